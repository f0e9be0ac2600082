"""More than 128 tokens: the plans over CTA pairs and single CTAs, at the edges of blocks and tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-2


@pytest.fixture(scope="module")
def d(b200_lib):
    import dexter_labs_b200

    return dexter_labs_b200


@pytest.mark.parametrize("m,k,n,bits,group,symmetric,why", [
    (129, 256, 14336, 4, 128, True, "one block of 160, a tile per pair"),
    (160, 3072, 14336, 4, 128, False, "one full block, two accumulators do not fit"),
    (256, 256, 14448, 4, 64, True, "largest block; the last pair tile has 112 columns, its second CTA none"),
    (257, 1024, 9232, 4, 128, False, "two blocks, last tile of 16 columns"),
    (512, 768, 9216, 8, 768, True, "blocks of 256, int8 per channel"),
    (700, 1280, 5136, 8, 128, False, "several rounds of tiles, int8 with zero points"),
    (913, 3072, 3072, 4, 128, True, "six blocks, one round"),
    (1000, 640, 10000, 4, 128, False, "many rounds with one accumulator, ragged last block and tile"),
    (2049, 256, 2048, 4, 128, True, "nine blocks"),
])
def test_many_tokens(m, k, n, bits, group, symmetric, why, d, oracle):
    torch.manual_seed(m)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, device="cuda") * 0.02).to(torch.bfloat16)
    q = d.quantize(w, bits=bits, group_size=group, symmetric=symmetric,
                   bias=torch.randn(n, device="cuda").to(torch.bfloat16))
    fn = d.w4a16 if bits == 4 else d.w8a16
    want = oracle.torch_wq_gemm(x, q.qweight, q.scales, q.zeros, q.bias, group, bits).float()
    for cap in (0, 40):
        y = fn(x, q.qweight, q.scales, q.zeros, q.bias, group, max_ctas=cap)
        assert (y.float() - want).abs().max() / want.abs().max() < TOL, (why, cap)
        assert torch.equal(fn(x, q.qweight, q.scales, q.zeros, q.bias, group, max_ctas=cap), y), "not deterministic: " + why
    gelu = (d.ops.w4a16_gelu if bits == 4 else d.ops.w8a16_gelu)(x, q.qweight, q.scales, q.zeros, q.bias, group)
    ref = torch.nn.functional.gelu(want, approximate="tanh")
    assert (gelu.float() - ref).abs().max() / ref.abs().max() < TOL, why
    assert d.ops.last_status() == 0
