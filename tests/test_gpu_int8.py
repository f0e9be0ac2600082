"""int8 weights inside the GEMM kernels, bit for bit: every byte, with scales and zero points on both sides of
what the short conversion takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SCALES = (0.0117, 1.9921875, 2.0, 300.0, 2.0 ** -100, -0.37, 0.0)
ZEROS = (0.0, 128.0, 255.0, 127.5, 256.0, -3.0, 100.25, 77.0)


@pytest.fixture(scope="module")
def d(b200_lib):
    import dexter_labs_b200

    return dexter_labs_b200


@pytest.mark.parametrize("m,n,why", [(8, 2048, "few tokens"), (96, 6144, "whole tiles or clusters"), (160, 8192, "CTA pairs")])
@pytest.mark.parametrize("zeros", [None, "whole", "any"])
def test_one_nonzero_activation_reads_back_the_exact_weight(m, n, why, zeros, d):
    k, group = 1024, 128
    gen = torch.Generator(device="cuda").manual_seed(m)
    q = torch.randint(0, 256, (k, n), dtype=torch.uint8, device="cuda", generator=gen)
    q[:, 0] = torch.arange(k, device="cuda") % 256  # every byte
    rows = torch.arange(k // group, device="cuda")[:, None] + torch.arange(n, device="cuda")[None, :] // 4
    # usual scales in the first half of the groups, all of them in the others: a warp takes either way
    usual = (torch.arange(k // group, device="cuda") < k // group // 2)[:, None]
    s = torch.where(usual, torch.tensor(0.0117, device="cuda"), torch.tensor(SCALES, device="cuda")[rows % len(SCALES)]).bfloat16()
    z = None
    if zeros is not None:
        pool = torch.tensor(ZEROS, device="cuda")[rows % len(ZEROS)]
        z = (torch.where(usual, pool.clamp(0, 255).floor(), pool) if zeros == "any" else pool.clamp(0, 255).floor()).bfloat16()
    full = lambda t: t.double().repeat_interleave(group, 0)
    # the difference and its product fit into 64 bits, so the rounding to bf16 is the only one
    want = ((q.double() - (128.0 if z is None else full(z))) * full(s)).bfloat16()
    for k0 in range(0, k, m):
        x = torch.zeros(m, k, device="cuda", dtype=torch.bfloat16)
        have = min(m, k - k0)
        x[torch.arange(have), k0 + torch.arange(have)] = 1
        y = d.w8a16(x, q, s, z, None, group)
        assert torch.equal(y[:have], want[k0:k0 + have]), why
        assert not y[have:].any()


@pytest.mark.parametrize("m,n,why", [(8, 2048, "few tokens"), (96, 6144, "whole tiles or clusters"), (160, 8192, "CTA pairs")])
@pytest.mark.parametrize("zero", [None, 3.0, 16.25])
def test_weights_are_exact_from_2_to_the_minus_120_on(m, n, why, zero, d):
    # every byte and every significand of the scale, two binades higher where the difference can be a quarter
    k, group = 256, 256
    low = -120 if zero is None or zero % 1 == 0 else -118
    q = torch.arange(256, dtype=torch.uint8, device="cuda")[:, None].repeat(1, n)
    s = ((1 + torch.arange(n, device="cuda") % 128 / 128).double() * 2.0 ** low).bfloat16()[None]
    z = None if zero is None else torch.full_like(s, zero)
    want = ((q.double() - (128.0 if zero is None else zero)) * s.double()).bfloat16()
    for k0 in range(0, k, m):
        have = min(m, k - k0)
        x = torch.zeros(m, k, device="cuda", dtype=torch.bfloat16)
        x[torch.arange(have), k0 + torch.arange(have)] = 1
        y = d.w8a16(x, q, s, z, None, group)
        assert torch.equal(y[:have], want[k0:k0 + have]), why
        assert not y[have:].any()


@pytest.mark.parametrize("k,n,group,m,why", [
    (256, 2048, 128, 8, "eight by eight weights a thread; few-token kernel"),
    (256, 33, 64, 8, "columns one by one; few-token kernel off the tiles"),
    (144, 24, 48, 8, "CUDA cores"),
    (1024, 6144, 1024, 96, "tcgen05 kernel"),
])
def test_zero_points_that_are_no_whole_numbers(k, n, group, m, why, d):
    pool = torch.tensor((127.5, 16.25, -0.375, 0.01171875, 300.0, 128.0, float("inf")), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(k)
    q = torch.randint(0, 256, (k, n), dtype=torch.uint8, device="cuda", generator=gen)
    rows = torch.arange(k // group, device="cuda")[:, None] + torch.arange(n, device="cuda")[None]
    z = pool[rows % len(pool)].bfloat16()
    s = (torch.rand(k // group, n, device="cuda", generator=gen) * 0.01 - 0.005).bfloat16()
    full = lambda t: t.double().repeat_interleave(group, 0)
    want = ((q.double() - full(z)) * full(s)).bfloat16()  # exact up to the rounding to bf16, as above
    # (as bytes: a zero has its sign)
    assert torch.equal(d.dequantize(q, s, z, group, 8).view(torch.int16), want.view(torch.int16)), why
    x = torch.zeros(m, k, device="cuda", dtype=torch.bfloat16)
    x[torch.arange(m), torch.arange(m) * (k // m)] = 1
    y, row = d.w8a16(x, q, s, z, None, group), want[::k // m][:m]
    finite = torch.isfinite(z).all(0)  # (an infinite weight times an activation of zero is no number)
    assert torch.equal(y[:, finite], row[:, finite]), why
