"""Several linears in one launch (``ops.gemm_group``) against the oracle, at the edges of its tiles and of what it takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def d(b200_lib):
    import dexter_labs_b200

    return dexter_labs_b200


def problems(d, m, k, widths, bits, group, symmetric, layout, seed=0):
    torch.manual_seed(seed)
    xs = [torch.randn(m, k + 8, device="cuda").to(torch.bfloat16)[:, :k], torch.randn(m, k, device="cuda").to(torch.bfloat16)]
    out = []
    for i, n in enumerate(widths):
        q = d.quantize((torch.randn(n, k, device="cuda") * 0.02).to(torch.bfloat16), bits=bits, group_size=group,
                       symmetric=symmetric, bias=torch.randn(n, device="cuda").to(torch.bfloat16) if i % 2 else None)
        packed = d.ops.relayout_w4(q.qweight) if layout == "b200" else q.qweight
        out.append(((xs[i % 2], packed, q.scales, q.zeros, q.bias), q.qweight))
    return out


@pytest.mark.parametrize("m,k,widths,bits,group,why", [
    (1, 256, (16,), 4, 128, "one item, one cut tile"),
    (83, 3072, (3072,) * 5, 4, 128, "the five linears a block starts with"),
    (128, 512, (144, 16, 2048, 128, 272, 4096, 112, 256), 4, 64, "eight items, cut tiles, two scale strides"),
    (96, 256, (16384, 7168), 4, 256, "more tiles than SMs"),
    (100, 1024, (1040, 3072), 8, 128, "int8, three activation stages"),
    (9, 256, (128, 640), 8, 256, "int8, one scale per channel, half a sixteen of tokens"),
])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("layout", ["dexter", "b200"])
def test_group_matches_the_oracle(m, k, widths, bits, group, why, symmetric, layout, d, oracle):
    if layout == "b200" and bits == 8:
        pytest.skip("int8 has one layout")
    made = problems(d, m, k, widths, bits, group, symmetric, layout, seed=m)
    outs = d.ops.gemm_group(bits, [p for p, _ in made], group, layout=layout)
    again = d.ops.gemm_group(bits, [p for p, _ in made], group, layout=layout)
    for y, y2, ((x, _, s, z, b), plain) in zip(outs, again, made):
        want = oracle.torch_wq_gemm(x, plain, s, z, b, group, bits).double()
        assert (y.double() - want).abs().max() <= 1e-2 * want.abs().max(), why
        assert torch.equal(y, y2), why


def test_what_cannot_go_together_is_declined(d):
    a = [p for p, _ in problems(d, 8, 256, (128, 128), 4, 128, True, "dexter")]
    b = [p for p, _ in problems(d, 8, 256, (128,), 4, 128, False, "dexter")]
    assert d.ops.gemm_group(4, a + b, 128) is None  # with and without zero points
    assert d.ops.gemm_group(4, a * 5, 128) is None  # ten items
    assert d.ops.gemm_group(4, [p for p, _ in problems(d, 129, 256, (128,), 4, 128, True, "dexter")], 128) is None
    assert d.ops.gemm_group(4, [p for p, _ in problems(d, 8, 256, (136,), 4, 128, True, "dexter")], 128) is None
    cpu = tuple(None if t is None else t.cpu() for t in a[0])
    assert d.ops.gemm_group(4, [cpu], 128) is None


def test_group_in_a_graph_follows_its_inputs(d, oracle):
    made = problems(d, 40, 512, (256, 1024), 4, 128, True, "b200")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            outs = d.ops.gemm_group(4, [p for p, _ in made], 128, layout="b200")
        for x in {id(p[0]): p[0] for p, _ in made}.values():
            x.copy_(torch.randn(x.shape, device="cuda").to(torch.bfloat16))
        graph.replay()
    stream.synchronize()
    for y, ((x, _, s, z, b), plain) in zip(outs, made):
        want = oracle.torch_wq_gemm(x, plain, s, z, b, 128, 4).double()
        assert (y.double() - want).abs().max() <= 1e-2 * want.abs().max()


def test_leading_dimensions_are_flattened_and_no_tokens_are_declined(d):
    made = [p for p, _ in problems(d, 40, 256, (128, 256), 4, 128, True, "dexter")]
    want = d.ops.gemm_group(4, made, 128)
    flat = [p[0].contiguous() for p in made]
    strided = torch.stack((flat[0], flat[0]), 1)[:, 0].view(5, 8, 256)  # rows 512 apart, in two dimensions
    shapes = [(flat[0].view(2, 20, 256), (2, 20)), (strided, (5, 8)), (flat[0].view(1, 40, 256), (1, 40))]
    for x, lead in shapes:
        got = d.ops.gemm_group(4, [(x, *made[0][1:]), (flat[1], *made[1][1:])], 128)
        assert [y.shape for y in got] == [(*lead, 128), (40, 256)]
        assert torch.equal(got[0].view(40, 128), want[0]) and torch.equal(got[1], want[1])
    empty = flat[0][:0]
    for x in (empty, empty.view(3, 0, 256)):
        assert d.ops.gemm_group(4, [(x, *p[1:]) for p in made], 128) is None
    assert d.ops.gemm_group(4, [], 128) is None
    assert d.ops.gemm_group(4, [(flat[0][0], *made[0][1:])], 128)[0].shape == (128,)
