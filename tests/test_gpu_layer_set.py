"""A one-GPU ``LayerSet`` in its concurrent schedule: each of its linears against the oracle, the flow between them, and
which of them went out as one launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DIM, FFN, BLOCKS = 256, 512, 2
FEEDS = {"self_o": "self_v", "cross_q": "self_o", "cross_o": "cross_v", "ffn_up": "cross_o", "ffn_down": "ffn_up"}


@pytest.fixture(scope="module")
def d(b200_lib):
    import dexter_labs_b200

    return dexter_labs_b200


def layer_set(bits, group, symmetric, relayout, dim=DIM, ffn=FFN):
    from dexter_labs_b200 import tp

    tp.PRESETS["test"] = (dim, ffn, BLOCKS)
    try:
        return tp.LayerSet.build("test", bits=bits, group_size=group, symmetric=symmetric, concurrent=True,
                                 relayout=relayout, weight_std=0.05)
    finally:
        del tp.PRESETS["test"]


def recorded(monkeypatch, ls):
    """(name, block) -> (input, output) of every linear that a pass runs, whichever way it is launched."""
    from dexter_labs_b200 import ops, tp

    names = {l.weight.scales.data_ptr(): (l.name, b) for b, row in enumerate(ls.layers) for l in row}
    seen, gemm, group = {}, tp._default_gemm, ops.gemm_group

    def one(x, w, max_ctas=0, **kwargs):
        y = gemm(x, w, max_ctas, **kwargs)
        assert seen.setdefault(names[w.scales.data_ptr()], (x, y))[1] is y, "run twice"
        return y

    def several(bits, problems, group_size, **kwargs):
        ys = group(bits, problems, group_size, **kwargs)
        for (x, _, scales, *_), y in zip(problems, ys or ()):
            assert seen.setdefault(names[scales.data_ptr()], (x, y))[1] is y, "run twice"
        return ys

    monkeypatch.setattr(tp, "_default_gemm", one)
    monkeypatch.setattr(ops, "gemm_group", several)
    ls.gemm = one
    return seen


@pytest.mark.parametrize("lead,ctx_lead,bits,group,symmetric,relayout,together", [  # together: blocks with one launch for five
    ((1,), (1,), 4, 128, True, True, 2),
    ((83,), (83,), 4, 64, False, True, 2),
    ((128,), (128,), 8, 128, False, True, 2),
    ((2, 20), (40,), 8, 0, True, True, 2),      # leading dimensions are flattened
    ((129,), (129,), 4, 128, True, True, 0),    # more than one token block
    ((40,), (17,), 4, 128, True, True, 1),      # a context of another length (a block's result has the context's)
    ((40,), (200,), 8, 128, True, True, 0),
    ((3, 7), (3, 7), 4, 128, True, False, 0),   # int4 in the reference layout
    ((0,), (0,), 4, 128, True, True, 0),        # no tokens
    ((2, 0), (2, 0), 8, 128, True, True, 0),
])
def test_concurrent_pass(lead, ctx_lead, bits, group, symmetric, relayout, together, d, oracle, monkeypatch):
    ls = layer_set(bits, group, symmetric, relayout)
    torch.manual_seed(len(lead) + lead[0])
    x = torch.randn(*lead, DIM, device="cuda").to(torch.bfloat16)
    ctx = torch.randn(*ctx_lead, DIM, device="cuda").to(torch.bfloat16)
    plain = {(l.name, b): d.ops.relayout_w4(l.weight.qweight, inverse=True) if l.layout == "b200" else l.weight.qweight
             for b, row in enumerate(ls.layers) for l in row}
    seen = recorded(monkeypatch, ls)
    y = ls.forward(x, ctx)
    assert len(seen) == ls.num_gemms
    assert ls.launches == ls.num_gemms - 4 * together
    assert y.shape == (*ctx_lead, DIM)
    assert torch.equal(y, seen["ffn_down", BLOCKS - 1][1])
    for b, row in enumerate(ls.layers):
        into = x if b == 0 else seen["ffn_down", b - 1][1]
        for l in row:
            a, got = seen[l.name, b]
            source = FEEDS.get(l.name)
            fed = seen[source, b][1] if source else ctx if l.name in ("cross_k", "cross_v") else into
            assert torch.equal(a, fed), (l.name, b)
            w = l.weight
            want = oracle.torch_wq_gemm(a, plain[l.name, b], w.scales, w.zeros, w.bias, w.group_size, bits).double()
            assert got.shape == want.shape
            if want.numel():
                assert (got.double() - want).abs().max() <= 1e-2 * want.abs().max(), (l.name, b)


def test_launches_are_those_of_the_last_pass(d):
    ls = layer_set(4, 128, True, True)
    x = torch.randn(24, DIM, device="cuda").to(torch.bfloat16)
    counts = []
    for concurrent in (True, True, False, True):
        ls.concurrent = concurrent
        ls.forward(x)
        counts.append(ls.launches)
    assert counts == [12, 12, 20, 12]
