"""The native eager call: taken for plain calls, declined for everything else, same results."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def d(b200_lib):
    import dexter_labs_b200

    return dexter_labs_b200


def weight(d, n=144, k=256, bits=4, group=128):
    torch.manual_seed(n + k)
    w = (torch.randn(n, k, device="cuda") * 0.02).to(torch.bfloat16)
    return d.quantize(w, bits=bits, group_size=group, bias=torch.randn(n, device="cuda").to(torch.bfloat16))


def native(d, x, q, **over):
    a = dict(x=x, w=q.qweight, s=q.scales, z=q.zeros, b=q.bias) | over
    return d.ops._CALL(q.bits, a["x"], a["w"], a["s"], a["z"], a["b"], q.group_size, 0, 0, 0, False)


@pytest.mark.parametrize("bits,n", [(4, 144), (4, 141), (8, 144)])  # 141: a width that is never repacked
def test_native_call_equals_the_general_path(bits, n, d, monkeypatch):
    q = weight(d, n=n, bits=bits)
    x = torch.randn(2, 3, 256, device="cuda").to(torch.bfloat16)
    y = d.linear(x, q.qweight, q.bias, scales=q.scales, zeros=q.zeros, group_size=128, bits=bits)
    got = native(d, x, q)  # workspace and repacked copy exist by now
    assert got is not None and got.shape == (2, 3, n)
    monkeypatch.setattr(d.ops, "_CALL", None)
    want = d.linear(x, q.qweight, q.bias, scales=q.scales, zeros=q.zeros, group_size=128, bits=bits)
    assert torch.equal(got, want) and torch.equal(y, want)


def test_native_call_declines_what_is_not_plain(d):
    q = weight(d)
    x = torch.randn(6, 256, device="cuda").to(torch.bfloat16)
    d.w4a16(x, q.qweight, q.scales, q.zeros, q.bias, 128)
    assert native(d, x, q) is not None
    wide = torch.randn(6, 512, device="cuda").to(torch.bfloat16)
    assert native(d, wide[:, :256], q) is not None                    # a row stride is plain
    assert native(d, x.t().contiguous().t(), q) is None               # inner stride
    assert native(d, wide[:, 4:260], q) is None                       # alignment
    assert native(d, x[:, :128].contiguous(), q) is None              # K mismatch
    assert native(d, x[:0], q) is None
    assert native(d, x.float(), q) is None
    assert native(d, x.cpu(), q) is None
    assert native(d, x, q, s=q.scales.t().contiguous().t()) is None
    assert native(d, x, q, w=q.qweight.clone()) is None               # never seen: no repacked copy yet
    before = d.w4a16(x, q.qweight, q.scales, q.zeros, q.bias, 128)
    q.qweight.zero_()                                                 # modified in place: the copy is stale
    assert native(d, x, q) is None
    assert not torch.equal(d.w4a16(x, q.qweight, q.scales, q.zeros, q.bias, 128), before)


def test_pin_and_platform_still_rule_the_call(d, monkeypatch):
    from dexter_labs_b200 import platform, registry

    q = weight(d)
    x = torch.randn(6, 256, device="cuda").to(torch.bfloat16)

    def linear():
        return d.linear(x, q.qweight, q.bias, scales=q.scales, zeros=q.zeros, group_size=128, bits=4)

    linear()
    monkeypatch.setenv("DEXTER_KERNEL", "gemm/w4a16:no_such_kernel")
    with pytest.raises(LookupError):
        linear()
    monkeypatch.delenv("DEXTER_KERNEL")
    linear()
    try:
        platform.override_platform(platform._cpu_platform())
        with pytest.raises(LookupError):
            linear()
    finally:
        platform.override_platform(None)
    linear()
    assert registry.leading("gemm/w4a16") is d.ops._SPECS[4]


def test_tensors_that_throw_reach_the_general_path(d):
    # their accessors throw C++ exceptions, which must not leave the native entries
    q = weight(d)
    x = torch.randn(3, 6, 256, device="cuda").to(torch.bfloat16)
    d.w4a16(x[0], q.qweight, q.scales, q.zeros, q.bias, 128)

    def plain(t):
        return d.w4a16(t, q.qweight, q.scales, q.zeros, q.bias, 128)

    for bad in (lambda: torch.vmap(plain)(x), lambda: plain(x[0].to_sparse()),
                lambda: torch.vmap(lambda s: d.dequantize(q.qweight, s, q.zeros, 128, 4))(q.scales.expand(2, -1, -1).contiguous()),
                lambda: d.dequantize(q.qweight.to_sparse(), q.scales, q.zeros, 128, 4)):
        with pytest.raises((RuntimeError, NotImplementedError)):
            bad()
    # quantize goes on with tensor expressions, which vmap can follow
    w = (torch.randn(2, 48, 256, device="cuda") * 0.02).to(torch.bfloat16)
    try:
        codes = torch.vmap(lambda t: d.quantize(t, bits=8).qweight)(w)
    except RuntimeError:
        pass
    else:
        assert torch.equal(codes[1], d.quantize(w[1], bits=8).qweight)
    assert torch.isfinite(plain(x[0]).float()).all()


def expected(oracle, x, q):
    return oracle.torch_wq_gemm(x, q.qweight, q.scales, q.zeros, q.bias, q.group_size, q.bits).float()


def close(got, want):
    return ((got.float() - want).abs().max() / want.abs().max()).item() < 1e-2


def test_a_repacked_weight_is_waited_for_on_other_streams(d, oracle):
    q = weight(d, n=2048, k=2048)
    x = torch.randn(83, 2048, device="cuda").to(torch.bfloat16)
    want = expected(oracle, x, q)
    first, second, third = (torch.cuda.Stream() for _ in range(3))
    torch.cuda.synchronize()
    with torch.cuda.stream(second):
        d.linear(x, weight(d, n=2048, k=2048).qweight, scales=q.scales, zeros=q.zeros)  # allocations, code
    torch.cuda.synchronize()
    junk = torch.full((1 << 21,), 0xFF, dtype=torch.uint8, device="cuda")  # what the copy's memory held
    del junk

    def linear():
        return d.linear(x, q.qweight, q.bias, scales=q.scales, zeros=q.zeros, group_size=128, bits=4)

    with torch.cuda.stream(first):
        torch.cuda._sleep(40_000_000)  # about 20 ms: the repack is queued behind it
        y1 = linear()
    with torch.cuda.stream(second):
        ys = [linear() for _ in range(2)]
    torch.cuda.synchronize()
    assert all(close(y, want) for y in (y1, *ys))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=third):  # a capture cannot wait for the copy, but sees that it is there
        y3 = linear()
    assert third.cuda_stream in d.ops._relaid[id(q.qweight)][4]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y3, y1)
    # written anew at the same address: the graph follows the weight
    q.qweight.bitwise_xor_(0x11)
    with torch.cuda.stream(first):
        first.wait_stream(torch.cuda.current_stream())
        y1 = linear()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert close(y1, expected(oracle, x, q)) and torch.equal(y3, y1)


def test_weights_made_under_inference_mode(d, oracle):
    with torch.inference_mode():
        q = weight(d)
        x = torch.randn(83, 256, device="cuda").to(torch.bfloat16)
        for _ in range(2):
            y = d.linear(x, q.qweight, q.bias, scales=q.scales, zeros=q.zeros, group_size=128, bits=4)
            assert close(y, expected(oracle, x, q))
            q.qweight.bitwise_xor_(0x11)  # no version counter tells of this


def test_a_weight_whose_storage_is_exchanged(d, oracle):
    q, other = weight(d, n=160), weight(d, n=160, k=256)
    x = torch.randn(83, 256, device="cuda").to(torch.bfloat16)
    d.w4a16(x, q.qweight, q.scales, q.zeros, q.bias, 128)
    q.qweight.data = other.qweight.bitwise_xor(0x11)
    for _ in range(2):
        assert close(d.w4a16(x, q.qweight, q.scales, q.zeros, q.bias, 128), expected(oracle, x, q))


@pytest.mark.parametrize("bits", [4, 8])
def test_operands_that_are_elsewhere_or_too_small_raise(bits, d):
    q = weight(d, bits=bits)
    x = torch.randn(6, 256, device="cuda").to(torch.bfloat16)
    fn = d.w4a16 if bits == 4 else d.w8a16
    fn(x, q.qweight, q.scales, q.zeros, q.bias, 128)
    for at in range(4):
        ops = [q.qweight, q.scales, q.zeros, q.bias]
        ops[at] = ops[at].cpu()
        with pytest.raises(RuntimeError):
            fn(x, *ops, 128)
        if at < 3:
            with pytest.raises(RuntimeError):
                d.dequantize(*ops[:3], 128, bits)
        if at == 0:
            continue
        ops = [q.qweight, q.scales, q.zeros, q.bias]
        ops[at] = ops[at][..., :-1].contiguous()
        with pytest.raises(ValueError):
            fn(x, *ops, 128)
        if at < 3:
            with pytest.raises(ValueError):
                d.dequantize(*ops[:3], 128, bits)
    with pytest.raises(ValueError):
        fn(x, q.qweight, q.scales, q.zeros, q.bias, 64)  # twice the groups that are there
    with pytest.raises(RuntimeError):
        fn(x, q.qweight, q.scales, q.zeros.float(), q.bias, 128)
