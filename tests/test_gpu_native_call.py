"""QuantizedLinear.__call__ in native code against the same call through ops.qlinear: equal bits, equal refusals, and None
(the Python path) for every form it does not cover."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(n=256, k=192, bits=4, bias=True, seed=0):
    from mflux_b200 import nn

    g = torch.Generator(device="cuda").manual_seed(seed)
    lin = nn.Linear(k, n, bias=bias, device="cuda")
    lin.weight.data.copy_((torch.randn(n, k, device="cuda", generator=g) * 0.02).to(torch.bfloat16))
    if bias:
        lin.bias.data.copy_(torch.randn(n, device="cuda", generator=g).to(torch.bfloat16))
    layer = lin.to_quantized(bits=bits)
    layer.prepared()
    return layer


def _native(layer, x, epilogue=None):
    from mflux_b200 import ops

    w, s, b, bias = layer._tensors()
    return ops.plain_qlinear(x, w, s, b, bias, layer._prepared, layer.bits, layer.group_size, epilogue)


def _python(layer, x, epilogue=None):
    from mflux_b200 import ops

    w, s, b, bias = layer._tensors()
    return ops.qlinear(x, w, s, b, bias, bits=layer.bits, epilogue=epilogue, prepared=layer.prepared())


@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("form", ["1d", "1row", "16rows", "17rows", "batch", "batch of one", "strided", "expanded"])
@pytest.mark.parametrize("epilogue", [None, "gelu", "silu", "swiglu"])
def test_equal_bits(lib_built, bits, bias, form, epilogue):
    from mflux_b200 import ops

    layer = _layer(bits=bits, bias=bias)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(3, 40, 192 + 64, device="cuda", generator=g).to(torch.bfloat16)
    x = {"1d": x[0, 0, :192].clone(), "1row": x[0, :1, :192].clone(), "16rows": x[0, :16, :192],
         "17rows": x[0, :17, 64:], "batch": x[..., :192].contiguous(), "batch of one": x[:1, :, :192].contiguous(),
         "strided": x[:, ::2, 64:], "expanded": x[:1, :, :192].expand(3, 40, 192)}[form]
    before = ops.LAUNCHES[0]
    y = _native(layer, x, epilogue)
    assert y is not None and ops.LAUNCHES[0] == before + 1
    ref = _python(layer, x, epilogue)
    assert y.shape == ref.shape and y.dtype == ref.dtype and y.stride() == ref.stride() and torch.equal(y, ref)
    assert torch.equal(layer(x, epilogue=epilogue), ref)


def test_forms_left_to_python(lib_built):
    from mflux_b200 import ops

    layer = _layer()
    x = torch.randn(2, 5, 192, device="cuda").to(torch.bfloat16)

    class Sub(torch.Tensor):
        pass

    for other in (x.float(), x.half(), x.transpose(0, 1).contiguous().transpose(0, 1)[..., ::1].mT.contiguous().mT,
                  x.unsqueeze(0), x.as_subclass(Sub)):
        assert _native(layer, other) is None
    assert torch.equal(layer(x.float()), _python(layer, x))
    assert torch.equal(layer(x.unsqueeze(0))[0], _python(layer, x))
    assert _native(layer, torch.nn.Parameter(x, requires_grad=False)) is not None
    with torch.inference_mode():
        xi = torch.ones(2, 192, device="cuda", dtype=torch.bfloat16)
        assert torch.equal(layer(xi), _python(layer, xi))
    y = layer(x.clone().requires_grad_())
    assert not y.requires_grad
    # enough rows for the two-launch form: scratch is the Python path's
    big = _layer(n=12288, k=3072, bits=8)
    rows = torch.randn(4608, 3072, device="cuda").to(torch.bfloat16)
    assert ops._scratch_bytes(4608, 1, 12288, 3072, 8) > 0
    assert _native(big, rows) is None
    assert torch.equal(big(rows), _python(big, rows))


def test_refusals(lib_built):
    layer = _layer()
    x = torch.randn(5, 192, device="cuda").to(torch.bfloat16)
    with pytest.raises(ValueError):
        layer(x[:, :128])
    with pytest.raises(ValueError):
        layer(x[:0])
    with pytest.raises(ValueError):
        layer(torch.randn(5, 196, device="cuda").to(torch.bfloat16)[:, 2:194])     # rows off the 16-byte boundary
    with pytest.raises(RuntimeError):
        layer(x.cpu())
    with pytest.raises(KeyError):
        layer(x, epilogue="relu")
    with pytest.raises(ValueError):
        layer(x, epilogue="gate_residual")
    assert torch.equal(layer(x), _python(layer, x))


def test_changed_weight_is_prepared_again(lib_built):
    a, b = _layer(seed=1), _layer(seed=2)
    x = torch.randn(5, 192, device="cuda").to(torch.bfloat16)
    ya, yb = a(x), b(x)
    assert not torch.equal(ya, yb)
    a.weight.data.copy_(b.weight.data)
    a.scales.data.copy_(b.scales.data)
    a.biases.data.copy_(b.biases.data)
    a.bias.data.copy_(b.bias.data)
    for p in (a.weight, a.scales, a.biases):
        torch._C._increment_version([p])          # .data leaves the counter alone
    assert torch.equal(a(x), yb)
    a.weight = torch.nn.Parameter(_layer(seed=1).weight.data, requires_grad=False)      # replaced
    assert not torch.equal(a(x), yb)


def test_streams_and_capture(lib_built):
    layer = _layer()
    x = torch.randn(5, 192, device="cuda").to(torch.bfloat16)
    ref = layer(x)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = layer(x)
    side.synchronize()
    assert torch.equal(y, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x)
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


def test_other_threads_run_while_a_launch_waits(lib_built):
    """With a full launch queue a call waits for the device; another Python thread goes on meanwhile."""
    import threading
    import time

    layer = _layer()
    x = torch.randn(2, 192, device="cuda").to(torch.bfloat16)
    layer(x)
    done, gaps = threading.Event(), []

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(1e-3)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    torch.cuda.synchronize()
    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(3_000_000_000)       # one and a half seconds and more
        longest = 0.0
        for _ in range(3000):                  # more launches than the queue holds
            begin = time.perf_counter()
            layer(x)
            longest = max(longest, time.perf_counter() - begin)
    finally:
        done.set()
        thread.join()
    torch.cuda.synchronize()
    assert longest > 0.5, "no call had to wait"
    assert max(gaps) < longest / 2, (max(gaps), longest)
