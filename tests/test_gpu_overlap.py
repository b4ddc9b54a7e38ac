"""Kernels that start while their predecessor drains: a chain in which each reads what the one before has just written, in
place and through reused buffers, gives the same bits with a synchronisation after every call, without one, on a side
stream and from a CUDA graph. Sizes from a single block to more than one wave."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(rows, d, heads, sync):
    from mflux_b200 import nn, ops

    g = torch.Generator(device="cuda").manual_seed(rows + d)

    def rnd(*shape, scale=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)

    def linear(n, k, bits):
        lin = nn.Linear(k, n, device="cuda")
        lin.weight.data.copy_(rnd(n, k, scale=0.02))
        layer = lin.to_quantized(bits=bits)
        layer.prepared()
        return layer

    qkv_l, out_l, up, down = (linear(3 * d, d, 4), linear(d, d, 8), linear(4 * d, d, 4), linear(d, 2 * d, 8))
    cond = linear(6 * d, 256, 8)
    x0, vec = rnd(2, rows, d, dtype=torch.float32), rnd(2, 256)
    ws = [rnd(128) for _ in range(4)]
    cs = torch.randn(rows, 64, 2, device="cuda", generator=g)
    nbuf, qkv = torch.empty(2, rows, d, device="cuda", dtype=torch.bfloat16), torch.empty(2, rows, 3 * d, device="cuda", dtype=torch.bfloat16)
    w = rnd(d)

    def step(x):
        def s(t):
            if sync:
                torch.cuda.synchronize()
            return t
        for _ in range(3):
            mod = s(cond(s(ops.vec_sum_act(vec, act="silu"))))
            s(ops.norm_modulate(x, mod[:, :d], mod[:, d:2 * d], out=nbuf))
            s(ops.qlinear(nbuf, *qkv_l._tensors(), bits=4, prepared=qkv_l.prepared(), out=qkv))
            s(ops.qknorm_rope(qkv, heads, *ws, rows // 3, cs))
            s(ops.fmha(qkv, heads, out=nbuf))
            s(out_l(nbuf, epilogue="gate_residual", gate=mod[:, 2 * d:3 * d], residual=x, out=x))
            s(ops.norm_modulate(x, mod[:, 3 * d:4 * d], mod[:, 4 * d:5 * d], out=nbuf))
            h = s(up(nbuf, epilogue="swiglu"))
            y = s(down(h))
            s(ops.norm_gate_residual(y, w, x, mod[:, 5 * d:], 1e-5, next_weight=w, next_out=nbuf, next_eps=1e-5))
            packed = s(ops.quantize_affine(nbuf[0].contiguous(), 64, 4))
            x[0] += s(ops.dequantize_affine(*packed, 64, 4)) * 0.01
        return x
    return step, x0


@pytest.mark.parametrize("rows,d,heads", [(1, 256, 2), (40, 256, 2), (300, 768, 6), (2100, 512, 4)])
def test_chain(lib_built, rows, d, heads):
    from mflux_b200 import ops

    step, x0 = _chain(rows, d, heads, True)
    ref = step(x0.clone())
    step, x0 = _chain(rows, d, heads, False)
    for _ in range(3):
        assert torch.equal(step(x0.clone()), ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = step(x0.clone())
    side.synchronize()
    assert torch.equal(y, ref)
    x = x0.clone()
    step(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step(x)
    for _ in range(2):
        x.copy_(x0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, ref)
    assert ops.poll_device_status() == 0
