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


def _large_chain(batch, rows, sync):
    """The kernels that only larger calls reach, each behind the producer of what it reads: few rows over weights of 24 M
    and more (the ring form), prepared beforehand and in the call, the decoded form, attention with a key bias (both
    kernels by the rows), an adapter, a fork to another stream and its join, and the element-wise kernels."""
    from mflux_b200 import nn, ops
    from mflux_b200.lora import LoRALinear

    d, heads, wide = 3072, 24, 12288
    g = torch.Generator(device="cuda").manual_seed(rows)

    def rnd(*shape, scale=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)

    def linear(n, k, bits):
        lin = nn.Linear(k, n, device="cuda")
        lin.weight.data.copy_(rnd(n, k, scale=0.02))
        layer = lin.to_quantized(bits=bits)
        layer.prepared()
        return layer

    cond, cond8, qkv_l, out_l, up, down = (linear(3 * d, d, 4), linear(3 * d, d, 8), linear(3 * d, d, 4),
                                           linear(d, d, 8), linear(wide, d, 8), linear(d, wide, 4))
    lora = LoRALinear.from_linear(linear(d, d, 4), r=16, scale=0.5)
    lora.lora_A.data.copy_(rnd(d, 16, scale=d ** -0.5))
    lora.lora_B.data.copy_(rnd(16, d, scale=0.02))
    assert bool(ops._scratch_bytes(rows, batch, wide, d, 8)) == (rows > 200)   # which of the cases decode
    x0, vec0 = rnd(batch, rows, d, dtype=torch.float32), rnd(batch, d)
    mask = torch.zeros(batch, rows, device="cuda")
    mask[:, rows - rows // 5:] = 1e9
    zeros, gates = torch.zeros_like(mask), rnd(batch, rows, d)
    other = torch.cuda.Stream()

    def step(x):
        def s(t):
            if sync:
                torch.cuda.synchronize()
            return t
        vec = vec0.clone()
        qkv, nbuf = x.new_empty(batch, rows, 3 * d, dtype=torch.bfloat16), x.new_empty(x.shape, dtype=torch.bfloat16)
        side_out = torch.zeros_like(nbuf[:, :64])
        for i in range(3):
            mod = s(cond(s(ops.vec_sum_act(vec, act="silu"))))
            mod8 = s(ops.qlinear(s(ops.vec_sum_act(vec, mod[:, :d].contiguous(), act="tanh")), *cond8._tensors(), bits=8))
            s(ops.norm_modulate(x, mod[:, :d], mod8[:, d:2 * d], out=nbuf))
            here = torch.cuda.current_stream()
            other.wait_stream(here)
            with torch.cuda.stream(other):
                s(ops.qlinear(nbuf[:, :64], *out_l._tensors(), bits=8, prepared=out_l.prepared(), out=side_out))
            s(qkv_l(nbuf, out=qkv))
            here.wait_stream(other)
            bias = s(ops.euler_step(zeros, mask, -1.0 if i < 2 else -1e-9))
            s(ops.fmha(qkv, heads, out=nbuf, key_bias=bias))
            s(ops.act_mul(nbuf, gates))
            s(ops.gate_residual(s(out_l(nbuf)), mod[:, 2 * d:], x))
            s(lora(nbuf, epilogue="gate_residual", gate=mod8[:, 2 * d:], residual=x, out=x))
            s(ops.norm_modulate(x, mod[:, d:2 * d], mod8[:, :d], out=nbuf))
            y = s(down(s(up(nbuf, epilogue="gelu"))))
            y[:, :64] += side_out
            comb = s(ops.cfg_combine(y[..., :64].contiguous(), nbuf[..., :64].contiguous(), 2.0))
            x[..., :64] += comb
            s(ops.gate_residual(y, mod8[:, :d], x))
            vec = s(ops.vec_sum_act(vec, nbuf[:, 0].contiguous()))
        return x
    return step, x0


def _same_bits(form, *args):
    from mflux_b200 import ops

    step, x0 = form(*args, True)
    ref = step(x0.clone())
    assert torch.isfinite(ref).all()
    step, x0 = form(*args, False)
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


@pytest.mark.parametrize("rows,d,heads", [(1, 256, 2), (40, 256, 2), (300, 768, 6), (2100, 512, 4)])
def test_chain(lib_built, rows, d, heads):
    _same_bits(_chain, rows, d, heads)


@pytest.mark.parametrize("batch,rows", [(2, 200), (2, 1100), (1, 4608)])
def test_large_chain(lib_built, batch, rows):
    _same_bits(_large_chain, batch, rows)
