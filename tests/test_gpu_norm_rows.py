"""Norm kernels whose blocks take several rows, of several samples: more rows than resident blocks, samples that change
inside a block's stride, the row lengths at which a kernel for shorter rows ends, every dtype of the row and of the vectors, strided rows. Against
float64; the bound is the bf16 rounding of the output (2^-8 of a value) and of float32 sums of up to 4096 terms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(x, shift, scale, weight, rms, eps):
    x = x.double()
    if not rms:
        x = x - x.mean(-1, keepdim=True)
    u = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    if weight is not None:
        u = u * weight.double()
    if scale is not None:
        u = u * (1 + scale.double()[:, None])
    return u if shift is None else u + shift.double()[:, None]


@pytest.mark.parametrize("batch,rows", [(1, 1), (1, 3001), (7, 401), (2500, 1)])
@pytest.mark.parametrize("d", [8, 3072, 3080, 4096])
@pytest.mark.parametrize("x_dtype,vec_dtype,form", [("float32", "bfloat16", "mod"), ("bfloat16", "bfloat16", "mod"),
                                                    ("float32", "bfloat16", "weight"), ("bfloat16", "bfloat16", "both"),
                                                    ("float32", "float32", "both"), ("bfloat16", "float16", "shift"),
                                                    ("float32", "bfloat16", "none")])
def test_norm_modulate(lib_built, batch, rows, d, x_dtype, vec_dtype, form):
    from mflux_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d + rows)
    vt = getattr(torch, vec_dtype)
    buf = torch.randn(batch, rows, d + 16, device="cuda", generator=g).to(getattr(torch, x_dtype))
    x = buf[..., 8:8 + d]                                   # strided rows
    mods = torch.randn(batch, 3 * d, device="cuda", generator=g).to(vt)
    shift = mods[:, d:2 * d] if form in ("mod", "both", "shift") else None
    scale = mods[:, :d] if form in ("mod", "both") else None
    weight = torch.randn(d, device="cuda", generator=g).to(vt) if form in ("weight", "both") else None
    rms = form == "weight"
    out = torch.full((batch, rows, d + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.norm_modulate(x, shift, scale, weight=weight, rms=rms, out=out[..., :d])
    ref = _ref(x, shift, scale, weight, rms, 1e-6)
    err = (out[..., :d].double() - ref).abs()
    assert (err <= 2 ** -8 * ref.abs() + 1e-3).all()        # terms of up to a few units cancel in u * (1 + scale) + shift
    assert (out[..., d:] == 7.0).all()


@pytest.mark.parametrize("rows,d", [(3, 64), (1700, 3840)])
@pytest.mark.parametrize("y_dtype,vec_dtype", [("bfloat16", "bfloat16"), ("float32", "bfloat16"), ("bfloat16", "float32")])
@pytest.mark.parametrize("two", [False, True])
def test_post_norm(lib_built, rows, d, y_dtype, vec_dtype, two):
    from mflux_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d)
    vt, b = getattr(torch, vec_dtype), 2
    y = torch.randn(b, rows, d, device="cuda", generator=g).to(getattr(torch, y_dtype))
    res = torch.randn(b, rows, d, device="cuda", generator=g)
    w, w2 = (torch.randn(d, device="cuda", generator=g).to(vt) for _ in range(2))
    gate, sc = (torch.randn(b, d, device="cuda", generator=g).to(vt) for _ in range(2))
    ref = res.double() + _ref(y, None, None, w, True, 1e-5) * gate.double()[:, None]
    nxt = torch.empty(b, rows, d, device="cuda", dtype=torch.bfloat16)
    kw = dict(next_weight=w2, next_scale=sc, next_out=nxt, next_eps=1e-5) if two else {}
    ops.norm_gate_residual(y, w, res, gate, 1e-5, **kw)
    assert ((res.double() - ref).norm() / ref.norm()).item() <= 1e-6
    if two:
        ref2 = _ref(ref, None, sc, w2, True, 1e-5)
        assert (nxt.double() - ref2).abs().le(2 ** -8 * ref2.abs() + 1e-4).all()
