"""The two-launch form of the quantized linear (decode once to bf16, then a bf16 contraction), which calls with many
activation rows take: on ragged tiles and slices, with every epilogue and the low-rank term, against the one-launch
kernel and the float32 oracle, and the rule that chooses it."""
import pytest
import torch

from oracle import quant

pytestmark = pytest.mark.gpu


def _both(monkeypatch, call, n, k):
    """The same call in the two-launch and in the one-launch form, whatever the rule says for its size."""
    from mflux_b200 import ops

    outs = []
    for need in (2 * n * k, 0):
        with monkeypatch.context() as m:
            m.setattr(ops, "_scratch_bytes", lambda *a, need=need: need)
            outs.append(call())
    torch.cuda.synchronize()
    return outs


@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("m", [17, 256, 257, 1300])
@pytest.mark.parametrize("nk", [(8, 64), (264, 192), (520, 1600), (1000, 4672)])
def test_matches_oracle_and_one_launch_kernel(lib_built, monkeypatch, bits, m, nk):
    """K = 64 (one stage), 192, 1600 (ragged 1536-wide decode slice), 4672 (four slices); N = 8, 264, 520, 1000 (ragged
    tiles); less than a tile of rows, one, one more, several. Same bf16 weights and the same order of products: the two
    kernels agree to the bit."""
    from mflux_b200 import ops

    n, k = nk
    g = torch.Generator(device="cpu").manual_seed(bits + n)
    w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    b = torch.randn(n, generator=g).to(torch.bfloat16)
    wq, s, bi = ops.quantize_affine(w.cuda(), 64, bits)
    buf = torch.full((m + 8, n + 8), 7.0, dtype=torch.float32, device="cuda")
    prep = ops.prepare_qlinear(wq, s, bi, bits)
    got, one = _both(monkeypatch, lambda: ops.qlinear(x.cuda(), wq, s, bi, b.cuda(), bits=bits, prepared=prep,
                                                      out=buf[:m, :n]).clone(), n, k)
    assert ops.poll_device_status() == 0
    assert torch.equal(got, one)
    assert (buf[m:] == 7.0).all() and (buf[:, n:] == 7.0).all()
    ref = quant.qlinear(x, wq.cpu().numpy(), s.float().cpu().numpy(), bi.float().cpu().numpy(), b, 64, bits)
    assert quant.rel_l2(got, ref) <= 1e-2


@pytest.mark.parametrize("epi", ["gelu", "gelu_approx", "silu", "gate_residual", "swiglu"])
@pytest.mark.parametrize("lora", [0, 16, 72, 200])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_epilogues_samples_and_adapters(lib_built, monkeypatch, epi, lora, dtype):
    """Samples that are row slices of a longer buffer, each with its own ragged tile; ranks inside one slab and across
    two and four. Both kernels run the adapters' products after the layer's, 16 columns at a time in the same order."""
    from mflux_b200 import ops

    bits, n, k, bsz, rows = 4, 528, 320, 3, 301
    g = torch.Generator(device="cpu").manual_seed(lora + len(epi))
    w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16)
    seq = torch.randn(bsz, rows + 7, k, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
    wq, s, bi = ops.quantize_affine(w.cuda(), 64, bits)
    kw = {}
    if epi == "gate_residual":
        kw = {"gate": torch.randn(bsz, n, generator=g).to(torch.bfloat16).cuda(),
              "residual": torch.randn(bsz, rows, n, generator=g).to(dtype).cuda()}
    if lora:
        ld = -(-lora // 64) * 64
        t = torch.zeros(bsz, rows, ld)
        t[..., :lora] = torch.randn(bsz, rows, lora, generator=g)
        lb = torch.zeros(n, ld)
        lb[:, :lora] = torch.randn(n, lora, generator=g) * 0.05
        kw |= {"lora_t": t.to(torch.bfloat16).cuda(), "lora_b": lb.to(torch.bfloat16).cuda(), "lora_r": lora}
    got, one = _both(monkeypatch, lambda: ops.qlinear(seq[:, 5:5 + rows], wq, s, bi, b, bits=bits, epilogue=epi,
                                                      out_dtype=dtype, **kw), n, k)
    assert ops.poll_device_status() == 0
    assert got.shape == (bsz, rows, n // 2 if epi == "swiglu" else n) and got.dtype == dtype
    assert torch.isfinite(got.float()).all()
    assert torch.equal(got, one)


def test_short_or_misaligned_scratch_is_not_used(lib_built):
    from ctypes import byref

    from mflux_b200 import _lib, ops

    lib = _lib.load()
    m, n, k, bits = 40, 264, 128, 4
    g = torch.Generator(device="cpu").manual_seed(3)
    w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16).cuda()
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    wq, s, bi = ops.quantize_affine(w, 64, bits)
    prep = ops.prepare_qlinear(wq, s, bi, bits)
    want = ops.qlinear(x, wq, s, bi, None, bits=bits, prepared=prep)
    need = 2 * n * k
    for offset, size, used in ((0, need, True), (0, need - 1, False), (16, need, False)):
        scratch = torch.full((need + 256,), 0x5A, dtype=torch.uint8, device="cuda")
        y = torch.empty_like(want)
        a = _lib.QLinearArgs()
        a.x, a.x_row_stride, a.rows, a.batch, a.K, a.N = x.data_ptr(), k, m, 1, k, n
        a.bits, a.group_size, a.prepared = bits, 64, prep.data_ptr()
        a.y, a.y_dtype, a.y_row_stride = y.data_ptr(), _lib.BF16, n
        rc = lib.mfx_qlinear_ex_scratch(byref(a), scratch.data_ptr() + offset, size,
                                        torch.cuda.current_stream().cuda_stream)
        _lib.check(rc, "mfx_qlinear_ex_scratch")
        torch.cuda.synchronize()
        assert torch.equal(y, want)
        assert bool((scratch[:need] == 0x5A).all()) != used and (scratch[need:] == 0x5A).all()


@pytest.mark.parametrize("bits,rows", [(4, 18432), (8, 2560)])
def test_rule_and_call_through_it(lib_built, bits, rows):
    """The rule asks for scratch on a wide layer with many rows and not below its limits; a call that it sends through
    the two launches, prepared on the fly."""
    from mflux_b200 import _lib, ops

    lib = _lib.load()
    n, k = 9216, 3072
    assert lib.mfx_qlinear_scratch_bytes(rows, n, k, bits) == 2 * n * k
    assert lib.mfx_qlinear_scratch_bytes(1024, n, k, bits) == 0
    assert lib.mfx_qlinear_scratch_bytes(rows, n, 64, bits) == 0
    assert lib.mfx_qlinear_scratch_bytes(rows, n, 100, bits) == 0
    assert lib.mfx_qlinear_scratch_bytes(rows, n, k, 7) == 0
    g = torch.Generator(device="cpu").manual_seed(bits)
    w = (torch.randn(n, k, generator=g) * 0.02).to(torch.bfloat16)
    x = torch.randn(rows, k, generator=g).to(torch.bfloat16).cuda()
    wq, s, bi = ops.quantize_affine(w.cuda(), 64, bits)
    before = ops.LAUNCHES[0]
    y = ops.qlinear(x, wq, s, bi, None, bits=bits)
    assert ops.LAUNCHES[0] - before == 4      # two to prepare, decode, contraction
    wd = ops.dequantize_affine(wq, s, bi, 64, bits, torch.float32).cpu()
    ref = x[::97].float().cpu() @ wd.t()
    assert quant.rel_l2(y[::97], ref.numpy()) <= 1e-2


def test_no_room_for_scratch_runs_without_it(lib_built, monkeypatch):
    from mflux_b200 import ops

    n, k = 264, 128
    g = torch.Generator(device="cpu").manual_seed(4)
    w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16).cuda()
    x = torch.randn(40, k, generator=g).to(torch.bfloat16).cuda()
    wq, s, bi = ops.quantize_affine(w, 64, 4)
    prep = ops.prepare_qlinear(wq, s, bi, 4)
    want = ops.qlinear(x, wq, s, bi, None, bits=4, prepared=prep)
    monkeypatch.setattr(ops, "_scratch_bytes", lambda *a: 1 << 50)      # a petabyte: the allocator refuses on the host
    monkeypatch.setattr(ops, "_REFUSED", {})
    before, refused = ops.LAUNCHES[0], torch.cuda.memory_stats()["num_ooms"]
    for _ in range(3):
        assert torch.equal(ops.qlinear(x, wq, s, bi, None, bits=4, prepared=prep), want)
    assert ops.LAUNCHES[0] - before == 3
    assert torch.cuda.memory_stats()["num_ooms"] - refused == 1      # asked once, not on every call


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("epi", [None, "gelu", "gate_residual", "lora"])
def test_several_bands_and_three_tiles_per_pair(lib_built, monkeypatch, bits, epi):
    """A bf16 weight past one band (37 column tiles, 19 and 18 to a band) and 222 tiles for 74 CTA pairs: accumulators,
    ring and bias vectors in turn. All rows, to the bit against the one-launch kernel."""
    from mflux_b200 import ops

    m, n, k = 6 * 256 - 50, 37 * 256 - 248, 3072
    g = torch.Generator(device="cuda").manual_seed(bits)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(n, generator=g, device="cuda")
    wq, s, bi = ops.quantize_affine(w, 64, bits)
    kw = {"out_dtype": torch.float32}
    if epi == "gate_residual":
        kw = {"epilogue": epi, "gate": b[None], "residual": torch.randn(m, n, generator=g, device="cuda")}
    elif epi == "lora":
        t = torch.zeros(m, 128, device="cuda", dtype=torch.bfloat16)
        lb = torch.zeros(n, 128, device="cuda", dtype=torch.bfloat16)
        t[:, :72] = torch.randn(m, 72, generator=g, device="cuda")
        lb[:, :72] = torch.randn(n, 72, generator=g, device="cuda") * 0.05
        kw |= {"lora_t": t, "lora_b": lb, "lora_r": 72}
    elif epi:
        kw |= {"epilogue": epi}
    two, one = _both(monkeypatch, lambda: ops.qlinear(x, wq, s, bi, b, bits=bits, **kw), n, k)
    assert ops.poll_device_status() == 0
    assert torch.isfinite(two).all() and torch.equal(two, one)
