"""A key bias that is zero in some 32- and 64-key pieces of the key loop and not in others: the kernels take the plain form
of a piece of zeros. Biases stand at the edges of the pieces, in one half of a tile only, behind the last full tile; some
are positive (the row maximum grows in a biased piece), some mask; scales of either sign. Against float64. The bound is
the bf16 rounding of P and of the output (2^-9 each, relative) over averages of values: 5e-3 in the 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu

PLACES = {"first": [(0, 1, 3.0)], "edges": [(31, 33, -2.0), (63, 65, 4.0), (127, 129, -1e9)],
          "second half": [(64, 128, -1e9), (200, 201, 30.0)], "leading": [(0, 160, -1e9)], "last": [(-1, None, 9.0)]}


@pytest.mark.parametrize("kernel", ["pair", "pingpong"])
@pytest.mark.parametrize("seq", [225, 1030])
@pytest.mark.parametrize("places,scale", [(name, 128 ** -0.5) for name in PLACES] + [("edges", -0.05)])
def test_mixed_pieces(lib_built, monkeypatch, kernel, seq, places, scale):
    from mflux_b200 import ops

    monkeypatch.setenv("MFX_FMHA_KERNEL", kernel)
    g = torch.Generator(device="cuda").manual_seed(seq)
    heads, batch = 2, 2
    qkv = torch.randn(batch, seq, 3 * heads * 128, device="cuda", generator=g).to(torch.bfloat16)
    kb = torch.zeros(batch, (seq + 3) // 4 * 4, device="cuda")[:, :seq]
    for first, last, value in PLACES[places]:
        kb[1, first:last] = value          # sample 0 stays without
    out = ops.fmha(qkv, heads, scale=scale, key_bias=kb)
    assert ops.poll_device_status() == 0
    for b in range(batch):
        for h in range(heads):
            q, k, v = (qkv[b, :, (i * heads + h) * 128:(i * heads + h + 1) * 128].double() for i in range(3))
            ref = torch.softmax(q @ k.t() * scale + kb[b].double(), dim=-1) @ v
            got = out[b, :, h * 128:(h + 1) * 128].double()
            assert ((got - ref).norm() / ref.norm()).item() <= 5e-3
