"""QuantizedLinear as a torch module, on the CPU with the kernels' entry points replaced by recorders."""
import pytest
import torch

from mflux_b200 import nn, ops


@pytest.fixture
def calls(monkeypatch):
    """Records what reaches ops.qlinear."""
    seen = []

    def qlinear(x, wq, scales, biases, bias=None, **kw):
        seen.append({"weight": wq, "scales": scales, "biases": biases, "bias": bias, **kw})
        return x

    monkeypatch.setattr(ops, "qlinear", qlinear)
    monkeypatch.setattr(ops, "prepare_qlinear", lambda wq, s, b, bits, gs: (wq, s, b))
    return seen


class _Twice(torch.nn.Module):
    def forward(self, t):
        return 2 * t


def _layer(bias=True):
    layer = nn.QuantizedLinear(64, 8, bias=bias)
    layer.scales.data.fill_(3.0)
    if bias:
        layer.bias.data.fill_(5.0)
    return layer


@pytest.mark.parametrize("name,value", [("bias", 10.0), ("scales", 6.0)])
def test_parametrized_tensors_reach_the_call(calls, name, value):
    layer = _layer()
    torch.nn.utils.parametrize.register_parametrization(layer, name, _Twice())
    layer(torch.zeros(1, 64))
    assert (calls[0][name] == value).all()
    if name == "scales":
        assert (calls[0]["prepared"][1] == value).all()


def test_a_bias_that_is_a_plain_attribute_reaches_the_call(calls):
    layer = _layer()
    del layer.bias
    layer.bias = torch.full((8,), 7.0)
    layer(torch.zeros(1, 64))
    assert (calls[0]["bias"] == 7.0).all()


def test_plain_parameters_and_no_bias(calls):
    layer = _layer(bias=False)
    layer(torch.zeros(1, 64))
    assert calls[0]["bias"] is None and calls[0]["scales"] is layer.scales
    layer.scales.data = layer.scales.data * 2     # replaced: the prepared form is built again
    layer(torch.zeros(1, 64))
    assert (calls[1]["prepared"][1] == 6.0).all()


class _OwnBlob(nn.QuantizedLinear):
    def prepared(self):
        return "own", super().prepared()


def test_a_subclass_with_a_prepared_form_of_its_own(calls, monkeypatch):
    monkeypatch.setattr(ops, "plain_qlinear", lambda *a: "the base class's form")
    layer = _OwnBlob(64, 8)
    for _ in range(2):       # the second time the base class's form is there, too
        layer(torch.zeros(1, 64))
    assert [c["prepared"][0] for c in calls] == ["own", "own"]
    plain = _layer()
    plain(torch.zeros(1, 64))
    assert plain(torch.zeros(1, 64)) == "the base class's form"


class _Tagged(nn.QuantizedLinear):
    def __init__(self, *args, **kw):
        super().__init__(*args, **kw)
        self.tag = "set up"


@pytest.mark.parametrize("cls", [nn.QuantizedLinear, _Tagged])
@pytest.mark.parametrize("bias", [False, True])
def test_from_linear_runs_the_setup_of_a_subclass(monkeypatch, cls, bias):
    packed = (torch.ones(8, 8, dtype=torch.uint32), torch.full((8, 1), 2.0), torch.full((8, 1), 3.0))
    monkeypatch.setattr(ops, "quantize_affine", lambda w, gs, bits, mode: packed)
    linear = nn.Linear(64, 8, bias=bias)
    layer = cls.from_linear(linear, bits=4)
    assert type(layer) is cls and getattr(layer, "tag", "set up") == "set up" and (cls is not _Tagged or layer.tag)
    for name, t in zip(("weight", "scales", "biases"), packed):
        p = getattr(layer, name)
        assert isinstance(p, torch.nn.Parameter) and not p.requires_grad and p.data_ptr() == t.data_ptr()
    assert (layer.bias is None) if not bias else layer.bias.data_ptr() == linear.bias.data_ptr()
    assert set(layer.state_dict()) == {"weight", "scales", "biases"} | ({"bias"} if bias else set())
