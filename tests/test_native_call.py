"""The native form of a quantized linear's call refuses (returns None) what is not a plain CUDA call, without a GPU."""
import torch


def test_none_for_anything_else(lib_built):
    from mflux_b200 import _lib

    _lib.load()
    linear = _lib._host().linear
    x, w = torch.zeros(2, 64, dtype=torch.bfloat16), torch.zeros(8, 8, dtype=torch.int32)
    s = torch.zeros(8, 1, dtype=torch.bfloat16)
    blob = torch.zeros(1024, dtype=torch.uint8)
    key = (w.data_ptr(), w._version, s.data_ptr(), s._version, s.data_ptr(), s._version)
    for args in ((x, w, s, s, None, (key, blob), 4, 64, 0), (None,) * 6 + (4, 64, 0), (x, w, s, s, None, None, 4, 64, 0),
                 (1, 2, 3, 4, 5, (6, 7), 4, 64, 0), (x.to("meta"), w, s, s, None, (key, blob), 4, 64, 0)):
        assert linear(*args) is None
