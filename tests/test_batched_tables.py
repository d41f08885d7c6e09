"""The tables of orders and offsets that batched_posv takes: any sequence of what int() takes, as before it converted
lists at once."""
import numpy as np
import pytest

from oocdag_gb300 import _int_table


class OnAnotherDevice:
    """Like a GPU scalar: it has an integer value and no array form."""

    def __init__(self, v):
        self.v = v

    def __int__(self):
        return self.v

    def __array__(self, *args, **kwargs):
        raise TypeError("can't convert a device scalar to an array")


def _torch(values):
    import torch

    return torch.tensor(values)


VALUES = [16, 512, 3, 77]
FORMS = {
    "list": list(VALUES), "tuple": tuple(VALUES), "int32": np.array(VALUES, np.int32), "uint64": np.array(VALUES, np.uint64),
    "floats": [16.0, 512.0, 3.9, 77.0], "float array": np.array([16.0, 512.0, 3.9, 77.0]), "numpy scalars": [np.int64(x) for x in VALUES],
    "tensor": _torch(VALUES), "tensors": list(_torch(VALUES)), "tensors of one": list(_torch([[x] for x in VALUES])),
    "device scalars": [OnAnotherDevice(x) for x in VALUES], "mixed": [16, 512.0, np.uint8(3), OnAnotherDevice(77)], "text": ["16", "512", "3", "77"],
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_forms(form, dtype):
    got = _int_table(FORMS[form], 4, dtype)
    assert got.dtype == dtype and got.tolist() == VALUES


def test_large_offsets_are_exact():
    big = 2**53 + 1
    assert _int_table([0, big], 2, np.int64).tolist() == [0, big]
    assert _int_table([np.uint64(big), -1], 2, np.int64).tolist() == [big, -1]


def test_lengths():
    assert _int_table([], 0, np.int32).tolist() == [0]
    assert _int_table([5], 3, np.int64).tolist() == [5, 0, 0]
    with pytest.raises((ValueError, IndexError)):
        _int_table([1, 2, 3], 2, np.int32)
