"""Scalar arguments are packed as their DSL types convert them, on the direct route too."""
import ctypes
import types

import numpy as np
import pytest

from xgrid_gb300.native import NativeKernel
from xgrid_gb300.types import Floating, Integer


def _kernel(kinds):
    k = NativeKernel.__new__(NativeKernel)
    args = [(f"a{i}", t) for i, t in enumerate(kinds)]
    k.module = types.SimpleNamespace(value_args=args)
    k.args_type = type("args", (ctypes.Structure,), {"_fields_": [(n, t.ctype) for n, t in args]})
    k.plain_values = True
    return k


@pytest.mark.parametrize("value", [1, True, 1.5, -2**40, np.float32(1.5), np.int64(7), np.array(2.0), "x", None,
                                   ctypes.c_float(1.0), ctypes.c_double(1.0), ctypes.c_int(1)])
@pytest.mark.parametrize("kind", [Floating(4), Floating(8), Integer(4)], ids=["float", "double", "int"])
def test_values_are_converted_or_refused_as_serialize_does(kind, value):
    k = _kernel([kind, kind])
    try:
        want = bytes(kind.serialize(value))
    except TypeError:
        with pytest.raises(TypeError):
            k.pack([1, value])
        return
    assert bytes(k.pack([1, value])) == bytes(kind.serialize(1)) + want
