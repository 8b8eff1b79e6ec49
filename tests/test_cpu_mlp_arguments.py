"""The forward pass refuses networks that its weights do not fit, before
anything is launched (no GPU needed)."""
import ctypes

import pytest

from cudadsmc_b200 import lib
from cudadsmc_b200._capi import Mlp

ERR_ARG = 1


@pytest.mark.parametrize("change", [dict(depth=0, hidden=8), dict(depth=0, hidden=32), dict(depth=-1),
                                    dict(n_in=17), dict(n_in=0)])
def test_refused(change):
    shape = dict(n_in=4, in_pad=16, hidden=64, depth=2, modes=32, fields=64)
    shape.update(change)
    net = Mlp(*[shape[k] for k in ("n_in", "in_pad", "hidden", "depth", "modes", "fields")])
    x = (ctypes.c_float * 4)()
    ptrs = (ctypes.c_void_p * 2)(16, 16)
    assert lib().dsmc_mlp_forward(ctypes.byref(net), x, 1, 16, None, ptrs, 16, None, None) == ERR_ARG
