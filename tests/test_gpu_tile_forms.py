"""A tiling of chi0's tau transform that the tuners time in one form's precision does not
change the other's chi0: the FP64 forms' default is another kernel than the mixed
form's, and theirs keeps the order of its sums to the last bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chi0(g, form):
    g.set_form(form)
    g.calc_chiqw_FFT_spline()
    c = g.chi0()
    return np.concatenate([c["chiqw"].ravel(), c["chi0_inf"], c["chi0_inf2"]])


@pytest.mark.parametrize("tuned", ["fp64", "mixed"])
@pytest.mark.parametrize("tuner", ["tpsc_tune_tau_tiles", "tpsc_tune_tau_plans"])
@pytest.mark.parametrize("nk0,nw0", [(8, 16), (16, 64), (32, 256), (64, 1024)])
def test_tuning_one_form_leaves_the_others_chi0(nk0, nw0, tuner, tuned):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Green

    lib = _lib.load()
    mixed = _lib.FORM_NEWTON | _lib.FORM_MIXED
    mine, other = (_lib.FORM_NEWTON, mixed) if tuned == "fp64" else (mixed, _lib.FORM_NEWTON)
    g = Green(nk0, nw0, 0.875, 0.3, 0.1, (-0.15, 0.0, 0.0, 2.0))
    want = _chi0(g, other)
    try:
        g.set_form(mine)
        g.solve()
        ms = np.zeros(9)
        assert getattr(lib, tuner)(g.ctx.h, 3, ms.ctypes.data_as(C.POINTER(C.c_double))) == 0
        print(ms)
        assert np.array_equal(_chi0(g, other), want)
    finally:
        for kind in range(3):
            assert lib.tpsc_set_tau_tile(kind, nw0, 0) == 0
