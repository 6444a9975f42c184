"""The grouped tau transforms (several column pairs per CTA, groups of one thread
and more, a last CTA with pairs to spare) against the pair-per-CTA kernels of the
FP64 form and the radix-8 plan: the mixed form's chi0, V and Sigma at every
frequency-grid size, and the same points through the shape groups.

Tolerances: the mixed form's stated 1e-6 against FP64 (its FP32 slices); 1e-11
between tau kernels on the same slices, as the tilings' test has it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = (0.87, 0.3, (-0.15, 0.03, 0.0, 2.4))


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def solved(nk0, nw0, form):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Green

    g = Green(nk0, nw0, M[0], M[1], 0.1, M[2])
    g.set_form({"fp64": _lib.FORM_REFERENCE, "mixed": _lib.FORM_NEWTON | _lib.FORM_MIXED}[form])
    g.solve()
    return g


@pytest.mark.parametrize("nw0", [16, 32, 64, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("nk0", [8, 32])
def test_every_frequency_grid(nk0, nw0):
    from tpsc_conductivity_b200 import _lib, api

    a, b = solved(nk0, nw0, "mixed"), solved(nk0, nw0, "fp64")
    assert rel(a.chi0()["chiqw"], b.chi0()["chiqw"]) < 1e-6
    assert rel(a.vertex(), b.vertex()) < 1e-6
    assert rel(a.sigma(), b.sigma()) < 1e-6
    lib = _lib.load()
    try:
        for kind in range(3):
            assert lib.tpsc_set_tau_tile(kind, nw0, 2) == 0
        c = solved(nk0, nw0, "mixed")
    finally:
        for kind in range(3):
            assert lib.tpsc_set_tau_tile(kind, nw0, 0) == 0
    assert rel(a.chi0()["chiqw"], c.chi0()["chiqw"]) < 1e-11
    assert rel(a.vertex(), c.vertex()) < 1e-11
    assert rel(a.sigma(), c.sigma()) < 1e-11
    res, st, _ = api.solve_points(np.tile([nk0, nw0, M[0], M[1], *M[2]], (3, 1)))
    assert not st.any()
    for k in ("Usp", "Uch", "mu", "dblOcc", "Sigma_inf"):
        v = a.scalars()[k]
        assert np.all(np.abs(res[:, _lib.SCALARS.index(k)] - v) < 1e-11 * max(1.0, abs(v))), k
