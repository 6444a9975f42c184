"""The tau transforms' rule on the size of a launch: the pair-per-CTA kernels where one
wave takes all column pairs, the grouped kernels beyond.  The grouped kernels at every
frequency-grid size on a lattice of 1074 pairs against the radix-8 pair kernels, and
batches of points on both sides of the line (78 pairs a point, 296 CTAs a wave) against
single solves.

Tolerance: 1e-11 between tau kernels on the same slices, as the tilings' test has it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = (0.87, 0.3, (-0.15, 0.03, 0.0, 2.4))
MIXED = 3


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def solved(nk0, nw0, form):
    from tpsc_conductivity_b200.api import Green

    g = Green(nk0, nw0, M[0], M[1], 0.1, M[2])
    g.set_form(form)
    g.solve()
    return g


@pytest.mark.parametrize("nw0", [16, 32, 64, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("form", [1, MIXED])
def test_grouped_kernels_at_every_size(form, nw0):
    from tpsc_conductivity_b200 import _lib

    lib = _lib.load()
    a = solved(128, nw0, form)
    try:
        for kind in range(3):
            assert lib.tpsc_set_tau_tile(kind, nw0, 2) == 0
        c = solved(128, nw0, form)
    finally:
        for kind in range(3):
            assert lib.tpsc_set_tau_tile(kind, nw0, 0) == 0
    assert rel(a.chi0()["chiqw"], c.chi0()["chiqw"]) < 1e-11
    assert rel(a.vertex(), c.vertex()) < 1e-11
    assert rel(a.sigma(), c.sigma()) < 1e-11


@pytest.mark.parametrize("nw0", [16, 128, 1024])
@pytest.mark.parametrize("points", [1, 3, 4, 9])
def test_batches_on_both_sides_of_a_wave(points, nw0):
    from tpsc_conductivity_b200 import _lib, api

    a = solved(32, nw0, MIXED)
    res, st, _ = api.solve_points(np.tile([32, nw0, M[0], M[1], *M[2]], (points, 1)))
    assert not st.any()
    for k in ("Usp", "Uch", "mu", "dblOcc", "Sigma_inf"):
        v = a.scalars()[k]
        assert np.all(np.abs(res[:, _lib.SCALARS.index(k)] - v) < 1e-11 * max(1.0, abs(v))), k
