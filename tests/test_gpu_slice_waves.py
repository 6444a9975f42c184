"""The slice kernels' wide blocks (launches that one block an SM, two in FP32, holds at
once) against the plans' own blocks: single points on both sides of the line at every
lattice size against the FP64 form's oracle-checked path, and batches wide enough for
the plans' blocks against single solves.

Tolerances: the transform is the same, only the threads that fill and store a slice
differ, so batch and single solve agree as the other batch tests have it (1e-11); the
mixed form's stated 1e-6 against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = (0.87, 0.3, (-0.15, 0.03, 0.0, 2.4))


def solved(nk0, nw0, form):
    from tpsc_conductivity_b200.api import Green

    g = Green(nk0, nw0, M[0], M[1], 0.1, M[2])
    g.set_form(form)
    g.solve()
    return g


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


# Nw0 + 1 slices of G and Sigma, Nw0/2 + 1 of chi0 and V: wide for all (16, 128), for the
# latter (256: FP64; 512: FP32), for none (1024)
@pytest.mark.parametrize("nw0", [16, 128, 256, 512, 1024])
@pytest.mark.parametrize("nk0", [8, 16, 32, 64])
def test_forms_agree_on_both_sides(nk0, nw0):
    a, b = solved(nk0, nw0, 3), solved(nk0, nw0, 1)
    assert rel(a.chi0()["chiqw"], b.chi0()["chiqw"]) < 1e-6
    assert rel(a.vertex(), b.vertex()) < 1e-6
    assert rel(a.sigma(), b.sigma()) < 1e-6


@pytest.mark.parametrize("nk0,nw0", [(8, 64), (16, 64), (32, 64), (64, 64), (64, 256)])
def test_batches_beyond_the_line_equal_single_solves(nk0, nw0):
    from tpsc_conductivity_b200 import _lib, api

    a = solved(nk0, nw0, 3).scalars()
    res, st, _ = api.solve_points(np.tile([nk0, nw0, M[0], M[1], *M[2]], (12, 1)))
    assert not st.any()
    for k in ("Usp", "Uch", "mu", "dblOcc", "Sigma_inf"):
        assert np.all(np.abs(res[:, _lib.SCALARS.index(k)] - a[k]) < 1e-11 * max(1.0, abs(a[k]))), k
