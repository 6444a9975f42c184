"""The find_mu moments' tail summed term by term (cold points, whose series does not
converge at the axis's end) with several columns per half warp, one after the other: a
batch wide enough for eight against single solves, which take one.

Tolerance: 1e-11, as the other batch tests have it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 12 points x 525 blocks of 16 tail columns: eight a block at 256^2; rho / w_NO > 0.05 at
# every T for the columns far from the Fermi surface
@pytest.mark.parametrize("nk0,nw0,T", [(256, 1024, 0.03), (256, 64, 0.2), (128, 256, 0.05)])
def test_wide_batch_of_cold_points_against_single_solves(nk0, nw0, T):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Green, solve_points

    rows = np.array([[nk0, nw0, 0.75 + 0.02 * i, T * (1.0 + 0.02 * i), -0.1, 0.0, 0.0, 1.0 + 0.1 * i]
                     for i in range(12)])
    res, st, _ = solve_points(rows)
    assert not st.any()
    names = list(_lib.SCALARS)
    for r, out in zip(rows[::4], res[::4]):
        g = Green(nk0, nw0, r[2], r[3], 0.1, (r[4], 0.0, 0.0, r[7]))
        g.set_form(_lib.FORM_NEWTON | _lib.FORM_MIXED)
        g.solve()
        ref = g.scalars()
        for k in ("Usp", "Uch", "mu", "trSG2"):
            assert abs(out[names.index(k)] - ref[k]) <= 1e-11 * max(1.0, abs(ref[k])), k
