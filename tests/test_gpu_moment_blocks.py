"""The find_mu moments with several column blocks and tail columns per block: single
Newton-form solves of the widest lattice at short frequency axes (rows of many column
blocks in one thread block, tail series and tail term by term) against the reference
form's direct traces, and a batch whose blocks are wider than a single point's
against single solves.

Tolerance: 1e-9, far above the moments' truncation (1e-12) and the roots' 1e-15; the
batch 1e-11 as the other batch tests have it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk0,Nw0,T", [(256, 16, 0.05), (256, 16, 1.0), (256, 64, 0.2), (256, 256, 0.5),
                                       (128, 128, 0.3), (8, 16, 0.4)])
def test_newton_against_reference_traces(nk0, Nw0, T):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Green

    got = []
    for form in (_lib.FORM_REFERENCE, _lib.FORM_NEWTON):
        g = Green(nk0, Nw0, 0.88, T, 0.1, (-0.2, 0.0, 0.0, 1.5))
        g.set_form(form)
        g.solve()
        got.append(g.scalars())
    for k in ("mu", "trSG2"):
        if k in got[0]:
            assert abs(got[0][k] - got[1][k]) <= 1e-9 * max(1.0, abs(got[0][k])), k


def test_wide_batch_against_single_points():
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Green, solve_points

    rows = np.array([[64, 32, 0.75 + 0.02 * i, 0.3 + 0.01 * i, -0.1, 0.0, 0.0, 1.0 + 0.1 * i] for i in range(12)])
    res, st, _ = solve_points(rows)
    assert not st.any()
    names = list(_lib.SCALARS)
    for r, out in zip(rows[::5], res[::5]):
        g = Green(64, 32, r[2], r[3], 0.1, (r[4], 0.0, 0.0, r[7]))
        g.set_form(_lib.FORM_NEWTON | _lib.FORM_MIXED)
        g.solve()
        ref = g.scalars()
        for k in ("Usp", "Uch", "mu", "dblOcc"):
            assert abs(out[names.index(k)] - ref[k]) <= 1e-11 * max(1.0, abs(ref[k])), k
