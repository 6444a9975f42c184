"""The reference form's root searches through slots on grids of a few blocks with many
column blocks each (the cap of many contexts, values kept in shared memory or read at
every evaluation) against one block per column block: the sums are taken in the order
of the column blocks, so the results are equal to the last bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [(8, 16, 0.9, 0.4), (16, 32, 0.85, 0.3), (32, 128, 1.1, 0.2), (64, 64, 0.8, 0.3), (64, 1024, 0.9, 0.1),
        (128, 32, 0.9, 0.4)]


def test_capped_grids_give_the_same_bits():
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Batch, Green

    rows = np.array([[k, w, n, T, -0.15, 0.0, 0.0, 2.0] for k, w, n, T in ROWS])
    res, st, _ = Batch(32).solve(rows, form=_lib.FORM_REFERENCE)
    assert not st.any()
    names = list(_lib.SCALARS)
    for r, out in zip(rows, res):
        g = Green(int(r[0]), int(r[1]), r[2], r[3], 0.1, (r[4], 0.0, 0.0, r[7]))
        g.set_form(_lib.FORM_REFERENCE)
        g.solve()
        ref = g.scalars()
        for k in ("mu0", "Usp", "Uch", "mu"):
            assert out[names.index(k)] == ref[k], (r[:2], k)
