"""chi_jj at every frequency-grid size of the tau kernel (groups of one thread to
a warp and more), with an odd number of columns and with angle bins that split
column pairs, against the CPU oracle at the parity tests' 1e-10."""
import numpy as np
import pytest

from oracle import tpsc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw0", [16, 32, 128, 256, 512, 1024])
@pytest.mark.parametrize("n,tp,bins", [(0.87, -0.15, 1), (1.13, 0.1, 4)])
def test_every_frequency_grid(nw0, n, tp, bins):
    from tpsc_conductivity_b200.api import CondOpt

    T, U = 0.25, 2.4
    ref = O.solve(U, tp, 0.02, 0.01, n, T, 16, nw0)
    want = O.conductivity(ref, tp, 0.02, 0.01, U, T, bins)
    g = CondOpt(16, nw0, n, T, 0.1, (tp, 0.02, 0.01, U))
    g.solve()
    for _ in range(2):
        r = g.calc_chijj_vertex_corr_all_optim(N_theta_k=bins)
        assert abs(r["kx0"] - want.kx0) < 1e-10 * abs(want.kx0)
        for k in ("chijj1", "chijj2", "chijj1_k", "chijj2_k"):
            v = getattr(want, k)
            assert np.max(np.abs(r[k] - v)) < 1e-10 * np.max(np.abs(v)), k
