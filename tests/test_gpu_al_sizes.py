"""The Aslamazov-Larkin term at the edges of its plans: the smallest lattices and
frequency grids (groups of one to four threads), one transform per warp and
per block, grids of one frequency, of none, and batches with a remainder,
against the CPU oracle.

Tolerance: the parity tests' 1e-9 of the largest |chijj3| (difference
quotients of nearly equal tails lose digits)."""
import numpy as np
import pytest

from oracle import tpsc_oracle as O

pytestmark = pytest.mark.gpu

M = dict(n=0.87, T=0.3, tp=-0.15, tpp=0.03, t3=0.0, U=2.4)


@pytest.mark.parametrize("nk0,nw0,mmin,bins", [(8, 16, 0, 1), (8, 16, 2, 2), (16, 16, 5, 1), (8, 32, 1, 1), (16, 64, 1, 3),
                                               (8, 128, 2, 1), (32, 64, 3, 2), (8, 512, 4, 1), (16, 1024, 6, 2),
                                               (64, 64, 3, 1)])
def test_every_plan(nk0, nw0, mmin, bins):
    from tpsc_conductivity_b200.api import CondOpt

    ref = O.solve(M["U"], M["tp"], M["tpp"], M["t3"], M["n"], M["T"], nk0, nw0)
    al = O.conductivity_al(ref, M["tp"], M["tpp"], M["t3"], M["U"], M["T"], mmin, bins)
    g = CondOpt(nk0, nw0, M["n"], M["T"], 0.1, (M["tp"], M["tpp"], M["t3"], M["U"]))
    g.solve()
    for _ in range(2):  # the second call reuses the buffers
        r = g.calc_chijj_vertex_corr_all_optim(True, mmin, bins)
        assert np.array_equal(r["ind_freq"], al.ind_freq)
        top = max(float(np.max(np.abs(al.chijj3))), 1e-300)
        assert np.max(np.abs(r["chijj3"] - al.chijj3)) < 1e-9 * top
        assert np.max(np.abs(r["chijj3_k"] - al.chijj3_k)) < 1e-9 * top
