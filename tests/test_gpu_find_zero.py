"""The reference form's root searches on the device (find_zero with grid-wide
evaluations): grids of one block, of a few and of many, against the CPU oracle
with the reference's control flow; a deferred or captured solve against the
same stages read back one by one.

Tolerance: the roots are zeros to 1e-15 of sums over the same chi0 and Sigma to
1e-10, as the parity tests have it."""
import numpy as np
import pytest

from oracle import tpsc_oracle as O

pytestmark = pytest.mark.gpu

MODELS = [dict(n=0.87, tp=-0.15, tpp=0.03, t3=0.0, U=2.4), dict(n=1.12, tp=-0.1, tpp=0.0, t3=0.02, U=3.1),
          dict(n=1.0, tp=0.0, tpp=0.0, t3=0.0, U=1.5)]


def green(m, nk0, nw0, T, ctx=None):
    from tpsc_conductivity_b200.api import Green

    return Green(nk0, nw0, m["n"], T, 0.1, (m["tp"], m["tpp"], m["t3"], m["U"]), ctx=ctx)


@pytest.mark.parametrize("m", MODELS)
@pytest.mark.parametrize("nk0,nw0,T", [(8, 16, 0.5), (16, 64, 0.3), (32, 256, 0.3), (64, 512, 0.25)])
def test_roots_equal_the_oracles(m, nk0, nw0, T):
    ref = O.solve(m["U"], m["tp"], m["tpp"], m["t3"], m["n"], T, nk0, nw0)
    g = green(m, nk0, nw0, T)
    g.solve()
    sc = g.scalars()
    for k, v in (("mu0", ref.mu0), ("Usp", ref.U.Usp), ("Uch", ref.U.Uch), ("mu", ref.mu),
                 ("trSG", ref.trace_self_G[0]), ("trSG_asymp", ref.trace_self_G[1]), ("trSG2", ref.trace_self_G2[0])):
        assert abs(sc[k] - v) <= 1e-10 * max(1.0, abs(v)), k
    # the search's own iteration limits: two ends, the start, 20 (12) steps of at most two evaluations
    assert 3 <= sc["evals_sp"] <= 50 and 3 <= sc["evals_ch"] <= 50 and 3 <= sc["evals_mu"] <= 50


@pytest.mark.parametrize("nk0,nw0", [(16, 64), (64, 512)])
def test_deferred_and_captured_solves_equal_the_stages(nk0, nw0):
    from tpsc_conductivity_b200.api import Context

    m, T = MODELS[0], 0.3
    keys = ("mu0", "chi0max", "Usp", "Uch", "dblOcc", "Sigma_inf", "mu", "trSG", "trSG_asymp", "trSG2", "evals_sp",
            "evals_ch", "evals_mu")
    g = green(m, nk0, nw0, T)
    g.calc_chiqw_FFT_spline()
    g.find_Usp_Uch_grid(nk0, nw0)
    g.calc_chirt()
    g.calc_self_energy()
    assert g.scalars()["trSG"] == 0.0
    g.find_mu()
    assert g.scalars()["trSG"] == 0.0
    g.traceSelfG()
    want, S = g.scalars(), g.self_energy()["S"]
    for mode in (0, 1, 2):
        ctx = Context()
        for _ in range(3):  # direct, captured, replayed (mode 1); updated in place (mode 2)
            h = green(m, nk0, nw0, T, ctx)
            h.set_graph_mode(mode)
            h.solve()
            h.solve()
            h.solve()
            got = h.scalars()
            assert all(got[k] == want[k] for k in keys if k != "dblOcc"), mode
            assert np.array_equal(h.self_energy()["S"], S)
