"""The model's tables made on the device: the dispersion of all four hoppings in a
batch of two points per shape and in single solves, and chi_jj's derivative tables
and angle bins through changes of the model and of the number of bins on one
context, against the CPU oracle.

Tolerance: scalars of the mixed solve 1e-6 and chi_jj of the FP64 solve 1e-10, as
the parity tests have them."""
import numpy as np
import pytest

from oracle import tpsc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk0,Nw0", [(8, 16), (16, 64), (32, 32)])
def test_batch_of_models(nk0, Nw0):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import solve_points

    pts = [(nk0, Nw0, 0.87, 0.3, -0.2, 0.05, 0.02, 2.0), (nk0, Nw0, 1.1, 0.4, 0.15, -0.04, 0.03, 1.5)]
    res, st, _ = solve_points(np.array(pts))
    assert not st.any()
    names = list(_lib.SCALARS)
    for p, r in zip(pts, res):
        _, _, n, T, tp, tpp, t3, U = p
        ref = O.solve(U, tp, tpp, t3, n, T, nk0, Nw0)
        for name, want in (("mu0", ref.mu0), ("Usp", ref.U.Usp), ("Uch", ref.U.Uch), ("mu", ref.mu)):
            assert abs(r[names.index(name)] - want) <= 1e-6 * max(1.0, abs(want))


@pytest.mark.parametrize("nk0,Nw0", [(8, 32), (16, 64)])
def test_bins_and_models_on_one_context(nk0, Nw0):
    from tpsc_conductivity_b200.api import Context, CondOpt

    ctx = Context()
    for n, tp, tpp, t3, bins in ((0.87, -0.15, 0.03, 0.02, 4), (0.87, -0.15, 0.03, 0.02, 1),
                                 (1.1, 0.1, -0.02, 0.01, 3), (1.1, 0.1, -0.02, 0.01, 4)):
        want = O.conductivity(O.solve(2.2, tp, tpp, t3, n, 0.25, nk0, Nw0), tp, tpp, t3, 2.2, 0.25, bins)
        g = CondOpt(nk0, Nw0, n, 0.25, 0.1, (tp, tpp, t3, 2.2), ctx=ctx)
        g.solve()
        r = g.calc_chijj_vertex_corr_all_optim(N_theta_k=bins)
        assert abs(r["kx0"] - want.kx0) < 1e-10 * abs(want.kx0)
        for k in ("chijj1_k", "chijj2_k"):
            v = getattr(want, k)
            assert np.max(np.abs(r[k] - v)) < 1e-10 * np.max(np.abs(v)), k
