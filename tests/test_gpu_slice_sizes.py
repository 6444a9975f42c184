"""Every compiled lattice size at the smallest frequency grids: the slice
kernels' block plans (groups, threads, rounds) against the CPU oracle.

Tolerances: the FP64 form's parity tolerances (chi_jj 1e-10, full Sigma 1e-10
of its maximum); the mixed form's stated 1e-6 against the FP64 form."""
import numpy as np
import pytest

from oracle import tpsc_oracle as O

pytestmark = pytest.mark.gpu

MODEL = dict(n=0.87, T=0.3, tp=-0.15, tpp=0.03, t3=0.0, U=2.4)


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(b)))


def solved(nk0, nw0, form):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import CondOpt

    m = MODEL
    g = CondOpt(nk0, nw0, m["n"], m["T"], 0.1, (m["tp"], m["tpp"], m["t3"], m["U"]))
    g.set_form({"fp64": _lib.FORM_REFERENCE, "mixed": _lib.FORM_NEWTON | _lib.FORM_MIXED}[form])
    g.solve()
    return g, g.calc_chijj_vertex_corr_all_optim(N_theta_k=2)


@pytest.mark.parametrize("nk0", [8, 16, 32, 64, 128])
@pytest.mark.parametrize("nw0", [16, 64])
def test_every_lattice_size(nk0, nw0):
    m = MODEL
    ref = O.solve(m["U"], m["tp"], m["tpp"], m["t3"], m["n"], m["T"], nk0, nw0)
    cond = O.conductivity(ref, m["tp"], m["tpp"], m["t3"], m["U"], m["T"], 2)
    g, r = solved(nk0, nw0, "fp64")
    assert rel(g.chi0()["chiqw"], ref.chi0.chiqw) < 1e-10
    assert rel(g.vertex(), ref.V) < 1e-10
    assert rel(g.sigma(), ref.sigma.sigma(m["T"])) < 1e-10
    for k in ("chijj1", "chijj2", "chijj1_k", "chijj2_k"):
        assert rel(r[k], getattr(cond, k)) < 1e-10, k
    gm, rm = solved(nk0, nw0, "mixed")
    assert rel(gm.sigma(), g.sigma()) < 1e-6
    for k in ("chijj1", "chijj2"):
        assert rel(rm[k], r[k]) < 1e-6, k
