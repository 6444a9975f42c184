"""The reverse pass of chi_jj at every length of the tau axis, from one thread per
transform to 256, on 15 and 63 columns (a last pair of one column): the gradient of a
combination of sigma(iq_1..4) against central differences of full device solves.

Tolerance: 1e-6 of the largest component, the differences' truncation, as the tests
of the ordinary sizes have it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk0,Nw0,T", [(8, 16, 0.5), (8, 32, 0.4), (8, 64, 0.3), (16, 128, 0.25), (8, 256, 0.2),
                                       (16, 512, 0.15), (8, 1024, 0.1), (16, 2048, 0.1), (8, 4096, 0.05)])
def test_reverse_pass_at_every_length(nk0, Nw0, T):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import CondOpt

    g = CondOpt(nk0, Nw0, 0.85, T, 0.1, (-0.2, 0.0, 0.0, 2.5))
    g.set_form(_lib.FORM_NEWTON)
    g.solve()
    g.ctx.call("tpsc_chijj", 1)
    g._nbins = 1
    ds, _ = g.sigma_qn_sensitivities(4)
    g.ctx.call("tpsc_chijj", 1)
    cot = np.random.default_rng(Nw0).standard_normal(4)
    grad, _ = g.sigma_qn_vjp(cot)
    ref = ds @ cot
    assert np.max(np.abs(grad - ref)) <= 1e-6 * np.max(np.abs(ref))
