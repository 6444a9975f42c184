"""Tangents and the reverse pass on the G(r, tau) that the solve has left.

The FP64 forms' chi0 stage leaves the FP64 G(r, tau) that the tangents need;
the mixed form's leaves its FP32 copy beside whatever the FP64 buffer held
before.  The calls must give what a fresh context gives, to the last bit, also
when models and forms change on one context.
"""
import numpy as np
import pytest

from tpsc_conductivity_b200 import _lib, api

pytestmark = pytest.mark.gpu

MIXED = _lib.FORM_NEWTON | _lib.FORM_MIXED
A = (0.875, 0.25, (-0.15, 0.02, 0.0, 3.0))
B = (0.8, 0.3, (-0.05, -0.03, 0.0, 2.5))


def sensitivities(ctx, nk0, nw0, form, model):
    ctx.call("tpsc_set_form", form)
    n, T, params = model
    g = api.CondOpt(nk0, nw0, n, T, 0.1, params, ctx=ctx)
    g.solve()
    t = g.sumrule_tangents()
    grad, dD = g.sigma_qn_vjp(np.array([0.0, 1.0]))
    return np.concatenate([[t[p][k] for p in ("U", "mu", "tp") for k in ("Usp", "Uch", "D")], grad, dD])


@pytest.mark.parametrize("nk0,nw0", [(8, 64), (32, 256), (128, 512)])
def test_models_and_forms_in_turn(nk0, nw0):
    steps = [(_lib.FORM_REFERENCE, A), (_lib.FORM_NEWTON, B), (MIXED, A), (MIXED, B), (_lib.FORM_NEWTON, A),
             (MIXED, B), (_lib.FORM_REFERENCE, A)]
    ctx = api.Context()
    for form, model in steps:
        got = sensitivities(ctx, nk0, nw0, form, model)
        np.testing.assert_array_equal(got, sensitivities(api.Context(), nk0, nw0, form, model))
