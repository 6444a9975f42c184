"""A solve or a root search that fails leaves no results behind it: the roots were not
found, so V, Sigma, mu and what is formed from them are refused until a search
succeeds, whatever the form and however the solve was launched (directly, captured,
replayed).  A solve queues every stage before it reads a result, so each of them has
run on the failed search's last iterate by then.

The failing model: U = 5e-324 (the smallest positive double), for which the spin sum
rule's term Us nsr^2 / (2U) overflows and the search has no root in any form."""
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

STATE = 5
NO_ROOT = 4


def _green(p, ctx, form, U=None):
    from tpsc_conductivity_b200.api import CondOpt

    g = CondOpt(int(p["nk0"]), int(p["Nw0"]), p["n"], p["T"], 0.1,
                (p["tp"], p["tpp"], p["t3"], p["U"] if U is None else U), ctx=ctx)
    g.set_form(form)
    return g


def _refused(call, status=STATE):
    from tpsc_conductivity_b200 import _lib

    with pytest.raises(_lib.TPSCError) as e:
        call()
    assert e.value.status == status


def _no_results(g, vertex=True):
    if vertex:
        _refused(g.vertex)
    _refused(g.self_energy)
    _refused(g.find_mu)
    _refused(g.traceSelfG)
    _refused(lambda: g.ctx.call("tpsc_chijj", 1))
    _refused(g.Gwn_local)
    _refused(g.sumrule_tangents)
    _refused(g.sp_corr_length)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("form", [0, 1, 3])
def test_failed_solve_leaves_no_results(form, mode):
    from tpsc_conductivity_b200.api import Context

    p = load_golden("l16_w128_n110")["p"]
    ctx = Context()
    good = _green(p, ctx, form)
    good.set_graph_mode(mode)
    good.solve()
    want = good.scalars()
    bad = _green(p, ctx, form, U=5e-324)
    for _ in range(4):  # direct, then captured, then replayed (mode 1)
        _refused(bad.solve, NO_ROOT)
        _no_results(bad)
    again = _green(p, ctx, form)
    again.solve()
    assert again.scalars() == want
    again.self_energy()
    again.sumrule_tangents()
    again.ctx.call("tpsc_chijj", 1)


@pytest.mark.parametrize("form", [0, 1])
def test_failed_search_on_a_grid_leaves_no_roots(form):
    from tpsc_conductivity_b200.api import Context

    p = load_golden("l16_w128_n110")["p"]
    nk0, nw0 = int(p["nk0"]), int(p["Nw0"])
    ctx = Context()
    bad = _green(p, ctx, form, U=5e-324)
    _refused(lambda: bad.find_Usp_Uch_grid(nk0, nw0), NO_ROOT)
    _refused(bad.sumrule_tangents)
    _refused(bad.sp_corr_length)
    # the vertex stage takes the last roots that were found: none in this context
    bad.calc_chirt()
    assert not bad.vertex().any()
    good = _green(p, ctx, form)
    good.find_Usp_Uch_grid(nk0, nw0)
    good.calc_chirt()
    want = good.vertex()
    bad = _green(p, ctx, form, U=5e-324)
    _refused(lambda: bad.find_Usp_Uch_grid(nk0, nw0), NO_ROOT)
    good = _green(p, ctx, form)
    good.calc_chiqw_FFT_spline()
    good.calc_chirt()
    assert (good.vertex() == want).all()
