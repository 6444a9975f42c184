"""A root search whose wait between blocks runs out is repeated in one block, which
waits for no other: the call succeeds with the same results (to the last bit in the
reference form, whose sums are in block order; the Newton form's sums take another
order, 1e-11 as for other grids).  When the repetition runs out too the call fails, and
leaves a context that solves.  The wait is made to run out on the host (the flag that
is read back counts as set)."""
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

CUDA = 2
KEYS = ("mu0", "Usp", "Uch", "mu", "trSG2", "dblOcc")


def _green(form, name="l32_w256_u4_tp", ctx=None):
    from tpsc_conductivity_b200.api import Green

    p = load_golden(name)["p"]
    g = Green(p["nk0"], p["Nw0"], p["n"], p["T"], 0.1, (p["tp"], p["tpp"], p["t3"], p["U"]), ctx=ctx)
    g.set_form(form)
    return g


def _same(got, want, form):
    for k in KEYS:
        assert got[k] == want[k] if form == 0 else abs(got[k] - want[k]) <= 1e-11 * max(1.0, abs(want[k])), k


# 8^2 to 32^2 exchange values through slots, 256^2 (golden 256^2 x 4096) at a barrier
@pytest.mark.parametrize("name", ["l16_w64_u2", "l32_w256_u4_tp", "l256_w4096_u4"])
@pytest.mark.parametrize("form", [0, 1, 3])
def test_a_search_that_ran_out_is_repeated_alone(form, name):
    g = _green(form, name)
    g.solve()
    want = g.scalars()
    for count in (1, 2):  # the sum rules' flag; both flags
        g.ctx.call("tpsc_inject_wait_timeouts", count)
        g.solve()
        _same(g.scalars(), want, form)
    g.solve()
    assert g.scalars() == want


@pytest.mark.parametrize("form", [0, 1])
def test_stage_by_stage(form):
    g = _green(form)
    g.solve()
    want = g.scalars()
    g.ctx.call("tpsc_inject_wait_timeouts", 1)
    g.find_Usp_Uch_grid(g.nk0, g.Nw0)
    g.calc_chirt()
    g.calc_self_energy()
    g.ctx.call("tpsc_inject_wait_timeouts", 1)
    g.find_mu()
    _same(g.scalars(), want, form)


@pytest.mark.parametrize("form", [0, 1, 3])
def test_a_repetition_that_runs_out_fails(form):
    from tpsc_conductivity_b200 import _lib

    g = _green(form)
    g.solve()
    want = g.scalars()
    g.ctx.call("tpsc_inject_wait_timeouts", 4)
    with pytest.raises(_lib.TPSCError) as e:
        g.solve()
    assert e.value.status == CUDA and "timed out" in str(e.value)
    with pytest.raises(_lib.TPSCError):
        g.self_energy()
    g.solve()
    assert g.scalars() == want
