"""The Fermi-surface hot spot searched on the device, one thread per line, against
the CPU oracle's find_FS and vF_hot_spots: surfaces that cross the zone's diagonal,
that do not, electron-like ones whose later lines have no root, and t'', t3.

Tolerance: vF is |grad eps| at the midpoint of two roots that the bounded search
finds to 1e-15 of eps: 1e-9 as the parity tests have it."""
import pytest

from oracle import tpsc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tp,tpp,t3", [(0.85, -0.2, 0.0, 0.0), (0.95, -0.3, 0.05, 0.0), (0.6, 0.0, 0.0, 0.0),
                                         (1.0, 0.0, 0.0, 0.0), (1.15, -0.25, 0.1, 0.02), (0.3, 0.1, 0.0, -0.03)])
def test_vf_equals_the_oracles(n, tp, tpp, t3):
    from tpsc_conductivity_b200.api import Green

    g = Green(16, 64, n, 0.4, 0.1, (tp, tpp, t3, 1.5))
    g.find_Usp_Uch()
    r = g.sp_corr_length()
    fs = O.find_fs(g.scalars()["mu0"], tp, tpp, t3)
    want = O.vf_hot_spots(fs, tp, tpp, t3)
    assert abs(r["vF"] - want) <= 1e-9 * max(1.0, abs(want))
