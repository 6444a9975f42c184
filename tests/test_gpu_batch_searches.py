"""Reference-form batches on many contexts: where a context's share of the GPU leaves its
root searches few blocks for the lattice, the host drives them.  Every result equals the
single solve's to the last bit (both sum in block order), point by point, also where a
search has no root; capped by 8 contexts (37 blocks on 148 SMs) lattices of up to 64^2
search on the device, by 16 (18 blocks) up to 32^2."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(8, 64), (32, 64), (64, 64), (128, 64), (256, 32)]


def _points(nk0, nw0):
    return np.array([[nk0, nw0, n, T, -0.1, 0.05, 0.0, U]
                     for n, T, U in ((0.85, 0.6, 2.0), (0.95, 0.5, 3.0), (1.1, 0.7, 1.5))])


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("nstreams", [8, 16])
@pytest.mark.parametrize("nk0,nw0", CASES)
def test_many_contexts_give_the_single_solves_bits(form, nstreams, nk0, nw0):
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Batch, Green

    pts = _points(nk0, nw0)
    b = Batch(nstreams=nstreams)
    res, st, _ = b.solve(pts, form=form)
    b.close()
    assert (st == 0).all()
    for p, r in zip(pts, res):
        g = Green(int(p[0]), int(p[1]), p[2], p[3], 0.1, tuple(p[4:]))
        g.set_form(form)
        g.solve()
        s = g.scalars()
        for i, k in enumerate(_lib.SCALARS):
            assert r[i] == s[k], (k, r[i], s[k])


@pytest.mark.parametrize("nk0", [64, 128])
def test_corr_length_rows(nk0):
    from tpsc_conductivity_b200.api import Batch

    a, many = Batch(nstreams=1), Batch(nstreams=16)
    args = (nk0, 64, (-0.1, 0.0, 0.0, 2.5), [0.8, 0.9], 2, [0.6, 0.5], 2)
    want, st0, _ = a.corr_length(*args, form=0)
    got, st1, _ = many.corr_length(*args, form=0)
    a.close()
    many.close()
    assert (st0 == 0).all() and (st1 == 0).all()
    assert np.array_equal(got, want)


def test_a_point_without_a_root_fails_alone():
    from tpsc_conductivity_b200.api import Batch

    pts = _points(128, 64)
    # Us nsr^2 / (2U) overflows: no Usp in any form
    bad = [128, 64, 0.9, 0.5, 0.0, 0.0, 0.0, 5e-324]
    pts = np.vstack([pts[:1], [bad], pts[1:]])
    out = []
    for S in (1, 16):
        b = Batch(nstreams=S)
        out.append(b.solve(pts, form=0)[:2])
        b.close()
    assert np.array_equal(out[0][1], out[1][1]) and out[0][1].tolist() == [0, 4, 0, 0]
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)


@pytest.mark.parametrize("nk0,nstreams,host", [(256, 4, False), (256, 8, True), (128, 8, True), (64, 8, False),
                                               (64, 16, True), (32, 16, False)])
def test_who_drives_the_searches(nk0, nstreams, host):
    """A search that the host drives launches a kernel for each evaluation."""
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    from tpsc_conductivity_b200 import _lib
    from tpsc_conductivity_b200.api import Batch

    lib, pts, n, launches = _lib.load(), _points(nk0, 64), C.c_longlong(), []
    for S in (1, nstreams):
        b = Batch(nstreams=S)
        b.set_graph_mode(0)
        b.solve(pts, form=0)
        lib.tpsc_launch_count(None, C.byref(n))
        k = n.value
        res, st, _ = b.solve(pts, form=0)
        lib.tpsc_launch_count(None, C.byref(n))
        launches.append(n.value - k)
        b.close()
        assert (st == 0).all()
    evals = sum(res[:, list(_lib.SCALARS).index(e)].sum() for e in ("evals_sp", "evals_ch", "evals_mu"))
    assert (launches[1] - launches[0] > evals / 2) == host and (launches[1] == launches[0]) != host
