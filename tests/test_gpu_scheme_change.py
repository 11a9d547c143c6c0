"""A context whose scheme is changed computes what a fresh context of the new
scheme computes: the viscous halves that HLLC with the stresses and WENO5 keep
beside their face fluxes enter no other family's residual."""
import numpy as np
import pytest

from codens_b200 import cases

from ._helpers import assert_equal_bits, real

pytestmark = pytest.mark.gpu


def _case(ischema, ns, precision):
    # a low Reynolds number: the viscous fluxes are far above rounding
    case = cases.box_case((9, 7, 5), seed=3, ns=bool(ns), skew=0.02, reynz=50.0, lmax=3)
    case.scheme.ischema = ischema
    case.scheme.precision = precision
    return case


def _march(torch, s, case, v0):
    with torch.cuda.stream(s.stream):
        s.v.copy_(v0)
    s.set_cycle(0, 0)
    s.atsch_num(2)
    ld, rc = case.layout.ld, real(case)
    return [t.cpu().numpy().reshape(-1, ld)[:5, rc] for t in (s.v, s.u)]


@pytest.mark.parametrize("before", [14, 12])
@pytest.mark.parametrize("ischema,ns,precision", [(7, 1, 0), (7, 1, 1), (7, 1, 2), (9, 1, 0),
                                                  (5, 1, 1), (14, 0, 0), (14, 1, 1)])
def test_scheme_after_one_with_viscous_halves(cuda, before, ischema, ns, precision):
    from codens_b200.solver import CodeNS
    torch = cuda
    old, case = _case(before, 1, 0), _case(ischema, ns, precision)
    s = CodeNS(old)
    s.metric()
    v0 = s.v.clone()
    torch.cuda.synchronize()
    _march(torch, s, old, v0)
    s.set_scheme(case.scheme)
    got = _march(torch, s, case, v0)
    s.close()
    f = CodeNS(case)
    f.metric()
    want = _march(torch, f, case, v0)
    f.close()
    for g, w, what in zip(got, want, ("state", "residual")):
        assert np.isfinite(w).all()
        assert_equal_bits(g, w, what)


def test_flux_routine_after_hllc(cuda):
    from codens_b200.solver import CodeNS
    case = _case(7, 1, 0)
    out = []
    for first in (False, True):
        s = CodeNS(case)
        s.metric()
        s.zpres(0, s.v, s.pression, s.ztemp, s.cson)
        s.zvismo(0, s.mu, s.v, s.ztemp)
        s.rbord(s.v, s.pression, s.ztemp, s.cson)
        s.zvisqc(s.v, s.mu, s.mut, s.tau, s.sn, s.vol, s.ztemp)
        if first:
            s.sch_hllc(1, s.u, s.v, s.tau, s.sn, s.pression)
        for routine in (s.sch_roe, s.sch_rusanov, s.sch_ausmp):
            routine(1, s.u, s.v, s.tau, s.sn, s.pression)
            s.sync()
            out.append(s.u.cpu().numpy().reshape(-1, case.layout.ld)[:5, real(case)])
        s.close()
    for q in range(3):
        assert_equal_bits(out[3 + q], out[q], "residual")


def test_setting_a_scheme_waits_for_no_iteration(cuda):
    """the block table follows the iterations in flight on the stream, so that the
    call returns while they run, and those after it see the new values"""
    import time

    from codens_b200.solver import CodeNS
    out = []
    for wait in (True, False):
        case = cases.box_case((96, 96, 96), seed=5, qfix_dfez=1, lmax=10)
        s = CodeNS(case)
        s.metric()
        s.set_sweep_tiles(0, 16, 8, 16)
        s.atsch_num(1)
        t = time.perf_counter()
        s.atsch_num_launch(200)
        if wait:
            s.sync()
            march = time.perf_counter() - t
        t = time.perf_counter()
        case.scheme.eta = 2.0
        s.set_scheme(case.scheme)
        if not wait:
            assert time.perf_counter() - t < 0.2 * march
        s.atsch_num(2)
        out.append(s.v.cpu().numpy().reshape(-1, case.layout.ld)[:, real(case)])
        s.close()
    assert np.isfinite(out[0]).all()
    assert_equal_bits(out[1], out[0], "state")
