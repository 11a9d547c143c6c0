"""The global time step (kdtl = 0, chrono.f90:113-151) in the fused
iteration and as its own entry point, against the oracle; the reference's
stop when the step falls below dt1min becomes CNS_EDT."""
import numpy as np
import pytest

from oracle.oracle import lib as orc_lib

from ._helpers import SMALL, assert_equal_bits, oracle_prepared, real

pytestmark = pytest.mark.gpu


def _min_local_dt(case):
    orc, st = oracle_prepared(case)
    L = orc_lib()
    for l in range(1, case.layout.nblk + 1):
        L.orc_zpres(l, st.v, st.ps, st.temp, st.cson)
        if case.scheme.ns:
            L.orc_zvismo(l, st.mu, st.temp)
        L.orc_chronos(l, st.mu, st.mut, st.v, st.dt, st.sn, st.vol, st.cson)
    return float(st.dt[real(case)].min()), float(st.dt[real(case)].max())


@pytest.mark.parametrize("name", ["box_ns", "box_eu_qfix"])
def test_global_dt_fused_parity(cuda, name):
    from codens_b200.solver import CodeNS
    case = SMALL[name]()
    lo, _ = _min_local_dt(case)
    case.scheme.kdtl = 0
    case.scheme.dt1min = 0.5 * lo
    orc, st = oracle_prepared(case)
    s = CodeNS(case)
    s.metric()
    ld = case.layout.ld
    rc = real(case)
    for it in range(4):
        u0 = st.v.copy()
        orc.step(st)
        no = orc.norms(u0, st)
        ng = s.atsch_num(1)
        assert_equal_bits(s.v.cpu().numpy().reshape(5, ld)[:, rc], st.v.reshape(5, ld)[:, rc],
                          f"v after step {it}")
        n = case.layout.ncells
        assert_equal_bits(s.dt.cpu().numpy()[:n], st.dt[:n], f"dt after step {it}")
        np.testing.assert_allclose(ng, no, rtol=1e-12, atol=0)
    s.close()


def test_global_dt_below_dt1min_is_an_error(cuda):
    from codens_b200 import abi
    from codens_b200.solver import CodeNS
    case = SMALL["box_ns"]()
    _, hi = _min_local_dt(case)
    case.scheme.kdtl = 0
    case.scheme.dt1min = 10.0 * hi
    s = CodeNS(case)
    s.metric()
    with pytest.raises(abi.CnsError) as ei:
        s.atsch_num(1)
    assert ei.value.code == abi.CNS_EDT
    s.close()


def test_adjoint_prepared_with_the_global_step(cuda):
    """as the first call on a context (its step reduction has no scratch yet) and
    after one that has made it: the same transposed implicit phase"""
    from codens_b200.solver import CodeNS
    torch = cuda
    case = SMALL["box_eu_qfix"]()
    case.scheme.kdtl = 0
    case.scheme.dt1min = 1e-9
    ld, rc = case.layout.ld, real(case)
    y = torch.zeros(5, ld, dtype=torch.float64, device="cuda")
    y[:, torch.as_tensor(rc, device="cuda")] = 1.0
    y = y.reshape(-1)
    outs = []
    for warm in (False, True):
        s = CodeNS(case)
        s.metric()
        if warm:
            s.dt.fill_(1.0)
            torch.cuda.synchronize()
            s.chrono_global(s.dt)
        s.adjoint_prepare()
        out = torch.zeros(5 * ld, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.adjoint_lt(y, out)
        s.sync()
        outs.append(out.cpu().numpy().reshape(5, ld)[:, rc])
        s.close()
    assert np.isfinite(outs[0]).all() and (outs[0] != 0.0).any()
    assert_equal_bits(outs[0], outs[1], "L^T y")
