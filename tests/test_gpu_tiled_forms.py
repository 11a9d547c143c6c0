"""The 2.5D tiles on layouts above the point sweeps' sizes: blocks of one to
five cells beside a large one, one plane of cells, columns many times deeper
than a tile.  FP64 iterations and one-block implicit calls equal the oracle
for every patch shape and for plane counts of one, odd ones and whole columns;
the reduced-precision forms give the same bits for every tiling and staging."""
import functools

import numpy as np
import pytest

from codens_b200 import cases
from oracle.oracle import lib as orc_lib

from ._helpers import assert_equal_bits, oracle_prepared, real

pytestmark = pytest.mark.gpu

WHOLE = 2**31 - 1  # past every block: whole columns (at most; the depth may be cut)
LARGE = {  # all above the largest layout of point sweeps
    "narrow": lambda: cases.channel_case([1, 2, 3, 5, 280], 45, 31, seed=13, reynz=1.0e3,
                                         lmax=3),
    "plane": lambda: cases.box_case((701, 601, 1), seed=11, skew=0.02, lmax=3, qfix_dfez=1),
    "deep": lambda: cases.box_case((9, 7, 6500), seed=12, ns=True, reynz=1.0e3, lmax=3),
}
TILINGS = [(32, 4, 1), (32, 8, 3), (16, 8, 7), (16, 16, WHOLE)]


@functools.lru_cache(maxsize=None)
def _oracle_state(name):
    case = LARGE[name]()
    assert case.layout.nreal > 370000
    orc, st = oracle_prepared(case)
    orc.step(st)
    return np.asarray(st.v).reshape(-1, case.layout.ld)[:5, real(case)].copy()


def _run(name, precision, tiles, staging=0):
    from codens_b200.solver import CodeNS
    case = LARGE[name]()
    case.scheme.precision = precision
    s = CodeNS(case)
    s.metric()
    if staging:
        s.set_sweep_staging(staging)
    s.set_sweep_tiles(precision, *tiles)
    s.atsch_num(1 if precision == 0 else 2)  # 2: a refresh and a regular defect iteration
    v = s.v.cpu().numpy().reshape(-1, case.layout.ld)[:5, real(case)]
    s.close()
    return v


@pytest.mark.parametrize("tiles", TILINGS)
@pytest.mark.parametrize("name", sorted(LARGE))
def test_fp64_tiles_equal_the_oracle(cuda, name, tiles):
    assert_equal_bits(_run(name, 0, tiles), _oracle_state(name), "state")


@pytest.mark.parametrize("name,precision", [("narrow", 1), ("narrow", 2), ("plane", 1),
                                            ("deep", 1), ("deep", 2)])
def test_reduced_precision_tiles_agree(cuda, name, precision):
    want = _run(name, precision, (32, 8, 16))
    assert np.isfinite(want).all()
    for staging in (0, 1):
        for tiles in TILINGS:
            assert_equal_bits(_run(name, precision, tiles, staging), want,
                              f"{tiles} staging {staging}")


@pytest.mark.parametrize("ns", [0, 1])
@pytest.mark.parametrize("tiles", [(32, 8, 3), (16, 8, 16)])
def test_one_block_calls_equal_the_oracle(cuda, ns, tiles):
    from codens_b200.solver import CodeNS
    torch = cuda
    case = LARGE["narrow"]()
    orc, st = oracle_prepared(case)
    L = orc_lib()
    blocks = range(1, case.layout.nblk + 1)
    for l in blocks:
        L.orc_zpres(l, st.v, st.ps, st.temp, st.cson)
        L.orc_zvismo(l, st.mu, st.temp)
        L.orc_chronos(l, st.mu, st.mut, st.v, st.dt, st.sn, st.vol, st.cson)
    L.orc_rbord(st.v, st.ps, st.temp, st.cson)
    ld = case.layout.ld
    u = np.random.default_rng(5).uniform(-1.0, 1.0, (5, ld)) * 1e-3 * np.asarray(st.vol)
    s = CodeNS(case)
    s.metric()
    s.set_sweep_tiles(0, *tiles)
    for t, a in ((s.v, st.v), (s.pression, st.ps), (s.cson, st.cson), (s.mu, st.mu),
                 (s.mut, st.mut), (s.dt, st.dt), (s.u, u)):
        t.copy_(torch.as_tensor(np.ascontiguousarray(a).reshape(-1)))
    torch.cuda.synchronize()
    u = np.ascontiguousarray(u).reshape(st.u.shape)
    for l in blocks:
        if ns:
            L.orc_implimf_3d(l, u, st.dt, st.v, st.d, st.mu, st.mut, st.sn, st.vol, st.ps,
                             st.cson, 3)
            s.implimf_3d(l, s.u, s.dt, s.v, s.d, s.mu, s.mut, s.sn, s.vol, s.pression, s.cson, 3)
        else:
            L.orc_implimf_eu(l, u, st.dt, st.v, st.d, st.sn, st.vol, st.ps, st.cson, 3)
            s.implimf_eu(l, s.u, s.dt, s.v, s.d, s.sn, s.vol, s.pression, s.cson, 3)
    s.sync()
    rc = real(case)
    for t, a, what in ((s.d, st.d, "d"), (s.v, st.v, "v")):
        a = np.asarray(a).reshape(5, ld)[:, rc]
        assert np.isfinite(a).all()
        assert_equal_bits(t.cpu().numpy().reshape(5, ld)[:, rc], a, what)
    s.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_tiles_after_a_change_of_equations_and_staging(cuda, precision):
    """the tile lists are cut for the equations and the staging: changed on one
    context, the state of a fresh one"""
    from codens_b200.solver import CodeNS
    torch = cuda
    want = _run("narrow", precision, (16, 8, 16), staging=1)
    case = LARGE["narrow"]()
    case.scheme.precision = precision
    case.scheme.ns = 0
    s = CodeNS(case)
    s.metric()
    s.set_sweep_tiles(precision, 16, 8, 16)
    v0 = s.v.clone()
    torch.cuda.synchronize()
    s.atsch_num(1)
    case.scheme.ns = 1
    s.set_scheme(case.scheme)
    s.set_sweep_staging(1)
    assert s.sweep_tiles(precision)[:3] == (16, 8, 16)
    with torch.cuda.stream(s.stream):
        s.v.copy_(v0)
    s.set_cycle(0, 0)
    s.atsch_num(1 if precision == 0 else 2)
    v = s.v.cpu().numpy().reshape(-1, case.layout.ld)[:5, real(case)]
    s.close()
    assert_equal_bits(v, want, "state")
