"""The injection condition's global sweep count (clidd.f90:96-113): cells of
reversed flow count as converged in their first sweep (the update is divided
by the signed velocity) and may still move when the others are done, so that
the boundary needs sweeps past every cell's first small update."""
import numpy as np
import pytest

from codens_b200 import cases
from oracle.oracle import lib as orc_lib

from ._helpers import assert_equal_bits, oracle_prepared


def reversed_case(seed, share, spread):
    """a channel whose inlet cells are within `spread` of the condition's own
    solution, but for a `share` of reversed ones"""
    case = cases.channel_case([6, 5], 9, 7, seed=3, reynz=1.0e3, noise=0.0)
    rng = np.random.default_rng(seed)
    bd = next(q for q, b in enumerate(case.boundaries) if b.kind == cases.BC_IDD)
    ba = case.boundary_arrays()
    ni = ba["ncin"][ba["mpb"][bd]:ba["mpb"][bd] + ba["mmb"][bd]]
    f = np.where(rng.random(ni.size) < share, rng.uniform(-1.2, -0.05, ni.size), 1.0)
    v = case.v0
    gam = case.phys.gam
    q = v[1, ni] / v[0, ni] * f
    # the pressure the condition itself gives at that velocity (no update), off
    # it by `spread`, or by up to half for the reversed cells
    p = case.phys.pa1 * (1.0 + 0.5 * (gam - 1.0) * q * q) ** (-gam / (gam - 1.0))
    p *= np.where(f < 0, rng.uniform(0.4, 1.0, ni.size),
                  1.0 + spread * rng.uniform(-1.0, 1.0, ni.size))
    v[1, ni] = v[0, ni] * q
    v[4, ni] = p / (gam - 1.0) + 0.5 * (v[1:4, ni] ** 2).sum(0) / v[0, ni]
    return case, ni


def sweeps(case, ni):
    """per cell, whether each of the 20 updates is above 1e-7 (omg = 0, the
    inlet normal (1, 0, 0))"""
    gam = case.phys.gam
    g1 = gam - 1.0
    v = case.v0[:, ni]
    q = v[1] / v[0]
    p = g1 * (v[4] - 0.5 * (v[1:4] ** 2).sum(0) / v[0])
    roc0 = -np.sqrt(gam * p * v[0])
    am0 = p + roc0 * q
    out = []
    for _ in range(20):
        b = 1.0 / (1.0 + 0.5 * g1 * q * q)
        pp = case.phys.pa1 * b ** (gam / g1)
        dq = -(pp + roc0 * q - am0) / (roc0 - gam * pp / b * q)
        out.append(np.abs(dq) / q > 1e-7)
        q = q + dq
    return np.array(out)


CASES = [(1, 0.3, 0.2), (2, 0.1, 1e-4), (3, 0.7, 1e-6), (4, 0.02, 1e-3), (5, 0.0, 0.3)]


def test_cases_need_late_sweeps():
    """some of the cases hold a cell whose update is large again after its
    first small one, at the sweep where every cell has had a small one"""
    late = []
    for seed, share, spread in CASES:
        big = sweeps(*reversed_case(seed, share, spread))
        first = np.argmin(big, axis=0)  # the first small update of each cell
        late.append(bool(big[first.max()].any()))
    assert any(late) and not all(late), late


@pytest.mark.gpu
@pytest.mark.parametrize("seed,share,spread", CASES)
def test_injection_ghosts_with_reversed_cells(cuda, seed, share, spread):
    from codens_b200.solver import CodeNS
    case, _ = reversed_case(seed, share, spread)
    orc, st = oracle_prepared(case)
    L = orc_lib()
    for l in range(1, case.layout.nblk + 1):
        L.orc_zpres(l, st.v, st.ps, st.temp, st.cson)
    L.orc_rbord(st.v, st.ps, st.temp, st.cson)
    s = CodeNS(case)
    s.metric()
    for _ in range(2):  # the second call finds the work words of the first
        s.zpres(0, s.v, s.pression, s.ztemp, s.cson)
        s.rbord(s.v, s.pression, s.ztemp, s.cson)
    s.sync()
    g = case.boundary_arrays()["ncbd"]
    ld = case.layout.ld
    assert_equal_bits(s.v.cpu().numpy().reshape(5, ld)[:, g], st.v.reshape(5, ld)[:, g], "v")
    for a, b in ((s.pression, st.ps), (s.ztemp, st.temp), (s.cson, st.cson)):
        assert_equal_bits(a.cpu().numpy()[g], b[g], "ps, temp, cson")
    s.close()
