"""The two forms of the Jacobi sweeps: point sweeps (small layouts) and 2.5D
tiles (larger ones) give the same bits.  Six independent boxes, each small
enough for point sweeps, together make a layout of 2.5D tiles: every box of
the batch must end as it does alone, for every patch shape and precision; and
boxes at the lines equal the oracle."""
import numpy as np
import pytest

from codens_b200 import cases

from ._helpers import assert_equal_bits, oracle_prepared, real

pytestmark = pytest.mark.gpu

# the largest layouts of point sweeps: FP64 Euler, FP64 Navier-Stokes, FP32
POINT_EULER64, POINT_NS64, POINT_32 = 180000, 270000, 370000


def _run(case, nsteps, precision, tiles=None):
    from codens_b200.solver import CodeNS
    case.scheme.precision = precision
    s = CodeNS(case)
    s.metric()
    if tiles:
        s.set_sweep_tiles(precision, *tiles)
    s.atsch_num(nsteps)
    v = s.v.cpu().numpy().reshape(5, case.layout.ld)
    s.close()
    return v


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ns", [0, 1])
def test_point_equals_tiled(cuda, precision, ns):
    def batch():
        bt = cases.batch_case(ncase=6, side=(40, 47), seed=6, qfix_dfez=1 - ns)
        bt.scheme.ns = ns
        bt.phys.reynz = 1.0e4
        return bt
    bt = batch()
    assert bt.layout.nreal > POINT_32 and max(b.nreal for b in bt.layout.blocks) < POINT_EULER64
    alone = []
    for ib in range(bt.layout.nblk):
        m = cases.batch_member(bt, ib)
        alone.append(_run(m, 3, precision)[:, m.layout.blocks[0].real_cells()])
    for tiles in ((32, 4, 3), (32, 8, 16), (16, 8, 5), (16, 16, 64)):
        v = _run(batch(), 3, precision, tiles)
        for ib, want in enumerate(alone):
            assert_equal_bits(v[:, bt.layout.blocks[ib].real_cells()], want, f"{tiles} box {ib}")


# the last point-sweep size and the first tiled one; odd sides, one-cell directions
@pytest.mark.parametrize("ns,cells", [
    (0, (60, 50, 60)), (0, (61, 59, 51)), (1, (100, 60, 45)), (1, (65, 65, 64)),
    (0, (129, 2, 3)), (1, (129, 2, 3)), (0, (1, 33, 5)), (1, (1, 33, 5))])
def test_fused_step_bits_at_the_line(cuda, ns, cells):
    case = cases.box_case(cells, seed=7, ns=bool(ns), skew=0.01, reynz=1.0e4,
                          qfix_dfez=1 - ns, lmax=4)
    orc, st = oracle_prepared(case)
    for _ in range(2):
        orc.step(st)
    rc = real(case)
    v = _run(case, 2, 0)
    assert_equal_bits(v[:, rc], np.asarray(st.v).reshape(-1, case.layout.ld)[:5, rc], "state")


@pytest.mark.parametrize("lmax", [0, 1, 2, 3])
def test_few_sweeps(cuda, lmax):
    case = cases.box_case((9, 7, 5), seed=8, ns=True, skew=0.02, lmax=lmax, reynz=1.0e3)
    orc, st = oracle_prepared(case)
    for _ in range(2):
        orc.step(st)
    rc = real(case)
    v = _run(case, 2, 0)
    assert_equal_bits(v[:, rc], np.asarray(st.v).reshape(-1, case.layout.ld)[:5, rc], "state")
    assert np.isfinite(_run(case, 2, 1)[:, rc]).all()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ns", [0, 1])
def test_one_wave_and_more(cuda, precision, ns):
    """FP32 point sweeps take another kernel once the cells are more than one
    wave (four CTAs of 128 cells an SM): each of two boxes just inside one wave
    ends in their common layout of two waves as it does alone"""
    import torch
    wave = 4 * 128 * torch.cuda.get_device_properties(0).multi_processor_count
    n = int(wave ** (1. / 3.))  # 42 on 148 SMs

    def batch():
        bt = cases.batch_case(ncase=2, side=(n, n), seed=9, qfix_dfez=1 - ns, mach_range=(0.4, 0.5))
        bt.scheme.ns = ns
        bt.phys.reynz = 1.0e4
        return bt
    bt = batch()
    v = _run(batch(), 2, precision)
    for ib in range(2):
        m = cases.batch_member(bt, ib)
        want = _run(m, 2, precision)[:, m.layout.blocks[0].real_cells()]
        assert_equal_bits(v[:, bt.layout.blocks[ib].real_cells()], want, f"box {ib}")


@pytest.mark.parametrize("precision", [0, 1])
def test_point_sweeps_take_no_scratch_of_their_own(cuda, precision):
    """the packed iterates lie in buffers that are free during the sweeps: a
    layout of point sweeps holds as much device scratch a cell as a tiled one (the
    tile and boundary lists weigh a little more on the smaller)"""
    from codens_b200.solver import CodeNS
    per_cell = []
    for cells in ((50, 50, 50), (80, 80, 80)):
        case = cases.box_case(cells, seed=7, qfix_dfez=1)
        case.scheme.precision = precision
        s = CodeNS(case)
        s.metric()
        s.atsch_num(1)
        per_cell.append(s.scratch_bytes / case.layout.ld)
        s.close()
    assert per_cell[0] < 1.1 * per_cell[1], per_cell
