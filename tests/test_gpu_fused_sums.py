"""The sums of the fused FP64 iteration: the residual u, formed from the face
fluxes by the coefficient kernel, has the oracle's bits for each flux family;
the residual norms equal the oracle's for one CTA of partials, several CTAs of
one block, and more blocks than a warp has lanes."""
import numpy as np
import pytest

from codens_b200 import cases

from ._helpers import assert_equal_bits, oracle_prepared, real

pytestmark = pytest.mark.gpu


def _solver(case):
    from codens_b200.solver import CodeNS
    s = CodeNS(case)
    s.metric()
    return s


@pytest.mark.parametrize("cells", [(1, 1, 1), (5, 3, 4), (33, 9, 2)])
@pytest.mark.parametrize("ns,flux", [(0, 7), (0, 14), (1, 7), (1, 14), (1, 9), (1, 5)])
def test_residual_of_the_fused_step(cuda, ns, flux, cells):
    case = cases.box_case(cells, seed=9, ns=bool(ns), skew=0.01, reynz=1.0e3, lmax=2)
    case.scheme.ischema = flux
    orc, st = oracle_prepared(case)
    orc.step(st)
    s = _solver(case)
    s.atsch_num(1)
    ld, rc = case.layout.ld, real(case)
    u = s.u.cpu().numpy().reshape(-1, ld)[:5, rc]
    s.close()
    assert_equal_bits(u, np.asarray(st.u).reshape(-1, ld)[:5, rc], "residual")


@pytest.mark.parametrize("make", [
    lambda: cases.box_case((3, 2, 2), seed=9, lmax=2),
    lambda: cases.box_case((129, 65, 16), seed=9, lmax=2),
    lambda: cases.batch_case(ncase=37, side=(3, 9), seed=9, lmax=2)],
    ids=["one tile", "several chunks", "37 blocks"])
def test_norms_of_the_fused_step(cuda, make):
    case = make()
    orc, st = oracle_prepared(case)
    s = _solver(case)
    v0 = st.v.copy()
    orc.step(st)  # one iteration: the 37 boxes diverge in the second, in the oracle too
    # sums of at most 134160 positive terms in two orders: 1e-12 is 4500 eps
    np.testing.assert_allclose(s.atsch_num(1), orc.norms(v0, st), rtol=1e-12, atol=0)
    s.close()
