"""PPCG inner steps and Chebyshev iterations without a preconditioner or with
the diagonal one, each in one pass, against the CPU oracle bit for bit: tile
edges (two cells, 31 to 33 and 255 to 257 columns, 1 to 5 rows past a strip),
odd inner step counts, halo depths, reflective faces and the three arithmetic
forms; and grids of more supertiles than SMs, where the products run on the
integer pipes, at three and at four blocks per SM, for these, Jacobi and CG."""
import pytest

from oracle import oracle
from tealeaf_opencl_gb300 import lib
from tests import scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["ppcg", "chebyshev"])
@pytest.mark.parametrize("prec", ["none", "jac_diag"])
@pytest.mark.parametrize("x,y,halo,form,reflective", [
    (2, 1, 1, 1, False), (31, 5, 2, 2, False), (33, 6, 1, 0, True), (255, 7, 1, 1, True),
    (257, 13, 3, 2, True), (300, 67, 1, 1, False),
])
def test_one_pass_steps_match_oracle(solver, prec, x, y, halo, form, reflective):
    args = (x, y, halo, lib.SOLVER[solver], lib.PREC[prec])
    recs = [scenarios.run(mod.Chunk(*args), x, y, solver, prec, halo=halo, inner=5,
                          cg_iters=4 if x * y > 8 else 0, lognormal_seed=3, fused=form,
                          reflective=reflective) for mod in (lib, oracle)]
    assert scenarios.compare(*recs) == []


@pytest.mark.parametrize("solver,prec", [("ppcg", "none"), ("ppcg", "jac_diag"),
                                         ("chebyshev", "none"), ("chebyshev", "jac_diag"),
                                         ("jacobi", "none"), ("cg", "jac_diag")])
@pytest.mark.parametrize("x,y,halo,form", [(520, 331, 1, 1), (520, 331, 2, 0),
                                           (2050, 623, 1, 2)])
def test_larger_grids_match_oracle(solver, prec, x, y, halo, form):
    args = (x, y, halo, lib.SOLVER[solver], lib.PREC[prec])
    recs = [scenarios.run(mod.Chunk(*args), x, y, solver, prec, halo=halo, inner=3, cg_iters=2,
                          cheby_iters=2, jacobi_iters=3, lognormal_seed=5, fused=form,
                          snapshots=x < 1000) for mod in (lib, oracle)]
    assert scenarios.compare(*recs) == []
