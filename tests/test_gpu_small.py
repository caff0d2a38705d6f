"""Smoother calls on levels that one block handles, and on the smallest ones that it does not: bits and
sweep counts against the oracle, at the edges of the size bound and of the row-width classes."""
import numpy as np
import pytest

from helpers import random_diag_dominant
from matlab_ufvm_b200 import case
from test_gpu_wave import grid, hub

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "two": lambda: grid(2, 1, 1), "line33": lambda: grid(33, 1, 1), "grid2048": lambda: grid(64, 32, 1),
    "grid2049": lambda: grid(683, 3, 1), "cube12": lambda: grid(12, 12, 12), "width10": lambda: random_diag_dominant(700, 21, nbr=8),
    "wide": lambda: random_diag_dominant(2000, 22, nbr=30), "hub": lambda: hub(300, 50),
}


@pytest.mark.parametrize("smoother", ["ILU", "SOR", "MCGS"])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_smoother_call(ufvm_mod, oracle_mod, name, smoother):
    rp, col, ac, anb, bc = SYSTEMS[name]()
    x0 = np.random.default_rng(3).normal(size=len(ac))
    for n_iter, rrf in ((0, 0.1), (1, 0.1), (7, 1e-6), (10, 0.1)):
        xg, r0, r1, it = ufvm_mod.cfdSolveAlgebraicSystem(rp, col, ac, anb, bc, x0, smoother, n_iter, rrf)
        xo, q0, q1, jt = oracle_mod.solve_algebraic_system(rp, col, ac, anb, bc, x0, case.SMOOTHER[smoother], n_iter, rrf,
                                                           case.QUIRKS_REFERENCE)
        assert it == jt
        assert np.array_equal(xg, xo)
        # sums of |r| over n rows in two orders: a few n eps apart at most
        tol = 4 * len(ac) * np.finfo(float).eps
        assert abs(r0 - q0) <= tol * abs(q0) and abs(r1 - q1) <= tol * abs(q1)
