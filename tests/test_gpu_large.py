"""The sweeps on systems of millions of rows, bit for bit against the oracle: chunks whose
levels do not fit in shared memory while the schedule is made (more than about a million rows, 4,000
levels), and chunks whose values do not either (more than 4.17 million rows)."""
import numpy as np
import pytest

from matlab_ufvm_b200 import case
from test_gpu_wave import from_pairs, grid, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2000, 2000), (2100, 2001)])
def test_sweeps_of_large_grids(ufvm_mod, oracle_mod, nx, ny):
    rp, col, ac, anb, bc = grid(nx, ny, 1)
    x0 = np.random.default_rng(4).normal(size=len(ac))
    same(ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0), oracle_mod.sor_sweep(rp, col, ac, anb, bc, x0), "SOR")
    dc = ufvm_mod.cfdFactorizeILU(rp, col, ac, anb, 0)
    same(dc, oracle_mod.ilu_factor(rp, col, ac, anb, 0), "factor")
    same(ufvm_mod.cfdSolveILU(rp, col, ac, anb, bc, dc, x0), oracle_mod.ilu_sweep(rp, col, ac, anb, bc, dc, x0), "ILU")


def test_a_chain_longer_than_the_bound_of_a_wait(ufvm_mod, oracle_mod):
    """1.3 million rows in one chain: finding its levels takes several seconds, more than the bound of
    a single wait, and the last chunk waits for all the others."""
    rp, col, ac, anb, bc = grid(1_300_000, 1, 1)
    x0 = np.random.default_rng(4).normal(size=len(ac))
    same(ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0), oracle_mod.sor_sweep(rp, col, ac, anb, bc, x0), "SOR")


@pytest.mark.parametrize("nx,ny", [(1000, 700), (70000, 9)])
def test_multicolour_call_of_large_grids(ufvm_mod, oracle_mod, nx, ny):
    """More rows than the threads that colour them."""
    rp, col, ac, anb, bc = grid(nx, ny, 1)
    x0 = np.random.default_rng(4).normal(size=len(ac))
    xg, _, _, it = ufvm_mod.cfdSolveAlgebraicSystem(rp, col, ac, anb, bc, x0, "MCGS", 2, 1e-9)
    xo, _, _, jt = oracle_mod.solve_algebraic_system(rp, col, ac, anb, bc, x0, case.SMOOTHER["MCGS"], 2, 1e-9, 0)
    assert it == jt
    same(xg, xo, "MCGS")


def coloured_grid(nx, ny, k):
    """A grid whose rows are numbered by (i + j) mod k first: about k dependency levels."""
    c = np.arange(nx * ny).reshape(ny, nx)
    key = np.add.outer(np.arange(ny), np.arange(nx)) % k
    num = np.empty(nx * ny, dtype=np.int64)
    num[np.lexsort((c.ravel(), key.ravel()))] = np.arange(nx * ny)
    own = num[np.concatenate([c[:, :-1].ravel(), c[:-1].ravel()])]
    nei = num[np.concatenate([c[:, 1:].ravel(), c[1:].ravel()])]
    return from_pairs(nx * ny, np.minimum(own, nei), np.maximum(own, nei), 9)


@pytest.mark.parametrize("nx,ny,k", [(553, 549, 2), (700, 601, 7), (1100, 1000, 3)])
def test_sweeps_of_few_wide_levels(ufvm_mod, oracle_mod, nx, ny, k):
    """More rows than one chunk of 2,048 for every SM, in levels wide enough for two chunks on each."""
    rp, col, ac, anb, bc = coloured_grid(nx, ny, k)
    x0 = np.random.default_rng(4).normal(size=len(ac))
    same(ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0), oracle_mod.sor_sweep(rp, col, ac, anb, bc, x0), "SOR")
    dc = ufvm_mod.cfdFactorizeILU(rp, col, ac, anb, 0)
    same(dc, oracle_mod.ilu_factor(rp, col, ac, anb, 0), "factor")
    same(ufvm_mod.cfdSolveILU(rp, col, ac, anb, bc, dc, x0), oracle_mod.ilu_sweep(rp, col, ac, anb, bc, dc, x0), "ILU")


def test_colours_of_a_large_clique(ufvm_mod, oracle_mod):
    """A row of more than 64 colours looks for its own colour by colour, so the last of 640 rows that are
    all coupled waits longer for the others than the bound of a wait."""
    n = 640
    own, nei = np.triu_indices(n, 1)
    rp, col, ac, anb, bc = from_pairs(n, own, nei, 8)
    x0 = np.random.default_rng(4).normal(size=n)
    xg, _, _, it = ufvm_mod.cfdSolveAlgebraicSystem(rp, col, ac, anb, bc, x0, "MCGS", 2, 1e-9)
    xo, _, _, jt = oracle_mod.solve_algebraic_system(rp, col, ac, anb, bc, x0, case.SMOOTHER["MCGS"], 2, 1e-9, 0)
    assert it == jt
    same(xg, xo, "MCGS")
