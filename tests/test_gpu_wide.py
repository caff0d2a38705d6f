"""Rows far wider than the others, and entries listed more than once, in the natural-order sweeps."""
import numpy as np
import pytest

from test_gpu_wave import from_pairs, grid, same

pytestmark = pytest.mark.gpu


def star(n, hub):
    """One row coupled to all others."""
    leaf = np.delete(np.arange(n), hub)
    return from_pairs(n, np.minimum(leaf, hub), np.maximum(leaf, hub), 3)


def repeated(n, both):
    """A line whose entries (i, i + 1) are listed twice, every third one in one direction only or (both)
    every one in both directions."""
    rp, col, ac, anb, bc = grid(n, 1, 1)
    row = np.repeat(np.arange(n), np.diff(rp))
    rep = np.where(both | ((col > row) & (row % 3 == 0)), 2, 1)
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(row, weights=rep, minlength=n))]).astype(np.int32)
    return rp2, np.repeat(col, rep), 2.5 * ac, np.repeat(anb, rep), bc


def check_sor(ufvm_mod, oracle_mod, sys_):
    rp, col, ac, anb, bc = sys_
    x0 = np.random.default_rng(2).normal(size=len(ac))
    want = oracle_mod.sor_sweep(rp, col, ac, anb, bc, x0)
    for _ in range(2):
        same(ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0), want, "SOR")
    return x0


@pytest.mark.parametrize("n", [3, 50, 9000])
@pytest.mark.parametrize("both", [False, True])
def test_repeated_entries(ufvm_mod, oracle_mod, n, both):
    check_sor(ufvm_mod, oracle_mod, repeated(n, both))


@pytest.mark.parametrize("n,hub", [(6000, 0), (6000, 5999), (9001, 4500), (131072, 0)])
def test_one_row_coupled_to_all(ufvm_mod, oracle_mod, n, hub):
    rp, col, ac, anb, bc = star(n, hub)
    x0 = check_sor(ufvm_mod, oracle_mod, (rp, col, ac, anb, bc))
    dc = ufvm_mod.cfdFactorizeILU(rp, col, ac, anb, 0)
    same(dc, oracle_mod.ilu_factor(rp, col, ac, anb, 0), "factor")
    same(ufvm_mod.cfdSolveILU(rp, col, ac, anb, bc, dc, x0), oracle_mod.ilu_sweep(rp, col, ac, anb, bc, dc, x0), "ILU")


@pytest.mark.parametrize("wide", [25, 32, 33, 41, 64, 65, 72, 73, 300])
def test_few_wide_rows(ufvm_mod, oracle_mod, wide):
    """Rows at the width that the sweeps' copies of the matrix end at, in one chunk and in several."""
    for n in (2100, 30000):
        rng = np.random.default_rng(wide)
        own, nei = [np.arange(n - 1)], [np.arange(1, n)]
        for h in (0, n // 2, n - 1):  # the line gives each of them one or two entries already
            far = rng.choice(np.setdiff1d(np.arange(n), [h - 1, h, h + 1]), wide - 1, replace=False)
            own.append(np.minimum(h, far))
            nei.append(np.maximum(h, far))
        own, nei = np.unique(np.stack([np.concatenate(own), np.concatenate(nei)]), axis=1)
        rp, col, ac, anb, bc = from_pairs(n, own, nei, wide)
        x0 = check_sor(ufvm_mod, oracle_mod, (rp, col, ac, anb, bc))
        dc = ufvm_mod.cfdFactorizeILU(rp, col, ac, anb, 0)
        same(dc, oracle_mod.ilu_factor(rp, col, ac, anb, 0), "factor")
        same(ufvm_mod.cfdSolveILU(rp, col, ac, anb, bc, dc, x0), oracle_mod.ilu_sweep(rp, col, ac, anb, bc, dc, x0), "ILU")
