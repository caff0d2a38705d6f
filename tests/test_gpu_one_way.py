"""Matrices with links in one direction only (an entry without its transposed one): Gauss-Seidel and
agglomeration give what the sequential loops give, the same in every run."""
import numpy as np
import pytest

from matlab_ufvm_b200 import case
from test_gpu_agg import one_way
from test_gpu_wave import grid, same

pytestmark = pytest.mark.gpu


def one_way_grid(nx, ny, seed):
    """A grid that lost a fifth of its entries, most of them without the transposed one."""
    rp, col, ac, anb, bc = grid(nx, ny, 1)
    row = np.repeat(np.arange(len(ac)), np.diff(rp))
    keep = np.random.default_rng(seed).random(len(col)) < 0.8
    keep[np.unique(row, return_index=True)[1]] = True  # no row without an entry
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=len(ac)))]).astype(np.int32)
    return rp2, col[keep], ac, anb[keep], bc


def upper_only(n):
    """Every row reads the next ones, no row reads an earlier one: all rows could go first."""
    d = (1, 2, 5, 3000)
    rows = [[i + s for s in d if i + s < n] for i in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.array([j for r in rows for j in r], dtype=np.int32)
    rng = np.random.default_rng(1)
    return rp, col, rng.uniform(1.0, 2.0, n), -rng.uniform(0.1, 0.4, col.size), rng.normal(size=n)


SYSTEMS = {
    "random900": lambda: one_way(900), "random12000": lambda: one_way(12000), "grid40x30": lambda: one_way_grid(40, 30, 1),
    "grid90x91": lambda: one_way_grid(90, 91, 2), "grid250x130": lambda: one_way_grid(250, 130, 3),
    "grid3x20000": lambda: one_way_grid(3, 20000, 4), "upper9000": lambda: upper_only(9000), "upper60": lambda: upper_only(60),
    "grid1100x1000": lambda: one_way_grid(1100, 1000, 5),
}


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_gauss_seidel(ufvm_mod, oracle_mod, name):
    rp, col, ac, anb, bc = SYSTEMS[name]()
    x0 = np.random.default_rng(2).normal(size=len(ac))
    want = oracle_mod.sor_sweep(rp, col, ac, anb, bc, x0)
    for _ in range(3):
        same(ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0), want, "SOR")
    xg, _, _, it = ufvm_mod.cfdSolveAlgebraicSystem(rp, col, ac, anb, bc, x0, "SOR", 3, 1e-9)
    xo, _, _, jt = oracle_mod.solve_algebraic_system(rp, col, ac, anb, bc, x0, case.SMOOTHER["SOR"], 3, 1e-9, 0)
    assert it == jt
    same(xg, xo, "smoother call")


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_agglomeration(ufvm_mod, oracle_mod, name):
    rp, col, ac, anb, _ = SYSTEMS[name]()
    for got, want in zip(ufvm_mod.cfdAgglomerateLevel(rp, col, ac, anb), oracle_mod.agglomerate(rp, col, ac, anb)):
        same(got, want, "agglomeration")


def orphan_chains(lengths):
    """Blocks of two pairs (0, 1) and (2, 3), each an aggregate, and a chain of orphans that prefers, one
    after another, the lower orphan beside it, and at its end a later orphan still (one-way link, 0.45
    against 0.4), which is attached to the other pair and waits for nobody."""
    rows, at = [], 0
    for m in lengths:
        rows += [[(at + 1, 10.0)], [(at, 10.0)], [(at + 3, 10.0)], [(at + 2, 10.0)]]
        for k in range(m):
            rows.append([(at, 1.0)] + ([(at + 3 + k, 0.4)] if k else []) + ([(at + 4 + m, 0.45)] if k == m - 1 else []))
        rows.append([(at + 2, 1.0)])
        at += 5 + m
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.array([j for r in rows for j, _ in r], dtype=np.int32)
    return rp, col, np.full(at, 12.0), -np.array([w for r in rows for _, w in r])


@pytest.mark.parametrize("lengths", [(60,), (2, 30, 200, 7), tuple(range(2, 90))])
def test_orphans_in_order(ufvm_mod, oracle_mod, lengths):
    rp, col, ac, anb = orphan_chains(lengths)
    want = oracle_mod.agglomerate(rp, col, ac, anb)
    at = 0
    for k, m in enumerate(lengths):
        assert (want[0][at + 4:at + 4 + m] == want[0][at]).all() and want[0][at + 4 + m] == want[0][at + 2]
        at += 5 + m
    for _ in range(3):
        for got, w in zip(ufvm_mod.cfdAgglomerateLevel(rp, col, ac, anb), want):
            same(got, w, "agglomeration")
