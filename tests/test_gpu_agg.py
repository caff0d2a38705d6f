"""Agglomeration and its Galerkin product against the sequential loops, at the sizes where their kernels
change: the one-block bound, rows with more than 32 links, coarse rows with more than 32 entries,
anisotropic couplings (few strong links, orphans), and a pattern that is not symmetric."""
import numpy as np
import pytest

from helpers import py_agglomerate, random_diag_dominant
from test_gpu_wave import from_pairs, grid, hub

pytestmark = pytest.mark.gpu


def aniso(nx, ny):
    rp, col, ac, anb, bc = grid(nx, ny, 1)
    row = np.repeat(np.arange(len(ac)), np.diff(rp))
    return rp, col, ac, np.where(np.abs(row - col) == 1, anb, 0.2 * anb), bc


def uniform(nx, ny, nz):
    rp, col, ac, anb, bc = grid(nx, ny, nz)
    return rp, col, ac, -np.ones_like(anb), bc


def one_way(n):
    """Random links, about a third of them without a transposed entry."""
    rp, col, ac, anb, bc = random_diag_dominant(n, 31, nbr=8)
    row = np.repeat(np.arange(n), np.diff(rp))
    keep = np.random.default_rng(32).random(len(col)) < 0.8
    keep[np.unique(row, return_index=True)[1]] = True  # no row without an entry
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=n))]).astype(np.int32)
    return rp2, col[keep], ac, anb[keep], bc


SYSTEMS = {
    "two": lambda: grid(2, 1, 1), "line40": lambda: uniform(40, 1, 1), "grid128x128": lambda: uniform(128, 128, 1),
    "grid2048": lambda: uniform(64, 32, 1), "grid2049": lambda: grid(683, 3, 1), "grid16385": lambda: grid(3277, 5, 1), "grid150x120": lambda: uniform(150, 120, 1), "aniso": lambda: aniso(131, 127),
    "cube28": lambda: uniform(28, 28, 28), "wide": lambda: random_diag_dominant(3000, 33, nbr=44), "hub": lambda: hub(100, 90),
    "one_way": lambda: one_way(900),
}


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_agglomerate(ufvm_mod, name):
    rp, col, ac, anb, _ = SYSTEMS[name]()
    parents, crp, ccol, cac, canb = ufvm_mod.cfdAgglomerateLevel(rp, col, ac, anb)
    want, nc = py_agglomerate(rp, col, anb)
    assert len(cac) == nc and np.array_equal(parents, want)
    conn = [[] for _ in range(nc)]
    val = [dict() for _ in range(nc)]
    diag = np.zeros(nc)
    for i in range(len(ac)):  # fine natural order (assembleAgglomeratedLHS.m:16-30)
        P = want[i]
        diag[P] += ac[i]
        for k in range(rp[i], rp[i + 1]):
            Q = int(want[col[k]])
            if Q == P:
                diag[P] += anb[k]
            else:
                if Q not in val[P]:
                    conn[P].append(Q)
                    val[P][Q] = 0.0
                val[P][Q] += anb[k]
    assert np.array_equal(np.diff(crp), [len(c) for c in conn])
    assert np.array_equal(ccol, np.array([q for c in conn for q in c], dtype=np.int32))
    assert np.array_equal(cac, diag)
    assert np.array_equal(canb, np.array([val[P][q] for P in range(nc) for q in conn[P]]))


def test_agglomerate_more_cells_than_the_lists(ufvm_mod, oracle_mod):
    """1.34M cells: a block's cells exceed its list, which it fills several times a round."""
    rp, col, ac, anb, _ = uniform(112, 110, 109)
    got = ufvm_mod.cfdAgglomerateLevel(rp, col, ac, anb)
    for a, b in zip(got, oracle_mod.agglomerate(rp, col, ac, anb)):
        assert np.array_equal(a, b)
