"""The chunked-wavefront sweeps (natural-order Gauss-Seidel, DILU) against the oracle, bit for bit, at
the sizes where their schedules change shape: two rows, partial tasks, the largest one-chunk level and
the smallest many-chunk one, wide levels, rows wider than the kernel's registers, levels that spread
over more than a chunk's counters, matrices that are not structurally symmetric, and operands far
outside the exponents of ordinary fields (the quotient's own path)."""
import numpy as np
import pytest

from helpers import random_diag_dominant
from matlab_ufvm_b200 import case

pytestmark = pytest.mark.gpu


def from_pairs(n, own, nei, seed):
    """cconn-ordered CSR of a symmetric pattern given by faces (own < nei), seeded values."""
    rng = np.random.default_rng(seed)
    own, nei = np.asarray(own, dtype=np.int64), np.asarray(nei, dtype=np.int64)
    f = np.arange(own.size)
    row, col, face = np.concatenate([own, nei]), np.concatenate([nei, own]), np.concatenate([f, f])
    o = np.lexsort((face, row))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    g = rng.uniform(0.1, 1.0, own.size)
    anb = -g[face[o]]
    ac = np.bincount(row, weights=g[face], minlength=n) * rng.uniform(1.05, 1.5, n) + 1e-3
    return rowptr, col[o].astype(np.int32), ac, anb, rng.normal(size=n)


def grid(nx, ny, nz):
    c = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    own = np.concatenate([c[:, :, :-1].ravel(), c[:, :-1, :].ravel(), c[:-1].ravel()])
    nei = np.concatenate([c[:, :, 1:].ravel(), c[:, 1:, :].ravel(), c[1:].ravel()])
    o = np.lexsort((nei, own))
    return from_pairs(nx * ny * nz, own[o], nei[o], 5)


def chain_and_loners(n):
    """Even rows form one chain, odd rows stand alone."""
    e = np.arange(0, n - 2, 2)
    return from_pairs(n, e, e + 2, 6)


def hub(n, width):
    """A few rows coupled to `width` others each."""
    own, nei = [], []
    for h in range(3):
        for k in range(width):
            own.append(h)
            nei.append(3 + (h * 7 + k) % (n - 3))
    return from_pairs(n, own, nei, 7)


SYSTEMS = {
    "two": lambda: grid(2, 1, 1), "line31": lambda: grid(31, 1, 1),
    "line33": lambda: grid(33, 1, 1), "grid90x91": lambda: grid(90, 91, 1), "grid91x91": lambda: grid(91, 91, 1),
    "grid8192": lambda: grid(128, 64, 1), "grid8193": lambda: grid(2731, 3, 1), "grid250x130": lambda: grid(250, 130, 1),
    "cube31": lambda: grid(31, 31, 31), "random4000": lambda: random_diag_dominant(4000, 11, nbr=6),
    "random12000": lambda: random_diag_dominant(12000, 12, nbr=40), "hub": lambda: hub(500, 60),
    "chain9000": lambda: chain_and_loners(9000), "chain60000": lambda: chain_and_loners(60000),
}


def same(a, b, what):
    assert np.array_equal(np.asarray(a), np.asarray(b)), (what, int(np.count_nonzero(a != b)))


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_sweeps_bit_exact(ufvm_mod, oracle_mod, name):
    rp, col, ac, anb, bc = SYSTEMS[name]()
    x0 = np.random.default_rng(2).normal(size=len(ac))
    same(ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0), oracle_mod.sor_sweep(rp, col, ac, anb, bc, x0), "SOR")
    for q in (case.QUIRKS_REFERENCE, 0):
        dc = ufvm_mod.cfdFactorizeILU(rp, col, ac, anb, q)
        same(dc, oracle_mod.ilu_factor(rp, col, ac, anb, q), "factor")
    same(ufvm_mod.cfdSolveILU(rp, col, ac, anb, bc, dc, x0), oracle_mod.ilu_sweep(rp, col, ac, anb, bc, dc, x0), "ILU")


@pytest.mark.parametrize("scale_a,scale_b", [(1.0, 0.0), (1e-280, 1e-300), (1e250, 1e-250), (1e-120, 1e180), (1.0, 5e-324),
                                             (1e-100, 1e-310), (1e160, 1e307)])
def test_quotient_outside_ordinary_exponents(ufvm_mod, oracle_mod, scale_a, scale_b):
    rp, col, ac, anb, bc = grid(40, 33, 1)
    rng = np.random.default_rng(8)
    x0 = rng.normal(size=len(ac)) * (scale_b if scale_b else 0.0)
    with np.errstate(all="ignore"):
        a, w, b = ac * scale_a, anb * scale_a, np.where(rng.random(len(ac)) < 0.5, bc * scale_b, 0.0)
        x0 = x0 / scale_a if np.isfinite(x0 / scale_a).all() else x0
    g, o = ufvm_mod.cfdSolveSOR(rp, col, a, w, b, x0), oracle_mod.sor_sweep(rp, col, a, w, b, x0)
    assert np.array_equal(g, o, equal_nan=True)


def test_pattern_that_is_not_symmetric(ufvm_mod):
    """DILU with lower entries only: dc = 1 / ac, a forward substitution, nothing backward."""
    n = 3000
    rng = np.random.default_rng(9)
    rows = [sorted(set(rng.integers(max(0, i - 40), i, size=3).tolist())) if i else [] for i in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.array([j for r in rows for j in r], dtype=np.int32)
    anb, ac, bc, x0 = -rng.uniform(0.1, 0.3, col.size), rng.uniform(1.0, 2.0, n), rng.normal(size=n), rng.normal(size=n)
    dc = ufvm_mod.cfdFactorizeILU(rp, col, ac, anb, 0)
    same(dc, 1.0 / ac, "factor")
    r = np.zeros(n)
    for i in range(n):
        v = -ac[i] * x0[i] + bc[i]
        for k in range(rp[i], rp[i + 1]):
            v = v - anb[k] * x0[col[k]]
        r[i] = v
    for i in range(n):
        for k in range(rp[i], rp[i + 1]):
            r[i] = r[i] - anb[k] * (dc[col[k]] * r[col[k]])
    same(ufvm_mod.cfdSolveILU(rp, col, ac, anb, bc, dc, x0), x0 + dc * r, "ILU")
