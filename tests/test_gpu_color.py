"""The multicolour sweep against the oracle's, where its colouring and its colour kernels change:
chains longer than the threads that colour them, more than 64 and more than 256 colours (the bit
mask's and the shared histogram's ends), rows at the ends of the load batches (4, 5, 12, 13 entries)."""
import numpy as np
import pytest

from helpers import random_diag_dominant
from test_gpu_wave import from_pairs, grid

pytestmark = pytest.mark.gpu


def clique(n, extra=0):
    i, j = np.triu_indices(n, 1)
    tail = np.arange(n, n + extra)
    return from_pairs(n + extra, np.concatenate([i, tail - 1]), np.concatenate([j, tail]), n)


def band(n, w):
    own = np.concatenate([np.arange(n - d) for d in range(1, w + 1)])
    nei = np.concatenate([np.arange(d, n) for d in range(1, w + 1)])
    return from_pairs(n, own, nei, w)


SYSTEMS = {
    "two": lambda: grid(2, 1, 1), "chain40000": lambda: band(40000, 1), "band2": lambda: band(5000, 2),
    "band6": lambda: band(1025, 6), "cube": lambda: grid(17, 19, 23), "clique5": lambda: clique(5),
    "clique13": lambda: clique(13), "clique14": lambda: clique(14), "clique64": lambda: clique(64, 3),
    "clique65": lambda: clique(65, 3), "clique300": lambda: clique(300, 4000),
    "wide": lambda: random_diag_dominant(6000, 41, nbr=30),
}


@pytest.mark.parametrize("which", list(SYSTEMS))
def test_multicolour_sweep_bits(ufvm_mod, oracle_mod, which):
    import torch
    rp, col, ac, anb, bc = SYSTEMS[which]()
    nc, color = oracle_mod.coloring(rp, col)
    x = np.random.default_rng(7).normal(size=len(ac))
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rp, col, ac, anb, bc)]
    xd = torch.from_numpy(x.copy()).cuda()
    ufvm_mod.profile_plain_kernel("MCGS", *dev, xd, 1)  # one untimed sweep and one timed
    for _ in range(2):
        x = oracle_mod.mcgs_sweep(rp, col, ac, anb, bc, color, nc, x)
    assert np.array_equal(xd.cpu().numpy(), x)
