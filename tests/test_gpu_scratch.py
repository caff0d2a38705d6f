"""The matrix functions' scratch can be given back by a program that has no case and no service."""
import numpy as np
import pytest

from test_gpu_wave import grid

pytestmark = pytest.mark.gpu


def test_release_scratch(ufvm_mod):
    import torch
    rp, col, ac, anb, bc = grid(700, 500, 1)
    x0 = np.zeros(len(ac))
    for _ in range(2):  # modules loaded, torch's own buffers allocated
        want = ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0)
    ufvm_mod.release_scratch()
    free = torch.cuda.mem_get_info()[0]
    got = ufvm_mod.cfdSolveSOR(rp, col, ac, anb, bc, x0)
    assert free - torch.cuda.mem_get_info()[0] > 32 << 20  # its ELL copies alone are 67 MB
    ufvm_mod.release_scratch()
    assert torch.cuda.mem_get_info()[0] == free
    assert np.array_equal(got, want)
    ufvm_mod.release_scratch()  # nothing to give back
