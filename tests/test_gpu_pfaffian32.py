"""GPU tests of the FP32 Pfaffian kernel at the edges of its forms: a single 32-row panel warp and
the first size beyond (32, 34), the last size of the 128-thread form (128, 130), of the 8-wide
panels (224, 226) and of the kernel (256).

Both thread counts run the same operations in the same order, so a matrix gives the same bits
whichever form the batch size selects; against the FP64 oracle the FP32 factorisation of Gaussian
matrices (condition ~ n^2) is held to the bar of the general Pfaffian tests, 1e-3 in the logarithm.
"""

import numpy as np
import pytest
import torch

import neuralhubbard_b200 as nh
from neuralhubbard_b200 import _lib
from oracle import pfaffian as opf

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [2, 16, 18, 32, 34, 126, 128, 130, 224, 226, 256])
def test_forms_agree(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(4, n, n)).astype(np.float32)
    A = A - np.swapaxes(A, 1, 2)
    few = nh.slogpf(torch.from_numpy(A).to(DEV), cond_tau=0.0)
    many = nh.slogpf(torch.from_numpy(np.tile(A, (100, 1, 1))).to(DEV), cond_tau=0.0)
    for x, y in zip(few, many):
        assert torch.equal(x.repeat(100), y)
    s0, l0 = opf.slogpf(A.astype(np.float64))
    assert np.array_equal(few[0].cpu().numpy(), s0)
    assert np.max(np.abs(few[1].cpu().numpy() - l0)) < 1e-3


def test_ties_zero_columns_and_nonfinite():
    """Equal magnitudes everywhere (every pivot search ties), a zero column met in the middle of
    the elimination, and an infinite entry; both forms give the same bits and flags."""
    n = 40
    rng = np.random.default_rng(5)
    A = np.zeros((4, n, n), np.float32)
    signs = np.triu(rng.choice([-1.0, 1.0], size=(n, n)), 1).astype(np.float32)
    A[0] = signs - signs.T
    B = rng.normal(size=(n, n)).astype(np.float32)
    A[1] = B - B.T
    A[1, :, 30] = A[1, 30, :] = 0.0
    A[2] = A[1]
    A[2, 3, 7], A[2, 7, 3] = np.inf, -np.inf
    A[3] = B - B.T
    few = nh.slogpf(torch.from_numpy(A).to(DEV), cond_tau=0.0)
    many = nh.slogpf(torch.from_numpy(np.tile(A, (100, 1, 1))).to(DEV), cond_tau=0.0)
    for x, y in zip(few, many):
        assert torch.equal(torch.nan_to_num(x.repeat(100)), torch.nan_to_num(y))
    sg, la, fl = (x.cpu().numpy() for x in few)
    s0, l0 = opf.slogpf(A[[0, 3]].astype(np.float64))
    assert np.array_equal(sg[[0, 3]], s0) and np.max(np.abs(la[[0, 3]] - l0)) < 1e-3
    assert sg[1] == 0 and la[1] == -np.inf and fl[1] & _lib.FLAG_ZERO_PIVOT
    assert fl[2] & (_lib.FLAG_NONFINITE | _lib.FLAG_ZERO_PIVOT)
