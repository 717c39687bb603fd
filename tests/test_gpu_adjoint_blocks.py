"""GPU tests of the Pfaffian adjoint at the edges of its blocks of eight pivot steps: matrices of
less than a block, a last block of two, four and six steps, a whole number of blocks, both sides of
each multiple of 32 (the register tile), the largest size; and a pivot that vanishes inside a block.

An FP32 Gauss-Jordan inverse with row pivoting is off by a small multiple of eps cond(A) relative
to its largest element: 2e-6 cond + 1e-6, the bar of the general adjoint tests.
"""

import numpy as np
import pytest
import torch

import neuralhubbard_b200 as nh
from neuralhubbard_b200 import _lib
from oracle import gradient as og

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [2, 4, 8, 10, 12, 30, 32, 34, 62, 64, 66, 96, 98, 128, 130, 160, 162,
                               190, 192, 194, 218, 220, 222, 224])
def test_block_edges(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(3, n, n))
    A = (A - np.swapaxes(A, 1, 2)).astype(np.float32)
    G, fl = nh.slogpf_adjoint(torch.from_numpy(A).to(DEV))
    G = G.cpu().numpy()
    G0 = og.slogpf_adjoint(A.astype(np.float64))
    cond = np.linalg.cond(A.astype(np.float64))
    assert np.all(fl.cpu().numpy() == 0)
    for b in range(A.shape[0]):
        scale = np.max(np.abs(G0[b]))
        assert np.max(np.abs(G[b] - G0[b])) <= 2e-6 * cond[b] * scale + 1e-6 * scale, b


@pytest.mark.parametrize("n,at", [(8, 0), (20, 11), (64, 37), (224, 223)])
def test_zero_column_inside_a_block(n, at):
    """A zero row and column gives an exact zero column at its step: flagged, zero cotangent; the
    other matrices of the launch are not touched by it."""
    rng = np.random.default_rng(n)
    A = rng.normal(size=(3, n, n))
    A = (A - np.swapaxes(A, 1, 2)).astype(np.float32)
    alone, _ = nh.slogpf_adjoint(torch.from_numpy(A).to(DEV))
    B = A.copy()
    B[1, at, :] = 0.0
    B[1, :, at] = 0.0
    G, fl = nh.slogpf_adjoint(torch.from_numpy(B).to(DEV))
    assert fl.cpu().tolist() == [0, _lib.FLAG_ZERO_PIVOT, 0]
    assert torch.all(G[1] == 0.0)
    assert torch.equal(G[0], alone[0]) and torch.equal(G[2], alone[2])
