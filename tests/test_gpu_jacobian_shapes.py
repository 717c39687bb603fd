"""GPU tests of the Jacobian's kernels at the sizes where their splits change: the gather's cotangents
at both sides of 64 and 128 rows (4, 8 and 16 rows per warp) on a rectangular lattice, for sorted
and unsorted mode lists, and whole Jacobians on lattices with Lx != Ly whose row count the split of
the weight cotangent does not divide.

Cotangents are FP32 sums of at most n products: 1e-5 of the largest value, the bar of the square
lattices.  Jacobian rows carry the FP32 inverse of the block: a small multiple of eps cond(F), held
to 2e-6 cond + 1e-5 of the row's largest entry.
"""

import numpy as np
import pytest
import torch

import neuralhubbard_b200 as nh
from neuralhubbard_b200 import _lib
from oracle import backflow as obf
from oracle import gradient as og
from oracle import lattice as olat

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 2, 31, 63, 64, 65, 127, 128, 129, 160, 224])
@pytest.mark.parametrize("d", [8, 16, 32])
def test_pairing_vjp_rows(n, d):
    if d == 32 and n > 160:
        pytest.skip("32 channels and 224 rows exceed shared memory")
    Lx, Ly = 14, 16
    N = Lx * Ly
    rng = np.random.default_rng(100 * n + d)
    idx = np.stack([rng.choice(2 * N, n, replace=False) for _ in range(3)])
    idx[:2].sort(axis=1)  # the third list mixes the spins
    Y = rng.normal(size=(3, n, d)).astype(np.float32)
    Wt = rng.normal(size=(4, N, d)).astype(np.float32)
    G = rng.normal(size=(3, n, n)).astype(np.float32)
    geom = nh.PairGeometry(Lx, Ly, d, n // 2, n - n // 2)
    dY, dWt = nh.pairing_occ_vjp(torch.from_numpy(Y).to(DEV),
                                 torch.from_numpy(idx.astype(np.int32)).to(DEV),
                                 torch.from_numpy(Wt).to(DEV), torch.from_numpy(G).to(DEV), geom)
    dY0, dWt0 = og.pairing_occ_vjp(Y.astype(np.float64), idx, Wt.astype(np.float64),
                                   G.astype(np.float64), Lx, Ly)
    assert np.max(np.abs(dY.cpu().numpy() - dY0)) <= 1e-5 * np.abs(dY0).max()
    assert np.max(np.abs(dWt.cpu().numpy() - dWt0)) <= 1e-5 * np.abs(dWt0).max()


@pytest.mark.parametrize("Lx,Ly,up,dn", [(3, 4, 2, 2), (5, 6, 12, 12), (6, 4, 9, 7), (7, 10, 30, 28),
                                         (10, 7, 30, 30), (13, 8, 40, 44)])
@pytest.mark.parametrize("channels,layers", [(16, 1), (16, 3), (32, 4)])
def test_jacobian_rectangular(Lx, Ly, up, dn, channels, layers):
    p = nh.init_params(Lx, Ly, channels=channels, layers=layers, std=0.2, seed=Lx * Ly + channels)
    op = dict(conv_w=[np.asarray(w, np.float64) for w in p["conv_w"]],
              conv_b=[np.asarray(b, np.float64) for b in p["conv_b"]],
              W=np.asarray(p["W"], np.float64), theta=float(p["theta"]), Lx=Lx, Ly=Ly)
    s = olat.random_configs(np.random.default_rng(Lx * Ly + layers), 5, Lx * Ly, up, dn)
    y = obf.cnn_forward(s, op["conv_w"], op["conv_b"], Lx, Ly)
    idx = obf.fermion_idx(s)
    F = obf.pairing_occ(obf.occupied_features(y, idx), idx,
                        obf.build_wtilde(op["W"], op["theta"], Lx, Ly), Lx, Ly)
    cond = np.linalg.cond(F)
    model = nh.PfaffianBackflow(Lx, Ly, up, dn, params=p)
    _, J = nh.Variational(model, symm=False).jacobian(s)
    J0 = og.log_jacobian(s, op, symm=False)[2]
    err = np.max(np.abs(J.cpu().numpy() - J0), axis=1) / np.max(np.abs(J0), axis=1)
    assert np.all(err <= 2e-6 * cond + 1e-5), (err, cond)


@pytest.mark.parametrize("Lx,Ly,up,dn,channels", [(4, 4, 5, 5, 32), (5, 6, 12, 12, 16),
                                                  (10, 11, 40, 40, 32), (10, 12, 40, 40, 32)])
def test_jacobian_many_samples(Lx, Ly, up, dn, channels):
    """More samples than SMs take the 256-thread form of the CNN cotangents where two CTAs fit (up to
    10x11): its rows against those of the 512-thread form, which sum the lattice's rows in another
    split.  FP32 sums of N terms: N eps of the row's largest entry, times ten for the layers."""
    N = Lx * Ly
    p = nh.init_params(Lx, Ly, channels=channels, layers=4, std=0.2, seed=N)
    state = nh.Variational(nh.PfaffianBackflow(Lx, Ly, up, dn, params=p), symm=False)
    s = olat.random_configs(np.random.default_rng(N), 30, N, up, dn)
    few = state.jacobian(s)[1].cpu().numpy()
    many = state.jacobian(np.tile(s, (20, 1)))[1].cpu().numpy()
    scale = np.max(np.abs(few), axis=1, keepdims=True)
    assert np.array_equal(many, np.tile(many[:30], (20, 1)))
    assert np.max(np.abs(many[:30] - few) / scale) <= 10 * N * np.finfo(np.float32).eps


@pytest.mark.parametrize("n", [8, 20, 64, 100, 222, 224])
def test_adjoint_ties_and_nonfinite(n):
    """Matrices with +-1 everywhere (the pivot searches tie) against the oracle, beside a zero, an
    infinite and a NaN entry's matrix, which are flagged and leave the others' bits alone."""
    rng = np.random.default_rng(n)
    U = np.triu(rng.choice([-1.0, 1.0], size=(5, n, n)), 1)
    A = (U - np.swapaxes(U, 1, 2)).astype(np.float32)
    A[2] = 0.0
    A[3, n - 1, 0], A[3, 0, n - 1] = np.inf, -np.inf
    A[4, n // 2, 1], A[4, 1, n // 2] = np.nan, np.nan
    G, fl = nh.slogpf_adjoint(torch.from_numpy(A).to(DEV))
    alone, _ = nh.slogpf_adjoint(torch.from_numpy(A[:2]).to(DEV))
    assert torch.equal(G[:2], alone)
    fl = fl.cpu().numpy()
    assert np.all(fl[:2] == 0) and fl[2] == _lib.FLAG_ZERO_PIVOT
    assert np.all(fl[3:] == _lib.FLAG_NONFINITE)
    assert torch.all(G[2] == 0.0)
    G0 = og.slogpf_adjoint(A[:2].astype(np.float64))
    cond = np.linalg.cond(A[:2].astype(np.float64))
    for b in range(2):
        scale = np.max(np.abs(G0[b]))
        assert np.max(np.abs(G[b].cpu().numpy() - G0[b])) <= (2e-6 * cond[b] + 1e-6) * scale
