"""GPU tests of the FP64 recompute kernels at the sizes where their tilings change, against the
FP64 oracle: lattices whose site count is not a multiple of the 8-site tile, the largest of each
thread-count variant and the first beyond it.

With cond_tau = 1 every image goes through FP64 features and an FP64 factorisation, so the result
carries FP64 rounding amplified by the block's condition (at most ~1e6 here): 1e-8 absolute in the
logarithm, signs exact.
"""

import numpy as np
import pytest
import torch

import neuralhubbard_b200 as nh
from oracle import bcs as obcs
from oracle import lattice as olat
from oracle import pfaffian as opf
from oracle import projection as oproj

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-8


def log_error(la, l0):
    """Largest difference of the finite logarithms; the infinite ones (a sum that vanishes by
    symmetry) have to be the same."""
    fin = np.isfinite(l0)
    assert np.array_equal(la[~fin], l0[~fin])
    return np.max(np.abs(la[fin] - l0[fin]), initial=0.0)


def params_for(Lx, Ly, seed, ansatz="pfaffian"):
    p = nh.init_params(Lx, Ly, channels=32, layers=4, std=0.1, seed=seed)
    if ansatz == "bcs":
        p["W"] = p["W"][0]
        p["delta_d"] = 0.1
    return p


def oracle_params(p, Lx, Ly):
    return dict(conv_w=[np.asarray(w, np.float64) for w in p["conv_w"]],
                conv_b=[np.asarray(b, np.float64) for b in p["conv_b"]],
                W=np.asarray(p["W"], np.float64), theta=float(p["theta"]), Lx=Lx, Ly=Ly,
                **({"delta_d": p["delta_d"]} if "delta_d" in p else {}))


# 128 and 256 sites are the largest of the 256- and 512-thread forms; 130 and 272 the first
# beyond; 12, 15 x 2 and 90 leave a partial site tile.
@pytest.mark.parametrize("Lx,Ly", [(3, 4), (5, 6), (9, 10), (8, 16), (10, 13), (16, 16), (16, 17)])
def test_fp64_features_through_bcs(Lx, Ly):
    """FP64 CNN kernel (determinant ansatz, every image recomputed)."""
    N = Lx * Ly
    ne = min(max(2, 7 * N // 16), 112)
    p = params_for(Lx, Ly, N, "bcs")
    s = olat.random_configs(np.random.default_rng(N), 3, N, ne, ne)
    s0, l0 = obcs.projected_amplitude(s, oracle_params(p, Lx, Ly))
    model = nh.BCSBackflow(Lx, Ly, ne, ne, params=p, cond_tau=1.0)
    sg, la = nh.Variational(model)(s).numpy()
    assert np.array_equal(sg, s0)
    assert log_error(la, l0) < TOL


@pytest.mark.parametrize("n", [2, 6, 8, 10, 56, 110, 142, 222, 224])
def test_refine_dense(n):
    """Static-pivot FP64 factorisation of dense matrices: partial last panels (n mod 8 != 0), one
    panel only, both thread counts and the largest n."""
    rng = np.random.default_rng(n)
    A = rng.normal(size=(5, n, n)).astype(np.float32)
    A = A - np.swapaxes(A, 1, 2)
    s0, l0 = opf.slogpf(A.astype(np.float64))
    sg, la, _ = nh.slogpf(torch.from_numpy(A).to(DEV), cond_tau=1.0)
    assert np.array_equal(sg.cpu().numpy(), s0)
    assert np.max(np.abs(la.cpu().numpy() - l0)) < 1e-9


# n = 2 and n = 224; a partial tile; unequal spins; few sites per block; a lattice whose FP64
# features take the scalar path (16x17); 16 channels (d = 8).
@pytest.mark.parametrize("Lx,Ly,up,dn,symm,channels", [
    (3, 4, 1, 1, True, 32), (4, 4, 5, 3, True, 32), (8, 8, 28, 28, True, 32),
    (5, 6, 0, 8, False, 32), (9, 12, 50, 44, False, 32), (10, 14, 61, 59, False, 32),
    (16, 16, 112, 112, False, 32), (16, 17, 100, 98, False, 32), (8, 10, 35, 35, False, 16)])
def test_refine_gather(Lx, Ly, up, dn, symm, channels):
    """FP64 features, gather and factorisation of every image (cond_tau = 1), the fused form."""
    N = Lx * Ly
    p = nh.init_params(Lx, Ly, channels=channels, layers=4, std=0.1, seed=N + up)
    s = olat.random_configs(np.random.default_rng(N), 3, N, up, dn)
    s0, l0 = oproj.projected_amplitude(s, oracle_params(p, Lx, Ly), symm=symm)
    model = nh.PfaffianBackflow(Lx, Ly, up, dn, params=p, cond_tau=1.0)
    sg, la = nh.Variational(model, symm=symm)(s).numpy()
    assert np.array_equal(sg, s0)
    assert log_error(la, l0) < TOL


def test_refine_refuses_wide_cnn():
    """64 channels: the FP64 weights of a layer alone exceed shared memory."""
    p = nh.init_params(6, 8, channels=64, layers=4, std=0.1, seed=1)
    s = olat.random_configs(np.random.default_rng(1), 3, 48, 20, 22)
    model = nh.PfaffianBackflow(6, 8, 20, 22, params=p, cond_tau=1.0)
    with pytest.raises(nh.NativeLibraryError):
        nh.Variational(model)(s)


@pytest.mark.parametrize("cnn_mode", [0, 2])
def test_refine_stored_features(cnn_mode):
    """The unfused gather from stored FP64 rows (tensor-core CNN form; the residual network's
    d = 32 with its wider rows), projected."""
    L, N, ne = 16, 256, 112
    rng = np.random.default_rng(3)
    if cnn_mode == 2:
        p = params_for(L, L, 5)
        op = oracle_params(p, L, L)
    else:
        p = dict(net="resconv", embed=rng.normal(size=(64, 4)).astype(np.float32),
                 conv_w=[(rng.normal(size=(64, 64, 3, 3)) * 0.04).astype(np.float32)] * 2,
                 conv_b=[(rng.normal(size=64) * 0.1).astype(np.float32)] * 2,
                 W=(rng.normal(size=(3, N, 32)) / np.sqrt(32)).astype(np.float32),
                 theta=float(np.float32(0.55)))
        op = dict(p, Lx=L, Ly=L, W=np.asarray(p["W"], np.float64))
    s = olat.random_configs(rng, 2, N, ne, ne)
    s0, l0 = oproj.projected_amplitude(s, op)
    model = nh.PfaffianBackflow(L, L, ne, ne, params=p, cond_tau=1.0, cnn_mode=cnn_mode)
    sg, la = nh.Variational(model)(s).numpy()
    assert np.array_equal(sg, s0)
    assert log_error(la, l0) < TOL


# 128-row blocks are the largest two CTAs share in FP32 and the largest in FP64; 33 and 65 open a
# new column group.
@pytest.mark.parametrize("Lx,Ly,nh_", [(4, 4, 1), (8, 8, 32), (8, 9, 33), (10, 13, 65),
                                       (16, 16, 128)])
def test_determinant_blocks(Lx, Ly, nh_):
    """BCS determinant at the edges of its register blocks: all FP64 against the oracle, and the
    default mixed path within the 1e-4 bar of the mixed forms."""
    N = Lx * Ly
    p = params_for(Lx, Ly, 7 * N + nh_, "bcs")
    s = olat.random_configs(np.random.default_rng(nh_), 2, N, nh_, nh_)
    s0, l0 = obcs.projected_amplitude(s, oracle_params(p, Lx, Ly))
    for tau, tol in ((1.0, TOL), (5.0, 1e-4)):
        model = nh.BCSBackflow(Lx, Ly, nh_, nh_, params=p, cond_tau=tau)
        sg, la = nh.Variational(model)(s).numpy()
        assert np.array_equal(sg, s0)
        assert log_error(la, l0) < tol


# 6 sites to a partial tile, 64 (half of the warps), 16 x 16 (the largest of the cluster form) and
# 10 x 28 beyond it.
@pytest.mark.parametrize("Lx,Ly,ne,blocks", [(3, 4, 3, 1), (5, 6, 10, 2), (8, 8, 28, 3),
                                             (16, 16, 100, 2), (10, 28, 60, 1)])
def test_resconv_fp64(Lx, Ly, ne, blocks):
    """FP64 residual network: one cluster of two CTAs per image, more images than clusters."""
    N = Lx * Ly
    rng = np.random.default_rng(N)
    p = dict(net="resconv", embed=rng.normal(size=(64, 4)).astype(np.float32),
             conv_w=[(rng.normal(size=(64, 64, 3, 3)) * 0.04).astype(np.float32)
                     for _ in range(2 * blocks)],
             conv_b=[(rng.normal(size=64) * 0.1).astype(np.float32) for _ in range(2 * blocks)],
             W=(rng.normal(size=(3, N, 32)) / np.sqrt(32)).astype(np.float32),
             theta=float(np.float32(0.55)))
    s = olat.random_configs(rng, 3, N, ne, ne)
    s0, l0 = oproj.projected_amplitude(s, dict(p, Lx=Lx, Ly=Ly, W=np.asarray(p["W"], np.float64)))
    model = nh.PfaffianBackflow(Lx, Ly, ne, ne, params=p, cond_tau=1.0)
    sg, la = nh.Variational(model)(np.tile(s, (6, 1))).numpy()
    assert np.array_equal(sg, np.tile(s0, 6))
    assert log_error(la, np.tile(l0, 6)) < TOL


# 238 is the first size of the form with its tiles in global memory (236 the last of the pivoted
# one); partial tiles; 16x17 with the table staged, 31x33 not; the largest n.
@pytest.mark.parametrize("Lx,Ly,up,dn,symm", [(16, 17, 118, 118, False), (16, 17, 120, 118, True),
                                              (18, 20, 121, 119, False), (20, 19, 180, 176, False),
                                              (24, 24, 252, 252, False), (32, 32, 512, 512, False)])
def test_refine_large(Lx, Ly, up, dn, symm):
    N = Lx * Ly
    p = nh.init_params(Lx, Ly, channels=32, layers=4, std=0.05, seed=N + up)
    s = olat.random_configs(np.random.default_rng(N), 2, N, up, dn)
    s0, l0 = oproj.projected_amplitude(s, oracle_params(p, Lx, Ly), symm=symm)
    model = nh.PfaffianBackflow(Lx, Ly, up, dn, params=p, cond_tau=1.0)
    sg, la = nh.Variational(model, symm=symm)(np.tile(s, (30, 1))).numpy()
    assert np.array_equal(sg, np.tile(s0, 30))
    assert log_error(la, np.tile(l0, 30)) < TOL
