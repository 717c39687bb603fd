"""GPU tests of the FP64 recompute beyond n = 236 where the pivot order of the FP32 factorisation is
of no use for the FP64 one: blocks whose FP32 entries overflow, and nearly singular ones.

Singlet pairing (uu and dd blocks zero): an order that pairs two up electrons meets an exactly zero
FP64 pivot.
"""

import numpy as np
import pytest

import neuralhubbard_b200 as nh
from neuralhubbard_b200 import _lib
from oracle import backflow as ob
from oracle import lattice as olat
from oracle import pfaffian as opf
from oracle import projection as oproj

pytestmark = pytest.mark.gpu


def singlet_params(Lx, Ly, seed, std, theta=0.55):
    p = nh.init_params(Lx, Ly, channels=32, layers=4, std=std, seed=seed)
    p["W"][1:] = 0.0
    p["theta"] = np.float32(theta)
    return p


def oracle_params(p, Lx, Ly):
    return dict(conv_w=[np.asarray(w, np.float64) for w in p["conv_w"]],
                conv_b=[np.asarray(b, np.float64) for b in p["conv_b"]],
                W=np.asarray(p["W"], np.float64), theta=float(p["theta"]), Lx=Lx, Ly=Ly)


def block64(s, op):
    """The oracle's occupied pairing blocks (B, n, n)."""
    y = ob.cnn_forward(s, op["conv_w"], op["conv_b"], op["Lx"], op["Ly"])
    idx = ob.fermion_idx(s)
    Wt = ob.build_wtilde(op["W"], op["theta"], op["Lx"], op["Ly"])
    return ob.pairing_occ(ob.occupied_features(y, idx), idx, Wt, op["Lx"], op["Ly"])


# 240: the FP32 matrix in shared memory; 300: in global memory.
@pytest.mark.parametrize("Lx,Ly,ne", [(16, 17, 120), (18, 18, 150)])
def test_fp32_overflow(Lx, Ly, ne):
    """Features scaled so that the largest FP32 products of two overflow: the FP32 order is arbitrary
    from the first infinity on, and the items it leaves with a pivot ratio of infinity (those with a
    finite pivot) are recomputed in FP64.  Well-conditioned blocks: the 1e-8 bar of the FP64 path."""
    p = singlet_params(Lx, Ly, 11, 0.3)
    N = Lx * Ly
    s = olat.random_configs(np.random.default_rng(11), 3, N, ne, ne)
    y = ob.cnn_forward(s, [np.asarray(w, np.float64) for w in p["conv_w"]],
                       [np.asarray(b, np.float64) for b in p["conv_b"]], Lx, Ly)
    scale = np.float32(1.3 * np.sqrt(float(np.finfo(np.float32).max)) / np.abs(y).max())
    p["conv_w"][-1] = p["conv_w"][-1] * scale
    p["conv_b"][-1] = p["conv_b"][-1] * scale
    s0, l0 = oproj.projected_amplitude(s, oracle_params(p, Lx, Ly), symm=False)
    psi = nh.Variational(nh.PfaffianBackflow(Lx, Ly, ne, ne, params=p), symm=False)(s)
    sg, la = psi.numpy()
    flags = psi.flags.cpu().numpy()
    redone = (flags & _lib.FLAG_REFINED != 0) & (flags & _lib.FLAG_NONFINITE == 0)
    assert redone.any(), flags
    assert np.array_equal(sg[redone], s0[redone])
    assert np.max(np.abs(la[redone] - l0[redone])) < 1e-8


@pytest.mark.parametrize("Lx,Ly,ne", [(16, 17, 120), (18, 18, 150)])
def test_near_singular(Lx, Ly, ne):
    """Short-ranged singlets: pivot ratios of 1e6 and more.  Whichever way they are factorised, the
    logarithm is held to n eps times the block's condition (plus the FP64 path's 1e-8)."""
    p = singlet_params(Lx, Ly, 5, 0.02, theta=4.0)
    s = olat.random_configs(np.random.default_rng(5), 12, Lx * Ly, ne, ne)
    op = oracle_params(p, Lx, Ly)
    F = block64(s, op)
    cond = np.linalg.cond(F)
    assert cond.max() > 1e6
    s0, l0 = oproj.projected_amplitude(s, op, symm=False)
    model = nh.PfaffianBackflow(Lx, Ly, ne, ne, params=p, cond_tau=1.0)
    sg, la = nh.Variational(model, symm=False)(s).numpy()
    assert np.array_equal(sg, s0)
    assert np.all(np.abs(la - l0) < 1e-8 + 2 * ne * np.finfo(np.float64).eps * cond)
