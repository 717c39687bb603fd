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
from oracle import projection as oproj

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-8


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
    assert np.max(np.abs(la - l0)) < TOL
