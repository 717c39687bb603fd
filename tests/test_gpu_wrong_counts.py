"""GPU tests of configurations whose particle numbers are not the state's, among them one without any
electron: amplitude 0, and the other configurations of the call keep their bits.
"""

import numpy as np
import pytest
import torch

import neuralhubbard_b200 as nh
from oracle import lattice as olat

pytestmark = pytest.mark.gpu


def resconv_params(L, rng):
    return dict(net="resconv", embed=rng.normal(size=(64, 4)).astype(np.float32),
                conv_w=[(rng.normal(size=(64, 64, 3, 3)) * 0.04).astype(np.float32)] * 2,
                conv_b=[(rng.normal(size=64) * 0.1).astype(np.float32)] * 2,
                W=(rng.normal(size=(3, L * L, 32)) / np.sqrt(32)).astype(np.float32),
                theta=float(np.float32(0.55)))


@pytest.mark.parametrize("L,ne,net,kw", [
    (4, 5, "cnn", {}), (8, 28, "cnn", {}), (8, 28, "cnn", dict(cond_tau=1.0)),
    (8, 28, "cnn", dict(refine_tau=1.0, cond_tau=0.0)), (8, 28, "cnn", dict(pf_mode=1)),
    (16, 112, "cnn", dict(cnn_mode=2)), (16, 128, "cnn", dict(cond_tau=1.0)),
    (18, 150, "cnn", dict(cond_tau=1.0)), (8, 28, "resconv", dict(cond_tau=1.0)),
    (16, 112, "resconv", dict(cnn_mode=2))])
@pytest.mark.parametrize("symm", [False, True])
def test_amplitude_zero(L, ne, net, kw, symm):
    N = L * L
    rng = np.random.default_rng(N + ne)
    p = resconv_params(L, rng) if net == "resconv" else nh.init_params(L, L, std=0.05, seed=N)
    state = nh.Variational(nh.PfaffianBackflow(L, L, ne, ne, params=p, **kw), symm=symm)
    right = olat.random_configs(rng, 3, N, ne, ne)
    wrong = np.concatenate([np.full((1, 2 * N), -1, np.int8), np.zeros((1, 2 * N), np.int8),
                            olat.random_configs(rng, 1, N, ne, 0),
                            olat.random_configs(rng, 1, N, 0, ne),
                            olat.random_configs(rng, 1, N, ne - 1, ne),
                            olat.random_configs(rng, 1, N, ne + 1, ne + 1)])
    alone = state(right)
    psi = state(np.concatenate([wrong[:3], right, wrong[3:]]))
    assert torch.equal(psi.sign[3:6], alone.sign) and torch.equal(psi.logabs[3:6], alone.logabs)
    bad = torch.cat([psi.sign[:3], psi.sign[6:]])
    assert torch.all(bad == 0)
    assert torch.all(torch.cat([psi.logabs[:3], psi.logabs[6:]]) == -np.inf)


def test_bcs_amplitude_zero():
    L, ne = 8, 28
    p = nh.init_params(L, L, std=0.05, seed=3)
    p["W"], p["delta_d"] = p["W"][0], 0.1
    s = np.concatenate([np.full((2, 128), -1, np.int8),
                        olat.random_configs(np.random.default_rng(1), 2, 64, ne, ne)])
    psi = nh.Variational(nh.BCSBackflow(L, L, ne, ne, params=p))(s)
    assert torch.all(psi.sign[:2] == 0) and torch.all(psi.sign[2:] != 0)
