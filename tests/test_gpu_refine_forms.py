"""GPU tests of the FP64 refinement's two thread counts: with more matrices than SMs it runs two CTAs
of 256 threads per SM where 111 KB of shared memory hold one, else one of 512.

Both run the same operations on a matrix, so a matrix gives the same bits whichever form the number
of matrices selects; against the FP64 oracle the factorisation of Gaussian matrices is held to 1e-9
and the amplitudes to 1e-8, as in the tests of few matrices.
"""

import numpy as np
import pytest
import torch

import neuralhubbard_b200 as nh
from neuralhubbard_b200 import _lib
from oracle import backflow as obf
from oracle import lattice as olat
from oracle import pfaffian as opf
from oracle import projection as oproj

pytestmark = pytest.mark.gpu
DEV = "cuda"


def oracle_params(p, Lx, Ly):
    return dict(conv_w=[np.asarray(w, np.float64) for w in p["conv_w"]],
                conv_b=[np.asarray(b, np.float64) for b in p["conv_b"]],
                W=np.asarray(p["W"], np.float64), theta=float(p["theta"]), Lx=Lx, Ly=Ly)


# 152 rows (19 tiles: 107 KB) are the largest of the 256-thread form, 154 the first beyond; 10 and 142
# leave a partial panel.
@pytest.mark.parametrize("n", [2, 10, 56, 142, 152, 154])
def test_dense(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(5, n, n)).astype(np.float32)
    A = A - np.swapaxes(A, 1, 2)
    few = nh.slogpf(torch.from_numpy(A).to(DEV), cond_tau=1.0)
    many = nh.slogpf(torch.from_numpy(np.tile(A, (80, 1, 1))).to(DEV), cond_tau=1.0)
    for x, y in zip(few, many):
        assert torch.equal(x.repeat(80), y)
    s0, l0 = opf.slogpf(A.astype(np.float64))
    assert np.array_equal(many[0][:5].cpu().numpy(), s0)
    assert np.max(np.abs(many[1][:5].cpu().numpy() - l0)) < 1e-9


def fp32_block_logabs(model, s, idx):
    """log|pf| in FP64 of the FP32 pairing blocks that the library factorises."""
    Y = obf.occupied_features(model.features(torch.from_numpy(s).to(DEV)).cpu().numpy(), idx)
    F = nh.pairing_occ(torch.from_numpy(Y).to(DEV),
                       torch.from_numpy(idx.astype(np.int32)).to(DEV), model.Wt, model.geom)
    return opf.slogpf(F.cpu().numpy().astype(np.float64))[1]


def check_forms(channels, Lx, Ly, up, dn, refine_tau, pf_mode):
    """All-FP64 (cond_tau = 1), or (refine_tau = 1, cond_tau off) the FP64 factorisation of every FP32
    block, against the oracle and between the two thread counts."""
    N = Lx * Ly
    p = nh.init_params(Lx, Ly, channels=channels, layers=4, std=0.1, seed=N + channels)
    s = olat.random_configs(np.random.default_rng(N), 6, N, up, dn)
    s0, l0 = oproj.projected_amplitude(s, oracle_params(p, Lx, Ly), symm=False)
    model = nh.PfaffianBackflow(Lx, Ly, up, dn, params=p, cond_tau=0.0 if refine_tau else 1.0,
                                refine_tau=refine_tau, pf_mode=pf_mode)
    if refine_tau:
        l0 = fp32_block_logabs(model, s, obf.fermion_idx(s))
    state = nh.Variational(model, symm=False)
    few, many = state(s), state(np.tile(s, (50, 1)))
    assert torch.equal(few.sign.repeat(50), many.sign)
    assert torch.equal(few.logabs.repeat(50), many.logabs)
    assert torch.all(few.flags & _lib.FLAG_REFINED != 0)
    sg, la = few.numpy()
    assert np.array_equal(sg, s0)
    assert np.max(np.abs(la - l0)) < 1e-8


# Features computed in the kernel (fused form, bare states): with 32 channels 8x8 at n = 56 and 8x10
# at n = 20 still take two CTAs, 8x10 at n = 68 the first that does not; with 16 channels (scalar FP64
# network) 12x14 does and 16x12 does not.
@pytest.mark.parametrize("channels,Lx,Ly,up,dn", [
    (32, 3, 4, 2, 2), (32, 6, 6, 17, 13), (32, 8, 8, 28, 28), (32, 8, 10, 10, 10),
    (32, 8, 10, 33, 35), (32, 8, 16, 55, 57), (16, 4, 4, 7, 7), (16, 8, 8, 28, 26),
    (16, 12, 14, 71, 69), (16, 16, 12, 84, 84)])
@pytest.mark.parametrize("refine_tau", [0.0, 1.0])
def test_in_kernel_features(channels, Lx, Ly, up, dn, refine_tau):
    check_forms(channels, Lx, Ly, up, dn, refine_tau, 0)


# Stored rows (the tensor-memory Pfaffian's form): the separate FP64 network takes two CTAs of 256
# threads up to 10x10 and one of 512 from 10x11 on, the refinement two up to 152 rows.
@pytest.mark.parametrize("Lx,Ly,up,dn", [(4, 4, 5, 5), (8, 8, 28, 26), (10, 10, 44, 44),
                                         (10, 11, 48, 46), (16, 12, 76, 76), (16, 12, 78, 76)])
@pytest.mark.parametrize("refine_tau", [0.0, 1.0])
def test_stored_features(Lx, Ly, up, dn, refine_tau):
    check_forms(32, Lx, Ly, up, dn, refine_tau, 1)


@pytest.mark.parametrize("channels,Lx,Ly,ne,kw,message", [
    (64, 6, 8, 20, dict(cond_tau=1.0), r"refine: n=40 needs \d+ B"),
    (32, 32, 32, 4, {}, r"fused amplitude: n=8, N=1024 needs \d+ B")])
def test_refusals_say_what_is_needed(channels, Lx, Ly, ne, kw, message):
    p = nh.init_params(Lx, Ly, channels=channels, layers=4, std=0.1, seed=1)
    s = olat.random_configs(np.random.default_rng(1), 2, Lx * Ly, ne, ne)
    with pytest.raises(nh.NativeLibraryError, match=message):
        nh.Variational(nh.PfaffianBackflow(Lx, Ly, ne, ne, params=p, **kw))(s)


@pytest.mark.parametrize("Lx,Ly,up,dn", [(8, 8, 28, 26), (12, 14, 71, 69)])
def test_few_of_many_listed(Lx, Ly, up, dn):
    """16 channels, more images than SMs of which fewer than SMs are listed: the 512-thread form then,
    as for few images; the same bits either way, and both lists' lengths occur."""
    N = Lx * Ly
    p = nh.init_params(Lx, Ly, channels=16, layers=4, std=0.1, seed=N)
    s = olat.random_configs(np.random.default_rng(N + 1), 6, N, up, dn)
    seen = set()
    for tau in (1.0, 5.0, 10.0, 20.0, 40.0, 80.0, 160.0, 320.0):
        state = nh.Variational(nh.PfaffianBackflow(Lx, Ly, up, dn, params=p, cond_tau=tau),
                               symm=False)
        few, many = state(s), state(np.tile(s, (50, 1)))
        assert torch.equal(few.sign.repeat(50), many.sign)
        assert torch.equal(few.logabs.repeat(50), many.logabs)
        assert torch.equal(few.flags.repeat(50), many.flags)
        seen.add(int((few.flags & _lib.FLAG_REFINED != 0).sum()))
    assert seen & {1, 2} and seen & {3, 4, 5, 6}, seen
