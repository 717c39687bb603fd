"""Workloads for timing the library's public entry points, with FP64 reference values.

A variational Monte Carlo program spends its time in five calls: ``state(spins)`` (amplitudes),
``sampler.sweep()`` (Metropolis steps), ``H.Oloc`` (local energies), ``state.jacobian`` (the
derivatives that stochastic reconfiguration consumes) and, for the released networks, the same
amplitudes through the residual network.  ``listed`` holds one or two cases of each over the sizes
such programs use, from a handful of configurations on an 8x8 lattice to the 8192 projected
configurations at 16x16 of ``bench.py``; ``draw`` gives more of the same kinds.  Weights are
random, as in the benchmark (N(0, 0.02) convolutions; LeCun-sized ones for the residual network),
and configurations uniform at fixed particle numbers.

``exact`` restates every path in plain torch FP64 (no code of this package): the networks, the
pairing block, a batched Parlett-Reid Pfaffian with sign, the projection, the hop enumeration and
autograd for the Jacobian.
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as tf

import neuralhubbard_b200 as nh

DEV = "cuda"
HOPS = ((1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (1, -1), (-1, 1), (-1, -1))
T_NN, T_NNN, U_HUB = 1.0, -0.2, 8.0


def _case(name, kind, Lx, Ly, n_up, n_dn, batch, symm, **kw):
    c = dict(kind=kind, Lx=Lx, Ly=Ly, n_up=n_up, n_dn=n_dn, batch=batch, symm=symm,
             net="cnn", ansatz="pfaffian", cnn_mode=0, blocks=0, steps=0, n_dirs=8)
    c.update(kw)
    if name:
        c = dict(name=name, **c)
    return c


def listed():
    return [
        # A few projected amplitudes on the 8x8 lattice of the tests: launches and latency.
        _case("amp_8x8_small", "amplitude", 8, 8, 28, 28, 16, True),
        # A rectangular lattice with odd counts, bare amplitudes (no projection).
        _case("amp_10x14_ragged", "amplitude", 10, 14, 61, 59, 777, False),
        # One sampler's chains at 16x16, projected, default (FP32 CNN) form.
        _case("amp_16_plain", "amplitude", 16, 16, 112, 112, 1024, True),
        # The benchmark's call: 8192 projected configurations, tensor-core CNN.
        _case("amp_16_chosen", "amplitude", 16, 16, 112, 112, 8192, True, cnn_mode=2),
        # Lattices beyond shared memory (the 24x24 and 32x32 states of the benchmark).
        _case("amp_24", "amplitude", 24, 24, 252, 252, 48, True),
        _case("amp_32", "amplitude", 32, 32, 448, 448, 24, True),
        # Local energies: the benchmark's 8x8 configuration (1024 samples, bare) and a batch of
        # 16x16 samples, t' included; the largest share of a measurement run.
        _case("eloc_8x8", "eloc", 8, 8, 28, 28, 1024, False),
        _case("eloc_16", "eloc", 16, 16, 112, 112, 64, False),
        # Mixed hop / site-exchange chains at 16x16 (the reference's sampler), tensor-core CNN.
        _case("sample_16", "sample", 16, 16, 112, 112, 1024, True, cnn_mode=2, steps=4),
        # Training: the per-sample Jacobian of one optimiser step's share of samples.
        _case("jacobian_16", "jacobian", 16, 16, 112, 112, 256, True),
        # The released states' residual network (16 blocks) on the tensor cores.
        _case("resconv_16", "amplitude", 16, 16, 112, 112, 256, True, net="resconv", blocks=16,
              cnn_mode=2),
        # The BCS-backflow ansatz, tensor-core CNN.
        _case("bcs_16", "amplitude", 16, 16, 112, 112, 512, True, ansatz="bcs", cnn_mode=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fill(rng, N, limit):
    """(n_up, n_dn) at 3/8, 7/16 or 1/2 filling, sometimes polarised by an electron, even sum."""
    ne = min(int(N * rng.choice((0.375, 0.4375, 0.4375, 0.5))), limit // 2)
    return (ne + 1, ne - 1) if rng.random() < 0.2 else (ne, ne)


def draw(rng):
    kind = rng.choice(("amp", "amp", "amp", "chosen", "large", "eloc", "sample", "jacobian",
                       "resconv", "bcs"))
    if kind == "chosen":
        up, dn = _fill(rng, 256, 224)
        return _case(None, "amplitude", 16, 16, up, dn, _log_int(rng, 1, 6000),
                     rng.random() < 0.7, cnn_mode=2)
    if kind == "resconv":
        up, dn = _fill(rng, 256, 224)
        return _case(None, "amplitude", 16, 16, up, dn, _log_int(rng, 2, 500), True,
                     net="resconv", blocks=rng.choice((4, 8, 16)), cnn_mode=2)
    if kind == "bcs":
        ne = rng.choice((96, 112, 128))
        return _case(None, "amplitude", 16, 16, ne, ne, _log_int(rng, 8, 1500), True,
                     ansatz="bcs", cnn_mode=rng.choice((0, 2)))
    if kind == "large":
        Lx = rng.randrange(18, 33)
        Ly = rng.randrange(max(18, Lx - 4), min(32, Lx + 4) + 1)
        Ly -= (Lx * Ly) % 2
        up, dn = _fill(rng, Lx * Ly, 1024)
        b = _log_int(rng, 2, max(3, int(60 * (504 / (up + dn)) ** 2)))
        return _case(None, "amplitude", Lx, Ly, up, dn, b, rng.random() < 0.7)
    if kind == "jacobian":
        Lx, Ly = rng.choice(((8, 8), (10, 8), (12, 12), (16, 12), (16, 16)))
        up, dn = _fill(rng, Lx * Ly, 224)
        return _case(None, "jacobian", Lx, Ly, up, dn, _log_int(rng, 8, 300), True)
    Lx, Ly = rng.randrange(4, 17), rng.randrange(4, 17)
    Ly -= (Lx * Ly) % 2
    up, dn = _fill(rng, Lx * Ly, 256)
    n = up + dn
    if kind == "eloc":
        top = min(1000.0, max(2.0, 5e4 / (4.5 * n) * min(5.0, (224 / n) ** 2)))
        return _case(None, "eloc", Lx, Ly, up, dn, _log_int(rng, 1, top), rng.random() < 0.1,
                     n_dirs=rng.choice((4, 8)))
    if kind == "sample":
        return _case(None, "sample", Lx, Ly, up, dn, _log_int(rng, 32, 1024), rng.random() < 0.5,
                     steps=rng.randrange(1, 9), n_dirs=rng.choice((4, 8)))
    return _case(None, "amplitude", Lx, Ly, up, dn, _log_int(rng, 1, 4000), rng.random() < 0.5)


# ------------------------------------------------------------------ inputs


def _params(case, seed):
    """Model parameters (host FP32 arrays) from the seed."""
    Lx, Ly = case["Lx"], case["Ly"]
    N = Lx * Ly
    if case["net"] == "resconv":
        rng = np.random.default_rng([seed, 2])
        C, d, nb = 64, 32, 2 * case["blocks"]
        w = (rng.normal(size=(nb, C, C, 3, 3)) * 0.04).astype(np.float32)
        b = (rng.normal(size=(nb, C)) * 0.1).astype(np.float32)
        return dict(net="resconv", embed=rng.normal(size=(C, 4)).astype(np.float32),
                    conv_w=list(w), conv_b=list(b),
                    W=(rng.normal(size=(3, N, d)) / np.sqrt(d)).astype(np.float32),
                    theta=float(np.float32(0.55)))
    p = nh.init_params(Lx, Ly, channels=32, layers=4, std=0.02, seed=seed)
    if case["ansatz"] == "bcs":
        p["W"] = p["W"][0]
        p["delta_d"] = 0.1
    return p


def _spins(case, seed):
    """(batch, 2N) int8 configurations, uniform at fixed particle numbers, on the GPU."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1000003 * (int(seed) % 1000003) + 17)
    N, B = case["Lx"] * case["Ly"], case["batch"]
    out = torch.full((B, 2 * N), -1, dtype=torch.int8, device=DEV)
    for half, ne in ((0, case["n_up"]), (1, case["n_dn"])):
        order = torch.rand((B, N), generator=gen, device=DEV).argsort(1)[:, :ne]
        out.scatter_(1, half * N + order, 1)
    return out


def prepare(case, seed):
    cls = nh.BCSBackflow if case["ansatz"] == "bcs" else nh.PfaffianBackflow
    model = cls(case["Lx"], case["Ly"], case["n_up"], case["n_dn"], params=_params(case, seed),
                cnn_mode=case["cnn_mode"], device=DEV)
    state = nh.Variational(model, symm=case["symm"])
    spins = _spins(case, seed)
    st = dict(case=case, state=state, spins=spins)
    nn = [1, 2] if case["n_dirs"] == 8 else 1
    if case["kind"] == "eloc":
        t = [T_NN, T_NNN] if case["n_dirs"] == 8 else T_NN
        st["H"] = nh.Hubbard(U=U_HUB, t=t, n_neighbor=nn)
        st["samples"] = nh.Samples(spins, state(spins))
    elif case["kind"] == "sample":
        half = case["batch"] // 2
        smp = nh.MixSampler([nh.ParticleHop(state, case["batch"] - half, n_neighbor=nn),
                             nh.SiteExchange(state, half, n_neighbor=nn)],
                            initial_spins=spins.clone(), seed=int(seed))
        smp.psi  # the chains' amplitudes, as after an earlier sweep
        st["sampler"] = smp
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "amplitude":
        psi = state["state"](state["spins"])
        return {"sign": psi.sign, "logabs": psi.logabs, "flags": psi.flags}
    if case["kind"] == "eloc":
        return {"eloc": state["H"].Oloc(state["state"], state["samples"])}
    if case["kind"] == "jacobian":
        psi, jac = state["state"].jacobian(state["spins"])
        return {"sign": psi.sign, "logabs": psi.logabs, "jac": jac}
    smp = state["sampler"]
    s = smp.sweep(case["steps"])
    return {"spins": s.spins, "sign": s.psi.sign, "logabs": s.psi.logabs,
            "accepted": smp.accepted}


def work(case):
    """Floating-point operations of one pass (convolutions, pairing block, n^3 / 3 per Pfaffian or
    2 m^3 / 3 per determinant, all once per image) and the bytes of its inputs and outputs."""
    N, n, B = case["Lx"] * case["Ly"], case["n_up"] + case["n_dn"], case["batch"]
    G = 8 if case["symm"] else 1
    d = 32 if case["net"] == "resconv" else 16
    if case["net"] == "resconv":
        conv, weights = 2 * N * 2 * case["blocks"] * 9 * 64 * 64, 2 * case["blocks"] * 9 * 64 * 64
    else:
        conv, weights = 2 * N * 9 * (2 * 32 + 3 * 32 * 32), 9 * (2 * 32 + 3 * 32 * 32)
    if case["ansatz"] == "bcs":
        m = case["n_up"]
        pf, gather, table = 2 * m ** 3 / 3, 3 * d * m * m, N * d
    else:
        pf, gather, table = n ** 3 / 3, 3 * d * n * n / 2, 4 * N * d
    amp = conv + gather + pf
    nbytes = 4 * (weights + table) + B * 2 * N
    if case["kind"] == "amplitude":
        return dict(bytes=nbytes + 16 * B, flops=B * G * amp)
    if case["kind"] == "eloc":
        conn = B * case["n_dirs"] * (case["n_up"] * (N - case["n_up"])
                                     + case["n_dn"] * (N - case["n_dn"])) / (N - 1)
        return dict(bytes=nbytes + 20 * B, flops=conn * G * amp)
    if case["kind"] == "jacobian":
        # forward, inverse (2 n^3), the gather's two cotangents, the convolutions' (twice)
        P = weights + 4 * 32 + 3 * N * d + 1
        return dict(bytes=nbytes + 12 * B + 4 * B * P,
                    flops=B * G * (amp + 2 * n ** 3 + 5 * d * n * n + 2 * conv))
    moved = 1.0 - 0.5 * (n / (2 * N)) - 0.25  # moves that are not null, roughly
    return dict(bytes=nbytes + B * (2 * N + 28), flops=case["steps"] * B * moved * G * amp)


# ------------------------------------------------------------------ FP64 reference values


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _conv(x, w, b):
    """Periodic 3x3 cross-correlation as one matrix product."""
    B, C, Lx, Ly = x.shape
    cols = tf.unfold(tf.pad(x, (1, 1, 1, 1), mode="circular"), 3)  # (B, C 9, N)
    return (torch.matmul(w.reshape(w.shape[0], -1), cols) + b[:, None]).reshape(B, -1, Lx, Ly)


def _features(s, p, Lx, Ly):
    """(B, 2N, d) features of +-1 configurations."""
    B, N = s.shape[0], Lx * Ly
    if p.get("net") == "resconv":
        occ = (s[:, :N] > 0).long() + 2 * (s[:, N:] > 0).long()
        x = p["embed"].t()[occ].transpose(1, 2).reshape(B, -1, Lx, Ly)
        nb = len(p["conv_w"]) // 2
        for k in range(nb):
            h = _gelu(x / torch.sqrt((x * x).mean((1, 2, 3), keepdim=True) + 1e-6))
            h = _gelu(_conv(h, p["conv_w"][2 * k], p["conv_b"][2 * k]))
            x = x + _conv(h, p["conv_w"][2 * k + 1], p["conv_b"][2 * k + 1])
        x = x / math.sqrt(nb + 1.0)
    else:
        x = s.reshape(B, 2, Lx, Ly).double()
        for k, (w, b) in enumerate(zip(p["conv_w"], p["conv_b"])):
            x = _conv(x, w, b)
            if k + 1 < len(p["conv_w"]):
                x = _gelu(x)
    d = x.shape[1] // 2
    return x.reshape(B, 2, d, N).transpose(2, 3).reshape(B, 2 * N, d)


def _tables(Lx, Ly):
    site = torch.arange(Lx * Ly, device=DEV)
    x, y = site // Ly, site % Ly
    disp = ((x[:, None] - x[None]) % Lx) * Ly + (y[:, None] - y[None]) % Ly
    neg = ((-x) % Lx) * Ly + (-y) % Ly
    mx, my = torch.minimum(x, Lx - x), torch.minimum(y, Ly - y)
    return disp, neg, torch.sqrt((mx * mx + my * my).double()), mx, my


def _table(W, theta, Lx, Ly):
    """The pairing table: (4, N, d) blocks [uu, ud, du, dd], or (N, d) for the BCS state."""
    _, neg, dist, _, _ = _tables(Lx, Ly)
    e = torch.exp(-tf.softplus(theta) * dist)
    pref = (e / (Lx * Ly * e.sum()))[:, None]
    if W.dim() == 2:
        return W * pref
    return torch.stack([(W[1] - W[1][neg]) / 2, W[0], -W[0][neg], (W[2] - W[2][neg]) / 2]) * pref


def _block(s, p, Lx, Ly):
    """The occupied pairing block F (B, n, n); up x down for the BCS state."""
    N = Lx * Ly
    disp, _, _, mx, my = _tables(Lx, Ly)
    y, Wt = _features(s, p, Lx, Ly), _table(p["W"], p["theta"], Lx, Ly)
    B = s.shape[0]
    idx = (s > 0).nonzero()[:, 1].reshape(B, -1)
    Y = torch.gather(y, 1, idx[:, :, None].expand(-1, -1, y.shape[2]))
    sp, site = idx // N, idx % N
    if Wt.dim() == 2:
        nu = int((s[0, :N] > 0).sum())
        r = disp[site[:, :nu, None], site[:, None, nu:]]
        fd = ((mx == 0) & (my == 1)).double() - ((mx == 1) & (my == 0)).double()
        return torch.einsum("bpa,bpqa,bqa->bpq", Y[:, :nu], Wt[r], Y[:, nu:]) \
            + p["delta_d"] * fd[r]
    r = disp[site[:, :, None], site[:, None, :]]
    F = (Y[:, :, None] * Wt[2 * sp[:, :, None] + sp[:, None, :], r] * Y[:, None]).sum(-1)
    return 0.5 * (F - F.transpose(1, 2))


def _slogpf(A):
    """(sign, log|pf|) of antisymmetric A (B, n, n): Parlett-Reid with partial pivoting."""
    B, n, _ = A.shape
    sign = torch.ones(B, dtype=torch.float64, device=A.device)
    log = torch.zeros(B, dtype=torch.float64, device=A.device)
    rows = torch.arange(B, device=A.device)
    A = A.clone()
    for _ in range(n // 2):
        q = 1 + A[:, 1:, 0].abs().argmax(1)
        r1, rq = A[:, 1].clone(), A[rows, q].clone()
        A[:, 1], A[rows, q] = rq, r1
        c1, cq = A[:, :, 1].clone(), A[rows, :, q].clone()
        A[:, :, 1], A[rows, :, q] = cq, c1
        piv = A[:, 0, 1]
        sign = sign * torch.sign(piv) * torch.where(q == 1, 1.0, -1.0)
        log = log + torch.log(piv.abs())
        tau, col = A[:, 0, 2:] / piv[:, None], A[:, 2:, 1]
        A = A[:, 2:, 2:] + tau[:, :, None] * col[:, None, :] - col[:, :, None] * tau[:, None, :]
    return sign, log


def _bare(s, p, Lx, Ly):
    """(sign, log|psi|) of configurations, without projection."""
    n = (s > 0).sum(1)
    F = _block(s, p, Lx, Ly)
    if p["W"].dim() == 2:
        sg, la = torch.linalg.slogdet(F)
        nu = F.shape[1]
        sg = sg * (-1.0) ** (nu * (nu - 1) // 2)
    else:
        sg, la = _slogpf(F)
    return sg * (1 - 2 * ((n * (n - 1) // 2) % 2)).double(), la


def _images(s, Lx, Ly):
    """(B, 8, 2N) symmetry images and their (B, 8) fermionic reordering signs."""
    N = Lx * Ly
    site = torch.arange(N, device=DEV)
    x, y = site // Ly, site % Ly
    idx = (s > 0).nonzero()[:, 1].reshape(s.shape[0], -1)
    later = torch.triu(torch.ones(idx.shape[1], idx.shape[1], dtype=torch.bool, device=DEV), 1)
    imgs, eta = [], []
    for g in range(8):
        t = ((-x) % Lx if g & 1 else x) * Ly + ((-y) % Ly if g & 2 else y)
        m = torch.cat([t + N, t]) if g & 4 else torch.cat([t, t + N])
        imgs.append(s[:, m])  # the maps are involutions
        to = m[idx]
        eta.append(1.0 - 2.0 * (((to[:, :, None] > to[:, None]) & later).sum((1, 2)) % 2).double())
    return torch.stack(imgs, 1), torch.stack(eta, 1)


def _amplitudes(s, p, Lx, Ly, symm):
    """(sign, log|psi|) of s, chunked."""
    n = int((s[0] > 0).sum())
    per = max(1, int(4e8 / (n * n * p["W"].shape[-1])) // (8 if symm else 1))
    out = []
    for c in s.split(per):
        if not symm:
            out.append(_bare(c, p, Lx, Ly))
            continue
        im, eta = _images(c, Lx, Ly)
        sg, la = _bare(im.reshape(-1, im.shape[2]), p, Lx, Ly)
        sg, la = sg.reshape(-1, 8) * eta, la.reshape(-1, 8)
        m = la.max(1, keepdim=True).values
        tot = (sg * torch.exp(la - m)).sum(1)
        out.append((torch.sign(tot), torch.log(tot.abs()) + m[:, 0] - math.log(8.0)))
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


def _params64(case, seed):
    p = _params(case, seed)
    q = {k: torch.from_numpy(np.asarray(p[k], np.float64)).to(DEV) for k in ("W", "theta")}
    for k in ("conv_w", "conv_b"):
        q[k] = [torch.from_numpy(np.asarray(a, np.float64)).to(DEV) for a in p[k]]
    if "embed" in p:
        q["net"], q["embed"] = "resconv", torch.from_numpy(p["embed"]).double().to(DEV)
    if "delta_d" in p:
        q["delta_d"] = float(p["delta_d"])
    return q


def _hop_list(s, Lx, Ly, n_dirs):
    """Connected configurations: owners, configurations (C, 2N) and matrix elements."""
    B, N = s.shape[0], Lx * Ly
    site = torch.arange(N, device=DEV)
    x, y = site // Ly, site % Ly
    occ = s > 0
    before = torch.cumsum(occ.long(), 1)  # occupied modes up to and including m
    own, conf, h = [], [], []
    for k in range(n_dirs):
        dx, dy = HOPS[k]
        t = ((x + dx) % Lx) * Ly + (y + dy) % Ly
        t = torch.cat([t, t + N])
        b, m = (occ & ~occ[:, t]).nonzero(as_tuple=True)
        lo, hi = torch.minimum(m, t[m]), torch.maximum(m, t[m])
        # occupied modes strictly between: the target is empty, the source occupied
        between = before[b, hi] - occ[b, hi].long() - before[b, lo]
        c = s[b].clone()
        i = torch.arange(b.numel(), device=DEV)
        c[i, m], c[i, t[m]] = -1, 1
        own.append(b)
        conf.append(c)
        h.append(-(T_NN if k < 4 else T_NNN) * (1.0 - 2.0 * (between % 2).double()))
    return torch.cat(own), torch.cat(conf), torch.cat(h)


def _jacobian(s, p, Lx, Ly):
    """(sign, logabs, J) of the projected state; J rows by autograd, one sample at a time."""
    leaves = []
    for w, b in zip(p["conv_w"], p["conv_b"]):
        leaves += [w, b]
    leaves += [p["W"], p["theta"]]
    for t in leaves:
        t.requires_grad_(True)
    sign, logabs = [], []
    J = torch.empty((s.shape[0], sum(t.numel() for t in leaves)), dtype=torch.float64, device=DEV)
    for k in range(s.shape[0]):
        im, eta = _images(s[k:k + 1], Lx, Ly)
        F = _block(im[0], p, Lx, Ly)
        with torch.no_grad():
            sg, la0 = _slogpf(F)
            n = F.shape[1]
            sg = sg * eta[0] * (-1.0) ** (n * (n - 1) // 2)
        la = 0.5 * torch.linalg.slogdet(F)[1]
        m = la0.max()
        tot = (sg * torch.exp(la - m)).sum()
        val = torch.log(tot.abs()) + m - math.log(8.0)
        g = torch.autograd.grad(val, leaves)
        J[k] = torch.cat([t.reshape(-1) for t in g])
        sign.append(torch.sign(tot.detach()))
        logabs.append(val.detach())
    return torch.stack(sign), torch.stack(logabs), J


def exact(case, seed):
    Lx, Ly, kind = case["Lx"], case["Ly"], case["kind"]
    if kind == "sample":
        return None  # the chains' decisions, not a computed number
    if kind == "jacobian" and not case["symm"]:
        return None
    p, s = _params64(case, seed), _spins(case, seed)
    if kind == "jacobian":
        sg, la, J = _jacobian(s, p, Lx, Ly)
        return {"sign": sg, "logabs": la, "jac": J}
    sg, la = _amplitudes(s, p, Lx, Ly, case["symm"])
    if kind == "amplitude":
        return {"sign": sg, "logabs": la, "flags": None}
    own, conf, h = _hop_list(s, Lx, Ly, case["n_dirs"])
    N = Lx * Ly
    e = U_HUB * ((s[:, :N] > 0) & (s[:, N:] > 0)).sum(1).double()
    sc, lc = _amplitudes(conf, p, Lx, Ly, case["symm"])
    e.index_add_(0, own, h * sc * sg[own] * torch.exp(lc - la[own]))
    return {"eloc": e}
