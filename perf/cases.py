"""Performance cases: the work that users of the subspace operators have the library do.

A reconstruction precomputes the Toeplitz kernel of its trajectory once (``kernel``),
backprojects its k-space data once (``backprojection``), then applies the normal operator
tens of times, alone (``apply``, a solver of the user's own) or inside ``cg`` (``cg``).
``forward`` synthesises data, ``grog`` shifts radial data onto the Cartesian grid.  All run
in float32: the reduced-precision operators are slower than the float32 one here and give
worse images, so programs run float32.

Every input is made with torch and numpy alone from the seed.  Values follow the path:
golden-angle radial trajectories, orthonormal bases of relaxation curves, smooth coil maps
of unit root-sum-of-squares, k-space data of objects made of point sources with 1% noise,
kernels with the density of radial sampling on its disc (ball) of support.
"""
import math

import numpy as np
import torch

from __graft_entry__ import package

C64, C128, F64 = torch.complex64, torch.complex128, torch.float64


def _case(name, kind, n, K, coils, nt=0, spokes=1, basis="real", iters=0):
    n = tuple(n)
    c = {"kind": kind, "n1": n[0], "n2": n[1], "n3": n[2] if len(n) == 3 else 0, "K": K, "coils": coils, "basis": basis,
         "nt": nt, "spokes": spokes, "iters": iters}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one operator product of a small 2D scan: all launches and host latency
        _case("apply_2d_64_k4_c4", "apply", (64, 64), 4, 4),
        # the usual 2D fingerprinting scan
        _case("apply_2d_256_k5_c20", "apply", (256, 256), 5, 20),
        # high resolution, all channels of a head array
        _case("apply_2d_384_k6_c32", "apply", (384, 384), 6, 32),
        # a rectangular field of view with a complex basis (phase-cycled sequences)
        _case("apply_2d_180x150_k3_c12_cplx", "apply", (180, 150), 3, 12, basis="complex"),
        # isotropic 3D volume: the largest product
        _case("apply_3d_128_k5_c16", "apply", (128, 128, 128), 5, 16),
        # Cartesian sampling (or GROG-gridded data): no oversampling, full complex kernel
        _case("apply_cart_256_k6_c32", "apply_cart", (256, 256), 6, 32, basis="complex"),
        # operator construction: kernel and mask of the usual 2D scan's trajectory
        _case("kernel_2d_256_k5", "kernel", (256, 256), 5, 1, nt=1000),
        # right-hand side of the usual 2D scan
        _case("backprojection_2d_256_k5_c20", "backprojection", (256, 256), 5, 20, nt=1000),
        # right-hand side of a 3D koosh-ball scan
        _case("backprojection_3d_64_k4_c8", "backprojection", (64, 64, 64), 4, 8, nt=400, spokes=6),
        # data synthesis on the usual 2D scan
        _case("forward_2d_256_k5_c20", "forward", (256, 256), 5, 20, nt=1000),
        # a whole iterative solve, the reference's 20 iterations
        _case("cg20_2d_192_k4_c12", "cg", (192, 192), 4, 12, iters=20),
        # GROG self-calibration and gridding of a 32-channel radial scan
        _case("grog_2d_256_c32", "grog", (256, 256), 1, 32, nt=500, spokes=2),
    ]


def _smooth(lo, hi):
    """Lengths with prime factors 2, 3, 5 only: what the transforms take."""
    out = []
    for v in range(lo, hi + 1):
        r = v
        for p in (2, 3, 5):
            while r % p == 0:
                r //= p
        if r == 1:
            out.append(v)
    return out


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    v = _log(rng, lo, hi)
    return min(_smooth(lo, hi), key=lambda s: (abs(s - v), s))


def draw(rng):
    kind = rng.choice(("apply", "apply", "apply", "apply_cart", "kernel", "backprojection", "backprojection", "forward", "cg", "grog"))
    basis = "complex" if rng.random() < 0.25 else "real"
    K = rng.randint(2, 6)
    if kind in ("apply", "kernel", "backprojection") and rng.random() < 0.3:  # 3D
        if kind == "apply":
            a, b = _length(rng, 32, 96), _length(rng, 32, 96)
            return _case(None, kind, (a, b, _length(rng, 32, 96)), K, rng.randint(1, 12), basis=basis)
        a = _length(rng, 32, 64)
        return _case(None, kind, (a, a, _length(rng, 32, 64)), min(K, 4), 1 if kind == "kernel" else rng.randint(2, 8),
                     nt=_log(rng, 100, 400), spokes=rng.randint(2, 6), basis=basis)
    a = _length(rng, 32, 384)
    b = a if rng.random() < 0.5 else _length(rng, max(32, a // 2), min(384, 2 * a))
    if kind in ("apply", "apply_cart"):
        return _case(None, kind, (a, b), K, _log(rng, 1, 32), basis="complex" if kind == "apply_cart" else basis)
    a, b = min(a, 256), min(b, 256)
    if kind == "cg":
        return _case(None, kind, (a, b), K, _log(rng, 2, 20), basis=basis, iters=rng.randint(5, 20))
    if kind == "grog":
        nc = rng.randint(6, 32)
        return _case(None, kind, (max(a, 64), max(a, 64)), 1, nc, nt=max(_log(rng, 100, 500), nc * nc // 2), spokes=rng.randint(1, 2))
    return _case(None, kind, (a, b), K, 1 if kind == "kernel" else _log(rng, 2, 20), nt=_log(rng, 200, 1000), basis=basis)


# ---------------------------------------------------------------- inputs ---


def _shape(case):
    return tuple(v for v in (case["n1"], case["n2"], case["n3"]) if v)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _basis(case, seed):
    """(nt, K) orthonormal basis of relaxation curves."""
    rng = np.random.default_rng(seed)
    nt, K = case["nt"], case["K"]
    t = 5.0 * np.arange(1, nt + 1)[:, None]
    t1 = np.exp(rng.uniform(np.log(100.0), np.log(3000.0), 4 * K))
    t2 = np.exp(rng.uniform(np.log(10.0), np.log(300.0), 4 * K))
    d = (1 - 2 * np.exp(-t / t1)) * np.exp(-t / t2) + 0.05 * np.cos(t * rng.uniform(0.0005, 0.02, 4 * K))
    if case["basis"] == "complex":
        d = d * np.exp(2j * np.pi * rng.uniform(0, 1, 4 * K) * t / t[-1])
    u = np.linalg.svd(d, full_matrices=False)[0][:, :K]
    return torch.from_numpy(np.ascontiguousarray(u.astype(np.complex64 if case["basis"] == "complex" else np.float32))).cuda()


def _trajectory(case, seed):
    """(d, samples, nt) float32: golden-angle spokes (2D) or golden-means koosh ball (3D), 2 n1 samples each."""
    n, nt, sp = _shape(case), case["nt"], case["spokes"]
    g = torch.Generator().manual_seed(int(seed))
    start = torch.rand(2, generator=g, dtype=F64) * (0.0 if case["kind"] == "kernel" else 1.0)
    nr = 2 * n[0]
    kr = ((torch.arange(nr, dtype=F64) - (nr - 1) / 2) / nr).cuda()
    i = torch.arange(sp * nt, dtype=F64).cuda()
    if len(n) == 2:
        phi = i * (math.pi / ((math.sqrt(5.0) + 1) / 2)) + 2 * math.pi * float(start[0])
        dirs = torch.stack([-torch.cos(phi), torch.sin(phi)])
    else:
        z = 2 * torch.remainder(i * 0.46557123187676 + float(start[0]), 1.0) - 1
        phi = 2 * math.pi * torch.remainder(i * 0.68232780382802 + float(start[1]), 1.0)
        s = torch.sqrt(1 - z * z)
        dirs = torch.stack([s * torch.cos(phi), s * torch.sin(phi), z])
    dirs = dirs.reshape(len(n), nt, sp, 1)
    if case["kind"] == "kernel":  # the frames in another order: the mask, and with it the output's size, stays
        dirs = dirs[:, torch.randperm(nt, generator=g).cuda()]
    k = dirs * kr
    return k.clamp(-0.5, 0.5).float().reshape(len(n), nt, sp * nr).transpose(1, 2)


def _coords(n, d):
    """Image coordinates in [-1, 1) along axis d."""
    return (torch.arange(n[d], device="cuda", dtype=torch.float32) - n[d] // 2) * (2.0 / n[d])


def _cmaps(case, seed):
    """(img..., coils) complex64: Gaussians on a ring with linear phases, unit root-sum-of-squares."""
    n, nc = _shape(case), case["coils"]
    g = torch.Generator().manual_seed(int(seed) + 17)
    slope = torch.rand((nc, 3), generator=g) * 2 - 1
    out = torch.empty((nc,) + n, dtype=C64, device="cuda")
    for c in range(nc):
        a = 2 * math.pi * c / nc
        ctr = (1.2 * math.cos(a), 1.2 * math.sin(a), -0.8 + 1.6 * (c + 0.5) / nc)
        v = torch.ones((), device="cuda", dtype=C64)
        for d in range(len(n)):
            x = _coords(n, d)
            e = torch.polar(torch.exp(-((x - ctr[d]) ** 2) / 1.62), math.pi * float(slope[c, d]) * x)
            v = v[..., None] * e
        out[c] = v
    out /= out.abs().square().sum(0, keepdim=True).sqrt()
    return torch.movedim(out, 0, -1)


def _image(case, seed):
    """(img..., K) complex64 piecewise-constant coefficient images of an ellipse phantom."""
    n, K = _shape(case), case["K"]
    rng = np.random.default_rng(seed + 3)
    out = torch.zeros(n + (K,), dtype=C64, device="cuda")
    for _ in range(8):
        r2 = torch.zeros((), device="cuda")
        for d in range(len(n)):
            q = ((_coords(n, d) - float(rng.uniform(-0.5, 0.5))) / float(rng.uniform(0.1, 0.45))) ** 2
            r2 = r2[..., None] + q
        coef = rng.standard_normal(K) * np.exp(-0.5 * np.arange(K)) + 0.2j * rng.standard_normal(K)
        out += (r2 <= 1.0).to(C64)[..., None] * torch.from_numpy(coef.astype(np.complex64)).cuda()
    return out + 0.01 * torch.randn(out.shape, dtype=C64, device="cuda", generator=_gen(seed + 4))


def _kdata(case, trj, seed):
    """(samples, nt, coils) complex64: 96 point sources seen by the coils, relaxing over the frames, 1% noise."""
    n, nc, nt = _shape(case), case["coils"], case["nt"]
    rng = np.random.default_rng(seed + 5)
    ns = trj.shape[1]
    pos = rng.uniform(-0.6, 0.6, (96, 3))
    r = torch.from_numpy((pos[:, : len(n)] * np.array([0.5 * v for v in n])).astype(np.float32)).cuda()
    sens = np.empty((96, nc), dtype=np.complex64)
    slope = rng.uniform(-1, 1, (nc, 3))
    for c in range(nc):
        a = 2 * math.pi * c / nc
        ctr = np.array((1.2 * math.cos(a), 1.2 * math.sin(a), -0.8 + 1.6 * (c + 0.5) / nc))[: len(n)]
        q = pos[:, : len(n)]
        sens[:, c] = np.exp(-((q - ctr) ** 2).sum(1) / 1.62 + 1j * np.pi * (q @ slope[c, : len(n)]))
    rho = rng.uniform(0.3, 1.0, 96) * np.exp(1j * rng.uniform(-0.5, 0.5, 96))
    t = np.arange(1, nt + 1)[:, None] * 5.0
    tc = np.exp(rng.uniform(np.log(300.0), np.log(3000.0), 96))
    curve = torch.from_numpy(((1 - 2 * np.exp(-t / (0.3 * tc))) * np.exp(-t / (3 * tc)) * rho).astype(np.complex64)).cuda()
    sens = torch.from_numpy(sens).cuda()
    out = torch.empty((nc, nt, ns), dtype=C64, device="cuda")
    step = max(1, (1 << 25) // (96 * ns))
    for t0 in range(0, nt, step):
        k = trj[:, :, t0:t0 + step].permute(2, 1, 0)
        ph = torch.polar(torch.ones((), device="cuda"), -2 * math.pi * (k.unsqueeze(-2) * r).sum(-1))  # (frames, ns, 96)
        ph = ph * curve[t0:t0 + step, None, :]
        out[:, t0:t0 + step] = torch.movedim(ph @ sens, -1, 0)
    out += (0.01 * float(out.abs().square().mean().sqrt())) * torch.randn(out.shape, dtype=C64, device="cuda", generator=_gen(seed + 6))
    return out.permute(2, 1, 0)


def _pairs(K):
    return [(k1, k2) for k2 in range(K) for k1 in range(k2 + 1)]


def _mixing(case, seed):
    """Eight K x K positive matrices and their angular phases: how frames mix coefficients around k-space."""
    K = case["K"]
    rng = np.random.default_rng(seed + 7)
    q = rng.standard_normal((8, K, K)) + (1j * rng.standard_normal((8, K, K)) if case["basis"] == "complex" else 0)
    b = np.einsum("mik,mjk->mij", q, q.conj()) / K + 0.5 * np.eye(K)
    return b, rng.uniform(0, 2 * math.pi, (8, 3))


def _toeplitz(case, seed):
    """Packed (pairs, cells) kernel on the disc (ball) of the twofold grid, and its 1-based cells."""
    n = _shape(case)
    G = [2 * v for v in n]
    f = [torch.fft.fftfreq(g, 1.0 / g).cuda().float() for g in reversed(G)]  # last axis first: flat = column-major
    grid = torch.meshgrid(*f, indexing="ij")
    rel = sum((x / (g / 2)) ** 2 for x, g in zip(grid, reversed(G))).reshape(-1)
    cells = torch.nonzero(rel <= (math.inf if case["kind"] == "cg" else 1.0))[:, 0]
    rad = rel[cells].sqrt() * (min(G) / 2)
    flat = 16.0 if case["kind"] == "cg" else 1.0  # a solve is density-compensated
    dens = (1000.0 / (rad + flat) ** (len(n) - 1) + 5.0) * (rel[cells] <= 1.0)
    dens = dens * (0.8 + 0.4 * torch.rand(dens.shape, device="cuda", generator=_gen(seed + 8)))
    b, ph = _mixing(case, seed)
    x = [grid[i].reshape(-1)[cells] / (G[len(n) - 1 - i] / 2) for i in range(len(n))]
    mix = [dens * (1.0 + torch.cos((m % 3 + 1) * 3.0 * x[m % len(n)] + float(ph[m, 0]))) for m in range(8)]
    cplx = case["basis"] == "complex"
    out = torch.zeros((cells.numel(), case["K"] * (case["K"] + 1) // 2), dtype=C64 if cplx else torch.float32, device="cuda")
    for p, (k1, k2) in enumerate(_pairs(case["K"])):
        for m in range(8):
            out[:, p] += mix[m] * (complex(b[m, k1, k2]) if cplx else float(b[m, k1, k2].real))
        if case["kind"] == "cg" and k1 == k2:
            out[:, p] += 30.0  # Tikhonov regularisation of a solve: a multiple of the identity on the whole grid
    return out.T, cells + 1


def _cartesian(case, seed):
    """(K, K, img...) complex64 kernel of a variable-density Cartesian mask (two thirds of the cells sampled)."""
    n, K = _shape(case), case["K"]
    b, _ = _mixing(case, seed)
    w = torch.rand((8,) + n, device="cuda", generator=_gen(seed + 9))
    keep = torch.rand(n, device="cuda", generator=_gen(seed + 10)) < 0.67
    out = torch.empty((K, K) + n, dtype=C64, device="cuda")
    for k1 in range(K):
        for k2 in range(K):
            v = torch.zeros(n, dtype=C64, device="cuda")
            for m in range(8):
                v += w[m] * complex(b[m, k1, k2])
            out[k1, k2] = v * keep
    return out


def _inputs(case, seed):
    """All inputs of a case as plain tensors."""
    kind = case["kind"]
    if kind == "apply_cart":
        return {"lam": _cartesian(case, seed), "cmaps": _cmaps(case, seed), "x": _image(case, seed)}
    if kind in ("apply", "cg"):
        lam, cells = _toeplitz(case, seed)
        d = {"lam": lam, "cells": cells, "cmaps": _cmaps(case, seed), "x": _image(case, seed)}
        if kind == "cg":  # the right-hand side of an object
            d["x"] = _apply_nfft(case, d["x"], lam, cells, d["cmaps"], C64) / (1000.0 * 4)
        return d
    trj = _trajectory(case, seed)
    if kind == "kernel":
        return {"trj": trj, "U": _basis(case, seed)}
    if kind == "backprojection":
        return {"trj": trj, "U": _basis(case, seed), "cmaps": _cmaps(case, seed), "data": _kdata(case, trj, seed)}
    if kind == "forward":
        return {"trj": trj, "U": _basis(case, seed), "cmaps": _cmaps(case, seed), "x": _image(case, seed)}
    return {"trj": trj, "data": _kdata(case, trj, seed)}


def prepare(case, seed):
    mr = package()
    s = {k: mr.to_jl(v, v.dtype) for k, v in _inputs(case, seed).items()}
    s["kind"], s["img"], s["iters"], s["nr"] = case["kind"], _shape(case), case["iters"], 2 * case["n1"]
    if s["kind"] in ("apply", "cg"):
        s["A"] = mr.NFFTNormalOp(s["img"], s.pop("lam"), s.pop("cells"), cmaps=s.pop("cmaps"))
    elif s["kind"] == "apply_cart":
        s["A"] = mr.FFTNormalOp(s.pop("lam"), cmaps=s.pop("cmaps"))
    if s["kind"] in ("apply", "apply_cart"):
        s["y"] = mr.jl_zeros(s["x"].shape, C64)
    return s


def run(s):
    mr = package()
    kind = s["kind"]
    if kind in ("apply", "apply_cart"):
        return s["A"].mul(s["y"], s["x"])
    if kind == "cg":
        return mr.cg(s["A"], s["x"], maxiter=s["iters"], reltol=0.0)
    if kind == "kernel":
        A = mr.NFFTNormalOp(s["img"], s["trj"], s["U"])
        return [A.Λ, A.kmask_indcs]
    if kind == "backprojection":
        return mr.calculate_backprojection(s["data"], s["trj"], s["cmaps"], U=s["U"])
    if kind == "forward":
        return mr.forward_model(s["x"], s["trj"], s["U"], cmaps=s["cmaps"])
    data = s["data"].clone()  # gridded in place
    lnG = mr.grog_calib(data, s["trj"], s["nr"])
    trj_cart = mr.grog_gridding(data, s["trj"], lnG, s["nr"], s["img"])
    return [torch.stack(lnG), data, trj_cart]


def work(case):
    n, K, nc = _shape(case), case["K"], case["coils"]
    d, img = len(n), math.prod(n)
    cx = case["basis"] == "complex"
    P = K * (K + 1) // 2
    if case["kind"] in ("apply", "apply_cart", "cg"):
        if case["kind"] == "apply_cart":
            G, cells, lam = img, 0.67 * img, 8 * K * K
        else:
            G = img * 2 ** d
            cells, lam = G * (math.pi / 4 if d == 2 else math.pi / 6), P * (8 if cx else 4)
        flops = nc * (K * 10 * G * math.log2(G) + cells * K * K * (8 if cx else 4))
        b = {"bytes": img * K * 16 + img * nc * 8 + cells * lam, "flops": flops}
        return dict(b, flops=flops * max(1, case["iters"]))
    ns = 2 * n[0] * case["spokes"] * case["nt"]
    if case["kind"] == "grog":
        return {"bytes": ns * (nc * 16 + d * 8), "flops": ns * nc * nc * 8 * (2 + 2 * d)}
    M = img * 2 ** d
    if case["kind"] == "kernel":
        G, parts = M, P * (2 if cx else 1)
        cells = G * (math.pi / 4 if d == 2 else math.pi / 6)
        return {"bytes": ns * d * 4 + cells * P * (8 if cx else 4), "flops": ns * 8 ** d * parts * 2 + P * 5 * G * 2 ** d * math.log2(G * 2 ** d)}
    return {"bytes": ns * (d * 4 + nc * 8) + img * (nc + K) * 8, "flops": ns * 8 ** d * (2 * K * nc) * 2 + nc * K * 5 * M * math.log2(M)}


# ------------------------------------------------- the values in 64 bits ---


def _apply_nfft(case, x, lam, cells, cmaps, dt):
    """sum_c conj(S_c) crop F^-1 Λ F pad (S_c x) on the twofold grid, in dtype dt."""
    n, K = _shape(case), case["K"]
    d = len(n)
    G = tuple(2 * v for v in n)
    out = torch.zeros(n + (K,), dtype=dt, device="cuda")
    low = tuple(slice(0, v) for v in n)
    idx = cells - 1
    for c in range(cmaps.shape[-1]):
        s = cmaps[..., c].to(dt)
        buf = []
        for k in range(K):
            g = torch.zeros(G, dtype=dt, device="cuda")
            g[low] = s * x[..., k].to(dt)
            buf.append(torch.fft.fftn(g).permute(*reversed(range(d))).reshape(-1)[idx])
        acc = [torch.zeros_like(b) for b in buf]
        for p, (k1, k2) in enumerate(_pairs(K)):
            l = lam[p].to(dt)
            acc[k1] += l * buf[k2]
            if k1 != k2:
                acc[k2] += l.conj() * buf[k1]
        for k in range(K):
            g = torch.zeros(math.prod(G), dtype=dt, device="cuda")
            g[idx] = acc[k]
            g = torch.fft.ifftn(g.reshape(G[::-1]).permute(*reversed(range(d))))
            out[..., k] += s.conj() * g[low]
    return out


def _apply_cart(x, lam, cmaps):
    d, K = x.dim() - 1, x.shape[-1]
    axes = tuple(range(d))
    out = torch.zeros(x.shape, dtype=C128, device="cuda")
    lam = lam.to(C128)
    for c in range(cmaps.shape[-1]):
        s = cmaps[..., c].to(C128)[..., None]
        f = torch.fft.fftn(s * x.to(C128), dim=axes)
        y = torch.stack([sum(lam[k1, k2] * f[..., k2] for k2 in range(K)) for k1 in range(K)], dim=-1)
        out += s.conj() * torch.fft.ifftn(y, dim=axes)
    return out


def _phi(z, beta):
    return torch.exp(beta * (torch.sqrt((1 - z * z).clamp(min=0.0)) - 1)) * (z.abs() < 1)


def _taps(k, M, w):
    """Cells (n, w) and weights (n, w) of the spreading kernel along one axis."""
    u = k * M
    l = torch.ceil(u - w / 2)[:, None] + torch.arange(w, device="cuda", dtype=F64)
    return torch.remainder(l, M).long(), _phi((l - u[:, None]) / (w / 2), 2.3 * w)


def _inv_psi(j, M, w):
    x, q = np.polynomial.legendre.leggauss(200)
    ph = np.exp(2.3 * w * (np.sqrt(1 - x * x) - 1)) * q
    v = 1.0 / (0.5 * w * (np.cos(np.pi * np.outer(j.cpu().numpy(), x) * w / M) @ ph))
    return torch.from_numpy(v).cuda()


def _cells(pts, M, w):
    """Flat C-order cells and weights of every tap of every point."""
    idx, wt = _taps(pts[0], M[0], w)
    for i in range(1, len(M)):
        a, b = _taps(pts[i], M[i], w)
        idx = (idx[:, :, None] * M[i] + a[:, None, :]).flatten(1)
        wt = (wt[:, :, None] * b[:, None, :]).flatten(1)
    return idx, wt


def _type1(pts, vals, modes, M, w):
    """sum_n vals[n, ch] exp(+2 pi i j . k_n) for j in modes: (ch, modes...) complex128.  vals: f(first, last) -> (n, ch)."""
    n, d = pts.shape[1], pts.shape[0]
    nch = vals(0, 1).shape[1]
    grid = torch.zeros((math.prod(M), 2 * nch), dtype=F64, device="cuda")
    step = max(256, (1 << 27) // (w ** d * 2 * nch))
    for a in range(0, n, step):
        b = min(n, a + step)
        idx, wt = _cells(pts[:, a:b], M, w)
        v = torch.view_as_real(vals(a, b).to(C128)).flatten(1)
        grid.index_add_(0, idx.reshape(-1), (wt[:, :, None] * v[:, None, :]).flatten(0, 1))
    out = torch.empty((nch,) + tuple(len(j) for j in modes), dtype=C128, device="cuda")
    for ch in range(nch):
        f = torch.fft.ifftn(torch.complex(grid[:, 2 * ch], grid[:, 2 * ch + 1]).reshape(M), norm="forward")
        for i, j in enumerate(modes):
            shape = [1] * d
            shape[i] = len(j)
            f = f.index_select(i, torch.remainder(j, M[i])) * _inv_psi(j, M[i], w).reshape(shape)
        out[ch] = f
    return out


def _type2(pts, f, modes, M, w):
    """sum_j f[ch, j] exp(-2 pi i j . k_n): (n, ch)."""
    d, nch = pts.shape[0], f.shape[0]
    grid = torch.empty((math.prod(M), nch), dtype=C128, device="cuda")
    for ch in range(nch):
        v = f[ch]
        g = torch.zeros(M, dtype=C128, device="cuda")
        for i, j in enumerate(modes):
            shape = [1] * d
            shape[i] = len(j)
            v = v * _inv_psi(j, M[i], w).reshape(shape)
        g[torch.meshgrid(*[torch.remainder(j, m) for j, m in zip(modes, M)], indexing="ij")] = v
        grid[:, ch] = torch.fft.fftn(g).reshape(-1)
    out = torch.empty((pts.shape[1], nch), dtype=C128, device="cuda")
    step = max(256, (1 << 26) // (w ** d * nch))
    for a in range(0, pts.shape[1], step):
        idx, wt = _cells(pts[:, a:a + step], M, w)
        out[a:a + step] = torch.einsum("nt,ntc->nc", wt.to(C128), grid[idx])
    return out


def _points(trj):
    """(d, samples * nt) in column-major order, and each one's frame."""
    d, ns, nt = trj.shape
    return trj.permute(0, 2, 1).reshape(d, -1).double(), torch.arange(nt, device="cuda").repeat_interleave(ns)


def _width(n):
    return 12 if len(n) == 2 else 10


def _exact_kernel(case, s):
    n, K = _shape(case), case["K"]
    d, w = len(n), _width(n)
    G = tuple(2 * v for v in n)
    trj, U = s["trj"], s["U"].to(C128)
    pts, fr = _points(trj)
    hit = torch.zeros(G, dtype=torch.bool, device="cuda")
    p32 = trj.permute(0, 2, 1).reshape(d, -1)
    i0 = [torch.floor(-p32[i] * float(G[i])).long() for i in range(d)]
    hit[tuple(torch.remainder(i0[i], G[i]) for i in range(d))] = True
    for i in range(d):
        acc = torch.zeros_like(hit)
        for o in range(-3, 5):
            acc |= torch.roll(hit, o, i)
        hit = acc
    cells = torch.nonzero(hit.permute(*reversed(range(d))).reshape(-1))[:, 0]
    real = case["basis"] != "complex"
    fft = [torch.cat([torch.arange(0, g // 2), torch.arange(-(g // 2), 0)]).cuda() for g in G]
    modes = [torch.arange(0, G[0] // 2 + 1).cuda() if real else fft[0]] + fft[1:]
    pr = _pairs(K)
    prod = torch.stack([U[:, k1].conj() * U[:, k2] for k1, k2 in pr], dim=1)
    c = _type1(pts, lambda a, b: prod[fr[a:b]], modes, tuple(2 * g for g in G), w)
    out = torch.empty((len(pr), cells.numel()), dtype=F64 if real else C128, device="cuda")
    for p in range(len(pr)):
        if real:
            ax = tuple(range(1, d)) + (0,)
            lam = torch.fft.irfftn(c[p].conj(), s=G[1:] + (G[0],), dim=ax, norm="forward")
        else:
            lam = torch.fft.fftn(c[p])
        out[p] = lam.permute(*reversed(range(d))).reshape(-1)[cells]
    return [out, cells + 1]


def _exact_backprojection(case, s):
    n, K, nc = _shape(case), case["K"], case["coils"]
    w = _width(n)
    pts, fr = _points(s["trj"])
    uc = s["U"].to(C128).conj()
    data = s["data"].permute(2, 1, 0).reshape(nc, -1)
    modes = [torch.arange(v).cuda() - v // 2 for v in n]
    out = torch.zeros(n + (K,), dtype=C128, device="cuda")
    for c in range(nc):
        img = _type1(pts, lambda a, b: data[c, a:b, None].to(C128) * uc[fr[a:b]], modes, tuple(2 * v for v in n), w)
        out += torch.movedim(img, 0, -1) * s["cmaps"][..., c, None].to(C128).conj()
    return out


def _exact_forward(case, s):
    n, nc = _shape(case), case["coils"]
    pts, fr = _points(s["trj"])
    U = s["U"].to(C128)
    modes = [torch.arange(v).cuda() - v // 2 for v in n]
    ns, nt = s["trj"].shape[1:]
    out = torch.empty((ns, nt, nc), dtype=C128, device="cuda")
    for c in range(nc):
        f = torch.movedim(s["x"].to(C128) * s["cmaps"][..., c, None].to(C128), -1, 0)
        z = _type2(pts, f, modes, tuple(2 * v for v in n), _width(n))
        out[..., c] = (z * U[fr]).sum(1).reshape(nt, ns).T
    return out


def _exact_cg(case, s):
    b = s["x"].to(C128)
    x, r, u, prev = torch.zeros_like(b), b.clone(), torch.zeros_like(b), 1.0
    res = float(torch.linalg.vector_norm(r))
    for _ in range(case["iters"]):
        u = r + (res * res / (prev * prev)) * u
        c = _apply_nfft(case, u, s["lam"], s["cells"], s["cmaps"], C128)
        a = res * res / torch.vdot(u.reshape(-1), c.reshape(-1))
        x, r = x + a * u, r - a * c
        prev, res = res, float(torch.linalg.vector_norm(r))
    return x


def _exact_grog(case, s):
    n, nc, nr = _shape(case), case["coils"], 2 * case["n1"]
    trj, data = s["trj"], s["data"].to(C128)
    ns, nt = trj.shape[1:]
    sp = data.permute(1, 0, 2).reshape(nt * (ns // nr), nr, nc)  # spokes in frame-major order
    d1, d2 = sp[:, :-1], sp[:, 1:]
    h = d1.mH
    g = torch.linalg.solve(h @ d1, h @ d2).mT.cpu().numpy()
    lam, v = np.linalg.eig(g)
    logs = torch.from_numpy((v * np.log(lam)[:, None, :]) @ np.linalg.inv(v)).cuda()
    k0 = trj.permute(2, 1, 0).reshape(nt * (ns // nr), nr, 2)
    nm = ((k0[:, 1] - k0[:, 0]) * float(nr)).double()
    lnG = torch.einsum("dp,pij->dij", torch.linalg.pinv(nm).to(C128), logs)
    cart = torch.empty((2, ns, nt), dtype=torch.int32, device="cuda")
    w = data.reshape(-1, nc)
    for d in range(2):
        t = (trj[d] * float(n[d])).double() + 0.5
        k = torch.round(t)
        cart[d] = k.int() + n[d] // 2
        shift = ((k - t) * nr / n[d]).reshape(-1, 1)
        term, acc = w, w
        for m in range(1, 61):  # exp(shift lnG) data, |shift lnG| well below 20
            term = (term @ lnG[d].mT) * (shift / m)
            acc = acc + term
        w = acc
    return [lnG, w.reshape(ns, nt, nc), cart]


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "apply":
        return _apply_nfft(case, s["x"], s["lam"], s["cells"], s["cmaps"], C128)
    if kind == "apply_cart":
        return _apply_cart(s["x"], s["lam"], s["cmaps"])
    return {"cg": _exact_cg, "kernel": _exact_kernel, "backprojection": _exact_backprojection, "forward": _exact_forward,
            "grog": _exact_grog}[kind](case, s)
