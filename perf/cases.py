"""Workloads of the reconstruction library, timed through its public entry points.

``listed()`` gives the standing set, ``draw(rng)`` one more workload of the same ranges,
``prepare(case, seed)`` what a caller holds before the call (seeded inputs on the GPU, a context
with k-space uploaded, a network with its weights), ``run(state)`` one pass through the public API
and its outputs, ``work(case)`` the bytes and operations the pass cannot do without, and
``exact(case, seed)`` the same outputs in 64-bit torch arithmetic, without the library.

Device images are torch tensors of shape (nq, nz, ny, nx): C order there is the library's
reference layout (x fastest, volume last).
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "llr-reco_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

_DEV = "cuda"


# ---------------------------------------------------------------------------------------
# the workloads
# ---------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # The smallest reconstruction (the size of the repository's smoke run): ten iterations in
        # which launches and dependent latencies are all there is.
        _recon("recon_tiny", (32, 32, 16), 1, 8, (8, 8, 8), accel=4.0, iters=10),
        # Benchmark configuration c1: one shell, 8^3 blocks; a preview-quality protocol.
        _recon("recon_c1", (64, 64, 64), 1, 16, (8, 8, 8), accel=4.0, iters=10),
        # Benchmark configuration c2, the headline workload: whole-brain, 61 volumes, 6^3 blocks.
        _recon("recon_c2", (192, 192, 96), 7, 54, (6, 6, 6), accel=8.0, iters=10),
        # The reference's default prox (hard rank 6) on a ragged volume the blocks do not tile, with
        # per-volume linear phase corrections: a clinical matrix that suits no power of two.
        _recon("recon_hard_ragged", (90, 75, 52), 3, 30, (7, 6, 5), accel=5.0, iters=5, mode="hard", rank=6,
               corrections=True),
        # Benchmark configuration c3 at half its slices: rank-7 temporal subspace, 3-level db4 shrink
        # of the coefficient volumes, 256 x 256 planes.
        _recon("recon_c3_half", (128, 256, 256), 1, 60, (8, 8, 8), accel=10.0, iters=2, srank=7, moments=4, levels=3),
        # Benchmark configuration c5_small: 106 volumes (multi-shell), overlapping 8^3 blocks at stride 4.
        _recon("recon_c5_small", (128, 128, 128), 6, 100, (8, 8, 8), accel=12.0, iters=1, stride=4),
        # The reference's operator loop on device buffers: lift blocks, batched rank truncation, un-lift.
        dict(name="op_lowrank", kind="lowrank", nx=96, ny=96, nz=48, b0=7, dirs=54, bx=6, by=6, bz=6, mode="hard",
             rank=6),
        # The reference's data-consistency loop on device buffers: A, hard projection, A^H.
        dict(name="op_dc", kind="dc", nx=144, ny=120, nz=90, b0=1, dirs=14, accel=4.0),
        # The reference's wavelet shrink (db2, all levels) on odd-sized image volumes.
        dict(name="op_wavelet", kind="wavelet", nx=113, ny=97, nz=61, nvol=6, moments=2, levels=0),
        # The learned warm start of c2: one forward pass of the network over the whole volume.
        dict(name="cnn_forward", kind="cnn", nx=192, ny=192, nz=96, grad=False),
        # One training subject (96^3): loss and every gradient.
        dict(name="cnn_grad", kind="cnn", nx=96, ny=96, nz=96, grad=True),
        # Scalar maps after a c2 reconstruction: tensor fit of 54 directions and 7 b0 volumes.
        dict(name="dti_fit", kind="dti", nx=192, ny=192, nz=96, b0=7, dirs=54),
    ]


def _recon(name, vol, b0, dirs, block, accel, iters, mode="soft", rank=6, srank=0, moments=2, levels=0, stride=0,
           corrections=False) -> dict:
    c = dict(kind="recon", nx=vol[0], ny=vol[1], nz=vol[2], b0=b0, dirs=dirs, bx=block[0], by=block[1], bz=block[2],
             accel=accel, iters=iters, mode=mode, rank=rank, srank=srank, moments=moments, levels=levels,
             stride=stride, corrections=corrections)
    return dict(c, name=name) if name else c


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _vol(rng, lo: int, hi: int, most: float, per: float) -> tuple:
    """Three extents spread over [lo, hi] on a log scale with nx ny nz per <= most."""
    while True:
        v = (_log(rng, lo, hi), _log(rng, lo, hi), _log(rng, lo, hi))
        if v[0] * v[1] * v[2] * per <= most:
            return v


def draw(rng) -> dict:
    kind = rng.choices(["recon", "subspace", "overlap", "lowrank", "dc", "wavelet", "cnn", "dti"],
                       [40, 10, 6, 12, 8, 8, 8, 8])[0]
    if kind == "recon":
        b0, dirs = rng.randint(1, 6), rng.randint(6, 57)
        vol = _vol(rng, 16, 192, 1.2e8, b0 + dirs)
        if rng.random() < 0.3:
            vol = tuple(max(16, v // 8 * 8) for v in vol)
        block = tuple(rng.randint(4, 8) for _ in range(3))
        if rng.random() < 0.6:
            block = (rng.choice([4, 6, 8]),) * 3
        mode = "hard" if rng.random() < 0.35 else "soft"
        return _recon(None, vol, b0, dirs, block, accel=round(rng.uniform(2.0, 10.0), 1), iters=rng.randint(2, 8),
                      mode=mode, rank=rng.randint(2, 6), corrections=rng.random() < 0.3)
    if kind == "subspace":
        b0, dirs = rng.randint(1, 4), rng.randint(20, 60)
        vol = tuple(max(3, v // 8) * 8 for v in _vol(rng, 32, 256, 1.5e8, b0 + dirs))
        return _recon(None, vol, b0, dirs, (8, 8, 8), accel=round(rng.uniform(4.0, 10.0), 1), iters=rng.randint(1, 4),
                      srank=rng.randint(4, 8), moments=rng.choice([2, 4]), levels=0)
    if kind == "overlap":
        b0, dirs = rng.randint(1, 6), rng.randint(60, 110)
        vol = tuple(max(2, v // 8) * 8 for v in _vol(rng, 24, 96, 0.5 * 128 ** 3 * 106, b0 + dirs))
        return _recon(None, vol, b0, dirs, (8, 8, 8), accel=round(rng.uniform(6.0, 12.0), 1), iters=1, stride=4)
    if kind == "lowrank":
        b0, dirs = rng.randint(1, 6), rng.randint(6, 57)
        vol = _vol(rng, 16, 128, 4e7, b0 + dirs)
        return dict(kind="lowrank", nx=vol[0], ny=vol[1], nz=vol[2], b0=b0, dirs=dirs, bx=rng.randint(4, 8),
                    by=rng.randint(4, 8), bz=rng.randint(4, 8), mode=rng.choice(["hard", "soft"]),
                    rank=rng.randint(2, 6))
    if kind == "dc":
        b0, dirs = 1, rng.randint(1, 40)
        vol = _vol(rng, 16, 192, 6e7, b0 + dirs)
        return dict(kind="dc", nx=vol[0], ny=vol[1], nz=vol[2], b0=b0, dirs=dirs, accel=round(rng.uniform(2.0, 10.0), 1))
    if kind == "wavelet":
        nvol = rng.randint(1, 12)
        vol = _vol(rng, 24, 224, 4e7, nvol)
        return dict(kind="wavelet", nx=vol[0], ny=vol[1], nz=vol[2], nvol=nvol, moments=rng.choice([1, 2, 2, 4]),
                    levels=0)
    if kind == "cnn":
        grad = rng.random() < 0.5
        vol = _vol(rng, 16, 160, 1.2e6 if grad else 3.5e6, 1)
        return dict(kind="cnn", nx=vol[0], ny=vol[1], nz=vol[2], grad=grad)
    b0, dirs = rng.randint(1, 7), rng.randint(7, 90)
    vol = _vol(rng, 16, 192, 2.2e8, b0 + dirs)
    return dict(kind="dti", nx=vol[0], ny=vol[1], nz=vol[2], b0=b0, dirs=dirs)


# ---------------------------------------------------------------------------------------
# synthetic acquisitions (torch, seeded)
# ---------------------------------------------------------------------------------------
def _dims(c: dict) -> tuple:
    return c["nx"], c["ny"], c["nz"]


def _nq(c: dict) -> int:
    return c["b0"] + c["dirs"]


def _b_table(c: dict, seed: int):
    """b0 volumes first, then the directions over up to three shells (s/mm^2)."""
    r = np.random.default_rng(seed)
    nd = c["dirs"]
    shells = [1000.0] if nd <= 16 else [3000.0] if nd == 54 else [1000.0, 2000.0] if nd <= 60 else [1000.0, 2000.0, 3000.0]
    b = np.array([0.0] * c["b0"] + [shells[i * len(shells) // nd] for i in range(nd)])
    g = r.standard_normal((len(b), 3))
    g /= np.linalg.norm(g, axis=1, keepdims=True)
    g[: c["b0"]] = 0.0
    return b, g, r


def _axes(c: dict):
    def one(n):
        return (torch.arange(n, device=_DEV, dtype=torch.float32) - n / 2 + 0.5) / (n / 2)
    nx, ny, nz = _dims(c)
    return one(nx)[None, None, :], one(ny)[None, :, None], one(nz)[:, None, None]


def _phantom(c: dict, seed: int) -> torch.Tensor:
    """Diffusion-weighted image (nq, nz, ny, nx) complex64: an isotropic object holding six
    anisotropic ellipsoids, every volume with its own smooth phase."""
    b, g, r = _b_table(c, seed)
    nx, ny, nz = _dims(c)
    X, Y, Z = _axes(c)
    nq = len(b)
    label = ((X / 0.9) ** 2 + (Y / 0.85) ** 2 + (Z / 0.8) ** 2 <= 1.0).to(torch.int64)
    sig = np.zeros((8, nq))
    sig[1] = r.uniform(0.5, 1.0) * np.exp(-b * 3.0e-3)
    outer = label > 0
    for i in range(6):
        ctr, rad = r.uniform(-0.45, 0.45, 3), r.uniform(0.12, 0.35, 3)
        q, _ = np.linalg.qr(r.standard_normal((3, 3)))
        P = [X - float(ctr[0]), Y - float(ctr[1]), Z - float(ctr[2])]
        d2 = sum(((P[0] * float(q[0, k]) + P[1] * float(q[1, k]) + P[2] * float(q[2, k])) / float(rad[k])) ** 2
                 for k in range(3))
        label[(d2 <= 1.0) & outer] = 2 + i
        v, _ = np.linalg.qr(r.standard_normal((3, 3)))
        D = v @ np.diag([1.7e-3, 0.3e-3, 0.3e-3]) @ v.T
        sig[2 + i] = r.uniform(0.5, 1.0) * np.exp(-b * np.einsum("qi,ij,qj->q", g, D, g))
    out = torch.empty((nq, nz, ny, nx), dtype=torch.complex64, device=_DEV)
    table = torch.tensor(sig, dtype=torch.float32, device=_DEV)
    mon = [X, Y, Z, X * X, Y * Y, Z * Z, X * Y, X * Z, Y * Z]
    for k in range(nq):
        cf = r.standard_normal(9) * (math.pi / 6.0)
        ph = sum(float(a) * m for a, m in zip(cf, mon)).expand(nz, ny, nx)
        out[k] = torch.polar(table[:, k][label], ph.contiguous())
    return out


def _noise(shape, sigma: float, seed: int) -> torch.Tensor:
    g = torch.Generator(device=_DEV).manual_seed(seed)
    n = torch.randn(tuple(shape) + (2,), device=_DEV, generator=g)
    return torch.view_as_complex(n) * sigma


def _ramp(c: dict, corr, dtype) -> torch.Tensor:
    """exp(+i theta) of one volume, theta_a(i) = 2 pi (corr_a + n_a / 2) (i - n_a / 2) / n_a."""
    def one(n, cr):
        i = torch.arange(n, device=_DEV, dtype=torch.float64) - n / 2.0
        return torch.polar(torch.ones_like(i), i * (2.0 * math.pi * (float(cr) + 0.5 * n) / n))
    nx, ny, nz = _dims(c)
    return (one(nz, corr[2])[:, None, None] * one(ny, corr[1])[None, :, None] * one(nx, corr[0])[None, None, :]).to(dtype)


def _signal(c: dict, x: torch.Tensor, lk, li, inverse: bool) -> torch.Tensor:
    """A (or A^H) of every volume, in x's precision."""
    out = torch.empty_like(x)
    for q in range(x.shape[0]):
        k, i = _ramp(c, lk[q], x.dtype), _ramp(c, li[q], x.dtype)
        if inverse:
            out[q] = torch.fft.ifftn(x[q] * i, norm="ortho") * k.conj()
        else:
            out[q] = torch.fft.fftn(x[q] * k, norm="ortho") * i.conj()
    return out


def _corrections(c: dict, seed: int):
    n = _nq(c)
    if not c.get("corrections"):
        return np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32)
    r = np.random.default_rng(seed + 77)
    return (r.integers(-2, 3, (n, 3)).astype(np.float32), r.uniform(-1.5, 1.5, (n, 3)).astype(np.float32))


def _lines(c: dict, seed: int) -> torch.Tensor:
    """Variable-density ky-kz sampling, one mask per volume, with a fully sampled centre (nq, nz, ny, 1)."""
    _, ny, nz = _dims(c)
    r = np.random.default_rng(seed + 5)
    dy = (np.arange(ny) - ny // 2) / (ny / 2.0)
    dz = (np.arange(nz) - nz // 2) / (nz / 2.0)
    w = np.maximum(1.0 - np.hypot(dz[:, None], dy[None, :]), 0.0) ** 2 + 0.02
    h = max(2, min(16, min(ny, nz) // 4)) // 2
    want = ny * nz / c["accel"]
    p = np.minimum(1.0, w * want / w.sum())
    for _ in range(6):
        p = np.minimum(1.0, p * want / p.sum())
    p[nz // 2 - h: nz // 2 + h, ny // 2 - h: ny // 2 + h] = 1.0
    m = r.random((_nq(c), nz, ny)) < p
    return torch.from_numpy(m).to(_DEV)[..., None]


def _kspace(c: dict, seed: int) -> torch.Tensor:
    """Measured k-space (nq, nz, ny, nx) complex64: SNR 30, unsampled x-lines zero."""
    x = _phantom(c, seed)
    lk, li = _corrections(c, seed)
    x = _signal(c, x, lk, li, False)
    x += _noise(x.shape, 0.02, seed + 1)
    return x.mul_(_lines(c, seed))


def _subspace(c: dict, seed: int) -> np.ndarray:
    """Temporal subspace (nq, srank): leading left singular vectors of simulated tensor signals."""
    b, g, _ = _b_table(c, seed)
    r = np.random.default_rng(seed + 9)
    n = 4000
    lam = r.uniform(0.1e-3, 3.0e-3, (n, 3))
    v = np.linalg.qr(r.standard_normal((n, 3, 3)))[0]
    D = np.einsum("nik,nk,njk->nij", v, lam, v)
    s = np.exp(-b[:, None] * np.einsum("qi,nij,qj->qn", g, D, g))
    return np.asfortranarray(np.linalg.svd(s, full_matrices=False)[0][:, : c["srank"]].astype(np.complex64))


def _image(c: dict, seed: int) -> torch.Tensor:
    """Noisy image volumes, as a reconstruction gives them."""
    x = _phantom(c, seed)
    x += _noise(x.shape, 0.02, seed + 1)
    return x


def _channels(c: dict, seed: int) -> torch.Tensor:
    """Network channels (nz, ny, nx, 14): smooth structure plus noise, unit RMS."""
    nx, ny, nz = _dims(c)
    g = torch.Generator(device=_DEV).manual_seed(seed)
    low = torch.randn((1, 14, max(2, nz // 8), max(2, ny // 8), max(2, nx // 8)), device=_DEV, generator=g)
    up = torch.nn.functional.interpolate(low, size=(nz, ny, nx), mode="trilinear", align_corners=False)[0]
    out = up.permute(1, 2, 3, 0).contiguous()
    out += 0.3 * torch.randn(out.shape, device=_DEV, generator=g)
    return out.div_(out.square().mean().sqrt())


def _weights_file() -> str:
    return os.path.join(_PKG, "llr_b200", "data", "warm_start_net.npz")


# ---------------------------------------------------------------------------------------
# what a caller holds before the call
# ---------------------------------------------------------------------------------------
def _ptr(t: torch.Tensor) -> C.c_void_p:
    return C.c_void_p(t.data_ptr())


def prepare(case: dict, seed: int) -> dict:
    return {"recon": _prepare_recon, "lowrank": _prepare_lowrank, "dc": _prepare_dc, "wavelet": _prepare_wavelet,
            "cnn": _prepare_cnn, "dti": _prepare_dti}[case["kind"]](case, seed)


def run(state: dict):
    return state["pass"](state)


def _prepare_recon(c, seed):
    from llr_b200 import LLR_PROX_HARD_RANK, LLR_PROX_SOFT_THRESH, ReconContext, ReconParams, _lib as L
    hard = c["mode"] == "hard"
    p = ReconParams(vol_size=_dims(c), nq=_nq(c), block_size=(c["bx"], c["by"], c["bz"]),
                    prox_mode=LLR_PROX_HARD_RANK if hard else LLR_PROX_SOFT_THRESH, rank=c["rank"], seed=seed,
                    block_stride=(c["stride"],) * 3 if c["stride"] else None)
    if c["srank"]:
        p.subspace_rank, p.wavelet_space, p.wavelet_alpha = c["srank"], 1, 0.005
        p.wavelet_moments, p.wavelet_levels = c["moments"], c["levels"]
    ctx = ReconContext(p)
    if c["corrections"]:
        ctx.set_linear_corrections(*_corrections(c, seed))
    y = _kspace(c, seed)
    torch.cuda.synchronize()
    L.check(L.lib.llr_upload_kspace_dev(ctx.h, _ptr(y)))
    if c["srank"]:
        ctx.upload_subspace(_subspace(c, seed))
    if not hard:
        ctx.init_zero_filled()
        ctx.set_lambda(0.02 * ctx.sigma_max((0, 0, 0)))
    return {"pass": _run_recon, "ctx": ctx, "iters": c["iters"], "image": y}


def _run_recon(s):
    """One reconstruction call: zero-filled start, the iterations, the image."""
    from llr_b200 import _lib as L
    ctx = s["ctx"]
    ctx.init_zero_filled()
    hist = ctx.iterate(s["iters"])
    L.check(L.lib.llr_download_image_dev(ctx.h, _ptr(s["image"])))
    return {"image": s["image"], "residual": hist.astype(np.float32)}


def _grid(c):
    return c["nx"] // c["bx"], c["ny"] // c["by"], c["nz"] // c["bz"]


def _prepare_lowrank(c, seed):
    gx, gy, gz = _grid(c)
    m, n, nb = c["bx"] * c["by"] * c["bz"], _nq(c), gx * gy * gz
    x = _image(c, seed)
    r = np.random.default_rng(seed + 3)
    shift = tuple(int(v) for v in r.integers(0, _dims(c)))
    return {"pass": _run_lowrank, "c": c, "x": x, "out": x.clone(), "shift": shift, "m": m, "nb": nb,
            "lam": _op_lambda(c, x, shift), "mats": torch.empty((nb, n, m), dtype=torch.complex64, device=_DEV)}


def _run_lowrank(s):
    from llr_b200 import _lib as L
    c, nq, nb = s["c"], _nq(s["c"]), s["nb"]
    vs, bs, sh = L.i32x3(_dims(c)), L.i32x3((c["bx"], c["by"], c["bz"])), L.i32x3(s["shift"])
    mats, out = _ptr(s["mats"]), _ptr(s["out"])
    L.check(L.lib.llr_lift_data_set_dev(_ptr(s["x"]), nq, mats, vs, bs, sh, 0, nb, None))
    if c["mode"] == "hard":
        L.check(L.lib.llr_low_rank_batch_dev(s["m"], nq, c["rank"], nb, mats, None))
    else:
        L.check(L.lib.llr_soft_threshold_batch_dev(s["m"], nq, s["lam"], nb, mats, None))
    L.check(L.lib.llr_un_lift_data_set_dev(out, nq, mats, vs, bs, sh, 0, nb, None))
    return s["out"]


def _prepare_dc(c, seed):
    return {"pass": _run_dc, "c": c, "x": _image(c, seed + 20), "y": _kspace(c, seed),
            "k": torch.empty((_nq(c), c["nz"], c["ny"], c["nx"]), dtype=torch.complex64, device=_DEV)}


def _run_dc(s):
    from llr_b200 import _lib as L
    c, k = s["c"], s["k"]
    dims, nq, err = L.i32x3(_dims(c)), _nq(c), C.c_double()
    k.copy_(s["x"])
    L.check(L.lib.llr_signal_model_dev(_ptr(k), dims, nq, None, None, L.LLR_FORWARD, None))
    L.check(L.lib.llr_hard_project_dev(_ptr(k), _ptr(s["y"]), k.numel(), C.byref(err), None))
    L.check(L.lib.llr_signal_model_dev(_ptr(k), dims, nq, None, None, L.LLR_INVERSE, None))
    return {"image": k, "error": np.float32(err.value)}


def _wavelet_image(c, seed):
    return _image(dict(c, b0=1, dirs=c["nvol"] - 1) if c["nvol"] > 1 else dict(c, b0=1, dirs=0), seed)


def _prepare_wavelet(c, seed):
    x = _wavelet_image(c, seed)
    return {"pass": _run_wavelet, "c": c, "x": x, "out": torch.empty_like(x)}


_ALPHA = 0.02   # about the noise level of one volume


def _run_wavelet(s):
    from llr_b200 import _lib as L
    c, out = s["c"], s["out"]
    out.copy_(s["x"])
    L.check(L.lib.llr_wavelet_denoise_dev(_ptr(out), L.i32x3(_dims(c)), c["nvol"], c["moments"], c["levels"], _ALPHA,
                                          None))
    return out


def _prepare_cnn(c, seed):
    from llr_b200.cnn import Cnn
    x = _channels(c, seed)
    s = {"pass": _run_cnn, "c": c, "net": Cnn.load(_weights_file()), "x": x}
    s["out" if not c["grad"] else "target"] = torch.empty_like(x) if not c["grad"] else _target(x, seed)
    return s


def _target(x, seed):
    g = torch.Generator(device=_DEV).manual_seed(seed + 50)
    return x * 0.9 + 0.05 * torch.randn(x.shape, device=_DEV, generator=g)


def _run_cnn(s):
    from llr_b200 import _lib as L
    c, net = s["c"], s["net"]
    dims = (C.c_int32 * 3)(*_dims(c))
    if not c["grad"]:
        L.check(L.lib.llr_cnn_forward_dev(net.h, _ptr(s["x"]), _ptr(s["out"]), dims, None))
        return s["out"]
    loss = C.c_double()
    L.check(L.lib.llr_cnn_loss_grad_dev(net.h, _ptr(s["x"]), _ptr(s["target"]), dims, C.byref(loss), None))
    return {"loss": np.float32(loss.value), "grads": net.grads}


def _prepare_dti(c, seed):
    b, g, _ = _b_table(c, seed)
    x = _image(c, seed)
    V = c["nx"] * c["ny"] * c["nz"]
    return {"pass": _run_dti, "c": c, "x": x, "V": V, "b": np.ascontiguousarray(b[c["b0"]:], np.float32),
            "g": np.ascontiguousarray(g[c["b0"]:], np.float32), "out": torch.empty((7, V), device=_DEV)}


def _run_dti(s):
    from llr_b200 import _lib as L
    c, x = s["c"], s["x"]
    L.check(L.lib.llr_dti_fit_dev(_ptr(x[c["b0"]:]), c["dirs"], _ptr(x), c["b0"], s["V"], L.fptr(s["b"]),
                                  L.fptr(s["g"]), _ptr(s["out"]), None))
    return s["out"]


# ---------------------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    c = case
    V = c["nx"] * c["ny"] * c["nz"]
    lg = math.log2(V)
    if c["kind"] == "recon":
        # Per iteration: the prox reads and writes the iterate, data consistency reads and writes it
        # and reads the sampled lines; once: the zero-filled start and the image.
        n, E, it = _nq(c), V * _nq(c), c["iters"]
        nb = V // (c["bx"] * c["by"] * c["bz"]) * ((c["bx"] // c["stride"]) ** 3 if c["stride"] else 1)
        m, k = c["bx"] * c["by"] * c["bz"], c["srank"] or n
        prox = nb * (4.0 * m * k * k + 16.0 * m * k * min(8, k) + (16.0 * m * n * k if c["srank"] else 0.0))
        return {"bytes": it * (32.0 * E + 8.0 * E / c["accel"]) + 8.0 * E + 16.0 * E,
                "flops": it * (prox + 10.0 * E * lg) + 5.0 * E * lg}
    if c["kind"] == "lowrank":
        n, m = _nq(c), c["bx"] * c["by"] * c["bz"]
        nb = math.prod(_grid(c))
        return {"bytes": 16.0 * m * n * nb, "flops": nb * (4.0 * m * n * n + 16.0 * m * n * c["rank"])}
    if c["kind"] == "dc":
        E = V * _nq(c)
        return {"bytes": 24.0 * E, "flops": 10.0 * E * lg}
    if c["kind"] == "wavelet":
        return {"bytes": 16.0 * V * c["nvol"], "flops": 2 * 3 * 4.0 * 2 * c["moments"] * V * c["nvol"] * 8 / 7}
    if c["kind"] == "cnn":
        f = 2.0 * 27 * (14 * 32 + 6 * 32 * 32 + 32 * 14) * V
        return {"bytes": 2 * 56.0 * V, "flops": 3 * f if c["grad"] else f}
    return {"bytes": V * (8.0 * _nq(c) + 28.0), "flops": V * (c["dirs"] * 20.0 + 200.0)}


# ---------------------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    c = case
    if c["kind"] == "recon":
        return _exact_recon(c, seed)
    if c["kind"] == "lowrank":
        if c["nx"] * c["ny"] * c["nz"] * _nq(c) > 3e7:
            return None
        x = _image(c, seed)
        r = np.random.default_rng(seed + 3)
        shift = tuple(int(v) for v in r.integers(0, _dims(c)))
        lam = _op_lambda(c, x, shift)
        out = x.to(torch.complex128)
        _prox(c, out, shift, lam)
        return out
    if c["kind"] == "dc":
        y, x = _kspace(c, seed).to(torch.complex128), _image(c, seed + 20).to(torch.complex128)
        z = np.zeros((_nq(c), 3))
        k = _signal(c, x, z, z, False)
        on = y != 0
        err = float((k - y)[on].abs().square().sum())
        return {"image": _signal(c, torch.where(on, y, k), z, z, True), "error": np.float64(err)}
    if c["kind"] == "wavelet":
        x = _wavelet_image(c, seed).to(torch.complex128)
        return torch.stack([_shrink_volume(v, _ALPHA, c["moments"], c["levels"]) for v in x])
    if c["kind"] == "cnn":
        return _exact_cnn(c, seed)
    return _exact_dti(c, seed)


def _blocks(c, x, shift):
    """(nb, m, n) view-copy of the shifted blocks of x (nq, nz, ny, nx), and the rolled array."""
    gx, gy, gz = _grid(c)
    n = x.shape[0]
    r = torch.roll(x, (-shift[2], -shift[1], -shift[0]), (1, 2, 3))
    v = r[:, : gz * c["bz"], : gy * c["by"], : gx * c["bx"]].reshape(n, gz, c["bz"], gy, c["by"], gx, c["bx"])
    return v.permute(1, 3, 5, 2, 4, 6, 0).reshape(gz * gy * gx, -1, n), r


def _op_lambda(c, x, shift) -> float:
    """0.02 of the largest block norm of the input."""
    B, _ = _blocks(c, x, shift)
    return float(np.float32(0.02 * math.sqrt(float(B.abs().square().double().sum((1, 2)).max()))))


def _low_rank(B, mode, rank, lam):
    """Rank truncation or singular-value soft threshold of every matrix of B (nb, m, n)."""
    out = torch.empty_like(B)
    step = max(1, int(2e8) // max(1, B.shape[1] * B.shape[2] * 16))
    for i in range(0, B.shape[0], step):
        b = B[i: i + step]
        w, v = torch.linalg.eigh(b.mH @ b)
        if mode == "hard":
            f = torch.zeros_like(w)
            f[:, -rank:] = 1.0
        else:
            s = w.clamp_min(0.0).sqrt()
            f = torch.where(s > lam, 1.0 - lam / s.clamp_min(1e-300), torch.zeros_like(s))
        out[i: i + step] = ((b @ v) * f[:, None, :]) @ v.mH
    return out


def _prox(c, x, shift, lam):
    """x <- un-lift(LR(lift(x))), in place; voxels no block covers keep their values."""
    gx, gy, gz = _grid(c)
    n = x.shape[0]
    B, r = _blocks(c, x, shift)
    B = _low_rank(B, c["mode"], c["rank"], lam)
    v = B.reshape(gz, gy, gx, c["bz"], c["by"], c["bx"], n).permute(6, 0, 3, 1, 4, 2, 5)
    r[:, : gz * c["bz"], : gy * c["by"], : gx * c["bx"]] = v.reshape(n, gz * c["bz"], gy * c["by"], gx * c["bx"])
    x.copy_(torch.roll(r, (shift[2], shift[1], shift[0]), (1, 2, 3)))


def _draw_shift(seed: int, it: int, dims) -> tuple:
    """Block shift of iteration ``it``: SplitMix64 keyed by (seed, iteration, axis)."""
    M, G = (1 << 64) - 1, 0x9E3779B97F4A7C15

    def mix(x):
        z = (x + G) & M
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
        return z ^ (z >> 31)
    return tuple(mix((seed + G * ((0x5348 << 32) + 3 * it + a + 1)) & M) % dims[a] for a in range(3))


def _exact_recon(c, seed):
    if c["stride"] or c["nx"] * c["ny"] * c["nz"] * _nq(c) * c["iters"] > 6e7:
        return None
    lk, li = _corrections(c, seed)
    y = _kspace(c, seed).to(torch.complex128)
    on = y != 0
    x = _signal(c, y, lk, li, True)
    lam, S = 0.0, None
    if c["mode"] == "soft":
        B, _ = _blocks(c, x, (0, 0, 0))
        fro = B.abs().square().sum((1, 2))
        top = B[torch.argsort(fro, descending=True)[:128]]
        lam = 0.02 * math.sqrt(float(torch.linalg.eigvalsh(top.mH @ top).max()))
    if c["srank"]:
        S = torch.from_numpy(_subspace(c, seed)).to(_DEV).to(torch.complex128)
    hist = []
    for it in range(c["iters"]):
        shift = _draw_shift(seed, it, _dims(c))
        if S is None:
            _prox(c, x, shift, lam)
        else:
            z = torch.einsum("qzyx,qk->kzyx", x, S).contiguous()
            _prox(c, z, shift, lam)
            z = torch.stack([_shrink_volume(v, 0.005, c["moments"], c["levels"]) for v in z])
            x = torch.einsum("kzyx,qk->qzyx", z, S.conj()).contiguous()
        k = _signal(c, x, lk, li, False)
        hist.append(float((k - y)[on].abs().square().sum()))
        x = _signal(c, torch.where(on, y, k), lk, li, True)
    return {"image": x, "residual": np.array(hist)}


def _scaling_filter(N: int) -> np.ndarray:
    """Minimum-phase Daubechies scaling filter by spectral factorisation, sum sqrt 2."""
    poly = np.array([1.0 + 0j])
    for _ in range(N):
        poly = np.convolve(poly, [1.0, 1.0])
    if N > 1:
        for y in np.roots([math.comb(N - 1 + k, k) for k in range(N)][::-1]):
            r = np.roots([1.0, -(2.0 - 4.0 * y), 1.0])
            poly = np.convolve(poly, [1.0, -r[np.argmin(np.abs(r))]])
    h = np.real(poly)
    return h * (math.sqrt(2.0) / h.sum())


def _banks(N: int, n: int):
    """Analysis (2 nc, n) and synthesis (n, 2 nc) matrices of one level along an axis of length n:
    half-sample symmetric extension, centre samples kept."""
    lo = _scaling_filter(N)
    F = 2 * N
    hi = np.array([(-1.0) ** k * lo[F - 1 - k] for k in range(F)])
    nc = (n + F - 1) // 2
    A, Sy = np.zeros((2 * nc, n)), np.zeros((n, 2 * nc))
    for r in range(nc):
        for j in range(F):
            i = 2 * r - F + 2 + j
            i = -i - 1 if i < 0 else i
            i = 2 * n - i - 1 if i >= n else i
            A[r, i] += lo[j]
            A[nc + r, i] += hi[j]
    for s in range(n):
        for j in range(F):
            i = (2 * nc + F - 1 - (2 * nc - F + 2)) // 2 + s - j
            if 0 <= i < 2 * nc and i % 2 == 0:
                Sy[s, i // 2] += lo[j]
                Sy[s, nc + i // 2] += hi[j]
    return (torch.from_numpy(A).to(_DEV).to(torch.complex128), torch.from_numpy(Sy).to(_DEV).to(torch.complex128), nc)


def _along(Mx, My, Mz, v):
    v = torch.einsum("ax,zyx->zya", Mx, v)
    v = torch.einsum("by,zya->zba", My, v)
    return torch.einsum("cz,zba->cba", Mz, v)


def _shrink(v, alpha):
    m = v.abs()
    return v * torch.where(m > 0, (m - alpha).clamp_min(0.0) / m.clamp_min(1e-300), torch.zeros_like(m))


def _shrink_volume(v, alpha, moments, levels):
    """Every detail band of every level and the last approximation shrunk by alpha."""
    if levels <= 0:
        q = min(v.shape) / (2 * moments - 1)
        levels = int(math.floor(math.log2(q))) if q >= 1 else 0
    if levels == 0:
        return v
    nz, ny, nx = v.shape
    (ax, sx, cx), (ay, sy, cy), (az, sz, cz) = _banks(moments, nx), _banks(moments, ny), _banks(moments, nz)
    d = _along(ax, ay, az, v)
    low = d[:cz, :cy, :cx].clone()
    d = _shrink(d, alpha)
    if levels > 1:
        d[:cz, :cy, :cx] = _shrink_volume(low, alpha, moments, levels - 1)
    return _along(sx, sy, sz, d)


def _exact_cnn(c, seed):
    z = np.load(_weights_file())
    ch, p = [int(v) for v in z["channels"]], torch.from_numpy(np.asarray(z["params"], np.float32))
    x = _channels(c, seed)
    layers, off = [], 0
    for ci, co in zip(ch[:-1], ch[1:]):
        W = p[off: off + 27 * ci * co].to(torch.bfloat16).double().reshape(3, 3, 3, ci, co)
        off += 27 * ci * co
        layers.append((W.permute(4, 3, 0, 1, 2).contiguous().to(_DEV).requires_grad_(c["grad"]),
                       p[off: off + co].double().to(_DEV).requires_grad_(c["grad"])))
        off += co
    with torch.set_grad_enabled(c["grad"]):
        h0 = x.double().permute(3, 0, 1, 2)[None]
        h = h0
        for i, (W, b) in enumerate(layers):
            h = _conv3(h, W, b)
            if i + 1 < len(layers):
                h = torch.relu(h)
        out = (h0 + h)[0].permute(1, 2, 3, 0)
        if not c["grad"]:
            return out.contiguous()
        loss = (out - _target(x, seed).double()).square().mean()
        loss.backward()
    g = []
    for W, b in layers:
        g += [W.grad.permute(2, 3, 4, 1, 0).reshape(-1), b.grad]
    return {"loss": np.float64(float(loss.detach())), "grads": torch.cat(g).cpu().numpy()}


def _conv3(h, W, b):
    """conv3d 3x3x3 with zero padding as 27 matrix products (64-bit convolutions are slow)."""
    _, ci, nz, ny, nx = h.shape
    p = torch.nn.functional.pad(h[0], (1, 1, 1, 1, 1, 1))
    out = b[:, None].expand(W.shape[0], nz * ny * nx)
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                out = out + W[:, :, dz, dy, dx] @ p[:, dz: dz + nz, dy: dy + ny, dx: dx + nx].reshape(ci, -1)
    return out.reshape(1, -1, nz, ny, nx)


def _exact_dti(c, seed):
    b, g, _ = _b_table(c, seed)
    b, g = (np.ascontiguousarray(v[c["b0"]:], np.float32).astype(np.float64) for v in (b, g))
    A = np.stack([-b * g[:, 0] ** 2, -b * g[:, 1] ** 2, -b * g[:, 2] ** 2, -2 * b * g[:, 0] * g[:, 1],
                  -2 * b * g[:, 0] * g[:, 2], -2 * b * g[:, 1] * g[:, 2]], 1)
    P = torch.from_numpy(np.linalg.pinv(A)).to(_DEV)
    x = _image(c, seed).reshape(_nq(c), -1)
    tiny = float(np.finfo(np.float32).tiny)
    out = torch.empty((7, x.shape[1]), dtype=torch.float64, device=_DEV)
    for i in range(0, x.shape[1], 1 << 19):
        m = x[:, i: i + (1 << 19)].to(torch.complex128).abs()
        s0 = m[: c["b0"]].mean(0)
        t = P @ (m[c["b0"]:] / s0.clamp_min(tiny)).clamp(tiny, 1.0).log()
        D = torch.stack([t[0], t[3], t[4], t[3], t[1], t[5], t[4], t[5], t[2]], -1).reshape(-1, 3, 3)
        e1, e2, e3 = _eig3(D)
        md = (e1 + e2 + e3) / 3.0
        num = ((e1 - md) ** 2 + (e2 - md) ** 2 + (e3 - md) ** 2).sqrt()
        fa = math.sqrt(1.5) * num / (e1 ** 2 + e2 ** 2 + e3 ** 2).sqrt()
        out[:, i: i + (1 << 19)] = torch.stack([s0, e1, e2, e3, md, 0.5 * (e2 + e3), fa])
    return out


def _eig3(D):
    """Eigenvalues of symmetric 3 x 3 matrices, descending (cyclic Jacobi rotations)."""
    D = D.clone()
    for _ in range(8):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            apq, app, aqq = D[:, p, q].clone(), D[:, p, p].clone(), D[:, q, q].clone()
            th = 0.5 * torch.atan2(2.0 * apq, aqq - app)
            cs, sn = torch.cos(th), torch.sin(th)
            arp, arq = D[:, r, p].clone(), D[:, r, q].clone()
            D[:, p, p] = cs * cs * app - 2 * cs * sn * apq + sn * sn * aqq
            D[:, q, q] = sn * sn * app + 2 * cs * sn * apq + cs * cs * aqq
            v = (cs * cs - sn * sn) * apq + cs * sn * (app - aqq)
            D[:, p, q], D[:, q, p] = v, v
            u, w = cs * arp - sn * arq, sn * arp + cs * arq
            D[:, r, p], D[:, p, r], D[:, r, q], D[:, q, r] = u, u, w, w
    e = torch.stack([D[:, 0, 0], D[:, 1, 1], D[:, 2, 2]], -1).sort(-1, descending=True).values
    return e[:, 0], e[:, 1], e[:, 2]
