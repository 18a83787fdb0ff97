"""Casorati matrices of 65 to 128 columns: the split path (tensor-core Gram, Jacobi eigen kernel with a rotation
log, apply kernel, wide kernel over the blocks handed back) against the FP64 oracle."""
import ctypes as C
import time

import numpy as np
import pytest

from conftest import crandn, rel_err
from oracle import llr_oracle as O

from llr_b200 import DeviceBuffer, ReconContext, ReconParams, _lib as L

pytestmark = pytest.mark.gpu


def _low_rank_mats(rng, m, n, k, batch, noise):
    """k components between 1 and 0.3 over noise, the last matrix noise alone."""
    out = noise * crandn(rng, (m, n, batch), np.complex128)
    for b in range(batch - 1):
        u = np.linalg.qr(crandn(rng, (m, k), np.complex128))[0]
        v = np.linalg.qr(crandn(rng, (n, k), np.complex128))[0]
        out[:, :, b] += (u * np.linspace(1.0, 0.3, k)) @ v.conj().T
    return np.asfortranarray(out.astype(np.complex64))


@pytest.mark.parametrize("m,n,k,batch", [(65, 65, 1, 3), (512, 106, 4, 7), (130, 128, 8, 5), (33, 127, 3, 4),
                                         (512, 107, 12, 2), (64, 80, 2, 700)])
@pytest.mark.parametrize("mode", ["soft", "hard"])
def test_wide_batch_matches_oracle(gpu, m, n, k, batch, mode):
    """Column counts at both ends and odd, more rows or fewer than columns, kept counts up to and beyond what a
    block's factor holds (8; 12 takes the wide kernel), blocks that are zero, more blocks than CTAs.  FP32 Gram and
    rotations: relative 5e-5, the prox tolerance."""
    rng = np.random.default_rng(m + n)
    x = _low_rank_mats(rng, m, n, k, batch, 1e-3)
    d = DeviceBuffer.from_array(x)
    if mode == "soft":
        L.check(L.lib.llr_soft_threshold_batch_dev(m, n, 0.1, batch, d.ptr, None))
        exp = O.low_rank_soft(x.astype(np.complex128), 0.1)
    else:
        L.check(L.lib.llr_low_rank_batch_dev(m, n, k, batch, d.ptr, None))
        exp = O.low_rank_hard(x.astype(np.complex128), k)
    got = d.download(np.empty_like(x, order="F"))
    d.close()
    cut = batch - 1 if mode == "hard" else batch      # the noise matrix has no gap for a rank cut
    assert rel_err(got[..., :cut], exp[..., :cut]) < 5e-5
    if mode == "soft":
        assert not got[..., -1].any()


@pytest.mark.parametrize("mode", ["soft", "hard"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_wide_batch_keeps_non_finite_matrices(gpu, mode, bad):
    """One element, and a whole matrix, that is not finite: those matrices stay so (the residual check of an
    iteration relies on it) and the others do not change by a bit."""
    m, n, batch = 96, 80, 6
    x = _low_rank_mats(np.random.default_rng(3), m, n, 3, batch, 1e-3)
    out = []
    for hurt in (False, True):
        y = x.copy(order="F")
        if hurt:
            y[5, 7, 1] = bad
            y[:, :, 3] = bad
        d = DeviceBuffer.from_array(y)
        if mode == "soft":
            L.check(L.lib.llr_soft_threshold_batch_dev(m, n, 10.0, batch, d.ptr, None))
        else:
            L.check(L.lib.llr_low_rank_batch_dev(m, n, 3, batch, d.ptr, None))
        out.append(d.download(np.empty_like(x, order="F")))
        d.close()
    for b in range(batch):
        if b in (1, 3):
            assert not np.isfinite(out[1][..., b]).all()
        else:
            assert np.array_equal(out[0][..., b], out[1][..., b])


@pytest.mark.parametrize("m,n", [(2048, 66), (512, 106), (128, 128)])
def test_wide_gram_sums_keep_fp32_accuracy(gpu, m, n):
    """Orthogonal columns: the Gram matrix is diagonal, no rotation acts, and the gains 1 - lambda / s show the error of
    its sums over all m rows alone.  Six kept columns with lambda = 0.9 s (the others below lambda): a relative error e of
    s^2 gives 4.5 e.  Sums of 32 products truncated in tensor memory (at most 2^-23 of the partial sum per eight) and m / 32
    FP32 additions stay below 1e-6, so 5e-6; sums truncated over 2048 rows were 4e-5 short."""
    H = np.ones((1, 1))
    while H.shape[0] < m:
        H = np.block([[H, H], [H, -H]])
    amp = np.where(np.arange(n) < 6, 0.3718, 0.05)
    x = np.asfortranarray((H[:m, :n] * amp * np.exp(0.7j))[..., None].astype(np.complex64))
    sv = np.linalg.norm(x[:, 0, 0].astype(np.complex128))
    lam = np.float32(0.9 * sv)
    d = DeviceBuffer.from_array(x)
    L.check(L.lib.llr_soft_threshold_batch_dev(m, n, float(lam), 1, d.ptr, None))
    got = d.download(np.empty_like(x, order="F"))
    d.close()
    exp = x.astype(np.complex128) * (1.0 - float(lam) / sv)
    assert rel_err(got[:, :6], exp[:, :6]) < 5e-6
    assert np.abs(got[:, 6:]).max() < 1e-6


@pytest.mark.parametrize("m,n,k,batch", [(512, 106, 9, 3), (216, 80, 33, 5), (130, 128, 64, 2), (300, 65, 65, 3), (96, 71, 40, 700)])
@pytest.mark.parametrize("mode", ["soft", "hard"])
def test_wide_batch_keeping_more_than_a_factor_holds(gpu, mode, m, n, k, batch):
    """Nine components, around one and two rounds of 32 columns, all of them (odd n), more blocks than CTAs: such blocks
    get W from the eigen kernel and only the product from the wide one.  Tolerance as above."""
    rng = np.random.default_rng(m + k)
    x = _low_rank_mats(rng, m, n, k, batch, 1e-4)
    d = DeviceBuffer.from_array(x)
    if mode == "soft":
        L.check(L.lib.llr_soft_threshold_batch_dev(m, n, 0.1, batch, d.ptr, None))
        exp = O.low_rank_soft(x.astype(np.complex128), 0.1)
    else:
        L.check(L.lib.llr_low_rank_batch_dev(m, n, k, batch, d.ptr, None))
        exp = O.low_rank_hard(x.astype(np.complex128), k)
    got = d.download(np.empty_like(x, order="F"))
    d.close()
    assert rel_err(got[..., :batch - 1], exp[..., :batch - 1]) < 5e-5


def _wide_ctx(gram_mode, lam=0.0, rank=0, stride=None, nq=70):
    rng = np.random.default_rng(11)
    vol = (16, 16, 16)
    y = crandn(rng, vol + (nq,)) * (rng.random((1, 16, 16, nq)) < 0.5)
    p = ReconParams(vol_size=vol, nq=nq, block_size=(8, 8, 8), prox_mode=0 if rank else 1, rank=max(rank, 1), lam=lam, seed=2,
                    gram_mode=gram_mode, block_stride=stride)
    ctx = ReconContext(p)
    ctx.upload_kspace(np.asfortranarray(y.astype(np.complex64)))
    ctx.init_zero_filled()
    return ctx


@pytest.mark.parametrize("stride", [None, (4, 8, 8)])
def test_wide_context_with_many_kept_components(gpu, stride):
    """Volume blocks, overlapping ones too (their results are accumulated), every component above the threshold: image,
    residual and objective against the FP32 Gram mode, whose blocks all take the wide kernel.  Two FP32 paths of error 5e-5
    each (prox tolerance); the objective's nuclear norms are sums of positive singular values."""
    out = []
    for gm in (0, 1):
        with _wide_ctx(gm, lam=2.0, stride=stride) as ctx:
            h = ctx.iterate(2)
            out.append((ctx.download_image(), h, ctx.objective_history(2)))
    assert rel_err(out[0][0], out[1][0]) < 1e-4
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=2e-4)
    if stride is None:
        np.testing.assert_allclose(out[0][2], out[1][2], rtol=2e-4)


@pytest.mark.parametrize("kw", [dict(rank=12), dict(lam=2.0)])
def test_wide_blocks_are_not_solved_twice(gpu, kw):
    """A hard rank above eight, or a threshold that keeps more, against the FP32 Gram mode, where one kernel does all: with
    the eigenproblem solved twice it took 1.3 times as long."""
    ms = {}
    for gm in (0, 1):
        with _wide_ctx(gm, **kw) as ctx:
            ctx.iterate(1)
            ms[gm] = min(ctx.iterate_timed(2) for _ in range(5))
    assert ms[0] < 1.1 * ms[1]


def test_wide_scratch_is_not_mapped_on_every_call(gpu):
    """600 blocks of 128 columns whose outputs are all zero against 100 of them: the rotation log (519 MB) outweighed what
    the scratch pool kept and was mapped anew by every call, 85 times as long."""
    best = {}
    for batch in (100, 600):
        x = _low_rank_mats(np.random.default_rng(1), 64, 128, 2, 1, 1e-3)
        x = np.asfortranarray(np.broadcast_to(x, (64, 128, batch)))
        d = DeviceBuffer.from_array(x)
        for _ in range(8):
            L.check(L.lib.llr_stream_sync(None))
            t0 = time.perf_counter()
            L.check(L.lib.llr_soft_threshold_batch_dev(64, 128, 100.0, batch, d.ptr, None))
            L.check(L.lib.llr_stream_sync(None))
            best[batch] = min(best.get(batch, 1.0), time.perf_counter() - t0)
        d.close()
    assert best[600] < 10 * best[100]


def test_wide_context_without_room_for_the_split_path(gpu):
    """128 volumes in blocks of one voxel: a Gram matrix per block would be 197 GB.  The context is created without it, as
    before there was a split path, and holds the image buffers, the tables and the wide kernel's scratch only."""
    p = ReconParams(vol_size=(144, 144, 144), nq=128, block_size=(1, 1, 1), prox_mode=1, lam=0.1)
    with ReconContext(p) as ctx:
        assert ctx.device_bytes() < 8 << 30
    y = np.zeros((4, 4, 4, 80), np.complex64, order="F")
    with ReconContext(ReconParams(vol_size=(4, 4, 4), nq=80, block_size=(2, 2, 2), prox_mode=1, lam=0.1)) as ctx:
        ctx.upload_kspace(y)      # the next allocations do not see the failed one
        ctx.init_zero_filled()
        ctx.iterate(1)


@pytest.mark.parametrize("kw", [dict(eig_solver=1), dict(gram_mode=1)])
def test_wide_context_takes_no_scratch_that_it_cannot_use(gpu, kw):
    """The Jacobi solver and the FP32 Gram mode run the wide kernel: no Gram matrices, no rotation log."""
    p = dict(vol_size=(16, 16, 16), nq=100, block_size=(4, 4, 4), prox_mode=1, lam=0.1)
    with ReconContext(ReconParams(**p)) as a, ReconContext(ReconParams(**p, **kw)) as b:
        assert a.device_bytes() - b.device_bytes() >= 64 * 5050 * 8


@pytest.mark.parametrize("n", [64, 65, 128])
def test_zero_threshold_is_the_identity(gpu, n):
    """A soft threshold of zero keeps every component: the matrices come back bit for bit, rank-deficient and not finite
    ones too, on both sides of the kernels' limit."""
    m, batch = 72, 5
    x = _low_rank_mats(np.random.default_rng(n), m, n, 5, batch, 0.0)
    x[0, 1, 2] = np.nan
    d = DeviceBuffer.from_array(x)
    L.check(L.lib.llr_soft_threshold_batch_dev(m, n, 0.0, batch, d.ptr, None))
    got = d.download(np.empty_like(x, order="F"))
    d.close()
    np.testing.assert_array_equal(got, x)


def test_zero_threshold_with_overlapping_blocks(gpu):
    """The mean over the tilings of an identity is the image itself, to the rounding of the scaled sum of eight."""
    rng = np.random.default_rng(4)
    vol, nq = (8, 16, 8), 66
    y = crandn(rng, vol + (nq,)) * (rng.random((1,) + vol[1:] + (nq,)) < 0.5)
    p = ReconParams(vol_size=vol, nq=nq, block_size=(4, 4, 4), block_stride=(2, 2, 2), lam=0.0, seed=1,
                    prox_mode=L.LLR_PROX_SOFT_THRESH)
    with ReconContext(p) as ctx:
        ctx.upload_kspace(np.asfortranarray(y.astype(np.complex64)))
        ctx.init_zero_filled()
        x0 = ctx.download_image()
        ctx.iterate(1)
        x1 = ctx.download_image()
    assert rel_err(x1, x0) < 2e-6
