"""Planes beyond shared memory: the row and column transforms (every length they can meet there is a product of two
factors of 8 to 16) and the k-space expansion of the subspace, with the path that ran read off the launches."""
import numpy as np
import pytest

from conftest import crandn, rel_err
from oracle import llr_oracle as O

from llr_b200 import ReconContext, ReconParams, _lib as L

pytestmark = pytest.mark.gpu


def _lines(rng, vol, nq):
    """Random data on 40 % of the lines, a volume without samples among them."""
    y = crandn(rng, vol + (nq,)) * (rng.random((1,) + vol[1:] + (nq,)) < 0.4)
    y[..., 1] = 0
    return np.asfortranarray(y.astype(np.complex64))


@pytest.mark.parametrize("ny,nz", [(256, 128), (117, 256), (240, 121), (140, 208), (144, 225), (169, 196), (112, 256),
                                   (165, 182), (256, 143), (256, 256)])
def test_row_and_column_lengths(gpu, ny, nz):
    """Register lengths 8 to 16 on both axes, ragged last tiles, against the cuFFT passes on the same data: one launch
    for data consistency there, three here.  FP32 transforms: relative 2e-6 for the zero-filled start, 6e-6 after three
    iterations; a residual of h inherits 2 x 6e-6 of sqrt(h) times the norm of the data."""
    vol, nq = (3, ny, nz), 4
    y = _lines(np.random.default_rng(ny + nz), vol, nq)
    out = {}
    for mode in (0, 1):
        p = ReconParams(vol_size=vol, nq=nq, block_size=(3, 4, 4), prox_mode=L.LLR_PROX_SOFT_THRESH, lam=0.3, seed=3,
                        fft_mode=mode)
        with ReconContext(p) as ctx:
            ctx.upload_kspace(y)
            ctx.init_zero_filled()
            x0 = ctx.download_image()
            h = np.asarray(ctx.iterate(3))
            out[mode] = (x0, ctx.download_image(), h, ctx.kernel_launches_per_iteration)
    assert out[0][3] == out[1][3] + 2
    assert rel_err(out[0][0], out[1][0]) < 2e-6
    assert rel_err(out[0][1], out[1][1]) < 6e-6
    assert (np.abs(out[0][2] - out[1][2]) < 12e-6 * np.sqrt(out[1][2]) * np.linalg.norm(y)).all()


@pytest.mark.parametrize("vol,bs,nq,srank,corr", [((8, 256, 128), (4, 8, 8), 9, 1, None), ((8, 144, 224), (8, 8, 8), 21, 7, "shared"),
                                                  ((8, 176, 169), (4, 11, 13), 19, 16, "shared"),
                                                  ((8, 256, 256), (8, 8, 8), 13, 7, None),
                                                  ((8, 196, 150), (4, 7, 5), 11, 5, "own")])
def test_kspace_expansion_matches_oracle(gpu, vol, bs, nq, srank, corr):
    """Coefficient-domain iterations whose image is expanded row by row in k-space (shared phases), ranks 1 to 16 and odd
    volume counts; volumes with phases of their own are expanded in the image and take the same row kernels.  Against the
    oracle (2e-4, the reconstruction tolerance) and the cuFFT passes (1e-5)."""
    rng = np.random.default_rng(vol[1] + srank)
    y = _lines(rng, vol, nq)
    S = np.asfortranarray(np.linalg.qr(crandn(rng, (nq, srank), np.complex128))[0].astype(np.complex64))
    lk = None
    if corr:
        lk = (np.tile([[1.0, -2.0, 1.0]], (nq, 1)) if corr == "shared" else rng.integers(-2, 3, (nq, 3))).astype(np.float32)
    ocfg = O.ReconConfig(block_size=bs, mode="soft", seed=5, wavelet_alpha=0.003, wavelet_moments=2, wavelet_levels=1,
                         wavelet_space="coeffs", lin_ksp=lk)
    ocfg.subspace = S.astype(np.complex128)
    x0 = O.zero_filled(y.astype(np.complex128), ocfg)
    ocfg.lam = 0.05 * O.sigma_max(x0, bs)
    out = {}
    for mode in (0, 1):
        p = ReconParams(vol_size=vol, nq=nq, block_size=bs, lam=ocfg.lam, seed=5, subspace_rank=srank, wavelet_space=1,
                        prox_mode=L.LLR_PROX_SOFT_THRESH, fft_mode=mode)
        p.wavelet_alpha, p.wavelet_moments, p.wavelet_levels = 0.003, 2, 1
        with ReconContext(p) as ctx:
            if corr:
                ctx.set_linear_corrections(lk, None)
            ctx.upload_kspace(y)
            ctx.upload_subspace(S)
            ctx.init_zero_filled()
            h = ctx.iterate(2)
            out[mode] = (ctx.download_image(), h, ctx.kernel_launches_per_iteration)
    # three transform launches for one of data consistency, and no expansion launch where k-space holds it
    assert out[0][2] == out[1][2] + (2 if corr == "own" else 1)
    assert rel_err(out[0][0], out[1][0]) < 1e-5
    ox, oh = O.recon(y.astype(np.complex128), ocfg, 2, x0=x0)
    assert rel_err(out[0][0], ox) < 2e-4
    np.testing.assert_allclose(out[0][1], oh, rtol=2e-4)


@pytest.mark.parametrize("ny,nz", [(16, 12), (256, 128)])
def test_coefficient_volumes_of_more_than_64_stay_refused(gpu, ny, nz):
    """The coefficient wavelet takes at most 64 volumes, on planes of either path."""
    rng = np.random.default_rng(3)
    vol, nq, srank = (8, ny, nz), 66, 4
    p = ReconParams(vol_size=vol, nq=nq, block_size=(4, 4, 4), lam=0.1, subspace_rank=srank, wavelet_space=1,
                    prox_mode=L.LLR_PROX_SOFT_THRESH)
    p.wavelet_alpha, p.wavelet_moments, p.wavelet_levels = 0.003, 2, 1
    with ReconContext(p) as ctx:
        ctx.upload_kspace(_lines(rng, vol, nq))
        ctx.upload_subspace(np.asfortranarray(np.linalg.qr(crandn(rng, (nq, srank)))[0].astype(np.complex64)))
        ctx.init_zero_filled()
        with pytest.raises(L.LlrError) as err:
            ctx.iterate(1)
    assert err.value.status == L.LLR_ERR_UNSUPPORTED
