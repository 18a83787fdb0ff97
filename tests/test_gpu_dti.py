"""DTI scalar maps on the GPU (llr_dti_fit, llr-dti-scalars) against the FP64 oracle
(diffusion_models.rs:21-129)."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, rel_err
from oracle import llr_oracle as O

pytestmark = pytest.mark.gpu


def _fit(dwi, b0, b, g):
    from llr_b200 import _lib as L
    V, nq = dwi.shape
    nb0 = b0.shape[1]
    out = np.empty((7, V), dtype=np.float32)
    dwi = np.asfortranarray(dwi.astype(np.complex64))
    b0 = np.asfortranarray(b0.astype(np.complex64))
    bb = np.ascontiguousarray(b, dtype=np.float32)
    gg = np.ascontiguousarray(g, dtype=np.float32)
    L.check(L.lib.llr_dti_fit(L.ptr(dwi), nq, L.ptr(b0) if nb0 else None, nb0, V, L.fptr(bb), L.fptr(gg), L.fptr(out)))
    return dict(zip(["b0av", "e1", "e2", "e3", "md", "rd", "fa"], out))


def test_dti_fit_matches_oracle_on_phantom(gpu):
    from llr_b200.phantom import make_dataset
    d = make_dataset((20, 20, 10), [(0, 3), (1000, 30), (2000, 30)], 2.0, 4, centre=4)
    x = d.x_true.reshape(-1, d.x_true.shape[3], order="F")
    rng = np.random.default_rng(1)
    x = x + 0.01 * (rng.standard_normal(x.shape) + 1j * rng.standard_normal(x.shape))
    dwi, b0 = x[:, d.b > 0], x[:, d.b == 0]
    got = _fit(dwi, b0, d.b[d.b > 0], d.g[d.b > 0])
    exp = O.dti_fit(dwi.astype(np.complex64).astype(np.complex128), b0.astype(np.complex64).astype(np.complex128),
                    d.b[d.b > 0], d.g[d.b > 0])
    for k in ("b0av", "e1", "e2", "e3", "md", "rd"):
        assert rel_err(got[k], exp[k]) < 1e-4, k
    ok = np.isfinite(exp["fa"])
    assert np.array_equal(np.isfinite(got["fa"]), ok)
    assert np.max(np.abs(got["fa"][ok] - exp["fa"][ok])) < 1e-3


def test_dti_fit_noise_free_tensor(gpu):
    from llr_b200.phantom import b_table, eigenvector_matrix, sample_unit_sphere, tensor_signal
    rng = np.random.default_rng(2)
    b, g = b_table([(0, 2), (1000, 15), (2000, 15)], rng)
    R = eigenvector_matrix(sample_unit_sphere(0.3, 0.7))
    D = R @ np.diag([1.7e-3, 0.5e-3, 0.3e-3]) @ R.T
    s = tensor_signal(np.array([0.8, 0.0]), np.stack([D, D]), b, g)     # second voxel: zero signal
    got = _fit(s[:, b > 0], s[:, b == 0], b[b > 0], g[b > 0])
    np.testing.assert_allclose([got["e1"][0], got["e2"][0], got["e3"][0]], [1.7e-3, 0.5e-3, 0.3e-3], rtol=2e-4)
    assert got["b0av"][1] == 0.0


def test_dti_scalars_cli(gpu, tmp_path):
    from llr_b200.cfl import read_cfl, write_cfl
    from llr_b200.phantom import make_dataset
    exe = os.path.join(PKG, "llr-dti-scalars")
    d = make_dataset((12, 10, 8), [(0, 2), (1000, 12)], 2.0, 5, centre=4)
    n = d.x_true.shape[3]
    for q in range(n):
        write_cfl(str(tmp_path / f"v{q:02d}"), d.x_true[..., q])
    with open(tmp_path / "bt.txt", "w") as f:
        for bv, gv in zip(d.b, d.g):
            f.write(f"{bv:g} {gv[0]:.9f} {gv[1]:.9f} {gv[2]:.9f}\n")
    out = tmp_path / "maps"
    out.mkdir()
    r = subprocess.run([exe, str(tmp_path), "v*", str(tmp_path / "bt"), str(out), str(n)], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    x = d.x_true.reshape(-1, n, order="F")
    exp = _fit(x[:, d.b > 0], x[:, d.b == 0], d.b[d.b > 0], d.g[d.b > 0])
    for k in ("b0av", "e1", "md", "fa"):
        m = read_cfl(str(out / k)).reshape(-1, order="F")
        assert np.all(m.imag == 0)
        np.testing.assert_allclose(m.real, exp[k], rtol=1e-6)   # the b-table went through text


@pytest.mark.parametrize("V,nq,scale", [(1, 6, 1.0), (255, 7, 1.0), (513, 8, 1e-18), (1025, 17, 1e18)])
def test_dti_fit_edges_and_extreme_scales(gpu, V, nq, scale):
    """Voxel counts around the two-voxel split, sample counts around the eight-sample batch, and signals
    whose squares leave the FP32 range (the ratio is formed without squares there).  Tolerance: the
    logarithm's argument carries a few FP32 roundings (5e-7), amplified by the fit's conditioning (the
    phantom test's 1e-4)."""
    rng = np.random.default_rng(V)
    g = rng.standard_normal((nq, 3))
    g /= np.linalg.norm(g, axis=1, keepdims=True)
    b = np.full(nq, 1000.0)
    s0 = rng.uniform(0.5, 1.0, (V, 2))
    lam = rng.uniform(0.2e-3, 2e-3, (V, nq))
    dwi = s0[:, :1] * np.exp(-1000.0 * lam) * np.exp(1j * rng.uniform(0, 6, (V, nq))) * scale
    dwi, b0 = dwi.astype(np.complex64), (s0 * scale).astype(np.complex64)
    got = _fit(dwi, b0, b, g)
    exp = O.dti_fit(dwi.astype(np.complex128), b0.astype(np.complex128), b, g)
    for k in ("b0av", "e1", "e2", "e3", "md", "rd"):
        assert rel_err(got[k], exp[k]) < 1e-4, k


def _masked(V, nq, nb0, rng):
    """Background of exact zeros in runs of 24 voxels, and single zero samples inside."""
    g = rng.standard_normal((nq, 3))
    g /= np.linalg.norm(g, axis=1, keepdims=True)
    s0 = rng.uniform(0.5, 1.0, (V, 1)) * np.ones((1, nb0))
    dwi = s0[:, :1] * np.exp(-1000.0 * rng.uniform(0.2e-3, 2e-3, (V, nq))) * np.exp(1j * rng.uniform(0, 6, (V, nq)))
    out = (np.arange(V) // 24) % 2 == 0
    dwi[out] = 0
    s0[out] = 0
    dwi[rng.random((V, nq)) < 0.01] = 0
    return dwi.astype(np.complex64), s0.astype(np.complex64), np.full(nq, 1000.0), g


def test_dti_fit_zero_samples_match_oracle(gpu):
    """Exact zeros clamp to the smallest normal number, in voxels with signal and in the background, where b0 is zero
    too.  The logarithm of that number is exact to a few roundings: the phantom test's 1e-4."""
    rng = np.random.default_rng(6)
    dwi, b0, b, g = _masked(1500, 19, 2, rng)
    got = _fit(dwi, b0, b, g)
    exp = O.dti_fit(dwi.astype(np.complex128), b0.astype(np.complex128), b, g)
    for k in ("b0av", "e1", "e2", "e3", "md", "rd"):
        assert rel_err(got[k], exp[k]) < 1e-4, k


def test_dti_fit_masked_volume_is_not_slower(gpu):
    """A volume that is half background of exact zeros against one without any: each batch with a zero formed its ratios
    one by one, 3.3 times as long."""
    import time
    from llr_b200 import DeviceBuffer, _lib as L
    rng = np.random.default_rng(7)
    V, nq = 1 << 20, 48
    _, _, b, g = _masked(8, nq, 1, rng)
    bb, gg = np.ascontiguousarray(b, np.float32), np.ascontiguousarray(g, np.float32)
    x = np.full((V, nq), 0.5, np.complex64, order="F")
    s0 = np.ones((V, 1), np.complex64, order="F")
    out = DeviceBuffer(4 * 7 * V)
    us = []
    for mask in (False, True):
        if mask:
            x[(np.arange(V) // 96) % 2 == 0] = 0
            s0[(np.arange(V) // 96) % 2 == 0] = 0
        dx, db = DeviceBuffer.from_array(x), DeviceBuffer.from_array(s0)
        best = 1.0
        for _ in range(10):
            L.check(L.lib.llr_stream_sync(None))
            t0 = time.perf_counter()
            L.check(L.lib.llr_dti_fit_dev(dx.ptr, nq, db.ptr, 1, V, L.fptr(bb), L.fptr(gg), out.ptr, None))
            L.check(L.lib.llr_stream_sync(None))
            best = min(best, time.perf_counter() - t0)
        us.append(best)
        dx.close()
        db.close()
    out.close()
    assert us[1] < 1.5 * us[0]


def test_dti_fit_infinite_reference(gpu):
    """With an infinite b0 every ratio clamps to the smallest normal number, finite / infinite and infinite / infinite
    alike (the maximum of NaN and a number is the number), so the maps are those of zero samples."""
    rng = np.random.default_rng(9)
    _, _, b, g = _masked(8, 16, 1, rng)
    V = 1024
    b0 = np.full((V, 1), np.inf, np.complex64)
    got = [_fit(np.full((V, 16), v, np.complex64), b0, b, g) for v in (0.0, 1.0, np.inf)]
    for k in ("e1", "e2", "e3", "md"):
        assert np.isfinite(got[0][k]).all()
        np.testing.assert_allclose(got[1][k], got[0][k], rtol=1e-4, atol=1e-6 * np.abs(got[0]["e1"]).max())
        np.testing.assert_allclose(got[2][k], got[0][k], rtol=1e-4, atol=1e-6 * np.abs(got[0]["e1"]).max())
