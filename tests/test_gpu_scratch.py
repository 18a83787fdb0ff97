"""The operators' scratch pool: what it keeps between calls is given back on request."""
import numpy as np
import pytest

from conftest import crandn

from llr_b200 import DeviceBuffer, _lib as L

pytestmark = pytest.mark.gpu


def test_kept_scratch_is_given_back(gpu):
    """A batch of 8192 matrices of 61 columns leaves its Gram scratch (124 MB) mapped; freeing a null pointer releases
    it, and the next call works as before."""
    import torch
    m, n, batch = 8, 61, 8192
    x = crandn(np.random.default_rng(0), (m, n, batch))
    d = DeviceBuffer.from_array(np.asfortranarray(x))
    L.check(L.lib.llr_device_free(None))
    free0 = torch.cuda.mem_get_info()[0]
    L.check(L.lib.llr_soft_threshold_batch_dev(m, n, 1.0, batch, d.ptr, None))
    L.check(L.lib.llr_stream_sync(None))
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert 100 << 20 < kept <= 288 << 20
    L.check(L.lib.llr_device_free(None))
    assert free0 - torch.cuda.mem_get_info()[0] < 40 << 20
    L.check(L.lib.llr_soft_threshold_batch_dev(m, n, 1.0, batch, d.ptr, None))
    L.check(L.lib.llr_stream_sync(None))
    d.close()


def test_calls_of_different_sizes_on_two_threads(gpu):
    """Two threads launch the same kernels with different amounts of shared memory: the DTI fit with 1600 and 2000
    directions (51 and 64 KB of weights) and the batched prox with 512 and 64 rows.  A limit set to one call's size made
    the other thread's launch fail."""
    import threading
    errors = []

    def work(nq, m):
        rng = np.random.default_rng(nq)
        g = rng.standard_normal((nq, 3)).astype(np.float32)
        g /= np.linalg.norm(g, axis=1, keepdims=True)
        b = np.full(nq, 1000.0, np.float32)
        d = DeviceBuffer.from_array(np.asfortranarray(np.full((64, nq), 0.5, np.complex64)))
        s0 = DeviceBuffer.from_array(np.ones((64, 1), np.complex64))
        out = DeviceBuffer(4 * 7 * 64)
        x = DeviceBuffer.from_array(np.asfortranarray(crandn(rng, (m, 61, 4))))
        try:
            for _ in range(300):
                L.check(L.lib.llr_dti_fit_dev(d.ptr, nq, s0.ptr, 1, 64, L.fptr(b), L.fptr(g), out.ptr, None))
                L.check(L.lib.llr_soft_threshold_batch_dev(m, 61, 0.1, 4, x.ptr, None))
            L.check(L.lib.llr_stream_sync(None))
        except L.LlrError as e:
            errors.append(str(e))
        for v in (d, s0, out, x):
            v.close()

    threads = [threading.Thread(target=work, args=a) for a in ((1600, 512), (2000, 64))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
