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
