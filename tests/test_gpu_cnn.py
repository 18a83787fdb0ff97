"""GPU checks of the learned warm start's own kernels: conv3d forward, backward (weight,
bias and input gradients through the whole residual network), subspace channel packing,
and Adam training, against the FP64 CNN oracle with the same BF16-rounded weights."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import cnn_oracle as CO

pytestmark = pytest.mark.gpu

CH = (14, 32, 32, 32, 32, 32, 32, 32, 14)


def _net(seed=1):
    from llr_b200.cnn import Cnn
    return Cnn(CH, seed=seed)


def test_forward_matches_oracle(gpu):
    rng = np.random.default_rng(5)
    x = rng.standard_normal((7, 6, 5, 14)).astype(np.float32)      # (nz, ny, nx, C), ragged tiles
    with _net() as net:
        p = net.params
        p[CO.layer_slices(CH)[0][0][1]:][:32] = rng.standard_normal(32) * 0.1   # non-zero biases
        net.params = p
        got = net.forward(x)
    exp, _ = CO.forward(p, CH, x.astype(np.float64))
    assert rel_err(got, exp) < 1e-5
    assert rel_err(got - x, exp - x) < 1e-4


@pytest.mark.parametrize("dims", [(1, 16, 8), (2, 17, 9), (3, 1, 1), (40, 205, 101), (97, 33, 7)])
def test_forward_runs_and_edges(gpu, dims):
    """One plane and two, a single voxel per plane, columns cut by the volume's edge, several runs per CTA with more
    output planes than tensor memory holds at once.  Large volumes are checked on crops (the network reaches
    8 voxels).  BF16 weights are exact on both sides, activations carry 24 bits: 1e-4 of the residual, as
    above, and the rounding of the sum with the input, which a thin volume's small residual lets show."""
    rng = np.random.default_rng(8)
    x = rng.standard_normal(dims + (14,)).astype(np.float32)
    with _net(seed=3) as net:
        p = net.params
        w0, b0 = CO.layer_slices(CH)[0][-1]                     # a last layer as large as the others: residual of order x
        p[w0:b0] = rng.standard_normal(b0 - w0) * np.sqrt(2 / (27 * CH[-2]))
        net.params = p
        got = net.forward(x)
    ny, nx = dims[1:]
    for y0, x0 in {(0, 0), (ny // 2, nx // 2), (max(ny - 4, 0), max(nx - 4, 0))}:
        y1, x1 = min(y0 + 4, ny), min(x0 + 4, nx)
        ya, xa = max(y0 - 8, 0), max(x0 - 8, 0)
        exp, _ = CO.forward(p, CH, x[:, ya:y1 + 8, xa:x1 + 8].astype(np.float64))
        exp = exp[:, y0 - ya:y1 - ya, x0 - xa:x1 - xa]
        res = np.linalg.norm(exp - x[:, y0:y1, x0:x1])
        assert np.linalg.norm(got[:, y0:y1, x0:x1] - exp) <= 1e-4 * res + 2.0 ** -24 * np.linalg.norm(exp)


@pytest.mark.parametrize("dims", [(1, 17, 9), (2, 5, 8), (3, 16, 16), (11, 18, 11)])
def test_forward_sums_of_one_sign(gpu, dims):
    """Positive activations and weights: every addition in tensor memory truncates in the same direction.  The high BF16
    parts take 27 additions in the first layer and 54 in the three others, a unit of 2^-23 of a sum that grows steadily
    at most and half of that on average: 189 x 2^-23 / 2 / 2 = 5.6e-6; the low parts' own sums lose 2^-8 of that.  7e-6
    (with one sum for all parts, three times as many additions: 1.2e-5)."""
    from llr_b200.cnn import Cnn
    rng = np.random.default_rng(11)
    ch = (14, 32, 32, 32, 14)
    x = rng.uniform(0.5, 1.0, dims + (14,)).astype(np.float32)
    with Cnn(ch, seed=2) as net:
        p = np.zeros(net.n_params, np.float32)
        for w0, b0 in CO.layer_slices(ch)[0]:
            p[w0:b0] = rng.uniform(0.0, 0.1, b0 - w0)
        net.params = p
        got = net.forward(x)
    exp, _ = CO.forward(p, ch, x.astype(np.float64))
    assert rel_err(got, exp) < 7e-6


@pytest.mark.parametrize("dims", [(4, 9, 10), (9, 8, 17)])
def test_gradients_match_oracle(gpu, dims):
    """dL/dW and dL/db of every layer for L = mean |out - target|^2."""
    from llr_b200.cnn import DeviceArray
    rng = np.random.default_rng(6)
    x = rng.standard_normal(dims + (14,)).astype(np.float32)
    t = rng.standard_normal(dims + (14,)).astype(np.float32)
    with _net(seed=2) as net:
        p = net.params
        dx, dt = DeviceArray.from_numpy(x), DeviceArray.from_numpy(t)
        loss = net.loss_grad_dev(dx, dt)
        g = net.grads
    el, eg = CO.loss_and_grads(p, CH, x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - el) <= 1e-5 * el
    for (w0, b0), co in zip(CO.layer_slices(CH)[0], CH[1:]):
        assert rel_err(g[w0:b0], eg[w0:b0]) < 1e-4
        assert rel_err(g[b0:b0 + co], eg[b0:b0 + co]) < 1e-4


def test_subspace_channels_and_image_match_oracle(gpu):
    import llr_b200
    from llr_b200 import DeviceBuffer
    from llr_b200.cnn import DeviceArray, subspace_channels_dev, subspace_image_dev
    rng = np.random.default_rng(7)
    vol, nq, r = (5, 6, 7), 11, 7
    S, _ = np.linalg.qr(rng.standard_normal((nq, r)) + 1j * rng.standard_normal((nq, r)))
    S = S.astype(np.complex64)
    x = (rng.standard_normal(vol + (nq,)) + 1j * rng.standard_normal(vol + (nq,))).astype(np.complex64)
    dx, dS = DeviceBuffer.from_array(x), DeviceBuffer.from_array(np.asfortranarray(S))
    ch = DeviceArray((vol[2], vol[1], vol[0], 2 * r))
    subspace_channels_dev(dx.ptr, vol, nq, dS.ptr, r, 3.0, ch)
    llr_b200._lib.check(llr_b200._lib.lib.llr_stream_sync(None))
    got = ch.numpy()
    assert rel_err(got, CO.subspace_channels(x.astype(np.complex128), S.astype(np.complex128), 3.0)) < 1e-6
    dy = DeviceBuffer(x.nbytes)
    subspace_image_dev(ch, vol, nq, dS.ptr, r, 3.0, dy.ptr)
    back = dy.download(np.empty_like(x, order="F"))
    assert rel_err(back, CO.subspace_image(got.astype(np.float64), S.astype(np.complex128), 3.0)) < 1e-6
    # demodulated by the unit phase u of a reference image: channels of u* x, image u (c S^H)
    ref = (rng.standard_normal(vol + (nq,)) + 1j * rng.standard_normal(vol + (nq,))).astype(np.complex64)
    ref[0, 0, 0, 0] = 0                                           # a zero reference maps to u = 1
    u = np.where(ref == 0, 1.0, ref / np.maximum(np.abs(ref), 1e-30))
    dref = DeviceBuffer.from_array(ref)
    subspace_channels_dev(dx.ptr, vol, nq, dS.ptr, r, 3.0, ch, dref.ptr)
    llr_b200._lib.check(llr_b200._lib.lib.llr_stream_sync(None))
    gotp = ch.numpy()
    assert rel_err(gotp, CO.subspace_channels(np.conj(u) * x.astype(np.complex128), S.astype(np.complex128), 3.0)) < 1e-6
    subspace_image_dev(ch, vol, nq, dS.ptr, r, 3.0, dy.ptr, d_phase_ref=dref.ptr)
    backp = dy.download(np.empty_like(x, order="F"))
    assert rel_err(backp, u * CO.subspace_image(gotp.astype(np.float64), S.astype(np.complex128), 3.0)) < 1e-6


def _adam_oracle(p, x, t, steps, lr, b1=0.9, b2=0.999, eps=1e-8):
    """FP64 Adam on the oracle's gradients, FP32 master weights rounded to BF16 in use."""
    p = p.astype(np.float64)
    m = np.zeros_like(p)
    v = np.zeros_like(p)
    losses = []
    for k in range(1, steps + 1):
        loss, g = CO.loss_and_grads(p.astype(np.float32), CH, x, t)
        losses.append(loss)
        m = b1 * m + (1 - b1) * g
        v = b2 * v + (1 - b2) * g * g
        p = p - lr * (m / (1 - b1 ** k)) / (np.sqrt(v / (1 - b2 ** k)) + eps)
    return np.asarray(losses)


def test_adam_steps_match_oracle(gpu):
    """Five Adam steps on the GPU follow the oracle's loss trajectory."""
    from llr_b200.cnn import Cnn, DeviceArray
    rng = np.random.default_rng(8)
    x = rng.standard_normal((6, 8, 8, 14)).astype(np.float32)
    t = 0.5 * x
    with Cnn(CH, seed=12) as net:
        p0 = net.params
        dx, dt = DeviceArray.from_numpy(x), DeviceArray.from_numpy(t)
        got = np.asarray([net.train_step_dev(dx, dt, 2e-3) for _ in range(5)])
    exp = _adam_oracle(p0, x.astype(np.float64), t.astype(np.float64), 5, 2e-3)
    np.testing.assert_allclose(got, exp, rtol=2e-3)


def test_adam_training_reduces_loss(gpu):
    """Adam on the GPU kernels fits a damping map (target = 0.5 x: the residual branch must
    learn -0.5 x) on a 6 x 8 x 8 volume; the oracle reaches 1e-2 of the first loss in 50 steps."""
    from llr_b200.cnn import Cnn, DeviceArray
    rng = np.random.default_rng(8)
    x = rng.standard_normal((6, 8, 8, 14)).astype(np.float32)
    t = 0.5 * x
    with Cnn(CH, seed=12) as student:
        dx, dt = DeviceArray.from_numpy(x), DeviceArray.from_numpy(t)
        first = student.loss_grad_dev(dx, dt)
        for _ in range(100):
            last = student.train_step_dev(dx, dt, 2e-3)
    assert np.isfinite(last) and last < 0.05 * first, (first, last)


def test_learned_warm_start_gain(gpu):
    """Train on the GPU (own kernels) on adjoint -> converged pairs of 16 subjects that share
    one protocol, then start a held-out subject's recon from the network's image (the demodulated
    subspace part of the zero-filled image replaced by the network's prediction): it starts closer
    to the converged image than the zero-filled start and needs strictly fewer iterations to reach
    NRMSE <= 1e-2 and <= 1e-3 (fixed partition, shared by both)."""
    from llr_b200 import warmstart as W
    from llr_b200.cnn import Cnn
    proto = W.Protocol(vol=(36, 36, 36), centre=9)      # 6^3 blocks tile the volume exactly
    codec = W.SubspaceCodec(proto)
    pairs = W.training_pairs(proto, codec, list(range(200, 216)), 400)
    with Cnn(seed=5) as net:
        losses = W.train(net, pairs, epochs=30, lr=1e-3)
        assert losses[-1] < 0.8 * losses[0]
        d = proto.subject(977)
        x_zf, x_ref, lam, energy, snap = W.reference(proto, d.y, 1600, snapshot=True)
        x0, ms = W.warm_start_image(net, codec, x_zf, energy, d.y)
    e_zf, e_ws = W.nrmse(x_zf, x_ref), W.nrmse(x0, x_ref)
    assert e_ws < e_zf, (e_ws, e_zf)
    plain, cp = W.time_to_targets(proto, d.y, lam, x_zf, snap, [1e-2, 1e-3], 300)
    learned, cl = W.time_to_targets(proto, d.y, lam, x0, snap, [1e-2, 1e-3], 300)
    snap.close()
    assert abs(cp[0][1] - e_zf) < 1e-4 and abs(cl[0][1] - e_ws) < 1e-4   # device distance = host NRMSE
    for t in (1e-2, 1e-3):
        assert plain[t] is not None and learned[t] is not None, (t, plain, learned)
        assert learned[t][0] < plain[t][0], (t, learned, plain)


@pytest.mark.parametrize("dims", [(41, 50, 40), (37, 33, 41), (75, 17, 9)])
def test_gradients_with_several_tiles_per_cta(gpu, dims):
    """Odd and even numbers of 8 x 16 x 1 tiles per CTA, ragged in x and y, in both passes of the convolution and in the
    weight gradient: every layer against the oracle.  FP32 sums over up to 82 k voxels of activations whose own error is
    4e-6 (through BF16-exact weights): relative 1e-4 for each layer's weights and biases.  Inputs, weights and biases are
    positive: an activation that rounds across zero would switch its ReLU, which alone moves the first layer's gradient
    by up to 1e-3 at these sizes."""
    from llr_b200.cnn import Cnn, DeviceArray
    rng = np.random.default_rng(dims[0])
    ch = (14, 32, 32, 14)
    x = rng.uniform(0.2, 1.0, dims + (14,)).astype(np.float32)
    t = rng.standard_normal(x.shape).astype(np.float32)
    with Cnn(ch, seed=2) as net:
        p = rng.uniform(0.0, 0.01, net.n_params).astype(np.float32)
        net.params = p
        dx, dt = DeviceArray.from_numpy(x), DeviceArray.from_numpy(t)
        net.loss_grad_dev(dx, dt)
        got = net.grads
        dx.close()
        dt.close()
    _, exp = CO.loss_and_grads(p, ch, x.astype(np.float64), t.astype(np.float64))
    sl, total = CO.layer_slices(ch)
    edges = [e for s in sl for e in s] + [total]
    for a, b in zip(edges[:-1], edges[1:]):
        assert rel_err(got[a:b], exp[a:b]) < 1e-4, (a, b)


def test_weight_gradient_error_does_not_grow_with_the_volume(gpu):
    """Positive activations and output gradients: every product of the weight gradient has the same sign, so what the
    running sums lose to truncation adds up.  120000 single-voxel planes are 811 tiles per CTA.  A sum over 64 tiles, six
    products each, loses at most 64 x 6 x 2^-23 / 2 = 2.3e-5, the activations of the layer below 1e-5 in the same way: 4e-5
    (a sum over all the CTA's tiles was 1.6e-4 short)."""
    from llr_b200.cnn import Cnn, DeviceArray
    rng = np.random.default_rng(4)
    ch, nz = (14, 32, 14), 120000
    x = rng.uniform(0.5, 1.0, (nz, 1, 1, 14)).astype(np.float32)
    t = np.full_like(x, -3.0)
    with Cnn(ch, seed=2) as net:
        p = np.zeros(net.n_params, np.float32)
        (w0, b0), (w1, b1) = CO.layer_slices(ch)[0]
        p[w0:b0] = rng.uniform(0.0, 0.1, b0 - w0)
        p[w1:b1] = rng.uniform(0.0, 0.1, b1 - w1)
        net.params = p
        dx, dt = DeviceArray.from_numpy(x), DeviceArray.from_numpy(t)
        net.loss_grad_dev(dx, dt)
        got = net.grads
        dx.close()
        dt.close()
    _, exp = CO.loss_and_grads(p, ch, x.astype(np.float64), t.astype(np.float64))
    assert rel_err(got[w1:b1], exp[w1:b1]) < 4e-5
    assert rel_err(got[w0:b0], exp[w0:b0]) < 4e-5
