"""The memory-bound passes of a training step (im2col, max-pool gradient, batch normalisation, dropout)
at ragged sizes, unaligned starts and both types (GPU tests against the CPU oracle)."""
import numpy as np
import pytest

from gorgonia_b200.engine import Tensor
from oracle import oracle
from tests import util
from tests.util import assert_bits_equal, assert_gemm_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("case", [
    # B, C, H, W, kernel, pad, stride, dil
    (2, 1, 5, 5, (3, 3), (1, 1), (1, 1), (1, 1)), (3, 4, 7, 6, (2, 5), (0, 2), (1, 1), (1, 1)),
    (2, 33, 9, 3, (1, 1), (0, 0), (1, 1), (1, 1)), (1, 8, 12, 13, (3, 3), (2, 2), (2, 3), (2, 1)),
    (5, 32, 14, 14, (3, 3), (1, 1), (1, 1), (1, 1)), (1, 300, 4, 4, (3, 3), (1, 1), (1, 1), (1, 1))])
def test_im2col_pieces(fresh, case, dt):
    e = fresh
    B, C, H, W, k, pad, stride, dil = case
    x = util.normal(5, (B, C, H, W), dt)
    Ho = (H + 2 * pad[0] - (dil[0] * (k[0] - 1) + 1)) // stride[0] + 1
    Wo = (W + 2 * pad[1] - (dil[1] * (k[1] - 1) + 1)) // stride[1] + 1
    p = np.zeros((B, C, H + 2 * pad[0], W + 2 * pad[1]), dt)
    p[:, :, pad[0]:pad[0] + H, pad[1]:pad[1] + W] = x
    want = np.empty((B, Ho, Wo, C, k[0], k[1]), dt)
    for r in range(k[0]):
        for s in range(k[1]):
            want[..., r, s] = p[:, :, r * dil[0]:r * dil[0] + (Ho - 1) * stride[0] + 1:stride[0],
                                s * dil[1]:s * dil[1] + (Wo - 1) * stride[1] + 1:stride[1]].transpose(0, 2, 3, 1)
    col = e.empty((B, Ho, Wo, C * k[0] * k[1]), dt)
    e.Im2Col(e.tensor(x), col, k, pad, stride, dil)
    assert_bits_equal(col.numpy(), want.reshape(col.shape))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("case", [
    # few images: rows cut into runs of positions, and the channels of a row shared between blocks
    (1, 3, 224, 224, (3, 3), (1, 1), (1, 1), (1, 1)), (1, 1, 3, 1001, (1, 3), (0, 1), (1, 2), (1, 3)),
    (1, 256, 13, 13, (3, 3), (1, 1), (1, 1), (1, 1)), (1, 40, 1, 9, (1, 2), (0, 0), (1, 1), (1, 1)),
    (2, 5, 31, 47, (3, 3), (2, 2), (2, 2), (1, 2))])
def test_im2col_few_images(fresh, case, dt):
    test_im2col_pieces(fresh, case, dt)


@pytest.mark.parametrize("shape", [(1, 1, 2, 2), (3, 5, 14, 14), (2, 7, 13, 6), (2, 3, 9, 8), (100, 64, 14, 14)])
def test_maxpool2x2_gradient(fresh, shape):
    e = fresh
    B, C, H, W = shape
    x = util.normal(7, shape)
    y, mask, dx = e.empty((B, C, H // 2, W // 2)), e.empty((B, C, H // 2, W // 2), np.int64), e.empty(shape)
    e.MaxPool2D(e.tensor(x), y, (2, 2), (0, 0), (2, 2), mask=mask)
    dy = util.normal(8, y.shape)
    dy.flat[0] = -0.0
    e.MaxPool2DDiff(e.tensor(dy), mask, dx, (2, 2), (0, 0), (2, 2))
    assert_bits_equal(dx.numpy(), oracle.maxpool2d_bwd(dy, mask.numpy(), shape))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(2, 1, 1, 1), (3, 5, 2, 2), (130, 3, 7, 7), (17, 20, 5, 4), (128, 64, 28, 28), (2, 2, 50, 50),
                                   (9, 700)])
def test_batchnorm_groups(fresh, shape, dt):
    e = fresh
    C = shape[1]
    x, dy = util.normal(9, shape, dt, 2.0) + dt(0.5), util.normal(10, shape, dt)
    rm, rv = e.tensor(np.zeros(C, dt)), e.tensor(np.ones(C, dt))
    sm, sv, y, dx = e.empty((C,), dt), e.empty((C,), dt), e.empty(shape, dt), e.empty(shape, dt)
    for training in (True, False, True):        # twice in training: the arrival counters must be back at zero
        rm.set(np.zeros(C, dt))
        rv.set(np.ones(C, dt))
        e.BatchNorm(e.tensor(x), y, rm, rv, sm, sv, training=training)
        wm, wv = np.zeros(C, dt), np.ones(C, dt)
        out = oracle.batchnorm(x, wm, wv, training=training)
        # the oracle sums in the tensor's own type: n additions of rounding error against double sums here
        n = x.size // C
        rel = max(2e-5 if dt == np.float32 else 1e-12, n * np.finfo(dt).eps * 0.05)
        assert_gemm_close(y.numpy(), out[0], rel)
        if training:
            e.BatchNormDiff(e.tensor(x), e.tensor(dy), dx, rv, sm, sv, training=True)
            want = oracle.batchnorm_bwd(x, dy, wv, sm.numpy(), sv.numpy(), training=True)
            if n > 2:       # two samples cancel to rounding noise
                assert_gemm_close(dx.numpy(), want, 10 * rel)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 100_001])
@pytest.mark.parametrize("start", [0, 1])
def test_dropout_pieces(fresh, n, dt, start):
    e = fresh
    whole = [util.normal(11, n + start, dt), util.uniform(12, (n + start,)).astype(dt), util.normal(13, n + start, dt)]
    size = np.dtype(dt).itemsize
    x, r, dy = (Tensor(e, e.tensor(a).ptr + start * size, (n,), dt, owned=False) for a in whole)
    y, dx = (Tensor(e, e.empty((n + start,), dt).ptr + start * size, (n,), dt, owned=False) for _ in range(2))
    for uniforms in (r, None):
        e.Dropout(x, y, 0.3, uniforms=uniforms, seed=5, offset=2)
        want = oracle.dropout(whole[0][start:], 0.3, uniforms=whole[1][start:] if uniforms else None, seed=5, offset=2)
        assert_bits_equal(y.numpy(), want)
        e.DropoutDiff(dy, y, dx, 0.3)
        assert_bits_equal(dx.numpy(), oracle.dropout_bwd(whole[2][start:], want, 0.3))
