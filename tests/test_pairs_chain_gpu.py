"""Convolutions on pairs of fp16: each kernel at the sizes where its tiles and rows meet, and whole chains whose
tensors do not fit fp16's range and have to come out as the TF32 chain makes them (GPU tests)."""
import numpy as np
import pytest

from gorgonia_b200 import B200Error, tapes
from oracle import oracle
from tests import util
from tests.util import assert_bits_equal, assert_gemm_close

pytestmark = pytest.mark.gpu


def _pairs(e, x):
    """x (B, C, H, W) in pairs form, made on the host, and its record."""
    amax = np.abs(x).max()
    exp = 14 - int(np.floor(np.log2(amax)))
    v = np.ascontiguousarray(x.transpose(0, 2, 3, 1)).astype(np.float64) * 2.0 ** exp
    h = v.astype(np.float16)
    l = ((v - h) * 2048).astype(np.float16)
    rec = np.array([np.float32(amax).view(np.int32), 0, 0, exp], np.int32)
    both = np.concatenate([h.ravel(), l.ravel()]).view(np.float32)
    return e.tensor(both), e.tensor(rec)


def _unpair(t, rec, shape):
    B, C, H, W = shape
    r = rec.numpy()
    v = t.numpy().view(np.float16).astype(np.float64).reshape(2, B, H, W, C)
    return ((v[0] + v[1] / 2048) * 2.0 ** -int(r[3])).transpose(0, 3, 1, 2), r


def _oracle(x, w, pad, bias, act, alpha, pool):
    y = oracle.conv2d(x, w, pad=pad)
    if bias is not None:
        y = (y + bias[None, :, None, None]).astype(np.float32)
    y = {"rectify": oracle.rectify, "leaky": lambda t: oracle.leaky_relu(t, alpha), None: lambda t: t}[act](y)
    return oracle.maxpool2d(y, (2, 2), (0, 0), (2, 2))[0] if pool else y


LINKS = [
    # B, C, H, W, K, kernel, pad, act, alpha, pool: the window kernel (32, 64 and 128-byte rows)
    (3, 16, 32, 32, 32, 3, 1, "leaky", 0.1, True), (2, 16, 48, 46, 24, 3, 1, None, 0.0, False),
    (4, 32, 28, 28, 64, 3, 1, "rectify", 0.0, True), (2, 32, 30, 32, 40, 5, 2, "leaky", 1.5, False),
    (2, 64, 16, 31, 72, 3, 1, "leaky", -0.5, False), (2, 64, 32, 32, 64, 3, 1, "leaky", -0.5, True),
    (9, 32, 14, 14, 64, 3, 1, "rectify", 0.0, True),
    # the im2col kernel (128 and 64-byte rows), k shared between blocks and not
    (5, 128, 13, 13, 256, 3, 1, "leaky", 0.1, False), (7, 96, 9, 11, 48, 3, 1, None, 0.0, False),
    (3, 128, 26, 26, 125, 1, 0, "leaky", 1.0, False), (40, 64, 7, 7, 128, 3, 1, "rectify", 0.0, False),
    (2, 512, 13, 13, 136, 3, 1, "leaky", 0.1, False), (30, 128, 26, 26, 512, 3, 0, "rectify", 0.0, False),
]


@pytest.mark.parametrize("case", LINKS)
@pytest.mark.parametrize("scale", [1.0, 3e-20])
def test_link(fresh, case, scale):
    e = fresh
    B, C, H, W, K, k, pad, act, alpha, pool = case
    if scale != 1.0 and B * C * K > 40000:
        pytest.skip("magnitudes are tried on the small links")
    x = (util.normal(41, (B, C, H, W)) * np.float32(scale)).astype(np.float32)
    w = util.normal(42, (K, C, k, k), scale=0.05)
    bias = (util.normal(43, K) * np.float32(scale)).astype(np.float32)
    want = _oracle(x, w, (pad, pad), bias, act, alpha, pool)
    tx, rx = _pairs(e, x)
    y, yp = e.empty(want.shape), e.empty((want.size,)) if K % 8 == 0 else None
    for _ in range(2):
        ry = e.tensor(np.zeros(4, np.int32))
        e.Conv2dPairs(None, e.tensor(w), y, x.shape, rx.ptr, ry.ptr, pad=(pad, pad), bias=e.tensor(bias), act=act,
                      alpha=alpha, pool2=pool, x_pairs=tx, y_pairs=yp)
    got = y.numpy()
    assert_gemm_close(got, want, 1e-5)
    if yp is not None:
        back, r = _unpair(yp, ry, want.shape)
        assert r[2] == 0 and np.int32(r[0]).view(np.float32) == np.abs(got).max()
        # heads and tails: 2^-22 of a value, or 2^-36 of the scaled range for the small ones
        assert (np.abs(back - got) <= 2.0 ** -22 * np.abs(got) + 2.0 ** (-36 - int(r[3]))).all()
        assert np.abs(back).max() * 2.0 ** int(r[3]) <= 65504


@pytest.mark.parametrize("C", [1, 2, 3])
def test_first_link_and_pool(fresh, C):
    e = fresh
    x, w, bias = util.uniform(51, (3, C, 28, 36)), util.normal(52, (16, C, 3, 3), scale=0.3), util.normal(53, 16)
    want = _oracle(x, w, (1, 1), bias, "leaky", 0.1, True)
    tx, recs = e.tensor(x), e.tensor(np.zeros(12, np.int32))
    e.pairs_magnitude(tx, recs.ptr)
    yp = e.empty((want.size,))
    e.Conv2dPairs(tx, e.tensor(w), None, x.shape, recs.ptr, recs.ptr + 16, pad=(1, 1), bias=e.tensor(bias), act="leaky",
                  alpha=0.1, pool2=True, y_pairs=yp)
    r1 = e.empty((4,), np.int32)
    r1.set(recs.numpy()[4:8])
    back, r = _unpair(yp, r1, want.shape)
    assert_gemm_close(back, want, 1e-6)
    # a pool in front of the next link, with gorgonia's explicit padding, and an odd number of channels
    z = util.normal(54, (2, 40, 13, 11))
    tz = e.tensor(z)
    rz = e.tensor(np.array([np.abs(z).max().view(np.int32), 0, 0, 0], np.int32))
    for kernel, pad, stride in (((2, 2), (1, 0, 1, 0), (1, 1)), ((2, 2), (0, 0), (2, 2)), ((3, 3), (1, 1), (2, 2))):
        p4 = pad if len(pad) == 4 else (pad[0], pad[0], pad[1], pad[1])
        Ho, Wo = (13 + p4[0] + p4[1] - kernel[0]) // stride[0] + 1, (11 + p4[2] + p4[3] - kernel[1]) // stride[1] + 1
        ref, got, rec = e.empty((2, 40, Ho, Wo)), e.empty((2 * 40 * Ho * Wo,)), e.tensor(np.zeros(4, np.int32))
        e.MaxPool2D(tz, ref, kernel, pad, stride)
        e.MaxPool2DPairs(tz, rz.ptr, got, rec.ptr, kernel, pad, stride)
        back, r = _unpair(got, rec, ref.shape)
        assert np.abs(back - ref.numpy()).max() <= 2.0 ** -22 * np.abs(z).max() and r[2] == 0


@pytest.mark.parametrize("constant", [False, True])
@pytest.mark.parametrize("case", [(32, 128, 26, 26, 256, 3, 1, 1), (128, 64, 32, 32, 64, 3, 1, 1), (32, 96, 40, 41, 250, 3, 2, 1),
                                  (48, 256, 13, 13, 256, 3, 1, 1)])
def test_single_convolutions(fresh, case, constant):
    # TF32 pairs, but the first case with constant filters: fp16 (the larger ones are further down); then values that
    # are out of fp16's range, which the TF32 launches behind it answer
    e = fresh
    B, C, H, W, K, k, stride, pad = case
    x, w, bias = util.normal(61, (B, C, H, W)), util.normal(62, (K, C, k, k), scale=0.05), util.normal(63, K)
    tx, tw, tb = e.tensor(x), e.tensor(w), e.tensor(bias)
    if constant:
        e.constant(tw)
    Ho, Wo = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    y = e.empty((B, K, Ho, Wo))

    def run():
        e.Conv2d(tx, tw, y, pad=(pad, pad), stride=(stride, stride), bias=tb, act="leaky", alpha=0.1)
        return y.numpy()

    def want(x):
        c = oracle.conv2d(x, w, pad=(pad, pad), stride=(stride, stride))
        return oracle.leaky_relu((c + bias[None, :, None, None]).astype(np.float32), 0.1)

    ref = want(x)
    assert_gemm_close(run(), ref, 1e-5)
    assert_gemm_close(run(), ref, 1e-5)
    wide = x.copy()
    wide[1] *= np.float32(1e-25)          # one image far below the others: exact in itself all the same
    wide[2, :, 3, 3] = np.float32(1e20)
    tx.set(wide)
    got, ref = run(), want(wide)
    for b in range(3):
        assert_gemm_close(got[b], ref[b], 1e-5)
    bad = x.copy()
    bad[0, 0, 0, 0], bad[3, 1, 5, 5] = np.inf, np.nan
    tx.set(bad)
    got, ref = run(), want(bad)
    assert np.isfinite(got).sum() == np.isfinite(ref).sum() and not np.isfinite(got[0]).all() and np.isfinite(got[1]).all()
    assert_gemm_close(got[1], ref[1], 1e-5)
    tx.set(x)                             # and back again
    assert_gemm_close(run(), want(x), 1e-5)


def _lenet(e, monkeypatch, flops, batch=40):
    monkeypatch.setattr(tapes._ConvChain, "PAIRS_FLOPS", flops)
    return tapes.LeNet(e, batch, seed=11)


def _yolo(e, monkeypatch, flops, batch=4):
    monkeypatch.setattr(tapes._ConvChain, "PAIRS_FLOPS", flops)
    m = tapes.TinyYolo(e, batch, seed=12, channels=(3, 16, 32, 64, 64, 128, 128, 256, 128, 24))
    for b in m.b:       # a bias would lift an image of 1e-25 into the others' range
        b.set(np.zeros(b.shape, np.float32))
    return m


@pytest.mark.parametrize("make", [_lenet, _yolo])
@pytest.mark.parametrize("kind", ["plain", "small", "large", "wide", "inf", "nan", "zero"])
def test_chains_against_tf32(fresh, monkeypatch, make, kind):
    e = fresh
    m16, m32 = make(e, monkeypatch, 0), make(e, monkeypatch, 1e30)
    assert m16.records is not None and m32.records is None
    x = util.uniform(71, m16.x.shape)
    x = {"small": lambda: x * np.float32(1e-12), "large": lambda: x * np.float32(1e12), "zero": lambda: x * 0,
         "wide": lambda: x * np.where(np.arange(len(x)) % 2, 1e-25, 1.0).astype(np.float32)[:, None, None, None]
         }.get(kind, lambda: x)()
    if kind in ("inf", "nan"):
        x[1, 0, 3, 3] = np.inf if kind == "inf" else np.nan
    out = []
    for m in (m16, m32):
        m.x.set(x)
        m.record()
        for _ in range(2):
            m.replay()
        out.append(m.out.numpy())
        redo = m.records.buf.numpy()[-4] if m.records is not None else None
        if m is m16:
            # what fp16's range is not enough for comes out as the TF32 chain makes it, to the bit
            assert redo == (1 if kind in ("wide", "inf", "nan") else 0)
    if kind in ("wide", "inf", "nan"):
        assert_bits_equal(out[0], out[1])
    else:
        rms = np.sqrt(np.mean(out[1].astype(np.float64) ** 2))
        assert np.abs(out[0] - out[1]).max() <= 4e-5 * max(rms, np.abs(out[1]).max())
    # a replay on ordinary values after one that was made over
    m16.x.set(util.uniform(72, m16.x.shape))
    m16.replay()
    first = m16.out.numpy()
    m32.x.set(util.uniform(72, m16.x.shape))
    m32.replay()
    second = m32.out.numpy()
    assert m16.records.buf.numpy()[-4] == 0
    assert np.abs(first - second).max() <= 4e-5 * np.abs(second).max()
    m16.close()
    m32.close()


def test_only_if_refuses_other_calls(fresh):
    e = fresh
    flag, a = e.tensor(np.zeros(4, np.int32)), e.tensor(util.normal(81, (64, 64)))
    with e.only_if(flag.ptr):
        with pytest.raises(B200Error):
            e.MatMul(a, a, e.empty((64, 64)))
        with pytest.raises(B200Error):
            e.DoWork()
    e.MatMul(a, a, e.empty((64, 64)))
    e.Signal()


@pytest.mark.parametrize("make", [_lenet, _yolo])
def test_failed_chain_leaves_its_records_clear(fresh, monkeypatch, make):
    e = fresh
    m = make(e, monkeypatch, 0)
    x = util.uniform(82, m.x.shape)
    m.x.set(x)
    want = m.forward().numpy()
    m.x.set(x * np.float32(1e6))
    links = []

    def fail(*a, **kw):
        links.append(0)
        if len(links) == 3:
            raise B200Error(2, "no room")
        return type(e).Conv2dPairs(e, *a, **kw)
    monkeypatch.setattr(e, "Conv2dPairs", fail, raising=False)
    with pytest.raises(B200Error):
        m.forward()
    monkeypatch.delattr(e, "Conv2dPairs")
    assert not m.records.buf.numpy()[:-4].any()
    m.x.set(x)
    assert_bits_equal(m.forward().numpy(), want)


# ---- values that are small but alone ---------------------------------------------------------------------------------
BIG = [(48, 128, 26, 26, 256, 3, 1), (96, 64, 32, 32, 128, 5, 2)]     # the im2col and the window kernel, 19 GFLOP and more


def _conv64(x, w, pad):
    import torch
    y = torch.nn.functional.conv2d(torch.from_numpy(x).cuda().double(), torch.from_numpy(w).cuda().double(), padding=pad)
    return y.cpu().numpy()


@pytest.mark.parametrize("case", BIG)
def test_large_single_convolutions_are_made_from_pairs(fresh, case):
    # ordinary values, to float64; constant filters, whose pairs are kept from the first call on, so that the second
    # launches the magnitude, the rewrite, the convolution and the check, and two of TF32 that find nothing to do
    e = fresh
    B, C, H, W, K, k, pad = case
    x, w = util.normal(91, (B, C, H, W)), util.normal(92, (K, C, k, k), scale=0.05)
    want = _conv64(x, w, pad)
    tx, tw, y = e.tensor(x), e.tensor(w), e.empty(want.shape)
    e.Conv2d(tx, tw, y, pad=(pad, pad))
    assert_gemm_close(y.numpy(), want, 1e-5)
    e.constant(tw)
    for _ in range(2):
        before = e.launches
        e.Conv2d(tx, tw, y, pad=(pad, pad))
        made = e.launches - before
    assert made == 6
    assert_gemm_close(y.numpy(), want, 1e-5)
    # a sprinkling of small values among ordinary ones changes nothing of that
    x.reshape(-1)[::x.size // 50] = np.float32(1e-13)
    tx.set(x)
    e.Conv2d(tx, tw, y, pad=(pad, pad))
    assert_gemm_close(y.numpy(), _conv64(x, w, pad), 1e-5)
    # an image far below the others and a value far above; then infinities and NaNs; then ordinary values again
    wide = x.copy()
    wide[1] *= np.float32(1e-25)
    wide[2, :, 3, 3] = np.float32(1e20)
    tx.set(wide)
    e.Conv2d(tx, tw, y, pad=(pad, pad))
    got, ref = y.numpy(), _conv64(wide, w, pad)
    for b in range(3):
        assert_gemm_close(got[b], ref[b], 1e-5)
    bad = x.copy()
    bad[0, 0, 0, 0], bad[3, 1, 5, 5] = np.inf, np.nan
    tx.set(bad)
    e.Conv2d(tx, tw, y, pad=(pad, pad))
    got, ref = y.numpy(), _conv64(bad, w, pad)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref)) and not np.isfinite(got[0]).all()
    assert_gemm_close(got[1], ref[1], 1e-5)
    tx.set(x)
    e.Conv2d(tx, tw, y, pad=(pad, pad))
    assert_gemm_close(y.numpy(), _conv64(x, w, pad), 1e-5)


@pytest.mark.parametrize("case", BIG)
@pytest.mark.parametrize("where", ["filter", "pixel", "corner"])
def test_small_values_alone_in_a_window_or_a_filter(fresh, case, where):
    # fewer of them than the allowance: a filter of one tap, an image of a few pixels
    e = fresh
    B, C, H, W, K, k, pad = case
    x, w = util.normal(93, (B, C, H, W)), util.normal(94, (K, C, k, k), scale=0.05)
    if where == "filter":
        w[5] = 0.0
        w[5, 0, 1, 1] = np.float32(1e-15)
        part = (slice(None), 5)
    else:
        x[1] = 0.0
        if where == "pixel":
            x[1, :20, 9, 7] = util.normal(95, 20) * np.float32(1e-14)
        else:
            x[1, C - 1, H - 1, W - 1] = np.float32(1e-16)
        part = (1,)
    want = _conv64(x, w, pad)
    y = e.empty(want.shape)
    e.Conv2d(e.tensor(x), e.tensor(w), y, pad=(pad, pad))
    got = y.numpy()
    assert_gemm_close(got, want, 1e-5)
    assert np.linalg.norm(got[part] - want[part]) <= 2e-6 * np.linalg.norm(want[part])


@pytest.mark.parametrize("case", [c for c in LINKS if c[4] % 8 == 0 and c[0] > 1])
def test_link_marks_a_place_where_every_channel_is_small(fresh, case):
    # the input is within range, the output's pairs (scaled by a bound) are not where all channels are small
    e = fresh
    B, C, H, W, K, k, pad, act, alpha, pool = case
    x = util.normal(96, (B, C, H, W))
    w = util.normal(97, (K, C, k, k), scale=0.05)
    marks = []
    for far in (False, True):
        z = x.copy()
        if far:
            z[1, :, H // 2 - k:H // 2 + k, W // 2 - k:W // 2 + k] *= np.float32(2.0 ** -26)
        tx, rx = _pairs(e, z)
        Ho, Wo = H + 2 * pad - k + 1, W + 2 * pad - k + 1
        shape = (B, K, Ho // 2, Wo // 2) if pool else (B, K, Ho, Wo)
        ry, yp = e.tensor(np.zeros(4, np.int32)), e.empty((int(np.prod(shape)),))
        e.Conv2dPairs(None, e.tensor(w), None, x.shape, rx.ptr, ry.ptr, pad=(pad, pad), act=act, alpha=alpha, pool2=pool,
                      x_pairs=tx, y_pairs=yp)
        marks.append(int(ry.numpy()[2]))
    assert marks == [0, 1]


def test_first_link_and_pool_mark_small_places(fresh):
    e = fresh
    w = util.normal(98, (16, 1, 3, 3), scale=0.3)
    for far in (False, True):
        x = util.uniform(99, (3, 1, 28, 28)) + np.float32(0.1)
        x[1, :, 20:] = 0.0      # nothing at all is not small
        if far:
            x[1, 0, 24, 13] = np.float32(1e-12)
        recs, yp = e.tensor(np.zeros(8, np.int32)), e.empty((3 * 16 * 14 * 14,))
        tx = e.tensor(x)
        e.pairs_magnitude(tx, recs.ptr)
        e.Conv2dPairs(tx, e.tensor(w), None, x.shape, recs.ptr, recs.ptr + 16, pad=(1, 1), act="rectify", pool2=True,
                      y_pairs=yp)
        assert recs.numpy()[6] == (1 if far else 0)
        z = util.normal(100, (2, 40, 12, 12))
        z[:, :, 4:6, 4:6] = 0.0
        if far:
            z[1, 3, 4, 5] = np.float32(1e-12)
        rz, ry = e.tensor(np.array([np.abs(z).max().view(np.int32), 0, 0, 0], np.int32)), e.tensor(np.zeros(4, np.int32))
        e.MaxPool2DPairs(e.tensor(z), rz.ptr, e.empty((2 * 40 * 36,)), ry.ptr, (2, 2), (0, 0), (2, 2))
        assert ry.numpy()[2] == (1 if far else 0)


def test_dark_image_of_a_large_batch(fresh):
    # one image in 8192 holds a single pixel of 1e-13: too few small values for the allowance at any link
    from gorgonia_b200 import Engine
    B = 8192
    x = util.uniform(101, (B, 1, 28, 28))
    x[7] = 0.0
    x[7, 0, 13, 13] = np.float32(1e-13)
    pooled, redo = [], []
    for flops in (0, 1e30):
        e = Engine(0, 4 << 30)
        with pytest.MonkeyPatch.context() as mp:
            m = _lenet(e, mp, flops, B)
        m.x.set(x)
        m.forward()
        a = m.chain.layers[-1]
        pooled.append((a["pooled"] or a["y"]).numpy()[7])
        if m.records is not None:
            redo.append(int(m.records.buf.numpy()[-4]))
            m.x.set(util.uniform(102, x.shape))
            m.forward()
            redo.append(int(m.records.buf.numpy()[-4]))
        e.Close()
    assert np.linalg.norm(pooled[0] - pooled[1]) <= 4e-6 * np.linalg.norm(pooled[1])
    assert redo == [1, 0]


def test_only_if_is_the_calling_threads(fresh):
    # another thread's calls on the same engine are neither refused nor made conditional, and a pointwise call
    # inside is refused like every other
    import threading
    e = fresh
    z = util.normal(103, (2, 16, 32, 32))
    flag, tz, ty = e.tensor(np.zeros(4, np.int32)), e.tensor(z), e.tensor(np.zeros((2, 16, 16, 16), np.float32))
    w = e.tensor(util.normal(104, (32, 16, 3, 3), scale=0.05))
    ts = tuple(e.tensor(np.zeros((2, 16, 16, 16), np.float32)) for _ in range(2))
    conv, inner, s = e.tensor(np.zeros((2, 32, 32, 32), np.float32)), e.tensor(np.zeros((2, 16, 16, 16), np.float32)), e.empty(z.shape)
    second, failed = e.tensor(np.zeros(4, np.int32)), []

    def other():
        try:
            e.MaxPool2D(tz, ty, (2, 2), (0, 0), (2, 2))
            e.MaxPool2DSplit(tz, None, ts, (2, 2), (0, 0), (2, 2))
            e.Conv2dChain(tz, w, conv, z.shape, pad=(1, 1))
            e.Unary("neg", tz, reuse=s)
            e.Signal()
            with e.only_if(second.ptr):     # a condition of its own at the same time
                e.MaxPool2D(tz, inner, (2, 2), (0, 0), (2, 2))
        except Exception as err:            # noqa: BLE001 - handed to the test's thread
            failed.append(err)

    with e.only_if(flag.ptr):
        t = threading.Thread(target=other)
        t.start()
        t.join()
        e.MaxPool2D(tz, inner, (2, 2), (0, 0), (2, 2))
        with pytest.raises(B200Error):
            e.Unary("neg", tz, reuse=s)
        with pytest.raises(B200Error):
            e.Add(tz, tz, reuse=s)
    assert not failed
    want = oracle.maxpool2d(z, (2, 2), (0, 0), (2, 2))[0]
    assert_bits_equal(ty.numpy(), want)
    assert np.abs(ts[0].numpy() + ts[1].numpy() - want.transpose(0, 2, 3, 1).reshape(ts[0].shape)).max() <= 2.0 ** -21 * np.abs(z).max()
    assert np.abs(conv.numpy()).max() > 0
    assert_bits_equal(s.numpy(), -z)
    assert not inner.numpy().any()


@pytest.mark.parametrize("alpha", [0.1, 0.001, 0.0003])
def test_many_small_values_among_ordinary_ones(fresh, alpha):
    # a slope that leaves many small values, each beside ordinary ones: the chain is not made over, and agrees with
    # the TF32 one
    e = fresh
    ch, g = (3, 16, 32, 64, 128), util.rng(105)
    ws = [e.constant(e.tensor((g.standard_normal((ch[i + 1], ch[i], 3, 3)) * np.sqrt(2 / (9 * ch[i]))).astype(np.float32)))
          for i in range(4)]
    chain = tapes._ConvChain(e, 8, (3, 128, 128), [
        {"w": ws[i], "pad": (1, 1), "bias": None, "act": "leaky", "alpha": alpha, "pool": "2x2/2" if i < 2 else None}
        for i in range(4)])
    assert chain.can_pairs()
    rec = tapes._Records(e)
    chain.plan_pairs(rec)
    tx = e.tensor(g.random((8, 3, 128, 128), dtype=np.float32) - np.float32(0.5))
    with rec.chain():
        got = chain.forward_pairs(tx).numpy()
        small = rec.buf.numpy().reshape(-1, 4)[:len(rec.counts), 1]
    assert rec.buf.numpy()[-4] == 0
    assert alpha > 0.05 or (small > np.array(rec.counts) >> 16).any()     # more than a matrix may hold
    want = chain.forward(tx).numpy()
    # both chains' sums end in float32 roundings: as the chains of the tapes
    assert np.abs(got - want).max() <= 4e-5 * np.abs(want).max()
