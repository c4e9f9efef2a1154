"""float32 products made from pairs of fp16 (large ones) and their way back to pairs of TF32 where fp16's
range is not enough (GPU tests against float64)."""
import numpy as np
import pytest

from tests import util
from tests.util import assert_gemm_close

pytestmark = pytest.mark.gpu


def _product(e, a, b, transA=False, transB=False, constant=False, **kw):
    ta, tb = e.tensor(a), e.tensor(b)
    if constant:
        e.constant(tb)
    M = a.shape[-1] if transA else a.shape[-2]
    N = b.shape[-2] if transB else b.shape[-1]
    tc = e.empty(a.shape[:-2] + (M, N))
    out = []
    for _ in range(2):      # twice: the operands' records must be clear again, a constant's must stay
        e.MatMul(ta, tb, tc, transA, transB, **kw)
        out.append(tc.numpy())
    for t in (ta, tb, tc):
        t.free()
    assert np.array_equal(out[0], out[1], equal_nan=True)
    return out[1]


def _want(a, b, transA=False, transB=False):
    a, b = a.astype(np.float64), b.astype(np.float64)
    return (np.swapaxes(a, -1, -2) if transA else a) @ (np.swapaxes(b, -1, -2) if transB else b)


@pytest.mark.parametrize("transA,transB", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(2048, 2048, 2048), (2051, 1999, 2309), (1030, 3001, 1000), (3000, 130, 9000)])
def test_large_products(fresh, shape, transA, transB):
    M, N, K = shape
    a = util.normal(1, (K, M) if transA else (M, K))
    b = util.normal(2, (N, K) if transB else (K, N), scale=0.02)
    want = _want(a, b, transA, transB)
    got = _product(fresh, a, b, transA, transB)
    assert_gemm_close(got, want, 1e-5)
    # sums of exact products of pairs: no worse than the TF32 pairs' 7e-7 of the result's norm
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


def test_large_batched_and_constant(fresh):
    a, b = util.normal(3, (6, 1024, 1100)), util.normal(4, (6, 1100, 1024), scale=0.02)
    assert_gemm_close(_product(fresh, a, b), _want(a, b), 1e-5)
    a, b = util.normal(5, (4000, 1152)), util.normal(6, (1152, 2000), scale=0.02)
    assert_gemm_close(_product(fresh, a, b, constant=True), _want(a, b), 1e-5)


@pytest.mark.parametrize("scale_a,scale_b", [(1e-30, 1.0), (1e30, 1e-30), (3e37, 1e-20), (1e-32, 1e30), (1e20, 1e15)])
def test_any_magnitude(fresh, scale_a, scale_b):
    # the whole operand far from 1: taken up by its power of two, or, near the ends of float32, by TF32 pairs,
    # which need their tails, 2^-11 of the values, above float32's smallest normal number, 1.2e-38
    a = (util.normal(7, (2048, 2048)).astype(np.float64) * scale_a).astype(np.float32)
    b = (util.normal(8, (2048, 2048)).astype(np.float64) * scale_b).astype(np.float32)
    want = _want(a, b)
    got = _product(fresh, a, b)
    assert_gemm_close(got, want, 1e-5)


@pytest.mark.parametrize("constant", [False, True])
def test_wide_range_rows_keep_their_precision(fresh, constant):
    # rows of A from 1e-18 to 1e18: each row of the result is as exact as its neighbours
    a = util.normal(9, (2048, 2048)) * (10.0 ** np.linspace(-18, 18, 2048)).astype(np.float32)[:, None]
    b = util.normal(10, (2048, 2048))
    want = _want(a, b)
    got = _product(fresh, a, b, constant=constant)
    row = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert row.max() < 2e-6
    # and the same in the other operand's columns
    want = _want(b, a.T)
    got = _product(fresh, b, np.ascontiguousarray(a.T), constant=constant)
    assert (np.linalg.norm(got - want, axis=0) / np.linalg.norm(want, axis=0)).max() < 2e-6


def test_lowest_value_masks(fresh):
    # a column of A near the type's lowest value meets a row of zeros: the others must not notice (the lowest
    # value itself rounds to an infinite TF32 head)
    low = np.float32(-3.0e38)
    a, b = util.normal(11, (2048, 2048)), util.normal(12, (2048, 2048))
    a[:, 7] = low
    b[7] = 0.0
    assert_gemm_close(_product(fresh, a, b), _want(a, b), 1e-5)
    a[:, 7] = util.normal(13, 2048)
    b[7] = 1.0
    a[5, 7] = low          # one element only: its row is that element's, the others as ever
    want = _want(a, b)
    got = _product(fresh, a, b)
    assert_gemm_close(np.delete(got, 5, 0), np.delete(want, 5, 0), 1e-5)
    assert_gemm_close(got[5], want[5], 1e-5)


def test_infinities_and_nans(fresh):
    a, b = util.normal(14, (2048, 2048)), util.normal(15, (2048, 2048))
    a[3, 9], a[4, 10], b[11, 6] = np.inf, np.nan, -np.inf
    got = _product(fresh, a, b)
    clean = np.ones((2048, 2048), bool)
    clean[3], clean[4], clean[:, 6] = False, False, False
    az, bz = np.nan_to_num(a, nan=0, posinf=0, neginf=0), np.nan_to_num(b, nan=0, posinf=0, neginf=0)
    want = _want(az, bz)
    assert np.isfinite(got[clean]).all() and not np.isfinite(got[~clean]).any()
    assert np.abs(got - want)[clean].max() <= 1e-5 * np.abs(want).max()


def test_all_zero_and_recorded(fresh):
    e = fresh
    z = np.zeros((2048, 2048), np.float32)
    assert not _product(e, z, util.normal(16, (2048, 2048))).any()
    # a recorded product replays on new operands, some within fp16's range and some not
    ta, tb, tc = e.tensor(z), e.tensor(z), e.empty((2048, 2048))
    e.MatMul(ta, tb, tc)
    e.Signal()
    e.tape_begin()
    e.MatMul(ta, tb, tc)
    tape = e.tape_end()
    b = util.normal(17, (2048, 2048))
    for k, spread in enumerate((0, 30, 0)):
        a = util.normal(18 + k, (2048, 2048)) * (10.0 ** np.linspace(0, spread, 2048)).astype(np.float32)[:, None]
        ta.set(a)
        tb.set(b)
        e.tape_launch(tape)
        e.Signal()
        want = _want(a, b)
        row = np.linalg.norm(tc.numpy() - want, axis=1) / np.linalg.norm(want, axis=1)
        assert row.max() < 2e-6
    e.tape_destroy(tape)


@pytest.mark.parametrize("which", ["a", "b", "both"])
def test_constant_met_in_a_full_arena(which):
    # at its first use the arena holds the TF32 pairs but not all that fp16 pairs need; with room again, the
    # second product must not find anything that was never made
    from gorgonia_b200 import Engine
    e = Engine(0, 256 << 20)
    a, b = util.normal(31, (2048, 2048)), util.normal(32, (2048, 2048), scale=0.02)
    ta, tb, tc = e.tensor(a), e.tensor(b), e.empty((2048, 2048))
    for t in {"a": [ta], "b": [tb], "both": [ta, tb]}[which]:
        e.constant(t)
    filler = e.Get(e.arena_stats()["largest_free"] - (70 << 20))
    want = _want(a, b)
    e.MatMul(ta, tb, tc)
    assert_gemm_close(tc.numpy(), want, 1e-5)
    free = e.arena_stats()["free"]
    e.Put(filler)
    for _ in range(2):
        e.MatMul(ta, tb, tc)
        assert_gemm_close(tc.numpy(), want, 1e-5)
    e.Close()
    # nothing but the constants' TF32 pairs (two blocks of 16 MB each) had stayed behind
    assert free == (70 << 20) - (32 << 20) * (2 if which == "both" else 1)


def test_failed_convolution_leaves_no_trace():
    # the pairs' records are the engine's: a call that runs out of room must hand them back clear
    from gorgonia_b200 import B200Error, Engine
    B, C, H, W, K = 48, 128, 26, 26, 256
    x, w = util.normal(33, (B, C, H, W)), util.normal(34, (K, C, 3, 3), scale=0.05)
    out = []
    for fail in (False, True):
        e = Engine(0, 512 << 20)
        tx, tw, y = e.tensor(x * np.float32(1e6)), e.tensor(w), e.empty((B, K, H, W))
        if fail:
            filler = e.Get(e.arena_stats()["largest_free"] - x.nbytes - (256 << 10))
            with pytest.raises(B200Error):
                e.Conv2d(tx, tw, y, pad=(1, 1))
            e.Put(filler)
        tx.set(x)
        e.Conv2d(tx, tw, y, pad=(1, 1))
        out.append(y.numpy())
        e.Close()
    util.assert_bits_equal(out[0], out[1])


@pytest.mark.parametrize("size", [256, 1024])
def test_constant_read_with_two_strides(fresh, size):
    # one constant as a batch of slices, as every second one of them, and as one slice for the whole batch (the
    # sizes take TF32 and fp16 pairs)
    from gorgonia_b200 import _lib
    e, n, batch = fresh, size, 4
    a, b = util.normal(35, (batch, n, n)), util.normal(36, (2 * batch, n, n), scale=0.05)
    ta, tb, tc = e.tensor(a), e.constant(e.tensor(b)), e.empty((batch, n, n))
    for step in (1, 2, 0, 1):
        _lib.check(_lib.lib.b200_gemm(e.h, _lib.F32, 0, 0, n, n, n, ta.ptr, n, tb.ptr, n, tc.ptr, n, batch, n * n,
                                      step * n * n, n * n, None), e.h)
        assert_gemm_close(tc.numpy(), _want(a, b[[step * i for i in range(batch)]]), 1e-5)


@pytest.mark.parametrize("tiny", [1e-14, 1e-16])
@pytest.mark.parametrize("count", [1, 64])
@pytest.mark.parametrize("transA,transB", [(False, False), (True, True)])
def test_small_values_that_are_alone_in_their_line(fresh, count, tiny, transA, transB):
    # a diagonal factor of ones and a few tiny entries: each of these is the largest of its row and column
    n = 2048
    diag = np.ones(n, np.float32)
    diag[np.linspace(0, n - 1, count).astype(int)] = np.float32(tiny)
    d, x = np.diag(diag), util.normal(21, (n, n))
    for a, b in ((d, x), (x, d)):
        want = _want(a, b, transA, transB)
        got = _product(fresh, a, b, transA, transB)
        for axis in (0, 1):
            assert (np.linalg.norm(got - want, axis=axis) / np.linalg.norm(want, axis=axis)).max() < 1e-6


def test_small_row_of_a_tall_matrix(fresh):
    # one row in 131072 far below the others: fewer values than a 65536th of the matrix
    e, M, n = fresh, 131072, 1024
    a, b = util.normal(22, (M, n)), util.normal(23, (n, n), scale=0.05)
    rows = [0, 77_777, M - 1]
    a[77_777] *= np.float32(1e-20)
    want = _want(a[rows], b)
    ta, tb, tc = e.tensor(a), e.tensor(b), e.empty((M, n))
    e.MatMul(ta, tb, tc)
    got = tc.numpy()[rows]
    assert (np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)).max() < 1e-6


@pytest.mark.parametrize("transA,transB", [(False, False), (True, False), (False, True), (True, True)])
def test_small_values_among_ordinary_ones_stay_with_fp16(fresh, transA, transB):
    # harmless along k: no line is made of them, and the product is made once
    e, n = fresh, 2048
    a, b = util.normal(24, (n, n)), util.normal(25, (n, n), scale=0.02)
    for k in range(60):
        a[(31 * k) % n, (57 * k) % n] = np.float32(1e-13)
        b[(17 * k) % n, (91 * k) % n] = np.float32(1e-15)
    want = _want(a, b, transA, transB)
    assert_gemm_close(_product(e, a, b, transA, transB), want, 1e-5)
    # the word behind the two records says whether the product was made over
    ta, tb, tc = e.tensor(a), e.tensor(b), e.empty((n, n))
    fp16, tf32 = [], []
    for spread in (False, True):
        if spread:
            ta.set(a * (10.0 ** np.linspace(0, 20, n)).astype(np.float32)[:, None])
        ev = [e.event() for _ in range(2)]
        for _ in range(3):
            e.MatMul(ta, tb, tc, transA, transB)
        e.record(ev[0])
        for _ in range(20):
            e.MatMul(ta, tb, tc, transA, transB)
        e.record(ev[1])
        (tf32 if spread else fp16).append(e.elapsed_ms(*ev))
    assert fp16[0] < 0.8 * tf32[0]


def test_one_summation_order_whatever_the_batch():
    # streamk=False promises that a shard of a batch and the whole batch agree to the bit, at sizes where the
    # choice of pairs or of a cut along k would depend on the batch
    from gorgonia_b200 import Engine, tapes
    e = Engine(0, 8 << 30, streamk=False)
    x = util.uniform(41, (1024, 1, 28, 28))
    out = []
    for lo, hi in ((0, 1024), (0, 512), (512, 1024)):
        m = tapes.LeNet(e, hi - lo)
        m.x.set(x[lo:hi])
        out.append(m.forward().numpy())
        e.Signal()
        e.ResetAllocator()
    util.assert_bits_equal(out[0], np.concatenate(out[1:]))

    def shards(make, rows, parts):
        whole = make(0, rows)
        cut = [make(rows * k // parts, rows * (k + 1) // parts) for k in range(parts)]
        util.assert_bits_equal(whole, np.concatenate(cut))
        e.Signal()
        e.ResetAllocator()

    a, w = util.normal(42, (4096, 2048)), util.normal(43, (2048, 2048), scale=0.02)
    a[0, 0] = 1e-14

    def product(dt):
        def make(lo, hi):
            c = e.empty((hi - lo, w.shape[1]), dt)
            return e.MatMul(e.tensor(a[lo:hi].astype(dt)), e.constant(e.tensor(w.astype(dt))), c).numpy()
        return make
    shards(product(np.float32), 4096, 4)
    a, w = a[:256, :784], w[:784, :300]
    shards(product(np.float64), 256, 4)
    img, f = util.normal(44, (64, 128, 26, 26)), util.normal(45, (256, 128, 3, 3), scale=0.05)

    def conv(lo, hi):
        return e.Conv2d(e.tensor(img[lo:hi]), e.constant(e.tensor(f)), e.empty((hi - lo, 256, 26, 26)), pad=(1, 1)).numpy()
    shards(conv, 64, 4)
    s = util.normal(46, (512, 1000, 12))

    def total(lo, hi):
        return e.Reduce("sum", e.tensor(s[lo:hi]), e.empty((hi - lo, 12)), 1).numpy()
    shards(total, 512, 8)
    e.Close()
