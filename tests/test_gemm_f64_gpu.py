"""The float64 product at the sizes where its tiles, k slabs and shared k ranges meet, against the CPU oracle (GPU tests)."""
import numpy as np
import pytest

from oracle import oracle
from tests import util
from tests.util import assert_gemm_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transA,transB", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(1, 17, 1), (31, 33, 15), (32, 32, 16), (65, 63, 129), (100, 300, 784), (257, 18, 2049),
                                   (1000, 1030, 70)])
def test_matmul_f64_tiles(fresh, shape, transA, transB):
    e = fresh
    M, N, K = shape
    a = util.normal(21 + M, (K, M) if transA else (M, K), np.float64)
    b = util.normal(22 + N, (N, K) if transB else (K, N), np.float64)
    bias, c0 = util.normal(23, N, np.float64), util.normal(24, (M, N), np.float64)
    ta, tb, tc = e.tensor(a), e.tensor(b), e.empty((M, N), np.float64)
    want = oracle.gemm(a, b, transA, transB)
    for _ in range(2):
        e.MatMul(ta, tb, tc, transA, transB)
        assert_gemm_close(tc.numpy(), want, 1e-12)
    e.MatMul(ta, tb, tc, transA, transB, bias=e.tensor(bias), act="rectify")
    assert_gemm_close(tc.numpy(), np.maximum(want + bias, 0), 1e-12)
    tc.set(c0)
    e.MatMul(ta, tb, tc, transA, transB, incr=True)
    assert_gemm_close(tc.numpy(), want + c0, 1e-12)


def test_matmul_f64_batched_and_unaligned(fresh):
    e = fresh
    a, b = util.normal(31, (5, 70, 45), np.float64), util.normal(32, (5, 45, 37), np.float64)
    tc = e.empty((5, 70, 37), np.float64)
    e.MatMul(e.tensor(a), e.tensor(b), tc)
    assert_gemm_close(tc.numpy(), a @ b, 1e-12)
    # an operand that starts on an 8-byte boundary only
    from gorgonia_b200.engine import Tensor
    flat = util.normal(33, 64 * 48 + 1, np.float64)
    t = e.tensor(flat)
    view = Tensor(e, t.ptr + 8, (64, 48), np.float64, owned=False)
    tc = e.empty((64, 37), np.float64)
    e.MatMul(view, e.tensor(np.ascontiguousarray(np.vstack([b[0], b[1][:3]]))), tc)
    assert_gemm_close(tc.numpy(), flat[1:].reshape(64, 48) @ np.vstack([b[0], b[1][:3]]), 1e-12)
