"""Fused runs of calls that do not fit one program, that release their temporaries, or that take the shared-memory
interpreter on small and unaligned tensors (GPU tests against the CPU oracle)."""
import numpy as np
import pytest

from gorgonia_b200.engine import Tensor
from oracle import oracle
from tests import util
from tests.util import assert_bits_equal, assert_pointwise_close

pytestmark = pytest.mark.gpu


def _at(e, a, start):
    """The array on the device, `start` elements into a larger buffer."""
    whole = np.concatenate([np.zeros(start, a.dtype), a])
    return Tensor(e, e.tensor(whole).ptr + start * a.itemsize, a.shape, a.dtype, owned=False)


SIZES = [1, 3, 127, 128 * 4, 128 * 4 + 1, 5000, 1 << 20, 3_000_001]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("start", [0, 1])
def test_gated_unit(fresh, n, dt, start):
    e = fresh
    v = {k: util.normal(100 + i, n, dt) for i, k in enumerate("ifgoc")}
    d = {k: _at(e, a, start) for k, a in v.items()}
    c, h = (_at(e, np.zeros(n, dt), start) for _ in range(2))
    e.Signal()
    i, f, g, q = (e.empty((n,), dt) for _ in range(4))
    e.Unary("sigmoid", d["i"], reuse=i)
    e.Unary("sigmoid", d["f"], reuse=f)
    e.Unary("tanh", d["g"], reuse=g)
    e.Mul(f, d["c"], reuse=c)
    e.Mul(i, g, unsafe=True)
    e.Add(c, i, unsafe=True)
    e.Unary("sigmoid", d["o"], reuse=q)
    e.Unary("tanh", c, reuse=h)
    e.Mul(h, q, unsafe=True)
    for t in (i, f, g, q):
        t.free()
    assert e.pending() == (9, 2)
    e.DoWork()
    un = oracle.unary
    wc = oracle.binary("add", oracle.binary("mul", un("sigmoid", v["f"]), v["c"]),
                       oracle.binary("mul", un("sigmoid", v["i"]), un("tanh", v["g"])))
    got = c.numpy()
    # each factor within 1e-6 (1e-13) of its own, and the sum may cancel
    rel = 4e-6 if dt == np.float32 else 4e-13
    assert (np.abs(got - wc) <= rel * (np.abs(v["c"]) + 1)).all()
    assert_pointwise_close(h.numpy(), oracle.binary("mul", un("tanh", got), un("sigmoid", v["o"])), rel)


@pytest.mark.parametrize("n", [777, 1 << 20])
@pytest.mark.parametrize("length", [7, 8, 9, 17, 30])
def test_runs_of_any_length(fresh, n, length):
    # a run in place; one that keeps every result; one whose temporaries are released at its end
    e = fresh
    x, y = util.normal(5, n), util.normal(6, n)
    want = [x]
    for k in range(length):
        want.append(oracle.binary("add" if k % 2 else "mul", want[-1], y))
    tx, ty = e.tensor(x), e.tensor(y)
    for k in range(length):
        (e.Add if k % 2 else e.Mul)(tx, ty, unsafe=True)
    e.DoWork()
    assert_bits_equal(tx.numpy(), want[-1])
    tx.set(x)
    kept = [e.empty(n) for _ in range(length)]
    e.Signal()
    a = tx
    for k in range(length):
        a = (e.Add if k % 2 else e.Mul)(a, ty, reuse=kept[k])
    e.DoWork()
    for k in range(length):
        assert_bits_equal(kept[k].numpy(), want[k + 1])
    out = e.empty(n)
    a = tx
    for k in range(length):
        a = (e.Add if k % 2 else e.Mul)(a, ty, reuse=kept[k] if k + 1 < length else out)
    for t in kept[:-1]:
        t.free()
    e.DoWork()
    assert_bits_equal(out.numpy(), want[-1])


def test_released_temporary_that_is_read_later_is_stored(fresh):
    # more results than one kernel stores, read again after the point where it has to end
    e = fresh
    n = 1 << 18
    xs = [util.normal(20 + k, n) for k in range(6)]
    ts = [e.tensor(a) for a in xs]
    tmp, out = [e.empty(n) for _ in range(6)], [e.empty(n) for _ in range(6)]
    e.Signal()
    for k in range(6):
        e.Unary("square", ts[k], reuse=tmp[k])
    for k in range(6):
        e.Add(tmp[k], ts[(k + 1) % 6], reuse=out[k])
    for t in tmp:
        t.free()
    again = e.empty(n)      # may well be one of the released buffers
    e.Unary("neg", out[0], reuse=again)
    e.DoWork()
    for k in range(6):
        assert_bits_equal(out[k].numpy(), oracle.binary("add", oracle.unary("square", xs[k]), xs[(k + 1) % 6]))
    assert_bits_equal(again.numpy(), oracle.unary("neg", out[0].numpy()))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [4097, 3_000_001])
@pytest.mark.parametrize("div,mod", [(1, 1), (1, 7), (3, 5), (4, 3), (49, 128), (784, 64), (1024, 1021), (1 << 20, 2), (999_999, 3)])
def test_broadcast_index(fresh, n, dt, div, mod):
    # two broadcast sources in one program; every element names its own
    e = fresh
    x, g, b = util.normal(31, n, dt), util.normal(32, mod, dt), util.normal(33, mod, dt)
    y = e.empty((n,), dt)
    e.BroadcastBinary("mul", e.tensor(x), e.tensor(g), div, mod, reuse=y)
    e.BroadcastBinary("add", y, e.tensor(b), div, mod, unsafe=True)
    at = np.arange(n) // div % mod
    assert_bits_equal(y.numpy(), oracle.binary("add", oracle.binary("mul", x, g[at]), b[at]))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [5, 1000, 3_000_001])
@pytest.mark.parametrize("start", [0, 1])
@pytest.mark.parametrize("n_src,n_instr", [(1, 2), (3, 4), (4, 4), (2, 5), (6, 8)])
def test_one_result_to_several_outputs(fresh, n, dt, start, n_src, n_instr):
    # programs of the register kernel and of the loop kernel, on small, unaligned and large tensors: the result of
    # the first instruction (kept for the last one) goes to two outputs, the last one's to two as well
    e = fresh
    xs = [util.normal(60 + k, n, dt) for k in range(n_src)]
    srcs = [_at(e, x, start) for x in xs]
    outs = [_at(e, np.zeros(n, dt), start) for _ in range(4)]
    SRC, INS = 0x00, 0x80
    instr, vals = [("neg", SRC | 0, SRC | 0)], [-xs[0]]
    for k in range(1, n_instr - 1):
        instr.append(("add" if k % 2 else "mul", INS | (k - 1), SRC | (k % n_src)))
        vals.append(oracle.binary("add" if k % 2 else "mul", vals[-1], xs[k % n_src]))
    instr.append(("sub", INS | (n_instr - 2), INS | 0))
    vals.append(oracle.binary("sub", vals[-1], vals[0]))
    last = n_instr - 1
    e.Pointwise({"instr": instr, "out": [0, last, 0, last]}, outs, srcs, n, dt)
    for o, k in zip(outs, (0, last, 0, last)):
        assert_bits_equal(o.numpy(), vals[k])
    for s, x in zip(srcs, xs):      # nothing was written where it does not belong
        assert_bits_equal(s.numpy(), x)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [4096, 3_000_001])
@pytest.mark.parametrize("chunk", [None, (784, 32), (3, 5)])
@pytest.mark.parametrize("instr", [3, 7])
def test_rows_and_scalars_with_and_without_divided_sources(fresh, n, dt, chunk, instr):
    # rows and scalars alone take the kernels without index divisions, a third kind of source the others
    e, SRC, INS = fresh, 0x00, 0x80
    x, row, one = util.normal(71, n, dt), util.normal(72, 64, dt), util.normal(73, 1, dt)
    srcs, bcast, third = [x, row, one], {1: (1, 64), 2: (1, 1)}, None
    if chunk:
        third = util.normal(74, chunk[1], dt)
        srcs, bcast = srcs + [third], {**bcast, 3: chunk}
    full = [x, row[np.arange(n) % 64], np.full(n, one[0], dt)] + ([third[np.arange(n) // chunk[0] % chunk[1]]] if chunk else [])
    prog, val = [("mul", SRC | 0, SRC | 1)], oracle.binary("mul", full[0], full[1])
    for k in range(1, instr):
        s = k % len(srcs) if k > 1 else 2
        prog.append(("add" if k % 2 else "mul", INS | (k - 1), SRC | s))
        val = oracle.binary("add" if k % 2 else "mul", val, full[s])
    out = e.empty((n,), dt)
    e.Pointwise({"instr": prog, "out": [instr - 1], "bcast": bcast}, [out], [e.tensor(a) for a in srcs], n, dt)
    assert_bits_equal(out.numpy(), val)
