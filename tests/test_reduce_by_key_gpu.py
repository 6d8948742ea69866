"""Reduce_By_Key in its one-pass form: tile edges, several turns of the stage ring, segments
shorter and longer than tiles, key and value widths, views, alignment, ordered operators.
Integer-valued data, so that every result is exact, against numpy's reduceat."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    return t


def run_keys(rng, n, mean, dtype):
    k = np.cumsum(rng.random(n) < 1.0 / mean) if mean else np.zeros(n)
    info = np.iinfo(dtype) if np.issubdtype(dtype, np.integer) else None
    k = k % (info.max if info else 1 << 20)
    return k.astype(dtype)


def expected(k, v, ufunc=np.add):
    heads = np.flatnonzero(np.concatenate([[True], k[1:] != k[:-1]]))
    return k[heads], ufunc.reduceat(v, heads).astype(v.dtype)  # (numpy widens integer sums)


def check(trtc, k, v, dk, dv, ufunc=np.add, op=None, pred=None, off=0):
    n = len(k)
    ko, vo = trtc.device_vector_from_numpy(np.zeros(n + 1, k.dtype)), trtc.device_vector_from_numpy(np.full(n + 1, 77, v.dtype))
    c = trtc.Reduce_By_Key(dk, dv, ko.range(0, n), vo.range(0, n), pred, op)
    ek, ev = expected(k, v, ufunc)
    assert c == len(ek)
    assert ko.to_host(0, c).tobytes() == ek.tobytes()
    assert vo.to_host(0, c).tobytes() == ev.astype(v.dtype).tobytes()
    assert vo.to_host()[c] == 77  # nothing written behind the last segment


SIZES = [1, 2, 19, 20, 5119, 5120, 5121, 5124, 5128, 10240, 15361, 40_001, 5120 * 4 * 300 + 5, 5120 * 148 * 40 + 9]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("mean", [0, 1, 3, 1000, 20_000])
def test_sizes_and_runs(trtc, n, mean):
    rng = np.random.default_rng(n + mean)
    k, v = run_keys(rng, n, mean, np.int32), rng.integers(0, 8, n).astype(np.float32)
    if mean == 0 or mean == 20_000:
        v[:] = 0
        v[::max(1, n // 1000)] = 1  # sums stay exact in float32
    check(trtc, k, v, trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v))


@pytest.mark.parametrize("kt", [np.int8, np.int16, np.uint32, np.int64, np.float64])
@pytest.mark.parametrize("vt", [np.int32, np.int64, np.float64])
@pytest.mark.parametrize("n", [2561, 50_000])
def test_types(trtc, kt, vt, n):
    rng = np.random.default_rng(n)
    k, v = run_keys(rng, n, 7, kt), rng.integers(-50, 50, n).astype(vt)
    check(trtc, k, v, trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v))
    check(trtc, k, v, trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v), np.maximum, trtc.Maximum(), trtc.EqualTo())


@pytest.mark.parametrize("off", [1, 2, 3, 4])
def test_unaligned_ranges(trtc, off):
    n = 20_011
    rng = np.random.default_rng(off)
    k, v = run_keys(rng, n, 5, np.int32), rng.integers(0, 9, n).astype(np.int32)
    pad = np.zeros(off, np.int32)
    dk = trtc.device_vector_from_numpy(np.concatenate([pad, k])).range(off, off + n)
    dv = trtc.device_vector_from_numpy(np.concatenate([pad, v])).range(off, off + n)
    check(trtc, k, v, dk, dv)
    check(trtc, k, v, dk, trtc.device_vector_from_numpy(v))


def test_views_and_functors(trtc):
    n = 30_007
    rng = np.random.default_rng(1)
    k, v = run_keys(rng, n, 9, np.int32), rng.integers(0, 9, n).astype(np.int32)
    dk, dv = trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v)
    ek, ev = expected(k, np.ones(n, np.int32))
    # counts of a histogram: a constant as the values
    ko, vo = trtc.device_vector("int32_t", n), trtc.device_vector("int32_t", n)
    c = trtc.Reduce_By_Key(dk, trtc.DVConstant(trtc.DVInt32(1), n), ko, vo)
    assert c == len(ek) and vo.to_host(0, c).tobytes() == ev.tobytes() and ko.to_host(0, c).tobytes() == ek.tobytes()
    # keys dropped
    c = trtc.Reduce_By_Key(dk, dv, trtc.DVDiscard("int32_t", n), vo)
    ek, ev = expected(k, v)
    assert c == len(ek) and vo.to_host(0, c).tobytes() == ev.tobytes()
    # a user's predicate, and operators whose result depends on the order of their operands
    half = trtc.Functor({}, ["a", "b"], "        return a / 2 == b / 2;\n")
    heads = np.flatnonzero(np.concatenate([[True], k[1:] // 2 != k[:-1] // 2]))
    last = np.concatenate([heads[1:] - 1, [n - 1]])
    for body, want in (("        return a;\n", v[heads]), ("        return b;\n", v[last])):
        c = trtc.Reduce_By_Key(dk, dv, ko, vo, half, trtc.Functor({}, ["a", "b"], body))
        assert c == len(heads)
        assert ko.to_host(0, c).tobytes() == k[last].tobytes() and vo.to_host(0, c).tobytes() == want.tobytes()
    # outputs shorter than the number of segments are filled to their end
    short = trtc.device_vector("int32_t", 10)
    assert trtc.Reduce_By_Key(dk, dv, ko, short) == len(ek) and short.to_host().tobytes() == ev[:10].tobytes()


def test_overlapping_output_takes_the_general_form(trtc):
    n = 10_000
    rng = np.random.default_rng(2)
    k, v = run_keys(rng, n, 4, np.int32), rng.integers(0, 9, n).astype(np.int32)
    dk, dv = trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v)
    c = trtc.Reduce_By_Key(dk, dv, dk, dv)
    ek, ev = expected(k, v)
    assert c == len(ek) and dk.to_host(0, c).tobytes() == ek.tobytes() and dv.to_host(0, c).tobytes() == ev.tobytes()
