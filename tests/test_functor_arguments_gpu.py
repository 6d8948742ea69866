"""A user's predicate is called on elements of the array only: it may index a captured vector by its
argument.  The functors here check their arguments themselves, count those that are not what the
call promises, and make no access with them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    return t


# the compaction pipeline starts at 2^22 elements; tiles of 5120 4-byte and 2560 8-byte elements
EDGE = -(-(1 << 22) // 5120) * 5120
SIZES = [1, 100, 5121, EDGE - 1, EDGE, EDGE + 1, EDGE + 20, EDGE + 2559, EDGE + 5119]
BASE = 1 << 20  # elements are BASE + their index: zeros and foreign words are none of them


def looked_up(trtc, n):
    """table[x - BASE] behind a check of x; calls[] counts per element, bad[0] the arguments that are none."""
    table = (np.arange(n) % 3 == 0).astype(np.int32)
    calls, bad = trtc.device_vector_from_numpy(np.zeros(n, np.int32)), trtc.device_vector_from_numpy(np.zeros(1, np.int32))
    f = trtc.Functor({"table": trtc.device_vector_from_numpy(table), "calls": calls, "bad": bad}, ["x"],
                     "        long long i = (long long)x - %d;\n"
                     "        if (i < 0 || i >= (long long)table.size()) { atomicAdd(&bad[0], 1); return false; }\n"
                     "        atomicAdd(&calls[i], 1);\n"
                     "        return table[i] != 0;\n" % BASE)
    return f, table != 0, calls, bad


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_selection_predicates(trtc, n, dtype):
    x = np.arange(BASE, BASE + n).astype(dtype)
    d, o, r = (trtc.device_vector_from_numpy(a) for a in (x, np.zeros(n, dtype), np.zeros(n, dtype)))
    f, keep, calls, bad = looked_up(trtc, n)
    assert trtc.Copy_If(d, o, f) == keep.sum() and o.to_host(0, int(keep.sum())).tobytes() == x[keep].tobytes()
    assert trtc.Remove_Copy_If(d, o, f) == n - keep.sum()
    if n > 1:
        assert o.to_host(0, int(n - keep.sum())).tobytes() == x[~keep].tobytes()
    assert trtc.Partition_Copy(d, o, r, f) == keep.sum()
    assert bad.to_host()[0] == 0
    c = calls.to_host()
    assert c.min() >= 3 and c.min() == c.max()  # no element more often than another


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_neighbour_predicate(trtc, n, dtype):
    x = np.arange(BASE, BASE + n).astype(dtype)
    d, o = trtc.device_vector_from_numpy(x), trtc.device_vector_from_numpy(np.zeros(n, dtype))
    bad = trtc.device_vector_from_numpy(np.zeros(1, np.int32))
    f = trtc.Functor({"bad": bad, "n": trtc.DVInt32(n)}, ["a", "b"],
                     "        if (a != b + 1 || b < %d || a >= %d + n) { atomicAdd(&bad[0], 1); return false; }\n"
                     "        return a / 2 == b / 2;\n" % (BASE, BASE))
    heads = np.concatenate([[True], x[1:] // 2 != x[:-1] // 2])
    assert trtc.Unique_Copy(d, o, f) == heads.sum() and o.to_host(0, int(heads.sum())).tobytes() == x[heads].tobytes()
    assert bad.to_host()[0] == 0


@pytest.mark.parametrize("n", [1, 2, 20, 2560, 2561, 5119, 5120, 5121, 5140, 10240, 20_483, EDGE + 7])
@pytest.mark.parametrize("dtype", [np.int16, np.int32, np.int64])
def test_key_predicate(trtc, n, dtype):
    # keys count up (modulo a range above zero): neighbours, or a key and itself, and nothing else
    m = min(n, 30_000)
    base = 1000 if dtype == np.int16 else BASE
    k = (base + np.arange(n) % m).astype(dtype)
    dk, dv = trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(np.ones(n, np.int32))
    ko, vo = trtc.device_vector_from_numpy(np.zeros(n, dtype)), trtc.device_vector_from_numpy(np.zeros(n, np.int32))
    bad = trtc.device_vector_from_numpy(np.zeros(1, np.int32))
    f = trtc.Functor({"bad": bad, "m": trtc.DVInt32(m)}, ["a", "b"],
                     "        long long i = (long long)a - %d, j = (long long)b - %d;\n"
                     "        if (i < 0 || i >= m || (j != (i + 1) %% m && j != i)) { atomicAdd(&bad[0], 1); return false; }\n"
                     "        return i / 2 == j / 2;\n" % (base, base))
    i = np.arange(n) % m
    heads = np.flatnonzero(np.concatenate([[True], (i[1:] // 2 != i[:-1] // 2)]))
    last = np.concatenate([heads[1:] - 1, [n - 1]])
    assert trtc.Reduce_By_Key(dk, dv, ko, vo, f) == len(heads)
    assert bad.to_host()[0] == 0
    assert ko.to_host(0, len(heads)).tobytes() == k[last].tobytes()
    assert vo.to_host(0, len(heads)).tobytes() == (last - heads + 1).astype(np.int32).tobytes()


@pytest.mark.parametrize("n", [1, 5121, 300_000, 8_000_003])
@pytest.mark.parametrize("run", [3, 7000, 1 << 30])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_value_operator(trtc, n, run, dtype):
    # values from one range under an operator that is only defined on it; the call before leaves other
    # words in the stream's workspace
    k = (np.arange(n) // run).astype(np.int32)
    v = (BASE + (np.arange(n) * 2654435761 >> 7) % 5000).astype(dtype)
    dk, dv = trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v)
    ko, vo = trtc.device_vector_from_numpy(np.zeros(n, np.int32)), trtc.device_vector_from_numpy(np.zeros(n, dtype))
    bad = trtc.device_vector_from_numpy(np.zeros(1, np.int32))
    f = trtc.Functor({"bad": bad}, ["a", "b"],
                     "        if (a < %d || a >= %d || b < %d || b >= %d) atomicAdd(&bad[0], 1);\n"
                     "        return a > b ? a : b;\n" % (BASE, BASE + 5000, BASE, BASE + 5000))
    heads = np.arange(0, n, run)
    want = np.maximum.reduceat(v, heads).astype(dtype)
    minus = trtc.device_vector_from_numpy(np.full(n, -7, dtype))
    for _ in range(5):
        trtc.Reduce_By_Key(dk, minus, ko, vo, trtc.EqualTo(), trtc.Minimum())
        assert trtc.Reduce_By_Key(dk, dv, ko, vo, trtc.EqualTo(), f) == len(heads)
        assert vo.to_host(0, len(heads)).tobytes() == want.tobytes()
    assert bad.to_host()[0] == 0
