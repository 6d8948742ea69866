"""The compaction pipeline at the edges of its range and tiles and over many turns of its ring: every
selection mode it takes, 4- and 8-byte elements, kept shares from none to all, partitions,
unaligned ranges, outputs that are too short, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    return t


# the pipeline starts at 2^22 elements; tiles of 5120 4-byte and 2560 8-byte elements
EDGE = -(-(1 << 22) // 5120) * 5120
SIZES = [1, 4097, (1 << 22) - 1, 1 << 22, EDGE - 1, EDGE, EDGE + 1, EDGE + 19, EDGE + 2559, EDGE + 2561, 5120 * 148 * 40 + 9]


def check(trtc, got, out, want):
    assert got == len(want)
    h = out.to_host()
    assert h[:got].tobytes() == want.tobytes()
    assert (h[got:] == 77).all()  # nothing written behind the end


def dest(trtc, n, dtype):
    return trtc.device_vector_from_numpy(np.full(n, 77, dtype))


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.int64, np.float64])
def test_modes(trtc, n, dtype):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 1000, n).astype(dtype)
    d = trtc.device_vector_from_numpy(x)
    for limit in (0, 50, 500, 1000):
        f = trtc.Functor({"l": trtc.DVInt32(limit)}, ["x"], "        return x < l;\n")
        o = dest(trtc, n, dtype)
        check(trtc, trtc.Copy_If(d, o, f), o, x[x < limit])
        o = dest(trtc, n, dtype)
        check(trtc, trtc.Remove_Copy_If(d, o, f), o, x[~(x < limit)])
        o, r = dest(trtc, n, dtype), dest(trtc, n, dtype)
        c = trtc.Partition_Copy(d, o, r, f)
        check(trtc, c, o, x[x < limit])
        check(trtc, n - c, r, x[~(x < limit)])
    y = x % 4
    d = trtc.device_vector_from_numpy(y)
    o = dest(trtc, n, dtype)
    check(trtc, trtc.Remove_Copy(d, o, trtc.DVInt32(2)), o, y[y != 2])
    z = np.sort(x)
    d = trtc.device_vector_from_numpy(z)
    heads = np.concatenate([[True], z[1:] != z[:-1]])
    o = dest(trtc, n, dtype)
    check(trtc, trtc.Unique_Copy(d, o), o, z[heads])
    o = dest(trtc, n, dtype)
    near = trtc.Functor({}, ["a", "b"], "        return (int)a / 2 == (int)b / 2;\n")
    w = z.astype(np.int64) // 2
    check(trtc, trtc.Unique_Copy(d, o, near), o, z[np.concatenate([[True], w[1:] != w[:-1]])])


@pytest.mark.parametrize("off", [1, 2, 3])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_unaligned_ranges_and_in_place(trtc, off, dtype):
    n = (1 << 22) + 33_333
    rng = np.random.default_rng(off)
    x = np.sort(rng.integers(0, 400_000, n + off)).astype(dtype)
    d = trtc.device_vector_from_numpy(x)
    v = x[off:]
    o = dest(trtc, n, dtype)
    heads = np.concatenate([[True], v[1:] != v[:-1]])
    check(trtc, trtc.Unique_Copy(d.range(off, n + off), o), o, v[heads])
    odd = trtc.Functor({}, ["x"], "        return (x & 1) != 0;\n")
    c = trtc.Remove_If(d.range(off, n + off), odd)
    want = v[(v & 1) == 0]
    assert c == len(want) and d.to_host()[off:off + c].tobytes() == want.tobytes()


def test_short_outputs_are_filled_to_their_end(trtc):
    x = np.arange(5_000_000, dtype=np.int32)
    d = trtc.device_vector_from_numpy(x)
    even = trtc.Functor({}, ["x"], "        return (x & 1) == 0;\n")
    o, r = dest(trtc, 7001, np.int32), dest(trtc, 333, np.int32)
    assert trtc.Copy_If(d, o, even) == 2_500_000 and o.to_host().tobytes() == x[::2][:7001].tobytes()
    assert trtc.Partition_Copy(d, o, r, even) == 2_500_000 and r.to_host().tobytes() == x[1::2][:333].tobytes()
