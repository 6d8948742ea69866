"""Reduce and Transform_Reduce around the steps of loads that a thread keeps in flight (1, 4 and 16
vectors of 16 bytes on the full grid), with and without an initial value: integers exactly, floats
(integer-valued, sums below 2^24) exactly as well."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = 148 * 4 * 256  # threads of the full grid


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    return t


SIZES = [1, 3, 4, 5, 1023, 1025] + [GRID * 4 * k + d for k in (1, 4, 5, 16, 21) for d in (-1, 0, 3)]


@pytest.mark.parametrize("n", SIZES)
def test_sums(trtc, n):
    rng = np.random.default_rng(n)
    x = rng.integers(-1000, 1001, n).astype(np.int32)
    d = trtc.device_vector_from_numpy(x)
    total = int(x.astype(np.int64).sum())
    wrap = lambda v: (v + 2**31) % 2**32 - 2**31  # noqa: E731
    assert trtc.Reduce(d) == wrap(total)
    assert trtc.Reduce(d, trtc.DVInt32(7), trtc.Plus()) == wrap(total + 7)
    assert trtc.Reduce(d, trtc.DVInt32(-2000), trtc.Maximum()) == int(x.max())
    if n > 1:  # an unaligned start
        assert trtc.Reduce(d.range(1, n)) == wrap(total - int(x[0]))
    sq = trtc.Functor({}, ["x"], "        return x * x;\n")
    want = int((x.astype(np.int64) ** 2).sum())
    assert trtc.Transform_Reduce(d, sq, trtc.DVInt64(5), trtc.Plus()) == want + 5  # (the map in 32 bits, the sum in 64)


@pytest.mark.parametrize("n", [1000, GRID * 4 * 5 + 3])
def test_map_in_the_type_of_the_initial_value(trtc, n):
    rng = np.random.default_rng(n)
    x = np.zeros(n, np.float32)
    x[rng.integers(0, n, 500)] = 3.0
    d = trtc.device_vector_from_numpy(x)
    half = trtc.Functor({}, ["x"], "        return x * 0.5f;\n")
    want = float((x * 0.5).astype(np.float64).sum())
    assert trtc.Transform_Reduce(d, half, trtc.DVFloat(1.0), trtc.Plus()) == want + 1.0
    assert trtc.Transform_Reduce(d, half, trtc.DVDouble(1.0), trtc.Plus()) == want + 1.0
    assert trtc.Transform_Reduce(d, half, trtc.DVInt32(0), trtc.Plus()) == int((x * 0.5).astype(np.int32).sum())
    assert trtc.Transform_Reduce(d, half, trtc.DVFloat(-1.0), trtc.Maximum()) == float((x * 0.5).max())
    # an operator of the user keeps its order
    last = trtc.Functor({}, ["a", "b"], "        return b;\n")
    assert trtc.Transform_Reduce(d, half, trtc.DVFloat(0.0), last) == float(x[-1] * 0.5)
