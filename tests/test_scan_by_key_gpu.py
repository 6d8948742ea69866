"""Scan_By_Key on the tile pipeline: tile edges, several turns of its ring, segments shorter and
longer than tiles, key and value widths, alignment, in place, both modes.  Integer-valued data, so
that every result is exact, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    return t


def expected(k, v, init=None):
    n = len(k)
    c = np.cumsum(v.astype(np.float64))
    heads = np.concatenate([[True], k[1:] != k[:-1]])
    start = np.maximum.accumulate(np.where(heads, np.arange(n), 0))
    before = np.where(start > 0, c[np.maximum(start, 1) - 1], 0.0)
    inc = c - before
    if init is None:
        return inc.astype(v.dtype)
    return (inc - v.astype(np.float64) + init).astype(v.dtype)


def run_keys(rng, n, mean, dtype):
    k = np.cumsum(rng.random(n) < 1.0 / mean) if mean else np.zeros(n)
    return k.astype(dtype)


# the pipeline starts at 48 MiB of keys and values (4 + 4 bytes: 6,291,456 elements); tiles of 5120
# elements, 2560 of more than 8 bytes
EDGE = -(-6_291_456 // 5120) * 5120
SIZES = [1, 5121, 6_291_455, 6_291_456, EDGE, EDGE + 1, EDGE + 19, EDGE + 2561, EDGE + 5119, 5120 * 148 * 40 + 9]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("mean", [0, 1, 3, 1000, 20_000])
def test_sizes_and_runs(trtc, n, mean):
    rng = np.random.default_rng(n + mean)
    k, v = run_keys(rng, n, mean, np.int32), rng.integers(0, 4, n).astype(np.float32)
    if mean == 0 or mean == 20_000:
        v[:] = 0
        v[:: max(1, n // 1000)] = 1  # sums stay exact in float32
    dk, dv, do = (trtc.device_vector_from_numpy(a) for a in (k, v, np.full(n, 77, np.float32)))
    trtc.Inclusive_Scan_By_Key(dk, dv, do)
    assert do.to_host().tobytes() == expected(k, v).tobytes()
    trtc.Exclusive_Scan_By_Key(dk, dv, do, trtc.DVFloat(5.0))
    assert do.to_host().tobytes() == expected(k, v, 5.0).tobytes()
    trtc.Exclusive_Scan_By_Key(dk, dv, do)
    assert do.to_host().tobytes() == expected(k, v, 0.0).tobytes()
    trtc.Inclusive_Scan_By_Key(dk, dv, dv)  # in place
    assert dv.to_host().tobytes() == expected(k, v).tobytes()


@pytest.mark.parametrize("kt", [np.int32, np.uint32, np.int64])
@pytest.mark.parametrize("vt", [np.int32, np.uint32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("n", [2561, 6_300_001])
def test_types(trtc, kt, vt, n):
    rng = np.random.default_rng(n)
    init = {np.int32: trtc.DVInt32, np.uint32: trtc.DVUInt32, np.int64: trtc.DVInt64, np.float32: trtc.DVFloat,
            np.float64: trtc.DVDouble}[vt]
    for mean in (0, 7, 5000):  # (one segment: few nonzero values, exact in float32)
        k, v = run_keys(rng, n, mean, kt), (rng.integers(0, 9, n) * (rng.random(n) < (1 if mean else 0.01))).astype(vt)
        dk, dv, do = (trtc.device_vector_from_numpy(a) for a in (k, v, np.zeros(n, vt)))
        trtc.Inclusive_Scan_By_Key(dk, dv, do)
        assert do.to_host().tobytes() == expected(k, v).tobytes()
        trtc.Exclusive_Scan_By_Key(dk, dv, do, init(3))
        assert do.to_host().tobytes() == expected(k, v, 3).tobytes()


@pytest.mark.parametrize("off", [1, 2, 3])
def test_unaligned_ranges(trtc, off):
    n = 7_000_011
    rng = np.random.default_rng(off)
    k, v = run_keys(rng, n + off, 9, np.int32), rng.integers(0, 9, n + off).astype(np.int32)
    dk, dv, do = (trtc.device_vector_from_numpy(a) for a in (k, v, np.full(n + off, 77, np.int32)))
    trtc.Inclusive_Scan_By_Key(dk.range(off, n + off), dv.range(off, n + off), do.range(off, n + off))
    out = do.to_host()
    assert (out[:off] == 77).all() and out[off:].tobytes() == expected(k[off:], v[off:]).tobytes()
    full = trtc.device_vector_from_numpy(np.zeros(n, np.int32))
    trtc.Exclusive_Scan_By_Key(dk.range(off, n + off), dv.range(off, n + off), full)
    assert full.to_host().tobytes() == expected(k[off:], v[off:], 0).tobytes()


def test_output_over_the_keys_takes_the_general_form(trtc):
    n = 20_000
    rng = np.random.default_rng(3)
    k, v = run_keys(rng, n, 5, np.int32), rng.integers(0, 9, n).astype(np.int32)
    dk, dv = trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v)
    trtc.Inclusive_Scan_By_Key(dk, dv, dk)
    assert dk.to_host().tobytes() == expected(k, v).tobytes()
