"""Sort / Sort_By_Key under a user comparator (the merge sort) at the edges of its tiles: one
element to several merge levels, every key width its tile shape depends on, against a stable
numpy sort of the same order.  Few distinct codes, so that ties show a lost stability."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    return t


SIZES = [2, 15, 17, 255, 4095, 4096, 4097, 8191, 8193, 12289, 40000, 4096 * 33 + 5]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.int64, np.float64, np.int16])
def test_pairs_by_magnitude(trtc, n, dtype):
    rng = np.random.default_rng(n)
    k = rng.integers(-300, 301, n).astype(dtype)
    v = np.arange(n, dtype=np.int64 if dtype == np.int32 else np.int32)
    comp = trtc.Functor({}, ["a", "b"], "        return (a < 0 ? -a : a) < (b < 0 ? -b : b);\n")
    dk, dv = trtc.device_vector_from_numpy(k), trtc.device_vector_from_numpy(v)
    trtc.Sort_By_Key(dk, dv, comp)
    order = np.argsort(np.abs(k.astype(np.float64)), kind="stable")
    assert dk.to_host().tobytes() == k[order].tobytes()
    assert dv.to_host().tobytes() == v[order].tobytes()


@pytest.mark.parametrize("n", SIZES)
def test_keys_only_and_ranges(trtc, n):
    rng = np.random.default_rng(n)
    k = rng.integers(0, 1 << 30, n).astype(np.int32)
    comp = trtc.Functor({}, ["a", "b"], "        return (a & 1023) < (b & 1023);\n")
    d = trtc.device_vector_from_numpy(np.concatenate([[7], k, [9]]).astype(np.int32))
    trtc.Sort(d.range(1, n + 1), comp)
    out = d.to_host()
    assert out[0] == 7 and out[-1] == 9
    assert out[1:-1].tobytes() == k[np.argsort(k & 1023, kind="stable")].tobytes()


@pytest.mark.parametrize("fields", [["int32_t"] * 2, ["double"] * 2, ["double"] * 4, ["double"] * 6, ["double"] * 9])
@pytest.mark.parametrize("n", [300, 2049, 5000])
def test_wide_keys(trtc, fields, n):
    """Zipped keys of 8 to 72 bytes: 16 to 1 elements per thread."""
    rng = np.random.default_rng(n + len(fields))
    cols = [rng.integers(0, 50, n).astype({"int32_t": np.int32, "double": np.float64}[f]) for f in fields]
    names = ["f%d" % i for i in range(len(fields))]
    vecs = [trtc.device_vector_from_numpy(c) for c in cols]
    v = np.arange(n, dtype=np.int32)
    dv = trtc.device_vector_from_numpy(v)
    comp = trtc.Functor({}, ["a", "b"], "        return a.f1 < b.f1;\n")
    trtc.Sort_By_Key(trtc.DVZipped(vecs, names), dv, comp)
    order = np.argsort(cols[1], kind="stable")
    assert dv.to_host().tobytes() == v[order].tobytes()
    for d, c in zip(vecs, cols):
        assert d.to_host().tobytes() == c[order].tobytes()


def test_inconsistent_comparator_stays_in_bounds(trtc):
    """A comparator that is no order leaves some arrangement of values of the input and no error."""
    n = 20000
    k = np.arange(n, dtype=np.int32)
    d = trtc.device_vector_from_numpy(k)
    trtc.Sort(d, trtc.Functor({}, ["a", "b"], "        return ((a * 2654435761u) ^ (b * 40503u)) & 1;\n"))
    out = d.to_host()
    assert out.min() >= 0 and out.max() < n
