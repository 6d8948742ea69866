"""Short sorts (one launch): both sides of every change of shape, all key types, payload widths
and orders, floats with -0.0 and NaN anywhere, against the oracle."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TC = {np.int8: 0, np.uint8: 1, np.int16: 2, np.uint16: 3, np.int32: 4, np.uint32: 5, np.int64: 6, np.uint64: 7,
      np.float32: 8, np.float64: 9}


@pytest.fixture(scope="module")
def N(cuda):
    from thrustrtc_b200 import _native as N
    return N


def _dev(a):
    import torch
    return torch.from_numpy(a.view(np.uint8).copy()).cuda()


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def keys_of(rng, dtype, n):
    if np.issubdtype(dtype, np.floating):
        x = (rng.standard_normal(n) * 3).astype(dtype)
        x[rng.random(n) < 0.1] = -0.0
        x[rng.random(n) < 0.1] = 0.0
        x[rng.random(n) < 0.1] = dtype(1.5)
        return x
    info = np.iinfo(dtype)
    return rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True)


def check(N, k, vsize, desc):
    n = len(k)
    tk = _dev(k)
    if vsize == 0:
        assert N.lib.trtc_raw_sort(TC[k.dtype.type], _p(tk), n, int(desc), None) == 0
        assert N.lib.trtc_raw_sync(None) == 0
        assert tk.cpu().numpy().tobytes() == O.sort(k, desc).tobytes()
        return
    v = np.arange(n, dtype=np.int64)
    ek, ev = O.sort_by_key(k, v, desc)
    raw = v.view(np.uint8).reshape(n, 8)
    raw = np.ascontiguousarray(raw[:, :vsize] if vsize <= 8 else np.concatenate([raw, raw[:, : vsize - 8]], 1))
    tv = _dev(raw.reshape(-1))
    assert N.lib.trtc_raw_sort_by_key(TC[k.dtype.type], _p(tk), _p(tv), vsize, n, int(desc), None) == 0
    assert N.lib.trtc_raw_sync(None) == 0
    assert tk.cpu().numpy().tobytes() == ek.tobytes()
    assert tv.cpu().numpy().tobytes() == raw[ev].tobytes()


@pytest.mark.parametrize("n", [2, 31, 33, 255, 257, 1023, 1024, 1025, 2048, 2049, 4097, 8191, 8192, 8193, 12289, 16384, 16385, 32768, 32769])
@pytest.mark.parametrize("dtype", [np.uint32, np.int64, np.float32])
def test_sizes(N, n, dtype):
    rng = np.random.default_rng(n)
    k = keys_of(rng, dtype, n)
    for vsize, desc in ((0, False), (4, False), (8, True)):
        check(N, k, vsize, desc)


@pytest.mark.parametrize("dtype", sorted(TC, key=TC.get))
@pytest.mark.parametrize("vsize", [0, 1, 4, 8, 12])
def test_types_and_payloads(N, dtype, vsize):
    rng = np.random.default_rng(vsize)
    for n in (700, 5000):
        for desc in (False, True):
            check(N, keys_of(rng, dtype, n), vsize, desc)
    # keys of one value, of few values, and with constant high bytes
    check(N, np.full(3000, 7, dtype), vsize, False)
    check(N, rng.integers(0, 3, 3000).astype(dtype), vsize, True)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 200, 256, 257, 3000, 8000, 30000])
@pytest.mark.parametrize("where", ["first", "some", "all"])
def test_nan(N, dtype, n, where):
    rng = np.random.default_rng(n)
    x = keys_of(rng, dtype, n)
    if where == "first":
        x[0] = np.nan
    elif where == "some":
        x[rng.random(n) < 0.05] = np.nan
        x[rng.random(n) < 0.02] = -np.nan
    else:
        x[:] = np.nan
    for desc in (False, True):
        check(N, x, 0, desc)
        check(N, x, 4, desc)
