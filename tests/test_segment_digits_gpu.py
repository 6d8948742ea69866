"""Segmented sort: segments sorted by the top bits of those that vary, their ties finished in
place, and the segments that have to take all bits (clustered keys, long tied runs).  Oracle:
the per-segment stable sort and prefix sum on the host, exact."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TC = {"uint32_t": 5, "int64_t": 6, "float": 8}
NP = {"uint32_t": np.uint32, "int64_t": np.int64, "float": np.float32}
# one warp's, a group's, the CTA's and the global path's ends; 2^14: three digits from here on
LENGTHS = [33, 100, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097, 16384, 16385, 40000]


def bits(rng, kind, n, width):
    """n unsigned codes of `width` bits."""
    u = rng.integers(0, 2**width, n, dtype=np.uint64, endpoint=False)
    if kind == "uniform":
        return u
    if kind == "ties":      # neighbours that agree in their top half, the larger one first
        u[1::2] = u[0:-1:2][:len(u[1::2])] & ~np.uint64(0xF)
        return u
    if kind == "hidden":    # the first 32 keys say nothing about the rest: four tied runs, reversed
        r = u.copy()
        m = max(0, n - 32)
        r[32:] = (np.arange(m, dtype=np.uint64) % np.uint64(4) << np.uint64(width - 4)) | \
            np.arange(m, 0, -1, dtype=np.uint64)
        return r
    if kind == "runs":      # tied runs of about 20, just past what is finished in place
        return (rng.integers(0, max(1, n // 20), n).astype(np.uint64) << np.uint64(width - 12)) ^ \
            (u & np.uint64(0xFF))
    if kind == "few":
        return rng.integers(0, 7, n).astype(np.uint64) << np.uint64(width - 3)
    if kind == "equal":
        return np.full(n, 5, np.uint64)
    if kind == "outlier":   # one key above all the others' bits, where no sample looks
        u >>= np.uint64(width - 16)
        u[n - 1] |= np.uint64(1) << np.uint64(width - 3)
        return u
    if kind == "narrow":    # 17 varying bits under a common top
        return (u & np.uint64(0x1FFFF)) | (np.uint64(1) << np.uint64(width - 2))
    return np.sort(u)[::-1].copy()


KINDS = ["uniform", "ties", "hidden", "runs", "few", "equal", "narrow", "outlier", "reversed"]


def keys_of(rng, name, kind, n):
    if name == "int64_t":
        return bits(rng, kind, n, 64).view(np.int64)
    u = bits(rng, kind, n, 32).astype(np.uint32)
    if name == "float":
        f = u.view(np.float32).copy()
        f[np.isnan(f)] = -0.0
        return f
    return u


@pytest.mark.parametrize("items", [8, 16])
@pytest.mark.parametrize("desc", [False, True])
@pytest.mark.parametrize("name", ["uint32_t", "int64_t", "float"])
def test_segments_by_their_top_bits(name, desc, items):
    import torch
    from oracle import oracle as O
    from thrustrtc_b200 import _native as N
    rng = np.random.default_rng(3)
    parts = [keys_of(rng, name, kind, n) for n in LENGTHS for kind in KINDS]
    parts = [parts[i] for i in rng.permutation(len(parts))]
    off = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.int64)
    keys = np.concatenate(parts)
    n, nseg = len(keys), len(parts)
    vals = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    ek, ev, es = keys.copy(), vals.copy(), np.zeros_like(vals)
    for a, b in zip(off[:-1], off[1:]):
        ek[a:b], ev[a:b] = O.sort_by_key(keys[a:b], vals[a:b], desc)
        c = np.cumsum(ev[a:b].astype(np.uint64)) & 0xFFFFFFFF
        es[a:b] = np.concatenate([[0], c[:-1]]).astype(np.uint32)

    L = N.lib
    L.trtc_raw_segmented_workspace_bytes.restype = ctypes.c_ulonglong
    L.trtc_raw_segmented_workspace_bytes.argtypes = [ctypes.c_int, ctypes.c_ulonglong, ctypes.c_ulonglong]
    L.trtc_raw_segmented_sort_scan.restype = ctypes.c_int
    L.trtc_raw_segmented_sort_scan.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 4 + \
        [ctypes.c_ulonglong, ctypes.c_ulonglong, ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_int, ctypes.c_void_p]
    L.trtc_raw_segmented_tuning_json.restype = ctypes.c_ulonglong
    L.trtc_raw_segmented_tuning_json.argtypes = [ctypes.c_char_p, ctypes.c_ulonglong]
    L.trtc_raw_segmented_tuning_load.restype = ctypes.c_int
    L.trtc_raw_segmented_tuning_load.argtypes = [ctypes.c_char_p]
    buf = ctypes.create_string_buffer(1 << 16)
    L.trtc_raw_segmented_tuning_json(buf, len(buf))
    saved = buf.value
    tk = torch.from_numpy(keys.view(np.int64 if keys.dtype.itemsize == 8 else np.int32)).cuda()
    tv = torch.from_numpy(vals.view(np.int32)).cuda()
    ts = torch.full_like(tv, -1)
    to = torch.from_numpy(off).cuda()
    wsb = L.trtc_raw_segmented_workspace_bytes(TC[name], n, nseg)
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    try:
        table = ('{"format": "thrustrtc_b200.segmented_tuning", "version": 1, "entries": '
                 '[{"key_type": %d, "items": %d, "warp_small": 32}]}' % (TC[name], items))
        assert L.trtc_raw_segmented_tuning_load(table.encode()) == 0
        rc = L.trtc_raw_segmented_sort_scan(TC[name], p(tk), p(tv), p(ts), p(to), nseg, n, p(ws), wsb, int(desc), None)
        assert rc == 0, N.last_error()
        torch.cuda.synchronize()
    finally:
        L.trtc_raw_segmented_tuning_load(saved)
    assert tk.cpu().numpy().tobytes() == ek.tobytes()
    assert np.array_equal(tv.cpu().numpy().view(np.uint32), ev)
    assert np.array_equal(ts.cpu().numpy().view(np.uint32), es)
