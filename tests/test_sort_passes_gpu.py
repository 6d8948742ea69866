"""The digit passes on both sides of one tile per resident CTA, with 0 to 3 digits that move data
(none, one -- whose result is copied back -- and an odd and an even number of passes), against
numpy's stable sort."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 4 CTAs on each of 148 SMs take tiles of 5120 4-byte or 3072 8-byte keys
EDGE32, EDGE64 = 592 * 5120, 592 * 3072


@pytest.fixture(scope="module")
def N(cuda):
    from thrustrtc_b200 import _native as N
    return N


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n", [300_001, EDGE32 - 1, EDGE32 + 1, 2 * EDGE32 + 7])
@pytest.mark.parametrize("mask", [0x0, 0xFF00, 0xFF0000FF, 0x00FFFFFF])
@pytest.mark.parametrize("pairs", [False, True])
def test_32_bit_keys(N, n, mask, pairs):
    import torch
    rng = np.random.default_rng(n)
    k = (rng.integers(0, 1 << 32, n, dtype=np.uint32) & np.uint32(mask)) | np.uint32(0x01020304 & ~mask & 0xFFFFFFFF)
    tk = torch.from_numpy(k.view(np.int32)).cuda()
    tv = torch.arange(n, dtype=torch.int32, device="cuda")
    if pairs:
        assert N.lib.trtc_raw_sort_by_key(5, _p(tk), _p(tv), 4, n, 0, None) == 0
    else:
        assert N.lib.trtc_raw_sort(5, _p(tk), n, 0, None) == 0
    assert N.lib.trtc_raw_sync(None) == 0
    order = np.argsort(k, kind="stable")
    assert tk.cpu().numpy().view(np.uint32).tobytes() == k[order].tobytes()
    if pairs:
        assert tv.cpu().numpy().tobytes() == order.astype(np.int32).tobytes()


@pytest.mark.parametrize("n", [EDGE64 - 1, EDGE64 + 1])
@pytest.mark.parametrize("mask", [0xFF000000, 0xFF000000FF00, 0x00FFFFFF])
def test_64_bit_keys(N, n, mask):
    import torch
    rng = np.random.default_rng(n)
    k = rng.integers(-(1 << 62), 1 << 62, n, dtype=np.int64) & np.int64(mask) | np.int64(0x0123 << 48)
    tk = torch.from_numpy(k).cuda()
    tv = torch.arange(n, dtype=torch.int32, device="cuda")
    assert N.lib.trtc_raw_sort_by_key(6, _p(tk), _p(tv), 4, n, 0, None) == 0
    assert N.lib.trtc_raw_sync(None) == 0
    order = np.argsort(k, kind="stable")
    assert tk.cpu().numpy().tobytes() == k[order].tobytes()
    assert tv.cpu().numpy().tobytes() == order.astype(np.int32).tobytes()
