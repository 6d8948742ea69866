"""Digit passes over many tiles per resident CTA: the payload stage is written by ordinary stores for one
tile and by a bulk copy for the next.  Payloads of 4 and 8 bytes, aligned (bulk copies) and not,
against numpy's stable sort."""
import ctypes
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_payload_stage_is_fenced_between_tiles():
    # a CTA barrier does not order ordinary shared-memory stores before a later bulk copy: a proxy fence
    # stands between the staging of a tile and the barrier that ends its turn of the tile loop
    src = open(os.path.join(ROOT, "thrustrtc_b200", "csrc", "device", "trtc_radix.cuh")).read()
    body = src[src.index("radix_pass_kernel(SortBufs"):]
    body = body[:re.search(r"^}", body, re.M).start()]
    assert body.count("bulk_load_g2s(s_vals") == 1
    turn_end = body[body.rindex("write_tile(BoolC<false>())"):]
    assert re.search(r"if constexpr \(VB\) smem_proxy_fence\(\);\s*__syncthreads\(\);\s*}\s*$", turn_end)


@pytest.mark.gpu
@pytest.mark.parametrize("kt,tc", [(np.uint32, 5), (np.float32, 8), (np.int64, 6)])
@pytest.mark.parametrize("vt", [np.int32, np.int64])
@pytest.mark.parametrize("off", [0, 1])
def test_many_tiles_per_cta(cuda, kt, tc, vt, off):
    import torch
    from thrustrtc_b200 import _native as N
    n = 592 * 5120 * 7 + 4099
    rng = np.random.default_rng(off)
    k = rng.standard_normal(n).astype(kt) if kt == np.float32 else rng.integers(0, 1 << 31, n).astype(kt)
    order = np.argsort(k, kind="stable")
    k0, v0 = torch.from_numpy(k.view({4: np.int32, 8: np.int64}[k.itemsize])).cuda(), torch.arange(off + n, device="cuda", dtype=torch.int32 if vt == np.int32 else torch.int64)
    for _ in range(3):
        tk, tv = k0.clone(), v0.clone()
        p = ctypes.c_void_p(tv.data_ptr() + off * vt().itemsize)
        assert N.lib.trtc_raw_sort_by_key(tc, ctypes.c_void_p(tk.data_ptr()), p, vt().itemsize, n, 0, None) == 0
        assert N.lib.trtc_raw_sync(None) == 0
        assert tk.cpu().numpy().tobytes() == k[order].tobytes()
        assert (tv[off:].cpu().numpy() == order + off).all()
