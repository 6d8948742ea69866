"""The tile pipeline finishes with one resident CTA, as the look-back kernels do: grids of one CTA (the
prefix CTA, which then does every tile itself) and of a few, against numpy."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hook(cuda):
    import torch
    from thrustrtc_b200 import _native as N
    f = N.lib.trtc_test_pipe_few_ctas
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_uint] + [ctypes.c_void_p] * 4 + [ctypes.c_ulonglong] + [ctypes.c_void_p] * 2

    def run(what, ctas, keys, x):
        n = len(x)
        dk, dx = torch.from_numpy(keys).cuda(), torch.from_numpy(x).cuda()
        a, b = torch.zeros_like(dx), torch.zeros_like(dx)
        c = ctypes.c_ulonglong(0)
        r = f(what, ctas, dk.data_ptr(), dx.data_ptr(), a.data_ptr(), b.data_ptr(), n, ctypes.addressof(c), None)
        assert r == 0, N.last_error()
        return a.cpu().numpy(), b.cpu().numpy(), c.value

    return run


def by_key(k, x, exclusive):
    heads = np.concatenate([[True], k[1:] != k[:-1]])
    s = np.cumsum(x, dtype=np.int64)
    start = np.flatnonzero(heads)[np.cumsum(heads) - 1]
    incl = s - (s[start] - x[start])
    return ((incl - x + 5) if exclusive else incl).astype(np.int32)


@pytest.mark.parametrize("ctas", [1, 2, 3])
@pytest.mark.parametrize("n,run", [(1, 1), (351, 3), (353, 5), (5119, 7), (5120, 9000), (5121, 2), (10_240, 33), (40_007, 1 << 30),
                                   (40_007, 4000), (300_001, 32)])
def test_grids_of_few_ctas(hook, ctas, n, run):
    if ctas > -(-n // 5120) + 1:
        pytest.skip("fewer tiles than workers")
    rng = np.random.default_rng(n + run)
    k = np.sort(rng.integers(0, max(1, n // run), n)).astype(np.int32)
    x = rng.integers(-1000, 1000, n).astype(np.int32)
    gone = 2**64 - 1
    for _ in range(2):
        # the scans are done by the prefix CTA alone
        assert hook(2, ctas, k, x)[0].tobytes() == by_key(k, x, False).tobytes()
        assert hook(3, ctas, k, x)[0].tobytes() == by_key(k, x, True).tobytes()
        # the others give up when it is alone, and leave the outputs as they were
        a, b, c = hook(0, ctas, k, x)
        odd = x[(x & 1) != 0]
        if ctas == 1:
            assert c == gone and not a.any() and not b.any()
        else:
            assert c == len(odd) and a[:c].tobytes() == odd.tobytes() and b[:n - c].tobytes() == x[(x & 1) == 0].tobytes()
        heads = np.flatnonzero(np.concatenate([[True], k[1:] != k[:-1]]))
        a, _, c = hook(1, ctas, k, k)
        assert c == gone if ctas == 1 else c == len(heads) and a[:c].tobytes() == k[heads].tobytes()
        a, b, c = hook(4, ctas, k, x)
        if ctas == 1:
            assert c == gone and not a.any() and not b.any()
        else:
            assert c == len(heads) and b[:c].tobytes() == k[heads].tobytes()
            assert a[:c].tobytes() == np.add.reduceat(x, heads).astype(np.int32).tobytes()


@pytest.mark.parametrize("call", ["copy_if", "remove", "reduce_by_key", "scan_by_key"])
def test_calls_beside_a_long_kernel(hook, call):
    # another stream's kernel holds the shared memory of all SMs but one for 400 ms: a call ends before it does
    import torch
    import thrustrtc_b200 as t
    from thrustrtc_b200 import _native as N
    N.lib.trtc_test_occupy.argtypes = [ctypes.c_uint] * 3 + [ctypes.c_void_p]
    t.init()
    n = 5_000_003 if call != "scan_by_key" else 7_000_003
    rng = np.random.default_rng(n)
    k = np.sort(rng.integers(0, n // 30, n)).astype(np.int32)
    x = rng.integers(0, 1000, n).astype(np.int32)
    dk, dx = t.device_vector_from_numpy(k), t.device_vector_from_numpy(x)
    a, b = t.device_vector_from_numpy(np.zeros(n, np.int32)), t.device_vector_from_numpy(np.zeros(n, np.int32))
    odd = t.Functor({}, ["x"], "        return (x & 1) != 0;\n")
    heads = np.flatnonzero(np.concatenate([[True], k[1:] != k[:-1]]))

    def run():
        if call == "copy_if":
            c = t.Copy_If(dx, a, odd)
            return c, x[(x & 1) != 0]
        if call == "remove":
            c = t.Remove_Copy(dx, a, t.DVInt32(7))
            return c, x[x != 7]
        if call == "reduce_by_key":
            c = t.Reduce_By_Key(dk, dx, b, a)
            return c, np.add.reduceat(x, heads).astype(np.int32)
        t.Inclusive_Scan_By_Key(dk, dx, a)
        t.Reduce(a.range(0, 1))  # (waits for the scan's stream only)
        return n, by_key(k, x, False)

    run()  # everything compiled and allocated
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    other, done = torch.cuda.Stream(), torch.cuda.Event()
    for warm in (True, False):  # (the first one compiles the general form)
        t.Fill(a, t.DVInt32(0))
        torch.cuda.synchronize()
        assert N.lib.trtc_test_occupy(sms - 1, 200 * 1024, 400_000, other.cuda_stream) == 0
        done.record(other)
        c, want = run()
        busy = not done.query()
        assert c == len(want) and a.to_host(0, c).tobytes() == want.tobytes()
        # (reduce_by_key's general form frees a vector, which waits for the whole device)
        assert warm or busy or call == "reduce_by_key"
    other.synchronize()
    c, want = run()
    assert c == len(want) and a.to_host(0, c).tobytes() == want.tobytes()


def test_waits_for_ring_room_do_not_hold_up_one_another(cuda):
    # runs whose results nearly fill the pipeline's ring three tiles deep: the longest waits for room.
    # 0.9 to 1.1 ms a call; up to 1.6 s while every waiting warp polled the error word in host memory
    # each 256 polls
    import torch
    import thrustrtc_b200 as t
    t.init()
    n = 50_000_000
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    k = torch.cumsum(torch.rand(n, device="cuda", generator=g) < 0.5, 0).to(torch.int64)
    x = torch.randint(0, 100, (n,), device="cuda", generator=g).to(torch.float64)
    ko, xo = torch.empty_like(k), torch.empty_like(x)
    v = [t.DVTorchVector(a, c) for a, c in ((k, "int64_t"), (x, "double"), (ko, "int64_t"), (xo, "double"))]
    t.Reduce_By_Key(*v)
    for _ in range(10):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        c = t.Reduce_By_Key(*v)
        b.record()
        torch.cuda.synchronize()
        assert a.elapsed_time(b) < 20
    keys, counts = torch.unique_consecutive(k, return_counts=True)
    assert c == keys.numel() and torch.equal(ko[:c], keys)
    assert float(xo[:c].sum()) == float(x.sum())
