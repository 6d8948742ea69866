"""The calls whose speed this repository is measured by: what a program does with the library,
through its public entry points, over the sizes, types and options that such programs use.

``listed()`` names one case (three for the pair sort, the library's headline) of each family:

* calls         a chain of small calls, where launches and latency count;
* sort_pairs    Sort_By_Key of a built-in key type with 4-byte values;
* sort_keys     Sort of a built-in key type;
* sort_functor  Sort_By_Key under a user's comparator;
* scan          Inclusive_Scan / Exclusive_Scan;
* scan_by_key   Inclusive_Scan_By_Key / Exclusive_Scan_By_Key;
* reduce        Reduce, and Transform_Reduce with a user's map;
* reduce_by_key Reduce_By_Key;
* select        Copy_If / Remove_Copy_If with a user's predicate, Remove_Copy, Unique_Copy,
                Partition_Copy;
* segments      many uneven segments sorted and scanned by one call.

``draw(rng)`` gives one more case of a family.  Calls that work in place first take a fresh
copy of their input with Copy, as a program does whose data arrives in a buffer of its own.
Floating-point keys and elements that a call only moves are returned as their bit patterns,
outputs of a length that depends on the data as the whole buffer (zeros behind the end) and
the length.
"""
import ctypes
import math

import torch

import thrustrtc_b200 as trtc

DEV = "cuda"
TORCH = {"int32_t": torch.int32, "uint32_t": torch.int32, "int64_t": torch.int64, "uint64_t": torch.int64,
         "float": torch.float32, "double": torch.float64}
SIZE = {"int32_t": 4, "uint32_t": 4, "int64_t": 8, "uint64_t": 8, "float": 4, "double": 8}
SEG_KEY_TYPE = {"uint32_t": 5, "int64_t": 6, "float": 8}


def listed():
    return [
        # a small chain, as one step of a host-driven loop takes it: four calls of 4,000 elements
        {"name": "calls_4k", "family": "calls", "n": 4000},
        # an ordinary pair sort: ids of one frame, particles by cell
        {"name": "pairs_u32_1m", "family": "sort_pairs", "key": "uint32_t", "dist": "uniform", "descending": False,
         "n": 1 << 20},
        # the headline: 2^28 uniform 32-bit keys with their indices
        {"name": "pairs_u32_256m", "family": "sort_pairs", "key": "uint32_t", "dist": "uniform", "descending": False,
         "n": 1 << 28},
        # 64-bit ids of a skewed popularity, three of eight bytes varying, a ragged size
        {"name": "pairs_i64_zipf", "family": "sort_pairs", "key": "int64_t", "dist": "zipf", "descending": False,
         "n": 50_000_003},
        # scores with duplicates, negative zeros and NaNs, keys only
        {"name": "keys_f32_30m", "family": "sort_keys", "key": "float", "dist": "special", "descending": False,
         "n": 30_000_017},
        # an order that only the user knows: floats by magnitude, with their indices
        {"name": "sort_functor_4m", "family": "sort_functor", "key": "float", "n": 4_194_301},
        # the plain prefix sum at the benchmark's size
        {"name": "scan_i32_256m", "family": "scan", "value": "int32_t", "op": "Plus", "exclusive": False,
         "n": 1 << 28},
        # running sums within groups of mean length 32
        {"name": "scan_by_key_f32", "family": "scan_by_key", "key": "int32_t", "value": "float", "mean_run": 32,
         "exclusive": False, "n": 100_000_007},
        # sums of groups of mean length 32 (the step after a sort in a group-by)
        {"name": "reduce_by_key_f32", "family": "reduce_by_key", "key": "int32_t", "value": "float", "mean_run": 32,
         "n": 50_000_011},
        # a filter with a user's predicate, half of the elements kept
        {"name": "copy_if_functor", "family": "select", "kind": "copy_if", "value": "int32_t", "keep": 0.5,
         "n": 134_217_731},
        # a sum read back by the host
        {"name": "reduce_f32_16m", "family": "reduce", "value": "float", "op": "Plus", "map": False,
         "n": 16_777_259},
        # 100,000 uneven segments in one call
        {"name": "segments_100k", "family": "segments", "key": "uint32_t", "median": 256, "sigma": 1.5,
         "segments": 100_000},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    family = rng.choice(["calls", "sort_pairs", "sort_pairs", "sort_keys", "sort_functor", "scan", "scan_by_key",
                         "reduce_by_key", "select", "select", "reduce", "segments"])
    c = {"family": family}
    if family == "calls":
        c["n"] = _log_uniform(rng, 64, 16384)
    elif family == "sort_pairs":
        c["key"] = rng.choice(["uint32_t", "uint32_t", "int32_t", "int64_t", "float"])
        c["dist"] = "special" if c["key"] == "float" else rng.choice(["uniform", "zipf", "few"])
        c["descending"] = rng.random() < 0.3
        c["n"] = _log_uniform(rng, 1 << 10, 1 << 27)
    elif family == "sort_keys":
        c["key"] = rng.choice(["float", "uint32_t", "int32_t", "int64_t"])
        c["dist"] = "special" if c["key"] == "float" else rng.choice(["uniform", "few"])
        c["descending"] = rng.random() < 0.3
        c["n"] = _log_uniform(rng, 1 << 10, 1 << 27)
    elif family == "sort_functor":
        c["key"] = rng.choice(["float", "int32_t"])
        c["n"] = _log_uniform(rng, 1 << 10, 1 << 23)
    elif family == "scan":
        c["value"] = rng.choice(["int32_t", "float", "double", "int64_t"])
        c["op"] = rng.choice(["Plus", "Plus", "Maximum"])
        c["exclusive"] = rng.random() < 0.5
        c["n"] = _log_uniform(rng, 1 << 12, 1 << 27)
    elif family == "scan_by_key":
        c["key"] = rng.choice(["int32_t", "uint32_t"])
        c["value"] = rng.choice(["float", "int32_t", "double"])
        c["mean_run"] = rng.choice([3, 32, 1000])
        c["exclusive"] = rng.random() < 0.5
        c["n"] = _log_uniform(rng, 1 << 12, 1 << 27)
    elif family == "reduce_by_key":
        c["key"] = rng.choice(["int32_t", "uint32_t", "int64_t"])
        c["value"] = rng.choice(["float", "int32_t", "double"])
        c["mean_run"] = rng.choice([3, 32, 1000])
        c["n"] = _log_uniform(rng, 1 << 12, 1 << 27)
    elif family == "select":
        c["kind"] = rng.choice(["copy_if", "remove_if", "remove", "unique", "partition"])
        c["value"] = rng.choice(["int32_t", "float", "int64_t"])
        c["keep"] = rng.choice([0.05, 0.5, 0.9])
        c["n"] = _log_uniform(rng, 1 << 12, 1 << 27)
    elif family == "reduce":
        c["value"] = rng.choice(["float", "int32_t", "double"])
        c["op"] = rng.choice(["Plus", "Plus", "Maximum"])
        c["map"] = rng.random() < 0.3
        c["n"] = _log_uniform(rng, 1 << 12, 1 << 28)
    else:
        c["key"] = rng.choice(["uint32_t", "uint32_t", "float"])
        c["median"] = rng.choice([16, 64, 256])
        c["sigma"] = rng.choice([0.5, 1.0, 1.5])
        c["segments"] = _log_uniform(rng, 100, 100_000)
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform_bits(n, dtype, g):
    """Every bit pattern of the type's width, equally likely."""
    if dtype == torch.int64:
        lo = torch.randint(0, 1 << 32, (n,), generator=g, device=DEV, dtype=torch.int64)
        hi = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int64)
        return (hi << 32) | lo
    return torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int32)


def _keys(cls, dist, n, g):
    dt = TORCH[cls]
    if dist == "special":  # normal, one in ten a duplicate, -0.0 and NaN among them
        x = torch.randn(n, generator=g, device=DEV, dtype=torch.float32)
        r = torch.rand(n, generator=g, device=DEV)
        x = torch.where(r < 0.1, torch.round(x * 64.0) / 64.0, x)
        x = torch.where((r >= 0.1) & (r < 0.11), torch.tensor(-0.0, device=DEV), x)
        return torch.where((r >= 0.11) & (r < 0.111), torch.tensor(float("nan"), device=DEV), x)
    if dist == "few":
        return torch.randint(0, 1000, (n,), generator=g, device=DEV, dtype=dt)
    if dist == "zipf":  # 2^20 ids of a Zipf(1.1) popularity, scattered; 64-bit ones in one high range
        cdf = torch.cumsum(torch.arange(1, (1 << 20) + 1, device=DEV, dtype=torch.float64) ** -1.1, 0)
        cdf = cdf / cdf[-1].clone()
        r = torch.empty(n, device=DEV, dtype=torch.int64)
        for a in range(0, n, 1 << 25):
            u = torch.rand(min(1 << 25, n - a), generator=g, device=DEV, dtype=torch.float64)
            r[a:a + u.numel()] = torch.searchsorted(cdf, u)
        r = ((r + 1) * 0x9E3B1) & ((1 << 20) - 1)
        return r + 0x0123456700000000 if dt == torch.int64 else r.to(dt)
    return _uniform_bits(n, dt, g)


def _values(cls, n, g):
    dt = TORCH[cls]
    if dt.is_floating_point:
        return torch.rand(n, generator=g, device=DEV, dtype=dt)
    return torch.randint(-1000, 1001, (n,), generator=g, device=DEV, dtype=dt)


def _run_keys(cls, mean, n, g):
    """Ascending keys in runs of geometric length."""
    heads = torch.rand(n, generator=g, device=DEV) < 1.0 / mean
    return torch.cumsum(heads, 0, dtype=torch.int64).to(TORCH[cls])


def _segment_offsets(case, g):
    """Lognormal lengths at evenly spaced quantiles, in an order of the seed's."""
    count = case["segments"]
    q = (torch.randperm(count, generator=g, device=DEV).to(torch.float64) + 0.5) / count
    z = math.sqrt(2.0) * torch.erfinv(2.0 * q - 1.0)
    lens = torch.clamp(torch.round(torch.exp(math.log(case["median"]) + case["sigma"] * z)), 1, 1 << 20)
    off = torch.zeros(count + 1, device=DEV, dtype=torch.int64)
    off[1:] = torch.cumsum(lens.to(torch.int64), 0)
    return off


def _inputs(case, seed):
    """The case's input tensors, from the seed alone."""
    g, f, n = _gen(seed), case["family"], case.get("n", 0)
    if f == "calls":
        return {"k": _keys("uint32_t", "uniform", n, g), "x": _values("int32_t", n, g), "y": _values("float", n, g)}
    if f in ("sort_pairs", "sort_keys"):
        return {"k": _keys(case["key"], case["dist"], n, g)}
    if f == "sort_functor":
        if case["key"] == "float":
            return {"k": torch.randn(n, generator=g, device=DEV)}
        return {"k": torch.randint(-(1 << 20), 1 << 20, (n,), generator=g, device=DEV, dtype=torch.int32)}
    if f in ("scan", "reduce"):
        return {"x": _values(case["value"], n, g)}
    if f in ("scan_by_key", "reduce_by_key"):
        return {"k": _run_keys(case["key"], case["mean_run"], n, g), "x": _values(case["value"], n, g)}
    if f == "select":
        dt, keep = TORCH[case["value"]], case["keep"]
        if case["kind"] == "unique":
            return {"x": (_run_keys("int64_t", 1.0 / keep, n, g) & 0xFFFFF).to(dt)}
        if case["kind"] == "remove":  # a share of the elements is the value that is removed
            x = torch.randint(1, 1 << 20, (n,), generator=g, device=DEV, dtype=torch.int32)
            return {"x": torch.where(torch.rand(n, generator=g, device=DEV) < keep, x, torch.zeros_like(x)).to(dt)}
        return {"x": torch.randint(0, 1 << 20, (n,), generator=g, device=DEV, dtype=torch.int32).to(dt)}
    off = _segment_offsets(case, g)
    return {"off": off, "k": _keys(case["key"], "special" if case["key"] == "float" else "uniform", int(off[-1]), g)}


# ---------------------------------------------------------------- what a program has in hand
def _vec(t, cls):
    return trtc.DVTorchVector(t, cls)


def prepare(case, seed):
    trtc.init()
    s = {"case": dict(case), **_inputs(case, seed)}
    f = case["family"]
    if f == "calls":
        n = case["n"]
        s["v"] = torch.arange(n, device=DEV, dtype=torch.int32)
        for name, cls in (("k", "uint32_t"), ("v", "int32_t"), ("x", "int32_t")):
            s["d" + name], s["o" + name] = _vec(s[name], cls), torch.empty_like(s[name])
            s["do" + name] = _vec(s["o" + name], cls)
        s["sel"] = torch.zeros_like(s["x"])
        s["dsel"], s["dy"] = _vec(s["sel"], "int32_t"), _vec(s["y"], "float")
        s["pred"] = trtc.Functor({}, ["x"], "        return x > 0;\n")
    elif f in ("sort_pairs", "sort_keys", "sort_functor"):
        s["dk"], s["ok"] = _vec(s["k"], case["key"]), torch.empty_like(s["k"])
        s["dok"] = _vec(s["ok"], case["key"])
        if f != "sort_keys":
            s["v"] = torch.arange(case["n"], device=DEV, dtype=torch.int32)
            s["ov"] = torch.empty_like(s["v"])
            s["dv"], s["dov"] = _vec(s["v"], "uint32_t"), _vec(s["ov"], "uint32_t")
        if f == "sort_functor":
            s["comp"] = trtc.Functor({}, ["a", "b"], "        return (a < 0 ? -a : a) < (b < 0 ? -b : b);\n")
        else:
            s["comp"] = trtc.Greater() if case["descending"] else None
    elif f == "scan":
        s["out"] = torch.empty_like(s["x"])
        s["dx"], s["dout"] = _vec(s["x"], case["value"]), _vec(s["out"], case["value"])
        s["op"] = trtc.Maximum() if case["op"] == "Maximum" else None
        init = {"int32_t": trtc.DVInt32, "int64_t": trtc.DVInt64, "float": trtc.DVFloat, "double": trtc.DVDouble}
        s["init"] = init[case["value"]](0)
    elif f in ("scan_by_key", "reduce_by_key"):
        s["dk"], s["dx"] = _vec(s["k"], case["key"]), _vec(s["x"], case["value"])
        s["out"] = torch.zeros_like(s["x"])
        s["dout"] = _vec(s["out"], case["value"])
        if f == "reduce_by_key":
            s["kout"] = torch.zeros_like(s["k"])
            s["dkout"] = _vec(s["kout"], case["key"])
    elif f == "reduce":
        s["dx"] = _vec(s["x"], case["value"])
        s["op"] = trtc.Maximum() if case["op"] == "Maximum" else trtc.Plus()
        s["map"] = trtc.Functor({}, ["x"], "        return x * x;\n")
        s["init"] = {"int32_t": trtc.DVInt32, "float": trtc.DVFloat, "double": trtc.DVDouble}[case["value"]](0)
    elif f == "select":
        cls = case["value"]
        s["out"], s["rest"] = torch.zeros_like(s["x"]), torch.zeros_like(s["x"])
        s["dx"], s["dout"], s["drest"] = _vec(s["x"], cls), _vec(s["out"], cls), _vec(s["rest"], cls)
        s["limit"] = trtc.DVInt32(int(case["keep"] * (1 << 20)))
        sign = ">=" if case["kind"] == "remove_if" else "<"
        s["pred"] = trtc.Functor({"limit": s["limit"]}, ["x"], "        return x %s limit;\n" % sign)
        s["zero"] = {"int32_t": trtc.DVInt32, "int64_t": trtc.DVInt64, "float": trtc.DVFloat}[cls](0)
    else:
        n = s["k"].numel()
        s["v"] = torch.arange(n, device=DEV, dtype=torch.int32)
        s["ok"], s["ov"], s["out"] = torch.empty_like(s["k"]), torch.empty_like(s["v"]), torch.empty_like(s["v"])
        for name, cls in (("k", case["key"]), ("v", "uint32_t")):
            s["d" + name], s["do" + name] = _vec(s[name], cls), _vec(s["o" + name], cls)
        lib = trtc.lib
        lib.trtc_raw_segmented_workspace_bytes.restype = ctypes.c_ulonglong
        lib.trtc_raw_segmented_workspace_bytes.argtypes = [ctypes.c_int] + [ctypes.c_ulonglong] * 2
        lib.trtc_raw_segmented_sort_scan.restype = ctypes.c_int
        lib.trtc_raw_segmented_sort_scan.argtypes = (
            [ctypes.c_int] + [ctypes.c_void_p] * 4 + [ctypes.c_ulonglong] * 2 +
            [ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_int, ctypes.c_void_p])
        s["ws_bytes"] = lib.trtc_raw_segmented_workspace_bytes(SEG_KEY_TYPE[case["key"]], n, case["segments"])
        s["ws"] = torch.empty(s["ws_bytes"], device=DEV, dtype=torch.uint8)
    return s


# ---------------------------------------------------------------- one pass
def _bits(t):
    return t.view(torch.int32) if t.dtype == torch.float32 else t.view(torch.int64) if t.dtype == torch.float64 else t


def run(s):
    return globals()["_run_" + s["case"]["family"]](s, s["case"])


def _run_calls(s, c):
    trtc.Copy(s["dk"], s["dok"])
    trtc.Copy(s["dv"], s["dov"])
    trtc.Sort_By_Key(s["dok"], s["dov"])
    trtc.Inclusive_Scan(s["dx"], s["dox"])
    total = trtc.Reduce(s["dy"])
    kept = trtc.Copy_If(s["dx"], s["dsel"], s["pred"])
    return {"keys": s["ok"], "values": s["ov"], "scan": s["ox"], "total": total, "selected": s["sel"], "kept": kept}


def _run_sort_pairs(s, c):
    trtc.Copy(s["dk"], s["dok"])
    trtc.Copy(s["dv"], s["dov"])
    trtc.Sort_By_Key(s["dok"], s["dov"], s["comp"])
    return {"keys": _bits(s["ok"]), "values": s["ov"]}


_run_sort_functor = _run_sort_pairs


def _run_sort_keys(s, c):
    trtc.Copy(s["dk"], s["dok"])
    trtc.Sort(s["dok"], s["comp"])
    return {"keys": _bits(s["ok"])}


def _run_scan(s, c):
    if c["exclusive"]:
        trtc.Exclusive_Scan(s["dx"], s["dout"], s["init"], s["op"])
    else:
        trtc.Inclusive_Scan(s["dx"], s["dout"], s["op"])
    return {"out": s["out"]}


def _run_scan_by_key(s, c):
    if c["exclusive"]:
        trtc.Exclusive_Scan_By_Key(s["dk"], s["dx"], s["dout"])
    else:
        trtc.Inclusive_Scan_By_Key(s["dk"], s["dx"], s["dout"])
    return {"out": s["out"]}


def _run_reduce_by_key(s, c):
    groups = trtc.Reduce_By_Key(s["dk"], s["dx"], s["dkout"], s["dout"])
    return {"keys": s["kout"], "out": s["out"], "groups": groups}


def _run_reduce(s, c):
    if c["map"]:
        return {"out": trtc.Transform_Reduce(s["dx"], s["map"], s["init"], s["op"])}
    return {"out": trtc.Reduce(s["dx"], s["init"], s["op"])}


def _run_select(s, c):
    kind = c["kind"]
    if kind == "copy_if":
        kept = trtc.Copy_If(s["dx"], s["dout"], s["pred"])
    elif kind == "remove_if":
        kept = trtc.Remove_Copy_If(s["dx"], s["dout"], s["pred"])
    elif kind == "remove":
        kept = trtc.Remove_Copy(s["dx"], s["dout"], s["zero"])
    elif kind == "unique":
        kept = trtc.Unique_Copy(s["dx"], s["dout"])
    else:
        kept = trtc.Partition_Copy(s["dx"], s["dout"], s["drest"], s["pred"])
        return {"out": _bits(s["out"]), "rest": _bits(s["rest"]), "kept": kept}
    return {"out": _bits(s["out"]), "kept": kept}


def _run_segments(s, c):
    trtc.Copy(s["dk"], s["dok"])
    trtc.Copy(s["dv"], s["dov"])
    trtc.check_i(trtc.lib.trtc_raw_segmented_sort_scan(
        SEG_KEY_TYPE[c["key"]], s["ok"].data_ptr(), s["ov"].data_ptr(), s["out"].data_ptr(), s["off"].data_ptr(),
        c["segments"], s["k"].numel(), s["ws"].data_ptr(), s["ws_bytes"], 0, None))
    return {"keys": _bits(s["ok"]), "values": s["ov"], "scan": s["out"]}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    f, n = case["family"], case.get("n", 0)
    if f == "calls":  # keys and values, the scan, the sum, the filter (half kept)
        return {"bytes": n * (16 + 8 + 4 + 6), "flops": 0}
    if f in ("sort_pairs", "sort_functor"):
        return {"bytes": 2 * n * (SIZE[case["key"]] + 4), "flops": 0}
    if f == "sort_keys":
        return {"bytes": 2 * n * SIZE[case["key"]], "flops": 0}
    if f == "scan":
        return {"bytes": 2 * n * SIZE[case["value"]], "flops": n}
    if f == "scan_by_key":
        return {"bytes": n * (SIZE[case["key"]] + 2 * SIZE[case["value"]]), "flops": n}
    if f == "reduce_by_key":
        return {"bytes": n * (SIZE[case["key"]] + SIZE[case["value"]]) * (1 + 1 / case["mean_run"]), "flops": n}
    if f == "reduce":
        return {"bytes": n * SIZE[case["value"]], "flops": n}
    if f == "select":
        kept = 1 if case["kind"] == "partition" else case["keep"]
        return {"bytes": n * SIZE[case["value"]] * (1 + kept), "flops": 0}
    mean = case["median"] * math.exp(case["sigma"] ** 2 / 2)  # of the lognormal lengths
    return {"bytes": case["segments"] * mean * (2 * (SIZE[case["key"]] + 4) + 4), "flops": 0}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """What run() computes (rather than moves), by torch in 64 bits; None where it only moves."""
    f = case["family"]
    if f == "calls":
        y = _inputs(case, seed)["y"]
        return {"keys": None, "values": None, "scan": None, "total": float(y.to(torch.float64).sum()),
                "selected": None, "kept": None}
    if f not in ("scan", "reduce", "scan_by_key", "reduce_by_key") or not TORCH[case["value"]].is_floating_point:
        return None
    i = _inputs(case, seed)
    x = i["x"].to(torch.float64)
    if f == "reduce":
        x = x * x if case["map"] else x
        return {"out": float(x.max() if case["op"] == "Maximum" else x.sum())}
    if f == "scan":
        y = torch.cummax(x, 0).values if case["op"] == "Maximum" else torch.cumsum(x, 0)
        if case["exclusive"]:
            y = torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), y[:-1]])
        return {"out": y}
    seg = (i["k"].to(torch.int64) - i["k"][0].to(torch.int64))
    groups = int(seg[-1]) + 1
    if f == "reduce_by_key":
        return {"keys": None, "out": torch.zeros_like(x).index_add_(0, seg, x), "groups": None}
    y = torch.cumsum(x, 0)
    before = torch.zeros(groups + 1, device=DEV, dtype=torch.float64)  # the sum before each group
    before[1:] = torch.zeros(groups, device=DEV, dtype=torch.float64).index_add_(0, seg, x).cumsum(0)
    y = y - before[seg]
    return {"out": y - x if case["exclusive"] else y}
