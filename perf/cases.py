"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the public entry points of gqs_ctypes (the binding of include/gqs.h):

  sort      Context.sort_dev: one array of keys in device memory, sorted in place
  pairs     Context.sort_pairs_dev: keys with their values, here the stable argsort (values 0..n-1)
  segments  Context.sort_segments_dev: many arrays in one buffer, each sorted by itself
  batch     Batch.launch: the same, replayed as a captured graph over the batch's own key arena
  host      Context.sort: the host-pointer call, keys in page-locked host memory
  server    Server.submit / drain: a burst of requests of mixed key types, from host to host

The sorts are in place, so a pass copies the unsorted keys into the buffer that it sorts first, as a
caller that keeps its input does. uint32 keys are held in int32 tensors (the same bits).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-quicksort_gb300"))
import gqs_ctypes  # noqa: E402

TORCH = {"u32": torch.int32, "f32": torch.float32, "f64": torch.float64}
SIZE = {"u32": 4, "f32": 4, "f64": 8}
DISTS = {"u32": ["uniform", "sorted", "reverse", "distinct16", "zipf", "gaussian"],
         "f32": ["gaussian", "uniform", "sorted", "reverse", "distinct16"],
         "f64": ["uniform", "gaussian", "sorted", "reverse", "distinct16"]}


def listed():
    return [
        # A few keys at a time inside a pipeline on the device: the calls queue up, launches count.
        {"name": "sort_u32_1k", "kind": "sort", "dtype": "u32", "dist": "uniform", "n": 1 << 10, "shift": 0, "sync": False},
        # A short ragged array that starts in the middle of a buffer, each call waited for (the default).
        {"name": "sort_f32_20k", "kind": "sort", "dtype": "f32", "dist": "gaussian", "n": 20_001, "shift": 1, "sync": True},
        # Doubles of an ordinary odd size.
        {"name": "sort_f64_300k", "kind": "sort", "dtype": "f64", "dist": "uniform", "n": 300_007, "shift": 0, "sync": True},
        # The reference's own size, as its driver calls it.
        {"name": "sort_u32_1m", "kind": "sort", "dtype": "u32", "dist": "uniform", "n": 1 << 20, "shift": 0, "sync": True},
        # The large sort, uniform keys.
        {"name": "sort_u32_268m", "kind": "sort", "dtype": "u32", "dist": "uniform", "n": 1 << 28, "shift": 0, "sync": True},
        # The large sort of few distinct values (labels, categories).
        {"name": "sort_u32_268m_16", "kind": "sort", "dtype": "u32", "dist": "distinct16", "n": 1 << 28, "shift": 0, "sync": True},
        # Large arrays of doubles.
        {"name": "sort_f64_67m", "kind": "sort", "dtype": "f64", "dist": "uniform", "n": 1 << 26, "shift": 0, "sync": True},
        # Stable argsort of skewed keys (ids by frequency), an odd size.
        {"name": "argsort_u32_8m", "kind": "pairs", "dtype": "u32", "dist": "zipf", "n": (1 << 23) + 5, "sync": True},
        # Thousands of short lists in one call, empty and single-key ones among them.
        {"name": "segments_f32_3000", "kind": "segments", "dtype": "f32", "dist": "gaussian", "segments": 3000, "lo": 0, "hi": 3000, "shape": 21, "sync": True},
        # The batched form: 4096 arrays of very uneven lengths, one graph replay.
        {"name": "batch_u32_4096", "kind": "batch", "dtype": "u32", "dist": "uniform", "segments": 4096, "lo": 32, "hi": 1 << 20, "shape": 4, "variant": -1},
        # The reference's calling convention: a large array in host memory, there and back.
        {"name": "host_f32_67m", "kind": "host", "dtype": "f32", "dist": "gaussian", "n": (1 << 26) + 1},
        # A burst of requests to the server, 60 % uint32, 30 % float, 10 % double.
        {"name": "server_96", "kind": "server", "requests": 96, "lo": 1 << 10, "hi": 1 << 20, "shape": 7},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["sort", "sort", "sort", "sort", "pairs", "segments", "batch", "host", "server"])
    dtype = rng.choice(["u32", "u32", "f32", "f64"])
    case = {"kind": kind, "dtype": dtype, "dist": rng.choice(DISTS[dtype])}
    most = (1 << 30) // SIZE[dtype]  # 1 GiB of keys
    if kind == "sort":
        n = _log_int(rng, 1 << 10, most // 2 if dtype == "f64" else most)
        case.update(n=n, shift=rng.choice([0, 0, 1, 3]), sync=rng.random() < 0.7)
    elif kind == "pairs":
        case["dtype"] = dtype = rng.choice(["u32", "f32"])
        case["dist"] = rng.choice(DISTS[dtype])
        case.update(n=_log_int(rng, 1 << 10, 1 << 25), sync=rng.random() < 0.7)
    elif kind in ("segments", "batch"):
        hi = _log_int(rng, 1 << 9, 1 << 20)
        lo = rng.choice([0, 1, 32]) if kind == "segments" else 32
        # as many as 2^27 keys in all, 4096 at most
        mean = (hi - max(lo, 1)) / math.log(hi / max(lo, 1))
        case.update(segments=_log_int(rng, 2, max(2, min(4096, int((1 << 27) / mean)))), lo=lo, hi=hi, shape=rng.randrange(1 << 16))
        if kind == "segments":
            case["sync"] = True
        else:
            # the batch's own choice of kernel, or one that its autotuner may have picked
            case["variant"] = rng.choice([-1, -1, 0, 3, 6])
    elif kind == "host":
        case["n"] = _log_int(rng, 1 << 10, (1 << 28) // SIZE[dtype])
    else:
        case = {"kind": kind, "requests": rng.randrange(8, 129), "lo": 1 << 10, "hi": _log_int(rng, 1 << 14, 1 << 20), "shape": rng.randrange(1 << 16)}
    return case


# ---- inputs -----------------------------------------------------------------

def _keys(dtype, dist, n, g):
    """n keys of one distribution on the GPU, in the raw type of the case."""
    dev = {"device": "cuda", "generator": g}
    if dist == "distinct16":
        return _keys(dtype, "uniform", 16, g)[torch.randint(0, 16, (n,), **dev)]
    if dtype == "u32":
        if dist in ("uniform", "sorted", "reverse"):
            k = torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, **dev)
            if dist == "uniform":
                return k
            k = torch.bitwise_xor(torch.sort(k, descending=dist == "reverse").values, -(1 << 31))
            return k  # signed order with the top bit flipped: ascending (descending) as unsigned
        if dist == "zipf":
            # s = 1.1 over 2^20 ranks, each rank a key of its own
            w = torch.arange(1, (1 << 20) + 1, dtype=torch.float64, device="cuda").pow(-1.1).cumsum(0)
            out = torch.empty(n, dtype=torch.int32, device="cuda")
            for a in range(0, n, 1 << 25):
                u = torch.rand(min(1 << 25, n - a), dtype=torch.float64, **dev) * w[-1]
                r = torch.searchsorted(w, u).clamp_(max=(1 << 20) - 1) + 1
                out[a:a + r.numel()] = ((r * 2654435761) & 0xFFFFFFFF).to(torch.uint32).view(torch.int32)
            return out
        k = torch.empty(n, dtype=torch.int32, device="cuda")  # rounded Gaussian, mean 2^31, sd 2^28
        for a in range(0, n, 1 << 25):
            x = torch.randn(min(1 << 25, n - a), dtype=torch.float64, **dev)
            k[a:a + x.numel()] = (x * 2.0**28).round().clamp(-(2.0**31), 2.0**31 - 1).to(torch.int32)
        return torch.bitwise_xor(k, -(1 << 31))
    t = TORCH[dtype]
    if dist == "gaussian":
        k = torch.randn(n, dtype=t, **dev) * 1e3
    else:
        k = (torch.rand(n, dtype=t, **dev) - 0.5) * 2e9
        if dist in ("sorted", "reverse"):
            k = torch.sort(k, descending=dist == "reverse").values
    return k + 0.0  # no -0.0


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _lengths(case, count):
    """Lengths log-uniform in [lo, hi] (the shape of the case: the same for every seed)."""
    r = np.random.RandomState(case["shape"])
    lo, hi = case["lo"], case["hi"]
    n = np.exp(r.uniform(math.log(max(lo, 1)), math.log(hi), count)).astype(np.int64)
    n = np.clip(n, max(lo, 1), hi)
    if lo == 0:
        n[r.rand(count) < 0.02] = 0
    return n


def _offsets(case):
    return np.concatenate([[0], np.cumsum(_lengths(case, case["segments"]))]).astype(np.int64)


def _requests(case):
    """(key type, first key, length) of every request; each key type has a buffer of its own."""
    lens = _lengths(case, case["requests"])
    types = np.random.RandomState(case["shape"] + 1).choice(["u32", "f32", "f64"], case["requests"], p=[0.6, 0.3, 0.1])
    at = {"u32": 0, "f32": 0, "f64": 0}
    out = []
    for t, n in zip(types, lens):
        out.append((str(t), at[t], int(n)))
        at[t] += int(n)
    return out, at


class _Arena:
    """The batch's key arena as a tensor, which keeps the batch (the arena's owner) alive."""

    def __init__(self, batch, n, dtype):
        self.batch = batch
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": {"u32": "<i4", "f32": "<f4", "f64": "<f8"}[dtype],
                                         "data": (batch.keys_ptr, False), "version": 2}


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "server":
        s["requests"], total = _requests(case)
        s["src"] = {t: _keys(t, "gaussian" if t == "f32" else "uniform", max(n, 1), g).cpu().pin_memory() for t, n in total.items()}
        s["out"] = {t: torch.zeros_like(x).pin_memory() for t, x in s["src"].items()}
        s["server"] = gqs_ctypes.Server(budget_bytes=8 << 30)
        return s
    t = case["dtype"]
    if kind in ("segments", "batch"):
        s["off"] = _offsets(case)
        n = max(int(s["off"][-1]), 1)
    else:
        n = case["n"]
    src = _keys(t, case["dist"], n, g)
    if kind == "host":
        s["src"] = src.cpu().pin_memory()
        s["out"] = torch.empty_like(s["src"]).pin_memory()
        keys = s["out"].numpy()
        s["keys"] = keys.view(np.uint32) if t == "u32" else keys
        s["ctx"] = gqs_ctypes.Context()
        s["ctx"].reserve(t, n, 1, True)
        return s
    s["src"] = src
    if kind == "batch":
        s["batch"] = gqs_ctypes.Batch(t, n, case["segments"], variant=case["variant"])
        s["batch"].set_segments(s["off"])
        s["keys"] = torch.as_tensor(_Arena(s["batch"], n, t), device="cuda")
        return s
    s["ctx"] = gqs_ctypes.Context(sync=case["sync"])
    if kind == "pairs":
        s["keys"] = torch.empty_like(src)
        s["values"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["iota"] = torch.arange(n, dtype=torch.int32, device="cuda")
        return s
    shift = case.get("shift", 0)
    s["keys"] = torch.empty(n + shift, dtype=TORCH[t], device="cuda")[shift:]
    if kind == "segments":
        s["ctx"].reserve(t, n, case["segments"])
        s["offsets"] = torch.from_numpy(s["off"]).cuda()
    else:
        s["ctx"].reserve(t, n)
    return s


# ---- one pass ---------------------------------------------------------------

def _ok(code):
    if code:
        raise gqs_ctypes.GqsError(code, "sort")


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "server":
        srv = s["server"]
        for t, first, n in s["requests"]:
            at = first * SIZE[t]
            srv.submit_raw(t, s["src"][t].data_ptr() + at, s["out"][t].data_ptr() + at, n)
        _ok(srv.drain())
        while srv.wait_any(0)[0] != 4:  # collect the finished requests
            pass
        return s["out"]
    if kind == "host":
        s["out"].copy_(s["src"])
        s["ctx"].sort(s["keys"])
        return s["out"]
    keys, n, stream = s["keys"], s["src"].numel(), torch.cuda.current_stream().cuda_stream
    keys.copy_(s["src"])
    if kind == "sort":
        _ok(s["ctx"].sort_dev(case["dtype"], keys.data_ptr(), None, n, stream))
        return keys
    if kind == "pairs":
        s["values"].copy_(s["iota"])
        _ok(s["ctx"].sort_pairs_dev(case["dtype"], keys.data_ptr(), s["values"].data_ptr(), n, stream))
        return [keys, s["values"]]
    if kind == "segments":
        _ok(s["ctx"].sort_segments_dev(case["dtype"], keys.data_ptr(), None, n, s["offsets"].data_ptr(), case["segments"], stream))
        return keys
    _ok(s["batch"].launch(case["segments"], stream))
    return keys


def work(case):
    """Every key read once and written once; no floating-point operations."""
    kind = case["kind"]
    if kind == "server":
        return {"bytes": 2 * sum(n * SIZE[t] for t, _, n in _requests(case)[0]), "flops": 0}
    if kind in ("segments", "batch"):
        return {"bytes": 2 * int(_offsets(case)[-1]) * SIZE[case["dtype"]] + 8 * (case["segments"] + 1), "flops": 0}
    return {"bytes": 2 * case["n"] * (SIZE[case["dtype"]] + (4 if kind == "pairs" else 0)), "flops": 0}


# ---- the same in 64 bits, without this library -----------------------------

def _wide(x):
    """Keys as 64-bit numbers in their own order."""
    return x.to(torch.int64) & 0xFFFFFFFF if x.dtype == torch.int32 else x.to(torch.float64)


def _narrow(x, dtype):
    return x.to(torch.uint32).view(torch.int32) if dtype == "u32" else x


def _sorted_segments(x, bounds, dtype):
    out = _wide(x)
    for a, b in zip(bounds[:-1], bounds[1:]):
        if b - a > 1:
            out[a:b] = torch.sort(out[a:b]).values
    return _narrow(out, dtype)


def exact(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "server":
        req, total = _requests(case)
        out = {}
        for t, n in total.items():
            x = _keys(t, "gaussian" if t == "f32" else "uniform", max(n, 1), g)
            if not n:
                out[t] = torch.zeros_like(x).cpu()
                continue
            out[t] = _sorted_segments(x, [0] + [a + m for u, a, m in req if u == t], t).cpu()
        return out
    t = case["dtype"]
    if kind in ("segments", "batch"):
        off = [int(v) for v in _offsets(case)]
        return _sorted_segments(_keys(t, case["dist"], max(off[-1], 1), g), off, t)
    x = _wide(_keys(t, case["dist"], case["n"], g))
    v, i = torch.sort(x, stable=True)
    if kind == "pairs":
        return [_narrow(v, t), i.to(torch.int32)]
    v = _narrow(v, t)
    return v.cpu() if kind == "host" else v
