"""GPU parity of the sampled split and its on-chip sort (csrc/gqs_split.cu), bit for bit, at the sizes where their paths meet:
the on-chip capacity, the two-kernel sorts' largest size, one and two counted levels, and tiles' edges around them; keys that
the map has to divide again (few values, clusters, one value, the type's extremes), and segments at the on-chip capacity."""
import numpy as np
import pytest

import gqs_ctypes

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "f32": np.float32, "f64": np.float64}
LOCAL = {"u32": 8192, "f32": 8192, "f64": 4096}          # keys that one thread block sorts
SMALL = {"u32": 1 << 21, "f32": 1 << 21, "f64": 1 << 19}  # the most that two kernels sort
ONE_LEVEL = 1024 * 1792                                   # the most f64 keys that one counted level splits


def ordered(a):
    """The keys as integers in the library's order (-0.0 before +0.0, NaNs by their bits)."""
    if a.dtype == np.uint32:
        return a
    u = a.view(np.uint32 if a.dtype == np.float32 else np.uint64)
    top = u.dtype.type(1 << (8 * u.dtype.itemsize - 1))
    return np.where(u & top, ~u, u | top)


def unordered(k, dtype):
    if dtype == "u32":
        return k
    top = k.dtype.type(1 << (8 * k.dtype.itemsize - 1))
    return np.where(k & top, k ^ top, ~k).view(NP[dtype])


def keys(dtype, kind, n):
    rng = np.random.default_rng(n)
    ut = np.uint64 if dtype == "f64" else np.uint32
    bits = 8 * ut().itemsize
    if kind == "uniform":
        k = rng.integers(0, 1 << bits, n, dtype=ut, endpoint=False) if bits < 64 else rng.integers(0, (1 << 64) - 1, n, dtype=ut, endpoint=True)
    elif kind == "values":  # a few values with most of the keys, close to each other and far apart
        v = np.array([0, 1, 2, 1 << 9, (1 << bits) - 1, (1 << (bits - 1)) + 5, (1 << (bits - 1)) + 6], dtype=ut)
        k = v[rng.integers(0, len(v), n)]
        odd = rng.integers(0, n, n // 50 + 1)
        k[odd] = rng.integers(0, 1 << 31, len(odd)).astype(ut) << ut(bits - 32)
    elif kind == "clusters":  # dense runs of words with wide gaps, of very different sizes
        k = (rng.zipf(1.3, n).astype(np.float64).clip(0, 255).astype(ut) << ut(bits - 8)) | rng.integers(0, 1 << 12, n).astype(ut)
    elif kind == "one":
        k = np.full(n, 12345, dtype=ut)
    else:  # "real": values around zero over many exponents, infinities among them
        v = rng.normal(size=n) * np.exp2(rng.integers(-60, 60, n).astype(np.float64))
        v[:: 997] = np.inf
        v[1 :: 997] = -np.inf
        v[2 :: 499] = -0.0
        return v.astype(NP[dtype]) if dtype != "u32" else np.abs(v).clip(0, 4e9).astype(np.uint32)
    return np.ascontiguousarray(unordered(k, dtype))


def expect(a):
    return unordered(np.sort(ordered(a)), {np.dtype(v): k for k, v in NP.items()}[a.dtype])


def same(got, want):
    return np.array_equal(got.view(np.uint8), want.view(np.uint8))


@pytest.mark.parametrize("kind", ["uniform", "values", "clusters", "one", "real"])
@pytest.mark.parametrize("dtype", ["u32", "f32", "f64"])
def test_split_paths_match_numpy(gpu_ctx, dtype, kind):
    sizes = [LOCAL[dtype], LOCAL[dtype] + 1, 3 * LOCAL[dtype] - 1, 152 * 2048 + 1, SMALL[dtype], SMALL[dtype] + 1]
    sizes += [ONE_LEVEL, ONE_LEVEL + 1] if dtype == "f64" else [(1 << 22) + 8191]
    for n in sizes:
        a = keys(dtype, kind, n)
        b = a.copy()
        gpu_ctx.sort(b)
        assert same(b, expect(a)), (dtype, kind, n)


@pytest.mark.parametrize("dtype", ["u32", "f32"])
@pytest.mark.parametrize("n", [4097, (1 << 19) + 1, 2_000_003])
def test_split_pairs_match_numpy(gpu_ctx, dtype, n):
    # values of few bits, of all bits, and a permutation, under keys with many duplicates
    rng = np.random.default_rng(n)
    k = unordered((rng.zipf(1.4, n).clip(0, 1 << 20)).astype(np.uint32) * np.uint32(4001), dtype)
    for v in (rng.integers(0, 3, n), rng.integers(0, 1 << 32, n), rng.permutation(n)):
        kk, vv = k.copy(), v.astype(np.uint32)
        gpu_ctx.sort_pairs(kk, vv)
        order = np.lexsort((v, ordered(k)))
        assert same(kk, k[order]) and np.array_equal(vv, v[order].astype(np.uint32)), (dtype, n)


@pytest.mark.parametrize("dtype", ["u32", "f32", "f64"])
def test_split_segments_match_numpy(gpu_ctx, dtype):
    L = LOCAL[dtype]
    lens = [0, 1, L, 2, L + 1, 0, 3 * L + 7, 130 * L + 1, 31, 1100 * 1792 + 5]
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    a = np.concatenate([keys(dtype, kind, n) for n, kind in zip(lens, ["one", "one", "values", "uniform", "clusters", "one", "real", "clusters", "values", "uniform"])])
    b = a.copy()
    gpu_ctx.sort_segments(b, off)
    want = np.concatenate([expect(a[int(s):int(e)]) for s, e in zip(off[:-1], off[1:])])
    assert same(b, want)


def test_reserve_covers_shorter_sorts(gpu_ctx):
    # a context reserved for a size sorts every shorter array without allocating (a capture would refuse to)
    torch = pytest.importorskip("torch")
    stream = torch.cuda.current_stream().cuda_stream
    arrays = [keys("u32", "uniform", n) for n in (1 << 21, 20_001)]
    on_gpu = [torch.from_numpy(a.view(np.int32)).cuda() for a in arrays]

    def run(ctx):
        out = []
        for t in on_gpu:
            w = t.clone()
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            assert ctx.sort_dev("u32", w.data_ptr(), None, w.numel(), stream) == 0
            torch.cuda.synchronize()
            out.append((before - torch.cuda.mem_get_info()[0], w.cpu().numpy().view(np.uint32)))
        return out

    with gqs_ctypes.Context() as first:  # loads the kernels
        run(first)
    with gqs_ctypes.Context() as ctx:
        ctx.reserve("u32", (1 << 21) + 4096, with_buffers=True)
        for a, (taken, got) in zip(arrays, run(ctx)):
            assert taken == 0, len(a)
            assert same(got, expect(a))
