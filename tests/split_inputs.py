"""Inputs that the split of csrc/gqs_split.cu cannot finish: the places that it samples are a fixed function of a segment's length,
so an array can show it evenly spread keys there and hold all its other keys, all different, in one narrow interval. One of the
split's ranges then gets nearly the whole array, and the persistent kernel has to sort it."""
import numpy as np

LOCAL = {"u32": 8192, "f32": 8192, "f64": 4096, "pairs": 4096}   # keys that one thread block sorts
TARGET = {k: v // 16 * 7 for k, v in LOCAL.items()}              # mean keys of a range
SMALL_MAX = {"u32": 1 << 21, "f32": 1 << 21, "f64": 1 << 19, "pairs": 1 << 19}
MAX_BINS = 1024


def ranges(kind, n, more_levels):
    want = -(-n // TARGET[kind])
    if want <= 2:
        return 2
    if want <= MAX_BINS:
        return want
    return min(MAX_BINS, int(np.ceil(np.sqrt(np.float32(want))))) if more_levels else MAX_BINS


def sample_places(kind, n, sms, plain=True, levels=None):
    """The indexes that the first map of n keys samples (a segment: plain=False, and how many levels its table may take)."""
    wide = kind in ("f64", "pairs")
    if plain and n <= SMALL_MAX[kind]:
        least, most = n // (LOCAL[kind] // 10 * 3) + 1, n // 1024 + 1
        k = min(MAX_BINS, max(2, least if sms * 3 < least else most if sms * 3 > most else sms * 3))
        s = min(max(10 * k, 1024), 3328 if wide else 5120)
    else:
        if levels is None:
            levels = 2 if n > MAX_BINS * TARGET[kind] or n > (1 << 21) else 1
        k = ranges(kind, n, levels > 1)
        most = (16384 if wide else 24576) if plain else (8192 if wide else 12288)
        s = min(max(32 * k, 1024), most)
    s = min(s, n)
    i = np.arange(s, dtype=np.uint64)
    h = (i * np.uint64(2654435761)) & np.uint64(0xffffffff)
    h ^= h >> np.uint64(15)
    h = (h * np.uint64(0x85ebca6b)) & np.uint64(0xffffffff)
    return (i * np.uint64(n) // np.uint64(s) + (h * np.uint64(n // s) >> np.uint64(32))).astype(np.int64)


def unfinishable(kind, n, sms, seed=1, **level):
    """n keys, as integers in the library's order (uint32; uint64 for f64)."""
    rng = np.random.default_rng(seed)
    ut = np.uint64 if kind == "f64" else np.uint32
    bits = 8 * ut().itemsize
    at = sample_places(kind, n, sms, **level)
    k = ut((1 << (bits - 1)) + (1 << (bits - 13))) + rng.permutation(n).astype(ut)
    s = len(at)
    spread = (np.arange(s, dtype=np.float64) * (2.0 ** bits / s)).astype(ut)
    spread[-1] = ut((1 << bits) - 1)
    k[at] = rng.permutation(spread)
    return k


def as_keys(k, dtype):
    """Integers in the library's order as keys of `dtype`."""
    if dtype == "u32":
        return k
    top = k.dtype.type(1 << (8 * k.dtype.itemsize - 1))
    return np.where(k & top, k ^ top, ~k).view(np.float32 if dtype == "f32" else np.float64)
