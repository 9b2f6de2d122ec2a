"""What the split leaves to the persistent kernel, on inputs that are sure to leave something (tests/split_inputs.py): a small sort
as a whole, ranges of one counted level (their keys are in the scratch) and of two, in plain sorts, pairs, segments and batches,
with calls that wait, calls that are queued and host-pointer calls, and with every kernel variant. That the persistent kernel did
sort is read from its own cycle counters, or from partition passes that the split alone does not make."""
import numpy as np
import pytest

import gqs_ctypes
from split_inputs import as_keys, unfinishable

pytestmark = pytest.mark.gpu

PLAIN = [("u32", 100_003), ("u32", 1 << 21), ("f32", 700_001), ("f64", 1 << 19),  # left as a whole
         ("f64", 1_500_001),                                                     # one counted level
         ("u32", (1 << 24) - 1000), ("f64", (1 << 23) + 77)]                     # two


@pytest.fixture(scope="module")
def sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


def to_gpu(a):
    import torch
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


def same(got, want):
    return np.array_equal(got.view(np.uint8), want.view(np.uint8))


def sort_on_gpu(ctx, dtype, a, off=None):
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    t = to_gpu(a)
    if off is None:
        assert ctx.sort_dev(dtype, t.data_ptr(), None, a.size, stream) == 0
    else:
        o = torch.from_numpy(off.view(np.int64)).cuda()
        assert ctx.sort_segments_dev(dtype, t.data_ptr(), None, a.size, o.data_ptr(), len(off) - 1, stream) == 0
    assert ctx.sync() == 0
    return t.cpu().numpy().view(a.dtype)


@pytest.mark.parametrize("dtype,n", PLAIN)
def test_plain_sort_leaves_a_range(sms, dtype, n):
    k = unfinishable(dtype, n, sms)
    a, want = as_keys(k, dtype), as_keys(np.sort(k), dtype)
    for waits in (True, False):
        with gqs_ctypes.Context(sync=waits) as ctx:
            for _ in range(2):
                assert same(sort_on_gpu(ctx, dtype, a), want)
                assert ctx.phases()["total_cycles"] > 0 and ctx.stats()["status"] == 0
            plain = as_keys(np.random.default_rng(2).permutation(k), dtype)  # and a sort that leaves nothing
            assert same(sort_on_gpu(ctx, dtype, plain), want)
    if n < 1 << 24:  # (longer ones are sorted in pieces from the host)
        with gqs_ctypes.Context() as ctx:
            b = a.copy()
            ctx.sort(b)
            assert same(b, want) and ctx.phases()["total_cycles"] > 0


@pytest.mark.parametrize("dtype", ["u32", "f32"])
@pytest.mark.parametrize("n", [300_001, 1_500_001, 1 << 23])
def test_pairs_leave_a_range(sms, dtype, n):
    import torch
    k = unfinishable("pairs", n, sms)
    a = as_keys(k, dtype)
    order = np.argsort(k, kind="stable")
    for waits in (True, False):
        with gqs_ctypes.Context(sync=waits) as ctx:
            t, v = to_gpu(a), torch.arange(n, dtype=torch.int32, device="cuda")
            assert ctx.sort_pairs_dev(dtype, t.data_ptr(), v.data_ptr(), n, torch.cuda.current_stream().cuda_stream) == 0
            assert ctx.sync() == 0
            assert same(t.cpu().numpy().view(a.dtype), a[order])
            assert np.array_equal(v.cpu().numpy(), order)
            assert ctx.phases()["total_cycles"] > 0


def segment_table(long, buffer):
    """Short segments around one long one, which starts at 1000; the buffer may end later."""
    off = np.array([0, 0, 100, 1000, 1000 + long, 1000 + long, 1300 + long, buffer], dtype=np.uint64)
    return off


def segments_case(dtype, long, sms, levels):
    buffer = 1400 + long
    off = segment_table(long, buffer)
    rng = np.random.default_rng(long)
    ut = np.uint64 if dtype == "f64" else np.uint32
    k = rng.integers(0, 1 << 31, buffer).astype(ut)
    k[1000:1000 + long] = unfinishable(dtype, long, sms, plain=False, levels=levels)
    want = k.copy()
    for s, e in zip(off[:-1], off[1:]):
        want[int(s):int(e)].sort()
    return as_keys(k, dtype), as_keys(want, dtype), off


@pytest.mark.parametrize("dtype,long,levels", [("u32", 200_003, 1), ("f32", 90_001, 1), ("f64", 200_003, 1),
                                               ("u32", 1 << 24, 2), ("f64", 1 << 23, 2)])
def test_segments_leave_a_range(sms, dtype, long, levels):
    a, want, off = segments_case(dtype, long, sms, levels)
    for waits in (True, False):
        with gqs_ctypes.Context(sync=waits) as ctx:
            assert same(sort_on_gpu(ctx, dtype, a, off), want)
            assert ctx.phases()["total_cycles"] > 0
    with gqs_ctypes.Batch(dtype, a.size, 16) as batch:
        nseg = batch.set_segments(off)
        for _ in range(2):
            batch.copy_in(a)
            assert batch.launch(nseg) == 0
            code, st = batch.wait()
            b = np.empty_like(a)
            batch.copy_out(b)
            assert code == 0 and same(b, want)
            # the split reads every key of the long segment once a level; a range left is partitioned again
            assert st["part_keys"] > levels * long


@pytest.mark.parametrize("dtype", ["u32", "f32", "f64"])
def test_every_variant_sorts_what_is_left(sms, dtype):
    """A fixed variant is the kernel that sorts what is left: every one of them, over one range in the scratch (segments, a batch)
    and over a whole small sort."""
    a, want, off = segments_case(dtype, 150_001, sms, 1)
    k = unfinishable(dtype, 300_007, sms)
    small, small_want = as_keys(k, dtype), as_keys(np.sort(k), dtype)
    with gqs_ctypes.Batch(dtype, a.size, 16) as batch:
        nseg = batch.set_segments(off)
        for v in range(len(gqs_ctypes.variants(dtype))):
            batch.set_variant(v)
            batch.copy_in(a)
            assert batch.launch(nseg) == 0
            code, st = batch.wait()
            b = np.empty_like(a)
            batch.copy_out(b)
            assert code == 0 and same(b, want) and st["variant"] == v and st["part_keys"] > 150_001, v
            with gqs_ctypes.Context(variant=v) as ctx:
                assert same(sort_on_gpu(ctx, dtype, a, off), want), v
                assert ctx.phases()["total_cycles"] > 0, v
                assert same(sort_on_gpu(ctx, dtype, small), small_want), v
                assert ctx.phases()["total_cycles"] > 0 and ctx.stats()["variant"] == v, v
