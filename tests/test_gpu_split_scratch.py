"""The counters that small sorts keep in their scratch (csrc/gqs_split.cu, Small): a context's first sorts are exact whatever its new
scratch held and whatever the default stream is busy with, which no other stream waits for."""
import numpy as np
import pytest

import gqs_ctypes

pytestmark = pytest.mark.gpu

N = 1 << 20


def leave_garbage(torch):
    """Device memory that the next allocations are given again, full of ones."""
    junk = [torch.full((1 << 24,), -1, dtype=torch.int32, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()


def keep_default_stream_busy(x):
    """Some 20 ms of ordinary work."""
    for _ in range(40):
        x.add_(1)


@pytest.mark.parametrize("reserve", [False, True])
@pytest.mark.parametrize("call", ["host", "dev"])
def test_first_small_sorts_beside_a_busy_default_stream(gpu_ctx, call, reserve):
    torch = pytest.importorskip("torch")
    a = gqs_ctypes.generate("u32", "uniform", 17, N)
    want = np.sort(a)
    gpu_ctx.sort(a.copy())  # loads the kernels
    busy = torch.zeros(1 << 29, dtype=torch.int32, device="cuda")
    side = torch.cuda.Stream()
    keys = [torch.from_numpy(a.view(np.int32)).cuda() for _ in range(2)]
    with gqs_ctypes.Context() as ctx:
        leave_garbage(torch)
        torch.cuda.synchronize()
        keep_default_stream_busy(busy)
        if reserve:
            ctx.reserve("u32", N, 1, True)
        for t in keys:  # the second one finds the counters as the first one left them
            if call == "host":
                got = a.copy()
                ctx.sort(got)
            else:
                assert ctx.sort_dev("u32", t.data_ptr(), None, N, side.cuda_stream) == 0
                got = t.cpu().numpy().view(np.uint32)
            assert np.array_equal(got, want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("variant", [-1, 0])
@pytest.mark.parametrize("nseg", [1, 3])
def test_reserve_covers_plain_and_segmented_sorts(variant, nseg):
    """What is reserved for n keys in nseg segments sorts n keys, and fewer, as one array or as segments, and allocates nothing."""
    torch = pytest.importorskip("torch")
    stream = torch.cuda.current_stream().cuda_stream
    n = 1 << 25
    keys = torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int64, device="cuda").to(torch.int32)
    order = torch.tensor([-(1 << 31)], dtype=torch.int32, device="cuda")  # signed order to unsigned
    want = torch.sort(keys ^ order).values ^ order

    def run(ctx, length, segments):
        t = keys[:length].clone()
        off = torch.tensor([length * i // max(segments, 1) for i in range(segments + 1)], device="cuda")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        if segments:
            code = ctx.sort_segments_dev("u32", t.data_ptr(), None, length, off.data_ptr(), segments, stream)
        else:
            code = ctx.sort_dev("u32", t.data_ptr(), None, length, stream)
        assert code == 0
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0], t

    with gqs_ctypes.Context(variant=variant) as ctx:
        first = run(ctx, n, 1)  # loads the kernels
        run(ctx, n, 0), run(ctx, 1 << 20, 0)
        assert torch.equal(first[1], want)
    with gqs_ctypes.Context(variant=variant) as ctx:
        ctx.reserve("u32", n, nseg)
        for length in (n, 1 << 20, 5000):
            for segments in (0, 1, nseg):
                taken, t = run(ctx, length, segments)
                assert taken == 0, (length, segments)
                if length == n and segments < 2:
                    assert torch.equal(t, want)
