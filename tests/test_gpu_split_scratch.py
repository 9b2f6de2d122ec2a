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
