"""What a server's lanes take out of its budget: job records and ticket rings. The split's tables, which are done with before the
first job record is made, lie in the same memory, so a budget that holds the records holds the server."""
import ctypes

import numpy as np
import pytest

import gqs_ctypes

JOB = 80      # bytes of a job record
GRAIN = 256   # the arena's unit


def lane_bytes(keys, segments):
    """Job records and ring entries of the most demanding variant of any key type."""
    jobs = ring = 0
    for t in ("u32", "f32", "f64"):
        for v in gqs_ctypes.variants(t):
            jobs = max(jobs, keys // v["tiny"] + 16 * (keys // v["tile"]) + keys // 32768 + 2 * segments + 4096)
            need = 2 * (keys // v["chunk"]) + keys // v["tiny"] + keys // 32768 + 2 * segments + 65536
            ring = max(ring, 1 << (need - 1).bit_length())
    return jobs * JOB, ring * 8


def test_split_tables_fit_in_the_job_records():
    lib = gqs_ctypes.load_library()
    scratch, keep = lib["_ZN3gqs19split_scratch_bytesEimmbi"], lib["_ZN3gqs16split_keep_bytesEimmi"]
    scratch.restype = keep.restype = ctypes.c_size_t
    scratch.argtypes = [ctypes.c_int, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_bool, ctypes.c_int]
    keep.argtypes = [ctypes.c_int, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_int]
    for keys in [1, 255, 2047, 2048, 4097, 8193, 100_003, 1 << 20, (1 << 22) - 1, 1 << 27, (1 << 31) - 1]:
        for segments in [1, 64, 4096, 1 << 20]:
            kept = max(keep(t, keys, segments, 152) for t in range(3))
            assert max(scratch(t, keys, segments, False, 152) for t in range(3)) - kept <= lane_bytes(keys, segments)[0]
            # what stays beside them: the ranges left, 16 bytes each, and a block of fixed size
            assert kept <= (keys // 4096 + 1) * 16 + 65536


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,keys,segments", [(3, 1 << 27, 4096), (2, 1 << 17, 64)])
def test_budget_of_the_records_holds_a_server(lanes, keys, segments):
    arena = 2 << 20
    budget = lanes * sum(lane_bytes(keys, segments)) + 2 * arena
    with gqs_ctypes.Server(budget_bytes=budget, batch_keys=keys, batch_segments=segments, lanes=lanes) as srv:
        assert srv.stats()["arena_bytes"] == arena // GRAIN * GRAIN
        a = gqs_ctypes.generate("f64", "uniform", 3, 120_001)
        b = np.empty_like(a)
        assert srv.wait(srv.submit(a, b))[0] == 0
        assert np.array_equal(b, np.sort(a))
