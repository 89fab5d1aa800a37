"""Calls on a greater-priority stream while a launch that fills the GPU runs."""
import time

import numpy as np
import pytest

from conftest import P, dev_empty, from_dev, rand_u64, to_dev

pytestmark = pytest.mark.gpu

TILE, GROUPS, CTA_PERMS = 128, 4, 38  # hash_mma.cu: rows per tile, tiles of a CTA at a time, permutations of a group


def test_opening_does_not_wait_for_a_whole_row_hash(tv):
    import torch
    rows, width = 1 << 21, 379
    x = torch.randint(0, 2**62, (width, rows), dtype=torch.int64, device="cuda")
    out = dev_empty(rows, 5)
    idx = np.arange(80) * 11 % 1024
    with tv.Commitment(rand_u64(1, (10, 256))) as c:
        want = c.auth_paths(idx)
        big = torch.cuda.Stream()
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        lat = []
        for _ in range(6):
            torch.cuda.synchronize()
            start.record(big)
            tv.hash_rows_gpu(x.data_ptr(), rows, width, out.data_ptr(), stream=big)
            end.record(big)
            time.sleep(1e-3)  # the row hash holds every SM
            t0 = time.perf_counter()
            got = c.auth_paths(idx)
            lat.append(1e3 * (time.perf_counter() - t0))
            assert (got == want).all()
        torch.cuda.synchronize()
        assert np.median(lat) < start.elapsed_time(end) / 4, lat


@pytest.mark.parametrize("width", [379, 99, 9])
@pytest.mark.parametrize("tiles", [-1, 0, 1, 150])
def test_row_hash_at_the_edges_of_a_round_of_ctas(tv, oracle, width, tiles):
    """One full round of CTAs, one tile less, and a little more."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    depth = max(1, CTA_PERMS // (width // 10 + 1))
    rows = (sms * GROUPS * depth + tiles) * TILE - 5
    x = torch.randint(0, 2**62, (width, rows), dtype=torch.int64, device="cuda")
    out = torch.full((rows, 5), -1, dtype=torch.int64, device="cuda")
    tv.hash_rows_gpu(x.data_ptr(), rows, width, out.data_ptr())
    pick = np.unique(np.concatenate([np.arange(0, rows, 1009), np.arange(max(0, rows - 300), rows)]))
    cells = from_dev(x[:, torch.from_numpy(pick).cuda()])
    assert (from_dev(out)[pick] == oracle.hash_rows_cm(np.ascontiguousarray(cells % P))).all()
    assert (from_dev(out) < P).all()  # every row was written
