"""The cell sort without allocation where few of its blocks run at once (the threads then stride over the
particles instead of holding them), and from two host threads, whose calls may overlap on the GPU.
"""
import ctypes
import threading

import numpy as np
import pytest

from solunar_b200.abi import PhysicsError

pytestmark = pytest.mark.gpu

RADIUS = 0.1


def arrays(n, seed):
    rng = np.random.default_rng(seed)
    pos = (rng.uniform(-0.5, 0.5, (n, 3)) * 0.04 * np.cbrt(n)).astype(np.float32)
    return pos, rng.permutation(n).astype(np.int32)


def expected(pos, ids):
    cell = np.floor(pos / np.float32(RADIUS)).astype(np.int64)
    return np.lexsort((ids, cell[:, 2], cell[:, 1], cell[:, 0]))


@pytest.mark.parametrize("blocks", [1, 2, 7, 100, 0])
@pytest.mark.parametrize("n", [1, 257, 2049, 20001, 1 << 18])
def test_any_number_of_blocks_sorts(gpu_lib, n, blocks):
    import torch

    pos, ids = arrays(n, n)
    d_pos, d_ids = torch.from_numpy(pos).cuda(), torch.from_numpy(ids).cuda()
    order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    status = gpu_lib.load_library().slf_debug_sort_by_cell_noalloc(
        ctypes.c_void_p(d_pos.data_ptr()), ctypes.c_void_p(d_ids.data_ptr()), n, RADIUS,
        ctypes.c_void_p(order.data_ptr()), None, blocks)
    assert status == 0
    assert np.array_equal(order.cpu().numpy(), expected(pos, ids))


def test_overlapping_calls_end_and_the_next_one_sorts(gpu_lib):
    import torch

    # the same box in both threads: what one call reads of the other's tables stays plausible, the
    # orders may be wrong, and neither call may wait for the other's blocks
    n = 20001
    pos, ids = arrays(n, 5)
    d_pos, d_ids = torch.from_numpy(pos).cuda(), torch.from_numpy(ids).cuda()
    orders = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    failures = []

    def call(k, times):
        for _ in range(times):
            try:
                gpu_lib.sort_by_cell_noalloc(d_pos.data_ptr(), d_ids.data_ptr(), n, RADIUS, orders[k].data_ptr(),
                                             streams[k].cuda_stream)
            except PhysicsError as e:
                failures.append(e.kind)

    threads = [threading.Thread(target=call, args=(k, 50)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert "Timeout" not in failures and "Cuda" not in failures
    call(0, 1)
    assert np.array_equal(orders[0].cpu().numpy(), expected(pos, ids))
