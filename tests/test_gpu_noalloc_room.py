"""The cell sort without allocation where few of its blocks run at once (the threads then stride over the
particles instead of holding them).
"""
import ctypes

import numpy as np
import pytest

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

