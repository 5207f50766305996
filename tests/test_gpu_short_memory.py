"""GPU: what the library's memory pool keeps is given back when memory is short.
The test holds most of the device's memory while it asks for more than is left
outside the pool.  Run with -m gpu on a B200."""
import numpy as np
import pytest

import oracle
from tests.knn_check import assert_knn_matches

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import curplsh_b200 as cb
    res = cb.DeviceResources(0)
    yield cb, torch, res
    res.close()


@pytest.fixture()
def short(env):
    """A small index and its rows, with about 700 MB freed into the pool and 250 MB
    left on the device."""
    cb, torch, res = env
    rng = np.random.default_rng(1)
    rows = rng.standard_normal((3000, 32)).astype(np.float32)
    ix = cb.IndexBF(res, 32)
    ix.add(len(rows), rows)
    ix.search_array(rows[:4], 5)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    big = cb.IndexBF(res, 128)
    big.add(500_000, torch.zeros((500_000, 128), device="cuda"))
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - 250 * MB, dtype=torch.uint8, device="cuda")
    big.close()
    assert torch.cuda.mem_get_info()[0] < 400 * MB
    yield ix, rows
    del hold
    torch.cuda.empty_cache()
    ix.close()


def test_server_arena(env, short):
    cb, torch, _ = env
    ix, rows = short
    server = cb.Server(ix, memory_budget=600 * MB)
    i, x = torch.empty((4, 5), dtype=torch.int32).pin_memory(), torch.empty((4, 5)).pin_memory()
    server.wait(server.submit(torch.tensor(rows[:4]).pin_memory(), 5, i, x))
    server.close()
    rd, ri = oracle.knn(rows, rows[:4], 6)
    assert_knn_matches(rows, rows[:4], x.numpy(), i.numpy(), rd, ri)


def test_batch_workspace(env, short):
    cb, torch, _ = env
    ix, rows = short
    q = torch.tensor(rows[:1500]).cuda()
    i, x = torch.empty((1500, 1000), dtype=torch.int32, device="cuda"), torch.empty((1500, 1000), device="cuda")
    cb.set_bound_estimate(False)
    try:
        batch = cb.SearchBatch([(ix, q, 1000, i, x)])
    finally:
        cb.set_bound_estimate(True)
    assert 300 * MB < batch.info()[1] < 700 * MB
    batch.run()
    batch.close()
    rd, ri = oracle.knn(rows, rows[:50], 1001)
    assert_knn_matches(rows, rows[:50], x[:50].cpu().numpy(), i[:50].cpu().numpy(), rd, ri)


def test_rows_right_after_an_index_closed(env, short):
    """Larger than the pool serves, and asked for before any wait for the frees."""
    cb, torch, res = env
    _, rows = short
    big = cb.IndexBF(res, 32)
    big.add(2_200_000, np.zeros((2_200_000, 32), np.float32))  # 282 MB of rows, 334 MB of operands
    assert big.getNumData() == 2_200_000
    big.close()
