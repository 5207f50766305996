"""GPU: the database norms inside the FP8 accumulator.

The norm of a row rides in units of 1 / (2 s_q s), s_q and s the scales of the
query and of the database, so a query many orders of magnitude smaller than the
rows must not overflow it: such a query's nearest rows are those of the smallest
norm.  Run with -m gpu on a B200."""
import numpy as np
import pytest

import oracle
from tests.knn_check import assert_knn_matches

pytestmark = pytest.mark.gpu

FP8 = 2


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import curplsh_b200 as cb
    res = cb.DeviceResources(0)
    yield cb, torch, res
    cb.set_coarse_check(True)
    res.close()


def _every_entry(env, base, queries, k):
    """(distances, indices) of the search, the batch, the serving loop and the
    allocation-free call."""
    cb, torch, res = env
    nq, d = queries.shape
    ix = cb.IndexBF(res, d, cb.IndexBFConfig(precision=FP8))
    ix.add(base.shape[0], base)
    out = {"search": [np.asarray(a) for a in ix.search_array(queries, k)]}
    q = torch.tensor(queries).cuda()

    def buffers():
        return torch.full((nq, k), -7, dtype=torch.int32, device="cuda"), torch.full((nq, k), -7.0, device="cuda")

    i, x = buffers()
    batch = cb.SearchBatch([(ix, q, k, i, x)])
    batch.run()
    out["batch"] = [x.cpu().numpy(), i.cpu().numpy()]
    batch.close()
    i, x = buffers()
    torch.cuda.synchronize()
    server = cb.Server(ix)
    server.wait(server.submit(q, k, i, x))
    out["server"] = [x.cpu().numpy(), i.cpu().numpy()]
    server.close()
    i, x = buffers()
    torch.cuda.synchronize()
    ix.search_noalloc(nq, q, k, i, x)
    out["noalloc"] = [x.cpu().numpy(), i.cpu().numpy()]
    ix.close()
    return out


# below and above the first size with a sample; codes that fill their last
# 128-byte chunk (the tail is a chunk of its own) and codes that do not
@pytest.mark.parametrize("n", [1000, 3000])
@pytest.mark.parametrize("d", [96, 128, 256])
@pytest.mark.parametrize("scale", [1e-12, 1e-30, 1e-33, 1e-36])
def test_queries_far_smaller_than_the_rows(env, n, d, scale):
    rng = np.random.default_rng(d + n)
    base = rng.random((n, d), dtype=np.float32)
    queries = (rng.random((5, d)) * scale).astype(np.float32)
    rd, ri = oracle.knn(base, queries, 11)
    for entry, (dist, idx) in _every_entry(env, base, queries, 10).items():
        assert (idx >= 0).all(), entry
        assert_knn_matches(base, queries, dist, idx, rd, ri)


# rows of 1e-19 have distances of 1e-36, in FP32's normal range, but a product of
# scales, 2 s_q s, below it; rows of 1e+16 the other way
@pytest.mark.parametrize("scale", [1e-19, 1e16])
@pytest.mark.parametrize("d", [96, 128])
def test_rows_at_the_ends_of_the_range(env, d, scale):
    rng = np.random.default_rng(d)
    base = (rng.random((1500, d)) * scale).astype(np.float32)
    queries = (rng.random((5, d)) * scale).astype(np.float32)
    queries[3] *= np.float32(1e-3)
    rd, ri = oracle.knn(base, queries, 11)
    for entry, (dist, idx) in _every_entry(env, base, queries, 10).items():
        assert (idx >= 0).all(), entry
        assert_knn_matches(base, queries, dist, idx, rd, ri)


# Rows whose codes are exact, with norms around 8e5 that differ by a few units
# (2^-18 of them): 16 bits of a norm hold 4 units of half of it, so all rows would
# tie and the lowest rows -- not the nearest, which come last -- be taken as the
# 480 candidates.  The distances of the 10 nearest are at most 1.5 and those of the
# other rows at least 2.5, and FP32 resolves 0.06 there.  `top` 448 and 300: a
# query scale of one, and one whose reciprocal is no short binary fraction.
@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("top", [448.0, 300.0])
def test_norms_keep_fp32_bits(env, d, top):
    cb, torch, res = env
    n, k = 2000, 10
    rng = np.random.default_rng(d)
    row = np.zeros(d, np.float32)
    row[:4] = 448.0
    row[4:8] = 40.0, 13.0, 4.0, 2.0  # half of the norm is 401,408 + 894.5
    base = np.tile(row, (n, 1))
    far = np.array([[1.5, 0.5, 0, 0], [1.5, 0.5, 0.5, 0], [1, 1, 0.5, 0.5], [1.5, 1, 0, 0], [2, 0.5, 0, 0]], np.float32)
    near = np.array([[0.5, 0, 0, 0], [0.5, 0.5, 0, 0], [1, 0, 0, 0], [1, 0.5, 0, 0], [1, 0.5, 0.5, 0]], np.float32)
    base[:, d - 4:] = far[rng.integers(0, 5, n)]
    base[n - k:, d - 4:] = np.repeat(near, 2, axis=0)
    queries = np.tile(row * np.float32(top / 448.0), (3, 1))
    rd, ri = oracle.knn(base, queries, k)
    cb.set_coarse_check(False)
    out = _every_entry(env, base, queries, k)
    cb.set_coarse_check(True)
    for entry, (_, idx) in out.items():
        np.testing.assert_array_equal(np.sort(idx, axis=1), np.tile(np.arange(n - k, n), (3, 1)), err_msg=entry)
    assert (np.sort(ri, axis=1) == np.arange(n - k, n)).all()
