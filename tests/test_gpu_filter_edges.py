"""GPU: edges of the fused pass's filter, its samples and the merge -- the
shortest searches that start from a sample and the ones just below, sample
blocks of eight rows (large k'), FP8 norm tails in a chunk of their own, query
counts at the edges of single and dual blocks, many short candidate lists per
query -- against the FP64 oracle and against the same search without a sample.
Run with -m gpu on a B200."""
import numpy as np
import pytest

import oracle
from tests.knn_check import assert_knn_matches

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import curplsh_b200 as cb
    res = cb.DeviceResources(0)
    yield cb, res
    cb.set_bound_estimate(True)
    res.close()


def _rows(rng, n, d, kind):
    if kind == "ties":  # few distinct distances: the lower row wins
        return rng.integers(0, 3, (n, d)).astype(np.float32)
    x = rng.standard_normal((n, d)).astype(np.float32)
    return x / np.linalg.norm(x, axis=1, keepdims=True) if kind == "sphere" else x


def _check(env, n, nq, d, k, form, kind, seed):
    cb, res = env
    rng = np.random.default_rng(seed)
    base, queries = _rows(rng, n, d, kind), _rows(rng, nq, d, kind)
    ix = cb.IndexBF(res, d, cb.IndexBFConfig(precision=form))
    ix.add(n, base)
    out = []
    for est in (True, False):
        cb.set_bound_estimate(est)
        out.append([np.asarray(a) for a in ix.search_array(queries, k)])
    cb.set_bound_estimate(True)
    ix.close()
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][0], out[1][0])
    rd, ri = oracle.knn(base, queries, min(k + 1, n))
    assert_knn_matches(base, queries, out[0][0], out[0][1], rd, ri)


# the first size with a sample and the last without; a ragged last tile; k' a
# quarter of the rows and just above; 8-row sample blocks at k' > 1,000
@pytest.mark.parametrize("n,nq,k", [(2047, 3, 5), (2048, 3, 5), (2305, 130, 1), (5000, 17, 1000), (4096, 1, 1000),
                                    (20011, 129, 300), (70001, 40, 1024)])
@pytest.mark.parametrize("kind", ["normal", "ties"])
def test_short_searches_and_large_k(env, n, nq, k, kind):
    _check(env, n, nq, 24, k, 0, kind, n + nq)


# the norm tail inside the last chunk, filling it, and as a chunk of its own;
# one, three (single) and eight (dual) query blocks
@pytest.mark.parametrize("d", [96, 97, 100, 128, 130, 256, 640])
@pytest.mark.parametrize("nq", [5, 300, 1024])
def test_fp8_norm_tails(env, d, nq):
    _check(env, 9000, nq, d, 10, 2, "sphere", d + nq)


# few queries over many units: up to 148 short lists per query, and lists that
# do not fit the merge's shared buffer
@pytest.mark.parametrize("nq,k", [(1, 1), (2, 10), (16, 100), (5, 1024)])
@pytest.mark.parametrize("form", [0, 1])
def test_many_lists(env, nq, k, form):
    _check(env, 150001, nq, 32, k, form, "normal", 7 * nq + k)


@pytest.mark.parametrize("form", [0, 1, 2])
def test_rows_without_a_distance(env, form):
    """Rows holding NaN or infinity are no neighbours of anything, in whole
    eights of columns, alone in one, and with fewer than k rows left."""
    cb, res = env
    rng = np.random.default_rng(5)
    for n, bad in ((6000, list(range(8, 24)) + [100, 4095, 5999]), (3000, list(range(3, 3000)))):
        base = rng.standard_normal((n, 40)).astype(np.float32)
        queries = rng.standard_normal((70, 40)).astype(np.float32)
        base[bad, 3] = np.where(np.arange(len(bad)) % 2, np.nan, np.inf)
        ix = cb.IndexBF(res, 40, cb.IndexBFConfig(precision=form))
        ix.add(n, base)
        dist, idx = (np.asarray(a) for a in ix.search_array(queries, 10))
        ix.close()
        good = np.setdiff1d(np.arange(n), bad)
        rd, ri = oracle.knn(np.ascontiguousarray(base[good]), queries, min(10, len(good)))
        m = rd.shape[1]
        np.testing.assert_array_equal(idx[:, :m], good[ri])
        np.testing.assert_allclose(dist[:, :m], rd, rtol=1e-4)
        assert (idx[:, m:] == -1).all()
