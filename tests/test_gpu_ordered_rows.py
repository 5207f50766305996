"""GPU: samples of rows that were added in some order.  A light sample must hold
its rank when a query's neighbours all lie in one part of the rows: the search
answers as without a sample, and (almost) no query is searched again.  Run with
-m gpu on a B200."""
import numpy as np
import pytest

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


def _check(env, base, queries, k):
    """Results with and without a sample are equal and no query fails its estimate
    (the rank's failure probability is at most 1e-6 a query)."""
    cb, res = env
    n, d = base.shape
    ix = cb.IndexBF(res, d, cb.IndexBFConfig(precision=0))
    ix.add(n, base)
    assert ix.estimate_plan(len(queries), k)[0] == 0 and ix.estimate_sample(len(queries), k)[0] > 0
    d1, i1 = ix.search_array(queries, k)
    failed = ix.fallback_count()
    cb.set_bound_estimate(False)
    d0, i0 = ix.search_array(queries, k)
    cb.set_bound_estimate(True)
    ix.close()
    np.testing.assert_array_equal(i1, i0)
    np.testing.assert_array_equal(d1, d0)
    assert failed == 0


# (rows, queries, k): sample blocks of 8 and of 128 rows, whose step used to be 1 and 3
SHAPES = [(30_000, 1000, 100), (300_000, 200, 1024), (100_000, 100, 10)]


@pytest.mark.parametrize("n,nq,k", SHAPES)
@pytest.mark.parametrize("first", [0.3, 0.5, 0.75, 1.0])
def test_two_sets_added_one_after_the_other(env, n, nq, k, first):
    rng = np.random.default_rng(n)
    base = rng.random((n, 48), dtype=np.float32)
    base[int(n * first):] += 3.0
    _check(env, base, rng.random((nq, 48), dtype=np.float32), k)


# periods that divide the old steps (2, 3, 4) and some that do not; the FP8 forms of
# one scale and of a scale per row read norms and scales at the sampled rows too
@pytest.mark.parametrize("n,nq,k", SHAPES)
@pytest.mark.parametrize("period", [2, 3, 4, 10])
def test_rows_interleaved_with_a_period(env, n, nq, k, period):
    rng = np.random.default_rng(n + period)
    base = rng.random((n, 48), dtype=np.float32) + np.float32(3.0) * (np.arange(n) % period)[:, None].astype(np.float32)
    _check(env, base, rng.random((nq, 48), dtype=np.float32), k)


@pytest.mark.parametrize("form,spread", [(0, 1.0), (1, 1.0), (2, 1.0), (2, 1000.0)])
@pytest.mark.parametrize("n,nq,k", [(2048, 600, 20), (20_011, 70, 50)])
def test_forms_agree_with_and_without_a_light_sample(env, form, spread, n, nq, k):
    cb, res = env
    rng = np.random.default_rng(n + form)
    base = rng.standard_normal((n, 72)).astype(np.float32)
    base[rng.random(n) < 0.5] *= np.float32(spread)
    queries = base[rng.choice(n, nq)] + rng.normal(0.0, 0.1, (nq, 72)).astype(np.float32)
    ix = cb.IndexBF(res, 72, cb.IndexBFConfig(precision=form, rerankFactor=6 if form else 0))
    ix.add(n, base)
    assert ix.estimate_plan(nq, k)[0] == 0 and ix.estimate_sample(nq, k)[0] > 0
    d1, i1 = ix.search_array(queries.astype(np.float32), k)
    failed = ix.fallback_count()
    cb.set_bound_estimate(False)
    d0, i0 = ix.search_array(queries.astype(np.float32), k)
    cb.set_bound_estimate(True)
    ix.close()
    np.testing.assert_array_equal(i1, i0)
    np.testing.assert_array_equal(d1, d0)
    assert failed == 0


def _sampled_rows(n, rows, step):
    """Database rows of a light sample (curplsh_index_estimate_sample)."""
    i = np.arange(rows, dtype=np.uint64)
    phase = ((i // 256 * 2654435769) % 2**32 * step) >> np.uint64(32) if n > 63 * 256 else 0
    return (i * step + phase).astype(np.int64)


# sample blocks of 8 and of 128 rows; host arrays (the host searches failed queries
# again) and device arrays (the stream does)
@pytest.mark.parametrize("n,nq,k", [(10_000, 2, 10), (300_000, 200, 10)])
@pytest.mark.parametrize("host", [True, False])
def test_a_light_sample_that_fails(env, n, nq, k, host):
    """Only the sampled rows are near the queries and the rank is below k' = 32, so
    every bound is too small."""
    import torch
    cb, res = env
    rng = np.random.default_rng(n)
    base = rng.random((n, 32), dtype=np.float32) + np.float32(50.0)
    queries = rng.random((nq, 32), dtype=np.float32)
    ix = cb.IndexBF(res, 32, cb.IndexBFConfig(precision=0))
    ix.add(n, base)
    assert ix.estimate_plan(nq, k)[0] == 0
    rows, step, _, rank = ix.estimate_sample(nq, k)
    at = _sampled_rows(n, rows, step)
    assert 0 < rank < 24 and at.max() < n and len(np.unique(at)) == rows
    ix.reset()
    base[at] -= np.float32(50.0)
    ix.add(n, base)

    def search():
        if host:
            return [np.asarray(a) for a in ix.search_array(queries, k)]
        i, x = torch.empty((nq, k), dtype=torch.int32, device="cuda"), torch.empty((nq, k), device="cuda")
        ix.search(nq, torch.tensor(queries).cuda(), k, i, x)
        torch.cuda.synchronize()
        return [x.cpu().numpy(), i.cpu().numpy()]

    d1, i1 = search()
    assert ix.fallback_count() == nq
    cb.set_bound_estimate(False)
    d0, i0 = search()
    cb.set_bound_estimate(True)
    ix.close()
    np.testing.assert_array_equal(i1, i0)
    np.testing.assert_array_equal(d1, d0)
