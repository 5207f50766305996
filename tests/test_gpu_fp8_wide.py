"""GPU: FP8 passes over wide rows, where the ring of a CTA of its own has three stages
or two (CTA pairs), with the norm tail inside the last chunk of codes and in a chunk
of its own, against the FP64 oracle.  Run with -m gpu on a B200."""
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


@pytest.mark.parametrize("d", [704, 736, 737, 768, 769, 896, 1024, 1300])
@pytest.mark.parametrize("estimate", [True, False])
def test_wide_rows(env, d, estimate):
    cb, res = env
    rng = np.random.default_rng(d)
    n, nq, k = 40_001, 513, 10
    base = rng.standard_normal((n, d)).astype(np.float32)
    queries = (base[rng.choice(n, nq)] + rng.normal(0.0, 0.2, (nq, d))).astype(np.float32)
    ix = cb.IndexBF(res, d, cb.IndexBFConfig(precision=2))
    ix.add(n, base)
    cb.set_bound_estimate(estimate)
    dist, idx = ix.search_array(queries, k)
    cb.set_bound_estimate(True)
    ix.close()
    rd, ri = oracle.knn(base, queries, k + 1)
    assert_knn_matches(base, queries, np.asarray(dist), np.asarray(idx), rd, ri)
