"""GPU: plans with less working memory.  A serving request whose ordinary plan is over
the server's budget runs on the lean plan, with the same results.  Run with -m gpu on
a B200."""
import re

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


# dual blocks, and CTA pairs (two pools per query and unit)
@pytest.mark.parametrize("form,d", [(2, 96), (1, 384)])
def test_request_between_the_two_plans_needs(env, form, d):
    cb, torch, res = env
    n, nq, k = 200_000, 600, 100
    rng = np.random.default_rng(d)
    base = rng.standard_normal((n, d)).astype(np.float32)
    queries = base[rng.choice(n, nq)] + rng.normal(0.0, 0.1, (nq, d)).astype(np.float32)
    queries = queries.astype(np.float32)
    ix = cb.IndexBF(res, d, cb.IndexBFConfig(precision=form))
    ix.add(n, base)
    q = torch.tensor(queries).cuda()
    i = torch.full((nq, k), -7, dtype=torch.int32, device="cuda")
    x = torch.full((nq, k), -7.0, device="cuda")
    torch.cuda.synchronize()
    batch = cb.SearchBatch([(ix, q, k, i, x)])
    ordinary = batch.info()[1]
    batch.close()
    server = cb.Server(ix, memory_budget=1 * MB)  # too small for either plan: the error says what the lean one needs
    with pytest.raises(cb.CurplshError) as err:
        server.submit(q, k, i, x)
    server.close()
    lean = int(re.search(r"needs (\d+) bytes", str(err.value)).group(1))
    assert lean < ordinary
    server = cb.Server(ix, memory_budget=(lean + ordinary) // 2)
    server.wait(server.submit(q, k, i, x))
    server.close()
    ix.close()
    rd, ri = oracle.knn(base, queries, k + 1)
    assert_knn_matches(base, queries, x.cpu().numpy(), i.cpu().numpy(), rd, ri)
