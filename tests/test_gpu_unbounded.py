"""GPU: searches whose candidate pools start without a bound (the estimate off, the
allocation-free call, batches): single blocks, CTA pairs and FP8 dual blocks, one
tile per unit and many, pools from nearly empty to full, against the FP64 oracle.
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
    cb.set_bound_estimate(False)
    yield cb, torch, res
    cb.set_bound_estimate(True)
    res.close()


# (form, d, rows, queries, k): d = 200 FP32-exact and 320 BF16 run 600 queries as
# pairs, FP8 as dual blocks; rows at the edges of a tile, of one tile per CTA and of
# pools that a unit's end selects or leaves; `spread` 100 gives FP8 a scale per row
CASES = [(0, 64, 255, 5, 1), (0, 64, 300, 600, 100), (0, 64, 20_011, 3, 1000), (0, 200, 257, 600, 10),
         (0, 200, 1500, 600, 100), (0, 200, 40_000, 513, 10), (1, 64, 1537, 600, 100), (1, 320, 9000, 600, 10),
         (1, 320, 700, 600, 200), (2, 64, 481, 600, 10), (2, 128, 8000, 600, 10), (2, 64, 2000, 5, 100)]


@pytest.mark.parametrize("form,d,n,nq,k,spread", [(*c, 1.0) for c in CASES] + [(*c, 100.0) for c in CASES if c[0] == 2])
def test_unbounded_searches(env, form, d, n, nq, k, spread):
    cb, torch, res = env
    rng = np.random.default_rng(n + d)
    base = rng.standard_normal((n, d)).astype(np.float32)
    base[::3] *= np.float32(spread)
    queries = rng.standard_normal((nq, d)).astype(np.float32)
    k = min(k, n)
    rd, ri = oracle.knn(base, queries, min(k + 1, n))
    ix = cb.IndexBF(res, d, cb.IndexBFConfig(precision=form))
    ix.add(n, base)
    out = {"search": ix.search_array(queries, k)}
    q = torch.tensor(queries).cuda()
    for entry in ("batch", "noalloc"):
        i = torch.full((nq, k), -7, dtype=torch.int32, device="cuda")
        x = torch.full((nq, k), -7.0, device="cuda")
        torch.cuda.synchronize()
        if entry == "batch":
            # the same rows in another index: a launch of several items
            other = cb.IndexBF(res, d, cb.IndexBFConfig(precision=form))
            other.add(n, base)
            i2, x2 = torch.full_like(i, -7), torch.full_like(x, -7.0)
            batch = cb.SearchBatch([(ix, q, k, i, x), (other, q, k, i2, x2)])
            batch.run()
            batch.close()
            other.close()
            out["second item"] = (x2.cpu().numpy(), i2.cpu().numpy())
        else:
            ix.search_noalloc(nq, q, k, i, x)
        out[entry] = (x.cpu().numpy(), i.cpu().numpy())
    ix.close()
    for entry, (dist, idx) in out.items():
        assert_knn_matches(base, queries, np.asarray(dist), np.asarray(idx), rd, ri)
