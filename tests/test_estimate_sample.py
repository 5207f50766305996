"""CPU: the estimate a search starts from, regular or light (host logic, no device
needed)."""
import math
import random

import pytest
from scipy.stats import binom

import curplsh_b200 as cb


@pytest.mark.parametrize("n,nq,kp", [(10**6, 10000, 128), (10**7, 100, 416)])
def test_regular_samples_are_reported_as_planned(n, nq, kp):
    rows, step, block_rows, rank = cb.estimate_sample_shape(n, nq, kp)
    assert (rows, step, rank) == cb.estimate_plan_shape(n, nq, kp) and rows > 0 and block_rows == 128


# k = 10 and 1,024, few rows and many; none below 2,048 rows or four times k'
@pytest.mark.parametrize("n,nq,kp", [(3000, 1, 32), (10**4, 100, 32), (300_000, 1000, 1056), (2 * 10**6, 16, 32)])
def test_light_samples_are_reported(n, nq, kp):
    assert cb.estimate_plan_shape(n, nq, kp)[0] == 0
    rows, step, block_rows, rank = cb.estimate_sample_shape(n, nq, kp)
    assert rows > 0 and rows % 256 == 0 and block_rows in (8, 128) and 1 <= rank <= rows // block_rows


@pytest.mark.parametrize("n,kp", [(2047, 32), (4000, 1056), (0, 1)])
def test_shapes_without_a_sample(n, kp):
    assert cb.estimate_sample_shape(n, 100, kp) == (0, 1, 0, 0)


def test_bad_shapes_are_refused():
    with pytest.raises(cb.CurplshError):
        cb.estimate_sample_shape(-1, 10, 100)
    with pytest.raises(cb.CurplshError):
        cb.estimate_sample_shape(10**6, 10, 100, num_sms=0)


def _light_shapes():
    r = random.Random(11)
    for _ in range(400):
        n = int(2048 * 2 ** r.uniform(0, 12))
        kp = max(1, min(n // 4, int(2 ** r.uniform(0, 11))))
        nq = int(2 ** r.uniform(0, 13))
        if cb.estimate_plan_shape(n, nq, kp)[0] == 0 and cb.estimate_sample_shape(n, nq, kp)[0]:
            yield n, nq, kp


def test_light_samples_are_spread_over_the_rows():
    """The sample covers the rows it is taken from evenly, four fifths of the
    database at the least, and its rank holds when all k' nearest lie among those:
    the chance that more blocks hold one of them is at most 1e-6."""
    shapes = list(_light_shapes())
    assert len(shapes) > 100
    for n, nq, kp in shapes:
        rows, step, block_rows, rank = cb.estimate_sample_shape(n, nq, kp)
        assert 0.8 * n <= rows * step <= n, (n, nq, kp, rows, step)
        q = -math.expm1(block_rows * math.log1p(-kp / (rows * step)))
        tail = binom.sf(rank - 1, rows // block_rows, q)
        assert tail <= 1e-6, (n, nq, kp, rows, step, block_rows, rank, tail)
