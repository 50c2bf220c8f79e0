"""Split precision with every digit next to its limit and of one sign: the largest sums the FP32
accumulators meet between two drains. Level 5 stays exact just below 2^24; levels 6 and 7 pass it (the
test checks from the digits that they do). There the accumulator holds multiples of two units, and a
16-wide MMA may drop a unit of each product and of the sum: 17 units an MMA, in the last 5 (level 6,
units 2^-48) and 12 (level 7, units 2^-56) of a full period's. Against the exact sum of the kept
products the result may be off by that, half a unit of 2^-50 a period for the conversion of levels 6
and 7, and one rounding to FP64 of 2^-53 per fold of 24 periods. A level 5 past 2^24 (160 k
stretched to 192, emulated) is off by fifteen times that."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

DRAIN, FOLD = 160, 24 * 160
WEIGHTS = 2.0 ** (-8.0 * np.arange(1, 7))


def _digits(rng, *shape):
    """Six digits per value, the first 254 or 255, the others 126 or 127: sums with all low bits."""
    d = rng.integers(126, 128, shape + (6,))
    d[..., 0] += 128
    return d


def _level(da, db, level):
    return sum(da[..., p - 1] @ db[..., level - p - 1] for p in range(1, level) if p <= 6 and level - p <= 6)


@pytest.mark.parametrize("signs", ["positive", "negative", "rows"])
@pytest.mark.parametrize("m,k,n", [(130, 160, 33), (20, 320, 24), (40, 1000, 17), (9, 4000, 10)])
def test_largest_level_sums(gpu, m, k, n, signs):
    rng = np.random.default_rng(k)
    da, db = _digits(rng, m, k), _digits(rng, k, n)
    full = [_level(da[:, :DRAIN], db[:DRAIN], level).max() / 2**24 for level in (5, 6, 7)]
    assert 0.9 < full[0] < 1.0 < full[1] < 1.08 and 1.2 < full[2] < 1.24
    sign = {"positive": np.ones(m), "negative": -np.ones(m), "rows": np.where(np.arange(m) % 2, 1.0, -1.0)}[signs]
    A, B = (da @ WEIGHTS) * sign[:, None], db @ WEIGHTS   # exact: 48 bits
    leg = lambda d, direction: Leg(direction, np.asarray([[0]]), np.asarray([d]))
    inner = leg(k, OUT)
    one = np.asarray([[0, 0]])
    a = BSTensor([leg(m, IN), inner], one, np.float64, A.ravel())
    b = BSTensor([inner.inverse(), leg(n, OUT)], one, np.float64, B.ravel())
    plan = ContractionPlan(a, b, [[1], [0]])
    c = plan.execute(DTensor.from_host(a), DTensor.from_host(b), mode="split")
    plan.device_status()
    # integers in units of 2^-56, then the difference to the result in the same units, exactly
    kept = sum(_level(da, db, level).astype(object) << (8 * (7 - level)) for level in range(2, 8))
    got = c.to_host().to_dense() * sign[:, None]
    off = np.abs(np.vectorize(lambda x: int(x * 2.0**56), otypes=[object])(got) - kept).astype(np.float64)
    periods, folds = -(-k // DRAIN), -(-k // FOLD)
    bound = periods * (5 * 17 * 2**8 + 12 * 17 + 2**5) + folds * np.abs(got) * 2.0**3
    assert np.all(off <= bound), float((off / bound).max())
