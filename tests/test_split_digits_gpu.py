"""Split precision at the edges of its digits and of its accumulation: contracted extents around
the 160 between two drains and the 1920 between two folds, row and column remainders of the
128 x 32 tiles, values whose digits are all at a limit.

Small integers have no digits below the ones kept, so their result must equal numpy's bit for
bit. Otherwise an element is off by at most 2^-49 of its scale (2^e, e the exponent of its row's
or column's largest value: at most twice that value), the products left out add at most
(5 x 2^14) 2^-64 of both scales and a hundredth more for the higher levels, level 6's rounding in
FP32 two units of 2^-48 per drain and level 7's conversion 2^-52: with k products,
    |error| <= (k (2 + 2.6) + 6 drains) 2^-49 x (2 max|a_i|) (2 max|b_j|) + folds 2^-52 |c|
"""
import numpy as np
import pytest

from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 9, 9), (129, 159, 33), (40, 160, 40), (5, 161, 31), (130, 176, 9), (24, 1920, 24), (24, 1921, 40),
          (9, 4000, 10)]
# (Y + bias) 2^-48 patterns: first digit 256, digits all -128, all 127, alternating, one ulp
LIMITS = np.concatenate([np.asarray([1 - 2.0**-53, 0.5, 1 - 2.0**-49, 2.0**-49, 2.0**-48]),
                         np.asarray([(255 << 40) - 0x8080808080, (255 << 40) + 0x7F7F7F7F7F,
                                     (200 << 40) + 0x7F7F7F7F7F - 0x7F807F807F, 0x7F7F7F7F7F], dtype=np.float64)
                         * 2.0**-48])


def _operands(m, k, n, kind, rng):
    if kind == "integers":
        return rng.integers(-100, 101, (m, k)).astype(float), rng.integers(-100, 101, (k, n)).astype(float)
    if kind == "normal":
        return rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if kind == "one value":     # every product the same: the largest level sums
        return np.full((m, k), LIMITS[5]), np.full((k, n), LIMITS[6])
    return (rng.choice(LIMITS, (m, k)) * rng.choice([-1, 1], (m, k)),
            rng.choice(LIMITS, (k, n)) * rng.choice([-1, 1], (k, n)))


@pytest.mark.parametrize("kind", ["integers", "normal", "one value", "limits"])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_digits(gpu, m, k, n, kind):
    A, B = _operands(m, k, n, kind, np.random.default_rng(m + 10 * k + n))
    leg = lambda d, direction: Leg(direction, np.asarray([[0]]), np.asarray([d]))
    inner = leg(k, OUT)
    one = np.asarray([[0, 0]])
    a = BSTensor([leg(m, IN), inner], one, np.float64, A.ravel())
    b = BSTensor([inner.inverse(), leg(n, OUT)], one, np.float64, B.ravel())
    plan = ContractionPlan(a, b, [[1], [0]])
    c = plan.execute(DTensor.from_host(a), DTensor.from_host(b), mode="split")
    plan.device_status()
    C = c.to_host().to_dense()
    if kind == "integers":
        assert np.array_equal(C, A @ B)
        return
    exact = A.astype(np.longdouble) @ B.astype(np.longdouble)
    bound = ((4.6 * k + 6 * -(-k // 160)) * 2.0**-47 * np.abs(A).max(1)[:, None] * np.abs(B).max(0)
             + -(-k // 1920) * 2.0**-52 * np.abs(exact))
    assert np.all(np.abs(C - exact) <= bound), float((np.abs(C - exact) / bound).max())


@pytest.mark.parametrize("m,k,n", [(1, 1, 9), (33, 3, 15), (130, 9, 16), (7, 63, 17), (40, 64, 33), (5, 66, 48), (129, 81, 10)])
def test_digits_complex(gpu, m, k, n):
    """Complex operands (B sliced as its real 2k x 2n form): column remainders of the 16-column
    tiles, row remainders of the 4-row pieces. Integers, and halves of them on one side in every
    third row, so rows and columns have different scales: the results are exact."""
    rng = np.random.default_rng(m + 10 * k + n)

    def ints(*shape):
        x = rng.integers(-90, 91, shape) + 1j * rng.integers(-90, 91, shape)
        x[::3] *= 0.5
        return x

    A, B = ints(m, k), ints(k, n)
    B[:, n // 2] = 0
    B[:, n - 1] = B[:, n - 1].real
    leg = lambda d, direction: Leg(direction, np.asarray([[0]]), np.asarray([d]))
    inner = leg(k, OUT)
    one = np.asarray([[0, 0]])
    a = BSTensor([leg(m, IN), inner], one, np.complex128, A.ravel())
    b = BSTensor([inner.inverse(), leg(n, OUT)], one, np.complex128, B.ravel())
    plan = ContractionPlan(a, b, [[1], [0]])
    c = plan.execute(DTensor.from_host(a), DTensor.from_host(b), mode="split")
    plan.device_status()
    assert np.array_equal(c.to_host().to_dense(), A @ B)
