"""The one rounding to FP64 of a split-precision sum: exact ties go to the even neighbour, whatever the
other outputs of the tile are (a tiny output beside them takes the kernel's general form of the
rounding, otherwise its short one runs). The sums are exact: ones, and one product of 2^-48 or
3 x 2^-48, half a last place of 32."""
from fractions import Fraction

import numpy as np
import pytest

from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("tiny_rows", [(), (3,), (3, 40, 77, 120)])
def test_ties_to_even(gpu, tiny_rows, sign):
    m, k, n = 130, 33, 17
    A = np.ones((m, k))
    A[:, -1] = 2.0**-23
    A[::2] *= sign
    for r in tiny_rows:
        A[r, :-1] = 0.0
    B = np.ones((k, n))
    B[-1] = 2.0**-25
    B[-1, 1::2] = 3 * 2.0**-25
    leg = lambda d, direction: Leg(direction, np.asarray([[0]]), np.asarray([d]))
    inner = leg(k, OUT)
    one = np.asarray([[0, 0]])
    a = BSTensor([leg(m, IN), inner], one, np.float64, A.ravel())
    b = BSTensor([inner.inverse(), leg(n, OUT)], one, np.float64, B.ravel())
    plan = ContractionPlan(a, b, [[1], [0]])
    c = plan.execute(DTensor.from_host(a), DTensor.from_host(b), mode="split")
    plan.device_status()
    F = np.vectorize(Fraction, otypes=[object])
    exact = (F(A) @ F(B)).astype(np.float64)   # a Fraction becomes a float by rounding to even
    assert np.array_equal(c.to_host().to_dense(), exact)
