"""Skinny output blocks (n, k <= 8) at their edges: every n, row counts around the 32 outputs of a lane
range, the 128 of a pass and the 512 of a long list's item, entry counts around the unrolled pair,
operands read in place with strides. Small integers: sums are exact, so the result must equal
numpy's bit for bit."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu


def _leg(d, direction):
    return Leg(direction, np.arange(len(d)).reshape(-1, 1), np.asarray(d))


def _tensor(rng, legs, coords, dtype):
    size = sum(int(np.prod([l.dims[c] for l, c in zip(legs, x)])) for x in coords)
    data = rng.integers(-8, 9, size).astype(dtype)
    if dtype is np.complex128:
        data += 1j * rng.integers(-8, 9, size)
    return BSTensor(legs, np.asarray(coords), dtype, data)


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("rows", [1, 31, 33, 127, 129, 513, 300000])
def test_every_width(gpu, rows, dtype):
    if rows == 300000 and dtype is np.complex128:
        rows = 100000
    rng = np.random.default_rng(rows)
    # x: the long leg between two contracted ones (strided reads); 8 output columns sectors 1 .. 8
    ks, ns = [1, 2, 7, 8], [1, 2, 3, 4, 5, 6, 7, 8]
    u, x, v, y = _leg(ks, OUT), _leg([rows, 3], IN), _leg([1, 1], OUT), _leg(ns, OUT)
    a = _tensor(rng, [u, x, v], [(i, j, l) for i in range(4) for j in range(2) for l in range(2)], dtype)
    b = _tensor(rng, [u.inverse(), v.inverse(), y],
                [(i, l, c) for i in range(4) for l in range(2) for c in range(8) if (i + l + c) % 2 == 0], dtype)
    plan = ContractionPlan(a, b, [[0, 2], [0, 1]])
    got = plan.execute(DTensor.from_host(a), DTensor.from_host(b)).to_host().to_dense()
    assert np.array_equal(got, np.tensordot(a.to_dense(), b.to_dense(), ([0, 2], [0, 1])))
