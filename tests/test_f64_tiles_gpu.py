"""FP64 GEMM tiles at their edges: blocks of one row or column, remainders of the 8 x 4 pieces and
of the 16-column tiles, tasks shorter and longer than the operand prefetch, few tiles (shared by a
CTA's warps) and many (one per warp). Operands are small integers, so every sum is exact in FP64
and the result must equal numpy's bit for bit."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

# (rows, contracted extent, columns): the last two have more tiles than four per sub-partition
SHAPES = [(9, 1, 9), (1, 130, 17), (7, 9, 31), (8, 3, 16), (33, 64, 12), (17, 513, 41), (485, 5, 661),
          (16, 33, 20000)]


def _leg(q, d, direction):
    return Leg(direction, np.asarray([[x] for x in q]), np.asarray(d))


@pytest.mark.parametrize("rows", [32, 64])
@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_tile_edges(gpu, m, k, n, dtype, rows):
    rng = np.random.default_rng(m * 1000 + k * 10 + n)

    def tensor(legs, coords):
        size = sum(int(np.prod([l.dims[c] for l, c in zip(legs, x)])) for x in coords)
        data = rng.integers(-8, 9, size).astype(dtype)
        if dtype is np.complex128:
            data += 1j * rng.integers(-8, 9, size)
        return BSTensor(legs, np.asarray(coords), dtype, data)

    # two contracted sectors feed one output block (two tasks), a third block stands alone
    x, y = _leg([0, 1], [m, 9], IN), _leg([0, 1], [n, 10], OUT)
    u, v = _leg([0, 1], [k, k + 1], OUT), _leg([0, 1], [1, 2], OUT)
    a = tensor([x, u, v], [(0, 0, 0), (0, 1, 1), (1, 1, 0)])
    b = tensor([u.inverse(), v.inverse(), y], [(0, 0, 0), (1, 0, 1), (1, 1, 0)])
    plan = ContractionPlan(a, b, [[1, 2], [0, 1]])
    plan.set_schedule(f64_tile_rows=rows)
    c = plan.execute(DTensor.from_host(a), DTensor.from_host(b)).to_host()
    ref = np.tensordot(a.to_dense(), b.to_dense(), ([1, 2], [0, 1]))
    assert np.array_equal(c.to_dense(), ref)
