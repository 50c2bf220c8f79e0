"""Complex tensors whose buffer starts at 8 modulo 16 bytes (any range of a float64 tensor): split
precision reads real values where nothing has to be transposed and no output block is skinny (small
integers, so the result must equal numpy's bit for bit); what works on whole elements refuses them."""
import numpy as np
import pytest
import torch

from tensortoolkit_gb300 import api
from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.capi import QltgError
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu


def _at_8(t):
    """t on the GPU, its buffer 8 bytes past a 16-byte boundary."""
    d = DTensor.from_host(t)
    buf = torch.empty(d.buf.numel() + 1, dtype=torch.float64, device=d.buf.device)[1:]
    buf.copy_(d.buf)
    assert buf.data_ptr() % 16 == 8
    return DTensor(d.meta, buf)


def _matrices(m, k, n):
    """A (m x k) and B (k x n) as tensors of one block each, complex integers."""
    rng = np.random.default_rng(m + k + n)

    def ints(*shape):
        return rng.integers(-90, 91, shape) + 1j * rng.integers(-90, 91, shape)

    leg = lambda d, direction: Leg(direction, np.asarray([[0]]), np.asarray([d]))
    inner = leg(k, OUT)
    one = np.asarray([[0, 0]])
    return (BSTensor([leg(m, IN), inner], one, np.complex128, ints(m, k).ravel()),
            BSTensor([inner.inverse(), leg(n, OUT)], one, np.complex128, ints(k, n).ravel()))


@pytest.mark.parametrize("m,k,n", [(1, 1, 9), (33, 3, 15), (130, 9, 16), (40, 64, 33), (5, 66, 48)])
def test_split_reads_real_values(gpu, m, k, n):
    a, b = _matrices(m, k, n)
    plan = ContractionPlan(a, b, [[1], [0]])
    da, db, out = _at_8(a), _at_8(b), _at_8(BSTensor(plan.result.legs, plan.result.coords, np.complex128,
                                                       np.zeros(m * n, np.complex128)))
    for x, y in [(DTensor.from_host(a), db), (da, DTensor.from_host(b)), (da, db)]:
        c = plan.execute(x, y, out, mode="split")
        plan.device_status()
        assert np.array_equal(c.to_host().to_dense(), a.to_dense() @ b.to_dense())


def test_whole_elements_refuse(gpu):
    a, b = _matrices(40, 24, 33)
    x, y = _at_8(a), _at_8(b)
    good_a, good_b = DTensor.from_host(a), DTensor.from_host(b)
    sa, sb = _matrices(24, 5, 6)   # k = 5, n = 6: a skinny block
    plan = ContractionPlan(a, b, [[1], [0]])
    out = plan.execute(good_a, good_b)
    skinny = ContractionPlan(sa, sb, [[1], [0]])
    swapped = api.TransposePlan(b, [1, 0])
    b_t = swapped.execute(good_b).to_host()
    transposing = ContractionPlan(a, b_t, [[1], [1]])
    refused = [lambda: plan.execute(x, good_b), lambda: plan.execute(good_a, y),
               lambda: plan.execute(good_a, good_b, _at_8(out.to_host())),
               lambda: skinny.execute(_at_8(sa), DTensor.from_host(sb), mode="split"),
               lambda: transposing.execute(good_a, _at_8(b_t), mode="split"),
               lambda: swapped.execute(y), lambda: api.Transpose(y, [1, 0]),
               lambda: api.LinearCombine([1.0, 2.0], [good_a, x]), lambda: api.AddScaledAssign(x, 2.0, good_a),
               lambda: api.ApplyAxisDiagonal(x, 0, np.ones(40)),
               lambda: api.ContractTailHeadContiguousAccumulate(good_a, good_b, 1, 0, 1, 1.0, 1.0, _at_8(out.to_host())),
               lambda: api.SVD(x, 1, [0], 0.0, 1, 40), lambda: api.QR(x, 1, [0])]
    for call in refused:
        with pytest.raises(QltgError, match="16-byte elements"):
            call()
    # nothing ran, the context is as it was
    assert np.array_equal(plan.execute(good_a, good_b).to_host().data, out.to_host().data)
