"""The SVD does not depend on the data's unit: scaled by a power of four (exact in every step, the
squared norms stay normal FP64 numbers), the singular values scale exactly and the vectors keep every
bit. The scales take the squared norms past FP32's range both ways. Pairs of nearly equal columns
become small ones by rotations that take away most of a column's norm."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import SVD, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

SHAPES = [(17, 16), (40, 33), (64, 64), (110, 111), (290, 200)]


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("near", [1e-6, 1e-9, 1e-12])
@pytest.mark.parametrize("power", [-100, 100])
def test_power_of_two_scale(gpu, power, near, dtype):
    rng = np.random.default_rng(5)
    mats = []
    for r, c in SHAPES:
        x, d = rng.standard_normal((r, c)).astype(dtype), rng.standard_normal((r, c)).astype(dtype)
        if dtype is np.complex128:
            x, d = x + 1j * rng.standard_normal((r, c)), d + 1j * rng.standard_normal((r, c))
        x[:, 1::2] = x[:, :c - c % 2:2] + near * d[:, 1::2]
        mats.append(x)
    n = len(SHAPES)
    qn = np.arange(n).reshape(-1, 1)
    legs = [Leg(IN, qn, [r for r, _ in SHAPES]), Leg(OUT, qn, [c for _, c in SHAPES])]
    data = np.concatenate([x.reshape(-1) for x in mats])

    def svd(values):
        t = BSTensor(legs, np.stack([np.arange(n)] * 2, 1), dtype, values)
        return [x.to_host().data for x in SVD(DTensor.from_host(t), 1, [0], 0.0, 0, 10 ** 6)[:3]]

    u, s, vt = svd(data)
    u2, s2, vt2 = svd(data * 2.0**power)
    assert np.array_equal(s2, s * 2.0**power)
    assert np.array_equal(u2, u) and np.array_equal(vt2, vt)
