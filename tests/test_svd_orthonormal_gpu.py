"""The SVD's left vectors are Q J with J the rotations of the FP32 start, made orthonormal by two
Newton-Schulz steps up to 256 columns and three past them, then rotated in FP64: at the sizes around
that line, on data that keep the FP32 start at work, J's columns must be orthonormal to FP64. Bound:
16 q eps (Householder Q and the products a few q eps, the last sweeps' rotations 2 eps each on a
column). A deviation of 1e-4 after the FP32 start is 4e-17 after two steps; one of 1.5e-3, or one step
too few, would miss the bound."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import SVD, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

EPS = 2.0**-52


def _matrix(rng, q, kind, dtype):
    x = rng.standard_normal((q + 3, q)).astype(dtype)
    if dtype is np.complex128:
        x = x + 1j * rng.standard_normal((q + 3, q))
    if kind == "pairs":         # small columns of FP32 rounding size appear
        x[:, 1::2] = x[:, :q - q % 2:2] + 1e-9 * x[:, 1::2]
    elif kind == "parallel":    # every angle near 45 degrees
        x = x[:, :1] + 1e-3 * x
    elif kind == "graded":
        x = x * np.exp(-30.0 * np.arange(q) / q)[rng.permutation(q)]
    return x


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("kind", ["normal", "pairs", "parallel", "graded"])
@pytest.mark.parametrize("q", [255, 256, 257, 400])
def test_left_vectors(gpu, q, kind, dtype):
    x = _matrix(np.random.default_rng(q), q, kind, dtype)
    one = np.asarray([[0, 0]])
    legs = [Leg(IN, [[0]], [q + 3]), Leg(OUT, [[0]], [q])]
    u, s, vt, _, kept = SVD(DTensor.from_host(BSTensor(legs, one, dtype, x.ravel())), 1, [0], 0.0, 0, q)
    assert kept == q
    ub, sb, vb = u.to_host().block(0), np.diagonal(s.to_host().block(0)), vt.to_host().block(0)
    assert np.abs(ub.conj().T @ ub - np.eye(q)).max() <= 16 * q * EPS
    assert np.linalg.norm((ub * sb) @ vb - x) <= 1e-12 * np.linalg.norm(x)
