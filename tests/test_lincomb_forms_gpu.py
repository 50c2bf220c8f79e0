"""LinearCombine over tensors that hold different blocks, at the kernel's work-item edges: FP64 and
complex, absent contributions, zero coefficients, a result kept at beta = 0 (its own blocks become
zeros: work items without contributions), results in place and expanded. Small integers: sums and
complex products are exact, so the result must equal numpy's bit for bit."""
import numpy as np
import pytest

from tensortoolkit_gb300 import api
from tensortoolkit_gb300.api import DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

FEW = [1, 31, 32, 33, 255, 256, 257, 513, 769, 1023, 1024, 1025, 2049, 4095, 4096, 4097, 9000]
MANY = [1 + (7 * i) % 300 for i in range(4000)] + [1025, 4097, 5000]


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("sizes", [FEW, MANY], ids=["few", "many"])
@pytest.mark.parametrize("beta,keep", [(0, False), (0, True), (2, False)])
def test_different_blocks(gpu, sizes, dtype, beta, keep):
    n = len(sizes)
    qn = np.arange(n).reshape(-1, 1)
    legs = [Leg(IN, qn, [1] * n), Leg(OUT, qn, sizes)]
    rng = np.random.default_rng(n)
    ints = lambda k: (rng.integers(-9, 10, k) + (1j * rng.integers(-9, 10, k) if dtype is np.complex128 else 0)).astype(dtype)

    def tensor(held):
        held = np.asarray(held)
        return BSTensor(legs, np.stack([held, held], 1), dtype, ints(sum(sizes[b] for b in held)))

    # the first contributes nothing, its own blocks do not appear
    ts = [tensor([b for b in range(n) if b % 5 != 0]), tensor([b for b in range(n) if b % 3 == 0]),
          tensor([b for b in range(n) if b % 4 == 1])]
    coefs = [0, 3 - 1j, -2j] if dtype is np.complex128 else [0, 3, -2]
    res = tensor([b for b in range(n) if b % 5 == 0 or b % 7 == 1])
    expect = {}
    for c, t in zip(coefs, ts):
        for i, b in enumerate(t.coords[:, 0] if c != 0 else []):
            x = c * t.block(i)
            expect[int(b)] = expect[int(b)] + x if int(b) in expect else x
    if beta or keep:
        for i, b in enumerate(res.coords[:, 0]):
            x = beta * res.block(i)
            expect[int(b)] = expect[int(b)] + x if int(b) in expect else x
    got = api.LinearCombine(coefs, [DTensor.from_host(t) for t in ts], beta, DTensor.from_host(res), keep).to_host()
    assert [int(b) for b in got.coords[:, 0]] == sorted(expect)
    assert np.array_equal(got.data, np.concatenate([expect[b].ravel() for b in sorted(expect)]))


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("sizes", [FEW, MANY], ids=["few", "many"])
def test_in_place(gpu, sizes, dtype):
    """x holds every other block of y: the sum goes into y's buffer, y's other blocks pass through."""
    n = len(sizes)
    qn = np.arange(n).reshape(-1, 1)
    legs = [Leg(IN, qn, [1] * n), Leg(OUT, qn, sizes)]
    rng = np.random.default_rng(n + 1)
    ints = lambda k: (rng.integers(-9, 10, k) + (1j * rng.integers(-9, 10, k) if dtype is np.complex128 else 0)).astype(dtype)
    half = np.arange(0, n, 2)
    y = BSTensor(legs, np.stack([np.arange(n)] * 2, 1), dtype, ints(sum(sizes)))
    x = BSTensor(legs, np.stack([half] * 2, 1), dtype, ints(sum(sizes[b] for b in half)))
    alpha = 2 - 3j if dtype is np.complex128 else -3
    dy = DTensor.from_host(y)
    got = api.AddScaledAssign(dy, alpha, DTensor.from_host(x))
    assert got is dy
    blocks = [y.block(b) + (alpha * x.block(b // 2) if b % 2 == 0 else 0) for b in range(n)]
    assert np.array_equal(got.to_host().data, np.concatenate([b.ravel() for b in blocks]))
