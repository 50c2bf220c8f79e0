"""LinearCombine at the edges of its work items: block sizes around a warp, around the 256 elements
between a thread's own, around 1024 and 4096; few items (four CTAs share one) and more than the GPU
holds CTAs. Every product and sum is rounded by itself in the order of the tensors, so the result
must equal numpy's bit for bit (real: complex products use multiply-adds)."""
import numpy as np
import pytest

from tensortoolkit_gb300 import api
from tensortoolkit_gb300.api import DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

FEW = [1, 31, 32, 33, 255, 256, 257, 512, 513, 768, 769, 1023, 1024, 1025, 2049, 4095, 4096, 4097, 9000]
MANY = [1 + (7 * i) % 300 for i in range(4000)] + [1025, 4097, 5000]


@pytest.mark.parametrize("sizes", [FEW, MANY], ids=["few", "many"])
@pytest.mark.parametrize("n", [1, 2, 5])
def test_block_sizes(gpu, sizes, n):
    qn = np.arange(len(sizes)).reshape(-1, 1)
    legs = [Leg(IN, qn, [1] * len(sizes)), Leg(OUT, qn, sizes)]
    rng = np.random.default_rng(n)
    data = [rng.standard_normal(sum(sizes)) for _ in range(n)]
    coefs = rng.standard_normal(n)
    ts = [DTensor.from_host(BSTensor(legs, np.stack([np.arange(len(sizes))] * 2, 1), np.float64, d)) for d in data]
    ref = coefs[0] * data[0]
    for c, d in zip(coefs[1:], data[1:]):
        ref = ref + c * d
    assert np.array_equal(api.LinearCombine(list(coefs), ts).to_host().data, ref)
    # into the first tensor's own buffer
    got = api.AddScaledAssign(ts[0], 0.75, ts[-1] if n > 1 else DTensor.from_host(ts[0].to_host())).to_host().data
    assert np.array_equal(got, 0.75 * data[-1] + data[0])
