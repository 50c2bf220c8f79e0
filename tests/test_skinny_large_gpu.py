"""A skinny output block of more than 2^31 elements (17 GB of FP64 values, 34 GB of complex ones): the
last outputs lie past 32-bit positions. Small integers, so the products must be exact."""
import numpy as np
import pytest
import torch

from tensortoolkit_gb300.api import ContractionPlan, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
def test_past_32_bits(gpu, dtype):
    m, n = 2**28 + 5, 8
    parts = 2 if dtype is np.complex128 else 1
    leg = lambda d, direction: Leg(direction, np.asarray([[0]]), np.asarray([d]))
    inner = leg(1, OUT)
    one = np.asarray([[0, 0]])
    ma = BSTensor([leg(m, IN), inner], one, dtype, None)
    B = np.arange(1, n + 1).astype(dtype) * (1 + 2j if parts == 2 else 1)
    b = BSTensor([inner.inverse(), leg(n, OUT)], one, dtype, B)
    plan = ContractionPlan(ma, b, [[1], [0]])
    gen = torch.Generator(device="cuda").manual_seed(1)
    buf = torch.randint(-99, 100, (m * parts,), generator=gen, device="cuda", dtype=torch.int8).double()
    out = DTensor.empty(plan.result)
    out.buf.fill_(float("nan"))
    plan.execute(DTensor(ma, buf), DTensor.from_host(b), out)
    col = torch.from_numpy(B).cuda()
    step = 2**25
    for r in range(0, m, step):
        rows = min(step, m - r)
        a = buf[r * parts:(r + rows) * parts]
        c = out.buf[r * n * parts:(r + rows) * n * parts]
        if parts == 2:
            a, c = torch.view_as_complex(a.view(-1, 2)), torch.view_as_complex(c.view(-1, 2))
        assert torch.equal(c.view(rows, n), a[:, None] * col[None]), r
    del out, buf, a, c
    torch.cuda.empty_cache()
