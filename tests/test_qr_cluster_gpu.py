"""QR where CTAs of a panel's cluster have no rows: a launch's cluster size comes from its tallest
block, so short blocks beside tall ones leave ranks idle, which reach the exchange with the other
CTAs' shared memory at once, while CTAs of the launch's later clusters are still starting. Many
clusters (more CTAs than the GPU holds), several calls. Compared with LAPACK (numpy) to 1e-11 relative:
the factors move by about eps times a block's condition number, below 400 for these."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import QR, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg, rel_frob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("tall", [65, 129, 300])   # clusters of 2, 4 and 8 CTAs
def test_ranks_without_rows(gpu, dtype, tall):
    shapes = [(1 + i % 9, 1 + i % 5) for i in range(400)]
    for i in range(0, 400, 57):
        shapes[i] = (tall - i % 3, 40)
    rng = np.random.default_rng(tall)
    data = rng.standard_normal(sum(m * n for m, n in shapes)).astype(dtype)
    if dtype is np.complex128:
        data += 1j * rng.standard_normal(data.size)
    qn = np.arange(len(shapes)).reshape(-1, 1)
    legs = [Leg(IN, qn, [m for m, _ in shapes]), Leg(OUT, qn, [n for _, n in shapes])]
    t = BSTensor(legs, np.stack([np.arange(len(shapes))] * 2, 1), dtype, data)
    refs = [np.linalg.qr(t.block(b)) for b in range(t.nblk)]
    d = DTensor.from_host(t)
    for _ in range(5):
        q, r = QR(d, 1, [0])
        q, r = q.to_host(), r.to_host()
        for b, (rq, rr) in enumerate(refs):
            assert rel_frob(q.block(b), rq) <= 1e-11, shapes[b]
            assert rel_frob(r.block(b), rr) <= 1e-11, shapes[b]
