"""Blocked Householder QR at its edges: one row or column, panels one short of and one past 32
columns, row counts around a cluster's share per CTA and around the update kernels' row chunks,
wide blocks, and panels too tall for shared memory. Compared per block with LAPACK (numpy), whose
reflector convention the kernels follow. Gaussian blocks: the factors of a square one move by
about eps times its condition number (below 1e4 at these sizes), hence 1e-11 relative."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import QR, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg, rel_frob

pytestmark = pytest.mark.gpu

SMALL = [(1, 1), (1, 7), (7, 1), (2, 2), (31, 32), (32, 31), (32, 32), (33, 33), (33, 70), (64, 33), (65, 32),
         (97, 65), (128, 40), (129, 33), (257, 64), (40, 200)]
TALL = {np.float64: [(513, 33), (6300, 34), (5, 5)], np.complex128: [(514, 33), (3100, 34), (5, 5)]}


def _blocks(shapes, dtype, seed):
    n = len(shapes)
    qn = np.arange(n).reshape(-1, 1)
    legs = [Leg(IN, qn, [m for m, _ in shapes]), Leg(OUT, qn, [k for _, k in shapes])]
    rng = np.random.default_rng(seed)
    data = rng.standard_normal(sum(m * k for m, k in shapes)).astype(dtype)
    if dtype is np.complex128:
        data += 1j * rng.standard_normal(data.size)
    return BSTensor(legs, np.stack([np.arange(n)] * 2, 1), dtype, data)


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("tall", [False, True])
def test_qr_block_shapes(gpu, dtype, tall):
    shapes = TALL[dtype] if tall else SMALL
    t = _blocks(shapes, dtype, 11)
    q, r = QR(DTensor.from_host(t), 1, [0])
    q, r = q.to_host(), r.to_host()
    for b, shape in enumerate(shapes):
        rq, rr = np.linalg.qr(t.block(b))
        if dtype is np.complex128:   # numpy's diagonal of R is real too (?geqrf)
            assert np.all(np.diagonal(rr).imag == 0)
        assert rel_frob(q.block(b), rq) <= 1e-11, shape
        assert rel_frob(r.block(b), rr) <= 1e-11, shape


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
def test_qr_panel_beside_update(gpu, dtype):
    """Enough work that the first updates are cut in two, the next panel running beside the second
    part (at least two 128-row items per SM), then not any more; some blocks have no second part,
    some no next panel. Tall blocks are well conditioned (below 20), the wide ones' leading squares
    at most 1e4: the bound above holds."""
    shapes = [(800, 640), (96, 640), (700, 500), (33, 600), (900, 420), (640, 96), (300, 65), (64, 64), (31, 40)]
    t = _blocks(shapes, dtype, 12)
    q, r = QR(DTensor.from_host(t), 1, [0])
    q, r = q.to_host(), r.to_host()
    for b, shape in enumerate(shapes):
        rq, rr = np.linalg.qr(t.block(b))
        assert rel_frob(q.block(b), rq) <= 1e-11, shape
        assert rel_frob(r.block(b), rr) <= 1e-11, shape
