"""SVD at the edges of its Jacobi stages: blocks of one row or column, odd and even sizes around one
CTA's and a cluster's column blocks, a block past 256 columns (one more orthonormalisation step),
steep and flat spectra, equal singular values, rank-deficient and zero blocks, and data far from 1.
Per block against LAPACK (numpy): singular values within 1e-12 of the largest, factors rebuilding the
block to 1e-11, and kept vectors orthogonal as far as the Jacobi's stopping rule goes: it leaves pairs
whose inner product is below 64 eps, or below 64 eps ||A||_F over the smaller singular value."""
import numpy as np
import pytest

from tensortoolkit_gb300.api import SVD, DTensor
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 5), (5, 1), (2, 2), (3, 3), (2, 9), (17, 16), (16, 33), (31, 31), (64, 48), (110, 111), (130, 257),
          (290, 270)]


def _block(rng, m, n, dtype, kind):
    k = min(m, n)

    def ortho(r):
        x = rng.standard_normal((r, k)).astype(dtype)
        if dtype is np.complex128:
            x = x + 1j * rng.standard_normal((r, k))
        return np.linalg.qr(x)[0]

    s = {"flat": 1.0 + 0.3 * rng.random(k), "steep": np.exp(-30.0 * np.arange(k) / k), "equal": np.ones(k),
         "deficient": np.where(np.arange(k) < (k + 1) // 2, 1.0 + rng.random(k), 0.0), "zero": np.zeros(k)}[kind]
    return (ortho(m) * s) @ ortho(n).conj().T


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("kind,scale", [("flat", 1.0), ("steep", 1.0), ("equal", 1.0), ("deficient", 1.0),
                                        ("flat", 1e60), ("steep", 1e-60), ("zero", 1.0)])
def test_svd_block_shapes(gpu, kind, scale, dtype):
    n = len(SHAPES)
    rng = np.random.default_rng(n)
    mats = [_block(rng, r, c, dtype, kind) * scale for r, c in SHAPES]
    if kind == "zero":   # a whole tensor of zeros has no SVD here: one block keeps values
        mats[0] = np.full((1, 1), 3.0, dtype)
    qn = np.arange(n).reshape(-1, 1)
    legs = [Leg(IN, qn, [r for r, _ in SHAPES]), Leg(OUT, qn, [c for _, c in SHAPES])]
    t = BSTensor(legs, np.stack([np.arange(n)] * 2, 1), dtype, np.concatenate([x.reshape(-1) for x in mats]))
    u, s, vt, _, kept = SVD(DTensor.from_host(t), 1, [0], 0.0, 0, 10 ** 6)
    u, s, vt = u.to_host(), s.to_host(), vt.to_host()
    bond = {int(c[0]): i for i, c in enumerate(u.coords)}   # row sector -> its block
    total = 0
    for b, x in enumerate(mats):
        ref = np.linalg.svd(x, compute_uv=False)
        if b not in bond:
            assert ref[0] == 0.0
            continue
        i = bond[b]
        j = int(u.coords[i][1])
        ub, vb = u.block(i), vt.block([int(c[0]) for c in vt.coords].index(j))
        sb = np.diagonal(s.block([int(c[0]) for c in s.coords].index(j)))
        k = len(sb)
        total += k
        assert np.max(np.abs(sb - ref[:k])) <= 1e-12 * ref[0]
        assert k == len(ref) or ref[k] <= 1e-12 * ref[0]
        assert np.linalg.norm((ub * sb) @ vb - x) <= 1e-11 * np.linalg.norm(x)
        live = sb > 1e-13 * ref[0]   # values at the rounding level have no vectors of their own
        low = np.minimum.outer(sb[live], sb[live])
        bound = 2 * 64 * 2.2e-16 * (1 + np.linalg.norm(x) / low) + 1e-13
        for f in (ub[:, live], vb[live].conj().T):
            assert np.all(np.abs(f.conj().T @ f - np.eye(f.shape[1])) <= bound)
    assert total == kept
