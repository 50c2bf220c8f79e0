"""Block permutation over the forms its work items take: every permutation of rank 2 to 4 (and some
of rank 5) blocks with unit, short, 16 / 17, tile-sized and long extents, real and complex with
fermionic signs. A permutation moves bits, so the result must equal numpy's exactly."""
import itertools

import numpy as np
import pytest

from tensortoolkit_gb300.api import DTensor, TransposePlan
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

pytestmark = pytest.mark.gpu

DIMS = {2: [(1, 5), (2, 700), (3, 3), (31, 33), (33, 65), (16, 17), (2000, 3), (177, 146), (1100, 1)],
        3: [(3, 40, 61), (61, 3, 40), (40, 61, 3), (5, 6, 7), (16, 33, 2), (2, 2, 600), (17, 18, 19), (1, 70, 4),
            (3, 1500, 2)],
        4: [(3, 20, 2, 33), (2, 3, 4, 5), (33, 2, 2, 40), (7, 1, 9, 30)],
        5: [(3, 12, 2, 2, 21), (2, 3, 2, 3, 2)]}


def _tensor(shapes, dtype, rng):
    """One tensor whose blocks have these shapes: sector i of every leg belongs to block i."""
    rank, n = len(shapes[0]), len(shapes)
    qn = np.stack([np.arange(n), np.arange(n)], 1)   # the second component's oddness is the parity
    legs = [Leg(IN if l % 2 else OUT, qn, [s[l] for s in shapes], 1 if dtype is np.complex128 else -1)
            for l in range(rank)]
    data = rng.standard_normal(sum(int(np.prod(s)) for s in shapes)).astype(dtype)
    if dtype is np.complex128:
        data += 1j * rng.standard_normal(data.size)
    return BSTensor(legs, np.tile(np.arange(n).reshape(-1, 1), (1, rank)), dtype, data)


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("rank", [2, 3, 4, 5])
def test_every_permutation(gpu, rank, dtype):
    rng = np.random.default_rng(rank)
    t = _tensor(DIMS[rank], dtype, rng)
    d = DTensor.from_host(t)
    perms = list(itertools.permutations(range(rank)))
    for perm in perms if rank < 5 else perms[::7]:
        got = TransposePlan(t, perm).execute(d).to_host()
        for b in range(t.nblk):
            ref = t.block(b).transpose(perm)
            if dtype is np.complex128 and b % 2:   # every leg odd: the sign of the permutation
                swaps = sum(perm[i] > perm[j] for i in range(rank) for j in range(i + 1, rank))
                ref = -ref if swaps & 1 else ref
            assert np.array_equal(got.block(b), ref), (perm, t.block(b).shape)
