"""Sector pairing on both sides of the line between its host and its device form (4096 pairs, 4096
blocks): task lists - blocks, shapes, fermionic signs, beta - and result topology equal the oracle's
exactly, for bosonic and fermionic tensors, in every matvec step, and down to a scalar result."""
import numpy as np
import pytest

from oracle import oracle
from tensortoolkit_gb300 import workloads
from tensortoolkit_gb300.api import ContractionPlan
from tensortoolkit_gb300.tensor import BSTensor, same_topology

pytestmark = pytest.mark.gpu

AXES = [[[0], [0]], [[0, 2], [0, 1]], [[4, 1], [0, 1]], [[4, 1], [1, 0]]]


def _check(a, b, ax):
    ref, tasks = oracle.contract(a, b, ax)
    plan = ContractionPlan(a, b, ax)
    assert np.array_equal(plan.tasks(), tasks)
    if ref.rank:
        assert same_topology(plan.result, ref)
    return ref, len(tasks)


@pytest.mark.parametrize("kind,size", [("u1", 400), ("fermionic", 3), ("fermionic", 5)])
def test_matvec_steps(gpu, kind, size):
    ops = workloads.heisenberg(size, 8, 2.5, 1) if kind == "u1" else workloads.hubbard(60 + 20 * size, size, 4)
    cur, pairs = ops[0], []
    for b, ax in zip(ops[1:], AXES):
        cur, n = _check(cur, b, ax)
        pairs.append(n)
    if kind == "fermionic":
        assert (max(pairs) < 4096) == (size == 3)   # one workload on each side of the line


@pytest.mark.parametrize("half", [2, 8])
def test_scalar_result(gpu, half):
    psi = workloads.hubbard(300, half, 4)[1]
    bra = BSTensor([leg.inverse() for leg in psi.legs], psi.coords, psi.dtype, np.conj(psi.data))
    _check(psi, bra, [[0, 1, 2, 3], [0, 1, 2, 3]])
