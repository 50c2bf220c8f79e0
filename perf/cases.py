"""What this framework is timed on: the calls of a DMRG sweep on block-sparse tensors.

A two-site sweep joins two site tensors (`contract`), applies the effective Hamiltonian
(`matvec`, `lanczos`), splits the state (`svd`, `qr`), grows an environment (`env`), reorders
legs for storage or for another code (`transpose`) and sums Krylov vectors (`lincomb`). Shapes
are the repository's own workloads: the U(1) Heisenberg chain (two-site sectors of Gaussian
degeneracies, MPO bond 5), the fermionic U(1)xU(1) complex Hubbard chain (400 sectors) and the
block-diagonal decomposition shapes; bond dimensions run from a chain's edge to D = 4000.
"""
from functools import lru_cache

import numpy as np
import torch

from tensortoolkit_gb300 import workloads
from tensortoolkit_gb300.api import (QR, SVD, AccumulatePlan, Contract, ContractionPlan, DTensor, Lanczos,
                                     LinearCombine, Matvec, TransposePlan)
from tensortoolkit_gb300.tensor import IN, OUT, BSTensor, Leg

HUBBARD_HALF = 10          # 20 x 20 sectors, the complex matvec's configuration
T0_LEGS = 5                # rank of lenv . psi, the largest tensor a sweep permutes


def listed():
    return [
        # a chain's edge: joining two small site tensors, planned and run once (latency)
        {"name": "contract_edge", "kind": "contract", "D": 37},
        # joining two site tensors in the middle of the chain, planned and run once
        {"name": "contract_bulk", "kind": "contract", "D": 1500},
        # growing the left environment by one site with kept plans (three contractions)
        {"name": "env_fp64", "kind": "env", "D": 640, "mode": "fp64"},
        # the largest real tensor of a D = 4000 sweep brought into another leg order
        {"name": "transpose_real", "kind": "transpose", "family": "u1", "D": 4000, "perm": "42310"},
        # a fermionic complex state (5544 small blocks) with its block signs
        {"name": "transpose_complex", "kind": "transpose", "family": "hubbard", "D": 4001, "perm": "2031"},
        # the effective Hamiltonian: small, plain FP64, and the headline size in split precision
        {"name": "matvec_small", "kind": "matvec", "family": "u1", "D": 250, "mode": "split"},
        {"name": "matvec_fp64", "kind": "matvec", "family": "u1", "D": 1000, "mode": "fp64"},
        {"name": "matvec_large", "kind": "matvec", "family": "u1", "D": 4000, "mode": "split"},
        # the same on the fermionic complex chain
        {"name": "matvec_hubbard", "kind": "matvec", "family": "hubbard", "D": 3000, "mode": "split"},
        # a bond's ground-state search: Krylov steps, then the lowest vector they span
        {"name": "lanczos", "kind": "lanczos", "D": 2000, "steps": 8},
        # splitting the two-site state and absorbing the singular values
        {"name": "svd", "kind": "svd", "D": 1501},
        # orthogonalising a site tensor of a wide bond: 41 block-matrices, 40 x 20 .. 1200 x 600
        {"name": "qr_wide", "kind": "qr", "blocks": 41, "lo": 20, "hi": 600},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["contract", "env", "transpose", "matvec", "matvec", "lanczos", "svd", "qr", "accumulate",
                       "lincomb"])
    if kind == "contract":
        return {"kind": kind, "D": _log(rng, 17, 1500)}
    if kind == "env":
        return {"kind": kind, "D": _log(rng, 60, 640), "mode": rng.choice(["fp64", "split"])}
    if kind == "transpose":
        family = rng.choice(["u1", "hubbard"])
        rank = T0_LEGS if family == "u1" else 4
        perm = list(range(rank))
        while perm == sorted(perm):
            rng.shuffle(perm)
        return {"kind": kind, "family": family, "D": _log(rng, 400, 4000), "perm": "".join(map(str, perm))}
    if kind == "matvec":
        family = rng.choice(["u1", "u1", "hubbard"])
        mode = rng.choice(["split", "split", "fp64"])
        hi = {("u1", "split"): 4000, ("u1", "fp64"): 1000, ("hubbard", "split"): 3000, ("hubbard", "fp64"): 1200}
        return {"kind": kind, "family": family, "D": _log(rng, 100 if family == "u1" else 450, hi[family, mode]),
                "mode": mode}
    if kind == "lanczos":
        return {"kind": kind, "D": _log(rng, 100, 2000), "steps": rng.randint(3, 8)}
    if kind == "svd":
        return {"kind": kind, "D": _log(rng, 60, 1501)}
    if kind == "qr":
        return {"kind": kind, "blocks": rng.randint(5, 41), "lo": rng.randint(1, 30), "hi": _log(rng, 40, 600)}
    if kind == "accumulate":
        return {"kind": kind, "D": _log(rng, 60, 640), "mode": rng.choice(["fp64", "split"])}
    return {"kind": kind, "D": _log(rng, 200, 4000), "n": rng.randint(2, 8)}


# ------------------------------------------------------------------ layouts
def _qmax(D):
    """Sectors of a U(1) bond: 61 at D = 4000, 41 at D = 2000 (the repository's cases), fewer below."""
    return max(3, min(30, int(round(30 * (D / 4000.0) ** 0.58))))


def _chain(D, seed):
    """(lenv, psi, mpo1, mpo2, renv) of the Heisenberg chain: symmetric environments, its MPO."""
    q = _qmax(D)
    return workloads.heisenberg(D, q, 0.3 * q, seed, hermitian=True)


@lru_cache(maxsize=4)
def _hubbard_layout(D):
    return workloads.hubbard(D, HUBBARD_HALF, 4)


@lru_cache(maxsize=8)
def _bond(D):
    psi = _chain(D, 1)[1]
    return psi.legs[0], psi.legs[1]


def _tensor(legs):
    """Every block of zero divergence over `legs`, in ascending block index."""
    tot = np.zeros([1] * len(legs), np.int64)
    for l, g in enumerate(legs):
        q = (g.qns[:, 0] if g.dir == OUT else -g.qns[:, 0]).astype(np.int64)
        tot = tot + q.reshape([-1 if i == l else 1 for i in range(len(legs))])
    return BSTensor(legs, np.argwhere(tot == 0), np.float64, None)


def _site(D):
    v, p = _bond(D)
    return _tensor([v, p, v.inverse()])


def _meta(t):
    return BSTensor(t.legs, t.coords, t.dtype, None, offsets=t.offsets, size=t.size)


def _normal(meta, g, scale=1.0):
    n = meta.size * (2 if meta.is_complex else 1)
    buf = torch.randn(max(n, 1), dtype=torch.float64, device="cuda", generator=g)
    return DTensor(_meta(meta), buf.mul_(scale))


def _dagger(m):
    return BSTensor([l.inverse() for l in m.legs], m.coords, m.dtype, None, offsets=m.offsets, size=m.size)


def _groups(t, ldims):
    """Block-matrices of the split after `ldims` legs: (blocks, row and column place of each, shape)."""
    out = {}
    shp = t.block_shapes()
    for b in range(t.nblk):
        c = tuple(int(x) for x in t.coords[b])
        flux = sum(int(t.legs[l].qns[c[l], 0]) * (1 if t.legs[l].dir == OUT else -1) for l in range(ldims))
        g = out.setdefault(flux, {"rows": {}, "cols": {}, "m": 0, "n": 0, "blk": []})
        m, n = int(np.prod(shp[b, :ldims])), int(np.prod(shp[b, ldims:]))
        if c[:ldims] not in g["rows"]:
            g["rows"][c[:ldims]] = g["m"]
            g["m"] += m
        if c[ldims:] not in g["cols"]:
            g["cols"][c[ldims:]] = g["n"]
            g["n"] += n
        g["blk"].append((b, g["rows"][c[:ldims]], g["cols"][c[ldims:]], m, n))
    return list(out.values())      # in order of first appearance


def _decaying_state(meta, seed):
    """A two-site state whose singular values fall off exponentially in every block-matrix (no two
    alike), between random orthonormal vectors."""
    rng = np.random.default_rng(seed)
    data = np.zeros(meta.size)
    for i, x in enumerate(_groups(meta, 2)):
        k = min(x["m"], x["n"])
        at = np.arange(k) + (0.618034 * i) % 1.0
        left = np.linalg.qr(rng.standard_normal((x["m"], k)))[0]
        right = np.linalg.qr(rng.standard_normal((x["n"], k)))[0]
        dense = (left * np.exp(at * (-7.0 / k))) @ right.T
        for b, r, c, m, n in x["blk"]:
            o = int(meta.offsets[b])
            data[o:o + m * n] = dense[r:r + m, c:c + n].reshape(-1)
    return DTensor.from_host(BSTensor(meta.legs, meta.coords, meta.dtype, data))


ENV_AXES = [[[0], [0]], [[0, 2], [0, 1]], [[0, 3, 1], [0, 1, 2]]]
MATVEC_AXES = [[[0], [0]], [[0, 2], [0, 1]], [[4, 1], [0, 1]], [[4, 1], [1, 0]]]


# ------------------------------------------------------------------ prepare and run
def _inputs(case, seed):
    """The tensors a program holds before the call, on the GPU, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "contract":
        m = _site(case["D"])
        return [_normal(m, g), _normal(m, g)]
    if kind in ("env", "accumulate"):
        lenv, psi, mpo, _, _ = _chain(case["D"], int(seed) % 1000003)
        if kind == "accumulate":
            lead = _normal(psi, g)
            return [DTensor.from_host(lenv), lead, _normal(_left_times_psi(case["D"]), g)]
        two = DTensor.from_host(psi)
        return [DTensor.from_host(lenv), two, DTensor.from_host(mpo), DTensor(_dagger(two.meta), two.buf)]
    if kind == "transpose":
        m = _left_times_psi(case["D"]) if case["family"] == "u1" else _hubbard_layout(case["D"])[1]
        return [_normal(m, g)]
    if kind == "matvec" and case["family"] == "hubbard":
        return [_normal(m, g, 1.0 if i != 1 else max(m.size, 1) ** -0.5) for i, m in
                enumerate(_hubbard_layout(case["D"]))]
    if kind in ("matvec", "lanczos"):
        return [DTensor.from_host(t) for t in _chain(case["D"], int(seed) % 1000003)]
    if kind == "svd":
        return [_decaying_state(_chain_psi(case["D"]), int(seed))]
    if kind == "qr":
        return [_normal(_qr_layout(case["blocks"], case["lo"], case["hi"]), g)]
    m = _chain_psi(case["D"])
    return [_normal(m, g, m.size ** -0.5) for _ in range(case["n"])]


@lru_cache(maxsize=8)
def _chain_psi(D):
    return _meta(_chain(D, 1)[1])


@lru_cache(maxsize=8)
def _left_times_psi(D):
    """Layout of lenv . psi over lenv's first leg: (M in, V in, P in, P in, V out)."""
    lenv, psi, _, _, _ = _chain(D, 1)
    return _tensor([lenv.legs[1], lenv.legs[2], psi.legs[1], psi.legs[2], psi.legs[3]])


def _qr_layout(nb, lo, hi):
    """Tall block-matrices (a site tensor with two physical states): `nb` sectors, sizes lo .. hi."""
    hi = max(hi, lo)
    dims = [lo + (hi - lo) * i // max(1, nb - 1) for i in range(nb)]
    v = Leg(IN, np.arange(nb).reshape(-1, 1), np.asarray(dims))
    p = Leg(IN, np.asarray([[0]]), np.asarray([2]))
    return _tensor([v, p, v.inverse()])


def _coefs(case):
    return [(-1.0) ** i / (1.0 + i) for i in range(case["n"])]


def prepare(case, seed):
    kind = case["kind"]
    t = _inputs(case, seed)
    st = {"kind": kind, "case": case, "t": t}
    if kind == "env":
        metas, plans = t[0].meta, []
        for other, ax in zip(t[1:], ENV_AXES):
            plans.append(ContractionPlan(metas, other.meta, ax))
            metas = plans[-1].result
        st["plans"] = plans
    elif kind == "transpose":
        st["plan"] = TransposePlan(t[0].meta, [int(c) for c in case["perm"]])
        st["out"] = DTensor.empty(st["plan"].result)
    elif kind == "matvec":
        st["mv"] = Matvec(t[0], t[1].meta, t[2], t[3], t[4], case["mode"])
        st["out"] = DTensor.empty(st["mv"].result)
    elif kind == "lanczos":
        st["mv"] = Matvec(t[0], t[1].meta, t[2], t[3], t[4], "split")
        st["lanczos"] = Lanczos(st["mv"], case["steps"])
    elif kind == "accumulate":
        # lenv's first leg against psi's first: the result joins an existing tensor
        st["plan"] = AccumulatePlan(t[0].meta, t[1].meta, 0, 0, 1, t[2].meta)
        st["out"] = DTensor.empty(st["plan"].result)
    return st


def _lowest(alpha, beta):
    """Lowest eigenvector of the Krylov tridiagonal matrix, its first entry positive."""
    off = beta[1:len(alpha)]
    _, y = np.linalg.eigh(np.diag(alpha) + np.diag(off, 1) + np.diag(off, -1))
    return y[:, 0] * (1.0 if y[0, 0] >= 0 else -1.0)


def run(st):
    kind, case, t = st["kind"], st["case"], st["t"]
    if kind == "contract":
        return Contract(t[0], t[1], [[2], [0]]).buf
    if kind == "env":
        cur = t[0]
        for plan, other in zip(st["plans"], t[1:]):
            cur = plan.execute(cur, other, mode=case["mode"])
        return cur.buf
    if kind == "transpose":
        return st["plan"].execute(t[0], st["out"]).buf
    if kind == "matvec":
        return st["mv"].apply(t[1], st["out"]).buf
    if kind == "lanczos":
        lz = st["lanczos"]
        lz.start(t[1])
        lz.step(case["steps"])
        alpha, beta = lz.coeffs()
        y = _lowest(alpha, beta)
        krylov = [DTensor(st["mv"].result, lz.vector(i)) for i in range(len(y))]
        return {"alpha": alpha, "beta": beta, "state": LinearCombine(list(y), krylov).buf}
    if kind == "svd":
        # singular vectors are unique up to a sign each: the kept state is what goes on
        u, s, vt, err, kept = SVD(t[0], 2, [0], 0.0, 1, case["D"])
        state = Contract(u, Contract(s, vt, [[1], [0]]), [[2], [0]])
        return {"state": state.buf, "s": s.buf, "err": err, "kept": kept}
    if kind == "qr":
        q, r = QR(t[0], 2, [0])
        return {"q": q.buf, "r": r.buf}
    if kind == "accumulate":
        return st["plan"].execute(t[0], t[1], t[2], 0.5, -1.0, out=st["out"], mode=case["mode"]).buf
    return LinearCombine(_coefs(case), t).buf


# ------------------------------------------------------------------ plain 64-bit values
class _Dense:
    """A block-sparse tensor as plain blocks: {sector coordinates: ndarray}."""

    def __init__(self, legs, blocks):
        self.legs, self.blocks = legs, blocks


def _plain(t):
    m = t.meta
    n = m.size * (2 if m.is_complex else 1)
    raw = t.buf[:n].cpu().numpy()
    raw = raw.view(np.complex128) if m.is_complex else raw
    shp = m.block_shapes()
    return _Dense(m.legs, {tuple(int(x) for x in m.coords[b]): raw[int(m.offsets[b]):int(m.offsets[b]) +
                                                                   int(np.prod(shp[b]))].reshape(shp[b])
                           for b in range(m.nblk)})


def _raw(d):
    flat = [d.blocks[c].reshape(-1) for c in sorted(d.blocks)]
    x = np.concatenate(flat) if flat else np.zeros(1)
    return torch.from_numpy(np.ascontiguousarray(x).view(np.float64).copy())


def _parity(legs, coords):
    return tuple(bool(g.parity_comp >= 0 and g.qns[c, g.parity_comp] % 2) for g, c in zip(legs, coords))


def _exchange(pa, pb, axa, axb, a_in, memo):
    """Sign of moving every contracted leg of B next to its partner in A (fermionic legs)."""
    key = (pa, pb)
    if key not in memo:
        order = [("a", i) for i in range(len(pa))] + [("b", i) for i in range(len(pb))]
        odd = {("a", i): p for i, p in enumerate(pa)}
        odd.update({("b", i): p for i, p in enumerate(pb)})
        n = 0
        for x, y, inward in zip(axa, axb, a_in):
            i, j = order.index(("a", x)), order.index(("b", y))
            if odd["b", y]:
                n += sum(odd[e] for e in order[i + 1:j]) + (1 if inward else 0)
            order.insert(i + 1, order.pop(j))
        memo[key] = -1 if n & 1 else 1
    return memo[key]


def _contract64(a, b, axes):
    axa, axb = axes
    sa = [i for i in range(len(a.legs)) if i not in axa]
    sb = [i for i in range(len(b.legs)) if i not in axb]
    fermionic = a.legs[0].parity_comp >= 0
    a_in = [a.legs[i].dir == IN for i in axa]
    by_key = {}
    for c, x in b.blocks.items():
        k = int(np.prod([x.shape[i] for i in axb]))
        mat = np.ascontiguousarray(x.transpose(list(axb) + sb)).reshape(k, -1)
        by_key.setdefault(tuple(c[i] for i in axb), []).append(
            (tuple(c[i] for i in sb), mat, tuple(x.shape[i] for i in sb), _parity(b.legs, c)))
    out, shapes, memo = {}, {}, {}
    for c, x in a.blocks.items():
        match = by_key.get(tuple(c[i] for i in axa))
        if not match:
            continue
        k = int(np.prod([x.shape[i] for i in axa]))
        mat = np.ascontiguousarray(x.transpose(sa + list(axa))).reshape(-1, k)
        ca, sha, pa = tuple(c[i] for i in sa), tuple(x.shape[i] for i in sa), _parity(a.legs, c)
        for cb, mb, shb, pb in match:
            r = mat @ mb
            if fermionic and _exchange(pa, pb, axa, axb, a_in, memo) < 0:
                r = -r
            if ca + cb in out:
                out[ca + cb] += r
            else:
                out[ca + cb] = r
                shapes[ca + cb] = sha + shb
    return _Dense([a.legs[i] for i in sa] + [b.legs[i] for i in sb],
                  {c: x.reshape(shapes[c]) for c, x in out.items()})


def _apply64(ops, psi):
    lenv, mpo1, mpo2, renv = ops
    cur = lenv
    for other, ax in zip((psi, mpo1, mpo2, renv), MATVEC_AXES):
        cur = _contract64(cur, other, ax)
    return cur


def _lanczos64(t, steps):
    ops = [_plain(t[i]) for i in (0, 2, 3, 4)]
    psi = _plain(t[1])
    keys = sorted(psi.blocks)
    shapes = [psi.blocks[k].shape for k in keys]
    cuts = np.cumsum([int(np.prod(s)) for s in shapes])[:-1]

    def apply(v):
        d = _Dense(psi.legs, {k: x.reshape(s) for k, x, s in zip(keys, np.split(v, cuts), shapes)})
        return _raw(_apply64(ops, d)).numpy()

    v = np.concatenate([psi.blocks[k].reshape(-1) for k in keys])
    beta = [np.linalg.norm(v)]
    vs, alpha = [v / beta[0]], []
    for j in range(steps):
        w = apply(vs[j])
        a = 0.0
        for _ in range(2):
            m = np.asarray(vs)
            c = m @ w
            w = w - c @ m
            a += c[j]
        alpha.append(a)
        beta.append(np.linalg.norm(w))
        vs.append(w / beta[-1])
    alpha, beta = np.asarray(alpha), np.asarray(beta)
    return {"alpha": alpha, "beta": beta, "state": torch.from_numpy(_lowest(alpha, beta) @ np.asarray(vs[:steps]))}


def _matrix64(d, g, meta):
    m = np.zeros((g["m"], g["n"]))
    for b, r, c, rows, cols in g["blk"]:
        m[r:r + rows, c:c + cols] = d.blocks[tuple(int(x) for x in meta.coords[b])].reshape(rows, cols)
    return m


def _svd64(t, kept):
    """The state kept by the `kept` largest singular values, those values, the lost weight."""
    meta, d = t.meta, _plain(t)
    gs = _groups(meta, 2)
    parts = [np.linalg.svd(_matrix64(d, g, meta), full_matrices=False) for g in gs]
    every = np.sort(np.concatenate([p[1] for p in parts]))[::-1]
    cut = every[min(kept, len(every)) - 1]
    state, diag = {}, {}
    for g, (u, s, vt) in zip(gs, parts):
        k = int(np.count_nonzero(s >= cut))
        if not k:
            continue
        x = (u[:, :k] * s[:k]) @ vt[:k]
        diag[(len(diag), len(diag))] = np.diag(s[:k])
        for b, r, c, rows, cols in g["blk"]:
            key = tuple(int(v) for v in meta.coords[b])
            state[key] = x[r:r + rows, c:c + cols].reshape(d.blocks[key].shape)
    w = np.square(every)
    return {"state": _raw(_Dense(meta.legs, state)), "s": _raw(_Dense(None, diag)),
            "err": float(w[kept:].sum() / w.sum()), "kept": min(kept, len(every))}


def _qr64(t):
    """Householder QR of every block-matrix (R's diagonal signed as LAPACK leaves it)."""
    meta, d = t.meta, _plain(t)
    q, r = {}, {}
    for x in _groups(meta, 2):
        (b, _, _, rows, cols), = x["blk"]
        c = tuple(int(v) for v in meta.coords[b])
        mq, mr = np.linalg.qr(d.blocks[c].reshape(rows, cols))
        q[(c[0], c[1], c[0])] = mq
        r[(c[0], c[0])] = mr
    return {"q": _raw(_Dense(None, q)), "r": _raw(_Dense(None, r))}


def exact(case, seed):
    kind = case["kind"]
    t = _inputs(case, seed)
    if kind == "contract":
        return _raw(_contract64(_plain(t[0]), _plain(t[1]), [[2], [0]]))
    if kind == "env":
        cur = _plain(t[0])
        for other, ax in zip(t[1:], ENV_AXES):
            cur = _contract64(cur, _plain(other), ax)
        return _raw(cur)
    if kind == "transpose":
        perm = [int(c) for c in case["perm"]]
        a = _plain(t[0])
        out = {}
        for c, x in a.blocks.items():
            p = _parity(a.legs, c)
            n = sum(p[i] and p[j] for k, i in enumerate(perm) for j in perm[k + 1:] if i > j)
            x = np.ascontiguousarray(x.transpose(perm))
            out[tuple(c[i] for i in perm)] = -x if n & 1 else x
        return _raw(_Dense([a.legs[i] for i in perm], out))
    if kind == "matvec":
        return _raw(_apply64([_plain(t[i]) for i in (0, 2, 3, 4)], _plain(t[1])))
    if kind == "lanczos":
        return _lanczos64(t, case["steps"])
    if kind == "svd":
        return _svd64(t[0], case["D"])
    if kind == "qr":
        return _qr64(t[0])
    if kind == "accumulate":
        prod, c = _contract64(_plain(t[0]), _plain(t[1]), [[0], [0]]), _plain(t[2])
        out = {k: -x for k, x in c.blocks.items()}
        for k, x in prod.blocks.items():
            out[k] = out[k] + 0.5 * x
        return _raw(_Dense(c.legs, out))
    acc = np.zeros(t[0].meta.size)
    for c, x in zip(_coefs(case), t):
        acc += c * x.buf[:acc.size].cpu().numpy()
    return torch.from_numpy(acc)


# ------------------------------------------------------------------ least bytes and operations
def _contraction_flops(a, b, axes, cplx):
    """Sum of 2 m k n (8 m k n complex) over the block pairs of a contraction, and its result's layout."""
    axa, axb = axes
    sa = [i for i in range(len(a.legs)) if i not in axa]
    sb = [i for i in range(len(b.legs)) if i not in axb]
    sha, shb = a.block_shapes(), b.block_shapes()
    n_of, saved = {}, {}
    for j in range(b.nblk):
        key = tuple(int(b.coords[j, i]) for i in axb)
        n_of[key] = n_of.get(key, 0) + int(np.prod(shb[j, sb]))
        saved.setdefault(key, []).append(tuple(int(b.coords[j, i]) for i in sb))
    total, coords = 0, set()
    for i in range(a.nblk):
        key = tuple(int(a.coords[i, x]) for x in axa)
        if key in n_of:
            total += int(np.prod(sha[i])) * n_of[key]
            c = tuple(int(a.coords[i, x]) for x in sa)
            coords.update(c + s for s in saved[key])
    legs = [a.legs[i] for i in sa] + [b.legs[i] for i in sb]
    return total * (8 if cplx else 2), BSTensor(legs, np.asarray(sorted(coords)), a.dtype, None)


@lru_cache(maxsize=64)
def _work(items):
    case = dict(items)
    kind = case["kind"]
    if kind == "contract":
        m = _site(case["D"])
        f, c = _contraction_flops(m, m, [[2], [0]], False)
        return 8 * (2 * m.size + c.size), f
    if kind in ("env", "accumulate"):
        lenv, psi, mpo, _, _ = _chain(case["D"], 1)
        if kind == "accumulate":
            f, c = _contraction_flops(lenv, psi, [[0], [0]], False)
            return 8 * (lenv.size + psi.size + 2 * c.size), f + 3 * c.size
        total, cur = 0, lenv
        for other, ax in zip((psi, mpo, _dagger(psi)), ENV_AXES):
            f, cur = _contraction_flops(cur, other, ax, False)
            total += f
        return 8 * (lenv.size + psi.size + mpo.size + cur.size), total
    if kind == "transpose":
        u1 = case["family"] == "u1"
        m = _left_times_psi(case["D"]) if u1 else _hubbard_layout(case["D"])[1]
        return 2 * m.size * (8 if u1 else 16), 0
    if kind in ("matvec", "lanczos"):
        cplx = case.get("family") == "hubbard"
        lenv, psi, mpo1, mpo2, renv = _hubbard_layout(case["D"]) if cplx else _chain(case["D"], 1)
        total, cur = 0, lenv
        for other, ax in zip((psi, mpo1, mpo2, renv), MATVEC_AXES):
            f, cur = _contraction_flops(cur, other, ax, cplx)
            total += f
        nbytes = (lenv.size + 2 * psi.size + mpo1.size + mpo2.size + renv.size) * (16 if cplx else 8)
        if kind == "matvec":
            return nbytes, total
        k = case["steps"]
        return nbytes + 8 * psi.size * k, k * total + sum(8 * (j + 1) for j in range(k)) * psi.size
    if kind == "svd":
        m = _chain_psi(case["D"])
        f = 0
        for g in _groups(m, 2):
            p, q = max(g["m"], g["n"]), min(g["m"], g["n"])
            f += 14 * p * q * q + 8 * q ** 3          # a thin SVD with both factors
        return 8 * 3 * m.size, f
    if kind == "qr":
        m = _qr_layout(case["blocks"], case["lo"], case["hi"])
        f = sum(4 * g["m"] * g["n"] ** 2 - 4 * g["n"] ** 3 / 3 for g in _groups(m, 2))
        return 8 * (2 * m.size + sum(g["n"] ** 2 for g in _groups(m, 2))), f
    m = _chain_psi(case["D"])
    return 8 * m.size * (case["n"] + 1), 2 * case["n"] * m.size


def work(case):
    nbytes, flops = _work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    return {"bytes": nbytes, "flops": flops}
