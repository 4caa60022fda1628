"""The framework's timed work: what a user of the Holstein TDVP library has it do, case by case.

Every case is one call (or one time step) through the public Python surface of
``libkvgpu`` on inputs of the shapes this repository names: the chains of
``holstein.config_chain`` (L8 one mode D = 32; L24 one mode D = 96; L32 two
modes D = 128; L64 four modes D = 512) and the disordered ensemble.  A local
problem (an H_eff apply, a Lanczos exponential, a split, an environment
update, an adjoint) is taken from the middle of a shorter chain of the same
model, whose bonds there have the long chain's sectors; its environments are
built on the device from the seeded state, as a sweep builds them.

Results stay on the device until they are looked up (:class:`Held`), as in a
program that passes them on to the next call.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "kylin_v_gb300" not in sys.modules:
        d = os.path.join(ROOT, "kylin-v_gb300")
        spec = importlib.util.spec_from_file_location("kylin_v_gb300", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        m = importlib.util.module_from_spec(spec)
        sys.modules["kylin_v_gb300"] = m
        spec.loader.exec_module(m)


_package()
from kylin_v_gb300 import holstein as H  # noqa: E402
from kylin_v_gb300 import kvgpu as G  # noqa: E402
from kylin_v_gb300.kvio import BlockTensor  # noqa: E402

PRECISION = {"fp64": G.KV_FP64, "mixed": G.KV_MIXED_3M_DIGITS}
DT, MAX_ITER, TOL_EXP, TOL_SVD = 0.05, 11, 1e-8, 1e-8  # the configurations' own settings
# mode frequencies and couplings by the number of modes: the L8 / L24, L32 and L64 chains
# (three modes: the L64 chain's first three)
MODES = {1: ([1.0], [1.0]), 2: ([0.2, 1.2], [0.5, 1.0]), 3: ([0.1, 0.4, 0.9], [0.3, 0.6, 0.8]),
         4: ([0.1, 0.4, 0.9, 1.5], [0.3, 0.6, 0.8, 1.0])}


def listed():
    return [
        # an environment update of the L8 chain: the smallest call a one-site sweep makes
        dict(name="env-fp64-D32", op="env", mol=6, modes=1, cutoff=8, D=32, site=9, l2r=True, precision="fp64"),
        # a forward one-site evolution of the L8 chain: a loop of small launches
        dict(name="krylov1-mixed-D32", op="krylov", nsite=1, mol=6, modes=1, cutoff=8, D=32, site=10, reverse=False,
             precision="mixed"),
        # one two-site H_eff apply of the L32 chain at an (auxiliary, phonon) pair: thousands of small blocks
        dict(name="apply2-mixed-D128", op="apply", nsite=2, mol=3, modes=2, cutoff=16, D=128, site=7,
             precision="mixed"),
        # the two-site evolution of the L32 chain at a (phonon, auxiliary) pair: its largest blocks
        dict(name="krylov2-mixed-D128", op="krylov", nsite=2, mol=3, modes=2, cutoff=16, D=128, site=8,
             reverse=False, precision="mixed"),
        # the backward one-site evolution of the FP64 differentiation chain (L24)
        dict(name="krylov1-fp64-D96", op="krylov", nsite=1, mol=6, modes=1, cutoff=12, D=96, site=10, reverse=True,
             precision="fp64"),
        # the two-site evolution of the L64 chain, the largest one here
        dict(name="krylov2-mixed-D512", op="krylov", nsite=2, mol=2, modes=4, cutoff=8, D=512, site=7,
             reverse=False, precision="mixed"),
        # the two-site split of the L32 chain, left to right
        dict(name="svd2-mixed-D128", op="svd", nsite=2, mol=3, modes=2, cutoff=16, D=128, site=8, l2r=True,
             precision="mixed"),
        # a two-site split in FP64 (the library's default precision) at an odd bond dimension, right to left
        dict(name="svd2-fp64-D101", op="svd", nsite=2, mol=3, modes=2, cutoff=16, D=101, site=8, l2r=False,
             precision="fp64"),
        # the energy of a 12-molecule piece of the L24 chain (36 sites): what is read after every step
        dict(name="energy-fp64-D96", op="energy", mol=12, modes=1, cutoff=12, D=96, precision="fp64"),
        # the reverse-mode derivative of a one-site H_eff apply, all cotangents
        dict(name="adjoint1-fp64-D96", op="adjoint", nsite=1, mol=6, modes=1, cutoff=12, D=96, site=9,
             precision="fp64"),
        # a whole two-site time step of the L32 model on 3 molecules, with its populations
        dict(name="step2-mixed-D128", op="step", mode=2, chains=1, mol=3, modes=2, cutoff=16, D=128,
             precision="mixed"),
        # a whole one-site step of a small disordered ensemble on concurrent streams, with its populations
        dict(name="ensemble1-mixed-D64", op="step", mode=1, chains=6, mol=8, modes=1, cutoff=8, D=64,
             precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the same calls at other bond dimensions, cutoffs, mode numbers, sites and options."""
    op = rng.choice(["env", "apply", "krylov", "krylov", "svd", "svd", "energy", "adjoint", "step", "step"])
    precision = rng.choice(["fp64", "mixed"])
    modes = rng.choice([1, 1, 2, 2, 4])
    cutoff = rng.randint(4, 12 if modes < 4 else 8)
    top = {"env": 256, "apply": 256, "krylov": 320, "svd": 144, "energy": 128, "adjoint": 160, "step": 96}[op]
    if precision == "fp64" and op in ("svd", "krylov", "step"):
        top //= 2
    D = _log(rng, 8, top)
    c = dict(op=op, modes=modes, cutoff=cutoff, D=D, precision="fp64" if op == "energy" else precision)
    if op == "energy":
        return dict(c, mol=rng.randint(2, 12 // modes + 2))
    if op == "step":
        mode = rng.choice([1, 2])
        return dict(c, mode=mode, chains=1 if mode == 2 else rng.choice([1, 1, 2, 4]),
                    mol=rng.randint(2, 3 if modes > 1 else 5))
    # enough molecules on both sides of the chosen one for its bonds to reach D
    side = min(4, max(1, math.ceil(math.log(D) / (modes * math.log(cutoff)))))
    unit = 1 + 2 * modes
    c.update(mol=2 * side + 1, site=side * unit + rng.randrange(unit))
    if op == "env":
        return dict(c, l2r=rng.choice([True, False]))
    if op in ("apply", "krylov"):
        c["nsite"] = rng.choice([0, 1, 2, 2])
    if op == "svd":
        return dict(c, nsite=rng.choice([1, 2]), l2r=rng.choice([True, False]))
    if op == "adjoint":
        c["nsite"] = rng.choice([1, 2])
    if op == "krylov":
        c["reverse"] = c["nsite"] < 2
    return c


# ------------------------------------------------------------------ inputs
def _chain(case, index=0, seed=0):
    omega, g = MODES[case["modes"]]
    if case.get("chains", 1) == 1:
        return H.HolsteinChain(case["mol"], list(omega), [list(g)] * case["mol"], cutoff=case["cutoff"])
    # a member of the disordered ensemble: eps ~ N(0, 0.5^2), g uniform in [0.5, 1.5], lengths spread about `mol`
    rng = np.random.default_rng([seed, index])
    L = max(2, case["mol"] + index % 3 - 1)
    return H.HolsteinChain(L, list(omega), [[float(x) for x in rng.uniform(0.5, 1.5, case["modes"])]
                                            for _ in range(L)], cutoff=case["cutoff"],
                           eps=[float(x) for x in rng.normal(0.0, 0.5, L)])


def _left_factor(t, carry):
    """Q and the triangular factors of one site with `carry` folded in from the left: Q is left-canonical."""
    blocks = [(q, np.einsum("ab,bsc->asc", carry[q[0]], a)) if carry else (q, a) for q, a in t.blocks]
    by_right = {}
    for i, (q, a) in enumerate(blocks):
        by_right.setdefault(q[2], []).append(i)
    out, r = [None] * len(blocks), {}
    for qr, idx in by_right.items():
        M = np.concatenate([blocks[i][1][:, 0, :] for i in idx], axis=0)
        Q, R = np.linalg.qr(M)
        row = 0
        for i in idx:
            n = blocks[i][1].shape[0]
            out[i] = (blocks[i][0], Q[row:row + n].reshape(n, 1, -1).copy())
            row += n
        r[qr] = R
    return BlockTensor(t.dirs, out), r


def _state(case, seed):
    """Host inputs of a local problem: the chain's MPS with its centre on site s (left-canonical before it,
    right-canonical after it, norm 1) and its MPO; for nsite = 0 the centre is the matrix on the bond after s."""
    ch = _chain(case)
    mps, mpo, s = H.random_mps(ch, case["D"], seed=seed), H.hamiltonian_mpo(ch), case["site"]
    carry = None
    for i in range(s):
        mps[i], carry = _left_factor(mps[i], carry)
    if carry:
        mps[s].blocks = [(q, np.einsum("ab,bsc->asc", carry[q[0]], a)) for q, a in mps[s].blocks]
    centre = None
    if case.get("nsite") == 0:
        mps[s], r = _left_factor(mps[s], None)
        centre = BlockTensor((1, -1), [((q, q), a) for q, a in sorted(r.items())])
    return mps, mpo, centre


def _cotangent(case, seed, like):
    rng = np.random.default_rng([seed, 7])
    return BlockTensor(like.dirs, [(q, rng.standard_normal(a.shape) + 1j * rng.standard_normal(a.shape))
                                   for q, a in like.blocks])


def _pair_layout(a, b):
    """The two-site tensor's blocks (zeros), from the bond structures of its two sites."""
    shapes = {}
    for qa, x in a.blocks:
        for qb, y in b.blocks:
            if qa[2] == qb[0]:
                shapes[(qa[0], qa[1], qb[1], qb[2])] = (x.shape[0], 1, 1, y.shape[2])
    return BlockTensor((1, 1, 1, -1), [(q, np.zeros(s)) for q, s in sorted(shapes.items())])


def _boundary(direction, q):
    return BlockTensor((direction, -direction, -direction), [((q, 0, q), np.ones((1, 1, 1), np.complex128))])


class Held(dict):
    """Named results; a device tensor is downloaded when it is looked up (its blocks in charge order)."""

    def __getitem__(self, k):
        v = dict.__getitem__(self, k)
        return _flat(v.to_host().as_dict()) if isinstance(v, G.Tensor) else v


def _flat(blocks):
    """Blocks keyed by (charges, shape), or by charges, as one array in key order."""
    return np.concatenate([np.asarray(blocks[k], np.complex128).ravel() for k in sorted(blocks)])


def prepare(case, seed):
    G.init(0)
    st = dict(case=case, precision=PRECISION[case["precision"]])
    if case["op"] == "energy":
        ch = _chain(case)
        st["mps"] = [G.Tensor.from_host(t) for t in H.random_mps(ch, case["D"], seed=seed)]
        st["mpo"] = [G.Tensor.from_host(t) for t in H.hamiltonian_mpo(ch)]
        return st
    if case["op"] == "step":
        st["chains"], st["density"], st["identity"] = [], [], []
        for i in range(case["chains"]):
            ch = _chain(case, i, seed)
            st["chains"].append(G.TDVP(H.random_mps(ch, case["D"], seed=seed * 64 + i), H.hamiltonian_mpo(ch), TOL_SVD,
                                       TOL_EXP, case["D"], MAX_ITER, DT, st["precision"]))
            st["identity"].append([G.Tensor.from_host(t) for t in H.identity_mpo(ch)])
            st["density"].append([(j, G.Tensor.from_host(H.density_mpo(ch, j)[j])) for j in ch.exciton_sites()])
        return st
    mps, mpo, centre = _state(case, seed)
    s, nsite = case["site"], case.get("nsite", 1)
    last = s if nsite == 0 else s + nsite - 1  # last site inside the local problem
    A = [G.Tensor.from_host(t) for t in mps]
    W = [G.Tensor.from_host(t) for t in mpo]
    L, R = G.Tensor.from_host(_boundary(1, 0)), G.Tensor.from_host(_boundary(-1, mps[-1].blocks[0][0][2]))
    for i in range(s + 1 if nsite == 0 else s):
        L = G.env_sweep(L, A[i], W[i], True)
    for i in range(len(mps) - 1, last, -1):
        R = G.env_sweep(R, A[i], W[i], False)
    psi = G.Tensor.from_host(centre) if nsite == 0 else A[s] if nsite == 1 else G.product(A[s], A[s + 1], 1)
    st.update(L=L, R=R, A=A[s], psi=psi, W1=W[s] if nsite >= 1 else None, W2=W[s + 1] if nsite == 2 else None)
    if case["op"] == "svd":  # what a sweep splits: the evolved tensor
        st["psi"] = G.local_krylov(nsite, L, psi, st["W1"], st["W2"], R, DT, MAX_ITER, TOL_EXP)[0]
    if case["op"] == "adjoint":
        like = mps[s] if nsite == 1 else _pair_layout(mps[s], mps[s + 1])
        st["ybar"] = G.Tensor.from_host(_cotangent(case, seed, like))
    return st


def run(st):
    case, prec = st["case"], st["precision"]
    op, nsite = case["op"], case.get("nsite", 1)
    if op == "env":
        env = st["L"] if case["l2r"] else st["R"]
        return Held(env=G.env_sweep(env, st["A"], st["W1"], case["l2r"], prec))
    if op == "apply":
        return Held(psi=G.heff_apply(nsite, st["L"], st["psi"], st["W1"], st["W2"], st["R"], 0.5 * DT, prec))
    if op == "krylov":
        t, dim = G.local_krylov(nsite, st["L"], st["psi"], st["W1"], st["W2"], st["R"], DT, MAX_ITER, TOL_EXP,
                                case["reverse"], prec)
        return Held(psi=t, dimension=dim)
    if op == "svd":
        # the factors are fixed up to a phase per state: their product is the truncated tensor
        U, V, kept, total = G.svd_impl(st["psi"], _split(case), case["l2r"], TOL_SVD, case["D"], prec)
        return Held(psi=G.product(U, V, 1), kept=kept, total=total)
    if op == "energy":
        return G.expectation(st["mps"], st["mpo"], st["mps"]).real
    if op == "adjoint":
        return Held(G.adjoint_heff(nsite, st["L"], st["psi"], st["W1"], st["W2"], st["R"], st["ybar"],
                                   precision=prec))
    if len(st["chains"]) == 1:
        st["chains"][0].sweep(case["mode"])
    else:
        G.sweep_batched(st["chains"], case["mode"], 1)
    out = {}
    for i, t in enumerate(st["chains"]):
        sites = t.sites()
        out["populations%d" % i] = np.array(
            [x.real for x in G.local_expectations(sites, st["identity"][i], st["density"][i])])
        out["energy%d" % i] = G.expectation(sites, t.mpo, sites).real
    return out


def _split(case):
    """Legs on the left of the split: after the first site of a pair; a one-site tensor towards the sweep."""
    return 2 if case["nsite"] == 2 or case["l2r"] else 1


# --------------------------------------------------- the same in 64-bit numpy
# A tensor here is a dict from leg charges to arrays; `contract` multiplies all blocks whose contracted legs carry
# equal charges and sums those with equal free charges.
def _blocks(t):
    return dict(t.blocks)


def _contract(x, lx, y, ly, out):
    """x with legs named lx times y with legs named ly, the shared names summed, legs ordered as in out."""
    shared = [c for c in lx if c in ly]
    fx, fy = [c for c in lx if c not in shared], [c for c in ly if c not in shared]
    ax = [lx.index(c) for c in fx] + [lx.index(c) for c in shared]
    ay = [ly.index(c) for c in shared] + [ly.index(c) for c in fy]
    perm = [(fx + fy).index(c) for c in out]
    index = {}
    for q, b in y.items():
        bt = b.transpose(ay)
        k = math.prod(bt.shape[:len(shared)])
        index.setdefault(tuple(q[ly.index(c)] for c in shared), []).append(
            (tuple(q[ly.index(c)] for c in fy), bt.shape[len(shared):], np.ascontiguousarray(bt).reshape(k, -1)))
    res = {}
    for q, a in x.items():
        todo = index.get(tuple(q[lx.index(c)] for c in shared))
        if not todo:
            continue
        at = a.transpose(ax)
        sa = at.shape[:len(fx)]
        m = np.ascontiguousarray(at).reshape(math.prod(sa), -1)
        qa = tuple(q[lx.index(c)] for c in fx)
        for qb, sb, n in todo:
            key = qa + qb
            v = m @ n
            if key in res:
                res[key][0] += v
            else:
                res[key] = [v, sa + sb]
    return {tuple(k[p] for p in perm): v.reshape(s).transpose(perm) for k, (v, s) in res.items()}


def _conj(x):
    return {k: v.conj() for k, v in x.items()}


def _env_l2r(L, A, W, bra=None):
    t = _contract(_contract(L, "pwx", A, "xsb", "pwsb"), "pwsb", W, "uwsv", "puvb")
    return _contract(_conj(A if bra is None else bra), "puq", t, "puvb", "qvb")


def _env_r2l(R, A, W):
    t = _contract(_contract(R, "qvy", A, "xsy", "qvsx"), "qvsx", W, "uwsv", "quwx")
    return _contract(_conj(A), "puq", t, "quwx", "pwx")


def _apply(nsite, L, psi, W1, W2, R):
    if nsite == 0:
        return _contract(_contract(L, "pwx", psi, "xb", "pwb"), "pwb", R, "qwb", "pq")
    if nsite == 1:
        t = _contract(_contract(L, "pwx", psi, "xsb", "pwsb"), "pwsb", W1, "uwsv", "puvb")
        return _contract(t, "puvb", R, "qvb", "puq")
    t = _contract(_contract(L, "pwx", psi, "xstb", "pwstb"), "pwstb", W1, "uwsv", "puvtb")
    t = _contract(t, "puvtb", W2, "zvty", "puzyb")
    return _contract(t, "puzyb", R, "qyb", "puzq")


def _axpy(x, c, y):
    """x + c y over the union of the blocks."""
    out = dict(x)
    for k, v in y.items():
        out[k] = out[k] + c * v if k in out else c * v
    return out


def _dot(x, y):
    return sum((np.vdot(x[k], v) for k, v in y.items() if k in x), 0.0 + 0.0j)


def _norm(x):
    return math.sqrt(sum(np.vdot(v, v).real for v in x.values()))


def _krylov(nsite, L, psi, W1, W2, R, reverse):
    """exp(-+i H dt/2) psi / |psi| as the Lanczos recurrence of local_krylov forms it."""
    n = _norm(psi)
    V, alpha, beta, err = [{k: v / n for k, v in psi.items()}], [], [], 1.0
    while True:
        hv = {k: 0.5 * DT * v for k, v in _apply(nsite, L, V[-1], W1, W2, R).items()}
        if len(V) > 1:
            beta.append(_dot(hv, V[-2]))
            hv = _axpy(hv, -beta[-1], V[-2])
        alpha.append(_dot(hv, V[-1]))
        hv = _axpy(hv, -alpha[-1], V[-1])
        n = _norm(hv)
        err *= n
        if err <= TOL_EXP or len(alpha) >= MAX_ITER - 1:
            break
        V.append({k: v / n for k, v in hv.items()})
    m = len(alpha)
    T = np.zeros((m, m), complex)
    for i in range(m):
        T[i, i] = alpha[i].real
        if i + 1 < m:
            T[i, i + 1], T[i + 1, i] = beta[i], np.conj(beta[i])
    lam, Z = np.linalg.eigh(T)
    c = Z @ (np.exp((1j if reverse else -1j) * lam) * Z[0].conj())
    out = {}
    for i in range(m):
        out = _axpy(out, c[i], V[i])
    return out, m


def _truncated(psi, split, D):
    """The block tensor with all but the D largest singular values (and those below the threshold) dropped."""
    sec = {}
    for q in psi:  # MPS legs run in, in, .., out: the bond's charge is the sum of the left ones
        sec.setdefault(sum(q[:split]), []).append(q)
    parts, vals, total = [], [], 0
    for qs in sec.values():
        rows, cols = {}, {}
        for q in sorted(qs):
            sh = psi[q].shape
            rows.setdefault(q[:split], math.prod(sh[:split]))
            cols.setdefault(q[split:], math.prod(sh[split:]))
        ro = dict(zip(rows, np.cumsum([0] + list(rows.values()))))
        co = dict(zip(cols, np.cumsum([0] + list(cols.values()))))
        M = np.zeros((sum(rows.values()), sum(cols.values())), complex)
        for q in qs:
            i, j = ro[q[:split]], co[q[split:]]
            M[i:i + rows[q[:split]], j:j + cols[q[split:]]] = psi[q].reshape(rows[q[:split]], -1)
        u, s, v = np.linalg.svd(M, full_matrices=False)
        total += len(s)
        parts.append((u, s, v, rows, cols, ro, co))
        vals += [(x, len(parts) - 1) for x in s]
    vals.sort(key=lambda t: -t[0])
    kept = max(1, min(D, sum(x > TOL_SVD for x, _ in vals)))
    count = [0] * len(parts)
    for _, p in vals[:kept]:
        count[p] += 1
    out = {}
    for (u, s, v, rows, cols, ro, co), k in zip(parts, count):
        if k == 0:
            continue
        M = (u[:, :k] * s[:k]) @ v[:k]
        for qr, nr in rows.items():
            for qc, nc in cols.items():
                out[qr + qc] = M[ro[qr]:ro[qr] + nr, co[qc]:co[qc] + nc]
    return out, kept, total


def exact(case, seed):
    op = case["op"]
    if op == "energy":
        ch = _chain(case)
        L = _blocks(_boundary(1, 0))
        for a, w in zip(H.random_mps(ch, case["D"], seed=seed), H.hamiltonian_mpo(ch)):
            L = _env_l2r(L, _blocks(a), _blocks(w))
        return float(sum(v.real.sum() for v in L.values()))
    # a whole step is thousands of the contractions below: minutes; so is an evolution over thousands of blocks
    if op == "step" or (op in ("krylov", "svd") and _pairs(case) > 3000):
        return None
    mps, mpo, centre = _state(case, seed)
    s, nsite = case["site"], case.get("nsite", 1)
    last = s if nsite == 0 else s + nsite - 1
    A, W = [_blocks(t) for t in mps], [_blocks(t) for t in mpo]
    L, R = _blocks(_boundary(1, 0)), _blocks(_boundary(-1, mps[-1].blocks[0][0][2]))
    if op != "env" or case["l2r"]:
        for i in range(s + 1 if nsite == 0 else s):
            L = _env_l2r(L, A[i], W[i])
    if op != "env" or not case["l2r"]:
        for i in range(len(mps) - 1, last, -1):
            R = _env_r2l(R, A[i], W[i])
    if op == "env":
        return dict(env=_flat(_env_l2r(L, A[s], W[s]) if case["l2r"] else _env_r2l(R, A[s], W[s])))
    W1, W2 = W[s] if nsite >= 1 else None, W[s + 1] if nsite == 2 else None
    psi = _blocks(centre) if nsite == 0 else A[s] if nsite == 1 else _contract(A[s], "xsm", A[s + 1], "mtb", "xstb")
    if op == "apply":
        y = {k: 0.5 * DT * v for k, v in _apply(nsite, L, psi, W1, W2, R).items()}
        return dict(psi=_flat({**{k: np.zeros_like(v) for k, v in psi.items()}, **y}))
    if op in ("krylov", "svd"):
        out, m = _krylov(nsite, L, psi, W1, W2, R, case.get("reverse", False))
        if op == "krylov":
            return dict(psi=_flat(out), dimension=m)
        out, kept, total = _truncated(out, _split(case), case["D"])
        return dict(psi=_flat(out), kept=kept, total=total)
    like = mps[s] if nsite == 1 else _pair_layout(mps[s], mps[s + 1])
    y = _blocks(_cotangent(case, seed, like))
    Lc, Rc, pc = _conj(L), _conj(R), _conj(psi)
    if nsite == 1:
        W1c = _conj(W1)
        left = _contract(Lc, "pwx", y, "puq", "wxuq")
        lw = _contract(left, "wxuq", W1c, "uwsv", "xqsv")
        Lp = _contract(Lc, "pwx", pc, "xsb", "pwsb")
        Lpy = _contract(Lp, "pwsb", y, "puq", "wsbuq")
        out = dict(psi=_contract(lw, "xqsv", Rc, "qvb", "xsb"), W1=_contract(Lpy, "wsbuq", Rc, "qvb", "uwsv"),
                   R=_contract(Lpy, "wsbuq", W1c, "uwsv", "qvb"),
                   L=_contract(_contract(_contract(y, "puq", Rc, "qvb", "puvb"), "puvb", W1c, "uwsv", "pbws"),
                               "pbws", pc, "xsb", "pwx"))
    else:
        W1c, W2c = _conj(W1), _conj(W2)
        lw = _contract(_contract(Lc, "pwx", y, "puzq", "wxuzq"), "wxuzq", W1c, "uwsv", "xzqsv")
        rw = _contract(_contract(Rc, "qyb", y, "puzq", "ybpuz"), "ybpuz", W2c, "zvty", "bputv")  # [b, p, u, t, v]
        Lp = _contract(Lc, "pwx", pc, "xstb", "pwstb")
        Lpw = _contract(Lp, "pwstb", W1c, "uwsv", "ptbuv")
        Ry = _contract(Rc, "qyb", y, "puzq", "ybpuz")
        out = dict(psi=_contract(_contract(lw, "xzqsv", W2c, "zvty", "xqsty"), "xqsty", Rc, "qyb", "xstb"),
                   L=_contract(_contract(rw, "bputv", W1c, "uwsv", "bptws"), "bptws", pc, "xstb", "pwx"),
                   W1=_contract(Lp, "pwstb", rw, "bputv", "uwsv"),
                   W2=_contract(Lpw, "ptbuv", Ry, "ybpuz", "zvty"),
                   R=_contract(_contract(Lpw, "ptbuv", y, "puzq", "tbvzq"), "tbvzq", W2c, "zvty", "qyb"))
    return {k: _flat(v) for k, v in out.items()}


# ------------------------------------------------------------------ work
class _Count:
    """Bond structures of a chain and the 8 M N K flops and 16-byte elements of its contractions."""

    def __init__(self, case, index=0):
        self.ch = _chain(case, index)
        self.bonds = H.random_mps_structure(self.ch, case["D"])
        self.dims = self.ch.site_dims()
        self.mpo = H.hamiltonian_mpo(self.ch)

    def site(self, i):
        L, R = self.bonds[i], self.bonds[i + 1]
        return {(l, s, l + s): (L[l], 1, R[l + s]) for l in L for s in range(self.dims[i]) if l + s in R}

    def pair(self, i):
        L, R = self.bonds[i], self.bonds[i + 2]
        return {(l, s, t, l + s + t): (L[l], 1, 1, R[l + s + t]) for l in L for s in range(self.dims[i])
                for t in range(self.dims[i + 1]) if l + s + t in R}

    def centre(self, i):
        return {(q, q): (d, d) for q, d in self.bonds[i + 1].items()}

    def channels(self, i):
        """MPO bond dimension per charge on bond i."""
        if i < self.ch.n_sites:
            return {q[1]: a.shape[1] for q, a in self.mpo[i].blocks}
        return {q[3]: a.shape[3] for q, a in self.mpo[i - 1].blocks}

    def env(self, i):
        b, w = self.bonds[i], self.channels(i)
        return {(p, c, p + s * c): (b[p], d, b[p + s * c]) for s in (1, -1) for p in b for c, d in w.items()
                if p + s * c in b}

    def apply(self, nsite, i):
        """(flops, elements in and out) of one H_eff apply at site i."""
        psi = self.centre(i) if nsite == 0 else self.site(i) if nsite == 1 else self.pair(i)
        lb, rb = (i + 1, i + 1) if nsite == 0 else (i, i + nsite)
        wl, wr = sum(self.channels(lb).values()), sum(self.channels(rb).values())
        n = sum(map(math.prod, psi.values()))
        envs = sum(map(math.prod, self.env(lb).values())) + sum(map(math.prod, self.env(rb).values()))
        # a block meets one charge of the other bond index per MPO channel: 8 (D' w) D N on each side
        left = right = 0.0
        dl, dr = self.bonds[lb], self.bonds[rb]
        for q, s in psi.items():
            for c, d in self.channels(lb).items():
                left += 8.0 * dl.get(q[0] - c, 0) * d * math.prod(s)
            for c, d in self.channels(rb).items():
                right += 8.0 * dr.get(q[-1] + c, 0) * d * math.prod(s)
        mix = 0.0 if nsite == 0 else 8.0 * nsite * n * min(wl, wr) * 2
        mpo = sum(a.size for j in range(i, i + nsite) for _, a in self.mpo[j].blocks)
        return left + right + mix, envs + mpo + 2.0 * n, n

    def svd(self, psi, split, D):
        """Dense factorisation of every charge sector (about 8 (2 m n k + 2 k^3) flops), truncated factors out."""
        sec = {}
        for q, s in psi.items():
            r, c = sec.setdefault(sum(q[:split]), ({}, {}))
            r[q[:split]], c[q[split:]] = math.prod(s[:split]), math.prod(s[split:])
        fl = 0.0
        for r, c in sec.values():
            m, n = sum(r.values()), sum(c.values())
            k = min(m, n)
            fl += 8.0 * (2.0 * m * n * k + 2.0 * k ** 3)
        n = sum(map(math.prod, psi.values()))
        return fl, 2.0 * n

    def step(self, mode, D):
        fl = by = 0.0
        ns = self.ch.n_sites
        for i in range(ns - mode + 1):
            f, e, n = self.apply(mode, i)
            g, h = self.svd(self.site(i) if mode == 1 else self.pair(i), 2, D)
            k, m, _ = self.apply(mode - 1, min(i, ns - 1 if mode == 2 else ns - 2))
            fl += 2 * ((MAX_ITER - 1) * (f + 44.0 * n + k) + g)
            by += 2 * (e + h + m)
        return fl, by


def _pairs(case):
    c = _Count(case)
    psi = c.site(case["site"]) if case.get("nsite", 1) <= 1 else c.pair(case["site"])
    return len(psi) * len(c.channels(case["site"]))


def work(case):
    """8 M N K per contraction; 16 bytes per complex element read or written once."""
    c, op, nsite = _Count(case), case["op"], case.get("nsite", 1)
    if op == "step":
        got = [_Count(case, i).step(case["mode"], case["D"]) for i in range(case["chains"])]
        return dict(flops=sum(f for f, _ in got), bytes=16.0 * sum(e for _, e in got))
    if op == "energy":
        fl = by = 0.0
        for i in range(c.ch.n_sites):
            f, _, n = c.apply(1, i)
            fl, by = fl + f, by + 2.0 * n + sum(a.size for _, a in c.mpo[i].blocks)
        return dict(flops=fl, bytes=16.0 * by)
    f, e, n = c.apply(nsite, case["site"])
    if op == "krylov":
        return dict(flops=(MAX_ITER - 1) * (f + 44.0 * n), bytes=16.0 * e)
    if op == "svd":
        f, e = c.svd(c.site(case["site"]) if nsite == 1 else c.pair(case["site"]), _split(case), case["D"])
        return dict(flops=f, bytes=16.0 * e)
    if op == "adjoint":
        return dict(flops=3.0 * f, bytes=16.0 * 2.0 * e)
    return dict(flops=f, bytes=16.0 * e)
