"""The calls a user of dmrg_c_gb300 makes, over the sizes they make them at.

A DMRG program makes, step by step, the ground state of a superblock ("solve"), the superblock
Hamiltonian before it ("build"), and after it the site observables ("expect"), the truncation of
the enlarged block ("truncate") and the renormalisation of the block operators ("renorm"); a
reference program that keeps its matrix on the host calls the drop-in product ("product").  An
exact-diagonalisation program builds and solves one chain ("ed") or many together ("batch").

The superblocks are the ones recorded from the reference's own DMRG runs (tests/golden): XXZ L=32
m=64, Kondo lattice L=24 m=127, Hubbard L=64 m=512.  A smaller m keeps the m block states of
largest weight in the recorded ground state, as a truncation does, and restricts every block
operator to them.  The seed scales the couplings between the positions (and draws start vectors,
chain parameters and observables), so every seed is another Hamiltonian of the same structure.
"""
import ctypes as C
import functools
import math
import os

import numpy as np
import torch

from dmrg_c_gb300 import abi, ed_models, sb_models
from dmrg_c_gb300 import lib as L

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(sb_models.__file__))), "tests", "golden")
FIXTURE = {"xxz": "dmrg_xxz_vf_sweep4.npz", "klm": "dmrg_klm_vf_sweep4.npz", "hubbard": "dmrg_hubbard_vf_sweep4.npz"}
M_RANGE = {"xxz": (20, 64), "klm": (24, 127), "hubbard": (48, 512)}
# operator applications of one FP64 ground state (Lanczos, then the CG of inverse iteration)
PRODUCTS = {"xxz": 90, "klm": 170, "hubbard": 250}


def listed():
    return [
        # every sweep of a small spin chain: a few thousand states, where a step is all latency
        {"name": "solve_xxz_m64", "kind": "solve", "model": "xxz", "m": 64, "mixed": 0},
        # the ordinary DMRG step: the matrix stays in L2
        {"name": "solve_klm_m127", "kind": "solve", "model": "klm", "m": 127, "mixed": 0},
        # the largest DMRG step: 56 M stored elements, streamed from HBM in every product
        {"name": "solve_hubbard_m512", "kind": "solve", "model": "hubbard", "m": 512, "mixed": 0},
        # the same in the mixed-precision form with full reorthogonalisation
        {"name": "solve_hubbard_m512_mixed", "kind": "solve", "model": "hubbard", "m": 512, "mixed": 1},
        # a reference program's MATRIX_VECTOR_PRODUCT_SYM on its host arrays (upload and expansion
        # of the symmetric half, product, download)
        {"name": "product_klm_m127", "kind": "product", "model": "klm", "m": 127},
        # GET_HAM_LLLRRRRL of the largest step: term list to operator, then the first product
        {"name": "build_hubbard_m512", "kind": "build", "model": "hubbard", "m": 512, "values": 1},
        # the truncation of the largest step: density blocks of up to 216 pairs
        {"name": "truncate_hubbard_m512", "kind": "truncate", "model": "hubbard", "m": 512},
        # the site observables of the largest step, on a resident vector
        {"name": "expect_hubbard_m512", "kind": "expect", "model": "hubbard", "m": 512, "sites": 31},
        # T^dagger O T of one block operator of the largest step
        {"name": "renorm_hubbard_m512", "kind": "renorm", "model": "hubbard", "m": 512},
        # a small exact diagonalisation, below the size where the reference goes dense
        {"name": "ed_xxz_L12", "kind": "ed", "model": "xxz", "L": 12, "mixed": 0},
        # a served request: Hubbard chain at half filling, built and solved in the mixed form
        {"name": "ed_hubbard_L12_mixed", "kind": "ed", "model": "hubbard", "L": 12, "mixed": 2},
        # XXZ chains of uneven length solved together in lock-step, FP64
        {"name": "batch_xxz_24", "kind": "batch", "count": 24, "Lmin": 12, "Lmax": 20, "mixed": 0},
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    def superblock(top=1.0):
        model = rng.choice(["xxz", "klm", "hubbard"])
        lo, hi = M_RANGE[model]
        return {"model": model, "m": log_int(lo, max(lo, int(hi * top)))}

    kind = rng.choice(["solve", "solve", "product", "build", "ed", "batch", "truncate", "expect", "renorm"])
    if kind == "solve":
        return {"kind": kind, **superblock(), "mixed": rng.choice([0, 0, 1, 2])}
    if kind == "product":
        return {"kind": kind, **superblock(0.5)}
    if kind == "build":
        return {"kind": kind, **superblock(), "values": rng.choice([1, 3])}
    if kind == "ed":
        model = rng.choice(["xxz", "hubbard"])
        L_ = 2 * rng.randint(4, 11) if model == "xxz" else rng.randint(4, 11)
        return {"kind": kind, "model": model, "L": L_, "mixed": rng.choice([0, 2])}
    if kind == "batch":
        lo = 2 * rng.randint(6, 8)
        return {"kind": kind, "count": log_int(2, 24), "Lmin": lo, "Lmax": 2 * rng.randint(lo // 2, 10), "mixed": rng.choice([0, 2])}
    if kind == "expect":
        return {"kind": kind, **superblock(), "sites": rng.randint(2, 31)}
    return {"kind": kind, **superblock()}


# ---------------------------------------------------------------------------------------
# Superblocks
# ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def recorded(model):
    return sb_models.load_dmrg_superblock(os.path.join(GOLDEN, FIXTURE[model]))


def restrict(op, keep):
    """The rows and columns `keep` (ascending) of a block operator, as a Crs."""
    n = len(op.row) - 1
    new = -np.ones(n, np.int64)
    new[keep] = np.arange(len(keep))
    rows = np.repeat(np.arange(n), np.diff(op.row))
    cols, vals = op.col[:op.nnz], op.val[:op.nnz]
    ok = (new[rows] >= 0) & (new[cols] >= 0)
    row = np.concatenate([[0], np.cumsum(np.bincount(new[rows[ok]], minlength=len(keep)))])
    return abi.Crs(row, new[cols[ok]], vals[ok], n=len(keep))


@functools.lru_cache(maxsize=32)
def parts(model, m):
    """(states, inv, ops, terms, ele, vector) of the recorded superblock with m states a block."""
    R = recorded(model)
    S, v2 = R.model, R.gs_vec ** 2
    keep = []
    for pos, dim in ((S.LL, S.dim_LL), (S.RR, S.dim_RR)):
        weight = np.bincount(pos, weights=v2, minlength=dim)
        keep.append(np.sort(np.argsort(-weight, kind="stable")[:m]))
    new = []
    for k, dim in zip(keep, (S.dim_LL, S.dim_RR)):
        a = -np.ones(dim, np.int64)
        a[k] = np.arange(len(k))
        new.append(a)
    ok = (new[0][S.LL] >= 0) & (new[1][S.RR] >= 0)
    states = (new[0][S.LL[ok]].astype(np.int16), S.LR[ok], new[1][S.RR[ok]].astype(np.int16), S.RL[ok])
    dims = (len(keep[0]), S.d, len(keep[1]), S.d)
    inv = -np.ones(int(np.prod(dims)), np.int32)
    inv[flat(states, dims)] = np.arange(len(states[0]), dtype=np.int32)
    ops, seen = list(S.ops), set()
    for p1, p2, o1, o2, *_ in S.terms:
        for p, o in ((p1, o1), (p2, o2)):
            if p in (0, 2) and o not in seen:
                seen.add(o)
                ops[o] = restrict(S.ops[o], keep[p // 2])
    ele = [None if e is None else (e[keep[p // 2]] if p in (0, 2) else e) for p, e in enumerate(S.ele)]
    return states, dims, inv, ops, list(S.terms), ele, R.gs_vec[ok]


def flat(states, dims):
    LL, LR, RR, RL = (np.asarray(a, np.int64) for a in states)
    return ((LL * dims[1] + LR) * dims[2] + RR) * dims[3] + RL


def terms_of(case, seed):
    """The term list with the coupling of each pair of positions scaled by the seed."""
    rng = np.random.default_rng(seed)
    scale = {p: 1.0 + 0.1 * rng.uniform(-1, 1) for p in ((0, -1), (2, -1), (1, -1), (3, -1), (0, 1), (2, 3), (1, 3))}
    return [(t[0], t[1], t[2], t[3], t[4] * scale[(t[0], t[1])], t[5], t[6]) for t in parts(case["model"], case["m"])[4]]


def superblock_model(case, seed):
    states, dims, inv, ops, _, ele, _ = parts(case["model"], case["m"])
    return sb_models.SBModel(len(states[0]), dims[0], dims[2], dims[1], *states, inv, ops, terms_of(case, seed), ele)


def block_vector(case, seed):
    """A normalised superblock vector with a ground state's Schmidt spectrum: the recorded one with
    the weights of the block states changed a little."""
    states, dims, _, _, _, _, v = parts(case["model"], case["m"])
    rng = np.random.default_rng(seed + 1)
    f, g = (1.0 + 0.2 * rng.uniform(-1, 1, size=n) for n in (dims[0], dims[2]))
    v = v * f[states[0]] * g[states[2]]
    return v / np.linalg.norm(v)


def lllr(case):
    """The LLLR list of the superblock: pairs (LL, LR), states of each, the index of its label.
    (Pairs of one label have the same (RR, RL) partners, of another label none of them.)"""
    states, dims, *_ = parts(case["model"], case["m"])
    pair = states[0].astype(np.int64) * dims[1] + states[1]
    first = np.flatnonzero(np.concatenate([[True], pair[1:] != pair[:-1]]))
    count = np.diff(np.concatenate([first, [len(pair)]]))
    partner = states[2][first].astype(np.int64) * dims[3] + states[3][first]
    label = np.cumsum(np.concatenate([[0], partner[1:] != partner[:-1]]))
    return states[0][first], states[1][first], count.astype(np.int32), label.astype(np.int32)


def density_blocks(case, v):
    """[(first pair, X_g)]: the vector as one dense pairs x partners matrix for each label."""
    _, _, count, label = lllr(case)
    at, out, p0 = 0, [], 0
    for g in range(int(label[-1]) + 1):
        P = int(np.sum(label == g))
        Q = int(count[p0])
        out.append((p0, v[at:at + P * Q].reshape(P, Q)))
        at, p0 = at + P * Q, p0 + P
    return out


def block_operators(case, seed, count):
    """Seeded symmetric operators on each block that conserve its labels (the sparsity of the block
    Hamiltonian), and one diagonal site operator."""
    states, dims, _, ops, terms, _, _ = parts(case["model"], case["m"])
    rng = np.random.default_rng(seed + 2)
    out = []
    for pos in (0, 2):
        H = ops[next(t[2] for t in terms if t[0] == pos and t[1] < 0)]
        n = dims[pos]
        rows, cols = np.repeat(np.arange(n), np.diff(H.row)), H.col[:H.nnz].astype(np.int64)
        for _ in range(count):
            A = rng.standard_normal((n, n))
            out.append(abi.Crs(H.row, H.col[:H.nnz], ((A + A.T) * 0.5)[rows, cols], n=n))
    d = dims[1]
    site = abi.Crs(np.arange(d + 1), np.arange(d, dtype=np.int32), rng.standard_normal(d), n=d)
    return out, site


def renorm_inputs(case, seed):
    """(T's columns' label blocks as CCS arrays, the operator on the LLLR pairs as CRS arrays)."""
    states, dims, _, ops, terms, _, _ = parts(case["model"], case["m"])
    LLp, LRp, _, _ = lllr(case)
    nl, cols = len(LLp), []
    for p0, X in density_blocks(case, block_vector(case, seed)):
        w, V = np.linalg.eigh(X @ X.T)
        cols += [(w[k], p0, V[:, k]) for k in range(len(w))]
    order = np.argsort([-c[0] for c in cols], kind="stable")[:case["m"]]
    kept = sorted((cols[k] for k in order), key=lambda c: c[1])
    T = (np.concatenate([[0], np.cumsum([len(c[2]) for c in kept])]),
         np.concatenate([c[1] + np.arange(len(c[2])) for c in kept]), np.concatenate([c[2] for c in kept]))
    pair = -np.ones((dims[0], dims[1]), np.int64)
    pair[LLp, LRp] = np.arange(nl)
    H = ops[next(t[2] for t in terms if t[0] == 0 and t[1] < 0)]
    hr, hc = np.repeat(np.arange(dims[0]), np.diff(H.row)), H.col[:H.nnz]
    r, c = pair[hr].ravel(), pair[hc].ravel()
    val = np.repeat(H.val[:H.nnz], dims[1])
    ok = (r >= 0) & (c >= 0)
    at = np.lexsort((c[ok], r[ok]))
    row = np.concatenate([[0], np.cumsum(np.bincount(r[ok], minlength=nl))])
    return nl, len(kept), T, (row, c[ok][at], val[ok][at])


def chain_parameters(case, seed, k=0):
    rng = np.random.default_rng([seed, k])
    if case.get("model", "xxz") == "xxz":
        return {"Jz": float(rng.uniform(0, 2)), "hz": float(rng.uniform(0, 1))}
    return {"U": float(rng.uniform(0, 8)), "hz": float(rng.uniform(0, 0.5))}


def chain(case, seed, k=0, length=None):
    p, n = chain_parameters(case, seed, k), length or case["L"]
    if case.get("model", "xxz") == "xxz":
        return ed_models.xxz_chain(n, Jxy=1.0, **p)
    return ed_models.hubbard_chain(n, t=-1.0, n_ele=n - n % 2, **p)


def batch_lengths(case):
    span = (case["Lmax"] - case["Lmin"]) // 2 + 1
    return [case["Lmin"] + 2 * (k % span) for k in range(case["count"])]


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ---------------------------------------------------------------------------------------
# What a program has in hand before the call
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": dict(case)}
    if kind == "solve":
        crs = L.SuperblockCRS(superblock_model(case, seed))
        s["matrix"] = crs.matrix(L.DG_VALUES_BOTH if case["mixed"] else L.DG_VALUES_F64)
        crs.close()
        s["params"] = L.default_params(seed=seed, mixed=case["mixed"])
        s["out"] = torch.empty(s["matrix"].n, dtype=torch.float64, device="cuda")
    elif kind == "product":
        crs = L.SuperblockCRS(superblock_model(case, seed))
        s["crs"] = abi.Crs(*crs.download())
        crs.close()
        s["x"] = np.random.default_rng(seed).standard_normal(s["crs"].n)
        s["out"] = np.empty(s["crs"].n)
    elif kind == "build":
        s["model"] = superblock_model(case, seed)
        s["x"] = cuda(np.random.default_rng(seed).standard_normal(s["model"].n))
        s["out"] = torch.empty_like(s["x"])
    elif kind == "ed":
        s["model"] = chain(case, seed)
        s["params"] = L.default_params(seed=seed, mixed=case["mixed"])
    elif kind == "batch":
        s["matrices"] = []
        for k, n in enumerate(batch_lengths(case)):
            ed = L.EDSystem(chain(case, seed, k, n))
            s["matrices"].append(ed.matrix(L.DG_VALUES_BOTH if case["mixed"] else L.DG_VALUES_F64))
            ed.close()
        s["params"] = L.default_params(seed=seed, mixed=case["mixed"])
    elif kind == "truncate":
        states, dims, inv, *_ = parts(case["model"], case["m"])
        LLp, LRp, count, label = lllr(case)
        v = block_vector(case, seed)
        basis = abi.DMRG_BASIS(LL_LLLRRRRL=abi.ptr(states[0], C.c_short), LR_LLLRRRRL=abi.ptr(states[1], C.c_short),
                               RR_LLLRRRRL=abi.ptr(states[2], C.c_short), RL_LLLRRRRL=abi.ptr(states[3], C.c_short),
                               Inv_LLLRRRRL=abi.ptr(inv, C.c_int), dim_LLLRRRRL=len(v), dim_LL=dims[0], dim_RR=dims[2],
                               dim_onsite=dims[1], LL_LLLR=abi.ptr(LLp, C.c_short), LR_LLLR=abi.ptr(LRp, C.c_short),
                               dim_LLLR=len(LLp), Sum_LLLR=abi.ptr(count, C.c_int))
        s.update(basis=basis, label=label, v=v, time=abi.DMRG_TIME(), largest=int(np.bincount(label).max()),
                 keep=(states, inv, LLp, LRp, count))
    elif kind == "expect":
        states, dims, inv, *_ = parts(case["model"], case["m"])
        k = case["sites"]
        ops, site = block_operators(case, seed, k)
        s["basis"] = L.superblock_states(states, dims[0], dims[2], dims[1], inv=inv)
        s["ops"] = L.BlockOperators(ops + [site], [dims[0]] * k + [dims[2]] * k + [dims[1]])
        s["terms"] = ([(0, i, 0, 0) for i in range(k)] + [(1, 2 * k, 0, 0), (3, 2 * k, 0, 0)]
                      + [(2, k + i, 0, 0) for i in range(k)])
        s["v"] = cuda(block_vector(case, seed))
    elif kind == "renorm":
        nl, nr, (tc, tr, tv), (row, col, val) = renorm_inputs(case, seed)
        s["args"] = (abi.Crs(tc, tr, tv, n=nr, ncol=nl), abi.Crs(row, col, val, n=nl), abi.Ccs(tc, tr, tv, nl, nr),
                     abi.Crs(np.zeros(nr + 1), np.zeros(nr * nr), np.zeros(nr * nr), n=nr), abi.Ccs.empty(nr, nl * nr))
        s["scratch"] = np.zeros(nl)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "solve":
        _, info = L.ground_state(s["matrix"], s["params"], out=s["out"])
        return {"energy": np.float64(info.eig_val), "vector": s["out"]}
    if kind == "product":
        L.load().MATRIX_VECTOR_PRODUCT_SYM(s["crs"].ref, abi.ptr(s["x"], C.c_double), abi.ptr(s["out"], C.c_double), None, 1)
        return s["out"]
    if kind == "build":
        crs = L.SuperblockCRS(s["model"])
        matrix = crs.matrix(s["case"]["values"])
        crs.close()
        matrix.spmv(s["x"], s["out"])
        n, nnz = matrix.n, matrix.nnz
        matrix.close()
        return {"n": n, "stored": nnz, "y": s["out"]}
    if kind == "ed":
        ed = L.EDSystem(s["model"])
        matrix = ed.matrix(L.DG_VALUES_BOTH if s["case"]["mixed"] else L.DG_VALUES_F64)
        ed.close()
        vector = torch.empty(matrix.n, dtype=torch.float64, device="cuda")
        _, info = L.ground_state(matrix, s["params"], out=vector)
        matrix.close()
        return {"energy": np.float64(info.eig_val), "vector": vector}
    if kind == "batch":
        vectors, infos = L.batch_ground_state(s["matrices"], s["params"])
        return {"energy": np.array([i.eig_val for i in infos]), "vector": vectors}
    if kind == "truncate":
        return truncate(s)
    if kind == "expect":
        return L.sb_expect(s["basis"], s["basis"], s["ops"], s["terms"], s["v"], s["v"])
    M1, M2, M3, out, work = s["args"]
    L.load().CRS_CRS_CCS_PRODUCT(M1.ref, M2.ref, M3.ref, out.ref, work.ref, abi.ptr(s["scratch"], C.c_double))
    return {"row": out.row, "col": out.col, "val": out.val, "work_col": work.col, "work_row": work.row, "work_val": work.val}


def truncate(s):
    lib, libc = L.load(), C.CDLL(None)
    libc.free.argtypes = [C.c_void_p]
    S = lib.DMRG_GET_SYSTEM_INFO_Q1(abi.ptr(s["label"], C.c_int), C.byref(s["basis"]), abi.ptr(s["v"], C.c_double),
                                    s["case"]["m"], 1, C.byref(s["time"])).contents
    T, k = S.Trans_Matrix.contents, S.dim_renorm
    nnz, m, most = T.Col[k], s["case"]["m"], s["case"]["m"] * s["largest"]

    def copy(p, n, room):   # the result in an array of the size it can reach, as a program keeps it
        a = np.zeros(room, np.ctypeslib.as_array(p, (1,)).dtype)
        a[:n] = np.ctypeslib.as_array(p, (n,))
        return a

    out = {"weights": copy(S.Val_DM_Dist, S.dim_LLLR, S.dim_LLLR), "label": copy(S.Q_Number1, k, m),
           "col": copy(T.Col, k + 1, m + 1), "row": copy(T.Row, nnz, most), "val": copy(T.Val, nnz, most)}
    for M in (T, S.Trans_Matrix_Dagger.contents):
        for a in (M.Val, M.Row, M.Col):
            libc.free(C.cast(a, C.c_void_p))
    for a in (S.Trans_Matrix, S.Trans_Matrix_Dagger, S.Val_DM_Dist, S.Q_Number1, S.Q_Number2, S.Q_Number3, C.pointer(S)):
        libc.free(C.cast(a, C.c_void_p))
    return out


# ---------------------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------------------
def chain_size(model, n):
    """(states of the sector, stored elements)."""
    if model == "xxz":
        dim = math.comb(n, n // 2)
        return dim, dim + (n - 1) * 2 * math.comb(n - 2, n // 2 - 1)
    h = n // 2 if n % 2 == 0 else (n - 1) // 2
    dim = math.comb(n, h) ** 2
    return dim, dim + 2 * (n - 1) * 2 * math.comb(n - 2, h - 1) * math.comb(n, h)


def work(case):
    kind = case["kind"]
    if kind in ("ed", "batch"):
        sizes = [chain_size(case["model"], case["L"])] if kind == "ed" else [chain_size("xxz", n) for n in batch_lengths(case)]
        n, nnz = (sum(v) for v in zip(*sizes))
        return {"bytes": 12 * nnz + 16 * n, "flops": 2 * nnz * 120}
    states, dims, inv, ops, *_ = parts(case["model"], case["m"])
    n = len(states[0])
    if kind in ("truncate", "expect", "renorm"):
        P = [(X.shape[0], X.shape[1]) for _, X in density_blocks(case, np.zeros(n))]
        if kind == "truncate":
            return {"bytes": 8 * (n + sum(p * p for p, _ in P)), "flops": sum(p * p * q + 9 * p ** 3 for p, q in P)}
        if kind == "expect":
            nnz = sum(o.nnz for o in ops[:2])
            return {"bytes": 8 * n + 12 * case["sites"] * nnz, "flops": sum(p * p * q + q * q * p for p, q in P) + 2 * case["sites"] * nnz}
        nl, nr, T, O = renorm_inputs(case, 0)
        flops = 2 * int(np.sum(np.diff(O[0])[T[1]])) + 2 * nr * len(T[2])
        return {"bytes": 12 * (2 * len(T[2]) + len(O[2])) + 12 * nr * nr // 4, "flops": flops}
    crs = L.SuperblockCRS(superblock_model(case, 0))
    lower = crs.nnz
    crs.close()
    full = 2 * lower - n
    if kind == "solve":
        return {"bytes": (8 if case["mixed"] else 12) * full + 16 * n, "flops": 2 * full * PRODUCTS[case["model"]]}
    if kind == "product":
        return {"bytes": 12 * lower + 24 * n, "flops": 2 * full}
    return {"bytes": 4 * len(inv) + 8 * n + sum(12 * o.nnz for o in ops) + 12 * full + 16 * n, "flops": 2 * full}


# ---------------------------------------------------------------------------------------
# The same in 64 bits, by plain torch and numpy
# ---------------------------------------------------------------------------------------
def superblock_product(case, seed):
    """v -> H v on the sector, term by term on the dense (LL, LR, RR, RL) tensor."""
    states, dims, _, ops, _, ele, _ = parts(case["model"], case["m"])
    at = cuda(flat(states, dims))
    dense = {}

    def matrix(o):
        if o not in dense:
            A = np.zeros((ops[o].n, ops[o].n))
            A[np.repeat(np.arange(ops[o].n), np.diff(ops[o].row)), ops[o].col[:ops[o].nnz]] = ops[o].val[:ops[o].nnz]
            dense[o] = cuda(A)
        return dense[o]

    def shaped(a, pos):
        return a.reshape([-1 if p == pos else 1 for p in range(4)])

    terms = []
    for p1, p2, o1, o2, coef, mask, even in terms_of(case, seed):
        sign = torch.ones(1, 1, 1, 1, dtype=torch.float64, device="cuda")
        for p in range(4):
            if mask & (1 << p):
                sign = sign * shaped(cuda(1.0 - 2.0 * (np.asarray(ele[p]) % 2)), p)
        terms.append((p1, p2, matrix(o1), matrix(o2) if p2 >= 0 else None, coef * (even if mask else 1) * sign))

    def apply(v):
        x = torch.zeros(int(np.prod(dims)), dtype=torch.float64, device="cuda")
        x[at] = v
        x = x.reshape(dims)
        y = torch.zeros_like(x)
        for p1, p2, A, B, f in terms:
            t = x if B is None else torch.movedim(torch.tensordot(B, x, dims=([1], [p2])), 0, p2)
            y += f * torch.movedim(torch.tensordot(A, t, dims=([1], [p1])), 0, p1)
        return y.reshape(-1)[at]

    return apply, len(at)


def chain_product(case, seed):
    """v -> H v of an open chain on its sector, bond by bond on the dense tensor of local states."""
    n, p = case["L"], chain_parameters(case, seed)
    if case["model"] == "xxz":
        d, sz = 2, np.array([0.5, -0.5])
        up = np.array([[0.0, 1.0], [0.0, 0.0]])
        bond = p["Jz"] * np.kron(np.diag(sz), np.diag(sz)) + 0.5 * (np.kron(up, up.T) + np.kron(up.T, up))
        local = p["hz"] * sz
        charge, target = [2 * sz], [0]
    else:
        d, Z, c, one = 4, np.diag([1.0, -1.0]), np.array([[0.0, 1.0], [0.0, 0.0]]), np.eye(2)
        mode = [functools.reduce(np.kron, [Z] * k + [c] + [one] * (3 - k)) for k in range(4)]
        bond = -sum(mode[k].T @ mode[k + 2] + mode[k + 2].T @ mode[k] for k in (0, 1))
        nd, nu = (np.array(a, float) for a in ([0, 1, 0, 1], [0, 0, 1, 1]))   # state 2 n_up + n_down
        local = p["U"] * nu * nd + 0.5 * p["hz"] * (nu - nd)
        charge, target = [nu + nd, nu - nd], [n - n % 2, 0]
    ok = torch.ones(d ** n, dtype=torch.bool, device="cuda")
    diag = torch.zeros(d ** n, dtype=torch.float64, device="cuda")
    for q, t in zip(charge, target):
        tot = torch.zeros(d ** n, dtype=torch.float64, device="cuda")
        for s in range(n):
            tot.reshape(d ** s, d, -1).add_(cuda(q)[None, :, None])
        ok &= tot == t
    for s in range(n):
        diag.reshape(d ** s, d, -1).add_(cuda(local)[None, :, None])
    at, B = torch.nonzero(ok).reshape(-1), cuda(bond)
    dd = diag[at]

    def apply(v):
        x = torch.zeros(d ** n, dtype=torch.float64, device="cuda")
        x[at] = v
        y = torch.zeros_like(x)
        for s in range(n - 1):
            y.reshape(d ** s, d * d, -1).add_(torch.matmul(B, x.reshape(d ** s, d * d, -1)))
        return y[at] + dd * v

    return apply, len(at)


def lowest_energy(apply, n):
    """Lanczos with full reorthogonalisation in 64 bits."""
    v = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    V, a, b, last = [v / v.norm()], [], [], math.inf
    for k in range(min(n, 400)):
        w = apply(V[k])
        a.append(float(V[k] @ w))
        basis = torch.stack(V)
        for _ in range(2):
            w = w - basis.T @ (basis @ w)
        beta = float(w.norm())
        if k % 10 == 9 or k == n - 1 or beta < 1e-12:
            e = float(np.linalg.eigvalsh(np.diag(a) + np.diag(b, 1) + np.diag(b, -1))[0])
            if abs(e - last) < 1e-13 * abs(e) or k == n - 1 or beta < 1e-12:
                return e
            last = e
        b.append(beta)
        V.append(w / beta)
    return None


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "ed"):   # an eigenvector has no value of its own: its sign is free
        apply, n = superblock_product(case, seed) if kind == "solve" else chain_product(case, seed)
        e = lowest_energy(apply, n)
        return {"energy": None if e is None else np.float64(e), "vector": None}
    if kind in ("product", "build"):
        apply, n = superblock_product(case, seed)
        y = apply(cuda(np.random.default_rng(seed).standard_normal(n)))
        return y.cpu().numpy() if kind == "product" else {"n": n, "stored": None, "y": y}
    if kind == "truncate":
        w = np.concatenate([np.linalg.svd(X, compute_uv=False)[:X.shape[0]] for _, X in density_blocks(case, block_vector(case, seed))])
        pairs = len(lllr(case)[0])
        weights = np.zeros(pairs)
        weights[:len(w)] = np.sort(w ** 2)[::-1]
        return {"weights": weights, "label": None, "col": None, "row": None, "val": None}
    if kind == "expect":
        states, dims, *_ = parts(case["model"], case["m"])
        k = case["sites"]
        ops, site = block_operators(case, seed, k)
        x = torch.zeros(int(np.prod(dims)), dtype=torch.float64, device="cuda")
        x[cuda(flat(states, dims))] = cuda(block_vector(case, seed))
        x = x.reshape(dims)
        rho = [torch.movedim(x, p, 0).reshape(dims[p], -1) for p in range(4)]
        rho = [(r @ r.T).cpu().numpy() for r in rho]

        def value(o, p):
            r = np.repeat(np.arange(o.n), np.diff(o.row))
            return float(np.sum(o.val[:o.nnz] * rho[p][r, o.col[:o.nnz]]))

        return np.array([value(o, 0) for o in ops[:k]] + [value(site, 1), value(site, 3)] + [value(o, 2) for o in ops[k:]])
    if kind == "renorm":
        nl, nr, (tc, tr, tv), (row, col, val) = renorm_inputs(case, seed)
        T, O = np.zeros((nl, nr)), np.zeros((nl, nl))
        T[tr, np.repeat(np.arange(nr), np.diff(tc))] = tv
        O[np.repeat(np.arange(nl), np.diff(row)), col] = val
        W = O @ T
        R = T.T @ W
        val, work_val = np.zeros(nr * nr), np.zeros(nl * nr)
        for out, a in ((val, R), (work_val, W.T)):
            a = a[np.abs(a) > 1e-15]
            out[:len(a)] = a
        return {"row": None, "col": None, "val": val, "work_col": None, "work_row": None, "work_val": work_val}
    return None
