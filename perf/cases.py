"""The measured cases: what a user's DMRG program asks of the library, step by step.

Every case starts from two renormalised blocks as a chain at that size has
them (``m`` kept states spread over the quantum-number sectors around the
target, a block Hamiltonian with a chain's low-lying spectrum in a rotated
basis, the operators of the block's last site), enlarged by one site each.
The operators are drawn from the seed with numpy; nothing in them comes from
the library, so two builds of it get the same inputs bit for bit.

Kinds, and what a program does with each:

``hv``     one superblock product on device vectors (the sparse_HxV callback)
``solve``  one ground-state solve (the sp_eigh call of sb_diag), FP64 or mixed
``rdm``    reduced density matrices, truncation and rotation matrices
``batch``  several small superblocks solved together (a parameter scan)
``setup``  a new superblock handed over, then one product (every DMRG step)
``chain``  a whole infinite-system run through the driver
"""
import math

import numpy as np
import torch

import nssdmrg_gb300 as nss

SPIN_HALF, SPIN_ONE, HUBBARD = "spin-1/2", "spin-1", "hubbard"


def listed():
    return [
        # a young chain's product: latency of one call
        {"name": "hv_spin_half_m24", "kind": "hv", "model": SPIN_HALF, "m": 24},
        # the benchmark's superblock size (Hubbard, m = 256: 39 sectors)
        {"name": "hv_hubbard_m256", "kind": "hv", "model": HUBBARD, "m": 256},
        # a turning point of the spin-1 sweeps, where the truncation's
        # degeneracy rule keeps ~880 states
        {"name": "hv_spin_one_m881", "kind": "hv", "model": SPIN_ONE, "m": 881},
        # a small chain's solve, two states wanted
        {"name": "solve_fp64_spin_half_m64", "kind": "solve", "model": SPIN_HALF, "m": 64, "precision": "fp64",
         "neigen": 2},
        # the benchmark's solve in both precisions
        {"name": "solve_fp64_hubbard_m256", "kind": "solve", "model": HUBBARD, "m": 256, "precision": "fp64",
         "neigen": 1},
        {"name": "solve_mixed_hubbard_m256", "kind": "solve", "model": HUBBARD, "m": 256, "precision": "mixed",
         "neigen": 1},
        # an ordinary step of the spin-1 m = 512 sweeps
        {"name": "solve_mixed_spin_one_m512", "kind": "solve", "model": SPIN_ONE, "m": 512, "precision": "mixed",
         "neigen": 1},
        # density matrices and truncation of the benchmark's step, and of a
        # spin-1 step (blocks beyond one SM's shared memory)
        {"name": "rdm_hubbard_m256", "kind": "rdm", "model": HUBBARD, "m": 256},
        {"name": "rdm_spin_one_m400", "kind": "rdm", "model": SPIN_ONE, "m": 400},
        # a scan over small chains, solved as one batch
        {"name": "batch_16", "kind": "batch", "model": HUBBARD, "m": 96, "count": 16},
        # what every step pays before its solve
        {"name": "setup_hubbard_m250", "kind": "setup", "model": HUBBARD, "m": 250},
        # a whole small run: blocks, products, solves, density matrices
        {"name": "chain_spin_half_L20_m40", "kind": "chain", "model": SPIN_HALF, "m": 40, "ldmrg": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hv", "hv", "solve", "solve", "solve", "rdm", "batch", "setup", "chain"])
    model = rng.choice([SPIN_HALF, SPIN_ONE, HUBBARD])
    if kind == "hv":
        return {"kind": kind, "model": model, "m": _log(rng, 8, {SPIN_HALF: 900, SPIN_ONE: 850, HUBBARD: 400}[model])}
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed"])
        top = {SPIN_HALF: 400, SPIN_ONE: 400, HUBBARD: 256}[model] if precision == "mixed" else 200
        return {"kind": kind, "model": model, "m": _log(rng, 12, top), "precision": precision,
                "neigen": rng.choice([1, 2]) if precision == "fp64" else 1}
    if kind == "rdm":
        return {"kind": kind, "model": model, "m": _log(rng, 16, {SPIN_HALF: 256, SPIN_ONE: 350, HUBBARD: 256}[model])}
    if kind == "batch":
        return {"kind": kind, "model": model, "m": _log(rng, 16, {SPIN_HALF: 128, SPIN_ONE: 96, HUBBARD: 96}[model]),
                "count": _log(rng, 2, 16)}
    if kind == "setup":
        return {"kind": kind, "model": model, "m": _log(rng, 16, 240)}
    return {"kind": kind, "model": SPIN_HALF, "m": _log(rng, 10, 40), "ldmrg": rng.randint(5, 10)}


# ---------------------------------------------------------------------------
# Blocks


class _Csr:
    """A CSR matrix with the attributes the library's Python view reads."""

    def __init__(self, dense):
        r, c = np.nonzero(dense)
        self.shape = dense.shape
        self.indices = c.astype(np.int32)
        self.data = dense[r, c]
        self.indptr = np.zeros(dense.shape[0] + 1, np.int32)
        np.cumsum(np.bincount(r, minlength=dense.shape[0]), out=self.indptr[1:])

    def tocsr(self):
        return self


def _site(model):
    """(QN per state, H, operators) of one site."""
    if model == HUBBARD:
        qn = np.array([[0, 0], [1, 0], [0, 1], [1, 1]], float)
        up, dw = np.zeros((4, 4)), np.zeros((4, 4))
        up[0, 1] = up[2, 3] = 1.0
        dw[0, 2], dw[1, 3] = 1.0, -1.0
        return qn, np.diag([0.0, -2.0, -2.0, 0.0]), {"C_l1_s1_n": up, "C_l1_s2_n": dw,
                                                    "P_n": np.diag([1.0, -1.0, -1.0, 1.0])}
    if model == SPIN_ONE:
        s = math.sqrt(2.0)
        sp = np.array([[0, s, 0], [0, 0, s], [0, 0, 0]])
        return np.array([[1.0], [0.0], [-1.0]]), np.zeros((3, 3)), {"S_z_n": np.diag([1.0, 0.0, -1.0]), "S_p_n": sp}
    sp = np.array([[0.0, 1.0], [0.0, 0.0]])
    return np.array([[0.5], [-0.5]]), np.zeros((2, 2)), {"S_z_n": np.diag([0.5, -0.5]), "S_p_n": sp}


def _sector_sizes(model, m):
    """{QN: kept states}, m states in all, spread as a chain's block has them."""
    if model == HUBBARD:
        qs, var = [(a, b) for a in range(-4, 5) for b in range(-4, 5)], 1.0
    else:
        qs, var = [(a,) for a in range(-7, 8)], 2.1 if model == SPIN_ONE else 1.1
    rng = np.random.default_rng([17, m])                # uneven, and the same for every seed
    w = np.array([math.exp(-sum(x * x for x in q) / (2.0 * var)) for q in qs])
    want = m * w / w.sum() + rng.uniform(-0.3, 0.3, len(qs)) * np.sqrt(m * w / w.sum())
    size = np.maximum(0, np.floor(want)).astype(int)
    for k in np.argsort(size - want, kind="stable")[: max(0, m - int(size.sum()))]:
        size[k] += 1
    size[int(np.argmax(w))] += m - int(size.sum())     # exact total
    return {q: int(n) for q, n in zip(qs, size) if n > 0}


def _block(model, m, rng):
    """A renormalised block of m states: QN per state, H, last-site operators."""
    size = _sector_sizes(model, m)
    qn = np.array([q for q, n in size.items() for _ in range(n)], float)
    dim = len(qn)
    mix = rng.permutation(dim)                          # kept states come ordered by weight, not by sector
    qn = qn[mix]
    at = {q: np.nonzero((qn == q).all(1))[0] for q in size}
    mirror = {q: [v / np.linalg.norm(v) for v in rng.standard_normal((2, n))] for q, n in size.items()}

    def rotated(x, p, q):
        """x, given between the energy states of sectors p and q, in the kept basis."""
        for v in mirror[p]:
            x = x - 2.0 * np.outer(v, v @ x)
        for v in mirror[q]:
            x = x - 2.0 * np.outer(x @ v, v)
        return x

    h = np.zeros((dim, dim))
    for q, n in size.items():
        e = 0.3 * sum(x * x for x in q) - 3.0 + 8.0 * (np.arange(n) / max(n, 8)) ** 0.6
        x = rotated(np.diag(e), q, q)
        h[np.ix_(at[q], at[q])] = 0.5 * (x + x.T)
    ops = {}

    def move(step, scale):
        o = np.zeros((dim, dim))
        for q, n in size.items():
            p = tuple(a + b for a, b in zip(q, step))
            if p in at:
                x = np.eye(size[p], n) + rng.standard_normal((size[p], n)) / (2.0 * math.sqrt(max(size[p], n)))
                o[np.ix_(at[p], at[q])] = scale * rotated(x, p, q)
        return o

    if model == HUBBARD:
        ops["C_l1_s1_n"] = move((-1, 0), 0.6)
        ops["C_l1_s2_n"] = move((0, -1), 0.6)
        p = np.zeros((dim, dim))
        for q in size:                                  # U^T P U: signs, and rounding beside them
            n = len(at[q])
            dust = rng.standard_normal((n, n)) * 1e-17 * (rng.random((n, n)) < 0.9)
            p[np.ix_(at[q], at[q])] = (-1.0) ** (sum(q) % 2) * np.eye(n) + np.triu(dust, 1) + np.triu(dust, 1).T
        ops["P_n"] = p
    else:
        s = 1.0 if model == SPIN_ONE else 0.5
        z = move((0,), 0.4 * s)
        ops["S_z_n"] = 0.5 * (z + z.T)
        ops["S_p_n"] = move((1,), 0.6 * s)
    return qn, h, ops


def _coupling(model):
    return np.array([[-1.0, 0.0], [0.0, -1.0]]) if model == HUBBARD else np.array([[1.0, 0.0], [0.0, 0.5]])


def _enlarged(model, m, rng, right):
    """Dense H and operators of the block with one more site, and its QNs."""
    qn, h, ops = _block(model, m, rng)
    sq, sh, sops = _site(model)
    d, dim, j = len(sq), len(qn), _coupling(model)

    def kron(a, b):                                     # block (x) site, or site (x) block
        return np.kron(b, a) if right else np.kron(a, b)

    ib, isite = np.eye(dim), np.eye(d)
    big = kron(h, isite) + kron(ib, sh)
    new = {}
    if model == HUBBARD:
        for c, t in (("C_l1_s1_n", j[0, 0]), ("C_l1_s2_n", j[1, 1])):
            first, second = (sops, ops) if right else (ops, sops)
            a = t * first[c].T @ first["P_n"]
            x = kron(second[c], a) if right else kron(a, second[c])
            big += x + x.T
            new[c] = kron(ib, sops[c]) if right else kron(ops["P_n"], sops[c])
        new["P_n"] = kron(ops["P_n"], sops["P_n"])
    else:
        x = 2.0 * 0.5 * kron(ops["S_p_n"], sops["S_p_n"].T) * j[1, 1]
        big += j[0, 0] * kron(ops["S_z_n"], sops["S_z_n"]) + x + x.T
        for key in ("S_z_n", "S_p_n"):
            new[key] = kron(ib, sops[key])
    big = 0.5 * (big + big.T)
    basis = (sq[:, None, :] + qn[None, :, :] if right else qn[:, None, :] + sq[None, :, :]).reshape(dim * d, -1)
    return {"basis": basis, "H": big, **new}


def _pair(model, m, seed):
    """Dense left and right enlarged blocks, target QN, couplings."""
    rng = np.random.default_rng([seed, m, len(model)])
    left, right = _enlarged(model, m, rng, False), _enlarged(model, m, rng, True)
    target = np.array([1.0, 1.0]) if model == HUBBARD else np.array([0.0])
    if model != HUBBARD and (left["basis"][0, 0] + right["basis"][0, 0]) % 1.0:
        target = target + 0.5
    return left, right, target, _coupling(model)


def _sectors(left, right, target):
    """[(left states, right states)] in the library's sector order."""
    got, seen = [], set()
    for q in map(tuple, left["basis"]):
        if q in seen:
            continue
        seen.add(q)
        r = np.nonzero((right["basis"] == target - np.array(q)).all(1))[0]
        if len(r):
            got.append((np.nonzero((left["basis"] == np.array(q)).all(1))[0], r))
    return got


def _terms(model, left, right, hij):
    """[(A, B)] with H_LR = sum A (x) B over the whole blocks."""
    if model == HUBBARD:
        got = []
        for k, c in enumerate(("C_l1_s1_n", "C_l1_s2_n")):
            a = hij[k, k] * left[c].T @ left["P_n"]
            got += [(a, right[c]), (a.T, right[c].T)]
        return got
    a = hij[1, 1] * left["S_p_n"]
    return [(hij[0, 0] * left["S_z_n"], right["S_z_n"]), (a, right["S_p_n"].T), (a.T, right["S_p_n"])]


def _hand_over(sb, model, left, right, target, hij):
    kind = nss.NSS_SITE_FERMION if model == HUBBARD else nss.NSS_SITE_SPIN
    sb.setup(kind, left, right, target, hij)


def _sparse(blk):
    return {k: v if k == "basis" else _Csr(v) for k, v in blk.items()}


def _superblock(model, m, seed):
    left, right, target, hij = _pair(model, m, seed)
    sb = nss.Superblock(0)
    _hand_over(sb, model, _sparse(left), _sparse(right), target, hij)
    return sb


def _state_vector(model, m, seed):
    """A normalised state whose sectors have decaying singular values, as a
    ground state's do: 4.5 decades of density-matrix weight in 40 states."""
    left, right, target, _ = _pair(model, m, seed)
    rng = np.random.default_rng([seed, 7, m])
    secs = _sectors(left, right, target)
    spread = np.random.default_rng([23, m])             # weights of the case, in the bases of the seed
    big = max(len(a) for a, _ in secs)
    parts = [None] * len(secs)
    for k in sorted(range(len(secs)), key=lambda k: tuple(left["basis"][secs[k][0][0]])):
        (a, b), n = secs[k], min(len(secs[k][0]), len(secs[k][1]))
        u = np.linalg.qr(rng.standard_normal((len(a), n)))[0]
        v = np.linalg.qr(rng.standard_normal((len(b), n)))[0]
        s = n / big * np.exp(-0.13 * np.arange(n) - 0.05 * spread.random(n))
        parts[k] = ((u * s) @ v.T).reshape(-1)
    psi = np.concatenate(parts)
    return psi / np.linalg.norm(psi), secs


def _kept(case):
    return max(4, (2 * case["m"]) // 5)


# ---------------------------------------------------------------------------
# The interface


def prepare(case, seed):
    kind, model, m = case["kind"], case["model"], case["m"]
    state = {"case": case}
    if kind == "hv":
        sb = _superblock(model, m, seed)
        v = np.random.default_rng([seed, 3]).standard_normal(sb.n)
        state["v"] = torch.from_numpy(v / np.linalg.norm(v)).cuda()
        state["hv"] = torch.empty_like(state["v"])
        state["sb"] = sb
        torch.cuda.synchronize()
    elif kind == "solve":
        state["sb"] = _superblock(model, m, seed)
    elif kind == "rdm":
        state["sb"] = _superblock(model, m, seed)
        state["psi"] = _state_vector(model, m, seed)[0]
    elif kind == "batch":
        state["sbs"] = [_superblock(model, _scan_m(m, k), seed + 1000 * k) for k in range(case["count"])]
    elif kind == "setup":
        left, right, target, hij = _pair(model, m, seed)
        state["blocks"] = (_sparse(left), _sparse(right), target, hij)
        state["sb"] = nss.Superblock(0)
        n = sum(len(a) * len(b) for a, b in _sectors(left, right, target))
        v = np.random.default_rng([seed, 3]).standard_normal(n)
        state["v"] = v / np.linalg.norm(v)
    else:
        state["sb"] = nss.Superblock(0)
        state["seed"] = 1000 + seed
    return state


def _scan_m(m, k):
    """The k-th chain of a scan keeps between half of m and m states."""
    return max(8, m - (5 * k) % max(1, m // 2))


def run(state):
    case = state["case"]
    kind, sb = case["kind"], state.get("sb")
    if kind == "hv":
        sb.hv_device(state["v"].data_ptr(), state["hv"].data_ptr())
        return state["hv"]
    if kind == "solve":
        mixed = case["precision"] == "mixed"
        # two wanted states: their energies (the vectors stay on the device)
        ev, vec, _ = sb.sb_diag(neigen=case["neigen"], precision=nss.NSS_PREC_MIXED if mixed else nss.NSS_PREC_FP64,
                                want_vectors=case["neigen"] == 1)
        return {"ev": ev} if vec is None else {"ev": ev, "vec": vec}
    if kind == "rdm":
        r = sb.sb_get_rdm(_kept(case), psi=state["psi"])
        return {"m_s": list(r.m_s), "trunc_err": np.array(r.trunc_err), "entropy": np.array(r.entropy),
                "lam_l": r.lambdas[0], "lam_r": r.lambdas[1], "kept_l": r.kept_blocks[0], "kept_r": r.kept_blocks[1],
                "u_l": r.u[0], "u_r": r.u[1]}
    if kind == "batch":
        return {"ev": nss.eigh_batch(state["sbs"])[0]}
    if kind == "setup":
        left, right, target, hij = state["blocks"]
        _hand_over(sb, case["model"], left, right, target, hij)
        return sb.spmatvec(state["v"])
    d = nss.DMRG(nss.MODEL_HEISENBERG_HALF, case["ldmrg"], case["m"], sb=sb, seed=state["seed"])
    rec = d.infinite()
    d.close()
    return {"energy": np.array([r["energy"][0] for r in rec]), "entropy": np.array([r["entropy_left"] for r in rec]),
            "trunc": np.array([r["trunc_left"] for r in rec]), "n": [r["n"] for r in rec]}


def work(case):
    """Operators, vectors and results once; the products' multiply-adds. A
    solve's or run's count takes the ~100 products that its Lanczos needs."""
    kind, model, m = case["kind"], case["model"], case["m"]
    if kind == "chain":
        steps, big = case["ldmrg"] - 1, {"kind": "solve", "model": model, "m": m, "precision": "fp64", "neigen": 1}
        w = work(big)
        return {"bytes": steps * w["bytes"], "flops": steps * w["flops"]}
    if kind == "batch":
        ws = [work({"kind": "solve", "model": model, "m": _scan_m(m, k), "precision": "mixed", "neigen": 1})
              for k in range(case["count"])]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    size = _sector_sizes(model, m)
    sq = [tuple(q) for q in _site(model)[0]]
    dims = {}
    for q, n in size.items():
        for s in sq:
            k = tuple(a + b for a, b in zip(q, s))
            dims[k] = dims.get(k, 0) + n
    target = (1.0, 1.0) if model == HUBBARD else (0.0,)
    pairs = [(n, dims.get(tuple(t - a for t, a in zip(target, q)), 0)) for q, n in dims.items()]
    pairs = [(a, b) for a, b in pairs if b]
    n = sum(a * b for a, b in pairs)
    ops = sum(a * a + b * b for a, b in pairs)
    dense = sum(2.0 * a * b * (a + b) for a, b in pairs)
    terms = (4 if model == HUBBARD else 3) * 2.0 * 2.0 * n
    if kind == "rdm":
        return {"bytes": 8.0 * (n + sum(dims.values()) * 2 * _kept(case)),
                "flops": dense + sum((4 / 3 + 4 * 0.4) * (a ** 3 + b ** 3) for a, b in pairs)}
    if kind == "solve":
        return {"bytes": 8.0 * (ops + n * (1 + case["neigen"])), "flops": 100 * (dense + terms)}
    return {"bytes": 8.0 * (ops + 2 * n), "flops": dense + terms}


def _product(secs, hl, hr, cross, x):
    """H x, sector by sector, in 64 bits."""
    w, at = [], 0
    for a, b in secs:
        w.append(x[at:at + len(a) * len(b)].reshape(len(a), len(b)))
        at += len(a) * len(b)
    out = [hl[k] @ w[k] + w[k] @ hr[k].T for k in range(len(secs))]
    for k, q, a, b in cross:
        out[k] += a @ w[q] @ b.T
    return torch.cat([o.reshape(-1) for o in out])


def _operators(model, m, seed):
    left, right, target, hij = _pair(model, m, seed)
    secs = _sectors(left, right, target)

    def part(o, i, j):
        return torch.from_numpy(np.ascontiguousarray(o[np.ix_(i, j)])).cuda()

    hl = [part(left["H"], a, a) for a, _ in secs]
    hr = [part(right["H"], b, b) for _, b in secs]
    cross = []
    for ta, tb in _terms(model, left, right, hij):
        for k, (a, b) in enumerate(secs):
            for q, (c, e) in enumerate(secs):
                x, y = ta[np.ix_(a, c)], tb[np.ix_(b, e)]
                if np.abs(x).max() > 1e-12 and np.abs(y).max() > 1e-12:
                    cross.append((k, q, part(ta, a, c), part(tb, b, e)))
    return secs, hl, hr, cross


def _lowest(model, m, seed, count):
    """Lowest eigenvalues by Lanczos with twofold full orthogonalisation in 64 bits."""
    secs, hl, hr, cross = _operators(model, m, seed)
    n = sum(len(a) * len(b) for a, b in secs)
    most = min(n, 320)
    basis = torch.zeros((most, n), dtype=torch.float64, device="cuda")
    v = torch.from_numpy(np.random.default_rng([seed, 5]).standard_normal(n)).cuda()
    basis[0] = v / v.norm()
    alpha, beta = [], []
    for j in range(most):
        w = _product(secs, hl, hr, cross, basis[j])
        alpha.append(float(basis[j] @ w))
        for _ in range(2):
            w = w - basis[: j + 1].T @ (basis[: j + 1] @ w)
        beta.append(float(w.norm()))
        if j + 1 == most or beta[-1] < 1e-13:
            break
        basis[j + 1] = w / beta[-1]
        if j % 8 == 7:
            ev, s = np.linalg.eigh(np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1))
            if np.abs(beta[-1] * s[-1, :count]).max() < 1e-13 * abs(ev[0]):
                break
    return np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta[:len(alpha) - 1], 1) + np.diag(beta[:len(alpha) - 1], -1))[:count]


def exact(case, seed):
    kind, model, m = case["kind"], case["model"], case["m"]
    if kind in ("hv", "setup"):
        secs, hl, hr, cross = _operators(model, m, seed)
        n = sum(len(a) * len(b) for a, b in secs)
        v = np.random.default_rng([seed, 3]).standard_normal(n)
        return _product(secs, hl, hr, cross, torch.from_numpy(v / np.linalg.norm(v)).cuda())
    if kind == "rdm":
        psi, secs = _state_vector(model, m, seed)
        lam, at = [], 0
        for a, b in secs:
            w = psi[at:at + len(a) * len(b)].reshape(len(a), len(b))
            at += w.size
            s2 = np.linalg.svd(w, compute_uv=False) ** 2
            lam.append((s2, len(a), len(b)))
        full = [np.sort(np.concatenate([np.pad(s, (0, d[k] - len(s))) for s, *d in lam]))[::-1] for k in (0, 1)]
        some = [x[x > 1e-300] for x in full]
        ent = np.array([-(x * np.log(x)).sum() for x in some])
        return {"m_s": None, "trunc_err": None, "entropy": ent, "lam_l": full[0], "lam_r": full[1],
                "kept_l": None, "kept_r": None, "u_l": None, "u_r": None}
    if kind == "solve":
        ev = _lowest(model, m, seed, case["neigen"])
        return {"ev": ev} if case["neigen"] > 1 else {"ev": ev, "vec": None}
    if kind == "batch":
        return {"ev": np.array([_lowest(model, _scan_m(m, k), seed + 1000 * k, 1)[0] for k in range(case["count"])])}
    return None
