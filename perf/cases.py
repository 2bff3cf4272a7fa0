"""Timing cases of the two-site DMRG hot path, through the Python binding of the C ABI.

Every case is a call that a program using this library makes, on sizes of the
workloads that the repository's benchmark and tests run: H_eff*psi on device
pointers (FP64 and split precision), the Lanczos ground state and the truncating
block SVD on host tensors, one environment update, the many-instance Lanczos
solve, and a whole sweep of a small chain from checkpoint files.

Problems are synthetic with the structure of real ones.  Sector dimensions follow
what a spin-1/2 chain's bond of D states (U(1)) or D multiplets (SU(2)) holds --
``shape`` jitters them, so that they are odd and ragged -- or are log-uniform, as
in the benchmark's ladder.  Operators are Hermitian as the chain's are, two-site
vectors have singular values that fall over several decades, and matrix product
states are random and canonical.  All values come from the seed.

The split-precision cases switch the schedule tuner off: a sweep's H_eff plans
take the same untimed rules, and the results then do not depend on a timing.
"""
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "symmetry-adapted-dmrg-library_b200"))
import sadmrg  # noqa: E402

U1, SU2 = 0, 1
MLANC = 40          # the library's default Lanczos length in a chain


def listed():
    """What each stands for in real use is said beside it."""
    return [
        # ground state of one bond of a small U(1) chain (L = 32, D = 64): some thousand elements,
        # the time is launches and round trips
        {"name": "lanczos_u1_D64", "kind": "lanczos", "sym": U1, "cplx": False, "D": 64, "terms": 1, "shape": 1},
        # the same for the SU(2) chain at D = 512 multiplets, the bond of a production sweep
        {"name": "lanczos_su2_D512", "kind": "lanczos", "sym": SU2, "cplx": False, "D": 512, "terms": 1, "shape": 2},
        # H_eff*psi of the 2 x 32 SU(2) ladder's centre, D = 2048 multiplets in 34 sectors of 8 to 512:
        # the benchmark's matvec, in both precisions
        {"name": "matvec_f64_ladder", "kind": "matvec", "sym": SU2, "cplx": False, "D": 2048, "terms": 2, "shape": 2024,
         "prec": 0, "logdims": True},
        {"name": "matvec_mixed_ladder", "kind": "matvec", "sym": SU2, "cplx": False, "D": 2048, "terms": 2, "shape": 2024,
         "prec": 1, "logdims": True},
        # H_eff*psi of the complex U(1) J1-J2 chain with a DM term: large sectors, four real products each
        {"name": "matvec_f64_u1c_D1024", "kind": "matvec", "sym": U1, "cplx": True, "D": 1024, "terms": 2, "shape": 3,
         "prec": 0, "logdims": False},
        {"name": "matvec_mixed_u1c_D1024", "kind": "matvec", "sym": U1, "cplx": True, "D": 1024, "terms": 2, "shape": 3,
         "prec": 1, "logdims": False},
        # truncation of one bond: SU(2) at D = 512 and at D = 2048 multiplets (most of a sweep's time there),
        # and the complex U(1) chain
        {"name": "svd_su2_D512", "kind": "svd", "sym": SU2, "cplx": False, "D": 512, "shape": 4, "decades": 5.0},
        {"name": "svd_su2_D2048", "kind": "svd", "sym": SU2, "cplx": False, "D": 2048, "shape": 5, "decades": 5.0},
        {"name": "svd_u1c_D384", "kind": "svd", "sym": U1, "cplx": True, "D": 384, "shape": 6, "decades": 5.0},
        # environment update of one site of a U(1) J1-J2 chain, new tensors read back
        {"name": "env_u1_D768", "kind": "env", "cplx": False, "D": 768, "shape": 7, "J2": 0.5},
        # 64 independent U(1) J1-J2 centre problems of D = 32 to 256 solved together
        {"name": "batch_lanczos_64", "kind": "batch", "count": 64, "Dlo": 32, "Dhi": 256, "shape": 8},
        # one whole sweep of a short SU(2) Heisenberg chain from checkpoint files: every part of the
        # library at small sizes (longer chains started at random amplify rounding until their
        # truncations keep other states, in any two runs)
        {"name": "sweep_su2_L24_D96", "kind": "sweep", "sym": SU2, "L": 24, "D": 96, "J2": 0.0, "shape": 9},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["lanczos", "matvec", "matvec", "matvec", "svd", "svd", "env", "batch", "sweep"])
    shape = rng.randrange(1, 1 << 20)
    sym = rng.choice([U1, SU2])
    cplx = rng.random() < 0.4

    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    if kind == "lanczos":
        return {"kind": kind, "sym": sym, "cplx": cplx, "D": logint(32, 512), "terms": rng.choice([1, 2]), "shape": shape}
    if kind == "matvec":
        if rng.random() < 0.3:
            return {"kind": kind, "sym": SU2, "cplx": False, "D": logint(512, 2048), "terms": 2, "shape": shape,
                    "prec": rng.choice([0, 1]), "logdims": True}
        return {"kind": kind, "sym": sym, "cplx": cplx, "D": logint(32, 1024), "terms": rng.choice([1, 2]),
                "shape": shape, "prec": rng.choice([0, 1]), "logdims": False}
    if kind == "svd":
        return {"kind": kind, "sym": sym, "cplx": cplx, "D": logint(24, 384 if cplx else 1024), "shape": shape,
                "decades": round(rng.uniform(4.0, 6.0), 2)}
    if kind == "env":
        return {"kind": kind, "cplx": cplx, "D": logint(32, 768), "shape": shape, "J2": rng.choice([0.0, 0.5])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randrange(8, 65), "Dlo": 32, "Dhi": logint(64, 256), "shape": shape}
    return {"kind": kind, "sym": sym, "L": 2 * rng.randrange(6, 13 if sym == SU2 else 9),
            "D": logint(32, 128 if sym == SU2 else 64), "J2": rng.choice([0.0, 0.3]), "shape": shape}


# ---------------------------------------------------------------------------
# sector structure
def bond_dims(sym, D, odd, shape):
    """{label: dimension} of a bond of about D states or multiplets: Gaussian weights in
    the charge; an SU(2) multiplet count is the difference of neighbouring charges'."""
    r = random.Random(f"{shape}-{int(odd)}")
    top = 2 * int(math.log2(D) + 1) + int(odd)

    def m(q):
        return math.exp(-q * q / 18.0)

    if sym == U1:
        lab = range(-top, top + 1, 2)
        w = {q: m(q) for q in lab}
    else:
        lab = range(int(odd), top + 1, 2)
        w = {q: m(q) - m(q + 2) for q in lab}
    tot = sum(w.values())
    d = {q: int(round(D * w[q] / tot * r.uniform(0.9, 1.1))) for q in lab}
    return {q: n for q, n in d.items() if n > 0}


def fused(sym, d):
    """A bond of dims d fused with a spin-1/2 site."""
    out = {}
    for q, n in d.items():
        for t in (q - 1, q + 1):
            if sym == U1 or t >= 0:
                out[t] = out.get(t, 0) + n
    return dict(sorted(out.items()))


def legs(case):
    """(left, right) fused legs of the two-site problem of a case: label -> dimension."""
    sym, D, shape = case["sym"], case["D"], case["shape"]
    if case.get("logdims"):
        lo, hi = 8, 512
        n = max(3, int(round(2 * D * math.log(hi / lo) / (hi - lo))))
        out = []
        for side in "lr":
            r = random.Random(f"{shape}{side}")
            out.append({2 * i: int(round(math.exp(r.uniform(math.log(lo), math.log(hi))))) for i in range(n)})
        return out
    a = fused(sym, bond_dims(sym, D, False, shape))
    b = fused(sym, bond_dims(sym, D, False, shape + 1))
    common = sorted(set(a) & set(b))
    return {q: a[q] for q in common}, {q: b[q] for q in common}


def channels(sym):
    return [-2, 0, 2] if sym == U1 else [2]


def op_pairs(sym, d):
    """(a, channel, a') labels of a spin operator's blocks on a leg of dims d."""
    if sym == U1:
        return [(a, c, a + c) for a in d for c in (-2, 0, 2) if a + c in d]
    return [(a, 2, b) for a in d for b in d if abs(a - b) <= 2 and a + b >= 2]


def factor(sym, a, c, a2):
    """SU(2) weight of one term of H_eff*psi: the fully contracted Clebsch-Gordan network
    of (a, c, a') with its three singlets, times sqrt(2c + 1)."""
    return math.sqrt((a2 + 1) / (a + 1)) if sym == SU2 else 1.0


def matvec_work(sym, cplx, dl, dr, terms):
    fl = 0
    el = sum(dl[q] * dr[q] for q in dl)
    n = el
    for q in dl:
        fl += 2 * dl[q] * dr[q] * (dl[q] + dr[q])
        el += dl[q] ** 2 + dr[q] ** 2
    for a, _, a2 in op_pairs(sym, dl):
        fl += terms * (2 * dl[a2] * dr[a] * dl[a] + 2 * dl[a2] * dr[a2] * dr[a])
        el += terms * (dl[a] * dl[a2] + dr[a] * dr[a2])
    k, s = (4, 16) if cplx else (1, 8)
    return fl * k, (el + n) * s, n


def work(case):
    k = case["kind"]
    if k == "matvec":
        fl, by, _ = matvec_work(case["sym"], case["cplx"], *legs(case), case["terms"])
        return {"bytes": by, "flops": fl}
    if k == "lanczos":
        fl, by, n = matvec_work(case["sym"], case["cplx"], *legs(case), case["terms"])
        c = 4 if case["cplx"] else 1
        return {"bytes": by, "flops": MLANC * (fl + c * 4 * n * (MLANC / 2 + 3))}
    if k == "svd":
        fl = by = 0
        c, s = (4, 16) if case["cplx"] else (1, 8)
        dl, dr = legs(case)
        for q in dl:
            a, b = max(dl[q], dr[q]), min(dl[q], dr[q])
            fl += c * (6 * a * b * b + 20 * b ** 3)
            by += s * (a * b + (a + b) * b // 2)
        return {"bytes": by, "flops": fl}
    if k == "env":
        t = env_dims(case)
        c, s = (4, 16) if case["cplx"] else (1, 8)
        fl = by = 0
        dr, dl = t["r"], t["l"]
        nop = 2 if case["J2"] else 1
        for p, r, l in t["u"]:
            by += s * dr[r] * dl[l]
            fl += c * 2 * dl[l] * dr[r] * (dr[r] + dl[l])                     # U^T hh U
            for q in (r - 2, r, r + 2):
                if q in dr:
                    fl += c * 2 * dl[l] * dr[r] * dr[q] * nop                   # U^T op
        for r in dr:
            by += s * (dr[r] ** 2 + nop * sum(dr[r] * dr.get(r + x, 0) for x in (-2, 0, 2)))
        for q in dl:
            by += s * (dl[q] ** 2 + nop * sum(dl[q] * dl.get(q + x, 0) for x in (-2, 0, 2)))
        return {"bytes": by, "flops": fl}
    if k == "batch":
        fl = by = 0
        for c in instances(case):
            w = work(c)
            fl += w["flops"]
            by += w["bytes"]
        return {"bytes": by, "flops": fl}
    # a sweep: at each of its 2 L - 9 two-site steps at least two check points (8 matvecs) and one SVD
    c = {"sym": case["sym"], "cplx": False, "D": case["D"], "terms": 1, "shape": case["shape"]}
    fl = (2 * case["L"] - 9) * (8 * matvec_work(c["sym"], False, *legs(c), 1)[0] + work(dict(c, kind="svd"))["flops"])
    return {"bytes": 8 * 2 * case["L"] * case["D"] * case["D"] // 4, "flops": fl}


# ---------------------------------------------------------------------------
# tensors
def gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def randn(g, shape, cplx):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.complex128 if cplx else torch.float64)


def btensor(dirs, bonds, blocks, cplx):
    """BlockTensorData of {labels: column-major block}; bonds: label -> dimension per leg."""
    qs = [list(b) for b in bonds]
    ds = [list(b.values()) for b in bonds]
    pos = [{q: i for i, q in enumerate(x)} for x in qs]

    def index(lab):
        i = 0
        for b in range(len(qs) - 1, -1, -1):
            i = i * len(qs[b]) + pos[b][lab[b]]
        return i

    order = sorted(blocks, key=index)
    if order:
        data = torch.cat([blocks[k].permute(*range(blocks[k].dim() - 1, -1, -1)).reshape(-1) for k in order])
        data = data.cpu().numpy()
    else:
        data = np.zeros(0, np.complex128 if cplx else np.float64)
    return sadmrg.BlockTensorData(list(dirs), qs, ds, 0, np.array([index(k) for k in order], np.int64), data)


def hermitian(g, d, cplx):
    out = {}
    for q, n in d.items():
        a = randn(g, (n, n), cplx)
        out[(q, q)] = (a + a.conj().T) / math.sqrt(8 * n)
    return out


def spin_operator(g, sym, d, cplx):
    """Blocks (a, 1, a') of a spin operator; the block of (a', a) is the adjoint of (a, a')'s
    (times the ratio of multiplet sizes for SU(2)), so that H_eff is Hermitian."""
    out = {}
    for a, c, a2 in op_pairs(sym, d):
        if a2 < a:
            continue
        m = randn(g, (d[a], d[a2]), cplx) / math.sqrt(4 * max(d[a], d[a2]))
        if a == a2:
            m = (m + m.conj().T) / 2
        out[(a, c, a2)] = m[:, None, :]
        if a != a2:
            back = m.conj().T * math.sqrt((a2 + 1) / (a + 1)) if sym == SU2 else m.conj().T
            out[(a2, -c if sym == U1 else c, a)] = back[:, None, :]
    return out


def problem(case, seed):
    """The two-site problem: psi and the operators as {labels: block} on the device."""
    g = gen(seed)
    sym, cplx = case["sym"], case["cplx"]
    dl, dr = legs(case)
    psi = {(q, q): randn(g, (dl[q], dr[q]), cplx) for q in dl}
    norm = math.sqrt(sum(float((b.abs() ** 2).sum()) for b in psi.values()))
    psi = {k: b / norm for k, b in psi.items()}
    hl, hr = hermitian(g, dl, cplx), hermitian(g, dr, cplx)
    ops = [(spin_operator(g, sym, dl, cplx), spin_operator(g, sym, dr, cplx)) for _ in range(case["terms"])]
    return dl, dr, psi, hl, hr, ops


def plan(h, case, parts):
    """heff_plan of a problem; returns psi as the host vector the library uses."""
    dl, dr, psi, hl, hr, ops = parts
    sym, cplx = case["sym"], case["cplx"]
    ch = {c: 1 for c in channels(sym)}
    sr = -1 if sym == U1 else 1      # direction of psi's right leg
    p = btensor([1, sr], [dl, dr], psi, cplx)
    tens = []
    for left, right in ops:
        tens.append(btensor([-1, -1, 1], [dl, ch, dl], left, cplx))
        tens.append(btensor([-sr, -sr, sr], [dr, ch, dr], right, cplx))
    h.heff_plan(p, btensor([-1, 1], [dl, dl], hl, cplx), btensor([-sr, sr], [dr, dr], hr, cplx), tens,
                [(2 * i, 2 * i + 1) for i in range(len(ops))])
    return p.data


def apply_plain(case, parts, psi):
    """H_eff*psi by plain matrix products on {labels: block}."""
    _, _, _, hl, hr, ops = parts
    out = {k: hl[k].T @ b + b @ hr[k] for k, b in psi.items()}
    for left, right in ops:
        for (a, c, a2), m in left.items():
            out[(a2, a2)] = out[(a2, a2)] + factor(case["sym"], a, c, a2) * (m[:, 0, :].T @ psi[(a, a)] @ right[(a, c, a2)][:, 0, :])
    return out


def flat(blocks):
    return torch.cat([blocks[k].T.reshape(-1) for k in blocks])


def unflat(vec, like):
    out, o = {}, 0
    for k, b in like.items():
        out[k] = vec[o:o + b.numel()].reshape(b.shape[1], b.shape[0]).T
        o += b.numel()
    return out


def lanczos_plain(case, parts, steps):
    """Lowest Ritz value of at most `steps` Lanczos steps with full reorthogonalisation, stopped
    like the library's solver: at every fourth step, once |<v|Hv>|/|Hv| is within 1e-8 of 1."""
    psi = parts[2]

    def mv(v):
        return flat(apply_plain(case, parts, unflat(v, psi)))

    v = flat(psi)
    basis = [v / v.norm()]
    al, be = [], []
    for m in range(steps):
        w = mv(basis[-1])
        al.append(float(torch.vdot(basis[-1], w).real))
        if m == steps - 1:
            break
        V = torch.stack(basis)
        for _ in range(2):
            w = w - (V.conj() @ w) @ V
        be.append(float(w.norm()))
        if (m + 1) % 4 == 0 and m < steps - 1:
            e, z = np.linalg.eigh(np.diag(al) + np.diag(be[:m], 1) + np.diag(be[:m], -1))
            y = torch.from_numpy(z[:, 0].copy()).to(V) @ V
            hy = mv(y)
            if abs(float(abs(torch.vdot(y, hy))) / float(y.norm()) / float(hy.norm()) - 1.0) < 1e-8:
                return float(e[0])
        basis.append(w / w.norm())
    return float(np.linalg.eigvalsh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))[0])


def instances(case):
    """The two-site problems of a batch: D log-uniform in [Dlo, Dhi]."""
    r = random.Random(case["shape"])
    return [{"kind": "lanczos", "sym": U1, "cplx": False, "terms": 2, "shape": r.randrange(1 << 20),
             "D": int(round(math.exp(r.uniform(math.log(case["Dlo"]), math.log(case["Dhi"])))))}
            for _ in range(case["count"])]


def two_site_vector(case, seed):
    """psi with singular values falling over case["decades"] decades in every sector, generic
    left and right vectors; its singular values per sector are returned beside it."""
    g = gen(seed)
    cplx = case["cplx"]
    dl, dr = legs(case)
    psi, sv = {}, {}
    for q in dl:
        m, n = dl[q], dr[q]
        k = min(m, n)
        u = torch.linalg.qr(randn(g, (m, k), cplx))[0]
        v = torch.linalg.qr(randn(g, (n, k), cplx))[0]
        r = random.Random(f"{case['shape']}s{q}")   # the seed moves the vectors, not what is kept
        e = torch.tensor([-case["decades"] * (i + r.uniform(0.0, 0.4)) / k - 0.15 * abs(q) for i in range(k)], dtype=torch.float64)
        s = 10.0 ** e.to("cuda")
        psi[(q, q)] = (u * s) @ v.conj().T
        sv[q] = s
    norm = math.sqrt(sum(float((s ** 2).sum()) for s in sv.values()))
    return {k: b / norm for k, b in psi.items()}, {q: s / norm for q, s in sv.items()}


def site_bonds(case):
    """Outer bonds (dims) of the two site tensors whose fused legs legs(case) gives."""
    sym, D, shape = case["sym"], case["D"], case["shape"]
    return bond_dims(sym, D, False, shape), bond_dims(sym, D, False, shape + 1)


# ---------------------------------------------------------------------------
# environment update of one site from the right (U(1))
def env_dims(case):
    r = bond_dims(U1, case["D"], False, case["shape"])
    l = bond_dims(U1, case["D"], True, case["shape"] + 1)
    u = [(p, x, x - p) for p in (-1, 1) for x in r if x - p in l]
    l = {q: n for q, n in l.items() if any(t[2] == q for t in u)}
    return {"r": r, "l": l, "u": u}


def env_tensors(case, seed):
    g = gen(seed)
    t = env_dims(case)
    cplx = case["cplx"]
    uu = {}
    for q, n in t["l"].items():
        rows = [x for x in t["u"] if x[2] == q]
        m = sum(t["r"][x[1]] for x in rows)
        w = randn(g, (m, n), cplx)
        w = torch.linalg.qr(w)[0] if n <= m else w / math.sqrt(n)
        o = 0
        for p, r, l in rows:
            uu[(p, r, l)] = w[o:o + t["r"][r]].reshape(1, t["r"][r], n)
            o += t["r"][r]
    hh = hermitian(g, t["r"], cplx)
    ops = [spin_operator(g, U1, t["r"], cplx) for _ in range(2 if case["J2"] else 1)]
    return t, uu, hh, ops


def env_plain(case, t, uu, hh, ops):
    """(hh, opr of the site, opr carried over or None) after the update, as {labels: block}."""
    def spin(p, p2):          # element of the site's spin operator in the channel that p -> p2 fixes
        return p / 2.0 if p == p2 else 1.0 / math.sqrt(2.0)

    summed = {k: ops[0][k] + (case["J2"] * ops[1][k] if len(ops) > 1 else 0.0) for k in ops[0]}
    h2 = {}
    o1, o2 = {}, {}
    for (p, r, l), u in uu.items():
        u = u[0]
        for (p2, r2, l2), v in uu.items():
            v = v[0].conj()
            if p == p2 and r == r2:
                h2[(l, l2)] = h2.get((l, l2), 0) + u.T @ hh[(r, r)] @ v
            if r2 - r == p2 - p and (r, r2 - r, r2) in summed:
                h2[(l, l2)] = h2.get((l, l2), 0) + spin(p, p2) * (u.T @ summed[(r, r2 - r, r2)][:, 0, :] @ v)
            if r == r2:
                k = (l, p - p2, l2)
                o1[k] = o1.get(k, 0) + spin(p, p2) * (u.T @ v)[:, None, :]
            if len(ops) > 1 and p == p2 and (r, r2 - r, r2) in ops[0]:
                k = (l, r2 - r, l2)
                o2[k] = o2.get(k, 0) + (u.T @ ops[0][(r, r2 - r, r2)][:, 0, :] @ v)[:, None, :]
    return h2, o1, (o2 if len(ops) > 1 else None)


# ---------------------------------------------------------------------------
# random canonical matrix product state as checkpoint files
def write_mps(case, seed, directory):
    sym, L, D = case["sym"], case["L"], case["D"]
    rng = np.random.default_rng([int(seed), 41])
    site = {-1: 1, 1: 1} if sym == U1 else {1: 1}

    def spin_sum(a, b):
        return [a + b] if sym == U1 else range(abs(a - b), a + b + 1, 2)

    def grow(first):
        """Bond dims outward from an edge and the isometries between them: to[label][(x, y)] rows."""
        bonds, iso = [first], []
        for i in range(1, L // 2):
            prev, rows = bonds[-1], {}
            for q in prev:
                for p in site:
                    for t in spin_sum(q, p):
                        rows.setdefault(t, []).append((q, p))
            want = bond_dims(sym, D, (i + 1) % 2 == 1, case["shape"])
            new = {}
            for t in sorted(rows):
                n = min(sum(prev[q] for q, _ in rows[t]), want.get(abs(t), 0))   # the same for t and -t
                if n > 0:
                    new[t] = n
            bonds.append(new)
            iso.append({t: rows[t] for t in new})
        return bonds, iso

    first = {-1: 1, 1: 1} if sym == U1 else {1: 1}
    bonds, iso = grow(first)
    half = L // 2

    def isometry(i, order, weights=None):
        """Blocks {(q, p, t): matrix} of the tensor between bonds i-1 and i; order: sort key of its rows."""
        out = {}
        prev, new = bonds[i - 1], bonds[i]
        for t, n in new.items():
            rows = sorted(iso[i - 1][t], key=order)
            m = np.linalg.qr(rng.standard_normal((sum(prev[q] for q, _ in rows), n)))[0]
            if weights is not None:
                m = m * weights[t]
            o = 0
            for q, p in rows:
                out[(q, p, t)] = m[o:o + prev[q]]
                o += prev[q]
        return out

    sv = {}
    for t, n in bonds[half - 1].items():
        sv[t] = np.exp(-8.0 * (np.arange(n) + rng.uniform(0, 0.5, n)) / n - 0.4 * abs(t))
    norm = math.sqrt(sum(float((s ** 2).sum()) for s in sv.values()))
    sv = {t: s / norm for t, s in sv.items()}

    def write(i, dirs, labs, blocks):
        base = os.path.join(directory, f"uu-{L}-{D}-0-0-{i}")
        with open(base + ".dat", "w") as f:
            f.write("3\t0\n")
            for dr, b in zip(dirs, labs):
                f.write(f"{dr}\t{len(b)}\n" + "\t".join(map(str, b)) + "\n" + "\t".join(map(str, b.values())) + "\n")
        qs = [list(b) for b in labs]
        order = sorted(blocks, key=lambda k: [qs[b].index(k[b]) for b in (2, 1, 0)])
        np.concatenate([blocks[k].reshape(-1, order="F") for k in order]).tofile(base + ".bin")

    def every(a, b, c, allowed, blocks, d):
        """All allowed blocks of a tensor, absent ones zero."""
        full = {}
        for x in a:
            for y in b:
                for z in c:
                    if allowed(x, y, z):
                        full[(x, y, z)] = blocks.get((x, y, z), np.zeros(d(x, y, z)))
        return full

    vac = {0: 1}
    neg = (lambda b: {-q: n for q, n in sorted(b.items(), reverse=True)}) if sym == U1 else (lambda b: dict(b))
    tri = (lambda x, y, z: abs(x - y) <= z <= x + y and (x + y + z) % 2 == 0)
    # the edge sites: identity embeddings
    one = np.ones((1, 1, 1))
    write(0, [1, 1, -1], [vac, site, first], {(0, p, p): one for p in site})
    if sym == U1:
        write(L - 1, [1, -1, 1], [site, vac, first], {(p, 0, -p): one for p in site})
    else:
        write(L - 1, [1, 1, -1], [site, vac, first], {(p, 0, p): one for p in site})
    for i in range(1, half):
        w = isometry(i, lambda t: (t[1], t[0]), sv if i == half - 1 else None)
        blk = {(q, p, t): m.reshape(m.shape[0], 1, m.shape[1]) for (q, p, t), m in w.items()}
        a, c = bonds[i - 1], bonds[i]
        ok = (lambda x, y, z: x + y == z) if sym == U1 else tri
        write(i, [1, 1, -1], [a, site, c], every(a, site, c, ok, blk, lambda x, y, z: (a[x], 1, c[z])))
    for i in range(1, half):
        w = isometry(i, lambda t: (t[0], t[1]))
        # mirrored: bonds outward from the right edge carry the opposite charge
        a, c = neg(bonds[i - 1]), neg(bonds[i])
        s = -1 if sym == U1 else 1
        blk = {(s * p, s * q, s * t): m.reshape(1, m.shape[0], m.shape[1]) for (q, p, t), m in w.items()}
        if sym == U1:
            # legs (site +, right -, left +): site - right + left = 0; the mirrored site charge enters reversed
            blk = {(-p, q, t): m for (p, q, t), m in blk.items()}
            ok = (lambda x, y, z: x - y + z == 0)
            write(L - 1 - i, [1, -1, 1], [site, a, c], every(site, a, c, ok, blk, lambda x, y, z: (1, a[y], c[z])))
        else:
            write(L - 1 - i, [1, 1, -1], [site, a, c], every(site, a, c, tri, blk, lambda x, y, z: (1, a[y], c[z])))


# ---------------------------------------------------------------------------
class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    k = case["kind"]
    if k in ("matvec", "lanczos"):
        s.h = sadmrg.Handle(sym=case["sym"], cplx=case["cplx"])
        s.h.set_autotune(False)
        psi = plan(s.h, case, problem(case, seed))
        if k == "matvec":
            s.x = torch.from_numpy(psi).to("cuda")
            s.y = torch.empty_like(s.x)
            torch.cuda.synchronize()
        else:
            s.psi = psi
    elif k == "svd":
        s.h = sadmrg.Handle(sym=case["sym"], cplx=case["cplx"])
        sym, cplx = case["sym"], case["cplx"]
        psi, _ = two_site_vector(case, seed)
        dl, dr = legs(case)
        bl, br = site_bonds(case)
        fl, fr = fused(sym, bl), fused(sym, br)
        psi = {q: psi[q] for q in psi}
        site = {-1: 1, 1: 1} if sym == U1 else {1: 1}
        sr = -1 if sym == U1 else 1
        s.psi = btensor([1, sr], [fl, fr], psi, cplx)
        s.tu = btensor([1, 1, -1], [bl, site, fl], {}, cplx)
        s.tv = btensor([1, sr, -sr], [site, br, fr], {}, cplx)
    elif k == "env":
        s.h = sadmrg.Handle(sym=U1, cplx=case["cplx"])
        t, uu, hh, ops = env_tensors(case, seed)
        cplx, ch = case["cplx"], {-2: 1, 0: 1, 2: 1}
        s.h.chain_create(1, 12, case["D"], 1, 0, True, case["J2"])
        s.site = 6
        s.h.chain_set_tensor(0, s.site, 0, btensor([1, -1, 1], [{-1: 1, 1: 1}, t["r"], t["l"]], uu, cplx))
        s.h.chain_set_tensor(1, s.site + 1, 0, btensor([1, -1], [t["r"], t["r"]], hh, cplx))
        for i, o in enumerate(ops):
            s.h.chain_set_tensor(2, s.site + 1, s.site + 1 + i, btensor([1, 1, -1], [t["r"], ch, t["r"]], o, cplx))
    elif k == "batch":
        s.h = sadmrg.Handle(sym=U1, cplx=False)
        psis = []
        for i, c in enumerate(instances(case)):
            one = sadmrg.Handle(sym=U1, cplx=False)
            one.set_autotune(False)
            psis.append(plan(one, c, problem(c, seed * 1000 + i)))
            s.h.batch_add(one)
            one.close()
        s.h.batch_finalize()
        s.psi = np.concatenate(psis)
    else:
        s.h = sadmrg.Handle(sym=case["sym"], cplx=False)
        s.dir = tempfile.TemporaryDirectory(prefix="sadmrg_mps_")
        write_mps(case, seed, s.dir.name)
    return s


def run(s):
    case, h = s.case, s.h
    k = case["kind"]
    if k == "matvec":
        h.heff_apply_device(s.x.data_ptr(), s.y.data_ptr(), case["prec"])
        return s.y
    if k == "lanczos":
        e, v, matvecs = h.heff_lanczos(s.psi, MLANC, sadmrg.PREC_FP64)
        return {"energy": e, "vector": v, "matvecs": matvecs}
    if k == "svd":
        u, v, kept, dw = h.svd_truncate(s.psi, s.tu, s.tv, 1.0, 0.0, case["D"])
        return {"u": u.data, "v": v.data, "kept": kept, "discarded": dw, "labels": np.array(u.qs[2]),
                "dims": np.array(u.ds[2])}
    if k == "env":
        h.chain_env_update(s.site, 1, True)
        out = [h.chain_get_tensor(1, s.site), h.chain_get_tensor(2, s.site, s.site)]
        if case["J2"]:
            out.append(h.chain_get_tensor(2, s.site, s.site + 1))
        return [t.data for t in out]
    if k == "batch":
        e, v, matvecs, _ = h.batch_lanczos(s.psi, MLANC, sadmrg.PREC_FP64)
        return {"energies": e, "vectors": v, "matvecs": matvecs}
    h.chain_create(1, case["L"], case["D"], 1, 0, True, case["J2"])
    h.chain_read_mps(s.dir.name, case["D"])
    h.chain_prepare_sweep()
    e = h.chain_sweep()
    bonds = np.zeros((case["L"], 128), np.int64)     # kept dimension per site and label
    for i in range(case["L"]):
        for q, n in h.chain_bond(i):
            bonds[i, q + 64] = n
    ww = np.zeros(8 * case["D"])                     # the chain's array, filled up to one length
    w = h.chain_ww()
    ww[:w.size] = w
    return {"energy": e, "singular_values": ww, "bonds": bonds}


def exact(case, seed):
    k = case["kind"]
    if k == "matvec":
        parts = problem(case, seed)
        return flat(apply_plain(case, parts, parts[2]))
    if k == "lanczos":
        # the sign of a Ritz vector is the solver's own
        return {"energy": lanczos_plain(case, problem(case, seed), MLANC), "vector": None, "matvecs": None}
    if k == "svd":
        # so are the signs and phases of singular vectors
        _, sv = two_site_vector(case, seed)
        every = torch.sort(torch.cat(list(sv.values())), descending=True)[0]
        w = (every ** 2).cpu().numpy()
        return {"u": None, "v": None, "kept": min(case["D"], len(w)), "labels": None, "dims": None,
                "discarded": float(math.fsum(w[case["D"]:]) / math.fsum(w))}
    if k == "env":
        t, uu, hh, ops = env_tensors(case, seed)
        out = []
        for b, d in zip(env_plain(case, t, uu, hh, ops), (2, 3, 3)):
            if b is None:
                continue
            bonds = [t["l"], t["l"]] if d == 2 else [t["l"], {-2: 1, 0: 1, 2: 1}, t["l"]]
            out.append(btensor([1] * d, bonds, b, case["cplx"]).data)
        return out
    if k == "batch":
        es = [lanczos_plain(c, problem(c, seed * 1000 + i), MLANC) for i, c in enumerate(instances(case))]
        return {"energies": np.array(es), "vectors": None, "matvecs": None}
    return None
