"""Performance cases of the engine's public entry points.

A case is one call that a DMRG, VUMPS or Chebyshev program makes for one site of its chain:

  hxv       H |v> on host vectors (PivotMatrix1 / PivotMatrix2 .apply), the inner call of any caller's eigensolver
  env       contract_L / contract_R, once per site and half sweep; new layouts every time, so the call plans and runs
  lanczos   the local ground state (.lanczos), once per site and half sweep
  cheb      Chebyshev moments of several start vectors (.chebyshev_moments), spectral functions
  transfer  the GMRES solve of a VUMPS environment (MpoTransferMatrix.solve_device)

The pivot is the middle of a seeded random MPS in mixed canonical form with environments contracted by the engine.
Chains are as short as the bond dimension in the middle allows; the sites further out do not enter the measured call.
`state` "start" is the two-site (one-site) tensor of the random MPS, which a first sweep meets; "converged" weights its
rows and columns with a Schmidt spectrum that decays over eight decades, which late sweeps meet.
"""
from __future__ import annotations

import functools
import math
from fractions import Fraction

import numpy as np

from vmps_gb300 import models
from vmps_gb300.blocks import Blocks
from vmps_gb300.mps import RandomMPS, bond_bases, contract_two_sites, site_layout, two_site_layout
from vmps_gb300.pivot import (Context, EnvUpdate, PivotMatrix1, PivotMatrix2, contract_L, contract_R, left_vacuum,
                              right_target)
from vmps_gb300.uniform import UniformMPS, bond_bases_su2
from vmps_gb300.vumps import MpoTransferMatrix

LANCZOS_C1 = dict(max_iter=100, tol_eigval=1e-12, tol_state=1e-8, refine_iters=0)      # dmrg1's defaults
LANCZOS_SWEEP = dict(max_iter=300, tol_eigval=1e-10, tol_state=1e-6, refine_iters=10)  # the sweep tolerances of the benchmark


def listed():
    return [
        # config C1, the smallest calls: a Heisenberg chain at D = 64, single-site; launches and latency
        dict(name="hxv1_heis_D64_fp64", op="hxv", model="heis", sites=1, D=64, precision="fp64", state="start"),
        dict(name="lanczos1_heis_D64_fp64", op="lanczos", model="heis", sites=1, D=64, precision="fp64",
             state="start", hxvs=40),
        # an odd, small two-site pivot in split precision: the growing bonds near the edges of a chain
        dict(name="hxv2_hubbard_D203_bf16x3", op="hxv", model="hubbard", sites=2, D=203, precision="bf16x3",
             state="converged"),
        # config C2: the Hubbard chain at D = 1024 and 4096, two-site; FP64 is the default precision of every call
        dict(name="hxv2_hubbard_D1024_fp64", op="hxv", model="hubbard", sites=2, D=1024, precision="fp64",
             state="converged"),
        dict(name="hxv2_hubbard_D4096_fp64", op="hxv", model="hubbard", sites=2, D=4096, precision="fp64",
             state="start"),
        dict(name="hxv2_hubbard_D4096_bf16x3", op="hxv", model="hubbard", sites=2, D=4096, precision="bf16x3",
             state="start"),
        dict(name="lanczos2_hubbard_D1024_bf16x3", op="lanczos", model="hubbard", sites=2, D=1024,
             precision="bf16x3", state="start", hxvs=80),
        # the environment updates of the same sweeps, both directions
        dict(name="env_L_hubbard_D1024_fp64", op="env", model="hubbard", side="L", D=1024, precision="fp64"),
        dict(name="env_R_hubbard_D300_fp64", op="env", model="hubbard", side="R", D=300, precision="fp64"),
        # config C3: Hubbard SU(2)xU(1) on a width-4 cylinder, single-site sweeps
        dict(name="hxv1_cylinder_D700_fp64", op="hxv", model="cylinder", sites=1, D=700, precision="fp64",
             state="start"),
        # config C4: the left environment of a two-site SU(2) Heisenberg cell, 256 multiplets per bond
        dict(name="transfer_heis_su2_D256_fp64", op="transfer", D=256, precision="fp64", hxvs=48),
        # config C5: Chebyshev moments of 16 start vectors; FP64, which 1000 moments need
        dict(name="cheb_hubbard_D256_16rhs_fp64", op="cheb", model="hubbard", sites=2, D=256, precision="fp64",
             state="converged", nrhs=16, nmom=32),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["hxv", "hxv", "hxv", "env", "env", "lanczos", "cheb", "transfer"])
    model = rng.choice(["heis", "hubbard", "hubbard", "cylinder"])
    state = rng.choice(["start", "converged"])
    if op == "hxv":
        hi = {"heis": 400, "hubbard": 4096, "cylinder": 900}[model]
        return dict(op=op, model=model, sites=1 if model == "cylinder" else rng.choice([1, 2]), D=size(24, hi),
                    precision=rng.choice(["fp64", "fp64", "bf16x3"]), state=state)
    if op == "env":
        hi = {"heis": 400, "hubbard": 1024, "cylinder": 500}[model]
        return dict(op=op, model=model, side=rng.choice(["L", "R"]), D=size(24, hi), precision="fp64")
    if op == "lanczos":
        model = "hubbard" if model == "cylinder" else model
        return dict(op=op, model=model, sites=rng.choice([1, 2]), D=size(24, 300 if model == "heis" else 900),
                    precision=rng.choice(["fp64", "bf16x3"]), state="start", hxvs=60)
    if op == "transfer":
        return dict(op=op, D=size(48, 256), precision="fp64", hxvs=48)
    return dict(op=op, model="hubbard", sites=2, D=size(24, 256), precision="fp64", state=state,
                nrhs=rng.randint(2, 16), nmom=2 * rng.randint(4, 16))


# ---- inputs -----------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    return Context(0)


@functools.lru_cache(maxsize=None)
def _model(kind, D):
    """(model, total quantum number, sigma of the sector profile): the shortest chain whose middle bonds hold D states"""
    if kind == "heis":
        m = models.heisenberg_u1(max(12, 2 * math.ceil(math.log2(D)) + 6))
        return m, (0,), [2.5]
    if kind == "hubbard":
        m = models.hubbard_u1xu1(max(8, 2 * math.ceil(math.log(D, 4)) + 4))
        return m, (m.L, 0), [2.5, 2.5]
    m = models.hubbard_su2xu1_lattice(16, models.cylinder_bonds(4, 4), U=8.0)
    return m, (1, 14), [3.0, 3.0]


def _pivot_sites(case, m):
    s = m.L // 2 - 1
    return s, s + case.get("sites", 1) - 1


def _mps(case, seed, lo, hi):
    m, qtot, sigma = _model(case["model"], case["D"])
    return RandomMPS(m, qtot, case["D"], seed=seed, profile="gaussian", sigma=sigma).canonicalize(lo, hi)


def _environments(m, mps, lo, hi):
    ctx = _context()
    L, R = left_vacuum(m.sym), right_target(m.sym, mps.Qtot)
    for side, sites in (("L", range(lo)), ("R", range(m.L - 1, hi, -1))):
        for l in sites:
            E = L if side == "L" else R
            e = EnvUpdate(ctx, m.sym, side, E, mps.A[l], m.W[l], mps.A[l])
            E = e.run(E, mps.A[l], mps.A[l])
            e.close()
            if side == "L":
                L = E
            else:
                R = E
    return L, R


def _pivot_problem(case, seed):
    m = _model(case["model"], case["D"])[0]
    lo, hi = _pivot_sites(case, m)
    mps = _mps(case, seed, lo, hi)
    L, R = _environments(m, mps, lo, hi)
    V = mps.A[lo] if lo == hi else contract_two_sites(m.sym, mps.A[lo], mps.A[hi], m.qloc, m.qloc, m.sym.nq)
    if case["state"] == "converged":
        for i in range(V.n):
            b = V.block(i)
            b *= 10.0 ** np.linspace(0, -4, b.shape[0])[:, None] * 10.0 ** np.linspace(0, -4, b.shape[1])[None, :]
    V.data /= np.linalg.norm(V.data)
    return m, L, R, [m.W[l] for l in range(lo, hi + 1)], V


def _vectors(case, V, seed):
    """start vectors of a Chebyshev case: the state and noise of its size (local operators applied to it)"""
    rng = np.random.default_rng(seed + 1)
    X = np.abs(V.data)[None, :] * rng.standard_normal((case["nrhs"], V.data.size))
    return X / np.linalg.norm(X, axis=1)[:, None]


def _window(case):
    """(a, b) of the expansion in (H - b) / a; |E| per site of the Hubbard chain stays below 4"""
    n = _model(case["model"], case["D"])[0].L
    return 4.0 * n, 0.0


def _uniform(D, seed):
    m = models.heisenberg_su2(8)
    u = UniformMPS(m, bond_bases_su2(D, 14), seed=seed)
    u.gauge(tol=1e-11)
    return m, u


def _transfer_problem(case, seed):
    m, u = _uniform(case["D"], seed)
    order, W, nq = m.basis_order_map(4), [m.W[4], m.W[5]], m.sym.nq
    slot = max(p for (q, _), p in order.items() if tuple(q) == m.sym.vacuum())
    q0, a = next(k for k, p in order.items() if p == slot)
    rho = {q: M @ M.T for q, M in u.C[0].items()}
    LR = Blocks.from_entries(nq, [(0, q, q, rho[q]) for q in sorted(rho)])
    rng = np.random.default_rng(seed + 1)
    Y = Blocks.from_entries(nq, [(a, q, q, tuple(q0), rng.standard_normal((n, n)))
                                 for q, n in sorted(u.dims[0].items())], tripod=True)
    e = sum(float(np.trace(Y.block(i) @ rho[tuple(Y.qin[i])])) * m.sym.dot_weight(tuple(Y.qin[i])) for i in range(Y.n))
    b = np.concatenate([(Y.block(i) - e * np.eye(Y.rows[i])).T.ravel() for i in range(Y.n)])
    return m, u, W, LR, slot, order, Y.like(), b


def prepare(case, seed):
    ctx, op = _context(), case["op"]
    if op == "env":
        m = _model(case["model"], case["D"])[0]
        lo, hi = _pivot_sites(case, m)
        at = lo + 1 if case["side"] == "L" else lo - 1
        mps = _mps(case, seed, at, at)   # site lo normalised towards the environment's side
        if case["side"] == "L":
            E = _environments(m, mps, lo, m.L)[0]
        else:
            E = _environments(m, mps, 0, lo)[1]
        return dict(case=case, m=m, E=E, A=mps.A[lo], W=m.W[lo])
    if op == "transfer":
        m, u, W, LR, slot, order, V, b = _transfer_problem(case, seed)
        T = MpoTransferMatrix(ctx, m.sym, "L", u.AL, u.AL, W, LR, slot, order, V)
        return dict(case=case, T=T, b=b)
    m, L, R, Ws, V = _pivot_problem(case, seed)
    H = (PivotMatrix1(ctx, m.sym, L, R, Ws[0], V) if len(Ws) == 1 else PivotMatrix2(ctx, m.sym, L, R, Ws[0], Ws[1], V))
    H.prepare(case["precision"], fp64_too=op == "lanczos")
    s = dict(case=case, H=H, v=V.data.copy())
    if op == "hxv":
        s["out"] = np.zeros_like(s["v"])
    elif op == "cheb":
        s["X"] = _vectors(case, V, seed)
    return s


def run(s):
    case = s["case"]
    op, prec = case["op"], case["precision"]
    if op == "hxv":
        return s["H"].apply(s["v"], prec, out=s["out"])
    if op == "env":
        f = contract_L if case["side"] == "L" else contract_R
        return f(_context(), s["m"].sym, s["E"], s["A"], s["W"], s["A"], prec).data
    if op == "lanczos":
        e, v, _ = s["H"].lanczos(s["v"], prec, **(LANCZOS_C1 if prec == "fp64" else LANCZOS_SWEEP))
        return {"energy": e, "vector": v}
    if op == "cheb":
        a, b = _window(case)
        return s["H"].chebyshev_moments(s["X"], case["nmom"], a, b, prec)[0]
    return s["T"].solve_device(s["b"], tol=1e-12, dimK=100, precision=prec)[0]


# ---- the same contractions in numpy -------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _delta(a, b, c):
    f = math.factorial
    if (a + b + c) % 2 or c < abs(a - b) or c > a + b:
        return Fraction(0)
    return Fraction(f((a + b - c) // 2) * f((a - b + c) // 2) * f((b + c - a) // 2), f((a + b + c) // 2 + 1))


@functools.lru_cache(maxsize=None)
def _sixj(a, b, c, d, e, f):
    """Racah's formula; arguments 2j"""
    t = [_delta(a, b, c), _delta(a, e, f), _delta(d, b, f), _delta(d, e, c)]
    if not all(t):
        return 0.0
    F = math.factorial
    lows = [(a + b + c) // 2, (a + e + f) // 2, (d + b + f) // 2, (d + e + c) // 2]
    highs = [(a + b + d + e) // 2, (b + c + e + f) // 2, (a + c + d + f) // 2]
    s = sum(Fraction((-1) ** k * F(k + 1), math.prod(F(k - x) for x in lows) * math.prod(F(x - k) for x in highs))
            for k in range(max(lows), min(highs) + 1))
    return float(s) * math.sqrt(math.prod(t))


@functools.lru_cache(maxsize=None)
def _ninej(a, b, c, d, e, f, g, h, j):
    s = 0.0
    for x in range(max(abs(a - j), abs(d - h), abs(b - f)), min(a + j, d + h, b + f) + 1):
        s += (-1) ** x * (x + 1) * _sixj(a, b, c, f, j, x) * _sixj(d, e, f, b, x, h) * _sixj(g, h, j, x, a, d)
    return s


def _coupling(sym, q9):
    """the recoupling factor of one site: a 9j symbol and root dimensions for each SU(2) component, else 1"""
    r = 1.0
    for i, kind in enumerate(sym.kinds):
        if kind == "SU2":
            q = [int(x[i]) for x in q9]
            r *= _ninej(*(x - 1 for x in q)) * math.sqrt(q[6] * q[7] * q[2] * q[5])
    return r


def _fuse(sym, a, b, sign=1):
    out = [()]
    for i, kind in enumerate(sym.kinds):
        vals = [a[i] + sign * b[i]] if kind == "U1" else range(abs(a[i] - b[i]) + 1, a[i] + b[i], 2)
        out = [q + (v,) for q in out for v in vals]
    return out


def _rows(B):
    keys = [list(map(tuple, x.tolist())) for x in (B.qin, B.qout)] + [B.leg.tolist()]
    return list(zip(*keys)) if B.qmid is None else list(zip(*keys, map(tuple, B.qmid.tolist())))


def _entries(W):
    return zip(W.s1, W.s2, W.k, W.qin, W.qout, W.row, W.col, W.val)


def _by_slot(B):
    by = {}
    for i, (qin, qout, leg, qmid) in enumerate(_rows(B)):
        by.setdefault((qmid, leg), []).append((i, qin, qout))
    return by


def _chains_hxv(sym, L, Ws, R, V):
    """{(out, l, v, r): factor} of out += factor * L[l] V[v] R[r]"""
    Lby = _by_slot(L)
    Vat = {(leg, qin, qout): i for i, (qin, qout, leg) in enumerate(_rows(V))}
    Rat = {k: i for i, k in enumerate(_rows(R))}
    ch = {}
    if len(Ws) == 1:
        W = Ws[0]
        for s1, s2, k, qa, qb, row, col, val in _entries(W):
            for l, lin, lout in Lby.get((qa, row), ()):
                for rout in _fuse(sym, lin, W.qloc[s1]):
                    o = Vat.get((s1, lin, rout))
                    for rin in _fuse(sym, lout, W.qloc[s2]) if o is not None else ():
                        v, r = Vat.get((s2, lout, rin)), Rat.get((rin, rout, col, qb))
                        if v is None or r is None:
                            continue
                        c = val * _coupling(sym, (lout, W.qloc[s2], rin, qa, W.qop[k], qb, lin, W.qloc[s1], rout))
                        if c:
                            ch[o, l, v, r] = ch.get((o, l, v, r), 0.0) + c
        return ch
    W, X = Ws
    # combined local states, by their sum, then by the two parts
    pairs = sorted((_fuse(sym, a, b)[0], a, b, i, j) for i, a in enumerate(W.qloc) for j, b in enumerate(X.qloc))
    leg = {(p[3], p[4]): n for n, p in enumerate(pairs)}
    right = {}
    for s3, s4, _, qb, qc, row, col, val in _entries(X):
        right.setdefault((qb, row), []).append((s3, s4, qc, col, val))
    for s1, s2, _, qa, qb, row, mid, val in _entries(W):
        for s3, s4, qc, col, val2 in right.get((qb, mid), ()):
            c13, c24 = leg[s1, s3], leg[s2, s4]
            for l, lin, lout in Lby.get((qa, row), ()):
                rout, rin = _fuse(sym, lin, pairs[c13][0])[0], _fuse(sym, lout, pairs[c24][0])[0]
                o, v, r = Vat.get((c13, lin, rout)), Vat.get((c24, lout, rin)), Rat.get((rin, rout, col, qc))
                if o is not None and v is not None and r is not None:
                    ch[o, l, v, r] = ch.get((o, l, v, r), 0.0) + val * val2
    return ch


def _chains_env(sym, side, E, Abra, W, Aket, keep=None):
    """[(output key, bra, e, ket, factor)] of out += factor * bra^T E ket (L) or ket E bra^T (R)"""
    Eby = _by_slot(E)
    bra = {(leg, qin, qout): i for i, (qin, qout, leg) in enumerate(_rows(Abra))}
    ket = {(leg, qin, qout): i for i, (qin, qout, leg) in enumerate(_rows(Aket))}
    ch = []
    for s1, s2, k, qa, qb, row, col, val in _entries(W):
        if keep is not None and not keep(qa, row, qb, col):
            continue
        if side == "L":
            for e, ein, eout in Eby.get((qa, row), ()):
                for rout in _fuse(sym, ein, W.qloc[s1]):
                    b = bra.get((s1, ein, rout))
                    for rin in _fuse(sym, eout, W.qloc[s2]) if b is not None else ():
                        t = ket.get((s2, eout, rin))
                        if t is None or rout not in _fuse(sym, rin, qb):
                            continue
                        c = val * _coupling(sym, (eout, W.qloc[s2], rin, qa, W.qop[k], qb, ein, W.qloc[s1], rout))
                        if c:
                            ch.append(((rout, rin, col, qb), b, e, t, c))
        else:   # abelian only: the SU(2) cases contract from the left
            for e, ein, eout in Eby.get((qb, col), ()):
                lin, lout = _fuse(sym, eout, W.qloc[s1], -1)[0], _fuse(sym, ein, W.qloc[s2], -1)[0]
                b, t = bra.get((s1, lin, eout)), ket.get((s2, lout, ein))
                if b is not None and t is not None and lin in _fuse(sym, lout, qa):
                    ch.append(((lout, lin, row, qa), b, e, t, val))
    return ch


def _mats(B, data=None):
    d = B.data if data is None else data
    return [d[..., o:o + r * c].reshape(d.shape[:-1] + (c, r)).swapaxes(-1, -2)
            for o, r, c in zip(B.offset.tolist(), B.rows.tolist(), B.cols.tolist())]


def _plan(ch):
    """the chains as (l, v) products, and for each (out, r) the products that are summed first"""
    lv, groups = {}, {}
    for (o, l, v, r), c in ch.items():
        groups.setdefault((o, r), []).append((lv.setdefault((l, v), len(lv)), c))
    return lv, groups


def _hxv(L, R, V, plan, x):
    """H x for x of shape (dim,) or (n, dim)"""
    Lm, Rm, Vm = _mats(L), _mats(R), _mats(V, x)
    T = [Lm[l] @ Vm[v] for l, v in plan[0]]
    out = np.zeros_like(x)
    Om = _mats(V, out)
    for (o, r), terms in plan[1].items():
        Om[o][...] += sum(c * T[t] for t, c in terms) @ Rm[r]
    return out


def _env(E, Abra, Aket, ch, side, Em=None):
    Em, Bm, Km = _mats(E) if Em is None else Em, _mats(Abra), _mats(Aket)
    out = {}
    for key, b, e, t, c in ch:
        p = c * (Bm[b].T @ (Em[e] @ Km[t]) if side == "L" else Km[t] @ (Em[e] @ Bm[b].T))
        if key in out:
            out[key] += p
        else:
            out[key] = p
    return out


def _ground_state(apply, v, iters):
    """full Lanczos from v; the vector's sign is the one in which its largest Krylov coefficient is positive"""
    K, al, be = [v / np.linalg.norm(v)], [], []
    for _ in range(iters):
        w = apply(K[-1])
        al.append(float(w @ K[-1]))
        for _ in range(2):
            B = np.array(K)
            w = w - B.T @ (B @ w)
        nw = float(np.linalg.norm(w))
        th, y = np.linalg.eigh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))
        if nw * abs(y[-1, 0]) < 1e-12 * max(1.0, abs(th[0])) or nw < 1e-13:
            break
        be.append(nw)
        K.append(w / nw)
    y = y[:, 0] * np.sign(y[np.argmax(np.abs(y[:, 0])), 0])
    x = np.array(K[:len(y)]).T @ y
    return float(th[0]), x / np.linalg.norm(x)


def _solve(apply, dot, b, tol, iters):
    Q, H = [b / math.sqrt(dot(b, b))], np.zeros((iters + 1, iters))
    for k in range(iters):
        w = apply(Q[k])
        for _ in range(2):
            for j in range(k + 1):
                h = dot(Q[j], w)
                H[j, k] += h
                w = w - h * Q[j]
        H[k + 1, k] = math.sqrt(dot(w, w))
        e = np.zeros(k + 2)
        e[0] = math.sqrt(dot(b, b))
        y = np.linalg.lstsq(H[:k + 2, :k + 1], e, rcond=None)[0]
        if np.linalg.norm(H[:k + 2, :k + 1] @ y - e) < tol * e[0] or H[k + 1, k] < 1e-14:
            break
        Q.append(w / H[k + 1, k])
    return sum(c * q for c, q in zip(y, Q))


def exact(case, seed):
    op = case["op"]
    if op == "transfer":
        m, u, W, LR, slot, order, V, b = _transfer_problem(case, seed)
        (at, row), rows = next(k for k, p in order.items() if p == slot), _rows(V)
        layouts = [V]
        first = _chains_env(m.sym, "L", V, u.AL[0], W[0], u.AL[0], lambda qa, r, qb, c: (qa, r) == (at, row))
        keys = sorted({c[0] for c in first})
        shape = {k: (int(u.AL[0].cols[c[1]]), int(u.AL[0].cols[c[3]])) for c in first for k in [c[0]]}
        layouts.append(Blocks(m.sym.nq, *zip(*[(k[0], k[1], k[2], *shape[k]) for k in keys]), qmid=[k[3] for k in keys]))
        second = _chains_env(m.sym, "L", layouts[1], u.AL[1], W[1], u.AL[1], lambda qa, r, qb, c: (qb, c) == (at, row))
        weight = [m.sym.dot_weight(r[1]) for r in rows]
        rho = {tuple(LR.qin[i]): LR.block(i) for i in range(LR.n)}
        w = np.concatenate([np.full(int(r * c), x) for r, c, x in zip(V.rows, V.cols, weight)])

        def apply(x):
            Xm = _mats(V, x)
            t = _env(V, u.AL[0], u.AL[0], first, "L", Xm)
            t = _env(layouts[1], u.AL[1], u.AL[1], second, "L", [t[k] for k in keys])
            s = sum(float(np.sum(X * rho[r[0]].T)) * f for X, r, f in zip(Xm, rows, weight))
            return np.concatenate([(X - t[r[0], r[1], r[2], r[3]] + s * np.eye(len(X))).T.ravel() if r in t else 0 * X.ravel()
                                   for X, r in zip(Xm, rows)])

        return _solve(apply, lambda p, q: float(np.sum(w * p * q)), b, 1e-14, 90)
    if op == "env":
        s = prepare(case, seed)
        if case["side"] == "R" and s["m"].sym.nonabelian:
            return None
        out = _env(s["E"], s["A"], s["A"], _chains_env(s["m"].sym, case["side"], s["E"], s["A"], s["W"], s["A"]), case["side"])
        sym = s["m"].sym
        e = EnvUpdate(_context(), sym, case["side"], s["E"], s["A"], s["W"], s["A"])   # the order of the blocks only
        lay = e.out_layout.like()
        e.close()
        for i, k in enumerate(_rows(lay)):
            lay.block(i)[...] = out[k]
        return lay.data
    if op == "lanczos" and case["D"] * case["sites"] > (400 if case["model"] == "heis" else 150):
        return None   # minutes
    m, L, R, Ws, V = _pivot_problem(case, seed)
    plan = _plan(_chains_hxv(m.sym, L, Ws, R, V))
    if op == "hxv":
        return _hxv(L, R, V, plan, V.data)
    if op == "lanczos":
        e, x = _ground_state(lambda x: _hxv(L, R, V, plan, x), V.data, 160)
        return {"energy": e, "vector": x}
    a, b = _window(case)
    t = [_vectors(case, V, seed)]
    t.append((_hxv(L, R, V, plan, t[0]) - b * t[0]) / a)
    mu = [np.sum(t[0] * t[0], axis=1), np.sum(t[1] * t[0], axis=1)]
    for n in range(1, (case["nmom"] + 1) // 2):
        t = [t[1], 2.0 / a * (_hxv(L, R, V, plan, t[1]) - b * t[1]) - t[0]]
        mu += [2 * np.sum(t[0] * t[0], axis=1) - mu[0], 2 * np.sum(t[1] * t[0], axis=1) - mu[1]]
    return np.stack(mu[:case["nmom"]], axis=1)


# ---- the work a pass cannot do without ------------------------------------------------------------------------------
def _tripod(sym, order, dims):
    ent = [(a, p, q, tuple(qm)) for (qm, a), _ in sorted(order.items(), key=lambda kv: kv[1])
           for q in sorted(dims) for p in _fuse(sym, q, qm) if p in dims]
    return Blocks(sym.nq, [e[1] for e in ent], [e[2] for e in ent], [e[0] for e in ent],
                  [dims[e[1]] for e in ent], [dims[e[2]] for e in ent], qmid=[e[3] for e in ent])


def _elements(B):
    return int(np.sum(B.rows * B.cols))


@functools.lru_cache(maxsize=None)
def _counts(model, D, sites, side):
    """(flops, elements of the fixed operands, elements of the vector, elements of the output) of one contraction"""
    m, qtot, sigma = _model(model, D)
    sym = m.sym
    dims = bond_bases(m.qloc, m.L, qtot, D, profile="gaussian", sigma=sigma, sym=sym if sym.nonabelian else None)
    lo, hi = m.L // 2 - 1, m.L // 2 - 2 + sites
    s = sym if sym.nonabelian else None
    left, right = (_tripod(sym, m.basis_order_map(b), dims[b]) for b in (lo, hi + 1))
    if side:
        E, F = (left, right) if side == "L" else (right, left)
        A = site_layout(m.qloc, dims[lo], dims[lo + 1], sym.nq, s)
        flops, pairs, outs = 0.0, set(), set()
        for o, b, e, t, _ in _chains_env(sym, side, E, A, m.W[lo], A):
            first = int(E.rows[e] * E.cols[e] * (A.cols[t] if side == "L" else A.rows[b]))
            second = int(A.rows[b] * A.cols[b] * A.cols[t]) if side == "L" else int(A.rows[t] * A.cols[t] * A.rows[b])
            flops += 2.0 * first * ((e, t) not in pairs) + 2.0 * second * ((o, b) not in outs)
            pairs.add((e, t))
            outs.add((o, b))
        return flops, _elements(A), _elements(E), _elements(F)
    if sites == 1:
        V = site_layout(m.qloc, dims[lo], dims[lo + 1], sym.nq, s)
    else:
        V = two_site_layout(sym, m.qloc, m.qloc, dims[lo], dims[hi + 1], sym.nq)[0]
    lv, groups = _plan(_chains_hxv(sym, left, [m.W[l] for l in range(lo, hi + 1)], right, V))
    flops = 2.0 * sum(int(left.rows[l] * left.cols[l] * V.cols[v]) for l, v in lv)
    flops += 2.0 * sum(int(V.rows[o] * right.rows[r] * right.cols[r]) for o, r in groups)
    return flops, _elements(left) + _elements(right), _elements(V), _elements(V)


@functools.lru_cache(maxsize=None)
def _transfer_counts(D):
    dims = bond_bases_su2(D, 14)
    n = [sum(d.values()) for d in dims]
    vec = sum(k * k for k in dims[0].values())
    flops = 0.0
    for d, e in ((dims[0], dims[1]), (dims[1], dims[0])):   # E A then A^T (E A), the idle slot through both sites
        for (q,), k in d.items():
            for p in (q - 1, q + 1):
                flops += 2.0 * k * e.get((p,), 0) * (k + e.get((p,), 0))
    return flops, 2 * n[0] * n[1], vec


def work(case):
    op = case["op"]
    if op == "transfer":
        flops, fixed, vec = _transfer_counts(case["D"])
        return {"bytes": 8.0 * (fixed + 2 * vec), "flops": case["hxvs"] * flops}
    flops, fixed, vec, out = _counts(case["model"], case["D"], case.get("sites", 1), case.get("side"))
    if op == "cheb":
        n = case["nrhs"]
        return {"bytes": 8.0 * (fixed + n * vec + n * case["nmom"]), "flops": (case["nmom"] + 1) // 2 * n * flops}
    return {"bytes": 8.0 * (fixed + vec + out), "flops": case.get("hxvs", 1) * flops}
