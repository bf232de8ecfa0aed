"""The work this library is used for, as measurable cases: `listed()` names them, `draw()` gives more
of the same ranges, `prepare()` makes what a program holds before a call, `run()` makes the call.

A program keeps its tensors on the device and calls the public functions of `mps_gb300`: the two-site
effective Hamiltonian (prepared, or one-shot for the post-truncation energy), environment updates, the
Krylov ground-state solve, the complex one-site Hamiltonian of time evolution, the two truncations and a
whole sweep. Sizes are those of the benchmark (chi = 2048 over 25 charges), of its smaller configurations
(chi = 512 TDVP, chi = 1024 cylinder, the L = 32, chi = 64 chain) and odd ones between them; precision 0
(FP64) is the default of every entry point, 5 and 7 slices are what the mixed-precision sweep uses.

`exact()` restates each case densely in 64-bit torch / numpy."""
import math

import numpy as np
import torch

import mps_gb300 as mg
from mps_gb300 import ctensor, dmrg, tdvp

BOND = ((-1, 1), (0, 3), (1, 1))  # bond space of the XXZ MPO
SITE = ((0, 1), (1, 1))
DELTA = 0.5


# ---- cases -----------------------------------------------------------------------------------------
def listed():
    return [
        # one Krylov matvec of the FP64 sweep at the benchmark's size, and of smaller chains: an
        # ordinary odd one, and the smallest, where launches and host work are what counts
        {"name": "heff fp64 2048", "kind": "heff", "chi": 2048, "charges": 25, "precision": 0},
        {"name": "heff fp64 517", "kind": "heff", "chi": 517, "charges": 13, "precision": 0},
        {"name": "heff fp64 48", "kind": "heff", "chi": 48, "charges": 7, "precision": 0},
        # one Krylov matvec of the mixed-precision sweep (5 slices), the benchmark's headline
        {"name": "heff s5 2048", "kind": "heff", "chi": 2048, "charges": 25, "precision": 5},
        # the mixed sweep's post-truncation energy matvec: one-shot, operator built in the call
        {"name": "energy s7 701", "kind": "energy", "chi": 701, "charges": 17, "precision": 7},
        # environment updates, left in FP64 (drop-in sweep), right with 7 slices (mixed sweep)
        {"name": "env left fp64 1024", "kind": "env", "side": "left", "chi": 1024, "charges": 17,
         "precision": 0},
        {"name": "env right s7 363", "kind": "env", "side": "right", "chi": 363, "charges": 11,
         "precision": 7},
        # ground-state solve of one bond of an FP64 sweep (thick-restart Lanczos)
        {"name": "eigsolve fp64 256", "kind": "eigsolve", "chi": 256, "length": 20, "precision": 0},
        # one matvec of one-site time evolution (complex state, FP64), the TDVP configuration
        {"name": "tdvp matvec fp64 512", "kind": "tdvp", "chi": 512, "charges": 15, "precision": 0},
        # truncation of a two-site tensor: exact SVD of a small chain, density matrix of a large one
        {"name": "truncate exact 128", "kind": "truncate", "chi": 128, "charges": 9, "method": "exact"},
        {"name": "truncate gram 1024", "kind": "truncate", "chi": 1024, "charges": 17,
         "method": "gram_left"},
        # a whole FP64 sweep of the CPU-sized chain
        {"name": "sweep fp64 L32 chi64", "kind": "sweep", "chi": 64, "length": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["heff", "heff", "heff", "energy", "env", "env", "eigsolve", "tdvp", "truncate",
                       "sweep"])
    c = {"kind": kind}
    if kind == "sweep":
        c.update(chi=_log(rng, 16, 64), length=2 * rng.randint(6, 16))
        return c
    if kind == "eigsolve":
        c.update(chi=_log(rng, 24, 256), length=2 * rng.randint(7, 12), precision=0)
        return c
    c["charges"] = rng.randint(5, 25)
    if kind == "heff":
        c.update(chi=_log(rng, 48, 2048), precision=rng.choice([0, 0, 5]))
    elif kind == "energy":
        c.update(chi=_log(rng, 64, 1400), precision=rng.choice([0, 7]))
    elif kind == "env":
        c.update(side=rng.choice(["left", "right"]), chi=_log(rng, 48, 1400),
                 precision=rng.choice([0, 7]))
    elif kind == "tdvp":
        c.update(chi=_log(rng, 48, 512), precision=0)
    else:
        method = rng.choice(["exact", "gram_left", "gram_right"])
        c.update(method=method, chi=_log(rng, 32, 160 if method == "exact" else 1024))
    return c


# ---- graded spaces, written out ----------------------------------------------------------------------
# a leg is ((charge, dim), ...) with a dual flag; a tensor stores its allowed blocks one after the
# other, first leg's charge fastest, each column-major
def _bond(c, extra=0):
    n = c["charges"] + extra
    return tuple(enumerate(dmrg.binomial_profile(max(c["chi"], n), n)))


def _sectors(legs):
    """[(dims, charges)] of the allowed blocks of a charge-0 tensor in storage order."""
    out = []

    def rec(k, rest, chosen):
        if k < 0:
            if rest == 0:
                out.append(tuple(reversed(chosen)))
            return
        leg, dual = legs[k]
        for q, d in leg:
            rec(k - 1, rest - (-q if dual else q), chosen + [(q, d)])

    rec(len(legs) - 1, 0, [])
    return out


def _numel(legs):
    return sum(math.prod(d for _, d in s) for s in _sectors(legs))


def _flops(legs_a, con_a, legs_b, con_b):
    """2 M N K summed over the charges of the fused contracted legs."""
    def fused(legs, which, sign):
        acc = {0: 1}
        for k in which:
            leg, dual = legs[k]
            new = {}
            for q0, d0 in acc.items():
                for q, d in leg:
                    e = q0 + sign * (-q if dual else q)
                    new[e] = new.get(e, 0) + d0 * d
            acc = new
        return acc

    rows = fused(legs_a, [k for k in range(len(legs_a)) if k not in con_a], 1)
    mid = fused(legs_a, con_a, -1)
    cols = fused(legs_b, [k for k in range(len(legs_b)) if k not in con_b], -1)
    return 2.0 * sum(rows[q] * mid[q] * cols[q] for q in rows if q in mid and q in cols)


def _dense(flat, legs):
    """The dense array of a block list (torch, on the GPU)."""
    at = [{} for _ in legs]
    for k, (leg, _) in enumerate(legs):
        p = 0
        for q, d in leg:
            at[k][q] = p
            p += d
    out = torch.zeros([sum(d for _, d in leg) for leg, _ in legs], dtype=torch.float64, device="cuda")
    x = torch.as_tensor(flat, dtype=torch.float64).to("cuda")
    p = 0
    for s in _sectors(legs):
        dims = [d for _, d in s]
        n = math.prod(dims)
        block = x[p:p + n].reshape(dims[::-1]).permute(*range(len(dims) - 1, -1, -1))
        out[tuple(slice(at[k][q], at[k][q] + d) for k, (q, d) in enumerate(s))] = block
        p += n
    return out


def _flat(dense, legs):
    at = [{} for _ in legs]
    for k, (leg, _) in enumerate(legs):
        p = 0
        for q, d in leg:
            at[k][q] = p
            p += d
    return torch.cat([dense[tuple(slice(at[k][q], at[k][q] + d) for k, (q, d) in enumerate(s))]
                      .permute(*range(len(s) - 1, -1, -1)).reshape(-1) for s in _sectors(legs)])


V, D = False, True  # plain and dual legs


def _legs(kind, c):
    """Legs of the operands of one contraction case."""
    if kind in ("heff", "energy"):
        b = _bond(c)
        return {"v": [(b, V), (SITE, V), (SITE, V), (b, D)], "L": [(b, D), (BOND, D), (b, V)],
                "R": [(b, V), (BOND, V), (b, D)], "W": [(BOND, V), (SITE, V), (BOND, D), (SITE, D)]}
    l, r = _bond(c), _bond(c, 1)  # a site tensor adds one charge
    return {"v": [(l, V), (SITE, V), (r, D)], "L": [(l, D), (BOND, D), (l, V)],
            "R": [(r, V), (BOND, V), (r, D)], "W": [(BOND, V), (SITE, V), (BOND, D), (SITE, D)]}


_MAT = [np.array([[1.0, 0, 0], [-0.5 * DELTA, 0, 0], [0, -0.5, 1]]),
        np.array([[1.0, 0, 0], [0.5 * DELTA, 0, 0], [0, 0.5, 1]])]
_W = {(0, 0, 0, 0): _MAT[0].reshape((3, 1, 3, 1), order="F"),
      (0, 1, 0, 1): _MAT[1].reshape((3, 1, 3, 1), order="F"),
      (0, 1, 1, 0): np.array([0.0, 0, 1]).reshape((3, 1, 1, 1)),
      (0, 0, -1, 1): np.array([0.0, 0, 1]).reshape((3, 1, 1, 1)),
      (1, 0, 0, 1): np.array([0.5, 0, 0]).reshape((1, 1, 3, 1)),
      (-1, 1, 0, 0): np.array([0.5, 0, 0]).reshape((1, 1, 3, 1))}


def _w_flat(legs):
    return np.concatenate([_W.get(tuple(q for q, _ in s), np.zeros([d for _, d in s])).ravel(order="F")
                           for s in _sectors(legs)])


# ---- inputs ------------------------------------------------------------------------------------------
def _rng(seed):
    return np.random.Generator(np.random.Philox(1911 + int(seed)))


def _contraction_inputs(c, seed):
    """Flat host arrays of a heff / energy / env / tdvp case: N(0,1) blocks, as the benchmark's."""
    legs = _legs(c["kind"], c)
    rng = _rng(seed)
    x = {k: rng.standard_normal(_numel(legs[k])) for k in ("v", "L", "R")}
    if c["kind"] == "tdvp":
        for k in ("v", "L", "R"):
            x[k + "i"] = rng.standard_normal(x[k].size)
    x["W"] = _w_flat(legs["W"])
    return legs, x


def _two_site(c):
    b = _bond(c)
    return [(b, V), (SITE, V), (SITE, V), (b, D)]


def _theta_blocks(c, seed):
    """A two-site wave function as the matrix (l s) x (t r) of norm 1: per charge, random orthonormal
    factors around a spectrum that falls over about seven decades, weighted by sector."""
    rng = _rng(seed)
    leg = {}
    for q, d in _bond(c):
        for s, _ in SITE:
            leg[q + s] = leg.get(q + s, 0) + d
    rows = tuple(sorted(leg.items()))
    out, mid = [], sum(q for q, _ in rows) / len(rows) + 0.137  # no two charges share values
    col = {}
    for q, d in _bond(c):
        for s, _ in SITE:
            col[q - s] = col.get(q - s, 0) + d
    for q, n in rows:
        m = col.get(q, 0)
        if m == 0:
            continue
        k = min(n, m)
        decay = np.exp(-16.0 * np.arange(k) / k) * math.exp(-0.3 * (q - mid) ** 2)
        a = np.linalg.qr(rng.standard_normal((n, k)))[0]
        b = np.linalg.qr(rng.standard_normal((m, k)))[0]
        out.append((q, (a * decay) @ b.T))
    norm = math.sqrt(sum(float(np.sum(t * t)) for _, t in out))
    return rows, tuple(sorted(col.items())), [(q, t / norm) for q, t in out]


def _chain_inputs(c, seed):
    """Both halves of a random canonical MPS (site matrices (l s) x r orthonormal) and the two-site
    start vector at the middle bond of an L-site chain at half filling."""
    lx, half, chi = c["length"], c["length"] // 2, c["chi"]
    rng = _rng(seed)
    bond = [((0, 1),)] + [tuple(dmrg.binomial_bond_dims(lx, k, half, chi)) for k in range(1, lx)] + \
        [((half, 1),)]

    def site(l, r, right):
        legs = [(l, V), (SITE, V), (r, D)]
        rows, cols = (dict(r), dict(l)) if right else (dict(l), dict(r))
        blocks = {}
        for q, n in (l if right else r):  # the bond whose states become orthonormal
            src = [(q + s if right else q - s, s) for s, _ in SITE]
            src = [(p, s) for p, s in src if p in rows]
            m = sum(rows[p] for p, _ in src)
            if m == 0:
                continue
            g = rng.standard_normal((m, n))
            g = np.linalg.qr(g)[0] if n <= m else g / math.sqrt(m)
            at = 0
            for p, s in src:
                g1 = g[at:at + rows[p]]
                at += rows[p]
                blocks[(q, s, p) if right else (p, s, q)] = (g1.T if right else g1)[:, None, :]
        return legs, np.concatenate([blocks[tuple(q for q, _ in x)].ravel(order="F")
                                     for x in _sectors(legs)])

    left = [site(bond[k], bond[k + 1], False) for k in range(half - 1)]
    right = [site(bond[k], bond[k + 1], True) for k in range(half + 1, lx)]
    legs = [(bond[half - 1], V), (SITE, V), (SITE, V), (bond[half + 1], D)]
    x = rng.standard_normal(_numel(legs))
    edge = [[(bond[0], D), (BOND, D), (bond[0], V)], [(bond[lx], V), (BOND, V), (bond[lx], D)]]
    ends = [np.array([0.0, 0, 1]), np.array([1.0, 0, 0])]  # the MPO's first row and last column
    return left, right, (legs, x / np.linalg.norm(x)), edge, ends


def _space(legs):
    return tuple(mg.VectorSpace(leg, dual) for leg, dual in legs)


def _up(legs, flat):
    return mg.from_flat(0, _space(legs), flat)


_W_LEGS = [(BOND, V), (SITE, V), (BOND, D), (SITE, D)]


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("heff", "energy", "env", "tdvp"):
        legs, x = _contraction_inputs(c, seed)
        t = {k: _up(legs[k], x[k]) for k in ("v", "L", "R", "W")}
        if kind == "heff":
            t["op"] = mg.Heff2(t["v"], t["L"], t["R"], t["W"], t["W"], precision=c["precision"])
        elif kind == "tdvp":
            t["ops"] = ctensor.gpu_ops(precision=c["precision"])
            for k in ("v", "L", "R"):
                t["c" + k] = ctensor.CTensor(t[k], _up(legs[k], x[k + "i"]))
    elif kind == "truncate":
        rows, cols, blocks = _theta_blocks(c, seed)
        legs = [(rows, V), (cols, D)]
        t = {"a": _up(legs, np.concatenate([b.ravel(order="F") for _, b in blocks]))}
    elif kind == "eigsolve":
        left, right, v, edge, ends = _chain_inputs(c, seed)
        W = _up(_W_LEGS, _w_flat(_W_LEGS))
        L, R = _up(edge[0], ends[0]), _up(edge[1], ends[1])
        for s in left:
            L = mg.mpsupdateleft(L, _up(*s), W)
        for s in reversed(right):
            R = mg.mpsupdateright(R, _up(*s), W)
        t = {"v": _up(*v), "L": L, "R": R, "W": W}
    else:
        mps = dmrg.mps_from_host(dmrg.random_mps_host(c["length"], c["length"] // 2,
                                                      max(2, c["chi"] // 8), seed=1911 + int(seed)))
        dmrg.center_at(mps, 1, normalize=True)
        Ws = dmrg.xxz_u1mpo(c["length"], 1.0)
        t = {"As": mps.As, "Ws": Ws, "env": dmrg.initialenv(mps, Ws, 1)}
    t["c"] = dict(c)
    return t


class _Result:
    """The device buffer of a result tensor, as any array library may read it in place."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": (t.numel(),), "typestr": "<f8", "version": 3,
                                         "data": (t.device_ptr(), False), "strides": None}


def _out(t):
    return torch.as_tensor(_Result(t), device="cuda")


def run(state):
    t, c = state, state["c"]
    kind = c["kind"]
    if kind == "heff":
        return _out(t["op"](t["v"]))
    if kind == "energy":
        return _out(mg.applymps2site(t["v"], t["L"], t["R"], t["W"], t["W"], precision=c["precision"]))
    if kind == "env":
        if c["side"] == "left":
            return _out(mg.mpsupdateleft(t["L"], t["v"], t["W"], precision=c["precision"]))
        return _out(mg.mpsupdateright(t["R"], t["v"], t["W"], precision=c["precision"]))
    if kind == "tdvp":
        y = tdvp.apply1(t["ops"], t["cv"], t["cL"], t["cR"], t["W"])
        return [_out(y.re), _out(y.im)]
    if kind == "eigsolve":
        e, x, _ = mg.eigsolve_heff2(t["v"], t["L"], t["R"], t["W"], t["W"], precision=c["precision"])
        return {"value": e, "vector": _out(x)}
    if kind == "truncate":  # u and v are free in sign: a sweep uses s and the truncated tensor
        u, s, v = mg.svdtrunc(t["a"], maxdim=c["chi"], tol=1e-9, method=c["method"])
        return {"s": _out(s), "usv": _out(mg.matmul(mg.matmul(u, s, precision=0), v, precision=0))}
    mps = dmrg.MPState(t["As"], center=1)
    env = list(t["env"])
    energies = dmrg.dmrg2sitesweep(mps, t["Ws"], env, maxdim=c["chi"], tieband=1e-9)
    # the new state, up to the free signs of its bonds: the density matrix of its first site
    return {"energies": np.array(energies), "density": _out(mg.contract(
        mps.As[0], (-1, 1, -2), mg.dual(mps.As[0]), (-1, 2, -2)))}


# ---- the same in 64 bits, densely --------------------------------------------------------------------
def _apply2(v, L, R, W):
    t = torch.einsum("amx,astb->xmstb", L, v)
    t = torch.einsum("xmstb,mpns->xpntb", t, W)
    t = torch.einsum("xpntb,nqot->xpqob", t, W)
    return torch.einsum("xpqob,boy->xpqy", t, R)


def _apply1(v, L, R, W):
    t = torch.einsum("amx,asb->xmsb", L, v)
    t = torch.einsum("xmsb,mpns->xpnb", t, W)
    return torch.einsum("xpnb,bny->xpy", t, R)


def _left(E, A, W):
    t = torch.einsum("amx,asr->rsmx", E, A)
    t = torch.einsum("rsmx,mpns->rpnx", t, W)
    return torch.einsum("rpnx,xpy->rny", t, A)


def _right(E, A, W):
    t = torch.einsum("rmx,lsr->lsmx", E, A)
    t = torch.einsum("lsmx,npms->lpnx", t, W)
    return torch.einsum("lpnx,ypx->lny", t, A)


def _lanczos(f, x, kd=5, maxiter=8, tol=1e-7):
    """Lowest eigenvalue by thick-restart Lanczos, keeping 3/5 of the basis."""
    basis, H = [x / x.norm()], np.zeros((kd + 1, kd + 1))

    def step():
        w = f(basis[-1])
        for _ in range(2):
            for j, c in enumerate([float(torch.sum(b * w)) for b in basis]):
                w = w - c * basis[j]
                if j == len(basis) - 1:
                    H[j, j] += c
        return w, float(w.norm())

    w, beta = step()
    it, arrow = 1, False
    while True:
        k = len(basis)
        if k == kd or beta <= tol:
            d, u = np.linalg.eigh(H[:k, :k])
            if abs(beta * u[k - 1, 0]) <= tol or beta <= tol or it >= maxiter:
                return float(d[0])
            keep = max(1, 3 * kd // 5)
            basis = [sum(float(u[j, i]) * basis[j] for j in range(k)) for i in range(keep)]
            H[:] = 0
            for i in range(keep):
                H[i, i] = d[i]
                H[keep, i] = H[i, keep] = beta * u[k - 1, i]
            it, arrow, k = it + 1, True, keep
        if not arrow:
            H[k, k - 1] = H[k - 1, k] = beta
        arrow = False
        basis.append(w / beta)
        w, beta = step()


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("heff", "energy", "env", "tdvp"):
        legs, x = _contraction_inputs(c, seed)
        d = {k: _dense(x[k], legs[k]) for k in ("v", "L", "R", "W")}
        if kind in ("heff", "energy"):
            return _flat(_apply2(d["v"], d["L"], d["R"], d["W"]), legs["v"])
        if kind == "env":
            out, at = (_left, "R") if c["side"] == "left" else (_right, "L")
            y = out(d["L" if c["side"] == "left" else "R"], d["v"], d["W"])
            new = [(leg, not dual) for leg, dual in legs[at]]
            return _flat(y, new)
        for k in ("v", "L", "R"):
            d[k] = torch.complex(d[k], _dense(x[k + "i"], legs[k]))
        y = _apply1(d["v"], d["L"], d["R"], d["W"].to(torch.complex128))
        return [_flat(y.real, legs["v"]), _flat(y.imag, legs["v"])]
    if kind == "truncate":
        _, _, blocks = _theta_blocks(c, seed)
        svd = [np.linalg.svd(b, full_matrices=False) for _, b in blocks]
        keep = sorted(((s, k) for k, (_, ss, _) in enumerate(svd) for s in ss if s >= 1e-9),
                      reverse=True)[:c["chi"]]
        n = [sum(1 for _, k in keep if k == j) for j in range(len(svd))]
        return {"s": np.concatenate([np.diag(s[:r]).ravel() for (_, s, _), r in zip(svd, n) if r]),
                "usv": np.concatenate([((u[:, :r] * s[:r]) @ v[:r]).ravel(order="F")
                                       for (u, s, v), r in zip(svd, n)])}
    if kind == "eigsolve":
        left, right, v, edge, ends = _chain_inputs(c, seed)
        W = _dense(_w_flat(_W_LEGS), _W_LEGS)
        L, R = _dense(ends[0], edge[0]), _dense(ends[1], edge[1])
        for legs, a in left:
            L = _left(L, _dense(a, legs), W)
        for legs, a in reversed(right):
            R = _right(R, _dense(a, legs), W)
        return {"value": _lanczos(lambda y: _apply2(y, L, R, W), _dense(v[1], v[0])), "vector": None}
    return None


# ---- what a pass cannot do without -------------------------------------------------------------------
def _apply2_work(legs):
    v, L, R, W = legs["v"], legs["L"], legs["R"], legs["W"]
    bl, br = L[2], R[2]
    t1 = [bl, L[1], v[1], v[2], v[3]]
    t2 = [bl, (SITE, V), W[2], v[2], v[3]]
    t3 = [bl, (SITE, V), (SITE, V), W[2], v[3]]
    f = _flops(L, [0], v, [0]) + _flops(t1, [1, 2], W, [0, 3]) + _flops(t2, [2, 3], W, [0, 3]) + \
        _flops(t3, [3, 4], R, [1, 0])
    return f, 8.0 * (2 * _numel(v) + _numel(L) + _numel(R) + 2 * _numel(W))


def _env_work(legs, side):
    v, E, W = legs["v"], legs["L" if side == "left" else "R"], legs["W"]
    k = 0 if side == "left" else 2
    bond, new = v[k], v[2 - k]
    bra = (bond[0], not E[0][1])
    f = _flops(E, [0], v, [k])
    t1 = [new, v[1], E[1], bra]
    out = (BOND, E[1][1])
    f += _flops(t1, [1, 2], W, [3, 0 if side == "left" else 2])
    t2 = [new, (SITE, V), out, bra]
    dual = [(leg, not d) for leg, d in v]
    f += _flops(t2, [1, 3], dual, [1, k])
    return f, 8.0 * (_numel(E) + _numel(v) + _numel(W) + _numel([new, out, (new[0], not new[1])]))


def work(case):
    c, kind = case, case["kind"]
    if kind in ("heff", "energy"):
        f, b = _apply2_work(_legs(kind, c))
        return {"bytes": b, "flops": f}
    if kind == "env":
        f, b = _env_work(_legs(kind, c), c["side"])
        return {"bytes": b, "flops": f}
    if kind == "tdvp":
        legs = _legs(kind, c)
        v, L, R, W = legs["v"], legs["L"], legs["R"], legs["W"]
        t1 = [L[2], L[1], v[1], v[2]]
        t2 = [L[2], (SITE, V), W[2], v[2]]
        f = 4 * _flops(L, [0], v, [0]) + 2 * _flops(t1, [1, 2], W, [0, 3]) + \
            4 * _flops(t2, [2, 3], R, [1, 0])
        return {"bytes": 16.0 * (2 * _numel(v) + _numel(L) + _numel(R)) + 8.0 * _numel(W), "flops": f}
    if kind == "truncate":
        rows, cols = _theta_shape(c)
        n = [(d, cols[q]) for q, d in rows.items() if q in cols]
        f = sum(6.0 * max(a, b) * min(a, b) ** 2 for a, b in n)
        return {"bytes": 8.0 * sum(2 * a * b + min(a, b) ** 2 for a, b in n), "flops": f}
    if kind == "eigsolve":
        lx, half = c["length"], c["length"] // 2
        bond = [tuple(dmrg.binomial_bond_dims(lx, k, half, c["chi"])) for k in (half - 1, half + 1)]
        f, b = _apply2_work({"v": [(bond[0], V), (SITE, V), (SITE, V), (bond[1], D)],
                             "L": [(bond[0], D), (BOND, D), (bond[0], V)],
                             "R": [(bond[1], V), (BOND, V), (bond[1], D)], "W": _W_LEGS})
        return {"bytes": b, "flops": 19 * f}  # matvecs of 8 rounds of a 5-dimensional basis
    lx, half, f, b = c["length"], c["length"] // 2, 0.0, 0.0
    for k in range(1, lx):  # each bond twice: one ground-state solve and one energy
        bond = [tuple(dmrg.binomial_bond_dims(lx, j, half, c["chi"])) if 0 < j < lx else
                (((0, 1),) if j <= 0 else ((half, 1),)) for j in (k - 1, k + 1)]
        f1, b1 = _apply2_work({"v": [(bond[0], V), (SITE, V), (SITE, V), (bond[1], D)],
                               "L": [(bond[0], D), (BOND, D), (bond[0], V)],
                               "R": [(bond[1], V), (BOND, V), (bond[1], D)], "W": _W_LEGS})
        f, b = f + 2 * 20 * f1, b + 2 * 2 * b1
    return {"bytes": b, "flops": f}


def _theta_shape(c):
    rows, cols = {}, {}
    for q, d in _bond(c):
        for s, _ in SITE:
            rows[q + s] = rows.get(q + s, 0) + d
            cols[q - s] = cols.get(q - s, 0) + d
    return rows, cols
