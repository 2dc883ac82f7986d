"""The calls that a program built on this package makes, as timed cases.

A case is a dict of sizes and options; ``listed()`` names the standing ones,
``draw()`` gives others of the same ranges.  ``prepare`` builds what the
program holds before the call (basis, operator, plan, vectors), ``run`` is the
call, ``work`` counts what the call cannot do without, and ``exact`` gives the
same outputs from plain torch in 64 bits.

Every operator is a seeded model of the package's benchmark family: HO modes
with nb(l) = l+1, nq(l) = l+2, a quartic force field, and either a constant
kinetic operator (type 1) or the Q-dependent metric (type 10).
"""
import math

import numpy as np
import torch

from elvibrot_gb300 import MultiOp, ParamOp, Polynomial, SG4Basis, sub_TabOpPsi

DEV = "cuda"


def listed():
    return [
        # one vector of a triatomic's 3-D operator: the smallest call, latency alone
        dict(name="hpsi_3d_L6_t1", kind="hpsi", D=3, L=6, type=1, nrhs=1),
        # the 6-D benchmark: a Davidson block of 20 vectors, Q-dependent metric
        dict(name="hpsi_6d_L8_t10_20", kind="hpsi", D=6, L=8, type=10, nrhs=20),
        # the same operator on one host vector (a Fortran caller's sub_OpPsi: copies in and out)
        dict(name="hpsi_6d_L8_t10_host", kind="hpsi", D=6, L=8, type=10, nrhs=1, host=True),
        # the adjoint of a 5-D operator on 7 complex packets
        dict(name="hpsi_5d_L6_t10_adj", kind="hpsi", D=5, L=6, type=10, nrhs=7, cplx=True, adjoint=True),
        # few modes with long 1-D grids, and a volume element (Jac and rho grids), scaled as in Chebyshev
        dict(name="hpsi_4d_L9_t10_jac", kind="hpsi", D=4, L=9, type=10, nrhs=5, jac=True, scaled=True),
        # 8 packets of a 7-D constant-G operator: the large instances of an uneven batch
        dict(name="hpsi_7d_L7_t1_8c", kind="hpsi", D=7, L=7, type=1, nrhs=8, cplx=True),
        # more modes than the narrow kernels take, type 10, 3 packets
        dict(name="hpsi_8d_L5_t10_3c", kind="hpsi", D=8, L=5, type=10, nrhs=3, cplx=True),
        # two coupled electronic states
        dict(name="hpsi_6d_L5_2states", kind="hpsi", D=6, L=5, type=1, nrhs=2, cplx=True, nb0=2),
        # independent Hamiltonians of unequal size in one call, 8 packets each
        dict(name="multi_uneven", kind="multi", sizes="3x9 4x8 5x7 6x6 7x5 9x4", type=1, nrhs=8),
        # Chebyshev propagation of one packet, order 30 (a whole call)
        dict(name="cheby_4d_L7", kind="cheby", D=4, L=7, type=1, nrhs=1, npoly=30, nsteps=10),
        # the optimal-control gradient: forward and adjoint RK4 sweeps (a whole call)
        dict(name="oc_gradient_4d_L7", kind="oc", D=4, L=7, type=1, samples=30, nsub=10, checkpoint=12),
        # a 12-D operator whose fields do not stay resident: streamed slice by slice
        dict(name="streamed_12d_L4_t10", kind="hpsi", D=12, L=4, type=10, nrhs=4, cplx=True, budget_mib=4096),
    ]


#: No drawn case does more than this many flops (the largest listed one).
MOST_FLOPS = 1.5e11


def draw(rng):
    """One more case of the same ranges: operators of 2 to 9 modes on 1 to 32 columns, uneven batches,
    propagations and gradients of small systems, streamed operators of 10 to 12 modes."""
    while True:
        kind = rng.choice(["hpsi"] * 6 + ["multi", "cheby", "rk4", "oc", "streamed"])
        if kind == "hpsi":
            D = rng.randint(2, 9)
            c = dict(kind="hpsi", D=D, L=rng.randint(3, 11 - D // 2), type=rng.choice([1, 10]),
                     nrhs=int(round(math.exp(rng.uniform(0.0, math.log(32.0))))))
            c["cplx"] = rng.random() < 0.5
            if rng.random() < 0.25:
                c["adjoint"] = True
            if c["type"] == 10 and rng.random() < 0.25:
                c["jac"] = True
            if rng.random() < 0.2:
                c["nb0"] = rng.randint(2, 3)
            elif not c["cplx"] and not c.get("adjoint") and rng.random() < 0.3:
                c["host"] = True
            if not c.get("host") and rng.random() < 0.3:
                c["scaled"] = True
        elif kind == "multi":
            sizes = []
            for _ in range(rng.randint(2, 9)):
                D = rng.randint(3, 8)
                sizes.append("%dx%d" % (D, rng.randint(3, 11 - D)))
            c = dict(kind="multi", sizes=" ".join(sizes), type=1, nrhs=rng.randint(1, 8))
        elif kind == "cheby":
            c = dict(kind="cheby", D=rng.randint(2, 5), L=rng.randint(4, 8), type=1, nrhs=rng.randint(1, 6),
                     npoly=rng.randint(28, 40), nsteps=rng.randint(2, 12))
        elif kind in ("rk4", "oc"):
            c = dict(kind=kind, D=rng.randint(2, 4), L=rng.randint(4, 7), type=1, samples=rng.randint(8, 40),
                     nsub=rng.choice([8, 10, 12]))
            if kind == "oc":
                c["checkpoint"] = rng.randint(5, 20)
        else:
            c = dict(kind="hpsi", D=rng.randint(10, 12), L=rng.randint(2, 3), type=10, nrhs=rng.randint(1, 8),
                     cplx=True, budget_mib=rng.choice([256, 512]))
        if work(c)["flops"] <= MOST_FLOPS:
            return c


# ------------------------------------------------------------- index sets
_cache = {}


def _terms(D, L):
    """The Smolyak terms l (max(0, L-D+1) <= |l| <= L), first index fastest, with their weights."""
    key = ("terms", D, L)
    if key not in _cache:
        rows = []

        def rec(head, left):
            if len(head) == D:
                if L - sum(head) <= D - 1:
                    rows.append(tuple(reversed(head)))
                return
            for v in range(left + 1):
                rec(head + [v], left - v)
        rec([], L)
        _cache[key] = [(t, (-1) ** (L - sum(t)) * math.comb(D - 1, L - sum(t))) for t in rows]
    return _cache[key]


def _basis_size(D, L):
    return math.comb(D + L, D)


def _functions(D, L):
    """Packed functions n (sum n <= L), last index fastest, as an [N, D] array."""
    rows = []

    def rec(head, left):
        if len(head) == D:
            rows.append(head)
            return
        for v in range(left + 1):
            rec(head + [v], left - v)
    rec([], L)
    return np.array(rows, dtype=np.int64).reshape(-1, D)


def _term_flops(l, type_op, nb0):
    """Flops of one column on one term: the basis<->grid maps in their cheapest order and the grid operator."""
    nb, nq = [v + 1 for v in l], [v + 2 for v in l]
    q = math.prod(nq)
    order = sorted(range(len(l)), key=lambda i: (nq[i] - nb[i]) / (nb[i] * nq[i]))
    cur, f = list(nb), 0.0
    for i in order:
        rest = math.prod(cur) / cur[i]
        f += 4.0 * nb[i] * nq[i] * rest  # the two directions cost the same
        cur[i] = nq[i]
    f += 2.0 * nb0 * q
    if type_op == 10:
        f += 4.0 * q * sum(nq) + 2.0 * len(l) ** 2 * q
    else:
        f += 2.0 * q * sum(nq)
    return f


def _hpsi_work(D, L, type_op, cols, nb0=1, resident=True):
    key = ("work", D, L, type_op, nb0)
    if key not in _cache:
        _cache[key] = (sum(_term_flops(l, type_op, nb0) for l, _ in _terms(D, L)),
                       sum(math.prod(v + 2 for v in l) for l, _ in _terms(D, L)))
    flops, pts = _cache[key]
    b = 16.0 * _basis_size(D, L) * cols
    if resident:
        b += 8.0 * pts * (nb0 * nb0 + (D * D if type_op == 10 else 0))
    return {"bytes": b, "flops": flops * cols}


def _cols(case):
    return case["nrhs"] * (2 if case.get("cplx") else 1) * case.get("nb0", 1)


def work(case):
    kind = case["kind"]
    if kind == "hpsi":
        return _hpsi_work(case["D"], case["L"], case["type"], _cols(case), case.get("nb0", 1),
                          "budget_mib" not in case)
    if kind == "multi":
        ws = [_hpsi_work(*map(int, s.split("x")), case["type"], 2 * case["nrhs"]) for s in case["sizes"].split()]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    w = _hpsi_work(case["D"], case["L"], case["type"], 2 * case.get("nrhs", 1))
    if kind == "cheby":
        return {"bytes": w["bytes"], "flops": w["flops"] * case["npoly"] * case["nsteps"]}
    stages = 4 * case["samples"] * case["nsub"]
    n = stages if kind == "rk4" else 3 * stages  # the gradient: forward, recomputed forward, adjoint
    w0 = _hpsi_work(case["D"], case["L"], 0, 2)
    return {"bytes": w["bytes"], "flops": n * (w["flops"] + w0["flops"])}


# ------------------------------------------------------------------ models
def _model(D, seed, nb0=1):
    """omega, s and the force field (cubic c3, quartic c4 per channel pair) and the metric's slopes g."""
    r = np.random.default_rng(seed)
    omega = r.uniform(0.005, 0.02, D)
    s = omega ** 0.25
    wbar = omega.mean()
    i = np.arange(D)
    up3 = (i[:, None, None] <= i[None, :, None]) & (i[None, :, None] <= i[None, None, :])
    c3 = np.where(up3, r.normal(0.0, 0.01 * wbar, (nb0, nb0, D, D, D)), 0.0)
    c4 = np.where(i[:, None] <= i[None, :], r.normal(0.0, 0.01 * wbar, (nb0, nb0, D, D)), 0.0)
    c3, c4 = 0.5 * (c3 + c3.transpose(1, 0, 2, 3, 4)), 0.5 * (c4 + c4.transpose(1, 0, 2, 3))
    g = r.normal(0.0, 1.0 / math.sqrt(D), (D, D, D))
    G1 = 0.05 * 0.5 * (g + g.transpose(1, 0, 2)) * s
    a, b = r.normal(0.0, 1.0, D), np.triu(r.normal(0.0, 0.1, (D, D)))
    return dict(D=D, nb0=nb0, omega=omega, s=s, c3=c3, c4=c4, G1=G1, mu1=a, mu2=b)


def _poly_terms(D, idx_sets, coefs):
    expo = np.zeros((len(idx_sets), D), dtype=np.int32)
    for t, ids in enumerate(idx_sets):
        for k in ids:
            expo[t, k] += 1
    return Polynomial(np.array(coefs), expo)


def _v_poly(m):
    D, n, s = m["D"], m["nb0"], m["s"]
    sets = [(i, i) for i in range(D)]
    sets += [(i, j, k) for i in range(D) for j in range(i, D) for k in range(j, D)]
    sets += [(i, i, j, j) for i in range(D) for j in range(i, D)]
    rows = []
    for a in range(n):
        for b in range(n):
            row = [0.5 * m["omega"][i] * (a == b) for i in range(D)]
            row += [m["c3"][a, b, i, j, k] * s[i] * s[j] * s[k]
                    for i in range(D) for j in range(i, D) for k in range(j, D)]
            row += [m["c4"][a, b, i, j] * s[i] ** 2 * s[j] ** 2 for i in range(D) for j in range(i, D)]
            rows.append(row)
    return _poly_terms(D, sets, rows[0] if n == 1 else rows)


def _mu_poly(m):
    D, s = m["D"], m["s"]
    sets = [(i,) for i in range(D)] + [(i, j) for i in range(D) for j in range(i, D)]
    return _poly_terms(D, sets, [m["mu1"][i] * s[i] for i in range(D)] +
                       [m["mu2"][i, j] * s[i] * s[j] for i in range(D) for j in range(i, D)])


def _jac_rho(y):
    """Smooth volume factors of the dimensionless coordinates y [points, D] (torch or numpy)."""
    return 1.0 + 0.1 * y[:, 0] / (1.0 + y[:, 0] ** 2), 1.0 + 0.05 / (1.0 + y[:, -1] ** 2)


def _operator(m, basis, case):
    kw = {}
    if case.get("budget_mib"):
        kw["field_budget"] = case["budget_mib"] << 20
    if case["type"] == 1:
        return ParamOp(basis, 1, V_poly=_v_poly(m), F2=-0.5 * np.eye(m["D"]), **kw)
    if case.get("jac"):
        kw["Jac"], kw["sqRho"] = _jac_rho(basis.grid_points() * m["s"])
    return ParamOp(basis, 10, V_poly=_v_poly(m), G0=np.eye(m["D"]), G1=m["G1"], **kw)


def _basis(m, L):
    return SG4Basis(m["D"], L, scaleQ=m["s"], nb0=m["nb0"])


def _vectors(n, rows, cplx, seed):
    """(rows, n) column-normalised N(0, 1) vectors on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    v = torch.randn((rows, n), generator=g, device=DEV, dtype=torch.complex128 if cplx else torch.float64)
    return v / torch.linalg.vector_norm(v, dim=1, keepdim=True)


def _packets(D, L, rows, seed):
    """(rows, N) packets of a propagation: coefficients that fall off with the excitation."""
    n = torch.from_numpy(_functions(D, L).sum(1)).to(DEV)
    v = _vectors(len(n), rows, True, seed) * torch.exp(-1.0 * n)
    return v / torch.linalg.vector_norm(v, dim=1, keepdim=True)


def _bounds(D, L):
    """Bounds of the model spectra (hartree): frequencies sqrt(omega) <= 0.142, and room for the couplings."""
    return 0.0, 0.142 * (0.5 * D + L) * 1.3


def _field(samples, seed):
    return np.random.default_rng(seed).normal(0.0, 1e-2, samples)


E0_ESC = (0.1, 0.7)  # the scaled operator (H - E0)/Esc of a case with "scaled"
DT = 5.0             # a.u. per propagation step and field sample


def prepare(case, seed):
    kind = case["kind"]
    if kind == "multi":
        ops = []
        for k, sz in enumerate(case["sizes"].split()):
            D, L = map(int, sz.split("x"))
            m = _model(D, 1000 * seed + k)
            ops.append(_operator(m, _basis(m, L), case))
        psis = [_vectors(op.basis.nvec, case["nrhs"], True, seed + k) for k, op in enumerate(ops)]
        return dict(kind=kind, plan=MultiOp(ops, [case["nrhs"]] * len(ops), complex_=True), psis=psis,
                    outs=[torch.empty_like(p) for p in psis])
    m = _model(case["D"], seed, case.get("nb0", 1))
    basis = _basis(m, case["L"])
    op = _operator(m, basis, case)
    st = dict(kind=kind, op=op, case=case)
    if kind == "hpsi":
        st["psi"] = _vectors(basis.nvec, case["nrhs"], bool(case.get("cplx")), seed)
        if case.get("host"):
            st["psi"] = np.asfortranarray(st["psi"].cpu().numpy().T)
        else:
            st["out"] = torch.empty_like(st["psi"])
        return st
    st["psi"] = _packets(case["D"], case["L"], case.get("nrhs", 1), seed)
    if kind == "cheby":
        st["range"] = _bounds(case["D"], case["L"])
        return st
    st["psi"] = st["psi"][0].contiguous()
    st["target"] = _packets(case["D"], case["L"], 1, seed + 1)[0].contiguous()
    st["mu"] = ParamOp(basis, 0, V_poly=_mu_poly(m))
    st["E"] = _field(case["samples"], seed)
    st["E0"] = 0.5 * _bounds(case["D"], case["L"])[1]
    return st


def run(state):
    kind = state["kind"]
    if kind == "multi":
        state["plan"].hpsi(state["psis"], state["outs"])
        return state["outs"]
    op, case = state["op"], state["case"]
    if kind == "hpsi":
        e0, esc = E0_ESC if case.get("scaled") else (0.0, 1.0)
        if case.get("host"):
            return sub_TabOpPsi(state["psi"], op)
        return op.hpsi_dev(state["psi"], state["out"], E0=e0, Esc=esc, transpose=bool(case.get("adjoint")))
    if kind == "cheby":
        psi = state["psi"].clone()
        ac, _ = op.cheby_propagate(psi, *state["range"], DT, case["npoly"], case["nsteps"])
        return psi, ac
    if kind == "rk4":
        return op.rk4_field(state["mu"], state["E"], state["psi"].clone(), DT, E0=state["E0"], nsub=case["nsub"])
    return op.oc_gradient(state["mu"], state["E"], state["psi"], state["target"], DT, checkpoint=case["checkpoint"],
                          E0=state["E0"], nsub=case["nsub"])


# ------------------------------------------------- the same in plain torch
def _hermite(nb, nq, s):
    """1-D matrices of nb scaled HO functions on nq Gauss-Hermite points: y, basis->grid B, its weighted
    transpose W, and the grid derivatives d1, d2."""
    key = ("1d", nb, nq, s)
    if key not in _cache:
        x, _ = np.polynomial.hermite.hermgauss(nq)
        x = 0.5 * (x - x[::-1])
        for _ in range(2):  # Newton steps to full precision
            p = _psi(nq + 1, x)
            x = x - p[nq] / (math.sqrt(2.0 * nq) * p[nq - 1])
            x = 0.5 * (x - x[::-1])
        p = _psi(max(nb + 1, nq), x)
        w = 1.0 / (p[:nq] ** 2).sum(0) / s
        k = np.arange(nb)[:, None]
        low = np.vstack([np.zeros((1, nq)), p[: nb - 1]]) if nb > 1 else np.zeros((1, nq))
        d1 = np.sqrt(k / 2.0) * low - np.sqrt((k + 1) / 2.0) * p[1: nb + 1]
        d2 = (x ** 2 - (2 * k + 1)) * p[:nb]
        B = p[:nb].T * math.sqrt(s)
        inv = np.linalg.pinv(B)
        mats = [x, B, B.T * w, (d1.T * s * math.sqrt(s)) @ inv, (d2.T * s * s * math.sqrt(s)) @ inv]
        _cache[key] = [torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in mats]
    return _cache[key]


def _psi(n, x):
    p = [math.pi ** -0.25 * np.exp(-0.5 * x * x)]
    p.append(math.sqrt(2.0) * x * p[0])
    for k in range(1, n):
        p.append(math.sqrt(2.0 / (k + 1)) * x * p[k] - math.sqrt(k / (k + 1)) * p[k - 1])
    return np.array(p[: n + 1])


def _along(a, mat, axis):
    return torch.movedim(torch.tensordot(a, mat, dims=([axis], [1])), -1, axis)


def _v_exact(m, y, a, b):
    c3, c4 = (torch.from_numpy(np.ascontiguousarray(m[k][a, b])).to(DEV) for k in ("c3", "c4"))
    D = m["D"]
    v = torch.einsum("pi,pij,pj->p", y, (y @ c3.permute(2, 0, 1).reshape(D, D * D)).reshape(-1, D, D), y)
    v = v + torch.einsum("pi,ij,pj->p", y * y, c4, y * y)
    if a == b:  # 1/2 omega Q^2 with Q = y / s
        v = v + (y * y) @ torch.from_numpy(0.5 * m["omega"] / m["s"] ** 2).to(DEV)
    return v


def _apply_exact(m, L, type_op, x, adjoint=False, jac=False, v=_v_exact):
    """H x of real columns x [cols, nb0 * N]: every Smolyak term in turn, added up with TwoSum."""
    D, nb0 = m["D"], m["nb0"]
    N = x.shape[1] // nb0
    place = torch.full((L + 1,) * D, -1, dtype=torch.int64) if (L + 1) ** D <= 1 << 27 else None
    fun = _functions(D, L)
    if place is None:  # many modes: look packed functions up by a key instead of in a table
        base = (L + 1) ** np.arange(D, dtype=np.int64)
        keys = fun @ base
        order = np.argsort(keys)
        keys, order = torch.from_numpy(keys[order]).to(DEV), torch.from_numpy(order).to(DEV)
    else:
        place[tuple(torch.from_numpy(fun[:, i].copy()) for i in range(D))] = torch.arange(N)
        place = place.to(DEV)
    s = torch.from_numpy(m["s"]).to(DEV)
    G1 = torch.from_numpy(m["G1"]).to(DEV)
    hi, lo = torch.zeros_like(x), torch.zeros_like(x)
    xc = x.reshape(-1, nb0, N)
    for l, weight in _terms(D, L):
        mats = [_hermite(k + 1, k + 2, float(m["s"][i])) for i, k in enumerate(l)]
        nq = [k + 2 for k in l]
        ax = [torch.arange(k + 1, device=DEV) for k in l]
        if place is None:
            k = sum((a * int(base[i])).reshape([-1 if j == i else 1 for j in range(D)]) for i, a in enumerate(ax))
            idx = order[torch.searchsorted(keys, k.reshape(-1))]
        else:
            idx = place[: l[0] + 1]
            for i in range(1, D):
                idx = idx.narrow(i, 0, l[i] + 1)
            idx = idx.reshape(-1)
        cur = xc[:, :, idx].reshape(-1, *[k + 1 for k in l])  # [cols * nb0, n_1 .. n_D]
        for i in range(D):
            cur = _along(cur, mats[i][2].T.contiguous() if adjoint else mats[i][1], i + 1)
        y = torch.stack(torch.meshgrid(*[a[0] for a in mats], indexing="ij"), -1).reshape(-1, D)
        rows = cur.shape[0]
        f = cur.reshape(-1, nb0, y.shape[0])
        V = [[v(m, y, a, b) for b in range(nb0)] for a in range(nb0)]
        out = torch.stack([sum((V[b][a] if adjoint else V[a][b]) * f[:, b] for b in range(nb0))
                           for a in range(nb0)], 1).reshape(cur.shape)
        pick = (lambda a: a.T.contiguous()) if adjoint else (lambda a: a)
        if type_op == 1:
            for i in range(D):
                out = out - 0.5 * _along(cur, pick(mats[i][4]), i + 1)
        elif type_op == 10:
            J, R = _jac_rho(y) if jac else (None, None)
            first, last = (R, -0.5 / (J * R)) if jac else (None, None)
            if adjoint and jac:
                first, last = last, first
            z = cur if first is None else cur * first.reshape(nq)
            G = torch.eye(D, device=DEV, dtype=torch.float64) + torch.einsum("ijk,pk->pij", G1, y / s)
            phi = torch.stack([_along(z, pick(mats[j][3]), j + 1).reshape(rows, -1) for j in range(D)])
            U = torch.einsum("pij,jrp->irp", G, phi)
            if jac:
                U = U * J
            t = sum(_along(U[i].reshape(cur.shape), pick(mats[i][3]), i + 1) for i in range(D))
            out = out + (-0.5 * t if last is None else t * last.reshape(nq))
        for i in reversed(range(D)):
            out = _along(out, mats[i][1].T.contiguous() if adjoint else mats[i][2], i + 1)
        t = weight * out.reshape(xc.shape[0], nb0, -1)
        h = hi.reshape(xc.shape)[:, :, idx]
        sm = h + t
        bb = sm - h
        hi.reshape(xc.shape)[:, :, idx] = sm
        lo.reshape(xc.shape)[:, :, idx] += (h - (sm - bb)) + (t - bb)
    return hi + lo


def _apply_cplx(m, L, type_op, x, **kw):
    if not x.is_complex():
        return _apply_exact(m, L, type_op, x, **kw)
    n = x.shape[0]
    h = _apply_exact(m, L, type_op, torch.cat([x.real, x.imag]).contiguous(), **kw)
    return torch.complex(h[:n], h[n:])


def _dense(m, L, type_op, v=_v_exact):
    """H as a matrix: H e_k in its columns."""
    return _apply_exact(m, L, type_op, torch.eye(_basis_size(m["D"], L), device=DEV, dtype=torch.float64), v=v).T


def _mu_exact(m, y, a, b):
    lin, quad = torch.from_numpy(m["mu1"]).to(DEV), torch.from_numpy(m["mu2"]).to(DEV)
    return y @ lin + torch.einsum("pi,ij,pj->p", y, quad, y)


def exact(case, seed):
    kind = case["kind"]
    if kind == "multi":
        out = []
        for k, sz in enumerate(case["sizes"].split()):
            D, L = map(int, sz.split("x"))
            m = _model(D, 1000 * seed + k)
            out.append(_apply_cplx(m, L, case["type"], _vectors(_basis_size(D, L), case["nrhs"], True, seed + k)))
        return out
    D, L, nb0 = case["D"], case["L"], case.get("nb0", 1)
    m = _model(D, seed, nb0)
    if kind == "hpsi":
        x = _vectors(nb0 * _basis_size(D, L), case["nrhs"], bool(case.get("cplx")), seed)
        h = _apply_cplx(m, L, case["type"], x, adjoint=bool(case.get("adjoint")), jac=bool(case.get("jac")))
        if case.get("scaled"):
            h = (h - E0_ESC[0] * x) / E0_ESC[1]
        return h.cpu().numpy().T if case.get("host") else h
    H = _dense(m, L, case["type"]).to(torch.complex128)
    psi = _packets(D, L, case.get("nrhs", 1), seed)
    if kind == "cheby":
        step = torch.linalg.matrix_exp(-1j * DT * H)
        ac, cur = [(psi.conj() * psi).sum(1)], psi
        for _ in range(case["nsteps"]):
            cur = cur @ step.T
            ac.append((psi.conj() * cur).sum(1))
        return cur, torch.stack(ac).cpu().numpy()
    mu = _dense(m, L, 0, _mu_exact).to(torch.complex128)
    E = torch.from_numpy(_field(case["samples"], seed)).to(DEV).requires_grad_(kind == "oc")
    E0, h = 0.5 * _bounds(D, L)[1], DT / case["nsub"]
    H = H - E0 * torch.eye(len(H), device=DEV, dtype=torch.float64)
    phase = complex(math.cos(E0 * h), -math.sin(E0 * h))
    y = psi[0]

    def rate(v, e):
        return -1j * (H @ v - e * (mu @ v))
    for k in range(case["samples"]):
        for _ in range(case["nsub"]):
            k1 = rate(y, E[k])
            k2 = rate(y + 0.5 * h * k1, E[k])
            k3 = rate(y + 0.5 * h * k2, E[k])
            k4 = rate(y + h * k3, E[k])
            y = (y + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)) * phase
    if kind == "rk4":
        return y
    target = _packets(D, L, 1, seed + 1)[0]
    J = (target.conj() * y).sum().abs() ** 2
    J.backward()
    return float(J.detach()), E.grad.cpu().numpy()
