"""The items in block fixed point (sg4_fixed.cuh), at the sizes and values where
they can go wrong, against the oracle: the smallest and largest terms and 1-D
grids, odd numbers of columns, metrics that are not symmetric or spread too far
for one exponent, steep potentials, and columns that the FP64 code takes over.

The tolerance is the parity tolerance of every H.psi test (1e-12): each stage
keeps 2^-55 of its largest value, a term runs at most 2 D + 3 <= 27 stages, and
the alternating Smolyak weights amplify a term's error by less than 10^3.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from elvibrot_gb300 import ParamOp, Polynomial, SG4Basis, SG4Tables, sub_TabOpPsi
from elvibrot_gb300.configs import make_model, random_psi
from oracle.oracle import OracleSG4, oracle_tables

from test_gpu_parity import gpu_apply, oracle_for, rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-12


def need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("D,L,type_op,nrhs", [
    (1, 0, 10, 1), (1, 9, 10, 3), (1, 14, 1, 2),      # one mode: nq 2 to 16
    (2, 14, 10, 2), (3, 13, 1, 3), (2, 0, 1, 5),      # the longest 1-D grids, the smallest terms
    (4, 6, 10, 5), (5, 5, 10, 1), (6, 5, 10, 2),      # tiles of 32 points left partly empty
    (7, 5, 10, 3), (9, 3, 10, 2), (12, 2, 10, 3),     # more modes than the register-resident sizes
    (12, 2, 1, 2), (11, 3, 1, 1)])
def test_fixed_point_matches_oracle(D, L, type_op, nrhs):
    need_cuda()
    m = make_model(D, L, type_op, 900 + 17 * D + L)
    O, kw = oracle_for(m)
    psi = random_psi(O.N, nrhs, 3)
    e = rel_err(gpu_apply(m.operator(), psi), O.hpsi(psi, **kw))
    print(f"D={D} L={L} type {type_op} nrhs={nrhs}: {e:.2e}")
    assert e <= TOL


def _grid_problem(D, L, seed):
    b = SG4Basis(D, L, scaleQ=np.full(D, 0.4))
    O = OracleSG4(D, L, L, 1, 1, 2, 1, scaleQ=np.full(D, 0.4))
    return b, O, np.random.default_rng(seed)


def test_metric_that_is_not_symmetric_and_its_transpose():
    need_cuda()
    b, O, rng = _grid_problem(5, 4, 11)
    V, G = rng.normal(size=b.sum_nq), rng.normal(size=b.sum_nq * 25)
    op = ParamOp(b, 10, V=V, G=G)
    psi = random_psi(b.N, 3, 5)
    H = O.hpsi(np.eye(b.N), type_op=10, V=V, G=G)
    assert rel_err(gpu_apply(op, psi), H @ psi) <= TOL
    P = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    out = torch.empty_like(P)
    op.hpsi_dev(P, out, transpose=True)
    assert rel_err(out.cpu().numpy().T, H.T @ psi) <= TOL


@pytest.mark.parametrize("case", ["metric", "potential", "type0"])
def test_fields_with_a_wide_range(case):
    """A metric spread over 2^20 inside a term, and potentials that grow by 10^8 or
    more towards the edge of the grid."""
    need_cuda()
    b, O, rng = _grid_problem(4, 6, 12)
    r = np.abs(b.grid_points() * 0.4).max(axis=1)
    G = rng.normal(size=b.sum_nq * 16) * 0.1 if case != "metric" else \
        np.exp(rng.uniform(-7.0, 7.0, size=b.sum_nq * 16))
    V = rng.normal(size=b.sum_nq) if case == "metric" else np.exp(6.0 * r * r)
    t = 0 if case == "type0" else 10
    kw = dict(V=V) if t == 0 else dict(V=V, G=G)
    psi = random_psi(b.N, 3, 6)
    assert rel_err(gpu_apply(ParamOp(b, t, **kw), psi), O.hpsi(psi, type_op=t, **kw)) <= TOL


@pytest.mark.parametrize("type_op", [1, 10])
def test_scaled_and_exceptional_columns(type_op):
    """H (2^k x) = 2^k H x to the bit (one exponent per column), to rounding where
    the FP64 code takes the column; a column that is not finite, or far from the
    others in scale, leaves the others' bits alone."""
    need_cuda()
    m = make_model(4, 5, type_op, 31)
    op = m.operator()
    psi = random_psi(op.basis.N, 4, 8)
    ref = gpu_apply(op, psi)
    for k in (-250, -30, 1, 250):
        assert np.array_equal(gpu_apply(op, np.ldexp(psi, k)), np.ldexp(ref, k))
    for k in (-600, -310, 310, 600):
        assert rel_err(np.ldexp(gpu_apply(op, np.ldexp(psi, k)), -k), ref) <= TOL
    mixed = psi.copy()
    mixed[:, 0] = np.ldexp(psi[:, 0], 700)
    mixed[:, 2] = 0.0
    mixed[3, 3] = np.inf
    got = gpu_apply(op, mixed)
    assert np.array_equal(got[:, 1], ref[:, 1])
    assert rel_err(np.ldexp(got[:, 0], -700), ref[:, 0]) <= TOL
    assert np.all(got[:, 2] == 0.0)
    assert not np.all(np.isfinite(got[:, 3]))
    mixed[3, 3] = np.nan
    got = gpu_apply(op, mixed)
    assert np.array_equal(got[:, 1], ref[:, 1]) and np.isnan(got[:, 3]).any()


def test_complex_pair_shares_an_item():
    need_cuda()
    m = make_model(5, 4, 10, 33)
    op = m.operator()
    psi = random_psi(op.basis.N, 3, 9, complex_=True)
    P = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    got = sub_TabOpPsi(P, op).cpu().numpy().T
    assert np.array_equal(got.real, gpu_apply(op, np.ascontiguousarray(psi.real)))
    assert np.array_equal(got.imag, gpu_apply(op, np.ascontiguousarray(psi.imag)))


@pytest.mark.parametrize("D,L,terms", [(1, 14, 5), (2, 14, 40), (3, 9, 70), (7, 3, 200)])
def test_polynomial_fields_match_grids(D, L, terms):
    """V from its monomials (tables over two halves of the modes: one mode, the
    longest grids, more factors than a table holds) and a metric that is affine
    and not symmetric, against the same fields given as grids; H^T as well."""
    need_cuda()
    b, O, rng = _grid_problem(D, L, 13)
    Q = b.grid_points()
    expo = rng.integers(0, 4, size=(terms, D)) * (rng.random((terms, D)) < min(1.0, 3.0 / D))
    poly = Polynomial(rng.normal(size=terms) * 0.1 ** expo.sum(axis=1), expo.astype(np.int32))
    G0, G1 = np.eye(D) + 0.1 * rng.normal(size=(D, D)), 0.02 * rng.normal(size=(D, D, D))
    nq = np.prod(b.tables()[0] + 2, axis=1)
    off = np.concatenate([[0], np.cumsum(nq)])
    g = G0 + np.einsum("ijk,pk->pij", G1, Q)
    G = np.concatenate([g[off[t]:off[t + 1]].transpose(1, 2, 0).ravel() for t in range(len(nq))])
    P = torch.from_numpy(np.ascontiguousarray(random_psi(b.N, 2, 4).T)).cuda()
    for tr in (False, True):
        outs = []
        for kw in (dict(V_poly=poly, G0=G0, G1=G1), dict(V=poly(Q), G=G)):
            out = torch.empty_like(P)
            ParamOp(b, 10, **kw).hpsi_dev(P, out, transpose=tr)
            outs.append(out.cpu().numpy())
        assert rel_err(outs[0], outs[1]) <= TOL


@pytest.mark.parametrize("nrhs", [2, 3, 5, 33, 70])
def test_sums_do_not_depend_on_the_number_of_columns(nrhs):
    """The accumulation groups columns (one, two, or four a block): every column has
    the bits of its own call, with lists from one term to all of them."""
    need_cuda()
    op = make_model(4, 6, 1, 41).operator()
    psi = random_psi(op.basis.N, nrhs, 10)
    got = gpu_apply(op, psi)
    for j in {0, 1, nrhs - 1}:
        assert np.array_equal(got[:, j], gpu_apply(op, psi[:, j:j + 1])[:, 0])


@pytest.mark.parametrize("D,nb,nq", [(5, 16, 16), (4, 16, 16)])
def test_long_grids_on_both_sides_of_the_shared_memory_bound(D, nb, nq):
    """One term of D long 1-D grids: the five modes' matrices (3840 values) do not
    fit in a fixed-point CTA, the four modes' ones (3072) do."""
    need_cuda()
    b = SG4Basis(D, 0, A_nb=nb, A_nq=nq, scaleQ=np.full(D, 0.5))
    O = OracleSG4(D, 0, 0, nb, 0, nq, 0, scaleQ=np.full(D, 0.5))
    Q = O.grid_points()
    V, F2 = 0.1 * (Q * Q).sum(axis=1), -0.5 * np.eye(D)
    psi = random_psi(b.N, 1, 21)
    assert rel_err(gpu_apply(ParamOp(b, 1, V=V, F2=F2), psi), O.hpsi(psi, type_op=1, V=V, F2=F2)) <= TOL


@pytest.mark.parametrize("type_op", [1, 10])
def test_subnormal_columns_and_blocks(type_op):
    """A column that has decayed below 2^-1022 beside a normal one, as a real column
    and as one part of a complex one; terms whose entries are all subnormal beside a
    normal function that they do not hold; a block with one subnormal entry.  H is
    linear, so the results are those of the scaled vectors, to the spacing of the
    subnormal numbers (2^-1074) times the values that a result adds."""
    need_cuda()
    m = make_model(4, 5, type_op, 31)
    op = m.operator()
    psi = random_psi(op.basis.N, 3, 8)
    ref = gpu_apply(op, psi)
    tiny = np.ldexp(1.0, -1074)
    x = psi.copy()
    x[:, 0] = np.ldexp(psi[:, 0], -1040)                      # 2^-1040: 34 bits left
    exact = np.ldexp(x[:, 0], 1040)                           # what those bits hold
    got = gpu_apply(op, x)
    assert np.array_equal(got[:, 1:], ref[:, 1:])
    assert np.max(np.abs(np.ldexp(got[:, 0], 1040) - gpu_apply(op, exact[:, None])[:, 0])) <= 1e5 * np.ldexp(tiny, 1040)
    z = psi[:, :1] + 1j * x[:, :1]
    P = torch.from_numpy(np.ascontiguousarray(z.T)).cuda()
    h = sub_TabOpPsi(P, op).cpu().numpy().T
    assert np.array_equal(h.real, ref[:, :1]) and np.max(np.abs(h.imag)) < 1e-300
    # one normal entry in the last function, 1e-310 elsewhere: H e_last everywhere
    last = np.zeros((op.basis.N, 1))
    last[-1] = 1.0
    y = np.where(last == 0.0, 1e-310, last)
    assert np.max(np.abs(gpu_apply(op, y) - gpu_apply(op, last))) < 1e-300
    one = np.zeros((op.basis.N, 1))
    one[0] = tiny
    assert np.max(np.abs(gpu_apply(op, one))) <= 1e5 * tiny


# ------------------------------------------------------------- smooth vectors
def _smooth_vectors(n):
    """Columns that fall off with the excitation sum(n), and one that does not: N(0, 1)
    entries times exp(-a sum(n)), the lowest function, a displaced ground state."""
    rng = np.random.default_rng(1)
    s = n.sum(axis=1)
    r = rng.normal(size=len(s))
    fact = np.cumprod(np.concatenate([[1.0], np.arange(1.0, n.max() + 1)]))
    cols = [r, r * np.exp(-1.0 * s), r * np.exp(-3.0 * s), r * np.exp(-6.0 * s), (s == 0) * 1.0,
            np.prod(0.7 ** n / np.sqrt(fact[n]), axis=1)]
    return np.stack([c / np.linalg.norm(c) for c in cols], axis=1)


def _metric(kind, Q, nq):
    """GGiq(iq, j, i) per term of the identity times a factor of the point."""
    D = Q.shape[1]
    f = 1.0 + 0.05 * Q.sum(axis=1) if kind == "affine" else np.exp(kind * (Q * Q).sum(axis=1))
    off = np.concatenate([[0], np.cumsum(nq)])
    return np.concatenate([(np.eye(D)[:, :, None] * f[a:b]).ravel() for a, b in zip(off[:-1], off[1:])])


POTENTIALS = {
    "none": None,
    "harmonic": lambda y: 0.5 * (y * y).sum(axis=1),
    "quartic": lambda y: 0.5 * (y * y).sum(axis=1) + 0.1 * (y ** 4).sum(axis=1),
    "morse": lambda y: ((1.0 - np.exp(-0.8 * y)) ** 2).sum(axis=1) / 1.28,
    "wall": lambda y: np.exp(0.3 * (y * y).sum(axis=1)),
}


def _errors_in_both_arithmetics(D, L, type_op, pot, rules=(1, 1, 2, 1), metric="affine"):
    """2-norm errors of each column against the long-double oracle, in fixed point and
    from the FP64 items, which the same operator with a vanishing F1 term (types 0 and
    1) or a unit Jacobian grid (type 10) keeps."""
    O = OracleSG4(D, L, L, *rules)
    T = SG4Tables(**oracle_tables(O))
    tab_l, _, _, packed = O.tables()
    Q, psi = O.grid_points(), _smooth_vectors(packed - 1)
    kw = {} if POTENTIALS[pot] is None else dict(V=POTENTIALS[pot](Q))
    if type_op == 1:
        kw["F2"] = (-0.5 * np.eye(D)).ravel()
    if type_op == 10:
        kw["G"] = _metric(metric, Q, np.prod(tab_l * rules[3] + rules[2], axis=1))
    ref = O.hpsi(psi, type_op=type_op, extended=True, **kw)
    twin = dict(Jac=np.ones(O.sum_nq)) if type_op == 10 else dict(F1=np.full(D, 1e-300))
    ops = ParamOp(T, type_op, **kw), ParamOp(T, 10 if type_op == 10 else 1, **kw, **twin)
    return [np.linalg.norm(gpu_apply(op, psi) - ref, axis=0) / np.linalg.norm(ref, axis=0) for op in ops]


def _no_less_precise(*args, **kw):
    """Fixed point is no further from the exact result than the FP64 items: on the
    geometric mean over the columns, and to a factor of four on any one of them (two
    sums of rounding errors, each known to about a factor of two; half an ulp of the
    result at least)."""
    fx, f64 = _errors_in_both_arithmetics(*args, **kw)
    r = np.maximum(fx, 2.0 ** -54) / np.maximum(f64, 2.0 ** -54)
    print(args, kw, "fixed point / FP64:", np.round(r, 2), "mean %.2f" % np.exp(np.log(r).mean()))
    assert np.exp(np.log(r).mean()) <= 1.0
    assert r.max() <= 4.0


@pytest.mark.parametrize("D,L,type_op,pot", [
    (4, 8, 0, "harmonic"), (4, 8, 10, "harmonic"),   # one rounding shared by a term
    (2, 13, 1, "none"), (2, 13, 1, "harmonic"), (3, 10, 1, "harmonic"),   # low and high levels in one sum
    (2, 13, 0, "harmonic"), (2, 13, 10, "harmonic"), (3, 8, 10, "quartic"),   # passes of many inputs
])
def test_smooth_vectors_keep_their_digits(D, L, type_op, pot):
    need_cuda()
    _no_less_precise(D, L, type_op, pot)


@pytest.mark.parametrize("D,L,rules,type_op,pot", [
    (2, 13, (1, 1, 2, 1), 0, "wall"), (2, 13, (1, 1, 2, 1), 1, "wall"), (2, 13, (1, 1, 2, 1), 1, "morse"),
    (2, 13, (1, 1, 2, 1), 10, "wall"), (3, 10, (1, 1, 2, 1), 1, "wall"), (3, 10, (1, 1, 2, 1), 10, "morse"),
    (1, 14, (1, 1, 2, 1), 1, "wall"), (1, 14, (1, 1, 2, 1), 10, "morse"),         # a single term
    (2, 0, (14, 1, 14, 1), 1, "wall"), (2, 0, (14, 1, 14, 1), 10, "morse")])
def test_potentials_that_the_tails_of_x_carry(D, L, rules, type_op, pot):
    """V large where x is small: the columns that fixed point would lose digits on go
    through the FP64 code, one or both of an item's two."""
    need_cuda()
    _no_less_precise(D, L, type_op, pot, rules=rules)


@pytest.mark.parametrize("D,L,slope,pot", [(2, 13, 0.12, "harmonic"), (2, 13, 0.04, "harmonic"), (3, 10, 0.12, "none")])
def test_metrics_that_grow_towards_the_edge(D, L, slope, pot):
    """G = exp(slope r^2), up to a hundred times its value at the centre: one exponent
    a term leaves the centre's elements that many fewer bits."""
    need_cuda()
    _no_less_precise(D, L, 10, pot, metric=slope)


@pytest.mark.parametrize("nrhs", [1, 2, 3])
@pytest.mark.parametrize("nb,nq", [(3, 4), (4, 5), (5, 6)])
def test_exceptional_columns_of_terms_around_the_shared_memory(nb, nq, nrhs):
    """A term whose arrays fit a CTA's shared memory twice, once, or not at all (4-D type
    10: 5 nq^4 values of 3776), with a column that the FP64 code takes, alone or as one
    or both of a pair."""
    need_cuda()
    b = SG4Basis(4, 0, A_nb=nb, A_nq=nq, scaleQ=np.full(4, 0.5))
    V = np.random.default_rng(nq).normal(size=b.sum_nq)
    op = ParamOp(b, 10, V=V, G0=np.eye(4), G1=np.zeros((4, 4, 4)))
    psi = random_psi(b.N, nrhs, 17)
    ref = gpu_apply(op, psi)
    for far in ([0], [nrhs - 1], list(range(nrhs))):
        x = psi.copy()
        x[:, far] = np.ldexp(x[:, far], 700)
        got = gpu_apply(op, x)
        near = [j for j in range(nrhs) if j not in far]
        assert np.array_equal(got[:, near], ref[:, near])
        assert rel_err(np.ldexp(got[:, far], -700), ref[:, far]) <= TOL


def _remainder(n):
    """n values of both signs, a hundred at a time of sizes down to 2^-59, that cancel but for 2^-108."""
    rng = np.random.default_rng(n)
    x = np.ldexp(rng.integers(1, 1 << 53, size=n).astype(np.float64), -53 - rng.integers(0, 7, size=n))
    return np.concatenate([x, -x[rng.permutation(n)], [2.0 ** -108]]).tolist()


@pytest.mark.parametrize("values,result", [
    ([1.0, -1.0, 2.0 ** -110], 2.0 ** -110),
    ([2.0 ** -115, 1.0, -1.0], 2.0 ** -115),
    ([1.0, 2.0 ** -60, 2.0 ** -110, -1.0, -2.0 ** -60], 2.0 ** -110),
    ([3.0, -2.0 ** -90, 5.0, -8.0, 2.0 ** -90, -2.0 ** -112] + [0.0] * 60, -2.0 ** -112),
    ([1.0, 2.0 ** -50, -1.0], 2.0 ** -50), ([0.0, -0.0], 0.0),
    (_remainder(255), 2.0 ** -108), (_remainder(256), 2.0 ** -108), (_remainder(2000), 2.0 ** -108)])
@pytest.mark.parametrize("nrhs", [1, 2, 5])
def test_sums_of_terms_that_cancel(values, result, nrhs):
    """One function held by one term per value, on one point each: H.psi is the sum of the
    weights times psi, here a remainder far below the terms that cancel, and above
    2^-116 of the largest (2^-113 in lists of up to 4096), where the sums are exact."""
    need_cuda()
    n = len(values)
    w = np.sign(values) + (np.asarray(values) == 0.0)
    one = np.ones(1)
    T = SG4Tables(1, 0, 0, [1], [1], np.zeros(1), one, one, np.zeros(1), np.zeros(1), np.zeros(n, dtype=np.int32),
                  w, np.ones(n, dtype=np.int32), 1)
    op = ParamOp(T, 0, V=np.abs(values))
    psi = np.ldexp(1.0, np.arange(nrhs))[None, :]
    assert np.array_equal(gpu_apply(op, psi), result * psi)


def test_slabs_of_large_terms_stay_within_their_limit():
    """One term of 8^6 points, type 10: two columns of 7 arrays take 29 MB a CTA, 31 GB on
    seven CTAs an SM.  The plan takes single columns, and no more CTAs than items; every
    column has the bits of a call on a few."""
    need_cuda()
    b = SG4Basis(6, 0, A_nb=2, A_nq=8, scaleQ=np.full(6, 0.5))
    V = np.random.default_rng(6).normal(size=b.sum_nq)
    op = ParamOp(b, 10, V=V, G0=np.eye(6), G1=np.zeros((6, 6, 6)))
    P = torch.randn((1300, b.N), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda",
                    dtype=torch.float64)
    few, out = torch.empty_like(P[:3]), torch.empty_like(P)
    free = [torch.cuda.mem_get_info()[0]]
    for x, y in ((P[:3].contiguous(), few), (P, out)):
        op.hpsi_dev(x, y)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    array = 8 * 7 * 8 ** 6
    assert free[0] - free[1] <= 6 * array + (64 << 20)      # three items
    assert free[0] - free[2] <= (16 << 30) + (64 << 20)
    assert torch.equal(out[:3], few)
    x = np.ascontiguousarray(P[:3].cpu().numpy().T)
    G = np.concatenate([np.repeat(np.eye(6).ravel(), b.sum_nq)])
    O = OracleSG4(6, 0, 0, 2, 0, 8, 0, scaleQ=np.full(6, 0.5))
    assert rel_err(few.cpu().numpy().T, O.hpsi(x, type_op=10, V=V, G=G)) <= TOL
