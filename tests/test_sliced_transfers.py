"""Transfers on the sliced views (rows sorted by length in windows, slices of 32 rows or of 8 or 4 rows with
several lanes each) against the scalar CSR products, in every value type and block size, where rows fill
the GPU (P from 32,768 rows, R from 4,096 and 16,384): odd row counts, a last slice that is not full, rows of
one to fifty blocks."""
import numpy as np
import pytest

from fhhos4_gb300 import hho

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-14, "df": 1e-13, "fp32": 2e-6}   # of the largest |R||r| or |x| + |P||e|


@pytest.mark.parametrize("precision", ["fp64", "df", "fp32"])
@pytest.mark.parametrize("dim,n,k", [(2, 112, 1), (2, 112, 2), (2, 106, 3), (3, 16, 1), (3, 16, 2), (3, 28, 1)])
def test_gpu_transfers_on_sliced_views(dim, n, k, precision):
    torch = pytest.importorskip("torch")
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    H = hho.Hierarchy(dim, n, k, max_levels=2)
    A, P, bs = H.A(0), H.P(0), H.block_size
    H.close()
    # a coarse operator of the right size that is cheap to invert: the transfers do not see it
    rng = np.random.default_rng(2)
    import scipy.sparse as sp
    top = P.shape[1]
    As, Ps = [A, sp.identity(top, format="csr") + sp.csr_matrix((top, top))], [P]
    # the dense limit of the coarsest level keeps large ones out: a third level of one block row
    nb = top // bs
    Q = sp.csr_matrix((np.ones(top), (np.arange(top), np.tile(np.arange(bs), nb))), shape=(top, bs))
    As.append(sp.identity(bs, format="csr"))
    Ps.append(Q)
    ctx = S.fcg_mg(As, Ps, bs, precision=precision, fused=False).Context()
    p0 = scalar_perm(ctx.permutation(0, A.shape[0] // bs), bs)
    p1 = scalar_perm(ctx.permutation(1, nb), bs)
    Pp = P.tocsr()[p0][:, p1]

    def put(v):
        if precision == "df":
            hi = v.astype(np.float32)
            return torch.tensor(np.stack([hi, (v - hi).astype(np.float32)], 1), device="cuda")
        return torch.tensor(v, dtype=torch.float64 if precision == "fp64" else torch.float32, device="cuda")

    def get(t):
        a = t.cpu().numpy().astype(np.float64)
        return a[:, 0] + a[:, 1] if precision == "df" else a

    rd, ed = put(rng.standard_normal(A.shape[0])), put(rng.standard_normal(top))
    r, e = get(rd), get(ed)
    out = torch.full_like(ed, float("nan"))
    torch.cuda.synchronize()   # the context has a stream of its own
    ctx.apply_internal(0, N.OP_RESTRICT, precision, rd.data_ptr(), None, out.data_ptr())
    scale = (abs(Pp).T @ np.abs(r)).max()
    assert np.abs(get(out) - Pp.T @ r).max() <= TOL[precision] * scale
    out = torch.full_like(rd, float("nan"))
    torch.cuda.synchronize()
    ctx.apply_internal(0, N.OP_PROLONG_ADD, precision, ed.data_ptr(), rd.data_ptr(), out.data_ptr())
    scale = np.abs(r).max() + (abs(Pp) @ np.abs(e)).max()
    assert np.abs(get(out) - (r + Pp @ e)).max() <= TOL[precision] * scale
    ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dim,n,k", [(2, 112, 1), (2, 106, 3), (3, 16, 1), (3, 16, 2)])
def test_gpu_prolongation_rounds_once_at_the_size_of_x(dim, n, k, precision):
    """x + P e with e a hundredth of x: P e is summed from zero and x added once, so an entry is off by half a unit
    in the last place of the result and the rounding of the row's m products, m u |P||e|, where summing from x on
    rounds m times at the size of x."""
    torch = pytest.importorskip("torch")
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    import scipy.sparse as sp
    H = hho.Hierarchy(dim, n, k, max_levels=2)
    A, P, bs = H.A(0), H.P(0).tocsr(), H.block_size
    H.close()
    top = P.shape[1]
    nb = top // bs
    Q = sp.csr_matrix((np.ones(top), (np.arange(top), np.tile(np.arange(bs), nb))), shape=(top, bs))
    ctx = S.fcg_mg([A, sp.identity(top, format="csr"), sp.identity(bs, format="csr")], [P, Q], bs, precision=precision,
                   fused=False).Context()
    p0 = scalar_perm(ctx.permutation(0, A.shape[0] // bs), bs)
    p1 = scalar_perm(ctx.permutation(1, nb), bs)
    rng = np.random.default_rng(4)
    dt = np.float64 if precision == "fp64" else np.float32
    x, e = rng.standard_normal(A.shape[0]).astype(dt), (0.01 * rng.standard_normal(top)).astype(dt)
    xd, ed = torch.tensor(x, device="cuda"), torch.tensor(e, device="cuda")
    out = torch.full_like(xd, float("nan"))
    torch.cuda.synchronize()
    ctx.apply_internal(0, N.OP_PROLONG_ADD, precision, ed.data_ptr(), xd.data_ptr(), out.data_ptr())
    Pp = P[p0][:, p1].tocsr()
    vals = Pp.data.astype(dt).astype(np.longdouble)   # the values as the view stores them
    terms = vals * e.astype(np.longdouble)[Pp.indices]
    full = np.diff(Pp.indptr) > 0

    def rows(t):
        s = np.zeros(Pp.shape[0], np.longdouble)
        s[full] = np.add.reduceat(t, Pp.indptr[:-1][full])
        return s

    ref, size = x.astype(np.longdouble) + rows(terms), rows(np.abs(terms))
    u = np.longdouble(2.0) ** (-53 if precision == "fp64" else -24)
    # a row's block columns hold bs products each, zeros of the blocks among them
    m = bs * 7
    err = np.abs(out.cpu().numpy().astype(np.longdouble) - ref)
    assert np.all(err <= (1 + u) * u * (np.abs(ref) + (m + 1) * size)), float((err / (u * np.abs(ref) + m * u * size)).max())
    ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "df", "fp32"])
@pytest.mark.parametrize("dim,n,k,p_lanes,r_lanes",
                         [(2, 96, 1, 0, 8), (2, 112, 1, 1, 8), (2, 112, 2, 1, 8), (2, 106, 3, 1, 8), (2, 160, 1, 1, 4),
                          (2, 160, 3, 1, 4), (3, 16, 1, 1, 8), (3, 24, 2, 1, 4), (3, 28, 1, 1, 4)])
def test_gpu_transfers_run_on_the_sliced_views_of_their_sizes(dim, n, k, p_lanes, r_lanes, precision):
    """The view that each size takes (P a thread per row from 32,768 rows, R four from 16,384 and eight from 4,096,
    CSR below), and R r, x + P e on it."""
    torch = pytest.importorskip("torch")
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    import scipy.sparse as sp
    H = hho.Hierarchy(dim, n, k, max_levels=2)
    A, P, bs = H.A(0), H.P(0).tocsr(), H.block_size
    H.close()
    top = P.shape[1]
    nb = top // bs
    Q = sp.csr_matrix((np.ones(top), (np.arange(top), np.tile(np.arange(bs), nb))), shape=(top, bs))
    ctx = S.fcg_mg([A, sp.identity(top, format="csr"), sp.identity(bs, format="csr")], [P, Q], bs, precision=precision,
                   fused=False).Context()
    info = ctx.view_info(0, precision)
    assert (info["p_lanes"], info["r_lanes"]) == (p_lanes, r_lanes)
    row = S.fcg_mg([A, sp.identity(top, format="csr"), sp.identity(bs, format="csr")], [P, Q], bs, precision=precision,
                   fused=False, gs_layout="row").Context()
    assert (row.view_info(0, precision)["p_lanes"], row.view_info(0, precision)["r_lanes"]) == (0, 0)
    rng = np.random.default_rng(2)
    pair = precision == "df"
    dt = torch.float64 if precision == "fp64" else torch.float32

    def put(v):
        return torch.tensor(np.stack([v.astype(np.float32), 0 * v.astype(np.float32)], 1) if pair else v, dtype=dt, device="cuda")

    def get(t):
        a = t.cpu().numpy().astype(np.float64)
        return a[:, 0] + a[:, 1] if pair else a

    p0 = scalar_perm(ctx.permutation(0, A.shape[0] // bs), bs)
    p1 = scalar_perm(ctx.permutation(1, nb), bs)
    Pp = P[p0][:, p1]
    rd, ed = put(rng.standard_normal(A.shape[0])), put(rng.standard_normal(top))
    out, aux = torch.full_like(ed, float("nan")), torch.full_like(rd, float("nan"))
    torch.cuda.synchronize()
    ctx.apply_internal(0, N.OP_RESTRICT, precision, rd.data_ptr(), None, out.data_ptr())
    ctx.apply_internal(0, N.OP_PROLONG_ADD, precision, ed.data_ptr(), rd.data_ptr(), aux.data_ptr())
    r, e = get(rd), get(ed)
    assert np.abs(get(out) - Pp.T @ r).max() <= TOL[precision] * (abs(Pp).T @ np.abs(r)).max()
    assert np.abs(get(aux) - (r + Pp @ e)).max() <= TOL[precision] * (np.abs(r).max() + (abs(Pp) @ np.abs(e)).max())
    ctx.close()
    row.close()


@pytest.mark.parametrize("dim,n,k", [(2, 160, 1), (2, 160, 3), (3, 16, 1), (3, 24, 2), (3, 28, 1)])
def test_gpu_restriction_in_pairs_rounds_as_with_a_warp_a_row(dim, n, k):
    """R r in pairs on the sliced view (four or eight lanes a row of 25 to 50 blocks) against the CSR form with a warp
    a row, both from the exact product of the same pairs: the root mean square error over the rows, relative to
    |R||r|, no more than 1.3 times (a restatement of both orders of summation gives 1.0 to 1.1, and 1.4 to 2.2 for
    running sums that are not normalised)."""
    torch = pytest.importorskip("torch")
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    import scipy.sparse as sp
    H = hho.Hierarchy(dim, n, k, max_levels=2)
    A, P, bs = H.A(0), H.P(0).tocsr(), H.block_size
    H.close()
    top = P.shape[1]
    nb = top // bs
    Q = sp.csr_matrix((np.ones(top), (np.arange(top), np.tile(np.arange(bs), nb))), shape=(top, bs))
    rng = np.random.default_rng(5)
    r = rng.standard_normal(A.shape[0])
    hi = r.astype(np.float32)
    lo = (r - hi).astype(np.float32)
    exact_r = hi.astype(np.longdouble) + lo.astype(np.longdouble)
    rms = {}
    for layout in ("auto", "row"):
        ctx = S.fcg_mg([A, sp.identity(top, format="csr"), sp.identity(bs, format="csr")], [P, Q], bs, precision="df",
                       fused=False, gs_layout=layout).Context()
        assert (ctx.view_info(0, "df")["r_lanes"] > 0) == (layout == "auto")
        p0 = scalar_perm(ctx.permutation(0, A.shape[0] // bs), bs)
        p1 = scalar_perm(ctx.permutation(1, nb), bs)
        R = P[p0][:, p1].T.tocsr()
        R.sort_indices()
        vh = R.data.astype(np.float32)
        vals = vh.astype(np.longdouble) + (R.data - vh).astype(np.float32).astype(np.longdouble)
        terms = vals * exact_r[R.indices]
        start = R.indptr[:-1]
        assert np.all(np.diff(R.indptr) > 0)
        ref, size = np.add.reduceat(terms, start), np.add.reduceat(np.abs(terms), start)
        rd = torch.tensor(np.stack([hi, lo], 1), device="cuda")
        out = torch.full((top, 2), float("nan"), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.apply_internal(0, N.OP_RESTRICT, "df", rd.data_ptr(), None, out.data_ptr())
        g = out.cpu().numpy().astype(np.longdouble)
        rms[layout] = float(np.sqrt(np.mean(((g[:, 0] + g[:, 1] - ref) / size) ** 2)))
        ctx.close()
    assert rms["auto"] <= 1.3 * rms["row"], rms
