"""Sweeps over long rows (Galerkin coarse operators, 25 to 130 blocks a row, in up to 60 colours) against the
oracle in FP64 and colour order, on every level and in every value type: the three widths of the
long-row kernel (32, 64 and 128 threads a row), rows shorter and longer than those, colours of one row."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# norm-wise: a few hundred products a row in FP64 (2^-53), pairs (2^-47), FP32 (2^-24)
TOL = {"fp64": 1e-12, "df": 1e-11, "fp32": 1e-4}


@pytest.fixture(scope="module", params=[(2, 48, 1, "lognormal_patches"), (2, 36, 2, "lognormal_patches"),
                                        (2, 48, 3, "lognormal_patches"), (3, 16, 1, "anisotropic"),
                                        (3, 8, 2, "checkerboard")], ids=str)
def hierarchy(request):
    from fhhos4_gb300 import hho
    dim, n, k, coefficient = request.param
    H = hho.Hierarchy(dim, n, k, coefficient=coefficient, contrast=100.0, checker_blocks=8 if dim == 2 else 4)
    A0, Ps, bs = H.A(0), [H.P(l) for l in range(H.levels - 1)], H.block_size
    H.close()
    As = [A0.tocsr()]
    for P in Ps:
        As.append((P.T @ As[-1] @ P).tocsr())
    return As, Ps, bs


@pytest.mark.parametrize("precision", ["fp64", "df", "fp32"])
def test_gpu_long_row_sweeps(hierarchy, precision):
    torch = pytest.importorskip("torch")
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    As, Ps, bs = hierarchy
    ctx = S.fcg_mg(As, Ps, bs, precision=precision, galerkin=True).Context()
    rng = np.random.default_rng(3)
    for l in range(1, len(As) - 1):
        rows = As[l].shape[0]
        assert ctx.level_info(l)["blocks"] / ctx.level_info(l)["block_rows"] > 18   # the long-row kernel's rows
        s = scalar_perm(ctx.permutation(l, rows // bs), bs)
        Ap = O.as_csr(As[l][s][:, s])
        x, b = rng.standard_normal(rows).astype(np.float32), rng.standard_normal(rows).astype(np.float32)

        def put(v):
            v = v.astype(np.float64)
            if precision == "df":
                return torch.tensor(np.stack([v, 0 * v], 1).astype(np.float32), device="cuda")
            return torch.tensor(v, dtype=torch.float64 if precision == "fp64" else torch.float32, device="cuda")

        xd, bd = put(x), put(b)
        out = torch.empty_like(xd)
        for op, backward in ((N.OP_GS_FORWARD, False), (N.OP_GS_BACKWARD, True)):
            ctx.apply_internal(l, op, precision, xd.data_ptr(), bd.data_ptr(), out.data_ptr())
            g = out.cpu().numpy().astype(np.float64)
            g = g[:, 0] + g[:, 1] if precision == "df" else g
            ref = O.block_gs(Ap, bs, b.astype(np.float64), x.astype(np.float64), backward=backward)
            assert np.linalg.norm(g - ref) <= TOL[precision] * np.linalg.norm(ref), (l, op)
    ctx.close()


def _block_sor(A, bs, b, x, omega, backward):
    """Block SOR row by row in FP64."""
    A = A.tobsr((bs, bs))
    A.sort_indices()
    y = x.reshape(-1, bs).copy()
    rhs = b.reshape(-1, bs)
    rows = range(len(y))
    for i in reversed(rows) if backward else rows:
        lo, hi = A.indptr[i], A.indptr[i + 1]
        cols, vals = A.indices[lo:hi], A.data[lo:hi]
        off = cols != i
        t = rhs[i] - np.einsum("prc,pc->r", vals[off], y[cols[off]])
        y[i] = omega * np.linalg.solve(vals[~off][0], t) + (1.0 - omega) * y[i]
    return y.ravel()


def _put(torch, v, precision):
    v = v.astype(np.float64)
    if precision == "df":
        return torch.tensor(np.stack([v, 0 * v], 1).astype(np.float32), device="cuda")
    return torch.tensor(v, dtype=torch.float64 if precision == "fp64" else torch.float32, device="cuda")


def _get(t, precision):
    g = t.cpu().numpy().astype(np.float64)
    return g[:, 0] + g[:, 1] if precision == "df" else g


@pytest.mark.parametrize("precision", ["fp64", "df", "fp32"])
def test_gpu_long_row_sor(hierarchy, precision):
    """omega = 1.3, forward and backward, on the coarse levels."""
    torch = pytest.importorskip("torch")
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    As, Ps, bs = hierarchy
    ctx = S.fcg_mg(As, Ps, bs, precision=precision, galerkin=True, omega=1.3).Context()
    rng = np.random.default_rng(13)
    for l in range(1, len(As) - 1):
        rows = As[l].shape[0]
        s = scalar_perm(ctx.permutation(l, rows // bs), bs)
        Ap = O.as_csr(As[l][s][:, s])
        x, b = rng.standard_normal(rows).astype(np.float32), rng.standard_normal(rows).astype(np.float32)
        xd, bd = _put(torch, x, precision), _put(torch, b, precision)
        out = torch.empty_like(xd)
        for op, backward in ((N.OP_GS_FORWARD, False), (N.OP_GS_BACKWARD, True)):
            ctx.apply_internal(l, op, precision, xd.data_ptr(), bd.data_ptr(), out.data_ptr())
            ref = _block_sor(Ap, bs, b.astype(np.float64), x.astype(np.float64), 1.3, backward)
            assert np.linalg.norm(_get(out, precision) - ref) <= TOL[precision] * np.linalg.norm(ref), (l, op)
    ctx.close()


def _band(nb, radius, bs, rng):
    """A block operator whose row i holds the blocks |i - j| <= radius (radius + 1 colours of equal size), diagonally
    dominant."""
    import scipy.sparse as sp
    j = np.arange(nb)[:, None] + np.arange(-radius, radius + 1)[None, :]
    keep = (j >= 0) & (j < nb)
    data = rng.uniform(-1, 1, (int(keep.sum()), bs, bs)) / (4 * radius * bs)
    data[(j == np.arange(nb)[:, None])[keep]] += np.eye(bs)
    indptr = np.concatenate([[0], np.cumsum(keep.sum(1))])
    return sp.bsr_matrix((data, j[keep], indptr), shape=(nb * bs, nb * bs)).tocsr()


@pytest.mark.parametrize("precision", ["fp64", "df", "fp32"])
@pytest.mark.parametrize("nb,radius,bs", [(176000, 17, 2), (900, 17, 6), (1500, 40, 3), (1501, 70, 4)])
def test_gpu_long_row_sweeps_of_bands(nb, radius, bs, precision):
    """Rows of 35, 81 and 141 blocks. The first: colours of 9,777 rows (above 9,728), a warp a row longer than the
    warp. A sweep from x, and from zero through the cycle (P of zeros: the coarse correction vanishes), whose first
    sweep leaves out the columns not yet set."""
    torch = pytest.importorskip("torch")
    import scipy.sparse as sp
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    from test_gpu_parity import scalar_perm
    rng = np.random.default_rng(17)
    A = _band(nb, radius, bs, rng)
    n = A.shape[0]
    P = sp.csr_matrix((np.zeros(n), (np.arange(n), np.tile(np.arange(bs), nb))), shape=(n, bs))
    for pre in ("bgs", "rbgs"):
        ctx = S.fcg_mg([A, sp.identity(bs, format="csr")], [P], bs, precision=precision, pre=pre, nu=(1, 0)).Context()
        assert ctx.level_info(0)["colours"] == radius + 1
        assert ctx.view_info(0, precision)["classes"] == 0
        s = scalar_perm(ctx.permutation(0, nb), bs)
        Ap = O.as_csr(A[s][:, s])
        x, b = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
        xd, bd = _put(torch, x, precision), _put(torch, b, precision)
        out = torch.empty_like(xd)
        op = N.OP_GS_FORWARD if pre == "bgs" else N.OP_GS_BACKWARD
        ctx.apply_internal(0, op, precision, xd.data_ptr(), bd.data_ptr(), out.data_ptr())
        ref = O.block_gs(Ap, bs, b.astype(np.float64), x.astype(np.float64), backward=pre == "rbgs")
        assert np.linalg.norm(_get(out, precision) - ref) <= TOL[precision] * np.linalg.norm(ref)
        r = np.empty(n)
        r[s] = b
        z = ctx.apply(0, N.OP_VCYCLE, r, None, n)
        ref = O.block_gs(Ap, bs, b.astype(np.float64), np.zeros(n), backward=pre == "rbgs")
        assert np.linalg.norm(z[s] - ref) <= TOL[precision] * np.linalg.norm(ref)
        ctx.close()
