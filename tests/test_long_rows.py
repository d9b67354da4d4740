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
