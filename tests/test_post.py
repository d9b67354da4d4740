"""Post-processing of a face solution (cell-unknown recovery, k+1 reconstruction, L2 error;
Diffusion_HHO.h:855-912 and :120-150): the generator's element tables evaluated in numpy reproduce
the host L2 error (which test_generator.py pins against the reference's own L2Error), the C ABI
validates its tables before any device call, and the GPU pass gives the host's cell unknowns and
L2 error."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse.linalg as sla

from fhhos4_gb300 import hho

CASES = [(3, 6, 1), (2, 16, 2), (3, 4, 2)]


def _solved(dim, n, k):
    H = hho.Hierarchy(dim, n, k)
    x = sla.spsolve(H.A(0).tocsc(), H.b())
    return H, x


def numpy_post(t, x):
    """Cell unknowns and relative L2 error of the reconstruction from the element tables."""
    dim, ne, nC, nFF, nR, nq = (t[k] for k in ("dim", "n_elements", "n_cell", "n_face_dofs", "n_recon", "n_points"))
    nF = dim + 1
    nf = nFF // nF
    cls = t["elem_class"]
    faces = t["elem_faces"].reshape(ne, nF)
    xf = np.zeros((ne, nFF))
    xb = x.reshape(-1, nf)
    for lf in range(nF):
        g = faces[:, lf]
        m = g >= 0
        xf[m, lf * nf:(lf + 1) * nf] = xb[g[m]]
    xc = t["cell_rhs"].reshape(ne, nC) + np.einsum("eij,ej->ei", t["solve_cells"].reshape(-1, nC, nFF)[cls], xf)
    coef = np.einsum("eij,ej->ei", t["recon"].reshape(-1, nR, nC + nFF)[cls], np.concatenate([xc, xf], 1))
    uh = np.einsum("eqi,ei->eq", t["basis"].reshape(-1, nq, nR)[cls], coef)
    X = t["elem_centre"].reshape(ne, 3)[:, None, :] + t["offsets"].reshape(-1, nq, 3)[cls]
    u = np.prod(np.sin(np.pi * X[:, :, :dim]), axis=2)
    W = t["weights"].reshape(-1, nq)[cls]
    return xc, float(np.sqrt((W * (uh - u) ** 2).sum()) / np.sqrt((W * u * u).sum()))


@pytest.mark.parametrize("dim,n,k", CASES)
def test_tables_reproduce_host_l2_error(dim, n, k):
    H, x = _solved(dim, n, k)
    try:
        t = H.post_tables()
        assert t["n_classes"] < t["n_elements"]   # translated elements share their tables
        _, err = numpy_post(t, x)
        assert err == pytest.approx(H.l2_error(x), rel=1e-11)
    finally:
        H.close()


def test_post_create_validates_tables():
    """Bad tables are refused with FHG_ERR_INVALID_ARG / FHG_ERR_UNSUPPORTED before any device call."""
    from fhhos4_gb300 import _native as N
    H = hho.Hierarchy(2, 4, 1)
    t = H.post_tables()
    H.close()
    bad = dict(t)
    bad["elem_class"] = t["elem_class"].copy()
    bad["elem_class"][3] = t["n_classes"]
    with pytest.raises(N.FhgError) as e:
        N.Post(bad)
    assert e.value.code == N.FHG_ERR_INVALID_ARG and "class" in str(e.value)
    big = dict(t, n_points=100000)
    with pytest.raises(N.FhgError) as e:
        N.Post(big)
    assert e.value.code == N.FHG_ERR_UNSUPPORTED


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n,k", CASES)
def test_gpu_post_matches_host(dim, n, k):
    import torch
    from fhhos4_gb300 import _native as N
    H, x = _solved(dim, n, k)
    try:
        t = H.post_tables()
        host_err = H.l2_error(x)
    finally:
        H.close()
    xc_ref, _ = numpy_post(t, x)
    post = N.Post(t)
    try:
        xd = torch.tensor(x, device="cuda")
        cells = torch.zeros(t["n_elements"] * t["n_cell"], dtype=torch.float64, device="cuda")
        err, ms = post.run(xd.data_ptr(), cells.data_ptr(), "sine")
        assert ms > 0
        assert err == pytest.approx(host_err, rel=1e-11)
        xc = cells.cpu().numpy().reshape(xc_ref.shape)
        assert np.abs(xc - xc_ref).max() <= 1e-12 * np.abs(xc_ref).max()
        # cell unknowns only
        cells.zero_()
        none, _ = post.run(xd.data_ptr(), cells.data_ptr(), "none")
        assert none is None
        assert np.abs(cells.cpu().numpy().reshape(xc_ref.shape) - xc).max() == 0.0
        # the same launch twice: the fixed-order reduction gives the same bits
        err2, _ = post.run(xd.data_ptr(), 0, "sine")
        assert err2 == err
    finally:
        post.close()


@pytest.mark.gpu
def test_gpu_post_of_gpu_solve():
    """The whole path on the device: FCG + V-cycle solve of the 3D sine problem, then its L2 error,
    equal to the host's evaluation of the same x."""
    import torch
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    H = hho.Hierarchy(3, 8, 1)
    try:
        As = [H.A(l) for l in range(H.levels)]
        Ps = [H.P(l) for l in range(H.levels - 1)]
        b = H.b()
        s = S.fcg_mg(As, Ps, H.block_size, precision="fp32")
        x = s.Solve(b)
        t = H.post_tables()
        host_err = H.l2_error(x)
    finally:
        H.close()
    post = N.Post(t)
    try:
        err, _ = post.run(torch.tensor(x, device="cuda").data_ptr(), 0, "sine")
        assert err == pytest.approx(host_err, rel=1e-11)
        assert 1e-4 < err < 1e-2   # the discretisation error of 8^3, k = 1
    finally:
        post.close()


@pytest.mark.gpu
@pytest.mark.parametrize("tables", ["shared", "distinct"])
@pytest.mark.parametrize("dim,n,k", [(2, 8, 1), (2, 12, 1), (2, 9, 2), (2, 12, 3), (3, 3, 1), (3, 4, 1), (3, 4, 2), (3, 4, 3)])
def test_gpu_post_with_factorised_and_pointwise_tables(dim, n, k, tables):
    """Both forms of the L2 sums against numpy at the points, for every element size: "shared" tables
    are factorised; "distinct" ones (another rule of weights per element) are factorised up to 256 of them
    (2D n = 8 and n = 9, 3D n = 3) and evaluated at the points above. Face values far from a solution, so
    nothing cancels: 1e-12 covers the rounding of sums of a few 10^4 positive terms."""
    import torch
    from fhhos4_gb300 import _native as N
    H = hho.Hierarchy(dim, n, k, max_levels=1)
    try:
        t = H.post_tables()
        rows = H.A_rows(0)
    finally:
        H.close()
    ne, nq = t["n_elements"], t["n_points"]
    rng = np.random.default_rng(11)
    if tables == "distinct":
        cls = t["elem_class"]
        for name, m in (("solve_cells", t["n_cell"] * t["n_face_dofs"]),
                        ("recon", t["n_recon"] * (t["n_cell"] + t["n_face_dofs"])), ("offsets", nq * 3),
                        ("basis", nq * t["n_recon"]), ("weights", nq)):
            t[name] = t[name].reshape(-1, m)[cls].copy()
        t["weights"] *= 1.0 + 1e-3 * np.arange(ne)[:, None]
        t["n_classes"], t["elem_class"] = ne, np.arange(ne, dtype=np.int32)
    x = rng.standard_normal(rows)
    xc_ref, err_ref = numpy_post(t, x)
    post = N.Post({k_: (v.ravel() if isinstance(v, np.ndarray) else v) for k_, v in t.items()})
    try:
        cells = torch.zeros(ne * t["n_cell"], dtype=torch.float64, device="cuda")
        err, _ = post.run(torch.tensor(x, device="cuda").data_ptr(), cells.data_ptr(), "sine")
    finally:
        post.close()
    assert np.abs(cells.cpu().numpy().reshape(xc_ref.shape) - xc_ref).max() <= 1e-12 * np.abs(xc_ref).max()
    assert err == pytest.approx(err_ref, rel=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n,k,tables", [(2, 16, 1, None), (3, 6, 1, None), (3, 6, 2, None), (3, 2, 3, 31), (3, 2, 1, 32),
                                            (3, 3, 1, 33), (2, 12, 1, 288), (2, 96, 2, 33), (2, 96, 1, 200)])
def test_gpu_post_factorises_on_the_first_exact_run_where_that_repays(dim, n, k, tables):
    """Quadrature tables are factorised by the first run with an exact solution, not at set-up and not for the cell
    unknowns alone, and only where they are few (32) or have 512 elements each; both forms against numpy at the
    points. `tables`: that many rules of weights in turn (None: the mesh's own few). 1e-12: sums of positive terms."""
    import torch
    from fhhos4_gb300 import _native as N
    H = hho.Hierarchy(dim, n, k, max_levels=1)
    try:
        t = H.post_tables()
        rows = H.A_rows(0)
    finally:
        H.close()
    ne, nq = t["n_elements"], t["n_points"]
    if tables:   # every element of one geometry, so that the weights alone tell the tables apart
        cls = np.zeros(ne, np.int32)
        for name, m in (("solve_cells", t["n_cell"] * t["n_face_dofs"]), ("recon", t["n_recon"] * (t["n_cell"] + t["n_face_dofs"])),
                        ("offsets", nq * 3), ("basis", nq * t["n_recon"]), ("weights", nq)):
            t[name] = np.repeat(t[name].reshape(-1, m)[:1], tables, axis=0)
        t["weights"] *= 1.0 + 1e-3 * np.arange(tables)[:, None]
        t["n_classes"], t["elem_class"] = tables, (cls + np.arange(ne) % tables).astype(np.int32)
    expect = (tables or t["n_classes"]) if not tables or tables <= 32 or ne >= 512 * tables else 0
    x = np.random.default_rng(3).standard_normal(rows)
    xc_ref, err_ref = numpy_post(t, x)
    post = N.Post({k_: (v.ravel() if isinstance(v, np.ndarray) else v) for k_, v in t.items()})
    try:
        assert post.factors() == 0
        xd = torch.tensor(x, device="cuda")
        cells = torch.zeros(ne * t["n_cell"], dtype=torch.float64, device="cuda")
        post.run(xd.data_ptr(), cells.data_ptr(), "none")
        assert post.factors() == 0
        assert np.abs(cells.cpu().numpy().reshape(xc_ref.shape) - xc_ref).max() <= 1e-12 * np.abs(xc_ref).max()
        err, _ = post.run(xd.data_ptr(), 0, "sine")
        assert 0 < post.factors() <= expect if expect else post.factors() == 0
        assert tables is None or post.factors() == expect
        assert err == pytest.approx(err_ref, rel=1e-12)
        assert post.run(xd.data_ptr(), 0, "sine")[0] == err
    finally:
        post.close()
