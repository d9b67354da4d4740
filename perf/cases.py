"""Performance cases of fhhos4_gb300: what a program that solves HHO face systems has it do.

Most cases are whole solves, one per kind of call that the framework's own configurations, tests and
benchmark make: the default FP64 method through ``Solve`` on host arrays, the pair and FP32 V-cycles on
device arrays, Galerkin coarse operators on heterogeneous coefficients, the p-multigrid, the learned
FP32 method at the benchmark's size, and many uneven problems in one batched solve. The others are the
steps around the solve: one application of the preconditioner, condensation and assembly of the system,
and post-processing of its solution.

A program sets a hierarchy up once and solves for many right-hand sides, so ``prepare`` keeps the
hierarchies of this process (bounded) and draws the right-hand side (for the condensation: the
coefficients and element sources; for the post-processing: the face solution) from the seed.
"""
import ctypes
from collections import OrderedDict

import numpy as np
import torch

from fhhos4_gb300 import _native as N
from fhhos4_gb300 import batch as BT
from fhhos4_gb300 import hho
from fhhos4_gb300 import learned as LN
from fhhos4_gb300 import solver as S

MAXIT = 200


def _solve(name, **kw):
    case = dict(name=name, kind="solve", dim=3, n=16, k=1, coefficient="identity", contrast=1.0, precision="fp64",
                nu=1, coarse_nu=-1, galerkin=False, p_multigrid=False, learned=False, autotune=False, tol=1e-8, io="device")
    case.update(kw)
    return case


def listed():
    return [
        # the smallest call: default options, host arrays, a 2D problem whose launches are all short
        _solve("solve2d_n32_k1_fp64", dim=2, n=32, k=1, io="host"),
        # one problem of the batched configuration on its own: log-uniform coefficient on patches,
        # Galerkin coarse operators, 4 x 4 blocks, FP32 V-cycle
        _solve("solve2d_n144_k3_fp32", dim=2, n=144, k=3, coefficient="lognormal_patches", contrast=1e3, galerkin=True,
               precision="fp32"),
        # p-multigrid (face blocks 6 -> 3, then the h-levels), FP64-class pair V-cycle
        _solve("solve3d_n16_k2_pmg_df", n=16, k=2, p_multigrid=True, precision="df"),
        # the reference's method as it is called by default: FP64 everywhere, host arrays
        _solve("solve3d_n32_k1_fp64", n=32, io="host"),
        # rotated anisotropic tensors with Galerkin coarse operators (rows of many blocks on the coarse levels)
        _solve("solve3d_n24_k1_aniso_df", n=24, coefficient="anisotropic", galerkin=True, precision="df"),
        # face blocks of 6 in FP32 with two smoothing steps, a size between powers of two
        _solve("solve3d_n24_k2_fp32", n=24, k=2, precision="fp32", nu=2, io="host"),
        # the FP64-class plain method on a mid-size system, launch shapes timed at setup
        _solve("solve3d_n48_k1_df", n=48, precision="df", autotune=True),
        # the benchmark's headline: 9.4 M unknowns, FP32 fast cycle with the learned step
        _solve("solve3d_n64_k1_learned", n=64, precision="fp32", nu=3, coarse_nu=4, learned=True, autotune=True),
        # many independent 2D problems of uneven size in one batched solve, right-hand sides and
        # solutions on the host
        dict(name="batch2d_24", kind="batch", problems=24, n_max=96, precision="fp32", spec_seed=20261203),
        # one application of the FP32 preconditioner, as an outer Krylov method of a caller's own uses it
        dict(name="precond3d_n32_k1_fp32", kind="precond", dim=3, n=32, k=1, nu=1, precision="fp32"),
        # static condensation and assembly of a 48^3 system (4 M unknowns)
        dict(name="condense3d_n48_k1", kind="condense", dim=3, n=48, k=1),
        # cell unknowns and L2 error of a 32^3 solution
        dict(name="post3d_n32_k1", kind="post", dim=3, n=32, k=1),
    ]


def _pick_n(rng, dim, top):
    """A mesh size that the geometric coarsening takes down to a small coarsest level: m * 2^j."""
    sizes = {3: [8, 12, 16, 24, 32, 48], 2: [o << j for o in (5, 6, 7, 8, 9, 10, 11, 13) for j in (2, 3, 4)]}[dim]
    sizes = sorted(s for s in sizes if s <= top)
    lo, hi = np.log(sizes[0]), np.log(sizes[-1])
    at = np.exp(lo + (hi - lo) * rng.random())
    return min(sizes, key=lambda s: abs(np.log(s / at)))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["solve"] * 7 + ["batch", "precond", "condense", "post"])
    if kind == "batch":
        return dict(kind="batch", problems=rng.randint(2, 32), n_max=16 * rng.randint(3, 6),
                    precision=rng.choice(["fp32", "df", "fp64"]), spec_seed=rng.randint(1, 10 ** 6))
    dim = rng.choice([2, 3, 3])
    k = rng.choice([1, 2, 3]) if dim == 2 else rng.choice([1, 1, 2])
    n = _pick_n(rng, dim, 208 if dim == 2 else 48 if k == 1 else 24)
    if kind == "precond":
        return dict(kind="precond", dim=dim, n=n, k=k, nu=rng.choice([1, 2, 3]), precision=rng.choice(["fp32", "df", "fp64"]))
    if kind in ("condense", "post"):   # no hierarchy below the mesh: any size
        lo, hi = (12, 256) if dim == 2 else (6, 48 if k == 1 else 24)
        return dict(kind=kind, dim=dim, n=int(round(lo * (hi / lo) ** rng.random())), k=k)
    case = _solve("", dim=dim, n=n, k=k, precision=rng.choice(["fp64", "df", "fp32"]), nu=rng.choice([1, 1, 2, 3]),
                  io=rng.choice(["host", "device"]), autotune=rng.random() < 0.25, tol=rng.choice([1e-6, 1e-7, 1e-8, 1e-8, 1e-9]))
    del case["name"]
    if case["nu"] == 3:
        case["coarse_nu"] = 4
    style = rng.choice(["identity", "identity", "coefficient", "p_multigrid" if k > 1 else "learned"])
    if style == "coefficient":
        case["coefficient"] = "lognormal_patches" if dim == 2 else "anisotropic" if k == 1 else "checkerboard"
        case["contrast"] = {"lognormal_patches": 1e3, "anisotropic": 1.0, "checkerboard": 1e2}[case["coefficient"]]
        case["galerkin"] = True
        if dim == 3:
            case["n"] = min(n, 24 if k == 1 else 16)
            case["precision"] = "df"
    elif style == "p_multigrid":
        case.update(p_multigrid=True, nu=1, coarse_nu=-1, n=min(n, 64 if dim == 2 else 24))
    elif style == "learned" and dim == 3:
        case.update(learned=True, precision="fp32", nu=3, coarse_nu=4)
    return case


# ---------------------------------------------------------------------------------------------------
# hierarchies kept by this process

_kept = OrderedDict()


def _keep(key, make):
    """make() once per key; the least recently used beyond 24 are let go (their contexts free the GPU)."""
    if key in _kept:
        _kept.move_to_end(key)
    else:
        _kept[key] = make()
        while len(_kept) > 24:
            _kept.popitem(last=False)
    return _kept[key]


def _key(case, *extra):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "io"))) + extra


def _checker_blocks(coefficient):
    return 8 if coefficient == "lognormal_patches" else 4


def _loads(dim, n, k, coefficient, contrast, seed):
    """Right-hand sides of the sources of one problem (sine, constant, random sine modes), scaled to norm 1."""
    out = []
    for source in ("sine", "one", "modes"):
        H = hho.Hierarchy(dim, n, k, max_levels=1, source=source, coefficient=coefficient, contrast=contrast,
                          checker_blocks=_checker_blocks(coefficient), seed=seed)
        b = H.b()
        H.close()
        out.append(b / np.linalg.norm(b))
    return np.stack(out)


def _mix(loads, seed):
    """A source of the same kind: a random combination of the loads."""
    c = np.random.default_rng(seed).standard_normal(len(loads))
    return c @ loads


def _hierarchy(case):
    """(A_0.., P_0.., block size(s), coarse smoothing) of a solve or preconditioner case."""
    if case.get("p_multigrid"):
        As, Ps, _, bss, cnu = hho.generate_p(case["dim"], case["n"], case["k"], "mg")
        return As, Ps, bss, cnu
    coefficient = case.get("coefficient", "identity")
    H = hho.Hierarchy(case["dim"], case["n"], case["k"], coefficient=coefficient, contrast=case.get("contrast", 1.0),
                      checker_blocks=_checker_blocks(coefficient))
    As = [H.A(l) for l in range(H.levels)]
    Ps = [H.P(l) for l in range(H.levels - 1)]
    bs = H.block_size
    tensors = H.face_tensors(0) if case.get("learned") else None
    H.close()
    c = case.get("coarse_nu", -1)
    return As, Ps, bs, (c, c), tensors


def _solver(case):
    def make():
        As, Ps, bs, cnu = (got := _hierarchy(case))[:4]
        solver = S.fcg_mg(As, Ps, bs, tol=case.get("tol", 1e-8), maxit=MAXIT, precision=case["precision"], nu=(case["nu"], case["nu"]),
                          coarse_nu=cnu, galerkin=case.get("galerkin", False), autotune=case.get("autotune", False),
                          replace_residual=case.get("galerkin", False))
        if case.get("learned"):
            solver.Context().set_face_tensors(got[4])
            solver.Context().set_learned(LN.load_params(LN.DEFAULT_WEIGHTS)[0], "fallback")
        loads = None
        if case["kind"] == "solve":
            loads = _loads(case["dim"], case["n"], case["k"], case["coefficient"], case["contrast"], 20261203)
        return solver, loads, As[0].shape[0]
    return _keep(_key(case), make)


class _DeviceArray:
    """A device buffer of the library as torch sees it; the tensor made from it keeps the owner alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(owner, ptr, n, typestr):
    return torch.as_tensor(_DeviceArray(owner, ptr, n, typestr), device="cuda")


# ---------------------------------------------------------------------------------------------------
# prepare and run, by kind

def _prepare_solve(case, seed):
    solver, loads, n = _solver(case)
    b = _mix(loads, seed)
    if case["io"] == "host":
        return dict(kind="solve", io="host", solver=solver, b=b)
    bd = torch.from_numpy(b).cuda()
    return dict(kind="solve", io="device", solver=solver, b=bd, x=torch.empty_like(bd))


def _run_solve(s):
    if s["io"] == "host":
        return {"x": s["solver"].Solve(s["b"])}
    ctx = s["solver"].Context()
    rc, _, _ = ctx.solve_device(s["b"].data_ptr(), s["x"].data_ptr(), MAXIT)
    ctx._check(rc)
    return {"x": s["x"]}


def _prepare_precond(case, seed):
    solver, _, n = _solver(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    if case["precision"] == "fp32":
        r = r.float()
    elif case["precision"] == "df":
        hi = r.float()
        r = torch.stack([hi, (r - hi.double()).float()], dim=1).contiguous()
    return dict(kind="precond", ctx=solver.Context(), precision=case["precision"], r=r, z=torch.empty_like(r))


def _run_precond(s):
    s["ctx"].apply_internal(0, N.OP_VCYCLE, s["precision"], s["r"].data_ptr(), None, s["z"].data_ptr())
    return {"z": s["z"]}


def _specs(case):
    return BT.batched_specs(case["problems"], seed=case["spec_seed"], n_max=case["n_max"])


def _batch(case):
    def make():
        specs = _specs(case)
        probs, batch, _ = BT.build(specs, precision=case["precision"])
        return probs, batch, [_loads(2, p.spec.n, p.spec.k, "lognormal_patches", 1e3, p.spec.seed) for p in probs]
    return _keep(_key(case), make)


def _prepare_batch(case, seed):
    probs, batch, loads = _batch(case)
    return dict(kind="batch", probs=probs, batch=batch, b=[_mix(l, seed + 1000 * i) for i, l in enumerate(loads)])


def _run_batch(s):
    for p, b in zip(s["probs"], s["b"]):
        p.ctx.io_upload(b)
    rc, _, _ = s["batch"].solve()
    s["batch"]._check(rc)
    return [p.x() for p in s["probs"]]


def _tables(case, which):
    def make():
        H = hho.Hierarchy(case["dim"], case["n"], case["k"], max_levels=1)
        t = H.condense_tables() if which == "condense" else H.post_tables()
        H.close()
        return t
    return _keep(("tables", which, case["dim"], case["n"], case["k"]), make)


def _condense_inputs(case, seed):
    """The tables with a coefficient per class and a source per element drawn from the seed."""
    t = dict(_tables(case, "condense"))
    rng = np.random.default_rng(seed)
    scale = np.exp(0.5 * rng.standard_normal(t["n_classes"]))
    t["local"] = (t["local"].reshape(t["n_classes"], -1) * scale[:, None]).ravel()
    t["b_cell"] = t["b_cell"] * (1.0 + 0.25 * rng.standard_normal(t["b_cell"].size))
    return t


def _prepare_condense(case, seed):
    t = _condense_inputs(case, seed)
    return dict(kind="condense", cond=N.Condense(t), rows=t["n_face_blocks"] * (t["n_face_dofs"] // (t["dim"] + 1)))


def _run_condense(s):
    cond = s["cond"]
    nnz, _ = cond.run()
    p = [ctypes.c_void_p() for _ in range(4)]
    cond._check(cond.lib.fhg_cond_result(cond.h, *[ctypes.byref(v) for v in p]))
    return {"rowptr": _view(cond, p[0].value, s["rows"] + 1, "<i4"), "colidx": _view(cond, p[1].value, nnz, "<i4"),
            "vals": _view(cond, p[2].value, nnz, "<f8"), "b": _view(cond, p[3].value, s["rows"], "<f8")}


def _face_solution(case):
    """The discrete solution of the sine source, in the given numbering."""
    def make():
        H = hho.Hierarchy(case["dim"], case["n"], case["k"], max_levels=1)
        A, b = H.A(0), H.b()
        H.close()
        return _pcg(A, b)
    return _keep(("face solution", case["dim"], case["n"], case["k"]), make)


def _prepare_post(case, seed):
    t = _tables(case, "post")
    x = _face_solution(case)
    x = x * (1.0 + 1e-5 * np.random.default_rng(seed).standard_normal(x.size))   # a solution to some accuracy
    post = _keep(("post", case["dim"], case["n"], case["k"]), lambda: N.Post(t))
    return dict(kind="post", post=post, x=torch.from_numpy(x).cuda(),
                cells=torch.empty(t["n_elements"] * t["n_cell"], dtype=torch.float64, device="cuda"))


def _run_post(s):
    err, _ = s["post"].run(s["x"].data_ptr(), s["cells"].data_ptr(), "sine")
    return {"cells": s["cells"], "l2_error": err}


_PREPARE = dict(solve=_prepare_solve, precond=_prepare_precond, batch=_prepare_batch, condense=_prepare_condense,
                post=_prepare_post)
_RUN = dict(solve=_run_solve, precond=_run_precond, batch=_run_batch, condense=_run_condense, post=_run_post)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------------------------------
# work and exact values

def _mesh(dim, n, k):
    """(interior faces, their coupled pairs, elements, face block size, cell unknowns, reconstruction size)."""
    faces = 12 * n ** 3 - 6 * n ** 2 if dim == 3 else 3 * n ** 2 - 2 * n
    blocks = faces * (7 if dim == 3 else 5)
    elems = 6 * n ** 3 if dim == 3 else 2 * n ** 2
    bs = hho.face_unknowns(dim, k)
    cell = (k + 1) * (k + 2) * (k + 3) // 6 if dim == 3 else (k + 1) * (k + 2) // 2
    recon = (k + 2) * (k + 3) * (k + 4) // 6 if dim == 3 else (k + 2) * (k + 3) // 2
    return faces, blocks, elems, bs, cell, recon


def _solve_work(dim, n, k, size, sweeps, iterations):
    """Every level's operators and the vectors once; the products of `iterations` iterations."""
    faces, blocks, _, bs, _, _ = _mesh(dim, n, k)
    below = 8.0 / 7.0 if dim == 3 else 4.0 / 3.0
    entries = blocks * bs * bs * below
    transfer = 0.8 * entries
    byts = (entries + transfer) * size + (blocks * below) * 4 + 16 * faces * bs
    flops = iterations * 2.0 * (entries * (sweeps + 1) + blocks * bs * bs + 2 * transfer)
    return byts, flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        byts = flops = 0.0
        for s in _specs(case):
            b, f = _solve_work(2, s.n, s.k, 4 if case["precision"] == "fp32" else 8, 2, 30)
            byts, flops = byts + b, flops + f
        return {"bytes": byts, "flops": flops}
    dim, n, k = case["dim"], case["n"], case["k"]
    faces, blocks, elems, bs, cell, recon = _mesh(dim, n, k)
    if kind in ("solve", "precond"):
        its = 1 if kind == "precond" else {1: 34, 2: 17, 3: 12}[case["nu"]] * (2 if case["coefficient"] == "anisotropic" else 1)
        size = 4 if case["precision"] == "fp32" else 8
        byts, flops = _solve_work(dim, n, k, size, 2 * case["nu"], its)
        if kind == "solve" and case["learned"]:
            flops += its * 49152.0 * faces
        return {"bytes": byts, "flops": flops}
    ff = bs * (dim + 1)
    if kind == "condense":
        return {"bytes": 12.0 * blocks * bs * bs + 4.0 * faces * bs + 8.0 * faces * bs + 4.0 * elems * (dim + 2) + 8.0 * elems * cell
                + 16.0 * faces, "flops": 2.0 * blocks * bs * bs + 2.0 * 2 * faces * bs * cell}
    points = 6 ** dim
    return {"bytes": 8.0 * (faces * bs + 2 * elems * cell + 3 * elems) + 4.0 * elems * (dim + 2),
            "flops": elems * (2.0 * cell * ff + 2.0 * recon * (cell + ff) + points * (2.0 * recon + 2.0 * dim + 6))}


def _pcg(A, b):
    """x of A x = b in 64 bits: Jacobi-preconditioned CG with residual restarts, to the rounding level."""
    At = torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)), torch.from_numpy(A.indices.astype(np.int64)),
                                 torch.from_numpy(A.data), size=A.shape, dtype=torch.float64).cuda()
    bt = torch.from_numpy(np.ascontiguousarray(b)).cuda()
    dinv = torch.from_numpy(1.0 / A.diagonal()).cuda()
    x = torch.zeros_like(bt)
    bn = float(bt.norm())
    for _ in range(3):
        r = bt - At @ x
        z = dinv * r
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(6000):
            Ap = At @ p
            alpha = rz / torch.dot(p, Ap)
            x = x + alpha * p
            r = r - alpha * Ap
            z = dinv * r
            rz_new = torch.dot(r, z)
            p = z + (rz_new / rz) * p
            rz = rz_new
            if it % 50 == 49 and float(r.norm()) < 1e-14 * bn:
                break
    return x.cpu().numpy()


def _exact_problem(dim, n, k, coefficient, contrast, seed, load_seed):
    H = hho.Hierarchy(dim, n, k, max_levels=1, coefficient=coefficient, contrast=contrast,
                      checker_blocks=_checker_blocks(coefficient), seed=seed)
    A = H.A(0)
    H.close()
    return _pcg(A, _mix(_loads(dim, n, k, coefficient, contrast, seed), load_seed))


def _exact_condense(case, seed):
    """S = A_FF - A_TF^T A_TT^-1 A_TF and G = -A_TF^T A_TT^-1 per class, added up face by face."""
    t = _condense_inputs(case, seed)
    nC, nFF, nF = t["n_cell"], t["n_face_dofs"], case["dim"] + 1
    nf, nH, ne, rows = nFF // nF, nC + nFF, t["n_elements"], t["n_face_blocks"] * (nFF // nF)
    L = torch.from_numpy(t["local"]).reshape(t["n_classes"], nH, nH).cuda()
    TT, TF, FF = L[:, :nC, :nC], L[:, :nC, nC:], L[:, nC:, nC:]
    inv = torch.linalg.inv(TT)
    Sc = FF - TF.transpose(1, 2) @ (inv @ TF)
    Gc = -TF.transpose(1, 2) @ inv
    cls = torch.from_numpy(t["elem_class"].astype(np.int64)).cuda()
    faces = torch.from_numpy(t["elem_faces"].astype(np.int64)).reshape(ne, nF).cuda()
    dof = (faces[:, :, None] * nf + torch.arange(nf, device="cuda")).reshape(ne, nFF)
    dof[(faces < 0).repeat_interleave(nf, dim=1)] = -1
    bT = torch.from_numpy(t["b_cell"]).reshape(ne, nC, 1).cuda()
    be = (Gc[cls] @ bT)[:, :, 0]
    b = torch.zeros(rows, dtype=torch.float64, device="cuda")
    b.index_add_(0, dof[dof >= 0], be[dof >= 0])
    keys, vals = [], []
    for e0 in range(0, ne, 100_000):
        d = dof[e0:e0 + 100_000]
        ok = (d[:, :, None] >= 0) & (d[:, None, :] >= 0)
        keys.append((d[:, :, None] * rows + d[:, None, :])[ok])
        vals.append(Sc[cls[e0:e0 + 100_000]][ok])
    key, where = torch.unique(torch.cat(keys), sorted=True, return_inverse=True)
    v = torch.zeros(key.numel(), dtype=torch.float64, device="cuda")
    v.index_add_(0, where, torch.cat(vals))
    return {"rowptr": None, "colidx": None, "vals": v, "b": b}


def _exact_post(case, seed):
    t = _tables(case, "post")
    x = prepare(case, seed)["x"]
    nC, nFF, nR, nq, nF = t["n_cell"], t["n_face_dofs"], t["n_recon"], t["n_points"], case["dim"] + 1
    nf, ne, ncls = nFF // nF, t["n_elements"], t["n_classes"]
    g = lambda name, *shape: torch.from_numpy(t[name]).reshape(shape).cuda()  # noqa: E731
    faces = g("elem_faces", ne, nF).long()
    xf = x.reshape(-1, nf)[faces.clamp(min=0)] * (faces >= 0)[:, :, None]
    xf = xf.reshape(ne, nFF)
    cls, centre = g("elem_class", ne).long(), g("elem_centre", ne, 3)
    sc, rc = g("solve_cells", ncls, nC, nFF), g("recon", ncls, nR, nC + nFF)
    w, off, basis = g("weights", ncls, nq), g("offsets", ncls, nq, 3), g("basis", ncls, nq, nR)
    cells = g("cell_rhs", ne, nC).clone()
    err = nrm = 0.0
    for c in range(ncls):
        at = torch.nonzero(cls == c)[:, 0]
        cells[at] += xf[at] @ sc[c].T
        coef = torch.cat([cells[at], xf[at]], dim=1) @ rc[c].T
        for a0 in range(0, at.numel(), 65536):
            a = at[a0:a0 + 65536]
            u = torch.ones(a.numel(), nq, dtype=torch.float64, device="cuda")
            for d in range(case["dim"]):
                u = u * torch.sin(torch.pi * (centre[a, d, None] + off[c, None, :, d]))
            uh = coef[a0:a0 + 65536] @ basis[c].T
            err += float(((uh - u) ** 2 * w[c]).sum())
            nrm += float((u ** 2 * w[c]).sum())
    return {"cells": cells.reshape(-1), "l2_error": float(np.sqrt(err) / np.sqrt(nrm))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return {"x": _exact_problem(case["dim"], case["n"], case["k"], case["coefficient"], case["contrast"], 20261203, seed)}
    if kind == "batch":
        if case["problems"] * case["n_max"] > 2400:
            return None
        return [_exact_problem(2, s.n, s.k, "lognormal_patches", 1e3, s.seed, seed + 1000 * i)
                for i, s in enumerate(_specs(case))]
    if kind == "condense":
        return _exact_condense(case, seed)
    if kind == "post":
        return _exact_post(case, seed)
    return None   # the preconditioner is defined by its own smoothing order
