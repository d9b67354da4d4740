"""The one-launch coarse sub-cycle with its first level, cluster and CTA size chosen by the test: several smoothed
levels in the launch (transfers between them, the W loop's restart from a kept x), levels whose phases take several
passes of a warp, more than 24 colours, clusters of 8 and 16 CTAs of 512 and 1024 threads, every block size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _galerkin(A0, Ps):
    As = [A0.tocsr()]
    for P in Ps:
        As.append((P.T @ As[-1] @ P).tocsr())
    return As


@pytest.fixture(scope="module", params=[(2, 128, 1), (2, 96, 2), (2, 128, 3), (3, 16, 1), (3, 16, 2)], ids=str)
def hierarchy(request):
    from fhhos4_gb300 import batch as BT
    from fhhos4_gb300 import hho
    dim, n, k = request.param
    if dim == 2:
        bs, A0, Ps, _, _ = BT.generate(BT.ProblemSpec(n, k, 4242))
    else:
        H = hho.Hierarchy(dim, n, k, coefficient="anisotropic" if k == 1 else "checkerboard", contrast=100.0, checker_blocks=4)
        A0, Ps, bs = H.A(0), [H.P(l) for l in range(H.levels - 1)], H.block_size
        H.close()
    return _galerkin(A0, Ps), Ps, bs


def _starts(ctx, precision, last, info, bs):
    """Every start of the sub-cycle that the context takes, set one after the other: (first level, CTAs, threads)."""
    from fhhos4_gb300 import _native as N
    for threads in (512, 1024):
        for ctas in (8, 16):
            for first in range(1, last):
                try:
                    ctx.set_fused_coarse(precision, first, ctas, threads)
                except N.FhgError as e:
                    assert e.code == N.FHG_ERR_UNSUPPORTED
                    # only the shared memory of a CTA (200 KB) keeps a level out: three vectors a level, b and x on
                    # the coarsest, its b in FP64
                    entry = 4 if precision == "fp32" else 8
                    rows = sum((3 if l < last else 2) * info[l]["block_rows"] for l in range(first, last + 1))
                    assert rows * bs * entry / ctas + 8 * info[last]["block_rows"] * bs > 190 * 1024, (first, ctas, threads)
                    continue
                assert ctx.fused_coarse_info(precision) == (first, ctas, threads)
                yield first, ctas, threads


def _assert_covers(ran, last, info):
    firsts = {f for f, _, _ in ran}
    assert min(firsts) <= last - 2                               # two smoothed levels or more in the launch
    assert {f for f, c, t in ran if (c, t) == (16, 512)} == firsts
    assert {(c, t) for f, c, t in ran if f == last - 1} == {(c, t) for c in (8, 16) for t in (512, 1024)}
    assert max(i["block_rows"] for i in info[min(firsts):last]) > 1024   # several passes of 8 x 512 threads


@pytest.mark.parametrize("precision", ["fp32", "df"])
def test_fused_levels_match_launch_by_launch(hierarchy, precision):
    """One V-cycle from level 0 in FP64, in `precision` launch by launch, and with the sub-cycle in one launch from
    every level that it can start from. Both forms carry the rounding of the same operations in another order of a
    row's sums, so their distances from the FP64 cycle are of one size: the fused one's within 4 times the other's."""
    from fhhos4_gb300 import _native as N
    from fhhos4_gb300 import solver as S
    As, Ps, bs = hierarchy
    last = len(As) - 1
    ctx = S.fcg_mg(As, Ps, bs, precision=precision, nu=(2, 2), galerkin=True).Context()
    info = [ctx.level_info(l) for l in range(len(As))]
    if len(As) == 4:   # the 3D ones: long rows
        assert max(i["colours"] for i in info[1:last]) > 24
    n = As[0].shape[0]
    r = np.random.default_rng(6).standard_normal(n)
    ctx.set_vcycle_precision("fp64")
    ref = ctx.apply(0, N.OP_VCYCLE, r, None, n)
    ctx.set_vcycle_precision(precision)
    ctx.set_fused_coarse(precision, -1)
    assert ctx.fused_coarse_info(precision)[0] == -1
    err = np.linalg.norm(ctx.apply(0, N.OP_VCYCLE, r, None, n) - ref)
    assert 0 < err <= (1e-3 if precision == "fp32" else 1e-9) * np.linalg.norm(ref)
    ran = set()
    for start in _starts(ctx, precision, last, info, bs):
        got = ctx.apply(0, N.OP_VCYCLE, r, None, n)
        assert np.linalg.norm(got - ref) <= 4 * err, start
        # again: nothing is left over from the first run
        assert np.array_equal(ctx.apply(0, N.OP_VCYCLE, r, None, n), got), start
        ran.add(start)
    _assert_covers(ran, last, info)
    with pytest.raises(N.FhgError) as e:
        ctx.set_fused_coarse(precision, last, 8, 512)            # the dense level alone
    assert e.value.code == N.FHG_ERR_UNSUPPORTED
    ctx.close()


@pytest.mark.parametrize("precision", ["df"])
def test_fused_levels_solve_with_w_cycles_as_launch_by_launch(hierarchy, precision):
    """Solves with W-cycles (the sub-cycle restarts a level from the x that the last coarse correction left) from
    every start, held to those launch by launch as test_fused_coarse_cycle_deep_hierarchy holds them: 1e-8 of the
    history in pairs. (A single W-cycle is no measure on the 2D fields: it amplifies a few modes, and the distance
    from FP64 of the launch-by-launch cycle itself changes severalfold with the order of its sums.)"""
    from test_gpu_parity import _check_fused_pair
    from fhhos4_gb300 import solver as S
    As, Ps, bs = hierarchy
    last = len(As) - 1
    b = np.random.default_rng(7).standard_normal(As[0].shape[0])
    kw = dict(precision=precision, cycle="W", nu=(2, 2), galerkin=True)
    plain = S.fcg_mg(As, Ps, bs, fused=False, **kw)
    fused = S.fcg_mg(As, Ps, bs, **kw)
    ctx = fused.Context()
    info = [ctx.level_info(l) for l in range(len(As))]
    ran = set()
    for start in _starts(ctx, precision, last, info, bs):
        if start[1:] in ((8, 512), (16, 1024)) or start[0] == last - 1 or start[1:] == (16, 512):
            _check_fused_pair(As[0], b, fused, plain, precision, rtol=1e-8)
        ran.add(start)
    _assert_covers(ran, last, info)
    for s in (plain, fused):
        s.Context().close()


def test_timed_choice_is_kept_apart_for_repeating_and_distinct_rows():
    """The timed choice of the sub-cycle is kept per process. Two systems of one structure, one with repeating block
    rows (row-class sweeps) and one without (stored blocks), have different launch-by-launch times, so the second
    is timed by itself; a third like the second is not timed again."""
    from fhhos4_gb300 import hho
    from fhhos4_gb300 import solver as S
    As, Ps, b, bs = hho.generate(3, 16, 1)
    rng = np.random.default_rng(8)
    noisy = []
    for A in As:
        B = A.copy()
        B.data = B.data * (1.0 + 1e-13 * rng.integers(0, 64, B.nnz))
        noisy.append(B)
    kw = dict(precision="fp32", autotune=True)
    ctxs = [S.fcg_mg(M, Ps, bs, **kw).Context() for M in (As, noisy, noisy)]
    assert ctxs[0].view_info(1, "fp32")["classes"] > 0
    assert ctxs[1].view_info(1, "fp32")["classes"] == 0 and ctxs[2].view_info(1, "fp32")["classes"] == 0
    launches = []
    for c in ctxs:
        before = c.kernel_launches()
        c.set_coarse_smoothing(3, 5)   # chosen anew for a cycle that nothing else here uses
        launches.append(c.kernel_launches() - before)
    assert launches[0] > 0 and launches[1] > 0 and launches[2] == 0
    for c in ctxs:
        c.close()
