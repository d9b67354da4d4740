"""The one-launch coarse sub-cycle: the process-wide record of the timed choice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
