"""Batches of mixed families on the kernels of long lists (here for lists of any
length) and in the second phase.  They evaluate point by point; single-family calls sum
products and corner peak's pairs from factors there: the same sums in another
order, so values agree to rounding (1e-11 of the value over some 1e5 regions)
and counts up to close calls of a region's test.  The second phase has the
bounds of tests/test_gpu_parity.py: a tie in a box's heap may go either way,
which changes the subregions within the error estimate (2 epsrel, 0.5% of the
counts)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FAMILIES = [("gaussian", 9.0, 0.45), ("product_peak", 14.0, 0.4), ("corner_peak", 1.5, 0.0),
            ("continuous", 3.0, 0.55), ("oscillatory", 1.2, 0.3)]


def _integrands(cub, n):
    rng = np.random.default_rng(n)
    return [cub.Integrand(f, n, list(a * rng.uniform(0.8, 1.2, n)),
                          [u] * n if f in ("corner_peak", "oscillatory")
                          else list(u + rng.uniform(-0.1, 0.1, n)))
            for f, a, u in FAMILIES for _ in range(8)]


@pytest.mark.parametrize("n,eps,policy,cap", [(3, 1e-6, "breadth", 0), (4, 1e-5, "reference", 2048),
                                              (5, 1e-4, "reference", 1024)])
def test_mixed_batch_on_long_lists(cub, ctx, n, eps, policy, cap):
    fs = _integrands(cub, n)
    opts = cub.options(policy=cub.POLICY_BREADTH if policy == "breadth" else cub.POLICY_REFERENCE,
                       phase1_cap=cap, phase2_max_regions=64, persistent=False)
    ctx.reset_stats()
    mixed = ctx.integrate_mixed(fs, eps, 1e-12, opts)
    st = ctx.stats()
    assert st["eval_launches"] > 0 and (policy == "breadth" or st["phase2_boxes"] > 0)
    for k in range(0, len(fs), 8):
        one = ctx.integrate_batch(fs[k].family, n, [f.params() for f in fs[k:k + 8]], eps, 1e-12,
                                  opts)
        for f, m, s in zip(fs[k:k + 8], mixed[k:k + 8], one):
            label = (f.family, n, policy)
            assert (m.status == 0) == (s.status == 0), label
            assert abs(m.nregions - s.nregions) <= 0.005 * s.nregions, label
            bound = 1e-11 if policy == "breadth" else 2 * eps
            assert abs(m.integral - s.integral) <= bound * abs(s.integral) + 1e-14, label
