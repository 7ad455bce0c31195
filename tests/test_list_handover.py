"""Lists that go from the kernels of long lists back to the replicated one.

Small batches on short lists run in the replicated kernel, which finds a
slot's integral from the segments; integrals that stopped while the list was
long must not own slots of the others (their tolerances would decide, and
children and leftover boxes of those slots would not be written).
"""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("family", ["gaussian", "product_peak", "oscillatory", "corner_peak"])
@pytest.mark.parametrize("hard", [(0,), (2,), (0, 5), (1, 2, 6)])
@pytest.mark.parametrize("policy", ["breadth", "two_phase"])
def test_stopped_integrals_own_no_slots(cub, ctx, family, hard, policy):
    n, count = 3, 8
    a = {"gaussian": (9.0, 0.3), "product_peak": (15.0, 0.3), "oscillatory": (9.0, 0.3),
         "corner_peak": (12.0, 0.1)}[family]
    params = [cub.make_params(n, [a[0] + 0.3 * k, a[0], a[0] - 1] if k in hard else a[1], 0.4)
              for k in range(count)]
    # the others stop in the first iteration, at a tolerance that would stop
    # the hard ones too
    epsrel = [1e-9 if k in hard else 1e-1 for k in range(count)]
    # 512 regions of the initial grids are a long list, the children of three
    # are not; and an integral has 64 regions, then up to 128 and 256: with a cap
    # of 160 it hands its boxes to the second phase after the list came back
    kw = dict(policy=cub.POLICY_BREADTH if policy == "breadth" else cub.POLICY_REFERENCE,
              phase1_cap=0 if policy == "breadth" else 160, persistent_max_n=400,
              phase2_max_regions=30)
    for device_loop in (True, False):
        ctx.reset_stats()
        got = ctx.integrate_batch(family, n, params, epsrel, 1e-15,
                                  cub.options(device_loop=device_loop, **kw))
        st = ctx.stats()
        assert st["eval_launches"] > 0 and st["replicated_launches"] > 0
        want = ctx.integrate_batch(family, n, params, epsrel, 1e-15,
                                   cub.options(device_loop=device_loop, replicated=False, **kw))
        assert got == want
        assert all(got[k].iterations > 1 for k in hard)
        assert all(got[k].iterations == 1 for k in range(count) if k not in hard)
