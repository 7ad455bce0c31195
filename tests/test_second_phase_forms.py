"""The second phase of product integrands gives a box the same result however
many boxes share the call.

Up to 65 536 boxes take 8 lanes per child (n >= 5), more boxes 4; in 2 to 4
dimensions up to 16 384 boxes take 16 lanes, more 4 or 2: whichever form refines
a box, its bisections and its bits are the same, so an integral's
counts and status do not depend on its batch neighbours or on the number of
shares of its leftover list.  Values and errors are sums over the boxes, per
integral in the order of its own boxes: the same bits too.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MANY = 1 << 16


def _integrals(cub, family, n, count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        a = rng.uniform(12, 25, n) if family == "product_peak" else rng.uniform(7, 11, n)
        out.append((list(a), list(rng.uniform(0.3, 0.7, n))))
    return out, [cub.make_params(n, a, u) for a, u in out]


@pytest.mark.parametrize("family", ["product_peak", "gaussian"])
@pytest.mark.parametrize("n,eps", [(5, 1e-8), (6, 1e-7), (7, 1e-6), (8, 1e-5)])
def test_integral_alone_and_in_a_batch(cub, ctx, family, n, eps):
    _, params = _integrals(cub, family, n, 24, n)
    # (one kernel per step in the first phase: the others sum a region's points
    # in an order that depends on the length of the list)
    opts = cub.options(phase1_cap=4096, phase2_max_regions=40, persistent=False)
    ctx.reset_stats()
    batch = ctx.integrate_batch(family, n, params, eps, 1e-15, opts)
    assert ctx.stats()["phase2_boxes"] > MANY
    for k in (0, 7, 16, 23):
        ctx.reset_stats()
        one = ctx.integrate_batch(family, n, [params[k]], eps, 1e-15, opts)[0]
        assert 0 < ctx.stats()["phase2_boxes"] < MANY
        assert one == batch[k], (family, n, k)


@pytest.mark.parametrize("family,a", [("product_peak", (15, 25)), ("gaussian", (9, 12))])
@pytest.mark.parametrize("n,eps,cap,count", [(2, 1e-11, 400, 60), (3, 1e-10, 800, 24),
                                             (4, 1e-7, 800, 24)])
def test_integral_alone_and_in_a_batch_low_dimensions(cub, ctx, family, a, n, eps, cap, count):
    rng = np.random.default_rng(10 * n)
    params = [cub.make_params(n, list(rng.uniform(*a, n)), list(rng.uniform(0.3, 0.7, n)))
              for _ in range(count)]
    opts = cub.options(phase1_cap=cap, persistent=False)
    ctx.reset_stats()
    batch = ctx.integrate_batch(family, n, params, eps, 1e-14, opts)
    assert ctx.stats()["phase2_boxes"] > 1 << 14
    ctx.reset_stats()
    for k in (0, 11, count - 1):
        one = ctx.integrate_batch(family, n, [params[k]], eps, 1e-14, opts)[0]
        assert one == batch[k], (family, n, k)
    assert 0 < ctx.stats()["phase2_boxes"] < 1 << 14


@pytest.mark.parametrize("cap", [126, 127, 128, 129])
def test_heap_sizes_of_the_form_for_many_boxes(cub, oracle, ctx, cap):
    """Bisection limits around the 127 heap entries that this form keeps in
    shared memory, on boxes that reach them, against the oracle."""
    n, eps = 5, 1e-9
    cases, params = _integrals(cub, "product_peak", n, 80, 1)
    kw = dict(phase1_cap=1024, phase2_max_regions=cap)
    ctx.reset_stats()
    batch = ctx.integrate_batch("product_peak", n, params, eps, 1e-15, cub.options(**kw))
    assert ctx.stats()["phase2_boxes"] > MANY
    for k in (3, 41):
        o = oracle.Rule(n).integrate_reference(
            oracle.make_integrand("product_peak", n, *cases[k]), eps, 1e-15, phase1_cap=1024,
            phase2_max=cap)
        assert batch[k].status == o["status"] > 0
        assert abs(batch[k].nregions - o["nregions"]) <= 0.005 * o["nregions"]
        assert abs(batch[k].integral - o["value"]) <= 1e-9 * abs(o["value"])


def test_shares_of_a_long_leftover_list(cub, ctx):
    """One integral whose leftover list is long and whose shares are short."""
    n, eps, world = 6, 1e-8, 4
    f = cub.Integrand("product_peak", n, [20.0, 25.0, 15.0, 22.0, 18.0, 24.0],
                      [0.3, 0.5, 0.7, 0.45, 0.6, 0.4])
    opts = cub.options(phase1_cap=70000, phase2_max_regions=20)
    ctx.reset_stats()
    whole = ctx.integrate(f, eps, 1e-15, opts)
    boxes = ctx.stats()["phase2_boxes"]
    assert MANY < boxes < world * MANY
    parts = [ctx.integrate_shard(f, eps, 1e-15, r, world, opts) for r in range(world)]
    first = parts[0][0]
    assert all(p1 == first for p1, _ in parts)
    assert first.nregions + sum(p.nregions for _, p in parts) == whole.nregions
    assert sum(p.status for _, p in parts) == whole.status > 0
    value = first.integral + sum(p.integral for _, p in parts)
    # up to 2.6e5 boxes of one sign, 8192 terms a lane in a row: at most
    # 8192 x 1.1e-16 by rounding
    assert abs(value - whole.integral) <= 1e-12 * abs(whole.integral)
