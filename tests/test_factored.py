"""Kernels that share work between the points of a region, at the sizes and
inputs where they can go wrong, against the point-by-point oracle.

Integrands that are products over the axes, those that depend on a sum over
the axes, and the 7-D table integrand are evaluated by one thread per region
from per-axis (per-group) quantities.  Values
and errors are sums of the same terms in another order: the tolerances are
those of tests/test_gpu_parity.py (1e-13 of the L1 magnitude of the rule sum
for the value, 1e-12 for the error), the split axes identical where the
oracle's two largest fourth differences are told apart.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from test_gpu_parity import FAMILY_PARAMS, compare_regions, refined_list  # noqa: E402


def _eval(cub, family, n, a, u, lo, ln, eps=1e-4):
    return cub.rule_eval(cub.Integrand(family, n, list(a), list(u)), torch.from_numpy(lo).cuda(),
                         torch.from_numpy(ln).cuda(), eps, 1e-12)


@pytest.mark.parametrize("family", ["gaussian", "product_peak"])
@pytest.mark.parametrize("n", range(2, 9))
@pytest.mark.parametrize("m", [1, 31, 33, 4097])
def test_product_rule_list_lengths(cub, oracle, ctx, family, n, m):
    rng = np.random.default_rng(100 * n + m)
    a, u = FAMILY_PARAMS[family](n, rng)
    level = rng.binomial(6, 0.5, (n, m))
    ln = np.ldexp(1.0, -level)
    lo = np.floor(rng.random((n, m)) / ln) * ln
    o = oracle.Rule(n).phase1_eval(oracle.make_integrand(family, n, a, u), lo, ln, 1e-4, 1e-12)
    compare_regions(o, _eval(cub, family, n, a, u, lo, ln), (family, n, m))


@pytest.mark.parametrize("family", ["corner_peak", "continuous"])
@pytest.mark.parametrize("n", range(2, 9))
@pytest.mark.parametrize("m", [33, 12321])
def test_sum_rule_list_lengths(cub, oracle, ctx, family, n, m):
    """12321 regions are past the length from which every family takes one
    thread per region, and no multiple of a block."""
    rng = np.random.default_rng(200 * n + m)
    a, u = FAMILY_PARAMS[family](n, rng)
    level = rng.binomial(6, 0.5, (n, m))
    ln = np.ldexp(1.0, -level)
    lo = np.floor(rng.random((n, m)) / ln) * ln
    o = oracle.Rule(n).phase1_eval(oracle.make_integrand(family, n, a, u), lo, ln, 1e-4, 1e-12)
    compare_regions(o, _eval(cub, family, n, a, u, lo, ln), (family, n, m))


@pytest.mark.parametrize("family,a,u", [
    ("continuous", [-2.0, 3.0, 1.0, -0.5], [0.3, 0.6, 0.5, 0.4]),  # factors above 1
    ("continuous", [2.0, 0.0, 1.0, 0.5], [0.3, 0.6, 0.5, 0.4]),    # ties, an idle axis
    ("corner_peak", [3.0, -0.2, 0.0, 1.0], [0.0] * 4),             # signs mixed, an idle axis
    ("corner_peak", [9.0, 7.0, 11.0, 8.0], [0.0] * 4),
])
def test_sum_rule_unusual_parameters(cub, ctx, family, a, u):
    """Against 32 lanes point by point in the engine: the same splits."""
    f = cub.Integrand(family, 4, a, u)
    opt = dict(policy=cub.POLICY_BREADTH, persistent=False)
    one = ctx.integrate(f, 1e-7, 1e-12, cub.options(lanes=1, **opt))
    many = ctx.integrate(f, 1e-7, 1e-12, cub.options(lanes=32, **opt))
    assert one.nregions == many.nregions and one.iterations == many.iterations
    assert one.status == many.status
    assert math.isclose(one.integral, many.integral, rel_tol=1e-12)


@pytest.mark.parametrize("family,n,a,eps", [("gaussian", 5, 5.0, 1e-5), ("gaussian", 3, 6.0, 1e-9),
                                            ("corner_peak", 4, 0.5, 1e-10),
                                            ("continuous", 3, 4.0, 1e-9),
                                            ("product_peak", 2, 20.0, 1e-10),
                                            ("product_peak", 6, 4.0, 1e-5)])
def test_tied_axes_split_as_point_by_point(cub, ctx, family, n, a, eps):
    """An integrand that is the same in every axis, on its symmetric grid:
    all fourth differences tie up to their last bits, and the axis is
    whichever the point values make the largest.  One thread per region and
    32 lanes point by point take the same splits."""
    f = cub.Integrand(family, n, a, 0.5)
    opt = dict(policy=cub.POLICY_BREADTH, persistent=False)
    one = ctx.integrate(f, eps, 1e-15, cub.options(lanes=1, **opt))
    many = ctx.integrate(f, eps, 1e-15, cub.options(lanes=32, **opt))
    assert one.nregions == many.nregions > (2 if n >= 5 else 4) ** n
    assert one.iterations == many.iterations and one.status == many.status
    assert math.isclose(one.integral, many.integral, rel_tol=1e-12)


def test_underflowing_centre_and_flat_regions(cub, oracle, ctx):
    """Gaussian regions so far from the peak that the centre's value is zero
    (or every point's is), and regions whose differences are all rounding."""
    n, a, u = 4, [60.0, 55.0, 1e-9, 1e-9], [0.5, 0.5, 0.5, 0.5]
    lo, ln = refined_list(oracle, n, 4, seed=11)
    o = oracle.Rule(n).phase1_eval(oracle.make_integrand("gaussian", n, a, u), lo, ln, 1e-4, 1e-12)
    compare_regions(o, _eval(cub, "gaussian", n, a, u, lo, ln), ("underflow",))


def test_tiles_of_long_lists(cub, oracle, ctx):
    """Integrals with more than 256 chunks beside short ones: whole tiles and
    the chunks after them, at segment starts that are no multiple of a tile.
    Tiles are counted from the segment's start, so an integral has the same
    bits in a batch as in a list of two of its own, host-driven and
    device-driven alike."""
    n, eps = 3, 1e-11
    rng = np.random.default_rng(5)
    cases = []
    for k in range(5):
        hard = k in (1, 3)
        a = rng.uniform(10, 25, n) if hard else rng.uniform(1, 2, n)
        cases.append((list(a), list(rng.uniform(0.3, 0.7, n))))
    params = [cub.make_params(n, a, u) for a, u in cases]
    opt = dict(policy=cub.POLICY_BREADTH, persistent=False)
    dev = ctx.integrate_batch("product_peak", n, params, eps, 1e-14, cub.options(**opt))
    host = ctx.integrate_batch("product_peak", n, params, eps, 1e-14,
                               cub.options(device_loop=False, **opt))
    assert dev == host
    assert max(r.nregions for r in dev) > 16 * 256 * 32
    for (a, u), p, r in zip(cases, params, dev):
        two = ctx.integrate_batch("product_peak", n, [p, p], eps, 1e-14, cub.options(**opt))
        assert two[0] == two[1] == r
        exact = oracle.exact(oracle.make_integrand("product_peak", n, a, u))
        assert r.status == 0 and abs(r.integral - exact) <= max(r.error, 1e-13 * exact)


@pytest.mark.parametrize("n", range(2, 9))
@pytest.mark.parametrize("family", ["gaussian", "product_peak"])
def test_second_phase_of_products(cub, oracle, ctx, family, n):
    """The second phase with a few lanes per box, in every dimension, against
    the oracle's (the bounds of tests/test_gpu_parity.py: values within 2
    epsrel, region counts within 0.5%)."""
    rng = np.random.default_rng(31 * n)
    eps = {2: 1e-9, 3: 1e-8, 4: 1e-7, 5: 1e-6, 6: 1e-5, 7: 1e-3, 8: 1e-3}[n]
    a = rng.uniform(8, 14, n) if family == "product_peak" else rng.uniform(6, 9, n)
    u = rng.uniform(0.3, 0.7, n)
    kw = dict(phase1_cap=256)
    ctx.reset_stats()
    r = ctx.integrate(cub.Integrand(family, n, list(a), list(u)), eps, 1e-14,
                      cub.options(**kw))
    assert ctx.stats()["phase2_boxes"] > 0
    o = oracle.Rule(n).integrate_reference(oracle.make_integrand(family, n, a, u), eps, 1e-14, **kw)
    assert r.status == o["status"]
    assert abs(r.integral - o["value"]) <= 2 * eps * abs(o["value"])
    assert abs(r.nregions - o["nregions"]) <= 0.005 * o["nregions"]


@pytest.mark.parametrize("cap", [7, 254, 255, 256, 600])
def test_second_phase_heap_sizes(cub, oracle, ctx, cap):
    """Bisection limits around the number of heap entries kept in shared
    memory, on boxes that reach them."""
    n, eps = 5, 1e-8
    a, u = [20.0, 30.0, 10.0, 25.0, 15.0], [0.3, 0.5, 0.7, 0.45, 0.6]
    r = ctx.integrate(cub.Integrand("product_peak", n, a, u), eps, 1e-14,
                      cub.options(phase1_cap=64, phase2_max_regions=cap))
    o = oracle.Rule(n).integrate_reference(oracle.make_integrand("product_peak", n, a, u), eps,
                                           1e-14, phase1_cap=64, phase2_max=cap)
    assert r.status == o["status"] > 0
    assert r.nregions == o["nregions"]
    assert abs(r.integral - o["value"]) <= 1e-9 * abs(o["value"])


def test_second_phase_wide_and_narrow(cub, ctx):
    """Few leftover boxes take more lanes per box than many: an integral by
    itself and in a batch whose boxes pass the limit gets the same answer."""
    n, eps = 3, 1e-10
    rng = np.random.default_rng(3)
    params = [cub.make_params(n, list(rng.uniform(15, 30, n)), list(rng.uniform(0.3, 0.7, n)))
              for _ in range(24)]
    opts = cub.options(phase1_cap=4096)
    ctx.reset_stats()
    batch = ctx.integrate_batch("product_peak", n, params, eps, 1e-15, opts)
    assert ctx.stats()["phase2_boxes"] > 1 << 16
    for k in (0, 11, 23):
        one = ctx.integrate_batch("product_peak", n, [params[k]], eps, 1e-15, opts)[0]
        assert one.status == batch[k].status
        assert abs(one.integral - batch[k].integral) <= 1e-11 * abs(one.integral)
        assert abs(one.nregions - batch[k].nregions) <= 0.005 * one.nregions


def test_table_regions_match_the_points(cub, oracle, ctx):
    """The table integrand by one thread per region (long lists) against the
    16- and 32-lane point-by-point forms: the same run, the same counts."""
    from cubature import tables as T

    d = T.table7_data(3)
    tab = T.Table7(d, 0)
    offs = [-0.7, 0.1, 0.9]
    thread = ctx.integrate_table7_batch(tab, offs, 1e-4, 1e-12, cub.options(
        policy=cub.POLICY_BREADTH, persistent=False))
    lanes = ctx.integrate_table7_batch(tab, offs, 1e-4, 1e-12, cub.options(
        policy=cub.POLICY_BREADTH, persistent=False, lanes=32))
    for t, w in zip(thread, lanes):
        assert t.status == w.status and t.nregions == w.nregions
        assert math.isclose(t.integral, w.integral, rel_tol=1e-12)
        assert math.isclose(t.error, w.error, rel_tol=1e-9)
