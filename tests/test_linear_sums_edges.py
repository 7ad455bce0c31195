"""Coefficients that the thread-per-region forms of continuous and corner peak
have to treat apart, against the point-by-point oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

U = 2.0 ** -53


def _boxes(n, m, seed):
    rng = np.random.default_rng(seed)
    ln = np.ldexp(1.0, -rng.binomial(3, 0.5, (n, m)))
    return np.floor(rng.random((n, m)) / ln) * ln, ln


def _eval(cub, family, n, a, u, lo, ln, eps=1e-4):
    return cub.rule_eval(cub.Integrand(family, n, list(a), list(u)), torch.from_numpy(lo).cuda(),
                         torch.from_numpy(ln).cuda(), eps, 1e-12)


@pytest.mark.parametrize("m", [33, 4097])
@pytest.mark.parametrize("a", [
    [-3.0, 2.0], [-1.0, -2.0, -0.5], [4.0, -0.0, -3.0, 1.0],
    [-3.0, 2.0, -1.5, 4.0, 0.5], [1.0, 2.0, 3.0, 1.0, 2.0, 1.0, 2.0, -1.0],
    [-840.0, 3.0], [400.0, -190.0, 1.0],       # inside the range of the products
    [-650.0, 700.0], [800.0, -790.0, 3.0],     # beyond it: point by point
    [-350.0, 350.0, -330.0, 320.0]])
def test_continuous_with_growing_axes(cub, oracle, ctx, a, m):
    """Coefficients below zero.  A value's exponent is a sum of n terms of at
    most `reach` together, each rounded (2 n reach roundings of u on either
    side); the rest are the bounds of tests/test_gpu_parity.py.  Split axes: the
    fourth difference of exp(-a x) over a side h is about 0.05 (a h)^4 of the
    value, above 1e-4 for the axis that has the largest here (a h >= 1 / 4),
    and carries a rounding of some 1e-15 + slack."""
    n = len(a)
    u = [0.3 + 0.1 * (i % 5) for i in range(n)]
    lo, ln = _boxes(n, m, 7 * n + m)
    o = oracle.Rule(n).phase1_eval(oracle.make_integrand("continuous", n, a, u), lo, ln, 1e-4,
                                   1e-12)
    avg, err, axis, active = [t.cpu().numpy() for t in _eval(cub, "continuous", n, a, u, lo, ln)]
    reach = sum(abs(x) * max(v, 1 - v) for x, v in zip(a, u))
    slack = 4 * n * reach * U
    scale = np.abs(o["avg"]) + o["mag"]
    assert np.all(np.abs(avg - o["avg"]) <= (1e-13 + slack) * scale + 1e-300)
    assert np.all(np.abs(err - o["err"]) <= (1e-12 + 10 * slack) * scale + 1e-12 * o["err"] + 1e-300)
    clear = o["margin"] > 1e-8 + 1e6 * slack
    assert clear.any() and np.array_equal(axis[clear], o["axis"][clear])


def test_growing_axes_cost_what_the_others_do(cub, ctx):
    """One negative coefficient does not send every region to its 1105 points."""
    n, m = 8, 512
    lo, ln = (torch.from_numpy(x).cuda() for x in _boxes(n, m, 1))

    def best(a0):
        f = cub.Integrand("continuous", n, [a0] + [2.0] * (n - 1), [0.4] * n)
        t = []
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record()
            for _ in range(4):
                cub.rule_eval(f, lo, ln, 1e-4, 1e-12)
            e[1].record()
            torch.cuda.synchronize()
            t.append(e[0].elapsed_time(e[1]))
        return min(t)

    best(2.0)
    assert best(-2.0) <= 2 * best(2.0)


@pytest.mark.parametrize("n,m", [(2, 100), (4, 4200), (8, 12400)])
def test_corner_peak_arguments_beyond_the_range(cub, oracle, ctx, n, m):
    """a x is infinite in all or some of the boxes: the values there are zero."""
    a = [1e308] + [1.0] * (n - 1)
    lo, ln = _boxes(n, m, n)
    lo[0] += np.where(np.arange(m) % 2, 5.0, 0.0)
    ln[0] *= np.where(np.arange(m) % 3, 8.0, 1.0)
    o = oracle.Rule(n).phase1_eval(oracle.make_integrand("corner_peak", n, a, [0.0] * n), lo, ln,
                                   1e-4, 1e-12)
    avg, err, axis, active = [t.cpu().numpy()
                              for t in _eval(cub, "corner_peak", n, a, [0.0] * n, lo, ln)]
    assert np.isfinite(o["avg"]).all() and (o["avg"] == 0).any()
    scale = np.abs(o["avg"]) + o["mag"]
    assert np.all(np.abs(avg - o["avg"]) <= 1e-13 * scale + 1e-300)
    assert np.all(np.abs(err - o["err"]) <= 1e-12 * scale + 1e-12 * o["err"] + 1e-300)
    assert np.array_equal(active, o["active"])
