"""The operation counts behind bench.py's roofline follow the evaluators that
the kernels use."""
import bench


def test_counts_follow_the_evaluators():
    points = {f: bench.flops_per_region(f, 8) for f in ("corner_peak", "oscillatory", "gaussian")}
    # corner peak: 552 pairs of a division and two powers instead of 1105 points
    assert bench.pair_flops(8) < points["corner_peak"] / 5
    split = {("corner_peak", 8): (0, 10, 3)}
    p, ml, p2 = bench.kernel_flops(split, 2, "k_persistent")
    assert (p, ml, p2) == (0, 20 * bench.pair_flops(8), 6 * points["corner_peak"])
    split = {("gaussian", 8): (5, 10, 3)}
    _, ml, p2 = bench.kernel_flops(split, 1, "k_replicated")
    assert ml / 10 == p2 / 3 == bench.FACTORED["gaussian"](8) < points["gaussian"] / 10


def test_regions_of_unknown_evaluator_have_no_count():
    split = {("gaussian", 8): (5, 0, 0), ("oscillatory", 8): (7, 0, 0)}
    assert bench.kernel_flops(split, 1, "k_persistent")[0] is None
    assert bench.kernel_flops(split, 3, "k_replicated")[0] == 3 * (
        5 * bench.flops_per_region("gaussian", 8) + 7 * bench.flops_per_region("oscillatory", 8))
    assert bench.kernel_flops({("oscillatory", 8): (7, 0, 0)}, 1, "k_persistent")[0] == (
        7 * bench.flops_per_region("oscillatory", 8))
