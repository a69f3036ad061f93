"""Host-side logic that needs no GPU: the learned angle's training targets, the bench's
launch count, and the universe sharding helpers."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def test_theta_target_monotone_and_interpolated():
    from nbh import learned as LR
    grid = (0.4, 0.5, 0.6, 0.7)
    # rows = grid angles, columns = samples
    E = np.array([[1, 1, 1, 9],
                  [2, 5, 1, 9],
                  [9, 2, 1, 9],
                  [20, 20, 1, 9]], float)
    mono = np.exp(LR.theta_target(E, 3.0, grid=grid))
    loose = np.exp(LR.theta_target(E, 3.0, grid=grid, monotone=False))
    # sample 0: passes at 0.4 and 0.5, fails at 0.6 -> between 0.5 and 0.6 (log-interpolated)
    assert 0.5 < mono[0] < 0.6 and mono[0] == loose[0]
    # sample 1: fails at 0.5, passes at 0.6 by luck -> monotone stops below 0.5
    assert 0.4 < mono[1] < 0.5 and loose[1] > 0.6
    # sample 2: passes everywhere -> the largest grid angle
    assert abs(mono[2] - 0.7) < 1e-12
    # sample 3: fails everywhere -> the floor
    assert abs(mono[3] - 0.3) < 1e-12


def test_graph_launch_count_follows_the_build_schedule():
    import bench
    # bbox, link, summarize, sort, force, item order, integrate = 7, plus the build
    assert bench.graph_launches() == 7 + 3 + 4                 # five phases, bucketed
    assert bench.graph_launches(3, 1) == 7 + 1 + 2 * 4              # one lock phase, two bucketed passes
    assert bench.graph_launches(5, 2) == 7 + 5
    assert bench.graph_launches(1, 2) == 7 + 1
    assert bench.graph_launches(1, 1) == 7 + 1                 # one pass has no bucketed completion


def test_step_launch_count_follows_the_reported_schedule():
    import bench
    tune = dict(build_phases=3, build_buckets=1, top_phase=4)
    staged = bench.graph_launches(3, 1) - 1                    # (the work-item order is part of integrate)
    assert bench.step_launches([1000]) == bench.step_launches([1000], tune) == 3
    assert bench.step_launches([1000, 50]) == bench.step_launches([1000, 50], tune) == 4
    assert bench.step_launches([1000], {**tune, "top_phase": 1}) == staged - 4   # the tuner left the one launch
    assert bench.step_launches([1000], {**tune, "top_phase": 2}) == staged
    assert bench.step_launches([6000]) == staged - 4           # the whole 1/16 sample in the first phase
    assert bench.step_launches([1 << 20], {**tune, "top_phase": 3}) == staged


def test_workload_shapes():
    import argparse
    import bench
    arrs, counts = bench.workload(argparse.Namespace(workload="ensemble", n=16, seed=5), 5)
    assert counts is not None and len(counts) == 16 and arrs[0].size == counts.sum()
    assert counts.min() >= 1024 and counts.max() <= 65536
    arrs, counts = bench.workload(argparse.Namespace(workload="ball", n=1000, seed=5), 5)
    assert counts is None and arrs[0].size == 1000
    r = np.sqrt(arrs[0] ** 2 + arrs[1] ** 2 + arrs[2] ** 2)
    assert r.max() <= 1.0 + 1e-6


def test_p99_ratio_interval_of_paired_errors():
    """The bootstrap interval of the learned-over-plain p99 ratio: identical arms give
    exactly 1; an arm scaled by 0.9 gives exactly 0.9 (every resample scales alike); and the
    interval of two unrelated arms holds their point ratio."""
    import numpy as np
    import bench
    rng = np.random.default_rng(3)
    ep = rng.lognormal(-7.0, 1.0, size=(8, 4096))
    assert bench._p99_ratio_interval(ep, ep, np) == [1.0, 1.0]
    lo, hi = bench._p99_ratio_interval(0.9 * ep, ep, np)
    assert abs(lo - 0.9) < 1e-12 and abs(hi - 0.9) < 1e-12
    el = rng.lognormal(-7.1, 0.9, size=(8, 4096))
    point = np.percentile(el, 99, axis=1).mean() / np.percentile(ep, 99, axis=1).mean()
    lo, hi = bench._p99_ratio_interval(el, ep, np)
    assert lo < point < hi and hi - lo < 0.2


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000])
def test_feature_normalisation(n):
    """Row after row in FP32; other memory orders and a column that divides by zero as in numpy."""
    from nbh import learned
    r = np.random.default_rng(n)
    X = (r.standard_normal((n, 12)) * np.exp(r.uniform(-4, 4, 12)) + 3).astype(np.float32)
    X[:, 5] = 2.0
    s = np.zeros(12, np.float32)
    for row in X:
        s += row
    mean = s / np.float32(n)
    s[:] = 0
    for row in (X - mean) * (X - mean):
        s += row
    std = np.maximum(np.sqrt(s / np.float32(n)), np.float32(0.05))
    got = learned._normalize(X, 0.05)
    for a, b in zip(got, (mean, std, (X - mean) / std)):
        assert a.dtype == np.float32 and a.flags.c_contiguous
        np.testing.assert_array_equal(a, b)
    other = learned._normalize(np.asfortranarray(X), 0.05)       # sums in another order
    bound = n * 2.0 ** -24 * np.abs(X).sum(0) / n                # of either order's sum
    assert (np.abs(other[0] - mean) <= 2 * bound).all() and other[2].flags.c_contiguous
    with np.errstate(invalid="ignore", divide="ignore"):
        assert np.isnan(learned._normalize(X, 0.0)[2][:, 5]).all()
