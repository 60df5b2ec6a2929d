"""The adjoint's waiting lists at the shortest and longest paths: a range priced whole gives its parts' Greeks, for paths
that are in the money seldom, half of the time and mostly, so that lists fill within a group, over groups and at a range's end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["gbm", "dupire", "lv"])
@pytest.mark.parametrize("steps", [32, 96, 512, 1024])
@pytest.mark.parametrize("moneyness", [0.8, 1.0, 1.6])
def test_range_equals_its_parts(gpu, model, steps, moneyness):
    m = {"gbm": lambda: gpu.gbm(100.0, 0.03, 0.25, 1.0), "dupire": lambda: gpu.dupire(100.0, 0.03, 0.25, 0.5, 0.7, 1.0),
         "lv": lambda: gpu.localvol_grid(*gpu.config4_surface(), 100.0, 0.03, 2.0)}[model]()
    p = gpu.asian(100.0 * moneyness)
    # 16 x 8100 points: items of two groups (148 x 24 items); cuts inside a group and at one point
    cuts = [0, 1, 33, 4096, 4127, 8100]
    whole, nodes = gpu.adjoint(m, p, steps, R=16, offset=7, n_points=cuts[-1])
    parts = [(b - a, gpu.adjoint(m, p, steps, R=16, offset=7 + a, n_points=b - a)) for a, b in zip(cuts, cuts[1:])]
    for k in ("price", "delta", "rho", "vega"):
        v = sum(n * g[k] for n, (g, _) in parts) / cuts[-1]
        assert abs(whole[k] - v) <= 2e-6 * max(abs(v), 1e-3), (k, whole[k], v)
    if nodes is not None:
        v = sum(n * x for n, (_, x) in parts) / cuts[-1]
        assert np.abs(nodes - v).max() <= 1e-5 * np.abs(v).max() + 1e-12
