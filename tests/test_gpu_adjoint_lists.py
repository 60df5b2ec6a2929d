"""The adjoint's waiting lists: paths of consecutive groups share a reverse sweep when they are in the
money, so a range priced whole, cut at odd places or point by point gives the same Greeks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["gbm", "lv", "heston"])
@pytest.mark.parametrize("pay", ["asian", "eur", "lookback"])
@pytest.mark.parametrize("moneyness", [0.5, 1.0, 1.3])
def test_range_equals_its_parts(gpu, model, pay, moneyness):
    m = {"gbm": lambda: gpu.gbm(100.0, 0.03, 0.25, 1.0), "heston": lambda: gpu.heston(100.0, 0.03, 2.0, 0.04, 0.3, -0.5, 0.04, 1.0),
         "lv": lambda: gpu.localvol_grid(*gpu.config4_surface(), 100.0, 0.03, 2.0)}[model]()
    K = 100.0 * moneyness
    p = {"asian": gpu.asian(K), "eur": gpu.european(K, 0.03, m.T), "lookback": gpu.lookback(0.25)}[pay]
    # 16 x 8100 points: items of two groups (148 x 24 items); cuts inside a group and at one point
    cuts = [0, 1, 33, 4096, 4127, 8100]
    whole, nodes = gpu.adjoint(m, p, 64, R=16, offset=7, n_points=cuts[-1])
    parts = [(b - a, gpu.adjoint(m, p, 64, R=16, offset=7 + a, n_points=b - a)) for a, b in zip(cuts, cuts[1:])]
    for k in ("price", "delta", "rho", "vega"):
        v = sum(n * g[k] for n, (g, _) in parts) / cuts[-1]
        assert abs(whole[k] - v) <= 2e-6 * max(abs(v), 1e-3), (k, whole[k], v)
    if nodes is not None:
        v = sum(n * x for n, (_, x) in parts) / cuts[-1]
        assert np.abs(nodes - v).max() <= 1e-5 * np.abs(v).max()
