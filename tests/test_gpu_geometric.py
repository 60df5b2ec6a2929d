"""The geometric average as a running product: per-replica sums against FP64 paths on the same normals, from one
step up, at prices far from 1 and with paths that leave the positive numbers (payoff 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 2, 31, 32, 33, 100, 500])
@pytest.mark.parametrize("S0,sigma", [(100.0, 0.25), (3e30, 0.25), (2e-30, 0.25), (100.0, 3.0)])
def test_geometric_sums_against_fp64(gpu, steps, S0, sigma):
    R, n, mu = 2, 3000, 0.03
    m, p = gpu.gbm(S0, mu, sigma, 1.0), gpu.geom_asian(S0)
    sums = np.asarray(gpu.qmc_pass(m, p, steps, R=R, offset=5, n_points=n))
    z = gpu.debug_pass_dump(m, steps, R=R, offset=5, n_points=n, flags=gpu.FLAG_DUMP_PRICED).astype(np.float64)
    S = S0 * np.cumprod(1.0 + mu / steps + sigma * z / np.sqrt(steps), axis=2)
    alive = (S > 0).all(axis=2)
    G = np.exp(np.log(np.where(S > 0, S, 1.0)).mean(axis=2))
    want = np.where(alive, np.maximum(G - S0, 0.0), 0.0).sum(axis=1)
    # the tolerance of the per-replica sums against the oracle
    np.testing.assert_allclose(sums[:, 0], want, rtol=1e-4)
