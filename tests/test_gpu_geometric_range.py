"""Geometric averages at the ends of the FP32 range, where prices leave [2^-126, 2^126) or overflow (payoff 0, as the
compensated sum of logarithms gives), and in every form that carries the running product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 16, 33, 100])
@pytest.mark.parametrize("S0,sigma", [(1.2e38, 0.05), (3e-39, 0.25), (1.1e-38, 0.25), (3e38, 0.4)])
def test_ends_of_the_range(gpu, steps, S0, sigma):
    # few points: a lane adds its paths' payoffs in FP32, and their sum must not overflow; in the money, so that the
    # payoffs' relative error is of the order of the prices'
    R, n, mu, K = 2, 90, 0.03, 0.9 * S0
    m, p = gpu.gbm(S0, mu, sigma, 1.0), gpu.geom_asian(K)
    sums = np.asarray(gpu.qmc_pass(m, p, steps, R=R, offset=5, n_points=n))
    z = gpu.debug_pass_dump(m, steps, R=R, offset=5, n_points=n, flags=gpu.FLAG_DUMP_PRICED).astype(np.float64)
    S = S0 * np.cumprod(1.0 + mu / steps + sigma * z / np.sqrt(steps), axis=2)
    ok = ((S > 0) & (S <= np.finfo(np.float32).max)).all(axis=2)
    assert ok.any() and (S0 < 3e38 or not ok.all())
    G = np.exp(np.log(np.where(S > 0, S, 1.0)).mean(axis=2))
    want = np.where(ok, np.maximum(G - K, 0.0), 0.0).sum(axis=1)
    # that of the other geometric sums; a price held to 2^-149 is off by 5e-7 a step, at random
    np.testing.assert_allclose(sums[:, 0], want, rtol=1e-4)


def make_model(gpu, name):
    return {"gbm": lambda: gpu.gbm(100.0, 0.05, 0.2, 1.0), "dupire": lambda: gpu.dupire(100.0, 0.05, 0.2, 0.5, 0.7, 1.0),
            "heston": lambda: gpu.heston(100.0, 0.02, 2.0, 0.04, 0.3, -0.7, 0.04, 1.0)}[name]()


def close(g, o, N, tol=2e-4):   # the tolerance of the passes against the oracle; levels have twice that
    return (np.abs(g[:, 0] - o[:, 0]) / N < tol * (1 + np.abs(o[:, 0]) / N)).all()


@pytest.mark.parametrize("model", ["gbm", "dupire", "heston"])
@pytest.mark.parametrize("steps", [1, 15, 32, 100, 300])
def test_raw(gpu, orc, model, steps):
    m, p, N = make_model(gpu, model), gpu.geom_asian(100.0), 640
    g = gpu.qmc_pass(m, p, steps, salt_base=7, R=2, offset=13, n_points=N)
    assert close(g, orc.qmc_sums(m, p, steps, None, salt_base=7, R=2, offset=13, N=N), N)


@pytest.mark.parametrize("model", ["gbm", "dupire"])
@pytest.mark.parametrize("noise,steps", [("BB", 16), ("BB", 64), ("PCA", 8), ("PCA", 64), ("PCA", 96), ("PCA", 256)])
def test_orderings(gpu, orc, model, noise, steps):
    m, p, N = make_model(gpu, model), gpu.geom_asian(100.0), 512
    mode = getattr(gpu, noise)
    h = (gpu.bb_create if noise == "BB" else gpu.pca_create)(steps, 1.0)
    g = gpu.qmc_pass(m, p, steps, noise=mode, salt_base=77, R=2, offset=64, n_points=N, **{noise.lower(): h})
    o = orc.qmc_sums(m, p, steps, orc.noise(mode, steps, 1.0), salt_base=77, R=2, offset=64, N=N)
    h.close()
    assert close(g, o, N)


@pytest.mark.parametrize("model", ["gbm", "dupire", "heston"])
@pytest.mark.parametrize("steps,M", [(4, 2), (16, 4), (256, 2)])
@pytest.mark.parametrize("sobol", [True, False])
def test_levels(gpu, orc, model, steps, M, sobol):
    m, p, N = make_model(gpu, model), gpu.geom_asian(100.0), 640
    g = gpu.level_pass(m, p, steps, M, use_sobol=sobol, seed=9, salt_base=3, R=2, offset=0, n_points=N)
    o = orc.level_sums(m, p, steps, M, use_sobol=sobol, seed=9, salt_base=3, R=2, offset=0, N=N)
    assert close(g[:, [0]], o[:, [0]], N, 4e-4) and close(g[:, [2]], o[:, [2]], N, 4e-4)


@pytest.mark.parametrize("model", ["gbm", "dupire", "heston"])
def test_monte_carlo(gpu, orc, model):
    m, p, N = make_model(gpu, model), gpu.geom_asian(100.0), 2000
    g = gpu.mc_pass(m, p, 50, seed=5, stream_id=2, first_path=11, n_paths=N)
    o = orc.mc_sums(m, p, 50, 5, 2, 11, N)
    assert close(np.reshape(g, (1, 2)), np.reshape(o, (1, 2)), N)
