"""Single-level basket passes of every register-resident width (tiles of whole steps) against the FP64
oracle on the same points: full and partial last tiles, multi-group items, correlated and not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", range(1, 17))
@pytest.mark.parametrize("kind", ["gbm", "dupire", "gbm_uncorrelated"])
def test_basket_width_vs_oracle(gpu, orc, n, kind):
    rng = np.random.default_rng(n)
    S0, sig = 100.0 * rng.uniform(0.8, 1.2, n), rng.uniform(0.1, 0.4, n)
    A = rng.normal(size=(n, n))
    C = A @ A.T + 0.5 * np.eye(n)
    L = np.linalg.cholesky(C / np.sqrt(np.outer(np.diag(C), np.diag(C))))
    if kind == "dupire":
        m = gpu.multi_dupire(S0, L=L, mu=0.03, sigma0=0.2, alpha=0.3, beta_d=0.8, T=1.0)
    elif kind == "gbm":
        m = gpu.basket_gbm(S0, sig, L=L, weights=rng.dirichlet(np.ones(n)), mu=0.03, T=1.0)
    else:
        m = gpu.basket_gbm(S0, sig, mu=0.03, T=1.0)
    p = gpu.basket(0.95 * float(S0.mean()), 0.03, 1.0, n)
    for n_steps, N, off in ((1, 97, 3), (32 // n, 256, 0), (2 * (32 // n) + 1, 1000, 4097)):
        g = gpu.qmc_pass(m, p, n_steps, salt_base=5, R=2, offset=off, n_points=N)
        o = orc.qmc_sums(m, p, n_steps, None, salt_base=5, R=2, offset=off, N=N)
        assert (np.abs(g - o)[:, 0] / N < 2e-4 * (1 + np.abs(o[:, 0]) / N)).all(), (n_steps, g, o)


def test_basket_items_of_several_groups(gpu, orc):
    """Carried start words with tiles of 30 dimensions: a pass whose items hold several groups equals its halves."""
    n = 5
    m = gpu.basket_gbm(np.linspace(90, 110, n), np.linspace(0.1, 0.3, n), mu=0.03, T=1.0)
    p = gpu.basket(100.0, 0.03, 1.0, n)
    N = 1 << 20
    whole = gpu.qmc_pass(m, p, 13, R=4, n_points=N)
    assert gpu.debug_last_pass_layout()[0] >= 2 and gpu.debug_last_pass_layout()[1] == 32 * 3
    parts = sum(gpu.qmc_pass(m, p, 13, R=4, offset=i * (N // 64), n_points=N // 64) for i in range(64))
    assert np.allclose(whole, parts, rtol=1e-6)
