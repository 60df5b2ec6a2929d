"""The adjoint at the limits of its range: 1024 steps with up to 4096 nodes, where fewer warps share an SM.  A surface
refined by whole cells is the same volatility, so the Greeks are those of the coarse one, whose node vegas are the
fine ones' gathered by the hat functions.  The surface is affine: a price on a kink has two derivatives, and which of
them a path takes depends on the last bit of its price."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def refine(x, k):
    """x on n uniform nodes, linearly on (n - 1) k + 1; and the weights W of x in the result (result = W x)."""
    n = len(x)
    pos = np.arange((n - 1) * k + 1) / k
    W = np.maximum(0.0, 1.0 - np.abs(pos[:, None] - np.arange(n)[None, :]))
    return W @ x, W


# 3836 nodes is the most that 24 warps hold at 1024 steps
@pytest.mark.parametrize("steps,nK,nt,kK,kt", [(1024, 22, 22, 3, 3), (1024, 28, 69, 1, 2), (1024, 28, 137, 1, 1), (1024, 28, 138, 1, 1),
                                              (992, 22, 22, 3, 3), (1024, 32, 32, 2, 2)])
@pytest.mark.parametrize("pay", ["asian", "eur"])   # (a lookback's step of the minimum may differ between the two)
def test_refined_surface(gpu, steps, nK, nt, kK, kt, pay):
    K, t = np.linspace(0.0, 400.0, nK), np.linspace(0.0, 2.0, nt)
    g = 0.2 + 0.0004 * (100.0 - K[None, :]) + 0.02 * t[:, None]
    (Kf, WK), (tf, Wt) = refine(K, kK), refine(t, kt)
    p = gpu.asian(95.0) if pay == "asian" else gpu.european(95.0, 0.03, 2.0)
    run = lambda K, t, g: gpu.adjoint(gpu.localvol_grid(K, t, g, 100.0, 0.03, 2.0), p, steps, R=2, offset=3, n_points=3000)
    fine, vf = run(Kf, tf, Wt @ g @ WK.T)
    if kK * kt > 1:
        few, vc = run(K, t, g)
        for k in ("price", "delta", "rho", "vega"):
            assert abs(fine[k] - few[k]) <= 2e-5 * max(1.0, abs(few[k])), (k, fine[k], few[k])
        assert np.abs(Wt.T @ vf @ WK - vc).max() <= 1e-4 * np.abs(vc).max()
    assert vf.shape == (len(tf), len(Kf)) and abs(vf.sum() - fine["vega"]) <= 1e-4 * abs(fine["vega"])
    q = gpu.qmc_pass(gpu.localvol_grid(Kf, tf, Wt @ g @ WK.T, 100.0, 0.03, 2.0), p, steps, R=2, offset=3, n_points=3000)
    assert abs(fine["price"] - q[:, 0].sum() / 6000) <= 2e-5 * fine["price"]
