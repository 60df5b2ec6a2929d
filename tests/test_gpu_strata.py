"""The normals that the priced passes form (one polynomial per 1/32 of the unit interval, points in
strata order) against AS241 of the same u, at the edges of tiles and points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Inside [1/32, 31/32): half an ulp of the last operation, at most half an ulp from the rounding of the
# term it adds, 0.12 ulp of fit, and AS241's own 1e-15: below 1.5 x 2^-23 relative.  The end strata add the
# documented 2^-22 of the hardware's base-2 logarithm, halved by the square root, and that root's 2^-23, each
# amplified by at most 1.5 (d log z / d log r at u = 1/32): below 5 x 2^-23, which is also normcdfinvf's
# documented maximum (the stream the second test compares with).
TOL_INNER, TOL_END = 1.5 * 2.0 ** -23, 5.0 * 2.0 ** -23


@pytest.mark.parametrize("n_steps,model", [(1, "gbm"), (16, "gbm"), (31, "gbm"), (32, "gbm"), (33, "gbm"),
                                           (50, "heston"), (512, "gbm")])
@pytest.mark.parametrize("offset", [0, 37, (1 << 22) - 3, (1 << 32) - 70])
def test_priced_normals_vs_as241(gpu, orc, n_steps, model, offset):
    m = gpu.gbm() if model == "gbm" else gpu.heston()
    D, R, n = n_steps * gpu.noise_dim(m), 2, 70
    dump = gpu.debug_pass_dump(m, n_steps, gpu.RAW, use_sobol=True, salt_base=42, R=R, offset=offset, n_points=n,
                               flags=gpu.FLAG_DUMP_PRICED)
    for r in range(R):
        ref = orc.sobol_hh_normal(42 + r, 0, D, offset, n).T
        x = orc.sobol_hh_u32(42 + r, 0, D, offset, n).T >> 27
        tol = np.where((x == 0) | (x == 31), TOL_END, TOL_INNER)
        err = np.abs(dump[r] - ref)
        assert (err <= tol * np.abs(ref)).all(), (r, np.argwhere(err > tol * np.abs(ref))[:3])


@pytest.mark.parametrize("model,n_steps,R,n,offset", [("gbm", 33, 2, 1 << 20, 5), ("heston", 32, 3, 700000, 1 << 21)])
def test_priced_normals_of_carried_groups(gpu, model, n_steps, R, n, offset):
    """Items of several groups carry each tile's packed start word: the same normals as the stream's."""
    m = gpu.gbm() if model == "gbm" else gpu.heston()
    dump = gpu.debug_pass_dump(m, n_steps, gpu.RAW, use_sobol=True, salt_base=11, R=R, offset=offset, n_points=n,
                               flags=gpu.FLAG_DUMP_PRICED)
    gpi, carry = gpu.debug_last_pass_layout()
    assert gpi >= 2 and carry > 0
    for r in range(R):
        ref = gpu.sobol_hh_normal(11 + r, 0, n_steps * gpu.noise_dim(m), offset, n).T.astype(np.float64)
        assert (np.abs(dump[r] - ref) <= (TOL_INNER + TOL_END) * np.abs(ref)).all()


@pytest.mark.parametrize("model,n_steps", [("gbm", 1), ("gbm", 33), ("heston", 50)])
@pytest.mark.parametrize("first", [0, 1000, (1 << 32) - 20])
def test_counter_based_normals_vs_fp64(gpu, orc, model, n_steps, first):
    """Box-Muller on Philox words: an ulp each from the logarithm's fit and rounding (halved by the root), the root,
    the sine or cosine and the product: below 4 x 2^-23 relative, plus the sine's 2^-23 2^-23 at its zeros."""
    m = gpu.gbm() if model == "gbm" else gpu.heston()
    D, n = n_steps * gpu.noise_dim(m), 40
    dump = gpu.debug_pass_dump(m, n_steps, gpu.RAW, use_sobol=False, seed=9, salt_base=3, R=2, offset=first & 0xffffffff,
                               n_points=n)
    for r in range(2):
        for i in range(n):
            ref = orc.philox_normals(9, 3 + r, (first & 0xffffffff) + i, D)
            assert (np.abs(dump[r, i] - ref) <= 4 * 2.0 ** -23 * np.abs(ref) + 2.0 ** -44).all(), (r, i)
