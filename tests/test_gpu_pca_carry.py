"""Start words carried from tile to tile of the tensor-core PCA pass: runs of many tiles that cross replicas give the
increments of short ones, which walk every word, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R,offset,n", [(64, 3, 37, 60001), (128, 2, 4096, 40000), (256, 2, 100001, 30001)])
def test_long_runs_give_the_increments_of_short_ones(gpu, N, R, offset, n):
    m, pca = gpu.gbm(100.0, 0.03, 0.25, 1.0), gpu.pca_create(N, 1.0)
    dump = lambda o, k: gpu.debug_pass_dump(m, N, noise=gpu.PCA, bb=pca, R=R, offset=o, n_points=k,
                                            flags=gpu.FLAG_DUMP_PRICED)
    full = dump(offset, n)
    for at in (0, 250, 1000, n // 3, n // 2 + 7, n - 300):
        assert np.array_equal(full[:, at:at + 300], dump(offset + at, 300))
