"""A driver that sizes its first pass by the free device memory takes the same size whatever ran before it: memory that
the engine keeps between calls counts as free."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(gpu):
    """The engine with nothing kept from earlier calls."""
    gpu.shutdown()
    gpu.init(0)
    return gpu


def cv_samples(gpu, n_steps):
    m = gpu.gbm(100.0, 0.03, 0.25, 1.0)
    cfg = gpu.qmc_cfg(R=2, max_doublings=1, N0_per_replica=0)
    return gpu.run_qmc_cv(m, m, gpu.asian(100.0), gpu.geom_asian(100.0), 4.0, 1.0, 1e-9, n_steps, cfg)["n_samples"]


def test_first_pass_after_an_adjoint(fresh):
    import torch
    m, p = fresh.gbm(100.0, 0.03, 0.25, 1.0), fresh.asian(100.0)
    fresh.adjoint(m, p, 32, R=2, n_points=64)   # (loads the kernels)
    cv_samples(fresh, 20000)
    # a step count at which the size, the largest power of two that fits, halves if 0.1 to 0.8 % of the memory goes
    budget = int(torch.cuda.mem_get_info()[0] * 0.8) // 4
    steps = next(n for n in range(300, 1500) if 1.001 < budget // n / 2.0 ** ((budget // n).bit_length() - 1) < 1.008)
    first = cv_samples(fresh, steps)
    free = torch.cuda.mem_get_info()[0]
    fresh.adjoint(m, p, 1024, R=16, n_points=30000)
    assert free - torch.cuda.mem_get_info()[0] > 0.009 * free   # 24 warps x 148 keep two stretches of 1024 steps each
    assert cv_samples(fresh, steps) == first
