"""Asynchronous passes on several callers' streams share the engine's scratch: each gives the sums of a synchronous
pass, in whatever order the streams take turns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turns", ["ab", "abab", "-a", "a-b", "aab-a"])   # streams a, b and the engine's own (-)
def test_passes_on_several_streams(gpu, turns):
    import torch
    K, t = np.linspace(50, 150, 9), np.linspace(0, 2, 5)
    lv = gpu.localvol_grid(K, t, 0.2 + 0.001 * np.abs(K[None, :] - 100) * (1 + t[:, None]), 100.0, 0.03, 1.0)
    # one request per turn: another model (its parameter arrays), salt (direction words) and size (item records)
    req = [(lv if i % 2 else gpu.gbm(100.0, 0.03, 0.25, 1.0), 192 - 32 * i, 1000 + 7 * i, (1 << 18) - 4096 * i)
           for i in range(len(turns))]
    p, R = gpu.asian(100.0), 16
    want = [gpu.qmc_pass(m, p, n, salt_base=s, R=R, n_points=k) for m, n, s, k in req]
    streams = {"a": torch.cuda.Stream(), "b": torch.cuda.Stream()}
    out = [torch.zeros(R, 2, dtype=torch.float64, device="cuda") for _ in req]
    torch.cuda.synchronize()
    for (m, n, s, k), o, who in zip(req, out, turns):
        gpu.qmc_pass_device(m, p, n, o.data_ptr(), streams[who].cuda_stream if who != "-" else 0, salt_base=s, R=R,
                            n_points=k)
    torch.cuda.synchronize()
    for o, w in zip(out, want):
        assert np.array_equal(o.cpu().numpy(), w)


def test_failed_pass_leaves_the_streams_ordered(gpu):
    """A request that is refused between good ones on other streams."""
    import torch
    m, p, R = gpu.gbm(100.0, 0.03, 0.25, 1.0), gpu.asian(100.0), 8
    want = gpu.qmc_pass(m, p, 128, salt_base=5, R=R, n_points=1 << 17)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    out = torch.zeros(2, R, 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    gpu.qmc_pass_device(m, p, 128, out[0].data_ptr(), a.cuda_stream, salt_base=5, R=R, n_points=1 << 17)
    with pytest.raises(gpu.MCQError):
        gpu.qmc_pass_device(m, p, 128, out[1].data_ptr(), b.cuda_stream, noise=gpu.BB, R=R, n_points=64)
    gpu.qmc_pass_device(m, p, 128, out[1].data_ptr(), b.cuda_stream, salt_base=5, R=R, n_points=1 << 17)
    torch.cuda.synchronize()
    assert np.array_equal(out[0].cpu().numpy(), want) and np.array_equal(out[1].cpu().numpy(), want)
