"""The no-allocation pass carries the start words of every path length it takes (up to 16 tiles), as the allocating
pass does, and gives its sums; also from a captured graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,steps", [("gbm", 384), ("gbm", 385), ("gbm", 512), ("heston", 256), ("dupire", 500)])
def test_long_paths_carry_their_start_words(gpu, model, steps):
    import torch
    m = {"gbm": lambda: gpu.gbm(100.0, 0.03, 0.25, 1.0), "dupire": lambda: gpu.dupire(100.0, 0.05, 0.2, 0.5, 0.7, 1.0),
         "heston": lambda: gpu.heston(100.0, 0.02, 2.0, 0.04, 0.3, -0.7, 0.04, 1.0)}[model]()
    p, R, n = gpu.asian(100.0), 32, 1 << 16   # 2 groups an item
    tiles = -(-steps * (2 if model == "heston" else 1) // 32)
    out = torch.zeros(2, R, 2, dtype=torch.float64, device="cuda")
    gpu.qmc_pass_noalloc(m, p, steps, out[0].data_ptr(), 0, salt_base=9, R=R, offset=77, n_points=n)
    assert gpu.debug_noalloc_layout() == (2, 32 * tiles)
    gpu.qmc_pass_device(m, p, steps, out[1].data_ptr(), 0, salt_base=9, R=R, offset=77, n_points=n)
    torch.cuda.synchronize()
    assert np.array_equal(out[0].cpu().numpy(), out[1].cpu().numpy())


@pytest.mark.parametrize("steps", [8, 100, 512])
def test_captured_pass(gpu, steps):
    import torch
    m, p, R = gpu.gbm(100.0, 0.03, 0.25, 1.0), gpu.asian(100.0), 32
    out = torch.zeros(R, 2, dtype=torch.float64, device="cuda")
    run = lambda s: gpu.qmc_pass_noalloc(m, p, steps, out.data_ptr(), s.cuda_stream, salt_base=5, R=R, n_points=1 << 16)
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    run(s)
    s.synchronize()
    want = out.cpu().numpy().copy()
    with torch.cuda.graph(g, stream=s):
        run(s)
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
