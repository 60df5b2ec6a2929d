"""Calls that run short of device memory (a limit on the engine's buffers stands in for a full device): what the engine
keeps for later calls gives way, and results keep their bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(gpu):
    """The engine with nothing kept from earlier calls; the limit is taken back at the end."""
    gpu.shutdown()
    gpu.init(0)
    yield gpu
    gpu.debug_device_memory(0)


def book(gpu, n, width, eps, seed=3):
    rng = np.random.default_rng(seed)
    return [gpu.book_option(100.0 * rng.uniform(0.8, 1.2, width), rng.uniform(0.1, 0.5, width), 100.0, 0.03, 1.0, eps, 5)
            for _ in range(n)]


def same(a, b):
    return all(x["price"] == y["price"] and x["std_error"] == y["std_error"] and np.array_equal(x["delta"], y["delta"])
               for x, y in zip(a, b))


@pytest.mark.parametrize("model,steps", [("gbm", 256), ("lv", 256), ("heston", 128)])
def test_adjoint_with_little_scratch(fresh, model, steps):
    gpu = fresh
    m = {"gbm": lambda: gpu.gbm(100.0, 0.03, 0.25, 1.0), "heston": lambda: gpu.heston(100.0, 0.03, 2.0, 0.04, 0.3, -0.5, 0.04, 1.0),
         "lv": lambda: gpu.localvol_grid(*gpu.config4_surface(), 100.0, 0.03, 2.0)}[model]()
    run = lambda: gpu.adjoint(m, gpu.asian(100.0), steps, R=16, offset=5, n_points=20000)
    want, nodes = run()
    full = gpu.debug_device_memory(0)
    gpu.shutdown()
    gpu.init(0)
    gpu.debug_device_memory(full // 5)
    got, got_nodes = run()
    assert gpu.debug_device_memory(0) <= full // 5
    assert all(got[k] == want[k] for k in ("price", "delta", "rho", "vega", "price_se"))
    if nodes is not None:
        assert np.abs(got_nodes - nodes).max() <= 1e-6 * np.abs(nodes).max()   # FP32 sums in another order
    gpu.debug_device_memory(1 << 20)
    gpu.shutdown()
    gpu.init(0)
    with pytest.raises(gpu.MCQError):   # not even one CTA's
        run()


def test_path_scratch_gives_way_to_a_pass(fresh):
    gpu = fresh
    m, p = gpu.gbm(100.0, 0.03, 0.25, 1.0), gpu.asian(100.0)
    want = gpu.qmc_pass(m, p, 256, R=32, n_points=1 << 15)
    gpu.shutdown()
    gpu.init(0)
    gpu.adjoint(m, p, 256, R=2, n_points=20000)
    held = gpu.debug_device_memory(0)
    gpu.debug_device_memory(held)
    assert np.array_equal(gpu.qmc_pass(m, p, 256, R=32, n_points=1 << 15), want)
    assert gpu.debug_device_memory(0) < held


def test_slabs_give_way_to_a_running_book(fresh):
    """A book that stores nothing itself, after one that left slabs of stored normals."""
    gpu = fresh
    first, second = book(gpu, 24, 6, 2e-2), book(gpu, 2, 16, 2e-2)
    want, _ = gpu.book_price(second)
    gpu.shutdown()
    gpu.init(0)
    gpu.book_price(first)
    held = gpu.debug_device_memory(0)
    assert held > 1 << 30
    gpu.debug_device_memory(held)
    got, _ = gpu.book_price(second)
    assert same(got, want) and gpu.debug_device_memory(0) < 1 << 30


def test_store_of_a_book_that_finds_no_room(fresh):
    gpu = fresh
    b = book(gpu, 24, 6, 2e-2)
    want, _ = gpu.book_price(b)
    full = gpu.debug_device_memory(0)
    gpu.shutdown()
    gpu.init(0)
    gpu.debug_device_memory(full - (1 << 29))   # one slab less at least
    got, _ = gpu.book_price(b)
    assert same(got, want) and gpu.debug_device_memory(0) <= full - (1 << 30)
