"""Books that do read stored normals: enough options of a level share its points, some end inside the stored range and
one goes far beyond it.  Bits as in the plain form, which stores nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths", [(1,) * 12, (2,) * 12, (3, 4) * 6, (5, 6, 7, 8) * 4, (9, 10) * 6, (11,) * 12, (12,) * 12,
                                    (13, 16, 14, 15) * 4, (16, 1, 12, 11, 8, 4, 16, 9, 10, 5) * 2])
def test_stored_ranges(gpu, widths):
    rng = np.random.default_rng(len(widths) + sum(widths))
    book = []
    for i, d in enumerate(widths):
        S0, sig = 100.0 * rng.uniform(0.8, 1.2, d), rng.uniform(0.2, 0.5, d)
        # the same tolerance for most: their slices are about as long; the first option's many times longer
        eps = 2e-2 * (0.25 if i == 0 else rng.uniform(1.0, 1.5))
        book.append(gpu.book_option(S0, sig, 100.0, 0.03, 1.0, eps, 5))
    a, _ = gpu.book_price(book, gpu.BOOK_BATCHED)
    stored = [gpu.debug_book_stored(l) for l in range(8)]
    assert stored[0] >= 1024 and all(s % 1024 == 0 for s in stored)
    assert 16 * sum(stored) < a[0]["n_samples"]   # (16 replicas)
    b, _ = gpu.book_price(book, gpu.BOOK_PLAIN)
    for x, y in zip(a, b):
        assert x["price"] == y["price"] and x["std_error"] == y["std_error"] and x["n_samples"] == y["n_samples"]
        assert np.array_equal(x["delta"], y["delta"])
