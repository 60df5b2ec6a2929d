"""Stored normals of the batched book: options of one level that share points read them from memory instead
of generating them.  The plain form stores nothing, so both must give the same bits, with slices that end
inside, at and beyond the stored range, and an option whose chunks lie partly beyond it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,eps", [((1, 2, 3, 4), 2e-2), ((5, 6, 8, 8, 7), 3e-2), ((9, 12, 11, 16, 3, 1), 4e-2),
                                        ((16, 16, 16), 5e-2)])
def test_stored_normals_give_the_same_bits(gpu, widths, eps):
    rng = np.random.default_rng(len(widths))
    book = []
    for i, d in enumerate(widths):
        S0, sig = 100.0 * rng.uniform(0.8, 1.2, d), rng.uniform(0.1, 0.5, d)
        book.append(gpu.book_option(S0, sig, 100.0, 0.03, 1.0, eps * (1.0 if i else 0.5), 5))
    a, sa = gpu.book_price(book, gpu.BOOK_BATCHED)
    b, _ = gpu.book_price(book, gpu.BOOK_PLAIN)
    assert max(x["n_samples"] for x in a) > 1 << 16
    for x, y in zip(a, b):
        assert x["price"] == y["price"] and x["std_error"] == y["std_error"] and x["n_samples"] == y["n_samples"]
        assert np.array_equal(x["delta"], y["delta"])
