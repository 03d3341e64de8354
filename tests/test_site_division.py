"""The division of a site by the row length as the sweep operator makes it,
site * ceil(2^20 / Y) >> 20 on 32 bits, for every lattice that it packs."""
import numpy as np
import pytest


@pytest.mark.parametrize("Y", range(2, 33))
def test_site_over_row_length(Y):
    site = np.arange(4096, dtype=np.uint64)
    product = site * np.uint64(((1 << 20) + Y - 1) // Y)
    assert product.max() < 1 << 32
    assert np.array_equal(product >> np.uint64(20), site // np.uint64(Y))
