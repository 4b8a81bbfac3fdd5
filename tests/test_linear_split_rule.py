"""Which 32-bit products go to the tensor cores: the rule against timings of both, and where the kernel's grid ends."""

import pytest

from freetoken_b200.kernels import ops


@pytest.mark.parametrize("rows,cols,k,split_us,library_us", [
    (600000, 8, 64, 155, 100), (600000, 8, 256, 292, 247), (75000, 16, 64, 21, 17.5), (75000, 32, 256, 40, 37), (300000, 32, 128, 106, 80),
    (100000, 64, 64, 36, 33), (100000, 64, 256, 63, 80), (100000, 128, 128, 58, 90), (100000, 129, 64, 110, 79), (100000, 129, 128, 127, 121),
    (100000, 129, 256, 159, 201), (8192, 1024, 16, 31.5, 20.6), (8192, 1024, 64, 33, 41), (65536, 1024, 128, 268, 359), (8192, 8192, 16, 210, 119),
    (2048, 4096, 1024, 126, 333), (60, 16384, 64, 8, 12), (60, 65536, 64, 25, 23), (60, 65536, 512, 67, 93), (130, 65536, 16, 45, 29),
    (130, 65536, 256, 79, 127), (4000, 300, 16, 9.6, 12.7), (6250, 96, 1024, 32, 38), (4688, 128, 64, 10.7, 15.3)])
def test_the_faster_product_is_named(rows, cols, k, split_us, library_us):
    assert ops.split_pays(rows, cols, k) == (split_us < library_us)


def test_more_rows_than_the_grid_holds_stay_with_the_library():
    most = 65535 * 128
    assert ops.split_pays(most, 128, 1024) and not ops.split_pays(most + 1, 128, 1024)
    assert not ops.split_pays(1 << 30, 4, 4096) and not ops.split_pays(47, 1 << 20, 1024)
