"""How the products of several rows are cut up (host side of lum_gemm.cu, no GPU): rows per chunk and ranges of the inner dimension."""
import ctypes as C
import math

import pytest

SMS = 148
# (outputs, inner dimension): the linear layers and heads of the configured decoders, a narrow and a long one
PRODUCTS = [(6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (128256, 4096), (6144, 2560), (2560, 4096), (19456, 2560), (2560, 9728), (9728, 2560),
            (512, 512), (28672, 14336), (16384, 16384), (65536, 16384)]
ROWS = [1, 2, 5, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 80, 81, 96, 112, 128, 129, 200, 256, 257, 300, 387, 512, 600, 1000, 1021, 2048, 4000, 4096]


class Shape(C.Structure):
    _fields_ = [("nc", C.c_int), ("ks", C.c_int)]


@pytest.fixture(scope="module")
def shape(pkg):
    f = pkg.load_library()["_ZN3lum10gemm_shapeEiiii"]              # lum::gemm_shape(outputs, rows, inner, SMs)
    f.restype, f.argtypes = Shape, [C.c_int] * 4
    return lambda n, m, k: f(n, m, k, SMS)


def coarse_split(n, m, k):
    """The split that chunks of 32, 64 or 128 rows and items of 128 or 256 outputs ask for: fewer ranges than this lengthen the tensor core's sums."""
    nc = 32 if m <= 32 else 64 if m <= 64 else 128
    items, tiles = math.ceil(n / (256 if m > 64 else 128)) * math.ceil(m / nc), k // 512
    tile_us, plane_us = (14.4 if m > 64 else 16 * (0.16 + 0.43 * nc / 128)), m * n * 8 / 6.5e6

    def cost(s):
        return math.ceil(items * s / SMS) * (tiles / s + 0.33) * tile_us + (s - 1) * plane_us

    best = 1
    for s in range(2, min(8, tiles) + 1):
        if cost(s) < cost(best) * 0.97:
            best = s
    return best


@pytest.mark.parametrize("n,k", PRODUCTS)
def test_ranges_are_never_longer_than_the_coarse_split(shape, n, k):
    for m in ROWS:
        s = shape(n, m, k)
        assert s.nc % 16 == 0 and (s.nc in (16, 32, 64) and s.nc >= m if m <= 64 else 80 <= s.nc <= 128)
        assert coarse_split(n, m, k) <= s.ks <= min(8, k // 512), f"{m} rows"


@pytest.mark.parametrize("n,k", PRODUCTS)
def test_shapes_hold_for_blocks_of_sixteen_rows(shape, n, k):
    for block in [0, 1, 2, 3, 4, 5, 7, 8, 15, 24, 31, 63, 127, 128, 200, 255]:
        first = shape(n, 16 * block + 1, k)
        assert all((s.nc, s.ks) == (first.nc, first.ks) for s in (shape(n, 16 * block + i, k) for i in range(2, 17))), f"rows from {16 * block + 1} on"


@pytest.mark.parametrize("n,k", PRODUCTS)
@pytest.mark.parametrize("cap", [1, 32, 33, 387, 1024, 4096])
def test_room_for_partial_sums_covers_every_row_count(pkg, shape, n, k, cap):
    f = pkg.load_library()["_ZN3lum15gemm_parts_rowsEiiii"]          # lum::gemm_parts_rows(outputs, inner, most rows, SMs)
    f.restype, f.argtypes = C.c_size_t, [C.c_int] * 4
    assert f(n, k, cap, SMS) == max(m * shape(n, m, k).ks for m in range(1, cap + 1))
