"""How kernels are cut up (host side of lum_gemm.cu and lum_moe.cu, no GPU): rows per chunk and ranges of the inner dimension of products of several
rows, rings of the expert kernels."""
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


def test_expert_kernels_take_every_size_whose_activations_fit(pkg):
    """200 KB of activation levels and block scales have always been taken, whatever else lies beside them."""
    lib = pkg.load_library()
    fit = lib["_ZN3lum12moe_ring_fitEmiPiS0_"]
    fit.restype, fit.argtypes = C.c_int, [C.c_size_t, C.c_int, C.POINTER(C.c_int), C.POINTER(C.c_int)]
    gate_up, down = lib["_ZN3lum17moe_gate_up_bytesEii"], lib["_ZN3lum14moe_down_bytesEiiii"]
    gate_up.restype, gate_up.argtypes, down.restype, down.argtypes = C.c_size_t, [C.c_int] * 2, C.c_size_t, [C.c_int] * 4
    stages, blocks = C.c_int(), C.c_int()

    def ring(act, k):
        ok = fit(act, k, C.byref(stages), C.byref(blocks))
        assert not ok or (1 <= stages.value <= 2 and 1 <= blocks.value <= min(96, k // 32) and act + 16 * 64 * stages.value * blocks.value <= 226 * 1024)
        return (stages.value, blocks.value) if ok else None

    for hidden in (32, 96, 2880, 4096, 16384, 47104, 50016, 65536):
        assert 3 * hidden + hidden // 8 <= 200 * 1024 and ring(gate_up(hidden, 8), hidden)
        for top_k in range(1, 9):
            most = max(f for f in range(32, 70000, 32) if top_k * ((3 * f + f // 8 + 15) // 16 * 16) <= 200 * 1024)
            for ffn in (32, 96, 2880, most):
                if ffn <= most:
                    assert ring(down(hidden, ffn, top_k, SMS), ffn), f"{hidden} x {ffn}, {top_k} experts"
    # the configured shape keeps whole rows in two stages
    assert ring(gate_up(2880, 4), 2880) == (2, 90) and ring(down(2880, 2880, 4, SMS), 2880) == (2, 90)
    assert ring(230 * 1024, 2880) is None
