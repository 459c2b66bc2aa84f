"""Kernels whose tile is chosen by size, at the sizes where a tile, a chunk or a group ends in the middle."""
import pytest

import darknet_b200 as dn
from conftest import parity
from test_gpu_layers import conv_case, oracle_conv, run_conv

pytestmark = pytest.mark.gpu

FP32_TILES = {   # tile of the fp32 GEMM -> cases; 296 blocks of 128 x 64 (or x 32) fill an SM twice
    "large_tile_64_filters_ragged": dict(b=5, c=5, h=89, w=87, n=65, size=3),
    "large_tile_32_filters": dict(b=5, c=9, h=90, w=86, n=31, size=3, stride=1, act="linear"),
    "large_tile_1x1_odd_channels": dict(b=6, c=21, h=81, w=83, n=70, size=1),
    "small_tile_one_pixel_over": dict(b=1, c=10, h=3, w=11, n=33, size=3),
    "small_tile_stride2": dict(b=2, c=24, h=9, w=13, n=17, size=3, stride=2),
    "small_tile_1x1_one_channel_over": dict(b=1, c=17, h=5, w=7, n=18, size=1),
    "groups_off_four_channel_boundary": dict(b=2, c=36, h=9, w=10, n=38, size=3, groups=2),
    "groups_of_four_channels": dict(b=2, c=16, h=9, w=10, n=40, size=3, groups=2),
    "slab_4": dict(b=2, c=24, h=7, w=9, n=9, size=3, groups=3),
    "slab_8": dict(b=2, c=12, h=7, w=9, n=15, size=3, groups=3),
    "slab_16": dict(b=1, c=6, h=9, w=15, n=15, size=3, pad=0),
}


@pytest.mark.parametrize("name", list(FP32_TILES))
@pytest.mark.parametrize("layouts", [("nchw", "nchw"), ("nchw", "nhwc"), ("nhwc", "nhwc")])
def test_fp32_gemm_tiles(name, layouts):
    """Tolerance: a sum of K fp32 products differs from the checker's by at most about K * 2^-24 of its largest partial sum
    (K <= 324 here: 2e-5 in the worst case, its square root typically), so 1e-5 of the layer's maximum as for the other fp32 cases."""
    case = conv_case(700, **FP32_TILES[name])
    plan, got, _ = run_conv(case, dn.MODE_FP32, layouts[0], layouts[1])
    assert plan.kernel == "direct_fp32"
    parity(got, oracle_conv(case), 1e-5)


@pytest.mark.parametrize("name", ["groups_of_four_channels", "groups_off_four_channel_boundary", "slab_4"])
def test_grouped_layers_with_bf16_storage(name):
    """A grouped layer of a BF16 network: bf16 in, fp32 sums, bf16 out.  The input is rounded first, so what is left is the
    output's rounding, 2^-9 of each value."""
    from gpu_util import bf16_round
    case = conv_case(701, **FP32_TILES[name])
    case["x"] = bf16_round(case["x"])
    _, got, _ = run_conv(case, dn.MODE_BF16, "nhwc", "nhwc")
    parity(got, oracle_conv(case), 2 ** -8)
