"""How a dense product is cut: tile width and ranges of the contraction (host code, no GPU)."""
import random

import pytest

from bux_b200.ops import kernels as K


@pytest.mark.parametrize("kind,step", [(K.KIND_BF16, 64), (K.KIND_MXFP8, 128)])
def test_no_range_of_the_contraction_is_empty(kind, step):
    """Ranges are equal numbers of steps, as the launch cuts them: all of them start inside K."""
    rng = random.Random(3)
    shapes = [(16, 256, 2880), (1, 2048, 2880), (128, 128, 45 * step), (16, 6144, 4096)]
    shapes += [(rng.randint(1, 600), 128 * rng.randint(1, 40), 8 * rng.randint(1, 4000)) for _ in range(500)]
    split = 0
    for m, n, k in shapes:
        _, splits, _ = K.ops().gemm_plan(kind, m, n, k)
        steps = -(-k // step)
        per = -(-steps // splits)
        assert (splits - 1) * per < steps, (m, n, k, splits)
        assert splits == 1 or (per >= 4 and splits * -(-m // 128) * -(-n // 128) <= 148)
        split += splits > 1
    assert split > 20


@pytest.mark.parametrize("m,n,k,pairs", [
    (8192, 14336, 4096, True), (4096, 151936, 2048, True), (256, 151936, 2048, True),
    (128, 18952, 2048, False), (16, 201088, 2880, False), (384, 151936, 2048, False),   # rows fill half of the tiles
    (776, 5120, 2048, False), (640, 14336, 4096, False),                                # a wave more
    (14336, 4096, 448, False), (14336, 4096, 512, True),                                # short contractions
    (2048, 2048, 4096, False)])                                                         # under a wave
def test_pairs_of_sms_take_what_fills_them(m, n, k, pairs):
    assert K.ops().gemm_plan(K.KIND_BF16, m, n, k)[2] == pairs
    assert not K.ops().gemm_plan(K.KIND_MXFP8, m, n, k)[2]


@pytest.mark.parametrize("m,n,k,a_mn,width", [(3000, 2048, 18952, False, 256), (3000, 2048, 18944, False, 128),
                                              (3000, 2048, 18952, True, 256), (3008, 2048, 18952, True, 128),
                                              (776, 2048, 5128, False, 128)])
def test_narrow_tiles_and_rows_off_whole_lines(m, n, k, a_mn, width):
    """Three narrow waves against two wide ones, unless A's rows start off 128-byte lines; one against one."""
    assert K.ops().gemm_plan(K.KIND_BF16, m, n, k, 0, a_mn)[0] == width


@pytest.mark.parametrize("kind,m,n,k,splits", [
    (K.KIND_BF16, 16, 6144, 4096, 3), (K.KIND_BF16, 1, 2048, 2880, 9), (K.KIND_MXFP8, 16, 4096, 6144, 4),
    (K.KIND_BF16, 128, 2048, 512, 1), (K.KIND_BF16, 16, 8192, 1024, 1), (K.KIND_MXFP8, 300, 1152, 2048, 1)])
def test_short_contractions_are_not_split(kind, m, n, k, splits):
    """The ranges have to save more than the second launch and the partial sums cost."""
    assert K.ops().gemm_plan(kind, m, n, k)[1] == splits


@pytest.mark.parametrize("groups,rows_each,n,width", [
    (4, 75, 2880, 128), (4, 194, 2880, 256), (16, 256, 896, 128), (16, 512, 896, 256), (8, 40, 640, 128),
    (32, 97, 2880, 256), (32, 16, 2880, 128), (32, 97, 5760, 256), (8, 4, 4992, 128), (8, 512, 4992, 256),
    (8, 512, 384, 128), (8, 4, 512, 256)])
def test_ragged_widths_of_grouped_products(groups, rows_each, n, width):
    """Widths that 256 does not divide take the tile whose waves are shorter; measured either way."""
    rows = groups * (rows_each + 127)
    assert K._tile_width(n, K.KIND_BF16, K._grouped_row_tiles(rows, groups), 1.05) == width
    assert K._tile_width(n, K.KIND_MXFP8, K._grouped_row_tiles(rows, groups), 1.05) == (256 if n % 256 == 0 else 128)


@pytest.mark.parametrize("groups,m,n,width", [(32, 2880, 2880, 256), (128, 2048, 640, 256), (8, 384, 640, 128), (16, 2048, 896, 256)])
def test_ragged_widths_of_grouped_weight_gradients(groups, m, n, width):
    assert K._tile_width(n, K.KIND_BF16, groups * -(-m // 128)) == width
