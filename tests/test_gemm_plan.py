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
        _, splits = K.ops().gemm_plan(kind, m, n, k)
        steps = -(-k // step)
        per = -(-steps // splits)
        assert (splits - 1) * per < steps, (m, n, k, splits)
        assert splits == 1 or (per >= 4 and splits * -(-m // 128) * -(-n // 128) <= 148)
        split += splits > 1
    assert split > 20
