"""Which layouts of [..., T, H, D] the norm + RoPE kernel may walk with one stride between tokens."""
import itertools

import pytest
import torch

from bux_b200.ops import kernels as K


def _layouts():
    base = torch.arange(6 * 5 * 4 * 64, dtype=torch.float32).to(torch.bfloat16)
    for b, t, h in itertools.product((1, 2), (1, 3), (1, 2)):
        dense = base[: b * t * h * 64].view(b, t, h, 64)
        yield "dense", dense
        yield "tokens of a longer row", base[: b * 5 * h * 64].view(b, 5, h, 64)[:, 1:1 + t]
        yield "columns of wider rows", base[: b * t * 3 * h * 64].view(b, t, 3 * h, 64)[:, :, h:2 * h]
        yield "some heads", base[: b * t * 2 * h * 64].view(b, t, 2 * h, 64)[:, :, ::2]
        yield "heads first", base[: b * t * h * 64].view(b, h, t, 64).transpose(1, 2)
        yield "batch inside", base[: b * t * h * 64].view(t, b, h, 64).transpose(0, 1)
        yield "every other column", base[: b * t * h * 128].view(b, t, h, 128)[..., ::2]
        yield "one token for all", dense[:, :1].expand(b, 3, h, 64)
        yield "one row for all", dense[:1].expand(3, t, h, 64)
        yield "between 16-byte boundaries", base[1:1 + b * t * h * 64].view(b, t, h, 64)
        yield "odd wide rows", base[: b * t * (h * 64 + 4)].view(b, t, h * 64 + 4)[..., : h * 64].unflatten(-1, (h, 64))


@pytest.mark.parametrize("name,x", list(_layouts()), ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v.shape)))
def test_a_walk_by_the_token_stride_reads_the_tensor(name, x):
    """A stride that is given reads x's tokens in order, inside its storage and on 16-byte boundaries;
    whatever has none is copied into a layout that has one, although PyTorch may call it contiguous."""
    for y in (x, K.walkable(x)):
        step = K.token_stride(y)
        if step is None:
            assert y is x
            continue
        tokens, heads = y.shape[0] * y.shape[1], y.shape[2]
        first = y.storage_offset()
        assert first + (tokens - 1) * step + heads * 64 <= y.untyped_storage().nbytes() // 2
        assert step >= heads * 64 and step % 8 == 0 and y.data_ptr() % 16 == 0
        assert torch.equal(y.as_strided((tokens, heads, 64), (step, 64, 1), first), x.reshape(tokens, heads, 64))
    assert K.token_stride(K.walkable(x)) is not None
    if name in ("dense", "columns of wider rows"):
        assert K.walkable(x) is x   # read in place


def test_fewer_than_three_dimensions_have_no_tokens():
    assert K.token_stride(torch.zeros(4, 64).bfloat16()) is None
