"""Every CUDA kernel against the plain PyTorch fp32 statement of the same op."""
import pytest
import torch

from bux_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-12)).item()


@pytest.fixture(autouse=True)
def _status(cuda):
    from bux_b200.ops import kernels as K

    yield
    torch.cuda.synchronize()
    K.check_status(cuda)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k,bn", [(256, 512, 256, 256), (304, 264, 200, 128), (1024, 768, 2048, 256)])
def test_gemm_bf16(cuda, a_mn, b_mn, m, n, k, bn):
    from bux_b200.ops import kernels as K

    torch.manual_seed(0)
    a = torch.randn(m, k, device=cuda).bfloat16()
    b = torch.randn(n, k, device=cuda).bfloat16()
    want = a.float() @ b.float().t()
    a_in = a.t().contiguous() if a_mn else a
    b_in = b.t().contiguous() if b_mn else b
    got = K.gemm_bf16(a_in, b_in, a_mn=a_mn, b_mn=b_mn, bn=bn)
    assert rel_err(got, want) < 1e-2
    acc = torch.ones(m, n, device=cuda)
    K.gemm_bf16(a_in, b_in, a_mn=a_mn, b_mn=b_mn, out=acc, accumulate=True, bn=bn)
    assert rel_err(acc, want + 1) < 1e-2


def test_quant_mxfp8_matches_reference(cuda):
    from bux_b200.ops import kernels as K

    torch.manual_seed(1)
    x = (torch.randn(200, 384, device=cuda) * torch.logspace(-3, 3, 384, device=cuda)).bfloat16()
    q_row, sf_row, q_col, sf_col = K.quant_mxfp8(x, rowwise=True, colwise=True)
    rq, re = ref.quant_mxfp8(x)
    assert torch.equal(ref.unswizzle_scales(sf_row, 200, 12), re)
    assert torch.equal(q_row.view(torch.uint8), rq.view(torch.uint8))
    xt = torch.zeros(384, 256, device=cuda, dtype=torch.bfloat16)
    xt[:, :200] = x.t()
    tq, te = ref.quant_mxfp8(xt)
    # scale blocks past the last row are never written (they keep the pad byte)
    assert torch.equal(ref.unswizzle_scales(sf_col, 384, 8)[:, :7], te[:, :7])
    assert torch.equal(q_col.view(torch.uint8), tq.view(torch.uint8))


@pytest.mark.parametrize("rows,cols", [(1, 32), (31, 96), (129, 160), (300, 416)])
@pytest.mark.parametrize("shift", [0, 8])
def test_quant_mxfp8_ragged_gathered_and_shifted(cuda, rows, cols, shift):
    """Partial tiles both ways, a row gather with absent rows, NaN and infinities, and outputs that do
    not start on the 32-byte boundaries of the wide stores: the reference's bytes."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(2)
    src = torch.randn(40, cols, device=cuda).bfloat16()
    src[3, 5], src[4, 7] = float("nan"), float("inf")
    index = torch.randint(-1, 40, (rows,), device=cuda, dtype=torch.int32)
    x = torch.where(index[:, None] >= 0, src[index.clamp_min(0).long()], torch.zeros(1, device=cuda, dtype=src.dtype))
    r_pad = -(-rows // 128) * 128

    def buffer(n):
        return torch.empty(n + shift, dtype=torch.uint8, device=cuda)[shift:]

    q_row, q_col = buffer(rows * cols), buffer(cols * r_pad)
    # the scale tiles are whole 16-byte stores whatever the values' start
    sf_row, sf_col = (torch.empty(K.sf_bytes(r, c), dtype=torch.uint8, device=cuda) for r, c in ((rows, cols), (cols, r_pad)))
    K.ops().quant_mxfp8(src, index, None, q_row, sf_row, q_col, sf_col, rows, cols, r_pad, 1, 0)
    xt = torch.zeros(cols, r_pad, device=cuda, dtype=torch.bfloat16)
    xt[:, :rows] = x.t()
    for got, sf, plain in ((q_row.view(rows, cols), sf_row, x), (q_col.view(cols, r_pad), sf_col, xt)):
        finite = plain.isfinite().unflatten(-1, (-1, 32)).all(-1)
        want, scales = ref.quant_mxfp8(plain.nan_to_num(0, 0, 0))
        r, c = scales.shape
        assert torch.equal(ref.unswizzle_scales(sf, r, c)[finite], scales[finite])
        same = (got == want.view(torch.uint8)).unflatten(-1, (-1, 32)).all(-1)
        assert same[finite].all()
        assert (got.view(torch.float8_e4m3fn).float().isnan() == plain.isnan()).all()


@pytest.mark.parametrize("m,n,k,bn", [(128, 128, 128, 128), (256, 384, 512, 128), (1000, 768, 2048, 128),
                                      (512, 512, 1024, 256)])
def test_gemm_mxfp8(cuda, m, n, k, bn):
    from bux_b200.ops import kernels as K

    torch.manual_seed(2)
    a = torch.randn(m, k, device=cuda).bfloat16()
    b = torch.randn(n, k, device=cuda).bfloat16()
    aq, asf, _, _ = K.quant_mxfp8(a)
    bq, bsf, _, _ = K.quant_mxfp8(b)
    want = ref.gemm_mxfp8(*ref.quant_mxfp8(a), *ref.quant_mxfp8(b))
    got = K.gemm_mxfp8(aq, asf, bq, bsf, m, n, k, bn=bn)
    assert rel_err(got, want) < 1e-2


@pytest.mark.parametrize("kind", ["bf16", "mxfp8"])
def test_grouped_gemm_rows(cuda, kind):
    from bux_b200.ops import kernels as K

    torch.manual_seed(3)
    counts = [128, 0, 384, 256]
    n, k = 256, 512
    offsets = torch.tensor([0, *torch.tensor(counts).cumsum(0).tolist()], dtype=torch.int32, device=cuda)
    rows = sum(counts)
    a = torch.randn(rows, k, device=cuda).bfloat16()
    w = torch.randn(len(counts), n, k, device=cuda).bfloat16()
    want = torch.cat([a[offsets[g]:offsets[g + 1]].float() @ w[g].float().t() for g in range(len(counts))])
    if kind == "bf16":
        got = K.grouped_gemm(a, w.view(-1, k), offsets, n, k)
        tol = 1e-2
    else:
        aq, asf, _, _ = K.quant_mxfp8(a)
        wq, wsf, _, _ = K.quant_mxfp8(w.view(-1, k))
        got = K.grouped_gemm(aq, wq, offsets, n, k, kind=K.KIND_MXFP8, asf=asf, bsf=wsf)
        tol = 6e-2
    assert rel_err(got, want) < tol


def test_grouped_gemm_contraction(cuda):
    from bux_b200.ops import kernels as K

    torch.manual_seed(4)
    counts = [128, 0, 256]
    m, n = 256, 128
    offsets = torch.tensor([0, *torch.tensor(counts).cumsum(0).tolist()], dtype=torch.int32, device=cuda)
    rows = sum(counts)
    dy = torch.randn(rows, m, device=cuda).bfloat16()
    x = torch.randn(rows, n, device=cuda).bfloat16()
    want = torch.stack([dy[offsets[g]:offsets[g + 1]].float().t() @ x[offsets[g]:offsets[g + 1]].float()
                        for g in range(len(counts))])
    got = K.grouped_gemm_k(dy, x, offsets, m, n, a_mn=True, b_mn=True)
    assert rel_err(got, want) < 1e-2
    # gradients kept in bf16: written by one call, added to by the next (the chunks of a step)
    first = K.grouped_gemm_k(dy, x, offsets, m, n, a_mn=True, b_mn=True, out_dtype=torch.bfloat16)
    assert first.dtype == torch.bfloat16 and rel_err(first, want) < 1e-2
    again = K.grouped_gemm_k(dy, x, offsets, m, n, a_mn=True, b_mn=True, out=first, accumulate=True)
    assert again is first and rel_err(first, 2 * want) < 1e-2
    assert first[1].abs().max() == 0   # the empty group stays zero


def test_quant_mxfp8_of_blocks_without_numbers(cuda):
    """A block of nothing but NaN has the scale of an empty one (byte 0, 2^-127), one with a single
    number that number's, one with an infinity the largest; every NaN stays one."""
    from bux_b200.ops import kernels as K

    x = torch.full((128, 128), float("nan"), device=cuda).bfloat16()
    x[0, 32], x[1, 64], x[2, 96] = 448.0, -3.5, float("inf")
    want = torch.zeros(128, 4, dtype=torch.uint8, device=cuda)
    want[0, 1], want[1, 2], want[2, 3] = 127, 120, 254
    q, sf, qt, sft = K.quant_mxfp8(x, rowwise=True, colwise=True)
    assert torch.equal(ref.unswizzle_scales(sf, 128, 4), want)
    assert torch.equal(q.float().isnan(), x.isnan()) and torch.equal(qt.float().isnan(), x.t().isnan())
    assert q[0, 32].float() == 448 and q[1, 64].float() == -448 and q[2, 96].float() == 448
    cols = torch.zeros(128, 4, dtype=torch.uint8, device=cuda)
    cols[32, 0], cols[64, 0], cols[96, 0] = 127, 120, 254
    assert torch.equal(ref.unswizzle_scales(sft, 128, 4), cols)


@pytest.mark.parametrize("m,n", [(32, 8), (160, 264), (224, 648), (72, 96)])
@pytest.mark.parametrize("dtype,accumulate", [(torch.bfloat16, False), (torch.float32, False), (torch.float32, True)])
def test_grouped_contraction_with_ragged_outputs(cuda, m, n, dtype, accumulate):
    """Stacked outputs whose rows do not fill the tiles: whole 32-row boxes, and rows that are none (72).
    Each group's gradient stays in its own rows. Bounds as for the dense products."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(20)
    offsets = torch.tensor([0, 128, 128, 320], dtype=torch.int32, device=cuda)
    a, b = torch.randn(320, m, device=cuda).bfloat16(), torch.randn(320, n, device=cuda).bfloat16()
    want = torch.stack([a[:128].double().t() @ b[:128].double(), torch.zeros(m, n, device=cuda, dtype=torch.float64),
                        a[128:].double().t() @ b[128:].double()])
    out = torch.ones(3, m, n, device=cuda, dtype=dtype) if accumulate else None
    got = K.grouped_gemm_k(a, b, offsets, m, n, a_mn=True, b_mn=True, out=out, accumulate=accumulate, out_dtype=dtype)
    for g in range(3):
        assert rel_err(got[g], want[g] + int(accumulate)) < (4e-3 if dtype == torch.bfloat16 else 1e-6)
    assert accumulate or (got[1] == 0).all()


def test_rmsnorm(cuda):
    from bux_b200.ops import kernels as K

    torch.manual_seed(5)
    x = torch.randn(300, 512, device=cuda).bfloat16().requires_grad_()
    w = torch.randn(512, device=cuda).requires_grad_()
    y, rstd = K.rmsnorm_fwd(x.detach(), w.detach(), 1e-6)
    want = ref.rmsnorm(x, w, 1e-6)
    assert rel_err(y, want) < 1e-2
    dy = torch.randn_like(want)
    want.backward(dy)
    dx, dw = K.rmsnorm_bwd(x.detach(), w.detach(), dy, rstd)
    assert rel_err(dx, x.grad) < 2e-2
    assert rel_err(dw, w.grad) < 2e-2


@pytest.mark.parametrize("rows,d", [(1, 8), (5, 504), (3, 512), (9, 1032), (2, 2056), (5, 2880), (3, 4104), (2, 8192), (3, 8200),
                                    (592, 520), (593, 520), (601, 1032), (593, 2048), (601, 4104)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rmsnorm_widths(cuda, rows, d, shift):
    """The edges of each way of splitting a row, and gains that start between 16-byte boundaries.
    Bounds: outputs are rounded to bf16 (2^-9); dw is an fp32 sum of products of bf16 values."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(5)
    x, dy = (torch.randn(rows, d, device=cuda).bfloat16() for _ in range(2))
    w = torch.randn(d + shift, device=cuda)[shift:]
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    want = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * wd
    want.backward(dy.double())
    y, rstd = K.rmsnorm_fwd(x, w, 1e-6)
    dx, dw = K.rmsnorm_bwd(x, w, dy, rstd)
    assert rel_err(y, want) < 4e-3 and rel_err(dx, xd.grad) < 4e-3 and rel_err(dw, wd.grad) < 1e-5
    plain, r2 = K.rmsnorm_fwd(x, None, 1e-6)
    assert rel_err(plain, want / wd) < 4e-3 and rel_err(K.rmsnorm_bwd(x, None, dy, r2)[0], K.rmsnorm_bwd(x, torch.ones_like(w), dy, r2)[0]) < 1e-6


@pytest.mark.parametrize("tokens,heads,d", [(1, 1, 64), (7, 3, 128), (33, 5, 256), (50, 6, 64),
                                            (5000, 1, 128), (1600, 7, 64), (700, 5, 256), (1000, 6, 128)])
def test_norm_rope_odd_heads(cuda, tokens, heads, d):
    """Heads go four (backward: two) at a time, few of them one by one: counts that they do not divide, and a slice of wider
    rows. Bounds as for the RMSNorm, with one rotation more."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(6)
    wide = torch.randn(1, tokens, (heads + 1) * d, device=cuda).bfloat16()
    x = wide[..., d:].view(1, tokens, heads, d) if tokens == 1 else wide[..., d:].unflatten(-1, (heads, d))
    dy, w = torch.randn(1, tokens, heads, d, device=cuda).bfloat16(), torch.randn(d, device=cuda)
    cos, sin = ref.rope_tables(torch.arange(tokens, device=cuda)[None], d, 10000.0)
    xr, wr = x.float().requires_grad_(), w.clone().requires_grad_()
    want = ref.rmsnorm_rope(xr, wr, cos, sin, 1e-6)
    want.backward(dy.float())
    c2, s2 = cos.reshape(-1, d // 2).contiguous(), sin.reshape(-1, d // 2).contiguous()
    y, rstd = K.norm_rope_fwd(x, w, c2, s2, 1e-6)
    dx, dw = K.norm_rope_bwd(x, w, c2, s2, rstd, dy, 1e-6)
    assert rel_err(y, want) < 4e-3 and rel_err(dx, xr.grad) < 4e-3 and rel_err(dw, wr.grad) < 1e-5


@pytest.mark.parametrize("m,n,k", [(1, 8, 512), (16, 6144, 4096), (130, 136, 1000), (128, 256, 2048), (3, 2048, 568), (509, 1024, 3072), (16, 256, 2880),
                                   (1, 8, 2048), (130, 136, 2504), (3, 2048, 4088)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_small_products_are_split(cuda, m, n, k, a_mn, b_mn, dtype):
    """Products too small to fill the SMs, split and too short to be: one row, ragged edges of the tiles
    and of the last range of the contraction. Bounds: bf16 outputs are rounded once (2^-9); in fp32 the tensor core cuts its
    accumulator's low bits once per 16 terms, 2^-23 of it each time (measured 1.4e-6 at k = 4096)."""
    from bux_b200.ops import kernels as K

    if a_mn and m % 8:
        pytest.skip("an MN-major operand's rows are whole 16-byte pieces")
    torch.manual_seed(16)
    a, b = torch.randn(m, k, device=cuda).bfloat16(), torch.randn(n, k, device=cuda).bfloat16()
    want = a.double() @ b.double().t()
    out = K.gemm_bf16(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, a_mn=a_mn, b_mn=b_mn, out_dtype=dtype)
    assert rel_err(out, want) < (4e-3 if dtype == torch.bfloat16 else k / 16 * 2 ** -23)
    again = K.gemm_bf16(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, a_mn=a_mn, b_mn=b_mn, out_dtype=dtype)
    assert torch.equal(out, again)


@pytest.mark.parametrize("m,n,k", [(2568, 2056, 584), (4224, 1288, 512), (136, 18952, 520), (2048, 2560, 1024),
                                   (2568, 2056, 200), (4224, 1288, 64), (8, 18952, 72)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("out", ["bf16", "f32", "f32 +="])
def test_products_on_pairs_of_sms(cuda, m, n, k, a_mn, b_mn, out):
    """Enough 256 x 256 tiles for CTA pairs: tiles of which one CTA's rows or columns lie outside, the
    shortest contraction and ragged steps, all layouts, stores and additions. The last three are what
    pairs leave to single CTAs: short contractions, rows that fill a sliver. Bounds as above."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(18)
    a, b = torch.randn(m, k, device=cuda).bfloat16(), torch.randn(n, k, device=cuda).bfloat16()
    want = a.double() @ b.double().t()
    into = torch.ones(m, n, device=cuda) if out == "f32 +=" else None
    got = K.gemm_bf16(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, a_mn=a_mn, b_mn=b_mn, bn=256, out=into,
                      out_dtype=torch.bfloat16 if out == "bf16" else torch.float32, accumulate=into is not None)
    assert rel_err(got, want + 1 if into is not None else want) < (4e-3 if out == "bf16" else 3e-6)


@pytest.mark.parametrize("m,n,k", [(1, 128, 1024), (100, 384, 2048), (128, 256, 4096), (1, 128, 4096), (100, 384, 6144)])
def test_small_mxfp8_products_are_split(cuda, m, n, k):
    from bux_b200.ops import kernels as K

    torch.manual_seed(17)
    aq, asf, _, _ = K.quant_mxfp8(torch.randn(m, k, device=cuda).bfloat16())
    bq, bsf, _, _ = K.quant_mxfp8(torch.randn(n, k, device=cuda).bfloat16())
    wide = [ref.dequant_mxfp8(q, ref.unswizzle_scales(sf, q.shape[0], k // 32)).double() for q, sf in ((aq, asf), (bq, bsf))]
    assert rel_err(K.gemm_mxfp8(aq, asf, bq, bsf, m, n, k), wide[0] @ wide[1].t()) < 4e-3


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("norm", [True, False])
def test_norm_rope(cuda, d, norm):
    from bux_b200.ops import kernels as K

    torch.manual_seed(6)
    x = torch.randn(2, 50, 4, d, device=cuda).bfloat16().requires_grad_()
    w = torch.randn(d, device=cuda).requires_grad_() if norm else None
    pos = torch.arange(50, device=cuda).repeat(2, 1)
    cos, sin = ref.rope_tables(pos, d, 10000.0)
    want = ref.rmsnorm_rope(x, w, cos, sin, 1e-6) if norm else ref.rope(x, cos, sin)
    c2, s2 = cos.reshape(-1, d // 2).contiguous(), sin.reshape(-1, d // 2).contiguous()
    y, rstd = K.norm_rope_fwd(x.detach(), None if w is None else w.detach(), c2, s2, 1e-6)
    assert rel_err(y, want) < 1e-2
    dy = torch.randn_like(want)
    want.backward(dy)
    dx, dw = K.norm_rope_bwd(x.detach(), None if w is None else w.detach(), c2, s2, rstd, dy, 1e-6)
    assert rel_err(dx, x.grad) < 2e-2
    if norm:
        assert rel_err(dw, w.grad) < 2e-2


@pytest.mark.parametrize("kind,limit,off", [("swish", 0.0, 0.0), ("quick_gelu", 7.0, 1.0)])
def test_glu(cuda, kind, limit, off):
    from bux_b200.ops import kernels as K

    torch.manual_seed(7)
    h = (torch.randn(100, 256, device=cuda) * 4).bfloat16().requires_grad_()
    rs = torch.rand(100, device=cuda).requires_grad_()
    want = ref.glu(h[:, :128], h[:, 128:], kind, limit or None, off).float() * rs[:, None]
    got = K.glu_fwd(h.detach(), kind, rs.detach(), limit, off)
    assert rel_err(got, want) < 1e-2
    dout = torch.randn(100, 128, device=cuda).bfloat16()
    want.backward(dout.float())
    dh, drs = K.glu_bwd(h.detach(), dout, kind, rs.detach(), limit, off)
    assert rel_err(dh, h.grad) < 2e-2
    assert rel_err(drs, rs.grad) < 2e-2


def test_cross_entropy(cuda):
    from bux_b200.ops import kernels as K

    torch.manual_seed(8)
    logits = (torch.randn(64, 1000, device=cuda) * 3).bfloat16()
    tgt = torch.randint(0, 1000, (64,), device=cuda, dtype=torch.int32)
    mask = (torch.rand(64, device=cuda) > 0.2).float()
    lf = logits.float().requires_grad_()
    total, count = ref.cross_entropy(lf, tgt, mask, z_weight=1e-4)
    (total / count).backward()
    work = logits.clone()
    loss = K.ce_fwd_bwd(work, tgt, mask, 1.0 / count.item(), z_weight=1e-4)
    assert abs(loss.sum().item() - total.item()) / total.item() < 1e-3
    assert rel_err(work, lf.grad) < 2e-2


@pytest.mark.parametrize("vocab,rows", [(8, 5), (1024, 5), (1032, 5), (4096, 5), (1032, 593), (4096, 600), (4104, 600),
                                        (16384 + 8, 5), (50304, 5)])
@pytest.mark.parametrize("case", ["plain", "masked", "softcap"])
def test_cross_entropy_rows_and_masked_logits(cuda, vocab, rows, case):
    """One pass keeps the maximum and the sum: the three widths of a block, rows shorter than its step,
    remainders of the unrolled walk, logits of -inf and of the type's lowest value, a maximum that comes last.
    Bounds: the loss is an fp32 sum, the gradient is rounded to bf16 (2^-9)."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(8)
    cap = 20.0 if case == "softcap" else 0.0
    logits = (torch.randn(rows, vocab, device=cuda) * 4).bfloat16()
    targets = torch.randint(0, vocab, (rows,), device=cuda, dtype=torch.int32)
    logits[1, -1] = 60.0
    if case == "masked":
        logits[2, : vocab // 2] = float("-inf")
        logits[3, 1:] = torch.finfo(torch.bfloat16).min
        targets[2], targets[3] = vocab - 1, 0
    z = logits.double()
    z = cap * torch.tanh(z / cap) if cap else z
    logp = torch.log_softmax(z, -1)
    want = -logp.gather(1, targets.long()[:, None])[:, 0]
    grad = logp.exp().scatter_add(1, targets.long()[:, None], -torch.ones(rows, 1, device=cuda, dtype=torch.float64))
    grad = grad * (1 - (z / cap) ** 2) if cap else grad
    loss = K.ce_fwd_bwd(logits, targets, None, 1.0, softcap=cap)
    assert rel_err(loss, want) < 1e-5
    # an entry p - 1 at the target cancels where p is near 1: its error is that of p, 2^-22
    assert torch.allclose(logits.double(), grad, rtol=2 ** -8, atol=4e-6)


@pytest.mark.parametrize("n", [1, 7, 8, 4099, 1 << 20])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_scale_to_bf16(cuda, n, dtype):
    from bux_b200.ops import kernels as K

    src, g = torch.randn(n, device=cuda).to(dtype), torch.tensor(0.37, device=cuda)
    assert torch.equal(K.scale_to_bf16(src, g), (src.float() * g).bfloat16())


@pytest.mark.parametrize("mom", ["f32", "bf16", "fp8"])
def test_adamw(cuda, mom):
    from bux_b200.ops import kernels as K

    torch.manual_seed(9)
    n = 5000
    p = torch.randn(n, device=cuda)
    g = torch.randn(n, device=cuda).bfloat16()
    rp, rm, rv = p.clone(), torch.zeros(n, device=cuda), torch.zeros(n, device=cuda)
    if mom == "fp8":
        m = torch.zeros(n, dtype=torch.uint8, device=cuda)
        v = torch.zeros(n, dtype=torch.uint8, device=cuda)
        msf = torch.ones((n + 31) // 32, dtype=torch.uint8, device=cuda)
        vsf = torch.ones((n + 31) // 32, dtype=torch.uint8, device=cuda)
    else:
        dt = torch.float32 if mom == "f32" else torch.bfloat16
        m, v, msf, vsf = torch.zeros(n, dtype=dt, device=cuda), torch.zeros(n, dtype=dt, device=cuda), None, None
    shadow = torch.empty(n, dtype=torch.bfloat16, device=cuda)
    for step in (1, 2, 3):
        K.adamw(p, g, m, v, lr=1e-2, b1=0.9, b2=0.95, eps=1e-8, wd=0.1, step=step, m_sf=msf, v_sf=vsf,
                shadow=shadow)
        ref.adamw_step(rp, g, rm, rv, lr=1e-2, b1=0.9, b2=0.95, eps=1e-8, wd=0.1, step=step)
    tol = {"f32": 1e-5, "bf16": 2e-3, "fp8": 2e-2}[mom]
    assert rel_err(p, rp) < tol
    assert rel_err(shadow, rp) < 1e-2


def test_gather_combine(cuda):
    from bux_b200.ops import kernels as K

    torch.manual_seed(10)
    x = torch.randn(40, 64, device=cuda).bfloat16()
    idx = torch.randint(-1, 40, (100,), device=cuda, dtype=torch.int32)
    got = K.gather_rows(x, idx, 100)
    want = torch.where(idx[:, None] >= 0, x[idx.clamp_min(0).long()], torch.zeros_like(x[:1]))
    assert torch.equal(got, want)
    pos = torch.randint(-1, 100, (30, 4), device=cuda, dtype=torch.int32)
    w = torch.rand(30, 4, device=cuda)
    out = K.combine_rows(got, pos, w, 30)
    gathered = torch.where(pos[..., None] >= 0, got[pos.clamp_min(0).long()].float(), torch.zeros(1, device=cuda))
    assert rel_err(out, (gathered * w[..., None]).sum(1)) < 1e-2


@pytest.mark.parametrize("t,k,e,align", [(1, 1, 1, 128), (5, 3, 7, 128), (777, 4, 32, 128), (1000, 8, 128, 16), (300, 2, 1024, 1), (40000, 8, 128, 128)])
def test_sorted_picks_match_the_plain_sort(cuda, t, k, e, align):
    """Blocks, warps and steps of 32 picks, empty experts and one that takes most picks: the same
    integers as the stable sort on the CPU."""
    from bux_b200.ops import fused

    torch.manual_seed(13)
    picks = torch.randint(0, e, (t, k))
    picks[torch.rand(t, k) < 0.5] = e // 2
    w = torch.rand(t, k)
    want = fused._sort_picks(picks, e, align, w)
    got = fused._sort_picks(picks.cuda(), e, align, w.cuda())
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)


def test_a_pick_of_no_expert_is_reported(cuda):
    from bux_b200.ops import kernels as K

    picks = torch.tensor([[0, 1], [1, 4], [-1, 0]], device=cuda)
    row_index, pos, offsets, _ = K.sort_picks(picks, 4, 1, 6)
    assert pos.tolist() == [[0, 2], [3, -2], [-2, 1]] and offsets.tolist() == [0, 2, 4, 4, 4]
    assert row_index.tolist() == [0, 2, 0, 1, -1, -1]
    out = K.combine_rows(torch.ones(6, 8, device=cuda).bfloat16(), pos, None, 3)
    assert out[0].eq(2).all() and out[1:].isnan().all()
    with pytest.raises(RuntimeError, match=r"picked an expert that does not exist \(2 picks"):
        K.check_status(cuda)


@pytest.mark.parametrize("rows,f", [(1, 8), (9, 248), (5, 264), (700, 768), (1300, 56), (1185, 64), (33, 128), (3, 136),
                                    (40000, 128), (1184, 768), (1185, 776), (2, 14336)])
def test_glu_backward_rows(cuda, rows, f):
    """One, eight, 32 or 256 threads per row: rows narrower than their step, remainders of it, blocks
    that walk several rows, and the widths and row counts where the split changes. Bounds: gradients
    are rounded to bf16 (2^-9); the row scale's is an fp32 sum."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(14)
    h, dout = torch.randn(rows, 2 * f, device=cuda).bfloat16(), torch.randn(rows, f, device=cuda).bfloat16()
    rs = torch.rand(rows, device=cuda)
    hd, rd = h.double().requires_grad_(), rs.double().requires_grad_()
    g, u = hd.clamp(max=1.5)[:, :f], hd.clamp(-1.5, 1.5)[:, f:]
    (g * torch.sigmoid(g) * (u + 1) * rd[:, None]).backward(dout.double())
    dh, drs = K.glu_bwd(h, dout, "swish", rs, 1.5, 1.0)
    assert rel_err(dh, hd.grad) < 4e-3 and rel_err(drs, rd.grad) < 1e-4
    into = torch.full((rows,), float("nan"), device=cuda)
    assert torch.equal(K.glu_bwd_into(h, dout, "swish", rs, into, 1.5, 1.0), dh) and torch.equal(into, drs)


@pytest.mark.parametrize("d,h,g", [(128, 4, 2), (64, 8, 2)])
@pytest.mark.parametrize("t,window,sinks", [(256, 0, False), (300, 0, False), (384, 128, True)])
def test_attention_fwd(cuda, d, h, g, t, window, sinks):
    from bux_b200.ops import kernels as K

    torch.manual_seed(11)
    q = torch.randn(2, t, h, d, device=cuda).bfloat16()
    k = torch.randn(2, t, g, d, device=cuda).bfloat16()
    v = torch.randn(2, t, g, d, device=cuda).bfloat16()
    sk = torch.randn(h, device=cuda) if sinks else None
    want, want_lse = ref.attention(q, k, v, causal=True, window=window or None, sinks=sk)
    got, lse = K.attn_fwd(q, k, v, causal=True, window=window, sinks=sk)
    assert rel_err(got, want) < 2e-2
    assert rel_err(lse, want_lse) < 1e-3


@pytest.mark.parametrize("t,s,causal,window,scale,spread", [
    (1, 1, True, 0, None, 1.0),          # one query, one key
    (127, 127, True, 0, None, 1.0),      # a tile that ends inside the row: no TMA store
    (129, 300, True, 0, None, 1.0),      # more keys than queries; the second tile holds one row
    (256, 191, False, 0, None, 1.0),     # no mask but the end of the keys, in a half tile
    (300, 300, True, 40, None, 1.0),     # windows inside one half tile
    (640, 640, True, 0, None, 40.0),     # scores of thousands: the rows' references move mid-way
    (256, 256, True, 0, 0.0, 1.0),       # every score equal
    (256, 256, True, 0, -0.1, 30.0),     # a negative scale
    (256, 1, True, 0, None, 1.0),        # more queries than keys: the first tile of a pair sees none, the second one key
    (383, 1, True, 0, None, 1.0),        # the last such length
    (512, 256, True, 0, None, 1.0),      # a pair without keys, then one whose first tile has none
    (640, 200, True, 64, None, 1.0),     # with a window, and a last pair of one tile
    (1024, 700, False, 0, None, 1.0),    # no mask: every query sees every key
])
@pytest.mark.parametrize("d", [64, 128])
def test_attention_fwd_edges(cuda, d, t, s, causal, window, scale, spread):
    """Half tiles, partial tiles, references that move, against fp64. Bounds: P and the output are
    rounded to bf16 (2^-9 each, against the largest probability)."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(15)
    q = torch.randn(2, t, 4, d, device=cuda).bfloat16()
    k = (torch.randn(2, s, 2, d, device=cuda) * torch.linspace(0.1, spread, s, device=cuda)[None, :, None, None]).bfloat16()
    v = torch.randn(2, s, 2, d, device=cuda).bfloat16()
    sc = d ** -0.5 if scale is None else scale
    z = torch.einsum("bthd,bshd->bhts", q.double(), k.double().repeat_interleave(2, 2)) * sc
    i, j = torch.arange(t, device=cuda)[:, None] + s - t, torch.arange(s, device=cuda)[None]
    hidden = (j > i) if causal else torch.zeros(t, s, dtype=torch.bool, device=cuda)
    if window:
        hidden = hidden | (j <= i - window)
    z = z.masked_fill(hidden, float("-inf"))
    want = torch.einsum("bhts,bshd->bthd", torch.softmax(z, -1).nan_to_num(0), v.double().repeat_interleave(2, 2))
    got, lse = K.attn_fwd(q, k, v, causal=causal, window=window, scale=sc)
    assert rel_err(got, want) < 6e-3
    seen = ~hidden.all(-1)
    ref_lse = torch.logsumexp(z, -1)
    assert torch.allclose(lse.double()[..., seen], ref_lse[..., seen], rtol=1e-5, atol=1e-3)
    assert (got[:, ~seen] == 0).all()


@pytest.mark.parametrize("d,h,g", [(128, 4, 2), (64, 4, 1)])
@pytest.mark.parametrize("t,window,sinks", [(256, 0, False), (300, 0, False), (384, 128, True)])
def test_attention_bwd(cuda, d, h, g, t, window, sinks):
    from bux_b200.ops import kernels as K

    torch.manual_seed(12)
    q = torch.randn(2, t, h, d, device=cuda).bfloat16().requires_grad_()
    k = torch.randn(2, t, g, d, device=cuda).bfloat16().requires_grad_()
    v = torch.randn(2, t, g, d, device=cuda).bfloat16().requires_grad_()
    sk = torch.randn(h, device=cuda).requires_grad_() if sinks else None
    want, _ = ref.attention(q, k, v, causal=True, window=window or None, sinks=sk)
    do = torch.randn_like(q)
    want.backward(do)
    with torch.no_grad():
        o, lse = K.attn_fwd(q, k, v, causal=True, window=window, sinks=sk)
        dq, dk, dv, dsk = K.attn_bwd(q, k, v, o, do, lse, causal=True, window=window, sinks=sk)
    assert rel_err(dv, v.grad) < 3e-2
    assert rel_err(dk, k.grad) < 3e-2
    assert rel_err(dq, q.grad) < 3e-2
    if sinks:
        assert rel_err(dsk, sk.grad) < 3e-2


@pytest.mark.parametrize("scale,peak", [(float("nan"), 1.0), (0.0, float("inf")), (0.0, float("nan")), (1.0, float("inf"))])
@pytest.mark.parametrize("d", [64, 128])
def test_attention_fwd_of_scores_that_are_no_numbers(cuda, d, scale, peak):
    """A maximum that is no number is none, and no sign that a wait ran out: rows that see the NaN are
    NaN, the rows before it are what they are without it, and the status word stays clear."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(21)
    q, k, v = (torch.rand(1, 300, 2, d, device=cuda).bfloat16() for _ in range(3))
    clean, _ = K.attn_fwd(q, k, v, scale=0.0 if scale != scale else scale)
    k[:, 200] = peak
    got, _ = K.attn_fwd(q, k, v, scale=scale)
    torch.cuda.synchronize()
    K.check_status(cuda)
    assert got[:, 200:].isnan().all()
    assert got[:, :200].isnan().all() if scale != scale else torch.equal(got[:, :200], clean[:, :200])


@pytest.mark.parametrize("d,h,g,t", [(64, 12, 4, 33), (128, 3, 1, 31), (64, 8, 8, 1), (128, 9, 3, 64), (64, 40, 8, 1895),
                                     (128, 33, 3, 1900), (64, 10, 2, 300)])
def test_attention_sink_gradient_at_the_edges_of_its_tiles(cuda, d, h, g, t):
    """8 (many rows: 32) tokens x 8 heads go together in the kernel that forms delta and the sinks' gradient.
    Bound: every term of d sink is a bf16 product, off by 2^-8, and the terms partly cancel."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(19)
    q, do = (torch.randn(2, t, h, d, device=cuda).bfloat16() for _ in range(2))
    k, v = (torch.randn(2, t, g, d, device=cuda).bfloat16() for _ in range(2))
    sk = torch.randn(h, device=cuda).requires_grad_()
    q.requires_grad_()
    want, _ = ref.attention(q, k, v, causal=True, sinks=sk)
    want.backward(do)
    with torch.no_grad():
        o, lse = K.attn_fwd(q, k, v, sinks=sk)
        at = torch.empty(o.numel() + 1, device=cuda, dtype=o.dtype)[1:].view_as(o).copy_(o)  # starts between 16-byte pieces
        for out in (o, at):
            dq, _, _, dsk = K.attn_bwd(q, k, v, out, do, lse, sinks=sk)
            assert rel_err(dsk, sk.grad) < 3e-2
            assert t == 1 or rel_err(dq, q.grad) < 3e-2


def _documents(t: int, lens, device):
    """Document ids [1, t] of a row packed with documents of the given lengths."""
    assert sum(lens) == t
    ids = torch.cat([torch.full((n,), i + 1) for i, n in enumerate(lens)])
    return ids[None].to(device)


@pytest.mark.parametrize("t,h,g,lens,window,sinks", [
    (4096, 8, 1, None, 0, False),                                             # the benchmark's shape: 8 heads per group
    (4096, 8, 1, [700, 130, 1, 255, 1000, 58, 512, 384, 999, 57], 0, False),  # ten documents, odd boundaries
    (1024, 4, 2, [300, 212, 128, 384], 256, True),                            # documents + window + sinks
    (2048, 4, 2, None, 512, False),                                           # a window far from the diagonal's tile
])
def test_attention_long_rows_documents(cuda, t, h, g, lens, window, sinks):
    """Forward and backward at the lengths the benchmark runs, with packed documents
    (every query sees only its own document), against the fp32 statement."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(13)
    d = 128
    q = torch.randn(1, t, h, d, device=cuda).bfloat16().requires_grad_()
    k = torch.randn(1, t, g, d, device=cuda).bfloat16().requires_grad_()
    v = torch.randn(1, t, g, d, device=cuda).bfloat16().requires_grad_()
    sk = torch.randn(h, device=cuda).requires_grad_() if sinks else None
    seg = _documents(t, lens, cuda) if lens else None
    want, want_lse = ref.attention(q, k, v, causal=True, window=window or None, sinks=sk, segments=seg)
    do = torch.randn_like(q)
    want.backward(do)
    row_lo, key_hi = K.document_bounds(seg) if seg is not None else (None, None)
    if seg is not None:
        assert row_lo[0, 0] == 0 and key_hi[0, 0] == lens[0] - 1 and row_lo[0, -1] == t - lens[-1]
    with torch.no_grad():
        o, lse = K.attn_fwd(q, k, v, causal=True, window=window, sinks=sk, row_lo=row_lo)
        dq, dk, dv, dsk = K.attn_bwd(q, k, v, o, do, lse, causal=True, window=window, sinks=sk,
                                     row_lo=row_lo, key_hi=key_hi)
    assert rel_err(o, want) < 2e-2
    assert rel_err(lse, want_lse) < 1e-3
    assert rel_err(dv, v.grad) < 3e-2
    assert rel_err(dk, k.grad) < 3e-2
    assert rel_err(dq, q.grad) < 3e-2
    if sinks:
        assert rel_err(dsk, sk.grad) < 3e-2


def test_attention_layer_takes_the_kernels_for_packed_rows(cuda):
    """`functional.attention` with segments runs the kernels (not the quadratic statement)."""
    from bux_b200.ops import functional as OF
    from bux_b200.ops import kernels as K

    torch.manual_seed(14)
    q = torch.randn(2, 512, 4, 64, device=cuda).bfloat16().requires_grad_()
    k = torch.randn(2, 512, 2, 64, device=cuda).bfloat16().requires_grad_()
    v = torch.randn(2, 512, 2, 64, device=cuda).bfloat16().requires_grad_()
    seg = torch.cat([_documents(512, [100, 156, 256], cuda), _documents(512, [512], cuda)])
    before = K.launches
    out = OF.attention(q, k, v, causal=True, segments=seg)
    out.backward(torch.ones_like(out))
    assert K.launches - before == 3  # forward, delta, backward
    want, _ = ref.attention(q.detach(), k.detach(), v.detach(), causal=True, segments=seg)
    assert rel_err(out, want) < 2e-2


@pytest.mark.parametrize("kind,limit,up_offset", [("swish", 0.0, 0.0), ("quick_gelu", 7.0, 1.0)])
def test_quantiser_that_computes_the_gated_activation_matches_two_passes(kind, limit, up_offset):
    """glu (and its gradient) computed inside the MXFP8 quantiser gives the bytes that the
    separate activation kernel followed by the quantiser gives."""
    from bux_b200.ops import kernels as K

    torch.manual_seed(0)
    rows, f = 1000, 256  # a ragged last row tile
    h = (torch.randn(rows, 2 * f, device="cuda") * 3).bfloat16()
    da = torch.randn(rows, f, device="cuda").bfloat16()
    a = K.glu_fwd(h, kind, None, limit, up_offset)
    want = K.quant_mxfp8(a, rowwise=True, colwise=True)
    got = K.quant_mxfp8_glu(h, None, kind, rowwise=True, colwise=True, limit=limit, up_offset=up_offset)
    for w, g in zip(want, got):
        assert torch.equal(w.view(torch.uint8), g.view(torch.uint8))
    dh, _ = K.glu_bwd(h, da, kind, None, limit, up_offset)
    want = K.quant_mxfp8(dh, rowwise=True, colwise=True)
    got = K.quant_mxfp8_glu(h, da, kind, rowwise=True, colwise=True, limit=limit, up_offset=up_offset)
    for w, g in zip(want, got):
        assert torch.equal(w.view(torch.uint8), g.view(torch.uint8))
    # and against the fp32 statement of the op: the dequantised copy is close to glu(h)
    ref_a = ref.glu(h[:, :f].float(), h[:, f:].float(), kind, limit or None, up_offset)
    aq, asf, _, _ = K.quant_mxfp8_glu(h, None, kind, limit=limit, up_offset=up_offset)
    back = ref.dequant_mxfp8(aq, ref.unswizzle_scales(asf, rows, f // 32))
    assert rel_err(back, ref_a) < 0.04


@pytest.mark.parametrize("n,k", [(128, 8), (32, 4), (200, 6), (512, 32)])
def test_topk_rows_matches_torch(n, k):
    from bux_b200.ops import kernels as K

    torch.manual_seed(0)
    scores = torch.randn(1000, n, device="cuda")
    scores[3, :5] = float("-inf")          # group-limited routing masks entries out
    got = K.topk_rows(scores, k)
    want = scores.topk(k, dim=-1)
    assert torch.equal(scores.gather(-1, got), want.values)   # same values in the same order
    assert torch.equal(got, want.indices)                      # distinct random values: same indices
    ties = torch.zeros(4, n, device="cuda")
    assert torch.equal(K.topk_rows(ties, k), torch.arange(k, device="cuda").expand(4, k))


def test_nvfp4_quantiser_matches_the_recipe(cuda):
    """The CUDA quantiser (hardware E2M1 conversion) writes the bytes the PyTorch statement
    of the recipe packs."""
    from bux_b200.ops import kernels as K
    from bux_b200.ops import nvfp4 as N

    torch.manual_seed(21)
    x = (torch.randn(300, 512, device=cuda) * torch.logspace(-2, 2, 512, device=cuda)).bfloat16()
    packed, scales, ts = K.quant_nvfp4(x)
    want = N.quantize(x.float())
    wp, ws = N.pack(want)
    assert torch.allclose(ts, want.tensor_scale.reshape(1))
    assert torch.equal(scales, ws)
    mism = (packed != wp).float().mean().item()
    assert mism < 1e-3, mism   # ties at a grid midpoint may round differently after the division


@pytest.mark.parametrize("taps,bias,packed", [(4, False, False), (3, True, True), (8, True, False), (1, False, True)])
def test_causal_conv_matches_the_shifted_sums(cuda, taps, bias, packed):
    """The causal depthwise convolution kernels (forward, dx, dw, db) against the PyTorch sum of
    shifted rows in fp32, with and without document starts inside the rows."""
    from bux_b200 import ops

    torch.manual_seed(0)
    b, t, c = 3, 200, 264
    x = torch.randn(b, t, c, device=cuda).bfloat16().requires_grad_()
    w = (torch.randn(c, taps, device=cuda) * 0.5).bfloat16().requires_grad_()
    bb = torch.randn(c, device=cuda).bfloat16().requires_grad_() if bias else None
    pos = None
    if packed:
        pos = torch.arange(t, device=cuda).repeat(b, 1)
        pos[0, 70:] -= 70
        pos[1, 5:] -= 5
        pos[1, 131:] -= 126
    dy = torch.randn(b, t, c, device=cuda).bfloat16()
    y = ops.causal_conv(x, w, bb, pos)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    br = bb.detach().float().requires_grad_() if bias else None
    yr = xr * wr[:, 0]
    for j in range(1, taps):
        shifted = torch.nn.functional.pad(xr[:, : t - j], (0, 0, j, 0))
        if pos is not None:
            shifted = shifted * (pos >= j).unsqueeze(-1).float()
        yr = yr + shifted * wr[:, j]
    if bias:
        yr = yr + br
    yr.backward(dy.float())
    assert rel_err(y, yr) < 1e-2
    assert rel_err(x.grad, xr.grad) < 1e-2
    assert rel_err(w.grad, wr.grad) < 1e-2
    if bias:
        assert rel_err(bb.grad, br.grad) < 1e-2
