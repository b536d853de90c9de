"""Differentiable CUDA ops (kernels behind autograd) against plain PyTorch in fp32."""
import pytest
import torch

from bux_b200 import ops
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


@pytest.mark.parametrize("fmt,tol", [("bf16", 2e-2), ("mxfp8", 8e-2)])
def test_linear(cuda, fmt, tol):
    torch.manual_seed(0)
    x = torch.randn(4, 96, 256, device=cuda).bfloat16().requires_grad_()
    w = (torch.randn(384, 256, device=cuda) * 0.05).bfloat16().requires_grad_()
    y = ops.linear(x, w, fmt=fmt)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = xr @ wr.t()
    yr.backward(dy.float())
    assert rel_err(y, yr) < tol
    assert rel_err(x.grad, xr.grad) < tol
    assert rel_err(w.grad, wr.grad) < tol


@pytest.mark.parametrize("passes", [("fprop",), ("dgrad", "wgrad"), ("fprop", "wgrad"), ("dgrad",)])
def test_linear_mxfp8_in_some_passes_only(cuda, passes):
    """The GEMMs that `passes` lists multiply in MXFP8, the others exactly as the bf16 linear does."""
    torch.manual_seed(0)
    x = torch.randn(4, 96, 256, device=cuda).bfloat16()
    w = (torch.randn(384, 256, device=cuda) * 0.05).bfloat16()
    dy = torch.randn(4, 96, 384, device=cuda).bfloat16()

    def run(fmt, only):
        xi, wi = x.clone().requires_grad_(), w.clone().requires_grad_()
        y = ops.linear(xi, wi, fmt=fmt, passes=only)
        y.backward(dy)
        return {"fprop": y.detach(), "dgrad": xi.grad, "wgrad": wi.grad}

    plain = run("bf16", ("fprop", "dgrad", "wgrad"))
    low = run("mxfp8", ("fprop", "dgrad", "wgrad"))
    got = run("mxfp8", passes)
    for name in ("fprop", "dgrad", "wgrad"):
        want = low if name in passes else plain
        assert torch.equal(got[name], want[name]), name
        assert rel_err(got[name], plain[name]) < 8e-2


def test_cross_entropy_head(cuda):
    torch.manual_seed(1)
    x = torch.randn(300, 128, device=cuda).bfloat16().requires_grad_()
    w = (torch.randn(1000, 128, device=cuda) * 0.1).bfloat16().requires_grad_()
    tgt = torch.randint(0, 1000, (300,), device=cuda)
    mask = (torch.rand(300, device=cuda) > 0.1).float()
    total, count = ops.cross_entropy_head(x, w, tgt, mask, z_weight=1e-4)
    (total / count).backward()
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    tr, cr = ref.cross_entropy(xr @ wr.t(), tgt, mask, 1e-4)
    (tr / cr).backward()
    assert abs(total.item() - tr.item()) / tr.item() < 5e-3
    assert rel_err(x.grad, xr.grad) < 3e-2
    assert rel_err(w.grad, wr.grad) < 3e-2


@pytest.mark.parametrize("fmt,tol", [("bf16", 3e-2), ("mxfp8", 1e-1)])
def test_moe_experts(cuda, fmt, tol):
    torch.manual_seed(2)
    t, d, f, e, k = 512, 256, 128, 8, 2
    x = torch.randn(t, d, device=cuda).bfloat16().requires_grad_()
    wgu = (torch.randn(e, 2 * f, d, device=cuda) * 0.06).bfloat16().requires_grad_()
    wd = (torch.randn(e, d, f, device=cuda) * 0.06).bfloat16().requires_grad_()
    logits = torch.randn(t, e, device=cuda)
    logits[:, 3] = -100.0  # an expert nobody picks
    wts, idx, _ = ref.router_topk(logits, k)
    wts = wts.requires_grad_()
    out = ops.moe_experts(x, wgu, wd, wts, idx, fmt=fmt)
    dout = torch.randn_like(out)
    out.backward(dout)
    xr = x.detach().float().requires_grad_()
    gr = wgu.detach().float().requires_grad_()
    dr = wd.detach().float().requires_grad_()
    wr = wts.detach().clone().requires_grad_()
    want = ops.moe_reference(xr, gr, dr, wr, idx)
    want.backward(dout.float())
    assert rel_err(out, want) < tol
    assert rel_err(x.grad, xr.grad) < tol
    assert rel_err(wgu.grad, gr.grad) < tol
    assert rel_err(wd.grad, dr.grad) < tol
    assert rel_err(wts.grad, wr.grad) < tol


def test_norm_glu_attention_autograd(cuda):
    torch.manual_seed(3)
    x = torch.randn(2, 64, 256, device=cuda).bfloat16().requires_grad_()
    w = torch.ones(256, device=cuda).requires_grad_()
    y = ops.rmsnorm(x, w, 1e-6)
    h = ops.glu(y.view(2, 64, 256))
    h.sum().backward()
    assert torch.isfinite(x.grad).all() and torch.isfinite(w.grad).all()
    q = torch.randn(1, 256, 4, 64, device=cuda).bfloat16().requires_grad_()
    k = torch.randn(1, 256, 2, 64, device=cuda).bfloat16().requires_grad_()
    v = torch.randn(1, 256, 2, 64, device=cuda).bfloat16().requires_grad_()
    o = ops.attention(q, k, v)
    o.float().square().sum().backward()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    orf, _ = ref.attention(qr, kr, vr)
    orf.square().sum().backward()
    assert rel_err(q.grad, qr.grad) < 4e-2 and rel_err(k.grad, kr.grad) < 4e-2


@pytest.mark.gpu
def test_linear_f32_matches_fp32_matmul():
    from bux_b200.ops import functional as F_

    torch.manual_seed(0)
    x = torch.randn(512, 256, device="cuda").bfloat16().requires_grad_(True)
    for dtype in (torch.float32, torch.bfloat16):
        w = (torch.randn(128, 256, device="cuda") * 0.05).to(dtype).requires_grad_(True)
        y = F_.linear_f32(x, w)
        want = x.float() @ w.float().t()
        assert y.dtype == torch.float32
        assert torch.allclose(y, want, atol=2e-4 if dtype == torch.float32 else 1e-5, rtol=1e-4)
        g = torch.randn_like(y)
        dx, dw = torch.autograd.grad(y, (x, w), g)
        gb = g.bfloat16().float()
        assert torch.allclose(dx.float(), (gb @ w.float()), atol=2e-2, rtol=2e-2)
        assert torch.allclose(dw.float(), gb.t() @ x.float(), atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
def test_remat_that_keeps_attention_outputs_matches_plain_remat():
    from bux_b200.lang import compile_runs
    from bux_b200.ops import kernels as K
    from bux_b200.train.trainer import Trainer

    src = """
d_model=256
vocab_size=512
n = rmsnorm
block = [n gqa(num_heads=4, num_kv_heads=2, head_dim=64, rope=rope())] [n gated_mlp(intermediate_size=512, activation=swish)]
model = embed block^2 n head
data = synthetic
optimizer = adamw(lr=1e-3)
seq_len = 256
batch = 4
steps = 4
precision = precision(compute=bfloat16)
"""
    run = compile_runs(src, filename="k.bux")[0]
    out = []
    for keep, offload in ((False, False), (True, False), (1, True)):
        tr = Trainer(run, device="cuda")
        tr.model.set_remat(True, offload=offload, keep_attention=keep)
        feed = iter(tr.batches())
        before = K.launches
        losses = [tr.train_step(next(feed))["loss"].item() for _ in range(2)]
        out.append((losses, K.launches - before, {n: p.detach().float().clone() for n, p in tr.model.named_parameters()}))
    (l0, n0, s0), (l1, n1, s1), (l2, n2, s2) = out
    assert l0 == pytest.approx(l1, abs=1e-3) and l0 == pytest.approx(l2, abs=1e-3)
    assert n1 == n0 - 2 * 2              # one attention forward less per block and step
    assert n2 == n0 - 2 * 1              # a count keeps the last so many blocks only (inputs on the host)
    assert all(torch.allclose(s0[k], s2[k], atol=2e-3, rtol=2e-2) for k in s0)
    # dQ is summed by fp32 reductions whose order varies from run to run: close, not bit-equal
    assert all(torch.allclose(s0[k], s1[k], atol=2e-3, rtol=2e-2) for k in s0)


@pytest.mark.parametrize("shape", [(512, 2048), (2048, 768), (3, 256, 512)])
def test_newton_schulz_on_the_tcgen05_gemm_matches_fp32(shape):
    """Muon's orthogonalisation through the framework's GEMM against the same iteration in
    fp32 PyTorch; the result is close to an orthogonal factor (singular values near 1)."""
    from bux_b200.ops import kernels as K
    from bux_b200.train import optim

    torch.manual_seed(0)
    g = torch.randn(*shape, device="cuda")
    before = K.launches
    got = optim.newton_schulz(g, steps=5, dtype=torch.bfloat16).float()
    want = optim.newton_schulz(g, steps=5, dtype=torch.float32)
    assert got.shape == want.shape
    assert (got - want).norm() / want.norm() < 0.06
    s = torch.linalg.svdvals(got.reshape(-1, *shape[-2:])[0])
    assert 0.5 < s.min() and s.max() < 1.3
    assert K.launches >= before + 15  # three GEMMs per step, per matrix


def test_interleaved_microbatches_match_a_plain_accumulation_on_two_streams(cuda):
    """``methods(interleave=true)`` on the GPU: every microbatch's forward is issued on one of two
    streams by its parity, beside the backward of the one before on the other. A mixture of
    experts, a value residual that crosses blocks and ``remat=full``: the parameters after two
    steps are those of the microbatches run one after another."""
    from bux_b200.lang import compile_runs
    from bux_b200.train.trainer import Trainer

    src = """
d_model=256
vocab_size=512
n = rmsnorm
a = gqa(num_heads=4, num_kv_heads=2, head_dim=64, rope=rope(), value_residual=learned)
e = moe(num_experts=8, top_k=2, expert=gated_mlp(intermediate_size=128, activation=swish))
first = [n a(v=@v)] [n e]
rest = [n a(v=$v)] [n e]
model = embed first rest^3 n head
data = synthetic
optimizer = adamw(lr=1e-3, eps=1.0)
seq_len = 256
batch = 8
steps = 4
precision = precision(compute=bfloat16)
methods = methods(microbatches=4, remat=full{more})
"""
    out = {}
    for name, more in (("plain", ""), ("interleaved", ", interleave=true")):
        tr = Trainer(compile_runs(src.format(more=more), filename="g.bux")[0], device=cuda)
        feed = iter(tr.batches())
        losses = [tr.train_step(next(feed))["loss"].item() for _ in range(2)]
        torch.cuda.synchronize()
        out[name] = (losses, {n: p.detach().float().cpu() for n, p in tr.model.named_parameters()}, tr._interleave)
    assert out["interleaved"][2] and out["interleaved"][2].ticks == 2 * 3 * 6      # two steps, three pairs, six pieces
    assert out["plain"][0] == pytest.approx(out["interleaved"][0], abs=1e-3)
    for name, p in out["plain"][1].items():
        assert rel_err(out["interleaved"][1][name], p) < 1e-3, name


def _layer_calls(cuda):
    """One call of each layer op on inputs that are odd on purpose: slices, transposes, other dtypes."""
    from bux_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(3)

    def rand(*shape, dtype=torch.bfloat16):
        return torch.randn(*shape, generator=g, device=cuda).to(dtype)

    qkv = rand(2, 40, 3 * 4 * 64)
    cos, sin = torch.rand(2, 40, 32, device=cuda).double(), torch.rand(2, 40, 32, device=cuda)
    seg = torch.tensor([[0] * 15 + [1] * 25, [0] * 40], device=cuda)
    return {
        "rmsnorm": ([rand(520, 6).t(), rand(520)], lambda x, w: ops.rmsnorm(x, w, 1e-5)),
        "rmsnorm plain": ([rand(2, 3, 64)], lambda x: ops.rmsnorm(x, None)),
        "rmsnorm zero-centred": ([rand(2, 3, 64), rand(64, dtype=torch.float32)], lambda x, w: ops.rmsnorm(x, w, 1e-6, True)),
        "norm + rope of a slice": ([qkv, rand(64)], lambda x, w: ops.rmsnorm_rope(x[..., 256:512].unflatten(-1, (4, 64)), w, cos, sin)),
        "rope": ([rand(2, 4, 40, 64)], lambda x: ops.rope(x.transpose(1, 2), cos, sin)),
        "glu": ([rand(2, 9, 48)], lambda h: ops.glu(h, "gelu_tanh", None, 7.0, 1.0)),
        "glu scaled": ([rand(9, 48), rand(9)], lambda h, s: ops.glu(h, "swish", s)),
        "linear": ([rand(2, 24, 9), rand(40, 24)], lambda x, w: ops.linear(x.transpose(1, 2), w)),
        "linear with bias": ([rand(3, 24), rand(40, 24), rand(40)], ops.linear),
        "attention": ([rand(2, 40, 4, 64), rand(2, 40, 2, 64), rand(2, 2, 40, 64)],
                      lambda q, k, v: ops.attention(q, k, v.transpose(1, 2), window=16)),
        "attention packed": ([rand(2, 40, 4, 64), rand(2, 40, 2, 64), rand(2, 40, 2, 64), rand(4)],
                             lambda q, k, v, s: ops.attention(q, k, v, sinks=s, segments=seg, scale=0.2)),
    }


@pytest.mark.parametrize("frozen", [None, 0, 1])
def test_native_autograd_functions_match_the_python_ones(cuda, frozen, monkeypatch):
    """The same kernels, casts and saved tensors: outputs, gradients, their dtypes and strides, launch
    counts; with any one input frozen, under saved-tensor hooks, without gradients. Bits, but for what
    the kernels themselves sum with atomics (dq, the gains of the rotation, the sinks)."""
    from bux_b200.ops import functional as F
    from bux_b200.ops import kernels as K

    def packed(x):
        return x.cpu()

    def run(name, inputs, fn, hooks):
        xs = [x.detach().clone().requires_grad_(i != frozen) for i, x in enumerate(inputs)]
        before = K.launches
        with torch.autograd.graph.saved_tensors_hooks(packed, lambda x: x.to(cuda)) if hooks else torch.enable_grad():
            y = fn(*xs)
        want = [x for x in xs if x.requires_grad]
        grads = torch.autograd.grad(y, want, torch.ones_like(y) * 0.1, allow_unused=True) if want else []
        with torch.no_grad():
            again = fn(*xs)
        assert torch.equal(again, y) and not again.requires_grad
        return [y, *grads], K.launches - before

    for name, (inputs, fn) in _layer_calls(cuda).items():
        for hooks in (False, True):
            got, n = run(name, inputs, fn, hooks)
            with monkeypatch.context() as m:
                m.setattr(F, "_native", lambda op: None)
                want, n_want = run(name, inputs, fn, hooks)
            assert n == n_want, name
            for a, b in zip(got, want):
                assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride(), name
                assert torch.equal(a, b) or torch.allclose(a.float(), b.float(), rtol=2 ** -7, atol=1e-5), name


def test_native_autograd_functions_refuse_and_recompute(cuda):
    """Forward-mode differentiation stays refused; a checkpointed call recomputes."""
    from torch.utils.checkpoint import checkpoint

    from bux_b200 import ops

    x = torch.randn(4, 64, device=cuda).bfloat16().requires_grad_()
    w = torch.randn(64, device=cuda).requires_grad_()
    plain = torch.autograd.grad(ops.rmsnorm(x, w).sum(), [x, w])
    for reentrant in (True, False):
        y = checkpoint(lambda a, b: ops.rmsnorm(a, b), x, w, use_reentrant=reentrant)
        if reentrant:
            x.grad = w.grad = None
            y.sum().backward()
            again = [x.grad, w.grad]
        else:
            again = torch.autograd.grad(y.sum(), [x, w])
        assert all(torch.equal(a, b) for a, b in zip(plain, again))
    with pytest.raises((NotImplementedError, RuntimeError)):
        with torch.autograd.forward_ad.dual_level():
            ops.rmsnorm(torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x)), w)


@pytest.mark.parametrize("layout", ["tokens of one longer row", "one head, heads first", "between 16-byte boundaries", "gradient between them"])
@pytest.mark.parametrize("weighted", [True, False])
def test_norm_rope_of_layouts_that_only_look_dense(cuda, layout, weighted, monkeypatch):
    """Tensors that PyTorch calls contiguous and the kernel cannot walk in place, through both forms of
    the function, with gradients. Bounds: outputs are rounded to bf16 (2^-9), with one rotation more."""
    from bux_b200.ops import functional as F

    g = torch.Generator(device=cuda).manual_seed(4)
    t, h, d = 60, 1 if layout.startswith("one head") else 4, 64
    base = torch.randn(2 * 100 * 4 * d, generator=g, device=cuda).bfloat16()
    if layout == "tokens of one longer row":
        x = base[: 100 * h * d].view(1, 100, h, d)[:, :t]
    elif h == 1:
        x = base[: 2 * t * d].view(2, 1, t, d).transpose(1, 2)
    else:
        x = base[layout.startswith("between"):][: t * h * d].view(1, t, h, d)
    w = torch.randn(d, generator=g, device=cuda)
    cos, sin = ref.rope_tables(torch.arange(t, device=cuda)[None].expand(x.shape[0], t), d, 10000.0)
    dy = torch.randn(x.numel() + 1, generator=g, device=cuda).bfloat16()[layout.startswith("gradient"):][: x.numel()].view(x.shape)
    xr, wr = x.float().requires_grad_(), w.clone().requires_grad_()
    want = ref.rmsnorm_rope(xr, wr, cos, sin, 1e-6) if weighted else ref.rope(xr, cos, sin)
    want.backward(dy.float())
    for python in (False, True):
        with monkeypatch.context() as m:
            if python:
                m.setattr(F, "_native", lambda op: None)
            xg, wg = x.detach().requires_grad_(), w.clone().requires_grad_()
            y = ops.rmsnorm_rope(xg, wg if weighted else None, cos, sin, 1e-6)
            grads = torch.autograd.grad(y, [xg, wg] if weighted else [xg], dy)
        assert rel_err(y, want) < 4e-3 and rel_err(grads[0], xr.grad) < 4e-3
        assert not weighted or rel_err(grads[1], wr.grad) < 1e-5


def test_norm_rope_refuses_what_it_cannot_walk(cuda):
    """The wrapper's own checks, below the functions that copy such tensors."""
    from bux_b200.ops import kernels as K

    x = torch.zeros(1, 8, 2, 64, device=cuda).bfloat16()
    y, c = torch.empty_like(x), torch.zeros(8, 32, device=cuda)

    def call(x=x, y=y, cos=c, sin=c, step=128, tokens=8, dy=None, bwd=False):
        K.ops().norm_rope(bwd, x, None, cos, sin, y, None, dy, None, tokens, 2, 64, step, 128, 1e-6)

    call()
    bad = torch.zeros(8 * 2 * 64 + 1, device=cuda).bfloat16()[1:].view(1, 8, 2, 64)
    for kw in ({"x": bad}, {"y": bad}, {"step": -1}, {"step": 64}, {"step": 256}, {"tokens": 9}, {"cos": c[:7]}, {"sin": c[:, :16]},
               {"bwd": True}, {"bwd": True, "dy": bad}, {"x": x.float()}):
        with pytest.raises(RuntimeError, match="norm_rope"):
            call(**kw)


@pytest.mark.parametrize("fmt", ["bf16", "mxfp8"])
@pytest.mark.parametrize("bad", [-1, 4, 1 << 40])
def test_a_pick_of_no_expert_spoils_its_own_token_alone(cuda, fmt, bad):
    """Its row of the output and of dx, and its weight's gradient, are NaN; every other token is what
    it is with valid picks; the status word says what happened."""
    from bux_b200.ops import kernels as K

    g = torch.Generator(device=cuda).manual_seed(6)
    x, dy = (torch.randn(40, 128, generator=g, device=cuda).bfloat16() for _ in range(2))
    w_gu = (torch.randn(4, 256, 128, generator=g, device=cuda) * 0.1).bfloat16()
    w_down = (torch.randn(4, 128, 128, generator=g, device=cuda) * 0.1).bfloat16()
    wts, good = torch.rand(40, 2, generator=g, device=cuda), torch.randint(0, 4, (40, 2), generator=g, device=cuda)

    def run(picks):
        xs = [t.detach().clone().requires_grad_() for t in (x, wts)]
        y = ops.moe_experts(xs[0], w_gu, w_down, xs[1], picks, fmt=fmt)
        return [y.detach(), *torch.autograd.grad(y, xs, dy)]

    want = run(good)
    picks = good.clone()
    picks[7, 1] = bad
    got = run(picks)
    with pytest.raises(RuntimeError, match=r"does not exist \(1 picks"):
        K.check_status(cuda)
    rest = torch.arange(40, device=cuda) != 7
    for a, b in zip(got, want):
        assert torch.equal(a[rest], b[rest])
    assert got[0][7].isnan().all() and got[1][7].isnan().all()
    assert got[2][7, 1].isnan() and got[2][7, 0] == want[2][7, 0]


def test_rows_without_elements_are_refused(cuda):
    """An exception, where a division by the width or the head count would end the process."""
    empty = torch.empty(4, 0, device=cuda, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="rmsnorm"):
        ops.rmsnorm(empty, None)
    with pytest.raises(RuntimeError, match="glu"):
        ops.glu(empty)
    table = torch.zeros(1, 3, 32, device=cuda)
    with pytest.raises(RuntimeError, match="norm_rope"):
        ops.rope(torch.empty(1, 3, 0, 64, device=cuda, dtype=torch.bfloat16), table, table)


def test_cross_entropy_head_takes_a_batch_of_gradients(cuda):
    """Several incoming gradients at once, as `jacobian(vectorize=True)` sends them: each one's result."""
    g = torch.Generator(device=cuda).manual_seed(7)
    x = torch.randn(9, 64, generator=g, device=cuda).bfloat16().requires_grad_()
    w = torch.randn(128, 64, generator=g, device=cuda).bfloat16().requires_grad_()
    tgt = torch.randint(0, 128, (9,), generator=g, device=cuda)
    scales = torch.tensor([1.0, 0.37, -2.0], device=cuda)
    many = torch.autograd.grad(ops.cross_entropy_head(x, w, tgt)[0], [x, w], scales, is_grads_batched=True)
    for i, s in enumerate(scales):
        one = torch.autograd.grad(ops.cross_entropy_head(x, w, tgt)[0], [x, w], s)
        for a, b in zip(many, one):
            assert a[i].dtype == b.dtype and torch.equal(a[i], b)


@pytest.mark.parametrize("constant", [True, False])
def test_gradients_of_native_functions_have_no_gradients(cuda, constant):
    """The backward kernels are not differentiable: under create_graph the gradients do not pretend to
    be, whether the incoming gradient depends on the inputs or not, and asking for theirs raises."""
    for name, (inputs, fn) in _layer_calls(cuda).items():
        xs = [x.detach().clone().requires_grad_() for x in inputs]
        y = fn(*xs)
        dx, = torch.autograd.grad(y, xs[:1], torch.ones_like(y) if constant else 2 * y, create_graph=True)
        assert not dx.requires_grad, name
        with pytest.raises(RuntimeError, match="does not require grad"):
            torch.autograd.grad(dx.float().sum(), xs[:1])
