"""Model kernels (norms, rotary, ReLU^2, embedding, fused lm_head + cross-entropy, Linear)
against fp32 PyTorch references, forward and backward."""
import pytest
import torch
import torch.nn.functional as F

from dion_b200.ops import nn as N


def _close(x, ref, tol):
    """max |x - ref| relative to the scale of ref (bf16 intermediates make per-element
    relative checks meaningless near zero)."""
    err = ((x.float() - ref.float()).abs().max() / ref.float().abs().max().clamp_min(1e-20)).item()
    assert err < tol, f"scaled max error {err:.3e} >= {tol}"


def _ref_rms(x, eps=N.RMS_EPS):
    xf = x.float()
    return xf * torch.rsqrt(xf.square().mean(-1, keepdim=True) + eps)


def test_cpu_paths_are_differentiable():
    x = torch.randn(2, 5, 16, requires_grad=True)
    w = torch.randn(24, 16, requires_grad=True)
    y = N.linear(N.rms_norm(x), w, act="relu2")
    y.sum().backward()
    assert x.grad is not None and w.grad is not None
    cos, sin = N.rotary_tables(5, 8, "cpu")
    q = torch.randn(2, 5, 2, 8)
    qo, ko = N.rope_qknorm(q, q.clone(), cos, sin)
    assert qo.shape == q.shape
    torch.testing.assert_close(qo.square().mean(-1), torch.ones(2, 5, 2), rtol=1e-3, atol=1e-3)
    t = torch.randint(0, 24, (2, 5))
    loss = N.linear_cross_entropy(torch.randn(2, 5, 16), w, t)
    assert loss.ndim == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [768, 64, 4096])
def test_rmsnorm_kernel(dim):
    x = torch.randn(37, 5, dim, device="cuda").bfloat16().requires_grad_()
    y = N.rms_norm(x)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    yr = _ref_rms(xr)
    yr.backward(g.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=3e-2, atol=3e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("head_dim", [64, 128])
def test_rope_qknorm_kernel(head_dim):
    B, T, H = 2, 48, 3
    cos, sin = N.rotary_tables(T, head_dim, "cuda")
    q = torch.randn(B, T, H, head_dim, device="cuda").bfloat16().requires_grad_()
    k = torch.randn(B, T, H, head_dim, device="cuda").bfloat16().requires_grad_()
    qo, ko = N.rope_qknorm(q, k, cos, sin)
    gq, gk = torch.randn_like(qo), torch.randn_like(ko)
    (qo * gq).sum().backward(retain_graph=True)
    (ko * gk).sum().backward()
    qr = q.detach().float().requires_grad_()
    kr = k.detach().float().requires_grad_()
    qro, kro = N._rope_qknorm_torch(qr, kr, cos, sin, N.RMS_EPS)
    ((qro * gq.float()).sum() + (kro * gk.float()).sum()).backward()
    torch.testing.assert_close(qo.float(), qro, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(ko.float(), kro, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(q.grad.float(), qr.grad, rtol=5e-2, atol=5e-2)
    torch.testing.assert_close(k.grad.float(), kr.grad, rtol=5e-2, atol=5e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("head_dim", [64, 128])
def test_rope_qknorm_kernel_on_views_that_are_only_8_byte_aligned(head_dim):
    """Inputs that start 8 bytes into an allocation take the kernels with 8-byte accesses; same results."""
    B, T, H = 2, 40, 3
    n = B * T * H * head_dim
    cos, sin = N.rotary_tables(T, head_dim, "cuda")
    qbuf = torch.randn(n + 4, device="cuda").bfloat16()
    kbuf = torch.randn(n + 4, device="cuda").bfloat16()
    q = qbuf[4:].view(B, T, H, head_dim).requires_grad_()
    k = kbuf[4:].view(B, T, H, head_dim).requires_grad_()
    assert q.data_ptr() % 16 == 8 and q.is_contiguous()
    qo, ko = N.rope_qknorm(q, k, cos, sin)
    gq, gk = torch.randn_like(qo), torch.randn_like(ko)
    ((qo * gq).sum() + (ko * gk).sum()).backward()
    qr = q.detach().float().requires_grad_()
    kr = k.detach().float().requires_grad_()
    qro, kro = N._rope_qknorm_torch(qr, kr, cos, sin, N.RMS_EPS)
    ((qro * gq.float()).sum() + (kro * gk.float()).sum()).backward()
    torch.testing.assert_close(qo.float(), qro, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(ko.float(), kro, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(q.grad.float(), qr.grad, rtol=5e-2, atol=5e-2)
    torch.testing.assert_close(k.grad.float(), kr.grad, rtol=5e-2, atol=5e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("head_dim", [64, 128])
def test_rope_alone_kernel(head_dim):
    """Rotary embedding of one tensor without the norm (the Llama-shaped model's use)."""
    B, T, H = 2, 33, 5
    cos, sin = N.rotary_tables(T, head_dim, "cuda")
    x = torch.randn(B, T, H, head_dim, device="cuda").bfloat16().requires_grad_()
    y = N.rope(x, cos, sin)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    d = head_dim // 2
    c, s_ = cos[None, :T, None, :].float(), sin[None, :T, None, :].float()
    yr = torch.cat([xr[..., :d] * c + xr[..., d:] * s_, xr[..., d:] * c - xr[..., :d] * s_], dim=-1)
    yr.backward(g.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=2e-2, atol=2e-2)


@pytest.mark.gpu
def test_relu2_kernel():
    x = torch.randn(64, 3072, device="cuda").bfloat16().requires_grad_()
    h = N.relu2(x)
    g = torch.randn_like(h)
    h.backward(g)
    xr = x.detach().float().requires_grad_()
    hr = torch.relu(xr).square()
    hr.backward(g.float())
    torch.testing.assert_close(h.float(), hr, rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=1e-2, atol=1e-2)


@pytest.mark.gpu
def test_embedding_kernel():
    table = torch.randn(1000, 768, device="cuda", requires_grad=True)
    idx = torch.randint(0, 1000, (4, 33), device="cuda")
    idx[0, :5] = 7  # repeated ids accumulate
    out = N.embedding(idx, table)
    g = torch.randn_like(out)
    out.backward(g)
    assert torch.equal(out, table.detach()[idx].bfloat16())
    ref = torch.zeros_like(table)
    ref.index_put_((idx.reshape(-1),), g.float().view(-1, 768), accumulate=True)
    torch.testing.assert_close(table.grad, ref, rtol=1e-4, atol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("residual", [False, True])
def test_linear_fn(residual):
    T, K, Nn = 300, 256, 520
    x = torch.randn(T, K, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(Nn, K, device="cuda") / K ** 0.5).requires_grad_()
    r = torch.randn(T, Nn, device="cuda").bfloat16().requires_grad_() if residual else None
    y = N.linear(x, w, residual=r)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().bfloat16().float().requires_grad_()
    yr = xr @ wr.t() + (r.detach().float() if residual else 0)
    yr.backward(g.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(w.grad, wr.grad, rtol=2e-2, atol=2e-2)
    assert w.grad.dtype == torch.float32
    if residual:
        assert torch.equal(r.grad, g)


@pytest.mark.gpu
def test_linear_relu2_and_split_k_weight_grad():
    T, K, Nn = 4096, 128, 256
    x = torch.randn(T, K, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(Nn, K, device="cuda") / K ** 0.5).requires_grad_()
    y = N.linear(x, w, act="relu2")
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().bfloat16().float().requires_grad_()
    pre = (xr @ wr.t()).bfloat16().float()
    # reference through the same bf16 rounding of the pre-activation
    yr = torch.relu(xr @ wr.t()).square()
    yr.backward(g.float())
    _close(y, torch.relu(pre).square(), 1e-2)
    _close(x.grad, xr.grad, 2e-2)
    _close(w.grad, wr.grad, 2e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [50304, 1024])
def test_linear_cross_entropy(vocab):
    T, K = 700, 256
    x = torch.randn(T, K, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(vocab, K, device="cuda") / K ** 0.5).requires_grad_()
    t = torch.randint(0, vocab, (T,), device="cuda")
    t[:9] = -1
    loss = N.linear_cross_entropy(x, w, t, ignore_index=-1, chunk_tokens=256)
    (loss * 0.5).backward()
    xr = x.detach().float().requires_grad_()
    wr = w.detach().bfloat16().float().requires_grad_()
    logits = (xr @ wr.t())
    lr = F.cross_entropy(logits, t, ignore_index=-1)
    (lr * 0.5).backward()
    torch.testing.assert_close(loss, lr, rtol=5e-3, atol=5e-3)
    _close(x.grad, xr.grad, 2e-2)
    _close(w.grad, wr.grad, 2e-2)
    with torch.no_grad():
        l2 = N.linear_cross_entropy(x, w, t, ignore_index=-1)
    torch.testing.assert_close(l2, lr, rtol=5e-3, atol=5e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [8, 2056, 24576, 24584, 32760, 65528, 65536, 100008, 131072])
@pytest.mark.parametrize("write_grad", [True, False])
def test_cross_entropy_rows(vocab, write_grad):
    """Every number of threads per row, at lengths that end in whole groups of vectors and in between."""
    torch.manual_seed(vocab)
    rows, pitch = 37, vocab + 8
    x = torch.full((rows, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
    x[:, :vocab] = 3 * torch.randn(rows, vocab, device="cuda")
    x[3, : vocab // 2] = -float("inf")              # a masked vocabulary
    x[4, : vocab // 2] = torch.finfo(torch.bfloat16).min
    x[5, :vocab] = 1e4
    t = torch.randint(vocab // 2, vocab, (rows,), device="cuda")
    t[0], t[1], t[2] = vocab - 1, vocab // 2, -1
    ref = x[:, :vocab].double()
    logits, loss = x.clone(), torch.empty(rows, device="cuda")
    scale = torch.tensor([0.25], device="cuda")
    assert N.runtime.use_cuda_kernels(x)
    torch.ops.dion_b200.cross_entropy_fwd_bwd(logits[:, :vocab], t, loss, scale, 3.0, -1, write_grad)
    want = F.cross_entropy(ref, t, ignore_index=-1, reduction="none")
    # maximum minus target rounds once (2^-24 of it), the sum of a thread has up to 128 terms, each exponential 2 ulp
    torch.testing.assert_close(loss.double(), want, rtol=2.0 ** -22, atol=128 * 2.0 ** -24 + 1e-5)
    if write_grad:
        p = 0.75 * (torch.softmax(ref, 1) - F.one_hot(t.clamp_min(0), vocab))
        p[t == -1] = 0
        # bf16: half of 2^-8; the target's p - 1 can cancel, to within the rounding of fp32
        torch.testing.assert_close(logits[:, :vocab].double(), p, rtol=2.0 ** -8, atol=1e-6 * float(p.abs().amax()))
    else:
        assert torch.equal(logits, x)
    assert bool((logits[:, vocab:] == 7.0).all())
    bad = x.clone()
    bad[0, vocab // 3], bad[1, 0], bad[6, vocab - 1] = float("nan"), float("inf"), float("nan")
    torch.ops.dion_b200.cross_entropy_fwd_bwd(bad[:, :vocab], t, loss, scale, 3.0, -1, write_grad)
    assert torch.equal(loss.isnan(), torch.isin(torch.arange(rows, device="cuda"), torch.tensor([0, 1, 6], device="cuda")))


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,chunk", [(256, 8192), (300, 128)])
def test_linear_cross_entropy_backward_twice_and_scaled(tokens, chunk):
    """The gradients kept by the forward pass are scaled in place only when nobody needs them again: a kept graph gives
    the same gradients in every pass, and a scaled loss the scaled ones (bf16 dx: the scale is a power of two)."""
    torch.manual_seed(3)
    x = torch.randn(tokens, 64, device="cuda").bfloat16().requires_grad_()
    # logits of about 0.8: rounded to bf16 they move by up to 2^-8, and so do the probabilities
    w = (0.1 * torch.randn(512, 64, device="cuda")).requires_grad_()
    t = torch.randint(0, 512, (tokens,), device="cuda")
    t[5] = -1
    run = lambda: N.linear_cross_entropy(x, w, t, chunk_tokens=chunk)
    gx, gw = torch.autograd.grad(run(), (x, w))
    logits = (x.detach().float() @ w.detach().bfloat16().float().t()).requires_grad_()
    F.cross_entropy(logits, t, ignore_index=-1).backward()
    _close(gw, logits.grad.t() @ x.detach().float(), 1e-2)
    loss = run()
    for _ in range(2):
        a, b = torch.autograd.grad(0.25 * loss, (x, w), retain_graph=True)
        assert torch.equal(a, 0.25 * gx) and torch.allclose(b, 0.25 * gw, rtol=1e-5, atol=1e-8)
    a, b = torch.autograd.grad(0.25 * loss, (x, w))
    assert torch.equal(a, 0.25 * gx) and torch.allclose(b, 0.25 * gw, rtol=1e-5, atol=1e-8)
    a, b = torch.autograd.grad(run(), (x, w), grad_outputs=torch.tensor([1.0, 0.25], device="cuda"), is_grads_batched=True)
    assert torch.equal(a[1], 0.25 * gx) and torch.allclose(b[1], 0.25 * gw, rtol=1e-5, atol=1e-8) and torch.equal(a[0], gx)
    held = []
    with torch.autograd.graph.saved_tensors_hooks(lambda v: held.append(v) or v, lambda v: v):
        loss = run()
    copies = [v.clone() for v in held]
    torch.autograd.grad(0.25 * loss, (x, w))
    assert all(torch.equal(a, b) for a, b in zip(held, copies))


@pytest.mark.gpu
def test_fused_mlp_matches_unfused_reference():
    T, D = 520, 256
    x = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    res = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    w_fc = (torch.randn(4 * D, D, device="cuda") / D ** 0.5).requires_grad_()
    w_pj = (torch.randn(D, 4 * D, device="cuda") / (4 * D) ** 0.5).requires_grad_()
    out = N.mlp(x, w_fc, w_pj, res)
    g = torch.randn_like(out)
    out.backward(g)
    xr = x.detach().float().requires_grad_()
    rr = res.detach().float().requires_grad_()
    fr = w_fc.detach().bfloat16().float().requires_grad_()
    pr = w_pj.detach().bfloat16().float().requires_grad_()
    ref = rr + torch.relu(xr @ fr.t()).square() @ pr.t()
    ref.backward(g.float())
    _close(out, ref, 2e-2)
    _close(x.grad, xr.grad, 3e-2)
    _close(w_fc.grad, fr.grad, 3e-2)
    _close(w_pj.grad, pr.grad, 3e-2)
    assert torch.equal(res.grad, g)


@pytest.mark.gpu
def test_norm_branch_adds_both_gradients():
    x = torch.randn(33, 768, device="cuda").bfloat16().requires_grad_()
    xp, h = N.norm_branch(x)
    g1, g2 = torch.randn_like(xp), torch.randn_like(h)
    (xp * g1).sum().backward(retain_graph=True)
    gx_pass = x.grad.clone()
    x.grad = None
    ((xp * g1).sum() + (h * g2).sum()).backward()
    xr = x.detach().float().requires_grad_()
    (_ref_rms(xr) * g2.float()).sum().backward()
    _close(x.grad, xr.grad + g1.float(), 2e-2)
    assert torch.equal(xp, x)
    _close(gx_pass, g1.float(), 1e-2)  # the pass-through output alone hands its gradient on unchanged


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 256, 3, 3, 128), (1, 1024, 4, 2, 128), (3, 384, 2, 2, 64), (2, 128, 2, 1, 64)])
def test_flash_attention_forward_matches_fp32_reference(shape):
    from dion_b200 import ops
    from dion_b200.ops.nn import flash_attention_forward

    B, T, H, Hkv, D = shape
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(B, T, H, D, device="cuda", generator=g).to(torch.bfloat16)
    k = torch.randn(B, T, Hkv, D, device="cuda", generator=g).to(torch.bfloat16)
    v = torch.randn(B, T, Hkv, D, device="cuda", generator=g).to(torch.bfloat16)
    out, lse = flash_attention_forward(q, k, v)
    ops.check_status()
    qf, kf, vf = (t.float().transpose(1, 2) for t in (q, k, v))
    kf = kf.repeat_interleave(H // Hkv, dim=1)
    vf = vf.repeat_interleave(H // Hkv, dim=1)
    s = (qf @ kf.transpose(-1, -2)) / D ** 0.5
    s = s.masked_fill(torch.triu(torch.ones(T, T, device="cuda", dtype=torch.bool), 1), float("-inf"))
    ref = torch.softmax(s, dim=-1) @ vf
    err = (out.float().transpose(1, 2) - ref).abs().max().item()
    assert err < 2e-2, err
    torch.testing.assert_close(lse, torch.logsumexp(s, dim=-1), rtol=1e-3, atol=1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 256, 3, 3, 128), (1, 1024, 4, 2, 128), (3, 384, 2, 2, 64), (2, 128, 4, 1, 64)])
def test_flash_attention_backward_matches_fp32_reference(shape):
    from dion_b200 import ops
    from dion_b200.ops.nn import flash_attention_backward, flash_attention_forward

    B, T, H, Hkv, D = shape
    g = torch.Generator(device="cuda").manual_seed(11)
    q = torch.randn(B, T, H, D, device="cuda", generator=g).to(torch.bfloat16)
    k = torch.randn(B, T, Hkv, D, device="cuda", generator=g).to(torch.bfloat16)
    v = torch.randn(B, T, Hkv, D, device="cuda", generator=g).to(torch.bfloat16)
    d_out = torch.randn(B, T, H, D, device="cuda", generator=g).to(torch.bfloat16)
    out, lse = flash_attention_forward(q, k, v)
    dq, dk, dv = flash_attention_backward(q, k, v, out, lse, d_out)
    ops.check_status()
    qf, kf, vf = (t.float().requires_grad_() for t in (q, k, v))
    kr = kf.transpose(1, 2).repeat_interleave(H // Hkv, dim=1)
    vr = vf.transpose(1, 2).repeat_interleave(H // Hkv, dim=1)
    s = (qf.transpose(1, 2) @ kr.transpose(-1, -2)) / D ** 0.5
    s = s.masked_fill(torch.triu(torch.ones(T, T, device="cuda", dtype=torch.bool), 1), float("-inf"))
    ref = (torch.softmax(s, dim=-1) @ vr).transpose(1, 2)
    ref.backward(d_out.float())
    for name, got, want in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
        err = (got.float() - want).abs().max().item() / want.abs().max().item()
        assert err < 2e-2, (name, err)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 128, 2, 64), (2, 64, 2, 64), (2, 256, 2, 64), (2, 128, 2, 128)])
def test_attention_backward_refuses_keys_of_other_sizes(shape):
    """Sequences, rows or columns that q does not have: the kernels would read k and v where they are not."""
    from dion_b200.ops.nn import flash_attention_backward

    q, k = torch.zeros(2, 128, 4, 64, device="cuda").bfloat16(), torch.zeros(shape, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="does not go with q"):
        flash_attention_backward(q, k, k, q, torch.zeros(2, 4, 128, device="cuda"), q)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [2047, 2048])
@pytest.mark.parametrize("vocab", [24576, 24584])
def test_the_loss_alone_of_many_rows(rows, vocab):
    """Both numbers of threads per row of a pass without a gradient.  A thread adds up to 97 exponentials of 2 ulp each."""
    torch.manual_seed(rows)
    x = 3 * torch.randn(rows, vocab, device="cuda").bfloat16()
    t, loss, before = torch.randint(0, vocab, (rows,), device="cuda"), torch.empty(rows, device="cuda"), x.clone()
    assert N.runtime.use_cuda_kernels(x)
    torch.ops.dion_b200.cross_entropy_fwd_bwd(x, t, loss, None, 1.0, -1, False)
    torch.testing.assert_close(loss.double(), F.cross_entropy(x.double(), t, reduction="none"), rtol=2.0 ** -22,
                               atol=97 * 2.0 ** -24 + 1e-5)
    assert torch.equal(x, before)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [
    (150, 128, 1, 1, 128),  # one tile per head; a head for every CTA and two left over
    (40, 256, 4, 4, 64),    # pairs of query tiles, 160 heads
    (5, 640, 40, 8, 64),    # an odd number of tiles: the last pair is a single one; grouped kv heads
    (1, 384, 2, 2, 128),    # fewer tiles than SMs: one query tile per work item
    (2, 896, 24, 2, 128),   # leftover heads over several rounds, back and forth over the CTAs
])
def test_flash_attention_work_split(shape):
    """Every (head, tile) of the persistent kernels is worked on exactly once, forward and backward.  Outputs are bf16
    (2^-9 of values up to about 4.5) of products with bf16 probabilities: 2e-2, as for the shapes above."""
    from dion_b200 import ops
    from dion_b200.ops.nn import flash_attention_backward, flash_attention_forward

    B, T, H, Hkv, D = shape
    g = torch.Generator(device="cuda").manual_seed(17)
    q, k, v, d_out = (torch.randn(B, T, h, D, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hkv, Hkv, H))
    out, lse = flash_attention_forward(q, k, v)
    grads = flash_attention_backward(q, k, v, out, lse, d_out)
    ops.check_status()
    qf, kf, vf = (t.float().requires_grad_() for t in (q, k, v))
    kr, vr = (t.transpose(1, 2).repeat_interleave(H // Hkv, dim=1) for t in (kf, vf))
    s = (qf.transpose(1, 2) @ kr.transpose(-1, -2)) / D ** 0.5
    s = s.masked_fill(torch.triu(torch.ones(T, T, device="cuda", dtype=torch.bool), 1), float("-inf"))
    ref = (torch.softmax(s, dim=-1) @ vr).transpose(1, 2)
    ref.backward(d_out.float())
    assert (out.float() - ref).abs().max().item() < 2e-2
    torch.testing.assert_close(lse, torch.logsumexp(s, dim=-1), rtol=1e-3, atol=1e-3)
    for name, got, want in zip(("dq", "dk", "dv"), grads, (qf.grad, kf.grad, vf.grad)):
        err = (got.float() - want).abs().max().item() / want.abs().max().item()
        assert err < 2e-2, (name, err)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 1, 2, 2, 64), (3, 17, 4, 2, 64), (4, 127, 3, 3, 128), (2, 129, 4, 4, 128), (64, 333, 6, 6, 128),
                                   (8, 777, 12, 12, 64), (1, 24, 6, 1, 128)])
def test_attention_of_any_length(shape):
    """Lengths around the edges of the tiles against fp32, forward and backward, and against NaN in what lies behind each
    sequence: nothing of the next sequence or of the padding may reach a result.  Bounds as for whole tiles."""
    B, T, H, Hkv, D = shape
    g = torch.Generator(device="cuda").manual_seed(29)
    q, k, v, d_out = (torch.randn(B, T, h, D, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
                      for h in (H, Hkv, Hkv, H))
    y = N.causal_attention(q, k, v)
    assert "AnyLength" in type(y.grad_fn.next_functions[0][0]).__name__
    y.backward(d_out.detach().view_as(y))
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    kr, vr = (t.transpose(1, 2).repeat_interleave(H // Hkv, dim=1) for t in (kf, vf))
    s = (qf.transpose(1, 2) @ kr.transpose(-1, -2)) / D ** 0.5
    s = s.masked_fill(torch.triu(torch.ones(T, T, device="cuda", dtype=torch.bool), 1), float("-inf"))
    ref = (torch.softmax(s, dim=-1) @ vr).transpose(1, 2)
    ref.backward(d_out.detach().float())
    assert (y.view_as(ref).float() - ref).abs().max().item() < 2e-2
    for name, got, want in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        if T == 1 and name != "dv":
            # P is 1 and O is V bit for bit, so dP - delta is the difference of one sum taken in two orders: up to
            # 2 D 2^-24 of sum |dO||V| < 100, times |k| or |q| < 5, over sqrt(D) = 8: 4.8e-4 at worst, 1e-6 as a rule
            assert got.float().abs().max().item() < 1e-4, name
            continue
        err = (got.float() - want).abs().max().item() / max(want.abs().max().item(), 1.0)
        assert err < 2e-2, (name, err)
    if B > 1:  # the first sequence alone gives the same, and is not touched by NaN in the second
        with torch.no_grad():
            alone = N.causal_attention(q[:1], k[:1], v[:1])
            for t in (q, k, v):
                t[1:] = float("nan")
            assert torch.equal(N.causal_attention(q, k, v)[:1], alone) and torch.equal(alone, y[:1])


@pytest.mark.gpu
def test_attention_of_other_lengths_keeps_what_the_library_takes_and_refuses():
    from torch.utils._python_dispatch import TorchDispatchMode

    from dion_b200.ops.nn import flash_attention_forward

    q = torch.randn(2, 100, 4, 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):
        flash_attention_forward(q, q, q)

    class Names(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Names() as names:
        N.causal_attention(q, q, q)
    assert not any("dion_b200" in n for n in names.seen)
    shifted = torch.randn(q.numel() + 1, device="cuda").bfloat16()[1:].view_as(q)  # rows on odd addresses
    assert torch.equal(N.causal_attention(shifted, shifted, shifted), N.causal_attention(*[shifted.clone()] * 3))
    x = q.clone().requires_grad_()
    grad, = torch.autograd.grad(N.causal_attention(x, x, x).float().square().sum(), x, create_graph=True)
    with pytest.raises(RuntimeError):
        grad.float().sum().backward()


def test_attention_takes_operands_of_one_device_only(monkeypatch):
    """The questions that come before the kernels, asked of tensors without memory."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    with FakeTensorMode():
        tiles, ragged = ({d: torch.empty(2, T, 4, 64, dtype=torch.bfloat16, device=d) for d in ("cuda:0", "cuda:1", "cpu")}
                         for T in (128, 100))
    monkeypatch.setattr(N, "_transformed", lambda t: False)  # a stand-in is a subclass
    for ask, t in ((N.flash_attention_supported, tiles), (N._any_length, ragged)):
        q = t["cuda:0"]
        assert ask(q, q, q)
        for other in (t["cuda:1"], t["cpu"]):
            assert not ask(q, other, q) and not ask(q, q, other)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [100, 128, 384])
def test_attention_of_tensors_on_odd_addresses(T):
    """q, k, v and the gradient that comes in, contiguous but shifted by one element: the bits of aligned copies."""
    def shifted(*shape):
        n = torch.Size(shape).numel()
        return torch.randn(n + 1, device="cuda").bfloat16()[1:].view(shape)

    def run(q, k, v, dy):
        q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
        y = N.causal_attention(q, k, v)
        return (y, *torch.autograd.grad(y, (q, k, v), dy))

    ts = shifted(2, T, 4, 64), shifted(2, T, 2, 64), shifted(2, T, 2, 64), shifted(2, T, 256)
    assert all(t.data_ptr() % 16 and t.is_contiguous() for t in ts)
    for got, want in zip(run(*ts), run(*(t.clone() for t in ts))):
        assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [128, 100])
def test_attention_refuses_operands_of_another_device(T):
    from dion_b200.ops import runtime

    q, far = torch.zeros(1, T, 2, 64, device="cuda").bfloat16(), torch.zeros(1, T, 2, 64).bfloat16()
    lse, stats, status = torch.zeros(1, 2, T, device="cuda"), torch.zeros(2, 1, 2, 128, device="cuda"), runtime.status_tensor(q.device)
    for k, v in ((far, far), (far, q), (q, far)):
        with pytest.raises(RuntimeError):
            N.causal_attention(q, k, v)
    op = torch.ops.dion_b200
    for args in ((q, far, q, q, lse), (q, q, far, q, lse), (q, q, q, far, lse), (q, q, q, q, lse.cpu()), (far, q, q, q, lse)):
        with pytest.raises(RuntimeError, match="attention operands must be"):
            op.attn_fwd(*args, 0.125, status)
    good = [q, q, q, q, q, lse, stats, q.clone(), q.clone(), q.clone()]
    for i in range(len(good)):
        args = good[:i] + [good[i].cpu()] + good[i + 1:]
        with pytest.raises(RuntimeError, match="attention operands must be"):
            op.attn_bwd(*args, 0.125, status)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 384, 6, 6, 128), (64, 512, 6, 3, 64), (2, 2048, 16, 4, 128), (64, 333, 6, 6, 128)])
def test_flash_attention_gives_the_same_bits_in_every_run(shape):
    """No sum depends on the order in which warps or CTAs run, so a difference between two runs is a race."""
    from dion_b200.ops.nn import _attention_backward as flash_attention_backward
    from dion_b200.ops.nn import _attention_forward as flash_attention_forward

    B, T, H, Hkv, D = shape
    g = torch.Generator(device="cuda").manual_seed(23)
    q, k, v, d_out = (torch.randn(B, T, h, D, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hkv, Hkv, H))
    first = None
    for _ in range(8):
        out, lse = flash_attention_forward(q, k, v)
        run = (out, lse, *flash_attention_backward(q, k, v, out, lse, d_out))
        first = first or run
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), first, run):
            assert torch.equal(a, b), name


@pytest.mark.gpu
def test_overlapping_launches_in_a_graph_and_between_streams():
    """Kernels that start before their predecessor has ended: a chain of this library's kernels and torch's, eagerly,
    captured in a graph and with its halves on two streams, gives the same bits."""
    from dion_b200.ops.nn import flash_attention_forward

    g = torch.Generator(device="cuda").manual_seed(3)
    w1, w2 = (torch.randn(512, 512, device="cuda", generator=g).bfloat16() * 0.05 for _ in range(2))

    def first(x, buf):
        buf.zero_()                                    # a plain launch before, between and after
        buf.add_(x)
        h = N.linear(N.rms_norm(buf), w1)
        q = h.view(2, 128, 8, 64)
        return N.linear(flash_attention_forward(q, q, q)[0].view(256, 512), w2)

    def second(y):
        return N.linear(torch.relu(N.rms_norm(y)), w1) + y

    with torch.no_grad():
        xs = [torch.randn(256, 512, device="cuda", generator=g).bfloat16() for _ in range(3)]
        buf = torch.empty_like(xs[0])
        want = [second(first(x, buf)).clone() for x in xs]
        x0 = xs[0].clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = second(first(x0, buf))
        for x, w in zip(xs, want):
            x0.copy_(x)
            graph.replay()
            assert torch.equal(got, w)
        side = torch.cuda.Stream()
        for x, w in zip(xs, want):
            y = first(x, buf)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                z = second(y)
            torch.cuda.current_stream().wait_stream(side)
            y.record_stream(side)
            assert torch.equal(z, w)


@pytest.mark.gpu
def test_linear_fanout_matches_separate_linears():
    x = torch.randn(640, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    ws = [torch.nn.Parameter(torch.randn(n, 256, device="cuda") * 0.05) for n in (256, 128, 384)]
    outs = N.linear_fanout(x, *ws)
    gs = [torch.randn_like(o) for o in outs]
    torch.autograd.backward(outs, gs)
    got = [x.grad.clone()] + [w.grad.clone() for w in ws]
    x.grad = None
    for w in ws:
        w.grad = None
    ref = [N.linear(x, w) for w in ws]
    torch.autograd.backward(ref, gs)
    for o, r in zip(outs, ref):
        assert torch.equal(o, r)
    want = [x.grad] + [w.grad for w in ws]
    for g, w in zip(got, want):
        err = (g.float() - w.float()).abs().max().item() / w.float().abs().max().item()
        assert err < 1e-2, err


@pytest.mark.gpu
@pytest.mark.parametrize("rows,dim", [(300, 768), (64, 4096), (1000, 1024), (5, 256)])
@pytest.mark.parametrize("gain_dtype", [torch.float32, torch.bfloat16])
def test_rms_norm_with_gain_kernels(rows, dim, gain_dtype):
    """RMSNorm with a learnable gain: forward, input gradient and the gain's gradient (per-block partial
    sums in a fixed order) against fp32 PyTorch; two backward passes give the same bits."""
    from dion_b200.ops import nn as N

    x = torch.randn(rows, dim, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).to(gain_dtype).requires_grad_()
    g = torch.randn(rows, dim, device="cuda").bfloat16()
    y = N.rms_norm_gain(x, w, 1e-5)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    yr = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-5) * wr
    yr.backward(g.float())
    _close(y, yr, 2e-2)
    _close(x.grad, xr.grad, 3e-2)
    _close(w.grad, wr.grad, 2e-2)
    first = w.grad.clone()
    w.grad = None
    x.grad = None
    N.rms_norm_gain(x, w, 1e-5).backward(g)
    assert torch.equal(w.grad, first)


@pytest.mark.gpu
def test_swiglu_kernels():
    from dion_b200.ops import nn as N

    g = torch.randn(257, 1024, device="cuda").bfloat16().requires_grad_()
    u = torch.randn(257, 1024, device="cuda").bfloat16().requires_grad_()
    d = torch.randn(257, 1024, device="cuda").bfloat16()
    h = N.swiglu(g, u)
    h.backward(d)
    gr, ur = g.detach().float().requires_grad_(), u.detach().float().requires_grad_()
    hr = torch.nn.functional.silu(gr) * ur
    hr.backward(d.float())
    _close(h, hr, 2e-2)
    _close(g.grad, gr.grad, 2e-2)
    _close(u.grad, ur.grad, 2e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("B,T,heads,head_dim", [(1, 24, 6, 128), (3, 77, 2, 64), (2, 256, 4, 64), (1, 40, 1, 64), (8, 640, 5, 64)])
def test_block_without_gradients_runs_natively_with_the_same_bits(B, T, heads, head_dim):
    """A pass that records no gradients takes one native call per block; a hook on a part of the block, and recorded
    gradients, take the general path.  Same kernels, same bits."""
    from dion_b200 import ops
    from dion_b200.models import GPT, GPTConfig

    with torch.device("cuda"):
        model = GPT(GPTConfig(sequence_len=T, vocab_size=512, n_layer=2, n_head=heads, n_embd=heads * head_dim))
    model.init_weights()
    idx = torch.randint(0, 512, (B, T), device="cuda")
    general = model(idx, return_logits=True)
    assert general.requires_grad
    with torch.no_grad():
        native = model(idx, return_logits=True)
        x = torch.randn(B, T, heads * head_dim, device="cuda").bfloat16()
        assert model.transformer.h[0]._forward_native(x) is not None
        seen = []
        handle = model.transformer.h[0].attn.register_forward_hook(lambda *a: seen.append(1))
        assert model.transformer.h[0]._forward_native(x) is None
        hooked = model(idx, return_logits=True)
        handle.remove()
    assert torch.equal(native, general) and torch.equal(hooked, general) and seen == [1]
    ops.check_status()


class _SeenDispatch(torch.utils._python_dispatch.TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


class _SeenFunction(torch.overrides.TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


def test_modes_tracers_and_transforms_observe_a_call():
    assert not N._observed()
    with torch.device("cpu"):  # a default device only acts on the creation of tensors
        assert not N._observed()
        with _SeenFunction():
            assert N._observed()
    for mode in (_SeenDispatch(), _SeenFunction(), torch.autograd.forward_ad.dual_level()):
        with mode:
            assert N._observed()
        assert not N._observed()
    answers = []
    torch.vmap(lambda v: answers.append(N._observed()) or v)(torch.zeros(2))
    torch.jit.trace(lambda v: answers.append(N._observed()) or v + 1, torch.zeros(2), check_trace=False)
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    answers.append(N._observed())
    handle.remove()
    assert answers == [True, True, True] and not N._observed()


@pytest.mark.gpu
def test_modes_see_the_operations_of_a_block_without_gradients():
    """A dispatch or function mode around a pass that records no gradients sees its products and norms, not one opaque call."""
    from dion_b200.models import GPT, GPTConfig

    with torch.device("cuda"):
        model = GPT(GPTConfig(sequence_len=40, vocab_size=512, n_layer=1, n_head=2, n_embd=128))
    model.init_weights()
    block, x = model.transformer.h[0], torch.randn(2, 40, 128, device="cuda").bfloat16()
    with torch.no_grad():
        plain = block(x)
        with _SeenDispatch() as d:
            assert torch.equal(block(x), plain)
        with _SeenFunction() as f:
            assert torch.equal(block(x), plain)
        with torch.device("cuda"):
            assert block._forward_native(x) is not None
    assert sum("dion_b200.gemm" in s for s in d.seen) >= 6 and not any("gpt_block_fwd" in s for s in d.seen)
    assert any("view" in s or "reshape" in s for s in f.seen) and not any("gpt_block_fwd" in s for s in f.seen)


_PRIVATE = [(torch._C._functorch, "peek_interpreter_stack"), (torch._C._functorch, "is_batchedtensor"),
            (torch._C._functorch, "is_legacy_batchedtensor"), (torch._C._autograd, "_top_saved_tensors_default_hooks"),
            (torch._C._autograd, "_get_current_graph_task_keep_graph")]


@pytest.mark.parametrize("how", ["missing", "other arguments"])
def test_interfaces_that_another_pytorch_lacks_mean_the_general_path(monkeypatch, how):
    """Every private interface that decides about a native call or a write in place may be absent or take other arguments."""
    def without(owner, name):
        if how == "missing":
            m.delattr(owner, name)
        else:
            m.setattr(owner, name, lambda one, two, three: None)

    t = torch.zeros(2)
    assert not N._observed() and not N._transformed(t)
    for owner, name in [(torch._C._functorch, "peek_interpreter_stack"), (torch._C, "_len_torch_dispatch_stack"),
                        (torch.nn.modules.module, "_has_any_global_hook")]:
        with monkeypatch.context() as m:
            without(owner, name)
            assert N._observed()
    with _SeenFunction():
        with monkeypatch.context() as m:  # either of the two tells of the mode
            without(torch._C, "_len_torch_function_stack")
            assert N._observed()
        with monkeypatch.context() as m:
            without(torch.overrides, "_get_current_function_mode_stack")
            assert N._observed()
    for name in ("peek_interpreter_stack", "is_batchedtensor", "is_legacy_batchedtensor"):
        with monkeypatch.context() as m:
            without(torch._C._functorch, name)
            assert N._transformed(t)
    assert not N._observed() and not N._transformed(t)


@pytest.mark.gpu
@pytest.mark.parametrize("owner,name", _PRIVATE)
def test_loss_gradients_where_pytorch_lacks_an_interface(monkeypatch, owner, name):
    x = torch.randn(256, 64, device="cuda").bfloat16().requires_grad_()
    w = (0.1 * torch.randn(512, 64, device="cuda")).requires_grad_()
    t = torch.randint(0, 512, (256,), device="cuda")
    want = torch.autograd.grad(0.25 * N.linear_cross_entropy(x, w, t), (x, w))
    kept = N.linear_cross_entropy(x, w, t)
    with monkeypatch.context() as m:
        m.delattr(owner, name)
        got = torch.autograd.grad(0.25 * N.linear_cross_entropy(x, w, t), (x, w))
        again = [torch.autograd.grad(0.25 * kept, (x, w), retain_graph=True) for _ in range(2)]
    for g in (got, *again):
        assert all(torch.equal(a, b) for a, b in zip(g, want))


@pytest.mark.gpu
@pytest.mark.parametrize("T", [256, 200])
def test_block_without_gradients_holds_no_more_than_its_single_operations(T):
    """The native block gives every intermediate back once its last reader is issued: its peak is at most that of the general
    path, which a hook selects."""
    from dion_b200.models import GPT, GPTConfig

    with torch.device("cuda"):
        model = GPT(GPTConfig(sequence_len=T, vocab_size=512, n_layer=1, n_head=4, n_embd=512))
    model.init_weights()
    block, x = model.transformer.h[0], torch.randn(8, T, 512, device="cuda").bfloat16()

    def peak():
        block(x)
        torch.cuda.synchronize()
        held = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        block(x)
        return torch.cuda.max_memory_allocated() - held

    with torch.no_grad():
        assert block._forward_native(x) is not None
        native = peak()
        block.attn.register_forward_hook(lambda *a: None)
        assert block._forward_native(x) is None
        general = peak()
    assert native <= general


def test_long_contractions_are_halved_where_the_last_wave_is_nearly_empty():
    halved = [(8192, 768, 50304), (8192, 640, 50304), (6144, 1024, 50304), (8192, 1280, 50304), (7000, 768, 50304),
              (8192, 768, 16384), (4096, 1280, 50304)]
    whole = [(8192, 512, 50304), (8192, 1024, 50304), (4096, 2048, 32000), (8192, 2048, 16384), (4096, 4096, 128256),
             (8192, 4096, 128256), (8192, 1536, 50304), (8192, 768, 16376), (300, 256, 50304)]
    assert all(N._halve_contraction(*s, 74) for s in halved) and not any(N._halve_contraction(*s, 74) for s in whole)
    assert not N._halve_contraction(8192, 768, 50304, 96)  # a device on which one wave takes the tiles


@pytest.mark.gpu
def test_halved_input_gradient_of_the_loss():
    """A whole and a ragged chunk whose gradient products are cut in two: dx against the fp32 statement, the same bits again."""
    T, K, V, chunk = 8192 + 6100, 768, 16384, 8192
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert N._halve_contraction(chunk, K, V, pairs) and -(-(T - chunk) // 256) * 3 < pairs  # the second chunk is not cut
    x = torch.randn(T, K, device="cuda").bfloat16().requires_grad_()
    w = (0.02 * torch.randn(V, K, device="cuda")).requires_grad_()
    t = torch.randint(0, V, (T,), device="cuda")
    runs = [torch.autograd.grad(N.linear_cross_entropy(x, w, t, chunk_tokens=chunk), (x, w)) for _ in range(3)]
    assert all(torch.equal(a, b) for r in runs[1:] for a, b in zip(r, runs[0]))
    wb = w.detach().bfloat16().float()
    logits = x.detach().float() @ wb.t()
    p = torch.softmax(logits, -1)
    p[torch.arange(T, device="cuda"), t] -= 1.0
    want = (p / T) @ wb
    # logits of about 0.55, the probabilities and dx are rounded to bf16 once each (2^-9 relative)
    assert ((runs[0][0].float() - want).norm() / want.norm()).item() < 3 * 2.0 ** -9


@pytest.mark.parametrize("sizes,kernels", [
    ((8, 777, 12, 12, 64), True),
    ((1, 1500, 12, 12, 64), True),      # a CTA for every tile
    ((1, 1700, 12, 12, 64), False),     # few heads, more tiles than SMs
    ((8, 1700, 12, 12, 64), True),
    ((8, 8100, 12, 12, 64), False),
    ((64, 333, 6, 6, 128), True),
    ((32, 500, 6, 6, 128), False),
    ((1, 700, 6, 6, 128), True),
    ((1, 1000, 6, 6, 128), False),
    ((1, 300, 32, 8, 128), False),      # a group's dK and dV are one CTA's
    ((8, 300, 32, 8, 128), True),
    ((1, 100, 32, 8, 128), True),
    ((1, 24, 6, 6, 128), True),         # waits for the host
    ((64, 17, 12, 12, 64), False),      # does not
])
def test_which_ragged_lengths_run_on_the_kernels(sizes, kernels, monkeypatch):
    """Where the library measured faster, the call goes to the library as it did before the kernels took every length."""
    assert N._ragged_on_kernels(*sizes) == kernels
    assert N.attention_on_kernels(*sizes) == kernels
    assert N.attention_on_kernels(sizes[0], 128 * (1 + sizes[1] // 128), *sizes[2:])  # whole tiles are never asked about
    monkeypatch.setattr(N, "ATTENTION_IMPL", "library")
    assert not N.attention_on_kernels(*sizes)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,kernels", [((1, 1700, 12, 12, 64), False), ((1, 1200, 12, 12, 64), True), ((1, 300, 8, 2, 128), False),
                                           ((2, 100, 8, 2, 128), True)])
def test_ragged_attention_takes_the_path_that_was_chosen(shape, kernels):
    """The same one with and without gradients."""
    from dion_b200 import ops

    B, T, H, Hkv, D = shape
    q, k, v = (torch.randn(B, T, h, D, device="cuda").bfloat16().requires_grad_() for h in (H, Hkv, Hkv))
    before = ops.launch_count()
    y = N.causal_attention(q, k, v)
    assert ops.launch_count() - before == int(kernels) and y.requires_grad
    with torch.no_grad():
        again = N.causal_attention(q, k, v)
    assert ops.launch_count() - before == 2 * int(kernels) and not again.requires_grad
    assert not kernels or torch.equal(again, y)
    kr, vr = (t.detach().double().transpose(1, 2).repeat_interleave(H // Hkv, dim=1) for t in (k, v))
    ref = F.scaled_dot_product_attention(q.detach().double().transpose(1, 2), kr, vr, is_causal=True).transpose(1, 2)
    # bf16 values up to about 4.5 of products with bf16 probabilities
    assert (y.detach().view(B, T, H, D).double() - ref).abs().max().item() < 2e-2


@pytest.mark.gpu
def test_every_launch_is_counted_once():
    """The count of a training step, and of Newton-Schulz with and without norms in hand, against a profile of the same."""
    from torch.profiler import ProfilerActivity, profile

    from dion_b200 import Dion, ops
    from dion_b200.models import GPT, GPTConfig
    from dion_b200.optim.newton_schulz import newton_schulz

    with torch.device("cuda"):
        model = GPT(GPTConfig(sequence_len=128, vocab_size=1024, n_layer=2, n_head=4, n_embd=256))
    model.init_weights()
    hidden = [p for p in model.parameters() if p.dim() == 2 and p.shape[0] <= 1024 and p.shape != (1024, 256)]
    rest = [p for p in model.parameters() if all(p is not h for h in hidden)]
    opt = Dion([dict(params=hidden), dict(params=rest, algorithm="lion")], lr=1e-3, rank_fraction=0.25)
    idx = torch.randint(0, 1024, (2, 128), device="cuda")
    g = torch.randn(2, 300, 520, device="cuda").bfloat16()

    def step():
        model(idx, idx).backward()
        opt.step()
        opt.zero_grad()
        newton_schulz(g)
        newton_schulz(g, sumsq=g.float().square().sum((1, 2)))

    for _ in range(2):
        step()
    torch.cuda.synchronize()
    before = ops.launch_count()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        step()
        torch.cuda.synchronize()
    kernels = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA and "dion::" in e.name]
    assert ops.launch_count() - before == len(kernels) > 100
