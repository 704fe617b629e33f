"""tcgen05 GEMM against a plain fp32 PyTorch reference of the same op."""
import pytest
import torch

from dion_b200 import ops
from dion_b200.ops.gemm import gemm


def _operand(rows, cols, dtype, transposed, batch=None, device="cuda"):
    """Logical [rows, cols] matrix, stored row-major or as the transpose of a row-major one."""
    shape = (cols, rows) if transposed else (rows, cols)
    if batch is not None:
        shape = (batch, *shape)
    t = torch.randn(shape, device=device, dtype=torch.float32).to(dtype)
    return t.transpose(-1, -2) if transposed else t


def _rel_err(x, ref):
    return ((x.float() - ref.float()).abs().max() / ref.float().abs().max().clamp_min(1e-20)).item()


def test_reference_semantics_cpu():
    a = torch.randn(5, 7)
    b = torch.randn(7, 3)
    c = torch.randn(5, 3)
    out = gemm(a, b, c=c, alpha=0.5, beta=2.0)
    torch.testing.assert_close(out, 0.5 * a @ b + 2.0 * c)
    out2 = torch.ones(5, 3)
    gemm(a, b, out=out2, accumulate=True)
    torch.testing.assert_close(out2, 1 + a @ b)
    out3 = gemm(a, b, act="relu2")
    torch.testing.assert_close(out3, torch.relu(a @ b) ** 2)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("shape", [(256, 256, 256), (384, 200, 328), (128, 64, 64), (1000, 520, 72)])
def test_gemm_layouts(dtype, ta, tb, shape):
    M, N, K = shape
    a = _operand(M, K, dtype, ta)
    b = _operand(K, N, dtype, tb)
    out = gemm(a, b, out_dtype=torch.float32)
    ref = a.float() @ b.float()
    tol = 2e-5 if dtype == torch.bfloat16 else 4e-3
    assert _rel_err(out, ref) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("block_n", [64, 128, 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemm_block_n_and_batch(block_n, dtype):
    a = _operand(300, 192, dtype, False, batch=3)
    b = _operand(192, 520, dtype, True, batch=3)
    out = gemm(a, b, out_dtype=torch.float32, block_n=block_n)
    ref = torch.matmul(a.float(), b.float())
    assert _rel_err(out, ref) < (2e-5 if dtype == torch.bfloat16 else 4e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("c_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_epilogue_alpha_beta(c_dtype, out_dtype):
    a = _operand(520, 256, torch.bfloat16, False)
    b = _operand(256, 392, torch.bfloat16, False)
    c = torch.randn(520, 392, device="cuda").to(c_dtype)
    shadow = torch.empty(520, 392, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, c=c, alpha=-0.25, beta=0.75, out_dtype=out_dtype, shadow=shadow)
    ref = -0.25 * (a.float() @ b.float()) + 0.75 * c.float()
    assert _rel_err(out, ref) < (1e-2 if out_dtype == torch.bfloat16 else 2e-5)
    assert torch.equal(shadow, out.to(torch.bfloat16))


@pytest.mark.gpu
def test_gemm_inplace_accumulate_into_c():
    a = _operand(256, 128, torch.float32, False)
    b = _operand(128, 256, torch.float32, True)
    m = torch.randn(256, 256, device="cuda")
    ref = m - 0.05 * (a @ b)
    gemm(a, b, c=m, out=m, alpha=-0.05, beta=1.0)
    assert _rel_err(m, ref) < 1e-3


@pytest.mark.gpu
def test_gemm_relu2():
    a = _operand(256, 128, torch.bfloat16, False)
    b = _operand(128, 512, torch.bfloat16, True)
    out = gemm(a, b, act="relu2", out_dtype=torch.float32)
    ref = torch.relu(a.float() @ b.float()) ** 2
    assert _rel_err(out, ref) < 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemm_symmetric(dtype):
    x = _operand(640, 328, dtype, False, batch=2)
    out = gemm(x, x.transpose(-1, -2), out_dtype=torch.float32, symmetric=True)
    ref = torch.matmul(x.float(), x.float().transpose(-1, -2))
    assert _rel_err(out, ref) < (2e-5 if dtype == torch.bfloat16 else 4e-3)
    assert torch.equal(out, out.transpose(-1, -2))


@pytest.mark.gpu
@pytest.mark.parametrize("split_k", [1, 3, 8])
def test_gemm_split_k_atomic(split_k):
    a = _operand(256, 4096, torch.bfloat16, True)
    b = _operand(4096, 384, torch.bfloat16, False)
    out = torch.ones(256, 384, device="cuda")
    gemm(a, b, out=out, accumulate=True, split_k=split_k, alpha=0.5)
    ref = 1 + 0.5 * (a.float() @ b.float())
    assert _rel_err(out, ref) < 1e-4


@pytest.mark.gpu
def test_gemm_pointer_array_outputs():
    B = 5
    a = _operand(256, 96, torch.float32, False, batch=B)
    b = _operand(96, 384, torch.float32, True, batch=B)
    xs = [torch.randn(256, 384, device="cuda") for _ in range(B)]
    sh = [torch.empty(256, 384, device="cuda", dtype=torch.bfloat16) for _ in range(B)]
    refs = [0.9 * x - 0.1 * (a[i] @ b[i]) for i, x in enumerate(xs)]
    ptrs = torch.tensor([x.data_ptr() for x in xs], dtype=torch.int64, device="cuda")
    sptrs = torch.tensor([x.data_ptr() for x in sh], dtype=torch.int64, device="cuda")
    gemm(a, b, c=xs[0], out=xs[0], c_ptrs=ptrs, out_ptrs=ptrs, shadow=sh[0], shadow_ptrs=sptrs, alpha=-0.1, beta=0.9)
    for x, r, s in zip(xs, refs, sh):
        assert _rel_err(x, r) < 2e-3
        assert torch.equal(s, x.to(torch.bfloat16))


@pytest.mark.gpu
def test_gemm_unaligned_falls_back_to_library():
    a = torch.randn(33, 17, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(17, 9, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, out_dtype=torch.float32)
    assert _rel_err(out, a.float() @ b.float()) < 2e-2


@pytest.mark.gpu
def test_gemm_status_word_stays_clear():
    from dion_b200.ops import runtime

    a = _operand(512, 512, torch.bfloat16, False)
    gemm(a, a)
    runtime.check_status()


@pytest.mark.gpu
def test_gemm_relu2_save_pre_and_backward_multiplier():
    a = _operand(300, 128, torch.bfloat16, False)
    b = _operand(128, 520, torch.bfloat16, True)
    h = torch.empty(300, 520, device="cuda", dtype=torch.bfloat16)
    pre = torch.empty_like(h)
    gemm(a, b, out=h, shadow=pre, act="relu2_save_pre")
    ref_pre = a.float() @ b.float()
    assert _rel_err(pre, ref_pre) < 1e-2
    assert _rel_err(h, torch.relu(ref_pre) ** 2) < 1e-2
    dy = _operand(300, 64, torch.bfloat16, False)
    w = _operand(64, 520, torch.bfloat16, False)
    dpre = torch.empty(300, 520, device="cuda", dtype=torch.bfloat16)
    gemm(dy, w, c=pre, out=dpre, act="mul_relu2_grad")
    ref = (dy.float() @ w.float()) * 2 * torch.relu(pre.float())
    assert _rel_err(dpre, ref) < 1e-2
    # the same multiplier recovered from the stored activation h = relu(pre)^2
    dpre2 = torch.empty_like(dpre)
    gemm(dy, w, c=h, out=dpre2, act="mul_relu2_grad_sq")
    assert _rel_err(dpre2, ref) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("shape", [(512, 512, 256), (640, 296, 200), (200, 1000, 72)])
def test_gemm_cta_pair_layouts(dtype, ta, tb, shape):
    """256-row tiles computed by two CTAs of a cluster (tcgen05 cta_group::2), forced on small shapes."""
    M, N, K = shape
    a = _operand(M, K, dtype, ta)
    b = _operand(K, N, dtype, tb)
    out = gemm(a, b, out_dtype=torch.float32, pair=1)
    ref = a.float() @ b.float()
    assert _rel_err(out, ref) < (2e-5 if dtype == torch.bfloat16 else 4e-3)


@pytest.mark.gpu
def test_gemm_cta_pair_epilogues_batch_and_many_tiles():
    # batched, with C / alpha / beta and the second output; more tiles than CTA pairs so that the
    # persistent loop and both accumulator buffers wrap around several times
    a = _operand(1100, 320, torch.bfloat16, False, batch=5)
    b = _operand(320, 2100, torch.bfloat16, True, batch=5)
    c = torch.randn(5, 1100, 2100, device="cuda").to(torch.bfloat16)
    shadow = torch.empty(5, 1100, 2100, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, c=c, alpha=0.5, beta=1.0, out_dtype=torch.float32, shadow=shadow, pair=1)
    ref = 0.5 * torch.matmul(a.float(), b.float()) + c.float()
    assert _rel_err(out, ref) < 2e-5
    assert torch.equal(shadow, out.to(torch.bfloat16))
    y = gemm(a, b, act="relu2", pair=1)
    assert _rel_err(y, torch.relu(torch.matmul(a.float(), b.float())) ** 2) < 1e-2
    # split-K accumulation with atomics
    acc = torch.zeros(5, 1100, 2100, device="cuda")
    gemm(a, b, out=acc, accumulate=True, split_k=3, pair=1)
    assert _rel_err(acc, torch.matmul(a.float(), b.float())) < 2e-5


@pytest.mark.gpu
def test_gemm_cta_pair_matches_single_cta_bitwise():
    a = _operand(4096, 768, torch.bfloat16, False)
    b = _operand(768, 3072, torch.bfloat16, True)
    y1 = gemm(a, b, pair=1)
    y0 = gemm(a, b, pair=-1)
    assert torch.equal(y0, y1)


def _split(x):
    hi = (x.contiguous().view(torch.int32) & -8192).view(torch.float32)
    return hi, x - hi


def test_gemm_hi_lo_operands_and_column_scale_cpu():
    a, b, c = torch.randn(2, 9, 12), torch.randn(2, 12, 5), torch.randn(2, 9, 5)
    a_hi, a_lo = _split(a)
    b_hi, b_lo = _split(b)
    out = gemm(a_hi, b_hi, a_lo=a_lo, b_lo=b_lo)
    torch.testing.assert_close(out, a_hi @ b_hi + a_lo @ b_hi + a_hi @ b_lo)
    s = torch.rand(2, 5)
    out = gemm(a, b, c=c, alpha=-1.0, beta=1.0, c_col_scale=s)
    torch.testing.assert_close(out, c * s.unsqueeze(1) - a @ b)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "relu2", "addc", "inplace", "grad_sq", "symmetric"])
@pytest.mark.parametrize("M,N,K,batch", [(1, 136, 64, 1), (24, 768, 768, 1), (300, 520, 72, 2), (129, 264, 200, 1),
                                         (2049, 1000, 1096, 1), (4100, 2056, 1024, 1), (777, 200, 768, 3)])
def test_tma_epilogue_moves_c_and_d_by_boxes(M, N, K, batch, mode):
    """bf16 C and D go through 32 x 64 boxes: ragged rows and columns are clipped, a row pitch above N leaves what lies
    between the rows alone, C may be D.  The result is the fp64 one rounded to bf16 once (2^-9) plus the error of the
    fp32 sum, K / 16 truncations of at most 2^-23 of the sum of magnitudes (of order sqrt(K) times an entry)."""
    if mode == "symmetric":
        N = M
    shape = lambda *s: s if batch == 1 else (batch, *s)
    a = torch.randn(*shape(M, K), device="cuda").bfloat16()
    w = a if mode == "symmetric" else torch.randn(*shape(N, K), device="cuda").bfloat16()
    pitch = (N + 7) // 8 * 8 + 16
    store = torch.full(shape(M, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
    out = store[..., :N]
    c = torch.zeros(*shape(M, pitch), device="cuda", dtype=torch.bfloat16)[..., :N]
    c.copy_(torch.randn(*shape(M, N), device="cuda").abs())
    ref = a.double() @ w.double().transpose(-1, -2)
    kw = {}
    if mode == "relu2":
        kw, ref = dict(act="relu2", alpha=0.5), torch.relu(0.5 * ref).square()
    elif mode == "addc":
        kw, ref = dict(c=c, beta=-1.5), ref - 1.5 * c.double()
    elif mode == "inplace":
        out.copy_(c)
        kw, ref = dict(c=out, beta=1.0), ref + c.double()
    elif mode == "grad_sq":
        kw, ref = dict(c=c, act="mul_relu2_grad_sq"), ref * 2 * c.double().sqrt()
    elif mode == "symmetric":
        c = (c + c.transpose(-1, -2)).contiguous() if N % 8 == 0 else None
        kw, ref = (dict(c=c, beta=2.0, symmetric=True), ref + 2 * c.double()) if c is not None else (dict(symmetric=True), ref)
    gemm(a, w.transpose(-1, -2), out=out, **kw)
    scale = ref.abs().amax().item()
    err = (out.double() - ref).abs()
    assert (err <= ref.abs() * 2 ** -8 + scale * 2 ** -14).all(), (err.max().item(), scale)
    assert torch.equal(store[..., N:], torch.full_like(store[..., N:], 7.0))
    from dion_b200 import ops

    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "inplace", "col_scale", "symmetric"])
@pytest.mark.parametrize("split3", [False, True])
@pytest.mark.parametrize("M,N,K,batch", [(1, 132, 40, 1), (300, 516, 72, 2), (2049, 1000, 1096, 1), (4100, 2056, 1024, 1),
                                         (777, 200, 768, 3)])
def test_tma_epilogue_fp32(M, N, K, batch, split3, mode):
    """The same for fp32 C and D.  tf32 operands lose up to 2^-10 of each factor (errors of K products add up like their
    squares), split ones 2^-21; the accumulator drops up to 2^-23 of its value with each of K / 8 multiplies."""
    if mode == "symmetric":
        N = M = M // 4 * 4 + 4
    shape = lambda *s: s if batch == 1 else (batch, *s)
    a = torch.randn(*shape(M, K), device="cuda")
    w = a if mode == "symmetric" else torch.randn(*shape(N, K), device="cuda")
    store = torch.full(shape(M, N + 20), 7.0, device="cuda")
    out = store[..., :N]
    ref = a.double() @ w.double().transpose(-1, -2)
    kw = {}
    if mode == "inplace":
        out.copy_(torch.randn_like(out))
        kw, ref = dict(c=out, beta=-0.5, alpha=2.0), 2 * ref - 0.5 * out.double()
    elif mode == "col_scale":
        c, d = torch.randn(*shape(M, N), device="cuda"), torch.rand(batch, N, device="cuda")
        kw, ref = dict(c=c, beta=1.0, alpha=-1.0, c_col_scale=d), c.double() * d.double().view(*shape(1, N)) - ref
    elif mode == "symmetric":
        kw = dict(symmetric=True)
    gemm(a, w.transpose(-1, -2), out=out, split3=split3, **kw)
    big = (a.double().norm(dim=-1).amax() * w.double().norm(dim=-1).amax()).item() * abs(kw.get("alpha", 1.0))
    bound = big * ((2 ** -20 + K / 8 * 2 ** -23) if split3 else 2 ** -8)
    assert (out.double() - ref).abs().amax().item() < bound + 1e-6
    assert torch.equal(store[..., N:], torch.full_like(store[..., N:], 7.0))
    from dion_b200 import ops

    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,split3", [(torch.bfloat16, False), (torch.float32, False), (torch.float32, True)])
@pytest.mark.parametrize("M,N,K,batch", [(300, 520, 72, 1), (4100, 2056, 1024, 1), (1300, 1032, 512, 6)])
def test_addend_with_broadcast_rows(dtype, split3, M, N, K, batch):
    """One row (or one matrix) added everywhere: a pitch of zero, which no tensor map describes.  The result is close to
    that with the addend written out (the same kernel arithmetic, one rounding to the result's type apart)."""
    shape = lambda *s: s if batch == 1 else (batch, *s)
    a = torch.randn(*shape(M, K), device="cuda").to(dtype)
    b = torch.randn(*shape(N, K), device="cuda").to(dtype).transpose(-1, -2)
    row = torch.randn(N, device="cuda").to(dtype)
    full = gemm(a, b, c=row.expand(*shape(M, N)).contiguous(), beta=2.0, split3=split3)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -22
    for c in ([row.expand(M, N)] if batch == 1 else [row.expand(batch, M, N), row.expand(M, N).contiguous().expand(batch, M, N)]):
        out = gemm(a, b, c=c, beta=2.0, split3=split3)
        assert ((out - full).abs() <= eps * full.abs() + eps).all()
    from dion_b200 import ops

    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("batch,rows,r", [(1, 40, 128), (12, 3072, 96), (4, 2056, 512), (3, 5000, 200), (1, 4096, 130),
                                          (2, 776, 8), (40, 160, 96), (48, 776, 520)])
def test_gram_of_tall_factors_sums_k_ranges_over_a_cluster(batch, rows, r):
    """P^T P with few tiles and long K: the CTAs of a cluster take K ranges (2, 4 or 8 of them, some of them empty) and
    add their partial tiles; the last shape has enough tiles for CTA pairs instead.  The tensor core's accumulator drops
    up to 2^-23 of its value with every multiply (8 rows each); splitting the operands and adding parts costs below 2^-21."""
    x = torch.randn(batch, rows, r, device="cuda") + 0.25
    pitch = (r + 3) // 4 * 4
    buf = torch.zeros(batch, rows, pitch, device="cuda")
    buf[..., :r] = x
    p = buf[..., :r]
    out = torch.full((batch, r, r), float("nan"), device="cuda")
    gemm(p.transpose(-1, -2), p, out=out, symmetric=True, split3=True)
    ref = x.double().transpose(-1, -2) @ x.double()
    assert ((out.double() - ref).abs().amax() / ref.abs().amax()).item() < rows / 8 * 2 ** -23 + 2 ** -21
    # 128 x 128 blocks off the diagonal are mirrored (on it the two cross terms are added in either order)
    for i in range(0, r, 128):
        assert torch.equal(out[:, i:i + 128, i + 128:], out[:, i + 128:, i:i + 128].transpose(-1, -2))
    # every K sum in one pass: the same bits from CTA pairs and from single tiles
    p2 = gemm(p.transpose(-1, -2), p, symmetric=True, split3=True, pair=2)
    assert torch.equal(p2, gemm(p.transpose(-1, -2), p, symmetric=True, split3=True, pair=-1, block_n=128))
    again = gemm(p.transpose(-1, -2), p, symmetric=True, split3=True)
    assert torch.equal(out, again)


@pytest.mark.gpu
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("shape,symmetric", [((384, 200, 328), False), ((512, 512, 1000), False), ((256, 256, 520), True)])
def test_gemm_hi_lo_operands_reach_fp32_accuracy_in_one_launch(ta, tb, shape, symmetric):
    """A product of split operands (three K-segments into one accumulator) against fp64: a single tf32
    pass is about 1e-3 off, the three-segment product is close to fp32 rounding."""
    M, N, K = shape
    B = 3
    if symmetric:
        if ta != tb:
            pytest.skip("a symmetric product multiplies an operand with its own transpose")
        x = _operand(M, K, torch.float32, ta, batch=B)
        a, b = x, x.transpose(-1, -2)
    else:
        a = _operand(M, K, torch.float32, ta, batch=B)
        b = _operand(K, N, torch.float32, tb, batch=B)

    def split_like(t):  # halves with the memory layout of t
        base = t.transpose(-1, -2) if t.stride(-1) != 1 else t
        hi, lo = _split(base)
        return (hi.transpose(-1, -2), lo.transpose(-1, -2)) if t.stride(-1) != 1 else (hi, lo)

    a_hi, a_lo = split_like(a)
    b_hi, b_lo = split_like(b)
    ref = a.double() @ b.double()
    one = gemm(a_hi, b_hi, symmetric=symmetric)
    three = gemm(a_hi, b_hi, a_lo=a_lo, b_lo=b_lo, symmetric=symmetric)
    e1, e3 = _rel_err(one, ref), _rel_err(three, ref)
    assert e3 < 2e-5, (e1, e3)
    assert e1 > 10 * e3, (e1, e3)  # the segments really were added
    if symmetric:
        # mirrored tiles are exact copies; inside a diagonal tile the two cross terms of an element and of its
        # mirror image are added in opposite order, which may differ in the last bit
        torch.testing.assert_close(three, three.transpose(-1, -2), rtol=0, atol=2e-6 * ref.abs().max().item())


@pytest.mark.gpu
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_column_scale_on_the_addend(out_dtype):
    B, M, N, K = 2, 300, 200, 96
    a = torch.randn(B, M, K, device="cuda")
    b = torch.randn(B, K, N, device="cuda") * 0.05
    c = torch.randn(B, M, N, device="cuda")
    s = torch.rand(B, N, device="cuda") + 0.5
    out = gemm(a, b, c=c, alpha=-1.0, beta=1.0, c_col_scale=s, out_dtype=out_dtype)
    ref = c * s.unsqueeze(1) - a @ b
    assert _rel_err(out, ref) < (2e-2 if out_dtype == torch.bfloat16 else 3e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,k,batch", [(1024, 1024, 2), (768, 3072, 6), (520, 1032, 5), (512, 2048, 3)])
def test_gemm_symmetric_long_k_on_cta_pairs_with_staged_mirror(dtype, n, k, batch):
    """Symmetric products with K >= 1024 take 256 x 256 tiles on CTA pairs; off-diagonal tiles are stored a
    second time transposed, through shared memory.  The result must be exactly symmetric and match the
    plain product, also with an addend (b A + c A A) and ragged edges."""
    x = torch.randn(batch, n, k, device="cuda").to(dtype) * 0.05
    out = gemm(x, x.transpose(1, 2), symmetric=True)
    ref = x.float() @ x.float().transpose(1, 2)
    tol = 2e-2 if dtype == torch.bfloat16 else 3e-3
    assert _rel_err(out, ref) < tol
    assert torch.equal(out, out.transpose(1, 2))
    a = out.clone()
    if n * 4 % 16 == 0 and a.shape[-1] >= 1024:
        poly = gemm(a, a.transpose(1, 2), c=a, alpha=0.5, beta=-1.5, symmetric=True)
        ref2 = 0.5 * a.float() @ a.float().transpose(1, 2) - 1.5 * a.float()
        assert _rel_err(poly, ref2) < tol
        assert torch.equal(poly, poly.transpose(1, 2))


@pytest.mark.gpu
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("shape,symmetric", [((384, 200, 328), False), ((512, 512, 1000), False), ((200, 64, 72), False),
                                             ((256, 256, 520), True), ((768, 768, 768), True)])
def test_gemm_split3_splits_fp32_operands_in_shared_memory(ta, tb, shape, symmetric):
    """3xTF32 product of plain fp32 operands: the kernel forms the tf32 halves of every tile itself.
    Against fp64, and against the product of operands that were split beforehand."""
    M, N, K = shape
    B = 3
    if symmetric:
        if ta != tb:
            pytest.skip("a symmetric product multiplies an operand with its own transpose")
        x = _operand(M, K, torch.float32, ta, batch=B)
        a, b = x, x.transpose(-1, -2)
    else:
        a = _operand(M, K, torch.float32, ta, batch=B)
        b = _operand(K, N, torch.float32, tb, batch=B)
    ref = a.double() @ b.double()
    one = gemm(a, b, symmetric=symmetric)
    three = gemm(a, b, symmetric=symmetric, split3=True)
    e1, e3 = _rel_err(one, ref), _rel_err(three, ref)
    assert e3 < 2e-5 and e1 > 10 * e3, (e1, e3)
    # epilogue options ride along: addend with column scale, alpha / beta, strided views as operands
    c = torch.randn(B, M, N, device="cuda")
    s = torch.rand(B, N, device="cuda") + 0.5
    if not symmetric:
        out = gemm(a, b, c=c, alpha=-1.0, beta=1.0, c_col_scale=s, split3=True)
        assert _rel_err(out, c.double() * s.unsqueeze(1).double() - ref) < 2e-5
        big = torch.randn(B, M + 40, K + 24, device="cuda")
        av = big[:, 8:8 + M, 16:16 + K]
        out = gemm(av, b, split3=True)
        assert _rel_err(out, av.double() @ b.double()) < 2e-5
    from dion_b200 import ops

    ops.check_status()


def _plan(a, b, d, c=None, **kw):
    from dion_b200.ops import _ext

    if not _ext.load(required=False):
        pytest.skip("extension not built")
    return list(torch.ops.dion_b200.gemm_plan(a, b, c, d, **kw))


def _shapes(B, M, N, K, dtype=torch.bfloat16, out=None, a_mn=False, b_mn=True):
    """Operands and result of a product, for their sizes and layouts alone (host memory that nothing touches)."""
    lead = (B,) if B else ()
    a = torch.empty(*lead, K, M, dtype=dtype).mT if a_mn else torch.empty(*lead, M, K, dtype=dtype)
    b = torch.empty(*lead, K, N, dtype=dtype) if b_mn else torch.empty(*lead, N, K, dtype=dtype).mT
    return a, b, torch.empty(*lead, M, N, dtype=out or dtype)


def test_sums_in_order_forbid_the_sharing_of_k_and_nothing_else():
    """pair=2: the tiling is the one the kernel takes by itself, for every kind of product; only a K range that CTAs of a
    cluster would share is summed by one of them."""
    for block_n in (0, 64, 128, 256):
        for B, M, N, K in [(0, 512, 768, 768), (0, 8192, 768, 768), (0, 24, 96, 3072), (0, 8192, 3072, 4096), (12, 768, 3072, 768)]:
            for dtype in (torch.bfloat16, torch.float32):
                t = _shapes(B, M, N, K, dtype)
                assert _plan(*t, block_n=block_n, pair=2) == _plan(*t, block_n=block_n), (B, M, N, K, block_n)
    p = torch.empty(4, 14336, 512)
    g = torch.empty(4, 512, 512)
    shared = _plan(p.mT, p, g, symmetric=True, split3=True)
    in_order = _plan(p.mT, p, g, symmetric=True, split3=True, pair=2)
    assert in_order[2] == 1 and (shared[2] > 1 or shared[1] == 1)
    p, g = torch.empty(12, 3072, 96), torch.empty(12, 96, 96)
    assert _plan(p.mT, p, g, symmetric=True, split3=True)[2] > 1
    assert _plan(p.mT, p, g, symmetric=True, split3=True, pair=2)[2] == 1


def test_short_k_takes_pairs_only_where_c_and_d_move_by_tma():
    """K from 512 to 1023: pairs pay behind the TMA epilogue and lose behind the generic one, whatever keeps a product from
    the former; from K = 1024 on both take them."""
    M, N, f32 = 50176, 1000, torch.float32
    a, b, d = _shapes(0, M, N, 768)
    assert _plan(a, b, d) == [256, 1, 1, 1] and _plan(a, b, d, torch.empty_like(d), beta=1.0) == [256, 1, 1, 1]
    generic = [(a, b, torch.empty(M, N + 3, dtype=d.dtype)[:, :N], None),               # pitch no multiple of 16 bytes
               (a, b, torch.empty(M, N, dtype=f32), None),                              # results of another type
               (a, b, d, torch.empty(M, N, dtype=f32)),                                 # addend of another type
               (a, b, d, torch.empty(1, N, dtype=d.dtype).expand(M, N)),                # addend with broadcast rows
               (*_shapes(0, M, N + 4, 768), None),                                      # rows that end inside 16 bytes
               (*_shapes(0, M, N, 768, a_mn=True), None)]
    for x, y, out, c in generic:
        assert _plan(x, y, out, c, beta=1.0)[1::2] == [0, 0], (out.shape, out.stride(), out.dtype)
    for x, y, out, c in [(*_shapes(0, M, N + 4, 1024), None), (*_shapes(0, M, N, 1024, a_mn=True), None)]:
        assert _plan(x, y, out, c)[1::2] == [1, 0]


def test_gather_plan_takes_row_blocks_of_128_at_short_k():
    """The all-gather variant stores with the generic epilogue: at K = 768 it is not paired, and row blocks that are a
    multiple of 128 but not of 256 are taken."""
    _plan(*_shapes(0, 64, 64, 64))
    plan = list(torch.ops.dion_b200.gemm_gather_plan(8 * 7808, 768, 768, 7808, 8, 3))
    assert plan and plan[0] == 128 and plan[2] == 0


@pytest.mark.parametrize("B,n,k,tall,pair", [(48, 768, 768, False, 1), (48, 768, 768, True, 1), (24, 768, 768, True, 1),
                                             (8, 1024, 768, False, 0), (8, 1024, 768, True, 0), (8, 520, 1000, False, 0),
                                             (8, 520, 1000, True, 0), (30, 512, 600, False, 1), (30, 512, 600, True, 0),
                                             (48, 512, 500, False, 0), (12, 768, 3072, True, 1), (1, 768, 3072, False, 0)])
def test_symmetric_products_with_short_k_take_pairs_for_fewer_waves(B, n, k, tall, pair):
    """K from 512 to 1023: pairs where their waves are few enough, which depends on the epilogue (X^T X has the generic one)."""
    x = torch.empty(B, n, k, dtype=torch.bfloat16) if not tall else torch.empty(B, k, n, dtype=torch.bfloat16).mT
    plan = _plan(x, x.mT, torch.empty(B, n, n, dtype=torch.bfloat16), symmetric=True)
    assert plan == [256 if pair else 128, pair, 1, 0 if tall else 1]
    # results of another type are not stored by TMA: pairs from K = 1024 on
    plan = _plan(x, x.mT, torch.empty(B, n, n), symmetric=True)
    assert plan[1] == (pair if k >= 1024 else 0) and plan[3] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("B,n,k", [(24, 768, 768), (40, 520, 600), (16, 512, 512)])
def test_symmetric_products_of_tall_matrices_with_short_k(B, n, k):
    """X^T X (MN-major operands, generic mirrored epilogue) on CTA pairs and on single tiles: the same bits, symmetric, within
    the rounding of the bf16 result."""
    x = torch.randn(B, k, n, device="cuda").bfloat16()
    got = gemm(x.mT, x, symmetric=True)
    assert torch.equal(got, gemm(x.mT, x, symmetric=True, pair=-1)) and torch.equal(got, got.mT)
    want = x.double().mT @ x.double()
    assert ((got.double() - want).norm() / want.norm()).item() < 2.0 ** -8


_LAYOUTS = {  # out, addend (or None) for an M x N product, B of them where the first is 3-D
    "slices of wider rows": lambda z, r: (z(256, 3, 256).transpose(0, 1), None),
    "slices of wider rows, addend too": lambda z, r: (z(256, 3, 256).transpose(0, 1), r(256, 3, 256).transpose(0, 1)),
    "slices with a gap": lambda z, r: (z(200, 3, 272)[:, :, :264].transpose(0, 1), None),
    "one row, odd pitch": lambda z, r: (torch.as_strided(z(512), (1, 256), (257, 1)), torch.as_strided(r(512), (1, 256), (259, 1))),
    "one row, pitch 1": lambda z, r: (torch.as_strided(z(512), (1, 256), (1, 1)), None),
    "one row each, odd pitch": lambda z, r: (torch.as_strided(z(1024), (2, 1, 256), (256, 257, 1)), None),
    "addend of one row": lambda z, r: (z(256, 256), r(256).expand(256, 256)),
    "addend of one matrix": lambda z, r: (z(3, 256, 256), r(256, 256).expand(3, 256, 256)),
    "batch of one, odd stride": lambda z, r: (torch.as_strided(z(65536), (1, 256, 256), (7, 256, 1)),
                                             torch.as_strided(r(65536), (1, 256, 256), (9, 256, 1))),
    "addend beside the result": lambda z, r: (lambda buf: (buf[:, :256], buf[:, 512:768]))(r(256, 1024)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout", list(_LAYOUTS))
def test_results_and_addends_in_any_layout(layout, dtype):
    """Batch strides below the row pitch, single rows of any pitch, broadcast addends, result and addend in one buffer: the
    epilogue that the layout selects stores what it should and nothing else."""
    out, c = _LAYOUTS[layout](lambda *s: torch.zeros(*s, device="cuda", dtype=dtype),
                              lambda *s: torch.randn(*s, device="cuda").to(dtype))
    lead, (M, N), K = out.shape[:-2], out.shape[-2:], 128
    a, b = torch.randn(*lead, M, K, device="cuda").to(dtype), torch.randn(*lead, K, N, device="cuda").to(dtype)
    want = a.double() @ b.double() + (0.0 if c is None else c.double())
    base = out if out._base is None else out._base
    before = base.clone()
    gemm(a, b, c=c, beta=0.0 if c is None else 1.0, out=out)
    # one rounding of the result to bf16 (2^-9), tf32 operands with 10 bits of mantissa
    assert ((out.double() - want).norm() / want.norm()).item() < 2.0 ** -8
    out.copy_(torch.as_strided(before, out.shape, out.stride(), out.storage_offset()))
    assert torch.equal(base, before)


@pytest.mark.gpu
def test_two_streams_at_a_time_give_the_bits_of_one():
    """Clusters that share K, split pairs, the TMA epilogue with mirrored boxes, the Cholesky inverse and the launch sequence
    of Newton-Schulz issued on two streams at once, each with inputs of its own: the kernels keep nothing between calls and
    what one stream holds on an SM never blocks the other for good."""
    from dion_b200.optim.newton_schulz import newton_schulz

    def inputs(seed):
        g = torch.Generator("cuda").manual_seed(seed)
        r = lambda *s: torch.randn(*s, generator=g, device="cuda")
        return r(12, 3072, 96), r(6, 768, 768), r(24, 768, 768).bfloat16(), r(2, 333, 330).bfloat16()

    def work(p, f, x, odd):
        G = gemm(p.mT, p, symmetric=True, split3=True)
        return [G, ops.linalg.chol_inverse(G)[0], gemm(f, f, split3=True), gemm(x, x.mT, symmetric=True),
                gemm(x, x, c=x, beta=1.0), newton_schulz(x), newton_schulz(odd)]

    sets = [inputs(1), inputs(2)]
    want = [work(*s) for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    got = [[], []]
    for _ in range(4):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(work(*sets[i]))
    torch.cuda.synchronize()
    for i in range(2):
        for outs in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(outs, want[i]))
    ops.check_status()


_F32_OUT = [
    (128, 256, 64, 1, 1),        # one tile
    (300, 260, 200, 1, 2),       # rows and columns that fill no box, batches
    (129, 132, 1000, 3, 1),      # parts of unequal length
    (768, 768, 4096, 4, 1),      # pairs
    (1000, 516, 2056, 2, 1),
    (384, 384, 16384, 17, 1),    # 17 parts of 16 blocks for 256 blocks: the last one is empty
    (256, 128, 1024, 7, 2),      # 6 parts of 3 blocks would do for 16
    (256, 250, 512, 2, 1),       # rows of 1000 bytes: the generic epilogue
]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,split_k,batch,ta,mode", [
    (*shape, ta, mode) for shape in _F32_OUT for ta in ((False, True) if shape[0] % 8 == 0 else (False,))  # rows of A^T: 16 bytes
    for mode in (("store", "relu2", "add", "slice") if shape[3] == 1 else ("add",))])  # parts are added
def test_fp32_results_of_bf16_operands_by_tma(M, N, K, split_k, batch, ta, mode):
    """Stored or added to D by the copy engine.  Products of bf16 are exact in fp32 and the sums run in fp32: against fp64
    K * 2^-24 of the largest partial sum bounds the error; 1e-5 of the result's largest value lies above that here."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    lead = (batch,) if batch > 1 else ()
    n_pad = (N + 7) // 8 * 8
    a = torch.randn(*lead, *((K, M) if ta else (M, K)), device="cuda", generator=g).bfloat16()
    b = torch.randn(*lead, K, n_pad, device="cuda", generator=g).bfloat16()[..., :N]
    a = a.transpose(-1, -2) if ta else a
    want = a.double() @ b.double()
    if mode == "add":
        out = torch.randn(*lead, M, N, device="cuda", generator=g)
        want = out.double() + 0.5 * want
        gemm(a, b, out=out, alpha=0.5, accumulate=True, split_k=split_k)
    elif mode == "slice":
        whole = torch.full((*lead, M, N + 24), 7.0, device="cuda")
        out = whole[..., 8:8 + N]
        gemm(a, b, out=out)
        assert (whole[..., :8] == 7).all() and (whole[..., 8 + N:] == 7).all()
    else:
        out = torch.empty(*lead, M, N, device="cuda")
        gemm(a, b, out=out, act=None if mode == "store" else "relu2")
        want = want if mode == "store" else want.clamp_min(0).square()
    assert (out.double() - want).abs().max().item() <= 1e-5 * want.abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("B,M,N,K", [(1, 128, 256, 64), (3, 131, 260, 96), (33, 256, 132, 40), (40, 96, 768, 200), (2, 520, 1000, 64),
                                     (2, 300, 64, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("copies", [False, True])
def test_updates_in_place_through_maps_of_their_own(B, M, N, K, dtype, copies):
    """More matrices than one launch has maps for, sizes that fill no box, bf16 copies whose rows are not 16 bytes wide, an
    address TMA cannot take, beta = 0 over NaN: the bits of the path with staged loads and stores."""
    g = torch.Generator(device="cuda").manual_seed(B + M + N + K)
    P, R = (torch.randn(B, n, K, device="cuda", generator=g).to(dtype) for n in (M, N))
    start = torch.randn(B, M, N, device="cuda", generator=g)

    def run(host, beta, shift=0):
        X = [torch.empty(M * N + 4, device="cuda")[shift:shift + M * N].view(M, N).copy_(x if beta else float("nan") * x)
             for x in start]
        S = [torch.zeros(M, N, device="cuda", dtype=torch.bfloat16) for _ in X]
        addresses = [x.data_ptr() for x in X]
        ptrs = torch.tensor(addresses, device="cuda")
        kw = dict(shadow=S[0], shadow_ptrs=torch.tensor([s.data_ptr() for s in S], device="cuda")) if copies else {}
        gemm(P, R.transpose(1, 2), c=X[0], out=X[0], c_ptrs=ptrs, out_ptrs=ptrs, alpha=-0.3, beta=beta,
             host_ptrs=addresses if host else None, **kw)
        return X + (S if copies else [])

    for beta, shift in ((0.9, 0), (0.0, 0), (0.9, 1)):
        if shift and (N * 4) % 16 == 0:
            shift = 4  # still aligned: other addresses than the first time
        for a, b in zip(run(True, beta, shift), run(False, beta, shift)):
            assert torch.equal(a, b) and a.isfinite().all()
    want = 0.9 * start.double() - 0.3 * (P.double() @ R.double().transpose(1, 2))
    bound = 1e-5 if dtype == torch.bfloat16 else 2.0 ** -9  # tf32 operands: 10 bits
    for a, w in zip(run(True, 0.9), want):
        assert (a.double() - w).abs().max().item() <= bound * w.abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("N,maps", [(128, False), (508, False), (512, True), (768, True)])
def test_matrices_below_512_kb_are_updated_without_maps(N, maps, monkeypatch):
    """Where a tensor map per matrix costs the host more than it saves; 256 x N, the limit lies at N = 512.  Operands in tf32: 10 bits."""
    from dion_b200 import ops
    from dion_b200.optim.functional import foreach_baddbmm_

    X = [torch.randn(256, N, device="cuda") for _ in range(3)]
    A, B = torch.randn(3, 256, 32, device="cuda"), torch.randn(3, N, 32, device="cuda")
    want = [0.9 * x.double() - 0.3 * (a.double() @ b.double().t()) for x, a, b in zip(X, A, B)]
    seen, plain = [], ops.gemm
    monkeypatch.setattr(ops, "gemm", lambda *args, **kw: (seen.append(kw.get("host_ptrs")), plain(*args, **kw))[1])
    foreach_baddbmm_(X, A, B, alpha=-0.3, beta=0.9)
    assert seen == [[x.data_ptr() for x in X] if maps else None]
    for x, w in zip(X, want):
        assert (x.double() - w).abs().max().item() <= 2.0 ** -9 * w.abs().max().item()


@pytest.mark.gpu
@pytest.mark.parametrize("B,launches", [(1, 1), (32, 1), (33, 2), (70, 3)])
def test_updates_of_more_matrices_than_a_launch_has_maps_are_counted(B, launches):
    from dion_b200 import ops
    from dion_b200.optim.functional import foreach_baddbmm_

    X = list(torch.zeros(B, 256, 512, device="cuda").unbind())
    A, P = torch.randn(B, 256, 16, device="cuda"), torch.randn(B, 512, 16, device="cuda")
    before = ops.launch_count()
    foreach_baddbmm_(X, A, P)
    assert ops.launch_count() - before == launches
    # tf32 operands: 10 bits
    assert all((x - a @ p.t()).abs().max() <= 2.0 ** -9 * x.abs().max() for x, a, p in zip(X, A, P))


@pytest.mark.gpu
def test_first_call_of_a_thread():
    """A thread that has made no CUDA call yet, as a backward pass may meet it, starts with a product or with attention."""
    import threading

    from dion_b200.ops import runtime

    a, b = (torch.randn(256, 256, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(1, 128, 2, 64, device="cuda").bfloat16()
    lse, status = torch.empty(1, 2, 128, device="cuda"), runtime.status_tensor(a.device)
    outs, errors = [torch.empty_like(a), torch.empty_like(q)], []

    def run(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 - handed to the test's thread
            errors.append(e)

    torch.cuda.synchronize()
    for f in (lambda: gemm(a, b, out=outs[0]),
              lambda: torch.ops.dion_b200.attn_fwd(q, q, q, outs[1], lse, 0.125, status)):
        t = threading.Thread(target=run, args=(f,))
        t.start()
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    assert torch.equal(outs[0], gemm(a, b, out=torch.empty_like(a)))
    assert outs[1].isfinite().all()
