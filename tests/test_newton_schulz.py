"""Newton-Schulz orthogonalisation: the tcgen05 path (symmetric X X^T tiles, fused b A + c A A and
a X + B X epilogues) against the plain PyTorch iteration of the same coefficients, as the reference
checks its Triton kernels against torch (tests/test_newton_shultz.py)."""
import pytest
import torch

from dion_b200.optim.newton_schulz import NS_COEFFS, newton_schulz, newton_schulz_torch


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def test_torch_iteration_orthogonalises_on_cpu():
    torch.manual_seed(0)
    for shape in [(48, 96), (96, 48), (3, 64, 64)]:
        X = newton_schulz_torch(torch.randn(shape)).float()
        m = min(shape[-2:])
        gram = X @ X.transpose(-1, -2) if shape[-2] <= shape[-1] else X.transpose(-1, -2) @ X
        # the quintic iteration drives singular values into a band around 1, not to 1 exactly
        assert (gram - torch.eye(m)).abs().max() < 0.45
    assert len(NS_COEFFS) == 5 and all(len(c) == 3 for c in NS_COEFFS)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(768, 768), (768, 3072), (3072, 768), (4, 256, 512), (3, 512, 256), (2, 200, 328)])
def test_kernel_matches_torch_iteration(shape):
    torch.manual_seed(1)
    G = torch.randn(shape, device="cuda")
    ours = newton_schulz(G)
    ref = newton_schulz_torch(G)
    assert ours.shape == G.shape and ours.dtype == torch.bfloat16
    # both run five bf16 iterations; rounding differs, the result agrees to bf16 accuracy
    assert _rel(ours, ref) < 3e-2
    # and it is an approximate orthogonal factor
    X = ours.float()
    small_first = shape[-2] <= shape[-1]
    gram = X @ X.transpose(-1, -2) if small_first else X.transpose(-1, -2) @ X
    eye = torch.eye(gram.shape[-1], device="cuda")
    assert (gram - eye).abs().max() < 0.5


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(333, 1001), (1001, 333), (2, 130, 64), (3, 64, 130), (7, 9), (1, 8), (2, 8, 1),
                                   (10, 9), (333, 330), (3, 1003, 1002), (1007, 1001), (64, 3, 2), (64, 2, 1),
                                   (16, 9, 10), (330, 333)])
def test_sides_that_are_no_multiple_of_eight_are_padded(shape):
    """Zero rows and columns stay zero in every product: the result is the iteration's, as close to its fp64 form as the
    same bf16 iteration on PyTorch's products is (whose roundings differ; small singular values amplify them)."""
    g = torch.randn(*shape, device="cuda").bfloat16()
    out = newton_schulz(g)
    assert out.shape == g.shape and out.is_contiguous() and out.dtype == torch.bfloat16
    assert not newton_schulz(g.clone().requires_grad_()).requires_grad

    def iterate(dtype):
        X = g.to(dtype)
        X = X.mT if g.size(-2) > g.size(-1) else X
        X = X / (X.norm(dim=(-2, -1), keepdim=True) + 1e-7)
        for a, b, c in NS_COEFFS:
            A = X @ X.mT
            X = a * X + (b * A + c * (A @ A)) @ X
        return X.mT if g.size(-2) > g.size(-1) else X

    ref = iterate(torch.float64)
    err = ((out.double() - ref).norm() / ref.norm()).item()
    lib = ((iterate(torch.bfloat16).double() - ref).norm() / ref.norm()).item()
    assert err < 1.5 * lib + 4e-3, (err, lib)  # one rounding of the result is 2^-9


@pytest.mark.gpu
@pytest.mark.parametrize("coeffs", [[(1.0, 2.0), (3.0, 4.0), (5.0, 6.0)], [(1.0, 2.0, 3.0, 4.0)] * 3])
def test_a_step_takes_three_coefficients(coeffs):
    with pytest.raises(ValueError):
        newton_schulz(torch.randn(16, 24, device="cuda"), coeffs=coeffs)
    with pytest.raises(ValueError):
        newton_schulz_torch(torch.randn(16, 24), coeffs=coeffs)


@pytest.mark.gpu
def test_muon_steps_a_slightly_tall_matrix():
    """Ten rows and nine columns: padded to sixteen columns the matrix is still multiplied from the right."""
    from dion_b200 import Muon

    p = torch.nn.Parameter(torch.randn(10, 9, device="cuda"))
    before = p.detach().clone()
    p.grad = torch.randn_like(p)
    Muon([dict(params=[p])], lr=0.02).step()
    assert torch.isfinite(p).all() and not torch.equal(p.detach(), before)


@pytest.mark.gpu
def test_kernel_handles_zero_and_tiny_inputs():
    Z = torch.zeros(2, 128, 256, device="cuda")
    out = newton_schulz(Z)
    assert torch.isfinite(out).all() and out.abs().max() == 0
    T = torch.randn(128, 256, device="cuda") * 1e-20
    assert torch.isfinite(newton_schulz(T)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(256, 256), (256, 1024), (200, 328)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_symmetric_gram_and_poly_match_torch(m, n, dtype):
    from dion_b200.optim.newton_schulz import ns_line_1, ns_line_2

    tol = 5e-2
    for batch in (None, 4):
        shape = (m, n) if batch is None else (batch, m, n)
        A = torch.randn(shape, dtype=dtype, device="cuda")
        got, want = ns_line_1(A), A @ A.mT
        assert got.dtype == dtype and got.shape == want.shape
        assert (got.float() - want.float()).abs().max() <= tol * want.float().abs().max()
        S = torch.randn(shape[:-1] + (m,), dtype=dtype, device="cuda")
        S = (S + S.mT) / 2
        alpha, beta = 0.7, -1.3
        got, want = ns_line_2(S, alpha, beta), alpha * (S @ S.mT) + beta * S
        assert (got.float() - want.float()).abs().max() <= tol * want.float().abs().max()


def test_symmetric_helpers_on_cpu():
    from dion_b200.optim.newton_schulz import ns_line_1, ns_line_2

    A = torch.randn(3, 16, 24)
    torch.testing.assert_close(ns_line_1(A), A @ A.mT)
    S = torch.randn(16, 16)
    S = S + S.T
    torch.testing.assert_close(ns_line_2(S, 0.5, 2.0), 0.5 * (S @ S.T) + 2.0 * S)


def _one_launch_per_product(g, coeffs, tall):
    """Scaling and products of ``newton_schulz``, each in a launch of its own; sides of a multiple of eight."""
    from dion_b200 import ops

    X = torch.empty_like(g)
    torch.ops.dion_b200.frob_scale(g, X, None, 1e-7)
    for a, b, c in coeffs:
        A = ops.gemm(X.mT, X, symmetric=True) if tall else ops.gemm(X, X.mT, symmetric=True)
        P = ops.gemm(A, A.mT, c=A, alpha=c, beta=b, symmetric=True)
        X = ops.gemm(X, P, c=X, beta=a) if tall else ops.gemm(P, X, c=X, beta=a)
    return X


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 2, 5])
@pytest.mark.parametrize("shape", [(1, 8, 8), (2, 8, 1024), (1, 72, 64), (5, 64, 72), (1, 128, 128), (3, 200, 264), (2, 264, 200),
                                   (1, 1003, 56), (12, 256, 512), (2, 511, 256), (13, 136, 128), (24, 128, 256), (25, 64, 256),
                                   (64, 128, 128), (65, 128, 128), (128, 64, 64), (129, 64, 64), (1, 256, 768)])
def test_small_matrices_take_one_launch_for_all_products(shape, steps):
    """Every number of CTAs per matrix, edges of the 128 x 64 tiles, both orientations, odd and even numbers of steps (the
    transposes change places), and sizes just beyond: the sums and roundings are those of single products."""
    from dion_b200.ops import runtime

    torch.manual_seed(sum(shape))
    g = torch.randn(*shape, device="cuda").bfloat16()
    tall = shape[1] > shape[2]
    before = runtime.launch_count()
    want = _one_launch_per_product(g, NS_COEFFS[:steps], tall)
    between = runtime.launch_count()
    out = newton_schulz(g, coeffs=NS_COEFFS[:steps])
    small = shape not in ((129, 64, 64), (1, 256, 768))
    assert runtime.launch_count() - between == between - before - (3 * steps - 1 if small else 0)
    assert torch.equal(out, want)
    runtime.check_status()


@pytest.mark.gpu
def test_small_matrices_under_capture_and_on_two_streams():
    gs = [torch.randn(3, 200, 264, device="cuda").bfloat16() for _ in range(2)]
    want = [newton_schulz(g) for g in gs]
    streams = [torch.cuda.Stream() for _ in gs]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(10):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(newton_schulz(gs[i]))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i]) for i in range(2) for o in got[i])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = newton_schulz(gs[0])
    gs[0].copy_(gs[1])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[1])
