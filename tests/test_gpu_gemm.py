"""tcgen05 GEMM against an fp32 PyTorch reference, for every operand-major combination used by the dense towers."""
import pytest
import torch

import recis_b200

pytestmark = pytest.mark.gpu
C = recis_b200.native()
DEV = "cuda:0"


def _ref(a, b, bias, relu, a_mn, b_mn):
    A = (a.t() if a_mn else a).float()
    B = (b.t() if b_mn else b).float()
    y = A @ B.t()
    if bias is not None:
        y = y + bias.float()
    return torch.relu(y) if relu else y


@pytest.mark.parametrize("shape", [(128, 128, 64), (256, 128, 128), (300, 200, 72), (8192, 512, 16), (1000, 1024, 480), (77, 8, 8)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_matches_fp32(shape, a_mn, b_mn):
    M, N, K = shape
    torch.manual_seed(M + N + K)
    a = (torch.randn(K, M) if a_mn else torch.randn(M, K)).to(DEV, torch.bfloat16)
    b = (torch.randn(K, N) if b_mn else torch.randn(N, K)).to(DEV, torch.bfloat16)
    if (a.shape[1] % 8) or (b.shape[1] % 8):
        pytest.skip("row pitch must be a multiple of 16 bytes for TMA")
    bias = torch.randn(N, device=DEV)
    for relu, out_fp32 in ((False, True), (True, False)):
        y = C.gemm_bf16(a, b, bias, relu, a_mn, b_mn, out_fp32, None)
        ref = _ref(a, b, bias, relu, a_mn, b_mn)
        tol = 2e-2 if not out_fp32 else 2e-3
        err = (y.float() - ref).abs().max().item() / max(ref.abs().max().item(), 1.0)
        assert err < tol, (shape, a_mn, b_mn, relu, err)
        # relative Frobenius norm: bf16 output rounding is 2^-9 per entry, fp32 output only carries accumulation order
        fro = ((y.float() - ref).norm() / ref.norm().clamp_min(1e-6)).item()
        assert fro < (4e-3 if not out_fp32 else 1e-4), (shape, a_mn, b_mn, relu, fro)
    assert C.dense_status(DEV) == 0


def test_gemm_accumulate():
    torch.manual_seed(0)
    a = torch.randn(256, 64, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(128, 64, device=DEV, dtype=torch.bfloat16)
    acc = torch.randn(256, 128, device=DEV)
    ref = acc + a.float() @ b.float().t()
    out = C.gemm_bf16(a, b, None, False, False, False, True, acc)
    assert out.data_ptr() == acc.data_ptr()
    assert torch.allclose(out, ref, atol=1e-2, rtol=1e-3)


@pytest.mark.parametrize("M,N,K,masked", [(8192, 1024, 512, True), (1000, 264, 520, True), (300, 64, 128, False), (8192, 512, 1024, True), (77, 8, 24, True)])
def test_dgrad_with_relu_mask_and_bias_gradient_in_the_epilogue(M, N, K, masked):
    """dx = (dy W) masked by the ReLU of the layer below, and its column sums, from one GEMM: against fp32 matmul + mask + sum,
    on shapes that take the one-CTA kernel and shapes that take the pair kernel."""
    C = recis_b200.native()
    g = torch.Generator().manual_seed(M + N + K)
    dy = torch.randn(M, N, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) * 0.1).to(torch.bfloat16)
    y_below = torch.randn(M, K, generator=g).to(torch.bfloat16)
    dx, db = C.gemm_dgrad_fused(dy.to(DEV), w.to(DEV), y_below.to(DEV) if masked else None)
    ref = dy.float() @ w.float()
    if masked:
        ref = ref * (y_below.float() > 0).float()
    rel = lambda a, b: float((a.float().cpu() - b).norm() / b.norm().clamp(min=1e-12))
    assert dx.dtype == torch.bfloat16 and rel(dx, ref) < 6e-3
    if masked:
        assert float(dx.float().cpu()[(y_below.float() <= 0)].abs().max()) == 0.0       # masked entries are exact zeros
    assert rel(db, ref.sum(0)) < 2e-3
    assert C.dense_status(DEV) == 0


@pytest.mark.parametrize("M,N,K", [(19001, 264, 72), (20480, 2312, 64), (9500, 520, 1000), (4700, 72, 264), (1100, 136, 200)])
@pytest.mark.parametrize("odd", [False, True])
def test_gemm_epilogues_over_several_rounds_of_tiles(M, N, K, odd):
    """Bias + ReLU, residual and mask + column sums where a pair of SMs walks several tiles (ten column tiles included) and where one
    CTA has one tile, with rows and columns that end inside a box. ``odd``: a bias off its 8-byte line, a residual and a mask off their
    16-byte lines, which the bindings copy to one. Bounds: bf16 rounding 2^-9 per entry of bf16 outputs, accumulation order in fp32 ones (as above)."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, w = rn(M, K).bfloat16(), (rn(N, K) * 0.1).bfloat16()
    bias = rn(N + 1)[1:] if odd else rn(N)
    res = rn(M * N + 1)[1:].view(M, N) if odd else rn(M, N)
    mask = rn(M, N + 1).bfloat16()[:, :N] if odd else rn(M, N).bfloat16()
    mask[0, 0], mask[M - 1, N - 1], mask[1, 0] = float("nan"), float("inf"), -0.0
    ref = x.float() @ w.float().t()
    rel = lambda a, b: float((a.float() - b).norm() / b.norm())
    assert rel(C.gemm_bf16(x, w, bias, True, False, False, False, None), torch.relu(ref + bias)) < 4e-3
    assert rel(C.gemm_bf16_residual(x, w, bias, res), ref + bias + res) < 1e-4
    dx, db = C.gemm_dgrad_fused(x, w.t().contiguous(), mask)
    keep = (mask > 0).float()
    assert rel(dx, ref * keep) < 4e-3 and float(dx[keep == 0].float().abs().max()) == 0.0
    assert rel(db, (ref * keep).sum(0)) < 1e-4
    assert C.dense_status(DEV) == 0


@pytest.mark.parametrize("N,K,M", [(1280, 1280, 16392), (1024, 1024, 8200), (2304, 768, 20000), (256, 512, 40008), (2048, 3200, 4104), (200, 264, 65544)])
def test_split_reductions_in_parts_of_any_length(N, K, M):
    """dW = dy^T x over many rows, cut into parts that fill whole rounds of SMs, with a last part that is shorter or empty, added to the output:
    against fp64 on the same bf16 values; sums of M products in fp32 in any order: 1e-5 by norm."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    dy, x = (torch.randn(M, n, generator=g, device=DEV).bfloat16() for n in (N, K))
    out = C.gemm_bf16(dy, x, None, False, True, True, True, None)
    ref = sum(a.double().t() @ b.double() for a, b in zip(dy.split(8192), x.split(8192)))
    assert float((out.double() - ref).norm() / ref.norm()) < 1e-5
    C.gemm_bf16(dy, x, None, False, True, True, True, out)                 # on top of itself
    assert float((out.double() - 2 * ref).norm() / (2 * ref).norm()) < 1e-5
    assert C.dense_status(DEV) == 0


@pytest.mark.parametrize("M,N,K", [(8191, 256, 256), (8192, 192, 64), (8200, 256, 72), (9001, 200, 264)])
def test_column_sums_of_one_column_tile(M, N, K):
    """Column sums on both sides of the rows from which a pair of SMs adds them up over its tiles; bounds as for the masked shapes above."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    dy, w = torch.randn(M, K, generator=g, device=DEV).bfloat16(), (torch.randn(K, N, generator=g, device=DEV) * 0.1).bfloat16()
    y = torch.randn(M, N, generator=g, device=DEV).bfloat16()
    dx, db = C.gemm_dgrad_fused(dy, w, y)
    ref = (dy.double() @ w.double()) * (y > 0)
    assert float((dx.double() - ref).norm() / ref.norm()) < 4e-3 and float((db.double() - ref.sum(0)).norm() / ref.sum(0).norm()) < 1e-4
    assert C.dense_status(DEV) == 0


@pytest.mark.parametrize("M,N,K", [(333, 201, 72), (20001, 203, 264), (1000, 1030, 128)])
def test_epilogues_of_outputs_that_no_map_takes(M, N, K):
    """Residual, mask and column sums of outputs whose rows start off a 16-byte line: read and written row by row. Bounds as above."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, w, bias, res, mask = rn(M, K).bfloat16(), (rn(N, K) * 0.1).bfloat16(), rn(N), rn(M, N), rn(M, N).bfloat16()
    wt = torch.zeros(K, (N + 7) // 8 * 8, device=DEV).bfloat16()
    wt[:, :N] = w.t()
    ref = x.double() @ w.double().t()
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    assert rel(C.gemm_bf16_residual(x, w, bias, res), ref + bias + res) < 1e-4
    dx, db = C.gemm_dgrad_fused(x, wt[:, :N], mask)
    ref = ref * (mask > 0)
    assert rel(dx, ref) < 4e-3 and rel(db, ref.sum(0)) < 1e-4 and torch.count_nonzero(dx[mask <= 0]) == 0
    assert C.dense_status(DEV) == 0
