"""Dense-tower kernels (tcgen05 Linear, interactions) against fp32 PyTorch references."""
import pytest
import torch

import recis_b200
from recis_b200.ops import dense as D

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ref_dot(x, cube):
    B, Fn, Dm = cube.shape
    z = torch.cat([x.unsqueeze(1), cube], dim=1)
    zz = torch.bmm(z, z.transpose(1, 2))
    li, lj = torch.tril_indices(Fn + 1, Fn + 1, offset=-1)
    return torch.cat([x, zz[:, li, lj]], dim=1)


@pytest.mark.parametrize("B,F,Dm", [(64, 26, 128), (130, 26, 64), (5, 31, 128), (33, 3, 16), (8, 1, 8)])
def test_dot_interaction_fwd_bwd(B, F, Dm):
    torch.manual_seed(0)
    x = torch.randn(B, Dm).to(torch.bfloat16)
    cube = torch.randn(B, F, Dm)
    xr = x.float().requires_grad_(True); cr = cube.clone().requires_grad_(True)
    ref = _ref_dot(xr, cr)
    xg = x.to(DEV).requires_grad_(True); cg = cube.to(DEV).requires_grad_(True)
    out = D.dot_interaction(xg, cg)
    n = ref.shape[1]
    assert out.shape[1] % 8 == 0 and out.shape[1] >= n
    got = out[:, :n].detach().float().cpu()
    assert torch.allclose(got, ref.detach(), atol=0.15, rtol=2e-2)
    # relative norm: a dropped 16-column k-block of the D = 128 reduction would cost about 1/8 of every entry's terms
    assert float((got - ref.detach()).norm() / ref.detach().norm()) < 1e-2
    assert float(out[:, n:].detach().abs().sum()) == 0
    go = torch.randn(B, out.shape[1]).to(torch.bfloat16)
    out.backward(go.to(DEV))
    ref.backward(go[:, :n].float())
    assert torch.allclose(cg.grad.cpu(), cr.grad, atol=0.1, rtol=2e-2)
    assert torch.allclose(xg.grad.float().cpu(), xr.grad, atol=0.3, rtol=3e-2)
    assert float((cg.grad.cpu() - cr.grad).norm() / cr.grad.norm()) < 1e-2
    assert float((xg.grad.float().cpu() - xr.grad).norm() / xr.grad.norm()) < 1.5e-2


def test_fm_interaction():
    torch.manual_seed(0)
    for shape in [(50, 7, 16), (1000, 39, 16), (33, 5, 12), (17, 3, 128), (9, 4, 7)]:
        cube = torch.randn(*shape)
        cr = cube.clone().requires_grad_(True)
        ref = D.fm_interaction(cr)
        cg = cube.to(DEV).requires_grad_(True)
        out = D.fm_interaction(cg)
        assert torch.allclose(out.cpu(), ref, atol=2e-4, rtol=1e-4), shape
        g = torch.randn(shape[0], 1)
        ref.backward(g); out.backward(g.to(DEV))
        assert torch.allclose(cg.grad.cpu(), cr.grad, atol=1e-4, rtol=1e-4), shape


def _torch_bf16_mlp(mlp, x):
    """The same network with plain PyTorch ops and the same rounding points (bf16 operands/activations, fp32 accumulation)."""
    import torch.nn.functional as F
    params = []
    h = x.to(torch.bfloat16)
    n = len(mlp.layers)
    for i, layer in enumerate(mlp.layers):
        w = layer.weight.detach().clone().requires_grad_(True)
        b = layer.bias.detach().clone().requires_grad_(True)
        params += [w, b]
        h = (F.linear(h.float(), w.to(torch.bfloat16).float()) + b)
        if layer.act:
            h = torch.relu(h)
        h = h.to(torch.bfloat16)
    return h, params


@pytest.mark.parametrize("dims", [(13, 512, 256, 128), (480, 1024, 1024, 512, 256, 1), (16, 8)])
def test_mlp_matches_reference(dims):
    torch.manual_seed(0)
    M = 1000
    mlp = D.MLP(list(dims), final_act=False).to(DEV)
    x = torch.randn(M, dims[0], device=DEV)
    y = mlp(x)
    yr, ref_params = _torch_bf16_mlp(mlp, x)
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-12))
    assert y.shape == yr.shape
    assert rel(y, yr) < 1e-2
    # and against a pure fp32 network (no bf16 anywhere): loose, it only guards against gross errors
    ref32 = D.MLP(list(dims), final_act=False, dtype=torch.float32).to(DEV)
    ref32.load_state_dict(mlp.state_dict())
    assert rel(y, ref32(x)) < 5e-2
    go = torch.randn(M, dims[-1], device=DEV).to(torch.bfloat16)
    y.backward(go)
    yr.backward(go)
    for (name, p), r in zip(mlp.named_parameters(), ref_params):
        assert rel(p.grad, r.grad) < 3e-2, (name, rel(p.grad, r.grad))
    assert recis_b200.native().dense_status(DEV) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("decoupled", [False, True])
def test_dense_adam_matches_torch(decoupled):
    """Native multi-tensor Adam/AdamW against torch.optim on the same gradients (30 tensors: two launches, odd sizes)."""
    from recis_b200.optim import DenseAdam
    torch.manual_seed(0)
    shapes = [(37,), (128, 65), (3,), (1024, 16)] * 7 + [(5, 5), (1,)]
    ours = [torch.randn(s, device="cuda").requires_grad_() for s in shapes]
    ref = [p.detach().clone().requires_grad_() for p in ours]
    wd = 0.01
    o1 = DenseAdam(ours, lr=1e-2, weight_decay=wd, decoupled=decoupled)
    o2 = (torch.optim.AdamW if decoupled else torch.optim.Adam)(ref, lr=1e-2, weight_decay=wd)
    for _ in range(5):
        for a, b in zip(ours, ref):
            g = torch.randn_like(a)
            a.grad = g.clone()
            b.grad = g.clone()
        o1.step()
        o2.step()
    for a, b in zip(ours, ref):
        torch.testing.assert_close(a, b, rtol=2e-5, atol=2e-6)


@pytest.mark.gpu
def test_adamw_tf_native_matches_cpu_foreach():
    from recis_b200.optim import AdamWTF
    torch.manual_seed(1)
    shapes = [(33, 7), (256,), (2, 3, 5)]
    cpu = [torch.randn(s).requires_grad_() for s in shapes]
    gpu = [p.detach().cuda().requires_grad_() for p in cpu]
    o1, o2 = AdamWTF(cpu, lr=1e-2, weight_decay=0.02), AdamWTF(gpu, lr=1e-2, weight_decay=0.02)
    for _ in range(4):
        for a, b in zip(cpu, gpu):
            g = torch.randn_like(a)
            a.grad = g.clone()
            b.grad = g.cuda()
        o1.step()
        o2.step()
    for a, b in zip(cpu, gpu):
        torch.testing.assert_close(a, b.cpu(), rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("rows,hidden,out_bf16", [(1000, 256, True), (333, 64, False), (77, 1024, True), (4097, 36, False), (5, 512, False)])
def test_layer_norm_kernels_match_fp32_reference(rows, hidden, out_bf16):
    """Forward (bf16 or fp32 output) and the one-pass backward (input gradient and both weight gradients) against torch's
    layer norm in fp32 on the CPU."""
    from recis_b200.ops.dense import LayerNorm
    g = torch.Generator().manual_seed(rows + hidden)
    x = torch.randn(rows, hidden, generator=g) * 2 + 0.5
    go = torch.randn(rows, hidden, generator=g)
    ref = torch.nn.LayerNorm(hidden)
    with torch.no_grad():
        ref.weight.copy_(torch.randn(hidden, generator=g) * 0.5 + 1)
        ref.bias.copy_(torch.randn(hidden, generator=g) * 0.1)
    ours = LayerNorm(hidden).to(DEV)
    ours.load_state_dict(ref.state_dict())
    xr = x.clone().requires_grad_(True)
    yr = ref(xr)
    yr.backward(go)
    xo = x.to(DEV).requires_grad_(True)
    yo = ours(xo, out_bf16=out_bf16)
    assert yo.dtype == (torch.bfloat16 if out_bf16 else torch.float32)
    yo.backward(go.to(DEV).to(yo.dtype))
    rel = lambda a, b: float((a.float().cpu() - b).norm() / b.norm().clamp(min=1e-12))
    tol = 6e-3 if out_bf16 else 2e-5           # bf16 output and bf16 upstream gradient round at 2^-9
    assert rel(yo.detach(), yr.detach()) < tol
    assert rel(xo.grad, xr.grad) < tol
    assert rel(ours.weight.grad, ref.weight.grad) < tol
    assert rel(ours.bias.grad, ref.bias.grad) < tol


@pytest.mark.parametrize("M,N,relu", [(5000, 256, True), (777, 1024, True), (4096, 768, False), (100, 8, True), (300, 64, True), (64, 24, True)])
def test_relu_backward_with_bias_gradient_all_widths(M, N, relu):
    """Widths served by the 16-byte kernel (powers of two below 256, multiples of 256) and one that falls back (24)."""
    C = recis_b200.native()
    g = torch.Generator().manual_seed(M + N)
    y = torch.randn(M, N, generator=g).to(torch.bfloat16)
    dout = torch.randn(M, N, generator=g).to(torch.bfloat16)
    dy, db = C.relu_bwd_bias(y.to(DEV), dout.to(DEV), relu)
    want = dout.float() * ((y.float() > 0).float() if relu else 1.0)
    assert torch.equal(dy.cpu().float(), want.to(torch.bfloat16).float())
    ref_db = want.to(torch.bfloat16).float().sum(0)
    assert float((db.cpu() - ref_db).norm() / ref_db.norm().clamp(min=1e-6)) < 1e-5


def test_linear_with_residual_in_the_epilogue_matches_fp32_reference():
    from recis_b200.ops.dense import Linear
    g = torch.Generator().manual_seed(3)
    M, K, N = 1000, 256, 256
    lin = Linear(K, N).to(DEV)
    x = torch.randn(M, K, generator=g)
    res = torch.randn(M, N, generator=g)
    go = torch.randn(M, N, generator=g)
    xo = x.to(DEV).to(torch.bfloat16).requires_grad_(True)
    ro = res.to(DEV).requires_grad_(True)
    out = lin.forward_residual(xo, ro)
    assert out.dtype == torch.float32
    out.backward(go.to(DEV))
    xb = x.to(torch.bfloat16).float().requires_grad_(True)
    rr = res.clone().requires_grad_(True)
    W, b = lin.weight.detach().cpu().to(torch.bfloat16).float().requires_grad_(True), lin.bias.detach().cpu().clone().requires_grad_(True)
    ref = rr + xb @ W.t() + b
    ref.backward(go)
    rel = lambda a, b_: float((a.float().cpu() - b_).norm() / b_.norm().clamp(min=1e-12))
    assert rel(out.detach(), ref.detach()) < 1e-5
    assert torch.equal(ro.grad.cpu(), go)
    assert rel(xo.grad, xb.grad) < 8e-3 and rel(lin.weight.grad, W.grad) < 8e-3 and rel(lin.bias.grad, b.grad) < 8e-3


def test_bf16_weight_copies_follow_the_optimizer_and_any_other_change():
    """The forward pass keeps a bf16 copy (padded to multiples of 8) of every weight; the native dense optimizer rewrites it
    together with the weight (no cast in the next forward), and a change made through torch invalidates it."""
    from recis_b200.optim import DenseAdam
    torch.manual_seed(0)
    mlp = D.MLP([64, 128, 24, 1]).to(DEV)
    opt = DenseAdam(mlp.parameters(), lr=1e-2)
    x = torch.randn(256, 64, device=DEV)
    C = recis_b200.native()
    for step in range(3):
        before = C.launch_count()
        loss = mlp(x)[:, :1].float().square().mean()
        launches_fwd = C.launch_count() - before
        opt.zero_grad()
        loss.backward()
        opt.step()
        for layer in mlp.layers:
            sh = D.bf16_shadow(layer.weight)
            N, K = layer.weight.shape
            assert sh is not None and sh.shape == ((N + 7) // 8 * 8, (K + 7) // 8 * 8)
            assert torch.equal(sh[:N, :K], layer.weight.detach().to(torch.bfloat16))            # rewritten by the optimizer
            assert float(sh[N:].abs().sum()) == 0.0 and float(sh[:, K:].abs().sum()) == 0.0     # the padding stays zero
        if step == 0:
            first = launches_fwd
        else:
            assert launches_fwd == first - 3          # no layer casts its weight any more
    with torch.no_grad():
        mlp.layers[0].weight.mul_(0.5)
    assert D.bf16_shadow(mlp.layers[0].weight) is None
    ref = torch.relu(torch.relu(x.to(torch.bfloat16).float() @ mlp.layers[0].weight.detach().to(torch.bfloat16).float().t() + mlp.layers[0].bias))
    out = mlp.layers[0](x.to(torch.bfloat16)).float()
    assert float((out - ref).norm() / ref.norm()) < 1e-2


@pytest.mark.parametrize("B,Nd,F,D,w", [(1, 1, 2, 8, 4), (5, 13, 26, 16, 4), (37, 3, 7, 32, 1), (1024, 13, 39, 16, 4), (9, 0, 3, 4, 2), (2500, 5, 2, 64, 4),
                                        (17, 2, 3, 128, 4)])
def test_fm_head_matches_tensor_ops(B, Nd, F, D, w):
    """The fused DeepFM head against the same computation with tensor ops in 64 bits, forward and backward. The tower input is bf16
    (2^-9 relative); everything else is fp32 over at most (Nd + F) * D products resp. B samples: 1e-5 of the sum of magnitudes."""
    from recis_b200.ops.dense import fm_head
    g = torch.Generator().manual_seed(B + D)
    dense = torch.randn(B, Nd, generator=g)
    leaves = [torch.randn(Nd, D, generator=g), torch.randn(Nd, generator=g), torch.randn(B, F, D, generator=g), torch.randn(B, F, w, generator=g)]
    g_lin = torch.randn(B, 1, generator=g)
    g_deep = torch.randn(B, (Nd + F) * D, generator=g).to(torch.bfloat16)
    gpu = [t.to("cuda").requires_grad_() for t in leaves]
    deep, lin = fm_head(dense.to("cuda"), *gpu)
    pad = deep.shape[1] - (Nd + F) * D
    assert deep.dtype == torch.bfloat16 and deep.shape[1] % 8 == 0 and torch.count_nonzero(deep[:, deep.shape[1] - pad:]) == 0
    torch.autograd.backward([deep, lin], [torch.nn.functional.pad(g_deep, (0, pad)).to("cuda"), g_lin.to("cuda")])
    ref = [t.double().requires_grad_() for t in leaves]
    cube = torch.cat([dense.double().unsqueeze(-1) * ref[0].unsqueeze(0), ref[2]], dim=1)
    s = cube.sum(1)
    lin_r = (dense.double() * ref[1]).sum(1, keepdim=True) + ref[3][:, :, 0].sum(1, keepdim=True) + 0.5 * (s * s - (cube * cube).sum(1)).sum(1, keepdim=True)
    torch.autograd.backward([cube.reshape(B, -1), lin_r], [g_deep.double(), g_lin.double()])
    assert torch.allclose(deep[:, :(Nd + F) * D].double().cpu(), cube.reshape(B, -1), rtol=2 ** -8, atol=1e-6)
    mag = float((cube.abs().sum(1) ** 2).sum(1).max()) + 1
    assert (lin.double().cpu() - lin_r).abs().max() < 1e-5 * mag
    for a, b in zip(gpu, ref):
        if a.numel():
            assert (a.grad.double().cpu() - b.grad).abs().max() < 1e-5 * (float(b.grad.abs().max()) * max(B, Nd + F) ** 0.5 + mag ** 0.5), b.shape


@pytest.mark.parametrize("M,N", [(1, 8), (5, 64), (77, 256), (3000, 256), (4097, 768), (100, 24), (33, 512)])
def test_cast_with_column_sums(M, N):
    """fp32 -> bf16 with the column sums of the fp32 values, on widths inside and outside the vector kernel's range. Sums of M terms."""
    x = torch.randn(M, N, generator=torch.Generator().manual_seed(M)).cuda()
    y, db = recis_b200.native().cast_colsum(x)
    assert torch.equal(y, x.to(torch.bfloat16))
    inside = (N // 8) % 32 == 0 if N >= 256 else ((N // 8) & (N // 8 - 1)) == 0
    ref, mag = (x if inside else y.float()).double().sum(0), x.double().abs().sum(0)
    assert ((db.double() - ref).abs() <= (M + 1) * 2.0 ** -24 * mag).all()


@pytest.mark.parametrize("T,H,ffn", [(1, 64, 128), (300, 256, 1024), (1000, 128, 264)])
def test_pre_norm_block_matches_separate_functions(T, H, ffn):
    """LayerNorm with the residual gradient added in its backward, and the feed-forward block as one function, against the same layers
    as separate functions. Both round the same operands to bf16 (so the ReLU masks agree); what differs is that the bias gradients sum
    values before instead of after their rounding to bf16 (2^-9 each, independent) and the order of fp32 additions: 2^-8 of the norm."""
    torch.manual_seed(T)
    norm, l0, l1 = D.LayerNorm(H).cuda(), D.Linear(H, ffn, act=True).cuda(), D.Linear(ffn, H).cuda()
    torch.nn.init.normal_(norm.weight, 1.0, 0.1)
    x, go = torch.randn(T, H, device="cuda"), torch.randn(T, H, device="cuda")
    params = [norm.weight, norm.bias, l0.weight, l0.bias, l1.weight, l1.bias]
    a = x.clone().requires_grad_()
    h, r = norm.forward_split(a, out_bf16=True)
    out = D.ffn_residual(h, r, l0, l1)
    got = torch.autograd.grad(out, [a] + params, go)
    b = x.clone().requires_grad_()
    ref_out = l1.forward_residual(l0(norm(b, out_bf16=True)), b)
    ref = torch.autograd.grad(ref_out, [b] + params, go)
    assert torch.equal(out, ref_out)
    for p, q in zip(got, ref):
        assert (p - q).norm() <= 2.0 ** -8 * q.norm(), p.shape
    F = torch.nn.functional
    only_norm = torch.autograd.grad(norm.forward_split(a)[0], a, go)[0]
    only_res = torch.autograd.grad(norm.forward_split(a)[1], a, go)[0]
    assert torch.equal(only_res, go) and (only_norm - torch.autograd.grad(F.layer_norm(b, (H,), norm.weight, norm.bias, norm.eps), b, go)[0]).abs().max() < 1e-4


@pytest.mark.parametrize("M,dims", [(1, [8, 16, 8]), (37, [100, 64, 1]), (1000, [480, 512, 256, 1]), (300, [264, 200])])
def test_mlp_input_gradient_of_an_fp32_input(M, dims):
    """An fp32 input gets the GEMM's fp32 accumulator as its gradient, a bf16 input the same rounded to bf16 (2^-9 relative, zero padding
    cut off in both)."""
    torch.manual_seed(M)
    mlp = D.MLP(dims).cuda()
    x = torch.randn(M, dims[0], device="cuda").to(torch.bfloat16)
    a, b = x.float().requires_grad_(), x.clone().requires_grad_()
    go = torch.randn(M, dims[-1], device="cuda").to(torch.bfloat16)
    mlp(a).backward(go)
    mlp(b).backward(go)
    assert a.grad.dtype == torch.float32 and a.grad.shape == b.grad.shape == x.shape
    assert torch.equal(a.grad.to(torch.bfloat16), b.grad) and not torch.equal(a.grad, b.grad.float())


def _at(t, first):
    """The values of ``t`` as a contiguous view that starts ``first`` elements into a buffer."""
    buf = torch.empty(t.numel() + first, dtype=t.dtype, device=t.device)
    return buf[first:].copy_(t.reshape(-1)).view(t.shape)


@pytest.mark.parametrize("first", [1, 2, 3])
def test_vector_readers_take_views_at_any_element(first):
    """Contiguous inputs and gradients that do not start on a 16-byte line (autograd hands such views in, see the concatenation) give the
    bits of aligned ones: norm with and without the residual gradient, means and target attention over sequences, the DeepFM head. Weight
    gradients meet in atomics: fp32 sums of 37 terms in any order."""
    from recis_b200.ops.attention import segment_mean, target_attention
    torch.manual_seed(first)
    H, T = 64, 37
    offs = torch.tensor([0, 5, 5, T], dtype=torch.int32, device=DEV)
    x, q, go = torch.randn(T, H, device=DEV), torch.randn(3, H, device=DEV), torch.randn(3, H, device=DEV)
    gy, gr = torch.randn(T, H, device=DEV), torch.randn(T, H, device=DEV)
    w, b = torch.randn(H, device=DEV), torch.randn(H, device=DEV)
    cube, bias, num = torch.randn(T, 3, 8, device=DEV), torch.randn(T, 3, 4, device=DEV), torch.randn(T, 2, device=DEV)
    table, table_bias = torch.randn(2, 8, device=DEV), torch.randn(2, device=DEV)
    g_deep, g_lin = torch.randn(T, 40, device=DEV).to(torch.bfloat16), torch.randn(T, 1, device=DEV)

    def grads(place):
        p = lambda t: place(t).detach().requires_grad_()
        res = []
        for dtype in (torch.float32, torch.bfloat16):
            leaves = [p(x), p(w), p(b)]
            y, r = D._LayerNormSplitFn.apply(*leaves, 1e-5, dtype == torch.bfloat16)
            res += [y] + list(torch.autograd.grad([y, r], leaves, [place(gy.to(dtype)), place(gr)]))
        leaves = [p(x), p(w), p(b)]
        y = D._LayerNormFn.apply(*leaves, 1e-5, False)
        res += [y] + list(torch.autograd.grad(y, leaves, place(gy)))
        for fn, leaves in ((lambda a: segment_mean(a, offs), [p(x)]), (lambda a, c: target_attention(a, c, offs), [p(x), p(q)])):
            y = fn(*leaves)
            res += [y] + list(torch.autograd.grad(y, leaves, place(go)))
        leaves = [p(table), p(table_bias), p(cube), p(bias)]
        y = D._FMHeadFn.apply(place(num), *leaves)
        return res + list(y) + list(torch.autograd.grad(y, leaves, [place(g_deep), place(g_lin)]))

    for a, b_ in zip(grads(lambda t: _at(t, first)), grads(lambda t: t)):
        if a.dim() == 1 and a.numel() == H:
            assert torch.allclose(a, b_, rtol=1e-4, atol=1e-4)
        else:
            assert torch.equal(a, b_), tuple(a.shape)
    # the same through autograd: what stands in front of a concatenation is an odd number of elements
    norm, a = D.LayerNorm(H).to(DEV), x.clone().requires_grad_()
    y, r = norm.forward_split(a)
    (torch.cat([a.new_ones(first), r.reshape(-1), y.reshape(-1)]) * torch.arange(1., 1 + first + 2 * T * H, device=DEV)).sum().backward()
    assert torch.isfinite(a.grad).all()


@pytest.mark.parametrize("B", [1, 37, 1000, 4096, 4097, 20000])
@pytest.mark.parametrize("with_extra", [False, True])
def test_click_loss_matches_the_tensor_library(B, with_extra):
    """Loss, logit and gradients of the fused last step against slice + cast + BCEWithLogitsLoss on the same tower output, with a gradient
    of the logit too; fp32 sums of B terms in another order: 1e-5."""
    from recis_b200.ops.dense import MLP, click_loss
    torch.manual_seed(B)
    mlp = MLP([24, 16, 1], final_act=False).to(DEV)
    torch.nn.init.normal_(mlp.layers[-1].bias)
    loss_fn = torch.nn.BCEWithLogitsLoss()
    x = torch.randn(B, 24, device=DEV) * 4
    label = (torch.rand(B, 1, device=DEV) < 0.3).float()
    res = []
    for fused in (True, False):
        xi = x.clone().requires_grad_()
        extra = torch.linspace(-60, 60, B, device=DEV).view(B, 1).requires_grad_() if with_extra else None
        mlp.zero_grad()
        if fused:
            loss, logit = click_loss(mlp, xi, label, loss_fn, extra)
            assert "ClickLoss" in loss.grad_fn.name() and "ClickLogit" in logit.grad_fn.name()
        else:
            y = mlp(xi)
            assert y.shape == (B, 1)
            logit = y.float() if extra is None else extra + y.float()
            loss = loss_fn(logit, label)
        (3 * loss + 1e-3 * logit.sin().sum()).backward()
        res.append([loss.detach(), logit.detach(), xi.grad, *[p.grad for p in mlp.parameters()]] + ([extra.grad] if with_extra else []))
    assert res[0][0].shape == res[1][0].shape and torch.equal(res[0][1], res[1][1])
    assert abs(float(res[0][0] - res[1][0])) <= 1e-5 * abs(float(res[1][0]))
    for a, b in zip(res[0][2:], res[1][2:]):
        # the gradient of the tower's output is rounded to bf16 in both: a last-bit difference in front of it moves single entries by 2^-8
        assert float((a - b).norm()) <= 2e-3 * float(b.norm()) + 1e-9


def test_click_loss_has_the_logit_in_its_graph():
    from recis_b200.ops.dense import MLP, click_loss
    torch.manual_seed(3)
    mlp, loss_fn = MLP([8, 1], final_act=False).to(DEV), torch.nn.BCEWithLogitsLoss()
    x, label = torch.randn(37, 8, device=DEV), (torch.rand(37, 1, device=DEV) < 0.5).float()
    loss, logit = click_loss(mlp, x, label, loss_fn)
    ref = logit.detach().clone().requires_grad_()
    want, = torch.autograd.grad(loss_fn(ref, label), ref, create_graph=True)
    got, = torch.autograd.grad(loss, logit, retain_graph=True)
    torch.testing.assert_close(got, want.detach(), rtol=1e-5, atol=1e-8)
    twice, = torch.autograd.grad(torch.autograd.grad(loss, logit, create_graph=True)[0].sum(), logit, retain_graph=True)
    torch.testing.assert_close(twice, torch.autograd.grad(want.sum(), ref)[0], rtol=1e-5, atol=1e-8)
    logit.register_hook(lambda g: g * 0)
    loss /= 2                                                     # as when gradients of several steps are summed
    loss.backward()
    assert float(mlp.layers[0].weight.grad.abs().sum()) == 0


def test_click_loss_leaves_other_losses_and_hooks_alone():
    from recis_b200.ops.dense import MLP, click_loss
    mlp = MLP([8, 1], final_act=False).to(DEV)
    x, label = torch.randn(5, 8, device=DEV), torch.ones(5, 1, device=DEV)
    calls = []
    handle = mlp.register_forward_hook(lambda m, i, o: calls.append(o.shape))
    loss, _ = click_loss(mlp, x, label, torch.nn.BCEWithLogitsLoss())
    assert calls == [(5, 1)]
    handle.remove()
    for fn in (torch.nn.BCEWithLogitsLoss(reduction="sum"), torch.nn.BCEWithLogitsLoss(pos_weight=torch.tensor([2.0], device=DEV)), torch.nn.MSELoss()):
        got, logit = click_loss(mlp, x, label, fn)
        assert torch.equal(got, fn(logit, label))
    with pytest.raises(ValueError):
        click_loss(mlp, x, torch.ones(5, device=DEV), torch.nn.BCEWithLogitsLoss())


@pytest.mark.parametrize("dims", [(24, 35, 100, 5), (16, 1), (7, 300, 201, 3), (64, 188, 191, 12), (480, 1024, 256, 1)])
@pytest.mark.parametrize("M", [1, 333])
def test_mlp_with_biases_of_any_width(dims, M):
    """Biases as large as the sums, in layers of 8 n and of other widths on both sides of 192, against plain torch on the same bf16 values, column by
    column: a bias that is left out, shifted, or read past its end is off by the size of the output. Each layer rounds to bf16 (2^-9 of an entry),
    a hidden entry may round the other way (2^-8) and three layers add up: 1e-2. The columns of the padding are zeros."""
    torch.manual_seed(sum(dims) + M)
    mlp = D.MLP(list(dims), final_act=False).to(DEV)
    for layer in mlp.layers:
        torch.nn.init.normal_(layer.bias)
    x = torch.randn(M, dims[0], device=DEV)
    h = x.bfloat16().double()
    for layer in mlp.layers:
        h = h @ layer.weight.detach().bfloat16().double().t() + layer.bias.detach().double()
        h = (torch.relu(h) if layer.act else h).bfloat16().double()
    y = mlp.forward_padded(x)
    assert y.shape == (M, D._pad8(dims[-1])) and torch.count_nonzero(y[:, dims[-1]:]) == 0
    err = (y[:, :dims[-1]].double() - h).norm(dim=0) / h.norm(dim=0).clamp_min(0.1 * M ** 0.5)
    assert float(err.max()) < 1e-2, err
    y.backward(torch.ones_like(y))
    last = mlp.layers[-1].bias.grad
    assert torch.equal(last, torch.full_like(last, M)) and recis_b200.native().dense_status(DEV) == 0


@pytest.mark.parametrize("B", [1, 1000])
def test_click_logit_matches_plain_torch(B):
    """Logit and loss of a tower with biases against plain torch from its weights; the last layer's output is rounded to bf16: 2^-8 of it."""
    torch.manual_seed(B)
    mlp = D.MLP([24, 16, 1], final_act=False).to(DEV)
    for layer in mlp.layers:
        torch.nn.init.normal_(layer.bias, std=3.0)
    x, extra = torch.randn(B, 24, device=DEV), torch.randn(B, 1, device=DEV)
    label = (torch.rand(B, 1, device=DEV) < 0.3).float()
    h = x.bfloat16().double()
    for layer in mlp.layers:
        h = h @ layer.weight.detach().bfloat16().double().t() + layer.bias.detach().double()
        h = torch.relu(h).bfloat16().double() if layer.act else h
    loss, logit = D.click_loss(mlp, x, label, torch.nn.BCEWithLogitsLoss(), extra)
    assert float((logit.double() - extra.double() - h).abs().max()) <= 2 ** -7 * float(h.abs().max())
    want = torch.nn.functional.binary_cross_entropy_with_logits(logit.detach().double(), label.double())
    assert abs(float(loss.detach()) - float(want)) <= 1e-5 * float(want)
