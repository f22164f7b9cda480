"""Ragged (unpadded) self-attention on the tcgen05 kernels against a plain fp32 PyTorch computation of the same thing:
per sequence and head, ``softmax(q k^T / sqrt(d)) v`` on the bf16 inputs widened to fp32. Forward and backward."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _oracle(qkv, lens, H, d_out=None):
    """fp32 reference; returns (out [T, H*64], dqkv or None)."""
    x = qkv.float().detach().requires_grad_(d_out is not None)
    T = x.shape[0]
    hidden = H * 64
    outs, s0 = [], 0
    for L in lens:
        blk = x[s0:s0 + L]
        q, k, v = (blk[:, i * hidden:(i + 1) * hidden].view(L, H, 64).transpose(0, 1) for i in range(3))   # [H, L, 64]
        att = torch.softmax(q @ k.transpose(1, 2) / 8.0, dim=-1)
        outs.append((att @ v).transpose(0, 1).reshape(L, hidden))
        s0 += L
    out = torch.cat(outs) if outs else x.new_zeros(0, hidden)
    if d_out is None:
        return out, None
    out.backward(d_out.float())
    return out.detach(), x.grad


def _case(lens, H, seed=0):
    g = torch.Generator().manual_seed(seed)
    T = sum(lens)
    offs = torch.zeros(len(lens) + 1, dtype=torch.int32)
    offs[1:] = torch.tensor(lens).cumsum(0)
    qkv = (torch.randn(T, 3 * H * 64, generator=g) * 0.7).to(torch.bfloat16)
    d_out = (torch.randn(T, H * 64, generator=g) * 0.2).to(torch.bfloat16)
    return qkv, offs, d_out


CASES = [([5], 1), ([128], 1), ([129], 2), ([5, 128, 129, 300, 1], 4), ([1000, 50], 2), ([64] * 7, 1), ([257, 3, 511], 3)]


@pytest.mark.parametrize("lens,H", CASES)
def test_ragged_attention_forward_matches_fp32(lens, H):
    import recis_b200
    C = recis_b200.native()
    qkv, offs, _ = _case(lens, H)
    out, lse = C.ragged_attention_fwd(qkv.to(DEV), offs.to(DEV), H, max(lens), 0.125)
    torch.cuda.synchronize()
    assert C.dense_status("cuda:0") == 0
    ref, _ = _oracle(qkv, lens, H)
    got = out.float().cpu()
    assert got.shape == ref.shape
    err = (got - ref).norm() / ref.norm()
    assert err < 1e-2 and float((got - ref).abs().max()) < 3e-2, (float(err), float((got - ref).abs().max()))


@pytest.mark.parametrize("lens,H", CASES)
def test_ragged_attention_backward_matches_fp32(lens, H):
    import recis_b200
    C = recis_b200.native()
    qkv, offs, d_out = _case(lens, H, seed=1)
    q_dev, o_dev = qkv.to(DEV), offs.to(DEV)
    out, lse = C.ragged_attention_fwd(q_dev, o_dev, H, max(lens), 0.125)
    dqkv = C.ragged_attention_bwd(q_dev, out, d_out.to(DEV), lse, o_dev, H, max(lens), 0.125)
    torch.cuda.synchronize()
    assert C.dense_status("cuda:0") == 0
    _, ref = _oracle(qkv, lens, H, d_out)
    got = dqkv.float().cpu()
    hidden = H * 64
    for name, sl in (("dq", slice(0, hidden)), ("dk", slice(hidden, 2 * hidden)), ("dv", slice(2 * hidden, 3 * hidden))):
        a, b = got[:, sl], ref[:, sl]
        err = (a - b).norm() / b.norm().clamp_min(1e-6)
        assert err < 2e-2, (name, float(err))


def test_module_path_uses_the_kernels_and_matches_the_padded_path():
    """``ragged_self_attention`` (what the sequence model calls) on the kernels against the padded SDPA path in fp32."""
    import os
    from recis_b200.ops import attention
    lens, H = [40, 200, 7], 2
    qkv, offs, d_out = _case(lens, H, seed=2)
    a = qkv.to(DEV).requires_grad_(True)
    out = attention.ragged_self_attention(a, offs.to(DEV), H, max(lens))
    out.backward(d_out.to(DEV))
    prev = os.environ.get("RECIS_ATTENTION")
    os.environ["RECIS_ATTENTION"] = "padded"
    try:
        b = qkv.float().to(DEV).requires_grad_(True)
        ref = attention.ragged_self_attention(b, offs.to(DEV), H, max(lens))
        ref.backward(d_out.float().to(DEV))
    finally:
        if prev is None:
            os.environ.pop("RECIS_ATTENTION", None)
        else:
            os.environ["RECIS_ATTENTION"] = prev
    assert (out.float() - ref).norm() / ref.norm() < 1e-2
    assert (a.grad.float() - b.grad).norm() / b.grad.norm() < 2e-2


@pytest.mark.parametrize("lens,hidden", [([5, 1, 300], 256), ([0, 17, 1000, 0, 64], 64), ([33] * 40, 128), ([700, 2], 1024), ([9], 8)])
def test_target_attention_kernels_match_tensor_ops(lens, hidden):
    """One query per sequence over packed tokens, forward and backward, against the segment-reduction formulation in fp32."""
    import os
    from recis_b200.ops import attention
    g = torch.Generator().manual_seed(len(lens) + hidden)
    T, B = sum(lens), len(lens)
    offs = torch.zeros(B + 1, dtype=torch.int32)
    offs[1:] = torch.tensor(lens).cumsum(0)
    x = torch.randn(T, hidden, generator=g)
    q = torch.randn(B, hidden, generator=g)
    go = torch.randn(B, hidden, generator=g)
    a, b = x.to(DEV).requires_grad_(True), q.to(DEV).requires_grad_(True)
    out = attention.target_attention(a, b, offs.to(DEV))
    out.backward(go.to(DEV))
    os.environ["RECIS_TARGET_ATTENTION"] = "eager"
    try:
        c, d = x.clone().requires_grad_(True), q.clone().requires_grad_(True)
        ref = attention.target_attention(c, d, offs)
        ref.backward(go)
    finally:
        os.environ.pop("RECIS_TARGET_ATTENTION", None)
    assert torch.allclose(out.cpu(), ref, atol=2e-5, rtol=1e-4), float((out.cpu() - ref).abs().max())
    assert torch.allclose(a.grad.cpu(), c.grad, atol=5e-5, rtol=1e-3), float((a.grad.cpu() - c.grad).abs().max())
    assert torch.allclose(b.grad.cpu(), d.grad, atol=5e-5, rtol=1e-3), float((b.grad.cpu() - d.grad).abs().max())


@pytest.mark.parametrize("longest,n,H", [(1, 700, 1), (16, 300, 2), (64, 200, 3), (65, 150, 2), (128, 120, 5), (129, 100, 2), (260, 90, 2)])
def test_backward_over_many_items_isolates_sequences(longest, n, H):
    """More work items than the persistent grid holds at once, lengths over the whole range, tokens in front of and behind the
    sequences, and one sequence of non-finite values: the others' gradients match the fp32 oracle (bf16 rounding of P, dS and the
    results, 2^-9 each, against sums of up to 260 terms: 2e-2 as above) and uncovered tokens get exact zeros."""
    import recis_b200
    C = recis_b200.native()
    g = torch.Generator().manual_seed(longest)
    lens = torch.randint(0, longest + 1, (n,), generator=g).tolist()
    lens[n // 2], lens[n // 3] = longest, 1
    pre, post = 3, 5
    qkv, offs, d_out = _case([pre] + lens + [post], H, seed=3)
    offs = offs[1:-1].contiguous()
    bad = n // 2
    b0, b1 = int(offs[bad]), int(offs[bad + 1])
    q_dev, o_dev, d_dev = qkv.to(DEV), offs.to(DEV), d_out.to(DEV)
    q_dev[b0:b1] = float("nan")
    d_dev[b0:b1] = float("inf")
    out, lse = C.ragged_attention_fwd(q_dev, o_dev, H, max(lens), 0.125)
    got = C.ragged_attention_bwd(q_dev, out, d_dev, lse, o_dev, H, max(lens), 0.125).float().cpu()
    torch.cuda.synchronize()
    assert C.dense_status("cuda:0") == 0
    T = qkv.shape[0]
    _, ref = _oracle(qkv[pre:T - post], lens, H, d_out[pre:T - post])
    assert torch.count_nonzero(got[:pre]) == 0 and torch.count_nonzero(got[T - post:]) == 0
    keep = torch.ones(T, dtype=torch.bool)
    keep[:pre] = keep[T - post:] = keep[b0:b1] = False
    a, b = got[keep], ref[keep[pre:T - post]]
    assert torch.isfinite(a).all()
    for name, sl in (("dq", slice(0, H * 64)), ("dk", slice(H * 64, 2 * H * 64)), ("dv", slice(2 * H * 64, 3 * H * 64))):
        # one-token sequences have dq = dk = 0 exactly in theory: their error is measured against the scale of dv
        scale = b[:, sl].norm() if longest > 1 or name == "dv" else b[:, 2 * H * 64:].norm()
        assert (a[:, sl] - b[:, sl]).norm() / scale < 2e-2, name


@pytest.mark.parametrize("lens,hidden", [([0, 5, 0, 1000, 1], 256), ([3] * 500, 8), ([700], 1024), ([1, 2, 3], 12), ([0], 64)])
def test_segment_mean_matches_tensor_ops(lens, hidden):
    """Means over packed sequences, forward and backward, with tokens around the sequences; fp32 sums of up to 1000 terms against 64 bits."""
    from recis_b200.ops.attention import segment_mean
    g = torch.Generator().manual_seed(hidden)
    pre, post = 2, 3
    T = pre + sum(lens) + post
    offs = torch.tensor([pre] + lens).cumsum(0).to(torch.int32)
    x, go = torch.randn(T, hidden, generator=g), torch.randn(len(lens), hidden, generator=g)
    a = x.to(DEV).requires_grad_()
    out = segment_mean(a, offs.to(DEV))
    out.backward(go.to(DEV))
    b = x.double().requires_grad_()
    ref = torch.stack([b[offs[i]:offs[i + 1]].sum(0) / max(n, 1) for i, n in enumerate(lens)])
    ref.backward(go.double())
    assert (out.double().cpu() - ref).abs().max() < 1e-5
    assert torch.allclose(a.grad.double().cpu(), b.grad, rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("lens,bound", [([5, 0, 33, 128], 128), ([1, 16, 17, 64, 65], 65), ([300, 7], 300), ([200, 128, 31], 100)])
def test_forward_writes_every_row(lens, bound):
    """The output memory is not cleared beforehand: tokens outside the sequences, and those past the tiles that the length bound asks for,
    read as zeros; all others match the oracle at the edges of the 16-key steps and 32-column quarters."""
    import recis_b200
    C = recis_b200.native()
    H, pre, post = 2, 3, 4
    qkv, offs, _ = _case([pre] + lens + [post], H, seed=5)
    offs = offs[1:-1].contiguous()
    T = qkv.shape[0]
    poison = [torch.full((T, H * 64), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    del poison
    out, lse = C.ragged_attention_fwd(qkv.to(DEV), offs.to(DEV), H, bound, 0.125)
    assert C.dense_status("cuda:0") == 0
    got, lse = out.float().cpu(), lse.cpu()
    ref = _oracle(qkv[pre:T - post], lens, H)[0]
    computed = torch.zeros(T, dtype=torch.bool)
    for i, n in enumerate(lens):
        computed[int(offs[i]):int(offs[i]) + min(n, (bound + 127) // 128 * 128)] = True
    assert torch.count_nonzero(got[~computed]) == 0 and torch.count_nonzero(lse[~computed]) == 0
    a, b = got[computed], ref[computed[pre:T - post]]
    assert (a - b).norm() / b.norm() < 1e-2 and (a - b).abs().max() < 3e-2 and torch.isfinite(lse).all()


@pytest.mark.parametrize("hinted", [False, True])
@pytest.mark.parametrize("lens,hidden,pre", [([1024, 1025], 64, 0), ([513, 1025, 511], 256, 0), ([1536], 128, 512), ([0, 5000, 0, 3, 4096, 0], 256, 7), ([1025] * 5, 1024, 511),
                                             ([2, 1030, 506, 2000], 4, 0), ([1], 8, 3000)])
def test_segment_mean_of_long_sequences(lens, hidden, pre, hinted):
    """Sequences on both sides of the length from which they are taken in pieces, starting and ending at and beside the pieces' edges, with
    tokens around them and a bound that holds or is too small. fp32 sums of up to 5000 terms in pieces, against 64 bits."""
    from recis_b200.ops.attention import segment_mean
    g = torch.Generator().manual_seed(hidden)
    T = pre + sum(lens) + 5
    offs = torch.tensor([pre] + lens).cumsum(0).to(torch.int32)
    x, go = torch.randn(T, hidden, generator=g), torch.randn(len(lens), hidden, generator=g)
    a = x.to(DEV).requires_grad_()
    out = segment_mean(a, offs.to(DEV), max_len=1000 if hinted else None)
    out.backward(go.to(DEV))
    b = x.double().requires_grad_()
    ref = torch.stack([b[offs[i]:offs[i + 1]].sum(0) / max(n, 1) for i, n in enumerate(lens)])
    ref.backward(go.double())
    assert (out.double().cpu() - ref).abs().max() < 1e-5
    assert torch.allclose(a.grad.double().cpu(), b.grad, rtol=1e-6, atol=1e-9)
    again = segment_mean(a, offs.to(DEV))
    assert torch.equal(again, segment_mean(a, offs.to(DEV)))


@pytest.mark.parametrize("lens,bound,H", [([200, 128, 31], 100, 2), ([5, 300, 129, 0, 700], 64, 3), ([129], 1, 1), ([700, 90, 257, 300, 256], 200, 2),
                                          ([1000, 3], 129, 1), ([130, 400] * 200, 128, 2)])
def test_backward_of_sequences_longer_than_the_bound(lens, bound, H):
    """The forward computes the queries in the bound's tiles of 128 over all keys and leaves zeros for the rest, so only those queries
    contribute to the gradients, to every key, and the others' own gradient is zero; the outputs' gradients there do not count, however
    large. Against the fp32 oracle with the same rows taken out; rounding as above."""
    import recis_b200
    C = recis_b200.native()
    qkv, offs, d_out = _case(lens, H, seed=7)
    T, hidden = qkv.shape[0], H * 64
    computed = torch.zeros(T, dtype=torch.bool)
    for i, n in enumerate(lens):
        computed[int(offs[i]):int(offs[i]) + min(n, (bound + 127) // 128 * 128)] = True
    _, ref = _oracle(qkv, lens, H, torch.where(computed[:, None], d_out, torch.zeros_like(d_out)))
    q_dev, o_dev = qkv.to(DEV), offs.to(DEV)
    out, lse = C.ragged_attention_fwd(q_dev, o_dev, H, bound, 0.125)
    got = C.ragged_attention_bwd(q_dev, out, torch.where(computed[:, None], d_out, d_out * 1e4).to(DEV), lse, o_dev, H, bound, 0.125)
    torch.cuda.synchronize()
    assert C.dense_status("cuda:0") == 0
    got = got.float().cpu()
    assert torch.count_nonzero(got[~computed][:, :hidden]) == 0 and torch.isfinite(got).all()
    for name, sl in (("dq", slice(0, hidden)), ("dk", slice(hidden, 2 * hidden)), ("dv", slice(2 * hidden, 3 * hidden))):
        assert (got[:, sl] - ref[:, sl]).norm() / ref[:, sl].norm() < 2e-2, name


@pytest.mark.parametrize("lens,H", [([1] * 900 + [64, 65, 33, 128, 129, 191, 193], 3), ([700, 31, 1000, 257, 96, 97], 2), ([64, 65, 127, 192, 16, 17] * 70, 5),
                                    ([90] * 200, 4)])
@pytest.mark.parametrize("spread", [1.0, 40.0])
def test_forward_on_every_work_split_and_with_growing_scores(lens, H, spread):
    """Items dealt out one per CTA and fetched from the counter, one and several at a time, and key counts on both sides of a step and of a
    32-column chunk. With ``spread`` the scores of a row reach hundreds and grow along the sequence, so that every step raises the reference
    exponent. The rows behind the last sequence are non-finite and must not reach anything. Bounds as above."""
    import recis_b200
    C = recis_b200.native()
    qkv, offs, _ = _case(lens, H, seed=len(lens))
    if spread > 1:
        pos = torch.cat([torch.arange(L) / max(L, 2) for L in lens])
        k = slice(H * 64, 2 * H * 64)
        qkv[:, k] = (qkv[:, k].float() * (1 + spread * pos[:, None])).to(torch.bfloat16)
    tail = torch.full((7, 3 * H * 64), float("nan")).to(torch.bfloat16)
    for bound in (max(lens), 4 * max(lens)):
        out, lse = C.ragged_attention_fwd(torch.cat([qkv, tail]).to(DEV), offs.to(DEV), H, bound, 0.125)
        assert C.dense_status("cuda:0") == 0
        ref, _ = _oracle(qkv, lens, H)
        got = out.float().cpu()
        assert float(got[len(qkv):].abs().max()) == 0.0 and float(lse[len(qkv):].abs().max()) == 0.0
        err = (got[:len(qkv)] - ref).norm() / ref.norm()
        assert err < 1e-2, (bound, float(err))


@pytest.mark.parametrize("repeat,H,bound", [(40, 8, 128), (100, 8, 60), (470, 8, 128)])
@pytest.mark.parametrize("spread", [1.0, 20.0])
def test_outputs_of_a_sequence_do_not_depend_on_its_batch(repeat, H, bound, spread):
    """Short sequences by the thousand (up to several items per fetch), with some longer than the bound among them: output and log-sum-exp are
    those of the same sequences in a batch of their own, to the bit, and of every length within the bounds above."""
    import recis_b200
    C = recis_b200.native()
    some = [1, 16, 17, 63, 64, 65, 96, 127, 128, 300]
    qkv, offs, _ = _case(some, H, seed=repeat)
    if spread > 1:
        pos = torch.cat([torch.arange(L) / max(L, 2) for L in some])
        k = slice(H * 64, 2 * H * 64)
        qkv[:, k] = (qkv[:, k].float() * (1 + spread * pos[:, None])).to(torch.bfloat16)
    T = sum(some)
    out, lse = C.ragged_attention_fwd(qkv.to(DEV), offs.to(DEV), H, bound, 0.125)
    all_offs = torch.cat([offs[:-1] + i * T for i in range(repeat)] + [torch.tensor([repeat * T], dtype=torch.int32)])
    many, many_lse = C.ragged_attention_fwd(qkv.to(DEV).repeat(repeat, 1), all_offs.to(DEV), H, bound, 0.125)
    assert C.dense_status("cuda:0") == 0
    assert torch.equal(many.view(repeat, T, -1), out.expand(repeat, T, -1)) and torch.equal(many_lse.view(repeat, T, -1), lse.expand(repeat, T, -1))
    ref, _ = _oracle(qkv, some, H)
    got = out.float().cpu()
    for s0, L in zip(offs.tolist(), some):
        n = min(L, 128)                                               # queries in the bound's one tile
        assert (got[s0:s0 + n] - ref[s0:s0 + n]).norm() / ref[s0:s0 + n].norm() < 1e-2, L
        assert torch.count_nonzero(got[s0 + n:s0 + L]) == 0


@pytest.mark.parametrize("lens,H", [([5], 1), ([100], 4), ([64, 1, 128] * 20, 4), ([300, 17], 8), ([1000, 400, 30, 999], 4), ([129, 0, 256] * 40, 2)])
def test_forward_does_not_depend_on_the_bound(lens, H):
    """The bound and the lengths decide which kernel runs and how work items are dealt out or fetched, on both sides of one, three and eight rounds
    of them, and nothing else."""
    import recis_b200
    C = recis_b200.native()
    qkv, offs, _ = _case(lens, H, seed=11)
    a = C.ragged_attention_fwd(qkv.to(DEV), offs.to(DEV), H, max(lens), 0.125)
    for factor in (2, 3, 5, 9, 16, 33, 150):
        b = C.ragged_attention_fwd(qkv.to(DEV), offs.to(DEV), H, factor * max(lens), 0.125)
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]), factor
    assert C.dense_status("cuda:0") == 0
    ref, _ = _oracle(qkv, [n for n in lens if n], H)
    assert (a[0].float().cpu() - ref).norm() / ref.norm() < 1e-2


@pytest.mark.parametrize("lens,H", [([191, 193], 1), ([193, 193], 1), ([128] * 111, 4), ([128] * 112, 4), ([1] * 888, 1), ([1] * 889, 1), ([0, 0, 90, 0], 3)])
def test_forward_on_both_sides_of_a_cta_per_item(lens, H):
    """Batches on both sides of the rule for small ones, with tokens in front of and behind the sequences: rows of every sequence against the
    fp32 computation, rows of none as zeros. Bounds as above."""
    import recis_b200
    C = recis_b200.native()
    qkv, offs, _ = _case(lens, H, seed=12)
    pad = torch.full((3, 3 * H * 64), float("nan")).to(torch.bfloat16)
    out, lse = C.ragged_attention_fwd(torch.cat([pad, qkv, pad]).to(DEV), (offs + 3).to(DEV), H, max(lens), 0.125)
    assert C.dense_status("cuda:0") == 0
    got = out.float().cpu()
    for rows in (slice(0, 3), slice(3 + len(qkv), None)):
        assert torch.count_nonzero(got[rows]) == 0 and torch.count_nonzero(lse[rows]) == 0
    ref, _ = _oracle(qkv, [n for n in lens if n], H)
    assert (got[3:3 + len(qkv)] - ref).norm() / ref.norm() < 1e-2


@pytest.mark.parametrize("bound", [2**31 - 128, 2**31 - 1, 2**33])
def test_bounds_at_the_end_of_32_bits(bound):
    """A bound that says "any length": the row numbers behind its last tile do not fit in 32 bits. Outputs and gradients are those of the tight one."""
    import recis_b200
    C = recis_b200.native()
    lens, H = [200, 3, 128], 2
    qkv, offs, d_out = (t.to(DEV) for t in _case(lens, H, seed=13))
    want = C.ragged_attention_fwd(qkv, offs, H, 256, 0.125)
    got = C.ragged_attention_fwd(qkv, offs, H, bound, 0.125)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
    a, b = (C.ragged_attention_bwd(qkv, got[0], d_out, got[1], offs, H, n, 0.125) for n in (256, bound))
    assert (a.float() - b.float()).norm() <= 1e-2 * a.float().norm() and C.dense_status("cuda:0") == 0
