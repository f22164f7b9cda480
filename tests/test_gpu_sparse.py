"""GPU tests: every sm_100a sparse kernel against the CPU implementation of the same operation."""
import pytest
import torch

import recis_b200
from recis_b200.nn import EmbeddingEngine, EmbeddingOption, HashTable, filter_out_sparse_param
from recis_b200.nn.hashtable_hook import FilterHook
from recis_b200.nn.initializers import NormalInitializer
from recis_b200.optim import SparseAdagrad, SparseAdam
from recis_b200.ragged import RaggedTensor

pytestmark = pytest.mark.gpu
C = recis_b200.native()
DEV = "cuda:0"


def make_store(device, dim=8, cap=64, kind=2):
    return C.EmbeddingStore(dim, cap, device, kind, 0.0, 0.05, -0.1, 0.1, 99, True, True, None)


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("n", [1, 1000, 300000])
def test_dedup_partition_gpu(world, n):
    torch.manual_seed(n + world)
    ids = (torch.randint(0, max(n // 3, 2), (n,), dtype=torch.int64) * 2654435761) - 7
    ids[::17] = -1
    uniq, rev, counts, offs = C.dedup_partition(ids.to(DEV), world)
    cu, crev, ccounts, coffs = C.dedup_partition(ids, world)
    assert torch.equal(counts.cpu(), ccounts) and torch.equal(offs.cpu(), coffs)
    nu = int(offs[-1])
    assert torch.equal(uniq[:nu][rev.long()].cpu(), ids)
    for r in range(world):
        a = uniq[offs[r]:offs[r + 1]].cpu().sort().values
        b = cu[coffs[r]:coffs[r + 1]].sort().values
        assert torch.equal(a, b)


@pytest.mark.parametrize("dim", [4, 16, 128, 7])
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_store_gpu_matches_cpu(dim, kind):
    torch.manual_seed(dim)
    g, c = make_store(DEV, dim, 32, kind), make_store("cpu", dim, 32, kind)
    ids = torch.randint(0, 1 << 40, (20000,), dtype=torch.int64)
    ids = torch.cat([ids, ids[:5000]])           # duplicates inside one call
    rg = g.lookup_or_insert(ids.to(DEV), None, None, 1)
    rc = c.lookup_or_insert(ids, None, None, 1)
    assert g.size() == c.size() == ids.unique().numel()
    assert int(rg.min()) >= 0
    eg = g.emb()[rg.long()].cpu(); ec = c.emb()[rc.long()]
    assert torch.allclose(eg, ec, atol=2e-6, rtol=1e-5)
    # same id -> same row
    assert torch.equal(rg[:5000], rg[20000:])
    assert torch.equal(g.find(ids.to(DEV), None), rg)
    er = g.erase(ids[:1000].unique().to(DEV))
    assert int(er.min()) >= 0 and g.size() == c.size() - ids[:1000].unique().numel()
    assert int(g.find(ids[:1000].to(DEV), None).max()) == -1
    k, r = g.snapshot(False, 0)
    assert k.numel() == g.size()
    assert g.counters()[3] == 0


def test_store_device_count_and_admission():
    g = make_store(DEV, 8, 1024)
    ids = torch.arange(100, dtype=torch.int64, device=DEV) * 31
    n_dev = torch.tensor([40], dtype=torch.int32, device=DEV)
    step = torch.tensor([3], dtype=torch.int64, device=DEV)
    r = g.lookup_or_insert(ids, n_dev, step, 1)
    assert g.size() == 40 and int(r[40:].max()) == -1 and int(r[:40].min()) >= 0
    assert int(g.last_seen()[r[:40].long()].min()) == 3
    g2 = make_store(DEV, 8, 1024)
    assert int(g2.lookup_or_insert(ids, None, step, 3).max()) == -1
    assert int(g2.lookup_or_insert(ids, None, step, 3).max()) == -1
    assert int(g2.lookup_or_insert(ids, None, step, 3).min()) >= 0 and g2.size() == 100


@pytest.mark.parametrize("dim", [4, 16, 64, 128, 256, 6])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_pool_and_grad_reduce_gpu(dim, mode):
    torch.manual_seed(dim + mode)
    U, S = 5000, 3000
    emb = torch.randn(U, dim)
    lens = torch.randint(0, 30, (S,))
    offsets = torch.zeros(S + 1, dtype=torch.int32); offsets[1:] = torch.cumsum(lens, 0)
    n = int(offsets[-1])
    raw = torch.randint(0, U, (n,))
    raw[: n // 3] = 7                                 # one very hot id: exercises the chunk-spanning path
    rev = torch.unique(raw, return_inverse=True)[1].to(torch.int32)
    w = torch.rand(n) + 0.5
    oc, gsrc_c, gscale_c = C.pool_forward(emb, None, rev, offsets, w, mode, 0, 0, True)
    og, gsrc_g, gscale_g = C.pool_forward(emb.to(DEV), None, rev.to(DEV), offsets.to(DEV), w.to(DEV), mode, 0, 0, True)
    assert torch.allclose(og.cpu(), oc, atol=1e-4, rtol=1e-4)
    assert torch.equal(gsrc_g.cpu(), gsrc_c) and torch.allclose(gscale_g.cpu(), gscale_c)
    cu_c = C.build_csr(rev); cu_g = C.build_csr(rev.to(DEV))
    for a, b in zip(cu_c[:2], cu_g[:2]):
        assert torch.equal(a, b.cpu())
    nu = int(rev.max()) + 1
    assert torch.equal(cu_c[2][: nu + 1], cu_g[2][: nu + 1].cpu())
    go = torch.randn(S, dim)
    args = (dim, None, False, 2, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0, None, None, None, nu)
    gu_c = C.grad_reduce(go, gsrc_c, gscale_c, *cu_c, *args)
    gu_g = C.grad_reduce(go.to(DEV), gsrc_g, gscale_g, *cu_g, *args)
    ref = torch.zeros(nu, dim, dtype=torch.float64).index_add_(0, rev.long(), (go[gsrc_c.long()] * gscale_c[:, None]).double())
    tol = 1e-5 * float(ref.abs().max()) + 1e-4        # fp32 accumulation over a very hot id: error scales with the sum
    assert torch.allclose(gu_c.double(), ref, atol=tol, rtol=1e-4)
    assert torch.allclose(gu_g.cpu().double(), ref, atol=tol, rtol=1e-4)


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_fused_reduce_apply_gpu(kind):
    torch.manual_seed(kind)
    dim, U, S = 32, 800, 600
    lens = torch.randint(1, 12, (S,))
    offsets = torch.zeros(S + 1, dtype=torch.int32); offsets[1:] = torch.cumsum(lens, 0)
    n = int(offsets[-1])
    raw = torch.randint(0, U, (n,)); raw[: n // 4] = 3
    rev = torch.unique(raw, return_inverse=True)[1].to(torch.int32)
    nu = int(rev.max()) + 1
    rows = torch.randperm(2000)[:nu].to(torch.int32)
    rows[5] = -1                                       # a not-admitted id: no update
    w0, m0, v0 = torch.randn(2000, dim), torch.rand(2000, dim), torch.rand(2000, dim)
    go = torch.randn(S, dim)
    hyper = (kind, 0.01, 0.9, 0.999, 1e-8, 0.99, -0.02, 0.5)
    res = []
    for dev in ("cpu", DEV):
        w, m, v = w0.clone().to(dev), m0.clone().to(dev), v0.clone().to(dev)
        _, gsrc, gscale = C.pool_forward(w, rows.to(dev), rev.to(dev), offsets.to(dev), None, 0, 0, 0, True)
        csr = C.build_csr(rev.to(dev))
        C.grad_reduce(go.to(dev), gsrc, gscale, *csr, dim, rows.to(dev), True, *hyper, w, m, v, 0)
        res.append((w.cpu(), m.cpu(), v.cpu()))
    for a, b in zip(*res):
        assert torch.allclose(a, b, atol=1e-4, rtol=1e-4)
    assert not torch.equal(res[0][0], w0)
    # two-step path (store per-unique gradient, then apply) agrees with the fused kernel
    w, m, v = w0.clone().to(DEV), m0.clone().to(DEV), v0.clone().to(DEV)
    _, gsrc, gscale = C.pool_forward(w, rows.to(DEV), rev.to(DEV), offsets.to(DEV), None, 0, 0, 0, True)
    csr = C.build_csr(rev.to(DEV))
    gu = C.grad_reduce(go.to(DEV), gsrc, gscale, *csr, dim, None, False, 2, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0, None, None, None, nu)
    C.sparse_apply(rows.to(DEV), gu, None, *hyper, w, m, v)
    assert torch.allclose(w.cpu(), res[1][0], atol=1e-4, rtol=1e-4)


def test_tile_and_perm_gpu():
    torch.manual_seed(0)
    emb = torch.randn(50, 16)
    B, F = 8, 3
    lens = torch.randint(0, 6, (B * F,))
    offsets = torch.zeros(B * F + 1, dtype=torch.int32); offsets[1:] = torch.cumsum(lens, 0)
    rev = torch.randint(0, 50, (int(offsets[-1]),), dtype=torch.int32)
    for fn_args in ((C.tile_forward, (4, True)), (C.pool_forward, (0, B, F, True))):
        fn, extra = fn_args
        c = fn(emb, None, rev, offsets, None, *extra)
        g = fn(emb.to(DEV), None, rev.to(DEV), offsets.to(DEV), None, *extra)
        assert torch.allclose(g[0].cpu(), c[0], atol=1e-5)
        assert torch.equal(g[1].cpu(), c[1])
    plain = C.pool_forward(emb, None, rev, offsets, None, 0, 0, 0, False)[0]
    perm = C.pool_forward(emb, None, rev, offsets, None, 0, B, F, False)[0]
    assert torch.equal(perm.view(B, F, 16).transpose(0, 1).reshape(B * F, 16), plain)


def _run_engine(device, steps=3):
    torch.manual_seed(0)
    from recis_b200.nn.modules.hashtable import HashtableRegister
    HashtableRegister().clear()
    init = NormalInitializer(0, 0.05)
    opts = {f"f{i}": EmbeddingOption(embedding_dim=32, shared_name=f"f{i}", combiner="sum" if i % 2 else "mean", initializer=init,
                                     device=device) for i in range(6)}
    eng = EmbeddingEngine(opts)
    opt = SparseAdam(filter_out_sparse_param(eng), lr=0.01)
    g = torch.Generator().manual_seed(1)
    outs = []
    for t in range(steps):
        feats, coefs = {}, {}
        for i in range(6):
            lens = torch.randint(1, 8, (64,), generator=g)
            off = torch.zeros(65, dtype=torch.int32); off[1:] = torch.cumsum(lens, 0)
            vals = torch.randint(0, 300, (int(off[-1]),), generator=g)
            feats[f"f{i}"] = RaggedTensor(vals, [off], weight=torch.rand(int(off[-1]), generator=g)).to(device)
            coefs[f"f{i}"] = torch.randn(64, 32, generator=g).to(device)
        out = eng(feats)
        loss = sum((out[k] * coefs[k]).sum() for k in out)
        opt.zero_grad(); loss.backward(); opt.step()
        outs.append(torch.stack([out[f"f{i}"].detach().cpu() for i in range(6)]))
    return outs


def test_engine_training_gpu_matches_cpu():
    a = _run_engine("cpu"); b = _run_engine(DEV)
    for x, y in zip(a, b):
        assert torch.allclose(x, y, atol=2e-4, rtol=1e-3)


def test_filter_hook_gpu():
    ht = HashTable([8], initializer=NormalInitializer(0, 1), name="gpu_ttl", device=DEV,
                   filter_hook=FilterHook("GlobalStepFilter", {"filter_step": 1}))
    ht(torch.arange(100, device=DEV))
    for _ in range(3):
        ht._filter_hook_impl.update_step()
        ht(torch.arange(10, device=DEV))
    assert ht._filter_hook_impl.do_filter() == 90 and ht.impl.size() == 10


def test_smoke_entry():
    import __graft_entry__ as ge
    ge.smoke()


@pytest.mark.gpu
def test_dedup_partition_overflow_is_flagged_and_memory_safe():
    """A unique-id buffer smaller than the batch's unique count: the status bit is set, boundaries are clamped to the
    buffer and the guard cells behind the buffer stay untouched."""
    C = recis_b200.native()
    ids = torch.arange(0, 5000, dtype=torch.int64, device="cuda") * 7919
    buf = torch.full((1200,), -7, dtype=torch.int64, device="cuda")
    window, guard = buf[:1000], buf[1000:]
    offsets = torch.zeros(5, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    _u, rev, _c, _o = C.dedup_partition(ids, 4, window, offsets, status)
    torch.cuda.synchronize()
    assert int(status.item()) & 8
    assert int(offsets.max()) <= 1000 and int(rev.max()) < 1000
    assert bool((guard == -7).all())
    # the same call with room for every id leaves the status word clean
    status.zero_()
    big = torch.empty(5000, dtype=torch.int64, device="cuda")
    C.dedup_partition(ids, 4, big, offsets, status)
    assert int(status.item()) == 0 and int(offsets[-1]) == 5000


@pytest.mark.gpu
def test_device_prefetcher_orders_and_copies():
    from recis_b200.io import DevicePrefetcher
    src = [{"a": (torch.arange(1000) + i).pin_memory(),
            "r": RaggedTensor((torch.arange(40) * i).pin_memory(), [torch.arange(0, 41, 4, dtype=torch.int32).pin_memory()])}
           for i in range(7)]
    got = []
    for b in DevicePrefetcher(src, "cuda", depth=3):
        assert b["a"].is_cuda and b["r"].values().is_cuda
        got.append((int(b["a"].sum()), int(b["r"].values().sum())))
    assert got == [(int((torch.arange(1000) + i).sum()), int((torch.arange(40) * i).sum())) for i in range(7)]


@pytest.mark.gpu
def test_store_grows_from_mirrored_history_with_device_counts():
    """Many calls with a device-side count and an oversized id buffer (the exchange-window shape): the store has to size its
    growth from the counters that come back asynchronously, never lose an id, and report no exhaustion."""
    torch.manual_seed(0)
    st = make_store(DEV, 8, 4096, 1)
    buf = torch.zeros(60000, dtype=torch.int64, device=DEV)
    seen = []
    for step in range(40):
        n = 1500 + 37 * step
        new = torch.randint(0, 1 << 50, (n,), dtype=torch.int64)
        ids = torch.cat([new, seen[-1][:500]]) if seen else new
        seen.append(new)
        buf[:ids.numel()] = ids.to(DEV)
        n_dev = torch.tensor([ids.numel()], dtype=torch.int32, device=DEV)
        rows = st.lookup_or_insert(buf, n_dev, None, 1)
        assert int(rows[:ids.numel()].min()) >= 0
        if step % 7 == 0:
            torch.cuda.synchronize()          # lets a few mirrors land at different lags
    all_ids = torch.cat(seen).unique()
    assert st.size() == all_ids.numel()
    assert int(st.find(all_ids.to(DEV), None).min()) >= 0
    assert st.capacity() >= all_ids.numel()


def test_table_grows_in_place_without_copying():
    """Row slabs live in reserved virtual ranges: growing maps pages behind the old end. The base address stays, the rows stay,
    and the time to grow does not depend on how many rows are live (an allocate-and-copy store pays for every live row)."""
    import time
    C = recis_b200.native()
    dim = 32

    def grow_time(fill_rows):
        store = C.EmbeddingStore(dim, 1_000_000, DEV, 2, 0.0, 0.05, 0.0, 0.0, 7, True, True, None)
        store.add_slot("state", 0.5)
        assert store.grows_in_place()
        ids = torch.arange(fill_rows, dtype=torch.int64, device=DEV) * 7919
        rows = store.lookup_or_insert(ids, None, None, 1) if fill_rows else None
        ptr = store.emb().data_ptr()
        probe = store.emb()[rows[:1000].long()].clone() if fill_rows else None
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        store.reserve(8_000_000)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
        assert store.capacity() == 8_000_000 and store.emb().shape[0] == 8_000_000
        assert store.emb().data_ptr() == ptr                                   # nothing moved
        if fill_rows:
            assert torch.equal(store.emb()[rows[:1000].long()], probe)         # old rows intact
            assert torch.equal(store.find(ids[:1000]), rows[:1000])
            more = torch.arange(fill_rows, fill_rows + 3_000_000, dtype=torch.int64, device=DEV) * 7919
            r2 = store.lookup_or_insert(more, None, None, 1)
            assert int(r2.min()) >= 0 and int(r2.max()) < 8_000_000 and store.size() == fill_rows + 3_000_000
            assert float(store.slot("state")[r2[-1].long()].min()) == 0.5      # new rows of a slot carry its fill value
        return dt
    grow_time(0)                                       # the process's first mapping pays one-off driver costs
    t_full, t_empty = min(grow_time(900_000) for _ in range(2)), min(grow_time(0) for _ in range(2))
    # the pointer checks above are the proof that nothing moved; the clock only has to rule out a copy of the filled rows
    assert t_full < 5 * t_empty + 0.05, (t_full, t_empty)


@pytest.mark.parametrize("n,D", [(1, 8), (7, 4), (8, 16), (9, 16), (31, 32), (33, 64), (2400, 128), (2048 * 148 * 8 // 32 * 32 // 128, 512),
                                 (2048 * 148 // 32 * 32 - 32, 128), (2048 * 148 // 32 * 32, 128), (2048 * 148 // 4 * 32 // 8 - 1, 8)])
def test_gradient_reduction_chunk_sizes(n, D):
    """Both chunk lengths of the segmented gradient reduction and the line between them (fewer groups of lanes than the GPU holds threads
    for), with ids that cross many chunks and ids that occur once, against an index_add in 64 bits. fp32 sums of c terms in any order
    differ by at most c * 2^-24 of the sum of magnitudes."""
    C = recis_b200.native()
    g = torch.Generator().manual_seed(n + D)
    rev = torch.randint(0, max(n // 3, 1), (n,), generator=g)
    rev[torch.rand(n, generator=g) < 0.3] = 0
    rev = torch.unique(rev, return_inverse=True)[1].to(torch.int32)
    segs = max(n // 4, 1)
    grad = torch.randn(segs, D, generator=g)
    gsrc = torch.randint(0, segs, (n,), generator=g).to(torch.int32)
    gscale = torch.rand(n, generator=g)
    n_u = int(rev.max()) + 1
    dev = [t.cuda() for t in (grad, gsrc, gscale, rev)]
    csr_u, csr_elem, start = C.build_csr(dev[3])
    gu = C.grad_reduce(dev[0], dev[1], dev[2], csr_u, csr_elem, start, D, None, False, 2, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0, None, None, None, n_u)
    terms = grad[gsrc.long()].double() * gscale.double().unsqueeze(1)
    ref = torch.zeros(n_u, D, dtype=torch.float64).index_add_(0, rev.long(), terms)
    mag = torch.zeros(n_u, D, dtype=torch.float64).index_add_(0, rev.long(), terms.abs())
    count = torch.bincount(rev.long(), minlength=n_u).double().unsqueeze(1)
    assert ((gu.double().cpu() - ref).abs() <= (count + 2) * 2.0 ** -24 * mag + 1e-30).all()


@pytest.mark.parametrize("n,world", [(1, 1), (257, 3), (1023, 1), (4 * 148 * 2048 - 1, 1), (4 * 148 * 2048 + 5, 1), (4 * 148 * 2048 + 1030, 8)])
def test_dedup_sizes_around_the_batched_probing(n, world):
    """Both probing variants and remainders of their blocks, with ids of every kind (0, -1, -2, the extremes): every unique id once, the
    reverse index leads back to it, owners in order, counts and offsets consistent."""
    C = recis_b200.native()
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(-n // 3 - 2, n // 3 + 2, (n,), generator=g)
    for k, v in enumerate((-1, -2, 0, -(1 << 63), (1 << 63) - 1)):
        ids[k::97] = v
    ids = ids.cuda()
    uniq, rev, counts, offs = C.dedup_partition(ids, world)
    n_u = int(offs[-1])
    assert torch.equal(uniq[rev.long()], ids) and n_u == int(counts.sum())
    assert torch.equal(torch.sort(uniq[:n_u]).values, torch.unique(ids))
    assert torch.equal(offs.cpu()[1:], counts.cpu().cumsum(0).to(torch.int32))
    ref = C.dedup_partition(ids.cpu(), world)
    assert torch.equal(ref[2], counts.cpu())
    for w in range(world):
        a, b = int(offs[w]), int(offs[w + 1])
        assert torch.equal(torch.sort(uniq[a:b]).values.cpu(), torch.sort(ref[0][a:b]).values)


@pytest.mark.parametrize("first", [1, 2, 3])
def test_lookup_kernels_take_views_at_any_element(first):
    """Rows and gradients that are contiguous but do not start on a 16-byte line give the bits of aligned ones; the packed result of an
    engine behind an odd number of elements of a concatenation hands such a gradient in."""
    def at(t):
        return torch.empty(t.numel() + first, dtype=t.dtype, device=DEV)[first:].copy_(t.reshape(-1)).view(t.shape)
    g = torch.Generator().manual_seed(first)
    D, n, U, S = 16, 500, 90, 60
    emb, grad = torch.randn(U, D, generator=g).to(DEV), torch.randn(S, D, generator=g).to(DEV)
    rev = torch.unique(torch.randint(0, U, (n,), generator=g), return_inverse=True)[1].to(torch.int32).to(DEV)
    offs = torch.linspace(0, n, S + 1).to(torch.int32).to(DEV)
    csr, n_u = C.build_csr(rev), int(rev.max()) + 1
    rows = torch.arange(n_u, dtype=torch.int32, device=DEV)
    got = []
    for place in (at, lambda t: t):
        pooled, gsrc, gscale = C.pool_forward(place(emb), None, rev, offs, None, 0, 0, 0, True)
        gu = C.grad_reduce(place(grad), gsrc, gscale, *csr, D, None, False, 2, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0, None, None, None, n_u)
        w, s1, s2 = emb.clone(), torch.zeros_like(emb), torch.zeros_like(emb)
        C.sparse_apply(rows, place(gu), None, 0, 0.01, 0.9, 0.999, 1e-8, 0.99, -0.02, 0.5, w, s1, s2)
        got.append([pooled, C.tile_forward(place(emb), None, rev, offs, None, 2, True)[0], w])
        half = place(emb.to(torch.bfloat16))
        got[-1].append(C.pool_forward(half, None, rev, offs, None, 1, 0, 0, False)[0])
    for a, b in zip(*got):
        assert torch.equal(a, b)
    opts = {k: EmbeddingOption(embedding_dim=8, shared_name=k, combiner="sum", use_weight=False, device=torch.device(DEV),
                               initializer=NormalInitializer(0.0, 1.0)) for k in "ab"}
    engine = EmbeddingEngine(opts, interleave=True)
    batch = {k: torch.randint(0, 9, (1, 3), device=DEV) for k in "ab"}
    opt = SparseAdagrad(filter_out_sparse_param(engine), lr=0.1)
    engine(batch)
    (cube, _), = engine.packed.values()
    before = cube.detach().clone()
    torch.cat([cube.new_ones(1, first), cube.view(1, -1)], 1).sum().backward()
    opt.step()
    engine(batch)
    (cube, _), = engine.packed.values()
    assert torch.isfinite(cube).all() and (cube < before).all()


@pytest.mark.parametrize("n,D", [(3000, 16), (70_001, 16), (30_000, 64), (9_999, 128), (20_000, 200)])
def test_gradient_sums_of_up_to_33_occurrences_repeat(n, D):
    """Rows of up to 33 occurrences give the same bits in every run, on either side of the chunk edges (longer ones meet in reductions of
    any order); chunks of 8 take the pieces of a row that crosses several of them in order."""
    g = torch.Generator().manual_seed(n)
    lens = torch.randint(1, 34, (n // 8,), generator=g)
    rev = torch.repeat_interleave(torch.arange(lens.numel()), lens)[:n]
    rev = rev[torch.randperm(rev.numel(), generator=g)].to(torch.int32).to(DEV)
    grad = torch.randn(rev.numel(), D, generator=g).to(DEV)
    gsrc = torch.randint(0, rev.numel(), (rev.numel(),), generator=g).to(torch.int32).to(DEV)
    gscale = torch.rand(rev.numel(), generator=g).to(DEV)
    csr = C.build_csr(rev)
    n_u = int(rev.max()) + 1
    sums = [C.grad_reduce(grad, gsrc, gscale, *csr, D, None, False, 2, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0, None, None, None, n_u) for _ in range(30)]
    assert all(torch.equal(s, sums[0]) for s in sums[1:])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("n", [148 * 2048 - 32, 148 * 2048])
def test_fused_update_on_both_sides_of_the_chunk_rule(n, kind, dtype):
    """The reduction with the row update in it, in chunks of 8 and of 32 (128 columns: the line is 148 * 2048 elements): rows that occur
    once, rows across several chunks, one of a thousand occurrences, rows that are not admitted. Against 64-bit sums and the CPU update;
    sums of at most 1000 fp32 terms, and one rounding of the row type."""
    D, g = 128, torch.Generator().manual_seed(kind)
    rev = torch.randint(0, n // 3, (n,), generator=g)
    rev[:1000] = 5
    rev[1000:60_000] = torch.randint(0, 3000, (59_000,), generator=g)            # about 20 occurrences each
    rev = torch.unique(rev[torch.randperm(n, generator=g)], return_inverse=True)[1].to(torch.int32)
    n_u, segs = int(rev.max()) + 1, n // 4
    rows = torch.randperm(n_u + 50, generator=g)[:n_u].to(torch.int32)
    rows[::97] = -1
    grad, gscale = torch.randn(segs, D, generator=g), torch.rand(n, generator=g)
    gsrc = torch.randint(0, segs, (n,), generator=g).to(torch.int32)
    w, s1, s2 = (torch.rand(n_u + 50, D, generator=g) for _ in range(3))
    hyper = (kind, 0.01, 0.9, 0.999, 1e-8, 0.99, -0.02, 0.5)
    dev = [t.to(DEV) for t in (w.to(dtype), s1, s2)]
    C.grad_reduce(grad.to(DEV), gsrc.to(DEV), gscale.to(DEV), *C.build_csr(rev.to(DEV)), D, rows.to(DEV), True, *hyper, *dev, 0)
    sums = torch.zeros(n_u, D, dtype=torch.float64).index_add_(0, rev.long(), grad[gsrc.long()].double() * gscale.double()[:, None])
    ref = [w.to(dtype), s1.clone(), s2.clone()]
    C.sparse_apply(rows, sums.float(), None, *hyper, *ref)
    ulp = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
    for a, b, rel in zip(dev, ref, (1e-4 + ulp, 1e-4, 1e-4)):
        assert torch.allclose(a.float().cpu(), b.float(), rtol=rel, atol=1e-4)
    assert not torch.equal(dev[0].cpu(), w.to(dtype))
