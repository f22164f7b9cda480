"""Performance cases: the work that users of the framework have it do, through its public entry points.

A case is a dict with a ``kind`` and the sizes of one call. ``listed`` names the cases that are tracked; ``draw`` makes one more
of the same ranges; ``prepare`` builds what a program has in hand before the call (a model with warm tables, a batch on the GPU);
``run`` is one pass; ``work`` and ``tolerance`` state what a pass cannot do without and how exact its outputs are.

Kinds (one group per way in which the framework is used):

  deepfm_train / dlrm_train / seq_train   one training step of a model: forward, loss, backward, sparse + dense optimizer step
  dlrm_serve / seq_serve                  one scoring call (evaluation mode, no gradients): small batches, latency counts
  embedding_train                         EmbeddingEngine alone: pooled lookup, backward, sparse optimizer, read-back of the updated
                                          rows (what an online learner publishes); row types, combiners, widths, weights
  features                                FeatureEngine: hash / mod / bucketize / truncation over many ragged features
  attention                               ragged self-attention, forward and backward
  tower                                   bf16 MLP over a wide input: forward, backward, dense Adam step

Ids follow Zipf(1.05 .. 1.1) as in the benchmarks, bags are ragged, sequence lengths are spread over their whole range.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from recis_b200.features import Bucketize, Feature, FeatureEngine, Hash, Mod, SelectField, SequenceTruncate
from recis_b200.models import DLRM, DeepFM, SequenceModel
from recis_b200.nn import EmbeddingEngine, EmbeddingOption, filter_out_sparse_param
from recis_b200.nn.initializers import NormalInitializer
from recis_b200.nn.modules.hashtable import ChildrenInfo, HashtableRegister
from recis_b200.ops.attention import ragged_self_attention
from recis_b200.ops.dense import MLP
from recis_b200.optim import DenseAdam, SparseAdagrad, SparseAdam
from recis_b200.ragged import RaggedTensor

_ROW_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
_ROW_BYTES = {"fp32": 4, "bf16": 2, "fp16": 2}


def listed():
    return [
        # the smallest training step: single-hot fields, narrow rows, a small tower (the example program's default shape)
        {"name": "deepfm_train_b1024", "kind": "deepfm_train", "batch": 1024, "fields": 26, "emb": 16},
        # the flagship click model at its benchmark batch: 26 multi-hot fields, one merged table of 128-wide rows
        {"name": "dlrm_train_b8192", "kind": "dlrm_train", "batch": 8192, "fields": 26, "bag": 20.0, "universe": 150_000},
        # the same model at an odd, smaller batch and fewer fields (the last batch of an epoch, a smaller job)
        {"name": "dlrm_train_b1777", "kind": "dlrm_train", "batch": 1777, "fields": 15, "bag": 11.0, "universe": 100_000},
        # online scoring of one request's candidates: the smallest call
        {"name": "dlrm_serve_b64", "kind": "dlrm_serve", "batch": 64, "fields": 26, "bag": 20.0, "universe": 150_000},
        # the long-behaviour-sequence model, training: ragged sequences of 50 .. 1000 tokens
        {"name": "seq_train_b512", "kind": "seq_train", "batch": 512, "min_len": 50, "max_len": 1000, "hidden": 256, "items": 2_000_000},
        # the same model scoring a small, odd batch
        {"name": "seq_serve_b37", "kind": "seq_serve", "batch": 37, "min_len": 1, "max_len": 1000, "hidden": 256, "items": 2_000_000},
        # many small tables merged into one physical table, Adagrad (the embedding microbenchmark), fp32 rows: the largest lookup
        {"name": "embedding_200x64", "kind": "embedding_train", "tables": 200, "dims": "64", "batch": 4096, "bag": 10.0, "combiner": "sum",
         "rows": "fp32", "weights": False, "opt": "adagrad", "universe": 400_000},
        # tables of mixed widths behind one engine (five physical tables), Adam, bf16 rows, weighted mean pooling, odd batch
        {"name": "embedding_mixed_bf16", "kind": "embedding_train", "tables": 60, "dims": "8-16-32-64-128", "batch": 3001, "bag": 5.0,
         "combiner": "mean", "rows": "bf16", "weights": True, "opt": "adam", "universe": 200_000},
        # raw features of a many-field model through the feature engine
        {"name": "features_50x8192", "kind": "features", "fields": 50, "batch": 8192, "mean_len": 20, "keep": 16},
        # a sequence encoder's attention core at the benchmark's lengths
        {"name": "attention_256seq_h4", "kind": "attention", "seqs": 256, "heads": 4, "min_len": 50, "max_len": 1000},
        # many short, ragged sequences (sessions)
        {"name": "attention_3000short_h8", "kind": "attention", "seqs": 3000, "heads": 8, "min_len": 1, "max_len": 90},
        # the dense tower of the many-field model: wide input, compute bound
        {"name": "tower_b16384", "kind": "tower", "batch": 16384, "dims": "3200-2048-1024-512-1"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["deepfm_train", "dlrm_train", "dlrm_serve", "seq_train", "seq_serve", "embedding_train", "embedding_train", "features",
                       "attention", "attention", "tower"])
    if kind == "deepfm_train":
        return {"kind": kind, "batch": _log_int(rng, 64, 8192), "fields": rng.randint(8, 39), "emb": rng.choice([8, 16, 32])}
    if kind in ("dlrm_train", "dlrm_serve"):
        return {"kind": kind, "batch": _log_int(rng, 300, 8192) if kind == "dlrm_train" else _log_int(rng, 1, 2048), "fields": rng.randint(6, 26),
                "bag": round(rng.uniform(2.0, 20.0), 1), "universe": _log_int(rng, 10_000, 150_000)}
    if kind in ("seq_train", "seq_serve"):
        lo, hi = rng.choice([(1, 1000), (50, 1000), (10, 200), (20, 600)])
        return {"kind": kind, "batch": _log_int(rng, 16, 512) if kind == "seq_train" else _log_int(rng, 1, 256), "min_len": lo, "max_len": hi,
                "hidden": rng.choice([128, 256]), "items": _log_int(rng, 100_000, 2_000_000)}
    if kind == "embedding_train":
        rows = rng.choice(["fp32", "fp32", "bf16", "fp16"])
        dims = rng.choice(["64", "16", "128", "32", "8-16-32-64-128", "24-200"])
        batch, bag = _log_int(rng, 256, 4096), round(rng.uniform(1.0, 10.0), 1)
        tables = max(1, min(_log_int(rng, 4, 200), int(1.6e6 * 64 / (batch * bag * max(int(d) for d in dims.split("-"))) * 4)))
        tables = max(1, min(tables, int(6e6 / (batch * bag))))
        combiner = rng.choice(["sum", "mean", "tile"])
        if combiner == "tile":
            tables = min(tables, 40)                     # every table comes back as a tensor of its own
        return {"kind": kind, "tables": tables, "dims": dims, "batch": batch, "bag": bag, "combiner": combiner,
                "rows": rows, "weights": rng.random() < 0.4, "opt": rng.choice(["adagrad", "adam"]), "universe": _log_int(rng, 5_000, 400_000)}
    if kind == "features":
        return {"kind": kind, "fields": rng.randint(4, 50), "batch": _log_int(rng, 128, 8192), "mean_len": rng.randint(1, 20), "keep": rng.randint(1, 32)}
    if kind == "attention":
        lo, hi = rng.choice([(1, 1000), (50, 1000), (1, 90), (100, 300), (129, 129), (64, 512)])
        heads = rng.choice([1, 2, 4, 8, 16])
        cap = 256 * 4 * 525.0 * 525.0 / (heads * (0.5 * (lo + hi)) ** 2)
        cap = min(cap, 256 * 4 * 525.0 / (heads * 0.5 * (lo + hi)))
        return {"kind": kind, "seqs": max(1, _log_int(rng, 1, max(2, cap))), "heads": heads, "min_len": lo, "max_len": hi}
    dims = rng.choice(["3200-2048-1024-512-1", "479-1024-1024-512-256-1", "1000-400-400-400-1", "256-1024-256", "13-512-256-128"])
    return {"kind": "tower", "batch": _log_int(rng, 100, 16384), "dims": dims}


# ---------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _zipf(n, a, universe, gen):
    """``n`` ids in [0, universe): Zipf(a) ranks (inverse of the continuous distribution), scattered over the range by an odd factor."""
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    e = 1.0 - a
    rank = torch.pow(1.0 + u * (float(universe) ** e - 1.0), 1.0 / e).floor().clamp_(1, float(universe)).to(torch.int64) - 1
    return (rank * 0x9E3779B1 + 0x7F4A7C15) % universe


def _spread(ids, salt):
    """Raw 40-bit ids as they come from logs: a bijection of the dense ids."""
    return ((ids + salt * 7_919_191) * 0x2545F4914F6CDD1D) & ((1 << 40) - 1)


def _shuffled(lens, gen):
    """Every row of ``lens`` in an order of its own: which sample is long comes from the seed, the totals are those of the case."""
    return lens.gather(-1, torch.rand(lens.shape, generator=gen, device="cuda").argsort(-1))


def _bags(fields, batch, mean, gen, lo=1, hi=100):
    """int32 offsets [fields, batch + 1] of Poisson bag lengths in [lo, hi] and the totals per field."""
    lens = torch.poisson(torch.full((fields, batch), float(mean), device="cuda"), generator=_gen(17)).clamp_(lo, hi).to(torch.int32)
    lens = _shuffled(lens, gen)
    offs = torch.zeros((fields, batch + 1), dtype=torch.int32, device="cuda")
    offs[:, 1:] = lens.cumsum(1)
    return offs, offs[:, -1].tolist()


def _multi_hot(names, batch, bag, universe, a, gen):
    offs, totals = _bags(len(names), batch, bag, gen)
    ids = _zipf(sum(totals), a, universe, gen)
    out, pos = {}, 0
    for i, name in enumerate(names):
        out[name] = RaggedTensor(_spread(ids[pos:pos + totals[i]], i), [offs[i].clone()], dense_shape=(batch, -1))
        pos += totals[i]
    return out


def _dlrm_batch(names, case, gen):
    B = case["batch"]
    batch = _multi_hot(names, B, case["bag"], case["universe"], 1.05, gen)
    batch["dense"] = torch.randn(B, 13, generator=gen, device="cuda").exp().log1p()
    batch["label"] = (torch.rand(B, 1, generator=gen, device="cuda") < 0.03).float()
    return batch


def _sequences(n, lo, hi, gen):
    """int32 offsets [n + 1] of sequence lengths spread uniformly over [lo, hi], and the longest length."""
    lens = torch.randint(lo, hi + 1, (n,), generator=_gen(23), device="cuda").to(torch.int32)
    offs = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    offs[1:] = _shuffled(lens, gen).cumsum(0)
    return offs, int(lens.max())


def _seq_batch(profile, case, gen):
    B = case["batch"]
    offs, longest = _sequences(B, case["min_len"], case["max_len"], gen)
    T = int(offs[-1])
    items = _zipf(T + B, 1.1, case["items"], gen)
    cates = items % 10_000
    batch = {"seq_item": RaggedTensor(items[:T], [offs], dense_shape=(B, -1)), "seq_cate": RaggedTensor(cates[:T], [offs], dense_shape=(B, -1)),
             "tgt_item": items[T:].clone(), "tgt_cate": cates[T:].clone(), "max_len": longest,
             "label": (torch.rand(B, 1, generator=gen, device="cuda") < 0.05).float()}
    for i, f in enumerate(profile):
        batch[f] = torch.randint(0, 1000 * (i + 1), (B,), generator=gen, device="cuda")
    return batch


def _warm(engine, batches):
    """Tables as training leaves them: the ids of earlier batches have rows."""
    engine.train()
    with torch.no_grad():
        for b in batches:
            engine(b)


def _feature_plan(case):
    return [("mod", "mod", "hash", "hash", "bucket")[i % 5] for i in range(case["fields"])]


# --------------------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    torch.manual_seed(1234)                         # weights are those of one model; ids, lengths and values come from the seed
    HashtableRegister().clear()                     # every state is a model of its own, under the same table names
    st = {"kind": kind}

    if kind in ("deepfm_train", "dlrm_train", "dlrm_serve", "seq_train", "seq_serve"):
        B = case["batch"]
        if kind == "deepfm_train":
            names = [f"c{i}" for i in range(case["fields"])]

            def make():
                ids = _zipf(B * len(names), 1.1, 1_000_000, gen).view(len(names), B)
                b = {f: ids[i].view(B, 1).clone() for i, f in enumerate(names)}
                b["dense"] = torch.randn(B, 13, generator=gen, device="cuda").exp().log1p()
                b["label"] = (torch.rand(B, 1, generator=gen, device="cuda") < 0.25).float()
                return b
            model = DeepFM(names, dense_dim=13, emb_dim=case["emb"], hidden=(400, 400, 400), device="cuda", capacity=16 * B * len(names)).to("cuda")
            history = [make() for _ in range(2)]
            st["batch"] = make()
            _warm(model.embedding_engine, [{n + s: b[n] for n in names for s in ("_emb", "_bias")} for b in history])
        elif kind in ("dlrm_train", "dlrm_serve"):
            names = [f"c{i}" for i in range(case["fields"])]
            model = DLRM(names, dense_dim=13, emb_dim=128, device="cuda", capacity=int(1.1 * case["universe"] * len(names)) + 100_000).to("cuda")
            big = dict(case, batch=max(B, 2048))
            history = [_dlrm_batch(names, big, gen) for _ in range(2)]
            st["batch"] = _dlrm_batch(names, case, gen)
            _warm(model.embedding_engine, [{n: b[n] for n in names} for b in history])
        else:
            profile = [f"profile_{i}" for i in range(20)]
            hidden = case["hidden"]
            model = SequenceModel(profile, hidden=hidden, heads=hidden // 64, layers=2, ffn=4 * hidden, device="cuda",
                                   item_capacity=case["items"] // 2, cate_capacity=20_000, profile_capacity=300_000, max_len=case["max_len"]).to("cuda")
            st["batch"] = _seq_batch(profile, case, gen)
            seen = _seq_batch(profile, dict(case, batch=max(B, 128)), gen)
            ids = {f: seen[f] for f in profile + ["tgt_item", "tgt_cate"]}
            _warm(model.embedding_engine, [dict(ids, seq_item=seen["seq_item"].values(), seq_cate=seen["seq_cate"].values())])
        st["model"] = model
        if kind.endswith("_serve"):
            model.eval()
        else:
            model.train()
            sparse = filter_out_sparse_param(model)
            st["sparse_opt"] = SparseAdagrad(sparse, lr=0.01) if kind == "deepfm_train" else SparseAdam(sparse, lr=1e-3)
            st["params"] = [p for p in model.parameters() if p.requires_grad]
            st["dense_opt"] = DenseAdam(st["params"], lr=1e-3)
        return st

    if kind == "embedding_train":
        names = [f"t{i}" for i in range(case["tables"])]
        dims = [int(d) for d in case["dims"].split("-")]
        kw = {"combiner_kwargs": {"tile_len": 4}} if case["combiner"] == "tile" else {}
        per_table = int(min(case["universe"], 2 * case["batch"] * case["bag"])) + 64
        opts = {n: EmbeddingOption(embedding_dim=dims[i % len(dims)], shared_name=n, combiner=case["combiner"], use_weight=case["weights"],
                                   device="cuda", initializer=NormalInitializer(0.0, 0.01), capacity=per_table, dtype=_ROW_DTYPES[case["rows"]], **kw)
                for i, n in enumerate(names)}
        engine = EmbeddingEngine(opts, interleave=case["combiner"] != "tile")
        _warm(engine, [_multi_hot(names, case["batch"], case["bag"], case["universe"], 1.05, gen)])
        batch = _multi_hot(names, case["batch"], case["bag"], case["universe"], 1.05, gen)
        if case["weights"]:
            for n in names:
                v = batch[n].values()
                batch[n] = RaggedTensor(v, batch[n].offsets(), torch.rand(v.numel(), generator=gen, device="cuda") + 0.5, dense_shape=(case["batch"], -1))
        cls = SparseAdagrad if case["opt"] == "adagrad" else SparseAdam
        st.update(engine=engine, batch=batch, opt=cls(filter_out_sparse_param(engine), lr=0.01), names=names, grads=None)
        # the distinct ids of the batch per physical table, whose updated rows are read back after the step
        touched = {}
        for n in names:
            table = engine.table_of(n)
            child = table.table.children_info().child_index(n)
            touched.setdefault(id(table), (table, []))[1].append(ChildrenInfo.encode(torch.unique(batch[n].values()), child))
        st["touched"] = []
        for table, ids in touched.values():
            ids = torch.cat(ids)
            # as many as the batch is expected to touch, some of them twice where it touches fewer
            n = int(sum(engine.table_of(n) is table for n in names) * _distinct(case["batch"] * max(1.0, case["bag"]), 1.05, case["universe"]))
            st["touched"].append((table.table, ids[torch.arange(n, device="cuda") % ids.numel()]))
        outs = _pooled(engine, batch, names)
        st["grads"] = [(torch.randn(o.shape, generator=gen, device="cuda") * 1e-3).to(o.dtype) for o in outs]
        return st

    if kind == "features":
        F, B = case["fields"], case["batch"]
        plan = _feature_plan(case)
        boundaries = torch.linspace(-3.0, 3.0, 200).tolist()
        feats, batch = [], {}
        offs, totals = _bags(F, B, case["mean_len"], gen, lo=0)
        ids = _zipf(sum(totals), 1.05, 1 << 40, gen)
        pos = 0
        for i, op in enumerate(plan):
            name, n = f"f{i}", totals[i]
            v = _spread(ids[pos:pos + n], i)
            pos += n
            o = offs[i].clone()
            f = Feature(name).add_op(SelectField(name, dtype=torch.float32 if op == "bucket" else torch.long))
            if op == "mod":
                f.add_op(Mod((1 << 31) - 1))
                batch[name] = RaggedTensor(v, [o], dense_shape=(B, -1))
            elif op == "hash":
                # strings of 1 .. 24 bytes
                slen = torch.randint(1, 25, (n,), generator=gen, device="cuda")
                inner = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
                inner[1:] = slen.cumsum(0)
                chars = torch.randint(32, 127, (int(inner[-1]),), generator=gen, device="cuda").to(torch.int8)
                f.add_op(Hash("farm" if i % 2 else "murmur"))
                batch[name] = RaggedTensor(chars, [o, inner], dense_shape=(B, -1, -1))
            else:
                f.add_op(Bucketize(boundaries))
                batch[name] = RaggedTensor(torch.randn(n, generator=gen, device="cuda"), [o], dense_shape=(B, -1))
            if i % 5 in (1, 3):
                f.add_op(SequenceTruncate(seq_len=case["keep"], truncate_side="left" if i % 2 else "right", n_dims=2))
            feats.append(f)
        st.update(engine=FeatureEngine(feats), batch=batch, names=[f"f{i}" for i in range(F)])
        return st

    if kind == "attention":
        H = case["heads"]
        offs, longest = _sequences(case["seqs"], case["min_len"], case["max_len"], gen)
        T = int(offs[-1])
        st["qkv"] = (torch.randn(T, 3 * H * 64, generator=gen, device="cuda") * 0.7).to(torch.bfloat16).requires_grad_()
        st["d_out"] = torch.randn(T, H * 64, generator=gen, device="cuda").to(torch.bfloat16)
        st.update(offsets=offs, heads=H, max_len=longest)
        return st

    dims = [int(d) for d in case["dims"].split("-")]
    mlp = MLP(dims, final_act=False).to("cuda")
    st.update(model=mlp, params=list(mlp.parameters()), x=torch.randn(case["batch"], dims[0], generator=gen, device="cuda").requires_grad_(),
              d_out=torch.randn(case["batch"], dims[-1], generator=gen, device="cuda") / case["batch"])
    st["dense_opt"] = DenseAdam(st["params"], lr=1e-3)
    return st


# ------------------------------------------------------------------------------------------------------------------- run
def _pooled(engine, batch, names):
    outs = engine(batch)
    if engine.packed and len(engine.packed) == len(engine.tables()):
        return [cube for cube, _ in engine.packed.values()]
    return [outs[n] for n in names]


def run(st):
    kind = st["kind"]
    if kind in ("deepfm_train", "dlrm_train", "seq_train"):
        model = st["model"]
        loss, logit = model(st["batch"])
        st["dense_opt"].zero_grad()
        st["sparse_opt"].zero_grad()
        loss.backward()
        st["sparse_opt"].step()
        st["dense_opt"].step()
        cubes = [c for c, _ in model.embedding_engine.packed.values()]
        return [loss.detach(), logit.detach(), [p.grad for p in st["params"]], [c.detach() for c in cubes]]
    if kind.endswith("_serve"):
        with torch.no_grad():
            loss, logit = st["model"](st["batch"])
        return [loss, logit]
    if kind == "embedding_train":
        outs = _pooled(st["engine"], st["batch"], st["names"])
        torch.autograd.backward(outs, st["grads"])
        st["opt"].step()
        st["opt"].zero_grad()
        rows = [table.impl.embedding_lookup(ids, readonly=True)[1] for table, ids in st["touched"]]
        return [[o.detach() for o in outs], rows]
    if kind == "features":
        out = st["engine"](st["batch"])
        vals = [out[n].values() for n in st["names"]]
        return vals + [out[n].offsets()[-1] for i, n in enumerate(st["names"]) if i % 10 in (1, 3)]
    if kind == "attention":
        qkv = st["qkv"]
        qkv.grad = None
        out = ragged_self_attention(qkv, st["offsets"], st["heads"], st["max_len"])
        out.backward(st["d_out"])
        return [out.detach(), qkv.grad]
    st["x"].grad = None
    y = st["model"](st["x"])
    st["dense_opt"].zero_grad()
    y.backward(st["d_out"].to(y.dtype))
    st["dense_opt"].step()
    return [y.detach(), st["x"].grad, [p.grad for p in st["params"]]]


# ------------------------------------------------------------------------------------------------------------------ work
def _distinct(n, a, universe):
    """Expected number of distinct ids among ``n`` draws of the continuous Zipf(a) over [1, universe]."""
    edges = np.unique(np.floor(np.logspace(0, math.log10(universe), 400)))
    e = 1.0 - a
    cdf = (edges ** e - 1.0) / (float(universe) ** e - 1.0)
    width = np.diff(edges)
    p = np.diff(cdf) / width
    return float((width * -np.expm1(n * np.log1p(-np.minimum(p, 1 - 1e-12)))).sum()) + 1.0


def _mlp_work(dims, M, train):
    params = sum(a * b + b for a, b in zip(dims, dims[1:]))
    flops = 2.0 * M * sum(a * b for a, b in zip(dims, dims[1:])) * (3 if train else 1)
    # optimizer: gradient, weight and both moments read, weight and moments written; scoring reads the bf16 weights
    return flops, params * (28 if train else 2)


def _embedding_work(nnz, segs, distinct, D, row_bytes, state, train):
    read = nnz * 8 + segs * 4 + distinct * D * row_bytes + segs * D * 4
    return read + (segs * D * 4 + distinct * D * (2 * row_bytes + 8 * state) if train else 0)


def work(case):
    kind = case["kind"]
    train = not kind.endswith("_serve")
    if kind == "deepfm_train":
        B, F, D = case["batch"], case["fields"], case["emb"]
        u = F * _distinct(B, 1.1, 1_000_000)
        flops, bytes_ = _mlp_work([(13 + F) * D, 400, 400, 400, 1], B, True)
        return {"bytes": bytes_ + _embedding_work(2 * B * F, 2 * B * F, u, D + 4, 4, 1, True), "flops": flops}
    if kind in ("dlrm_train", "dlrm_serve"):
        B, F, D = case["batch"], case["fields"], 128
        nnz = B * F * case["bag"]
        u = F * _distinct(nnz / F, 1.05, case["universe"])
        top = D + (F + 1) * F // 2
        f1, b1 = _mlp_work([13, 512, 256, 128], B, train)
        f2, b2 = _mlp_work([top, 1024, 1024, 512, 256, 1], B, train)
        pair = 2.0 * B * (F + 1) * (F + 1) * D * (3 if train else 1)
        return {"bytes": b1 + b2 + _embedding_work(nnz, B * F, u, D, 4, 2, train), "flops": f1 + f2 + pair}
    if kind in ("seq_train", "seq_serve"):
        B, h, heads = case["batch"], case["hidden"], case["hidden"] // 64
        lo, hi = case["min_len"], case["max_len"]
        T, L2 = B * (lo + hi) / 2.0, B * ((hi - lo) ** 2 / 12.0 + ((lo + hi) / 2.0) ** 2)
        gemm = 2.0 * T * (128 * h + 2 * (12 * h * h)) * (3 if train else 1)
        att = 4.0 * 64 * heads * L2 * 2 * (3.5 if train else 1)
        f_head, b_head = _mlp_work([3 * h + 640, 512, 256, 1], B, train)
        u = _distinct(T, 1.1, case["items"]) + 10_000 + B * 20
        return {"bytes": b_head + (28.0 if train else 2.0) * 24 * h * h + _embedding_work(2 * T + B * 22, 2 * T + B * 22, u, 64, 4, 2, train), "flops": gemm + att + f_head}
    if kind == "embedding_train":
        dims = [int(d) for d in case["dims"].split("-")]
        bag = max(1.0, case["bag"])
        total = 0.0
        for i in range(case["tables"]):
            D, nnz = dims[i % len(dims)], case["batch"] * bag
            u = _distinct(nnz, 1.05, case["universe"])
            segs = case["batch"] * (4 if case["combiner"] == "tile" else 1)
            total += _embedding_work(nnz * (1.5 if case["weights"] else 1), segs, u, D, _ROW_BYTES[case["rows"]], 1 if case["opt"] == "adagrad" else 2, True)
            total += u * (8 + 2 * D * _ROW_BYTES[case["rows"]])
        return {"bytes": total, "flops": 0}
    if kind == "features":
        plan = _feature_plan(case)
        n = case["batch"] * case["mean_len"]
        per = {"mod": 16, "hash": 12.5 + 4 + 8, "bucket": 12}
        total = sum(n * per[p] for p in plan)
        total += sum(case["batch"] * (min(case["mean_len"], case["keep"]) * 16 + 8) for i in range(len(plan)) if i % 5 in (1, 3))
        return {"bytes": total, "flops": 0}
    if kind == "attention":
        H, n, lo, hi = case["heads"], case["seqs"], case["min_len"], case["max_len"]
        T, L2 = n * (lo + hi) / 2.0, n * (((hi - lo + 1) ** 2 - 1) / 12.0 + ((lo + hi) / 2.0) ** 2)
        return {"bytes": T * H * 64 * 2 * (3 + 1 + 1 + 3), "flops": 4.0 * 64 * H * L2 * 3.5}
    dims = [int(d) for d in case["dims"].split("-")]
    M = case["batch"]
    flops, bytes_ = _mlp_work(dims, M, True)
    return {"bytes": bytes_ + M * (dims[0] * 8 + dims[-1] * 6), "flops": flops}


def tolerance(case):
    """About four times what was measured between two correct implementations of a case: bf16 towers against other tile orders and
    an fp32 tower, attention against 64-bit arithmetic, fp32 sums of rows in another order (Adam and Adagrad turn a rounding
    difference of a near-zero gradient into a step of the other sign)."""
    kind = case["kind"]
    if kind == "features":
        return "exact"
    if kind == "embedding_train":
        return {"rel": 1e-4 if case["rows"] == "fp32" else 2e-4, "max": 0.6}
    if kind == "attention":
        return {"rel": 1e-2, "max": 0.2}
    # the bias of the key projection has a gradient that is zero but for rounding: it sets the figure of the sequence model
    return {"rel": 3e-2 if kind == "seq_train" else 2e-2, "max": 0.5}
