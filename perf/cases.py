"""Performance cases: passes through the public entry points that a user of this framework has it do.

A case is a plain dict; `kind` says which path it takes and the other fields give sizes, types and options.

  train     pooled lookups: forward + fused backward with the sparse optimizer, through the module
  sequence  unpooled lookups padded to a dense [bag, length, dim] block, forward and backward
  serve     pooled lookups without a backward (evaluation, inference)
  hashed    hash-keyed tables: keys -> slots + unique + inverse (IdsMapper), then forward + backward on them
  dynamic   a cached dynamic table: timestamps, counts, admission, slot policy, eviction, then forward + backward
  hybrid    a table larger than its HBM cache: slot policy, rows swapped with the host store, forward + backward
  rowwise   the row-wise sharded lookup on one rank: deduplicated fetch, local and owner backward phases
  input     input distribution of a jagged batch: offsets, feature permute, row-hash bucketize

Ids are Zipf distributed (hot rows spread over the table), gradients are N(0, 1), weights start uniform.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from recsdk_b200 import AdmitAndEvictConfig, EmbcacheManager, EmbConfig, ops, torch_ops
from recsdk_b200.hybrid_cache import HybridCacheEmbeddingBag
from recsdk_b200.rowwise import RowWiseShardedEmbeddingBag
from recsdk_b200.synthetic import table_rows_log_uniform, zipf_ids
from recsdk_b200.tbe import EmbOptimType, HybridSplitTableBatchedEmbeddingBagsCodegen, PoolingMode

DEV = "cuda"
OPTIM = {"adagrad": EmbOptimType.EXACT_ADAGRAD, "adam": EmbOptimType.ADAM, "sgd": EmbOptimType.EXACT_SGD}
STATES = {"adagrad": 1, "adam": 2, "sgd": 0}
POOL = {"sum": PoolingMode.SUM, "mean": PoolingMode.MEAN, "none": PoolingMode.NONE}


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one small table, one id per sample: a step of a dozen short kernels, launches and host work decide
        dict(name="train_small", kind="train", tables=1, rows_lo=1_000_000, rows_hi=1_000_000, dims="16", batch=4096,
             bag_lo=1, bag_hi=1, alpha=1.05, pooling="sum", optim="adagrad", plan_ahead=False),
        # click-model training: 26 categorical fields, one id each, large batch, Adam; the index work planned ahead
        dict(name="train_onehot", kind="train", tables=26, rows_lo=1_000, rows_hi=1_500_000, dims="128", batch=65536,
             bag_lo=1, bag_hi=1, alpha=1.1, pooling="sum", optim="adam", plan_ahead=True),
        # multi-hot training: long bags, many ids per row, 20 M ids per step
        dict(name="train_multihot", kind="train", tables=26, rows_lo=250_000, rows_hi=2_500_000, dims="64",
             batch=16384, bag_lo=1, bag_hi=100, alpha=1.2, pooling="sum", optim="adagrad", plan_ahead=True),
        # tables of different widths (some no multiple of 4 or a power of two), odd batch, empty bags, MEAN, no plan ahead
        dict(name="train_mixed", kind="train", tables=11, rows_lo=2_000, rows_hi=300_000, dims="8,32,20,64,128,48,18",
             batch=3001, bag_lo=0, bag_hi=20, alpha=1.05, pooling="mean", optim="sgd", plan_ahead=False),
        # behaviour sequences for a sequence model: unpooled rows, padded to a dense block
        dict(name="train_sequence", kind="sequence", tables=4, rows_lo=100_000, rows_hi=1_000_000, dims="64",
             batch=2048, bag_lo=0, bag_hi=50, alpha=1.05, pooling="none", optim="adam", plan_ahead=False),
        # online inference: a handful of samples, latency counts
        dict(name="serve_small", kind="serve", tables=26, rows_lo=1_000, rows_hi=500_000, dims="128", batch=37,
             bag_lo=0, bag_hi=10, alpha=1.1, pooling="sum", optim="sgd", plan_ahead=False),
        # batch inference / evaluation: bandwidth counts
        dict(name="serve_large", kind="serve", tables=12, rows_lo=50_000, rows_hi=1_000_000, dims="256", batch=8192,
             bag_lo=1, bag_hi=30, alpha=1.05, pooling="mean", optim="sgd", plan_ahead=False),
        # hash-keyed tables: every step maps its keys table by table
        dict(name="train_hashed", kind="hashed", tables=8, rows_lo=500_000, rows_hi=500_000, dims="64", batch=16384,
             bag_lo=1, bag_hi=3, alpha=1.05, pooling="sum", optim="adagrad", plan_ahead=False),
        # dynamic table with admission (count >= 2) and eviction (idle > 50 steps), 30 % new keys per step
        dict(name="train_dynamic", kind="dynamic", cache=1 << 23, dim=32, keys=131072, pool=1_000_000),
        # working set four times the HBM cache: rows swap with the host store every step
        dict(name="train_hybrid", kind="hybrid", tables=2, cache=65536, dim=64, keys=8192, universe=262144),
        # a rank of the row-wise sharded giant table
        dict(name="train_rowwise", kind="rowwise", rows=20_000_000, dim=64, batch=262144, alpha=1.05, optim="adam"),
        # jagged batch on its way to the row-wise owners: 26 features, deduplicated per owner
        dict(name="input_dist", kind="input", tables=26, batch=8192, bag_lo=0, bag_hi=8, vocab=1_000_000, alpha=1.1,
             world=8, unique=True),
    ]


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    kind = rng.choices(["train", "sequence", "serve", "hashed", "dynamic", "hybrid", "rowwise", "input"],
                       [8, 2, 3, 2, 1, 1, 1, 2])[0]
    if kind == "dynamic":
        return dict(kind=kind, cache=1 << rng.randint(20, 23), dim=rng.choice([16, 32, 64]),
                    keys=_log_int(rng, 4096, 131072), pool=_log_int(rng, 50_000, 900_000))
    if kind == "hybrid":
        cache = _log_int(rng, 16384, 65536)
        return dict(kind=kind, tables=rng.randint(1, 2), cache=cache, dim=rng.choice([16, 32, 64]),
                    keys=cache // rng.randint(8, 16), universe=cache * rng.randint(2, 4))
    if kind == "rowwise":
        return dict(kind=kind, rows=_log_int(rng, 1e6, 2e7), dim=rng.choice([32, 64, 128 if rng.random() < 0.5 else 16]),
                    batch=_log_int(rng, 2048, 262144), alpha=round(rng.uniform(1.02, 1.2), 3),
                    optim=rng.choice(["adam", "adagrad"]))
    bag_lo = rng.randint(0, 1)
    bag_hi = 1 if rng.random() < 0.4 else _log_int(rng, 2, 100)
    bag_lo = 1 if bag_hi == 1 else bag_lo
    if kind == "sequence":
        bag_lo, bag_hi = 0, _log_int(rng, 5, 100)
    tables = rng.choice([1, 2, 3, 8, 13, 26]) if kind != "hashed" else rng.randint(1, 8)
    if kind == "sequence":
        tables = min(tables, 8)
    if kind == "input":
        bag_hi = min(bag_hi, 20)
        batch = max(1, min(_log_int(rng, 64, 65536), 1_500_000 // (tables * bag_hi)))
        return dict(kind=kind, tables=tables, batch=batch, bag_lo=bag_lo, bag_hi=bag_hi, vocab=_log_int(rng, 1e4, 5e6),
                    alpha=round(rng.uniform(1.02, 1.2), 3), world=rng.choice([2, 3, 4, 8]), unique=rng.random() < 0.6)
    dims = rng.choice(["8", "16", "32", "64", "128", "256", "36", "20", "512"])
    if kind in ("train", "serve") and rng.random() < 0.25:
        dims = rng.choice(["16,64,128", "8,20,36,64", "128,32,18", "64,1024,8"])
    if kind in ("sequence", "hashed"):
        dims = rng.choice(["16", "32", "64", "128"])
    optim = rng.choice(["adagrad", "adam", "sgd"])
    widest = max(int(d) for d in dims.split(","))
    # bounds: ids per step, floats gathered per step, bytes of table state
    batch = _log_int(rng, 16 if kind == "serve" else 128, 65536)
    batch = max(1, min(batch, 4_000_000 // (tables * bag_hi), 200_000_000 // (tables * bag_hi * widest)))
    rows_hi = min(_log_int(rng, 5e3, 2e6), int(8e9 / (tables * widest * 4 * (1 + STATES[optim]))))
    return dict(kind=kind, tables=tables, rows_lo=min(1000, rows_hi), rows_hi=rows_hi, dims=dims, batch=batch,
                bag_lo=bag_lo, bag_hi=bag_hi, alpha=round(rng.uniform(1.02, 1.2), 3),
                pooling="none" if kind == "sequence" else rng.choice(["sum", "sum", "mean"]), optim=optim,
                plan_ahead=kind == "train" and rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ inputs
def _rows(case):
    return table_rows_log_uniform(2025, case["tables"], case["rows_lo"], case["rows_hi"])


def _dims(case):
    d = [int(x) for x in case["dims"].split(",")]
    return [d[i % len(d)] for i in range(case["tables"])]


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _ragged(gen, vocab, batch, lo, hi, alpha, draw_no=0):
    """(ids [N] feature-major, lengths [T, batch], offsets [T * batch + 1], ids per table).  How many ids, and how many
    distinct ones, is the case's: lengths and ids are drawn for the case, then shuffled and shifted by `gen`, so that
    outputs whose size depends on the data have one size."""
    base = _gen(1000 + draw_no)
    lens = torch.randint(lo, hi + 1, (len(vocab), batch), generator=base, device=DEV)
    lens[0, 0] = max(1, lo)  # never an empty step
    per_table = lens.sum(1).tolist()
    lens = lens.gather(1, torch.rand(lens.shape, generator=gen, device=DEV).argsort(1)).contiguous()
    offs = torch.zeros(lens.numel() + 1, dtype=torch.int64, device=DEV)
    offs[1:] = torch.cumsum(lens.view(-1), 0)
    ids = []
    for n, v in zip(per_table, vocab):
        shift = int(torch.randint(0, v, (1,), generator=gen, device=DEV))
        drawn = zipf_ids(base, n, v, alpha, DEV)[torch.randperm(n, generator=gen, device=DEV)]
        ids.append((drawn + shift) % v)
    return torch.cat(ids).contiguous(), lens, offs, per_table


def _module(case, seed, rows=None):
    rows = _rows(case) if rows is None else rows
    module = HybridSplitTableBatchedEmbeddingBagsCodegen(
        list(zip(rows, _dims(case))), optimizer=OPTIM[case["optim"]], pooling_mode=POOL[case["pooling"]], device=DEV,
        learning_rate=0.01, eps=1e-8, beta1=0.9, beta2=0.999,
        initial_accumulator_value=0.1 if case["optim"] == "adagrad" else 0.0, weights_init=(-0.05, 0.05), seed=seed,
        plan_ahead=case["plan_ahead"])
    # the registered operators have one switch for all modules of the process: what this program wants
    torch.ops.recsdk.set_plan_ahead(case["plan_ahead"])
    return module


def _trained(module, out):
    return [out.detach(), module.weights_dev.detach(), *module.get_momentum()]


def prepare(case, seed):
    torch_ops.load()
    return {"kind": case["kind"], "case": dict(case), **_PREPARE[case["kind"]](case, seed)}


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_train(case, seed):
    gen = _gen(seed)
    module = _module(case, seed)
    ids, _, offs, _ = _ragged(gen, _rows(case), case["batch"], case["bag_lo"], case["bag_hi"], case["alpha"])
    grad = torch.randn((case["batch"], sum(_dims(case))), generator=gen, device=DEV)
    return dict(module=module, ids=ids, offs=offs, grad=grad)


def _run_train(s):
    out = s["module"](s["ids"], s["offs"])
    out.backward(s["grad"])
    return _trained(s["module"], out)


def _prepare_sequence(case, seed):
    gen = _gen(seed)
    module = _module(case, seed)
    ids, _, offs, _ = _ragged(gen, _rows(case), case["batch"], case["bag_lo"], case["bag_hi"], case["alpha"])
    length, dim = case["bag_hi"], _dims(case)[0]
    grad = torch.randn((case["tables"] * case["batch"], length, dim), generator=gen, device=DEV)
    return dict(module=module, ids=ids, offs=offs, grad=grad, length=length)


def _run_sequence(s):
    rows = s["module"](s["ids"], s["offs"])
    dense = torch.ops.fbgemm.jagged_to_padded_dense(rows, [s["offs"]], s["length"], 0.0)
    dense.backward(s["grad"])
    return [rows.detach(), *_trained(s["module"], dense)]


def _prepare_serve(case, seed):
    gen = _gen(seed)
    module = _module(case, seed)
    ids, _, offs, _ = _ragged(gen, _rows(case), case["batch"], case["bag_lo"], case["bag_hi"], case["alpha"])
    return dict(module=module, ids=ids, offs=offs)


def _run_serve(s):
    with torch.no_grad():
        return s["module"](s["ids"], s["offs"])


def _key_of(ids):
    """A 62-bit key for every id (odd multiplier: distinct ids keep distinct keys)."""
    return (ids * 0x1E3779B97F4A7C15) & ((1 << 62) - 1)


def _prepare_hashed(case, seed):
    gen = _gen(seed)
    rows = _rows(case)
    module = _module(case, seed, rows)
    mappers = [torch.classes.hybrid.IdsMapper(r, True) for r in rows]
    batches = [_ragged(gen, rows, case["batch"], case["bag_lo"], case["bag_hi"], case["alpha"], k) for k in range(3)]
    s = dict(module=module, mappers=mappers)
    for ids, _, offs, per_table in batches:  # the table has seen two batches before; the third is the case's own
        n = ids.numel()
        s.update(keys=_key_of(ids), offs=offs,
                 table_offs=torch.tensor([0, *np.cumsum(per_table).tolist()], dtype=torch.int64),
                 hash_idx=torch.zeros(n, dtype=torch.int64, device=DEV), uniq=torch.zeros(n, dtype=torch.int64, device=DEV),
                 uniq_keys=torch.zeros(n, dtype=torch.int64, device=DEV), inverse=torch.zeros(n, dtype=torch.int64, device=DEV),
                 uniq_offs=torch.zeros(case["tables"] + 1, dtype=torch.int64, device=DEV))
        if ids is not batches[-1][0]:
            _map_keys(s)
    s["grad"] = torch.randn((case["batch"], sum(_dims(case))), generator=gen, device=DEV)
    return s


def _map_keys(s):
    torch.classes.hybrid.IdsMapper.parallel_ids2indices_unique_out(
        s["mappers"], s["keys"], s["hash_idx"], s["table_offs"], s["uniq"], s["uniq_keys"], s["inverse"], s["uniq_offs"])


def _run_hashed(s):
    _map_keys(s)
    out = s["module"](s["keys"], s["offs"], s["hash_idx"], s["uniq"], s["uniq_offs"], s["inverse"])
    out.backward(s["grad"])
    return [*_trained(s["module"], out), s["hash_idx"], s["uniq"], s["uniq_keys"], s["inverse"], s["uniq_offs"]]


EVICT_IDLE, EVICT_EVERY, WARM_STEPS = 50, 10, 64


def _prepare_dynamic(case, seed):
    gen = _gen(seed)
    n = case["keys"]
    cfg = EmbConfig("dynamic", emb_dim=case["dim"], optim_num=2, cache_size=case["cache"], weight_init_max=1.0,
                    admit_and_evict_config=AdmitAndEvictConfig(2, 0.0, EVICT_IDLE, EVICT_EVERY),
                    filter_capacity=1 << 23)
    module = HybridSplitTableBatchedEmbeddingBagsCodegen(
        [(case["cache"], case["dim"])], optimizer=EmbOptimType.ADAM, pooling_mode=PoolingMode.SUM, device=DEV,
        learning_rate=0.001, eps=1e-8, beta1=0.9, beta2=0.999, weights_init=(-0.01, 0.01), seed=seed)
    torch.ops.recsdk.set_plan_ahead(False)
    pool = torch.randint(0, 1 << 60, (case["pool"],), generator=gen, device=DEV)
    # 30 % of the positions hold a key never seen before, 10 % a key that lives for 16 steps, the others old keys
    base = _gen(1000)  # which positions, and which keys come again, is the case's; the keys are the seed's
    old = pool[torch.randint(0, case["pool"], (4, n), generator=base, device=DEV)]
    kind = torch.rand((n,), generator=base, device=DEV)
    stride = torch.randint(1, 1 << 40, (n,), generator=gen, device=DEV)
    s = dict(mgr=EmbcacheManager([cfg], device=DEV), module=module, n=n, old=[o.contiguous() for o in old],
             span=torch.tensor([0, n]), fresh=torch.where(kind < 0.3, stride, 0), slow=torch.where((kind >= 0.3) & (kind < 0.4), stride, 0), step=0,
             offs=torch.arange(n + 1, dtype=torch.int64, device=DEV),
             grad=torch.randn((n, case["dim"]), generator=gen, device=DEV))
    for _ in range(WARM_STEPS):  # a table in use: keys admitted, idle keys evicted
        _policy_step(s)
    return s


def _policy_step(s):
    mgr, step = s["mgr"], s["step"]
    s["step"] += 1
    keys = torch.add(s["old"][step % 4], s["fresh"], alpha=step).add_(s["slow"], alpha=step // 16)  # the loader's batch
    mgr.record_timestamp(keys, [0, s["n"]], torch.full_like(keys, step))
    if step > 0 and (step + 1) % EVICT_EVERY == 0:
        mgr.evict_features()
        mgr.remove_embedding_table_info()
    mgr.statistics_key_count(keys, s["span"], None, 0)
    uniq, inverse, count = ops.unique_sorted(keys)
    n_uniq = int(count.item())
    info = mgr.compute_swap_info(uniq[:n_uniq], [0, n_uniq])
    return info, info.batch_offs[inverse]


def _run_dynamic(s):
    info, slots = _policy_step(s)
    out = s["module"](slots, s["offs"])
    out.backward(s["grad"])
    return [*_trained(s["module"], out), slots, info.swapin_keys[0], info.swapin_offs, info.swapout_offs]


def _prepare_hybrid(case, seed):
    gen = _gen(seed)
    cfgs = [EmbConfig("table%d" % i, initializer_type=0, emb_dim=case["dim"], optim_num=2, cache_size=case["cache"],
                      weight_init_min=-0.05, weight_init_max=0.05, seed=i) for i in range(case["tables"])]
    bag = HybridCacheEmbeddingBag(cfgs, optimizer=EmbOptimType.ADAM, pooling_mode=PoolingMode.SUM, device=DEV,
                                  learning_rate=0.001, eps=1e-8, beta1=0.9, beta2=0.999)
    torch.ops.recsdk.set_plan_ahead(False)
    n, t = case["keys"], case["tables"]
    s = dict(bag=bag, universe=case["universe"], stride=case["keys"] // 2, step=0,
             base=[zipf_ids(gen, n, case["cache"] // 2, 1.05, DEV) for _ in range(t)],
             offs=torch.arange(t * n + 1, dtype=torch.int64, device=DEV),
             grad=torch.randn((n, t * case["dim"]), generator=gen, device=DEV))
    for _ in range(2 * case["universe"] // max(1, s["stride"])):  # two rounds: the host store holds every row
        _run_hybrid(s)
    return s


def _run_hybrid(s):
    step = s["step"]
    s["step"] += 1
    keys = [torch.remainder(b + step * s["stride"], s["universe"]) for b in s["base"]]  # the loader's batch
    out = s["bag"].forward(keys, s["offs"])
    out.backward(s["grad"])
    return _trained(s["bag"].module, out)


def _prepare_rowwise(case, seed):
    gen = _gen(seed)
    bag = RowWiseShardedEmbeddingBag([case["rows"]], case["dim"], 1, 0, batch_size=case["batch"],
                                     optimizer=OPTIM[case["optim"]], pooling_mode=PoolingMode.SUM, device=DEV,
                                     learning_rate=0.001, eps=1e-8, beta1=0.9, beta2=0.999, weights_init=(-0.01, 0.01),
                                     initial_accumulator_value=0.1 if case["optim"] == "adagrad" else 0.0, seed=seed,
                                     one_hot=True)
    return dict(bag=bag, ids=zipf_ids(gen, case["batch"], case["rows"], case["alpha"], DEV),
                offs=torch.arange(case["batch"] + 1, dtype=torch.int64, device=DEV),
                grad=torch.randn((case["batch"], case["dim"]), generator=gen, device=DEV))


def _run_rowwise(s):
    bag = s["bag"]
    out = bag.forward(s["ids"], s["offs"])
    bag.backward(s["grad"])
    return [out, bag.weights_dev, bag.momentum1_dev, bag.momentum2_dev]


def _prepare_input(case, seed):
    gen = _gen(seed)
    ids, lens, _, per_table = _ragged(gen, [case["vocab"]] * case["tables"], case["batch"], case["bag_lo"], case["bag_hi"],
                                      case["alpha"])
    perm = torch.randperm(case["tables"], generator=gen, device=DEV).to(torch.int32)
    return dict(ids=ids, lens=lens, total=sum(per_table), perm=perm, world=case["world"], unique=case["unique"],
                blocks=torch.full((case["tables"],), -(-case["vocab"] // case["world"]), dtype=torch.int64, device=DEV))


def _run_input(s):
    offs = torch.ops.fbgemm.asynchronous_complete_cumsum(s["lens"].view(-1))
    lens, ids, _ = torch.ops.fbgemm.permute_2D_sparse_data(s["perm"], s["lens"], s["ids"], None, s["total"])
    new_lens, new_ids, _, _, unbucketize, _, counts = torch.ops.hybrid.block_bucketize_sparse_features_cpu(
        lens.view(-1), ids, False, s["unique"], s["blocks"], s["world"], None, None, None, 0, None, False, False,
        s["unique"], s["unique"])
    return [offs, lens, ids, new_lens, new_ids, unbucketize, counts]


_PREPARE = dict(train=_prepare_train, sequence=_prepare_sequence, serve=_prepare_serve, hashed=_prepare_hashed,
                dynamic=_prepare_dynamic, hybrid=_prepare_hybrid, rowwise=_prepare_rowwise, input=_prepare_input)
_RUN = dict(train=_run_train, sequence=_run_sequence, serve=_run_serve, hashed=_run_hashed, dynamic=_run_dynamic,
            hybrid=_run_hybrid, rowwise=_run_rowwise, input=_run_input)


# ------------------------------------------------------------------------------------------------ what a pass needs
def _distinct(n, vocab, alpha):
    """Expected distinct ids of n draws from Zipf(alpha) over [0, vocab): exact head, the tail in geometric bins."""
    head = np.arange(1, min(vocab, 4096) + 1, dtype=np.float64)
    edges = np.unique(np.geomspace(4096, max(vocab, 4096), 2048).astype(np.int64)) if vocab > 4096 else np.array([4096])
    width = np.diff(edges).astype(np.float64)
    mid = edges[:-1] + (width + 1) / 2
    rank, weight = np.concatenate([head, mid]), np.concatenate([np.ones_like(head), width])
    p = rank ** -alpha
    p /= (p * weight).sum()
    return float((weight * -np.expm1(-n * p)).sum())


def _lookup_work(n, bags, uniq_dim, out_floats, row_floats, states):
    """n ids in `bags` bags; uniq_dim: floats in the distinct rows; out_floats: of the output (and of its gradient);
    row_floats: floats gathered."""
    return dict(bytes=8 * n + 8 * (bags + 1) + 8 * out_floats + 8 * uniq_dim * (1 + states),
                flops=2 * row_floats + (2 + 6 * states) * uniq_dim)


def work(case):
    kind = case["kind"]
    if kind == "dynamic":
        n, d = case["keys"], case["dim"]
        uniq = 0.3 * n + _distinct_uniform(0.6 * n, case["pool"]) + _distinct_uniform(0.1 * n, case["pool"])
        w = _lookup_work(n, n, 0.7 * uniq * d, n * d, n * d, 2)
        # per key: the key, its timestamp, a filter entry read and written, unique + inverse, a slot entry, its slot
        return dict(bytes=w["bytes"] + n * (8 + 8 + 64 + 8) + uniq * (8 + 16 + 8), flops=w["flops"])
    if kind == "hybrid":
        n, d, t = case["keys"], case["dim"], case["tables"]
        uniq = t * _distinct(n, case["cache"] // 2, 1.05)
        w = _lookup_work(n * t, n * t, uniq * d, n * t * d, n * t * d, 2)
        # keys, inverse and slots, and the rows that cross to the host and back (half of the distinct ones)
        return dict(bytes=w["bytes"] + n * t * 24 + uniq * 32 + uniq * d * 4 * 3, flops=w["flops"])
    if kind == "rowwise":
        n, d = case["batch"], case["dim"]
        return _lookup_work(n, n, _distinct(n, case["rows"], case["alpha"]) * d, n * d, n * d, STATES[case["optim"]])
    n_mean = (case["bag_lo"] + case["bag_hi"]) / 2 * case["batch"]
    t, bags = case["tables"], case["tables"] * case["batch"]
    if kind == "input":
        n = t * n_mean
        uniq = t * _distinct(n_mean, case["vocab"], case["alpha"]) if case["unique"] else n
        # ids read, permuted and bucketized ids written, the permute; lengths read, permuted and per-bucket written; offsets
        return dict(bytes=8 * (2 * n + 2 * uniq + n) + 8 * bags * (3 + case["world"]), flops=0)
    dims = _dims(case)
    uniq = [_distinct(n_mean, r, case["alpha"]) for r in _rows(case)]
    uniq_dim = sum(u * d for u, d in zip(uniq, dims))
    row_floats = sum(n_mean * d for d in dims)
    if kind == "serve":
        return dict(bytes=8 * t * n_mean + 8 * (bags + 1) + 4 * uniq_dim + 4 * case["batch"] * sum(dims), flops=row_floats)
    if kind == "sequence":
        padded = bags * case["bag_hi"] * dims[0]
        w = _lookup_work(t * n_mean, bags, uniq_dim, row_floats, row_floats, STATES[case["optim"]])
        return dict(bytes=w["bytes"] + 8 * padded, flops=w["flops"])
    w = _lookup_work(t * n_mean, bags, uniq_dim, case["batch"] * sum(dims), row_floats, STATES[case["optim"]])
    if kind == "hashed":
        # key read, slot entry read, slot and inverse written; unique slots and keys written
        w["bytes"] += t * n_mean * (8 + 16 + 8 + 8) + sum(uniq) * 16
    return w


def _distinct_uniform(n, vocab):
    return float(-vocab * np.expm1(-n / vocab))


def tolerance(case):
    if case["kind"] == "input":
        return "exact"
    # against the same pass in 64 bits: pooled rows differ by 2e-7; the squared gradient sums of the hottest rows, which
    # decide the norm of the optimizer state, by 1.6e-6.  Slots, keys and counts are whole numbers and stay the same.
    return {"rel": 8e-7 if case["kind"] == "serve" else 6e-6}
