"""The work that users of this framework have it do on one GPU, as cases that can be timed and compared.

Six kinds of work, each through the calls a program makes:

* ``train``     sparse logistic regression, one minibatch per pass through ``SparseLRWorker.submit``
                (localise, pull + margins, push, optimiser): the workload of ``bench.py`` and of the
                ``async_sgd`` application
* ``evaluate``  forward only: margins of a minibatch against a loaded model (``run_evaluation``)
* ``kv``        ``DeviceKVVector``: push, pull that waits for it, result
* ``layers``    ``DeviceKVLayer``: dense layers pushed, applied and pulled
* ``wide``      a training step with 64-wide bf16 values per key (``WidePlane``)
* ``darlin``    one pass over the data by block coordinate descent (``DarlinRank``)
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from parameter_server_b200.models.darlin import DarlinConfig, DarlinRank, darlin_heap_bytes
from parameter_server_b200.models.sparse_lr import SparseLRConfig, SparseLRWorker
from parameter_server_b200.ops import _lib
from parameter_server_b200.ops.localize import LocalBatch
from parameter_server_b200.parallel.dataplane import DataPlane, OptimizerConfig, PlaneConfig, heap_layout
from parameter_server_b200.parallel.fabric import Fabric
from parameter_server_b200.parallel.wide import WideConfig, WidePlane, wide_layout
from parameter_server_b200.parameter.kv import DeviceKVVector
from parameter_server_b200.parameter.kv_layer import DeviceKVLayer
from parameter_server_b200.utils.idpack import PackedIds, bits_for
from parameter_server_b200.utils.synthetic import gen_batch

ALEXNET = "11616,6400,2556,2304,177209344,16777216,4096000"


def listed():
    return [
        # The headline workload: a 64k-row minibatch of 200 binary features out of 2^26, FTRL, ids on the GPU;
        # the program looks at every minibatch before it submits the next one.
        dict(name="ftrl_64k_rows", kind="train", source="device_ids", rows=65536, nnz=200, features=26, zipf=1.05,
             values=False, ragged=False, algo="ftrl", tau=4, wait=True),
        # The same minibatches as a loader ships them, a bit stream of ids in pinned memory, streamed without waiting.
        dict(name="ftrl_64k_rows_from_host", kind="train", source="host_packed", rows=65536, nnz=200, features=26,
             zipf=1.05, values=False, ragged=False, algo="ftrl", tau=0, wait=False),
        # The async_sgd application at its default minibatch of 1000 rows: hashed 64-bit keys from text, AdaGrad.
        dict(name="adagrad_1000_rows", kind="train", source="host_keys", rows=1000, nnz=64, features=20, zipf=1.1,
             values=False, ragged=False, algo="adagrad", tau=0, wait=False),
        # The application on rows of different lengths with real values; every minibatch has another size.
        dict(name="ftrl_ragged_values", kind="train", source="host_keys", rows=10000, nnz=39, features=22, zipf=1.1,
             values=True, ragged=True, algo="ftrl", tau=0, wait=False),
        # Scoring held-out rows against a trained model, a chunk of 100,000 rows as the application reads them.
        dict(name="evaluate_100k_rows", kind="evaluate", rows=100000, nnz=39, features=22, zipf=1.1, values=True,
             ragged=True, model=1 << 20),
        # A small request: latency of one push and the pull that follows it.
        dict(name="kv_1k", kind="kv", keys=1000, width=1, mode="none"),
        # A worker that trains on one fixed feature set: the key list repeats and the key-caching filter is on.
        dict(name="kv_1m_w8_key_caching", kind="kv", keys=1000000, width=8, mode="key_caching"),
        # Embedding-like rows with the fixed-point filter; an odd number of keys.
        dict(name="kv_262k_w64_int8", kind="kv", keys=262145, width=64, mode="int8"),
        # The largest request of the key/value probe.
        dict(name="kv_16m", kind="kv", keys=16000000, width=1, mode="none"),
        # The dense layers of the layer probe (AlexNet): four of a few KB, three of 16 to 709 MB.
        dict(name="layers_alexnet", kind="layers", sizes=ALEXNET, updater="add"),
        # The wide-value model: 32k rows of 40 keys, 64 contexts, AdaGrad on the owner.
        dict(name="wide_32k_rows", kind="wide", rows=32768, nnz=40, features=24, zipf=1.2, contexts=64),
        # L1 logistic regression by block coordinate descent: 256 feature blocks one after another, real values. (With
        # a bounded delay the blocks overlap, and two runs on the same data do not give the same weights.)
        dict(name="darlin_1m25_rows", kind="darlin", rows=1250000, nnz=100, features=24, zipf=1.1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "evaluate", "kv", "kv", "kv", "layers", "wide", "darlin"])
    if kind == "train":
        source = rng.choice(["device_ids", "host_packed", "host_keys"])
        rows, nnz = _log(rng, 500, 65536), _log(rng, 8, 200)
        values = source == "host_keys" and rng.random() < 0.5
        if source == "host_keys":
            rows = min(rows, 20000)
        wait = source == "device_ids"
        return dict(kind=kind, source=source, rows=rows, nnz=nnz, features=rng.randint(20, 26),
                    zipf=round(rng.uniform(1.02, 1.2), 3), values=values,
                    ragged=source == "host_keys" and rng.random() < 0.7, algo=rng.choice(["ftrl", "adagrad", "sgd"]),
                    tau=rng.randint(0, 8) if wait else 0, wait=wait)
    if kind == "evaluate":
        return dict(kind=kind, rows=_log(rng, 2000, 100000), nnz=_log(rng, 8, 80), features=rng.randint(20, 24),
                    zipf=round(rng.uniform(1.02, 1.2), 3), values=rng.random() < 0.5, ragged=True,
                    model=_log(rng, 1 << 16, 1 << 21))
    if kind == "kv":
        width = rng.choice([1, 1, 8, 64, 3])
        mode = rng.choice(["none", "key_caching", "int8", "fp16"])
        return dict(kind=kind, keys=_log(rng, 1000, 16000000 // (width if width < 64 else 32)), width=width, mode=mode)
    if kind == "layers":
        sizes = [_log(rng, 100, 20000000) for _ in range(rng.randint(1, 7))]
        return dict(kind=kind, sizes=",".join(map(str, sizes)), updater=rng.choice(["add", "assign", "sgd"]))
    if kind == "wide":
        return dict(kind=kind, rows=_log(rng, 1000, 32768), nnz=rng.randint(10, 60), features=rng.randint(20, 24),
                    zipf=round(rng.uniform(1.05, 1.3), 3), contexts=rng.choice([64, 128]))
    return dict(kind=kind, rows=_log(rng, 50000, 1250000), nnz=rng.randint(20, 100), features=rng.randint(20, 24),
                zipf=round(rng.uniform(1.05, 1.2), 3))


# ------------------------------------------------------------------ inputs
class State:
    """What a program keeps between calls."""


def _release(bases):
    torch.cuda.synchronize()
    for p in bases:
        _lib.lib().psb_heap_free(p)


def _heap(nbytes):
    """A one-GPU symmetric heap that is given back when nothing refers to it any more."""
    fab = Fabric.single(nbytes)
    weakref.finalize(fab, _release, list(fab.bases))
    return fab


def _pow2(n):
    return 1 << max(0, int(n) - 1).bit_length()


def _hash(ids, bits=64):
    """Feature ids (int64, on the GPU) to uint64 keys; ``bits`` significant bits at the top."""
    keys = torch.empty_like(ids)
    _lib.check(_lib.lib().psb_hash_ids(0, _lib.ptr(ids), _lib.ptr(keys), ids.numel(), (bits % 64) << 56, _lib.stream_ptr()), "hash")
    return keys


def _rows(case, seed, batch, ids64):
    """(ids, y, vals or None, row_ptr or None) on the GPU. Ragged rows have 1 to 2 * nnz - 1 nonzeros."""
    r, z = case["rows"], case["nnz"]
    zz = 2 * z - 1 if case.get("ragged") else z
    ids, y, vals = gen_batch(r, zz, 1 << case["features"], case["zipf"], seed=seed, batch=batch, ids64=ids64,
                             real_values=bool(case.get("values")))
    if not case.get("ragged"):
        return ids, y, vals, None
    g = torch.Generator(device="cuda").manual_seed(seed * 31 + batch)
    n = torch.randint(1, 2 * z, ((r + 1) // 2,), device="cuda", generator=g)
    n = torch.cat([n, 2 * z - n])[:r]            # r * nnz nonzeros in all, whatever the seed
    keep = (torch.arange(zz, device="cuda")[None, :] < n[:, None]).flatten()
    rp = torch.zeros(r + 1, dtype=torch.int32, device="cuda")
    rp[1:] = torch.cumsum(n, 0)
    return ids[keep], y, None if vals is None else vals[keep], rp


def _fix_unique(ids, case):
    """The number of different ids in a minibatch is made the same for every seed, three per cent below what the
    law gives on average: the rest of the rare ones become the most frequent id."""
    want = int(0.97 * _unique(case["rows"] * case["nnz"], case["features"], case["zipf"]))
    uniq, inverse, count = torch.unique(ids, return_inverse=True, return_counts=True)
    drop = torch.sort(count, stable=True)[1][:max(0, uniq.numel() - want)]
    uniq[drop] = 0
    return uniq[inverse]


def _first_places(keys):
    """Sorted positions at which a key of the list appears for the first time: the number of them below n
    is the number of unique keys among the first n."""
    _, inverse = torch.unique(keys, return_inverse=True)
    first = torch.full((int(inverse.max()) + 1,), keys.numel(), dtype=torch.int64, device=keys.device)
    first.scatter_reduce_(0, inverse, torch.arange(keys.numel(), device=keys.device), "amin")
    return torch.sort(first)[0]


def _prepare_train(case, seed):
    s = State()
    rows, z, src = case["rows"], case["nnz"], case["source"]
    nnz = rows * (2 * z - 1 if case["ragged"] else z)
    opt = {"ftrl": OptimizerConfig(algo="ftrl", alpha=0.1, beta=1.0, l1=1.0, l2=0.1),
           "adagrad": OptimizerConfig(algo="adagrad", alpha=0.1, beta=1.0, l1=0.0, l2=0.01),
           "sgd": OptimizerConfig(algo="sgd", alpha=0.1, beta=1.0, l1=0.0, l2=0.01)}[case["algo"]]
    app = src == "host_keys"                     # the application: keys hashed by the parser, no ordered slots
    cap = _pow2(2 << case["features"])
    pc = PlaneConfig(table_capacity=cap, inbox_cap=nnz, ring=case["tau"] + 2, pull_cap=nnz, ordered_slots=not app)
    s.plane = DataPlane(_heap(heap_layout(pc, 1).total()), pc, opt)
    s.worker = SparseLRWorker(s.plane, SparseLRConfig(
        max_rows=rows, max_nnz=nnz, tau=case["tau"], hash_seed=None if app else 0, hash_bits=0 if app else 40,
        pipeline=2 if app else 3, auc=app, real_values=case["values"]))
    s.pool, s.i, s.wait = [], 0, case["wait"]
    for k in range(4):                           # two minibatches trained on before, two that the passes use in turn
        ids, y, vals, rp = _rows(case, seed, k, ids64=app)
        ids = _fix_unique(ids, case)
        keys = _hash(ids) if app else ids
        if app and rp is None:
            rp = torch.arange(rows + 1, dtype=torch.int32, device="cuda") * z
        if k < 2:
            s.worker.step(keys, y, fixed_z=0 if app else z, row_ptr=rp, vals=vals)
            continue
        places = _first_places(keys)
        if case["ragged"]:
            # the loader's minibatches vary in size: a pass takes the first n rows, another n every time
            n_rows = [rows - (7 * j) % min(251, rows // 2) for j in range(251)]
        else:
            n_rows = [rows]
        ends = [nnz] if rp is None else rp[torch.tensor(n_rows, device="cuda")].tolist()
        unique = torch.searchsorted(places, torch.tensor(ends, device="cuda")).tolist()
        b = dict(sizes=list(zip(n_rows, ends, unique)), z=0 if app else z)
        if src == "device_ids":
            b.update(ids=ids, y=y)
        elif src == "host_packed":
            b.update(ids=PackedIds.from_ids(ids, bits_for((1 << case["features"]) - 1)), y=y.cpu().pin_memory())
        else:
            b.update(ids=keys.cpu().pin_memory(), y=y.cpu().pin_memory(), rp=rp.cpu().pin_memory(),
                     vals=None if vals is None else vals.cpu().pin_memory())
        s.pool.append(b)
    return s


def _run_train(s):
    m = s.pool[s.i % len(s.pool)]
    rows, nnz, unique = m["sizes"][s.i % len(m["sizes"])]
    s.i += 1
    if "rp" in m:
        b = s.worker.submit(m["ids"][:nnz], m["y"][:rows], row_ptr=m["rp"][:rows + 1],
                            vals=None if m["vals"] is None else m["vals"][:nnz])
    else:
        b = s.worker.submit(m["ids"], m["y"], fixed_z=m["z"])
    if s.wait:
        s.worker.wait()
    return {"keys": b.ukeys[:unique], "gradient": b.grad[:unique], "margin": b.margin[:rows]}


def _prepare_evaluate(case, seed):
    s = State()
    cap = _pow2(2 * case["model"])
    pc = PlaneConfig(table_capacity=cap, inbox_cap=16, ring=2)
    s.plane = DataPlane(_heap(heap_layout(pc, 1).total()), pc, OptimizerConfig())
    g = torch.Generator(device="cuda").manual_seed(seed)
    model_keys = _hash(torch.arange(case["model"], dtype=torch.int64, device="cuda"))
    s.plane.load_state(model_keys.cpu().numpy().view(np.uint64),
                       w=torch.randn(case["model"], device="cuda", generator=g) * 0.1)
    s.pool, s.i = [], 0
    for k in range(2):
        ids, y, vals, rp = _rows(case, seed, k, ids64=True)
        s.pool.append((_hash(ids), y, rp, vals))
    s.rows = case["rows"]
    s.worker = SparseLRWorker(s.plane, SparseLRConfig(max_rows=s.rows, max_nnz=s.rows * (2 * case["nnz"] - 1),
                                                      hash_seed=None, pipeline=1, real_values=True))
    return s


def _run_evaluate(s):
    keys, y, rp, vals = s.pool[s.i % len(s.pool)]
    s.i += 1
    b = s.worker.prepare(keys, y, row_ptr=rp, vals=vals)
    s.plane.pull_margin(b)
    return b.margin[:s.rows]


def _prepare_kv(case, seed):
    s = State()
    n, k, mode = case["keys"], case["width"], case["mode"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s.pool, s.i = [], 0
    for _ in range(1 if mode == "key_caching" else 2):
        keys = torch.unique(torch.randint(0, 1 << 40, (n + n // 20 + 64,), device="cuda", generator=g))
        keys = torch.sort(keys[torch.randperm(keys.numel(), device="cuda", generator=g)[:n]])[0]
        s.pool.append((keys, torch.randn(n, k, device="cuda", generator=g)))
    pc = PlaneConfig(table_capacity=max(4096, _pow2(4 * n)), inbox_cap=n, ring=4, pull_cap=n, width=k,
                     quant=mode if mode in ("int8", "fp16") else "none", key_cache=mode == "key_caching")
    s.kv = DeviceKVVector.create(_heap(heap_layout(pc, 1).total()), table_capacity=pc.table_capacity, max_keys=n,
                                 quant=pc.quant, k=k, key_cache=pc.key_cache)
    return s


def _run_kv(s):
    keys, vals = s.pool[s.i % len(s.pool)]
    s.i += 1
    pushed = s.kv.push(keys, vals)
    pulled = s.kv.pull(keys, wait=[pushed])
    s.kv.wait(pulled)
    s.kv.discard(pushed)
    return s.kv.result(pulled)


def _sizes(case):
    return [int(x) for x in case["sizes"].split(",")]


def _prepare_layers(case, seed):
    s = State()
    layers = dict(enumerate(_sizes(case)))
    s.kv = DeviceKVLayer(_heap(DeviceKVLayer.heap_bytes(layers, 1)), layers, updater=case["updater"], lr=0.1)
    g = torch.Generator(device="cuda").manual_seed(seed)
    s.data = [torch.randn(n, device="cuda", generator=g) for n in layers.values()]
    s.out = [torch.empty(n, device="cuda") for n in layers.values()]
    s.rounds = 0
    for lid in layers:
        s.kv.segment(lid).zero_()
    return s


def _run_layers(s):
    s.rounds += 1
    for lid, (data, out) in enumerate(zip(s.data, s.out)):
        s.kv.push(lid, data)
        s.kv.apply(lid)
        s.kv.pull(lid, out, wait_for_round=s.rounds)
    return s.out


def _prepare_wide(case, seed):
    s = State()
    rows, z, n_ctx = case["rows"], case["nnz"], case["contexts"]
    cfg = WideConfig(table_capacity=_pow2(2 << case["features"]), inbox_cap=rows * z, ring=10, pull_cap=rows * z)
    s.plane = WidePlane(_heap(wide_layout(cfg, 1).total()), cfg)
    s.bufs = [LocalBatch(rows, rows * z, 1, "cuda") for _ in range(2)]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s.pool, s.z, s.i, s.n_ctx = [], z, 0, n_ctx
    for k in range(2):
        ids, y, _ = gen_batch(rows, z, 1 << case["features"], case["zipf"], seed=seed, batch=k)
        ids = _fix_unique(ids, case)
        b = s.bufs[k].localize(ids, y, s.plane.bounds, fixed_z=z, hash_seed=0, hash_bits=40)
        u = int(b.n_unique.item())
        s.plane.load(b.ukeys[:u].cpu().numpy().view(np.uint64), torch.randn(u, 64, device="cuda", generator=g) * 0.1)
        s.pool.append((ids, y, u))
    s.ctx = (torch.randn(n_ctx, 64, device="cuda", generator=g) * 0.3).to(torch.bfloat16)
    s.products = torch.zeros(rows * z, n_ctx, device="cuda")
    return s


def _run_wide(s):
    ids, y, unique = s.pool[s.i % 2]
    b = s.bufs[s.i % 2].localize(ids, y, s.plane.bounds, fixed_z=s.z, hash_seed=0, hash_bits=40)
    s.plane.pull_xgemm(b, s.ctx, s.products, s.i)
    s.plane.rowsum(b, s.products, s.n_ctx)
    s.plane.push(b, s.ctx, s.i)
    s.plane.apply(s.i)
    rows = s.plane.pulled_rows(s.i, unique)
    s.i += 1
    return {"rows": rows, "products": s.products[:unique], "margin": b.margin[:b.n_rows], "gcoef": b.gcoef[:b.n_rows]}


def _prepare_darlin(case, seed):
    s = State()
    nf = 1 << case["features"]
    ids, y, vals = gen_batch(case["rows"], case["nnz"], nf, case["zipf"], seed=seed, batch=0, ids64=True, real_values=True)
    keys = _hash(ids, 40)
    sign = -(1 << 63)                            # signed order of (k ^ sign) is the unsigned order of k
    every = torch.sort(_hash(torch.arange(nf, dtype=torch.int64, device="cuda"), 40) ^ sign)[0] ^ sign
    cfg = DarlinConfig(lambda_l1=1.0, eta=0.9, block_cols=1 << 16)
    s.r = DarlinRank(_heap(darlin_heap_bytes(cfg, 1)), cfg, keys, y, fixed_z=case["nnz"], vals=vals, global_keys=every)
    s.it, s.ts = 0, 0
    _run_darlin(s)                               # the passes measured are the ones after the first
    return s


def _run_darlin(s):
    r = s.r
    order = list(range(len(r.blocks)))
    np.random.default_rng(1000 + s.it).shuffle(order)
    r.run_pass(order, s.ts, r.cfg.tau)
    s.it += 1
    s.ts += len(order)
    progress = r.evaluate()
    r.kkt_threshold = progress[4] / max(1, r.n_rows) * r.cfg.kkt_ratio
    return {"progress": progress[:2], "weights": r.w_cur[:r.n_cols], "margin": r.margin}


def prepare(case, seed):
    make, state_run = _KINDS[case["kind"]]
    state = make(case, seed)
    state.run = state_run
    return state


def run(state):
    return state.run(state)


_KINDS = {"train": (_prepare_train, _run_train), "evaluate": (_prepare_evaluate, _run_evaluate), "kv": (_prepare_kv, _run_kv),
          "layers": (_prepare_layers, _run_layers), "wide": (_prepare_wide, _run_wide), "darlin": (_prepare_darlin, _run_darlin)}


# ------------------------------------------------------------------ what a pass cannot do without
def _unique(nnz, features, s):
    """Expected number of different ids among ``nnz`` draws from the Zipf-like law over 2^features ids."""
    n = 1 << features
    edges = np.unique(np.round(np.exp(np.linspace(0, math.log(n + 1), 4000))))
    a, b = edges[:-1], edges[1:]
    p = (b ** (1 - s) - a ** (1 - s)) / ((n + 1.0) ** (1 - s) - 1)          # of the ids a .. b - 1 together
    each = p / (b - a)
    return float(np.sum((b - a) * -np.expm1(nnz * np.log1p(-np.minimum(each, 0.999999)))))


def work(case):
    kind = case["kind"]
    if kind == "kv":
        # in: keys and values; the table's keys read, its values read and written; out: values
        n, k = case["keys"], case["width"]
        return {"bytes": n * (16 + 16 * k), "flops": n * k}
    if kind == "layers":
        # in: the pushed layer; state read and written; out: the pulled layer
        n = sum(_sizes(case))
        return {"bytes": 16 * n, "flops": n}
    rows, nnz = case["rows"], case["rows"] * case["nnz"]
    u = _unique(nnz, case["features"], case["zipf"])
    if kind == "train":
        id_bytes = {"device_ids": 4, "host_packed": case["features"] / 8, "host_keys": 8}[case["source"]]
        # in: ids (and values), labels; per unique key: key, weight and two state words read, the three written,
        # key and gradient out; margins out
        return {"bytes": nnz * (id_bytes + 4 * case["values"]) + rows * 12 + u * (8 + 12 + 12 + 12), "flops": 4 * nnz + 12 * u}
    if kind == "evaluate":
        return {"bytes": nnz * (8 + 4 * case["values"]) + rows * 12 + u * 12, "flops": 2 * nnz}
    if kind == "wide":
        # in: ids, labels; per unique key: key, row (bf16) and accumulators (fp32) read and written, the pulled row
        # and the row of products out; margins and coefficients out
        n_ctx = case["contexts"]
        return {"bytes": nnz * 4 + rows * 12 + u * (8 + 2 * 128 + 2 * 256 + 128 + 4 * n_ctx),
                "flops": 2 * u * 64 * n_ctx + 2 * nnz * 64 + nnz}
    # darlin: row, value and column of every nonzero; labels and margins; per column weight, trust region and active flag
    return {"bytes": nnz * 10 + rows * 12 + (1 << case["features"]) * 18, "flops": 12 * nnz}


def tolerance(case):
    """About four times what two runs on the same inputs, or sums in another order, were seen to differ by."""
    kind = case["kind"]
    if kind == "kv":
        # plain sums are one addition per push; a block-scaled code may be rounded the other way where it lies between two
        return {"rel": 1e-4, "max": 0.05} if case["mode"] in ("int8", "fp16") else {"rel": 1e-6}
    if kind in ("evaluate", "layers"):
        return {"rel": 2e-6}
    if kind == "wide":
        # 32-bit sums in varying order, rounded to bf16: now and then a weight moves by one bf16 step
        return {"rel": 1e-4, "max": 0.03}
    if kind == "darlin":
        # 32-bit sums in varying order; a weight close to the soft threshold moves by more than the rest
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-5}                         # 32-bit sums in varying order


# ------------------------------------------------------------------ the same results in 64 bits
def _uindex(keys_list):
    """Sorted (as unsigned numbers) different keys of the lists, and every list as indices into them."""
    sign = -(1 << 63)
    u, inv = torch.unique(torch.cat(keys_list) ^ sign, return_inverse=True)
    return u ^ sign, torch.split(inv, [k.numel() for k in keys_list])


def _row_sums(x, rp, z, rows):
    if rp is None:
        return x.view(rows, z).sum(1)
    row = torch.repeat_interleave(torch.arange(rows, device=x.device), (rp[1:] - rp[:-1]).long())
    return torch.zeros(rows, dtype=torch.float64, device=x.device).index_add_(0, row, x)


def _exact_train(case, seed):
    rows, z, app, algo = case["rows"], case["nnz"], case["source"] == "host_keys", case["algo"]
    batches = []
    for k in range(3):
        ids, y, vals, rp = _rows(case, seed, k, ids64=app)
        ids = _fix_unique(ids, case)
        batches.append((_hash(ids) if app else _hash(ids.long(), 40), y.double(), None if vals is None else vals.double(), rp))
    u, index = _uindex([b[0] for b in batches])
    w, s0, s1 = (torch.zeros(u.numel(), dtype=torch.float64, device="cuda") for _ in range(3))
    alpha, beta, l1, l2 = (0.1, 1.0, 1.0, 0.1) if algo == "ftrl" else (0.1, 1.0, 0.0, 0.01)
    for at, (_, y, vals, rp) in zip(index, batches):
        margin = _row_sums(w[at] if vals is None else w[at] * vals, rp, z, rows)
        coef = -y * torch.sigmoid(-y * margin)
        coef = coef.repeat_interleave(z) if rp is None else torch.repeat_interleave(coef, (rp[1:] - rp[:-1]).long())
        g = torch.zeros_like(w).index_add_(0, at, coef if vals is None else coef * vals)
        mine = torch.unique(at)
        gm, wm, am, bm = g[mine], w[mine], s0[mine], s1[mine]
        if algo == "ftrl":
            n = torch.sqrt(bm * bm + gm * gm)
            am, bm = am + gm - (n - bm) / alpha * wm, n
            eta = alpha / (n + beta)
            step = -am * eta
        else:
            am = am + (gm * gm if algo == "adagrad" else 1.0)
            eta = alpha / (torch.sqrt(am) + beta)
            step = wm - eta * gm
        w[mine] = torch.sign(step) * (step.abs() - l1 * eta).clamp(min=0) / (1 + l2 * eta)
        s0[mine], s1[mine] = am, bm
    return {"keys": u[mine], "gradient": gm, "margin": margin}


def _exact_evaluate(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    model = _hash(torch.arange(case["model"], dtype=torch.int64, device="cuda"))
    weights = (torch.randn(case["model"], device="cuda", generator=g) * 0.1).double()
    ids, _, vals, rp = _rows(case, seed, 0, ids64=True)
    u, (mine, at) = _uindex([model, _hash(ids)])
    w = torch.zeros(u.numel(), dtype=torch.float64, device="cuda")
    w[mine] = weights
    return _row_sums(w[at] if vals is None else w[at] * vals.double(), rp, case["nnz"], case["rows"])


def exact(case, seed):
    """What the first pass on ``prepare(case, seed)`` returns, in 64 bits."""
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "evaluate":
        return _exact_evaluate(case, seed)
    if kind == "kv":                             # one push into an empty table, pulled back
        n, g = case["keys"], torch.Generator(device="cuda").manual_seed(seed)
        keys = torch.unique(torch.randint(0, 1 << 40, (n + n // 20 + 64,), device="cuda", generator=g))
        torch.randperm(keys.numel(), device="cuda", generator=g)
        values = torch.randn(n, case["width"], device="cuda", generator=g).double()
        return values if case["width"] > 1 else values.flatten()
    if kind == "layers":                         # one push into zeros
        g = torch.Generator(device="cuda").manual_seed(seed)
        return [torch.randn(n, device="cuda", generator=g).double() * (-0.1 if case["updater"] == "sgd" else 1.0)
                for n in _sizes(case)]
    return None                                  # wide: bf16 state rounded on the way; darlin: 512 dependent blocks
