"""Performance cases: what a program that uses this framework has it do, through its public entry points.

Four kinds of pass, all on one GPU:

* ``train``    ``Model.fit`` over a few batches in pinned host memory, every step's loss read back;
* ``predict``  ``Model.predict`` over a few batches in pinned host memory;
* ``serve``    ``InferenceEngine.infer`` on one request and its probabilities back on the host;
* ``embed``    an ``EmbeddingFeatures`` layer on its own: forward, backward, sparse update (a custom training loop).

Ids are Zipf(1.05) ranks over 2^40 per slot, ranks beyond the resident signs of a slot folded onto them, hashed to
64 bits; every sign has its row before anything is measured, as in the steady state of a long job.
"""
from __future__ import annotations

import gc
import math
import weakref

import numpy as np
import torch

import tensornet_b200 as tn
from tensornet_b200.layers import DenseHead, EmbeddingFeatures, MLP
from tensornet_b200.serving import EmbeddingDictionary, InferenceEngine

_ODD = -7046029254386353131          # odd: x -> x * _ODD is a bijection on 2^64


# ------------------------------------------------------------------------------------------------------------- cases
def listed():
    """``bags``: mean number of ids per slot and example (1: exactly one id; above: Poisson, at least one, ragged).
    ``rows``: signs with a row in the table.  ``form``: one packed buffer per batch, or one tensor per slot.
    ``losses``: the loss of every step is read back, not only the last one of the pass."""
    return [
        # one request of a ranking service: latency is everything
        dict(name="serve one", do="serve", batch=1, slots=200, dim=32, hidden="1024-512-256", bags=1, rows=2_000_000),
        # a request batch of the serving benchmark
        dict(name="serve 512", do="serve", batch=512, slots=200, dim=32, hidden="1024-512-256", bags=1, rows=2_000_000),
        # multi-hot requests: ids with bag offsets, mean pooling
        dict(name="serve multi-hot", do="serve", batch=333, slots=100, dim=32, hidden="1024-512-256", bags=5, rows=2_000_000),
        # the quick-start tutorial's Wide&Deep: tiny batches, ragged slots, batch norm: launches and host time count
        dict(name="wide&deep 32", do="train", model="wide_deep", batch=32, slots=4, dim=8, dense=0, hidden="512-256-256",
             sparse="adagrad", bags=2, cvm=False, shared=False, form="packed", rows=400_000, steps=32, losses=True),
        # a small Wide&Deep job whose reader hands over one tensor per slot
        dict(name="wide&deep 1024", do="train", model="wide_deep", batch=1024, slots=10, dim=8, dense=4, hidden="64-32",
             sparse="adagrad", bags=1, cvm=False, shared=False, form="columns", rows=2_000_000, steps=16, losses=False),
        # the headline job: DeepFM, 26 single-hot slots, sparse Adam
        dict(name="deepfm 8192", do="train", model="deepfm", batch=8192, slots=26, dim=16, dense=13, hidden="400-400-400",
             sparse="adam", bags=1, cvm=False, shared=True, form="packed", rows=20_000_000, steps=16, losses=True),
        # sizes nobody tuned for: odd batch, dim that is no multiple of four, separate AdaGrad tables
        dict(name="deepfm odd", do="train", model="deepfm", batch=2999, slots=39, dim=10, dense=5, hidden="300-150-75",
             sparse="adagrad", bags=1, cvm=False, shared=False, form="packed", rows=4_000_000, steps=8, losses=False),
        # multi-hot Deep&Cross with show / click columns, as the example driver builds it
        dict(name="deep&cross 4096", do="train", model="deep_cross", batch=4096, slots=20, dim=8, dense=0, hidden="512-256-256",
             sparse="adagrad", bags=3, cvm=True, shared=False, form="packed", rows=4_000_000, steps=8, losses=False),
        # multi-hot DCN-v2: 4 M ids per step, FTRL, cross layers 6413 wide: the largest step there is
        dict(name="dcn-v2 8192", do="train", model="dcn_v2", batch=8192, slots=100, dim=64, dense=13, hidden="1024-512-256",
             sparse="ftrl", bags=5, cvm=False, shared=False, form="packed", rows=8_000_000, steps=2, losses=False),
        # scoring a day's data with the headline model
        dict(name="predict 8192", do="predict", model="deepfm", batch=8192, slots=26, dim=16, dense=13, hidden="400-400-400",
             sparse="adam", bags=1, cvm=False, shared=True, form="packed", rows=20_000_000, steps=8),
        # the sparse exchange on its own, short rows and a small batch
        dict(name="embed 64K x 8", do="embed", batch=8192, slots=8, dim=8, sparse="adagrad", bags=1, rows=4_000_000),
        # and long rows with many ids per step
        dict(name="embed 2M x 128", do="embed", batch=65536, slots=32, dim=128, sparse="adagrad", bags=1, rows=8_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: batch 1 to 1024 when serving, 32 to 16384 when training or scoring, up to 2 M
    ids per step through an embedding layer, single- and multi-hot, every model, optimizer and input form."""
    do = rng.choice(["serve", "train", "train", "train", "predict", "embed"])
    if do == "serve":
        bags = rng.choice([1, 1, 2, 5])
        slots = _log(rng, 16, 200 if bags < 5 else 120)
        return dict(do=do, batch=_log(rng, 1, 1024), slots=slots, dim=rng.choice([8, 16, 32]), bags=bags,
                    hidden=rng.choice(["256-128", "512-256-128", "1024-512-256"]), rows=_log(rng, 200_000, 2_000_000))
    if do == "embed":
        ids, slots, bags = _log(rng, 20_000, 2_000_000), _log(rng, 4, 64), rng.choice([1, 1, 3])
        return dict(do=do, batch=max(1, ids // (slots * bags)), slots=slots, dim=rng.choice([8, 10, 16, 32, 64, 128]),
                    sparse=rng.choice(["adagrad", "adam", "ftrl"]), bags=bags, rows=_log(rng, 500_000, 4_000_000))
    model = rng.choice(["wide_deep", "deepfm", "deepfm", "deep_cross", "dcn_v2"])
    batch, dim = _log(rng, 32, 16384), rng.choice([8, 8, 10, 16, 32])
    slots = _log(rng, 4, 48)
    bags = rng.choice([1, 1, 3])
    sparse = "adagrad" if model == "wide_deep" else rng.choice(["adagrad", "adagrad", "adam", "ftrl"])     # as the tutorial has it
    cvm = sparse == "adagrad" and rng.random() < 0.3
    shared = model == "deepfm" and sparse != "adagrad" and not cvm and rng.random() < 0.5
    form = rng.choice(["packed", "packed", "columns"])
    case = dict(do=do, model=model, batch=batch, slots=slots, dim=dim, dense=rng.choice([0, 4, 13]),
                hidden=rng.choice(["64-32", "128-128", "300-150-75", "400-400-400", "512-256-256"]), sparse=sparse, bags=bags,
                cvm=cvm, shared=shared, form=form, rows=_log(rng, 400_000, 4_000_000), steps=32 if batch < 512 else 8)
    if do == "train":
        case["losses"] = form == "packed" and rng.random() < 0.5
    return case


# ------------------------------------------------------------------------------------------------------------- inputs
def _zipf_signs(gen, n, slot, per_slot, dev):
    """``n`` signs; ``slot``: int64 tensor of ``n`` slot numbers."""
    u = torch.rand(n, generator=gen, device=dev, dtype=torch.float64)
    x = torch.floor((1.0 - 0.75 * u) ** -20.0).to(torch.int64).clamp_(1, 1 << 40)      # Zipf(1.05) over [1, 2^40]
    folded = (((x * _ODD) >> 20) & ((1 << 40) - 1)) % per_slot + 1
    return _sign(torch.where(x > per_slot, folded, x), slot)


def _sign(rank, slot):
    return (rank + ((slot + 1) << 42)) * _ODD


def _ids(case, gen, dev):
    """``(ids [S, B], None)`` or ``(values [nnz], offsets [S * B + 1])``, slot after slot."""
    S, B = case["slots"], case["batch"]
    per_slot = _per_slot(case)
    if case["bags"] == 1:
        slot = torch.arange(S, device=dev).repeat_interleave(B)
        return _zipf_signs(gen, S * B, slot, per_slot, dev).view(S, B), None
    mean = torch.full((S * B,), float(case["bags"]), device=dev)
    lens = torch.poisson(mean, generator=gen).clamp_(1, 3 * case["bags"]).to(torch.int64)
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64, device=dev), lens.cumsum(0)])
    slot = torch.arange(S * B, device=dev).repeat_interleave(lens) // B
    return _zipf_signs(gen, int(slot.numel()), slot, per_slot, dev), offsets.to(torch.int32)


def _per_slot(case):
    return max(1, case["rows"] // case["slots"])


def _bucket(case):
    """Bound on the distinct ids of one slot in one batch, with room for the spread of the bag lengths."""
    return case["batch"] if case["bags"] == 1 else int(case["batch"] * case["bags"] * 1.2) + 64


def _batch(case, gen, dev):
    """One batch in pinned host memory, as a reader hands it over: (features, labels)."""
    B, slots = case["batch"], _slots(case)
    ids, offsets = _ids(case, gen, dev)
    y = (torch.rand(B, generator=gen, device=dev) < 0.25).float().cpu().pin_memory()
    if case["form"] == "packed":
        host = ids.cpu().pin_memory()
        if offsets is None:
            f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=host)}
        else:
            f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, values=host, offsets=offsets.cpu().pin_memory(), batch_size=B)}
    elif offsets is None:
        f = {s: ids[k].cpu().pin_memory() for k, s in enumerate(slots)}
    else:
        host, off = ids.cpu(), offsets.cpu()
        f = {}
        for k, s in enumerate(slots):
            o = off[k * B: (k + 1) * B + 1]
            f[s] = tn.data.Ragged(host[int(o[0]): int(o[-1])].pin_memory(), (o - o[0]).pin_memory())
    if case["dense"]:
        f["dense"] = torch.log1p(torch.empty((B, case["dense"]), device=dev).exponential_(1.0, generator=gen)).cpu().pin_memory()
    if case["cvm"]:
        f["label"] = y
    return f, y


def _slots(case):
    return [str(i + 1) for i in range(case["slots"])]


# ------------------------------------------------------------------------------------------------------------- state
class _State:
    """What a program holds before a pass.  The framework's registries keep every table for the life of the process;
    the tables of a state that is gone are taken out of them, so that states can be made one after the other."""

    def __init__(self, case):
        self.case = case
        core = tn.core
        at = (len(core._sparse_tables), len(core._dense_tables), len(core._bn_tables))
        weakref.finalize(self, _State._forget, at, self.__dict__.setdefault("_upto", []))

    def built(self):
        core = tn.core
        self._upto[:] = [len(core._sparse_tables), len(core._dense_tables), len(core._bn_tables)]

    @staticmethod
    def _forget(at, upto):
        core = tn.core
        for reg, lo, hi in zip((core._sparse_tables, core._dense_tables, core._bn_tables), at, upto):
            for k in range(lo, min(hi, len(reg))):
                reg[k] = None


def _sparse_opt(kind):
    core = tn.core
    if kind == "adam":
        return core.Adam(learning_rate=2e-4, initial_scale=0.1)
    if kind == "ftrl":
        return core.Ftrl(learning_rate=5.0, lambda1=1e-4, lambda2=1e-3, initial_scale=0.05)
    return core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.1)


def _fill(link, case, dev):
    """Give every sign of every slot its row (what earlier training has done)."""
    S, per_slot = case["slots"], _per_slot(case)
    piece = max(1, min(link.max_unique, 1 << 22))
    total = S * per_slot
    for lo in range(0, total, piece):
        k = torch.arange(lo, min(lo + piece, total), device=dev)
        link.pull(_sign(k % per_slot + 1, k // per_slot), training=False)


def _build(case, dev):
    hidden = tuple(int(h) for h in case["hidden"].split("-"))
    slots = _slots(case)
    kw = dict(dnn_hidden_units=hidden, embedding_dim=case["dim"], dense_dim=case["dense"], sparse_opt=_sparse_opt(case["sparse"]),
              bucket_size=_bucket(case), combiner="sum", table_rows=int(case["rows"] * 1.25) + 4096,
              target_columns=["label"] if case["cvm"] else None)
    with torch.device(dev):
        if case["model"] == "wide_deep":
            m = tn.models.WideDeep(slots, slots, **kw)
        elif case["model"] == "deepfm":
            m = tn.models.DeepFM(slots, slots, share_linear_table=case["shared"], **kw)
        elif case["model"] == "deep_cross":
            m = tn.models.DeepCross(slots, **kw)
        else:
            m = tn.models.DCNv2(slots, **kw)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=2e-4)), loss="binary_crossentropy")
    return m


def prepare(case, seed):
    gc.collect()
    tn.core.init()
    dev = tn.core.runtime().device
    torch.manual_seed(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    s = _State(case)
    if case["do"] == "serve":
        _prepare_serve(s, case, gen, dev)
    elif case["do"] == "embed":
        _prepare_embed(s, case, gen, dev)
    else:
        s.model = _build(case, dev)
        s.layers = [l for l in s.model.sparse_layers()]
        for l in s.layers:
            _fill(l.link, case, dev)
        s.batches = [_batch(case, gen, dev) for _ in range(case["steps"])]
        signs = _touched(case, torch.cat([_all_ids(f, _slots(case)).to(dev) for f, _ in s.batches]), case["steps"])
        s.at = [l.table.lookup_rows(signs).long() for l in s.layers]
        # a job in its steady state has its first steps behind it
        if case["do"] == "train":
            s.model.fit((s.batches * 6)[:6], record_step_loss=case["losses"])
        else:
            s.model.predict(s.batches[:2])
    s.built()
    torch.cuda.synchronize()
    return s


def _touched(case, ids, steps):
    """The distinct signs of a pass, brought to a length that depends on the case alone (a little above what is
    expected; the last sign repeats), so that results of different inputs have one shape."""
    signs = torch.unique(ids)
    n = int(1.02 * _distinct(case, steps)) + 256
    return torch.cat([signs, signs[-1:].expand(max(0, n - signs.numel()))])[:n]


def _all_ids(f, slots):
    p = f.get(tn.data.PACKED_KEY)
    if p is not None:
        return (p.values if p.ids is None else p.ids).reshape(-1)
    return torch.cat([f[s].values if isinstance(f[s], tn.data.Ragged) else f[s] for s in slots])


def _prepare_serve(s, case, gen, dev):
    S, per_slot = case["slots"], _per_slot(case)
    k = torch.arange(S * per_slot, device=dev)
    signs = _sign(k % per_slot + 1, k // per_slot)
    weights = torch.randn((S * per_slot, case["dim"]), generator=gen, device=dev) * 0.05
    hidden = [int(h) for h in case["hidden"].split("-")]
    with torch.device(dev):
        mlp, head = MLP(S * case["dim"], hidden), DenseHead(hidden[-1])
    s.engine = InferenceEngine(EmbeddingDictionary(signs.cpu().numpy().view(np.uint64), weights.cpu().numpy()), mlp, head, S)
    ids, offsets = _ids(case, gen, dev)
    unknown = torch.rand(ids.shape, generator=gen, device=dev) < 0.1            # signs the dictionary does not hold
    ids = torch.where(unknown, ids ^ 0x5555, ids)
    s.ids = ids.cpu().pin_memory()
    s.offsets = None if offsets is None else offsets.cpu().pin_memory()
    s.engine.infer(s.ids, s.offsets)


def _prepare_embed(s, case, gen, dev):
    slots = _slots(case)
    cols = [tn.feature_column.embedding_column(tn.feature_column.category_column(key=k, bucket_size=_bucket(case)), case["dim"], "sum")
            for k in slots]
    s.layer = EmbeddingFeatures(cols, _sparse_opt(case["sparse"]), name="emb", is_concat=True, rows=int(case["rows"] * 1.25) + 4096)
    _fill(s.layer.link, case, dev)
    ids, offsets = _ids(case, gen, dev)
    p = (tn.data.PackedFeatures(slots, ids=ids) if offsets is None else
         tn.data.PackedFeatures(slots, values=ids, offsets=offsets, batch_size=case["batch"]))
    s.features = {tn.data.PACKED_KEY: p}
    s.grad = torch.randn((case["batch"], case["slots"] * case["dim"]), generator=gen, device=dev) * 1e-2
    s.at = s.layer.table.lookup_rows(_touched(case, ids.reshape(-1), 1)).long()


# ------------------------------------------------------------------------------------------------------------- passes
def run(state):
    do = state.case["do"]
    if do == "serve":
        return state.engine.infer(state.ids, state.offsets).cpu()
    if do == "embed":
        out = state.layer(state.features, training=True)
        out.backward(state.grad)
        state.layer.backwards()
        return {"pooled": out.detach(), "rows": state.layer.table.rows[state.at]}
    if do == "predict":
        return state.model.predict(state.batches)[1]
    hist = state.model.fit(state.batches, record_step_loss=state.case["losses"])
    d = state.model.optimizer.table
    # (not the first moments: where training has driven a gradient to nothing they hold rounding and no more)
    return {"loss": torch.tensor(hist["step_loss" if state.case["losses"] else "loss"]), "weights": d.W, "moments": d.s1,
            "rows": [l.table.rows[at] for l, at in zip(state.layers, state.at)]}


# ------------------------------------------------------------------------------------------------------------- work
def _distinct(case, steps=1):
    """Expected number of distinct signs in ``steps`` batches: per slot, over logarithmic bins of the Zipf ranks."""
    R = _per_slot(case)
    n = case["batch"] * _mean_len(case) * steps
    edges = np.unique(np.concatenate([np.arange(1, 257), np.geomspace(256, R + 1, 400)]).astype(np.int64))
    edges = edges[edges <= R + 1].astype(np.float64)
    if edges[-1] < R + 1:
        edges = np.append(edges, R + 1.0)
    width = edges[1:] - edges[:-1]
    mass = (edges[:-1] ** -0.05 - edges[1:] ** -0.05) / 0.75
    p = mass / width + (1.0 - mass.sum()) / R                   # ranks beyond the resident ones are folded evenly
    return case["slots"] * float((width * -np.expm1(n * np.log1p(-np.minimum(p, 0.999999)))).sum())


def _mean_len(case):
    return 1.0 if case["bags"] == 1 else case["bags"] + math.exp(-case["bags"])


def _row_floats(kind, dim):
    return dim + 4 if kind == "adagrad" else 3 * dim + 2


def work(case):
    """Bytes: ids, labels and dense features once; every distinct row of a batch read (and, when training, written with
    its optimizer state) once; dense weights once per pass, or with their optimizer state read and written once per
    step; results once.  Flops: the products of the towers and cross layers, three times when training."""
    B, S, dim = case["batch"], case["slots"], case["dim"]
    ids = B * S * _mean_len(case)
    hot = _distinct(case)
    if case["do"] == "embed":
        row = 4 * _row_floats(case["sparse"], dim)
        return {"bytes": 8 * ids + hot * 2 * row + 2 * 4 * B * S * dim, "flops": 2 * 2 * ids * dim}
    train = case["do"] == "train"
    width = S * (dim + (2 if case.get("cvm") else 0)) + case.get("dense", 0)
    dims = [width] + [int(h) for h in case["hidden"].split("-")]
    params = sum((a + 1) * b for a, b in zip(dims, dims[1:])) + dims[-1] + 1
    if case.get("model") == "dcn_v2":
        params += 3 * (width + 1) * width
    if case["do"] == "serve":
        return {"bytes": 8 * ids + hot * 4 * dim + 2 * params + 4 * B, "flops": 2 * B * params}
    step_in = 8 * ids + 4 * B * (1 + case["dense"])
    if not train:
        return {"bytes": case["steps"] * (step_in + hot * 4 * dim + 4 * B) + 2 * params, "flops": case["steps"] * 2 * B * params}
    rows = hot * 2 * 4 * _row_floats(case["sparse"], dim + (1 if case["shared"] else 0))
    if case["model"] in ("wide_deep", "deepfm") and not case["shared"]:
        rows += hot * 2 * 4 * _row_floats(case["sparse"], 1)
    return {"bytes": case["steps"] * (step_in + rows + 24 * params), "flops": case["steps"] * 6 * B * params}


def tolerance(case):
    """Towers compute in bf16 (8 bits); the embedding layer sums 32-bit floats, in no fixed order."""
    if case["do"] == "embed":
        return {"rel": 1e-5}
    return {"rel": 1e-2}
