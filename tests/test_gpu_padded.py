"""Ragged batches of many lengths share captured steps whose buffers have room to spare."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batches(tn, slots, B, n, form, seed=3):
    g = torch.Generator().manual_seed(seed)
    out = []
    for k in range(n):
        most = 1 if k == 1 else 4                      # one batch of the shortest length there is
        lens = torch.randint(0 if k else 1, most + 1, (len(slots), B), generator=g)
        offs = torch.cat([torch.zeros(1, dtype=torch.long), lens.reshape(-1).cumsum(0)])
        vals = torch.randint(0, 400, (int(offs[-1]),), generator=g) * 7919 + 11
        y = (torch.rand(B, generator=g) < 0.3).float()
        if form == "packed":
            f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, values=vals, offsets=offs.int(), batch_size=B)}
        else:
            f = {}
            for s, name in enumerate(slots):
                o = offs[s * B: (s + 1) * B + 1]
                f[name] = tn.data.Ragged(vals[int(o[0]): int(o[-1])].to(torch.int32 if s == 1 else torch.int64),
                                         (o - o[0]).to(torch.int64 if s == 2 else torch.int32))
        f["label"] = y
        out.append((f, y))
    return out


@pytest.mark.parametrize("form,cvm,n_slots,B", [("packed", False, 3, 33), ("packed", True, 3, 64), ("columns", False, 3, 33), ("columns", True, 70, 17)])
def test_padded_capture_follows_the_eager_steps(tn_gpu, status_ok, form, cvm, n_slots, B):
    """70 columns: more than one packing launch takes.  The steps agree as far as fp32 sums in another order allow,
    fed back through a dozen updates (the bound of the other captured-against-eager tests)."""
    tn = tn_gpu
    slots = [f"s{k}" for k in range(n_slots)]
    data = _batches(tn, slots, B, 16, form)
    runs, rows = [], []
    for graph in (False, True):
        torch.manual_seed(1)
        m = tn.models.WideDeep(slots, slots, dnn_hidden_units=(32, 16), embedding_dim=4, bucket_size=5 * B, table_rows=1 << 13,
                               use_bn=False, target_columns=["label"] if cvm else None)
        m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=2e-3)), cuda_graph=graph)
        runs.append([float(m.train_on_batch(f, y)) for f, y in data])
        rows.append(m.deep_emb.table.n_rows)
        if graph:
            assert 1 <= len(m._graphs) <= 3 and not m._padded_off
    assert rows[0] == rows[1]                          # nothing but the batch's own ids reached the table
    for a, b in zip(*runs):
        assert abs(a - b) < 5e-2 * max(1.0, abs(a)), runs


def test_a_model_that_reads_exact_lengths_is_not_padded(tn_gpu, status_ok):
    tn = tn_gpu
    slots = ["a", "b"]

    class Mean(tn.models.DeepCross):
        def forward(self, features):
            return super().forward(features) + features["a"].values.numel() * 0.0

    data = _batches(tn, slots, 16, 8, "columns")
    m = Mean(slots, dnn_hidden_units=(16,), embedding_dim=4, bucket_size=128, table_rows=1 << 12)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)))
    losses = [float(m.train_on_batch(f, y)) for f, y in data]
    assert m._padded_off and all(l == l for l in losses)


@pytest.mark.parametrize("form", ["packed", "columns", "single"])
def test_captured_scoring_equals_the_eager_scoring(tn_gpu, status_ok, form):
    """More batches than there are pinned buffers, a shorter last batch, training in between (whose run-ahead front the
    scoring must not take for its own).  Same kernels on the same numbers: equal to bf16 rounding of the towers."""
    tn = tn_gpu
    slots, B = ["a", "b", "c"], 48
    if form == "single":
        g = torch.Generator().manual_seed(5)
        data = [({tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=torch.randint(0, 300, (3, B if k < 21 else 7), generator=g))},
                 (torch.rand(B if k < 21 else 7, generator=g) < 0.3).float()) for k in range(22)]
    else:
        data = _batches(tn, slots, B, 22, form)
    torch.manual_seed(2)
    m = tn.models.DeepFM(slots, slots, dnn_hidden_units=(32, 16), embedding_dim=8, bucket_size=5 * B, table_rows=1 << 13)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)))
    for _ in range(2):
        m.fit(data[:10])
        y, p = m.predict(data)
        assert m._predict_sets and not m._predict_off
        want = torch.cat([m.predict_on_batch(f).cpu() for f, _ in data])
        assert p.shape == want.shape and torch.equal(y, torch.cat([l for _, l in data]))
        assert torch.allclose(p, want, atol=1e-5), float((p - want).abs().max())


def _count(monkeypatch, tn, name):
    made, orig = [], getattr(tn.model.Model, name)

    def counted(self, *a, **kw):
        made.append(1)
        return orig(self, *a, **kw)

    monkeypatch.setattr(tn.model.Model, name, counted)
    return made


def _model(tn, slots, B, cls=None):
    torch.manual_seed(1)
    m = (cls or tn.models.WideDeep)(slots, slots, dnn_hidden_units=(16,), embedding_dim=4, bucket_size=40 * B, table_rows=1 << 14, use_bn=False)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=2e-3)))
    return m


def test_the_number_of_captures_is_bounded(tn_gpu, status_ok, monkeypatch):
    """Twelve batch sizes in turn, more than are captured: the rest runs eagerly, no capture makes way for another."""
    tn = tn_gpu
    slots = ["a", "b"]
    data = [_batches(tn, slots, B, 4, "packed", seed=B)[k] for k in range(4) for B in range(20, 32)]
    made = _count(monkeypatch, tn, "_capture")
    m = _model(tn, slots, 32)
    for _ in range(3):
        m.fit(data)
    assert 1 <= len(made) <= 8 and len(m._graphs) <= 8
    made = _count(monkeypatch, tn, "_capture_predict")
    for _ in range(3):
        p = m.predict(data)[1]
    want = torch.cat([m.predict_on_batch(f).cpu() for f, _ in data])
    assert 1 <= len(made) <= 8 and torch.allclose(p, want, atol=1e-5)
    for B in range(200, 300):                            # sizes that never come back leave nothing behind
        f, y = _batches(tn, slots, B, 1, "packed", seed=B)[0]
        m.train_on_batch(f, y)
    assert len(m._padded_kinds) <= 80


def test_lengths_of_a_heavy_tail(tn_gpu, status_ok, monkeypatch):
    """Now and then one column many times its usual length: a handful of captures, and the steps of an eager run."""
    tn = tn_gpu
    slots, B = [f"s{k}" for k in range(12)], 16
    g = torch.Generator().manual_seed(8)
    data = []
    for _ in range(60):
        f = {}
        for s in slots:
            most = int(torch.empty(1).exponential_(1.0, generator=g).exp().clamp(1, 30))
            lens = torch.randint(1, most + 1, (B,), generator=g)
            offs = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)])
            f[s] = tn.data.Ragged(torch.randint(0, 400, (int(offs[-1]),), generator=g), offs)
        data.append((f, (torch.rand(B, generator=g) < 0.3).float()))
    made = _count(monkeypatch, tn, "_capture")
    m = _model(tn, slots, B)
    got = m.fit(data, epochs=2, record_step_loss=True)["step_loss"]
    assert 1 <= len(made) <= 3
    e = _model(tn, slots, B)
    e._use_graph = False
    want = e.fit(data, epochs=2, record_step_loss=True)["step_loss"]
    assert all(abs(a - b) < 5e-2 * max(1.0, abs(a)) for a, b in zip(want, got)), (want, got)


def test_lengths_within_a_fifth_of_one_another_share_a_capture(tn_gpu, status_ok, monkeypatch):
    tn = tn_gpu
    slots, B = ["a", "b"], 64
    g = torch.Generator().manual_seed(9)
    data = []
    for k in range(40):
        lens = torch.poisson(torch.full((2 * B,), 3.0 + 0.3 * (k % 2)), generator=g).long().clamp_(min=1)
        offs = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)])
        p = tn.data.PackedFeatures(slots, values=torch.randint(0, 400, (int(offs[-1]),), generator=g), offsets=offs.int(), batch_size=B)
        data.append(({tn.data.PACKED_KEY: p}, (torch.rand(B, generator=g) < 0.3).float()))
    made = _count(monkeypatch, tn, "_capture")
    m = _model(tn, slots, B)
    m.fit(data)
    assert len(made) == 1
    made = _count(monkeypatch, tn, "_capture_predict")
    m.predict(data[:7])
    assert not made                                      # a short pass does not pay for captures
    m.predict(data)
    assert len(made) == 1


@pytest.mark.parametrize("name", ["_capture", "_capture_predict"])
def test_a_capture_that_fails_says_so(tn_gpu, status_ok, monkeypatch, name):
    """Out of memory: eager for a while, then tried again.  Anything else: no padding and no captured scoring for good
    (training goes on at exact lengths), with the reason."""
    import warnings

    tn = tn_gpu
    slots, B = ["a", "b"], 32
    data = _batches(tn, slots, B, 24, "packed")
    orig = getattr(tn.model.Model, name)
    step = (lambda m: m.fit(data)) if name == "_capture" else (lambda m: m.predict(data))
    captured = (lambda m: m._graphs) if name == "_capture" else (lambda m: m._predict_sets)
    for error, again in ((torch.OutOfMemoryError("no memory for it"), True), (ValueError("no such thing"), False)):
        tries = []

        def fails_once(self, *a, **kw):
            tries.append(1)
            if len(tries) == 1:
                raise error
            return orig(self, *a, **kw)

        monkeypatch.setattr(tn.model.Model, name, fails_once)
        monkeypatch.setattr(tn.model.model, "_OOM_HOLD", 30, raising=False)
        m = _model(tn, slots, B)
        with warnings.catch_warnings(record=True) as said:
            warnings.simplefilter("always")
            step(m)
            assert any(str(error) in str(w.message) for w in said)
            assert (m._padded_off or m._predict_off) != again
            if again:
                assert len(tries) == 1 and not captured(m)
                for _ in range(3):
                    step(m)
                assert len(tries) == 2 and captured(m)


@pytest.mark.parametrize("why", ["exact lengths", "too many kinds"])
def test_batches_that_run_uncaptured_are_staged_ahead(tn_gpu, status_ok, monkeypatch, why):
    """``fit`` hands them over on the device, copied beside the step before."""
    tn = tn_gpu
    slots = ["a", "b"]

    class Mean(tn.models.WideDeep):
        def forward(self, features):
            return super().forward(features) + features["a"].values.numel() * 0.0

    sizes = [16] * 40 if why == "exact lengths" else list(range(16, 56))
    data = [_batches(tn, slots, B, 1, "columns", seed=k)[0] for k, B in enumerate(sizes)]
    m = _model(tn, slots, 56, Mean if why == "exact lengths" else None)
    step, on_gpu = tn.model.Model.train_step, []

    def seen(self, batch, next_batch=None):
        on_gpu.append(batch[0]["a"].values.is_cuda)
        return step(self, batch, next_batch)

    monkeypatch.setattr(tn.model.Model, "train_step", seen)
    assert all(l == l for l in m.fit(data, record_step_loss=True)["step_loss"])
    assert len(on_gpu) == 40 and not on_gpu[0] and all(on_gpu[-15:])
