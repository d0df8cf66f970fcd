"""``Model.predict`` by replaying captured scoring steps: what a caller could rely on while every batch was scored eagerly."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SLOTS = ["a", "b", "c"]


def _data(tn, n, B=48, seed=5, ragged=False, labels=True):
    g = torch.Generator().manual_seed(seed)
    out = []
    for _ in range(n):
        if ragged:
            lens = torch.randint(1, 4, (len(SLOTS) * B,), generator=g)
            offs = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)]).int()
            p = tn.data.PackedFeatures(SLOTS, values=torch.randint(0, 300, (int(offs[-1]),), generator=g), offsets=offs, batch_size=B)
        else:
            p = tn.data.PackedFeatures(SLOTS, ids=torch.randint(0, 300, (3, B), generator=g))
        y = (torch.rand(B, generator=g) < 0.3).float()
        out.append(({tn.data.PACKED_KEY: p}, y if labels else None))
    return out


def _model(tn, cls=None, B=48, compiled=True, **kw):
    torch.manual_seed(2)
    m = (cls or tn.models.DeepFM)(SLOTS, SLOTS, dnn_hidden_units=(32, 16), embedding_dim=8, bucket_size=5 * B, table_rows=1 << 13, **kw)
    if compiled:
        m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-2)))
    return m


def _eager(m, data):
    """The predictions batch by batch; the same kernels on the same numbers, so equal to bf16 rounding of the towers."""
    return torch.cat([m.predict_on_batch(f).cpu() for f, _ in data])


def _same(got, want):
    assert got.shape == want.shape and torch.allclose(got, want, atol=1e-5), float((got - want).abs().max())


def test_code_of_the_users_runs_for_every_batch(tn_gpu, status_ok):
    """An overridden ``predict_step``, a forward pass or a hook of the user's: called once per batch, its result kept."""
    tn = tn_gpu
    data = _data(tn, 12)

    class Calibrated(tn.models.DeepFM):
        def predict_step(self, batch):
            y, p = super().predict_step(batch)
            return y, p * 0.5

    class Counting(tn.models.DeepFM):
        def forward(self, features):
            seen.append(1)
            return super().forward(features)

    m = _model(tn, Calibrated)
    for _ in range(2):
        got = m.predict(data)[1]
        _same(got, _eager(m, data))
        assert float(got.max()) <= 0.5
    seen = []
    m = _model(tn, Counting)
    m.predict(data)
    assert len(seen) == 12
    m = _model(tn)
    handle = m.sub_model.head.register_forward_hook(lambda *_: seen.append(1))
    del seen[:]
    m.predict(data)
    assert len(seen) == 12
    handle.remove()
    m.predict(data)
    m.predict_step = lambda batch: (batch[1], torch.full((48, 1), 0.25))
    assert float(m.predict(data)[1].max()) == 0.25


def _held(m):
    """Keeps the storage a model scores from alive, so that a step captured from it reads what it read before."""
    return [p.data for p in m.parameters()] + [getattr(p, "_tn_bf16", None) for p in m.parameters()]


def test_scoring_follows_what_the_model_is_made_of(tn_gpu, status_ok):
    """Parameters re-pointed by an optimizer, a replaced sub-module, an attribute the forward pass goes by."""
    from tensornet_b200.layers import DenseHead

    tn = tn_gpu
    data = _data(tn, 20)
    m = _model(tn, compiled=False)
    m.compile()
    keep = [_held(m)]
    m.predict(data)
    for _ in range(2):
        keep.append((m.optimizer, _held(m)))
        m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=3e-2)))
        before = m.predict(data)[1]
        _same(before, _eager(m, data))
        m.fit(data)
        after = m.predict(data)[1]
        _same(after, _eager(m, data))
        assert float((after - before).abs().max()) > 1e-3
    keep.append(m.sub_model.head)
    m.sub_model.head = DenseHead(m.sub_model.head.in_dim).cuda()
    _same(m.predict(data)[1], _eager(m, data))
    m.sub_model.mlp.relu_last = False
    _same(m.predict(data)[1], _eager(m, data))
    m.predict(data)
    sets = dict(m._predict_sets)
    m.fit(data)                                       # training writes the weights in place: nothing to capture again
    _same(m.predict(data)[1], _eager(m, data))
    assert sets == m._predict_sets and not m._predict_off


def test_training_follows_a_second_optimizer(tn_gpu, status_ok):
    tn = tn_gpu
    data = _data(tn, 12)
    m = _model(tn)
    m.fit(data)
    keep = (m.optimizer, _held(m))
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-2)))
    before = [p.detach().clone() for p in m.parameters()]
    m.fit(data, epochs=2)
    assert m._graphs or m._rings
    assert all(not torch.equal(a, b) for a, b in zip(before, m.parameters()))
    del keep


@pytest.mark.parametrize("pinned", [False, True])
def test_a_reader_may_fill_the_same_buffers_again(tn_gpu, status_ok, pinned):
    """Ids and labels of every batch in one buffer each, overwritten as soon as the next batch is asked for."""
    tn = tn_gpu
    data = _data(tn, 30)
    m = _model(tn)
    want = _eager(m, data)
    ids = torch.empty((3, 48), dtype=torch.int64, pin_memory=pinned)
    y = torch.empty(48, pin_memory=pinned)

    def reader():
        for f, labels in data:
            ids.copy_(f[tn.data.PACKED_KEY].ids)
            y.copy_(labels)
            yield {tn.data.PACKED_KEY: tn.data.PackedFeatures(SLOTS, ids=ids)}, y
        ids.fill_(7)
        y.fill_(0.5)

    for _ in range(2):
        labels, got = m.predict(reader())
        _same(got, want)
        assert torch.equal(labels, torch.cat([l for _, l in data]))


def test_predictions_outlive_the_captures_they_came_from(tn_gpu, status_ok, monkeypatch):
    """Captured steps that go while the copies of their predictions still wait for their turn on the read-back stream."""
    tn = tn_gpu
    data = _data(tn, 40, B=512)
    m = _model(tn, B=512)
    want = _eager(m, data)
    m.predict(data)
    issue = type(m)._predict_captured

    def late(self, features, *a):
        got = issue(self, features, *a)
        with torch.cuda.stream(self._read_stream):
            torch.cuda._sleep(2_000_000)               # about a millisecond: the copy of this batch's predictions is late
        if len(calls) % 5 == 4:
            torch.cuda.current_stream().synchronize()  # the replays are over, the copies are not
            self._predict_sets.clear()                 # the last reference but the one predict holds for this batch
            torch.full((512, 1), 9.0, device="cuda")   # whoever gets the memory next writes it at once
            torch.full((512, 1), 9.0, device="cuda")
        calls.append(got is not None)
        return got

    calls = []
    monkeypatch.setattr(tn.model.Model, "_predict_captured", late)
    _same(m.predict(data)[1], want)
    assert sum(calls) >= 10
