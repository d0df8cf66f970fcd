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
