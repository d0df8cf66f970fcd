"""Weight gradients that run beside the gradients of a step's inputs, and the launches that follow them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SLOTS = ["a", "b", "c"]


def _model(tn, kind, seed=3):
    torch.manual_seed(seed)
    kw = dict(dnn_hidden_units=(48, 24), embedding_dim=8, dense_dim=3, bucket_size=1 << 14, table_rows=1 << 12)
    m = getattr(tn.models, kind)(*([SLOTS, SLOTS] if kind in ("DeepFM", "WideDeep") else [SLOTS]), **kw)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.AdaGrad(learning_rate=0.05)), cuda_graph=False)
    return m


def _batch(tn, B):
    g = torch.Generator().manual_seed(B)
    ids = torch.randperm(1 << 13, generator=g)[: len(SLOTS) * B].view(len(SLOTS), B)      # no sign twice: no sum of a free order
    f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(SLOTS, ids=ids), "dense": torch.randn((B, 3), generator=g)}
    return f, (torch.rand(B, generator=g) < 0.4).float()


@pytest.mark.parametrize("kind", ["DeepFM", "WideDeep", "DeepCross", "DCNv2"])
@pytest.mark.parametrize("B", [1, 33, 1000])
def test_weights_are_those_of_the_joined_pass(tn_gpu, status_ok, monkeypatch, kind, B):
    """The same kernels on the same operands: the tower's weights after a step to the bit."""
    tn = tn_gpu
    F = tn.ops.functional
    held, hold = [], F.LateGrads.hold
    monkeypatch.setattr(F.LateGrads, "hold", lambda self, *a: held.append(1) or hold(self, *a))
    got = []
    for late in (True, False):
        m = _model(tn, kind)
        f, y = _batch(tn, B)
        with monkeypatch.context() as mp:
            if not late:
                mp.setattr(m, "_step_body", lambda *a, body=m._step_body: (object.__setattr__(m, "_late_grads", _Never()), body(*a))[1])
            m.train_on_batch(f, y)
        assert m._late_grads is None and len(held) == 1
        got.append([w.detach().clone() for w in m.sub_model.mlp.weights])
    for a, b in zip(*got):
        assert torch.equal(a, b)


class _Never:
    """Stands in for the holder: the backward pass finds that it may not leave anything to it."""

    def __new__(cls):
        from tensornet_b200.ops import functional as F

        class Joined(F.LateGrads):
            def hold(self, side, *tensors):
                torch.cuda.current_stream().wait_stream(side)
        return Joined()


@pytest.mark.parametrize("joins", [True, False])
def test_a_failed_step_leaves_nothing_behind(tn_gpu, status_ok, monkeypatch, joins):
    """Its own error comes through, also where the streams cannot be joined any more."""
    tn = tn_gpu
    m = _model(tn, "DeepFM")
    f, y = _batch(tn, 33)
    layer = m.sparse_layers()[0]
    real = layer.backwards

    def fails(*a):
        raise ValueError("on purpose")
    layer.backwards = fails
    if not joins:
        def cannot(self):
            raise RuntimeError("capture has ended")
        monkeypatch.setattr(tn.ops.functional.LateGrads, "join", cannot)
    with pytest.raises(ValueError):
        m.train_on_batch(f, y)
    assert m._late_grads is None
    layer.backwards = real
    torch.cuda.synchronize()
    assert torch.isfinite(torch.as_tensor(m.train_on_batch(f, y))).all()


def test_a_step_of_the_users_runs_behind_the_gradients(tn_gpu, status_ok):
    """An optimizer whose ``step`` is replaced reads whole gradients on the caller's stream."""
    tn = tn_gpu
    norms = []
    for own in (False, True):
        m = _model(tn, "DeepFM")
        f, y = _batch(tn, 1000)
        real, opt = m.optimizer.step, m.optimizer
        if own:
            opt.step = lambda *a: (norms.append(opt.table.G.double().norm().item()), real(*a))[1]
        else:
            opt.table.ctx, ctx = _Spy(opt.table, norms), opt.table.ctx
            opt.table.ctx.real = ctx
        m.train_on_batch(f, y)
    assert norms[0] > 0 and abs(norms[0] - norms[1]) <= 1e-6 * norms[0]


@pytest.mark.parametrize("how", ["subclass", "instance"])
def test_backwards_of_the_users_finds_the_gradients(tn_gpu, status_ok, how):
    """``Model.backwards`` replaced: called between the backward pass and the update, on a stream behind the weights' gradients."""
    tn = tn_gpu
    seen = []

    def look(m, *a):
        seen.append((m.optimizer.table.G.double().norm().item(), m.optimizer.iterations))
        return tn.models.DeepFM.backwards(m, *a)
    m = _model(tn, "DeepFM")
    f, y = _batch(tn, 1000)
    m.train_on_batch(f, y)                                       # (the gradients' memory is there)
    ref = _model(tn, "DeepFM")
    ref.train_on_batch(f, y)
    ref.optimizer.table.ctx, ctx = _Spy(ref.optimizer.table, want := []), ref.optimizer.table.ctx
    ref.optimizer.table.ctx.real = ctx
    ref.train_on_batch(f, y)
    if how == "subclass":
        m.__class__ = type("Own", (type(m),), {"backwards": look})
    else:
        m.backwards = lambda *a: look(m, *a)
    m.train_on_batch(f, y)
    (norm, before), = seen
    assert before == 1 and m.optimizer.iterations == 2 and abs(norm - want[0]) <= 1e-6 * want[0] and want[0] > 0


class _Spy:
    def __init__(self, table, out):
        self.table, self.out = table, out

    def step(self, *a):
        self.out.append(self.table.G.double().norm().item())
        return self.real.step(*a)

    def __getattr__(self, k):
        return getattr(self.real, k)


@pytest.mark.parametrize("kind", ["AdaGrad", "Ftrl"])
@pytest.mark.parametrize("rows", [1000, 90000])
def test_pushes_small_and_large(tn_gpu, status_ok, kind, rows):
    """Launched to overlap with the kernel ahead and not: the first rows of a push as those of a push of ten, to the bit."""
    tn = tn_gpu
    opt = getattr(tn.core, kind)()
    got = []
    for n in (rows, 10):
        cols = [tn.feature_column.embedding_column(tn.feature_column.category_column(key="a", bucket_size=1 << 20), 128, "sum")]
        layer = tn.layers.EmbeddingFeatures(cols, opt, name="large", is_concat=True, rows=1 << 17)
        layer.train()
        out = layer({tn.data.PACKED_KEY: tn.data.PackedFeatures(["a"], ids=torch.arange(n).view(1, n))})
        out.backward(torch.ones_like(out) * torch.linspace(0.1, 1, 128, device=out.device))
        layer.backwards()
        layer.eval()
        with torch.no_grad():
            got.append(layer({tn.data.PACKED_KEY: tn.data.PackedFeatures(["a"], ids=torch.arange(n).view(1, n))})[:10].clone())
    assert torch.equal(got[0], got[1])
