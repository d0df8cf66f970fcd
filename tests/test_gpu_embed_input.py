"""The dense part's input straight from the pulled rows against the layers it takes the place of."""
import pytest
import torch

import tensornet_b200 as tn
from tensornet_b200.core.config import config
from tensornet_b200.layers import EmbeddingFeatures
from tensornet_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _layer(S, dim, cvm, B, combiner, kind="adagrad"):
    opt = tn.core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.5) if kind == "adagrad" else tn.core.Adam(learning_rate=1e-3, initial_scale=0.5)
    cols = [tn.feature_column.embedding_column(tn.feature_column.category_column(key=str(k), bucket_size=8 * B + 64), dim, combiner) for k in range(S)]
    return EmbeddingFeatures(cols, opt, name="emb", is_concat=True, target_columns=["label"] if cvm else None, rows=1 << 15)


def _features(S, B, bags, gen):
    slots = [str(k) for k in range(S)]
    y = (torch.rand(B, generator=gen) < 0.4).float().cuda()
    if bags == 1:
        p = tn.data.PackedFeatures(slots, ids=torch.randint(0, 300, (S, B), generator=gen).cuda())
    else:
        lens = torch.randint(0, bags * 2, (S * B,), generator=gen)              # empty bags among them
        off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).int()
        p = tn.data.PackedFeatures(slots, values=torch.randint(0, 300, (int(off[-1]),), generator=gen).cuda(), offsets=off.cuda(), batch_size=B)
    return {tn.data.PACKED_KEY: p, "label": y}


def _grads(link):
    """The rows' gradients in the order of their signs: positions are handed out anew by every pull."""
    n = link.unique_counts()[0]
    return link.gU[:n][torch.argsort(link._loc["stage_ids"][:n])].clone()


# slots, width, show / click columns, rows, ids per bag, dense columns
CASES = [(4, 8, False, 32, 2, 0), (1, 1, False, 1, 1, 0), (39, 10, False, 301, 1, 5), (26, 16, False, 700, 1, 13), (33, 3, False, 65, 3, 4),
         (65, 4, False, 40, 1, 2), (48, 32, False, 33, 1, 0), (7, 8, True, 100, 3, 1), (20, 16, True, 50, 1, 0), (3, 128, False, 37, 1, 3),
         (5, 100, False, 20, 4, 0), (100, 64, False, 9, 5, 7), (26, 16, False, 3000, 1, 0)]


@pytest.mark.parametrize("S,dim,cvm,B,bags,Dd", CASES)
@pytest.mark.parametrize("combiner", ["sum", "mean", "sqrtn"])
@pytest.mark.parametrize("staged", [False, True])
def test_against_the_layers(S, dim, cvm, B, bags, Dd, combiner, staged, monkeypatch):
    tn.core.init()
    if staged:                                       # rows in the per-batch matrix, as on several GPUs
        monkeypatch.setattr(config, "staged_row_return", 1)
    gen = torch.Generator().manual_seed(S * 31 + B)
    layer = _layer(S, dim, cvm, B, combiner)
    f = _features(S, B, bags, gen)
    dense = torch.randn(B, Dd, generator=gen).cuda() if Dd else None
    W = layer.out_dim
    layer(f, training=True)                          # every sign has its row
    layer.link.cnts.zero_()
    layer.link.gU.zero_()

    out = layer(f, training=False)
    pieces = [out] + ([dense] if Dd else [])
    want = F.concat_cast(pieces, ones=True)
    fm_want = F.fm(out, S, W)
    gx = torch.randn(want.shape, generator=gen).cuda().to(torch.bfloat16)
    gfm = torch.randn(B, 1, generator=gen).cuda()
    gp = torch.randn(B, S * W + Dd, generator=gen).cuda()
    torch.autograd.backward([want, fm_want, out], [gx, gfm, gp[:, : S * W]])
    g_want = _grads(layer.link)
    layer.link.gU.zero_()

    x0, fm, lin, pooled = layer.operand(f, False, dense, fm=True, pooled=True)
    assert lin is None and torch.equal(x0, want) and torch.equal(pooled, torch.cat([p.detach() for p in pieces], 1))
    x = out.detach().double().view(B, S, W)
    fm64 = 0.5 * (x.sum(1).square() - x.square().sum(1)).sum(1)
    bound = 2.0 ** -23 * (S + W) * (x.abs().sum(1).square() + x.square().sum(1)).sum(1)      # sums of S and of W terms
    assert bool(((fm.view(-1).double() - fm64).abs() <= bound + 1e-12).all())
    torch.autograd.backward([x0, fm, pooled], [gx, gfm, gp])
    g = _grads(layer.link)
    assert float((g - g_want).norm()) <= 1e-5 * float(g_want.norm()) + 1e-12      # sums of 32-bit floats in another order
    layer.link.gU.zero_()
    x0, fm, _, pooled = layer.operand(f, False, dense)
    assert fm is None and pooled is None and torch.equal(x0, want)
    with torch.no_grad():
        assert torch.equal(layer.operand(f, False, dense, fm=True)[0], want)
    tn.core.runtime().check_status()


@pytest.mark.parametrize("S,D,B,bags", [(26, 16, 500, 1), (40, 8, 33, 1), (5, 4, 64, 3), (70, 12, 20, 1)])
def test_linear_weights_in_the_rows(S, D, B, bags):
    tn.core.init()
    gen = torch.Generator().manual_seed(S)
    layer = _layer(S, D + 4, False, B, "mean", "adam")
    f = _features(S, B, bags, gen)
    layer(f, training=True)
    layer.link.gU.zero_()
    both = layer(f, training=False).view(B, S, D + 4)
    gx = torch.randn(B, F.pad8(S * D + 1), generator=gen).cuda().to(torch.bfloat16)
    gl = torch.randn(B, S, generator=gen).cuda()
    deep = both[:, :, :D].reshape(B, -1)
    torch.autograd.backward([F.concat_cast([deep], ones=True), both[:, :, D]], [gx, gl])
    g_want = _grads(layer.link)
    layer.link.gU.zero_()
    x0, fm, lin, _ = layer.operand(f, False, None, True, D, D)
    assert torch.equal(x0, F.concat_cast([deep.detach()], ones=True))
    assert torch.allclose(lin, both[:, :, D].detach(), rtol=1e-6, atol=1e-7) and torch.allclose(fm, F.fm(deep.detach(), S, D), rtol=1e-4, atol=1e-4)
    torch.autograd.backward([x0, lin], [gx, gl])
    assert float((_grads(layer.link) - g_want).norm()) <= 1e-5 * float(g_want.norm())


@pytest.mark.parametrize("kind", ["wide_deep", "deepfm", "deep_cross", "dcn_v2"])
@pytest.mark.parametrize("dim,frozen", [(132, ()), (8, ("head",)), (8, ("mlp",)), (132, ("head", "mlp"))])
def test_own_steps_that_the_kernels_do_not_take_whole(kind, dim, frozen):
    """Slots wider than the kernel's columns are pooled, a frozen head or tower goes through the layers: the same steps as one by one,
    and what is frozen stays as it is."""
    tn.core.init()
    S, B, slots, runs = 3, 40, ["0", "1", "2"], []
    for fused in (True, False):
        torch.manual_seed(2)
        kw = dict(dnn_hidden_units=(32, 16), embedding_dim=dim, dense_dim=3, bucket_size=B, table_rows=1 << 12)
        cls = {"wide_deep": tn.models.WideDeep, "deepfm": tn.models.DeepFM, "deep_cross": tn.models.DeepCross, "dcn_v2": tn.models.DCNv2}[kind]
        with torch.device("cuda"):
            m = cls(*([slots, slots] if kind in ("wide_deep", "deepfm") else [slots]), **kw)
        for part in frozen:
            for p in getattr(m.sub_model, part).parameters():
                p.requires_grad_(False)
        kept = [p.detach().clone() for part in frozen for p in getattr(m.sub_model, part).parameters()]
        m.compile(optimizer=tn.optimizer.Optimizer(tn.core.AdaGrad(learning_rate=0.05)), cuda_graph=False)
        m.use_fused = fused
        assert m.deep_emb.gives_operand() == (m.deep_emb.out_dim <= 128)
        g = torch.Generator().manual_seed(5)
        losses = []
        for _ in range(3):
            f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=torch.randint(0, 90, (S, B), generator=g)), "dense": torch.randn(B, 3, generator=g)}
            losses.append(float(m.train_on_batch(f, (torch.rand(B, generator=g) < 0.4).float())))
        now = [p.detach() for part in frozen for p in getattr(m.sub_model, part).parameters()]
        assert all(torch.equal(a, b) for a, b in zip(kept, now))
        runs.append((losses, torch.cat([p.detach().flatten() for p in m.sub_model.parameters()])))
        tn.core.runtime().check_status()
    assert runs[0][0] == pytest.approx(runs[1][0], rel=5e-3)
    assert float((runs[0][1] - runs[1][1]).norm()) <= 1e-2 * float(runs[1][1].norm())
