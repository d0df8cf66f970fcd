"""The Dense(1) head over the pieces of its operand against float64, and models with and without it."""
import pytest
import torch

import tensornet_b200 as tn
from tensornet_b200.layers import DenseHead
from tensornet_b200.ops import functional as F

pytestmark = pytest.mark.gpu

# (rows, bf16 piece's width, fp32 pieces' widths): one block, its first batch with several, both row counts, rows on no
# boundary, more units than threads, the widest that fits
CASES = [(1, 8, ()), (16, 256, (4,)), (17, 75, (39, 1)), (333, 400, (26, 1)), (4000, 400, (26, 1)), (700, 60, (1,)), (2400, 120, (100, 1)), (33, 257, (33,)), (1024, 32, ()), (1185, 256, (200,)), (2999, 75, (39, 1)),
         (4096, 256, (203,)), (300, 512, (1632,)), (40, 1024, (3064, 1))]


def _pieces(B, nh, widths, gen, requires_grad=True):
    h = torch.relu(torch.randn(B, F.pad8(nh + 1), generator=gen, device="cuda"))
    h[:, nh] = 1.0
    h[:, nh + 1:] = 0.0
    out = [h.to(torch.bfloat16)] + [torch.randn(B, w, generator=gen, device="cuda") for w in widths]
    return [p.requires_grad_(requires_grad) for p in out]


@pytest.mark.parametrize("B,nh,widths", CASES)
@pytest.mark.parametrize("bins", [0, 8])
def test_head_loss_and_gradients(B, nh, widths, bins):
    tn.core.init()
    gen = torch.Generator(device="cuda").manual_seed(B + nh)
    pieces = _pieces(B, nh, widths, gen)
    ks = [nh, *widths]
    K = sum(ks)
    w = (torch.randn(K + 1, generator=gen, device="cuda") / K ** 0.5).requires_grad_()
    y = (torch.rand(B, generator=gen, device="cuda") < 0.3).float()
    before = torch.randn(K + 1, generator=gen, device="cuda")
    w.grad = before.clone()
    sums = torch.zeros(4 + 2 * bins, device="cuda")
    scratch = F.head_scratch(ks, "cuda")
    for turn in range(2):                           # the second call finds the scratch as the first has left it
        for p in pieces:
            p.grad = None
        loss = F.head_loss(pieces, ks, w, y, sums, scratch)
        loss.backward()
    assert not scratch.any()

    z = torch.cat([p.detach()[:, :k].double() for p, k in zip(pieces, ks)], 1)
    logit = z @ w.detach()[:K].double() + w.detach()[K].double()
    want = torch.nn.functional.binary_cross_entropy_with_logits(logit, y.double())
    dl = (torch.sigmoid(logit) - y.double()) / B
    eps = 2.0 ** -23
    # sums of K products in 32 bits: at most K roundings of the sum of magnitudes
    assert abs(float(loss) - float(want)) <= K * eps * float((z.abs() @ w.detach()[:K].double().abs()).max() + 1)
    gw = torch.cat([z.t() @ dl, dl.sum()[None]])
    bound = (K + B + 64) * eps * torch.cat([z.abs().t() @ dl.abs(), dl.abs().sum()[None]]) * 2 + 4 * eps * before.abs() + 1e-9
    assert bool(((w.grad.double() - before.double() - 2 * gw).abs() <= 2 * bound + 1e-6 * gw.abs().max()).all())
    off = 0
    for i, (p, k) in enumerate(zip(pieces, ks)):
        g = dl[:, None] * w.detach()[off:off + k].double()
        if i == 0:
            g = torch.where(p.detach()[:, :k] > 0, g, 0.0)
            assert not p.grad[:, k:].any()
        tol = 2.0 ** -8 if p.dtype == torch.bfloat16 else 1e-4      # one rounding to bf16; dlogit through exp in 32 bits
        assert float((p.grad[:, :k].double() - g).norm()) <= tol * float(g.norm()) + 1e-12
        off += k
    assert abs(float(sums[0]) - 2 * float(want)) < 1e-3 * float(want) and float(sums[3]) == 2 * B
    assert float(sums[1]) == 2 * float(y.sum())
    if bins:
        hist = sums[4:].view(torch.int32).view(2, bins).sum(1)
        assert hist.tolist() == [2 * int(y.sum()), 2 * int((1 - y).sum())]


@pytest.mark.parametrize("B,nh,widths", CASES + [(5000, 400, (26, 1))])
def test_head_score(B, nh, widths):
    tn.core.init()
    gen = torch.Generator(device="cuda").manual_seed(B)
    pieces = _pieces(B, nh, widths, gen, False)
    ks = [nh, *widths]
    w = torch.randn(sum(ks) + 1, generator=gen, device="cuda")
    got = F.head_score(pieces, ks, w)
    z = torch.cat([p[:, :k].double() for p, k in zip(pieces, ks)] + [torch.ones(B, 1, device="cuda").double()], 1)
    bound = (sum(ks) + 2) * 2.0 ** -23 * (z.abs() @ w.double().abs())
    assert bool(((got.view(-1).double() - z @ w.double()).abs() <= bound).all())


@pytest.mark.parametrize("B,nh,widths", [(1, 8, ()), (17, 75, (39, 1)), (700, 60, (1,)), (33, 257, (33,)), (2999, 75, (39, 1)), (1185, 256, (200,)),
                                         (300, 512, (1632,)), (40, 1017, (3064, 1)), (5000, 401, (26, 1))])
@pytest.mark.parametrize("relu", [True, False])
def test_what_lies_behind_a_pieces_columns_is_left_out(B, nh, widths, relu):
    """Infinities and NaN there change nothing, to the bit."""
    tn.core.init()
    gen = torch.Generator(device="cuda").manual_seed(B)
    pieces, ks = _pieces(B, nh, widths, gen, False), [nh, *widths]
    w = (torch.randn(sum(ks) + 1, generator=gen, device="cuda") / sum(ks) ** 0.5).requires_grad_()
    y = (torch.rand(B, generator=gen, device="cuda") < 0.3).float()
    got = []
    for fill in (0.0, float("nan"), float("inf")):
        h = pieces[0].clone()
        h[:, nh:] = fill
        h.requires_grad_()
        w.grad = torch.zeros_like(w)
        pred = torch.empty(B, device="cuda")
        F.head_loss([h, *pieces[1:]], ks, w, y, torch.zeros(4, device="cuda"), F.head_scratch(ks, "cuda"), relu, pred).backward()
        # (the weight's gradient is a sum of blocks in no fixed order)
        got.append((pred, h.grad, F.head_score([h.detach(), *pieces[1:]], ks, w), w.grad.clone()))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0][:3], other[:3]))
        assert torch.allclose(got[0][3], other[3], rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("B,K", [(1, 8), (32, 260), (33, 42), (70, 127), (500, 319), (2048, 500)])
@pytest.mark.parametrize("relu", [False, True])
def test_small_head_is_the_layer_to_the_bit(B, K, relu):
    """Logits (and with them the operand's gradient) of a small batch are those of the layers one by one."""
    tn.core.init()
    gen = torch.Generator(device="cuda").manual_seed(B * K)
    z = torch.relu(torch.randn(B, F.pad8(K + 1), generator=gen, device="cuda"))
    z[:, K] = 1.0
    z[:, K + 1:] = 0.0
    z = z.to(torch.bfloat16)
    w = torch.randn(K + 1, generator=gen, device="cuda").requires_grad_()
    y = (torch.rand(B, generator=gen, device="cuda") < 0.3).float()
    grads = []
    for fused in (True, False):
        zz = z.clone().requires_grad_()
        w.grad = None
        if fused:
            pred = torch.empty(B, device="cuda")
            F.head_loss([zz], [K], w, y, torch.zeros(4, device="cuda"), F.head_scratch([K], "cuda"), relu, pred).backward()
        else:
            loss, want = F.bce_with_logits(F.head(zz, w), y, torch.zeros(4, device="cuda"))
            loss.backward()
            assert torch.equal(pred, want.view(-1))
        g = zz.grad[:, :K]
        grads.append(torch.where(z[:, :K] > 0, g, 0) if relu else g)
    assert torch.equal(*grads)


def test_head_takes_pieces_in_other_forms():
    """Strided, half-precision or unpadded pieces are brought to a form that the kernel reads, gradients included."""
    tn.core.init()
    gen = torch.Generator(device="cuda").manual_seed(5)
    wide = torch.randn(50, 40, generator=gen, device="cuda").requires_grad_()
    h = torch.randn(50, 21, generator=gen, device="cuda").to(torch.bfloat16).requires_grad_()
    head = DenseHead(13 + 17).cuda()
    y = (torch.rand(50, generator=gen, device="cuda") < 0.5).float()
    sums = torch.zeros(4, device="cuda")
    head.loss([h, wide[:, 3:20]], [13, 17], y, sums, relu_first=False).backward()
    z = torch.cat([h.detach()[:, :13].double(), wide.detach()[:, 3:20].double()], 1)
    dl = (torch.sigmoid(z @ head.weight.detach()[:30].double() + head.weight.detach()[30].double()) - y.double()) / 50
    assert torch.allclose(wide.grad[:, 3:20].double(), dl[:, None] * head.weight.detach()[13:30].double(), rtol=1e-4, atol=1e-8)
    assert not wide.grad[:, :3].any() and not h.grad[:, 13:].any()
    assert torch.allclose(h.grad[:, :13].double(), dl[:, None] * head.weight.detach()[:13].double(), rtol=2.0 ** -7, atol=1e-8)


def _model(kind, S, dim, hidden, B, bags, cvm):
    slots = [str(i + 1) for i in range(S)]
    kw = dict(dnn_hidden_units=hidden, embedding_dim=dim, dense_dim=3, bucket_size=B * bags * 3, table_rows=1 << 16, combiner="sum",
              target_columns=["label"] if cvm else None)
    with torch.device("cuda"):
        torch.manual_seed(3)
        m = (tn.models.WideDeep(slots, slots, **kw) if kind == "wide_deep" else tn.models.DeepFM(slots, slots, **kw) if kind == "deepfm" else
             tn.models.DeepCross(slots, **kw) if kind == "deep_cross" else tn.models.DCNv2(slots, **kw))
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)), cuda_graph=False)
    return m, slots


@pytest.mark.parametrize("kind,S,dim,hidden,bags,cvm", [
    ("wide_deep", 5, 8, (32, 16), 1, False), ("deepfm", 7, 10, (40, 24), 1, False), ("deepfm", 40, 8, (64,), 1, False),
    ("deepfm", 6, 8, (40,), 3, True), ("deep_cross", 6, 8, (48, 24), 3, True), ("dcn_v2", 5, 8, (32,), 1, False)])
def test_models_with_the_head_in_one_kernel(kind, S, dim, hidden, bags, cvm):
    """A few steps with and without the fused kernels; and a hook on the head is called, as it always was."""
    tn.core.init()
    B = 70
    runs = []
    for fused in (True, False):
        m, slots = _model(kind, S, dim, hidden, B, bags, cvm)
        m.use_fused = fused
        g = torch.Generator().manual_seed(1)
        losses = []
        for _ in range(4):
            if bags == 1:
                f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=torch.randint(0, 500, (S, B), generator=g))}
            else:
                lens = torch.randint(1, bags * 2, (S * B,), generator=g)
                off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).int()
                f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, values=torch.randint(0, 500, (int(off[-1]),), generator=g), offsets=off,
                                                                batch_size=B)}
            f["dense"] = torch.randn(B, 3, generator=g)
            y = (torch.rand(B, generator=g) < 0.3).float()
            if cvm:
                f["label"] = y
            losses.append(float(m.train_on_batch(f, y)))
        tn.core.runtime().check_status()
        with torch.no_grad():
            m.eval()
            dev = {k: v.to("cuda") for k, v in f.items()}
            logits = m(dev).detach().clone()
        runs.append((losses, m.optimizer.table.W.detach().clone(), logits))
    (l0, w0, p0), (l1, w1, p1) = runs
    assert l0 == pytest.approx(l1, rel=5e-3)
    assert float((w0 - w1).norm()) <= 1e-2 * float(w1.norm()) and float((p0 - p1).norm()) <= 5e-2 * float(p1.norm()) + 1e-2
    seen = []
    m.use_fused = True
    m.train()
    hook = m.sub_model.head.register_forward_hook(lambda *a: seen.append(1))
    m.train_on_batch(f, y)
    assert seen
    hook.remove()


@pytest.mark.parametrize("kind", ["wide_deep", "deep_cross"])
def test_own_steps_add_to_the_gradients_and_hooks_still_see_them(kind):
    """A model's own step adds the gradients of the cross network and of the batch norm to ``.grad`` in the kernels; a hook on one
    of those parameters gets the gradient as before, and the steps are the same."""
    tn.core.init()
    B, seen, runs = 64, [], []
    for hooked in (False, True):
        m, slots = _model(kind, 5, 8, (32, 16), B, 1, False)
        p = m.sub_model.bn.gamma if kind == "wide_deep" else m.sub_model.cross.W[1]
        if hooked:
            p.register_hook(lambda g: seen.append(g.clone()))
        g = torch.Generator().manual_seed(2)
        for _ in range(3):
            f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=torch.randint(0, 300, (5, B), generator=g)), "dense": torch.randn(B, 3, generator=g)}
            m.train_on_batch(f, (torch.rand(B, generator=g) < 0.3).float())
        runs.append(m.optimizer.table.W.clone())
    assert len(seen) == 3 and all(bool(g.abs().sum() > 0) for g in seen)
    assert float((runs[0] - runs[1]).norm()) <= 1e-3 * float(runs[1].norm())


@pytest.mark.parametrize("kind", ["wide_deep", "deepfm", "deep_cross", "dcn_v2"])
@pytest.mark.parametrize("fused", [True, False])
def test_labels_of_another_length(kind, fused):
    """Labels beyond the examples are not looked at, as ever; too few are refused before a kernel reads behind them."""
    tn.core.init()
    B, got = 48, []
    g = torch.Generator().manual_seed(4)
    ids, dense = torch.randint(0, 300, (5, B), generator=g), torch.randn(B, 3, generator=g)
    y = (torch.rand(B, 2, generator=g) < 0.3).float()
    for labels in (y, y.reshape(-1)[:B]):
        m, slots = _model(kind, 5, 8, (32, 16), B, 1, False)
        m.use_fused = fused
        f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=ids), "dense": dense}
        m.train_on_batch(f, labels)
        got.append(m.optimizer.table.W.clone())
    assert float((got[0] - got[1]).norm()) <= 1e-4 * float(got[1].norm())
    with pytest.raises(RuntimeError, match="label"):
        m.train_on_batch(f, y.reshape(-1)[: B - 1])
    assert torch.isfinite(m.train_on_batch(f, y.reshape(-1)[:B]))
    tn.core.runtime().check_status()
