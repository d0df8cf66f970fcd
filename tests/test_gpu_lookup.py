"""Pulls that no backward pass follows: the rows straight from the table's index, against the pull with its dedup."""
import pytest
import torch

import tensornet_b200 as tn
from tensornet_b200.layers import EmbeddingFeatures
from tensornet_b200.layers.embedding_features import pulled_together
from tensornet_b200.ops.sparse_table_gpu import GpuSparseLink

pytestmark = pytest.mark.gpu


def _layer(dim, S, bucket, rows=1 << 14, cvm=False, opt=None):
    opt = opt or tn.core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.3)
    cols = [tn.feature_column.embedding_column(tn.feature_column.category_column(key=str(k), bucket_size=bucket), dim, "sum") for k in range(S)]
    return EmbeddingFeatures(cols, opt, name="emb", is_concat=True, rows=rows, target_columns=["label"] if cvm else None)


def _packed(ids):
    return {tn.data.PACKED_KEY: tn.data.PackedFeatures([str(k) for k in range(ids.shape[0])], ids=ids)}


@pytest.mark.parametrize("n", [1, 31, 33, 257, 5000, 60_000])
@pytest.mark.parametrize("dim,cvm", [(8, False), (10, True), (128, False)])
def test_rows_are_those_of_the_pull(n, dim, cvm, monkeypatch):
    """Signs with a row, signs without (several times over), and the key that stands for an empty slot."""
    tn.core.init()
    g = torch.Generator().manual_seed(n)
    layer = _layer(dim, 1, n, cvm=cvm, rows=1 << 17)
    known = torch.randint(0, 1 << 62, (max(1, n // 2),), generator=g)
    layer.link.pull(known.cuda(), training=False)
    have = layer.table.n_rows
    pool = torch.cat([known, torch.randint(0, 1 << 62, (max(1, n // 3),), generator=g), torch.tensor([0, -1])])
    ids = pool[torch.randint(0, pool.numel(), (1, n), generator=g)].cuda()
    f = dict(_packed(ids), label=torch.zeros(n, device="cuda"))
    with torch.no_grad():
        got = layer(f, training=False).clone()
        assert layer.table.n_rows == have + len(set(ids.flatten().tolist()) - set(known.tolist()))
        again = layer(f, training=False).clone()
        monkeypatch.setattr(GpuSparseLink, "looks_up", lambda *a: False)
        want = layer(f, training=False)
    assert torch.equal(got, want) and torch.equal(again, want)
    # the table's own answer: every sign once
    rows = layer.table.lookup_rows(torch.unique(ids))
    assert int(rows.min()) >= 0 and rows.unique().numel() == rows.numel()
    tn.core.runtime().check_status()


@pytest.mark.parametrize("n", [1, 33, 5000])
@pytest.mark.parametrize("dim,cvm,kind", [(8, False, "adagrad"), (10, True, "adagrad"), (3, False, "adam"), (64, False, "ftrl"), (128, False, "adam")])
@pytest.mark.parametrize("zeros", [False, True])
def test_a_new_row_starts_as_the_one_a_pull_makes(n, dim, cvm, kind, zeros):
    """Two layers of one optimizer: the new signs of a batch, several times over, get their rows by lookup in one and by a pull in
    the other.  Values depend on key and column alone (a table in inference mode starts rows at zero), so whole rows agree, the
    optimizer's state included."""
    tn.core.init()
    opts = {"adagrad": tn.core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.3), "adam": tn.core.Adam(initial_scale=0.3),
            "ftrl": tn.core.Ftrl(initial_scale=0.3)}
    g = torch.Generator().manual_seed(n + dim)
    pool = torch.cat([torch.randint(0, 1 << 62, (max(1, n // 2),), generator=g), torch.tensor([0, -1])])
    ids = pool[torch.randint(0, pool.numel(), (n,), generator=g)].cuda()
    got = []
    for by_lookup in (True, False):
        layer = _layer(dim, 1, n, cvm=cvm, opt=opts[kind])
        layer.table.set_training(not zeros)
        with torch.no_grad():
            if by_lookup:
                found = layer.link.lookup_in_place(ids).long()
            else:
                layer.link.pull_in_place(ids, training=False)
        at = layer.table.lookup_rows(torch.unique(ids)).long()
        assert int(at.min()) >= 0 and layer.table.n_rows == at.numel()
        if by_lookup:
            assert torch.equal(found, layer.table.lookup_rows(ids).long())
        got.append(layer.table.rows[at].clone())
    assert torch.equal(*got) and bool((got[0][:, :dim] != 0).any()) != zeros
    tn.core.runtime().check_status()


def test_two_tables_in_one_launch_and_a_front_that_waits():
    tn.core.init()
    g = torch.Generator().manual_seed(1)
    layers = [_layer(4, 3, 400), _layer(8, 3, 400)]
    ids = torch.randint(0, 900, (3, 400), generator=g).cuda()
    nxt = torch.randint(0, 900, (3, 400), generator=g).cuda()
    layers[0](_packed(ids), training=True)
    layers[0].link.cnts.zero_()
    layers[0].link.prefetch(nxt.reshape(-1))                   # the next training batch's front is there, with signs of no row yet
    with torch.no_grad(), pulled_together(layers, _packed(ids), False):
        assert all(l.link._pulled.direct for l in layers)
        a = [l(_packed(ids), training=False).clone() for l in layers]
        b = [l(_packed(nxt), training=False).clone() for l in layers]
    assert layers[0].link._front is not None
    out = layers[0](_packed(nxt), training=True)              # takes the front; its new signs have got their rows meanwhile
    assert layers[0].link.front_hits == 1 and torch.equal(out.detach(), b[0])
    for l, x in zip(layers, a):
        assert torch.equal(l(_packed(ids), training=False).detach(), x)
    assert layers[0].table.n_rows == len(set(ids.flatten().tolist()) | set(nxt.flatten().tolist()))
    tn.core.runtime().check_status()


def test_a_table_that_runs_full_is_reported():
    tn.core.init()
    layer = _layer(8, 1, 4096, rows=1024)
    cap = int(layer.table.rows.shape[0])
    ids = torch.arange(1, cap + 500).view(1, -1).cuda()
    with torch.no_grad():
        out = layer(_packed(ids[:, :4000]), training=False)
        assert int((out.abs().sum(1) > 0).sum()) <= cap
    with pytest.raises(RuntimeError, match="full"):
        tn.core.runtime().check_status()
    tn.core.recover()


def test_a_gradient_still_finds_its_rows():
    """Inference of a layer inside a graph that is differentiated keeps the pull, whose positions the gradients go by."""
    tn.core.init()
    layer = _layer(8, 2, 64)
    ids = torch.arange(128).view(2, 64).cuda()
    out = layer(_packed(ids), training=False)
    out.backward(torch.ones_like(out))
    n = layer.link.unique_counts()[0]
    assert n == 128 and torch.equal(layer.link.gU[:n, :8], torch.ones(n, 8, device="cuda"))
    layer.link.gU.zero_()
