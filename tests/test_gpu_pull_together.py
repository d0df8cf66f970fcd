"""Pulls of several layers that are run ahead of their forward passes count what the layers are given and nothing else."""
import numpy as np
import pytest
import torch
from torch.nn.modules import module as torch_module

pytestmark = pytest.mark.gpu

SLOTS, B = ["a", "b"], 300


def _features(tn, seed, columns=False):
    g = torch.Generator().manual_seed(seed)
    dev = tn.core.runtime().device
    ids = torch.randint(0, 400, (len(SLOTS), B), generator=g) * 7919 + 11 * seed
    y = (torch.rand(B, generator=g) < 0.4).float().to(dev)
    f = {s: ids[k].to(dev) for k, s in enumerate(SLOTS)} if columns else {tn.data.PACKED_KEY: tn.data.PackedFeatures(SLOTS, ids=ids.to(dev))}
    return dict(f, label=y), ids, y


def _counted(layer, batches):
    """Rows, shows and clicks (AdaGrad) of a layer's table against the batches it was given."""
    ids = np.concatenate([i.numpy().reshape(-1) for i, _ in batches])
    clicks = np.concatenate([np.tile(y.cpu().numpy(), len(SLOTS)) for _, y in batches])
    signs, at = np.unique(ids, return_inverse=True)
    assert layer.table.n_rows == len(signs)
    rows = layer.table.rows[layer.table.lookup_rows(torch.from_numpy(signs).to(layer.table.dev)).long()].cpu().numpy()
    assert np.array_equal(rows[:, layer.dim + 1], np.bincount(at))
    assert np.array_equal(rows[:, layer.dim + 2], np.bincount(at, clicks) if layer.use_cvm else np.zeros(len(signs)))
    assert float(layer.link.cnts.abs().sum()) == 0.0


@pytest.mark.parametrize("family", ["wide_deep", "deepfm", "deepfm_cvm"])
@pytest.mark.parametrize("how", ["none", "pre_hook", "copy", "instance", "global"])
def test_layers_whose_input_somebody_changes(tn_gpu, status_ok, family, how):
    tn = tn_gpu
    torch.manual_seed(0)
    kw = dict(dnn_hidden_units=(16, 8), embedding_dim=8, dense_dim=0, bucket_size=4 * B, table_rows=1 << 14,
              sparse_opt=tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.1),
              target_columns=None if family == "deepfm" else ["label"])
    m = (tn.models.WideDeep if family == "wide_deep" else tn.models.DeepFM)(SLOTS, SLOTS, **kw)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)), cuda_graph=False)
    columns = how == "copy"
    other, ids2, y2 = _features(tn, 2, columns)
    lin, undo = m.linear_emb, None
    if how == "pre_hook":
        lin.register_forward_pre_hook(lambda mod, args: (other,) + args[1:])
    elif how == "copy":                        # the same batch in another dict
        lin.register_forward_pre_hook(lambda mod, args: (dict(args[0]),) + args[1:])
    elif how == "instance":
        lin.forward = lambda features, training=None: type(lin).forward(lin, other, training)
    elif how == "global":
        undo = torch_module.register_module_forward_pre_hook(lambda mod, args: (other,) + args[1:] if mod is lin else None)
    try:
        given = []
        for seed in (5, 6):
            f, ids, y = _features(tn, seed, columns)
            m.train_on_batch(f, y)
            given.append((ids, y))
    finally:
        if undo is not None:
            undo.remove()
    _counted(m.deep_emb, given)
    _counted(m.linear_emb, given if how in ("none", "copy") else [(ids2, y2)] * 2)


@pytest.mark.parametrize("change", ["ids", "contents", "labels", "again", "inference"])
def test_a_pull_run_ahead_that_nobody_takes_counts_nothing(tn_gpu, status_ok, change):
    from tensornet_b200.layers.embedding_features import pull_together

    tn = tn_gpu
    layers = []
    for name, dim in (("p", 8), ("q", 1)):
        cols = [tn.feature_column.embedding_column(tn.feature_column.category_column(key=s, bucket_size=4 * B), dim, "sum") for s in SLOTS]
        layers.append(tn.layers.EmbeddingFeatures(cols, tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.1), name=name,
                                                  is_concat=True, target_columns=["label"], rows=1 << 14))
    f, ids, y = _features(tn, 1)
    f2, ids2, y2 = _features(tn, 2)
    assert pull_together(layers, f, True) and all(l.link._pulled is not None for l in layers)
    created, given, use = np.unique(ids.numpy()), [(ids2, y2)], f2
    if change == "contents":                   # the same buffers, filled again in between
        f[tn.data.PACKED_KEY].ids.copy_(f2[tn.data.PACKED_KEY].ids)
        f["label"].copy_(y2)
        use = f
    elif change == "labels":                   # the same ids
        use, given = dict(f, label=y2), [(ids, y2)]
    elif change == "again":
        assert pull_together(layers, f2, True)
    elif change == "inference":
        for l in layers:
            l(f, training=False)
    for l in layers:
        out = l(use, training=True)
        assert l.link._pulled is None
        out.backward(torch.zeros_like(out))
        l.backwards()
        signs = np.concatenate([i.numpy().reshape(-1) for i, _ in given])
        clicks = np.concatenate([np.tile(v.cpu().numpy(), len(SLOTS)) for _, v in given])
        every = np.union1d(created, signs)     # rows of signs that were pulled in vain stay, with nothing counted
        rows = l.table.rows[l.table.lookup_rows(torch.from_numpy(every).to(l.table.dev)).long()].cpu().numpy()
        at = np.searchsorted(every, signs)
        assert l.table.n_rows == len(every)
        assert np.array_equal(rows[:, l.dim + 1], np.bincount(at, minlength=len(every)))
        assert np.array_equal(rows[:, l.dim + 2], np.bincount(at, clicks, minlength=len(every)))
        assert float(l.link.cnts.abs().sum()) == 0.0


def test_a_forward_pass_that_fails_leaves_no_pull_behind(tn_gpu, status_ok):
    tn = tn_gpu
    m = tn.models.WideDeep(SLOTS, SLOTS, dnn_hidden_units=(16, 8), embedding_dim=8, bucket_size=4 * B, table_rows=1 << 14, use_bn=False,
                           sparse_opt=tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.1))
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)), cuda_graph=False)
    m.train()
    f, ids, y = _features(tn, 1)
    combiner, m.linear_emb.combiner = m.linear_emb.combiner, "no such combiner"
    with pytest.raises(Exception):
        m(f)
    m.linear_emb.combiner = combiner
    assert m.deep_emb.link._pulled is None and float(m.deep_emb.link.cnts.abs().sum()) == 0.0
