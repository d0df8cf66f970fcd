"""One GPU: the pull that leaves rows in the table (two ordinary kernels, pooling reads the rows in place) against the exchange
kernel that writes them to the per-batch matrix (``staged_row_return``), over every form a batch can have."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(tn, dim, kind, cvm, combiner, slots, bucket, staged, rows=1 << 14):
    old, tn.core.config.staged_row_return = tn.core.config.staged_row_return, int(staged)
    try:
        cols = [tn.feature_column.embedding_column(tn.feature_column.category_column(key=s, bucket_size=bucket), dim, combiner) for s in slots]
        opt = {"adagrad": tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.3),
               "adam": tn.core.Adam(learning_rate=0.01, initial_scale=0.3), "ftrl": tn.core.Ftrl(learning_rate=0.05, initial_scale=0.3)}[kind]
        layer = tn.layers.EmbeddingFeatures(cols, opt, name="e", is_concat=True, target_columns=["label"] if cvm else None, rows=rows)
    finally:
        tn.core.config.staged_row_return = old
    assert layer.link.ctx.in_place() == (not staged)
    return layer


def _batch(tn, g, slots, B, ragged, top, dev):
    S = len(slots)
    lens = torch.randint(0, 6, (S * B,), generator=g) if ragged else torch.ones(S * B, dtype=torch.long)
    offs = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)])
    ids = (torch.randint(0, top, (int(offs[-1]),), generator=g) ** 2 // top * 104729 + 5).to(dev)
    y = (torch.rand(B, generator=g) < 0.4).float().to(dev)
    p = (tn.data.PackedFeatures(slots, values=ids, offsets=offs.int().to(dev), batch_size=B) if ragged else
         tn.data.PackedFeatures(slots, ids=ids.view(S, B)))
    return {tn.data.PACKED_KEY: p, "label": y}, torch.unique(ids)


@pytest.mark.parametrize("dim,kind,cvm", [(1, "adagrad", False), (1, "adagrad", True), (2, "adagrad", True), (3, "adam", False),
                                          (8, "adagrad", True), (10, "ftrl", False), (12, "adam", False), (38, "adagrad", True),
                                          (64, "ftrl", False), (128, "adagrad", False), (140, "adam", False)])
@pytest.mark.parametrize("ragged,combiner,B", [(False, "sum", 1), (False, "mean", 700), (True, "sum", 333), (True, "mean", 40), (True, "sqrtn", 2050)])
def test_in_place_pull_matches_the_exchange_kernel(tn_gpu, status_ok, dim, kind, cvm, ragged, combiner, B):
    tn = tn_gpu
    dev = tn.core.runtime().device
    slots = ["a", "b", "c"]
    got = []
    for staged in (True, False):
        layer = _layer(tn, dim, kind, cvm, combiner, slots, 6 * B + 8, staged)
        g = torch.Generator().manual_seed(dim * 7 + B)
        outs = []
        for step in range(4):                    # new signs in every step; the third one is inference, which makes zero rows
            f, signs = _batch(tn, g, slots, B, ragged, 200 * (step + 1), dev)
            train = step != 2
            out = layer(f, training=train)
            outs.append(out.detach().clone())
            assert layer.link.unique_counts()[0] == signs.numel()
            if not train:
                continue
            grad = ((torch.arange(out.numel(), device=dev) % 13).float() - 6).view_as(out) / 4      # sums of quarters: exact in any order
            out.backward(grad)
            layer.backwards()
            assert float(layer.link.gU.abs().sum()) == 0.0 and float(layer.link.cnts.abs().sum()) == 0.0
            rows = layer.table.lookup_rows(signs).long()
            assert signs.numel() == 0 or int(rows.min()) >= 0
            outs.append(layer.table.rows[rows][:, : dim + 3 if kind == "adagrad" else 3 * dim].clone())
        outs.append(torch.tensor(float(layer.table.n_rows)))
        got.append(outs)
    # single ids and plain sums: gradients are sums of quarters, exact in any order, and all is the same to the bit.  With a
    # scale the sums of the gradients depend on their order, so only what comes before the first update is compared.
    exact = not ragged or combiner == "sum"
    assert len(got[0]) == len(got[1]) == 8
    for a, b in list(zip(*got))[: None if exact else 1]:
        assert torch.equal(a, b), float((a - b).abs().max())
    assert float(got[0][-1]) == float(got[1][-1])


@pytest.mark.parametrize("n", [1, 33, 5000, 151553, 460001])
@pytest.mark.parametrize("lookup_only", [False, True])
def test_in_place_pull_of_every_batch_size(tn_gpu, status_ok, n, lookup_only):
    """One to four ids per lane, half of the signs known: rows found, created or (``lookup_only``) left out."""
    from tensornet_b200.ops.sparse_table_gpu import GpuSparseTable

    tn = tn_gpu
    t = GpuSparseTable(tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.3), 6, rows=1 << 20)
    lk = t.link(n)
    g = torch.Generator(device=t.dev).manual_seed(n)
    ids = torch.randint(0, max(2, n), (n,), generator=g, device=t.dev) * 7919 + 3
    uniq = torch.unique(ids)
    known = uniq[::2].contiguous()
    lk.pull(known, training=False)
    assert t.n_rows == known.numel()
    inv = lk.pull_in_place(ids, training=False, lookup_only=lookup_only)
    out = torch.empty((n, 6), device=t.dev)
    lk.ctx.pool_fwd(inv, None, n, 1, 0, out, lk.req)
    assert t.n_rows == (known.numel() if lookup_only else uniq.numel())
    rows = t.lookup_rows(ids).long()
    want = torch.where((rows >= 0)[:, None], t.rows[rows.clamp(min=0), :6], torch.zeros(1, device=t.dev))
    assert torch.equal(out, want)
    assert torch.equal(rows < 0, ~torch.isin(ids, known)) or not lookup_only
    lk.pull(ids, training=False, lookup_only=lookup_only, inverse=inv)
    assert torch.equal(lk.U[inv.long(), :6], want)
    assert bool((lk.comm["dd_keys"] == -1).all())


def test_front_that_has_looked_its_signs_up_meets_a_changed_table(tn_gpu, status_ok):
    """Between a front and its pull rows may be loaded, the shard may grow, and compaction moves rows: the pull finds them all."""
    import numpy as np
    from tensornet_b200.ops.sparse_table_gpu import GpuSparseTable, row_floats

    tn = tn_gpu
    t = GpuSparseTable(tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.3), 4, rows=1 << 10)
    lk = t.link(600)
    a = torch.arange(1, 501, device=t.dev) * 7919
    lk.pull(a[:300].contiguous(), training=False)
    shows = torch.zeros(600, device=t.dev)

    def check(ids):
        inv = lk.pull_in_place(ids, training=True)
        out = torch.empty((ids.numel(), 4), device=t.dev)
        lk.ctx.pool_fwd(inv, None, ids.numel(), 1, 0, out, lk.req)
        rows = t.lookup_rows(ids).long()
        assert int(rows.min()) >= 0 and torch.equal(out, t.rows[rows, :4])
        lk.push()
        shows[ids // 7919] += 1
        assert torch.equal(t.rows[t.lookup_rows(ids).long(), 5], shows[ids // 7919])

    lk.prefetch(a)
    extra = np.zeros((50, row_floats(t.kind, 4)), np.float32)
    extra[:, :4] = 7.0
    t.load_rows((np.arange(400, 450) * 7919).astype(np.uint64), extra)
    check(a)
    assert float(t.rows[t.lookup_rows(a[399:400]).long(), 0]) == 7.0
    lk.prefetch(a)
    t.grow(1 << 12)
    check(a)
    lk.prefetch(a)
    keep = torch.ones(t.n_rows, dtype=torch.bool, device=t.dev)
    keep[::3] = False
    shows[t.row_keys[: t.n_rows][::3] // 7919] = 0
    t.compact(keep)
    check(a)
    lk.prefetch(a)
    t.clear()
    shows.zero_()
    check(a)


@pytest.mark.parametrize("ragged", [False, True])
def test_pulls_of_two_layers_side_by_side(tn_gpu, status_ok, ragged):
    """One launch for both tables against one pull after the other; with fronts ahead of both, of one and of none."""
    from tensornet_b200.layers.embedding_features import pull_together

    tn = tn_gpu
    dev = tn.core.runtime().device
    slots, B = ["a", "b"], 500
    got = []
    for together in (False, True):
        layers = [_layer(tn, 1, "adagrad", True, "sum", slots, 6 * B + 8, False), _layer(tn, 12, "adam", False, "sum", slots, 6 * B + 8, False)]
        g = torch.Generator().manual_seed(3)
        outs = []
        batches = [_batch(tn, g, slots, B, ragged, 300 * (k + 1), dev) for k in range(5)]
        for k, (f, signs) in enumerate(batches):
            if not ragged:
                for layer in layers[: {3: 1, 4: 2}.get(k, 0)]:
                    layer.link.prefetch(layer.ids_pulled_for(f))
            if together:
                pull_together(layers, f, k != 2)
                assert all(layer.link._pulled is not None for layer in layers)
            for layer in layers:
                out = layer(f, training=k != 2)
                assert layer.link._pulled is None
                outs.append(out.detach().clone())
                if k != 2:
                    out.backward(((torch.arange(out.numel(), device=dev) % 13).float() - 6).view_as(out) / 4)
            for layer in layers:
                layer.backwards()
                outs.append(layer.table.rows[layer.table.lookup_rows(signs).long()][:, : 4 if layer.dim == 1 else 36].clone())
        got.append(outs)
    for a, b in zip(*got):
        assert torch.equal(a, b)
    # a pull that was run ahead is for that batch only: other ids are pulled again
    (f, _), (f2, s2) = batches[0], batches[1]
    pull_together(layers, f, True)
    for layer in layers:
        out = layer(f2, training=False)
        assert layer.link.unique_counts()[0] == s2.numel() and out.shape[0] == B
