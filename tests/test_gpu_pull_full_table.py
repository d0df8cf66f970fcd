"""A table that runs full in a pull on one GPU: what the pull does not depend on how its blocks come to run."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _table(tn, rows, n):
    from tensornet_b200.ops.sparse_table_gpu import GpuSparseTable

    t = GpuSparseTable(tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.3), 8, rows=rows)
    return t, t.link(n)


@pytest.mark.parametrize("healthy_first", [False, True])
@pytest.mark.parametrize("front", [False, True])
def test_full_table_leaves_everything_else_of_the_step_whole(tn_gpu, healthy_first, front):
    """Two tables in one launch of many blocks.  The one that is full has rows for the signs it knew and none for the others;
    shows are counted and the scratch is put back; the other table's pull is complete."""
    from tensornet_b200.ops.sparse_table_gpu import GpuSparseLink

    tn = tn_gpu
    n = 400_000
    (full, fl), (well, wl) = _table(tn, 1 << 12, n), _table(tn, 1 << 20, n)
    dev, cap = full.dev, full.row_cap
    g = torch.Generator(device=dev).manual_seed(1)
    known = torch.arange(1, cap - 100, device=dev) * 7919
    fl.pull(known, training=False)
    a = torch.randint(1, 300_000, (n,), generator=g, device=dev) * 7919            # most of them new to the full table
    b = torch.randint(1, 500_000, (n,), generator=g, device=dev) * 104729
    calls = [(fl, a, None, 0, True, None), (wl, b, None, 0, True, None)]
    try:
        if front:
            for lk, ids, *_ in calls:
                lk.prefetch(ids)
        assert GpuSparseLink.pull_many(calls[::-1] if healthy_first else calls)
        for lk, t, ids in ((fl, full, a), (wl, well, b)):
            inv = lk.pull_in_place(ids, training=True)
            out = torch.empty((n, 8), device=dev)
            lk.ctx.pool_fwd(inv, None, n, 1, 0, out, lk.req)
            signs, at, count = torch.unique(ids, return_inverse=True, return_counts=True)
            rows = t.lookup_rows(signs).long()
            has = rows >= 0
            assert lk.unique_counts()[0] == signs.numel() and int(inv.min()) >= 0
            assert bool(has[torch.isin(signs, known)].all()) and (t is full or bool(has.all()))
            want = torch.where(has[:, None], t.rows[rows.clamp(min=0), :8], torch.zeros(1, device=dev))
            assert torch.equal(out, want[at])
            pos = torch.empty(signs.numel(), dtype=torch.long, device=dev)
            pos[at] = inv.long()
            shows = lk.cnts[pos, 0]
            assert torch.equal(shows, count.float())
            assert bool((lk.comm["dd_keys"] == -1).all())
        assert full.n_rows == cap and well.n_rows == torch.unique(b).numel()
        with pytest.raises(tn.core.DeviceError):
            tn.core.runtime().check_status()
        # until recover() no id has a row
        inv = wl.pull_in_place(b, training=True)
        assert wl.unique_counts()[0] == 0 and int(inv.max()) < 0
    finally:
        tn.core.recover()
    inv = wl.pull_in_place(b, training=False)
    assert int(inv.min()) >= 0 and wl.unique_counts()[0] == torch.unique(b).numel()
    tn.core.runtime().check_status()
