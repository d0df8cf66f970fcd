"""AdaGrad row updates of one GPU where the width is no multiple of four, against the same mathematics in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(1, 1), (1, 40001), (2, 513), (3, 77), (5, 3000), (6, 31), (7, 2), (10, 90000), (29, 700), (61, 100), (122, 5000),
                                   (123, 3), (125, 200), (127, 90)])
def test_adagrad_push_of_odd_widths(tn_gpu, status_ok, dim, n):
    from tensornet_b200.ops.sparse_table_gpu import GpuSparseTable

    tn = tn_gpu
    opt = tn.core.AdaGrad(learning_rate=0.05, initial_g2sum=0.1, initial_scale=0.3)
    t = GpuSparseTable(opt, dim, rows=1 << 17)
    lk = t.link(n)
    ids = (torch.arange(n, device=t.dev) * 104729 + 5) * 1000003
    labels = (torch.arange(n, device=t.dev) % 3 == 0).float()
    g = torch.Generator(device=t.dev).manual_seed(dim)
    for _ in range(2):
        lk.pull(ids, labels=labels, training=True)
        at = t.lookup_rows(lk.comm["stage_ids"][:n]).long()
        t.rows[at, dim + 3] = 7.0
        before, rest = t.rows[at].double(), t.rows[at][:, dim + 4:].clone()
        lk.gU[:n, :dim] = torch.randn((n, dim), generator=g, device=t.dev)
        x, clicks = lk.gU[:n, :dim].double(), lk.cnts[:n, 1].double()
        lk.push()
        got = t.rows[at]
        assert float(lk.gU.abs().sum()) == 0.0 and float(lk.cnts.abs().sum()) == 0.0
        acc = before[:, dim] + (x * x).mean(1)
        step = opt.learning_rate * x / (opt.epsilon + acc.sqrt())[:, None]
        # a sum of 128 squares, a root and a quotient: below 2^-19 of the magnitudes that enter
        for a, b, size in ((got[:, :dim], before[:, :dim] - step, before[:, :dim].abs() + step.abs()), (got[:, dim], acc, acc)):
            assert bool(((a.double() - b).abs() <= 2.0 ** -19 * size + 1e-12).all())
        assert torch.equal(got[:, dim + 1].double(), before[:, dim + 1] + 1) and torch.equal(got[:, dim + 2].double(), before[:, dim + 2] + clicks)
        assert not bool(got[:, dim + 3].any()) and torch.equal(got[:, dim + 4:], rest)
