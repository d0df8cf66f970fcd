"""The batch norm's training step in one launch against its three kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,n_h,L", [(1, 5, 1), (32, 256, 4), (33, 0, 3), (64, 16, 7), (65, 9, 8), (256, 250, 26), (257, 64, 40), (1024, 40, 1),
                                     (1025, 3, 2), (2048, 30, 5), (2049, 30, 5)])
@pytest.mark.parametrize("affine,max_count", [(True, 1000000), (False, 3)])
def test_one_launch_matches_three(tn_gpu, status_ok, B, n_h, L, affine, max_count):
    """Operand and moments to the bit (the sums are of 64 bits, in another order), totals to 64-bit rounding, over batches that are kept
    for an exchange and one that drops them, with the moving window (``max_count`` of 3) and without."""
    from tensornet_b200.ops.bn_table import GpuBnTable

    F = tn_gpu.ops.functional
    dev = tn_gpu.core.runtime().device
    C = n_h + L
    ldz, ldh = F.pad8(C + 1), F.pad8(n_h + 1)
    gen = torch.Generator().manual_seed(B + L)
    gamma = (torch.rand(C, generator=gen) + 0.5).to(dev) if affine else None
    beta = torch.randn(C, generator=gen).to(dev) if affine else None
    tables = [GpuBnTable(f"t{k}", C, True, 0.9, max_count) for k in range(2)]
    for step in range(4):
        h = torch.relu(torch.randn((B, ldh), generator=gen) * (1 + step)).to(dev).bfloat16()
        x = (torch.randn((B, L + 3), generator=gen) * 2 + step).to(dev)[:, 1:L + 1]
        out = []
        for k, t in enumerate(tables):
            z = torch.full((B, ldz), 7.0, dtype=torch.bfloat16, device=dev)
            moments = torch.full((2 * C,), 7.0, device=dev)
            if k:
                t.ctx.join_train(h, n_h, x, gamma, beta, 1e-5, step == 2, z, moments)
            else:
                t.push_batch(x, False, step == 2, h, n_h)
                t.ctx.join_fwd(h, n_h, x, gamma, beta, 1e-5, z, moments)
            out.append((z, moments, t.mean.clone(), t.var.clone()))
        for a, b in zip(out[0][1:] + out[0][:1], out[1][1:] + out[1][:1]):
            assert torch.equal(a, b), (step, a.shape, (a.float() - b.float()).abs().max())
        for name in ("total_count", "total_sum", "total_sq", "inc"):
            a, b = [getattr(t, name) for t in tables]
            assert bool(((a - b).abs() <= 1e-12 * B * (1 + a.abs())).all()), (name, step)
        assert torch.equal(tables[0].total_count, tables[1].total_count)
        assert all(float(t.batch.abs().sum()) == 0.0 for t in tables)
