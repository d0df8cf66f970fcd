"""Device-resident batch-norm table and layer against the host table (numpy, float64) and plain PyTorch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _host_table(pctr=False, max_count=100000, moment=0.99, C=7):
    from tensornet_b200.ops.bn_table import BnTable

    return BnTable("ref", C, False, moment, max_count, pctr)


@pytest.mark.parametrize("max_count", [100000, 300])
def test_bn_table_matches_host_table(tn_gpu, status_ok, max_count):
    from tensornet_b200.ops.bn_table import GpuBnTable

    C = 37
    dev = tn_gpu.core.runtime().device
    g = GpuBnTable("t", C, False, 0.9, max_count)
    h = _host_table(max_count=max_count, moment=0.9, C=C)
    gen = torch.Generator().manual_seed(3)
    for step in range(8):
        B = [128, 257, 64, 1000][step % 4]
        x = torch.randn(B, C, generator=gen) * (1 + step) + step
        g.push_batch(x.to(dev))
        xd = x.double()
        h.append(xd.sum(0).numpy(), (xd * xd).sum(0).numpy(), np.full(C, float(B)))
        mean_g, var_g = g.get_moments()
        mean_h, var_h = h.get_moments()
        assert np.allclose(mean_g, mean_h, rtol=1e-6, atol=1e-6)
        assert np.allclose(var_g, var_h, rtol=1e-5, atol=1e-5)
    s, q, c = g.totals()
    hs, hq, hc = h.totals()
    assert np.allclose(s, hs, rtol=1e-12) and np.allclose(q, hq, rtol=1e-12) and np.array_equal(c, hc)
    assert float(g.batch.abs().sum()) == 0.0          # per-step scratch comes back clean
    inc = g.take_increments()
    hinc = h.take_increments()
    for a, b in zip(inc, hinc):
        assert np.allclose(a, b, rtol=1e-12)


def test_bn_layer_forward_backward_and_checkpoint(tn_gpu, status_ok, tmp_path):
    tn = tn_gpu
    dev = tn.core.runtime().device
    C, B = 45, 512
    bn = tn.layers.TNBatchNormalization(C, name="bn_gpu_test")
    assert bn._on_device
    bn.train()
    torch.manual_seed(0)
    x = (torch.randn(B, C, device=dev) * 3 + 1).requires_grad_(True)
    with torch.no_grad():
        bn.gamma.copy_(torch.rand(C, device=dev) + 0.5)
        bn.beta.copy_(torch.randn(C, device=dev))
    y = bn(x)
    mean, var = x.detach().mean(0), x.detach().var(0, unbiased=False)
    assert torch.allclose(bn.moving_mean, mean, atol=1e-5) and torch.allclose(bn.moving_variance, var, rtol=1e-4, atol=1e-4)
    ref = (x.detach() - mean) * torch.rsqrt(var + bn.epsilon) * bn.gamma.detach() + bn.beta.detach()
    assert torch.allclose(y, ref, rtol=1e-4, atol=1e-4)
    w = torch.randn(B, C, device=dev)
    (y * w).sum().backward()
    rs = torch.rsqrt(var + bn.epsilon)
    assert torch.allclose(x.grad, w * bn.gamma.detach() * rs, rtol=1e-4, atol=1e-4)
    assert torch.allclose(bn.beta.grad, w.sum(0), rtol=1e-4, atol=1e-3)
    assert torch.allclose(bn.gamma.grad, (w * (x.detach() - mean) * rs).sum(0), rtol=1e-4, atol=1e-2)
    bn.save_bn_table(str(tmp_path))
    bn2 = tn.layers.TNBatchNormalization(C, name="bn_gpu_test2")
    bn2.table.handle = bn.table.handle
    bn2.bn_table_handle = bn.bn_table_handle
    tn.core.load_bn_table(bn.bn_table_handle, str(tmp_path))
    assert torch.allclose(bn.moving_mean, mean, atol=1e-5)
    bn.eval()
    y2 = bn(x.detach())
    assert torch.allclose(y2, ref, rtol=1e-4, atol=1e-4)


def test_pctr_bn_accumulates_deviation_from_current_mean(tn_gpu, status_ok):
    tn = tn_gpu
    dev = tn.core.runtime().device
    C = 9
    bn = tn.layers.PCTRDNNBatchNormalization(C, name="pctr_gpu_test")
    bn.train()
    h = _host_table(pctr=True, C=C)
    gen = torch.Generator().manual_seed(5)
    for _ in range(3):
        x = torch.randn(200, C, generator=gen) + 2
        mean_before = torch.from_numpy(h.get_moments()[0])
        y = bn(x.to(dev))
        xd = x.double()
        h.append(xd.sum(0).numpy(), ((xd - mean_before.double()) ** 2).sum(0).numpy(), np.full(C, 200.0))
    mg, vg = bn.table.get_moments()
    mh, vh = h.get_moments()
    assert np.allclose(mg, mh, rtol=1e-6, atol=1e-6) and np.allclose(vg, vh, rtol=1e-5)


@pytest.mark.parametrize("B,n_h,L", [(1, 5, 1), (33, 32, 3), (700, 250, 26), (129, 64, 40)])
@pytest.mark.parametrize("training", [False, True])
def test_join_matches_the_steps_in_between(tn_gpu, status_ok, B, n_h, L, training):
    """``join_operand`` against normalising the concatenation and building the operand: the same operand, gradients and
    table to the bit but for gamma's and beta's gradients, sums of B 32-bit terms."""
    tn = tn_gpu
    dev = tn.core.runtime().device
    F = tn.ops.functional
    g = torch.Generator().manual_seed(B)
    ldh = F.pad8(n_h + 1)
    h0 = torch.relu(torch.randn((B, ldh), generator=g)).to(dev).bfloat16()
    h0[:, n_h:] = 0
    h0[:, n_h] = 1
    x0 = torch.randn((B, L), generator=g).to(dev)
    C = n_h + L
    gz = torch.randn((B, F.pad8(C + 1)), generator=g).to(dev).bfloat16()
    got = []
    for joined in (False, True):
        bn = tn.layers.TNBatchNormalization(C, synchronized=True, sync_freq=4, max_count=1000000, name=f"join{joined}{B}{training}")
        with torch.no_grad():
            bn.gamma.copy_(torch.linspace(0.5, 1.5, C))
            bn.beta.copy_(torch.linspace(-0.5, 0.5, C))
        bn.table.push_batch(torch.randn((50, C), generator=torch.Generator().manual_seed(1)).to(dev) * 2 + 1)
        bn.train(training)
        h, x = h0.clone().requires_grad_(), x0.clone().requires_grad_()
        for _ in range(5):                               # across an exchange of the increments
            h.grad = x.grad = bn.gamma.grad = bn.beta.grad = None
            if joined:
                z = bn.join_operand(h, n_h, x, masked=True)
            else:
                z = F.concat_cast([bn(torch.cat([h[:, :n_h].float(), x], dim=1))], ones=True)
            z.backward(gz)
        gh = h.grad.clone()
        if not joined:
            gh[:, :n_h] = torch.where(h0[:, :n_h] > 0, gh[:, :n_h], torch.zeros_like(gh[:, :n_h]))
        got.append((z.detach(), gh, x.grad, bn.table.inc.clone(), bn.table.total_sum.clone(), bn.gamma.grad, bn.beta.grad, bn.batch_counter))
    a, b = got
    assert a[-1] == b[-1]
    for k in range(3):
        assert torch.equal(a[k], b[k]), k
    for k in (3, 4):                                     # 64-bit sums whose order is free
        assert bool(((a[k] - b[k]).abs() <= 1e-12 * (1 + a[k].abs())).all())
    for k in (5, 6):
        assert bool(((a[k] - b[k]).abs() <= B * 2.0 ** -23 * 20 + 1e-6).all())


def test_use_fused_holds_for_the_joint_kernels(tn_gpu, status_ok):
    """``use_fused = False`` keeps Wide&Deep's tower, batch norm and head apart, in training and in scoring."""
    tn = tn_gpu
    torch.manual_seed(1)
    slots, B = ["a", "b"], 40
    m = tn.models.WideDeep(slots, slots, dnn_hidden_units=(16, 8), embedding_dim=8, bucket_size=4 * B, table_rows=1 << 12)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)), cuda_graph=False)
    f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=torch.arange(2 * B).view(2, B) % 50)}
    y = (torch.arange(B) % 3 == 0).float()
    joined, join = [], m.sub_model.bn.join_operand
    m.sub_model.bn.join_operand = lambda *a, **k: joined.append(1) or join(*a, **k)
    for fused, seen in ((True, 2), (False, 2), (True, 4)):
        m.use_fused = fused
        m.train_on_batch(f, y)
        m.predict_step((f, y))
        assert len(joined) == seen
