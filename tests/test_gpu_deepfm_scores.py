"""DeepFM scores through the fused input kernel it trains with."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [False, True])
@pytest.mark.parametrize("dense_dim", [0, 5])
def test_deepfm_scores_through_the_fused_input(tn_gpu, status_ok, share, dense_dim):
    """Scores with the fused input kernel against those of the layers one by one (a hook on the sub-model keeps them apart),
    signs the table does not hold among them; ragged batches take the general path."""
    tn = tn_gpu
    dev = tn.core.runtime().device
    torch.manual_seed(3)
    slots, B = [str(i) for i in range(6)], 301
    opt = tn.core.Adam(learning_rate=1e-2, initial_scale=0.3) if share else tn.core.AdaGrad(learning_rate=1e-2, initial_scale=0.3)
    m = tn.models.DeepFM(slots, slots, dnn_hidden_units=(32, 16), embedding_dim=8, dense_dim=dense_dim, sparse_opt=opt, bucket_size=4 * B,
                         table_rows=1 << 14, share_linear_table=share)
    m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-2)), cuda_graph=False)
    g = torch.Generator().manual_seed(5)
    ids = torch.randint(0, 3000, (6, B), generator=g)
    f = {tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=ids)}
    if dense_dim:
        f["dense"] = torch.randn((B, dense_dim), generator=g)
    y = (torch.rand(B, generator=g) < 0.3).float()
    for _ in range(3):
        m.train_on_batch(f, y)
    f2 = dict(f)
    f2[tn.data.PACKED_KEY] = tn.data.PackedFeatures(slots, ids=torch.cat([ids[:, :200], ids[:, 200:] + 10 ** 6], 1).to(dev))
    if dense_dim:
        f2["dense"] = f["dense"].to(dev)
    m.eval()
    with torch.no_grad():
        assert m._scores(f2) is not None
        fused = m(f2)
        seen = []
        handle = m.sub_model.register_forward_hook(lambda *a: seen.append(1))
        assert m._scores(f2) is None
        plain = m(f2)
        handle.remove()
        assert seen
        lens = torch.full((6 * B,), 2)
        offs = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)]).int()
        f3 = dict(f2)
        f3[tn.data.PACKED_KEY] = tn.data.PackedFeatures(slots, values=ids.reshape(-1).repeat_interleave(2).to(dev), offsets=offs.to(dev), batch_size=B)
        assert m._scores(f3) is None and m(f3).shape == fused.shape
    assert m._scores(f2) is None                                     # gradients are wanted
    # the operands are the same bf16 values but for the FM term's order of 32-bit sums: one step of bf16 in one of 23 inputs
    assert bool(((fused - plain).abs() <= 2.0 ** -8 * (1 + plain.abs())).all())
