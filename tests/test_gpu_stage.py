"""Inputs of captured steps on their way to the device: many small ones in one launch, columns one behind the other."""
import pytest
import torch

import tensornet_b200 as tn
from tensornet_b200 import _build
from tensornet_b200.data.features import adjacent_columns, gather_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("shift", [0, 1, 4, 8])          # bytes from a 16-byte boundary
def test_staged_inputs_arrive_whole(pinned, shift):
    tn.core.init()
    ext = _build.cuda_ext()
    # nothing, a byte, odd tails, exactly a block, one over, larger than what a kernel reads, and more pieces than a launch takes
    sizes = [0, 1, 15, 16, 17, 4095, 8192, 8193, 100_000, 256 * 1024, 256 * 1024 + 16, 1_000_001] + [33] * 120
    g = torch.Generator().manual_seed(shift)
    whole = [torch.randint(0, 255, (n + shift,), generator=g, dtype=torch.uint8) for n in sizes]
    whole = [w.pin_memory() if pinned and w.numel() else w for w in whole]
    srcs = [w[shift:] for w in whole]
    dsts = [torch.zeros(n + shift + 7, dtype=torch.uint8, device="cuda")[shift: shift + n] for n in sizes]
    room = [torch.full((n + 5,), 9, dtype=torch.uint8, device="cuda") if n % 2 else d for n, d in zip(sizes, dsts)]      # buffers with room to spare
    copy, done = torch.cuda.Stream(), torch.cuda.Event()
    done.record()
    for _ in range(2):
        ext.stage_inputs(room, srcs, copy.cuda_stream, torch.cuda.current_stream().cuda_stream, 0, done.cuda_event, 0)
    for d, s in zip(room, srcs):
        assert torch.equal(d[: s.numel()].cpu(), s) and bool((d[s.numel():] == 9).all())


def test_memory_that_is_page_locked_in_part_is_not_read_by_a_kernel():
    """A leaf of which only the first page is registered: copied, or refused by the copy; and the context is as before."""
    tn.core.init()
    ext = _build.cuda_ext()
    page = 4096
    room = torch.arange(6 * page, dtype=torch.int64).to(torch.uint8)
    at = -room.data_ptr() % page
    part = room[at: at + 2 * page + 8]
    srcs = [torch.full((100,), k, dtype=torch.uint8).pin_memory() for k in range(4)] + [part]
    dsts = [torch.zeros(s.numel(), dtype=torch.uint8, device="cuda") for s in srcs]
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(part.data_ptr(), page, 0)) == 0
    try:
        copy, done = torch.cuda.Stream(), torch.cuda.Event()
        done.record()
        try:
            ext.stage_inputs(dsts, srcs, copy.cuda_stream, torch.cuda.current_stream().cuda_stream, 0, done.cuda_event, 0)
        except RuntimeError as e:
            assert "cudaMemcpyAsync" in str(e)
        else:
            torch.cuda.synchronize()
            assert all(torch.equal(d.cpu(), s) for d, s in zip(dsts, srcs))
        torch.cuda.synchronize()
    finally:
        rt.cudaHostUnregister(part.data_ptr())
    assert float(torch.ones(4, device="cuda").sum()) == 4.0


def test_columns_next_to_each_other_are_taken_as_they_lie():
    tn.core.init()
    ids = torch.randint(0, 100, (4, 10), device="cuda")
    f = {str(k): ids[k] for k in range(4)}
    got, offsets, B = gather_columns(f, ["0", "1", "2", "3"], ids.device)
    assert got.data_ptr() == ids.data_ptr() and offsets is None and B == 10 and torch.equal(got, ids.reshape(-1))
    got, _, _ = gather_columns(f, ["1", "0", "2"], ids.device)                   # another order: packed anew
    assert torch.equal(got, ids[[1, 0, 2]].reshape(-1))
    assert adjacent_columns([ids[0], ids[2]]) is None and adjacent_columns([ids[0], ids[1].clone()]) is None
    assert adjacent_columns([ids[0].int(), ids[1].int()]) is None and adjacent_columns([ids[0], ids[1][:5]]) is None
    assert adjacent_columns([ids[:, 0], ids[:, 1]]) is None
    assert torch.equal(adjacent_columns([ids[1].view(10, 1), ids[2].view(10, 1)]), ids[1:3].reshape(-1))


@pytest.mark.parametrize("model", ["wide_deep", "deepfm"])
def test_fit_and_predict_over_columns_match_packed_batches(model):
    """One tensor per slot and one packed buffer: the same steps."""
    tn.core.init()
    S, B, slots = 6, 130, [str(k) for k in range(6)]
    g = torch.Generator().manual_seed(3)
    data = [(torch.randint(0, 400, (S, B), generator=g), torch.randn(B, 3, generator=g), (torch.rand(B, generator=g) < 0.3).float()) for _ in range(12)]
    runs = []
    for packed in (True, False):
        torch.manual_seed(1)
        cls = tn.models.WideDeep if model == "wide_deep" else tn.models.DeepFM
        with torch.device("cuda"):
            m = cls(slots, slots, dnn_hidden_units=(32, 16), embedding_dim=8, dense_dim=3, bucket_size=B, table_rows=1 << 14)
        m.compile(optimizer=tn.optimizer.Optimizer(tn.core.Adam(learning_rate=1e-3)))
        batches = []
        for ids, dense, y in data:
            f = ({tn.data.PACKED_KEY: tn.data.PackedFeatures(slots, ids=ids.pin_memory())} if packed else
                 {s: ids[k].clone().pin_memory() for k, s in enumerate(slots)})
            f["dense"] = dense.pin_memory()
            batches.append((f, y.pin_memory()))
        hist = m.fit(batches, epochs=2, record_step_loss=True)
        runs.append((torch.tensor(hist["step_loss"]), m.predict([(f, y) for f, y in batches])[1]))
        tn.core.runtime().check_status()
    assert torch.allclose(runs[0][0], runs[1][0], rtol=2e-3, atol=1e-4)
    assert torch.allclose(torch.as_tensor(runs[0][1]), torch.as_tensor(runs[1][1]), rtol=2e-2, atol=1e-2)
