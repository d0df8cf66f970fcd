"""The native request path against the module path (same dictionary, same tower)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 3, 17, 130, 1024])
@pytest.mark.parametrize("where", ["pinned", "pageable", "device"])
@pytest.mark.parametrize("ragged", [False, True])
def test_native_requests_equal_the_modules(tn_gpu, status_ok, B, where, ragged):
    """Both round rows and weights to bf16 and accumulate in fp32: logits differ by the order of the sums and by roundings
    of the hidden activations that flip with it, a bf16 step (2^-8) of a few of them; probabilities by a quarter of that."""
    from tensornet_b200.layers import DenseHead, MLP
    from tensornet_b200.serving import EmbeddingDictionary, InferenceEngine

    tn = tn_gpu
    dev = tn.core.runtime().device
    S, D = 37, 12
    rng = np.random.default_rng(B)
    signs = np.unique(rng.integers(1, 2 ** 40, 20_000).astype(np.uint64))
    torch.manual_seed(B)
    mlp, head = MLP(S * D, [200, 64, 33]).to(dev), DenseHead(33).to(dev)
    d = EmbeddingDictionary(signs, rng.standard_normal((len(signs), D)).astype(np.float32))
    eng = InferenceEngine(d, mlp, head, S, combiner="mean")
    assert eng._ctx is not None
    lens = torch.from_numpy(rng.integers(0, 40 if B < 20 else 6, S * B)) if ragged else torch.ones(S * B, dtype=torch.int64)
    offs = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).int()
    n = int(offs[-1])
    ids = np.where(rng.random(n) < 0.8, signs[rng.integers(0, len(signs), n)].view(np.int64), rng.integers(2 ** 41, 2 ** 42, n))
    ids = torch.from_numpy(ids)
    with torch.no_grad():
        want = eng._forward_gpu(ids.to(dev), offs.to(dev) if ragged else None, B)
    if not ragged:
        ids = ids.view(S, B)
    move = {"pinned": lambda t: t.pin_memory(), "pageable": lambda t: t, "device": lambda t: t.to(dev)}[where]
    got = eng.infer(move(ids), move(offs) if ragged else None)
    assert torch.allclose(got, want, atol=2 ** -10), float((got - want).abs().max())


def test_weights_written_between_requests_are_seen(tn_gpu, status_ok):
    from tensornet_b200.layers import DenseHead, MLP
    from tensornet_b200.serving import EmbeddingDictionary, InferenceEngine

    dev = tn_gpu.core.runtime().device
    mlp, head = MLP(8, [16]).to(dev), DenseHead(16).to(dev)
    eng = InferenceEngine(EmbeddingDictionary(np.arange(1, 9, dtype=np.uint64), np.ones((8, 4), np.float32)), mlp, head, 2)
    for B in (1, 40):
        ids = torch.randint(1, 9, (2, B))
        a = eng.infer(ids).clone()
        mlp.weights[0].data.mul_(-1.0)
        assert not torch.equal(a, eng.infer(ids))


def test_requests_follow_what_the_engine_is_made_of(tn_gpu, status_ok):
    """Another dictionary, another tower, an attribute of it, a hook on it: between two requests, ragged and not."""
    from tensornet_b200.layers import DenseHead, MLP
    from tensornet_b200.serving import EmbeddingDictionary, InferenceEngine

    dev = tn_gpu.core.runtime().device
    torch.manual_seed(1)
    make = lambda: (MLP(8, [16, 8]).to(dev), DenseHead(8).to(dev))
    signs = np.arange(1, 9, dtype=np.uint64)
    rows = lambda seed: np.random.default_rng(seed).standard_normal((8, 4)).astype(np.float32)
    mlp, head = make()
    eng = InferenceEngine(EmbeddingDictionary(signs, rows(0)), mlp, head, 2)
    ids = torch.randint(1, 9, (2, 40))
    offs = torch.arange(81, dtype=torch.int32)

    def follows():
        with torch.no_grad():
            want = eng._forward_gpu(ids.to(dev).reshape(-1), offs.to(dev), 40)
        for got in (eng.infer(ids), eng.infer(ids.reshape(-1), offs)):
            assert torch.allclose(got, want, atol=2 ** -10), float((got - want).abs().max())      # bound: see above
        return want

    seen = [follows()]

    def changed():
        seen.append(follows())
        assert not torch.allclose(seen[-1], seen[-2], atol=2 ** -8)

    eng.dict = EmbeddingDictionary(signs, rows(1))
    changed()
    eng.mlp, eng.head = make()
    changed()
    eng.mlp.relu_last = False
    changed()
    flat = torch.zeros(16 * 16 + 1, device=dev)[1:].view(16, 16)          # weights off the 16-byte boundary
    flat.copy_(eng.mlp.weights[0].detach())
    eng.mlp.weights[0].data = flat
    follows()
    calls = []
    handle = eng.mlp.register_forward_hook(lambda *_: calls.append(1))
    for k in range(3):
        eng.infer(ids.reshape(-1), offs)
    assert len(calls) == 3
    handle.remove()
    follows()


@pytest.mark.parametrize("B", [2, 40, 700])
@pytest.mark.parametrize("ragged", [False, True])
def test_page_locked_buffers_may_be_filled_again(tn_gpu, status_ok, B, ragged):
    """A request with offsets, or one outside a graph, that is queued behind other work: its buffers are written over as
    soon as the call returns.  2: read in place; 40: in place, layers on the tensor cores; 700: copied."""
    from tensornet_b200.layers import DenseHead, MLP
    from tensornet_b200.serving import EmbeddingDictionary, InferenceEngine

    dev = tn_gpu.core.runtime().device
    S = 40
    torch.manual_seed(B)
    mlp, head = MLP(S * 4, [32, 16]).to(dev), DenseHead(16).to(dev)
    rows = np.random.default_rng(0).standard_normal((100, 4)).astype(np.float32)
    eng = InferenceEngine(EmbeddingDictionary(np.arange(1, 101, dtype=np.uint64), rows), mlp, head, S)
    ids = torch.randint(1, 101, (S, B)).pin_memory()
    offs = torch.arange(S * B + 1, dtype=torch.int32).pin_memory()
    args = (ids.reshape(-1), offs) if ragged else (ids,)
    want = eng.infer(*args, use_graph=False).clone()
    for _ in range(3):
        keep = ids.clone(), offs.clone()
        torch.cuda._sleep(1_000_000)                  # half a millisecond of other work in front
        got = eng.infer(*args, use_graph=False)
        ids.fill_(7)
        offs.fill_(0)
        assert torch.equal(got, want)
        ids.copy_(keep[0])
        offs.copy_(keep[1])
