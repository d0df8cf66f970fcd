"""The rank-1 cross network as a whole against its layers in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 3, 8])
@pytest.mark.parametrize("B,D", [(1, 1), (3, 31), (37, 200), (4096, 200), (300, 256), (515, 257), (70, 512), (90, 800), (33, 1024), (20, 1030)])
def test_cross_network_matches_its_layers(tn_gpu, status_ok, B, D, L):
    tn = tn_gpu
    F = tn.ops.functional
    dev = tn.core.runtime().device
    g = torch.Generator(device=dev).manual_seed(B + D + L)
    x = torch.randn((B, D), generator=g, device=dev)
    ws = [torch.randn((D, 1), generator=g, device=dev) * (0.5 / D ** 0.5) for _ in range(L)]
    bs = [torch.randn(D, generator=g, device=dev) * 0.1 for _ in range(L)]
    gy = torch.randn((B, D), generator=g, device=dev)

    def run(dtype, net):
        p = [t.to(dtype).requires_grad_() for t in (x, *ws, *bs)]
        y = net(p[0], p[1:1 + L], p[1 + L:])
        y.backward(gy.to(dtype))
        return [y.detach()] + [q.grad for q in p]

    def layers(step):
        def net(x0, w, b):
            c = x0
            for k in range(L):
                c = step(x0, c, w[k], b[k])
            return c
        return net

    want = run(torch.float64, layers(lambda x0, c, w, b: x0 * (c @ w) + b + c))
    one = run(torch.float32, layers(F.cross_v1))
    got = run(torch.float32, F.cross_v1_net)
    for a, o, w in zip(got, one, want):
        assert a.shape == w.shape
        err, before = float((a.double() - w).norm() / w.norm()), float((o.double() - w).norm() / w.norm())
        assert err <= 2 * before + 1e-7, (err, before)         # no further from 64 bits than the layers one by one (1e-7: ulp)
