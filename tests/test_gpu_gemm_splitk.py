"""GEMMs whose output tile is shared by a cluster that splits K."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,BN", [(2, 64), (4, 128), (8, 64), (8, 256)])
@pytest.mark.parametrize("M,N,K,b_mn", [(1, 64, 1024, False), (130, 200, 1030, False), (128, 263, 1025, True), (257, 72, 2111, False)])
def test_cluster_split_matches_fp32(tn_gpu, status_ok, S, BN, M, N, K, b_mn):
    """Edges of the tiles, a ragged last k-block, the ones column inside and beyond the last tile, ReLU and the ReLU mask.
    Operands are bf16 and sums fp32; what is left is the rounding of the result, at most 2^-9 of each value."""
    from tensornet_b200 import _build

    kt = (K + 63) // 64
    if kt < 2 * S or -(-kt // -(-kt // S)) != S:
        pytest.skip("not every CTA of the cluster would have two k-blocks")
    ext, rt = _build.cuda_ext(), tn_gpu.core.runtime()
    g = torch.Generator(device=rt.device).manual_seed(M + N + K)
    pad = lambda n: (n + 7) // 8 * 8
    lda, ldc = pad(K), pad(N + 1)
    A = torch.randn((M, lda), generator=g, device=rt.device).bfloat16()
    W = torch.randn((K, pad(N)) if b_mn else (N, lda), generator=g, device=rt.device).bfloat16()
    ref = A[:, :K].float() @ (W[:, :N].float() if b_mn else W[:, :K].float().t())
    for mask in (None, torch.randn((M, ldc), generator=g, device=rt.device).bfloat16()):
        C = torch.full((M, ldc), 7.0, dtype=torch.bfloat16, device=rt.device)
        ext.gemm(A, W, C, M, N, K, lda, int(W.stride(0)), ldc, False, b_mn, False, mask is None, None, mask, None, None,
                 ldc if mask is not None else 0, N, ldc, 1, BN, rt.status, cluster_k=S)
        want = torch.relu(ref) if mask is None else torch.where(mask[:, :N].float() > 0, ref, torch.zeros_like(ref))
        err = (C[:, :N].float() - want).abs()
        assert bool((err <= want.abs() * 2 ** -8 + 1e-3 * K ** 0.5).all()), float(err.max())
        assert bool((C[:, N] == 1).all()) and bool((C[:, N + 1:] == 0).all())
