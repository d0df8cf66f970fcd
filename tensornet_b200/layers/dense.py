"""Dense building blocks that run on the tcgen05 GEMM family.

The reference builds its towers from Keras ``Dense`` layers, ``FMLayer`` and ``DeepCrossLayer``
(examples/models/deepfm.py:37-57, examples/common/layers.py:21-103).  Here activations travel
between layers as bf16 matrices padded to a multiple of 8 columns whose first pad column is
the constant 1, so every layer is one GEMM with the bias folded into the weight matrix.
"""
from __future__ import annotations

import math
from typing import Optional, Sequence

import torch
from torch import nn

from .. import _build
from ..ops import functional as F
from ..utils.hooks import unobserved


def _glorot_aug(n_out: int, n_in: int) -> torch.Tensor:
    """[n_out, pad8(n_in + 1)]: glorot-uniform weights, zero bias column, zero padding."""
    w = torch.zeros(n_out, F.pad8(n_in + 1))
    limit = math.sqrt(6.0 / (n_in + n_out))
    w[:, :n_in].uniform_(-limit, limit)
    return w


class MLP(nn.Module):
    """``in_dim -> hidden_units[0] -> ...`` with ReLU after every layer (optionally not the last).
    Input and output are padded bf16 operands (see :func:`tensornet_b200.ops.functional.concat_cast`)."""

    def __init__(self, in_dim: int, hidden_units: Sequence[int], relu_last: bool = True):
        super().__init__()
        self.in_dim = int(in_dim)
        self.hidden_units = [int(h) for h in hidden_units]
        self.relu_last = relu_last
        dims = [self.in_dim] + self.hidden_units
        self.weights = nn.ParameterList([nn.Parameter(_glorot_aug(dims[i + 1], dims[i])) for i in range(len(self.hidden_units))])
        # set by Model.compile on multi-GPU runs when this tower is the first reader of the dense weights in a step:
        # its first GEMM then waits for the optimizer's all-gather instead of the optimizer kernel waiting for everyone
        self.weight_gate = None

    @property
    def out_dim(self) -> int:
        return self.hidden_units[-1]

    def forward(self, x: torch.Tensor, grad_premasked: bool = False, late: Optional[F.LateGrads] = None) -> torch.Tensor:
        return F.mlp(x, list(self.weights), self.in_dim, self.relu_last, grad_premasked, gate=self.weight_gate, late=late)

    def weight(self, i: int) -> torch.Tensor:
        dims = [self.in_dim] + self.hidden_units
        return self.weights[i][:, : dims[i]]

    def bias(self, i: int) -> torch.Tensor:
        dims = [self.in_dim] + self.hidden_units
        return self.weights[i][:, dims[i]]


class DenseHead(nn.Module):
    """``Dense(1)`` on a padded bf16 operand: returns fp32 logits ``[B, 1]``."""

    _scratch = None          # of the head kernels; no part of a saved or copied layer

    def __init__(self, in_dim: int):
        super().__init__()
        self.in_dim = int(in_dim)
        w = torch.zeros(in_dim + 1)
        limit = math.sqrt(6.0 / (in_dim + 1))
        w[:in_dim].uniform_(-limit, limit)
        self.weight = nn.Parameter(w)

    def __getstate__(self):
        return {k: v for k, v in self.__dict__.items() if k != "_scratch"}

    def forward(self, z: torch.Tensor) -> torch.Tensor:
        return F.head(z, self.weight)

    # ---- straight from the pieces of the operand, without assembling it (GPU) -------------------------------------
    def fits(self, widths: Sequence[int], rows: int) -> bool:
        """Whether the head kernels take pieces of these widths."""
        w = self.weight
        return (type(self) is DenseHead and w.is_cuda and w.dtype == torch.float32 and w.is_contiguous() and sum(widths) == w.numel() - 1
                and 0 < len(widths) <= 4 and min(widths) > 0 and rows > 0 and F.head_span(widths) <= _build.cuda_ext().HEAD_MAX_SPAN)

    def on_pieces(self, pieces, widths: Sequence[Optional[int]]) -> torch.Tensor:
        """The logits of ``[piece[:, :width] ...]``; scoring does without the operand where nobody looks at it."""
        widths = [int(p.shape[1]) if k is None else int(k) for p, k in zip(pieces, widths)]
        if not torch.is_grad_enabled() and pieces[0].is_cuda and unobserved(self) and self.fits(widths, pieces[0].shape[0]):
            return F.head_score([_head_piece(p, k) for p, k in zip(pieces, widths)], widths, self.weight)
        return self(F.concat_cast(pieces, ones=True, widths=widths))

    def loss(self, pieces, widths: Sequence[int], label: torch.Tensor, sums: torch.Tensor, relu_first: bool) -> torch.Tensor:
        """Mean sigmoid cross-entropy of the logits, see :func:`tensornet_b200.ops.functional.head_loss`; for pieces that fit."""
        key = (F.head_span(widths), self.weight.device)
        if self._scratch is None or self._scratch[0] != key:      # one per layer: two models may train side by side
            self._scratch = (key, F.head_scratch(widths, self.weight.device))
        s = self._scratch[1]
        label = label.to(self.weight.device, non_blocking=True).contiguous().view(-1).float()
        return F.head_loss([_head_piece(p, k) for p, k in zip(pieces, widths)], widths, self.weight, label, sums, s, relu_first)


def _head_piece(p: torch.Tensor, width: int) -> torch.Tensor:
    """``p`` in a form that the head kernels read: padded bf16 rows of whole 16-byte pieces, or fp32 of exactly its width."""
    p = p if p.dim() == 2 else p.reshape(p.shape[0], -1)
    if p.dtype == torch.bfloat16 and p.shape[1] % 8 == 0 and p.is_contiguous() and p.data_ptr() % 16 == 0:
        return p
    return (p if p.shape[1] == width else p[:, :width]).float().contiguous()


def tower_loss(head: DenseHead, mlp: MLP, widths: Sequence[int], pieces, labels: torch.Tensor, sums: torch.Tensor,
               late: Optional[F.LateGrads] = None) -> torch.Tensor:
    """A training step's loss for a head over ``[mlp output | ...]``, with the head's backward pass in the same kernel where
    that takes it.  ``pieces(**kw)`` runs the layers before it and returns the pieces; ``kw`` are for ``mlp``.
    ``late``: of the model whose own step this is."""
    B = int(labels.numel())
    masked = type(mlp) is MLP and mlp.relu_last and unobserved(mlp, backward=True)      # the kernel masks the gradient of the last ReLU
    if head.weight.requires_grad and head.fits(widths, B):
        got = pieces(grad_premasked=True, late=late) if masked else pieces()
        rows = int(got[0].shape[0])      # (labels beyond the examples are not looked at, here as in the layers one by one)
        return head.loss(got, widths, labels if B <= rows else labels.reshape(-1)[:rows], sums, masked)
    return F.bce_with_logits(head(F.concat_cast(pieces(), ones=True, widths=widths)), labels, sums)[0]


class FMLayer(nn.Module):
    """Second-order factorisation-machine term without linear part and bias.
    Input ``[B, fields, dim]`` (or ``[B, fields*dim]`` with ``fields`` given), output ``[B, 1]``."""

    def __init__(self, fields: int = 0, dim: int = 0):
        super().__init__()
        self.fields, self.dim = fields, dim

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if x.dim() == 3:
            return F.fm(x.reshape(x.shape[0], -1), x.shape[1], x.shape[2])
        if x.dim() != 2 or not self.fields:
            raise ValueError("Unexpected inputs dimensions %d, expect to be 3 dimensions" % x.dim())
        return F.fm(x, self.fields, self.dim)


class DeepCrossLayer(nn.Module):
    """DCN-v1 cross network: ``x_{l+1} = x_0 * (x_l . w_l) + b_l + x_l`` (rank-1 cross)."""

    def __init__(self, input_dim: int, num_layer: int = 3):
        super().__init__()
        self.num_layer = num_layer
        limit = math.sqrt(6.0 / (input_dim + 1))
        self.W = nn.ParameterList([nn.Parameter(torch.empty(input_dim, 1).uniform_(-limit, limit)) for _ in range(num_layer)])
        self.bias = nn.ParameterList([nn.Parameter(torch.zeros(input_dim)) for _ in range(num_layer)])

    def forward(self, inputs: torch.Tensor) -> torch.Tensor:
        return F.cross_v1_net(inputs, list(self.W), list(self.bias))
