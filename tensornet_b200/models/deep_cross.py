"""Deep & Cross networks.

``DeepCross`` is the reference's example (examples/models/deep_cross.py): DCN-v1 rank-1 cross layers
next to a ReLU MLP.  ``DCNv2`` is the full-matrix variant ``x_{l+1} = x0 * (W_l x_l + b_l) + x_l``
whose cross layers are tcgen05 GEMMs with the Hadamard-residual fused into the epilogue.
"""
from __future__ import annotations

import math
from typing import Sequence

import torch
from torch import nn

from .. import core, feature_column as fc
from ..layers import DeepCrossLayer, DenseHead, EmbeddingFeatures, MLP
from ..layers.dense import tower_loss
from ..model import Model
from ..ops import functional as F
from ..utils.hooks import own_step, unobserved


class DeepCrossSubModel(nn.Module):
    def __init__(self, in_dim: int, hidden_units: Sequence[int], num_cross: int = 3):
        super().__init__()
        self.in_dim = in_dim
        self.cross = DeepCrossLayer(in_dim, num_cross)
        self.mlp = MLP(in_dim, hidden_units)
        self.head = DenseHead(self.mlp.out_dim + in_dim)

    def _head_pieces(self, x: torch.Tensor, x0=None, own: bool = False, **kw):
        """``x0``: ``x`` as the tower's operand, where that is there already.  ``own``: for the backward pass of a model's own step."""
        net = self.cross
        if own and type(net) is DeepCrossLayer and unobserved(net, backward=True):
            cross = F.cross_v1_net(x, list(net.W), list(net.bias), into_grads=True)
        else:
            cross = net(x)
        return [self.mlp(F.concat_cast([x], ones=True) if x0 is None else x0, **kw), cross]

    def forward(self, x: torch.Tensor, x0=None):
        return self.head.on_pieces(self._head_pieces(x, x0), [self.mlp.out_dim, None])

    def train_loss(self, x, x0, labels, sums, late=None):
        return tower_loss(self.head, self.mlp, [self.mlp.out_dim, x.shape[1]], lambda **kw: self._head_pieces(x, x0, True, **kw), labels, sums,
                          late)


class CrossV2(nn.Module):
    """Stack of DCN-v2 cross layers on a padded bf16 operand ``[B, pad8(D + 1)]``."""

    def __init__(self, dim: int, num_layer: int = 3):
        super().__init__()
        self.dim, self.num_layer = dim, num_layer
        limit = math.sqrt(6.0 / (2 * dim))
        self.weights = nn.ParameterList()
        for _ in range(num_layer):
            w = torch.zeros(dim, F.pad8(dim + 1))
            w[:, :dim].uniform_(-limit, limit)
            self.weights.append(nn.Parameter(w))

    def forward(self, x0: torch.Tensor) -> torch.Tensor:
        return F.cross_v2(x0, list(self.weights), self.dim)


class DCNv2SubModel(nn.Module):
    def __init__(self, in_dim: int, hidden_units: Sequence[int], num_cross: int = 3):
        super().__init__()
        self.in_dim = in_dim
        self.cross = CrossV2(in_dim, num_cross)
        self.mlp = MLP(in_dim, hidden_units)
        self.head = DenseHead(self.mlp.out_dim)

    def _tower(self, x, x0=None, **kw):
        if x0 is None:
            x0 = F.concat_cast(list(x) if isinstance(x, (list, tuple)) else [x], ones=True)
        return self.mlp(self.cross(x0), **kw)          # stacked structure: cross network feeds the deep network

    def forward(self, x, x0=None):
        """``x``: the input matrix, or its column blocks (embeddings, dense features): the blocks go straight into
        the padded bf16 operand, without an fp32 concatenation in between (a 210 MB copy each way at width 6413).  ``x0``: that
        operand, where it is there already."""
        return self.head(self._tower(x, x0))

    def train_loss(self, x, x0, labels, sums, late=None):
        return tower_loss(self.head, self.mlp, [self.mlp.out_dim], lambda **kw: [self._tower(x, x0, **kw)], labels, sums, late)


class _CrossModel(Model):
    def __init__(self, sub_cls, features: Sequence[str], dnn_hidden_units, embedding_dim, dense_dim, dense_key, sparse_opt,
                 bucket_size, target_columns, combiner, num_cross, table_rows):
        super().__init__(name="full_model")
        sparse_opt = sparse_opt or core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.1)
        cols = [fc.embedding_column(fc.category_column(key=s, bucket_size=bucket_size), embedding_dim, combiner) for s in features]
        self.dense_key, self.dense_dim = dense_key, dense_dim
        self.deep_emb = EmbeddingFeatures(cols, sparse_opt, name="deep_input", is_concat=True, target_columns=target_columns,
                                          rows=table_rows)
        self.sub_model = sub_cls(len(features) * self.deep_emb.out_dim + dense_dim, dnn_hidden_units, num_cross)

    def _inputs(self, features):
        x = self.deep_emb(features)
        if self.dense_dim:
            dense = features[self.dense_key].to(x.device, non_blocking=True).float()
            if x.is_cuda and isinstance(self.sub_model, DCNv2SubModel):
                return [x, dense]
            x = torch.cat([x, dense], dim=1)
        return x

    def _own(self) -> bool:
        return type(self.sub_model) in (DeepCrossSubModel, DCNv2SubModel) and own_step(self, _CrossModel, self.sub_model, type(self.sub_model))

    def _operands(self, features):
        """``(x, x0)``: the input matrix and the same as the tower's operand; for DCN-v2 the operand alone."""
        dense = features[self.dense_key] if self.dense_dim else None
        if not self.deep_emb.gives_operand() or (dense is not None and (dense.requires_grad or dense.dim() != 2)):
            return self._inputs(features), None
        x0, _, _, x = self.deep_emb.operand(features, self.deep_emb.training, dense, pooled=type(self.sub_model) is DeepCrossSubModel)
        return x, x0

    def fused_train_loss(self, features, labels, sums):
        """Training loss with the operand straight from the rows, and the head, its loss and its backward pass in one kernel; None
        where somebody looks at what passes in between."""
        return self.sub_model.train_loss(*self._operands(features), labels, sums, self._late_grads) if self._own() else None

    def forward(self, features):
        if not torch.is_grad_enabled() and self.use_fused and self._own():
            return self.sub_model(*self._operands(features))
        return self.sub_model(self._inputs(features))


class DeepCross(_CrossModel):
    def __init__(self, features, dnn_hidden_units=(128, 128), embedding_dim=8, dense_dim=0, dense_key="dense", sparse_opt=None,
                 bucket_size=1024, target_columns=None, combiner="mean", num_cross=3, table_rows=None):
        super().__init__(DeepCrossSubModel, features, dnn_hidden_units, embedding_dim, dense_dim, dense_key, sparse_opt, bucket_size,
                         target_columns, combiner, num_cross, table_rows)


class DCNv2(_CrossModel):
    def __init__(self, features, dnn_hidden_units=(1024, 512, 256), embedding_dim=64, dense_dim=13, dense_key="dense",
                 sparse_opt=None, bucket_size=1024, target_columns=None, combiner="sum", num_cross=3, table_rows=None):
        super().__init__(DCNv2SubModel, features, dnn_hidden_units, embedding_dim, dense_dim, dense_key, sparse_opt, bucket_size,
                         target_columns, combiner, num_cross, table_rows)
