"""Wide & Deep (examples/models/wide_deep.py in the reference): dim-1 "wide" embeddings concatenated
with a ReLU MLP over the deep embeddings (plus optional dense features), normalised by a
synchronised TNBatchNormalization, then ``Dense(1)``."""
from __future__ import annotations

from typing import Optional, Sequence

import torch
from torch import nn

from .. import core, feature_column as fc
from ..layers import DenseHead, EmbeddingFeatures, MLP, TNBatchNormalization
from ..layers.embedding_features import pulled_together
from ..model import Model
from ..ops import functional as F
from ..utils.hooks import own_step, unobserved


class WideDeepSubModel(nn.Module):
    def __init__(self, n_linear: int, deep_in: int, dense_dim: int, hidden_units: Sequence[int], use_bn: bool = True):
        super().__init__()
        self.n_linear, self.deep_in, self.dense_dim = n_linear, deep_in, dense_dim
        self.mlp = MLP(deep_in + dense_dim, hidden_units)
        width = self.mlp.out_dim + n_linear
        self.bn = TNBatchNormalization(width, synchronized=True, sync_freq=4, max_count=1000000, name="both_bn") if use_bn else None
        self.head = DenseHead(width)

    def _joins(self, x0, linear_emb) -> bool:
        """Whether the tower's output and the batch norm go through the joint kernels: the layers are the package's own and
        nobody looks at what passes between them."""
        bn, mlp = self.bn, self.mlp
        return (type(bn) is TNBatchNormalization and type(mlp) is MLP and bn.bn_table_handle is not None and bn._on_device and mlp.relu_last
                and x0.is_cuda and x0.shape[0] > 0 and linear_emb.dim() == 2 and linear_emb.dtype == torch.float32 and linear_emb.stride(1) == 1
                and unobserved(bn, mlp, backward=True))

    def _operand(self, deep_emb, dense):
        return F.concat_cast([deep_emb] + ([dense.float()] if self.dense_dim else []), ones=True)

    def _head_operand(self, linear_emb, x0, fused: bool, own_step: bool = False, late=None):
        """Padded bf16 operand of the head; ``x0``: of the tower.  ``own_step``: for the backward pass of a model's own step, which
        may see to ``late`` weight gradients."""
        if fused and self._joins(x0, linear_emb):
            # normalisation straight from the tower's output to the head's operand; its gradient comes back masked
            h = self.mlp(x0, grad_premasked=True, late=late)
            return self.bn.join_operand(h, self.mlp.out_dim, linear_emb, masked=True, into_grads=own_step)
        h = self.mlp(x0)
        if self.bn is None:
            return F.concat_cast([h, linear_emb], ones=True, widths=[self.mlp.out_dim, None])
        both = torch.cat([h[:, : self.mlp.out_dim].float(), linear_emb], dim=1)
        return F.concat_cast([self.bn(both)], ones=True)

    def forward(self, linear_emb, deep_emb, dense=None, fused: bool = True):
        """``fused``: the joint kernels may be used (a model's ``use_fused``)."""
        return self.head(self._head_operand(linear_emb, self._operand(deep_emb, dense), fused))

    def train_loss(self, linear_emb, x0, labels, sums, late=None):
        """Loss of a step's logits with the head's backward pass in the same kernel."""
        z = self._head_operand(linear_emb, x0, True, own_step=True, late=late)
        if self.head.weight.requires_grad and labels.numel() == z.shape[0] and self.head.fits([self.head.in_dim], z.shape[0]):
            return self.head.loss([z], [self.head.in_dim], labels, sums, relu_first=False)
        return F.bce_with_logits(self.head(z), labels, sums)[0]


class WideDeep(Model):
    def __init__(self, linear_features: Sequence[str], dnn_features: Sequence[str], dnn_hidden_units: Sequence[int] = (128, 128),
                 embedding_dim: int = 8, dense_dim: int = 0, dense_key: str = "dense", sparse_opt=None, bucket_size: int = 1024,
                 target_columns: Optional[Sequence[str]] = None, combiner: str = "mean", use_bn: bool = True,
                 table_rows: Optional[int] = None):
        super().__init__(name="full_model")
        sparse_opt = sparse_opt or core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.1)
        cols = {s: fc.category_column(key=s, bucket_size=bucket_size) for s in dict.fromkeys(list(linear_features) + list(dnn_features))}
        self.dense_key, self.dense_dim = dense_key, dense_dim
        self.linear_emb = EmbeddingFeatures([fc.embedding_column(cols[s], 1, combiner) for s in linear_features], sparse_opt,
                                            name="linear_input", is_concat=True, target_columns=target_columns, rows=table_rows)
        self.deep_emb = EmbeddingFeatures([fc.embedding_column(cols[s], embedding_dim, combiner) for s in dnn_features], sparse_opt,
                                          name="deep_input", is_concat=True, target_columns=target_columns, rows=table_rows)
        self.sub_model = WideDeepSubModel(len(linear_features) * self.linear_emb.out_dim, len(dnn_features) * self.deep_emb.out_dim,
                                          dense_dim, dnn_hidden_units, use_bn)

    def _inputs(self, features):
        with pulled_together([self.linear_emb, self.deep_emb], features):
            lin = self.linear_emb(features)
            deep = self.deep_emb(features)
        return lin, deep, features[self.dense_key].to(deep.device, non_blocking=True) if self.dense_dim else None

    def _operands(self, features):
        """``(linear embeddings, operand of the tower)``."""
        dense = features[self.dense_key] if self.dense_dim else None
        if not self.deep_emb.gives_operand() or (dense is not None and (dense.requires_grad or dense.dim() != 2)):
            lin, deep, dense = self._inputs(features)
            return lin, self.sub_model._operand(deep, dense)
        with pulled_together([self.linear_emb, self.deep_emb], features):
            lin = self.linear_emb(features)
            return lin, self.deep_emb.operand(features, self.deep_emb.training, dense)[0]

    def fused_train_loss(self, features, labels, sums):
        """Training loss with the tower's operand straight from the rows, and the head, its loss and its backward pass in one
        kernel; None where somebody looks at what passes in between."""
        if not own_step(self, WideDeep, self.sub_model, WideDeepSubModel):
            return None
        return self.sub_model.train_loss(*self._operands(features), labels, sums, self._late_grads)

    def forward(self, features):
        sub = self.sub_model
        if not torch.is_grad_enabled() and self.use_fused and own_step(self, WideDeep, sub, WideDeepSubModel):
            return sub.head(sub._head_operand(*self._operands(features), True))
        lin, deep, dense = self._inputs(features)
        if not self.use_fused and type(sub) is WideDeepSubModel and "forward" not in sub.__dict__:
            return sub(lin, deep, dense, fused=False)
        return sub(lin, deep, dense)
