"""DeepFM (examples/models/deepfm.py in the reference): a linear term over dim-1 embeddings,
a second-order FM term and a ReLU MLP over the concatenated deep embeddings (plus optional
dense features), joined by a final ``Dense(1)``.

As in the reference the model is split into an embedding part (``emb_model``: the two
EmbeddingFeatures layers) and a pure dense ``sub_model`` (what gets exported for serving).
"""
from __future__ import annotations

from typing import Optional, Sequence

import torch
from torch import nn

from .. import core, feature_column as fc
from ..layers import DenseHead, EmbeddingFeatures, MLP
from ..layers.dense import tower_loss
from ..layers.embedding_features import pulled_together
from ..model import Model
from ..ops import functional as F
from ..utils.hooks import own_step, unobserved


class DeepFMSubModel(nn.Module):
    """Dense part: inputs are the pooled embeddings, output is the logit."""

    def __init__(self, n_linear: int, n_fields: int, emb_dim: int, dense_dim: int, hidden_units: Sequence[int]):
        super().__init__()
        self.n_linear, self.n_fields, self.emb_dim, self.dense_dim = n_linear, n_fields, emb_dim, dense_dim
        self.mlp = MLP(n_fields * emb_dim + dense_dim, hidden_units)
        self.head = DenseHead(self.mlp.out_dim + n_linear + 1)

    def _head_pieces(self, linear_emb, deep_emb, dense, **kw):
        fm = F.fm(deep_emb, self.n_fields, self.emb_dim)
        pieces = [deep_emb] + ([dense.float()] if self.dense_dim else [])
        h = self.mlp(F.concat_cast(pieces, ones=True), **kw)
        return [h] + ([linear_emb] if self.n_linear else []) + [fm]

    def _head_widths(self):
        return [self.mlp.out_dim] + ([self.n_linear] if self.n_linear else []) + [1]

    def forward(self, linear_emb: Optional[torch.Tensor], deep_emb: torch.Tensor, dense: Optional[torch.Tensor] = None):
        return self.head.on_pieces(self._head_pieces(linear_emb, deep_emb, dense), self._head_widths())

    def train_loss(self, linear_emb, deep_emb, dense, labels, sums, late=None):
        return tower_loss(self.head, self.mlp, self._head_widths(), lambda **kw: self._head_pieces(linear_emb, deep_emb, dense, **kw),
                          labels, sums, late)


class DeepFM(Model):
    def __init__(self, linear_features: Sequence[str], dnn_features: Sequence[str], dnn_hidden_units: Sequence[int] = (128, 128),
                 embedding_dim: int = 8, dense_dim: int = 0, dense_key: str = "dense", sparse_opt=None, linear_sparse_opt=None,
                 bucket_size: int = 1024, target_columns: Optional[Sequence[str]] = None, combiner: str = "mean",
                 table_rows: Optional[int] = None, share_linear_table: bool = False):
        super().__init__(name="full_model")
        sparse_opt = sparse_opt or core.AdaGrad(learning_rate=0.01, initial_g2sum=0.1, initial_scale=0.1)
        linear_sparse_opt = linear_sparse_opt or sparse_opt
        cols = {s: fc.category_column(key=s, bucket_size=bucket_size) for s in dict.fromkeys(list(linear_features) + list(dnn_features))}
        self.dense_key, self.dense_dim = dense_key, dense_dim
        self.linear_emb = None
        # One table for both parts: a slot's linear weight is stored as an extra column of its embedding row, so
        # the batch is deduplicated, pulled and pushed once.  Exact for element-wise sparse optimizers (Adam, Ftrl);
        # AdaGrad keeps one accumulator per row and therefore needs separate tables.
        self.share_linear_table = bool(share_linear_table and linear_features and list(linear_features) == list(dnn_features)
                                       and sparse_opt.kind != 0 and not target_columns)
        self.emb_dim = embedding_dim
        if self.share_linear_table:
            self.deep_emb = EmbeddingFeatures([fc.embedding_column(cols[s], embedding_dim + 4, combiner) for s in dnn_features],
                                              sparse_opt, name="deep_input", is_concat=True, rows=table_rows)
            self.sub_model = DeepFMSubModel(len(linear_features), len(dnn_features), embedding_dim, dense_dim, dnn_hidden_units)
            return
        if linear_features:
            self.linear_emb = EmbeddingFeatures([fc.embedding_column(cols[s], 1, combiner) for s in linear_features],
                                                linear_sparse_opt, name="linear_input", is_concat=True,
                                                target_columns=target_columns, rows=table_rows)
        self.deep_emb = EmbeddingFeatures([fc.embedding_column(cols[s], embedding_dim, combiner) for s in dnn_features],
                                          sparse_opt, name="deep_input", is_concat=True, target_columns=target_columns,
                                          rows=table_rows)
        n_lin = len(linear_features) * (self.linear_emb.out_dim if self.linear_emb else 0)
        self.sub_model = DeepFMSubModel(n_lin, len(dnn_features), self.deep_emb.out_dim, dense_dim, dnn_hidden_units)

    def first_dense_tower(self):
        """The embedding pooling, FM term and input assembly read no dense parameter: the MLP is the first reader."""
        return self.sub_model.mlp

    def fused_train_loss(self, features, labels, sums):
        """Training loss through the fused kernels: gather + FM + operand build in one kernel where the inputs qualify (no
        ragged slots, no CVM columns); head, loss and head backward in one kernel.  None: the caller uses the generic path."""
        sub = self.sub_model
        if not own_step(self, DeepFM, sub, DeepFMSubModel):
            return None
        got = self._fused_inputs(features, True)
        if got is None:
            return sub.train_loss(*self._inputs(features), labels, sums, self._late_grads)
        x0, rest = got
        return tower_loss(sub.head, sub.mlp, sub._head_widths(), lambda **kw: [sub.mlp(x0, **kw), *rest], labels, sums,
                          self._late_grads)

    def _fused_inputs(self, features, training):
        """``(x0, [linear weights, FM term])``: the first layer's operand and what goes to the head beside the tower's output,
        through the fused input kernel; None when the layers are not the package's own or somebody looks on."""
        emb = [self.deep_emb] + ([self.linear_emb] if self.linear_emb is not None else [])
        dense = features[self.dense_key] if self.dense_dim else None
        if (not isinstance(features, dict) or not all(type(e) is EmbeddingFeatures and unobserved(e, backward=True) for e in emb)
                or not self.deep_emb.gives_operand(self.emb_dim if self.share_linear_table else None)
                or (dense is not None and (dense.requires_grad or dense.dim() != 2))):
            return None
        if self.share_linear_table:
            x0, fm, lin, _ = self.deep_emb.operand(features, training, dense, True, self.emb_dim, self.emb_dim)
            return x0, [lin, fm]
        if self.linear_emb is None:
            x0, fm, _, _ = self.deep_emb.operand(features, training, dense, True)
            return x0, [fm]
        with pulled_together([self.linear_emb, self.deep_emb], features, training):
            lin = self.linear_emb(features, training=training)
            x0, fm, _, _ = self.deep_emb.operand(features, training, dense, True)
        return x0, [lin, fm]

    def _scores(self, features, ragged: bool = False):
        """The logits by way of the fused input kernel (scoring: no gradients, layers in inference mode), or None when the
        batch does not qualify or somebody looks at what passes between the layers.  ``ragged``: bags of ids qualify too."""
        own = [self.deep_emb, self.sub_model] + ([self.linear_emb] if self.linear_emb is not None else [])
        if (torch.is_grad_enabled() or not self.use_fused or type(self.sub_model) is not DeepFMSubModel or not isinstance(features, dict)
                or any(m.training for m in own) or not unobserved(*own)):
            return None
        if not ragged and self.deep_emb.stash_pull_args(features, False)[1] is not None:
            self.deep_emb._args_cache = None
            return None
        got = self._fused_inputs(features, False)
        if got is None:
            return None
        x0, rest = got
        return self.sub_model.head.on_pieces([self.sub_model.mlp(x0), *rest], self.sub_model._head_widths())

    def _inputs(self, features):
        """The dense part's inputs through the layers one by one."""
        if self.share_linear_table:
            both = self.deep_emb(features)
            both = both.view(both.shape[0], -1, self.emb_dim + 4)
            lin = both[:, :, self.emb_dim].contiguous()
            deep = both[:, :, : self.emb_dim].reshape(both.shape[0], -1)
            dense = features[self.dense_key].to(deep.device, non_blocking=True) if self.dense_dim else None
            return lin, deep, dense
        if self.linear_emb is not None:
            with pulled_together([self.linear_emb, self.deep_emb], features):
                lin = self.linear_emb(features)
                deep = self.deep_emb(features)
        else:
            lin, deep = None, self.deep_emb(features)
        dense = None
        if self.dense_dim:
            dense = features[self.dense_key].to(deep.device, non_blocking=True)
        return lin, deep, dense

    def forward(self, features):
        logits = self._scores(features, ragged=True)
        if logits is not None:
            return logits
        return self.sub_model(*self._inputs(features))
