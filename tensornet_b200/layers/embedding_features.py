"""``tn.layers.EmbeddingFeatures``: the first layer of every model.

Creates one sparse table for the layer (or shares one through ``embedding_share``), and on
every call dedups the batch's signs, pulls their rows from the owning shards into the small
per-batch matrix and pools them per example - the reference's EmbeddingFeatures /
StateManagerImpl (tensornet/layers/embedding_features.py:36-177,180-406).  ``backwards()``
pushes the gradient of that per-batch matrix to the owners, where the sparse optimizer runs.

With ``target_columns`` the table counts show / click per sign and every embedding gets two
extra, gradient-free columns ``show`` and ``ln(click+1) - ln(show+1)`` (the CVM plug-in,
embedding_features.py:288-295, core/ps/optimizer/ada_grad_kernel.cc:121-128).
"""
from __future__ import annotations

import contextlib
from typing import Dict, Optional, Sequence

import torch
from torch import nn

from .. import _build, core
from ..data.features import PACKED_KEY, adjacent_columns, gather_columns, padded_columns
from ..feature_column import EmbeddingColumn
from ..ops import functional as F
from ..ops.embedding import COMBINERS, expand_bag_labels, pull_pool
from ..utils.hooks import unobserved


class EmbeddingFeatures(nn.Module):
    def __init__(self, feature_columns: Sequence[EmbeddingColumn], sparse_opt, trainable: bool = True,
                 name: Optional[str] = None, is_concat: bool = False, target_columns: Optional[Sequence[str]] = None,
                 embedding_share: Optional[str] = None, rows: Optional[int] = None):
        super().__init__()
        assert len(feature_columns) != 0, "feature_columns must not empty"
        dim = feature_columns[0].dimension
        combiner = feature_columns[0].combiner
        for c in feature_columns:
            if not isinstance(c, EmbeddingColumn):
                raise ValueError(f"Items of feature_columns must be a {EmbeddingColumn}. Given: {c}")
            assert c.dimension == dim, "currently we only support feature_columns with same dimension in EmbeddingFeatures"
            assert c.combiner == combiner, "all columns of one EmbeddingFeatures layer must use the same combiner"
        if target_columns and len(target_columns) > 1:
            raise ValueError(f"For now cvm plugin only support one column, Given: {target_columns}")
        self.layer_name = name or ""
        self.trainable = trainable
        self.is_concat = is_concat
        self._sparse_opt = sparse_opt
        self._feature_columns = list(feature_columns)
        self._target_columns = list(target_columns) if target_columns else None
        self._keys = [c.categorical_column.name for c in feature_columns]
        self.dim = dim
        self.combiner = combiner
        self.use_cvm = bool(target_columns)
        self.embedding_share = embedding_share
        self.sparse_table_handle = core.create_sparse_table(sparse_opt, self.layer_name, dim, self.use_cvm,
                                                            embedding_share or "", rows=rows)
        self.table = core.sparse_table(self.sparse_table_handle)
        max_unique = sum(c.categorical_column.bucket_size for c in feature_columns)
        self.link = self.table.link(max_unique)
        self.out_dim = dim + (2 if self.use_cvm else 0)
        self._anchor = torch.zeros(1, requires_grad=True, device=core.runtime().device)
        self._pending_push = False
        self._args_cache = None

    # --------------------------------------------------------------------------------
    @property
    def feature_columns(self):
        return self._feature_columns

    def filter_not_used_features(self, features: Dict) -> Dict:
        """The entries of ``features`` that this layer's columns read (embedding_features.py:314-319)."""
        return {k: features[k] for k in self._keys}

    def get_sparse_pulling_feature(self, features: Dict):
        """``(pulled, targets)``: the id features of ``features`` split into those whose signs are looked up and the
        target columns that only feed the show / click counters (embedding_features.py:321-334)."""
        pulled, targets = {}, {}
        for k, v in features.items():
            if self._target_columns and k in self._target_columns:
                targets[k] = v
            elif k in self._keys:
                pulled[k] = v
        return pulled, targets

    def get_config(self) -> Dict:
        """Constructor arguments as plain data (embedding_features.py:369-379); ``from_config`` builds the layer again."""
        return {"name": self.layer_name, "trainable": self.trainable, "is_concat": self.is_concat,
                "target_columns": self._target_columns, "embedding_share": self.embedding_share,
                "feature_columns": [c.get_config() for c in self._feature_columns], "sparse_opt": self._sparse_opt.get_config()}

    @classmethod
    def from_config(cls, config: Dict, sparse_opt=None):
        """``sparse_opt`` overrides the optimizer described in ``config`` (a learning-rate schedule is not part of a
        configuration)."""
        from ..core.optimizers import optimizer_from_config
        from ..feature_column import EmbeddingColumn
        cfg = dict(config)
        cols = [EmbeddingColumn.from_config(c) for c in cfg.pop("feature_columns")]
        opt = sparse_opt or optimizer_from_config(cfg.pop("sparse_opt"))
        cfg.pop("sparse_opt", None)
        return cls(cols, opt, **cfg)

    def _pull_args(self, features: Dict, training: bool):
        """What this layer's pull needs from a batch: ``(ids, offsets, B, labels, label_mod, count)``.  A model that
        runs several layers' pulls with shared round trips asks for them first; the ``forward`` of the same batch
        then finds them here (once) instead of gathering the columns again."""
        c, self._args_cache = self._args_cache, None
        if c is not None and c[0] is features and c[1] == training:
            return c[2]
        dev = core.runtime().device
        ids, offsets, B = gather_columns(features, self._keys, dev)
        S = len(self._keys)
        labels, label_mod = None, 0
        if self._target_columns:
            y = features[self._target_columns[0]].to(dev, non_blocking=True).reshape(-1).float().contiguous()
            if offsets is None:
                labels, label_mod = y, B
            elif ids.is_cuda:
                labels = expand_bag_labels(y, offsets, S, int(ids.numel()))
            else:
                lens = (offsets[1:] - offsets[:-1]).long()
                labels = torch.repeat_interleave(y.repeat(S), lens, output_size=int(ids.numel()))
        return ids, offsets, B, labels, label_mod, training and self.trainable

    def stash_pull_args(self, features: Dict, training: bool):
        args = self._pull_args(features, training)
        self._args_cache = (features, training, args)
        return args

    def _n_dev(self, features, offsets):
        """A captured step's buffers have room to spare: the last offset is the number of ids of this batch."""
        return offsets[-1:] if offsets is not None and padded_columns(features, self._keys) else None

    def forward(self, features: Dict, training: Optional[bool] = None):
        if not isinstance(features, dict):
            raise ValueError("We expected a dictionary here. Instead we got: ", features)
        training = self.training if training is None else bool(training)
        self.table.set_training(training)
        ids, offsets, B, labels, label_mod, count = self._pull_args(features, training)
        S = len(self._keys)
        n_dev = self._n_dev(features, offsets)
        out = pull_pool(self._anchor, self.link, ids, offsets, B, S, self.combiner, labels, label_mod, count, n_dev)
        self._pending_push = count
        if self.is_concat:
            return out
        pd = self.out_dim
        return [out[:, s * pd:(s + 1) * pd] for s in range(S)]

    def gives_operand(self, width: Optional[int] = None) -> bool:
        """Whether :meth:`operand` may stand in for a call of this layer: on a GPU, with nobody looking on."""
        return (core.runtime().on_gpu and type(self) is EmbeddingFeatures and self.is_concat
                and (width or self.out_dim) <= _build.cuda_ext().EMBED_INPUT_COLUMNS and unobserved(self, backward=True))

    def operand(self, features: Dict, training: bool, dense: Optional[torch.Tensor] = None, fm: bool = False, width: Optional[int] = None,
                lin_col: int = -1, pooled: bool = False):
        """``(x0, fm, lin, pooled)`` of :func:`tensornet_b200.ops.functional.embed_input` for a batch, in place of pooling its
        slots and assembling the dense part's operand from them.  ``width``: only the first columns of a slot."""
        self.table.set_training(training)
        ids, offsets, B, labels, label_mod, count = self._pull_args(features, training)
        if dense is not None:
            dense = dense.to(ids.device, non_blocking=True).float().contiguous()
        self._pending_push = count
        return F.embed_input(self._anchor, self.link, ids, offsets, B, len(self._keys), width or self.out_dim, COMBINERS[self.combiner],
                             labels, label_mod, count, self._n_dev(features, offsets), dense, fm, lin_col, pooled)

    def ids_pulled_for(self, features: Dict):
        """The id tensor this layer's next training pull will receive for ``features``, when that is known ahead
        without any work: the packed single-hot ids of exactly this layer's slots, or its columns one behind the other, already
        on the device (the tensor the pull gets is then a view of them, same address).  None otherwise, and for layers
        whose table serves several links (their pulls share one step counter)."""
        rt = core.runtime()
        if not (rt.on_gpu and self.trainable and isinstance(features, dict)) or not hasattr(self.link, "prefetch"):
            return None
        if len(getattr(self.table, "links", ())) != 1:
            return None
        packed = features.get(PACKED_KEY)
        if packed is None:
            cols = [features.get(k) for k in self._keys]
            return adjacent_columns(cols) if torch.is_tensor(cols[0]) and cols[0].is_cuda and cols[0].numel() > 0 else None
        if list(packed.keys) != list(self._keys) or packed.ids is None or not packed.ids.is_cuda:
            return None
        return packed.ids.reshape(-1)

    def backwards(self, grads_and_vars=None):
        """Push this step's sparse gradients to the owning shards and apply the sparse optimizer."""
        if self._pending_push:
            self.link.push()
            self._pending_push = False

    # --------------------------------------------------------------------------------
    def save_sparse_table(self, filepath: str, mode: str = "txt"):
        return core.save_sparse_table(self.sparse_table_handle, filepath, mode)

    def load_sparse_table(self, filepath: str, mode: str = "txt"):
        return core.load_sparse_table(self.sparse_table_handle, filepath, mode)

    def show_decay(self, delta_days: int = 0):
        return core.show_decay(self.sparse_table_handle, delta_days)


@contextlib.contextmanager
def pulled_together(layers: Sequence[EmbeddingFeatures], features: Dict, training: Optional[bool] = None):
    """:func:`pull_together` around the forward passes that use it: a pull that none of them took is undone at the end."""
    pulled = pull_together(layers, features, training)
    try:
        yield
    finally:
        if pulled:
            for l in layers:
                l.link.drop_pulled()


def pull_together(layers: Sequence[EmbeddingFeatures], features: Dict, training: Optional[bool] = None) -> bool:
    """Run the pulls of several layers over one batch side by side (one GPU; their ids are all they need).  The
    forward pass of every one of them has to follow; it then finds its pull done.  A training pull counts shows and clicks
    and creates rows, so it is run for ``features`` only where that is what the layers will be given: not when a hook or a
    ``forward`` set on an instance comes in between."""
    rt = core.runtime()
    if (not rt.on_gpu or rt.world > 1 or not isinstance(features, dict) or not all(type(l) is EmbeddingFeatures for l in layers)
            or not unobserved(*layers)):
        return False
    if training is None:
        training = layers[0].training
        if any(l.training != training for l in layers):
            return False
    if len({id(l.table) for l in layers}) < len(layers) or not all(l.link.ctx.in_place() for l in layers):
        return False
    calls, first = [], layers[0]
    for l in layers:
        l.table.set_training(training)
        if l is not first and l._keys == first._keys and l._target_columns == first._target_columns:
            # the same slots: gathered once (columns of a batch are packed by a kernel)
            l._args_cache = (features, training, (*first._args_cache[2][:5], training and l.trainable))
            ids, offsets, _, labels, label_mod, count = l._args_cache[2]
        else:
            ids, offsets, _, labels, label_mod, count = l.stash_pull_args(features, training)
        calls.append((l.link, ids, labels, label_mod, count, l._n_dev(features, offsets)))
    return layers[0].link.pull_many(calls)
