"""Input containers for categorical features.

A model input is a dict ``{slot name: feature}`` where a feature is
* an int64 tensor ``[B]`` / ``[B, 1]``   one sign per example,
* an int64 tensor ``[B, L]``            exactly L signs per example,
* a :class:`Ragged` ``(values, offsets)``  a variable number of signs per example
  (the SparseTensor inputs of the reference, tensornet/layers/embedding_features.py:252-284).

:class:`PackedFeatures` carries several slots in one buffer so a batch costs one host->device
copy instead of one per slot; layers pick the slots they need out of it.
"""
from __future__ import annotations

from typing import Dict, List, NamedTuple, Optional, Sequence, Tuple

import torch


class Ragged(NamedTuple):
    values: torch.Tensor   # int64 [nnz]
    offsets: torch.Tensor  # int32/int64 [B + 1]


class PackedFeatures:
    """Slots ``keys`` stored together.  Single-hot: ``ids [S, B]``.  Ragged: ``values [nnz]`` with
    ``offsets [S*B + 1]`` where bag ``s*B + b`` belongs to slot s, example b."""

    def __init__(self, keys: Sequence[str], ids: Optional[torch.Tensor] = None, values: Optional[torch.Tensor] = None,
                 offsets: Optional[torch.Tensor] = None, batch_size: Optional[int] = None):
        self.keys = [str(k) for k in keys]
        self.ids, self.values, self.offsets = ids, values, offsets
        if ids is not None:
            assert ids.dim() == 2 and ids.shape[0] == len(self.keys)
            self.batch_size = int(ids.shape[1])
        else:
            assert values is not None and offsets is not None and batch_size is not None
            self.batch_size = int(batch_size)

    def to(self, device, non_blocking: bool = True) -> "PackedFeatures":
        mv = lambda t: None if t is None else t.to(device, non_blocking=non_blocking)
        return PackedFeatures(self.keys, mv(self.ids), mv(self.values), mv(self.offsets), self.batch_size)

    def pin_memory(self) -> "PackedFeatures":
        pm = lambda t: None if t is None else t.pin_memory()
        return PackedFeatures(self.keys, pm(self.ids), pm(self.values), pm(self.offsets), self.batch_size)


PACKED_KEY = "__packed__"


class NeedsExactLengths(RuntimeError):
    """Code other than the embedding layers looked into a padded feature of a captured step."""


class PaddedRagged(Ragged):
    """The stand-in for a :class:`Ragged` column inside a captured step: ``values`` has room for more ids than the
    batch holds, the last offset says how many are there.  Only :func:`gather_columns` reads it.  It is a ``Ragged`` to
    code that looks at the type, and tells whatever asks for ``values`` / ``offsets`` that exact lengths are not to be
    had (the model then runs such batches uncaptured)."""

    def __new__(cls, values: torch.Tensor, offsets: torch.Tensor):
        self = super().__new__(cls, None, None)
        self._values, self._offsets = values, offsets
        return self

    def _refuse(self, *_, **__):
        raise NeedsExactLengths("padded feature")

    values = offsets = property(_refuse)
    __getitem__ = __iter__ = __len__ = __eq__ = __ne__ = __hash__ = __contains__ = _refuse
    _replace = _asdict = index = count = _refuse


class PaddedPacked(PackedFeatures):
    """:class:`PackedFeatures` of the ragged form with room for more ids than the batch holds; see :class:`PaddedRagged`."""

    def __init__(self, keys: Sequence[str], values: torch.Tensor, offsets: torch.Tensor, batch_size: int):
        self.keys, self.ids, self.batch_size = [str(k) for k in keys], None, int(batch_size)
        self._values, self._offsets = values, offsets

    def _refuse(self, *_):
        raise NeedsExactLengths("padded features")

    values = offsets = property(_refuse)
    to = pin_memory = _refuse


def padded_columns(features: Dict, keys: List[str]) -> bool:
    """Do the slots ``keys`` come with room for more ids than the batch holds?  The last offset is then the count."""
    packed = features.get(PACKED_KEY)
    if packed is not None and packed.keys == keys:
        return isinstance(packed, PaddedPacked)
    return any(isinstance(features.get(k), PaddedRagged) for k in keys)


def batch_size_of(feature) -> int:
    if isinstance(feature, PaddedRagged):
        return int(feature._offsets.numel()) - 1
    if isinstance(feature, Ragged) or (isinstance(feature, (tuple, list)) and len(feature) == 2):
        return int(feature[1].numel()) - 1
    return int(feature.shape[0])


def adjacent_columns(cols) -> Optional[torch.Tensor]:
    """Columns of int64 ids, one each per example, that lie one behind the other in one piece of memory, as a view of it; else
    None.  (A captured step's static columns do: they need no concatenation.)"""
    first = cols[0]
    if not all(torch.is_tensor(c) and c.dtype == torch.int64 and c.is_contiguous() and c.dim() in (1, 2) and c.device == first.device for c in cols):
        return None
    n, at, base = first.numel(), first.data_ptr(), first.untyped_storage().data_ptr()
    for k, c in enumerate(cols):
        if c.numel() != n or (c.dim() == 2 and c.shape[1] != 1) or c.data_ptr() != at + 8 * n * k or c.untyped_storage().data_ptr() != base:
            return None
    return first.as_strided((n * len(cols),), (1,), first.storage_offset())


def gather_columns(features: Dict, keys: List[str], device) -> Tuple[torch.Tensor, Optional[torch.Tensor], int]:
    """Collect the slots ``keys`` as ``(ids, offsets, B)`` in the column-after-column layout the
    pull kernel expects; ``offsets`` is None when every bag holds exactly one id."""
    packed = features.get(PACKED_KEY) if isinstance(features, dict) else None
    if packed is not None and packed.keys == keys:
        if packed.ids is not None:
            return packed.ids.to(device, non_blocking=True).reshape(-1), None, packed.batch_size
        if isinstance(packed, PaddedPacked):
            return packed._values, packed._offsets.int(), packed.batch_size
        return (packed.values.to(device, non_blocking=True), packed.offsets.to(device, non_blocking=True).int(),
                packed.batch_size)
    if packed is not None and packed.ids is not None and all(k in packed.keys for k in keys):
        idx = [packed.keys.index(k) for k in keys]
        ids = packed.ids.to(device, non_blocking=True)
        return ids[idx].reshape(-1).contiguous(), None, packed.batch_size
    cols = [features[k] for k in keys]
    single = all(torch.is_tensor(c) and (c.dim() == 1 or (c.dim() == 2 and c.shape[1] == 1)) for c in cols)
    B = batch_size_of(cols[0])
    if single:
        if cols[0].is_cuda and B > 0:
            ids = adjacent_columns(cols)
            if ids is not None:
                return ids, None, B
        ids = torch.stack([c.reshape(-1).to(device, non_blocking=True).long() for c in cols]).reshape(-1)
        return ids, None, B
    if any(isinstance(c, PaddedRagged) for c in cols):
        return _gather_padded(cols, B, device)
    vals, offs, base = [], [], 0
    for c in cols:
        if torch.is_tensor(c):
            c = c.to(device, non_blocking=True).long()
            c2 = c.reshape(B, -1)
            L = c2.shape[1]
            v = c2.reshape(-1)
            o = torch.arange(0, B * L + 1, L, device=device, dtype=torch.int64)
        else:
            v = c[0].to(device, non_blocking=True).long().reshape(-1)
            o = c[1].to(device, non_blocking=True).long().reshape(-1)
        vals.append(v)
        offs.append(o[:-1] + base)
        base += int(v.numel())
    offs.append(torch.tensor([base], device=device, dtype=torch.int64))
    return torch.cat(vals), torch.cat(offs).int(), B


def _gather_padded(cols, B: int, device) -> Tuple[torch.Tensor, torch.Tensor, int]:
    """Columns of a captured step -> packed layout.  Where a column starts depends on how many ids the columns before
    it hold in THIS batch, so the packing is a kernel that reads the counts on the device."""
    from .. import _build

    vals, offs, lens, room = [], [], [], 0
    for c in cols:
        if isinstance(c, PaddedRagged):
            v, o, n = c._values, c._offsets, 0
        elif torch.is_tensor(c):
            v, o = c.to(device, non_blocking=True).contiguous(), None
            n = int(v.numel()) // B
        else:
            v, o, n = c[0].to(device, non_blocking=True).contiguous(), c[1].to(device, non_blocking=True).contiguous(), 0
        if v.dtype not in (torch.int32, torch.int64):
            v = v.long()
        if o is not None and o.dtype not in (torch.int32, torch.int64):
            o = o.long()
        vals.append(v.reshape(-1))
        offs.append(o)
        lens.append(n)
        room += int(v.numel())
    values = torch.empty(room, dtype=torch.int64, device=device)
    offsets = torch.empty(len(cols) * B + 1, dtype=torch.int32, device=device)
    _build.cuda_ext().pack_columns(vals, offs, lens, B, values, offsets)
    return values, offsets, B
