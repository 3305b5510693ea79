"""Recognising the tensors that a kept copy was made from."""
from __future__ import annotations

import torch

from . import _native


class Origin:
    """``Origin(*tensors).still(*others)``: whether ``others`` are those tensors with the same contents, as far as their version
    counters tell.  Assigning ``p.data`` moves no counter, so the storage is compared, and by its identity: an address is
    given out again once its storage is gone, and two assignments can bring a parameter back to where it was.  Only a weak
    reference is held, which keeps the identity from being given out again, not the memory.  A copy or an unpickled one
    matches nothing."""

    __slots__ = ("_stamps",)

    def __init__(self, *tensors: torch.Tensor) -> None:
        self._stamps = _native.bind().stamps(*tensors) if tensors else None

    def still(self, *tensors: torch.Tensor) -> bool:
        return self._stamps is not None and _native.bind().still(self._stamps, *tensors)

    def __deepcopy__(self, memo) -> "Origin":
        return Origin()

    def __reduce__(self):
        return Origin, ()
