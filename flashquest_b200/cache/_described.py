"""What the three persistent caches share: the C record of their storage that the native calls take."""
from __future__ import annotations

from transformers.cache_utils import Cache

from .._lib import bind


class DescribedCache(Cache):
    """_storage (an attrgetter) names the tensors whose addresses _describe() puts into the record.  The record is made when first asked for
    and again whenever one of those tensors has been replaced; neither it nor the step objects built on it belong to a copied
    or saved cache (they hold addresses)."""
    _desc = None
    _desc_of = None

    def desc(self):
        at = bind().addresses(self._storage(self), self._desc_of)      # one native call: this runs for every token and layer
        if at is not self._desc_of:
            self._desc, self._desc_of = self._describe(), at
        return self._desc

    def __getstate__(self):
        state = dict(self.__dict__)
        for name in ("_desc", "_desc_of", "_fq_engines"):
            state.pop(name, None)
        return state
