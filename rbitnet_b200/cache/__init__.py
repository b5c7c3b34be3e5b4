from .allocator import FreeList, SlotBook, CacheFull, ContextOverflow
from .cache import SequenceCache, CacheLayerView, CacheGroup, PAGE_SIZE
from .upload import upload

__all__ = ["FreeList", "SlotBook", "CacheFull", "ContextOverflow", "SequenceCache", "CacheLayerView",
           "CacheGroup", "PAGE_SIZE", "upload"]
