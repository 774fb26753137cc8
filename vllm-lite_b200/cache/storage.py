"""Device tensors behind the cache manager's bookkeeping.

A paged group with c entries of the running order is one tensor
[c, 2, pages, kv_heads, page_size, head_dim] (keys at [:, 0], values at [:, 1]):
a (kv head, page) tile of page_size x head_dim is contiguous, which is what the
attention kernels read.  A group of latent rows (`PagedLatent`) has one plane,
[c, 1, pages, 1, page_size, width], handed out both as keys and as values.  A fixed-state group is [c, slots, *shape].  Pages are
never cleared when they change hands: attention reads only what the block table
and the positions name.  State slots are zeroed when they are handed out.
"""
from __future__ import annotations

import torch

from ..parts.base import CallCache
from .manager import CacheLayout

FILL_RUNS = 3        # most runs of neighbouring slots that are filled one by one
_STATE_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "int32": torch.int32}


class CacheStorage:
    def __init__(self, layout: CacheLayout, page_size: int, num_pages, max_requests: int, dtype, device):
        self.layout = layout
        counts = [int(num_pages)] * len(layout.paged_groups) if isinstance(num_pages, int) else list(num_pages)
        self.paged = [torch.zeros((len(members), need.planes, n, need.num_kv_heads, page_size, need.head_dim),
                                  dtype=dtype, device=device)
                      for need, members, n in zip(layout.paged_groups, layout.paged_members, counts)]
        self.state = [torch.zeros((len(members), max_requests) + tuple(need.shape),
                                  dtype=_STATE_DTYPES[need.dtype], device=device)
                      for need, members in zip(layout.state_groups, layout.state_members)]
        self.call_caches = []
        for place in layout.call_place:
            if place is None:
                self.call_caches.append(CallCache())
            elif place[0] == "several":
                self.call_caches.append(CallCache(parts=[self._call_cache(p) for p in place[1]]))
            else:
                self.call_caches.append(self._call_cache(place))

    def _call_cache(self, place) -> CallCache:
        kind, g, idx, owns = place
        if kind == "paged":
            return CallCache(group=g, k=self.paged[g][idx, 0], v=self.paged[g][idx, self.paged[g].shape[1] - 1], writes=owns)
        return CallCache(group=g, state=self.state[g][idx], writes=owns)

    def zero_slots(self, slots):
        if not slots:
            return
        runs = []                                    # of neighbouring slots: a fill each, and no list of indices to upload
        for s in sorted(slots):
            if runs and runs[-1][1] == s:
                runs[-1][1] = s + 1
            else:
                runs.append([s, s + 1])
        if len(runs) <= FILL_RUNS:
            for t in self.state:
                for lo, hi in runs:
                    t[:, lo:hi].zero_()
        elif self.state:
            # scattered slots: one launch a tensor, the list uploaded once and, from pinned memory, without waiting for the steps before
            index, device = torch.tensor(sorted(slots)), self.state[0].device
            if device.type == "cuda":
                index = index.pin_memory().to(device, non_blocking=True)
            for t in self.state:
                t.index_fill_(1, index, 0)

    def bytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in self.paged + self.state)
