"""Device memory of the cache groups: page pools and state slots."""

from __future__ import annotations

import torch

from .manager import CacheManager, PagedGroup


class CacheStorage:
    """One tensor for each group.

    Paged group: ``[slots, 2, num_pages, kv_heads, page_size, head_dim]`` (keys at
    index 0 of the second axis, values at 1); a page of one kv-head is contiguous,
    so a tile of keys is a run of ``page_size * head_dim`` elements.  Where a value
    row has another size than a key row, keys and values are two tensors,
    ``[slots, num_pages, kv_heads, page_size, head_dim]`` and ``[..., value_dim]``; where
    the values are part of the key rows (``PagedNeed.value_in_key``) there is the key
    tensor alone, handed out as both.  The
    reference keeps ``[num_blocks, 16, kv_heads, head_dim]`` per layer
    (acvram/memory/kvcache.py:463-469).  State group:
    ``[slots, max_requests + 1, *shape]`` (the last slot belongs to nobody: padding rows of a
    fixed-shape batch work on it).  Everything starts at zero, so that a key
    that is masked out never brings a NaN into a product.

    Beside its pages a paged group has its block table on the device, int32
    ``[max_requests + 1, width]``: row r belongs to the request that the manager gave row r, the last row to
    nobody; all entries start at -1 ("no page").  ``max_len`` (tokens) decides the width."""

    def __init__(self, manager: CacheManager, device, dtype: torch.dtype, max_len: int | None = None) -> None:
        self.manager = manager
        self.device = torch.device(device)
        self.dtype = dtype
        self.tensors: list[torch.Tensor] = []
        self.value_tensors: dict[int, torch.Tensor] = {}    # group index -> values, where their rows differ from the keys'
        self.tables: dict[int, torch.Tensor] = {}       # group index -> the group's block table on the device
        self.keys_only: set[int] = set()                # groups whose values live inside their key rows
        for gi, g in enumerate(manager.groups):
            if isinstance(g, PagedGroup):
                pages = max(g.pool.num_pages, 1)
                if getattr(g.need, "value_in_key", False):
                    # one kept row per token serves as key and as value: keys only
                    shape = (g.num_slots, pages, g.need.num_kv_heads, g.page_size, g.need.head_dim)
                    self.tensors.append(torch.zeros(shape, device=self.device, dtype=dtype))
                    self.keys_only.add(gi)
                elif g.need.value_size == g.need.head_dim:
                    shape = (g.num_slots, 2, pages, g.need.num_kv_heads, g.page_size, g.need.head_dim)
                    self.tensors.append(torch.zeros(shape, device=self.device, dtype=dtype))
                else:
                    shape = (g.num_slots, pages, g.need.num_kv_heads, g.page_size)
                    self.tensors.append(torch.zeros((*shape, g.need.head_dim), device=self.device, dtype=dtype))
                    self.value_tensors[gi] = torch.zeros((*shape, g.need.value_size), device=self.device, dtype=dtype)
                # a request that keeps all its keys can never hold more pages than the pool has
                tokens = max_len if max_len else g.pool.num_pages * g.page_size
                if g.need.keeps_all:
                    tokens = min(tokens, g.pool.num_pages * g.page_size)
                width = max(1, g.pages_for(tokens))
                self.tables[gi] = torch.full((manager.max_requests + 1, width), -1, device=self.device, dtype=torch.int32)
            else:
                sdtype = getattr(torch, g.need.dtype)
                self.tensors.append(torch.zeros((g.num_slots, g.max_requests + 1, *g.need.shape), device=self.device,
                                                dtype=sdtype))
        self._pages: dict[int, tuple[torch.Tensor, torch.Tensor]] = {}      # cache slot -> its views, once asked for

    def bytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in (*self.tensors, *self.value_tensors.values()))

    @property
    def max_tokens(self) -> int:
        """The longest request that every block table has columns for."""
        return min((t.shape[1] * self.manager.page_size for t in self.tables.values()), default=1 << 30)

    def pages(self, cache_slot: int) -> tuple[torch.Tensor, torch.Tensor]:
        """(keys, values) of a cache slot, ``[num_pages, kv_heads, page_size, head_dim]`` (values: ``value_dim``)."""
        got = self._pages.get(cache_slot)
        if got is None:
            got = self._pages[cache_slot] = self._pages_of(cache_slot)
        return got

    def _pages_of(self, cache_slot: int) -> tuple[torch.Tensor, torch.Tensor]:
        plan = self.manager.plan
        g, i = plan.group_of_slot[cache_slot], plan.index_in_group[cache_slot]
        if g in self.value_tensors:
            return self.tensors[g][i], self.value_tensors[g][i]
        if g in self.keys_only:
            return self.tensors[g][i], self.tensors[g][i]
        t = self.tensors[g][i]
        return t[0], t[1]

    def state(self, cache_slot: int) -> torch.Tensor:
        """State of a cache slot for all request slots: ``[max_requests + 1, *shape]``."""
        plan = self.manager.plan
        return self.tensors[plan.group_of_slot[cache_slot]][plan.index_in_group[cache_slot]]

    def zero_state(self, group: int, slot: int) -> None:
        self.tensors[group][:, slot].zero_()
