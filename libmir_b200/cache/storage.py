"""Device memory behind the cache manager's ids.

Per group one allocation for the keys, [entries, pages * page_size, kv_heads, head_dim], and one for the
values, [entries, pages * page_size, kv_heads, value_dim], in the engine's dtype, so a page id is the same
offset in every layer run of the group (libmir keeps one K and one V buffer per layer with widths of their
own, cuda/src/backend/kv/storage/mod.rs:17-25,47-89; token-major NHD layout as there).
Per schedule entry with fixed-size state: [max_requests, *shape], one record per request slot.
"""

from __future__ import annotations

from dataclasses import dataclass, replace
from typing import Dict, Optional, Tuple

import torch

from .. import kernels
from .manager import CacheManager

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "int32": torch.int32}


@dataclass
class CacheView:
    """What one schedule entry's mixer gets."""

    group: Optional[int] = None            # index of the paged group, None if the entry has no pages
    k_pages: Optional[torch.Tensor] = None  # [pages * page_size, kv_heads, head_dim]
    v_pages: Optional[torch.Tensor] = None
    page_size: int = 0
    writes: bool = True                     # False: the entry reads another entry's cache
    state: Optional[torch.Tensor] = None    # [max_requests, *shape] fixed-size state, indexed by slot (the first one)
    states: Tuple[torch.Tensor, ...] = ()   # every fixed-size state of the entry, in the order they were asked for

    def part(self, pages: bool, first_state: int, state_count: int) -> "CacheView":
        """What one mechanism of a mixer made of several sees: the pages (or none) and its own run of the states."""
        mine = tuple(self.states[first_state:first_state + state_count])
        view = replace(self, states=mine, state=mine[0] if mine else None)
        if not pages:
            view.group, view.k_pages, view.v_pages = None, None, None
        return view


class CacheStorage:
    def __init__(self, manager: CacheManager, plan, dtype: torch.dtype, device: torch.device):
        self.manager = manager
        self.key_buffers, self.value_buffers = [], []
        for group in manager.groups:
            r = group.requirement
            rows = group.pool.count * manager.page_size
            self.key_buffers.append(torch.zeros((len(group.entries), rows, r.kv_heads, r.head_dim), dtype=dtype,
                                                device=device))
            self.value_buffers.append(torch.zeros((len(group.entries), rows, r.kv_heads, r.value_dim), dtype=dtype,
                                                  device=device))
        self.buffers = self.key_buffers + self.value_buffers
        self.states: Dict[int, object] = {}        # entry -> tensor, or tuple of tensors where the entry has several
        make = lambda requirement: torch.zeros((manager.max_requests, *requirement.shape),
                                               dtype=_DTYPES[requirement.dtype], device=device)
        for entry, requirement in manager.state_entries.items():
            self.states[entry] = tuple(make(r) for r in requirement) if isinstance(requirement, tuple) else make(requirement)
        tensors = self._state_tensors()
        if tensors and tensors[0].device.type == "cuda":       # where each state's records are, for the kernel that zeroes them
            record = [t[0].numel() * t.element_size() for t in tensors]
            self._regions = torch.tensor([[t.data_ptr(), size] for t, size in zip(tensors, record)], device=device)
            self._largest = max(record)
        self.views: Dict[int, CacheView] = {}
        for item in plan:
            view = CacheView(writes=item.source == item.entry)
            if item.entry in manager.entry_group:
                group = manager.entry_group[item.entry]
                local = manager.entry_local[item.entry]
                view.group = group
                view.k_pages = self.key_buffers[group][local]
                view.v_pages = self.value_buffers[group][local]
                view.page_size = manager.page_size
            if item.source in self.states:
                held = self.states[item.source]
                view.states = held if isinstance(held, tuple) else (held,)
                view.state = view.states[0]
            self.views[item.entry] = view

    def zero_slots(self, slots) -> None:
        """Fixed-size state of newly admitted requests starts at zero."""
        if not slots or not self.states:
            return
        tensors = self._state_tensors()
        if tensors[0].device.type != "cuda":
            index = torch.tensor(slots, dtype=torch.long)
            for state in tensors:
                state.index_fill_(0, index, 0)
            return
        limit = self.manager.max_requests
        if any(not 0 <= slot < limit for slot in slots):
            raise IndexError(f"state slots {list(slots)} are not all within 0 .. {limit - 1}")
        kernels.zero_slots(self._regions, self._largest, slots)

    def _state_tensors(self):
        return [t for held in self.states.values() for t in (held if isinstance(held, tuple) else (held,))]

    def bytes(self) -> int:
        return sum(b.numel() * b.element_size() for b in self.buffers) + \
            sum(t.numel() * t.element_size() for t in self._state_tensors())
