"""The cache: a slot for each live sequence, keys and values for each schedule entry that keeps
its own, and a fixed-size state per sequence for mixers that have one.

Storage is paged: a page holds `TOKENS_PER_PAGE` consecutive positions of one sequence for one
kv head, [tokens, head_dim] contiguous, so a decode kernel streams whole pages. Entries with the
same need (kv heads, head size, window) form a group with pools of their own,
[entries, pages, kv heads, tokens per page, head_dim] for keys and for values, one page table
[slots, pages per sequence] and one free list. A windowed group keeps only as many pages per
sequence as its window can touch and uses them as a ring.

abacus keeps one sequence, [layers][seq_len][kv_dim] float32 (src/model.c:112-113, 256-258);
the slot, the pages and the groups are this library's own.
"""
from dataclasses import dataclass

import torch

from ..kernels import guards
from .need import CacheNeed
from .pages import CacheFull, FreeList, PageBook

TOKENS_PER_PAGE = 64


@dataclass
class LayerKV:
    """What the kernels need to find a sequence's keys and values for one schedule entry."""
    k: torch.Tensor  # [pages, kv heads, tokens per page, head_dim]
    v: torch.Tensor
    page_table: torch.Tensor  # int32 [slots, table_width]
    table_width: int
    ring_pages: int
    tokens_per_page: int
    window: object
    pinned_pages: int = 0  # a windowed group that also keeps a sequence's first pages (they come before the ring)
    values_in_keys: bool = False  # v is k: a value is the first elements of its key row


@dataclass
class EntryView:
    owns_storage: bool  # False: the entry reads the cache of another entry
    kv: object  # LayerKV or None
    state: object  # float32 [slots, *state_shape] or None
    states: dict = None  # further states by name, [slots, *shape] each


class _Group:
    def __init__(self, need, entries, n_pages, max_slots, max_context, dtype, device):
        tpp = TOKENS_PER_PAGE
        self.need, self.entries = need, entries
        self.ring_pages = 0 if need.window is None else (need.window + tpp - 2) // tpp + 1
        self.pinned_pages = -(-need.keep_first // tpp) if self.ring_pages else 0
        per_seq = -(-max_context // tpp)
        if self.ring_pages:
            per_seq = min(per_seq, self.pinned_pages + self.ring_pages)
            n_pages = min(n_pages, max_slots * (self.pinned_pages + self.ring_pages))
        self.table_width = max(1, min(per_seq, n_pages))
        self.book = PageBook(n_pages, tpp, self.ring_pages, self.pinned_pages)
        shape = (len(entries), n_pages, need.n_kv_heads, tpp, need.head_dim)
        self.k = guards.zeros(shape, dtype, device, what="cache keys")  # guard words around the pools
        if need.values_in_keys:  # one pool: a value is the first v_head_dim elements of its key row
            self.v = self.k
        else:
            self.v = guards.zeros(shape[:-1] + (need.v_head_dim or need.head_dim,), dtype, device, what="cache values")
        # the tables as the host has them; what changes goes to the device as arguments of a kernel (no copy from a host
        # buffer, which would have to be kept as it is, or waited for, while earlier steps are in flight)
        self.table_host = torch.zeros((max_slots, self.table_width), dtype=torch.int32)
        self._table_rows = self.table_host.numpy()
        self.table = torch.zeros((max_slots, self.table_width), dtype=torch.int32, device=device)

    def grow(self, slot, new_length):
        """Pages for the sequence to hold new_length tokens, set in the host's table; what changed, flat: word of the table,
        page, word, page, .."""
        added = self.book.grow(slot, new_length)
        if not added:
            return []
        first, pages = added[0][0], [page for _, page in added]
        self._table_rows[slot, first:first + len(pages)] = pages  # (new pages follow those a slot has)
        word = slot * self.table_width + first
        return [x for pair in zip(range(word, word + len(pages)), pages) for x in pair]

    def send(self, changes):
        """The device's table follows; on the table's own device, in the order of the current stream."""
        if not changes:
            return
        if self.table.is_cuda and self.table.get_device() == torch.cuda.current_device():
            from ..kernels import ops
            ops.set_words(self.table, changes)
        else:
            self.table.copy_(self.table_host)


_STATE_TYPES = {"float32": torch.float32, "int32": torch.int32}


class SequenceCache:
    """needs: one CacheNeed (or None) per schedule entry; sources: per entry, None or the entry it reads.
    frame_need: what the model's frame keeps per sequence (a CacheNeed with states only), or None."""

    def __init__(self, needs, sources, max_tokens, dtype, device, max_slots=None, max_context=None, frame_need=None):
        tpp = TOKENS_PER_PAGE
        self.device, self.dtype = torch.device(device), dtype
        self.n_pages = max(1, -(-max_tokens // tpp))
        self.max_slots = max_slots or min(self.n_pages, 4096)
        self.max_context = min(max_context or self.n_pages * tpp, self.n_pages * tpp)
        self.slots = FreeList(self.max_slots, "cache slot")
        self.length = {}
        self.groups, self._of_entry, self.states, self.named_states = [], {}, {}, {}
        by_need = {}
        for e, (need, source) in enumerate(zip(needs, sources)):
            if source is not None or need is None:
                continue
            if need.n_kv_heads > 0:
                keep_first = need.keep_first if need.window is not None else 0
                key = (need.n_kv_heads, need.head_dim, need.window, need.v_head_dim or need.head_dim, keep_first,
                       need.values_in_keys)
                by_need.setdefault(key, []).append(e)
            if need.state_shape:
                self.states[e] = guards.zeros((self.max_slots, *need.state_shape), torch.float32, device,
                                              what=f"state of entry {e}")
            if need.states:
                self.named_states[e] = self._named(need, f"entry {e}")
        self.frame = EntryView(True, None, None, self._named(frame_need, "the frame") if frame_need is not None else {})
        for (hkv, hd, window, vd, keep_first, in_keys), entries in by_need.items():
            g = _Group(CacheNeed(hkv, hd, window, v_head_dim=vd, keep_first=keep_first, values_in_keys=in_keys), entries, self.n_pages,
                       self.max_slots, self.max_context, dtype, self.device)
            self.groups.append(g)
            for i, e in enumerate(entries):
                self._of_entry[e] = (g, i)
        self.sources = list(sources)
        self.views = [self._view(e) for e in range(len(needs))]

    def _named(self, need, whose):
        return {name: guards.zeros((self.max_slots, *shape), _STATE_TYPES[kind], self.device,
                                   what=f"state {name} of {whose}") for name, shape, kind in need.states}

    def _all_states(self):
        yield from self.states.values()
        for named in list(self.named_states.values()) + [self.frame.states]:
            yield from named.values()

    def _view(self, e):
        owner = e if self.sources[e] is None else self.sources[e]
        kv = None
        if owner in self._of_entry:
            g, i = self._of_entry[owner]
            kv = LayerKV(g.k[i], g.v[i], g.table, g.table_width, g.ring_pages, TOKENS_PER_PAGE, g.need.window,
                         g.pinned_pages, g.need.values_in_keys)
        return EntryView(self.sources[e] is None, kv, self.states.get(owner), self.named_states.get(owner, {}))

    # ------------------------------------------------------------ slots
    def open_slot(self):
        """A slot for a new sequence: no tokens, state zeroed."""
        slot = self.slots.take()
        self.length[slot] = 0
        for g in self.groups:
            g.book.open(slot)
        for state in self._all_states():
            state[slot].zero_()
        return slot

    def close_slot(self, slot):
        """Give the slot and all it holds back."""
        self.slots.give_back(slot)
        del self.length[slot]
        for g in self.groups:
            g.book.close(slot)

    def pages_short(self, slot, new_length):
        """How many pages the group that is shortest of them lacks for the slot to grow to new_length (0: it fits)."""
        short = 0
        for g in self.groups:
            want = g.book.pages_for(new_length) - len(g.book.of_slot[slot])
            short = max(short, want - g.book.pages.n_free)
        return short

    def reserve(self, slot, new_length):
        """Room for the sequence to grow to new_length tokens; page tables on the device follow. All groups
        get their pages or none does: a refused call leaves the cache as it was."""
        if new_length > self.max_context:
            raise CacheFull(f"context is full: {new_length} tokens, the cache holds {self.max_context} per sequence")
        short = self.pages_short(slot, new_length)
        if short > 0:
            raise CacheFull(f"the cache lacks {short} free pages of {TOKENS_PER_PAGE} tokens for slot {slot} to hold "
                            f"{new_length} tokens")
        for g in self.groups:
            g.send(g.grow(slot, new_length))

    def reserve_all(self, wanted):
        """reserve() for several slots at once, [(slot, new_length)]: either every one gets its room or the cache
        is left as it was (a step is refused whole, not from its third sequence on)."""
        for slot, new_length in wanted:
            if new_length > self.max_context:
                raise CacheFull(f"context is full: {new_length} tokens, the cache holds {self.max_context} per sequence")
        for g in self.groups:
            need = sum(max(0, g.book.pages_for(n) - len(g.book.of_slot[slot])) for slot, n in wanted)
            if need > g.book.pages.n_free:
                raise CacheFull(f"the cache has {g.book.pages.n_free} free pages of {TOKENS_PER_PAGE} tokens; this step "
                                f"needs {need} more")
        for g in self.groups:
            g.send([x for slot, n in wanted for x in g.grow(slot, n)])

    def save_states(self, slots):
        """Copies of every per-sequence state of these slots (of the mixers' and of the frame's), for restore_states.
        Keys and values need none: writing a position twice leaves the same bytes, running a recurrence twice does not."""
        index = torch.tensor(list(slots), dtype=torch.int64, device=self.device)
        return index, [state.index_select(0, index) for state in self._all_states()]

    def restore_states(self, saved):
        index, copies = saved
        for state, copy in zip(self._all_states(), copies):
            state.index_copy_(0, index, copy)

    def advance(self, slot, n_new):
        self.length[slot] += n_new

    @property
    def free_pages(self):
        return min((g.book.pages.n_free for g in self.groups), default=0)

    def bytes(self):
        total = sum((g.k.numel() + (0 if g.need.values_in_keys else g.v.numel())) * g.k.element_size() for g in self.groups)
        return total + sum(s.numel() * 4 for s in self._all_states())
