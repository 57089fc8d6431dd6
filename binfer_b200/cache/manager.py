"""The cache manager: paged keys and values with a block table per request, in groups.

A *group* is a set of schedule entries (layer executions) whose caches have the
same geometry and the same retention rule: same kv heads, head size and window.
Each group has a page pool and block tables of its own.  A page id is valid for
every entry of its group (the reference's one pool works the same way across
all layers, src/kv/paged.ts:71-81).  In a windowed group the pages that every
later query has passed are given back while the request is still running.

Beside the pages, every live request holds one *slot*: an index into
fixed-size per-request state tensors that mixers may ask for (this
architecture asks for none, so those tensors are empty).

Pages are allocated by ``reserve`` before a step for exactly the tokens the
step writes; a failure raises :class:`OutOfPages` and changes nothing (the
reference ignores the failure of ``extendSequence``, src/serve.ts:390,476).
"""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import Dict, Hashable, List, Optional, Sequence, Tuple

from .pages import OutOfPages, PagePool, SlotPool


@dataclass(frozen=True)
class KVNeed:
    """What one layer execution asks of the paged cache.

    ``value_dim``: size of a value head where it differs from a key head's (None: the same).
    ``pools``: block sizes P for which, beside the tokens, one mean key and value per P
    tokens is kept for as long as the request lives (attention that sees pooled blocks of
    the keys behind its window); each P gets a *summary group* of its own, in which a
    request holds ``length // P`` entries.  A token's page is then kept until the token has
    left the window AND its block's mean is taken.  ``stride`` > 1 marks such a summary
    group's own need (made by the manager, not by mixers).  ``keep_first``: with a window,
    the request's first that many tokens stay visible for good, so the pages that hold them
    are never given back while the request lives."""

    num_kv_heads: int
    head_dim: int
    window: Optional[int] = None     # None: every key is kept
    value_dim: Optional[int] = None
    pools: Tuple[int, ...] = ()
    stride: int = 1
    keep_first: int = 0

    @property
    def v_dim(self) -> int:
        return self.head_dim if self.value_dim is None else self.value_dim

    @property
    def group_key(self) -> Tuple:
        if (self.value_dim is None and not self.pools and self.stride == 1
                and not self.kept_tokens):
            return (self.num_kv_heads, self.head_dim, self.window)
        return (self.num_kv_heads, self.head_dim, self.window, self.v_dim, self.pools,
                self.stride, self.kept_tokens)

    @property
    def kept_tokens(self) -> int:
        """First tokens that stay behind the window (nothing without a window: all stay)."""
        return int(self.keep_first) if self.window is not None else 0

    def merged(self, other: "KVNeed") -> "KVNeed":
        """The need of a cache that serves this execution and another that reads it: the
        wider window, the pools of both."""
        if (self.num_kv_heads, self.head_dim, self.v_dim) != (other.num_kv_heads,
                                                              other.head_dim, other.v_dim):
            raise ValueError("an execution that reads another's cache must have its head "
                             "count and head sizes")
        window = (None if self.window is None or other.window is None
                  else max(self.window, other.window))
        pools = tuple(sorted(set(self.pools) | set(other.pools))) if window is not None else ()
        return KVNeed(self.num_kv_heads, self.head_dim, window, self.value_dim, pools,
                      keep_first=max(self.kept_tokens, other.kept_tokens))


@dataclass(frozen=True)
class StateNeed:
    """Per-request state of fixed size that one layer execution keeps."""

    shape: Tuple[int, ...]
    dtype: str = "float32"


@dataclass
class RequestCache:
    rid: Hashable
    slot: int
    length: int = 0                            # tokens whose keys/values are cached
    tables: List[List[int]] = field(default_factory=list)   # per group: page id or -1
    fresh: bool = True                         # state slot not yet zeroed on the device
    # per group: the table as an int32 array for the step's batch description, kept in step
    # with `tables` (entries appended; rebuilt after a windowed page was released)
    np_tables: List[object] = field(default_factory=list)
    np_valid: List[int] = field(default_factory=list)

    def table_array(self, g: int):
        """``tables[g]`` as a numpy int32 array (a view of a cached buffer)."""
        import numpy as np
        table = self.tables[g]
        n = len(table)
        while len(self.np_tables) <= g:
            self.np_tables.append(None)
            self.np_valid.append(0)
        arr, valid = self.np_tables[g], self.np_valid[g]
        if arr is None or arr.shape[0] < n or valid < 0:
            arr = np.zeros(max(16, 2 * n), dtype=np.int32)
            arr[:n] = table
            self.np_tables[g] = arr
        elif valid < n:
            arr[valid:n] = table[valid:n]
        self.np_valid[g] = n
        return arr[:n]


def plan_pages(kv_needs: Sequence[Optional[KVNeed]], page_size: int, budget_bytes: int,
               element_size: int, max_requests: int, max_seq_len: int,
               max_tokens_per_step: int):
    """Share ``budget_bytes`` out among the cache groups; returns ``need -> pages`` for
    :class:`CacheManager`.

    A group that keeps every key needs ``max_seq_len`` tokens per request at most; a windowed
    one needs its window plus the longest portion a step may write (pages behind the window
    are given back before a step's new ones are taken) plus a page's slack at either end.
    Groups get pages in proportion to those needs, the windowed ones never more than
    ``max_requests`` requests can use; what that saves goes to the others.  (The reference
    has one pool, every layer alike: src/kv/paged.ts:55-62.)"""
    per_request, page_bytes = {}, {}
    for need in kv_needs:
        if need is None:
            continue
        key = need.group_key
        tokens = max_seq_len if need.window is None else min(
            max_seq_len, need.window + max(need.pools, default=0) + need.kept_tokens
            + max_tokens_per_step)
        per_request[key] = -(-tokens // page_size) + 2
        page_bytes[key] = page_bytes.get(key, 0) + (
            need.num_kv_heads * (need.head_dim + need.v_dim) * page_size * element_size)
        for P in need.pools:         # the summary group of this pool size
            sk = summary_need(need, P).group_key
            per_request[sk] = -(-(max_seq_len // P) // page_size) + 1
            page_bytes[sk] = page_bytes.get(sk, 0) + (
                need.num_kv_heads * (need.head_dim + need.v_dim) * page_size * element_size)
    # pages per unit of "request": scale every group's need by the same factor f
    unit = sum(per_request[k] * page_bytes[k] for k in per_request)
    f = min(float(max_requests), budget_bytes / unit) if unit else 0.0
    pages = {k: max(1, int(f * per_request[k])) for k in per_request}
    return lambda need: pages[need.group_key]


def summary_need(need: KVNeed, pool: int) -> KVNeed:
    """The need of the summary group that holds one mean key and value per ``pool`` tokens
    for caches of ``need``'s geometry."""
    return KVNeed(need.num_kv_heads, need.head_dim, None, need.value_dim, (), int(pool))


class CacheGroup:
    def __init__(self, index: int, need: KVNeed, num_pages: int, page_size: int):
        self.index = index
        self.need = need
        self.page_size = page_size
        self.stride = max(1, int(need.stride))   # tokens per entry (a summary group: the pool)
        # pages of one 128-key attention tile lie side by side in the pool where they can
        self.pool = PagePool(num_pages, run=max(1, 128 // page_size))
        self.entries: List[int] = []           # schedule entries stored here, in order
        self.storage = None                    # device tensor, see allocate_storage()

    def first_needed_page(self, length: int) -> int:
        """Index of the first logical page that a query at position >= ``length`` reads."""
        w = self.need.window
        if w is None:
            return 0
        first_key = max(0, length - w + 1)
        for P in self.need.pools:        # tokens of a block whose mean is not yet taken stay
            first_key = min(first_key, (length // P) * P)
        return first_key // self.page_size

    @property
    def kept_pages(self) -> int:
        """Logical pages at a request's start that are never given back: those that hold
        the first tokens a window keeps."""
        return -(-self.need.kept_tokens // self.page_size)

    def entries_for(self, length: int) -> int:
        """Entries (tokens; blocks in a summary group) that a request of ``length`` tokens holds."""
        return length // self.stride


class CacheManager:
    """Host-side bookkeeping; device storage is attached by ``allocate_storage``."""

    def __init__(self, kv_needs: Sequence[Optional[KVNeed]],
                 state_needs: Sequence[Optional[StateNeed]] = (),
                 page_size: int = 16, num_pages=64, max_requests: int = 64):
        """``num_pages``: pages of every group's pool, or a function of a group's
        :class:`KVNeed` that gives its pool's pages (a windowed group keeps far fewer keys
        per request than one that keeps them all: see :func:`plan_pages`)."""
        if page_size < 1:
            raise ValueError("page_size must be positive")
        self.page_size = int(page_size)
        pages_of = num_pages if callable(num_pages) else (lambda need: int(num_pages))
        self.groups: List[CacheGroup] = []
        # schedule entry -> (group index, index of the entry inside its group)
        self.entry_location: List[Optional[Tuple[int, int]]] = []
        # (schedule entry, pool size) -> (summary group index, index of the entry inside it)
        self.summary_location: Dict[Tuple[int, int], Tuple[int, int]] = {}
        by_key: Dict[Tuple, CacheGroup] = {}
        for e, need in enumerate(kv_needs):
            if need is None:
                self.entry_location.append(None)
                continue
            g = by_key.get(need.group_key)
            if g is None:
                g = CacheGroup(len(self.groups), need, int(pages_of(need)), self.page_size)
                by_key[need.group_key] = g
                self.groups.append(g)
            self.entry_location.append((g.index, len(g.entries)))
            g.entries.append(e)
            for P in need.pools:
                sn = summary_need(need, P)
                sg = by_key.get(sn.group_key)
                if sg is None:
                    sg = CacheGroup(len(self.groups), sn, int(pages_of(sn)), self.page_size)
                    by_key[sn.group_key] = sg
                    self.groups.append(sg)
                self.summary_location[(e, P)] = (sg.index, len(sg.entries))
                sg.entries.append(e)
        self._plain = (len(self.groups) == 1 and self.groups[0].need.window is None
                       and self.groups[0].stride == 1)
        # the largest pool (what a request that keeps every key can draw on)
        self.num_pages = max([g.pool.num_pages for g in self.groups], default=0)
        self.state_needs = list(state_needs) + [None] * (len(kv_needs) - len(state_needs))
        self.slots = SlotPool(max_requests)
        self.requests: Dict[Hashable, RequestCache] = {}
        self.state_storage: List[object] = [None] * len(self.state_needs)

    # ------------------------------------------------------------- requests
    def add_request(self, rid: Hashable) -> RequestCache:
        if rid in self.requests:
            raise ValueError(f"request {rid!r} is already live")
        rc = RequestCache(rid, self.slots.alloc(), 0, [[] for _ in self.groups])
        self.requests[rid] = rc
        return rc

    def get(self, rid: Hashable) -> RequestCache:
        return self.requests[rid]

    def free_request(self, rid: Hashable) -> None:
        """Give back every page and the slot of ``rid``."""
        rc = self.requests.pop(rid)
        for g, table in zip(self.groups, rc.tables):
            for p in table:
                if p > 0:
                    g.pool.free(p)
            table.clear()
        self.slots.free(rc.slot)

    # ---------------------------------------------------------------- pages
    def pages_to_add(self, rc: RequestCache, new_len: int) -> List[int]:
        """Pages each group must newly allocate so that positions < ``new_len`` are
        covered, counting the pages that the step will release first."""
        out = []
        for g, table in zip(self.groups, rc.tables):
            want = -(-g.entries_for(new_len) // g.page_size)
            add = max(0, want - len(table))
            first = g.first_needed_page(rc.length)
            if first > g.kept_pages:
                add -= sum(1 for p in table[g.kept_pages:first] if p > 0)
            out.append(add)
        return out

    def free_after(self, wants: Sequence[Tuple[Hashable, int]]) -> List[int]:
        """Free pages each group would have left after reserving every ``(rid, new_len)``
        (negative: that many pages short)."""
        need = [0] * len(self.groups)
        for rid, new_len in wants:
            rc = self.requests[rid]
            for i, n in enumerate(self.pages_to_add(rc, new_len)):
                need[i] += n
        return [g.pool.num_free - n for n, g in zip(need, self.groups)]

    def can_reserve(self, wants: Sequence[Tuple[Hashable, int]], spare: int = 0) -> bool:
        """Whether ``reserve`` would succeed for all ``(rid, new_len)`` together and still
        leave ``spare`` pages free in every group."""
        return all(n >= spare for n in self.free_after(wants))

    def reserve_all(self, wants: Sequence[Tuple[Hashable, int]]) -> bool:
        """``reserve`` for every ``(rid, new_len)``; False, with nothing changed, where their pages
        together are lacking."""
        if not self._plain:
            if not self.can_reserve(wants):
                return False
            for rid, new_len in wants:
                self.reserve(rid, new_len)
            return True
        # one group that keeps every key: nothing to give back, and a step's single tokens rarely
        # begin a page (32 requests: 100 us of a step's host time less)
        g, ps, need, todo = self.groups[0], self.page_size, 0, []
        for rid, new_len in wants:
            rc = self.requests[rid]
            if new_len < rc.length:
                raise ValueError(f"request {rid!r} holds {rc.length} tokens, cannot shrink to {new_len}")
            table = rc.tables[0]
            want = -(-new_len // ps)
            if want > len(table):
                need += want - len(table)
                todo.append((table, want))
        if need > g.pool.num_free:
            return False
        for table, want in todo:
            while len(table) < want:
                table.append(g.pool.alloc(after=max(table[-1], 0) if table else 0, index=len(table)))
        return True

    def reserve(self, rid: Hashable, new_len: int) -> None:
        """Make the block tables of ``rid`` cover positions < ``new_len``.

        Pages of a windowed group that lie wholly before the window of the
        request's next query are released first.  Raises :class:`OutOfPages`,
        with nothing changed, if any group lacks pages.
        """
        rc = self.requests[rid]
        if new_len < rc.length:
            raise ValueError(f"request {rid!r} holds {rc.length} tokens, cannot shrink to {new_len}")
        for g, n in zip(self.groups, self.pages_to_add(rc, new_len)):
            if n > g.pool.num_free:
                raise OutOfPages(
                    f"request {rid!r} needs {n} more pages in cache group {g.index}, "
                    f"{g.pool.num_free} free of {g.pool.num_pages}")
        for g, table in zip(self.groups, rc.tables):
            self._release_passed(g, rc, table)
            want = -(-g.entries_for(new_len) // g.page_size)
            while len(table) < want:
                table.append(g.pool.alloc(after=max(table[-1], 0) if table else 0,
                                          index=len(table)))

    def _release_passed(self, g: CacheGroup, rc: RequestCache, table: List[int]) -> None:
        first = min(g.first_needed_page(rc.length), len(table))
        for i in range(g.kept_pages, first):
            if table[i] > 0:
                g.pool.free(table[i])
                table[i] = -1
                if len(rc.np_valid) > g.index:
                    rc.np_valid[g.index] = -1      # the cached array is stale

    def commit(self, rid: Hashable, new_len: int) -> None:
        """Record that the step wrote keys/values up to ``new_len``."""
        rc = self.requests[rid]
        assert new_len >= rc.length
        for g, table in zip(self.groups, rc.tables):
            assert len(table) * g.page_size >= g.entries_for(new_len), \
                "commit beyond the reserved pages"
        rc.length = new_len

    def commit_all(self, rcs: Sequence[RequestCache], new_lens: Sequence[int]) -> None:
        """``commit`` for every request of a step."""
        if not self._plain:
            for rc, new_len in zip(rcs, new_lens):
                self.commit(rc.rid, new_len)
            return
        ps = self.page_size
        for rc, new_len in zip(rcs, new_lens):
            assert new_len >= rc.length and len(rc.tables[0]) * ps >= new_len, \
                "commit beyond the reserved pages"
            rc.length = new_len

    def release_passed(self, rid: Hashable) -> None:
        """Give back windowed pages that the request's next query no longer reads."""
        rc = self.requests[rid]
        for g, table in zip(self.groups, rc.tables):
            self._release_passed(g, rc, table)

    # ---------------------------------------------------------------- views
    def num_free_pages(self) -> List[int]:
        return [g.pool.num_free for g in self.groups]

    def pages_for_tokens(self, n: int) -> int:
        """Pages one full-attention group needs for ``n`` tokens (src/kv/paged.ts:180)."""
        return -(-n // self.page_size)

    def can_ever_hold(self, n: int) -> bool:
        """Whether a lone request of ``n`` tokens fits every group's pool: all of its pages
        where every key is kept, its window's pages (and the one being written) elsewhere,
        where a long prompt can always come in short portions."""
        for g in self.groups:
            w = g.need.window
            if w is not None:
                w += max(g.need.pools, default=0)
            m = g.entries_for(n)
            need = -(-m // g.page_size) if w is None else min(
                -(-m // g.page_size), -(-min(m, w + 1) // g.page_size) + 1 + g.kept_pages)
            if need > g.pool.num_pages:
                return False
        return True

    def check_consistent(self) -> None:
        """Every page is either free or held by exactly one live request."""
        for gi, g in enumerate(self.groups):
            seen = set()
            for rc in self.requests.values():
                for p in rc.tables[gi]:
                    if p > 0:
                        assert p not in seen, f"page {p} of group {gi} is held twice"
                        assert g.pool.is_held(p), f"page {p} of group {gi} is in a table but free"
                        seen.add(p)
            assert len(seen) == g.pool.num_held, (
                f"group {gi}: {g.pool.num_held} pages held, {len(seen)} in tables (a page is lost)")
        assert len(self.requests) == self.slots.num_slots - self.slots.num_free

    # -------------------------------------------------------------- storage
    def allocate_storage(self, dtype, device) -> None:
        """Device tensors: per group ``[entries, 2, pages + 1, kv_heads, page_size, head_dim]``
        (keys at index 0, values at 1; page 0 is scratch), or, where keys and values differ in
        size, a pair of tensors ``[entries, pages + 1, kv_heads, page_size, d]``; and per
        schedule entry with a :class:`StateNeed` a tensor ``[slots + 1, *shape]`` (the last
        slot is scratch: padded rows of a captured step use it)."""
        import torch
        for g in self.groups:
            n = g.need
            shape = (len(g.entries), g.pool.num_pages + 1, n.num_kv_heads, g.page_size)
            if n.v_dim == n.head_dim:
                g.storage = torch.zeros((shape[0], 2) + shape[1:] + (n.head_dim,),
                                        dtype=dtype, device=device)
            else:
                g.storage = (torch.zeros(shape + (n.head_dim,), dtype=dtype, device=device),
                             torch.zeros(shape + (n.v_dim,), dtype=dtype, device=device))
        for e, need in enumerate(self.state_needs):
            if need is not None:
                self.state_storage[e] = torch.zeros(
                    (self.slots.num_slots + 1,) + tuple(need.shape),
                    dtype=getattr(torch, need.dtype), device=device)

    def zero_fresh_state(self, rc: RequestCache) -> None:
        """Clear the state slot of a newly admitted request (its last owner's state is stale)."""
        if rc.fresh:
            for st in self.state_storage:
                if st is not None:
                    st[rc.slot].zero_()
            rc.fresh = False

    def kv_view(self, entry: int):
        """(keys, values) storage of schedule entry ``entry``: each
        ``[pages + 1, kv_heads, page_size, head_dim]``; and its group index."""
        gi, ei = self.entry_location[entry]
        return self._kv_of(gi, ei) + (gi,)

    def _kv_of(self, gi: int, ei: int):
        st = self.groups[gi].storage
        if isinstance(st, tuple):
            return st[0][ei], st[1][ei]
        return st[ei, 0], st[ei, 1]

    def summary_views(self, entry: int) -> Dict[int, Tuple]:
        """Per pool size kept for schedule entry ``entry``: (mean keys, mean values, group
        index), each tensor ``[pages + 1, kv_heads, page_size, d]`` with one entry per block."""
        out = {}
        for (e, P), (gi, ei) in self.summary_location.items():
            if e == entry:
                out[P] = self._kv_of(gi, ei) + (gi,)
        return out

    @property
    def scratch_slot(self) -> int:
        """The state slot that belongs to no request."""
        return self.slots.num_slots

    def storage_bytes(self) -> int:
        total = 0
        for g in self.groups:
            for st in (g.storage if isinstance(g.storage, tuple) else (g.storage,)):
                if st is not None:
                    total += st.numel() * st.element_size()
        return total
