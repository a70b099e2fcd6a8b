"""One step's rows on the device: what the cache manager planned, copied over in one piece.

Kapel uploads `ids, positions, lines, pages, rows, slots` as separate small tensors
(crates/kapel-models/src/cache.rs:822-842). Here they are slices of one int32 buffer that
crosses from pinned host memory in a single copy.
"""
from __future__ import annotations

from typing import Dict, List, Optional, Sequence

import numpy as np
import torch

from ..cache import Plan
from ..kernels import row_tile_blocks, sm_count


class GroupBatch:
    __slots__ = ("lines", "block_table")

    def __init__(self, lines, block_table):
        self.lines = lines                # [rows] int32 on the device
        self.block_table = block_table    # [entries, width] int32 on the device


def _chunks_touched(row_count: np.ndarray, window: Optional[int], chunk: int) -> int:
    """The most key chunks (cut at absolute multiples of `chunk`) any row of the step reads."""
    c = row_count[row_count > 0].astype(np.int64)
    if c.size == 0:
        return 1
    first = np.maximum(0, c - window) if window else np.zeros_like(c)
    return int(((c - 1) // chunk - first // chunk + 1).max())


SPLIT_STEP = 64          # splits are multiples of the kernels' key tile


def decode_split(pairs: int, longest: int, sms: int, window: Optional[int] = None, relative: bool = False):
    """(split, slots) of the decode attention kernel, which runs one block a multiprocessor.
    Keys are cut at multiples of `split`, counted from key 0 (`slots` then covers the longest
    request, `longest` positions) or, with `relative`, from each row's first visible key (`slots`
    covers what a row can see). A row reads at most `window` keys, so only about window / split of the
    slots do work. The split is chosen so that the working blocks (`pairs` (tile, kv head)
    pairs times working slots) take as little time as possible: waves of blocks times the keys a
    block walks plus what a block costs to start and to merge (about 192 keys' worth)."""
    pairs = max(1, pairs)
    span = min(longest, window) if window else longest
    best = None
    most = max(1, -(-span // SPLIT_STEP))
    for want in range(1, min(most, 4 * sms) + 1):
        split = max(SPLIT_STEP, -(-(-(-span // want)) // SPLIT_STEP) * SPLIT_STEP)
        working = -(-span // split) + (1 if (window and longest > window and not relative) else 0)
        cost = -(-(pairs * working) // sms) * (split + 192)
        if best is None or cost < best[0]:
            best = (cost, split)
    split = best[1]
    return split, max(1, -(-(span if relative else longest) // split))


# Latent attention: a request's rows from which its keys and values are made for every head: that costs about 6 ns a position (16 heads of
# 128 / 128 from 512 components), and then a pair of a row and a key costs 0.02 ns instead of the 0.4 that it costs over the cached
# lines, so a portion of some twenty rows pays for it; 64 leaves room for the launches. And the most positions laid out so in a pass
# (the part bounds their bytes).
LATENT_PROMPT_ROWS = 64
LATENT_PROMPT_POSITIONS = 131072

# The 32-bit attention by tiles: rows a tile, and the fewest tokens a request may bring.
ROW_TILE = 32
ROW_TILE_TOKENS = 16


def row_tiles_pay(row_count, tile_row0, tile_nq, kv_heads: int, heads_per_kv: int, head_dim: int, window: Optional[int], sms: int,
                  positions: Optional[int] = None) -> bool:
    """Whether the 32-bit attention of these rows is faster by tiles than row by row; `positions`: what a request's block table holds (None: the longest
    row's). A block of the tile kernel walks all the keys of its tile, 64 a step, however few its rows: few tiles behind a long history leave
    the GPU idle, where the row-wise kernel has a block a row, kv head and 256 keys. By tiles a step takes 17.0 us (heads of 256) or 11.4 (of 128), a block a
    multiprocessor; with two blocks a tile (`kernels.row_tile_blocks`) half the steps of 17.2 or 12.9. Row by row the longest block's keys take 0.08 us (one head of
    128) to 0.17 (two of 256, four of 128) each, or all keys 0.018 to 0.051 us a key and multiprocessor, and a quarter of the shorter.
    As measured on a B200, 8 heads over 4 of 256, by tiles and row by row, in us: 500 tokens 99 and 215; 16 tokens behind 256, 1,024 and 4,096 positions
    60 and 47, 164 and 51, 579 and 110; 128 tokens behind 0, 1,024 and 4,096 27 and 27, 166 and 206, 582 and 731; 500 behind 1,024 373 and 895."""
    count = np.asarray(row_count, np.int64)
    row0 = np.asarray(tile_row0, np.int64)
    first, last = count[row0], count[row0 + np.asarray(tile_nq, np.int64) - 1]
    steps = -(-(last - (np.maximum(0, first - window) if window else 0)) // 64)
    if row_tile_blocks(len(steps), kv_heads, head_dim, window, int(count.max()) if positions is None else positions, sms) == 2:
        by_tiles = 3.0 + 0.02 * head_dim + (8.6 + 0.0337 * head_dim) * max(-(-float(steps.max()) // 2), 1.1 * float(steps.sum()) * kv_heads / sms)
    else:
        by_tiles = 6.0 + (5.8 + 0.0438 * head_dim) * max(float(steps.max()), 1.1 * float(steps.sum()) * kv_heads / sms)
    seen = np.where(count > window, window + 200, count) if window else count      # a window begins within a block's keys: one more, partly idle
    slices, heads = -(-heads_per_kv // 8), min(heads_per_kv, 8)      # the row-wise kernel's blocks have up to eight heads
    longest = (0.00046 * head_dim + 0.0293 * heads - 0.008) * min(256.0, float(count.max()))
    every = head_dim * (0.0000794 + 0.000065 * heads) * float(seen.sum()) * kv_heads * slices / sms
    return by_tiles <= 3.0 + max(longest, every) + 0.25 * min(longest, every)


# What a block costs beyond its 64-key steps, what the merge of partial sums costs beyond its traffic
# (both in steps), microseconds a step, and how many multiprocessors a block takes, by prompt kernel;
# from sweeps of the split at Gemma 2 2B head sizes with 2,048 tokens behind 4,096 to 129,024 (a block
# that starts among running ones costs 20 to 27 us before its first and after its last step, twice
# what it costs in a launch of its own). The tcgen05 kernels' steps are short, so their fixed costs
# weigh more and they are cut into slots only when a few tiles face a long history; "tcgen05_pair" is
# the kernel on pairs of blocks (a tile of 256 rows on two multiprocessors, half the time a step). "flash", the kernel without a soft cap, has
# the tcgen05 kernel's fixed costs and half its step, not fitted but measured after: of 48 shapes (128, 512 and 2,048 tokens behind 0 to 30,720, 8 to 32
# heads of 64 and 128, with a window and without) the choice is the fastest split in 42 and within 7 us of it in the others.
PROMPT_KERNEL_COSTS = {"mma": (0.5, 1.0, 4.5, 1), "flash": (18.0, 15.0, 0.6, 1), "tcgen05": (18.0, 15.0, 1.2, 1), "tcgen05_pair": (32.0, 18.0, 0.85, 2)}


def prompt_costs_of(prompt_kernel: str, head_dim: int, pairs: Optional[int] = None) -> str:
    """The entry of PROMPT_KERNEL_COSTS for the kernel that will run prompt portions of this head size."""
    from .. import kernels as K

    if prompt_kernel == "tcgen05" and K.attention_tile_rows(False, prompt_kernel, head_dim, pairs) > 128:
        return "tcgen05_pair"
    return prompt_kernel


def prompt_split(first_counts, last_counts, pairs_per_tile: int, sms: int, window: Optional[int], rows: int, hq: int, d: int,
                 kernel: str = "mma"):
    """(split, slots) of the prompt attention kernel. A tile of a long prompt walks all the keys
    before it, so late tiles work many times longer than early ones; cutting the keys into slots
    of `split` positions evens the blocks out at the price of partial sums that a second kernel
    merges. The choice minimises an estimate of the time: the longest block or the mean load of a
    multiprocessor, whichever is larger, plus the merge, all counted in 64-key steps."""
    block_cost, merge_cost, step_us, sms_a_block = PROMPT_KERNEL_COSTS[kernel]
    sms = max(1, sms // sms_a_block)                     # blocks (or pairs of blocks) that run at once
    first = np.asarray(first_counts, np.int64)
    last = np.asarray(last_counts, np.int64)
    lo = np.maximum(0, first - window) if window else np.zeros_like(first)
    longest = int(last.max()) if last.size else 0
    best = None
    for split in (0, 4096, 2048, 1024, 512, 256, 128):
        if split == 0:
            steps = -(-(last - lo // 64 * 64) // 64)
            work = steps.astype(np.float64)
            slots = 1
            merge = 0.0
        else:
            if split >= longest:
                continue
            slots = -(-longest // split)
            z = np.arange(slots)[None, :]
            a = np.maximum(lo[:, None], z * split)
            b = np.minimum(last[:, None], (z + 1) * split)
            steps = np.where(b > a, -(-(b - a // 64 * 64) // 64), 0)
            work = steps.astype(np.float64).reshape(-1)
            # what the partial sums cost to write and read back (at ~5 TB/s), in steps, plus a launch
            merge = merge_cost + slots * rows * hq * (d + 2) * 8 / 5e12 / (step_us * 1e-6)
        work = work[work > 0] + block_cost               # what it costs to start and finish a block
        if work.size == 0:
            continue
        cost = max(float(work.max()), float(work.sum()) * pairs_per_tile / sms * 1.1) + merge
        if best is None or cost < best[0]:
            best = (cost, split, slots)
    return (best[1], best[2]) if best else (0, 1)


def pooled_slices(rows: int, longest: int, window: Optional[int], pool: int, sms: int, chunk: int):
    """(slices, keys a slice) of the attention kernel over a window and pooled blocks, which runs one
    block a row: with few rows, the keys a row can see (the window's tokens and the blocks below it) are
    cut into slices of a multiple of `chunk` keys so that about two blocks a multiprocessor run."""
    tokens = min(longest, window) if window else longest
    keys = tokens + (max(0, longest - window) // pool if (window and pool) else 0)
    if rows <= 0 or rows >= 2 * sms or keys <= chunk:
        return 1, 0
    want = min(-(-keys // chunk), max(1, (2 * sms) // rows))
    split_keys = -(-(-(-keys // want)) // chunk) * chunk
    slices = -(-keys // split_keys)
    return (slices, split_keys) if slices > 1 else (1, 0)


def cut_tiles(q_start, q_len, tokens_per_tile: int):
    """(tile_entry, tile_row0, tile_nq): each request's rows in runs of at most `tokens_per_tile`."""
    entry, row0, nq = [], [], []
    for e, (start, n) in enumerate(zip(q_start.tolist(), q_len.tolist())):
        for at in range(0, n, tokens_per_tile):
            entry.append(e)
            row0.append(start + at)
            nq.append(min(tokens_per_tile, n - at))
    return np.asarray(entry, np.int32), np.asarray(row0, np.int32), np.asarray(nq, np.int32)


class StepBatch:
    """Device views of a step. `memo` holds what parts share within the step (rotary tables)."""

    def __init__(self, plan: Plan, ids: Sequence[int], want_rows: Sequence[int], device, chunk: int,
                 fixed_slots: Optional[int] = None, into: Optional[torch.Tensor] = None):
        """`into`: a device buffer of a recorded pass of the same shape (the same number of values), to
        be rewritten in place instead of a new one."""
        self.plan = plan
        self.rows = plan.rows
        self.entries = len(plan.entries)
        self.chunk = chunk
        self.fixed_slots = fixed_slots
        self.memo: Dict[object, object] = {}
        self._slots_memo: Dict[Optional[int], int] = {}
        parts: List[np.ndarray] = [
            np.asarray(ids, np.int32), plan.positions, plan.row_entry, plan.row_count,
            np.asarray(want_rows, np.int32), plan.slots,
        ]
        for g in plan.groups:
            parts.append(g.lines)
            parts.append(g.block_table.reshape(-1))
        sizes = [p.size for p in parts]
        total = sum(sizes)
        host = torch.empty((max(total, 1),), dtype=torch.int32, pin_memory=(device.type == "cuda"))
        flat = host.numpy()
        at = 0
        for p in parts:
            flat[at : at + p.size] = p
            at += p.size
        self.h2d_bytes = total * 4
        if into is not None:
            if into.numel() != host.numel():
                raise ValueError(f"a recorded pass of {into.numel()} input values was offered a pass of {host.numel()}")
            into.copy_(host, non_blocking=True)
            dev = into
        else:
            dev = host.to(device, non_blocking=True)
        self.dev = dev
        self.sizes = sizes
        self._host = host                 # keeps the pinned buffer alive until the copy is done
        self._assign(dev, sizes, [g.block_table.shape for g in plan.groups])

    def _assign(self, dev, sizes, table_shapes):
        views, at = [], 0
        for n in sizes:
            views.append(dev[at : at + n])
            at += n
        self.ids, self.positions, self.row_entry, self.row_count, self.want_rows, self.slots = views[:6]
        self.groups = []
        for i, shape in enumerate(table_shapes):
            self.groups.append(GroupBatch(views[6 + 2 * i], views[7 + 2 * i].view(shape)))

    def attention_tiles(self, heads_per_kv: int, kv_heads: int, window: Optional[int] = None, head_dim: int = 256,
                        prompt_kernel: str = "mma", keep_first: int = 0):
        """How the tensor-core attention kernel cuts this step: (decode, (tile_entry, tile_row0,
        tile_nq) on the device, split, slots). `decode` is the most rows (tokens x query heads of a
        kv head) of any request when that is at most 16, which selects the decode kernel, else 0.
        The keys are split across blocks when the tiles alone are too few to fill the GPU;
        `prompt_kernel` names the kernel whose costs decide that for prompt portions. A fifth
        value says whether the slots are counted from each row's first visible key (every
        request brings one token) or from key 0. With `keep_first` (keys that stay visible below
        the window) prompt portions are not cut into slots."""
        key = ("tiles", heads_per_kv, kv_heads, window, head_dim, prompt_kernel, keep_first)
        if key not in self.memo:
            from .. import kernels as K

            plan = self.plan
            pairs = K.prompt_pairs(plan.rows, int(plan.row_count.max()))
            self.pairs = pairs                              # the attention part hands it to the kernel
            costs_of = prompt_costs_of(prompt_kernel, head_dim, pairs)
            most = int(plan.q_len.max()) * heads_per_kv
            decode = most if most <= K.attention_mma_rows(True) else 0      # rows a tile in decode mode, else 0
            per_tile = max(1, K.attention_tile_rows(bool(decode), prompt_kernel, head_dim, pairs) // heads_per_kv)
            arrays = cut_tiles(plan.q_start, plan.q_len, per_tile)
            n = arrays[0].size
            host = torch.from_numpy(np.concatenate(arrays)).pin_memory() if self.ids.is_cuda else torch.from_numpy(np.concatenate(arrays))
            dev = host.to(self.ids.device, non_blocking=True)
            tiles = (dev[:n], dev[n : 2 * n], dev[2 * n :])
            longest = int(plan.row_count.max())
            relative = bool(decode) and int(plan.q_len.max()) == 1
            if decode:
                split, slots = decode_split(n * kv_heads, longest, sm_count(self.ids.device), window, relative)
            elif keep_first and window:
                split, slots = 0, 1
            else:
                firsts = plan.row_count[arrays[1]]
                split, slots = prompt_split(firsts, firsts + arrays[2] - 1, kv_heads, sm_count(self.ids.device), window,
                                            plan.rows, heads_per_kv * kv_heads, head_dim, costs_of)
            self.memo[key] = (decode, tiles, split, slots, relative, host)
        return self.memo[key][:5]

    def mixed_tiles(self, heads_per_kv: int, kv_heads: int, window: Optional[int], head_dim: int, prompt_kernel: str):
        """How a pass of single tokens ahead of prompt portions is cut in two, or None where it is not: (rows of the first part, its
        (decode, tiles, split, slots, relative) as `attention_tiles` gives them for a decoding step, the second part's with rows counted from
        its first). Cut only where the single tokens' tiles, a handful of rows each, would be a wave of their own on the prompt
        kernel, which takes some 20 us a block whatever its rows: 32 single tokens behind 500 to 1,500 positions beside a prompt
        of 2,016, 16 heads over 8 of 256: 194 us a layer as one, 74 and 60 cut in two."""
        key = ("mixed", heads_per_kv, kv_heads, window, head_dim, prompt_kernel)
        if key not in self.memo:
            from .. import kernels as K

            plan = self.plan
            q_len = np.asarray(plan.q_len, np.int64)
            single = int(np.argmax(q_len > 1)) if (q_len > 1).any() else 0        # requests of one token ahead of the first portion
            costs = prompt_costs_of(prompt_kernel, head_dim, K.prompt_pairs(plan.rows, int(plan.row_count.max())))
            few = single == 0 or single * kv_heads * PROMPT_KERNEL_COSTS[costs][3] < sm_count(self.ids.device)
            if few or int(q_len[single:].min()) * heads_per_kv <= K.attention_mma_rows(True) or not self.ids.is_cuda:
                self.memo[key] = None
            else:
                pairs = K.prompt_pairs(plan.rows, int(plan.row_count.max()))
                per_tile = max(1, K.attention_tile_rows(False, prompt_kernel, head_dim, pairs) // heads_per_kv)
                tiles = cut_tiles(plan.q_start[single:], plan.q_len[single:], per_tile)
                every = np.arange(single, dtype=np.int32)
                parts = [every, every, np.ones(single, np.int32), tiles[0] + single, tiles[1] - single, tiles[2]]
                host = torch.from_numpy(np.concatenate([a.astype(np.int32) for a in parts])).pin_memory()
                views = host.to(self.ids.device, non_blocking=True).split([a.size for a in parts])
                views = [v.clone() if v.data_ptr() % 16 else v for v in views]
                first = decode_split(single * kv_heads, int(plan.row_count[:single].max()), sm_count(self.ids.device), window, True)
                firsts = plan.row_count[tiles[1]]
                second = prompt_split(firsts, firsts + tiles[2] - 1, kv_heads, sm_count(self.ids.device), window, plan.rows - single,
                                      heads_per_kv * kv_heads, head_dim, costs)
                self.memo[key] = (single, (heads_per_kv, tuple(views[:3]), *first, True), (0, tuple(views[3:]), *second, False), pairs, host)
        return self.memo[key][:4] if self.memo[key] is not None else None

    def attention_slots(self, window: Optional[int], keep_first: int = 0) -> int:
        """Chunk slots the row-wise attention kernel needs for a layer with this window; with
        `keep_first` the slots of the kept first keys come on top."""
        if window not in self._slots_memo:
            if self.fixed_slots is not None:
                n = self.fixed_slots
                if window:
                    n = min(n, (window - 1) // self.chunk + 2)
            else:
                n = _chunks_touched(self.plan.row_count, window, self.chunk)
            self._slots_memo[window] = max(1, n)
        extra = -(-keep_first // self.chunk) if (window and keep_first) else 0
        return self._slots_memo[window] + extra

    def pooled_slices(self, window: Optional[int], pool: int):
        """How the attention kernel over a window and pooled blocks cuts this step's keys: (slices, keys a slice)."""
        key = ("pooled_slices", window, pool)
        if key not in self.memo:
            from .. import kernels as K

            longest = int(self.plan.row_count.max()) if self.plan.rows else 0
            self.memo[key] = pooled_slices(self.plan.rows, longest, window, pool, sm_count(self.ids.device), K.pooled_attention_chunk())
        return self.memo[key]

    def pooled_tiles(self):
        """(tile_entry, tile_row0, tile_nq) on the device for the tensor-core kernel of the attention over
        a window and pooled blocks: each request's rows in runs of that kernel's tile. None in a step
        where every request brings one token (the kernel that cuts the keys into slices takes those)."""
        key = "pooled_tiles"
        if key not in self.memo:
            from .. import kernels as K

            plan = self.plan
            if not len(plan.q_len) or int(plan.q_len.max()) <= 1 or not self.ids.is_cuda:
                self.memo[key] = None
            else:
                arrays = cut_tiles(plan.q_start, plan.q_len, K.pooled_attention_tile_rows())
                n = arrays[0].size
                host = torch.from_numpy(np.concatenate(arrays)).pin_memory()
                dev = host.to(self.ids.device, non_blocking=True)
                self.memo[key] = (dev[:n], dev[n : 2 * n], dev[2 * n :], host)
        tiles = self.memo[key]
        return tiles[:3] if tiles is not None else None

    def row_tiles(self, heads_per_kv: int, kv_heads: int, head_dim: int, window: Optional[int], positions: Optional[int] = None):
        """(tile_entry, tile_row0, tile_nq) on the device for the 32-bit attention by tiles of ROW_TILE rows (tokens x query heads of a kv
        head), or None where some request brings fewer than ROW_TILE_TOKENS tokens (its tile would hold a few rows and walk all its keys
        alone) or the tiles take longer than row by row (`row_tiles_pay`)."""
        key = ("row_tiles", heads_per_kv, kv_heads, head_dim, window, positions)
        if key not in self.memo:
            plan = self.plan
            arrays = None
            if len(plan.q_len) and self.shortest_portion() >= ROW_TILE_TOKENS and heads_per_kv <= ROW_TILE and self.ids.is_cuda:
                arrays = cut_tiles(plan.q_start, plan.q_len, ROW_TILE // heads_per_kv)
                if not row_tiles_pay(plan.row_count, arrays[1], arrays[2], kv_heads, heads_per_kv, head_dim, window, sm_count(self.ids.device), positions):
                    arrays = None
            if arrays is None:
                self.memo[key] = None
            else:
                n = arrays[0].size
                host = torch.from_numpy(np.concatenate(arrays)).pin_memory()
                dev = host.to(self.ids.device, non_blocking=True)
                self.memo[key] = (dev[:n], dev[n : 2 * n], dev[2 * n :], host)
        tiles = self.memo[key]
        return tiles[:3] if tiles is not None else None

    def latent_tiles(self):
        """How the prompt path of latent attention cuts this step, or None where no request brings enough rows for it: (rows before
        the first such request's, requests before it, the most rows one of those brings, (tile_entry, tile_row0, tile_nq), entry_base,
        entry_length, positions, longest): tiles of 128 rows, counted from the first such request's; where each request's positions begin
        among those laid out densely, and how many it has there (none where it brings few rows). Each begins at a multiple of the positions
        that the kernel reads at a time, so that it reads zeros behind a request's last and nothing of the next request's."""
        key = "latent_tiles"
        if key not in self.memo:
            from .. import kernels as K

            plan = self.plan
            q_len = np.asarray(plan.q_len, np.int64)
            many = q_len >= LATENT_PROMPT_ROWS
            first = int(np.argmax(many)) if many.any() else 0
            lengths = np.where(many, plan.row_count[np.asarray(plan.q_start, np.int64) + np.maximum(q_len, 1) - 1], 0) if q_len.size else q_len
            room = -(-lengths // K.LATENT_KEYS) * K.LATENT_KEYS
            positions = int(room.sum())
            # Requests with few rows have to lie before the others (as the scheduler orders a pass).
            if not many.any() or not many[first:].all() or positions > LATENT_PROMPT_POSITIONS or not self.ids.is_cuda:
                self.memo[key] = None
            else:
                base = np.cumsum(room) - room
                tiles = cut_tiles(plan.q_start[first:], plan.q_len[first:], 128)
                arrays = [tiles[0] + first, tiles[1] - int(plan.q_start[first]), tiles[2], base.astype(np.int32), lengths.astype(np.int32)]
                host = torch.from_numpy(np.concatenate([a.astype(np.int32) for a in arrays])).pin_memory()
                views = host.to(self.ids.device, non_blocking=True).split([a.size for a in arrays])
                self.memo[key] = (int(plan.q_start[first]), first, int(q_len[:first].max()) if first else 0, tuple(v.contiguous() for v in views[:3]), views[3].contiguous(), views[4].contiguous(),
                                  positions, int(lengths.max()), host)
        return self.memo[key][:8] if self.memo[key] is not None else None

    def longest_count(self) -> int:
        """The most positions any row of this step has seen (its own included)."""
        return int(self.plan.row_count.max()) if self.plan.rows else 0

    def longest_portion(self) -> int:
        """The most rows any request brings in this step (what sizes a launch of a block a run of a request's rows)."""
        return int(self.plan.q_len.max()) if len(self.plan.q_len) else 0

    def shortest_portion(self) -> int:
        """The fewest rows any request brings in this step."""
        return int(self.plan.q_len.min()) if len(self.plan.q_len) else 0

    def entry_ranges(self):
        """(start, end) on the device: rows [start[e], end[e]) are request e's. Made once a step."""
        if "entry_ranges" not in self.memo:
            from .. import kernels as K

            self.memo["entry_ranges"] = K.entry_ranges(self.row_entry, self.entries)
        return self.memo["entry_ranges"]
