"""What one step needs on the device: the batch's index arrays and scratch.

The reference rebuilds and uploads its index tables layer by layer with
synchronous copies (token/position arrays src/model/gpt2_model.cu:391-392;
token_to_block/offset per layer :214-248; flat block table, offsets and lengths
per layer in decode :544-588: 63 copies per decode step).  Here all of a step's
integers are packed into one pinned buffer and go to the device in one
asynchronous copy; every layer of a cache group reads the same block table.
"""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import Dict, List, Optional, Sequence, Tuple

import numpy as np
import torch

from .. import ops


def _pad4(n: int) -> int:
    return (n + 3) & ~3


@dataclass
class GroupView:
    """Block tables and cache slots of the step's tokens, for one cache group."""

    block_table: torch.Tensor      # int32 [S, max_pages]
    slot_mapping: torch.Tensor     # int32 [T]; page * page_size + offset of every token
    max_pages: int


@dataclass
class StepLayout:
    """Offsets (in int32 elements) of every section of the packed buffer."""

    T: int
    S: int
    R: int
    max_pages: Tuple[int, ...]
    n_tiles: int = 0
    n_tiles_wide: int = 0
    single_runs: Tuple[Tuple[int, int], ...] = ()
    offsets: Dict[str, int] = field(default_factory=dict)
    total: int = 0

    @classmethod
    def make(cls, T: int, S: int, R: int, max_pages: Sequence[int], n_tiles: int = 0,
             n_tiles_wide: int = 0, single_runs: Sequence[Tuple[int, int]] = ()) -> "StepLayout":
        lay = cls(T, S, R, tuple(max_pages), n_tiles, n_tiles_wide, tuple(single_runs))
        off = 0
        for name, n in (("token_ids", T), ("positions", T), ("token_seq", T), ("logit_rows", R),
                        ("state_slots", S), ("cu_q", S + 1), ("q_start", S), ("ctx_len", S),
                        ("attn_tiles", 3 * n_tiles), ("attn_tiles_wide", 3 * n_tiles_wide)):
            lay.offsets[name] = off
            off += _pad4(n)
        for g, mp in enumerate(max_pages):
            lay.offsets[f"slot_mapping.{g}"] = off
            off += _pad4(T)
            lay.offsets[f"block_table.{g}"] = off
            off += _pad4(S * mp)
        lay.total = off
        return lay

    def key(self):
        return (self.T, self.S, self.R, self.max_pages, self.n_tiles, self.n_tiles_wide, self.single_runs)


class Workspace:
    """Scratch tensors by name, allocated once at their largest size.

    ``buf`` returns the first ``rows`` rows of a [max_tokens, cols] buffer, so
    addresses stay the same from step to step (which captured graphs rely on).
    """

    def __init__(self, device, max_tokens: int):
        self.device = device
        self.max_tokens = int(max_tokens)
        self._bufs: Dict[Tuple[str, int, torch.dtype], torch.Tensor] = {}
        self._logits: Optional[torch.Tensor] = None
        self.version = 0       # bumped when a buffer is replaced by a larger one

    def buf(self, name: str, rows: int, cols: int, dtype: torch.dtype) -> torch.Tensor:
        key = (name, cols, dtype)
        t = self._bufs.get(key)
        if t is None or t.shape[0] < rows:
            cap = max(rows, self.max_tokens)
            t = torch.empty((cap, cols), dtype=dtype, device=self.device)
            self._bufs[key] = t
            self.version += 1
        return t[:rows]

    def flat(self, name: str, n: int) -> torch.Tensor:
        """At least ``n`` 32-bit floats, in a buffer that grows by powers of two (sizes that vary from call to call
        replace it rarely)."""
        key = (name, 0, torch.float32)
        t = self._bufs.get(key)
        if t is None or t.numel() < n:
            t = torch.empty(max(1 << (int(n) - 1).bit_length(), 1 << 20), dtype=torch.float32, device=self.device)
            self._bufs[key] = t
            self.version += 1
        return t

    def zeroed(self, name: str, n: int) -> torch.Tensor:
        """``n`` int32 words that are zero when first handed out; kernels that use them as
        counters leave them zero."""
        key = (name, 0, torch.int32)
        t = self._bufs.get(key)
        if t is None or t.numel() < n:
            t = torch.zeros(max(n, 4096), dtype=torch.int32, device=self.device)
            self._bufs[key] = t
            self.version += 1
        return t[:n]

    def logits(self, rows: int, vocab: int) -> torch.Tensor:
        t = self._logits
        if t is None or t.shape[0] < rows or t.shape[1] != vocab:
            cap = 1
            while cap < rows:
                cap *= 2
            t = torch.empty((cap, vocab), dtype=torch.float32, device=self.device)
            self._logits = t
            self.version += 1
        return t[:rows]


class StepContext:
    """Device views of one step's packed integers, plus host-side facts about it."""

    def __init__(self, layout: StepLayout, dev: torch.Tensor, ws: Workspace, *, q_lens: Sequence[int],
                 q_starts: Sequence[int]):
        self.layout = layout
        self.T, self.S, self.R = layout.T, layout.S, layout.R
        self.ws = ws
        o = layout.offsets

        def sec(name, n):
            return dev[o[name]:o[name] + n]

        self.token_ids = sec("token_ids", self.T)
        self.positions = sec("positions", self.T)
        self.token_seq = sec("token_seq", self.T)
        self.logit_rows = sec("logit_rows", self.R)
        self.state_slots = sec("state_slots", self.S)
        self.cu_q = sec("cu_q", self.S + 1)
        self.q_start = sec("q_start", self.S)
        self.ctx_len = sec("ctx_len", self.S)
        # query tiles of the tensor-core attention: (request index, first flat token, rows)
        self.attn_tiles = sec("attn_tiles", 3 * layout.n_tiles)
        self.n_tiles = layout.n_tiles
        # the same tokens cut into tiles of ATTN_TILE_WIDE rows, for the tcgen05 attention
        self.attn_tiles_wide = sec("attn_tiles_wide", 3 * layout.n_tiles_wide)
        self.n_tiles_wide = layout.n_tiles_wide
        # runs (first flat row, rows) of requests that bring one token to a step in which others bring more; where there are
        # any, their tiles stand at the end of both lists
        self.single_runs = layout.single_runs
        self.groups: List[GroupView] = []
        for g, mp in enumerate(layout.max_pages):
            bt = dev[o[f"block_table.{g}"]:o[f"block_table.{g}"] + self.S * mp].view(self.S, mp)
            self.groups.append(GroupView(block_table=bt, slot_mapping=sec(f"slot_mapping.{g}", self.T), max_pages=mp))
        self.set_host_facts(q_lens, q_starts)

    def set_host_facts(self, q_lens: Sequence[int], q_starts: Sequence[int]) -> None:
        """What the host knows about the step (never read back from the device)."""
        self.q_lens = list(q_lens)
        self.q_starts = list(q_starts)
        self.max_q_len = max(self.q_lens) if self.q_lens else 0
        self.max_ctx_len = max((a + b for a, b in zip(self.q_starts, self.q_lens)), default=0)
        self.max_single_ctx_len = max((a + 1 for a, b in zip(self.q_starts, self.q_lens) if b == 1), default=0)
        self.decode_only = self.max_q_len == 1
        # what a layer's arrangement leaves for the next one within the step (a residual write that the next layer's
        # read takes along); nothing is carried from one step to the next
        self.carry = None


ATTN_TILE = 64      # query rows per tile of csrc/attention_flash.cu and attention_tiled.cu
ATTN_TILE_WIDE = 128     # query rows per tile of csrc/attention_tcgen05.cu


MAX_SINGLE_RUNS = 4      # runs of single tokens that a mixed step hands to the decode attention, a launch each


def single_runs(q_lens: Sequence[int]) -> List[Tuple[int, int]]:
    """Runs (first flat row, rows) of neighbouring requests with one new token each; none where there are more than
    MAX_SINGLE_RUNS of them."""
    runs: List[Tuple[int, int]] = []
    base = 0
    for n in q_lens:
        if n == 1:
            if runs and sum(runs[-1]) == base:
                runs[-1] = (runs[-1][0], runs[-1][1] + 1)
            else:
                runs.append((base, 1))
        base += n
    return runs if len(runs) <= MAX_SINGLE_RUNS else []


def singles_pay(q_lens: Sequence[int], q_starts: Sequence[int], heads: int, float32: bool, wide: bool = True,
                window: Optional[int] = None, sms: int = 148) -> bool:
    """Whether the single tokens of a mixed step are worth launches of their own, one per run.

    As a tile of the portions' launch a single token costs little while the launch neither lasts longer for it nor needs
    another wave, and while the bfloat16 portions keep their 128-row tiles (``wide``: a kernel for those takes these heads and
    pages), whose rule wants them mostly full.  Both are estimated in blocks of keys: a tile takes some blocks to start (4 of
    128 keys, 3 of 64) and one per block it walks; a launch takes its longest tile, or all tiles of all heads over the places
    on the GPU (a tile of 128 rows per SM, two of 64).  A block of 128 keys takes 4 us in 32-bit, 1.3 in bfloat16, like one of 64
    there; a launch of its own costs about 4 us.
    Fitted while those launches came after the portions' attention: GPT-2 small, medium and XL, portions of 64 to 1,024 tokens
    beside 1 to 32 single ones in 1 to 4 runs at contexts of 150 to 900, 292 steps, 0.1 % slower than the better of the two (3.6 % at
    most).  They run beside it now, so a run costs less than the rule charges, and the rule has not been fitted again: of 26 steps
    measured so, it picks the slower way in two.  Us a call of the runner, together / apart, * where the rule picks the slower:
      small, bfloat16  512 tokens beside one at 200 707 / 720, at 900 756 / 725, beside 8 at 500 907 / 822 *, beside 32 at 500 1,344 /
                       1,220; 4 x 256 beside 4 runs at 500 859 / 874; 700 beside 6 at 400 965 / 835; 128 beside 4 at 700 781 / 672
      small, 32-bit    512 beside 8 at 500 1,857 / 1,900, beside 16 at 900 2,795 / 2,109; 4 x 256 beside 4 runs 2,633 / 2,558 *
      medium           512 behind 450 beside 40 at 225 to 888, bfloat16 3,190 / 2,777, 32-bit 8,296 / 5,855"""
    ones = [start + 1 for n, start in zip(q_lens, q_starts) if n == 1]
    portions = [(n, start) for n, start in zip(q_lens, q_starts) if n > 1]
    tokens = sum(n for n, _ in portions)
    runs = sum(n == 1 and (i == 0 or q_lens[i - 1] != 1) for i, n in enumerate(q_lens))
    n_wide = sum(-(-n // ATTN_TILE_WIDE) for n, _ in portions)

    def launch(rows, start, places, singles):
        keys = [first + min(n, r + rows) for n, first in portions for r in range(0, n, rows)] + singles
        cost = [start - (-(k if window is None else min(k, window + rows)) // rows) for k in keys]
        return max(max(cost), sum(cost) * heads / places)

    def attention(singles):
        if float32 or (wide and ops.wide_tiles_full(tokens + len(singles), n_wide + len(singles))):
            return launch(ATTN_TILE_WIDE, 4, sms, singles)
        return launch(ATTN_TILE, 3, 2 * sms, singles)

    return attention(ones) - attention([]) > (1 if float32 else 3) * runs


def attention_tiles(q_lens: Sequence[int], q_starts: Optional[Sequence[int]] = None,
                    tile_rows: int = ATTN_TILE, singles_last: bool = False) -> List[int]:
    """Cut every request's new tokens into tiles of at most ``tile_rows`` rows: triples of
    (request index in the batch, flat index of the tile's first token, rows).  With the
    positions at which the portions start, the tiles that see the most keys come first,
    so that the longest walks of the attention kernel start earliest.  ``singles_last``: requests with
    one new token come after all others, so that a launch over the others takes the head of the list."""
    tiles = []
    base = 0
    for s, n in enumerate(q_lens):
        start = 0 if q_starts is None else int(q_starts[s])
        for q0 in range(0, n, tile_rows):
            rows = min(tile_rows, n - q0)
            tiles.append((start + q0 + rows, s, base + q0, rows))
        base += n
    if q_starts is not None:
        tiles.sort(key=lambda t: -t[0])          # stable: equal lengths keep the batch order
    if singles_last:
        tiles.sort(key=lambda t: q_lens[t[1]] == 1)
    out: List[int] = []
    for _, s, t0, rows in tiles:
        out += [s, t0, rows]
    return out


def pack_step(layout: StepLayout, host: np.ndarray, *, token_ids, positions, token_seq, logit_rows, state_slots,
              cu_q, q_start, ctx_len, slot_mappings, block_tables, attn_tiles=(), attn_tiles_wide=()) -> None:
    """Write every section into the int32 array ``host`` (length >= layout.total)."""
    o = layout.offsets

    def put(name, values):
        a = np.asarray(values, dtype=np.int32).reshape(-1)
        host[o[name]:o[name] + a.size] = a

    put("token_ids", token_ids)
    put("positions", positions)
    put("token_seq", token_seq)
    put("logit_rows", logit_rows)
    put("state_slots", state_slots)
    put("cu_q", cu_q)
    put("q_start", q_start)
    put("ctx_len", ctx_len)
    if layout.n_tiles:
        put("attn_tiles", attn_tiles)
    if layout.n_tiles_wide:
        put("attn_tiles_wide", attn_tiles_wide)
    for g, mp in enumerate(layout.max_pages):
        put(f"slot_mapping.{g}", slot_mappings[g])
        bt = np.zeros((layout.S, mp), dtype=np.int32)
        for s, row in enumerate(block_tables[g]):
            n = min(len(row), mp)
            if n:
                r = np.asarray(row[:n], dtype=np.int32)
                bt[s, :n] = np.where(r < 0, 0, r)
        host[o[f"block_table.{g}"]:o[f"block_table.{g}"] + bt.size] = bt.reshape(-1)
