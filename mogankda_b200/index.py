"""Chunk / segment tables (host logic).

Mirrors what ``prepare_chunk_indices`` / ``prepare_chunk_offsets`` give the reference kernels
(mogan_kda/utils/index.py:93-116): chunks never straddle a sequence and are numbered sequence-major.  On top of
that a sequence can be cut into *segments* of a fixed number of chunks; the serial recurrences then run per segment
and the segments are stitched by the state-combine kernel (the same mechanism carries context parallelism across
GPUs).  The segment length never depends on the sequence length, so a prefix of a sequence is segmented exactly
like the full sequence (bitwise prefix invariance).
"""
import threading
from dataclasses import dataclass, field

import numpy as np
import torch

from ._lib import ENUMS

CHUNK = 64


@dataclass
class Layout:
    B: int
    T: int
    N: int                      # sequences
    NC: int                     # chunks
    NS: int                     # segments
    NG: int                     # groups of segments (= sequences)
    chunk_start: torch.Tensor   # int32 [NC]
    chunk_len: torch.Tensor     # int32 [NC]
    seg_chunk_off: torch.Tensor  # int32 [NS+1]
    grp_seg_off: torch.Tensor   # int32 [N+1]
    seq_chunk_off: torch.Tensor  # int32 [N+1]  (segments == sequences view)
    seg_first: torch.Tensor     # int32 [NS]: sequence id if the segment opens its sequence, else -1
    seg_last: torch.Tensor      # int32 [NS]: sequence id if the segment closes its sequence, else -1
    seg_order: torch.Tensor     # int32 [NS]: the segments, longest first
    segmented: bool
    covers_all: bool            # every token of [0, B*T) belongs to a sequence
    host: dict = field(default_factory=dict)
    tables: torch.Tensor = None  # int32: the eight tables above, one after the other (what the native host path takes)
    dims: tuple = ()            # (NC, NS, N, segmented, covers_all, tokens of the longest sequence,
    #                             chunks of the longest segment, sequences of 1 to MKDA_STEP_MAX_TOKENS tokens)

    @property
    def TT(self):
        return self.B * self.T


def build_tables(B, T, cu, seg_chunks=0):
    """Tables as lists.  ``cu`` is a list of ints or None; ``seg_chunks`` = chunks per segment (0 = no cut)."""
    if cu is None:
        bounds = [(b * T, b * T + T) for b in range(B)]
    else:
        if B != 1:
            raise ValueError("cu_seqlens requires B == 1")
        if len(cu) < 1 or cu[0] != 0 or any(cu[i + 1] < cu[i] for i in range(len(cu) - 1)) or cu[-1] > T:
            raise ValueError("cu_seqlens must start at 0, be non-decreasing and end within T")
        bounds = list(zip(cu[:-1], cu[1:]))
    s, e = np.array(bounds, dtype=np.int64).reshape(-1, 2).T
    N = len(s)
    nc = -(-(e - s) // CHUNK)                                  # chunks per sequence
    seq_off = np.concatenate([[0], np.cumsum(nc)])
    within = np.arange(seq_off[-1]) - np.repeat(seq_off[:-1], nc)          # index of a chunk inside its sequence
    start = np.repeat(s, nc) + within * CHUNK
    length = np.minimum(CHUNK, np.repeat(e, nc) - start)
    step = np.full(N, seg_chunks, dtype=np.int64) if seg_chunks and seg_chunks > 0 else np.maximum(nc, 1)
    ns = np.maximum(-(-nc // step), 1)                         # segments per sequence (an empty sequence keeps one)
    grp_off = np.concatenate([[0], np.cumsum(ns)])
    seq_of = np.repeat(np.arange(N), ns)
    j = np.arange(grp_off[-1]) - grp_off[seq_of]
    seg_end = seq_off[seq_of] + np.minimum((j + 1) * step[seq_of], nc[seq_of])
    seg_off = np.concatenate([[0], seg_end])
    seg_first = np.where(j == 0, seq_of, -1)
    seg_last = np.where(j == ns[seq_of] - 1, seq_of, -1)
    tb = dict(chunk_start=start, chunk_len=length, seq_chunk_off=seq_off, seg_chunk_off=seg_off,
              grp_seg_off=grp_off, seg_first=seg_first, seg_last=seg_last, seg_order=np.argsort(-np.diff(seg_off), kind="stable"))
    return dict({n: t.tolist() for n, t in tb.items()}, N=N, covers_all=int((e - s).sum()) == B * T)


def _sm_count(device=None):
    """SMs of the device the kernels will run on (the library asks the runtime in the same way for its persistent
    grids); 148 (B200) when no device is visible, so that the host logic stays testable on CPU."""
    if torch.cuda.is_available():
        return torch.cuda.get_device_properties(device if device is not None else torch.cuda.current_device()).multi_processor_count
    return 148


def wants_segments(chunks_per_seq, HV, seg_chunks, sm_count=None, cost_ratio=2.5):
    """Segment-parallelism chooser: should sequences be cut into segments of ``seg_chunks`` chunks?

    The serial kernels run one CTA per (sequence or segment, v-head), one chunk step after another.  Uncut, their time is
    set by the longest sequence (critical path) unless there is so much work that the even share of all chunk steps over
    the SMs is longer still.  Cutting spreads the steps evenly but adds the state + transition pre-pass in the forward
    direction and a second pass in the backward direction, about 2.5 x the serial work over a layer step, plus the prefix
    combine.  So: cut when the critical path is longer than 2.5 even shares (``cost_ratio``; 1.25 when the caller allows
    warm-up truncation, which shortens the two extra passes to a few chunks wherever the gate decays).  With few chains the four passes of a
    cut call take a segment each however small the share is, so sequences of up to 1.85 segments (1.2 where truncation is allowed) are left alone.
    The line is older than chains shared by two CTAs, by which uncut calls gained most.  Time uncut / cut now, one sequence x 4, 8, 16, 32, 48 heads: training
    0.90 0.92 0.93 0.94 0.89 at 58 chunks, 0.95 0.96 0.96 0.95 0.92 at 62, 1.03 1.02 1.00 0.92 0.91 at 72, 1.20 1.17 1.11 1.01 0.96 at 90, 1.68 1.51 1.27 0.92
    0.98 at 160; forward only 0.91 0.92 0.93 0.95 1.02 at 58, 0.94 0.95 0.96 0.98 1.05 at 62, 1.03 1.03 1.01 1.00 1.10 at 72, 1.71 1.48 1.43 1.04 1.18 at 160;
    with truncation at 40 chunks 1.03 1.02 1.02 1.00 0.91 and 1.02 1.02 1.02 0.93 1.04.  So up to 70 chunks, and in training with 32 heads and more also
    beyond, the cut costs up to 13 %.  Decided from the
    lengths alone (host), never from data; it plays the role of the reference's intra-card CP decision
    (mogan_kda/ops/gated_delta_rule/chunk/cp/context.py:252-283, cp/autocp/decision.py:54-123)."""
    longest = max(chunks_per_seq, default=0)
    if seg_chunks <= 0 or longest <= seg_chunks:
        return False
    even_share = sum(chunks_per_seq) * HV / (sm_count or _sm_count())
    return longest > max(cost_ratio * even_share, (0.55 + 0.52 * cost_ratio) * seg_chunks)


# Entries: (static key, the cu_seqlens tensor itself, its version counter, layout).  The entry keeps the tensor alive
# and is matched by identity, as the reference's ``tensor_cache`` does (mogan_kda/utils/index.py:33-85): a fresh
# ``cu_seqlens`` that happens to land at the address of a freed one (the caching allocator hands blocks back in that
# way every step) can never hit an old entry, and an in-place edit changes the version.
_cache = []
_CACHE_MAX = 16
_cache_lock = threading.Lock()      # held for list operations only, never for a read-back or an upload


def _cached(key, cu_seqlens, ver):
    with _cache_lock:
        for i in range(len(_cache) - 1, -1, -1):
            k, ref, v, lay = _cache[i]
            if ref is cu_seqlens and v == ver and k == key:
                if i != len(_cache) - 1:
                    _cache.append(_cache.pop(i))          # most recently used last
                return lay
    return None


def get_layout(B, T, cu_seqlens, device, seg_chunks=0, auto_heads=0, cost_ratio=2.5):
    """Device tables, cached on (shape, identity + version of ``cu_seqlens``, segment policy) like the reference's
    ``tensor_cache`` (mogan_kda/utils/index.py:19-90).  A cache miss reads ``cu_seqlens`` back to the host.
    ``auto_heads`` > 0 lets ``wants_segments`` decide, for that many v-heads, whether ``seg_chunks`` is applied."""
    key = (B, T, device, seg_chunks, auto_heads, cost_ratio)
    ver = None if cu_seqlens is None else cu_seqlens._version
    lay = _cached(key, cu_seqlens, ver)
    if lay is not None:
        return lay
    cu = None if cu_seqlens is None else [int(x) for x in cu_seqlens.tolist()]
    lens = [T] * B if cu is None else [e - s for s, e in zip(cu[:-1], cu[1:])]
    if auto_heads > 0:
        if not wants_segments([-(-n // CHUNK) for n in lens], auto_heads, seg_chunks, _sm_count(device) if str(device) != "cpu" else None,
                              cost_ratio):
            seg_chunks = 0
    tb = build_tables(B, T, cu, seg_chunks)
    # one upload for all eight tables, each padded to a multiple of four entries (16 bytes)
    names = ("chunk_start", "chunk_len", "seg_chunk_off", "grp_seg_off", "seq_chunk_off", "seg_first", "seg_last", "seg_order")
    flat, at = [], {}
    for n in names:
        at[n] = (len(flat), len(tb[n]))
        flat += tb[n] + [0] * (-len(tb[n]) % 4)
    tables = torch.tensor(flat or [0], dtype=torch.int32, device=device)
    longest = T if cu is None else max(lens, default=0)
    few = sum(0 < n <= ENUMS["MKDA_STEP_MAX_TOKENS"] for n in lens)
    so = tb["seg_chunk_off"]
    chain = max((b - a for a, b in zip(so[:-1], so[1:])), default=0)
    part = {n: tables[o:o + m] for n, (o, m) in at.items()}
    NC, NS, segmented = len(tb["chunk_start"]), len(tb["seg_first"]), len(tb["seg_first"]) != tb["N"]
    lay = Layout(B=B, T=T, N=tb["N"], NC=NC, NS=NS, NG=tb["N"], segmented=segmented, covers_all=tb["covers_all"], host=tb, tables=tables,
                 dims=(NC, NS, tb["N"], int(segmented), int(tb["covers_all"]), longest, chain, few), **part)
    with _cache_lock:
        if len(_cache) >= _CACHE_MAX:
            _cache.pop(0)
        _cache.append((key, cu_seqlens, ver, lay))
    return lay
