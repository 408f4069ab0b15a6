"""The level driver: ET-Miner's GPU mining loop on one GB300, over the C-ABI library.

Restates the behaviour of ``_apriori_row_split_multi_gpu``
(gpu/row_split.py:229-1185) for one device: K=1 popcounts and the free
items, then level by level the prefix groups of the generating level, the
subset test / count inference, the counting kernels, the survivor
compaction and the free-set test. Every step runs on the device; the host
only plans candidate chunks from the group sizes and reads the totals it
needs to size the next allocation.

Differences from the reference's internals (results are identical):

* The level's itemsets never leave the device between levels: candidates
  are decoded into the next level's rows by the compaction kernel, already in
  lexicographic order, so there is no host decode, lexsort or group build.
* Levels are held in "generator index" space: column ids 0..n_g-1 index the
  engine's padded copy of the generating columns (``fbv``); results map back
  to the caller's columns through ``gen_cols``.

Forms:
    "batched"  one launch per candidate chunk and kernel kind (default)
    "plain"    one counting launch per prefix group: the one-launch-per-group
               comparator the batched form is measured against
"""

from __future__ import annotations

import ctypes
import gc
import math
import threading
import time
import weakref
from dataclasses import dataclass, field
from fractions import Fraction

import numpy as np
import torch

from . import _lib
from ._lib import check, load_library
from .autotune import Autotuner

#: A prefix group with at most this many members is counted from its columns (etm_count_groups), where ``project_pays``
#: does not decide.
SMALL_GROUP = 16
#: Suffixes per tile side of the tile-pair kernel.
TILE = 64
#: Candidates per chunk (int32 count + uint8 class each): bounds the level's dense scratch.
CHUNK_CANDS = 1 << 29
#: A group of more than SMALL_GROUP members is counted on its prefix's rows only when the prefix
#: holds less than this fraction of the transactions.
PROJ_DENSITY = 0.5
#: Device bytes of projected suffix words per chunk (two such sets alternate between the streams).
PROJ_BYTES = 16 << 30
#: Members per block of the tensor-core Gram kernel (e4m3 and f16 operands; packed e2m1 blocks hold 240):
#: a block pair (ua <= ub) is one work item.
TC_TILE = 256
#: Largest group (rows) the tensor-core Gram counts exactly: f32 holds every integer up to 2^24.
TC_MAX_ROWS = 1 << 24
PROJ_SEG_WORDS = 1024  # ETM_PROJ_SEG_WORDS: bitvector words per projection segment
GROUP_TILE = 8  # members per tile side of etm_count_groups
GROUP_SLAB_WORDS = 2048  # words etm_count_groups counts without partial sums
OCC_TILE_WORDS = 32  # ETM_OCC_TILE_WORDS: bitvector words per occupancy tile
#: Row-wise K=2 crossover: rows' pair increments over pairs x words (the reference's K2_ROWS_MAX_R).
K2_ROWS_MAX_R = 3.95e-3
#: Row-wise K=3 crossover: rows' pair increments over K=3 candidates x words, with every candidate in one
#: chunk (the reference's K3_ROWS_MAX_R, gpu/row_split_chunks.py:145-159).
K3_ROWS_MAX_R = 2.5e-4
#: Levels counted by etm_mine_direct: longest itemset (ETM_DIRECT_LEVELS), and the candidate words (candidates x words
#: of a column, projected or not) of a level, past which the general path counts it.
DIRECT_LEVELS = 64
DIRECT_WORDS = 1 << 30
#: Candidate words of a level past K=2 from which a mine that started direct goes on over generators by support, where the
#: columns are worth cutting to the first item: the turn costs some 0.5 ms (7.6e8 words 16.5 -> 7.4 ms with the levels after
#: it; 2.0e8 words, few levels after it, 1.0 -> 1.7).
DIRECT_TURN = 1 << 28
#: Its memory: rows and candidates of a level, and the levels' counts and items of one launch; DIRECT_SCALE times that
#: (4 times the candidates) for columns of DIRECT_LARGE words in all, and DIRECT_MOST times (8 times the candidates) for a
#: mine that such a launch has stopped in for want of it, on columns cut to the first item.
DIRECT_ROWS = 1 << 16
DIRECT_CANDS = 1 << 22
DIRECT_COUNTS_CAP = 1 << 18
DIRECT_ROWS_CAP = 1 << 20
DIRECT_SCALE = 16
DIRECT_MOST = 128
DIRECT_LARGE = 1 << 21
DIRECT_HEADER = 2 * (8 + 4 * (DIRECT_LEVELS + 1))  # 32-bit words
#: Counts and items of its outputs fetched along with the header: all of a small mine's, whose frame is then built on the
#: host. 8,192 itemsets of 4 items take 105 us there and 142 on the device, 16,384 take 205 and 146.
DIRECT_FETCH_COUNTS = 1 << 13
DIRECT_FETCH_ROWS = 1 << 15
#: Words of the columns it projects: none below DIRECT_PROJ_MIN words of columns in all, else at most half of those.
DIRECT_PROJ_MIN = 1 << 18
DIRECT_PROJ_WORDS = 1 << 25
#: Pair words of the K=2 level (pairs x words of a column) from which the generators are numbered by ascending support
#: while the mine counts: those whose K=2 level etm_mine_direct leaves. Above it every measured mine got faster or stayed
#: (3.7e9 pair words 8.7 -> 8.3 ms, 2.8e10 16.6 -> 11.1 ms, 2.6e11 515 -> 278 ms; 1.1e10 of a wide vocabulary 18.2 ->
#: 18.2 ms); below it the mine is direct, bound by launches and barriers, and the levels' reordering would add to them.
ORDER_WORDS = 1 << 30
#: Rows of a level that are put into the columns' order at once; past them, the rows of a piece and those looked over at a
#: time.
ORDER_ROWS = (1 << 31) - 1
ORDER_PIECE = 1 << 27
ORDER_STEP = 1 << 24
#: Counting method for tile-pairs: "popcount" or "tensor".
DEFAULT_METHOD = "tensor"


def min_count(min_support: float, n_rows: int) -> int:
    """ceil(s * N), s read as its shortest round-tripping decimal (core/result.py:57-79)."""
    return math.ceil(Fraction(str(min_support)) * n_rows)


def mining_min_count(min_support: float, n_rows: int) -> int:
    """The threshold the levels apply: ``min_count``, at least 1, as the CPU route does
    (core/cpu_miner.py:967-970); at 0 every pair would be "frequent" with count 0."""
    return max(1, min_count(min_support, n_rows))


def proj_stride(pcnt: np.ndarray, n_words: int) -> np.ndarray:
    """Words per member of a projected group: its prefix rows in whole words, plus up to four padded words
    per segment of PROJ_SEG_WORDS bitvector words (each segment's piece ends on a 4-word chunk), rounded up
    to 32 (at least 32)."""
    n_seg = max(1, -(-int(n_words) // PROJ_SEG_WORDS))
    return np.maximum(32, ((np.asarray(pcnt, np.int64) + 63) // 64 + 4 * n_seg + 31) // 32 * 32)


TC_MXF4 = 4  # ETM_TC_MXF4: packed e2m1 operands under kind::mxf4 (tc_elem code)
TC_WIDE = 16  # ETM_TC_WIDE: accepted in tc_elem and ignored (every code runs the block-pair kernel)
TC_BLOCKED = 32  # ETM_TC_BLOCKED: the Gram reads member rows in the projection's blocked layout
#: Packed e2m1 operands: the fastest exact form measured on GB300 (0.86 s per dense K=2 mine against 1.11 s
#: with e4m3 operands).
DEFAULT_TC_ELEM = TC_MXF4


def tc_block(tc_elem: int = DEFAULT_TC_ELEM) -> int:
    """Members per block of the Gram kernel for an element code: 240 for packed e2m1, else 256."""
    return 240 if (tc_elem & ~TC_WIDE) == TC_MXF4 else TC_TILE


def _tile_items(m: np.ndarray, method: int, tc_elem: int = DEFAULT_TC_ELEM) -> np.ndarray:
    """Work items of groups of m members: 64 x 64 tile-pairs (popcount) or Gram block pairs ua <= ub (tensor)."""
    if method == 1:
        t = tc_block(tc_elem)
        nb = (m + t - 1) // t
        return nb * (nb + 1) // 2
    nt = (m + TILE - 1) // TILE
    return nt * (nt + 1) // 2


#: Fewest stages (256 rows each) of a Gram work item cut from a longer block pair: about 12 us, several times the
#: item's start, its accumulator read and the additions of its counts.
GRAM_MIN_STAGES = 24


def direct_bytes(scale: int, cands: int, n_cols: int, n_words: int, proj_words: int) -> int:
    """Device bytes of the buffers that an engine keeps for direct launches of ``scale`` over such columns."""
    words, proj = ctypes.c_int64(), ctypes.c_int64()
    check(load_library().etm_direct_scratch_words(DIRECT_ROWS * scale, cands, n_cols, n_words, proj_words,
                                                  ctypes.byref(words), ctypes.byref(proj)), "etm_direct_scratch_words")
    out = DIRECT_HEADER + (DIRECT_COUNTS_CAP + DIRECT_ROWS_CAP) * scale
    return 5 * (words.value + proj.value + out) + 256  # with the quarter more that the scratch takes


def direct_scale(n_cols: int, n_words: int) -> int:
    """How many times the smallest levels' memory a direct launch gets, by its columns' size."""
    return DIRECT_SCALE if n_cols * n_words >= DIRECT_LARGE else 1


def direct_cands(scale: int, chunk_cands: int) -> int:
    """Candidates of a level that a direct launch of ``scale`` holds: four times as many as the smallest launch from four
    times its memory on, eight times in the largest, and no more than a chunk of the general path."""
    times = scale if scale < 4 else 4 if scale < DIRECT_MOST else 8
    return max(1, min(DIRECT_CANDS * times, chunk_cands))


def direct_proj(n_cols: int, n_words: int, proj_bytes: int) -> int:
    """Words of columns that a direct launch over such columns may project."""
    total = n_cols * n_words
    return min(total // 2, DIRECT_PROJ_WORDS, proj_bytes // 8) if total >= DIRECT_PROJ_MIN else 0


def direct_need(n_cols: int, n_gen: int, n_words: int, chunk_cands: int, proj_bytes: int) -> int:
    """``direct_bytes`` of all that a mine over such columns and generating columns may launch."""
    proj = direct_proj(n_gen, n_words, proj_bytes)
    scale = DIRECT_MOST if proj else max(direct_scale(n_cols, n_words), direct_scale(n_gen, n_words))
    return direct_bytes(scale, direct_cands(scale, chunk_cands), n_gen, n_words, proj)


def project_pays(m: np.ndarray, prefix_rows: np.ndarray, plen: int, n_words: int, n_cols: int,
                 copied: bool) -> np.ndarray:
    """Whether each group of m members over a prefix of ``plen`` columns and ``prefix_rows`` rows is counted on its prefix's
    rows (projected, then the Gram) rather than from its columns (etm_count_groups).

    In bytes through L2. From the columns: tiles of 8 x 8 members each read their members and the prefix, or count 64
    pairs a word, which takes as long as 3.3 bytes a pair. On the prefix's rows: the prefix is read twice, a row
    brings its words of every column in 16-byte pieces, the members' bits are written and read, and a Gram stage of 256
    rows (0.45 us of one SM) stands for 22 KB, an item's start and end for 250 KB. The row-major copy the projection
    reads is charged to the groups where the mine has not made it yet. Against a fixed line at 16 members (before):
    1M rows of sparse prefixes 18.1 -> 17.1 ms, 400K 11.7 -> 11.2 ms, 20M rows of prefixes of a million rows
    9.6 -> 8.6 ms, where the best fixed lines would be 8, 12 and 24.
    """
    m, rows = np.asarray(m, np.float64), np.asarray(prefix_rows, np.float64)
    nb = np.ceil(m / GROUP_TILE)
    last = m - (nb - 1) * GROUP_TILE
    # Members read by the tiles: a triangle reads its block, a pair of blocks both.
    members = (nb - 1) * GROUP_TILE + last + (nb * (nb - 1) / 2) * GROUP_TILE + (
        (nb - 1) * (nb - 2) / 2 * GROUP_TILE + (nb - 1) * last)
    columns = n_words * np.maximum(8 * (members + plen * nb * (nb + 1) / 2), 3.3 * m * (m - 1) / 2)
    blocks = np.ceil(m / 240)
    pairs = blocks * (blocks + 1) / 2
    projected = (16.0 * plen * n_words + rows * (16 * -(-n_cols // 128) + m / 4) +
                 pairs * (22e3 / 256 * rows + 250e3))
    pays = projected < columns
    if not copied and pays.any() and (columns - projected)[pays].sum() < 2.5 * 8 * n_cols * n_words:
        pays[:] = False
    return pays


def gram_parts(pairs: np.ndarray, stages: np.ndarray, sms: int) -> np.ndarray:
    """Parts into which the block pairs of each work entry are cut along their rows: ``pairs`` block pairs of
    ``stages`` stages each on ``sms`` CTAs.

    A pair is cut where it would keep its CTA busy after the others are done, that is where it takes more than half
    of the level's stages per SM, into items of a quarter of those (or GRAM_MIN_STAGES). A level of many pairs stays
    whole: its counts are then thresholded as they leave the accumulators, without a pass over every candidate. A
    part holds at most TC_MAX_ROWS rows (exact sums in f32).
    """
    pairs, stages = np.asarray(pairs, np.int64), np.asarray(stages, np.int64)
    most = max(1, TC_MAX_ROWS // 256)
    total = int((pairs * stages).sum())
    per = np.int64(most)
    if stages.size and 2 * sms * int(stages.max()) > total:
        per = min(per, max(GRAM_MIN_STAGES, -(-total // (4 * sms))))
    return np.maximum(1, -(-stages // per))


def _p(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _allocated_gb(device: torch.device) -> float:
    """Device memory allocated through torch, in GB (``torch.cuda.memory_allocated`` without its flattened copy of every
    statistic, which takes 0.15 ms a call)."""
    stats = torch.cuda.memory_stats_as_nested_dict(device)
    return (stats["allocated_bytes"]["all"]["current"] if stats else 0) / (1 << 30)


@dataclass
class Level:
    """One level on the device: rows int32 [n, k] in generator-index space, counts int32 [n], free flags."""

    rows: torch.Tensor
    counts: torch.Tensor
    free: torch.Tensor | None = None
    #: The counts are the rows' supports in the mine's columns, counted by it: block pairs may be bounded by them.
    counted: bool = False

    @property
    def n(self) -> int:
        return int(self.rows.shape[0])

    @property
    def k(self) -> int:
        return int(self.rows.shape[1])


@dataclass
class LevelStats:
    k: int
    n_candidates: int
    n_frequent: int
    ms: float
    n_groups: int = 0
    n_chunks: int = 0
    launches: int = 0
    row_wise: bool = False  # counted from the transactions (row-wise K=2 / K=3 kernels)
    n_inferred: int = 0  # candidates whose count the subset test or the deduction bounds settled (class_stats)
    n_skipped: int = 0  # candidates the subset test or the bounds showed infrequent (class_stats)


@dataclass
class MineOutput:
    """Emitted levels (device tensors in generator-index space) and how to map them back.

    ``gen_cols[g]`` is the caller's column of generator index g. Level 1 is
    held as the caller's columns directly (``level1_cols``) because under the
    free-set prune it differs from the generators only by nothing, and in a
    complete run every frequent column is both.
    """

    n_rows: int
    min_count: int
    gen_cols: np.ndarray
    level1_cols: np.ndarray
    level1_counts: np.ndarray
    levels: list[Level] = field(default_factory=list)
    stats: list[LevelStats] = field(default_factory=list)
    #: (rows, counts) of levels 2 .. one after another on the host, when one direct launch mined them all and they came
    #: back with its header: the frame of a small result is built from them without further device work.
    host: tuple[np.ndarray, np.ndarray] | None = None

    def host_levels(self) -> list[tuple[np.ndarray, np.ndarray]]:
        """Every emitted level as (caller column ids int64 [n, k], counts int64 [n]) on the host."""
        out = []
        if len(self.level1_cols):
            out.append((self.level1_cols[:, None].astype(np.int64), self.level1_counts.astype(np.int64)))
        for lv in self.levels:
            if lv.n == 0:
                continue
            rows = lv.rows.cpu().numpy()
            out.append((self.gen_cols[rows].astype(np.int64), lv.counts.cpu().numpy().astype(np.int64)))
        return out

    def n_itemsets(self) -> int:
        return len(self.level1_cols) + sum(lv.n for lv in self.levels)

    def frame_arrays(self, item_of_col: np.ndarray) -> tuple[np.ndarray, np.ndarray, np.ndarray, int]:
        """The result as flat arrays, built on the device and copied back once: (offsets int64 [n + 1],
        item ids [offsets[-1]] (int64, or uint64 when ``item_of_col`` is), support float64 [n]) for
        every emitted itemset in level order, and the bytes copied device to host.

        ``item_of_col[c]`` is the item id of the caller's column c.
        """
        wide = item_of_col.dtype == np.uint64

        def as_i64(a: np.ndarray) -> np.ndarray:
            a = np.ascontiguousarray(a)
            return a.view(np.int64) if wide else a.astype(np.int64)

        n1 = len(self.level1_cols)
        lv_on = [lv for lv in self.levels if lv.n > 0]
        if not lv_on:
            values = as_i64(item_of_col[self.level1_cols])
            offsets = np.arange(n1 + 1, dtype=np.int64)
            support = self.level1_counts.astype(np.float64) / max(1, self.n_rows)
            return offsets, values.view(np.uint64) if wide else values, support, 0
        if self.host is not None:
            table = item_of_col[self.gen_cols]
            rows, counts = self.host
            values = np.concatenate([as_i64(item_of_col[self.level1_cols]), as_i64(table[rows])])
            offsets = np.zeros(n1 + len(counts) + 1, np.int64)
            np.cumsum(np.concatenate([np.ones(n1, np.int64), *(np.full(lv.n, lv.k) for lv in lv_on)]), out=offsets[1:])
            support = np.concatenate([self.level1_counts, counts]).astype(np.float64) / max(1, self.n_rows)
            return offsets, values.view(np.uint64) if wide else values, support, 0
        dev = lv_on[0].rows.device
        ng, n = len(self.gen_cols), n1 + sum(lv.n for lv in lv_on)
        n_values = n1 + sum(lv.k * lv.n for lv in lv_on)
        # The generators' items, level 1's items and its counts (int32), in one copy.
        host = np.zeros(ng + n1 + (n1 + 1) // 2, np.int64)
        host[:ng] = as_i64(item_of_col[self.gen_cols])
        host[ng:ng + n1] = as_i64(item_of_col[self.level1_cols])
        host[ng + n1:].view(np.int32)[:n1] = self.level1_counts
        given = torch.from_numpy(host).pin_memory().to(dev, non_blocking=True)
        frame = torch.empty(n_values + 2 * n + 1, dtype=torch.int64, device=dev)
        values_d, offsets_d = frame[:n_values], frame[n_values:n_values + n + 1]
        support_d = frame[n_values + n + 1:].view(torch.float64)
        lib, stream = load_library(), torch.cuda.current_stream(dev).cuda_stream
        parts = [(None, _p(given[ng + n1:]), n1, 1, _p(given[ng:]))]
        parts += [(_p(lv.rows), _p(lv.counts), lv.n, lv.k, _p(given)) for lv in lv_on]
        row0 = value0 = 0
        for rows_p, counts_p, m, k, table_p in parts:
            check(lib.etm_frame_level(rows_p, counts_p, m, k, table_p, max(1, self.n_rows), row0, value0, _p(values_d),
                                      _p(offsets_d), _p(support_d), stream), "etm_frame_level")
            row0, value0 = row0 + m, value0 + m * k
        if frame.numel() * 8 < PINNED_MEDIUM_BYTES:
            host = frame.cpu().numpy()
            values, offsets = host[:n_values], host[n_values:n_values + n + 1]
            support = host[n_values + n + 1:].view(np.float64)
        else:
            values, support, offsets = _copy_to_host(values_d, support_d, offsets_d)
        d2h = values.nbytes + support.nbytes + offsets.nbytes
        return offsets, values.view(np.uint64) if wide else values, support, d2h


#: Results at least this large come back through page-locked host memory.
PINNED_RESULT_BYTES = 64 << 20
#: Results from this size on do where a page-locked buffer is at hand or there is room for another of theirs (a quarter of
#: the time of a pageable copy at 40 MB); they take at most PINNED_MEDIUM_BUFFERS buffers and collect no garbage for one.
PINNED_MEDIUM_BYTES = 4 << 20
PINNED_MEDIUM_BUFFERS = 2


class _PinnedPool:
    """Page-locked host buffers for results, shared by the engines of the process. A buffer is handed out again
    only once every numpy array made from it has been dropped (weak references), so a result never shares
    memory with a live earlier result, and steady-state calls pin nothing new; at most ``max_buffers`` are
    kept (past that, results come back through pageable memory)."""

    def __init__(self, max_buffers: int = 4):
        self.lock = threading.Lock()
        self.entries: list[list] = []  # [uint8 page-locked tensor, [weak references or a busy marker]]
        self.medium: list[list] = []   # the same for results below PINNED_RESULT_BYTES
        self.max_buffers = max_buffers

    @staticmethod
    def _free(entry) -> bool:
        return all(r() is None for r in entry[1])

    def arrays(self, tensors: list[torch.Tensor], large: bool = True) -> list[np.ndarray] | None:
        """Host arrays of the tensors, or None. A result that is not ``large`` takes a buffer of its own kind only."""
        sizes = [t.numel() * t.element_size() for t in tensors]
        offs, total = [], 0
        for n in sizes:
            offs.append(total)
            total += -(-n // 256) * 256
        if large:
            with self.lock:
                have = any(e[0].numel() >= total and self._free(e) for e in self.entries)
                busy = bool(self.entries)
            if not have and busy:
                # A dropped result held in a reference cycle is freed only by the collector: collect once (outside
                # the lock: finalizers may run) before pinning another buffer, which takes longer than a collection.
                gc.collect()
        with self.lock:
            entries = self.entries if large else self.medium
            entry = next((e for e in entries if e[0].numel() >= total and self._free(e)), None)
            if entry is None:
                if len(entries) >= (self.max_buffers if large else PINNED_MEDIUM_BUFFERS):
                    free = [e for e in entries if self._free(e)]
                    if not free:
                        return None
                    entries[:] = [e for e in entries if e is not free[0]]
                entry = [torch.empty(total, dtype=torch.uint8, pin_memory=True), []]
                entries.append(entry)
            entry[1] = [lambda: True]  # busy while the copies run
        buf = entry[0]
        views = [buf[o:o + n].view(t.dtype).view(t.shape) for o, n, t in zip(offs, sizes, tensors)]
        for v, t in zip(views, tensors):
            v.copy_(t, non_blocking=True)
        torch.cuda.current_stream().synchronize()
        out = [v.numpy() for v in views]
        with self.lock:
            entry[1] = [weakref.ref(a) for a in out]
        return out


_PINNED = _PinnedPool()


def _copy_to_host(*tensors: torch.Tensor) -> list[np.ndarray]:
    """Device tensors as host numpy arrays: large results through the page-locked pool (full-rate copies, no
    page faults on fresh memory), small ones (or with the pool exhausted) through ``.cpu()``."""
    nbytes = sum(t.numel() * t.element_size() for t in tensors)
    if nbytes >= min(PINNED_RESULT_BYTES, PINNED_MEDIUM_BYTES):
        got = _PINNED.arrays(list(tensors), nbytes >= PINNED_RESULT_BYTES)
        if got is not None:
            return got
    return [t.cpu().numpy() for t in tensors]


class _Scratch:
    """Reusable device buffers, grown on demand (torch allocations: plumbing only)."""

    def __init__(self, device: torch.device):
        self.device = device
        self.bufs: dict[str, torch.Tensor] = {}

    def get(self, name: str, n: int, dtype: torch.dtype) -> torch.Tensor:
        t = self.bufs.get(name)
        n = max(int(n), 1)
        if t is None or t.dtype != dtype or t.numel() < n:
            t = torch.empty(int(n * 1.25) + 16, dtype=dtype, device=self.device)
            self.bufs[name] = t
        return t[:n]


def host_rss_gb() -> float:
    """Resident set size of this process in GB (/proc/self/status; 0 where it cannot be read)."""
    try:
        with open("/proc/self/status") as f:
            for line in f:
                if line.startswith("VmRSS:"):
                    return int(line.split()[1]) / (1 << 20)
    except OSError:
        pass
    return 0.0


def check_memory_guard(k: int, ram_gb: float, vram_gb: float, max_ram_gb: float | None,
                       max_vram_gb: float | None) -> None:
    """Raise MemoryError when a level left the process over a memory limit (gpu/row_split.py:467-487): the
    lattice is incomplete at that point, so it is not returned."""
    for used, limit, what, remedy in (
        (ram_gb, max_ram_gb, "RAM", "lower max_length or mine fewer levels per call"),
        (vram_gb, max_vram_gb, "VRAM", "lower max_length, or lower the engine's chunk and projection budgets"),
    ):
        if limit is not None and used > limit:
            raise MemoryError(
                f"Memory guard tripped after K={k}: {what}={used:.1f}GB exceeds max_{what.lower()}_gb={limit}GB. "
                f"The lattice is INCOMPLETE at this point, so it is not returned. Raise max_{what.lower()}_gb, "
                f"or {remedy}.")


def scan_words(n: int) -> int:
    return (max(n, 1) + 4095) // 4096 + 2


def as_device_bitvecs(bitvecs) -> tuple[int, tuple[int, int], object]:
    """(device pointer, (n_cols, n_words), owner) of a C-contiguous uint64 device array.

    Accepts a torch CUDA tensor (uint64 or int64) or any object exposing
    ``__cuda_array_interface__`` with typestr ``<u8``.
    """
    if isinstance(bitvecs, torch.Tensor):
        if not bitvecs.is_cuda:
            raise TypeError("bitvecs must live on a CUDA device")
        if bitvecs.dtype not in (torch.uint64, torch.int64):
            raise ValueError(f"bitvecs must be uint64, got {bitvecs.dtype}")
        if bitvecs.dim() != 2 or not bitvecs.is_contiguous():
            raise ValueError("bitvecs must be a C-contiguous 2-D array")
        return bitvecs.data_ptr(), (int(bitvecs.shape[0]), int(bitvecs.shape[1])), bitvecs
    cai = getattr(bitvecs, "__cuda_array_interface__", None)
    if cai is None:
        raise TypeError(f"bitvecs must expose __cuda_array_interface__, got {type(bitvecs).__name__}")
    shape = tuple(cai["shape"])
    if len(shape) != 2:
        raise ValueError(f"bitvecs must be 2D (n_cols, n_u64s), got {len(shape)}D")
    if cai["typestr"] not in ("<u8", "|u8"):
        raise ValueError(f"bitvecs must be uint64, got {cai['typestr']}")
    strides = cai.get("strides")
    if strides is not None and tuple(strides) != (shape[1] * 8, 8):
        raise ValueError("bitvecs must be C-contiguous")
    return int(cai["data"][0]), (int(shape[0]), int(shape[1])), bitvecs


class Engine:
    """One device's mining state: the library, scratch buffers and the counting choices."""

    def __init__(self, device: torch.device | int | None = None, *, method: str = DEFAULT_METHOD,
                 form: str = "batched", chunk_cands: int = CHUNK_CANDS, small_group: int = SMALL_GROUP,
                 project: bool = True, proj_density: float = PROJ_DENSITY, proj_bytes: int = PROJ_BYTES,
                 tc_elem: int = DEFAULT_TC_ELEM, pipeline: bool = True, autotune: "Autotuner | bool | None" = None,
                 fused: bool = True, deduction_bounds: bool = True, proj_rows: bool = True):
        if not torch.cuda.is_available():
            raise RuntimeError("the GB300 engine needs a CUDA device; there is no CPU fallback")
        self.lib = load_library()
        self.device = torch.device("cuda", torch.cuda.current_device() if device is None else
                                   (device.index if isinstance(device, torch.device) else int(device)))
        if method not in ("popcount", "tensor"):
            raise ValueError(f"method must be 'popcount' or 'tensor', got {method!r}")
        if form not in ("batched", "plain"):
            raise ValueError(f"form must be 'batched' or 'plain', got {form!r}")
        self.method = method
        self.form = form
        self.chunk_cands = int(chunk_cands)
        self.small_group = int(small_group)
        self.project = bool(project)
        self.proj_density = float(proj_density)
        self.proj_bytes = int(proj_bytes)
        #: Tensor-core operand element: 1 = e4m3 (kind::f8f6f4), 2 = f16 (kind::f16), 4 = packed e2m1 (kind::mxf4).
        if (int(tc_elem) & ~TC_WIDE) not in (1, 2, TC_MXF4):
            raise ValueError(f"tc_elem must be 1 (e4m3), 2 (f16) or 4 (e2m1), optionally | 16; got {tc_elem}")
        self.tc_elem = int(tc_elem)
        #: Batched form with the column projection (proj_rows=False): project chunk c+1 on a side stream while
        #: chunk c is counted.
        self.pipeline = bool(pipeline)
        #: Fused threshold: the counting kernels write only the counts reaching min_count and a survivor bit each;
        #: compaction scans the bitmask (a 32nd of the dense counts). False: dense counts, dense compaction.
        self.fused = bool(fused)
        #: Under count inference, settle candidates by the deduction bounds of depth <= 3 from levels k-2 and
        #: k-3 (on by default in the reference's GPU route, gpu/row_split.py:541-546, 629); needs fused.
        self.deduction_bounds = bool(deduction_bounds)
        #: Projection from a row-major copy of the generating columns (etm_project_rows, 32 x 32 bit transposes
        #: over the prefix rows) instead of gathering every member's segment words (etm_project); the copy is
        #: built once per mine and skipped when it would exceed ``rows_copy_max_bytes``.
        self.proj_rows = bool(proj_rows)
        #: Row order of the bitvectors that ``apriori(transactions, ...)`` builds for this engine: "keep" (input
        #: order) or "lex" (the rows sorted by their most frequent columns, with the tile-occupancy skip; the
        #: reference's choice). Counts never depend on it. Measured on the deep sparse transactions (2M rows),
        #: lex halves the per-candidate counting but gathers each prefix's rows into few projection segments,
        #: whose units then run unbalanced, and its levels do not go through the direct launch: 4.3 against 14.9 ms
        #: per call, so the input order is the default.
        self.row_order = "keep"
        #: Under "lex", fewer rows than this keep their order: a few tiles per column leave the occupancy little
        #: to skip, and the keys, sorts and permutation would cost more than they save.
        self.lex_min_rows = 1 << 18
        self.rows_copy_max_bytes = 32 << 30
        self._xt = None
        self._xt_key = None
        #: (occupancy, words per column) of the mine's generating columns, when it asked for one.
        self._occ = None
        #: (level k-2, level k-3 or None, N) of the level being counted, for the deduction bounds.
        self._deep = None
        #: The level of the prefixes of the level being counted (two below it), when the mine has it.
        self._prefix_level = None
        #: When set, each level's stats count the candidates classified INFER and SKIP (one extra pass per chunk).
        self.class_stats = False
        #: K=2 counts row-wise from the transactions (when given) while
        #: sum C(len,2) / (pairs x words) is below this (gpu/row_split_chunks.py:130-142); 0 disables.
        self.k2_rows_max_r = K2_ROWS_MAX_R
        self.k3_rows_max_r = K3_ROWS_MAX_R
        self._k2_rows = None
        self._rows_input = None
        #: Small levels go through etm_mine_direct (one launch for as many as follow one another) where the engine has
        #: its default form; False: every level takes the general path.
        self.direct = True
        #: A block pair of the Gram stops once none of its candidates can be frequent; False: every one runs to its last
        #: row, for the rate of the work.
        self.early_stop = True
        #: Device bytes that the direct launches' buffers may take (None: as many as the mine's own limit leaves). Below
        #: what a large launch needs the engine takes small ones, below that the general path.
        self.direct_max_bytes: int | None = None
        #: Number the generators by ascending support while counting (larger mines in the engine's default form): a
        #: candidate's prefix is then its rarest items, which holds the fewest rows. False: the columns' order.
        self.by_support = True
        self._fetched: torch.Tensor | None = None  # page-locked: the start of a direct launch's outputs
        #: Counting settings chosen per level shape by timing (None: the fixed defaults).
        self.autotuner = Autotuner() if autotune is True else (autotune or None)
        self.scratch = _Scratch(self.device)
        self.launches = 0
        #: When set, every counting / compaction launch is bracketed by CUDA events on its stream.
        self.profile_kernels = False
        self._events: list[tuple] = []
        self.used_tensor = False
        #: Set when a kernel with bounded device waits (the Gram, the projection) ran since the last status read.
        self._waits_pending = False
        self._side: torch.cuda.Stream | None = None

    def _sms(self) -> int:
        if getattr(self, "_sm_count", None) is None:
            self._sm_count = max(1, int(self.lib.etm_device_sm_count()))
        return self._sm_count

    def _side_stream(self) -> torch.cuda.Stream:
        """The stream projection runs on beside the counting kernels (created on first use)."""
        if self._side is None:
            self._side = torch.cuda.Stream(device=self.device)
        return self._side

    # -- kernel timing ----------------------------------------------------------
    def _launch(self, name: str, nbytes: int, fn, flops: float = 0.0):
        """Run ``fn`` (one library call), timing it with CUDA events when profiling."""
        if not self.profile_kernels:
            return fn()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        st = fn()
        e1.record()
        self._events.append((name, e0, e1, int(nbytes), float(flops)))
        return st

    def reset_kernel_times(self) -> None:
        self._events = []

    def kernel_report(self) -> dict:
        """Per kernel: launches, total ms (CUDA events on the launching stream), algorithmic bytes and operations (of the
        Gram every pair over every row, also where a block pair stopped early)."""
        torch.cuda.synchronize()
        out: dict[str, dict] = {}
        for name, e0, e1, nbytes, flops in self._events:
            r = out.setdefault(name, {"name": name, "launches": 0, "ms": 0.0, "bytes": 0, "flops": 0.0})
            r["launches"] += 1
            r["ms"] += e0.elapsed_time(e1)
            r["bytes"] += nbytes
            r["flops"] += flops
        for r in out.values():
            r["gbs"] = r["bytes"] / (r["ms"] / 1e3) / 1e9 if r["ms"] > 0 else 0.0
            r["tflops"] = r["flops"] / (r["ms"] / 1e3) / 1e12 if r["ms"] > 0 else 0.0
        return out

    # -- K = 1 -----------------------------------------------------------------
    def _column_counts(self, ptr: int, n_cols: int, n_words: int, ld: int) -> torch.Tensor:
        out = self.scratch.get("colcounts", n_cols, torch.int64)
        check(self.lib.etm_popcount_cols(ptr, n_cols, n_words, ld, _p(out), _stream()), "etm_popcount_cols")
        self.launches += 1
        return out

    def column_counts(self, ptr: int, n_cols: int, n_words: int, ld: int) -> np.ndarray:
        return self._column_counts(ptr, n_cols, n_words, ld).cpu().numpy().copy()

    def gather(self, ptr: int, ld: int, cols: np.ndarray, n_words: int,
               cols_d: torch.Tensor | None = None) -> tuple[torch.Tensor, int]:
        """The listed columns (``cols_d``: int32 on the device, if it is there) one after another, padded."""
        ldp = max(32, (n_words + 31) // 32 * 32)
        fbv = torch.empty((max(len(cols), 1), ldp), dtype=torch.int64, device=self.device)
        if cols_d is None:
            cols_d = torch.from_numpy(cols.astype(np.int32)).to(self.device)
        check(self.lib.etm_gather_cols(ptr, ld, _p(cols_d), len(cols), n_words, _p(fbv), ldp, _stream()),
              "etm_gather_cols")
        self.launches += 1
        return fbv, ldp

    # -- K >= 2 ----------------------------------------------------------------
    def groups(self, gen: Level):
        n, width = gen.n, gen.k
        grp_first = self.scratch.get("grp_first", n, torch.int64)
        grp_size = self.scratch.get("grp_size", n, torch.int32)
        cand_off = self.scratch.get("cand_off", n + 1, torch.int64)
        counters = self.scratch.get("counters", 2, torch.int64)
        ws = self.scratch.get("ws_groups", 3 + scan_words(n), torch.int64)
        check(self.lib.etm_level_groups(_p(gen.rows), n, width, _p(grp_first), _p(grp_size), _p(cand_off),
                                        _p(counters), _p(ws), ws.numel(), _stream()), "etm_level_groups")
        self.launches += 10
        G, total = (int(x) for x in counters.cpu().tolist())
        return G, total, grp_first, grp_size, cand_off

    def _to_device(self, host: np.ndarray) -> torch.Tensor:
        """A work list on the device, in stream order. Through page-locked memory: a pageable copy of any size waits here
        for the work before it on the stream (the copy engine reads the pages in place), the whole of a level's first
        kernels, 0.3 ms a list."""
        return torch.from_numpy(host).pin_memory().to(self.device, non_blocking=True)

    def _work(self, ids: np.ndarray, weights: np.ndarray) -> tuple[torch.Tensor, torch.Tensor]:
        off = np.zeros(len(ids) + 1, dtype=np.int64)
        np.cumsum(weights, out=off[1:])
        both = torch.from_numpy(np.concatenate([ids.astype(np.int64), off])).to(self.device, non_blocking=False)
        return both[: len(ids)], both[len(ids):]

    def prefix_counts(self, fbv, ldp: int, n_words: int, gen: Level, grp_first, ids: np.ndarray) -> np.ndarray:
        """Rows holding each listed group's prefix (popcount of the AND of its prefix columns)."""
        wg = torch.from_numpy(ids.astype(np.int64)).to(self.device)
        out = self.scratch.get("prefix_counts", len(ids), torch.int64)
        st = self._launch("prefix_counts", len(ids) * (gen.k - 1) * n_words * 8, lambda: self.lib.etm_prefix_counts(
            _p(fbv), ldp, n_words, _p(gen.rows), gen.k, _p(grp_first), _p(wg), len(ids), _p(out), *self._occ_args(),
            _stream()))
        check(st, "etm_prefix_counts")
        self.launches += 1
        return out.cpu().numpy().copy()

    def _prefix_support(self, gen: Level, grp_first, G: int) -> np.ndarray | None:
        """The support of every group's prefix from the level the mine counted it in (etm_prefix_lookup), or None where
        that level is not at hand: then the rows are counted (``prefix_counts``)."""
        prev = self._prefix_level
        if prev is None or not prev.counted or prev.k != gen.k - 1:
            return None
        out = self.scratch.get("prefix_counts", G, torch.int64)
        st = self._launch("prefix_lookup", G * (gen.k * 4 + 16), lambda: self.lib.etm_prefix_lookup(
            _p(gen.rows), gen.k, _p(grp_first), G, _p(prev.rows), _p(prev.counts), prev.n, _p(out), _stream()))
        check(st, "etm_prefix_lookup")
        self.launches += 1
        known = out.cpu().numpy().copy()
        return None if (known < 0).any() else known

    def tile_occupancy(self, fbv: torch.Tensor, ldp: int, n_words: int) -> tuple[torch.Tensor, int]:
        """(occ int64 [n_cols][occ_ld], occ_ld): per generating column, one bit per tile of ETM_OCC_TILE_WORDS
        words holding a row of it (etm_tile_occupancy; gpu/kernels/occupancy.py:37-58)."""
        n_g = int(fbv.shape[0])
        occ_ld = max(1, -(-(-(-n_words // OCC_TILE_WORDS)) // 64))
        occ = torch.empty((n_g, occ_ld), dtype=torch.int64, device=self.device)
        st = self._launch("tile_occupancy", n_g * (n_words + occ_ld) * 8, lambda: self.lib.etm_tile_occupancy(
            _p(fbv), n_g, n_words, ldp, _p(occ), occ_ld, _stream()))
        check(st, "etm_tile_occupancy")
        self.launches += 1
        return occ, occ_ld

    def _occ_args(self) -> tuple:
        """The (occ, occ_ld) arguments of the prefix and per-candidate kernels: the mine's tile occupancy, or none."""
        return (None, 0) if self._occ is None else (_p(self._occ[0]), self._occ[1])

    def _rows_copy(self, fbv: torch.Tensor, ldp: int, n_words: int):
        """(xt, ldr): the row-major copy of the mine's generating columns that etm_project_rows reads (word c of
        row r holds bit r of columns 32 c .. 32 c + 31), built on the current stream at its first use in a mine;
        None when it would exceed ``rows_copy_max_bytes``."""
        n_g = int(fbv.shape[0])
        key = (fbv.data_ptr(), n_words, n_g)
        if self._xt_key == key:
            return self._xt
        ldr = max(4, -(-(-(-n_g // 32)) // 4) * 4)
        nbytes = n_words * 64 * ldr * 4
        self._xt, self._xt_key = None, key
        if nbytes > self.rows_copy_max_bytes:
            return None
        xt = torch.empty((n_words * 64, ldr), dtype=torch.int32, device=self.device)
        st = self._launch("rows_transpose", n_g * n_words * 8 + nbytes, lambda: self.lib.etm_rows_transpose(
            _p(fbv), ldp, n_words, n_g, _p(xt), ldr, _stream()))
        check(st, "etm_rows_transpose")
        self.launches += 1
        self._xt = (xt, ldr)
        return self._xt

    def _prep_projected(self, fbv, ldp, n_words, gen, grp_first, grp_size, gids, sizes, pcnt, method, buf: int = 0,
                        xt=None):
        """Segment offsets and projected member words of the listed groups (two launches on the current stream).

        Returns what ``_count_prepped`` needs. ``buf`` selects one of two scratch sets, so the
        projection of the next chunk can run while the current one is counted. ``xt``: the row-major copy
        (``_rows_copy``) for the row-major projection, else the column form runs.
        """
        width = gen.k
        # Longest prefixes first: the Gram's CTAs claim block pairs in this order, so the last ones are short.
        gids = gids[np.argsort(-pcnt[gids], kind="stable")]
        m = sizes[gids]
        cnt = pcnt[gids]
        n_seg = max(1, -(-n_words // PROJ_SEG_WORDS))
        cl = proj_stride(cnt, n_words)
        # The Gram reads blocked rows (blocks of its block size, chunk by chunk); rows past m are not written.
        blk = tc_block(self.tc_elem) if method == 1 else 0
        m_rows = -(-m // blk) * blk if blk else m
        cb = np.zeros(len(gids) + 1, np.int64)
        np.cumsum(m_rows * cl, out=cb[1:])
        parts = self._parts(m, -(-cnt // 256) + n_seg) if method == 1 else None
        toff = np.zeros(len(gids) + 1, np.int64)
        np.cumsum(_tile_items(m, method, self.tc_elem) * (1 if parts is None else parts), out=toff[1:])
        n = len(gids)
        # cwords starts as the bound (whole words of the prefix rows plus one padded word per segment);
        # etm_prefix_segments overwrites it with the exact padded length.
        host = np.concatenate([gids.astype(np.int64), toff, cb[:-1], (cnt + 63) // 64 + 4 * n_seg, cl,
                               cl[:0] if parts is None else parts])
        d = self._to_device(host)
        wg, wo = d[:n], d[n:2 * n + 1]
        cbase, cwords, cld = d[2 * n + 1:3 * n + 1], d[3 * n + 1:4 * n + 1], d[4 * n + 1:5 * n + 1]
        parts = None if parts is None or parts.max() == 1 else d[5 * n + 1:]
        seg_off = self.scratch.get(f"proj_seg_{buf}", n * (n_seg + 1), torch.int64)
        proj_counter = self.scratch.get(f"proj_counter_{buf}", 1, torch.int64)
        cbuf = self.scratch.get(f"proj_cbuf_{buf}", int(cb[-1]), torch.int64)
        st = self._launch("prefix_segments", int(n * (width - 1) * n_words * 8),
                          lambda: self.lib.etm_prefix_segments(_p(fbv), ldp, n_words, _p(gen.rows), width,
                                                               _p(grp_first), _p(wg), n, _p(seg_off), _p(cwords),
                                                               *self._occ_args(), _stream()))
        check(st, "etm_prefix_segments")
        self.launches += 1
        if xt is not None:
            # Algorithmic bytes: the prefix columns' words and the prefix rows' row-major words read once, the
            # member strides written.
            xt_t, ldr = xt
            st = self._launch("project_rows", int(n * (width - 1) * n_words * 8 + (cnt * ldr).sum() * 4
                                                  + (m * cl).sum() * 8),
                              lambda: self.lib.etm_project_rows(
                                  _p(fbv), ldp, n_words, _p(xt_t), ldr, _p(gen.rows), width, _p(grp_first),
                                  _p(grp_size), _p(wg), n, _p(seg_off), _p(cbase), _p(cld), blk, _p(cbuf),
                                  _stream()))
            check(st, "etm_project_rows")
            xt_t.record_stream(torch.cuda.current_stream())
            self._waits_pending = True
            self.launches += 2
            return dict(d=d, cbuf=cbuf, cbase=cbase, cwords=cwords, cld=cld, wg=wg, wo=wo, n=n,
                        n_tiles=int(toff[-1]), blocked=bool(blk), parts=parts, nbytes=int((m * ((cnt + 63) // 64)).sum() * 8),
                        macs=float((m * (m - 1) / 2 * cnt.astype(np.float64)).sum()))
        # Algorithmic bytes: every member's column words and the prefix words read once, the strides written.
        st = self._launch("project", int(((m + width - 1) * n_words).sum() * 8 + (m * cl).sum() * 8),
                          lambda: self.lib.etm_project_blocked(
                              _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(wg), n,
                              _p(seg_off), _p(cbase), _p(cld), blk, _p(cbuf), _p(proj_counter), _stream())
                          if blk else self.lib.etm_project(
                              _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(wg), n,
                              _p(seg_off), _p(cbase), _p(cld), _p(cbuf), _p(proj_counter), _stream()))
        check(st, "etm_project")
        self._waits_pending = True
        self.launches += 2
        return dict(d=d, cbuf=cbuf, cbase=cbase, cwords=cwords, cld=cld, wg=wg, wo=wo, n=n, n_tiles=int(toff[-1]),
                    blocked=bool(blk), parts=parts,
                    nbytes=int((m * ((cnt + 63) // 64)).sum() * 8),
                    macs=float((m * (m - 1) / 2 * cnt.astype(np.float64)).sum()))

    def _parts(self, m: np.ndarray, stages: np.ndarray) -> np.ndarray | None:
        """``gram_parts`` of groups of m members over ``stages`` stages, where the Gram can cut its block pairs: the
        batched form over packed e2m1 operands in blocked rows. None elsewhere."""
        if self.form != "batched" or tc_block(self.tc_elem) == TC_TILE:
            return None
        return gram_parts(_tile_items(m, 1, self.tc_elem), stages, self._sms())

    def _bound(self, gen: Level, grp_first: torch.Tensor) -> tuple | None:
        """What block pairs may stop by (``_count_words``): the counts of a level that this mine counted."""
        return (grp_first, gen.counts) if gen.counted and self.early_stop else None

    def _blocked_cols(self, fbv: torch.Tensor, ldp: int) -> torch.Tensor:
        """The columns fbv [n][ldp] in the Gram's blocked member layout (etm_block_cols): K=2 counts from it."""
        n, blk = int(fbv.shape[0]), tc_block(self.tc_elem)
        out = torch.empty(-(-n // blk) * blk * ldp, dtype=torch.int64, device=self.device)
        st = self._launch("block_cols", 16 * n * ldp, lambda: self.lib.etm_block_cols(
            _p(fbv), ldp, n, blk, _p(out), _stream()))
        check(st, "etm_block_cols")
        self.launches += 1
        return out

    def _count_small(self, fbv, ldp, n_words, gen, grp_first, grp_size, cand_off, gids, weights, m, base, cls, counts,
                     sel) -> None:
        """The candidates of groups of few members (etm_count_groups): each group's columns read once per tile."""
        n = len(gids)
        nb = -(-m // GROUP_TILE)
        both = np.zeros((2, n + 1), np.int64)
        np.cumsum(weights, out=both[0, 1:])
        np.cumsum(nb * (nb + 1) // 2, out=both[1, 1:])
        d = self._to_device(np.concatenate([gids.astype(np.int64), both.ravel()]))
        n_cands, n_tiles = int(both[0, -1]), int(both[1, -1])
        partial = self.scratch.get("cands_partial", n_cands, torch.int32) if n_words > GROUP_SLAB_WORDS else None
        # Every group's prefix and member columns, once.
        st = self._launch("count_groups", int((m + gen.k - 1).sum()) * n_words * 8, lambda: self.lib.etm_count_groups(
            _p(fbv), ldp, n_words, _p(gen.rows), gen.k, _p(grp_first), _p(grp_size), _p(cand_off), _p(d),
            _p(d[n:]), _p(d[2 * n + 1:]), n, n_cands, n_tiles, base, _p(cls), 0 if sel is None else sel[0], _p(counts),
            None if sel is None else _p(sel[1]), _p(partial), _stream()))
        check(st, "etm_count_groups")
        self.launches += 1 if partial is None else 2

    def _count_prepped(self, prep, grp_size, cand_off, base, cls, counts, method, sel=None, bound=None):
        """The tile-pair counts of a prepared projection (one launch on the current stream).

        Every tensor the projection made on the side stream and the counting reads here is recorded on this
        stream, so the caching allocator does not hand its memory to a later side-stream allocation (a grown
        scratch buffer) while this stream may still read it.
        """
        cur = torch.cuda.current_stream()
        prep["d"].record_stream(cur)
        prep["cbuf"].record_stream(cur)
        self._count_words(prep["cbuf"], prep["cbase"], prep["cwords"], prep["cld"], grp_size, cand_off, prep["wg"],
                          prep["wo"], prep["n"], prep["n_tiles"], base, cls, counts, method, prep["nbytes"],
                          prep["macs"], sel, prep["blocked"], prep["parts"], bound)

    def _count_projected(self, fbv, ldp, n_words, gen, grp_first, grp_size, cand_off, gids, sizes, pcnt, base, cls,
                         counts, method, sel=None, xt=None):
        """Row lists, projected suffix words and tile-pair counts of the listed groups (one launch each)."""
        prep = self._prep_projected(fbv, ldp, n_words, gen, grp_first, grp_size, gids, sizes, pcnt, method, 0, xt)
        self._count_prepped(prep, grp_size, cand_off, base, cls, counts, method, sel, self._bound(gen, grp_first))

    def _count_words(self, cbuf, cbase, cwords, cld, grp_size, cand_off, wg, wo, n, n_tiles, base, cls, counts,
                     method, nbytes, macs, sel=None, blocked: bool = False, parts=None, bound=None):
        """Tile-pair counts over member words laid out as cbuf[cbase[wi] + i * cld[wi]]: tensor or popcount.

        ``macs`` is the useful work: one multiply-add per candidate pair and row (sum of C(m,2) x rows).
        ``sel`` = (min_count, survivor bitmask) selects the fused-threshold form; ``blocked``: the rows are in
        the projection's blocked layout (tensor method); ``parts``: its block pairs are cut along their rows and
        the counts added (dense, over counts the caller zeroed); ``bound`` = (groups' first rows, the level's counts):
        block pairs stop where these show that none of their candidates is frequent (packed e2m1, blocked, fused).
        """
        elem = self.tc_elem | (TC_BLOCKED if blocked else 0)
        if method == 1:
            # The work counter lets the Gram's CTAs claim block pairs dynamically (one per engine: the Gram
            # launches of an engine run in turn on its main stream).
            counter = self.scratch.get("tc_work_counter", 1, torch.int64)
            if parts is not None:
                fn = lambda: self.lib.etm_count_tiles_tc_parts(  # noqa: E731
                    _p(cbuf), _p(cbase), _p(cwords), _p(cld), _p(grp_size), _p(cand_off), _p(wg), _p(wo), _p(parts), n,
                    n_tiles, base, _p(cls), _p(counts), _p(counter), _stream())
            elif bound is not None and blocked and sel is not None and tc_block(self.tc_elem) != TC_TILE:
                fn = lambda: self.lib.etm_count_tiles_tc_bound(  # noqa: E731
                    _p(cbuf), _p(cbase), _p(cwords), _p(cld), _p(grp_size), _p(cand_off), _p(wg), _p(wo), n, n_tiles,
                    base, _p(cls), sel[0], _p(counts), _p(sel[1]), _p(bound[0]), _p(bound[1]), _p(counter), _stream())
            elif sel is None:
                fn = lambda: self.lib.etm_count_tiles_tc(  # noqa: E731
                    _p(cbuf), _p(cbase), _p(cwords), _p(cld), _p(grp_size), _p(cand_off), _p(wg), _p(wo), n, n_tiles,
                    base, _p(cls), elem, _p(counts), _p(counter), _stream())
            else:
                fn = lambda: self.lib.etm_count_tiles_tc_sel(  # noqa: E731
                    _p(cbuf), _p(cbase), _p(cwords), _p(cld), _p(grp_size), _p(cand_off), _p(wg), _p(wo), n, n_tiles,
                    base, _p(cls), elem, sel[0], _p(counts), _p(sel[1]), _p(counter), _stream())
            check(self._launch("gram_tc", nbytes, fn, flops=2 * macs), "etm_count_tiles_tc")
            self.used_tensor = True
            self._waits_pending = True
        else:
            if sel is None:
                fn = lambda: self.lib.etm_count_tiles_proj(  # noqa: E731
                    _p(cbuf), _p(cbase), _p(cwords), _p(cld), _p(grp_size), _p(cand_off), _p(wg), _p(wo), n, base,
                    _p(cls), 0, _p(counts), _stream())
            else:
                fn = lambda: self.lib.etm_count_tiles_proj_sel(  # noqa: E731
                    _p(cbuf), _p(cbase), _p(cwords), _p(cld), _p(grp_size), _p(cand_off), _p(wg), _p(wo), n, base,
                    _p(cls), sel[0], _p(counts), _p(sel[1]), _stream())
            check(self._launch("count_tiles_proj", nbytes, fn), "etm_count_tiles_proj")
        self.launches += 1

    def count_level(self, gen: Level, fbv: torch.Tensor, ldp: int, n_words: int, mc: int,
                    infer: bool, prune: bool, n_rows: int | None = None) -> tuple[Level, LevelStats]:
        """Count every candidate of the level generated by ``gen``; returns the survivors (k = gen.k + 1).

        Groups with at most ``small_group`` members (in a mine, those where it costs less: ``project_pays``) are
        counted from their columns; larger groups by 64 x 64 tile-pairs, on the prefix's rows
        only (projected) when the prefix holds less than ``proj_density`` of the
        transactions, else on the full bitvectors with the prefix ANDed in.
        Chunks of whole groups bound the dense count scratch (``chunk_cands``)
        and the projection scratch (``proj_bytes``).
        """
        t0 = time.perf_counter()
        width = gen.k
        n_rows = n_words * 64 if n_rows is None else n_rows
        if width == 1 and gen.n > 1:
            # One group of every generator: nothing to search, and nothing to wait for.
            n = gen.n
            G, total = 1, n * (n - 1) // 2
            d = self._to_device(np.array([0, n, 0, total], np.int64))
            grp_first, grp_size, cand_off = d[:1], d[1:2].view(torch.int32), d[2:]
        else:
            G, total, grp_first, grp_size, cand_off = self.groups(gen)
        stats = LevelStats(width + 1, total, 0, 0.0, G)
        if total == 0:
            stats.ms = (time.perf_counter() - t0) * 1e3
            empty = Level(torch.empty((0, width + 1), dtype=torch.int32, device=self.device),
                          torch.empty(0, dtype=torch.int32, device=self.device))
            return empty, stats
        sizes = np.array([gen.n], np.int64) if width == 1 else grp_size[:G].cpu().numpy().astype(np.int64)
        offs = np.zeros(G + 1, np.int64)
        np.cumsum(sizes * (sizes - 1) // 2, out=offs[1:])
        args = (gen, fbv, ldp, n_words, mc, infer, prune, n_rows, G, total, grp_first, grp_size, cand_off, sizes,
                offs, stats)
        tuner = self.autotuner
        if tuner is None or total < tuner.min_candidates:
            level = self._count_groups(*args)
        else:
            key = tuner.key(width + 1, n_words, sizes, total, self.method)
            if key in tuner.cache:
                with self._settings(tuner.cache[key]):
                    level = self._count_groups(*args)
            else:
                # First level of this shape: count it under every setting, keep the fastest.
                best = None
                for setting in tuner.settings(self.method):
                    with self._settings(setting):
                        torch.cuda.synchronize()
                        t1 = time.perf_counter()
                        trial = self._count_groups(*args)
                        torch.cuda.synchronize()
                        dt = time.perf_counter() - t1
                    tuner.trials.append({"key": key, **setting, "s": dt})
                    if best is None or dt < best[0]:
                        best = (dt, setting, trial)
                tuner.cache[key] = best[1]
                level = best[2]
        stats.ms = (time.perf_counter() - t0) * 1e3
        stats.n_frequent = level.n
        return level, stats

    def _settings(self, setting: dict):
        """Context manager applying tuned attributes (small_group, proj_density) for one count."""
        engine = self

        class _Apply:
            def __enter__(self):
                self.saved = {k: getattr(engine, k) for k in setting}
                for k, v in setting.items():
                    setattr(engine, k, v)

            def __exit__(self, *exc):
                for k, v in self.saved.items():
                    setattr(engine, k, v)

        return _Apply()

    def _count_groups(self, gen, fbv, ldp, n_words, mc, infer, prune, n_rows, G, total, grp_first, grp_size,
                      cand_off, sizes, offs, stats) -> Level:
        """The counting of a level's candidates given its groups (see ``count_level``)."""
        width = gen.k
        stats.n_chunks = 0
        out_rows = torch.empty((0, width + 1), dtype=torch.int32, device=self.device)
        out_counts = torch.empty(0, dtype=torch.int32, device=self.device)
        # The subset test has prefix subsets to look up only from K=3 on.
        classify = (infer or prune) and width >= 2
        mode = (1 if prune or infer else 0) | (2 if infer else 0)
        deep = self._deep if (infer and self.deduction_bounds and self.fused and width + 1 <= 24) else None
        if deep is not None:
            mode |= 4  # ETM_SUBSET_BOUNDS
        big = sizes > self.small_group
        tensor = self.method == "tensor"
        pcnt = np.zeros(G, np.int64)
        proj = np.zeros(G, bool)
        ri = self._rows_input
        # K=3 from the transactions: each row adds 1 to the candidates it holds (sparse rows, one chunk).
        k3_rows = (width == 2 and ri is not None and self.k3_rows_max_r > 0 and total <= self.chunk_cands
                   and ri["pair_work"] < self.k3_rows_max_r * total * n_words)
        stats.row_wise = stats.row_wise or k3_rows
        # The Gram may cut its block pairs along their rows (``_parts``).
        cut = tensor and self._parts(sizes[:0], pcnt[:0]) is not None
        # With every prefix's rows at hand each group goes where it costs less, not by its members alone.
        by_cost = (cut and self.small_group == SMALL_GROUP and self.proj_rows and self._occ is None
                   and self._prefix_level is not None)
        if not k3_rows and (self.project or tensor) and width >= 2 and (big.any() or by_cost):
            ids_big = np.flatnonzero(big)
            known = self._prefix_support(gen, grp_first, G)
            if known is not None and by_cost:
                n_cols = int(fbv.shape[0])
                big = project_pays(sizes, known, width - 1, n_words, n_cols, self._xt_key == (
                    fbv.data_ptr(), n_words, n_cols))
                ids_big = np.flatnonzero(big)
            pcnt[ids_big] = (self.prefix_counts(fbv, ldp, n_words, gen, grp_first, ids_big) if known is None
                             else known[ids_big])
            if tensor:
                # The tensor cores count projected words; a prefix past 2^24 rows stays on popcount where the Gram
                # does not cut it into parts of fewer rows.
                proj = big if cut else big & (pcnt <= TC_MAX_ROWS)
            else:
                proj = big & (pcnt < self.proj_density * n_rows)
        pwords = proj_stride(pcnt, n_words)
        blk = tc_block(self.tc_elem) if tensor else 0
        pbytes = np.where(proj, (-(-sizes // blk) * blk if blk else sizes) * pwords * 8, 0)
        pcum = np.zeros(G + 1, np.int64)
        np.cumsum(pbytes, out=pcum[1:])
        cap = int(min(total, max(1 << 16, 2 * gen.n)))
        out_rows = torch.empty((cap, width + 1), dtype=torch.int32, device=self.device)
        out_counts = torch.empty(cap, dtype=torch.int32, device=self.device)
        acc = self.scratch.get("acc", 1, torch.int64)
        acc.zero_()
        n_out = 0
        method = 1 if tensor else 0
        n_seg = max(1, -(-n_words // PROJ_SEG_WORDS))
        blocked = None  # K=2: the columns in the Gram's member layout
        if width == 1 and cut and big.any() and self._k2_rows is None:
            try:
                blocked = self._blocked_cols(fbv, ldp)
            except torch.OutOfMemoryError:
                cut = False  # no room for another copy of them: from the columns as they are, in whole block pairs
        # K=2 on the tensor cores: the one group of every generator, its members the padded columns.
        whole_tc = tensor and width == 1 and (cut or n_rows <= TC_MAX_ROWS)
        # Chunks: whole groups within both budgets (at least one group each).
        chunks = []
        g0 = 0
        while g0 < G:
            g1c = int(np.searchsorted(offs, offs[g0] + self.chunk_cands, side="right")) - 1
            g1p = int(np.searchsorted(pcum, pcum[g0] + self.proj_bytes, side="right")) - 1
            g1 = max(min(g1c, g1p), g0 + 1)
            chunks.append((g0, g1))
            g0 = g1
        # The row-major copy for the projection, made on the main stream before any side-stream work reads it.
        xt = self._rows_copy(fbv, ldp, n_words) if (self.proj_rows and proj.any()) else None
        # Batched form with the column projection: the projection of chunk c+1 runs on a side stream while chunk
        # c is counted; two scratch sets alternate. The row-major projection stays on the main stream: it is
        # short, and the Gram's CTAs leave no room on their SMs for it (measured: 0.563 s per dense K=2 mine
        # with the side stream, 0.545 s without).
        pipelined = self.pipeline and self.form == "batched" and proj.any() and xt is None
        main = torch.cuda.current_stream()
        side = self._side_stream() if pipelined else None
        prep_done = [torch.cuda.Event(), torch.cuda.Event()]
        buf_free = [torch.cuda.Event(), torch.cuda.Event()]
        preps: dict[int, dict] = {}

        def proj_ids(c):
            a, b = chunks[c]
            sel = proj[a:b]
            return np.arange(a, b, dtype=np.int64)[sel]

        def prep(c):
            ids_c = proj_ids(c)
            if len(ids_c) == 0:
                return
            buf = c % 2
            with torch.cuda.stream(side):
                side.wait_event(buf_free[buf])
                preps[c] = self._prep_projected(fbv, ldp, n_words, gen, grp_first, grp_size, ids_c, sizes, pcnt,
                                                method, buf, xt)
                prep_done[buf].record(side)

        if pipelined:
            start_ev = torch.cuda.Event()
            start_ev.record(main)
            side.wait_event(start_ev)  # the generating level and group tables come from the main stream
            prep(0)
        grp_of = None
        for c, (g0, g1) in enumerate(chunks):
            base = int(offs[g0])
            n_c = int(offs[g1] - base)
            counts = self.scratch.get("chunk_counts", n_c, torch.int32)
            cls = self.scratch.get("chunk_cls", n_c, torch.uint8) if classify else None
            k2_rows = width == 1 and self._k2_rows is not None
            row_wise = k2_rows or k3_rows
            # Fused threshold: the counting kernels set survivor bits (the row-wise kernels count densely and a
            # threshold pass sets the bits after them).
            bits = None
            if self.fused:
                bits = self.scratch.get("chunk_bits", (n_c + 31) // 32 + 1, torch.int32)
                bits.zero_()
            sel = (mc, bits) if (self.fused and not row_wise) else None
            m = sizes[g0:g1]
            ids = np.arange(g0, g1, dtype=np.int64)
            small = ~big[g0:g1]
            pr = proj[g0:g1]
            # Tile groups too few to fill the GPU (few members over many rows) split their word ranges across
            # CTAs, which add partial counts: the chunk's counts start at zero and its bits come from a
            # threshold pass at the end (the fused kernels leave non-survivors at zero, so the pass agrees).
            tile_ids = ids[~small & ~pr] if not row_wise else ids[:0]
            n_split = 1
            if len(tile_ids):
                nt_t = (sizes[tile_ids] + TILE - 1) // TILE
                n_tp = int((nt_t * (nt_t + 1) // 2).sum())
                n_split = int(max(1, min(-(-n_words // 32), (6 * self._sms()) // max(1, n_tp))))
            # So do the Gram's block pairs where few of them hold most of the rows.
            k2_parts = self._parts(m[tile_ids - g0], np.full(len(tile_ids), -(-n_words // 4))) if whole_tc and cut else None
            g_split = not row_wise and (
                (k2_parts is not None and len(tile_ids) > 0 and k2_parts.max() > 1) or
                (cut and bool(pr.any()) and self._parts(m[pr], -(-pcnt[g0:g1][pr] // 256) + n_seg).max() > 1))
            added = g_split or (n_split > 1 and not whole_tc)
            if added:
                counts.zero_()
            if classify:
                if sel is None:
                    fn = lambda: self.lib.etm_classify(  # noqa: E731
                        _p(gen.rows), width, gen.n, _p(gen.counts), _p(gen.free), _p(grp_first), _p(grp_size),
                        _p(cand_off), g0, g1, mode, _p(cls), _p(counts), _stream())
                else:
                    d2, d3, n_tot = deep if deep is not None else (None, None, n_rows)
                    fn = lambda: self.lib.etm_classify_sel(  # noqa: E731
                        _p(gen.rows), width, gen.n, _p(gen.counts), _p(gen.free), _p(grp_first), _p(grp_size),
                        _p(cand_off), g0, g1, mode if sel is not None else mode & ~4, mc,
                        _p(d2.rows) if d2 is not None else None, d2.n if d2 is not None else 0,
                        _p(d2.counts) if d2 is not None else None, _p(d3.rows) if d3 is not None else None,
                        d3.n if d3 is not None else 0, _p(d3.counts) if d3 is not None else None, n_tot, _p(cls),
                        _p(counts), _p(bits), _stream())
                check(self._launch("classify", n_c * 5, fn), "etm_classify")
                self.launches += 1
                if self.class_stats:
                    by_class = torch.bincount(cls[:n_c].to(torch.int64), minlength=3).cpu().tolist()
                    stats.n_skipped += int(by_class[1])
                    stats.n_inferred += int(by_class[2])
            if k2_rows:
                stats.row_wise = True
                # K=2 from the transactions (one group of every generator): pair counts by row-wise increments.
                rp, cl, nnz, lut, n_r = self._k2_rows
                n_g = int(sizes[0])
                st = self._launch("pair_counts_rows", nnz * 8 + n_r * 8 + n_c * 4, lambda: self.lib.etm_pair_counts_rows(
                    _p(rp), _p(cl), nnz, _p(lut), lut.numel(), n_r, n_g, _p(counts), _stream()))
                check(st, "etm_pair_counts_rows")
                self.launches += 1
            if k3_rows:
                if grp_of is None:
                    grp_of = torch.full((ri["ng"],), -1, dtype=torch.int32, device=self.device)
                    grp_of[gen.rows[grp_first[:G], 0].long()] = torch.arange(G, dtype=torch.int32, device=self.device)
                st = self._launch("triple_counts_rows", ri["nnz"] * 8 + ri["n_r"] * 8 + n_c * 4,
                                  lambda: self.lib.etm_triple_counts_rows(
                                      _p(ri["rp"]), _p(ri["cl"]), ri["nnz"], _p(ri["lut"]), ri["lut"].numel(),
                                      ri["n_r"], _p(gen.rows), _p(grp_of), ri["ng"], _p(grp_first), _p(grp_size),
                                      _p(cand_off), base, n_c, _p(cls), _p(counts), _stream()))
                check(st, "etm_triple_counts_rows")
                self.launches += 2
            for kind, which in (() if (k2_rows or k3_rows) else
                                (("cands", small), ("tiles", ~small & ~pr), ("proj", pr & ~small))):
                gids = ids[which]
                if len(gids) == 0:
                    continue
                if kind == "proj":
                    if pipelined:
                        main.wait_event(prep_done[c % 2])
                        self._count_prepped(preps.pop(c), grp_size, cand_off, base, cls, counts, method, sel,
                                            self._bound(gen, grp_first))
                        buf_free[c % 2].record(main)
                        continue
                    groups = [gids] if self.form == "batched" else [gids[q:q + 1] for q in range(len(gids))]
                    for bg in groups:
                        self._count_projected(fbv, ldp, n_words, gen, grp_first, grp_size, cand_off, bg, sizes, pcnt,
                                              base, cls, counts, method, sel, xt)
                    continue
                if kind == "tiles" and whole_tc:
                    mg = sizes[gids]
                    toff = np.zeros(len(gids) + 1, np.int64)
                    np.cumsum(_tile_items(mg, 1, self.tc_elem) * (1 if k2_parts is None else k2_parts), out=toff[1:])
                    n = len(gids)
                    src, blocked = blocked if cut else fbv, None
                    host = np.concatenate([gids, toff, np.zeros(n, np.int64), np.full(n, n_words, np.int64),
                                           np.full(n, ldp, np.int64), gids[:0] if k2_parts is None else k2_parts])
                    d = self._to_device(host)
                    self._count_words(src, d[2 * n + 1:3 * n + 1], d[3 * n + 1:4 * n + 1], d[4 * n + 1:5 * n + 1],
                                      grp_size, cand_off, d[:n], d[n:2 * n + 1], n, int(toff[-1]), base, cls, counts,
                                      1, int(mg.sum()) * n_words * 8,
                                      float((mg * (mg - 1) / 2).astype(np.float64).sum() * n_rows), sel, cut,
                                      d[5 * n + 1:] if g_split else None, self._bound(gen, grp_first))
                    continue
                if kind == "cands":
                    w = m[which] * (m[which] - 1) // 2
                else:
                    nt = (m[which] + TILE - 1) // TILE
                    w = nt * (nt + 1) // 2
                batches = [(gids, w)] if self.form == "batched" else [(gids[q:q + 1], w[q:q + 1]) for q in range(len(gids))]
                for bg, bw in batches:
                    mg = sizes[bg]
                    if kind == "cands" and self._occ is None:
                        self._count_small(fbv, ldp, n_words, gen, grp_first, grp_size, cand_off, bg, bw, mg, base, cls,
                                          counts, sel)
                        continue
                    wg, wo = self._work(bg, bw)
                    if kind == "cands":
                        # Every candidate reads its k columns.
                        nbytes = int((mg * (mg - 1) // 2).sum()) * (width + 1) * n_words * 8
                        if sel is None:
                            fn = lambda: self.lib.etm_count_cands(  # noqa: E731
                                _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off),
                                _p(wg), _p(wo), len(bg), base, _p(cls), _p(counts), _stream())
                        else:
                            fn = lambda: self.lib.etm_count_cands_sel(  # noqa: E731
                                _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off),
                                _p(wg), _p(wo), len(bg), base, _p(cls), mc, _p(counts), _p(bits), *self._occ_args(),
                                _stream())
                        st = self._launch("count_cands", nbytes, fn)
                    else:
                        # Each group's prefix and suffix columns, once (the same-data minimum). Groups that reach
                        # this kind under the tensor method hold more than 2^24 rows (past the f32-exact range
                        # of the Gram), so these tiles always count on the CUDA cores.
                        nbytes = int((mg + width - 1).sum()) * n_words * 8
                        if n_split > 1:
                            fn = lambda: self.lib.etm_count_tiles_split(  # noqa: E731
                                _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off),
                                _p(wg), _p(wo), len(bg), int(bw.sum()), base, _p(cls), n_split, _p(counts), _stream())
                        elif sel is None:
                            fn = lambda: self.lib.etm_count_tiles(  # noqa: E731
                                _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off),
                                _p(wg), _p(wo), len(bg), base, _p(cls), 0, _p(counts), _stream())
                        else:
                            fn = lambda: self.lib.etm_count_tiles_sel(  # noqa: E731
                                _p(fbv), ldp, n_words, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off),
                                _p(wg), _p(wo), len(bg), base, _p(cls), mc, _p(counts), _p(bits), _stream())
                        st = self._launch("count_tiles", nbytes, fn)
                    check(st, f"etm_count_{kind}")
                    self.launches += 1
            if pipelined and c + 1 < len(chunks):
                prep(c + 1)  # overlaps this chunk's counting and the host wait in its compaction
            if self.fused and (row_wise or added):
                check(self._launch("threshold_bits", n_c * (5 if classify else 4), lambda: self.lib.etm_threshold_bits(
                    _p(counts), _p(cls), n_c, mc, _p(bits), _stream())), "etm_threshold_bits")
                self.launches += 1
            n_scan = (n_c + 31) // 32 if self.fused else n_c
            ws = self.scratch.get("ws_compact", scan_words(n_scan), torch.int64)
            while True:
                if self.fused:
                    # Reads the bitmask, and the counts of the survivors only.
                    fn = lambda: self.lib.etm_level_compact_bits(  # noqa: E731
                        _p(bits), _p(counts), n_c, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off),
                        g0, g1, _p(out_rows), _p(out_counts), cap, _p(acc), _p(ws), ws.numel(), _stream())
                    nbytes = (n_c + 7) // 8
                else:
                    fn = lambda: self.lib.etm_level_compact(  # noqa: E731
                        _p(counts), _p(cls), n_c, _p(gen.rows), width, _p(grp_first), _p(grp_size), _p(cand_off), g0,
                        g1, mc, _p(out_rows), _p(out_counts), cap, _p(acc), _p(ws), ws.numel(), _stream())
                    nbytes = n_c * (5 if classify else 4)
                check(self._launch("level_compact", nbytes, fn), "etm_level_compact")
                self.launches += 3
                new_total = int(acc.item())
                if new_total <= cap:
                    break
                # Grow to the level's survivors extrapolated from the candidates counted so far, so that the
                # later chunks compact once.
                done = max(1, int(offs[g1] - offs[0]))
                projected = int(new_total * (total / done) * 1.1)
                cap = int(min(total, max(2 * cap, int(new_total * 1.25), projected)))
                grown_r = torch.empty((cap, width + 1), dtype=torch.int32, device=self.device)
                grown_c = torch.empty(cap, dtype=torch.int32, device=self.device)
                grown_r[:n_out] = out_rows[:n_out]
                grown_c[:n_out] = out_counts[:n_out]
                out_rows, out_counts = grown_r, grown_c
                acc.fill_(n_out)
            n_out = new_total
            stats.n_chunks += 1
        self.check_device_status()
        return Level(out_rows[:n_out], out_counts[:n_out], counted=True)

    def check_device_status(self) -> None:
        """Raise if a Gram or projection launch since the last check gave up a bounded device wait.

        The kernels record the give-up in device status words instead of hanging; their counts are then
        incomplete, so the level is not returned. The projection's give-up leaves the device in an unknown
        state (bulk copies may still be landing): the caller should stop using the device.
        """
        if not self._waits_pending:
            return
        if self._side is not None:
            torch.cuda.current_stream().wait_stream(self._side)
        self._waits_pending = False
        st = self.lib.etm_device_status(_stream())
        if st != 0:
            raise RuntimeError(f"device counting failed: {self.lib.etm_last_error().decode()}")

    def _free_flags(self, new: Level, gen: Level, with_present: bool = False):
        """(free, present or None) of the rows of ``new`` against the level before it: no (k-1)-subset of the same
        count; every (k-1)-subset a row of ``gen``."""
        free = torch.empty(new.n, dtype=torch.uint8, device=self.device)
        present = torch.empty(new.n, dtype=torch.uint8, device=self.device) if with_present else None
        check(self.lib.etm_level_subsets(_p(new.rows), _p(new.counts), new.n, gen.k, _p(gen.rows), _p(gen.counts),
                                         gen.n, _p(free), _p(present), _stream()), "etm_level_subsets")
        self.launches += 1
        return free, present

    def _free_of(self, hist: list, prune: bool) -> torch.Tensor:
        """The free flags of the latest of these levels: under the free-set prune every row of it is free."""
        if prune:
            return torch.ones(hist[-1].n, dtype=torch.uint8, device=self.device)
        return self._free_flags(hist[-1], hist[-2])[0]

    def finish_level(self, new: Level, gen: Level, track_free: bool, prune: bool) -> Level:
        """Free flags against the generating level; under the free-set prune keep the free rows
        whose subsets are all generators (gpu/row_split.py:1075-1100)."""
        if not track_free or new.n == 0:
            if track_free:
                new.free = torch.zeros(0, dtype=torch.uint8, device=self.device)
            return new
        free, present = self._free_flags(new, gen, prune)
        if not prune:
            new.free = free
            return new
        out_r = torch.empty_like(new.rows)
        out_c = torch.empty_like(new.counts)
        out_f = torch.empty_like(free)
        acc = self.scratch.get("acc_sel", 1, torch.int64)
        acc.zero_()
        ws = self.scratch.get("ws_select", scan_words(new.n), torch.int64)
        check(self.lib.etm_select_rows(_p(new.rows), _p(new.counts), _p(free), _p(present), new.n, new.k, _p(out_r),
                                       _p(out_c), _p(free), _p(out_f), new.n, _p(acc), _p(ws), ws.numel(),
                                       _stream()), "etm_select_rows")
        self.launches += 3
        kept = int(acc.item())
        return Level(out_r[:kept], out_c[:kept], out_f[:kept], new.counted)

    # -- small levels ------------------------------------------------------------
    def _form_ok(self, max_k: int) -> bool:
        """Whether this engine's form and thresholds are the defaults (an engine set up to count otherwise does), and
        nothing asks for a level's classes, tunes it or reads an occupancy."""
        return (self.direct and self.method == "tensor" and self.form == "batched" and self.fused and self.project
                and self.proj_rows and self.small_group == SMALL_GROUP and self.autotuner is None
                and not self.class_stats and self._occ is None and self.k2_rows_max_r == K2_ROWS_MAX_R
                and self.k3_rows_max_r == K3_ROWS_MAX_R and max_k >= 2)

    def _direct_ok(self, max_k: int) -> bool:
        """Whether its small levels may go through etm_mine_direct as well: with the default operands, since the launch
        has none. Its budgets (``chunk_cands``, ``proj_bytes``) bound the launch; without ``pipeline`` or
        ``deduction_bounds`` it is as good, as it overlaps nothing and settles nothing by bounds."""
        return self.tc_elem & ~TC_WIDE == DEFAULT_TC_ELEM and self._form_ok(max_k)

    def _direct_cands(self, scale: int) -> int:
        return direct_cands(scale, self.chunk_cands)

    def _direct_proj(self, n_cols: int, n_words: int) -> int:
        return direct_proj(n_cols, n_words, self.proj_bytes)

    def _direct_held(self) -> int:
        return sum(t.numel() * t.element_size() for k, t in self.scratch.bufs.items() if k.startswith("direct"))

    def _direct_room(self, max_vram_gb: float | None) -> float:
        """Device bytes that the direct launches' buffers, those held among them, may take."""
        room = math.inf if self.direct_max_bytes is None else float(self.direct_max_bytes)
        if max_vram_gb is not None:
            room = min(room, (max_vram_gb - _allocated_gb(self.device)) * (1 << 30) + self._direct_held())
        return room

    def _drop_direct(self) -> float:
        """Gives the direct launches' buffers back; their size in GB."""
        held, stream = self._direct_held(), torch.cuda.current_stream(self.device)
        for k in [k for k in self.scratch.bufs if k.startswith("direct")]:
            self.scratch.bufs.pop(k).record_stream(stream)  # which may not be the one they were made on
        return held / (1 << 30)

    def _mine_direct(self, ptr: int, ld: int, n_words: int, n_cols: int, n_rows: int, mc: int, prune: bool, max_k: int,
                     col_counts: torch.Tensor | None = None, start: Level | None = None, turn: bool = False,
                     scale: int | None = None, projected: bool = False, max_vram_gb: float | None = None):
        """One etm_mine_direct launch and its header: (done, level 1 or None, the levels it counted, their (candidates,
        groups), the outputs (rows, counts) on the host if they are few, else those of level 1 there, whether all are,
        whether a capacity that the largest launch has more of stopped it on projected columns), or None when it gave up
        a wait. ``done``: no level follows. ``projected``: the columns are those that the mine's launch before left
        projected. Where its limits leave no room for the memory of a large launch it is a small one, on full columns;
        None where there is none for that either, where the start level does not fit it, or where the device has no
        memory left."""
        width = 0 if start is None else start.k
        scale = scale or direct_scale(n_cols, n_words)
        proj_words = self._direct_proj(n_cols, n_words) if width == 2 or projected else 0
        if not projected and (self.direct_max_bytes is not None or max_vram_gb is not None and (scale > 1 or proj_words)):
            room = self._direct_room(max_vram_gb)
            if direct_bytes(scale, self._direct_cands(scale), n_cols, n_words, proj_words) > room:
                scale, proj_words = 1, 0
            if self.direct_max_bytes is not None and direct_bytes(1, self._direct_cands(1), n_cols, n_words, 0) > room:
                return None
        if start is not None and start.n > DIRECT_ROWS * scale:
            return None
        cap_rows, cap_cands = DIRECT_ROWS * scale, self._direct_cands(scale)
        n_head, n_counts, n_items = DIRECT_HEADER, DIRECT_COUNTS_CAP * scale, DIRECT_ROWS_CAP * scale
        n_scratch, n_proj = ctypes.c_int64(), ctypes.c_int64()
        check(self.lib.etm_direct_scratch_words(cap_rows, cap_cands, n_cols, n_words, proj_words, ctypes.byref(n_scratch),
                                                ctypes.byref(n_proj)), "etm_direct_scratch_words")
        n_scratch, n_proj = n_scratch.value, n_proj.value
        try:
            buf = self.scratch.get("direct_out", n_head + n_counts + n_items, torch.int32)
            scratch = self.scratch.get("direct", n_scratch, torch.int32)
            proj = self.scratch.get("direct_proj", n_proj, torch.int32) if proj_words else None
            few = torch.empty(DIRECT_FETCH_COUNTS + DIRECT_FETCH_ROWS, dtype=torch.int32, device=self.device)
        except torch.OutOfMemoryError:
            buf = scratch = proj = None
            self._drop_direct()  # the general path needs less
            return None
        header_p = buf.data_ptr()
        counts_p, rows_p = header_p + 4 * n_head, header_p + 4 * (n_head + n_counts)
        last_k = min(max_k, DIRECT_LEVELS - 2)
        st = self._launch("mine_direct", 0, lambda: self.lib.etm_mine_direct(
            ptr, ld, n_words, n_cols, _p(col_counts), n_rows, mc, int(prune), last_k, DIRECT_WORDS,
            min(DIRECT_WORDS, DIRECT_TURN) if turn else DIRECT_WORDS, None if start is None else _p(start.rows),
            None if start is None else _p(start.counts),
            0 if start is None else start.n, width, header_p, counts_p, n_counts, rows_p, n_items,
            cap_rows, cap_cands, proj_words, int(projected), _p(scratch), n_scratch, _p(proj), n_proj, _stream()))
        check(st, "etm_mine_direct")
        self.launches += 1
        # The header and the start of the outputs (a page-locked buffer of the engine's, read out before it is used again),
        # and that start in memory of its own: a result outlives the launch.
        if self._fetched is None:
            self._fetched = torch.empty(n_head + DIRECT_FETCH_COUNTS + DIRECT_FETCH_ROWS, dtype=torch.int32,
                                        pin_memory=True)
        check(self.lib.etm_direct_take(header_p, counts_p, DIRECT_FETCH_COUNTS, rows_p, DIRECT_FETCH_ROWS,
                                       _p(self._fetched), _p(few), _stream()), "etm_direct_take")
        fetched = self._fetched.numpy()
        head = fetched[:n_head].view(np.int64).copy()
        if head[0] < 0:
            return None
        last = int(head[1])
        level1 = None
        r_at = c_at = 0
        if start is None:
            n1 = int(head[12]) if last >= 1 else cap_rows + 1
            if n1 > cap_rows:
                return False, None, [], [], None, False, False
            r_at = c_at = n1
        sizes = {k: int(head[8 + 4 * k]) for k in range(max(2, width + 1), last + 1)}
        n_c, n_r = c_at + sum(sizes.values()), r_at + sum(n * k for k, n in sizes.items())
        on_host = n_c <= DIRECT_FETCH_COUNTS and n_r <= DIRECT_FETCH_ROWS
        counts, rows = (few.split([DIRECT_FETCH_COUNTS, DIRECT_FETCH_ROWS]) if on_host else
                        (buf[n_head:n_head + n_c].clone(), buf[n_head + n_counts:n_head + n_counts + n_r].clone()))
        if start is None:
            level1 = (rows[:n1], counts[:n1])
        h_c, h_r = (n_c, n_r) if on_host else (n1, n1) if start is None else (0, 0)
        if max(h_c, h_r) <= DIRECT_FETCH_COUNTS or on_host:
            host = (fetched[n_head + DIRECT_FETCH_COUNTS:][:h_r].copy(), fetched[n_head:n_head + h_c].copy())
        else:
            host = (rows[:h_r].cpu().numpy(), counts[:h_c].cpu().numpy())
        levels, seen = [], []
        for k, n in sizes.items():
            levels.append(Level(rows[r_at:r_at + n * k].view(n, k), counts[c_at:c_at + n], counted=True))
            seen.append((int(head[9 + 4 * k]), int(head[10 + 4 * k])))
            r_at, c_at = r_at + n * k, c_at + n
        # A level follows the launch's own last one where the mine's is past it.
        done = int(head[0]) == 0 and (last < last_k or last_k == max_k or sizes[last] == 0)
        larger = bool(head[3]) and (head[2] == 2 or (head[2] == 1 and self._direct_cands(DIRECT_MOST) > cap_cands))
        return done, level1, levels, seen, host, on_host, larger

    def _order_rows(self, rows: torch.Tensor, counts: torch.Tensor, order: torch.Tensor, out_rows: torch.Tensor,
                    out_counts: torch.Tensor) -> None:
        """The rows over the generator indices ``order`` gives their items, sorted within and among each other
        (etm_order_level), with their counts."""
        n, k = rows.shape
        bits = max(1, (int(order.numel()) - 1).bit_length())
        nbytes = ctypes.c_int64()
        check(self.lib.etm_order_level_bytes(n, k, bits, ctypes.byref(nbytes)), "etm_order_level_bytes")
        scratch = torch.empty(nbytes.value, dtype=torch.uint8, device=self.device)
        # Each row read and written once.
        st = self._launch("order_level", 8 * n * (k + 1), lambda: self.lib.etm_order_level(
            _p(rows), _p(counts), n, k, _p(order), bits, _p(out_rows), _p(out_counts), _p(scratch), nbytes.value,
            _stream()))
        check(st, "etm_order_level")
        self.launches += self.lib.etm_order_level_launches(n, k, bits)

    def _order_pieces(self, level: Level, order: torch.Tensor, rows: torch.Tensor, counts: torch.Tensor) -> None:
        """``_order_rows`` of a level by ranges of the rows' first items, in a few bytes a row beside the output."""
        ng, first = int(order.numel()), torch.empty(level.n, dtype=torch.int32, device=self.device)
        seen = torch.zeros(ng, dtype=torch.int64, device=self.device)
        steps = [slice(a, min(a + ORDER_STEP, level.n)) for a in range(0, level.n, ORDER_STEP)]
        for s in steps:
            first[s] = order[level.rows[s].long()].amin(1)
            seen += torch.bincount(first[s], minlength=ng)
        seen = seen.cpu().numpy()
        at = lo = 0
        while lo < ng:
            hi, m = lo + 1, int(seen[lo])
            while hi < ng and m + seen[hi] <= ORDER_PIECE:
                m, hi = m + int(seen[hi]), hi + 1
            if m:
                part = [((first[s] >= lo) & (first[s] < hi)).nonzero().view(-1) + s.start for s in steps]
                part = torch.cat([p for p in part if p.numel()])
                self._order_rows(level.rows[part], level.counts[part], order, rows[at:at + m], counts[at:at + m])
            at, lo = at + m, hi

    def _named_level(self, level: Level, order: torch.Tensor) -> Level:
        """A level counted over generators in ``order`` (the generator index of each place), over the generator indices
        themselves: rows sorted within and among each other. A level of more rows than etm_order_level takes, or that
        leaves no room for its scratch (24 bytes a row), goes piece by piece."""
        rows, counts = torch.empty_like(level.rows), torch.empty_like(level.counts)
        whole = level.n <= ORDER_ROWS
        if level.n and whole:
            try:
                self._order_rows(level.rows, level.counts, order, rows, counts)
            except torch.OutOfMemoryError:
                whole = False
        if not whole:
            self._order_pieces(level, order, rows, counts)
        return Level(rows, counts)

    def _named_levels(self, levels: list[Level], order: torch.Tensor, named: Level, totals: torch.Tensor) -> list[Level]:
        """``_named_level`` of the levels of one direct launch (one after another in memory, from ``named.k + 1`` on) in one
        call, and the candidates and groups of each, from the level before it in the columns' order, to ``totals``."""
        sizes = np.array([lv.n for lv in levels], np.int64)
        k0 = levels[0].k
        items = sizes * (k0 + np.arange(len(levels)))
        rows = torch.empty(int(items.sum()), dtype=torch.int32, device=self.device)
        counts = torch.empty(int(sizes.sum()), dtype=torch.int32, device=self.device)
        bits = max(1, (int(order.numel()) - 1).bit_length())
        need, nbytes = 1, ctypes.c_int64()
        for lv in levels:
            check(self.lib.etm_order_level_bytes(lv.n, lv.k, bits, ctypes.byref(nbytes)), "etm_order_level_bytes")
            need = max(need, nbytes.value)
        scratch = torch.empty(need, dtype=torch.uint8, device=self.device)
        st = self._launch("order_level", int(8 * (items + sizes).sum()), lambda: self.lib.etm_order_levels(
            _p(levels[0].rows), _p(levels[0].counts), sizes.ctypes.data, len(levels), k0, _p(order), bits, _p(named.rows),
            named.n, _p(rows), _p(counts), _p(totals[k0]), _p(scratch), need, _stream()))
        check(st, "etm_order_levels")
        before = [named.n, *(lv.n for lv in levels[:-1])]
        self.launches += sum(self.lib.etm_order_level_launches(lv.n, lv.k, bits) + (n > 0) for lv, n in zip(levels, before))
        out, r, c = [], 0, 0
        for lv, m in zip(levels, items.tolist()):
            out.append(Level(rows[r:r + m].view(lv.n, lv.k), counts[c:c + lv.n]))
            r, c = r + m, c + lv.n
        return out

    # -- the whole mine ----------------------------------------------------------
    def mine(self, bitvecs, n_rows: int, min_support: float, max_length: int | None = None, *,
             prune_equal_support: bool = False, use_generator_pruning: bool = False,
             level_callback=None, n_cols_logical: int | None = None, rows=None, max_ram_gb: float | None = None,
             max_vram_gb: float | None = None, on_level=None, resume=None, keep_levels: bool = True,
             occupancy: bool = False, free_flags: bool = True) -> MineOutput:
        """Mine device bitvectors. ``rows`` = (row_ptr int64, cols int32, host row lengths) on the device,
        the transactions the bitvectors were built from, lets K=2 count row-wise when its rows are short
        against the pair space (the reference's rule, gpu/row_split_chunks.py:124-142). A fourth element
        (int32, -1 for none) makes the entries codes mapped to columns through it; the lengths then count
        only the entries that map to a column. A number in place of the lengths is the rows' pairs in all, the sum
        of L (L - 1) / 2.

        ``max_ram_gb`` / ``max_vram_gb``: for every level, the process's resident memory and the device
        memory allocated through torch (every engine buffer) are checked against them; over a limit the mine raises
        MemoryError instead of returning a partial lattice (gpu/row_split.py:467-487).

        Small levels come out of one launch several at a time (``direct``): their callbacks and checks, level by level
        as ever, then follow after the launch, and its time is shared out evenly over their ``LevelStats.ms``.

        ``on_level(k, caller_cols int64 [n, k], counts int64 [n])`` receives every emitted level on the host
        as soon as it is final (the per-level flush); with ``keep_levels=False`` the emitted levels are not kept
        in the output (only the few the next levels need stay on the device).

        ``resume = (k, caller_cols [n, k], counts [n])``: start from a complete emitted level k read back from a
        flush (gpu/row_split.py:546-606): levels 1..k are neither counted nor emitted again; the first resumed
        level has no free flags to infer from, and the deduction bounds wait for levels k-2 and k-3.

        ``occupancy``: build the generating columns' tile occupancy once, and let the prefix and per-candidate
        kernels skip the tiles where a prefix (or a candidate's) column holds no row. It pays when the rows
        are in the input layer's lex order, where deep itemsets' rows gather (gpu/row_split.py:397-413).

        ``free_flags``: under generator pruning or the free-set prune the returned levels carry their free flags; a caller
        that does not read them saves a launch a level with False.
        """
        ptr, (n_cols, ld), _owner = as_device_bitvecs(bitvecs)
        self._k2_rows = None
        self._rows_input = None
        self._xt, self._xt_key = None, None  # the row-major copy belongs to one mine's generating columns
        self._occ = None  # so does the tile occupancy
        self._prefix_level = None
        if self.direct_max_bytes is not None and self._direct_held() > self.direct_max_bytes:
            self._drop_direct()  # of a mine that had more room
        if n_rows >= 2**31:
            raise ValueError(f"n_transactions={n_rows:,} exceeds int32 max: the count arrays are int32")
        n_words = (n_rows + 63) // 64
        if ld < n_words:
            raise ValueError(f"bitvecs has {ld} words per column, fewer than ceil({n_rows}/64)")
        mc = mining_min_count(min_support, n_rows)
        prune, infer = bool(prune_equal_support), bool(use_generator_pruning) and not prune_equal_support
        track_free = prune or bool(use_generator_pruning)
        n_logical = n_cols if n_cols_logical is None else n_cols_logical
        max_k = min(max_length if max_length else n_logical, n_logical)
        t0 = time.perf_counter()
        # A mine that starts small is done in one launch, K=1 included, or as far as its levels stay small.
        first = None
        if resume is None and not occupancy and n_cols and n_words and self._direct_ok(max_k):
            counts_d = self._column_counts(ptr, n_cols, n_words, ld)
            first = self._mine_direct(ptr, ld, n_words, n_cols, n_rows, mc, prune, max_k, col_counts=counts_d,
                                      turn=self.by_support, max_vram_gb=max_vram_gb)
            if first is not None and first[1] is None:
                first = None
        if first is not None:
            t_first = (time.perf_counter() - t0) * 1e3 / (1 + len(first[2]))
            host_rows, host_counts = first[4]
            ng = len(first[1][0])
            gen_cols, gen_counts = host_rows[:ng].astype(np.int64), host_counts[:ng].astype(np.int64)
        else:
            col_counts = self.column_counts(ptr, n_cols, n_words, ld) if n_cols else np.zeros(0, np.int64)
            freq = np.flatnonzero(col_counts >= mc)
            gen_cols = freq[col_counts[freq] < n_rows] if prune else freq
            gen_counts = col_counts[gen_cols].astype(np.int64)
            t_first = (time.perf_counter() - t0) * 1e3
        r_k = int(resume[0]) if resume is not None else 0
        if resume is not None:
            out = MineOutput(n_rows, mc, gen_cols.astype(np.int64), np.zeros(0, np.int64), np.zeros(0, np.int64))
        else:
            out = MineOutput(n_rows, mc, gen_cols.astype(np.int64), gen_cols.astype(np.int64), gen_counts)
        out.stats.append(LevelStats(1, n_cols, len(gen_cols), t_first))
        #: The level stats of the latest mine (the same list as its MineOutput's).
        self.last_stats = out.stats
        if level_callback and resume is None:
            level_callback(1, n_cols, len(gen_cols), out.stats[-1].ms)
        if on_level is not None and resume is None and len(gen_cols):
            on_level(1, gen_cols[:, None].astype(np.int64), gen_counts)

        def leave_order() -> None:
            """The mine goes on in the columns' order, so that it holds each level once and not in both."""
            nonlocal order, fbv, gen, new, d2, d3
            gen = new = d2 = d3 = self._prefix_level = self._deep = None
            for i, lv in enumerate(hist):
                if i == 0 and lv is not None:
                    hist[i] = Level(lv.rows, counts_c, (counts_c < n_rows).to(torch.uint8), True)
                elif lv is not None:
                    hist[i] = out.levels[i - 1] if keep_levels else self._named_level(lv, order)
                    hist[i].counted = True
            order = fbv = self._xt = self._xt_key = None
            fbv = self.gather(ptr, ld, gen_cols, n_words)[0]

        def over_vram(held: list) -> bool:
            """Whether the mine holds too much device memory, the direct launches' buffers given back if that helps."""
            if max_vram_gb is not None and held[1] > max_vram_gb:
                held[1] -= self._drop_direct()
            return max_vram_gb is not None and held[1] > max_vram_gb

        def flag(levels: list[Level], prev: Level | None) -> None:
            """The free flags of returned levels one after another in memory (``prev``: the level before them in the same
            order, None for level 1)."""
            if not flagged or levels[0].free is not None:
                return
            n = [lv.n for lv in levels]
            if not sum(n):
                return
            if prune:
                free = torch.ones(sum(n), dtype=torch.uint8, device=self.device)
            else:
                prev = prev or Level(None, hist[0].counts if order is None else counts_c)
                free, sizes = torch.empty(sum(n), dtype=torch.uint8, device=self.device), np.array(n, np.int64)
                check(self.lib.etm_level_flags(_p(levels[0].rows), _p(levels[0].counts), sizes.ctypes.data, len(n), levels[0].k,
                                               _p(prev.rows), _p(prev.counts), len(prev.counts), _p(free), _stream()),
                      "etm_level_flags")
                self.launches += 1
            for lv, f in zip(levels, free.split(n)):
                lv.free = f

        def emit(k: int, new: Level, stats: LevelStats, held: list | None = None, ordered: Level | None = None) -> Level:
            """A final level: its stats, callbacks, memory guards and place in the output, in the columns' order
            (``ordered``: the level in that order, its totals taken; ``held``: the guards' readings). Returns the level
            to go on from."""
            nonlocal named
            go_on, prev = new, named
            if ordered is not None:
                new = named = ordered
                renumbered.append(stats)
            elif order is not None:
                if named is not None and k > 2:
                    # The candidates and groups of the columns' order, from the level before in that order.
                    check(self.lib.etm_group_totals(_p(named.rows), named.n, named.k, _p(totals[k]), _stream()),
                          "etm_group_totals")
                    self.launches += 1
                    renumbered.append(stats)
                new = named = self._named_level(new, order)
                flag([new], prev)
            if level_callback and renumbered and renumbered[-1] is stats:
                stats.n_candidates, stats.n_groups = (int(x) for x in totals[k].cpu())
            out.stats.append(stats)
            n = stats.n_frequent
            if level_callback:
                level_callback(k, stats.n_candidates, n, stats.ms)
            if max_ram_gb is not None or max_vram_gb is not None:
                held = held or [host_rss_gb(), _allocated_gb(self.device)]
                if over_vram(held) and order is not None:
                    go_on = new
                    leave_order()
                    go_on.counted = True
                    held[1] = _allocated_gb(self.device)
                check_memory_guard(k, *held, max_ram_gb, max_vram_gb)
            if n and on_level is not None:
                on_level(k, out.gen_cols[new.rows.cpu().numpy()], new.counts.cpu().numpy().astype(np.int64))
            if n and keep_levels:
                out.levels.append(new)
            return go_on

        def emit_direct(k: int, levels: list[Level], seen, ms: float) -> None:
            ordered = (self._named_levels(levels, order, named, totals) if order is not None and levels
                       and named is not None and named.k == k - 1 else [None] * len(levels))
            if levels:
                if ordered[0] is not None:
                    flag(ordered, named)
                elif order is None:
                    flag(levels, None if hist[-1].rows is None else hist[-1])
            # One launch made the levels: after each of them the mine would hold what it holds now without the ones past
            # it. One reading does for all of them where nothing of the caller's runs between.
            guarded = max_ram_gb is not None or max_vram_gb is not None
            rows_of = [lv.n for lv in levels]
            size = guarded and [4 * n * (k + i + 1) * (1 if ordered[0] is None else 2) / (1 << 30)
                                for i, n in enumerate(rows_of)]
            held = None
            for i, n in enumerate(rows_of):
                if guarded:
                    if held is None or on_level is not None or level_callback:
                        held = [host_rss_gb(), _allocated_gb(self.device) - sum(size[i:])]
                    held[1] += size[i]
                    if over_vram(held) and order is not None and ordered[i] is not None:
                        level, levels[:] = None, ordered  # nothing of the launch's own stays
                        leave_order()
                        size = [x / 2 for x in size]
                        held[1] = _allocated_gb(self.device) - sum(size[i + 1:])
                level = emit(k + i, levels[i], LevelStats(k + i, seen[i][0], n, ms, seen[i][1], 1), held, ordered[i])
                level.counted = True
                if n:
                    hist.append(level)
                if len(hist) > 4:
                    hist[-5] = None

        ng = len(gen_cols)
        order = named = None  # the order of the generators while counting; the latest level in the columns' order
        flagged = track_free and free_flags and keep_levels
        renumbered = []  # the stats of the levels whose candidates and groups in the columns' order are among the totals
        #: Complete levels 1, 2, ... (under inference without the free-set prune: every frequent set).
        hist: list[Level | None] = []
        if first is not None:
            hist.append(Level(None, first[1][1]))
            emit_direct(2, first[2], first[3], t_first)
            if first[0]:
                if keep_levels and first[5]:
                    out.host = (host_rows[ng:], host_counts[ng:])
                return out
        if ng < 2 or max_k < max(2, r_k + 1):
            return out
        if rows is not None:
            lens = rows[2]
            # The rows' pairs, given or from their lengths.
            pair_work = (float(lens) if np.ndim(lens) == 0 else
                         float((lens.astype(np.float64) * (lens - 1) / 2).sum()))
            k2_by_rows = (resume is None and self.k2_rows_max_r > 0 and
                          pair_work / max(1.0, ng * (ng - 1) / 2 * n_words) < self.k2_rows_max_r)
        if self.by_support and resume is None and not occupancy and self._form_ok(max_k) and (
                len(hist) == 2 or (not hist[1:] and not (rows is not None and k2_by_rows)
                                   and ng * (ng - 1) // 2 * n_words >= ORDER_WORDS)):
            by_support = np.argsort(gen_counts, kind="stable")
            gen_counts = gen_counts[by_support]
        else:
            by_support = None
        # What the levels need of the generators, in one copy: the levels' totals, the order and its inverse (place),
        # columns, numbers, counts (those in the columns' order too) and free flags (a copy each, and the kernels to make
        # these there, took 0.2 ms a mine).
        n_tot = 4 * (DIRECT_LEVELS + 2)
        n_at = n_tot + 6 * ng
        packed = np.zeros(n_at + (ng + 3) // 4, np.int32)
        order_h, place_h, cols_h, iota_h, counts_h, counts_ch = packed[n_tot:n_at].reshape(6, ng)
        iota_h[:] = np.arange(ng)
        order_h[:] = iota_h if by_support is None else by_support
        place_h[order_h] = iota_h
        cols_h[:] = gen_cols[order_h]
        counts_h[:] = gen_counts
        counts_ch[order_h] = gen_counts
        packed[n_at:].view(np.uint8)[:ng] = gen_counts < n_rows
        packed = self._to_device(packed)
        order_d, place, cols_d, iota, counts1, counts_c = packed[n_tot:n_at].view(6, ng).unbind()
        if by_support is not None:
            order = order_d
            totals = packed[:n_tot].view(torch.int64).view(DIRECT_LEVELS + 2, 2)
        fbv, ldp = self.gather(ptr, ld, gen_cols, n_words, cols_d)
        if occupancy:
            self._occ = self.tile_occupancy(fbv, ldp, n_words)
        # The row-wise kernels take a row's items in the columns' order.
        if rows is not None and order is None:
            rp, cl, lens = rows[:3]
            lut = torch.full((max(1, n_cols),), -1, dtype=torch.int32, device=self.device)
            lut[torch.from_numpy(gen_cols.astype(np.int64)).to(self.device)] = torch.arange(
                ng, dtype=torch.int32, device=self.device)
            if len(rows) > 3:
                # The entries hold codes and rows[3] their columns (-1 for none): compose code -> generator.
                col_of = rows[3]
                lut = torch.where(col_of >= 0, lut[col_of.clamp(min=0).long()], col_of).contiguous()
            self._rows_input = dict(rp=rp, cl=cl, nnz=int(cl.numel()), lut=lut, n_r=int(rp.numel()) - 1,
                                    pair_work=pair_work, ng=ng)
            if k2_by_rows:
                self._k2_rows = (rp, cl, int(cl.numel()), lut, int(rp.numel()) - 1)
        direct = False  # whether the next level may be small: not the one a direct launch has just stopped before
        if resume is None:
            level1 = Level(iota[:, None], counts1, packed[n_at:].view(torch.uint8)[:ng], True)
            if hist:
                hist[0] = level1
                if order is not None and len(hist) == 2:
                    # Level 2 is there in the columns' order: on from it in the order of the generators.
                    named = hist[1]
                    hist[1] = self._named_level(named, place)
                    hist[1].counted = True
                    direct = True
                gen = hist[-1]
                if track_free and len(hist) > 1 and gen.free is None:
                    gen.free = self._free_of(hist, prune)
            else:
                hist.append(level1)
                gen = level1
            k = len(hist) + 1
        else:
            cols_r = np.asarray(resume[1], np.int64)
            counts_r = np.asarray(resume[2], np.int64)
            gidx = np.searchsorted(gen_cols, cols_r)
            if cols_r.size and (gidx.max() >= ng or (gen_cols[np.minimum(gidx, ng - 1)] != cols_r).any()):
                raise ValueError(f"the level-{r_k} itemsets to resume from hold items that are not frequent here")
            lex = np.lexsort(gidx.T[::-1]) if gidx.size else np.zeros(0, np.int64)
            gen = Level(torch.from_numpy(np.ascontiguousarray(gidx[lex], dtype=np.int32)).to(self.device),
                        torch.from_numpy(counts_r[lex].astype(np.int32)).to(self.device), None)
            hist = [None] * (r_k - 1) + [gen]  # levels 1..k-1 are not at hand: no bounds until three follow
            k = r_k + 1
            direct = True
        most = False  # whether the mine's direct launches have the most memory, and go on on projected columns
        while k <= max_k and gen.n >= k:
            if direct and 3 <= k <= DIRECT_LEVELS - 2 and self._direct_ok(max_k) and (
                    gen.n <= DIRECT_ROWS * (DIRECT_MOST if most else direct_scale(ng, n_words))):
                t_level = time.perf_counter()
                rest = self._mine_direct(_p(fbv), ldp, n_words + n_words % 2, ng, n_rows, mc, prune, max_k, start=gen,
                                         scale=DIRECT_MOST if most else None, projected=most, max_vram_gb=max_vram_gb)
                full = rest is not None and rest[6] and direct_bytes(
                    DIRECT_MOST, self._direct_cands(DIRECT_MOST), ng, n_words + n_words % 2,
                    self._direct_proj(ng, n_words + n_words % 2)) <= self._direct_room(max_vram_gb)
                if rest is not None and (rest[0] or rest[2]):
                    emit_direct(k, rest[2], rest[3], (time.perf_counter() - t_level) * 1e3 / max(1, len(rest[2])))
                    if rest[0]:
                        break
                    gen = hist[-1]
                    k += len(rest[2])
                    if track_free and gen.free is None:
                        gen.free = self._free_of(hist, prune)
                if full and (not most or rest[2]) and "direct_proj" in self.scratch.bufs:
                    most = True
                    continue
                most = False
            t_level = time.perf_counter()
            # Levels k-2 and k-3 for the deduction bounds of level k (k >= 3), when both are at hand.
            d2 = hist[k - 3] if k >= 3 else None
            d3 = hist[k - 4] if k >= 4 else None
            self._prefix_level = d2
            self._deep = (d2, d3, n_rows) if d2 is not None and (k == 3 or d3 is not None) else None
            # The first resumed level has no free flags: inference waits one level.
            level_infer = infer and gen.free is not None
            new, stats = self.count_level(gen, fbv, ldp, n_words, mc, level_infer, prune, n_rows)
            new = self.finish_level(new, gen, track_free, prune)
            stats.n_frequent = new.n
            stats.ms = (time.perf_counter() - t_level) * 1e3
            new = emit(k, new, stats)
            if new.n == 0:
                break
            hist.append(new)
            if len(hist) > 4:
                hist[-5] = None  # the bounds read at most three levels back
            gen = new
            if track_free and gen.free is None:
                gen.free = self._free_of(hist, prune)
            k += 1
            direct = True
        if renumbered and not level_callback:
            seen = totals.cpu().numpy()
            for stats in renumbered:
                stats.n_candidates, stats.n_groups = int(seen[stats.k, 0]), int(seen[stats.k, 1])
        self._deep = self._prefix_level = None
        self._xt, self._xt_key = None, None
        self._occ = None
        return out


def mine(bitvecs, n_rows: int, min_support: float, max_length: int | None = None, **kw) -> MineOutput:
    """Mine device bitvectors [n_cols, ceil(N/64)] with a fresh ``Engine`` (see ``Engine.mine``)."""
    engine_kw = {k: kw.pop(k) for k in ("method", "form", "chunk_cands", "small_group", "device", "project",
                                        "proj_density", "proj_bytes", "tc_elem", "pipeline", "autotune", "fused",
                                        "deduction_bounds", "proj_rows") if k in kw}
    return Engine(**engine_kw).mine(bitvecs, n_rows, min_support, max_length, **kw)
