"""The calls a user of this package makes, over the range they are made in: whole mines through ``apriori`` and
``Engine.mine``, from a few thousand rows to the full dense and deep sparse workloads.

A case is one mining call. ``call`` says which:

* ``bitvecs``       ``apriori(bitvecs=(array, col_to_item, N))``: resident column bitvectors in, the frame out;
* ``transactions``  ``apriori(csr, use_gpu=True)``: a transaction list on the host in, the frame out;
* ``mine``          ``Engine.mine`` on resident bitvectors by an engine the program keeps, levels left on the device
                    (the serving loop's call).

``data`` says what the transactions look like (sizes and laws of the repository's workloads): ``zipf`` (a shop's
baskets: 1 + Poisson(8) draws by a Zipf(1.1) popularity), ``wide`` (log-normal lengths, Zipf(1.0) over a wide
vocabulary), ``dense`` (independent items, p ~ Beta(2, 30)), ``patterns`` (planted patterns and noise).
"""

from __future__ import annotations

import math
from fractions import Fraction
from types import SimpleNamespace

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.package()

#: Most rows for which ``exact`` mines the case again in plain torch.
EXACT_ROWS = 130_000


def _case(name, call, data, rows, items, support, length, **kw):
    c = dict(name=name, call=call, data=data, rows=rows, items=items, support=support, length=length, prune=False,
             infer=False, keep_engine=call == "mine", order="ascending", ids="int64")
    c.update(kw)
    return c


def listed():
    return [
        # One interactive call on a small table: what counts is latency and the number of launches.
        _case("call_tiny", "bitvecs", "zipf", 2_000, 100, 0.05, 4),
        # The smallest resident dataset of the serving set, with an engine kept between calls.
        _case("mine_small", "mine", "zipf", 10_000, 500, 0.01, 8),
        # Free itemsets of an odd-sized table.
        _case("call_free_odd", "bitvecs", "zipf", 33_333, 1_111, 0.004, 0, prune=True),
        # The plain transactions workload: 60,000 baskets from the host, every length.
        _case("transactions_60k", "transactions", "zipf", 60_000, 1_000, 0.01, 0, keep_engine=True),
        # A wide vocabulary from the host, at the workload's support.
        _case("transactions_wide", "transactions", "wide", 1_000_000, 50_000, 0.004, 0),
        # The same kind of input at a low support, its rows in the order they were recorded (not sorted) and
        # its ids unsigned: thousands of frequent items, few rows holding each.
        _case("transactions_low", "transactions", "wide", 400_000, 20_000, 0.0008, 4, order="recorded", ids="uint64"),
        # Deep itemsets from the host, counts inferred from generators.
        _case("transactions_deep", "transactions", "patterns", 2_000_000, 2_000, 0.005, 16, infer=True,
              keep_engine=True),
        # A serving request on a large resident dataset.
        _case("mine_serving", "mine", "zipf", 1_000_001, 6_000, 0.003, 6),
        # Dense pairs and triples whose result is copied back whole, ragged in rows and items.
        _case("call_dense_odd", "bitvecs", "dense", 300_007, 1_255, 0.003, 3),
        # The dense workload at its middle size.
        _case("mine_dense_mid", "mine", "dense", 1_000_000, 2_048, 0.002, 3),
        # The dense workload at full size: the benchmark's headline.
        _case("mine_dense", "mine", "dense", 2_000_000, 4_096, 0.002, 3),
        # The deep sparse workload at full size.
        _case("mine_deep", "mine", "patterns", 20_000_000, 2_000, 0.005, 16, infer=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choice(["bitvecs", "transactions", "mine"])
    data = rng.choice(["zipf", "wide", "patterns"] if call == "transactions" else ["zipf", "dense", "patterns"])
    if data == "zipf":
        rows, items, support, length = _log(rng, 2_000, 2_000_000), _log(rng, 100, 20_000), _log(rng, 0.003, 0.05), 0
        length = rng.choice([0, 2, 3, 4, 5, 6, 7, 8])
    elif data == "wide":
        rows, items, support = _log(rng, 20_000, 1_000_000), _log(rng, 2_000, 50_000), _log(rng, 0.001, 0.01)
        length = rng.choice([0, 3, 4])
    elif data == "dense":
        rows, items, support = _log(rng, 20_000, 2_000_000), _log(rng, 100, 4_096), _log(rng, 0.002, 0.02)
        length = rng.choice([2, 3, 3])
        if call == "bitvecs":  # the frame of a call is copied to the host: results of a few gigabytes at most
            items = min(items, 1_500)
    else:
        rows, items, support, length = _log(rng, 50_000, 20_000_000), 2_000, _log(rng, 0.005, 0.02), 16
        if call == "transactions":
            rows = min(rows, 2_000_000)
    option = rng.choice(["none", "none", "prune", "infer"])
    recorded = call == "transactions" and rng.random() < 0.3
    return dict(call=call, data=data, rows=int(rows) | 1, items=int(items), support=round(support, 5), length=length,
                prune=option == "prune", infer=option == "infer", keep_engine=call == "mine" or rng.random() < 0.5,
                order="recorded" if recorded else "ascending",
                ids="uint64" if call == "transactions" and rng.random() < 0.2 else "int64")


# ---- inputs ------------------------------------------------------------------------------------------------------
#
# A case is one table: its lattice, and so the size of a call's result, belongs to the case. The seed deals it out
# anew: which column (or id) each item gets, and the order of the transactions.

TABLE_SEED = 12345


def _popularity(case):
    """P(a draw is item i), i = 0 .. items - 1: a Zipf law by rank."""
    w = np.arange(1, case["items"] + 1, dtype=np.float64) ** (-1.1 if case["data"] == "zipf" else -1.0)
    return w / w.sum()


def _dense_probs(case):
    return pkg.synthetic.dense_k2_probs(case["items"], seed=0)


def _deal(n, seed, what):
    gen = torch.Generator(device="cuda").manual_seed(2 * seed + what)
    return torch.randperm(n, device="cuda", generator=gen)


def _drawn_rows(case, seed):
    """(rows, items) of every entry on the device, by row then item, repeats within a row dropped."""
    gen = torch.Generator(device="cuda").manual_seed(TABLE_SEED)
    n, m = case["rows"], case["items"]
    if case["data"] == "zipf":
        lens = 1 + torch.poisson(torch.full((n,), 8.0, device="cuda"), generator=gen).long()
    else:
        normal = torch.randn(n, device="cuda", generator=gen)
        lens = (normal * 1.2 + math.log(8.0)).exp().round().clamp(1, 500).long()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    cdf = torch.from_numpy(np.cumsum(_popularity(case))).cuda()
    u = torch.rand(row.numel(), device="cuda", generator=gen, dtype=torch.float64)
    item = torch.searchsorted(cdf, u * cdf[-1], right=True).clamp(max=m - 1)
    key = torch.unique(_deal(n, seed, 0)[row] * m + _deal(m, seed, 1)[item])
    return key // m, key % m


def _made_bits(case, seed):
    """Column bitvectors of the hash-defined data, its columns and its whole words of transactions dealt out."""
    lib = pkg.load_library()
    n, m = case["rows"], case["items"]
    if case["data"] == "patterns":
        spec = pkg.synthetic.pattern_spec(n_items=m, hash_seed=TABLE_SEED)
        bits = pkg.synthetic.patterns_bitvecs_device(lib, spec, n).view(torch.int64)
    else:
        thr = torch.from_numpy(pkg.synthetic.bernoulli_thresholds(_dense_probs(case)).view(np.int64)).cuda()
        bits = torch.empty((m, -(-n // 64)), dtype=torch.int64, device="cuda")
        if lib.etm_synth_bernoulli(thr.data_ptr(), m, n, TABLE_SEED, bits.data_ptr(), bits.shape[1],
                                   torch.cuda.current_stream().cuda_stream) != 0:
            raise RuntimeError("etm_synth_bernoulli failed")
    bits = bits[_deal(m, seed, 1)]
    turn = seed % max(1, n // 64)
    return torch.cat([bits[:, turn:n // 64], bits[:, :turn], bits[:, n // 64:]], dim=1)


def _bits(case, seed):
    """Column bitvectors int64 [items, ceil(rows / 64)]."""
    if case["data"] in ("dense", "patterns"):
        return _made_bits(case, seed)
    row, item = _drawn_rows(case, seed)
    words = -(-case["rows"] // 64)
    bits = torch.zeros(case["items"] * words, dtype=torch.int64, device="cuda")
    # Every (row, item) is there once: adding the bits of a word sets them.
    bits.scatter_add_(0, item * words + (row >> 6), torch.ones_like(row) << (row & 63))
    return bits.view(case["items"], words)


def _entries(case, seed):
    """(rows, items) of every entry on the device, by row then item."""
    if case["data"] != "patterns":
        return _drawn_rows(case, seed)
    bits = _made_bits(case, seed)
    at = bits.view(-1).nonzero().view(-1)
    item, word = at // bits.shape[1], at % bits.shape[1]
    hit, bit = ((bits.view(-1)[at][:, None] >> torch.arange(64, device="cuda")) & 1).nonzero(as_tuple=True)
    key = torch.sort((word[hit] * 64 + bit) * case["items"] + item[hit]).values
    return key // case["items"], key % case["items"]


def prepare(case, seed):
    engine = pkg.Engine() if case["keep_engine"] else None
    if case["call"] != "transactions":
        bits = _bits(case, seed).view(torch.uint64)
        return dict(case=case, bits=bits, items={c: 3 * c + 11 for c in range(case["items"])}, engine=engine)
    row, item = _entries(case, seed)
    if case["order"] == "recorded":
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        item = item[torch.argsort(row * (1 << 22) + torch.randint(0, 1 << 22, row.shape, device="cuda", generator=gen))]
    ids = (item * 5 + 100).cpu().numpy().astype(case["ids"])
    indptr = np.zeros(case["rows"] + 1, np.int64)
    indptr[1:] = torch.bincount(row, minlength=case["rows"]).cumsum(0).cpu().numpy()
    return dict(case=case, csr=SimpleNamespace(indptr=indptr, items=ids), engine=engine)


def run(state):
    case = state["case"]
    options = dict(prune_equal_support=case["prune"], use_generator_pruning=case["infer"])
    length = case["length"] or None
    if case["call"] == "mine":
        out = state["engine"].mine(state["bits"], case["rows"], case["support"], length, **options)
        got = {"items": out.level1_cols, "counts": out.level1_counts, "generators": out.gen_cols}
        for level in out.levels:
            got["rows%d" % level.k], got["counts%d" % level.k] = level.rows, level.counts
        return got
    if case["call"] == "bitvecs":
        frame = pkg.apriori(bitvecs=(state["bits"], state["items"], case["rows"]), min_support=case["support"],
                            max_length=length, warn_complexity=False, engine=state["engine"], **options)
    else:
        frame = pkg.apriori(state["csr"], use_gpu=True, min_support=case["support"], max_length=length,
                            warn_complexity=False, engine=state["engine"], **options)
    return {"offsets": frame.offsets, "values": frame.values.view(np.int64), "support": frame.support}


def work(case):
    """The input read once and, for the counting, two operations for every transaction of every pair of frequent
    items (and, of the dense data, of every pair of an item's more frequent partners within its transactions)."""
    n = float(case["rows"])
    if case["data"] == "dense":
        p = _dense_probs(case)
        entries = p.sum() * n
    elif case["data"] == "patterns":
        entries = 11.0 * n
        p = np.full(int(423 * 0.005 / case["support"]), 1.0)  # the frequent items of the pattern pool, about
    else:
        draws = 9.0 if case["data"] == "zipf" else 16.0
        p = 1.0 - np.exp(-draws * _popularity(case))
        entries = p.sum() * n
    s = case["support"]
    p = np.sort(p[p >= s])
    flops = len(p) * (len(p) - 1.0) * n
    if case["data"] == "dense" and case["length"] >= 3:
        partners = len(p) - np.maximum(np.searchsorted(p, s / p), np.arange(1, len(p) + 1))
        flops += float((partners * (partners - 1.0) * p).sum()) * n
    size = entries * 8 + n * 8 if case["call"] == "transactions" else case["items"] * n / 8
    return {"bytes": float(size), "flops": float(flops)}


# ---- the same mine in 64 bits ------------------------------------------------------------------------------------

def _levels64(x, n_rows, mc, longest, free_only):
    """Frequent itemsets of the 0/1 matrix x [items, rows] level by level, in lexicographic order: (itemsets of
    column indices, counts); the free ones alone under ``free_only``."""
    counts = x.sum(1).tolist()
    cols = [c for c, v in enumerate(counts) if v >= mc and (v < n_rows or not free_only)]
    level = [((c,), int(counts[c])) for c in cols]
    k = 1
    while level:
        yield level
        if k >= longest:
            return
        known = dict(level)
        groups = {}
        for itemset, _ in level:
            groups.setdefault(itemset[:-1], []).append(itemset[-1])
        level = []
        for prefix, last in groups.items():
            if len(last) < 2:
                continue
            y = x[last]
            if prefix:
                y = y[:, x[list(prefix)].all(0)]
            y = y.double()
            pair = (y @ y.T).cpu().numpy()
            for i, j in zip(*np.nonzero(np.triu(pair >= mc, 1))):
                itemset, c = prefix + (last[i], last[j]), int(pair[i, j])
                if free_only:
                    below = [known.get(itemset[:d] + itemset[d + 1:]) for d in range(k + 1)]
                    if any(b is None or b == c for b in below):
                        continue
                level.append((itemset, c))
        k += 1


def exact(case, seed):
    if case["rows"] > EXACT_ROWS or case["call"] == "mine" or case["rows"] * case["items"] > 4e8:
        return None  # of ``mine`` every output is a whole number
    n = case["rows"]
    if case["call"] == "bitvecs":
        bits, ids = _bits(case, seed), 3 * np.arange(case["items"]) + 11
        x = ((bits[:, :, None] >> torch.arange(64, device="cuda")) & 1).bool().view(case["items"], -1)[:, :n]
    else:
        row, item = _entries(case, seed)
        ids = 5 * np.arange(case["items"]) + 100
        x = torch.zeros((case["items"], n), dtype=torch.bool, device="cuda")
        x[item, row] = True
    mc = max(1, math.ceil(Fraction(str(case["support"])) * n))
    offsets, values, support = [0], [], []
    for level in _levels64(x, n, mc, case["length"] or case["items"], case["prune"]):
        for itemset, c in level:
            values.extend(itemset)
            offsets.append(len(values))
            support.append(c)
    return {"offsets": np.array(offsets, np.int64), "values": ids[np.array(values, np.int64)],
            "support": np.array(support, np.float64) / n}
