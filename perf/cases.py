"""Timed cases: the work a clustering or search program has this package do.

Every case is one pass through public entry points -- the clustkit-named
Python functions, ``search_batch`` over a ``DeviceDatabase``, or the C ABI of
``libckgpu.so`` on resident tensors, as INTEGRATION.md wires them.  The sizes
are those of the benchmark's workloads (2,000 / 50,000 / 20,000 / 1,000,000
sequences, a resident search database) or a fraction that keeps a pass within
some tens of milliseconds; ``draw`` spreads them over the whole range.

Sequences are synthetic protein families, generated on the GPU from the seed:
lognormal or Pareto lengths, residues and substitutions from the frequencies
BLOSUM62 implies (``clustkit_gb300.synth``), 10-70 % divergence within a
family, indels of geometric length (mean 3) at 0.05 a residue.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from clustkit_gb300 import _lib, graph, lsh, pairwise, search, synth
from clustkit_gb300.blosum import BLOSUM62

DEV = "cuda"
SUB = np.ascontiguousarray(BLOSUM62, np.int8)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # Align of a small protein set (200 families of 10) through clustkit's own Python function on host
        # arrays, at its default band width: the smallest clustering run, where launches and copies count.
        {"name": "align_small", "kind": "align_host", "families": 200, "median": 300, "lo": 50, "hi": 800,
         "pairs": 12000, "within": 0.75, "band": 50, "threshold": 0.5},
        # Align at clustering scale: 50,000 sequences, the pairs that LSH and the Jaccard pre-filter leave.
        {"name": "align_cluster", "kind": "align", "families": 5000, "median": 350, "lo": 30, "hi": 2000,
         "dist": "lognormal", "pairs": 700000, "within": 0.32, "ratio": 0.0, "band": 100, "threshold": 0.3},
        # Align of heavy-tailed lengths (30 to 8,000) in a narrow band.
        {"name": "align_uneven", "kind": "align", "families": 2000, "median": 300, "lo": 30, "hi": 8000,
         "dist": "pareto", "pairs": 500000, "within": 0.5, "ratio": 0.5, "band": 32, "threshold": 0.3},
        # MinHash sketches of a resident protein set, at clustkit's default k and sketch size.
        {"name": "sketch", "kind": "sketch", "families": 20000, "median": 300, "lo": 30, "hi": 1500, "k": 5,
         "size": 128, "alphabet": 20},
        # The Jaccard pre-filter over LSH candidates (most of them chance collisions).
        {"name": "jaccard", "kind": "jaccard", "families": 10000, "median": 300, "lo": 30, "hi": 1500, "k": 5,
         "size": 128, "pairs": 4000000, "within": 0.11, "threshold": 0.4},
        # LSH candidates at threshold 0.4, high sensitivity: one band, 448 tables.
        {"name": "lsh", "kind": "lsh", "families": 10000, "median": 300, "lo": 30, "hi": 1500, "k": 5, "size": 128,
         "tables": 448, "bands": 1},
        # Building the k-mer index of a search database (with its compact target list).
        {"name": "index", "kind": "index", "families": 10000, "median": 350, "lo": 30, "hi": 2000, "k": 5},
        # One query, answered alone: exact 5-mers, then banded SW of its candidates.
        {"name": "search_one", "kind": "search", "families": 20000, "queries": 1, "mode": "exact", "cands": 500},
        # A serving batch: exact 5-mers.
        {"name": "search_exact", "kind": "search", "families": 20000, "queries": 64, "mode": "exact", "cands": 500},
        # A serving batch in clustkit's default mode: BLOSUM62-similar 5-mers at threshold 13.
        {"name": "search_similar", "kind": "search", "families": 20000, "queries": 64, "mode": "similar",
         "cands": 500},
        # A whole call in clustkit's C-path mode (Phase B, hinted SW at band 50): query list in, ranked hits out.
        {"name": "search_call", "kind": "search_call", "families": 20000, "queries": 64, "cands": 500, "top_k": 10},
        # After Align: the similarity graph of the passing pairs and its connected components.
        {"name": "graph", "kind": "graph", "families": 10000, "pairs": 250000, "within": 0.97},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["align_host", "align", "align", "sketch", "jaccard", "lsh", "index", "search", "search",
                       "search_call", "graph"])
    if kind == "align_host":
        fam = _log(rng, 20, 600)
        return {"kind": kind, "families": fam, "median": rng.randint(120, 400), "lo": 30, "hi": rng.randint(600, 2000),
                "pairs": _log(rng, 300, 30000), "within": rng.uniform(0.3, 0.9),
                "band": rng.choice([20, 50, 77, 100]), "threshold": rng.choice([0.3, 0.4, 0.5, 0.7])}
    if kind == "align":
        pareto = rng.random() < 0.4
        return {"kind": kind, "families": _log(rng, 100, 5000), "median": rng.randint(150, 400), "lo": 30,
                "hi": rng.randint(3000, 8000) if pareto else rng.randint(800, 2000),
                "dist": "pareto" if pareto else "lognormal", "pairs": _log(rng, 500, 400000),
                "within": rng.uniform(0.2, 0.7), "ratio": rng.choice([0.0, 0.5]),
                "band": rng.choice([16, 32, 50, 64, 100, 117, 128]), "threshold": rng.choice([0.3, 0.4, 0.5])}
    if kind == "sketch":
        alphabet = rng.choice([20, 20, 4])
        return {"kind": kind, "families": _log(rng, 30, 15000), "median": rng.randint(100, 500), "lo": 20,
                "hi": rng.randint(1000, 4000), "k": rng.randint(3, 7) if alphabet == 20 else rng.randint(9, 21),
                "size": rng.choice([32, 64, 100, 128, 128, 200, 256, 500, 1000]), "alphabet": alphabet}
    if kind == "jaccard":
        return {"kind": kind, "families": _log(rng, 100, 10000), "median": rng.randint(100, 400), "lo": 30,
                "hi": 1500, "k": 5, "size": rng.choice([32, 64, 100, 128, 128, 200, 256]),
                "pairs": _log(rng, 2000, 1500000), "within": rng.uniform(0.05, 0.6),
                "threshold": rng.choice([0.3, 0.4, 0.5, 0.7])}
    if kind == "lsh":
        bands = rng.choice([1, 1, 2, 3])
        return {"kind": kind, "families": _log(rng, 100, 8000), "median": rng.randint(150, 400), "lo": 30, "hi": 1500,
                "k": 5, "size": rng.choice([64, 128, 256]), "tables": rng.randint(8, 448), "bands": bands}
    if kind == "index":
        return {"kind": kind, "families": _log(rng, 100, 10000), "median": rng.randint(150, 350), "lo": 30,
                "hi": 2000, "k": rng.choice([3, 4, 5, 5])}
    if kind == "search":
        return {"kind": kind, "families": _log(rng, 500, 20000), "queries": _log(rng, 1, 64),
                "mode": rng.choice(["exact", "similar", "cpath"]), "cands": rng.choice([200, 500, 1000])}
    if kind == "search_call":
        return {"kind": kind, "families": _log(rng, 500, 10000), "queries": _log(rng, 1, 64),
                "cands": rng.choice([200, 500]), "top_k": rng.choice([5, 10, 50])}
    fam = _log(rng, 50, 10000)
    return {"kind": "graph", "families": fam, "pairs": fam * rng.randint(5, 25), "within": rng.uniform(0.5, 1.0)}


# ------------------------------------------------------------------ sequences
PER_FAMILY = 10


@functools.lru_cache(maxsize=1)
def _cdfs():
    bg, cond = synth.substitution_cdf()
    cond = np.minimum(cond, 1.0)
    cond[:, -1] = 1.0
    flat = torch.from_numpy(cond + np.arange(20)[:, None]).reshape(-1)  # row a in (a, a + 1]
    return torch.from_numpy(np.ascontiguousarray(bg)).to(DEV), flat.to(DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _uniform(g, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64)


def _background(g, n):
    return torch.searchsorted(_cdfs()[0], _uniform(g, n)).clamp_(max=19)


def _lengths(g, n, median, lo, hi, dist):
    if dist == "pareto":
        x = lo * _uniform(g, n).clamp_(min=1e-9) ** (-1.0 / 1.5)
    else:
        x = median * torch.exp(0.5 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64))
    return x.round().clamp_(lo, hi).to(torch.int64)


def _starts(lengths):
    return torch.cumsum(lengths, 0) - lengths


def _families(g, n_fam, median, lo, hi, dist="lognormal", chunk=4000):
    """(flat uint8, offsets int64, lengths int32) of n_fam x PER_FAMILY sequences on the GPU, families contiguous."""
    flats, lens = [], []
    anc_all = _lengths(g, n_fam, median, lo, hi, dist)
    div_all = 0.1 + 0.6 * _uniform(g, n_fam)
    for f in range(0, n_fam, chunk):
        anc_len, div = anc_all[f:f + chunk], div_all[f:f + chunk]
        anc = _background(g, int(anc_len.sum()))
        fam = torch.arange(anc_len.numel(), device=DEV).repeat_interleave(PER_FAMILY)
        length = anc_len[fam]
        total = int(length.sum())
        start = _starts(length)
        seq = torch.arange(fam.numel(), device=DEV).repeat_interleave(length)
        res = anc[torch.arange(total, device=DEV) - start[seq] + _starts(anc_len)[fam][seq]]
        new = torch.searchsorted(_cdfs()[1], res + _uniform(g, total).clamp_(min=1e-12)) - 20 * res
        res = torch.where(_uniform(g, total) < div[fam][seq], new.clamp_(0, 19), res)
        # indels: runs dropped from an event on, or background residues put before it
        event = torch.nonzero(_uniform(g, total) < 0.05).reshape(-1)
        run = (torch.log(_uniform(g, event.numel()).clamp_(min=1e-9)) / math.log(2.0 / 3.0)).floor().to(torch.int64) + 1
        drop = _uniform(g, event.numel()) < 0.5
        d0, d1 = event[drop], torch.minimum(event[drop] + run[drop], (start + length)[seq[event[drop]]])
        edge = torch.zeros(total + 1, dtype=torch.int64, device=DEV)
        edge.index_add_(0, d0, torch.ones_like(d0))
        edge.index_add_(0, d1, -torch.ones_like(d1))
        copies = (torch.cumsum(edge[:-1], 0) == 0).to(torch.int64)
        copies[event[~drop]] += run[~drop]
        own = torch.cumsum(copies, 0) - 1  # the residue itself follows what is put before it
        kept = torch.cumsum(edge[:-1], 0) == 0
        out = _background(g, int(copies.sum()))
        out[own[kept]] = res[kept]
        out_seq = seq.repeat_interleave(copies)
        length = torch.bincount(out_seq, minlength=fam.numel())
        pos = torch.arange(out.numel(), device=DEV) - _starts(length)[out_seq]
        out = out[pos < hi]
        flats.append(out.to(torch.uint8))
        lens.append(length.clamp(max=hi))
    lengths = torch.cat(lens)
    return torch.cat(flats), _starts(lengths), lengths.to(torch.int32)


def _pairs(g, lengths, m, within, ratio=0.0):
    """m candidate pairs (i < j) in order of i: a share `within` families, the others of unrelated sequences."""
    n = lengths.numel()
    got = []
    for want, same in ((int(round(m * within)), True), (m - int(round(m * within)), False)):
        while want > 0:
            k = 2 * want + 1024
            i = torch.randint(0, n, (k,), generator=g, device=DEV)
            if same:
                step = torch.randint(1, PER_FAMILY, (k,), generator=g, device=DEV)
                j = i - i % PER_FAMILY + (i % PER_FAMILY + step) % PER_FAMILY
            else:
                j = torch.randint(0, n, (k,), generator=g, device=DEV)
            a, b = lengths[i].double(), lengths[j].double()
            ok = (i != j) & (torch.minimum(a, b) >= ratio * torch.maximum(a, b))
            p = torch.stack([torch.minimum(i, j), torch.maximum(i, j)], 1)[ok][:want]
            got.append(p)
            want -= p.shape[0]
    p = torch.cat(got)
    return p[torch.argsort(p[:, 0] * n + p[:, 1])].to(torch.int32).contiguous()


def _sketches(flat, off, length, k, size):
    out = torch.empty((length.numel(), size), dtype=torch.int64, device=DEV)
    _lib.check(_lib.load().ck_sketch_device(flat.data_ptr(), flat.numel(), off.data_ptr(), length.data_ptr(),
                                            length.numel(), k, size, 20, 42, out.data_ptr(), _stream()))
    return out


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _queries(g, flat, off, length, n):
    """n encoded queries (host): half mutated database members at 30-90 % identity, half background."""
    out = []
    want = _lengths(g, n, 300, 50, 2000, "lognormal").tolist()
    member = torch.randint(0, length.numel(), (n,), generator=g, device=DEV).tolist()
    identity = (0.3 + 0.6 * _uniform(g, n)).tolist()
    for q in range(n):
        if q % 2 == 0:
            o, size = int(off[member[q]]), int(length[member[q]])
            r = flat[o:o + size].to(torch.int64)
            new = torch.searchsorted(_cdfs()[1], r + _uniform(g, size).clamp_(min=1e-12)) - 20 * r
            r = torch.where(_uniform(g, size) < 1.0 - identity[q], new.clamp_(0, 19), r)
        else:
            r = _background(g, want[q])
        out.append(r.to(torch.uint8).cpu().numpy())
    return out


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return PREPARE[case["kind"]](case, _gen(seed))


def _prepare_align_host(c, g):
    flat, off, length = _families(g, c["families"], c["median"], c["lo"], c["hi"])
    pairs = _pairs(g, length, c["pairs"], c["within"])
    return {"case": c, "pairs": pairs.cpu().numpy(), "flat": flat.cpu().numpy(), "off": off.cpu().numpy(),
            "len": length.cpu().numpy(), "kept": np.zeros((c["pairs"], 2), np.int32),
            "sims": np.zeros(c["pairs"], np.float32)}


def _prepare_align(c, g):
    flat, off, length = _families(g, c["families"], c["median"], c["lo"], c["hi"], c["dist"])
    pairs = _pairs(g, length, c["pairs"], c["within"], c["ratio"])
    m = pairs.shape[0]
    buf = {"sims": torch.empty(m, dtype=torch.float32, device=DEV),
           "scores": torch.empty(m, dtype=torch.int32, device=DEV),
           "matches": torch.empty(m, dtype=torch.int32, device=DEV),
           "shorter": torch.empty(m, dtype=torch.int32, device=DEV),
           "mask": torch.empty(m, dtype=torch.uint8, device=DEV)}
    return {"case": c, "pairs": pairs, "flat": flat, "off": off, "len": length, "out": buf}


def _prepare_sketch(c, g):
    flat, off, length = _families(g, c["families"], c["median"], c["lo"], c["hi"])
    if c["alphabet"] == 4:
        flat = flat % 4
    out = torch.empty((length.numel(), c["size"]), dtype=torch.int64, device=DEV)
    return {"case": c, "flat": flat, "off": off, "len": length, "out": out}


def _prepare_jaccard(c, g):
    flat, off, length = _families(g, c["families"], c["median"], c["lo"], c["hi"])
    pairs = _pairs(g, length, c["pairs"], c["within"])
    return {"case": c, "pairs": pairs, "sk": _sketches(flat, off, length, c["k"], c["size"]),
            "sims": torch.empty(pairs.shape[0], dtype=torch.float32, device=DEV),
            "mask": torch.empty(pairs.shape[0], dtype=torch.uint8, device=DEV)}


def _prepare_lsh(c, g):
    flat, off, length = _families(g, c["families"], c["median"], c["lo"], c["hi"])
    return {"case": c, "sk": _sketches(flat, off, length, c["k"], c["size"]),
            "pairs": torch.zeros((_lsh_room(c), 2), dtype=torch.int32, device=DEV)}


def _lsh_room(c):
    return 400 * c["families"] * PER_FAMILY


def _prepare_index(c, g):
    flat, off, length = _families(g, c["families"], c["median"], c["lo"], c["hi"])
    nk = 20 ** c["k"]
    positions = int((length.to(torch.int64) - c["k"] + 1).clamp(min=0).sum())
    room = 2 * c["families"] * PER_FAMILY * c["median"]  # the same for every seed; the index fills the front
    assert positions <= room
    return {"case": c, "flat": flat, "off": off, "len": length, "positions": positions,
            "offsets": torch.empty(nk + 1, dtype=torch.int64, device=DEV),
            "freqs": torch.empty(nk, dtype=torch.int32, device=DEV),
            "entries": torch.zeros(room, dtype=torch.int64, device=DEV),
            "targets": torch.zeros(room, dtype=torch.int32, device=DEV),
            "total": np.zeros(1, np.int64)}


def _database(c, g):
    flat, off, length = _families(g, c["families"], 350, 30, 2000)
    queries = _queries(g, flat, off, length, c["queries"])
    db = search.DeviceDatabase(flat.cpu().numpy(), off.cpu().numpy(), length.cpu().numpy(), arena_slots=1,
                               arena_queries=64, arena_residues=64 * 2000)
    return db, queries


def _prepare_search(c, g):
    """A resident database, one batch of queries in pinned host memory, and the buffers of a search chain."""
    db, queries = _database(c, g)
    n, k = len(queries), c["cands"]
    sizes = np.array([len(q) for q in queries], np.int32)
    offs = (np.cumsum(sizes) - sizes).astype(np.int64) + db.arena_res0
    zeros = functools.partial(torch.zeros, device=DEV)
    return {"case": c, "db": db, "n": n, "longest": int(sizes.max()), "residues": int(sizes.sum()),
            "h_res": torch.from_numpy(np.concatenate(queries)).pin_memory(),
            "h_off": torch.from_numpy(offs).pin_memory(), "h_len": torch.from_numpy(sizes).pin_memory(),
            "targets": zeros(n * k, dtype=torch.int32), "counts": zeros(n * k, dtype=torch.int32),
            "diags": zeros(n * k, dtype=torch.int32), "found": zeros(n, dtype=torch.int32),
            "pairs": zeros((n * k, 2), dtype=torch.int32), "sims": zeros(n * k, dtype=torch.float32),
            "scores": zeros(n * k, dtype=torch.int32), "mask": zeros(n * k, dtype=torch.uint8)}


def _prepare_search_call(c, g):
    db, queries = _database(c, g)
    return {"case": c, "db": db, "queries": queries}


def _prepare_graph(c, g):
    n = c["families"] * PER_FAMILY
    pairs = torch.unique(_pairs(g, torch.full((n,), 300, device=DEV), 3 * c["pairs"], c["within"]), dim=0)
    keep = torch.randperm(pairs.shape[0], generator=g, device=DEV)[:c["pairs"]]
    pairs = pairs[torch.sort(keep)[0]].contiguous()
    sims = (0.4 + 0.6 * _uniform(g, pairs.shape[0])).to(torch.float32)
    return {"case": c, "n": n, "pairs": pairs, "sims": sims}


PREPARE = {"align_host": _prepare_align_host, "align": _prepare_align, "sketch": _prepare_sketch,
           "jaccard": _prepare_jaccard, "lsh": _prepare_lsh, "index": _prepare_index, "search": _prepare_search,
           "search_call": _prepare_search_call, "graph": _prepare_graph}


# ------------------------------------------------------------------ run
def run(state):
    return RUN[state["case"]["kind"]](state["case"], state)


def _run_align_host(c, s):
    pairs, sims = pairwise.compute_pairwise_alignment(s["pairs"], None, s["len"], c["threshold"],
                                                      band_width=c["band"], device="cpu", flat_sequences=s["flat"],
                                                      offsets=s["off"], use_sw=True, use_c_sw=True)
    s["kept"][:len(sims)] = pairs  # arrays of one size, whatever the seed
    s["sims"][:len(sims)] = sims
    return s["kept"], s["sims"], len(sims)


def _run_align(c, s):
    o = s["out"]
    _lib.check(_lib.load().ck_sw_batch_device(
        s["pairs"].data_ptr(), s["pairs"].shape[0], s["flat"].data_ptr(), s["flat"].numel(), s["off"].data_ptr(),
        s["len"].data_ptr(), s["len"].numel(), c["band"], SUB.ctypes.data, c["threshold"], None, _lib.PASS_CPU,
        _lib.ENGINE_BATCHED, o["sims"].data_ptr(), o["scores"].data_ptr(), o["matches"].data_ptr(),
        o["shorter"].data_ptr(), o["mask"].data_ptr(), _stream()))
    return o


def _run_sketch(c, s):
    _lib.check(_lib.load().ck_sketch_device(s["flat"].data_ptr(), s["flat"].numel(), s["off"].data_ptr(),
                                            s["len"].data_ptr(), s["len"].numel(), c["k"], c["size"], c["alphabet"],
                                            42, s["out"].data_ptr(), _stream()))
    return s["out"]


def _floor(c):
    return max(0.001, 0.3 * c["threshold"] ** 5)


def _run_jaccard(c, s):
    _lib.check(_lib.load().ck_jaccard_device(s["pairs"].data_ptr(), s["pairs"].shape[0], s["sk"].data_ptr(),
                                             s["sk"].shape[0], s["sk"].shape[1], _floor(c), s["sims"].data_ptr(),
                                             s["mask"].data_ptr(), _stream()))
    return s["sims"], s["mask"]


def _run_lsh(c, s):
    pairs = lsh.lsh_candidates_device(s["sk"], c["tables"], c["bands"])
    s["pairs"][:pairs.shape[0]] = pairs[:s["pairs"].shape[0]]
    return s["pairs"], pairs.shape[0]


def _run_index(c, s):
    lib = _lib.load()
    _lib.check(lib.ck_kmer_index_build_device(0, s["flat"].data_ptr(), s["flat"].numel(), s["off"].data_ptr(),
                                              s["len"].data_ptr(), s["len"].numel(), c["k"], 20,
                                              s["offsets"].data_ptr(), s["entries"].data_ptr(), s["positions"],
                                              s["freqs"].data_ptr(), s["total"].ctypes.data, _stream()))
    n = int(s["total"][0])
    _lib.check(lib.ck_kmer_targets_device(0, s["entries"].data_ptr(), n, s["targets"].data_ptr(), _stream()))
    return s["offsets"], s["freqs"], s["entries"], s["targets"], n


def _run_search(c, s):
    db, n, k, st, lib = s["db"], s["n"], c["cands"], _stream(), _lib.load()
    seq0 = db.arena_seq0
    db.d_flat[db.arena_res0:db.arena_res0 + s["residues"]].copy_(s["h_res"], non_blocking=True)
    db.d_offsets[seq0:seq0 + n].copy_(s["h_off"], non_blocking=True)
    db.d_lengths[seq0:seq0 + n].copy_(s["h_len"], non_blocking=True)
    q_off, q_len = db.d_offsets.data_ptr() + 8 * seq0, db.d_lengths.data_ptr() + 4 * seq0
    index = (db.d_kmer_offsets.data_ptr(), db.d_kmer_entries.data_ptr(), db.kmer_targets_ptr,
             db.d_kmer_freqs.data_ptr(), db.freq_thresh, db.n)
    found = (s["targets"].data_ptr(), s["counts"].data_ptr())
    query = (0, db.d_flat.data_ptr(), db.flat_len, q_off, q_len, n, s["longest"])
    band, hints = db.band_width, None
    if c["mode"] == "similar":
        _lib.check(lib.ck_search_phase_a_similar_device(*query, SUB.ctypes.data, 13, *index, 2, k, *found,
                                                        s["found"].data_ptr(), -1, st))
    elif c["mode"] == "cpath":
        band, hints = 50, s["diags"].data_ptr()
        bins = 10000 * ((s["residues"] + n * db.max_len) // 10 + n)
        _lib.check(lib.ck_search_kmer_candidates_device(*query, db.k, db.alpha, *index, db.d_lengths.data_ptr(), 2, 2,
                                                        10, k, 10000, *found, hints, s["found"].data_ptr(),
                                                        bins if bins <= 1 << 29 else -1, st))
    else:
        _lib.check(lib.ck_search_phase_a_device(*query, db.k, db.alpha, *index, 2, k, *found, s["found"].data_ptr(),
                                                st))
    _lib.check(lib.ck_search_pairs_device(n, k, seq0, db.empty_idx, s["found"].data_ptr(), s["targets"].data_ptr(),
                                          s["pairs"].data_ptr(), st))
    _lib.check(lib.ck_sw_batch_device_ctx(0, s["pairs"].data_ptr(), n * k, db.d_flat.data_ptr(), db.flat_len,
                                          db.d_offsets.data_ptr(), db.d_lengths.data_ptr(), db.n_all, band,
                                          SUB.ctypes.data, 0.0, hints, _lib.PASS_SCORE, _lib.ENGINE_BATCHED,
                                          s["sims"].data_ptr(), s["scores"].data_ptr(), None, None,
                                          s["mask"].data_ptr(), st))
    out = {x: s[x] for x in ("found", "targets", "counts", "pairs", "sims", "scores", "mask")}
    if hints:
        out["diags"] = s["diags"]
    return out


def _run_search_call(c, s):
    hits = search.search_batch(s["db"], s["queries"], top_k=c["top_k"], max_cands=c["cands"], kmer_score_thresh=0,
                               min_diag_hits=2, use_c_scoring=True, use_c_sw=True)
    found = np.full((len(hits), c["top_k"], 2), -1, np.int64)
    value = np.zeros((len(hits), c["top_k"], 2), np.float32)
    for q, per_query in enumerate(hits):
        found[q, :len(per_query)] = [(h.target, h.score) for h in per_query] or np.empty((0, 2))
        value[q, :len(per_query)] = [(h.identity, h.rank) for h in per_query] or np.empty((0, 2))
    return found, value


def _run_graph(c, s):
    indptr, indices, data = graph.graph_csr_device(s["pairs"], s["sims"], s["n"])
    count, labels, _ = graph.connected_components_device(s["pairs"], s["n"])
    return {"indptr": indptr, "indices": indices, "data": data, "count": count, "labels": labels}


RUN = {"align_host": _run_align_host, "align": _run_align, "sketch": _run_sketch, "jaccard": _run_jaccard,
       "lsh": _run_lsh, "index": _run_index, "search": _run_search, "search_call": _run_search_call,
       "graph": _run_graph}


# ------------------------------------------------------------------ work
def _mean_length(c):
    r = np.random.default_rng(0)
    if c.get("dist") == "pareto":
        x = c["lo"] * (1.0 - r.random(20000)) ** (-1.0 / 1.5)
    else:
        x = c.get("median", 350) * np.exp(0.5 * r.standard_normal(20000))
    return float(np.clip(x, c.get("lo", 30), c.get("hi", 2000)).mean())


def _cells(c, pairs, band, rows=None):
    """About the cells of `pairs` banded alignments of this case's sequences."""
    r = np.random.default_rng(1)
    x = (c["lo"] * (1.0 - r.random((2, 20000))) ** (-1.0 / 1.5) if c.get("dist") == "pareto"
         else c.get("median", 350) * np.exp(0.5 * r.standard_normal((2, 20000))))
    x = np.clip(x, c.get("lo", 30), c.get("hi", 2000))
    a, b = x.min(0), x.max(0)
    keep = a >= c.get("ratio", 0.0) * b
    a, b = a[keep], b[keep]
    w = np.where(b <= 50, b, band)
    lost = np.minimum(w, b) ** 2 / 2 + np.maximum(0, np.minimum(w, a + w - b)) ** 2 / 2
    return pairs * float(np.maximum(a * np.minimum(2 * w + 1, b) - np.where(2 * w + 1 < b, lost, 0), a).mean())


def work(case):
    c, kind = case, case["kind"]
    n = c["families"] * PER_FAMILY
    mean = _mean_length(c)
    if kind in ("align", "align_host"):
        # pairs and sequences in, five outputs a pair out; six max-plus operations a cell
        return {"bytes": 25.0 * c["pairs"] + n * (mean + 12), "flops": 6.0 * _cells(c, c["pairs"], c["band"])}
    if kind == "sketch":
        # a multiply-add a residue of each k-mer and a 64-bit mixing (about ten operations) a k-mer
        return {"bytes": n * (mean + 12 + 8 * c["size"]), "flops": 12.0 * n * mean}
    if kind == "jaccard":
        return {"bytes": 13.0 * c["pairs"] + 8.0 * n * c["size"], "flops": 2.0 * c["pairs"] * c["size"]}
    if kind == "lsh":
        # the band columns in, each family's pairs out
        cols = min(c["size"], c["tables"] * c["bands"])
        return {"bytes": 8.0 * n * cols + 8.0 * c["families"] * 45,
                "flops": float(n) * c["tables"] * (2 * c["bands"] + 5)}
    if kind == "index":
        return {"bytes": n * mean * (1 + 8 + 4 + 8) + 12.0 * 20 ** c["k"], "flops": 2.0 * n * mean}
    if kind == "graph":
        return {"bytes": 2 * 12.0 * c["pairs"] + 16.0 * c["pairs"] + 12.0 * n, "flops": 2.0 * c["pairs"]}
    # a query's posting lists (its residues times the mean list of the index) and its candidates' cells
    q = c["queries"]
    lists = q * 330.0 * n * mean / 20 ** 5
    if c.get("mode") == "similar":
        lists *= 3000
    band = 50 if kind == "search_call" or c["mode"] == "cpath" else 200
    cells = _cells({"median": 320}, q * min(c["cands"], 300), band)
    return {"bytes": 4.0 * lists + q * c["cands"] * 25.0 + 700.0 * q * c["cands"], "flops": lists + 6.0 * cells}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """The floating outputs in 64 bits.  Whole numbers have no such value; neither have the searches, whose
    identities are quotients of matches over candidates that only the search itself finds."""
    if case["kind"] == "jaccard":
        s = prepare(case, seed)
        return _exact_jaccard(s["pairs"], s["sk"]), None
    if case["kind"] == "graph":
        s = prepare(case, seed)
        return {"indptr": None, "indices": None, "data": _exact_weights(s), "count": None, "labels": None}
    if case["kind"] == "align" and _cells(case, case["pairs"], case["band"]) < 5e9 and case["dist"] != "pareto":
        s = prepare(case, seed)
        score, matches = _exact_sw(s["flat"], s["off"], s["len"], s["pairs"], case["band"])
        short = torch.minimum(s["len"][s["pairs"][:, 0].long()], s["len"][s["pairs"][:, 1].long()])
        return {"sims": torch.where(score > 0, matches.double() / short, 0.0), "scores": None, "matches": None,
                "shorter": None, "mask": None}
    if case["kind"] == "align_host" and _cells(case, case["pairs"], case["band"]) < 5e9:
        s = prepare(case, seed)
        d = {x: torch.from_numpy(s[x]).to(DEV) for x in ("flat", "off", "len", "pairs")}
        score, matches = _exact_sw(d["flat"], d["off"], d["len"], d["pairs"], case["band"])
        short = torch.minimum(d["len"][d["pairs"][:, 0].long()], d["len"][d["pairs"][:, 1].long()])
        sims = torch.where(score > 0, matches.double() / short, 0.0)
        sims = sims[sims.float() >= np.float32(case["threshold"])]
        return None, torch.cat([sims, sims.new_zeros(case["pairs"] - sims.numel())]), None
    return None


def _exact_jaccard(pairs, sk, chunk=500000):
    """clustkit's walk over two sorted sketches, one step of every pair at a time."""
    out = []
    big = torch.iinfo(torch.int64).max
    sk = sk ^ torch.iinfo(torch.int64).min  # unsigned order
    n, size = sk.shape
    sk = torch.cat([sk, torch.full((n, 1), big, dtype=torch.int64, device=DEV)], 1)
    for p in torch.split(pairs.long(), chunk):
        a, b = sk[p[:, 0]], sk[p[:, 1]]
        x, y, shared, steps = (torch.zeros(p.shape[0], dtype=torch.int64, device=DEV) for _ in range(4))
        for _ in range(size):
            u = a.gather(1, x[:, None])[:, 0]
            v = b.gather(1, y[:, None])[:, 0]
            go = ~((u == big) & (v == big))
            shared += go & (u == v)
            steps += go
            x += go & (u <= v)
            y += go & (v <= u)
        out.append(torch.where(steps > 0, shared.double() / steps.clamp(min=1), 0.0))
    return torch.cat(out)


def _exact_weights(s):
    p = torch.cat([s["pairs"], s["pairs"].flip(1)]).long()
    key = p[:, 0] * s["n"] + p[:, 1]
    uniq, at = torch.unique(key, return_inverse=True)
    w = torch.zeros(uniq.numel(), dtype=torch.float64, device=DEV)
    return w.index_add_(0, at, torch.cat([s["sims"], s["sims"]]).double())


def _exact_sw(flat, off, length, pairs, band, budget=40_000_000):
    """(score, matches) of clustkit's banded Smith-Waterman, anti-diagonal by anti-diagonal in 64-bit integers.

    A value holds score << 32 | rank << 28 | matches, so that one maximum also settles the ties: zero before
    diagonal before E before F, and a longer gap before a new one.
    """
    one, rank, low = 1 << 32, 1 << 28, (1 << 28) - 1
    table = torch.full((32, 32), -4, dtype=torch.int64)
    table[:20, :20] = torch.from_numpy(SUB.astype(np.int64))
    table = (table * one + torch.eye(32, dtype=torch.int64)).to(DEV).reshape(-1)
    flat, length = flat.long(), length.long()
    swap = length[pairs[:, 0].long()] > length[pairs[:, 1].long()]
    row = torch.where(swap, pairs[:, 1], pairs[:, 0]).long()
    col = torch.where(swap, pairs[:, 0], pairs[:, 1]).long()
    score = torch.zeros(pairs.shape[0], dtype=torch.int64, device=DEV)
    matches = torch.zeros_like(score)
    order = torch.argsort(length[row])
    sizes = length[row][order].tolist()
    at = 0
    while at < len(sizes):
        end = at + 1
        while end < len(sizes) and (end + 1 - at) * (sizes[end] + 1) <= budget:
            end += 1
        idx = order[at:end]
        at = end
        la, lb = length[row[idx]], length[col[idx]]
        w = torch.where(lb <= 50, lb, band)[:, None]
        rows = int(la.max())
        if rows == 0:
            continue
        i = torch.arange(1, rows + 1, device=DEV)[None, :]
        a = flat[(off[row[idx]][:, None] + torch.minimum(i, la[:, None]) - 1).clamp(min=0)] * 32
        floor = torch.full_like(a, -1_000_000 * one)
        zero = torch.zeros_like(a)
        h1, h2, e1, f1, best = zero, zero, floor, floor, zero

        def above(x, fill):  # the row above's value
            return torch.cat([torch.full_like(x[:, :1], fill), x[:, :-1]], 1)

        for d in range(2, int((la + lb).max()) + 1):
            j = d - i
            inside = (i <= la[:, None]) & (j >= 1) & (j <= lb[:, None]) & ((j - i).abs() <= w)
            b = flat[(off[col[idx]][:, None] + j.clamp(min=1) - 1).clamp(max=flat.numel() - 1)]
            e = torch.maximum(above(e1, -1_000_000 * one) - one + rank, above(h1, 0) - 11 * one) & ~(15 * rank)
            f = torch.maximum(f1 - one + rank, h1 - 11 * one) & ~(15 * rank)
            diag = above(h2, 0) + table[a + b]
            h = torch.maximum(torch.maximum(diag + 2 * rank, e + rank), f).clamp(min=3 * rank) & ~(15 * rank)
            h2, h1 = h1, torch.where(inside, h, 0)
            e1, f1 = torch.where(inside, e, floor), torch.where(inside, f, floor)
            best = torch.where(h1 // one > best // one, h1, best)
        # the first row that holds the largest score
        pick = torch.argmax((best // one) * 65536 - i, 1)
        v = best.gather(1, pick[:, None])[:, 0]
        score[idx], matches[idx] = v // one, v & low
    return score, matches
