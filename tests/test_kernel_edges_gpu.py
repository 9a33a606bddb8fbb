"""Kernels at the sizes where their forms change or their tiles end, against
the oracle (bit for bit)."""
import numpy as np
import pytest

import oracle
from clustkit_gb300 import synth
from clustkit_gb300.lsh import band_parameters, lsh_candidates, lsh_candidates_device
from clustkit_gb300.pairwise import batch_jaccard
from clustkit_gb300.sketch import sketch_flat

pytestmark = pytest.mark.gpu


def _pack(seqs):
    lengths = np.array([len(x) for x in seqs], np.int32)
    offsets = (np.cumsum(lengths) - lengths).astype(np.int64)
    return np.concatenate(seqs).astype(np.uint8), offsets, lengths


@pytest.mark.parametrize("s", [1, 2, 31, 32, 33, 64, 100, 128, 129, 256, 500, 1000, 1861, 1862, 4096])
@pytest.mark.parametrize("k,alphabet", [(5, 20), (3, 20), (7, 20), (11, 4), (32, 4)])
def test_sketch_sizes(ck, s, k, alphabet):
    """Sequences with as many k-mers as the threshold form's buffers hold, one
    more and one fewer; repeats that leave no threshold between too few and
    too many; codes outside the alphabet."""
    rng = np.random.default_rng(s + k)
    seqs = []
    for c in (0, 1, s - 1, s, s + 1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1025, 2047, 2048,
              2049, 5000):
        seqs.append(rng.integers(0, alphabet, max(0, c + k - 1)))
    for n in (300, 3000, 6000):  # one value, two values, a few, and a repeat among others
        seqs.append(np.zeros(n, np.int64))
        seqs.append(rng.integers(0, 2, n))
        seqs.append(np.tile(rng.integers(0, alphabet, 9), n // 9))
        x = rng.integers(0, alphabet, n)
        x[n // 4: n // 2] = 3
        seqs.append(x)
    seqs.append(rng.integers(0, 256, 2500))
    flat, off, lens = _pack(seqs)
    got = sketch_flat(flat, off, lens, k, s, alphabet)
    assert np.array_equal(got, oracle.sketches(flat, off, lens, k, s, alphabet))


@pytest.mark.parametrize("s", [1, 2, 31, 32, 33, 63, 65, 100, 127, 128, 129, 255, 256, 257])
@pytest.mark.parametrize("m", [1, 31, 33, 2431, 2433, 80000])
def test_jaccard_runs(ck, s, m):
    """Pair lists of every run length, sorted by the first sequence and not,
    over sketches with repeats, padding and values that differ in the high
    bits alone (the bitmap reads the low ones)."""
    rng = np.random.default_rng(s * 7 + m)
    mx = np.uint64(np.iinfo(np.uint64).max)
    rows = []
    for r in range(120):
        n = int(rng.integers(0, s + 1)) if r % 3 else s
        hi = [4, 3 * s, 2 ** 40, 2 ** 63][r % 4]
        x = rng.integers(0, hi, n).astype(np.uint64)
        if r % 5 == 0:
            x <<= np.uint64(20)
        rows.append(np.concatenate([np.sort(x), np.full(s - n, mx, np.uint64)]))
    sk = np.stack(rows)
    sk[60:90] = np.sort(np.where(rng.random((30, s)) < 0.5, sk[:30], sk[60:90]), 1)
    pairs = rng.integers(0, 120, size=(m, 2)).astype(np.int32)
    if m % 2 == 0:
        pairs = pairs[np.argsort(pairs[:, 0], kind="stable")]
    sims, mask = batch_jaccard(pairs, sk, 0.25)
    ref = oracle.jaccard(pairs, sk)
    assert np.array_equal(sims, ref)
    assert np.array_equal(mask, ref >= np.float32(0.25))


@pytest.mark.parametrize("tables,bands,size", [(1, 1, 1), (40, 1, 8), (64, 2, 3), (200, 1, 128), (30, 3, 4)])
def test_lsh_repeated_tables(ck, tables, bands, size):
    """Tables that read the same columns (most of them, here) add nothing; the
    same columns in another order are another table."""
    ss = synth.generate_families(150, 6, median=120, lo=5, hi=400, seed=tables + size)
    sk = sketch_flat(ss.flat, ss.offsets, ss.lengths, 4, size)
    idx, _ = band_parameters(size, tables, bands, 5)
    assert tables == 1 or len(np.unique(idx, axis=0)) < tables
    got = lsh_candidates_device(sk, tables, bands, 5).cpu().numpy()
    assert np.array_equal(got, lsh_candidates(sk, tables, bands, 5))


def _similar(db, qs, top_k, sub, thresh, entries=None, compact=True, list_capacity=-1):
    """ck_search_phase_a_similar_device in the default context: rows of (ids, scores)."""
    import torch
    from clustkit_gb300 import _lib
    lib, nq = db.lib, len(qs)
    lens = np.array([len(q) for q in qs], np.int32)
    offs = (np.cumsum(lens) - lens).astype(np.int64)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d_q, d_off, d_len = dev(np.concatenate(qs).astype(np.uint8)), dev(offs), dev(lens)
    d_ent = db.d_kmer_entries if entries is None else dev(entries)
    d_tgt = dev((d_ent.cpu().numpy() >> 32).astype(np.int32)) if compact else None
    out_t = torch.zeros(nq * top_k, dtype=torch.int32, device="cuda")
    out_s, out_n = torch.zeros_like(out_t), torch.zeros(nq, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.ck_search_phase_a_similar_device(
        0, d_q.data_ptr(), int(lens.sum()), d_off.data_ptr(), d_len.data_ptr(), nq, int(lens.max()), sub.ctypes.data,
        thresh, db.d_kmer_offsets.data_ptr(), d_ent.data_ptr(), d_tgt.data_ptr() if compact else None,
        db.d_kmer_freqs.data_ptr(), db.freq_thresh, db.n, 2, top_k, out_t.data_ptr(), out_s.data_ptr(),
        out_n.data_ptr(), list_capacity, st))
    _lib.check(lib.ck_ctx_status(0, st))
    n, t, s = out_n.cpu().numpy(), out_t.cpu().numpy().reshape(nq, -1), out_s.cpu().numpy().reshape(nq, -1)
    return [(t[q, :n[q]], s[q, :n[q]]) for q in range(nq)]


def _matrix(kind):
    from clustkit_gb300.blosum import BLOSUM62
    if kind == "blosum":
        return np.ascontiguousarray(BLOSUM62, np.int8)
    if kind == "flat":  # one score: no bins between the least and the most
        return np.full((20, 20), 3, np.int8)
    return np.random.default_rng(3).integers(-128, 128, (20, 20)).astype(np.int8)  # every int8 score


@pytest.fixture(scope="module")
def small_db():
    from clustkit_gb300.search import DeviceDatabase
    ss = synth.generate_families(300, 4, median=120, lo=3, hi=300, seed=4)
    return DeviceDatabase(ss.flat, ss.offsets, ss.lengths, arena_queries=8, arena_residues=8 * 400), ss


@pytest.mark.parametrize("kind,thresh", [("blosum", 13), ("blosum", 3), ("blosum", 60), ("flat", 15), ("flat", 16),
                                         ("wide", 330), ("wide", 636)])
def test_similar_listing(ck, small_db, kind, thresh):
    """Every 5-mer at or above the threshold, for matrices of the least and the
    largest score range and thresholds that most, few and no 5-mers reach."""
    db, ss = small_db
    off, ent, fr = db.index_arrays()
    sub = _matrix(kind)
    rng = np.random.default_rng(9)
    qs = [ss.seq(7)[:5].copy(), np.zeros(4, np.uint8), np.full(12, 18, np.uint8),  # 18: a large diagonal score
          np.concatenate([ss.seq(40)[:20], [20], ss.seq(41)[:11]]).astype(np.uint8),
          rng.integers(0, 20, 9).astype(np.uint8)]
    if thresh > 10:
        qs.append(ss.seq(100).copy())
    for part in (qs, qs[:1]):
        lens = np.array([len(q) for q in part], np.int32)
        offs = (np.cumsum(lens) - lens).astype(np.int64)
        want = oracle.similar_candidates_batch(np.concatenate(part), offs, lens, sub, thresh, off, ent, fr,
                                               db.freq_thresh, db.n, 2, 50)
        got = _similar(db, part, 50, sub, thresh)
        for g, w in zip(got, want):
            assert np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1])


@pytest.mark.parametrize("n_db,shuffled,compact", [(57344, False, True), (57345, False, True), (57345, False, False),
                                                   (120001, False, True), (120001, True, True), (1, False, True)])
def test_similar_target_ranges(ck, n_db, shuffled, compact):
    """The posting walk by target ranges: one range that is just full, two,
    three, one target; and lists that are not in target order, which it leaves
    to the walk on the count rows."""
    from clustkit_gb300 import _lib
    from clustkit_gb300.search import DeviceDatabase
    rng = np.random.default_rng(n_db)
    lens = rng.integers(5, 14, n_db).astype(np.int32)
    off = (np.cumsum(lens) - lens).astype(np.int64)
    flat = rng.integers(0, 20, int(lens.sum())).astype(np.uint8)
    db = DeviceDatabase(flat, off, lens, arena_queries=8, arena_residues=8 * 400)
    koff, ent, fr = db.index_arrays()
    if shuffled:  # each list's entries reversed
        at = np.repeat(koff[:-1] + koff[1:] - 1, np.diff(koff)) - np.arange(len(ent))
        ent = ent[at]
    qs = [flat[off[i]:off[i] + lens[i]].copy() for i in (0, n_db // 2, n_db - 1)]
    qs += [rng.integers(0, 20, 150).astype(np.uint8), np.zeros(3, np.uint8)]
    sub = _matrix("blosum")
    qlen = np.array([len(q) for q in qs], np.int32)
    qoff = (np.cumsum(qlen) - qlen).astype(np.int64)
    want = oracle.similar_candidates_batch(np.concatenate(qs), qoff, qlen, sub, 13, koff, ent, fr, db.freq_thresh,
                                           n_db, 2, 300)
    for cap in (-1, 4_000_000):
        got = _similar(db, qs, 300, sub, 13, entries=ent, compact=compact, list_capacity=cap)
        for g, w in zip(got, want):
            assert np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1])
    with pytest.raises(_lib.CkError) as e:
        _similar(db, qs, 300, sub, 13, entries=ent, compact=compact, list_capacity=10)
    assert e.value.status == _lib.CK_ERR_CAPACITY


@pytest.mark.parametrize("bw", [1, 8, 31, 32, 59, 60, 127, 128, 263])
@pytest.mark.parametrize("hinted,long_rows", [(False, 0), (True, 0), (False, 2100)])
def test_wave_group_shapes(ck, bw, hinted, long_rows):
    """The streamed schedule at the band widths where its lanes per group and
    rows per strip change: pairs of one strip, of just a group's lanes, and of
    many rotations, with and without hints; rows above 2,047 take the wide key
    for every pair."""
    from clustkit_gb300 import _lib
    from clustkit_gb300.blosum import BLOSUM62
    from clustkit_gb300.pairwise import batch_sw
    rng = np.random.default_rng(bw + long_rows)
    lens = [1, 2, 15, 16, 17, 49, 50, 51, 52, 64, 127, 128, 129, 130, 255, 256, 257, 258, 511, 513, 900, 1300]
    if long_rows:
        lens += [long_rows, long_rows + 40]
    base = rng.integers(0, 20, max(lens) + 60)
    seqs = []
    for n in lens:
        for v in range(3):  # related, shifted and unrelated
            x = base[5 * v: 5 * v + n].copy() if v < 2 else rng.integers(0, 20, n)
            x[rng.random(n) < 0.25] = rng.integers(0, 20)
            seqs.append(x)
    flat, off, length = _pack(seqs)
    pairs = rng.integers(0, len(seqs), (2500, 2)).astype(np.int32)
    pairs = np.concatenate([pairs, np.stack([np.arange(len(seqs) - 1), np.arange(1, len(seqs))], 1).astype(np.int32)])
    hints = rng.integers(-80, 81, len(pairs)).astype(np.int32) if hinted else None
    want = oracle.sw_batch(pairs, flat, off, length, bw, BLOSUM62, diag_hints=hints)
    keep = _lib.get_config(_lib.CFG_WAVE_STREAM)
    try:
        for stream in (2, 0):
            _lib.set_config(_lib.CFG_WAVE_STREAM, stream)
            got = batch_sw(pairs, flat, off, length, bw, BLOSUM62, 0.3, diag_hints=hints)
            for k in ("scores", "matches", "shorter", "sims"):
                assert np.array_equal(got[k], want[k]), (k, stream)
            assert _lib.sw_counters()["wave"] > 2000
    finally:
        _lib.set_config(_lib.CFG_WAVE_STREAM, keep)


def test_context_scratch_is_handed_on_clean(ck, small_db):
    """A context takes over the last destroyed one's scratch: its unread errors
    and its Phase-B bins (left by a call that ran out of them) must not show,
    and contexts alive at the same time share nothing."""
    from clustkit_gb300 import _lib
    from clustkit_gb300.search import Scoring, _Slot, search_batch
    db, ss = small_db
    qs = [ss.seq(i).copy() for i in (5, 300, 900)]
    kw = dict(top_k=10, max_cands=100, kmer_score_thresh=0, min_diag_hits=2, use_c_scoring=True, use_c_sw=True)
    hits = lambda res: [[(h.target, h.score, h.identity, h.rank) for h in q] for q in res]
    first = hits(search_batch(db, qs, **kw))
    slot = _Slot(db, 0, 100)
    slot.bins_bound = lambda nq, res, sc: 3  # far too few bins: the call leaves them dirty and an error unread
    slot.launch(qs, 2, 0, min_diag_hits=2, use_c_scoring=True, use_c_sw=True)
    slot.event.synchronize()
    slot.close()
    assert hits(search_batch(db, qs, **kw)) == first
    a, b = _Slot(db, 0, 100), _Slot(db, 0, 100)
    try:
        assert a.ctx != b.ctx
        for s in (a, b):
            assert hits(search_batch(db, qs[::-1], slot=s, **kw)) == first[::-1]
    finally:
        a.close()
        b.close()
    assert _lib.load().ck_ctx_status(a.ctx or 1 << 20, None) == _lib.CK_ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 65536, 65537])
def test_graph_key_widths(ck, n):
    """Rows and columns packed in as many bits as n needs, n at powers of two;
    chains, repeats and self-loops hooked in one pass."""
    import oracle.graph_oracle as go
    from clustkit_gb300 import graph
    rng = np.random.default_rng(n)
    ends = np.stack([np.arange(n), np.minimum(np.arange(n) + 1, n - 1)], 1)[rng.permutation(n)]
    pairs = np.concatenate([ends[: 3 * n // 4 + 1], rng.integers(0, n, (n // 8 + 1, 2)), ends[:2]]).astype(np.int32)
    w = rng.random(len(pairs)).astype(np.float32)
    got, want = graph.build_similarity_graph(n, pairs, w), go.build_similarity_graph(n, pairs, w)
    assert np.array_equal(got.indptr, want.indptr) and np.array_equal(got.indices, want.indices)
    assert np.allclose(got.data, want.data, rtol=1e-6)
    k, labels, _ = graph.connected_components_device(pairs, n)
    ref = go.cluster_connected_components(want)
    assert np.array_equal(labels.cpu().numpy(), ref) and k == int(ref.max()) + 1
    with pytest.raises(Exception):
        graph.connected_components_device(np.array([[0, n]], np.int32), n)
    k, labels, _ = graph.connected_components_device(pairs, n)  # the error above is not seen again
    assert np.array_equal(labels.cpu().numpy(), ref)


@pytest.mark.parametrize("n", [32, 33, 160, 1000, 1001, 1300])
def test_lsh_large_buckets(ck, n):
    """Buckets either side of the one-thread limit and of the cap, several at once."""
    rng = np.random.default_rng(n)
    sk = rng.integers(0, 2 ** 60, (2 * n + 50, 4)).astype(np.uint64)
    sk[:n, 0] = 7
    sk[n:2 * n, 1] = 9
    got = lsh_candidates_device(sk, 12, 1, 3).cpu().numpy()
    k = min(n, 1000)
    a, b = np.triu_indices(k, 1)
    want = np.concatenate([np.stack([a, b], 1), np.stack([a, b], 1) + n]).astype(np.int32)
    idx, _ = band_parameters(4, 12, 1, 3)
    assert {0, 1} <= set(idx[:, 0].tolist())
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [2, 3, 40, 1500])
def test_lsh_ids_that_share_their_upper_bits(ck, n):
    """Bucket ids of a table that differ in their lowest bits only, the members
    of one between those of another; the second table's are random."""
    rng = np.random.default_rng(n)
    idx, seeds = band_parameters(2, 8, 1, 4)
    col = int(idx[0, 0])
    m64 = (1 << 64) - 1

    def sketch_value(h):  # the value with bucket id h in table 0
        h ^= h >> 33
        h = h * pow(0xC4CEB9FE1A85EC53, -1, 1 << 64) & m64
        h ^= h >> 33
        return (h - int(seeds[0]) * 0x517CC1B727220A95) & m64

    low = rng.integers(0, max(2, n // 9), n)
    sk = rng.integers(0, max(2, n // 2), (n, 2)).astype(np.uint64)
    sk[:, col] = [sketch_value((0x0123456789AB << 16) | int(x)) for x in low]
    got = lsh_candidates_device(sk, 8, 1, 4).cpu().numpy()
    want = lsh_candidates(sk, 8, 1, 4)
    same = low[:, None] == low[None, :]
    a, b = np.nonzero(np.triu(same | (sk[:, None, 1 - col] == sk[None, :, 1 - col]), 1))
    assert set(idx[:, 0].tolist()) == {0, 1}
    assert np.array_equal(want, np.stack([a, b], 1)) and np.array_equal(got, want)


@pytest.mark.parametrize("members,rest,tables", [(1000, 0, 20), (900, 2000, 20), (760, 1, 40)])
def test_lsh_repeated_pairs(ck, members, rest, tables):
    """Pairs that every table finds, by the million, beside buckets of each
    small size that differ from table to table."""
    rng = np.random.default_rng(members)
    size = 64
    sk = rng.integers(0, 2 ** 62, (members + rest, size)).astype(np.uint64)
    sk[rng.permutation(members + rest)[:members]] = 5
    idx, _ = band_parameters(size, tables, 1, 8)
    columns = len(np.unique(idx))
    assert columns >= 12 and members * (members - 1) // 2 * columns >= 1 << 22
    for c in range(size if rest > 1 else 0):
        own = np.flatnonzero(sk[:, c] != 5)
        cut = np.sort(rng.choice(len(own), 120, replace=False))
        for x, y in zip(cut[:-1], cut[1:]):
            sk[own[x:y], c] = 1000 + x
    got = lsh_candidates_device(sk, tables, 1, 8).cpu().numpy()
    assert np.array_equal(got, lsh_candidates(sk, tables, 1, 8))


@pytest.mark.parametrize("n,lo,hi,k,alpha,letters", [
    (1, 5, 5, 5, 20, 20), (1, 8, 8, 5, 20, 20), (3, 0, 9, 3, 20, 25), (40, 1, 300, 2, 6, 6), (7, 60, 61, 3, 20, 1),
    (300, 0, 90, 4, 20, 21), (900, 30, 700, 5, 20, 22), (2500, 30, 700, 5, 20, 3), (64, 4, 130, 1, 20, 30),
    (50, 10, 400, 7, 4, 4), (2, 3, 4, 5, 20, 20), (5, 20, 30, 2, 20, 255)])
def test_kmer_index(ck, n, lo, hi, k, alpha, letters):
    """Offsets and frequencies counted and read off the sorted k-mers: few and
    many occurrences, long runs without a k-mer, residues that belong to none."""
    torch = pytest.importorskip("torch")
    from clustkit_gb300 import _lib
    rng = np.random.default_rng(n + k)
    flat, off, length = _pack([rng.integers(0, letters, rng.integers(lo, hi + 1)).astype(np.uint8) for _ in range(n)])
    keys, entries = [], []
    for q in range(n):
        s = flat[off[q]:off[q] + length[q]].astype(np.int64)
        for p in range(len(s) - k + 1):
            w = s[p:p + k]
            keys.append(int(w @ alpha ** np.arange(k)[::-1]) if (w < alpha).all() else alpha ** k)
            entries.append(q << 32 | p)
    keys, entries, nk = np.array(keys, np.int64), np.array(entries, np.int64), alpha ** k
    want_freqs = np.bincount(keys, minlength=nk + 1)[:nk]
    want_offsets = np.concatenate([[0], np.cumsum(want_freqs)])
    want_entries = entries[np.argsort(keys, kind="stable")]
    flat = np.concatenate([flat, np.zeros(1, np.uint8)])
    d = [torch.from_numpy(x).cuda() for x in (flat, off, length)]
    offsets = torch.full((nk + 1,), -1, dtype=torch.int64, device="cuda")
    freqs = torch.full((nk,), -1, dtype=torch.int32, device="cuda")
    out = torch.zeros(max(len(keys), 1), dtype=torch.int64, device="cuda")
    total = np.zeros(1, np.int64)
    _lib.check(_lib.load().ck_kmer_index_build_device(
        0, d[0].data_ptr(), d[0].numel(), d[1].data_ptr(), d[2].data_ptr(), n, k, alpha, offsets.data_ptr(),
        out.data_ptr(), len(keys), freqs.data_ptr(), total.ctypes.data, torch.cuda.current_stream().cuda_stream))
    assert total[0] == want_offsets[-1]
    assert np.array_equal(offsets.cpu().numpy(), want_offsets)
    assert np.array_equal(freqs.cpu().numpy(), want_freqs)
    assert np.array_equal(out.cpu().numpy()[:len(keys)], want_entries)
