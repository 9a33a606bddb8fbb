"""Kernels where a rule of their dispatch changes sides, and inputs that a rule
tuned on ordinary ones could lose on, against the oracle (bit for bit)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _pack(seqs):
    lengths = np.array([len(x) for x in seqs], np.int32)
    offsets = (np.cumsum(lengths) - lengths).astype(np.int64)
    return np.concatenate(seqs).astype(np.uint8), offsets, lengths


def _repeat(rng, n, period, changed):
    x = np.tile(rng.integers(0, 20, period), n // period + 1)[:n]
    m = rng.random(n) < changed
    x[m] = rng.integers(0, 20, int(m.sum()))
    return x


@pytest.mark.parametrize("s", [22, 23, 65, 66, 128, 163, 164, 377, 378, 829, 830, 1768, 1769])
@pytest.mark.parametrize("k", [5, 3, 8])
def test_sketch_buffer_edges(ck, s, k):
    """The largest sketch of each buffer size and the next: ordinary sequences
    of many lengths, and repeats of which no threshold leaves s to C hashes."""
    from clustkit_gb300.sketch import sketch_flat
    rng = np.random.default_rng(s * 10 + k)
    seqs = [rng.integers(0, 20, n) for n in list(rng.integers(s // 2 + 8, 6 * s + 100, 200)) + [9000]]
    for period in (1, 2, 4, 9, 30):
        for changed in (0.0, 0.02, 0.1, 0.4):
            for n in (s + 70, 2000, 7000):
                seqs.append(_repeat(rng, n, period, changed))
    for n in (3000, 6000):  # a repeat before and behind ordinary residues
        seqs.append(np.concatenate([_repeat(rng, n, 4, 0.02), rng.integers(0, 20, n)]))
        seqs.append(np.concatenate([rng.integers(0, 20, n), _repeat(rng, n, 4, 0.02)]))
    flat, off, lens = _pack(seqs)
    assert np.array_equal(sketch_flat(flat, off, lens, k, s), oracle.sketches(flat, off, lens, k, s, 20))


def test_sketch_time_of_repeats(ck):
    """A sequence takes at most two passes over its k-mers, and the second sorts
    the buffer a few times: repeats stay within 8 times the time of as many
    random residues (a threshold search by bisection took up to 66 passes)."""
    import torch
    from clustkit_gb300 import _lib
    lib, rng, n, length = _lib.load(), np.random.default_rng(2), 4000, 2000
    stream = torch.cuda.current_stream().cuda_stream
    off = torch.arange(n, device="cuda") * length
    lens = torch.full((n,), length, dtype=torch.int32, device="cuda")
    out = torch.empty((n, 128), dtype=torch.int64, device="cuda")

    def ms(period, changed):
        flat = torch.from_numpy(np.concatenate([_repeat(rng, length, period, changed) for _ in range(n)])
                                .astype(np.uint8)).cuda()
        best = np.inf
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            _lib.check(lib.ck_sketch_device(flat.data_ptr(), flat.numel(), off.data_ptr(), lens.data_ptr(), n, 5, 128,
                                            20, 42, out.data_ptr(), stream))
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    random = ms(1, 1.0)
    for period, changed in ((4, 0.02), (4, 0.1), (9, 0.02), (9, 0.0), (30, 0.05)):
        assert ms(period, changed) < 8 * random, (period, changed)


def test_similar_index_of_almost_2_to_32_postings(ck):
    """The walk by target ranges numbers postings in 32 bits, eight at a time;
    an index that ends a few short of 2^32 is left to the other walk."""
    import torch
    from clustkit_gb300 import _lib
    from clustkit_gb300.blosum import BLOSUM62
    lib, total, nk, nq, top_k = _lib.load(), 2 ** 32 - 4, 20 ** 5, 4, 5
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    sub = np.ascontiguousarray(BLOSUM62, np.int8)
    targets = torch.zeros(total, dtype=torch.int32, device="cuda")
    targets[-6:] = torch.tensor([0, 0, 1, 2, 2, 2], dtype=torch.int32)
    offsets = torch.full((nk + 1,), total - 6, dtype=torch.int64, device="cuda")
    offsets[0], offsets[-1] = 0, total  # all but six are the first 5-mer's, the six the last one's
    freqs = torch.zeros(nk, dtype=torch.int32, device="cuda")
    freqs[0], freqs[-1] = 2 ** 31 - 1, 6
    queries = [[19] * 5, [0] * 9, [19] * 6, [0] * 5]
    lens = np.array([len(q) for q in queries], np.int32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d_q, d_len = dev(np.concatenate(queries).astype(np.uint8)), dev(lens)
    d_off = dev((np.cumsum(lens) - lens).astype(np.int64))
    out_t = torch.zeros(nq * top_k, dtype=torch.int32, device="cuda")
    out_s, out_n = torch.zeros_like(out_t), torch.zeros(nq, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.ck_search_phase_a_similar_device(
        0, d_q.data_ptr(), int(lens.sum()), d_off.data_ptr(), d_len.data_ptr(), nq, int(lens.max()), sub.ctypes.data,
        13, offsets.data_ptr(), None, targets.data_ptr(), freqs.data_ptr(), 1000, 3, 2, top_k, out_t.data_ptr(),
        out_s.data_ptr(), out_n.data_ptr(), -1, st))
    _lib.check(lib.ck_ctx_status(0, st))
    w = 5 * int(sub[19, 19])
    assert w >= 13 and 5 * int(sub[0, 19]) < 13
    got = [list(zip(t[:n], s[:n])) for t, s, n in zip(out_t.view(nq, -1).tolist(), out_s.view(nq, -1).tolist(),
                                                      out_n.tolist())]
    assert got == [[(0, 2 * w), (1, w), (2, 3 * w)], [], [(0, 4 * w), (1, 2 * w), (2, 6 * w)], []]


@pytest.mark.parametrize("n_db,mean,nq,shuffled,compact", [
    (57344, 100, 64, False, True), (57344, 300, 4, False, True), (57345, 160, 70, False, True),
    (57345, 160, 64, False, False), (57345, 160, 64, True, True), (120001, 150, 64, False, True),
    (57345, 160, 3, False, True), (57345, 80, 64, False, True)])
def test_similar_ranges_of_long_lists(ck, n_db, mean, nq, shuffled, compact):
    """The walk by target ranges on indexes with enough postings for it: one
    range that is just full, two, three, more queries than are held at a time;
    lists out of target order, and calls either side of its rule."""
    import torch
    from clustkit_gb300 import _lib
    from clustkit_gb300.blosum import BLOSUM62
    from clustkit_gb300.search import DeviceDatabase
    rng = np.random.default_rng(n_db + nq)
    lens = rng.integers(mean // 2, mean + mean // 2 + 1, n_db).astype(np.int32)
    off = (np.cumsum(lens) - lens).astype(np.int64)
    flat = rng.integers(0, 20, int(lens.sum())).astype(np.uint8)
    db = DeviceDatabase(flat, off, lens, arena_queries=8, arena_residues=8 * 400)
    koff, ent, fr = db.index_arrays()
    ranges = -(-n_db // 57344)
    enough = (0.05 * ranges ** 2 + 2e-5 * n_db + (1.5 + 2 * ranges + 2.5 * ranges ** 2) / nq) * 20 ** 5
    assert (int(koff[-1]) >= enough and nq >= 4) == (mean != 80 and nq > 3)
    if shuffled:  # each list's entries reversed
        ent = ent[np.repeat(koff[:-1] + koff[1:] - 1, np.diff(koff)) - np.arange(len(ent))]
    at = rng.integers(0, n_db, nq)
    qs = [flat[off[i]:off[i] + int(rng.integers(20, 50))].copy() for i in at]
    qs[0], qs[1] = flat[off[-1]:off[-1] + lens[-1]].copy(), np.zeros(3, np.uint8)
    sub = np.ascontiguousarray(BLOSUM62, np.int8)
    qlen = np.array([len(q) for q in qs], np.int32)
    qoff = (np.cumsum(qlen) - qlen).astype(np.int64)
    want = oracle.similar_candidates_batch(np.concatenate(qs), qoff, qlen, sub, 13, koff, ent, fr, db.freq_thresh,
                                           n_db, 2, 300)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d_q, d_off, d_len, d_ent = dev(np.concatenate(qs)), dev(qoff), dev(qlen), dev(ent)
    d_tgt = dev((ent >> 32).astype(np.int32)) if compact else None
    out_t = torch.zeros(nq * 300, dtype=torch.int32, device="cuda")
    out_s, out_n = torch.zeros_like(out_t), torch.zeros(nq, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(db.lib.ck_search_phase_a_similar_device(
        0, d_q.data_ptr(), int(qlen.sum()), d_off.data_ptr(), d_len.data_ptr(), nq, int(qlen.max()), sub.ctypes.data,
        13, db.d_kmer_offsets.data_ptr(), d_ent.data_ptr(), d_tgt.data_ptr() if compact else None,
        db.d_kmer_freqs.data_ptr(), db.freq_thresh, n_db, 2, 300, out_t.data_ptr(), out_s.data_ptr(),
        out_n.data_ptr(), -1, st))
    _lib.check(db.lib.ck_ctx_status(0, st))
    t, s, n = out_t.cpu().numpy().reshape(nq, -1), out_s.cpu().numpy().reshape(nq, -1), out_n.cpu().numpy()
    for q in range(nq):
        assert np.array_equal(t[q, :n[q]], want[q][0]) and np.array_equal(s[q, :n[q]], want[q][1])


def test_components_of_chains_and_stars(ck):
    """A chain and a star of a million nodes: one component, in at most 2.4 times
    the time of a chain whose labels are in random order (a chain walked to its
    end from every node took 4.9 times as long, a star with an atomic for every
    edge 2.8)."""
    import time

    import torch
    from clustkit_gb300 import graph
    n = 1_000_000
    rng = np.random.default_rng(0)
    chain = np.stack([np.arange(n - 1), np.arange(1, n)], 1).astype(np.int32)
    star = np.stack([np.full(n - 1, n // 2), np.delete(np.arange(n), n // 2)], 1).astype(np.int32)
    two = np.concatenate([chain[:n // 2 - 1], chain[n // 2:]])  # and two chains side by side

    def run(edges, parts):
        pairs = torch.from_numpy(edges).cuda()
        best = np.inf
        for _ in range(8):
            torch.cuda.synchronize()
            t = time.perf_counter()
            k, labels, _ = graph.connected_components_device(pairs, n)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        assert k == parts
        return best, labels.cpu().numpy()

    random, labels = run(rng.permutation(n).astype(np.int32)[chain], 1)
    assert not labels.any()
    for edges in (chain[rng.permutation(n - 1)], chain, chain[::-1].copy(), star, star[rng.permutation(n - 1)]):
        seconds, labels = run(edges, 1)
        assert not labels.any() and seconds < 2.4 * random
    _, labels = run(two[rng.permutation(len(two))], 2)
    assert np.array_equal(labels, (np.arange(n) >= n // 2).astype(np.int32))


@pytest.mark.parametrize("bw", [16, 50, 128])
@pytest.mark.parametrize("setting,adaptive,routed", [
    (450, 0, 450), (450, 1, 450), (512, 0, 512), (3, 0, 3), (8192, 0, None), (8192, 1, None), (9000, 1, None)])
def test_wave_row_bound_is_taken_as_given(ck, bw, setting, adaptive, routed):
    """Pairs run one warp per pair from the row bound that was set, at every
    band; 8192 and more is never."""
    from clustkit_gb300 import _lib
    from clustkit_gb300.blosum import BLOSUM62
    from clustkit_gb300.pairwise import batch_sw
    rng = np.random.default_rng(setting)
    rows = np.array([2, 3, 4, 100, 337, 338, 380, 400, 449, 450, 511, 512, 600, 6200, 8000])
    flat, off, lens = _pack([rng.integers(0, 20, n) for n in rows for _ in range(2)])
    pairs = np.stack([np.arange(0, len(lens), 2), np.arange(1, len(lens), 2)], 1).astype(np.int32)
    keys = {_lib.CFG_WAVE_ALL_BELOW: 0, _lib.CFG_WAVE_MIN_ROWS: setting, _lib.CFG_WAVE_ADAPTIVE: adaptive}
    keep = {k: _lib.get_config(k) for k in keys}
    try:
        for k, v in keys.items():
            _lib.set_config(k, v)
        got = batch_sw(pairs, flat, off, lens, bw, BLOSUM62, 0.3)
        wave = _lib.sw_counters()["wave"]
    finally:
        for k, v in keep.items():
            _lib.set_config(k, v)
    want = oracle.sw_batch(pairs, flat, off, lens, bw, BLOSUM62)
    assert np.array_equal(got["scores"], want["scores"]) and np.array_equal(got["matches"], want["matches"])
    # the adaptive rule may raise the bound, here never above the two longest pairs
    at_least = int((rows >= routed).sum()) if routed else 0
    assert wave == at_least if not adaptive or not routed else 0 < wave <= at_least


def test_lsh_room_of_a_short_last_batch(ck):
    """1,000,000 sequences are worked on in batches of 107 tables: for 124 the
    raw pairs' room follows the tables, not two batches' worth.  In bytes: 40 an
    item of a batch, the sketches, 16 a raw pair with a quarter and 5 % to spare,
    the places of pairs seen, and 300 MB for the sorts."""
    import ctypes

    import torch
    from clustkit_gb300 import _lib
    from clustkit_gb300.lsh import band_parameters
    lib, n, s, tables, values = _lib.load(), 1_000_000, 16, 124, 500
    per_batch = (4 << 30) // (40 * n)
    idx, seeds = band_parameters(s, tables * 2, 2, 3)
    _, first = np.unique(idx, axis=0, return_index=True)
    idx = np.ascontiguousarray(idx[np.sort(first)[:tables]], np.int32)  # distinct ones
    seeds = np.ascontiguousarray(seeds[:tables], np.uint64)
    assert len(idx) == tables and tables // 2 < per_batch < tables
    sk = torch.randint(0, values, (n, s), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    if torch.cuda.mem_get_info()[0] < 32 << 30:
        pytest.skip("needs 32 GB of device memory")
    ctx, count = ctypes.c_int32(), np.zeros(1, np.int64)
    _lib.check(lib.ck_ctx_create(ctypes.byref(ctx)))
    try:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        status = lib.ck_lsh_candidates_device(ctx.value, sk.data_ptr(), n, s, tables, 2, idx.ctypes.data,
                                              seeds.ctypes.data, None, 0, count.ctypes.data,
                                              torch.cuda.current_stream().cuda_stream)
        assert status == _lib.CK_ERR_OUT_OF_MEMORY and count[0] > 0  # no room for the output: counted
        held = before - torch.cuda.mem_get_info()[0]
    finally:
        _lib.check(lib.ck_ctx_destroy(ctx.value))
    # raw pairs: every table's n(n - 1)/2 comparisons, one in values^2 of which agree in two
    # different columns, one in values where both bands read one column
    same = int((idx[:, 0] == idx[:, 1]).sum())
    raw = n * (n - 1) / 2 * ((tables - same) / values ** 2 + same / values)
    assert held < 40 * per_batch * n + n * s * 8 + 16 * 1.25 * 1.05 * raw + (64 << 20) + (300 << 20)


@pytest.mark.parametrize("bw", [35, 36, 63, 64, 75, 76, 135, 136, 155, 156, 263])
@pytest.mark.parametrize("hinted,long_rows", [(False, 0), (True, 0), (False, 2100), (True, 2100)])
def test_wave_groups_at_their_band_limits(ck, bw, hinted, long_rows):
    """The bands where strips of 8 and of 16 rows take the next larger group of
    lanes (where a lane's next strip starts right after its last one), in calls
    of more pairs than the kernel has warps; with a pair of more than 2,047 rows
    the default schedule takes strips of 8 rows in each of these groups."""
    from clustkit_gb300 import _lib
    from clustkit_gb300.blosum import BLOSUM62
    from clustkit_gb300.pairwise import batch_sw
    rng = np.random.default_rng(2 * bw + long_rows + hinted)
    lens = [1, 7, 8, 9, 16, 17, 50, 51, 52, 64, 65, 127, 128, 129, 255, 256, 257, 400, 512, 513, 700]
    if long_rows:
        lens += [long_rows, long_rows + 37]
    base = rng.integers(0, 20, max(lens) + 40)
    seqs = []
    for n in lens:
        for v in range(3):  # related, shifted and unrelated
            x = base[7 * v: 7 * v + n].copy() if v < 2 else rng.integers(0, 20, n)
            x[rng.random(n) < 0.2] = rng.integers(0, 20)
            seqs.append(x)
    flat, off, length = _pack(seqs)
    pairs = rng.integers(0, len(seqs), (2900, 2)).astype(np.int32)
    pairs = np.concatenate([pairs, np.stack([np.arange(len(seqs) - 1), np.arange(1, len(seqs))], 1).astype(np.int32)])
    hints = rng.integers(-120, 121, len(pairs)).astype(np.int32) if hinted else None
    want = oracle.sw_batch(pairs, flat, off, length, bw, BLOSUM62, diag_hints=hints)
    keep = _lib.get_config(_lib.CFG_WAVE_STREAM)
    try:
        for stream in (1, 2, 0):
            _lib.set_config(_lib.CFG_WAVE_STREAM, stream)
            got = batch_sw(pairs, flat, off, length, bw, BLOSUM62, 0.3, diag_hints=hints)
            for k in ("scores", "matches", "shorter", "sims"):
                assert np.array_equal(got[k], want[k]), (k, stream)
            assert _lib.sw_counters()["wave"] > 2432  # more than 16 warps on each of 152 SMs
    finally:
        _lib.set_config(_lib.CFG_WAVE_STREAM, keep)
