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
