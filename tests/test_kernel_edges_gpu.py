"""Kernels at the sizes where their forms change or their tiles end, against
the oracle (bit for bit)."""
import numpy as np
import pytest

import oracle
from clustkit_gb300 import synth
from clustkit_gb300.lsh import band_parameters, lsh_candidates, lsh_candidates_device
from clustkit_gb300.sketch import sketch_flat

pytestmark = pytest.mark.gpu


def _pack(seqs):
    lengths = np.array([len(x) for x in seqs], np.int32)
    offsets = (np.cumsum(lengths) - lengths).astype(np.int64)
    return np.concatenate(seqs).astype(np.uint8), offsets, lengths


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
