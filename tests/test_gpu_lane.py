"""Edges of the one-request-per-lane kernels against the oracle.

Key rests and values that end at, before and after the 30 data words of a
suffix slab (and at the 8-word parts that lanes read), key lengths shared by
few and many requests, requests of one warp and of more warps than the launch
has, with and without length arrays.  Integer results: compared exactly.
"""
import numpy as np
import pytest

from indexes import GpuIndex, OracleIndex

pytestmark = pytest.mark.gpu


def _edge_keys(n, maxK, maxV, seed):
    """Distinct keys: the first two slices from small ranges (shared layers),
    lengths and value lengths at the slab edges where the rows allow them."""
    rng = np.random.default_rng(seed)
    edges = [1, 2, 3, 7, 8, 9, 10, 16, 17, 24, 25, 29, 30, 31, 32, 33, 60, 61, 62, 63]
    kl = rng.choice([e for e in edges if e <= maxK] + [maxK], n).astype(np.uint32)
    vl = rng.choice([e for e in edges if e <= maxV] + [maxV], n).astype(np.uint32)
    keys = rng.integers(0, 1 << 32, (n, maxK), dtype=np.uint64).astype(np.uint32)
    keys[:, 0] = rng.choice(np.array([0, 1, 5, 0xFFFFFFFE, 0xFFFFFFFF], np.uint32), n)
    if maxK > 1:
        keys[:, 1] = rng.integers(0, 50, n)
    keys[np.arange(maxK)[None, :] >= kl[:, None]] = 0
    _, first = np.unique(np.concatenate([keys, kl[:, None]], axis=1), axis=0, return_index=True)
    first = np.sort(first)
    vals = rng.integers(1, 1 << 32, (n, maxV), dtype=np.uint64).astype(np.uint32)
    vals[np.arange(maxV)[None, :] >= vl[:, None]] = 0
    return keys[first], kl[first], vals[first], vl[first]


@pytest.mark.parametrize("n", [1, 31, 33, 5000, 150000])
@pytest.mark.parametrize("maxK,maxV", [(1, 1), (9, 8), (32, 30), (63, 62)])
def test_finds_at_slab_edges(n, maxK, maxV):
    keys, kl, vals, vl = _edge_keys(min(n, 20000), maxK, maxV, 7 * n + maxK)
    m = len(kl)
    held = max(1, m * 2 // 3)
    g, o = GpuIndex(pool_bytes=256 << 20), OracleIndex()
    try:
        np.testing.assert_array_equal(g.insert(keys[:held], kl[:held], vals[:held], vl[:held]),
                                      o.insert(keys[:held], kl[:held], vals[:held], vl[:held]))
        pick = np.random.default_rng(n).integers(0, m, n)
        fk, fl = keys[pick], kl[pick]
        near = np.arange(n) % 5 == 0  # a key that differs in its last slice
        fk[near, fl[near] - 1] ^= 1
        for lens in (fl, None):
            for maxv in (maxV, 1):
                ov, ol = o.find(fk, lens, maxv)
                for conc in (False, True):
                    gv, gl = g.find(fk, lens, maxv, concurrent=conc)
                    np.testing.assert_array_equal(gl, ol)
                    np.testing.assert_array_equal(gv, ov)
    finally:
        g.close()
