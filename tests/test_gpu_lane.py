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


def _same_contents(g, o, n, maxK, maxV):
    lower, one = np.zeros((1, maxK), np.uint32), np.ones(1, np.uint32)
    for x, y, what in zip(g.scan(lower, one, n + 2, maxV=maxV), o.scan(lower, one, n + 2, maxV=maxV),
                          ("counts", "values", "value lengths", "keys", "key lengths")):
        np.testing.assert_array_equal(x, y, err_msg=what)
    ok, keys, msg = g.t.validate()
    assert ok and keys == len(o.dump(maxK, maxV)[1]), msg


@pytest.mark.parametrize("n", [1, 33, 4000, 120000])
@pytest.mark.parametrize("maxK,maxV", [(1, 1), (9, 8), (32, 30), (63, 62)])
def test_mixed_batches_at_slab_edges(n, maxK, maxV):
    # Touch-once batches of every kind: each request's result is defined.
    keys, kl, vals, vl = _edge_keys(n, maxK, maxV, 11 * n + maxV)
    m = len(kl)
    rng = np.random.default_rng(n)
    g, o = GpuIndex(pool_bytes=512 << 20), OracleIndex()
    try:
        held = rng.permutation(m)[:m // 2]
        if len(held):
            np.testing.assert_array_equal(g.insert(keys[held], kl[held], vals[held], vl[held]),
                                          o.insert(keys[held], kl[held], vals[held], vl[held]))
        for _ in range(3):
            types = rng.integers(0, 4, m).astype(np.uint8)
            v = rng.integers(1, 1 << 32, (m, maxV), dtype=np.uint64).astype(np.uint32)
            l = rng.permutation(vl)
            order = rng.permutation(m)
            gv, gl, gr = g.mixed(types, keys[order], kl[order], v, l)
            ov, ol, orr = o.mixed(types, keys[order], kl[order], v, l)
            find = types == 2
            np.testing.assert_array_equal(gr[~find], orr[~find])
            np.testing.assert_array_equal(gl[find], ol[find])
            live = np.arange(maxV)[None, :] < np.minimum(ol, maxV)[:, None]
            assert (np.where(live, gv, 0)[find] == np.where(live, ov, 0)[find]).all()
        _same_contents(g, o, m, maxK, maxV)
    finally:
        g.close()


@pytest.mark.parametrize("upsert", [False, True])
def test_writes_that_meet_in_one_node(upsert):
    # Ascending keys inserted beside each other split the same nodes again and
    # again; many requests then write and erase few keys.
    n = 30000
    g, o = GpuIndex(pool_bytes=256 << 20), OracleIndex()
    try:
        keys = np.arange(3 * n, dtype=np.uint32)[:, None]
        one = np.ones(n, np.uint32)
        for i in range(3):  # the first call builds, the others insert between and after
            k = keys[i::3] if i < 2 else keys[2::3] + np.uint32(5 * n)
            np.testing.assert_array_equal(g.insert(k, one, k + 1, one, upsert=upsert),
                                          o.insert(k, one, k + 1, one, upsert=upsert))
        _same_contents(g, o, 3 * n, 1, 1)
        few = np.repeat(keys[:60][np.arange(60) % 3 != 2], 200, axis=0)  # 40 keys
        ones = np.ones(len(few), np.uint32)
        assert g.update(few, ones, few + 7, ones).all()
        o.update(few, ones, few + 7, ones)
        _same_contents(g, o, 3 * n, 1, 1)
        erased = g.erase(few, ones)
        o.erase(few, ones)
        assert int(erased.sum()) == 40 and (np.bincount(few[:, 0], erased)[np.unique(few)] == 1).all()
        _same_contents(g, o, 3 * n, 1, 1)
        added = g.insert(few, ones, few + 9, ones, upsert=upsert)
        o.insert(few, ones, few + 9, ones, upsert=upsert)
        assert int(added.sum()) == (len(few) if upsert else 40)
        _same_contents(g, o, 3 * n, 1, 1)
    finally:
        g.close()


@pytest.mark.parametrize("n", [1, 5, 37, 400])
@pytest.mark.parametrize("maxK,maxV", [(150, 80), (92, 1), (2, 121)])
def test_plain_calls_on_chains_of_many_slabs(n, maxK, maxV):
    # Warps with one request and with 32; key rests and values that end beside
    # slab edges; keys that differ from a held one in their last slice only.
    rng = np.random.default_rng(n + maxK)
    ends = [e for e in (1, 2, 3, 31, 32, 33, 61, 62, 63, 64, 91, 92, 93, 121, 122, 149, 150) if e <= maxK]
    vends = [e for e in (1, 2, 29, 30, 31, 59, 60, 61, 80, 90, 119, 120, 121) if e <= maxV]
    kl, vl = rng.choice(ends, n).astype(np.uint32), rng.choice(vends, n).astype(np.uint32)
    keys = rng.integers(0, 1 << 32, (n, maxK), dtype=np.uint64).astype(np.uint32)
    keys[:, 0] = np.arange(n) // 3
    keys[np.arange(maxK)[None, :] >= kl[:, None]] = 0
    near = keys.copy()
    near[np.arange(n), kl - 1] ^= 1
    keys, kl, vl = np.concatenate([keys, near]), np.concatenate([kl, kl]), np.concatenate([vl, vl[::-1]])
    _, first = np.unique(np.concatenate([keys, kl[:, None]], axis=1), axis=0, return_index=True)
    keys, kl, vl = keys[first], kl[first], vl[first]
    m = len(kl)
    g, o = GpuIndex(pool_bytes=128 << 20), OracleIndex()

    def values():
        v = rng.integers(1, 1 << 32, (m, maxV), dtype=np.uint64).astype(np.uint32)
        l = rng.permutation(vl)
        v[np.arange(maxV)[None, :] >= l[:, None]] = 0
        return v, l

    try:
        half, some = rng.permutation(m)[:(m + 1) // 2], rng.permutation(m)[:(m + 1) // 2]
        v, l = values()
        np.testing.assert_array_equal(g.insert(keys[half], kl[half], v[half], l[half]),
                                      o.insert(keys[half], kl[half], v[half], l[half]))
        for upsert in (False, True):
            v, l = values()
            np.testing.assert_array_equal(g.update(keys, kl, v, l), o.update(keys, kl, v, l))
            np.testing.assert_array_equal(g.erase(keys[some], kl[some]), o.erase(keys[some], kl[some]))
            for maxv in (maxV, 1):
                for x, y in zip(g.find(keys, kl, maxv), o.find(keys, kl, maxv)):
                    np.testing.assert_array_equal(x, y)
            v, l = values()
            np.testing.assert_array_equal(g.insert(keys, kl, v, l, upsert=upsert), o.insert(keys, kl, v, l, upsert=upsert))
            _same_contents(g, o, m, maxK, maxV)
    finally:
        g.close()


@pytest.mark.parametrize("n", [2, 255, 256, 257, 1025, 75775, 75776, 151553, 227328, 310000])
@pytest.mark.parametrize("mixed", [False, True])
def test_updates_of_one_key_in_one_call(n, mixed):
    # Chunks of 256 to 1,024 requests per block, whole and ragged; a call
    # after smaller and larger ones (the table keeps the entries of earlier
    # calls).  Updates of one key have no order: the result is every request's,
    # the value one of theirs.
    g = GpuIndex(pool_bytes=64 << 20)
    rng = np.random.default_rng(n)
    held = 5000
    try:
        keys = np.stack([np.arange(held), np.arange(held) % 7], 1).astype(np.uint32)
        two, one = np.full(held, 2, np.uint32), np.ones(held, np.uint32)
        assert g.insert(keys, two, np.zeros((held, 1), np.uint32), one).all()
        for size in (n, 3, n):
            ids = rng.integers(0, held + 50, size)
            k = np.stack([ids, ids % 7], 1).astype(np.uint32)
            v = (np.arange(size, dtype=np.uint32) + 1)[:, None]
            l2, l1 = np.full(size, 2, np.uint32), np.ones(size, np.uint32)
            if mixed:
                types = np.where(np.arange(size) % 3 == 0, 2, 3).astype(np.uint8)
                res = np.array(g.mixed(types, k, l2, v, l1)[2])
                upd = types == 3
            else:
                res, upd = np.array(g.update(k, l2, v, l1)), np.ones(size, bool)
            np.testing.assert_array_equal(res[upd] != 0, ids[upd] < held)
            got, gl = g.find(keys, two, 1)
            assert (gl == 1).all()
            touched = np.unique(ids[upd & (ids < held)])
            written = got[touched, 0].astype(np.int64) - 1
            assert (ids[written] == touched).all() and upd[written].all()
            g.update(keys, two, np.zeros((held, 1), np.uint32), one)
    finally:
        g.close()


@pytest.mark.parametrize("form", ["insert", "upsert", "mixed", "batches", "grouped"])
@pytest.mark.parametrize("held,n", [(1, 3000), (14, 20000), (100, 80000), (3000, 150000)])
def test_one_call_grows_a_small_tree(form, held, n):
    # Nearly every insert needs a root or a full parent split, or a new layer
    # (keys in a few shared prefixes), and the nodes that lanes read first are
    # split again and again by other warps of the launch.
    rng = np.random.default_rng(held)
    keys = np.zeros((held + n, 5), np.uint32)
    keys[:, 0] = rng.integers(0, 3, held + n)
    keys[:, 1] = rng.permutation(held + n)
    keys[:, 2:] = rng.integers(0, 4, (held + n, 3))
    kl = rng.integers(2, 6, held + n).astype(np.uint32)
    keys[np.arange(5)[None, :] >= kl[:, None]] = 0
    vals, vl = np.arange(1, held + n + 1, dtype=np.uint32)[:, None], np.ones(held + n, np.uint32)
    g, o = GpuIndex(pool_bytes=256 << 20), OracleIndex()
    try:
        for x in (g, o):
            assert x.insert(keys[:held], kl[:held], vals[:held], vl[:held]).all()
        k, l, v, w = keys[held:], kl[held:], vals[held:], vl[held:]
        if form in ("insert", "upsert"):
            res = g.insert(k, l, v, w, upsert=form == "upsert")
        elif form == "mixed":
            res = g.mixed(np.zeros(n, np.uint8), k, l, v, w)[2]
        else:
            import torch
            from indexingpu_b200.masstree import pack_subbatches
            d = [torch.from_numpy(x).cuda() for x in (np.zeros(n, np.uint8), k, l, v, w)]
            out = torch.zeros(n, dtype=torch.bool, device="cuda")
            subs = [dict(zip(("types", "keys", "lens", "vals", "vlens", "results", "n"),
                             [x[p] for x in d] + [out[p], p.stop - p.start])) for p in (slice(0, n // 3), slice(n // 3, n))]
            g.t.reserve_batches(2, n)
            g.t.mixed_batches(torch.from_numpy(pack_subbatches(subs)).cuda(), 2, 5, 1, group_by_key=form == "grouped")
            g.t.sync()
            res = out.cpu().numpy()
        assert np.array(res).all() and o.insert(k, l, v, w).all()
        _same_contents(g, o, held + n, 5, 1)
    finally:
        g.close()


def test_one_call_of_ascending_keys():
    # More leaves come off one node during the launch than a walk may visit, and
    # more requests are left to tiles than the list for them has room for.
    n = 1200000
    g = GpuIndex(pool_bytes=48 << 20)
    try:
        keys = np.arange(n + 40, dtype=np.uint32)[:, None]
        one = np.ones(n + 40, np.uint32)
        assert g.insert(keys[:40], one[:40], keys[:40], one[:40]).all()
        assert g.insert(keys[40:], one[40:], keys[40:], one[40:]).all()
        got, gl = g.find(keys, one, 1)
        assert (gl == 1).all() and (got == keys).all()
        ok, count, msg = g.t.validate()
        assert ok and count == n + 40, msg
    finally:
        g.close()


@pytest.mark.parametrize("n,maxV,pool_mb", [(1500, 620, 8), (90000, 110, 96)])
def test_slabs_of_inserts_that_lanes_cannot_place(n, maxV, pool_mb):
    # The chains (of 21 and of 4 slabs) fill half of the pool.  Into a tree of 14
    # keys, lanes place few of them; what they took for the others has to serve
    # these in the same call (of the second one: in its second kernel).
    g, o = GpuIndex(pool_bytes=pool_mb << 20), OracleIndex()
    try:
        rng = np.random.default_rng(5)
        keys = rng.permutation(1 << 20)[:n + 14].astype(np.uint32)[:, None]
        vals = rng.integers(0, 1 << 32, (n + 14, maxV), dtype=np.uint64).astype(np.uint32)
        one, vl = np.ones(n + 14, np.uint32), np.full(n + 14, maxV, np.uint32)
        for x in (g, o):
            assert x.insert(keys[:14], one[:14], vals[:14], vl[:14]).all()
            assert x.insert(keys[14:], one[14:], vals[14:], vl[14:]).all()
        _same_contents(g, o, n + 14, 1, maxV)
    finally:
        g.close()


def test_a_chain_longer_than_a_shard():
    # A pool of 64 shards of 961 slabs; a value of 30,000 slices takes 1,000.
    maxV = 30000
    g, o = GpuIndex(pool_bytes=8 << 20), OracleIndex()
    try:
        rng = np.random.default_rng(6)
        keys = np.arange(20, dtype=np.uint32)[:, None]
        one = np.ones(20, np.uint32)
        short = np.full(20, 1, np.uint32)
        long = np.where(np.arange(20) % 5 == 0, maxV, 40).astype(np.uint32)
        for vl in (short, long, long):
            vals = rng.integers(0, 1 << 32, (20, maxV), dtype=np.uint64).astype(np.uint32)
            vals[np.arange(maxV)[None, :] >= vl[:, None]] = 0
            for x in (g, o):
                assert (x.insert if vl is short else x.update)(keys, one, vals, vl).all()
            _same_contents(g, o, 20, 1, maxV)
        more = keys + np.uint32(100)
        for x in (g, o):
            assert x.insert(more, one, vals, long).all()
        _same_contents(g, o, 40, 1, maxV)
    finally:
        g.close()


@pytest.mark.parametrize("last", [0xFFFFFFFD, 0xFFFFFFFE, 0xFFFFFFFF])
def test_combining_when_its_count_comes_round(last):
    # Request 0 is a find of the key that the others update: taken for their
    # leader (entries never written read as request 0 of call 0), it would keep
    # them from running.  The entries of the tree's own calls 1 and 2, of more
    # requests than the later ones, must be gone as well.
    g = GpuIndex(pool_bytes=64 << 20)
    try:
        held = 4000
        keys, one = np.arange(held, dtype=np.uint32)[:, None], np.ones(held, np.uint32)
        assert g.insert(keys, one, keys, one).all()
        for _ in range(2):
            assert g.update(keys, one, keys + 1, one).all()
        assert g.t._lib.mt_set_combine_epoch(g.t._h, last) == 0
        for call in range(4):
            n = 300
            ids = np.concatenate([[call], np.full(9, call), np.arange(10, n)]).astype(np.uint32)
            types = np.full(n, 3, np.uint8)
            types[0] = 2
            vals = (ids + np.uint32(1000 * (call + 1)))[:, None]
            res = np.array(g.mixed(types, ids[:, None], np.ones(n, np.uint32), vals, np.ones(n, np.uint32))[2])
            assert res[1:].all()
            got, gl = g.find(keys, one, 1)
            assert (gl == 1).all() and (got[ids, 0] == vals[:, 0]).all()
    finally:
        g.close()


@pytest.mark.parametrize("maxK,maxV", [(40, 8), (8, 40), (31, 17), (48, 48), (49, 48), (70, 30)])
@pytest.mark.parametrize("count", [1, 14, 60])
def test_scan_rows_around_the_width_of_one_lane(maxK, maxV, count):
    # Rows of 48, 96 and 97 slices, of keys alone and of values alone; chains that
    # end at and beside slab edges.
    import torch
    keys, kl, vals, vl = _edge_keys(2500, maxK, maxV, maxK + count)
    rng = np.random.default_rng(count)
    g, o = GpuIndex(pool_bytes=128 << 20), OracleIndex()
    try:
        for x in (g, o):
            x.insert(keys, kl, vals, vl)
        pick = rng.integers(0, len(kl), 300)
        lower, ll = keys[pick], kl[pick].copy()
        ll[::7] = np.minimum(ll[::7], 2)
        upper = lower.copy()
        upper[:, 1] = np.minimum(upper[:, 1].astype(np.int64) + 3, 0xFFFFFFFF).astype(np.uint32)
        ul = np.minimum(ll + 1, maxK).astype(np.uint32)
        for up, ulen in ((None, None), (upper, ul)):
            want = o.scan(lower, ll, count, up, ulen, maxV=maxV)
            got = g.scan(lower, ll, count, up, ulen, maxV=maxV)
            for x, y in zip(got, want):
                np.testing.assert_array_equal(x, y)
            d = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
            z = lambda *s: torch.zeros(s, dtype=torch.uint32, device="cuda")  # noqa: E731
            n = len(ll)
            okeys, oval = z(n, count, maxK), z(n, count, maxV)
            g.t.scan(d(lower), d(ll), maxK, count, n, d(up), d(ulen), out_keys=okeys)
            g.t.scan(d(lower), d(ll), maxK, count, n, d(up), d(ulen), values=oval, max_value_length=maxV)
            g.t.sync()
            np.testing.assert_array_equal(oval.cpu().numpy(), want[1])
            np.testing.assert_array_equal(okeys.cpu().numpy(), want[3])
    finally:
        g.close()


@pytest.mark.parametrize("n", [18944, 18945, 20011])
@pytest.mark.parametrize("count", [1, 2, 3, 4])
def test_many_scans_of_few_results(n, count):
    keys, kl, vals, vl = _edge_keys(4000, 17, 9, 3)
    rng = np.random.default_rng(n)
    g, o = GpuIndex(pool_bytes=64 << 20), OracleIndex()
    try:
        for x in (g, o):
            x.insert(keys, kl, vals, vl)
        pick = rng.integers(0, len(kl), n)
        lower, ll = keys[pick], kl[pick]
        near = np.arange(n) % 3 == 0
        lower[near, ll[near] - 1] ^= 1
        upper, ul = lower.copy(), ll.copy()
        upper[:, 0] = np.minimum(upper[:, 0].astype(np.int64) + np.arange(n) % 2, 0xFFFFFFFF).astype(np.uint32)
        for up, ulen in ((None, None), (upper, ul)):
            want = o.scan(lower, ll, count, up, ulen, maxV=9)
            for conc in (False, True):
                for x, y in zip(g.scan(lower, ll, count, up, ulen, maxV=9, concurrent=conc), want):
                    np.testing.assert_array_equal(x, y)
    finally:
        g.close()
