"""What a program using this index spends its time on, as measurable cases.

Each case is one pass through the public entry points of
`indexingpu_b200.GpuMasstree` on a tree that the program already holds: batched
finds, mixed batches from device and from host buffers, many sub-batches in one
call, range scans, the plain write calls, a request stream through the serving
loop, and building an index from nothing.  Keys and values are u32 slices, made
on the GPU from the seed:

  short     1..maxk random slices (the plain small workload)
  prefixed  2..maxk slices, the first (up to) four shared by many keys (the
            mixed workload: 4096 prefixes under a 16M-key tree)
  pair      two slices of a random 64-bit number (the scan workload)
  fixed     exactly maxk random slices, length arrays left out
  long      1..maxk slices, the first two shared; with long values, so that a
            key's rest and value fill several slabs

A pass leaves the tree with the keys it found (what it inserts it erases again,
what it erases it puts back), so that passes can follow each other on one tree,
and no two requests of one unordered batch conflict, so that every result is
defined: ids are divided by `id % 4` into keys that are only found, keys that
one batch updates and the next one finds, keys that are only updated, and keys
that one batch erases and the next one inserts again.
"""
import math

import numpy as np
import torch

from indexingpu_b200 import GpuMasstree
from indexingpu_b200.masstree import pack_subbatches

INSERT, ERASE, FIND, UPDATE = 0, 1, 2, 3
FRESH = 1 << 30   # ids from here on are not in the tree between passes
ABSENT = 1 << 31  # ids from here on are never in the tree


def listed():
    return [
        # A small lookup call (a service answering one request): launch and
        # latency of one dependent walk.
        dict(name="find-small", op="find", keys="short", maxk=8, maxv=2, tree=50000, n=1000, theta=0.0, hits=0.9,
             concurrent=False),
        # The plain small workload: 1M finds, half of them misses, 1M keys.
        dict(name="find-1m", op="find", keys="short", maxk=8, maxv=2, tree=1 << 20, n=1 << 20, theta=0.0, hits=0.5,
             concurrent=False),
        # A small mixed batch, as an online store sends them.
        dict(name="mixed-small", op="mixed", keys="prefixed", maxk=16, maxv=8, tree=200000, n=2000, theta=0.99,
             host=False),
        # The headline workload: mixed batches of 1M on 16M keys
        # (50/30/10/10 find/insert/update/erase, Zipf 0.99).
        dict(name="mixed-1m", op="mixed", keys="prefixed", maxk=16, maxv=8, tree=1 << 24, n=1 << 20, theta=0.99,
             host=False),
        # The same requests from pinned host buffers, results read back.
        dict(name="mixed-host", op="mixed", keys="prefixed", maxk=16, maxv=8, tree=1 << 22, n=500000, theta=0.99,
             host=True),
        # Long documents' keys and values (multi-slab chains), ragged.
        dict(name="mixed-long", op="mixed", keys="long", maxk=100, maxv=60, tree=100000, n=50021, theta=0.5, host=False),
        # Many uneven sub-batches in one call, the requests on a key in order.
        dict(name="batches", op="batches", keys="prefixed", maxk=16, maxv=8, tree=1 << 22, pairs=10, least=1024,
             most=1 << 17, theta=0.99, grouped=True),
        # Short range reads over 32M fixed two-slice keys.
        dict(name="scan-100", op="scan", keys="pair", maxk=2, maxv=1, tree=1 << 25, n=400000, count=100, upper=False),
        # Bounded ranges over ragged keys that share prefixes (trie layers).
        dict(name="scan-range", op="scan", keys="prefixed", maxk=16, maxv=8, tree=1 << 20, n=30011, count=13,
             upper=True),
        # The plain calls one after the other: insert, update (Zipf 0.99),
        # find, erase; keys of fixed length without length arrays.
        dict(name="writes", op="writes", keys="fixed", maxk=8, maxv=1, tree=1 << 22, n=300000, theta=0.99,
             upsert=False),
        # A stream of small requests through the device-resident loop.
        dict(name="serve", op="serve", keys="prefixed", maxk=16, maxv=8, tree=1 << 21, n=200000, most=1024, theta=0.99),
        # An index made from nothing, looked at once and dropped.
        dict(name="build", op="build", keys="short", maxk=8, maxv=2, tree=1 << 20),
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("find", "find", "mixed", "mixed", "mixed", "batches", "scan", "scan", "writes", "serve", "build"))
    keys = rng.choice(("short", "prefixed", "fixed", "long"))
    c = dict(op=op, keys=keys)
    if keys == "short":
        c.update(maxk=rng.randint(2, 12), maxv=rng.randint(1, 8))
    elif keys == "prefixed":
        c.update(maxk=rng.randint(6, 24), maxv=rng.randint(1, 12))
    elif keys == "fixed":
        c.update(maxk=rng.randint(2, 12), maxv=rng.randint(1, 4))
    else:
        c.update(maxk=rng.randint(40, 150), maxv=rng.randint(1, 80))
    big = keys != "long"
    c["tree"] = _between(rng, 5000, 1 << 23 if big else 100000)
    n = _between(rng, 500, 1 << 20 if big else 60000)
    theta = rng.choice((0.0, 0.5, 0.99))
    if op == "find":
        c.update(n=n, theta=theta, hits=round(rng.uniform(0.1, 1.0), 2), concurrent=rng.random() < 0.5)
    elif op == "mixed":
        c.update(n=min(n, 500000), theta=theta, host=rng.random() < 0.3)
    elif op == "batches":
        c.update(pairs=rng.randint(2, 12), least=rng.randint(300, 1500), most=_between(rng, 2000, 1 << 17 if big else 8000),
                 theta=theta, grouped=rng.random() < 0.6)
    elif op == "scan":
        c.update(n=_between(rng, 300, 60000 if big else 3000), count=_between(rng, 1, 100), upper=rng.random() < 0.5)
        if rng.random() < 0.4:
            c.update(keys="pair", maxk=2, maxv=1)
    elif op == "writes":
        c.update(n=min(n, 300000), theta=theta, upsert=rng.random() < 0.5)
    elif op == "serve":
        c.update(n=_between(rng, 2000, 200000 if big else 20000), most=_between(rng, 4, 2048), theta=theta)
    else:
        c["tree"] = _between(rng, 2000, 1 << 20 if big else 50000)
    return c


# ---- inputs ------------------------------------------------------------------

def _lsr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _mix(x):
    """A bijection of 64-bit words (splitmix64's finalizer)."""
    x = (x ^ _lsr(x, 30)) * -0x40A7B892E31B1A47
    x = (x ^ _lsr(x, 27)) * -0x6B2FB644ECCEEE15
    return x ^ _lsr(x, 31)


def _rnd(seed, stream, ids):
    """64 random bits for (seed, stream, id)."""
    return _mix(_mix(ids * 0x2545F4914F6CDD1D + stream * 1000003 + 17) + seed * 7919)


def _u32(x):
    return _lsr(x, 32)


def _below(seed, stream, ids, n):
    return _u32(_rnd(seed, stream, ids)) * n >> 32


def _word(x):
    """Low 32 bits as an int32 tensor."""
    return ((x << 32) >> 32).to(torch.int32)


def _unique32(ids):
    """A bijection of 32-bit ids."""
    m = 0xFFFFFFFF
    u = (ids * 0x9E3779B1) & m
    u = ((u ^ (u >> 16)) * 0x7FEB352D) & m
    u = ((u ^ (u >> 15)) * 0x846CA68B) & m
    return u ^ (u >> 16)


def _prefixes(case):
    return max(16, min(4096, case["tree"] // 64))


def _keys(case, seed, ids):
    """Keys of ids (distinct ids, distinct keys): rows and lengths (None: all maxk)."""
    kind, maxk, n = case["keys"], case["maxk"], ids.numel()
    rows = torch.zeros((n, maxk), dtype=torch.int32, device=ids.device)
    if kind == "pair":
        x = _mix(_unique32(ids) + (_unique32(ids ^ 0x55AA55AA) << 32) + seed)
        rows[:, 0], rows[:, 1] = _word(_u32(x)), _word(x)
        return rows, torch.full((n,), 2, dtype=torch.int32, device=ids.device)
    shared, prefixes, least = 0, 1, 1
    if kind == "prefixed":
        shared, prefixes, least = 4, _prefixes(case), 2
    elif kind == "long":
        shared, prefixes = 2, 512
    lens = least + _below(seed, 1, ids, maxk - least + 1)
    if kind == "fixed":
        lens = torch.full_like(ids, maxk)
    prefix = _below(seed, 2, ids, prefixes)
    uid = _word(_unique32(ids))
    for s in range(maxk):
        col = _word(_u32(_rnd(seed, 10 + s, prefix + (1 << 40) if s < shared else ids)))
        col = torch.where(lens == s + 1, uid, col)
        rows[:, s] = torch.where(lens > s, col, torch.zeros_like(col))
    return rows, None if kind == "fixed" else lens.to(torch.int32)


def _values(case, seed, ids, version):
    """Values of ids in a version (0: as first inserted): rows and lengths."""
    maxv = case["maxv"]
    key = ids * 4 + version
    lens = 1 + _below(seed, 5, key, maxv)
    if case["keys"] == "fixed":
        lens = torch.full_like(ids, maxv)
    rows = torch.zeros((ids.numel(), maxv), dtype=torch.int32, device=ids.device)
    for s in range(maxv):
        col = _word(_u32(_rnd(seed, 1000 + s, key)))
        rows[:, s] = torch.where(lens > s, col, torch.zeros_like(col))
    return rows, lens.to(torch.int32)


def _ranks(n, theta, u):
    """Zipf(theta) ranks in [0, n) from uniforms (theta 0: uniform)."""
    if theta == 0.0 or n < 3:
        return (u * n).long().clamp_(0, max(0, n - 1))
    i = torch.arange(1, n + 1, dtype=torch.float64, device=u.device)
    zeta = float((i ** -theta).sum())
    zeta2 = 1.0 + 0.5 ** theta
    eta = (1 - (2.0 / n) ** (1 - theta)) / (1 - zeta2 / zeta)
    r = (n - 1) * (eta * u - eta + 1).clamp_(min=0) ** (1.0 / (1.0 - theta))
    r = torch.where(u * zeta < 1.0, torch.zeros_like(r), torch.where(u * zeta < zeta2, torch.ones_like(r), r))
    return r.long().clamp_(0, n - 1)


def _arange(first, n):
    return torch.arange(first, first + n, dtype=torch.int64, device="cuda")


def _uniform(seed, stream, n):
    return _lsr(_rnd(seed, stream, _arange(0, n)), 11).double() * (1.0 / (1 << 53))


def _shuffled(seed, stream, n):
    return torch.argsort(_rnd(seed, stream, _arange(0, n)))


def _pool(case, extra):
    """Pool bytes for the case's keys and `extra` more, with room to spare."""
    chain = 1 + (case["maxk"] + case["maxv"]) // 30
    return int(136 * 1.5 * (chain + 1) * (case["tree"] + 2 * extra)) + (64 << 20)


def _tree(case, seed, extra):
    t = GpuMasstree(pool_bytes=_pool(case, extra), tile_size=8)
    t.set_write_tile_size(32)
    t.set_scan_tile_size(4)
    n = case["tree"]
    for first in range(0, n, 1 << 24):
        ids = _arange(first, min(n - first, 1 << 24))
        k, l = _keys(case, seed, ids)
        v, vl = _values(case, seed, ids, 0)
        t.insert(k, case["maxk"], l, v, case["maxv"], vl, ids.numel())
        t.sync()
    return t


def _batch(case, seed, parts, number):
    """One unordered batch of (kind, ids, value version) parts, shuffled."""
    kind = torch.cat([torch.full((p[1].numel(),), p[0], dtype=torch.int64, device="cuda") for p in parts])
    ids = torch.cat([p[1] for p in parts])
    version = torch.cat([torch.full_like(p[1], p[2]) for p in parts])
    order = _shuffled(seed, 77 + number, ids.numel())
    kind, ids, version = kind[order], ids[order], version[order]
    keys, lens = _keys(case, seed, ids)
    vals, vlens = _values(case, seed, ids, version)
    blank = (kind == FIND) | (kind == ERASE)
    vals[blank] = 0
    vlens[blank] = 0
    return dict(types=kind.to(torch.uint8), keys=keys, lens=lens, vals=vals, vlens=vlens,
                results=torch.zeros(ids.numel(), dtype=torch.bool, device="cuda"), n=ids.numel())


def _pair(case, seed, n, at):
    """Two batches of n requests, half of them finds: the second one undoes what
    the first one inserted and erased.  `at`: the pair's number among the
    case's (pairs use other fresh and erased keys)."""
    quarter = max(1, case["tree"] // 4)
    theta = case["theta"]
    n_erase = max(1, min(n // 10, quarter // 4))
    n_insert = max(1, n * 3 // 10)
    n_update = max(1, n // 10)
    s = seed + 1000 * (at + 1)

    def some(stream, m, cls):
        return 4 * _ranks(quarter, theta, _uniform(s, stream, m)) + cls

    fresh = FRESH + (at << 21) + _arange(0, n_insert)
    erased = torch.unique(4 * ((_arange(0, n_erase) * 7 + at * 1009) % quarter) + 3)
    first_upd, second_upd = some(1, n_update, 1), some(2, n_update, 2)
    # A twentieth of the inserts meet a key that is there, and of the updates
    # and erases one that is not.
    there = 4 * (_below(s, 3, _arange(0, n_insert // 20 + 1), quarter))
    gone = ABSENT + _arange(0, max(1, n_update // 20))
    m = n - n_insert - n_update - erased.numel() - there.numel() - 2 * gone.numel()
    finds = some(4, max(1, m), 0)
    finds[::16] = ABSENT + (1 << 20) + finds[::16]
    fwd = [(FIND, finds, 0), (INSERT, fresh, 0), (INSERT, there, 0), (UPDATE, first_upd, 1), (UPDATE, gone, 1),
           (ERASE, erased, 0), (ERASE, gone + (1 << 19), 0)]
    m = n - n_insert - n_update - erased.numel()
    finds = torch.cat([some(5, max(1, m - m // 4), 0),
                       first_upd[_below(s, 6, _arange(0, max(1, m // 4)), first_upd.numel())]])
    inv = [(FIND, finds, 0), (ERASE, fresh, 0), (UPDATE, second_upd, 1), (INSERT, erased, 0)]
    return _batch(case, seed, fwd, 2 * at), _batch(case, seed, inv, 2 * at + 1)


def _sizes(case):
    """Sizes of the sub-batch pairs, spread over the logarithm of [least, most]."""
    return [int(case["least"] * (case["most"] / case["least"]) ** (0.5 + 0.618034 * i - int(0.5 + 0.618034 * i)))
            for i in range(case["pairs"])]


def prepare(case, seed):
    op, maxk, maxv = case["op"], case["maxk"], case["maxv"]
    s = dict(case=case, maxk=maxk, maxv=maxv)
    if op == "find":
        s["tree"] = _tree(case, seed, 0)
        n = case["n"]
        ids = _ranks(case["tree"], case["theta"], _uniform(seed, 3, n))
        miss = _uniform(seed, 4, n) >= case["hits"]
        ids = torch.where(miss, ABSENT + _arange(0, n), ids)
        s["keys"], s["lens"] = _keys(case, seed, ids)
        s["vals"] = torch.zeros((n, maxv), dtype=torch.int32, device="cuda")
        s["vlens"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif op in ("mixed", "serve"):
        s["tree"] = _tree(case, seed, case["n"])
        s["batches"] = _pair(case, seed, case["n"], 0)
        if op == "serve":
            s["requests"] = [_requests(case, seed + k, b["n"]) for k, b in enumerate(s["batches"])]
        elif case["host"]:
            s["batches"] = [{k: v.cpu().pin_memory() if torch.is_tensor(v) else v for k, v in b.items()}
                            for b in s["batches"]]
    elif op == "batches":
        sizes = _sizes(case)
        s["tree"] = _tree(case, seed, 2 * sum(sizes))
        subs = [b for i, n in enumerate(sizes) for b in _pair(case, seed, n, i)]
        s["subs"] = subs
        # The rows of all sub-batches in one buffer per field, as a program
        # that gathers them would lay them out.
        for f in ("types", "keys", "lens", "vals", "vlens", "results"):
            if subs[0][f] is None:
                continue
            s[f] = torch.cat([b[f] for b in subs])
            at = 0
            for b in subs:
                b[f] = s[f][at:at + b["n"]]
                at += b["n"]
        s["desc"] = torch.from_numpy(pack_subbatches(subs)).cuda()
        s["tree"].reserve_batches(len(subs), sum(b["n"] for b in subs))
    elif op == "scan":
        s["tree"] = _tree(case, seed, 0)
        n, count = case["n"], case["count"]
        ids = _below(seed, 3, _arange(0, n), case["tree"])
        # Half of the lower bounds are keys, half lie between keys.
        ids = torch.where(_uniform(seed, 4, n) < 0.5, ids, ABSENT + ids)
        s["lower"], s["lower_lens"] = _keys(case, seed, ids)
        s["upper"] = s["upper_lens"] = None
        if case["upper"]:
            # Up to about `count` keys further on: a step in the slice after
            # the shared ones (or the key's last one).
            s["upper"], s["upper_lens"] = s["lower"].clone(), s["lower_lens"]
            at = 4 if case["keys"] == "prefixed" else (2 if case["keys"] == "long" else 0)
            lens = s["lower_lens"].long() if s["lower_lens"] is not None else torch.full_like(ids, maxk)
            at = torch.clamp(lens - 1, max=at)[:, None]
            among = {"prefixed": case["tree"] // _prefixes(case), "long": case["tree"] // 512}.get(case["keys"], case["tree"])
            step = (1 << 32) * count // max(count, among)
            x = s["upper"].gather(1, at).long() & 0xFFFFFFFF
            s["upper"].scatter_(1, at, _word((x + step).clamp_(max=0xFFFFFFFF)))
        z = lambda *shape: torch.zeros(shape, dtype=torch.int32, device="cuda")  # noqa: E731
        s.update(counts=z(n), vals=z(n, count, maxv), vlens=z(n, count), okeys=z(n, count, maxk), oklens=z(n, count))
    elif op == "writes":
        n = case["n"]
        s["tree"] = _tree(case, seed, n)
        quarter = max(1, case["tree"] // 4)
        fresh = FRESH + _arange(0, n)
        fresh[::20] = 4 * _below(seed, 3, fresh[::20], quarter)
        upd = 4 * _ranks(quarter, case["theta"], _uniform(seed, 4, n)) + 1
        upd[::32] = ABSENT + upd[::32]
        gone = torch.where(fresh < FRESH, fresh + ABSENT, fresh)
        for at, (name, ids, version) in enumerate((("ins", fresh, 0), ("upd", upd, 1), ("era", gone, 0))):
            order = _shuffled(seed, 9 + at, n)
            k, l = _keys(case, seed, ids[order])
            v, vl = _values(case, seed, ids[order], version)
            if case["keys"] == "fixed":
                vl = None
            s[name] = (k, l, v, vl, torch.zeros(n, dtype=torch.bool, device="cuda"))
        s["vals"] = torch.zeros((n, maxv), dtype=torch.int32, device="cuda")
        s["vlens"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif op == "build":
        n = case["tree"]
        order = _shuffled(seed, 9, n)
        s["keys"], s["lens"] = _keys(case, seed, order)
        s["in_vals"], s["in_vlens"] = _values(case, seed, order, 0)
        s["results"] = torch.zeros(n, dtype=torch.bool, device="cuda")
        s["vals"] = torch.zeros((n, maxv), dtype=torch.int32, device="cuda")
        s["vlens"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


def _requests(case, seed, total):
    """Requests of 1..most ops (log-uniform), all there at the start: the first
    op and the ops of each, and arrival times (host arrays)."""
    rng = np.random.default_rng(seed & 0x7FFFFFFF)
    n = np.exp(rng.random(total) * math.log(case["most"] + 1)).astype(np.int64).clip(1, case["most"])
    n = n[:int(np.searchsorted(np.cumsum(n), total)) + 1]
    first = np.concatenate([[0], np.cumsum(n)[:-1]])
    n = np.minimum(n, total - first)
    return first.astype(np.uint32), n.astype(np.uint32), np.zeros(len(n), np.uint64)


# ---- one pass ------------------------------------------------------------------

def run(s):
    case, maxk, maxv = s["case"], s["maxk"], s["maxv"]
    op = case["op"]
    if op == "find":
        s["tree"].find(s["keys"], maxk, s["lens"], s["vals"], maxv, s["vlens"], case["n"], concurrent=case["concurrent"])
        return s["vals"], s["vlens"]
    if op == "mixed":
        call = s["tree"].mixed_batch_host if case["host"] else s["tree"].mixed_batch
        for b in s["batches"]:
            call(b["types"], b["keys"], maxk, b["lens"], b["vals"], maxv, b["vlens"], b["results"], b["n"])
        if case["host"]:
            s["tree"].sync()  # the results are read on the host
        return [(b["vals"], b["vlens"], b["results"]) for b in s["batches"]]
    if op == "batches":
        s["tree"].mixed_batches(s["desc"], len(s["subs"]), maxk, maxv, group_by_key=case["grouped"])
        return s["vals"], s["vlens"], s["results"]
    if op == "scan":
        s["tree"].scan(s["lower"], s["lower_lens"], maxk, case["count"], case["n"], upper_keys=s["upper"],
                       upper_key_lengths=s["upper_lens"], counts=s["counts"], values=s["vals"], max_value_length=maxv,
                       value_lengths=s["vlens"], out_keys=s["okeys"], out_key_lengths=s["oklens"])
        return s["counts"], s["vals"], s["vlens"], s["okeys"], s["oklens"]
    if op == "writes":
        t, n = s["tree"], case["n"]
        k, l, v, vl, r = s["ins"]
        t.insert(k, maxk, l, v, maxv, vl, n, update_if_exists=case["upsert"], results=r)
        k, l, v, vl, r = s["upd"]
        t.update(k, maxk, l, v, maxv, vl, n, results=r)
        t.find(k, maxk, l, s["vals"], maxv, s["vlens"], n)
        k, l, v, vl, r = s["era"]
        t.erase(k, maxk, l, n, results=r)
        return s["ins"][4], s["upd"][4], s["vals"], s["vlens"], s["era"][4]
    if op == "serve":
        for b, (first, nops, arrival) in zip(s["batches"], s["requests"]):
            s["tree"].serve(b["types"], b["keys"], maxk, b["lens"], b["vals"], maxv, b["vlens"], b["results"], first,
                            nops, arrival)
        return [(b["vals"], b["vlens"], b["results"]) for b in s["batches"]]
    n = case["tree"]
    with GpuMasstree(pool_bytes=_pool(case, 0), tile_size=8) as t:
        t.set_write_tile_size(32)
        t.insert(s["keys"], maxk, s["lens"], s["in_vals"], maxv, s["in_vlens"], n, results=s["results"])
        t.find(s["keys"], maxk, s["lens"], s["vals"], maxv, s["vlens"], n)
        t.sync()
    return s["results"], s["vals"], s["vlens"]


# ---- what a pass cannot do without ----------------------------------------------

def work(case):
    """Each request's key, value and result once, and once more the key and value
    that the index holds for it (read by a find, written by an insert)."""
    maxk, maxv, kind = case["maxk"], case["maxv"], case["keys"]
    klen = maxk if kind in ("fixed", "pair") else (maxk + (2 if kind == "prefixed" else 1)) / 2
    vlen = maxv if kind == "fixed" else (maxv + 1) / 2
    row = 4 * (klen + vlen)
    one = 2 * row + 9  # in or out, in the index, lengths and kind
    op = case["op"]
    if op == "find":
        n = case["n"] * (4 * klen + 8 + case["hits"] * (4 * klen + 8 * vlen))
    elif op in ("mixed", "serve"):
        n = 2 * case["n"] * one
    elif op == "batches":
        n = 2 * sum(_sizes(case)) * one
    elif op == "scan":
        n = case["n"] * (4 * klen + 8 + case["count"] * (2 * row + 8))
    elif op == "writes":
        n = 4 * case["n"] * one
    else:
        n = 2 * case["tree"] * one
    return {"bytes": float(n), "flops": 0.0}


def tolerance(case):
    return "exact"  # words, lengths and truth values
