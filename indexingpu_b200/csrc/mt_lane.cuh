// One request per thread: the batch kernels' way through the tree.
//
// A lane walks its request's path alone, with the whole 128-byte node in its
// registers (four 32-byte loads), so a warp has 32 independent walks in flight
// where the tile code (mt_tree.cuh) has 32 / T, and a node visit costs no
// shuffle, vote or reduction.  What benefits from neighbouring lanes reading
// neighbouring words (suffix chains, key rests, values) is done by eight lanes
// per request, four requests at a time (warp_chains).
#pragma once
#include "mt_internal.cuh"

namespace mtb {

// Loads of node images by single lanes.  With concurrent writers the first
// attempt is a plain load, which may hit L1: an image of an earlier moment of
// this launch is as good as any (B-link nodes are never unlinked while a launch
// runs, so a stale interior node still leads to its key through sibling links,
// and requests of one batch have no order), and the checksum rejects a torn
// one, which is then read again from L2.  The upper levels of the tree, which
// every request passes, thus come from L1 instead of one L2 line each.
MT_DEV void lane_load_weak(const uint32_t* a, uint32_t (&w)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    asm volatile("ld.global.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[8 * q]), "=r"(w[8 * q + 1]), "=r"(w[8 * q + 2]), "=r"(w[8 * q + 3]), "=r"(w[8 * q + 4]),
                   "=r"(w[8 * q + 5]), "=r"(w[8 * q + 6]), "=r"(w[8 * q + 7])
                 : "l"(a + 8 * q) : "memory");
}
MT_DEV void lane_load_relaxed(const uint32_t* a, uint32_t (&w)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    asm volatile("ld.relaxed.gpu.global.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[8 * q]), "=r"(w[8 * q + 1]), "=r"(w[8 * q + 2]), "=r"(w[8 * q + 3]), "=r"(w[8 * q + 4]),
                   "=r"(w[8 * q + 5]), "=r"(w[8 * q + 6]), "=r"(w[8 * q + 7])
                 : "l"(a + 8 * q) : "memory");
}

MT_DEV uint32_t lane_checksum(const uint32_t (&w)[32]) {
  uint32_t h = 0;
#pragma unroll
  for (int g = 0; g < 32; ++g) h += csum_term((uint32_t)g, w[g]);
  return h;
}

// A verified image of node i (bounded reloads, as node::load_verified).
template <bool CONC>
MT_DEV bool lane_read_node(const pool_view& p, uint32_t i, uint32_t (&w)[32]) {
  lane_load_weak(p.addr(i), w);
  if (!CONC) return true;
  for (uint32_t r = 0; lane_checksum(w) != w[WORD_CSUM]; ++r) {
    if (r >= kTornRetries) {
      record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
      return false;
    }
    lane_load_relaxed(p.addr(i), w);
  }
  return true;
}

// The same from L2: the node's latest published image.
MT_DEV bool lane_read_fresh(const pool_view& p, uint32_t i, uint32_t (&w)[32]) {
  lane_load_relaxed(p.addr(i), w);
  for (uint32_t r = 0; lane_checksum(w) != w[WORD_CSUM]; ++r) {
    if (r >= kTornRetries) {
      record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
      return false;
    }
    lane_load_relaxed(p.addr(i), w);
  }
  return true;
}

// Bits 2e of the entries e < n of a border node whose key continues past its
// slice (more) or ends at it (!more).
MT_DEV uint32_t lane_eligible(uint32_t meta, uint32_t ks, bool more) {
  const uint32_t n = meta & META_COUNT;
  return (more ? ks : ~ks) & 0x01555555u & ((1u << (2u * n)) - 1u);
}

// Where a request's key belongs: the border node of its last layer and, when
// the node has an entry for (slice, continues), that entry.
struct lane_place {
  uint32_t idx;     // the border node
  uint32_t parent;  // the interior node the walk came through to its level (kInvalid: none, or not known)
  uint32_t root;    // root slab of the border node's layer
  uint32_t layer;   // trie layer (the key's slice index) of the border node
  uint32_t state;   // the entry's key state
  uint32_t val;     // the entry's value word
  bool found;
};

// Walk from the root of layer 0 to the key's place.  False on a (recorded)
// error.
template <bool CONC>
MT_DEV bool lane_locate(const tree_view& tv, const uint32_t* key, uint32_t klen, lane_place& at) {
  const pool_view& p = tv.pool;
  uint32_t idx = tv.root, layer = 0, hops = 0;
  uint32_t slice = key[0];
  bool more = klen > 1u;
  uint32_t w[32];
  at.found = false;
  at.layer = 0;
  at.parent = kInvalid;
  at.root = idx;
  while (true) {
    if (!p.valid(idx) || ++hops > kMaxHops) {
      record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
      return false;
    }
    if (!lane_read_node<CONC>(p, idx, w)) return false;
    const uint32_t meta = w[WORD_META];
    if ((meta & META_SIB) && slice > w[WORD_HIGH]) {
      idx = w[WORD_SIB];
      continue;
    }
    if (!(meta & META_BORDER)) {
      // The first separator >= slice; separators past the count are skipped.
      const uint32_t n = meta & META_COUNT;
      uint32_t child = kInvalid;
#pragma unroll
      for (int e = kMaxEntries - 1; e >= 0; --e)
        if ((uint32_t)e < n && slice <= w[2 * e]) child = w[2 * e + 1];
      at.parent = idx;
      idx = child;  // none: caught as an invalid slab above
      continue;
    }
    const uint32_t ok = lane_eligible(meta, w[WORD_KS], more);
    uint32_t hit = 0, val = 0;
#pragma unroll
    for (int e = 0; e < kMaxEntries; ++e)
      if (w[2 * e] == slice && (ok & (1u << (2 * e)))) {
        hit = 1u << (2 * e);
        val = w[2 * e + 1];
      }
    at.layer = layer;
    at.idx = idx;
    if (!hit) return true;
    const uint32_t state = (more ? KS_MORE : 0u) | ((w[WORD_KS] & (hit << 1)) ? KS_SLAB : 0u);
    if (state != KS_LINK) {
      at.found = true;
      at.state = state;
      at.val = val;
      return true;
    }
    idx = val;
    at.root = val;
    at.parent = kInvalid;
    ++layer;
    slice = key[layer];
    more = layer + 1u < klen;
  }
}

// For every lane with `want`: compare its key rest K[0..lk) with that of the
// chain at `head` (lk 0 for a chain that holds a value only) and, where equal
// and out is not null, copy at most maxV value slices.  Eight lanes serve one
// request, lane r of them the words r, r+8, r+16 and r+24 of a slab: every load
// and store covers whole 32-byte sectors of four requests' lines.  Only the
// sectors that the key rest and maxV value slices can reach are read, and four
// requests' loads (per eight lanes) are in flight together.  Called by the
// whole warp; eq and vlen are set for the lanes with want.
template <bool VALUES>
MT_DEV void warp_chains(const pool_view& p, bool want, uint32_t head, const uint32_t* K, uint32_t lk, uint32_t* out,
                        uint32_t maxV, bool& eq, uint32_t& vlen) {
  constexpr int kRound = 4;
  const uint32_t lane = lane_id();
  const uint32_t r8 = lane & 7u, first = lane & 24u;
  const uint32_t todo = __ballot_sync(0xFFFFFFFFu, want);
  if (todo == 0u) return;
  const uint32_t columns = todo | (todo >> 8) | (todo >> 16) | (todo >> 24);  // bit i: lane i of some eight lanes
  for (int base = 0; base < 8; base += kRound) {
    if (!((columns >> base) & ((1u << kRound) - 1u))) continue;
    uint32_t c[kRound][4], kw[kRound][4];
#pragma unroll
    for (int i = 0; i < kRound; ++i) {
      const uint32_t src = first + base + i;
      const uint32_t hd = __shfl_sync(0xFFFFFFFFu, head, src);
      const uint32_t need = __shfl_sync(0xFFFFFFFFu, lk, src) + (VALUES ? maxV : 0u);
      const uint32_t n = min(__shfl_sync(0xFFFFFFFFu, lk, src), kSufData);
      const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
      const bool act = (todo >> src) & 1u;
      const uint32_t* a = p.addr(act ? hd : 0u) + r8;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;
        c[i][q] = 0u;
        if (act && (g < need || g >= kSufData)) c[i][q] = a[8 * q];
        kw[i][q] = (act && g < n) ? k[g] : 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < kRound; ++i) {
      const uint32_t src = first + base + i;
      const bool act = (todo >> src) & 1u;
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
      const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
      const uint32_t hdr = __shfl_sync(0xFFFFFFFFu, c[i][3], first + SUF_WORD_HDR % 8);
      uint32_t nx = __shfl_sync(0xFFFFFFFFu, c[i][3], first + SUF_WORD_NEXT % 8);
      const uint32_t vl = hdr >> 16;
      bool same = (hdr & kMaxLen16) == n;
      bool differs = false;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;
        if (act && g < kSufData && g < n) differs |= c[i][q] != kw[i][q];
      }
      const uint32_t other = __ballot_sync(0xFFFFFFFFu, differs);  // by every lane, whatever `same` is
      same = same && !((other >> first) & 0xFFu);
      uint32_t* o = nullptr;
      uint32_t last = n;  // data slices [0, n) are compared, [n, last) copied
      if (VALUES) {
        o = reinterpret_cast<uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(out), src));
        if (o != nullptr) last = n + min(vl, maxV);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t g = r8 + 8u * q;
          if (act && same && g < kSufData && g >= n && g < last) o[g - n] = c[i][q];
        }
      }
      // Chains of several slabs.
      for (uint32_t at = kSufData; __any_sync(0xFFFFFFFFu, act && same && at < last); at += kSufData) {
        const bool on = act && same && at < last && p.valid(nx);
        same = same && (on || at >= last || at >= n);  // a chain cut short cannot hold the key
        uint32_t d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = on ? p.addr(nx)[r8 + 8u * q] : 0u;
        differs = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t g = r8 + 8u * q;
          if (on && g < kSufData && at + g < n) differs |= d[q] != k[at + g];
        }
        const uint32_t rest = __ballot_sync(0xFFFFFFFFu, differs);
        same = same && !((rest >> first) & 0xFFu);
        if (VALUES) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t g = r8 + 8u * q;
            if (on && same && g < kSufData && at + g >= n && at + g < last) o[at + g - n] = d[q];
          }
        }
        nx = __shfl_sync(0xFFFFFFFFu, d[3], first + SUF_WORD_NEXT % 8);
        if (!on) nx = kInvalid;
      }
      if ((lane & 7u) == (uint32_t)(base + i)) {
        eq = same;
        vlen = vl;
      }
    }
  }
}

// Requests per warp and round: 32 on large batches; fewer on small ones, so
// that every warp of the launch gets work and the batch ends after one walk's
// latency.  Slot j of a round is served by lane (j % 4) * 8 + j / 4, which
// spreads few requests over the four groups of warp_chains.
MT_DEV uint32_t lane_slot(uint32_t lane) { return (lane & 7u) * 4u + (lane >> 3); }

// Finds.  1M finds (half of them misses) on 1M keys of 1-8 slices: 235 us, from
// 357 us with eight lanes per request (55 warp instructions per find instead
// of 587).  What bounds it now: a lane's 32-byte loads touch 32 lines per
// instruction, so the load path moves one sector per cycle (62% busy); the
// occupancy (4, 6 or 8 blocks per SM) changes nothing.
template <bool CONC>
MT_DEV void lane_find(const tree_view& tv, const batch_args& a) {
  const uint32_t slot = lane_slot(lane_id());
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32u;
  const uint32_t warps = (gridDim.x * blockDim.x) / 32u;
  const pool_view& p = tv.pool;
  const uint32_t nf = a.n_dev ? *a.n_dev : a.n;
  const uint32_t nb = a.n_back_dev ? *a.n_back_dev : 0u;
  const uint32_t n = nf + nb;
  const uint32_t per = max(1u, min(32u, (n + warps - 1u) / warps));
  uint32_t* values = a.values_out ? a.values_out : a.values;
  for (uint32_t base = warp * per; base < n; base += warps * per) {
    if (__any_sync(0xFFFFFFFFu, slot == 0u && fatal_error(p))) break;
    const uint32_t pos = base + slot;
    const bool valid = slot < per && pos < n;
    uint32_t i = pos, klen = 0;
    if (valid) {
      if (a.index) i = a.index[pos < nf ? pos : a.region - nb + (pos - nf)];
      klen = a.key_lengths ? a.key_lengths[i] : a.max_key_length;
    }
    const bool bad = valid && klen > a.max_key_length;
    if (bad) record_error(p, ERR_INVALID_ARG);
    const uint32_t* key = a.keys + (size_t)i * a.max_key_length;
    uint32_t* out = values ? values + (size_t)i * a.max_value_length : nullptr;
    lane_place at;
    at.found = false;
    at.layer = 0;
    if (valid && !bad && klen > 0u && !lane_locate<CONC>(tv, key, klen, at)) at.found = false;
    uint32_t vlen = 0;
    bool chain = at.found && at.state != KS_VALUE;
    if (chain && !p.valid(at.val)) {
      record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
      chain = false;
    }
    if (at.found && at.state == KS_VALUE) {
      if (out != nullptr && a.max_value_length > 0u) out[0] = at.val;
      vlen = 1u;
    }
    const uint32_t lk = (chain && at.state == KS_SUFFIX) ? klen - at.layer - 1u : 0u;
    bool eq = false;
    uint32_t cv = 0;
    warp_chains<true>(p, chain, at.val, key + at.layer + 1u, lk, out, a.max_value_length, eq, cv);
    if (chain && eq) vlen = cv;
    if (valid && a.value_lengths_out) a.value_lengths_out[i] = vlen;
  }
}

// ---- writes ------------------------------------------------------------------------

MT_DEV void fence_release() { asm volatile("fence.release.gpu;" ::: "memory"); }
MT_DEV uint32_t atom_or_relaxed(uint32_t* p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.relaxed.gpu.global.or.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
MT_DEV void red_and_relaxed(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.and.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
MT_DEV void lane_store_weak(uint32_t* a, const uint32_t (&w)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    asm volatile("st.global.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(a + 8 * q), "r"(w[8 * q]),
                 "r"(w[8 * q + 1]), "r"(w[8 * q + 2]), "r"(w[8 * q + 3]), "r"(w[8 * q + 4]), "r"(w[8 * q + 5]),
                 "r"(w[8 * q + 6]), "r"(w[8 * q + 7])
                 : "memory");
}

// Attempts of a lane on its border node (each one a read and perhaps an
// atomic) before the request goes to the tile kernel that follows, which
// waits for locks, splits roots and full parents, and makes new layers.
constexpr uint32_t kLaneTries = 24;

// Slabs that a warp took together; one lane's are the positions
// [first, first + its need).
struct lane_slabs {
  uint32_t shard;
  uint32_t lo;       // free-stack position of position 0
  uint32_t n_stack;  // positions below come from the free stack,
  uint32_t bump;     // the others from the shard's slabs bump, bump + 1, ...
  uint32_t first;
};
MT_DEV uint32_t lane_slab(const pool_view& p, const lane_slabs& s, uint32_t q) {
  const uint32_t k = s.first + q;
  if (k < s.n_stack) return ld_relaxed_u32(p.free_stack + (size_t)s.shard * p.shard_slabs + s.lo + k);
  return s.shard * p.shard_slabs + s.bump + (k - s.n_stack);
}

// Take `need` slabs for every lane of the warp (0: none): one atomic or two
// for the whole warp per shard asked.  A shard that cannot serve everyone
// serves the first lanes; the next shards serve the others.  Returns whether
// the lane got its slabs (no error is recorded: the caller hands the request
// on).
MT_DEV bool warp_take_slabs(const pool_view& p, uint32_t need, uint32_t& shard, lane_slabs& s) {
  const uint32_t lane = lane_id();
  bool got = need == 0u;
  for (uint32_t k = 0; k < p.num_shards; ++k) {
    const uint32_t want = got ? 0u : need;
    uint32_t incl = want;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= (uint32_t)d) incl += up;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (total == 0u) break;
    int lo = 0, n_stack = 0, bump = 0, n_bump = 0;
    if (lane == 0u) {
      int left = (int)total;
      int* topp = p.top(shard);
      if ((int)ld_relaxed_u32((const uint32_t*)topp) > 0) {
        const int old = atomicSub(topp, left);
        if (old > 0) {
          lo = max(old - left, 0);
          n_stack = old - lo;
          left -= n_stack;
        }
      }
      int* bp = p.bump(shard);
      if (left > 0 && (int)ld_relaxed_u32((const uint32_t*)bp) < (int)p.shard_slabs) {
        const int b = atomicAdd(bp, left);
        if (b < (int)p.shard_slabs) {
          bump = b;
          n_bump = min(left, (int)p.shard_slabs - b);
        }
      }
    }
    lo = __shfl_sync(0xFFFFFFFFu, lo, 0);
    n_stack = __shfl_sync(0xFFFFFFFFu, n_stack, 0);
    bump = __shfl_sync(0xFFFFFFFFu, bump, 0);
    n_bump = __shfl_sync(0xFFFFFFFFu, n_bump, 0);
    const uint32_t have = (uint32_t)(n_stack + n_bump);
    if (want != 0u) {
      lane_slabs g;
      g.shard = shard;
      g.lo = (uint32_t)lo;
      g.n_stack = (uint32_t)n_stack;
      g.bump = (uint32_t)bump;
      g.first = incl - want;
      if (incl <= have) {
        s = g;
        got = true;
      } else {
        // The part of a lane's need that this shard covered goes back.
        for (uint32_t q = g.first; q < have; ++q) retire_slab(p, lane_slab(p, g, q - g.first));
      }
    }
    if (__all_sync(0xFFFFFFFFu, got)) break;
    shard = (shard + 1u) % p.num_shards;
  }
  return got;
}

// Write the chain of every lane with `want` into its slabs: key rest K[0..lk),
// value V[0..vlen), both from the request's rows.  Eight lanes per request, as
// in warp_chains; whole 32-byte sectors are stored.
MT_DEV void warp_write_chains(const pool_view& p, bool want, const lane_slabs& s, const uint32_t* K, uint32_t lk,
                              const uint32_t* V, uint32_t vlen, uint32_t& head) {
  constexpr int kRound = 4;
  const uint32_t lane = lane_id();
  const uint32_t r8 = lane & 7u, first = lane & 24u;
  const uint32_t todo = __ballot_sync(0xFFFFFFFFu, want);
  if (todo == 0u) return;
  const uint32_t total = want ? lk + vlen : 0u;
  uint32_t next = kInvalid;
  if (want) {
    head = lane_slab(p, s, 0u);
    if (total > kSufData) next = lane_slab(p, s, 1u);
  }
  const uint32_t columns = todo | (todo >> 8) | (todo >> 16) | (todo >> 24);
  for (int base = 0; base < 8; base += kRound) {
    if (!((columns >> base) & ((1u << kRound) - 1u))) continue;
    uint32_t c[kRound][4];
#pragma unroll
    for (int i = 0; i < kRound; ++i) {
      const uint32_t src = first + base + i;
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
      const uint32_t all = __shfl_sync(0xFFFFFFFFu, total, src);
      const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
      const uint32_t* v = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(V), src));
      const bool act = (todo >> src) & 1u;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;
        c[i][q] = 0u;
        if (act && g < kSufData && g < all) c[i][q] = g < n ? k[g] : v[g - n];
      }
    }
#pragma unroll
    for (int i = 0; i < kRound; ++i) {
      const uint32_t src = first + base + i;
      const bool act = (todo >> src) & 1u;
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
      const uint32_t all = __shfl_sync(0xFFFFFFFFu, total, src);
      const uint32_t hd = __shfl_sync(0xFFFFFFFFu, head, src);
      const uint32_t nx = __shfl_sync(0xFFFFFFFFu, next, src);
      if (r8 == SUF_WORD_HDR % 8) c[i][3] = n | ((all - n) << 16);
      if (r8 == SUF_WORD_NEXT % 8) c[i][3] = nx;
      uint32_t* a = p.addr(act ? hd : 0u) + r8;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (act) a[8 * q] = c[i][q];
      if (!__any_sync(0xFFFFFFFFu, act && all > kSufData)) continue;
      // Further slabs.
      const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
      const uint32_t* v = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(V), src));
      lane_slabs o;
      o.shard = __shfl_sync(0xFFFFFFFFu, s.shard, src);
      o.lo = __shfl_sync(0xFFFFFFFFu, s.lo, src);
      o.n_stack = __shfl_sync(0xFFFFFFFFu, s.n_stack, src);
      o.bump = __shfl_sync(0xFFFFFFFFu, s.bump, src);
      o.first = __shfl_sync(0xFFFFFFFFu, s.first, src);
      uint32_t cur = nx;
      for (uint32_t at = kSufData, sl = 2u; act && at < all; at += kSufData, ++sl) {
        const uint32_t after = at + kSufData < all ? lane_slab(p, o, sl) : kInvalid;
        uint32_t* b = p.addr(cur) + r8;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t g = r8 + 8u * q, di = at + g;
          uint32_t x = 0u;
          if (g < kSufData && di < all) x = di < n ? k[di] : v[di - n];
          if (g == (uint32_t)SUF_WORD_NEXT) x = after;
          b[8 * q] = x;
        }
        cur = after;
      }
      __syncwarp();
    }
  }
}

// Retire a chain (one lane; as suffix_retire).
MT_DEV void lane_retire_chain(const pool_view& p, uint32_t head) {
  if (!p.valid(head)) return;
  const uint32_t hdr = ld_relaxed_u32(p.addr(head) + SUF_WORD_HDR);
  const uint32_t nn = suf_nodes(hdr & kMaxLen16, hdr >> 16);
  uint32_t c = head;
  for (uint32_t q = 0; q < nn; ++q) {
    if (!p.valid(c)) break;
    const uint32_t nx = ld_relaxed_u32(p.addr(c) + SUF_WORD_NEXT);
    retire_slab(p, c);
    c = nx;
  }
  if (c != kInvalid) record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
}

// x = v where c holds, as a select: a conditional store would make the compiler
// index the image (and move it to local memory).
MT_DEV void lane_set_if(bool c, uint32_t& x, uint32_t v) {
  const uint32_t old = x;
  x = c ? v : old;
}

// Entry edits of an image in one lane's registers (header words w[30], w[31]
// included; the count goes with them).
MT_DEV void lane_insert_entry(uint32_t (&w)[32], uint32_t pos, uint32_t key, uint32_t val, uint32_t state) {
#pragma unroll
  for (int e = kMaxEntries - 1; e >= 0; --e) {
    if (e > 0 && (uint32_t)e > pos) {
      w[2 * e] = w[2 * (e > 0 ? e - 1 : 0)];
      w[2 * e + 1] = w[2 * (e > 0 ? e - 1 : 0) + 1];
    } else if ((uint32_t)e == pos) {
      w[2 * e] = key;
      w[2 * e + 1] = val;
    }
  }
  const uint32_t low = (1u << (2u * pos)) - 1u;
  const uint32_t ks = w[WORD_KS];
  w[WORD_KS] = ((ks & low) | ((ks & ~low) << 2) | (state << (2u * pos))) & 0x0FFFFFFFu;
  w[WORD_META] += 1u;
}
MT_DEV void lane_remove_entry(uint32_t (&w)[32], uint32_t pos) {
#pragma unroll
  for (int e = 0; e < kMaxEntries; ++e)
    if ((uint32_t)e >= pos) {
      w[2 * e] = e + 1 < kMaxEntries ? w[2 * (e + 1 < kMaxEntries ? e + 1 : e)] : 0u;
      w[2 * e + 1] = e + 1 < kMaxEntries ? w[2 * (e + 1 < kMaxEntries ? e + 1 : e) + 1] : 0u;
    }
  const uint32_t low = (1u << (2u * pos)) - 1u;
  const uint32_t ks = w[WORD_KS];
  w[WORD_KS] = (ks & low) | ((ks >> 2) & ~low);
  w[WORD_META] -= 1u;
}
// Publish the edited image of a locked node; the stored meta keeps LOCK set.
MT_DEV void lane_publish_locked(const pool_view& p, uint32_t idx, uint32_t (&w)[32]) {
  w[WORD_META] = (w[WORD_META] | META_LOCK) + META_VERSION_ONE;
  w[WORD_CSUM] = lane_checksum(w);
  lane_store_weak(p.addr(idx), w);
}

// Write the upper half of the full border node w (entries sp.., sp 6 or 7) to
// slab R as a new node, with the new entry at position pos of the old order
// (pos >= sp) when it belongs there.
MT_DEV void lane_store_right_half(const pool_view& p, uint32_t R, const uint32_t (&w)[32], uint32_t sp, bool with_new,
                                  uint32_t pos, uint32_t key, uint32_t val, uint32_t state) {
  uint32_t r[32];
  const uint32_t cnt = (uint32_t)kMaxEntries - sp;
  const bool seven = sp == 7u;
  // Entries 0..6 of the half (at most 7), then the new one shifted in.
#pragma unroll
  for (int k = 14; k < 28; ++k) r[k] = 0u;
#pragma unroll
  for (int e = 0; e < 7; ++e) {
    // (By value: a conditional over array elements would index the array.)
    const uint32_t k6 = w[2 * (e + 6)], v6 = w[2 * (e + 6) + 1];
    const uint32_t k7 = e + 7 < kMaxEntries ? w[2 * (e + 7 < kMaxEntries ? e + 7 : 0)] : 0u;
    const uint32_t v7 = e + 7 < kMaxEntries ? w[2 * (e + 7 < kMaxEntries ? e + 7 : 0) + 1] : 0u;
    r[2 * e] = seven ? k7 : k6;
    r[2 * e + 1] = seven ? v7 : v6;
  }
  r[WORD_HIGH] = w[WORD_HIGH];
  r[WORD_SIB] = w[WORD_SIB];
  r[WORD_META] = META_BORDER | (w[WORD_META] & META_SIB) | cnt;
  r[WORD_KS] = w[WORD_KS] >> (2u * sp);
  if (with_new) lane_insert_entry(r, pos - sp, key, val, state);
  r[WORD_CSUM] = lane_checksum(r);
  lane_store_weak(p.addr(R), r);
}

// What a lane has to do at its border node.
enum lane_job : uint32_t { JOB_NONE = 0, JOB_ADD = 1, JOB_SET = 2, JOB_DEL = 3 };

struct defer_list {
  uint32_t* list;   // requests handed to the tile kernel
  uint32_t* count;
};

// Serve the requests [a.first, a.first + a.n) (through a.index where given),
// one per lane and round:
//   1. the lane walks to its border node without locks (lane_locate);
//   2. eight lanes per request compare suffix chains, copy found values, and
//      write the chains of inserts and updates (their slabs are taken with one
//      atomic for the warp); one fence covers all of them;
//   3. lanes that change a node read its image again, decide, and set its LOCK
//      bit with one atomic: the old word it returns equals the image's (the
//      version moves with every publication) exactly if the image is current, so
//      nothing is read under the lock.  Then they publish the new image, and
//      after one fence for the whole warp release their locks.  A lane holds
//      its locks only inside one round of this loop and never waits for one, so
//      lanes cannot block each other.
//   4. A full border node below a parent with room is split in the same way.
// What does not fit (roots and parents to be split, entries that become new
// layers, nodes that stay locked) goes to the defer list.
// A pair of 1M mixed batches on 16M keys: 2.72 ms, from 4.94 ms with one
// kernel per class and 32 lanes per write (1,505 warp instructions and two
// fences per insert; now about 500, and the fences serve 32 requests); insert +
// update + find + erase of 300K keys each on 4M keys 1.58 -> 0.65 ms.
template <int OP>
MT_DEV void lane_serve(const tree_view& tv, const batch_args& a, const defer_list& dl) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  constexpr bool kFinds = OP == OP_MIXED, kInserts = OP == OP_MIXED || OP == OP_INSERT || OP == OP_UPSERT;
  constexpr bool kErases = OP == OP_MIXED || OP == OP_ERASE, kUpdates = OP == OP_MIXED || OP == OP_UPDATE;
  constexpr bool kChains = kInserts || kUpdates;
  const uint32_t slot = lane_slot(lane_id());
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32u;
  const uint32_t warps = (gridDim.x * blockDim.x) / 32u;
  const pool_view& p = tv.pool;
  const uint32_t per = max(1u, min(32u, (a.n + warps - 1u) / warps));
  uint32_t shard = (warp * 0x9E3779B1u) % p.num_shards;
  for (uint32_t base = warp * per; base < a.n; base += warps * per) {
    if (__any_sync(kAll, slot == 0u && fatal_error(p))) break;
    const uint32_t pos = base + slot;
    const bool valid = slot < per && pos < a.n;
    uint32_t i = 0, kind = 0, klen = 0, vlen = 0;
    if (valid) {
      i = a.index ? a.index[a.first + pos] : a.first + pos;
      kind = OP == OP_MIXED ? (uint32_t)a.types[i]
                            : (uint32_t)(kInserts ? MT_REQ_INSERT : (kUpdates ? MT_REQ_UPDATE : MT_REQ_ERASE));
      klen = a.key_lengths ? a.key_lengths[i] : a.max_key_length;
      if (kChains && (kind == MT_REQ_INSERT || kind == MT_REQ_UPDATE))
        vlen = a.value_lengths_in ? a.value_lengths_in[i] : a.max_value_length;
    }
    const bool bad = valid && (klen > a.max_key_length || vlen > a.max_value_length || kind > MT_REQ_UPDATE);
    if (bad) record_error(p, ERR_INVALID_ARG);
    bool combined = false;
    if (kUpdates && valid && a.leader_of != nullptr) combined = a.leader_of[i] != kInvalid;
    const bool act = valid && !bad && !combined;
    const uint32_t* key = a.keys + (size_t)i * a.max_key_length;
    uint32_t* val = a.values + (size_t)i * a.max_value_length;
    const bool find = kFinds && act && kind == MT_REQ_FIND;
    const bool insert = kInserts && act && kind == MT_REQ_INSERT;
    const bool update = kUpdates && act && kind == MT_REQ_UPDATE;
    const bool erase = kErases && act && kind == MT_REQ_ERASE;
    if (kChains && (insert || update)) asm volatile("prefetch.global.L2 [%0];" ::"l"(val));
    bool defer = (insert || update) && (klen == 0u || klen > kMaxLen16 || vlen > kMaxLen16);
    bool go = act && !defer && klen > 0u;

    // 1. To the border node.
    lane_place at;
    at.found = false;
    at.layer = 0;
    at.idx = at.parent = at.root = 0;
    if (go && !lane_locate<true>(tv, key, klen, at)) go = false;
    bool chain = go && at.found && (at.state == KS_SUFFIX || (find && at.state == KS_LONGVAL));
    if (chain && !p.valid(at.val)) {
      record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
      chain = go = false;
    }

    // 2. Chains: compare and copy, then write.
    const bool more = at.layer + 1u < klen;
    const uint32_t rest = more ? klen - at.layer - 1u : 0u;
    bool eq = false;
    uint32_t cv = 0, res = 0, found_len = 0;
    warp_chains<kFinds>(p, chain, at.val, key + at.layer + 1u, rest, find ? val : nullptr, a.max_value_length, eq, cv);
    const bool present = go && at.found && (at.state != KS_SUFFIX || eq);
    if (find && present) {
      if (at.state == KS_VALUE) {
        val[0] = at.val;
        found_len = 1u;
      } else {
        found_len = cv;
      }
    }
    uint32_t job = JOB_NONE;
    if (erase && present) job = JOB_DEL;
    if (update && present) job = JOB_SET;
    if (insert && go) {
      if (present) {
        if (OP == OP_UPSERT) job = JOB_SET;
      } else if (at.found) {
        defer = true;  // a chain of another key: both move to a new layer
      } else {
        job = JOB_ADD;
      }
    }
    uint32_t nv = kInvalid, ns = KS_VALUE;
    if (kChains) {
      uint32_t need = 0;
      if (job == JOB_ADD || job == JOB_SET) {
        ns = more ? KS_SUFFIX : (vlen == 1u ? KS_VALUE : KS_LONGVAL);
        if (ns == KS_VALUE) nv = val[0];
        else need = suf_nodes(rest, vlen);
      }
      lane_slabs sl{};
      if (!warp_take_slabs(p, need, shard, sl)) {
        job = JOB_NONE;
        defer = true;
        need = 0;
      }
      warp_write_chains(p, need != 0u, sl, key + at.layer + 1u, rest, val, vlen, nv);
      __syncwarp();
      fence_release();
    }

    // 3. The border node.
    const uint32_t slice = klen > 0u && act ? key[at.layer] : 0u;
    uint32_t idx = at.idx, tries = 0, spare = kInvalid, old_chain = kInvalid;
    bool want_spare = false;
    while (__any_sync(kAll, job != JOB_NONE)) {
      if (kInserts && __any_sync(kAll, want_spare && spare == kInvalid)) {
        lane_slabs sl{};
        const uint32_t need = want_spare && spare == kInvalid ? 1u : 0u;
        if (warp_take_slabs(p, need, shard, sl)) {
          if (need) spare = lane_slab(p, sl, 0u);
        } else {
          job = JOB_NONE;
          defer = true;
          want_spare = false;
        }
      }
      uint32_t w[32];
      bool won = false, split = false;
      uint32_t pslot = 0, e = 0, st = 0, sp = 0;
      if (job != JOB_NONE) {
        uint32_t pmeta = 0;
        bool parent_ok = true;
        if (++tries > kLaneTries) {
          job = JOB_NONE;
          defer = true;
        }
        if (kInserts && job != JOB_NONE && want_spare) {
          // The node was full: its parent must list it and have room.
          parent_ok = lane_read_fresh(p, at.parent, w);
          pmeta = w[WORD_META];
          uint32_t hits = 0;
#pragma unroll
          for (int k = 0; k < kMaxEntries; ++k)
            if ((uint32_t)k < (pmeta & META_COUNT) && w[2 * k + 1] == idx) hits |= 1u << k;
          parent_ok = parent_ok && hits != 0u && !(pmeta & META_BORDER) && (pmeta & META_COUNT) < (uint32_t)kMaxEntries;
          pslot = hits ? (uint32_t)__ffs(hits) - 1u : 0u;
        }
        if (job != JOB_NONE && !lane_read_fresh(p, idx, w)) job = JOB_NONE;  // error recorded
        const uint32_t meta = w[WORD_META];
        if (job == JOB_NONE) {
        } else if ((meta & META_SIB) && slice > w[WORD_HIGH]) {
          idx = w[WORD_SIB];
          if (!p.valid(idx)) {
            record_error(p, ERR_CORRUPT, MT_AT(SRC_LANE));
            job = JOB_NONE;
          }
        } else if (!(meta & META_BORDER)) {
          job = JOB_NONE;  // a layer root that was split meanwhile
          defer = true;
        } else if (!(meta & META_LOCK)) {
          const uint32_t ks = w[WORD_KS];
          const uint32_t okm = lane_eligible(meta, ks, more);
          uint32_t hit = 0, v = 0, before = 0;
#pragma unroll
          for (int k = 0; k < kMaxEntries; ++k) {
            if ((uint32_t)k < (meta & META_COUNT) &&
                (w[2 * k] < slice || (more && w[2 * k] == slice && !(ks & (1u << (2 * k))))))
              ++before;
            if (w[2 * k] == slice && (okm & (1u << (2 * k)))) {
              hit = 1u << (2 * k);
              v = w[2 * k + 1];
            }
          }
          st = (more ? KS_MORE : 0u) | ((ks & (hit << 1)) ? KS_SLAB : 0u);
          e = before;  // entries before it: the entry's own position if there is one
          bool lock = false;
          if (job == JOB_ADD) {
            if (hit) {
              job = JOB_NONE;  // the slice was taken meanwhile
              defer = true;
            } else if ((meta & META_COUNT) < (uint32_t)kMaxEntries) {
              lock = true;
            } else if ((meta & META_ROOT) || at.parent == kInvalid || !parent_ok) {
              job = JOB_NONE;
              defer = true;
            } else if (spare == kInvalid) {
              want_spare = true;
            } else if (!(pmeta & META_LOCK)) {
              lock = split = true;
            }
          } else if (!hit) {
            // Erased meanwhile: updates and erases miss, an upsert starts again.
            defer = insert;
            job = JOB_NONE;
          } else if ((st == KS_SUFFIX && v != at.val) || st == KS_LINK) {
            job = JOB_NONE;  // another chain: compare again
            defer = true;
          } else {
            lock = true;
          }
          if (lock) {
            uint32_t* mw = p.addr(idx) + WORD_META;
            const uint32_t old = atom_or_relaxed(mw, META_LOCK);
            won = old == meta;
            if (!won && !(old & META_LOCK)) red_and_relaxed(mw, ~META_LOCK);  // changed since the read
            if (kInserts && won && split) {
              uint32_t* pw = p.addr(at.parent) + WORD_META;
              const uint32_t pold = atom_or_relaxed(pw, META_LOCK);
              if (pold != pmeta) {
                if (!(pold & META_LOCK)) red_and_relaxed(pw, ~META_LOCK);
                red_and_relaxed(mw, ~META_LOCK);
                won = false;
              }
            }
            if (won && job != JOB_ADD && (st & KS_SLAB)) old_chain = v;
          }
        }
      }
      if (kInserts && __any_sync(kAll, won && split)) {
        if (won && split) {
          // Never part the two entries of one slice.
          sp = w[2 * (kMaxEntries / 2 - 1)] == w[2 * (kMaxEntries / 2)] ? kMaxEntries / 2 + 1 : kMaxEntries / 2;
          const uint32_t h6 = w[10], h7 = w[12];
          const uint32_t left_high = sp == 7u ? h7 : h6;
          lane_store_right_half(p, spare, w, sp, slice > left_high, e, slice, nv, ns);
        }
        __syncwarp();
        fence_release();
      }
      if (won) {
        if (kInserts && split) {
          const uint32_t h6 = w[10], h7 = w[12];
          const uint32_t left_high = sp == 7u ? h7 : h6;
#pragma unroll
          for (int k = 6; k < kMaxEntries; ++k)
            if ((uint32_t)k >= sp) w[2 * k] = w[2 * k + 1] = 0u;
          w[WORD_KS] &= (1u << (2u * sp)) - 1u;
          w[WORD_META] = (w[WORD_META] & ~META_COUNT) | META_SIB | sp;
          w[WORD_HIGH] = left_high;
          w[WORD_SIB] = spare;
          if (slice <= left_high) lane_insert_entry(w, e, slice, nv, ns);
          lane_publish_locked(p, idx, w);
          lane_load_relaxed(p.addr(at.parent), w);  // locked: as read above
          lane_insert_entry(w, pslot, left_high, idx, 0u);
#pragma unroll
          for (int k = 1; k < kMaxEntries; ++k)
            lane_set_if((uint32_t)k == pslot + 1u, w[2 * k + 1], spare);
          lane_publish_locked(p, at.parent, w);
          spare = kInvalid;
        } else {
          if (job == JOB_ADD) {
            lane_insert_entry(w, e, slice, nv, ns);
          } else if (job == JOB_SET) {
#pragma unroll
            for (int k = 0; k < kMaxEntries; ++k)
              lane_set_if((uint32_t)k == e, w[2 * k + 1], nv);
            w[WORD_KS] = (w[WORD_KS] & ~(3u << (2u * e))) | (ns << (2u * e));
          } else {
            lane_remove_entry(w, e);
          }
          lane_publish_locked(p, idx, w);
        }
      }
      if (__any_sync(kAll, won)) fence_release();
      if (won) {
        red_and_relaxed(p.addr(idx) + WORD_META, ~META_LOCK);
        if (kInserts && split) red_and_relaxed(p.addr(at.parent) + WORD_META, ~META_LOCK);
        if (kErases && job == JOB_DEL) {
          const uint32_t left = w[WORD_META] & META_COUNT;
          const bool is_root = (w[WORD_META] & META_ROOT) != 0u;
          if (tv.merge_log != nullptr && !is_root && (left == kMergeAt || left == 0u)) {
            const uint32_t r = atomicAdd(tv.merge_log, 1u);
            if (r < tv.merge_cap) {
              tv.merge_log[2u + 2u * r] = at.root;
              tv.merge_log[3u + 2u * r] = slice;
            }
          }
          if (tv.layer_log != nullptr && at.layer >= 1u && at.layer < kLayerRecWords && left == 0u &&
              !(w[WORD_META] & META_SIB) && (is_root || tv.merge_log != nullptr)) {
            const uint32_t r = atomicAdd(tv.layer_log, 1u);
            if (r < tv.layer_cap) {
              uint32_t* rec = tv.layer_log + 2u + (size_t)kLayerRecWords * r;
              rec[0] = at.layer;
              for (uint32_t q = 0; q < at.layer; ++q) rec[1u + q] = key[q];
            }
          }
        }
        if (old_chain != kInvalid) lane_retire_chain(p, old_chain);
        nv = kInvalid;  // in the tree now
        res = 1u;
        job = JOB_NONE;
      }
    }
    // Slabs taken in vain.
    if (kChains && nv != kInvalid && (ns & KS_SLAB)) lane_retire_chain(p, nv);
    if (kInserts && spare != kInvalid) retire_slab(p, spare);

    // 4. Results, and the requests left to the tile kernel.
    const uint32_t dm = __ballot_sync(kAll, defer);
    if (dm) {
      uint32_t at0 = 0;
      if (lane_id() == 0u) at0 = atomicAdd(dl.count, (uint32_t)__popc(dm));
      at0 = __shfl_sync(kAll, at0, 0);
      if (defer) dl.list[at0 + __popc(dm & ((1u << lane_id()) - 1u))] = i;
    }
    if (valid && !combined && !defer) {
      if (kFinds && kind == MT_REQ_FIND) {
        if (a.value_lengths_out) a.value_lengths_out[i] = found_len;
      } else if (a.results) {
        a.results[i] = res != 0u;
      }
    }
  }
}

}  // namespace mtb
