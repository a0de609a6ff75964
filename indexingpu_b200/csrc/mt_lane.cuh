// One request per thread: the batch kernels' way through the tree.
//
// A lane walks its request's path alone: eight lanes bring the node to the
// lane's line of shared memory, the lane searches it in its registers.  So a
// warp has 32 independent walks in flight where the tile code (mt_tree.cuh) has
// 32 / T, and a node visit costs no vote or reduction.  What benefits from
// neighbouring lanes reading neighbouring words (suffix chains, key rests,
// values) is done by eight lanes per request, four requests at a time
// (warp_chains).  The few requests that need more than one node and its parent
// are served by the whole warp as one tile.
#pragma once
#include "mt_internal.cuh"

namespace mtb {

// Images of nodes.  Walks read them with plain loads, which may hit L1: with
// concurrent writers an image of an earlier moment of this launch is as good
// as any (B-link nodes are never unlinked while a launch runs, so a stale
// interior node still leads to its key through sibling links, and requests of
// one batch have no order), and the checksum rejects a torn one, which is then
// read again from L2.  A node that was split again and again since its parent
// came to L1 would be a long way from its last half: after kMaxSideways moves
// the walk starts its layer again, from L2.  The upper levels of the tree, which every request
// passes, thus come from L1 (reading them all from L2 costs a pair of 1M mixed
// batches 3.39 instead of 2.79 ms).
MT_DEV void lane_load_relaxed(const uint32_t* a, uint32_t (&w)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    asm volatile("ld.relaxed.gpu.global.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[8 * q]), "=r"(w[8 * q + 1]), "=r"(w[8 * q + 2]), "=r"(w[8 * q + 3]), "=r"(w[8 * q + 4]),
                   "=r"(w[8 * q + 5]), "=r"(w[8 * q + 6]), "=r"(w[8 * q + 7])
                 : "l"(a + 8 * q) : "memory");
}

// Out of line: errors are rare, and inlined recording would crowd the
// instruction cache.
static __device__ __noinline__ void lane_error(uint32_t* err, uint32_t code, uint32_t site) {
  pool_view p{};
  p.err = err;
  record_error(p, code, site);
}

// Node images of a warp's 32 walks in shared memory: line l holds lane l's
// node, its 16-byte part c at place c ^ (l & 7), so that eight lanes reading the
// same part of their lines meet no bank twice.
MT_DEV uint32_t* warp_lines() {
  __shared__ __align__(128) uint32_t lines[kBlock / 32][32 * 32];
  return lines[threadIdx.x / 32u];
}
MT_DEV void copy_async16(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
MT_DEV void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Bring the nodes `idx` of the lanes with `want` to their lines (called by the
// whole warp).  Eight lanes copy one node: one request per 128-byte line,
// where a lane loading its own node makes one per 32-byte part.
// The load path takes requests per line, not bytes: with a lane's own four
// 32-byte loads no occupancy from 4 to 8 blocks per SM moved the 225 us of 1M
// finds on 1M keys; staged they take 123 us, and a pair of 1M mixed batches on
// 16M keys 1.22 ms instead of 2.59.
MT_DEV void warp_load_nodes(const pool_view& p, uint32_t* lines, bool want, uint32_t idx) {
  const uint32_t lane = lane_id();
  const uint32_t m = __ballot_sync(0xFFFFFFFFu, want);
#pragma unroll
  for (uint32_t q = 0; q < 8u; ++q) {
    const uint32_t l = 4u * q + (lane >> 3), c = lane & 7u;
    const uint32_t i = __shfl_sync(0xFFFFFFFFu, idx, l);
    if ((m >> l) & 1u) copy_async16(lines + 32u * l + 4u * (c ^ (l & 7u)), p.addr(i) + 4u * c);
  }
  copy_async_wait();
  __syncwarp();
}
MT_DEV void lane_take_line(const uint32_t* lines, uint32_t (&w)[32]) {
  const uint32_t lane = lane_id();
#pragma unroll
  for (uint32_t c = 0; c < 8u; ++c) {
    const uint4 x = *reinterpret_cast<const uint4*>(lines + 32u * lane + 4u * (c ^ (lane & 7u)));
    w[4 * c] = x.x;
    w[4 * c + 1] = x.y;
    w[4 * c + 2] = x.z;
    w[4 * c + 3] = x.w;
  }
}

MT_DEV uint64_t lane_checksum(const uint32_t (&w)[32]) {
  uint64_t h = kCsumInit;
#pragma unroll
  for (int g = 0; g < 32; ++g) h += csum_term((uint32_t)g, w[g]);
  return h;
}
MT_DEV bool lane_verify(const uint32_t (&w)[32]) {
  return lane_checksum(w) == ((uint64_t)w[WORD_CSUM + 1] << 32 | w[WORD_CSUM]);
}
MT_DEV void lane_seal(uint32_t (&w)[32]) {
  const uint64_t h = lane_checksum(w);
  w[WORD_CSUM] = (uint32_t)h;
  w[WORD_CSUM + 1] = (uint32_t)(h >> 32);
}

// First entry at or after (slice, more) in an image's order: its position (the
// count if there is none), and its words.  An interior node's separators count
// as continuing keys, so the first one >= slice is found, whose child covers it.
// (Entry words past the count are 0 and never precede a found entry.)
MT_DEV uint32_t lane_search(const uint32_t (&w)[32], uint32_t slice, bool more, uint32_t& key, uint32_t& val) {
  uint32_t pos = kMaxEntries;
  key = val = 0u;
#pragma unroll
  for (int e = kMaxEntries - 1; e >= 0; --e) {
    const bool c = w[2 * e] >= slice;
    pos = c ? (uint32_t)e : pos;
    key = c ? w[2 * e] : key;
    val = c ? w[2 * e + 1] : val;
  }
  if (more && key == slice && (w[WORD_META] & META_BORDER) && pos < (w[WORD_META] & META_COUNT) &&
      !(ks_get(w[WORD_KS], pos) & KS_MORE)) {
    // The key that ends at this slice comes first: the next entry.
    ++pos;
    key = val = 0u;
#pragma unroll
    for (int e = 1; e < kMaxEntries; ++e) {
      key = (uint32_t)e == pos ? w[2 * e] : key;
      val = (uint32_t)e == pos ? w[2 * e + 1] : val;
    }
  }
  return min(pos, w[WORD_META] & META_COUNT);
}
// Whether the entry a search ended at is the one for (slice, more).
MT_DEV bool lane_is_entry(uint32_t meta, uint32_t ks, uint32_t pos, uint32_t key, uint32_t slice, bool more) {
  return pos < (meta & META_COUNT) && key == slice && ((ks_get(ks, pos) & KS_MORE) != 0u) == more;
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
  bool full;        // the border node has no room
  bool stuck;       // and is a root, or its parent has no room either: only a tile can split it
};

constexpr uint32_t kMaxSideways = 8;

// Walk from the root of layer 0 to the key's place, for the lanes with `go`
// (klen > 0); called by the whole warp.  The warp goes round the loop together,
// one node visit per lane and round: left to themselves, lanes in interior and
// border nodes drift apart and run the loop one after the other.  go is
// cleared after a (recorded) error.
template <bool CONC>
MT_DEV void lane_locate(const tree_view& tv, bool& go, const uint32_t* key, uint32_t klen, lane_place& at) {
  const pool_view& p = tv.pool;
  uint32_t idx = tv.root, hops = 0, torn = 0, sideways = 0;
  bool parent_full = true;  // (or there is none)
  bool from_l2 = false;
  uint32_t slice = go ? key[0] : 0u;
  bool more = klen > 1u;
  bool walk = go;
  at.found = false;
  at.layer = 0;
  at.parent = kInvalid;
  at.root = idx;
  uint32_t* lines = warp_lines();
#pragma unroll 1
  while (__any_sync(0xFFFFFFFFu, walk)) {
    const bool ok = p.valid(idx);
    warp_load_nodes(p, lines, walk && ok && torn == 0u && !from_l2, idx);
    if (walk) {
      uint32_t err = ERR_NONE;
      if (!ok || ++hops > kMaxHops) {
        err = ERR_CORRUPT;
      } else {
        uint32_t w[32];
        if (CONC && (torn != 0u || from_l2)) lane_load_relaxed(p.addr(idx), w);
        else lane_take_line(lines, w);
        if (CONC && !lane_verify(w)) {  // read again, from L2 (bounded, as node::load_verified)
          --hops;
          if (++torn > kTornRetries) err = ERR_CORRUPT;
        } else {
          torn = 0;
          const uint32_t meta = w[WORD_META];
          const bool border = (meta & META_BORDER) != 0u;
          uint32_t k, v;
          const uint32_t pos = lane_search(w, slice, more, k, v);
          if ((meta & META_SIB) && slice > w[WORD_HIGH]) {
            idx = w[WORD_SIB];
            if (CONC && ++sideways > kMaxSideways && !from_l2) {
              from_l2 = true;
              idx = at.root;
              at.parent = kInvalid;
              parent_full = true;
            }
          } else if (!border) {
            at.parent = idx;
            parent_full = (meta & META_COUNT) >= (uint32_t)kMaxEntries;
            idx = pos < (meta & META_COUNT) ? v : kInvalid;  // none: caught as an invalid slab above
          } else {
            const uint32_t state = ks_get(w[WORD_KS], pos);
            const bool hit = lane_is_entry(meta, w[WORD_KS], pos, k, slice, more);
            if (hit && state == KS_LINK) {
              idx = v;
              at.root = v;
              at.parent = kInvalid;
              parent_full = true;
              ++at.layer;
              slice = key[at.layer];
              more = at.layer + 1u < klen;
            } else {
              at.idx = idx;
              at.full = (meta & META_COUNT) >= (uint32_t)kMaxEntries;
              at.stuck = at.full && ((meta & META_ROOT) || parent_full);
              at.found = hit;
              at.state = state;
              at.val = v;
              walk = false;
            }
          }
        }
      }
      if (err != ERR_NONE) {
        lane_error(p.err, err, MT_AT(SRC_LANE));
        walk = go = false;
      }
    }
    __syncwarp();
  }
}

// For every lane with `want`: compare its key rest K[0..lk) with that of the
// chain at `head` (lk 0 for a chain that holds a value only) and, where equal
// and out is not null, copy at most maxV value slices.  Eight lanes serve one
// request, lane r of them the words r, r+8, r+16 and r+24 of a slab: every load
// and store covers whole 32-byte sectors of four requests' lines.  Only the
// sectors that the key rest and maxV value slices can reach are read, and two
// requests' loads (per eight lanes) are in flight together.  Called by the
// whole warp; eq and vlen are set for the lanes with want.  (Every vote and
// shuffle stands alone: none may be skipped by a lane's && or ?:.)
template <bool VALUES>
MT_DEV void warp_chains(const pool_view& p, bool want, uint32_t head, const uint32_t* K, uint32_t lk, uint32_t* out,
                        uint32_t maxV, bool& eq, uint32_t& vlen) {
  constexpr int kRound = MT_CHAIN_ROUND;
  const uint32_t lane = lane_id();
  const uint32_t r8 = lane & 7u, first = lane & 24u;
  const uint32_t todo = __ballot_sync(0xFFFFFFFFu, want);
  if (todo == 0u) return;
  const uint32_t columns = todo | (todo >> 8) | (todo >> 16) | (todo >> 24);  // bit i: lane i of some eight lanes
#pragma unroll 1
  for (int base = 0; base < 8; base += kRound) {
    if (!((columns >> base) & ((1u << kRound) - 1u))) continue;
    uint32_t c[kRound][4], kw[kRound][4];
#pragma unroll
    for (int i = 0; i < kRound; ++i) {
      const uint32_t src = first + base + i;
      const uint32_t hd = __shfl_sync(0xFFFFFFFFu, head, src);
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
      const uint32_t need = n + (VALUES ? maxV : 0u);
      const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
      const bool act = (todo >> src) & 1u;
      const uint32_t* a = p.addr(act ? hd : 0u) + r8;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;
        c[i][q] = 0u;
        if (act && (g < need || g >= kSufData)) c[i][q] = a[8 * q];
        kw[i][q] = (act && g < n && g < kSufData) ? k[g] : 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < kRound; ++i) {
      const uint32_t src = first + base + i;
      const bool act = (todo >> src) & 1u;
      const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
      const uint32_t hdr = __shfl_sync(0xFFFFFFFFu, c[i][3], first + SUF_WORD_HDR % 8);
      bool differs = act && (hdr & kMaxLen16) != n;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;
        differs |= act && g < kSufData && g < n && c[i][q] != kw[i][q];
      }
      const uint32_t other = __ballot_sync(0xFFFFFFFFu, differs);
      const bool same = !((other >> first) & 0xFFu);
      if (VALUES) {
        uint32_t* o = reinterpret_cast<uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(out), src));
        const uint32_t last = n + min(hdr >> 16, maxV);  // data slices [0, n) are compared, [n, last) copied
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t g = r8 + 8u * q;
          if (act && same && o != nullptr && g < kSufData && g >= n && g < last) o[g - n] = c[i][q];
        }
      }
      if (r8 == (uint32_t)(base + i)) {
        eq = same;
        vlen = hdr >> 16;
      }
    }
  }
  // Chains of several slabs: the slabs after the head, one request per eight
  // lanes at a time.
  uint32_t last = want && eq ? lk + (VALUES && out != nullptr ? min(vlen, maxV) : 0u) : 0u;
  const uint32_t longer = __ballot_sync(0xFFFFFFFFu, last > kSufData);
  if (longer == 0u) return;
#pragma unroll 1
  for (uint32_t i = 0; i < 8u; ++i) {
    const uint32_t src = first + i;
    const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
    const uint32_t hd = __shfl_sync(0xFFFFFFFFu, head, src);
    const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
    uint32_t* o = reinterpret_cast<uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(out), src));
    const uint32_t end = __shfl_sync(0xFFFFFFFFu, last, src);
    bool same = end > kSufData;
    uint32_t nx = same ? p.addr(hd)[SUF_WORD_NEXT] : kInvalid;
#pragma unroll 1
    for (uint32_t at = kSufData; __any_sync(0xFFFFFFFFu, same && at < end); at += kSufData) {
      const bool on = same && at < end && p.valid(nx);
      if (same && !on && at < n) same = false;  // a chain cut short cannot hold the key
      uint32_t d[4];
      bool differs = false;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;
        d[q] = on ? p.addr(nx)[g] : 0u;
        if (on && g < kSufData && at + g < n) differs |= d[q] != k[at + g];
      }
      const uint32_t rest = __ballot_sync(0xFFFFFFFFu, differs);
      if ((rest >> first) & 0xFFu) same = false;
      if (VALUES) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t g = r8 + 8u * q;
          if (on && same && g < kSufData && at + g >= n && at + g < end) o[at + g - n] = d[q];
        }
      }
      nx = __shfl_sync(0xFFFFFFFFu, d[3], first + SUF_WORD_NEXT % 8);
      if (!on) nx = kInvalid;
    }
    if (r8 == i && last > kSufData) eq = same;
  }
}

// Requests per warp and round: 32 on large batches; fewer on small ones, so
// that every warp of the launch gets work and the batch ends after one walk's
// latency.  Slot j of a round is served by lane (j % 4) * 8 + j / 4, which
// spreads few requests over the four groups of warp_chains.
MT_DEV uint32_t lane_slot(uint32_t lane) { return (lane & 7u) * 4u + (lane >> 3); }

// ---- requests --------------------------------------------------------------------

// One request as a lane serves it.  `val`: the value rows of inserts and
// updates (input) and finds (output; may be null).
struct lane_request {
  uint32_t id;
  uint32_t kind, klen, vlen;
  const uint32_t* key;
  uint32_t* val;
  uint32_t* out_len;  // for sources that do not derive their result addresses from id
  bool* out_ok;
};
enum lane_fetch : uint32_t { LANE_SKIP = 0, LANE_SERVE = 1, LANE_REFUSED = 2 };  // refused: recorded, reported as failed

// Where a kernel's requests come from and its results go to.  fetch is called
// by single lanes; lane_serve calls found for finds and result for the others.
struct batch_source {
  batch_args a;
  MT_DEV uint32_t size() const { return a.n_dev ? *a.n_dev : a.n; }
  MT_DEV uint32_t max_value_length() const { return a.max_value_length; }
  template <int OP>
  MT_DEV uint32_t fetch(const pool_view& p, uint32_t pos, lane_request& r) const {
    const uint32_t i = a.index ? a.index[pos] : pos;
    r.id = i;
    r.kind = MT_REQ_FIND;
    if (OP == OP_MIXED) r.kind = a.types[i];
    else if (OP == OP_INSERT || OP == OP_UPSERT) r.kind = MT_REQ_INSERT;
    else if (OP == OP_UPDATE) r.kind = MT_REQ_UPDATE;
    else if (OP == OP_ERASE) r.kind = MT_REQ_ERASE;
    r.klen = a.key_lengths ? a.key_lengths[i] : a.max_key_length;
    r.vlen = 0;
    if (r.kind == MT_REQ_INSERT || r.kind == MT_REQ_UPDATE)
      r.vlen = a.value_lengths_in ? a.value_lengths_in[i] : a.max_value_length;
    r.key = a.keys + (size_t)i * a.max_key_length;
    r.val = a.values ? a.values + (size_t)i * a.max_value_length : nullptr;
    // Lengths beyond the row stride (or unknown kinds) would read outside the
    // caller's buffers: such requests are skipped and reported.
    if (r.klen > a.max_key_length || r.vlen > a.max_value_length || r.kind > MT_REQ_UPDATE) {
      lane_error(p.err, ERR_INVALID_ARG, MT_AT(SRC_LANE));
      return LANE_REFUSED;
    }
    if ((OP == OP_MIXED || OP == OP_UPDATE) && a.leader_of != nullptr && a.leader_of[i] != kInvalid) return LANE_SKIP;
    return LANE_SERVE;
  }
  MT_DEV void found(uint32_t, const lane_request& r, bool, uint32_t len) const {
    if (a.value_lengths_out) a.value_lengths_out[r.id] = len;
  }
  MT_DEV void result(uint32_t, const lane_request& r, bool ok) const {
    if (a.results) a.results[r.id] = ok;
  }
};

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
// atomic) before the whole warp serves the request as a tile, which waits for
// locks, splits roots and full parents, and makes new layers.
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

// Keep a chain of n slabs that nothing leads to in the warp's slab cache, or
// (TAIL) give it back for the kernel that follows (one lane).
template <bool TAIL>
MT_DEV void lane_keep_slabs(const pool_view& p, uint32_t head, uint32_t n, slab_cache<32>& cache) {
  if (TAIL) {
#pragma unroll 1
    for (uint32_t q = 0; q < n; ++q) {
      const uint32_t next = q + 1u < n ? ld_relaxed_u32(p.addr(head) + kNextWord) : kInvalid;
      return_unused(p, head);
      head = next;
    }
    return;
  }
  uint32_t tail = head;
#pragma unroll 1
  for (uint32_t q = 1; q < n; ++q) tail = ld_relaxed_u32(p.addr(tail) + kNextWord);
  st_relaxed_u32(p.addr(tail) + kNextWord, cache.vain);
  cache.vain = head;
  cache.vain_n += n;
}

// Take `need` slabs for every lane of the warp (0: none): one atomic or two
// for the whole warp per shard asked.  A shard that cannot serve everyone
// serves the first lanes; the next shards serve the others.  Returns whether
// the lane got its slabs (no error is recorded: a tile, which takes one slab
// after the other from any shard, serves the request then).
template <bool TAIL>
MT_DEV bool warp_take_slabs(const pool_view& p, uint32_t need, slab_cache<32>& cache, lane_slabs& s) {
  const uint32_t lane = lane_id();
  uint32_t& shard = cache.shard;
  bool got = need == 0u;
#pragma unroll 1
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
    // A shard that cannot cover the first lane's need is left as it is.
    const uint32_t least = __shfl_sync(0xFFFFFFFFu, want, __ffs(__ballot_sync(0xFFFFFFFFu, want != 0u)) - 1);
    int lo = 0, n_stack = 0, bump = 0, n_bump = 0;
    if (lane == 0u) {
      int* topp = p.top(shard);
      int* bp = p.bump(shard);
      const int on_stack = max((int)ld_relaxed_u32((const uint32_t*)topp), 0);
      const int above = max((int)p.shard_slabs - (int)ld_relaxed_u32((const uint32_t*)bp), 0);
      int left = (uint32_t)(on_stack + above) >= least ? (int)total : 0;
      if (left > 0 && on_stack > 0) {
        const int old = atomicSub(topp, left);
        if (old > 0) {
          lo = max(old - left, 0);
          n_stack = old - lo;
          left -= n_stack;
        }
      }
      if (left > 0 && above > 0) {
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
        // The part of a lane's need that this shard covered is kept, or given back.
#pragma unroll 1
        for (uint32_t q = g.first; q < have; ++q) {
          const uint32_t x = lane_slab(p, g, q - g.first);
          lane_keep_slabs<TAIL>(p, x, 1u, cache);
        }
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
  constexpr int kRound = MT_CHAIN_ROUND;
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
#pragma unroll 1
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
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q;  // all: 0 for a request without a chain
        c[i][q] = 0u;
        if (g < kSufData && g < all) c[i][q] = *(g < n ? k + g : v + (g - n));
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
    }
  }
  // Further slabs: slab after slab of all chains, four at a time (eight lanes
  // each), so that one long chain is written by the whole warp and four loads of
  // rows are under way.  (One chain per eight lanes, slab after slab, took 17 of
  // the 28 us of 1,000 inserts with keys to 150 and values to 80 slices, now 39
  // -> 28 us a call; 50,000 mixed requests of 100 and 60 slices 213 -> 191 us a pair.)
  const uint32_t more = total > kSufData ? (total - 1u) / kSufData : 0u;
  uint32_t end = more;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, end, d);
    if (lane >= (uint32_t)d) end += up;
  }
  const uint32_t all_more = __shfl_sync(0xFFFFFFFFu, end, 31);
#pragma unroll 1
  for (uint32_t base = 0; base < all_more; base += 4u) {
    const uint32_t item = base + (lane >> 3);
    // The chain it belongs to: the first lane whose end lies beyond it.
    uint32_t src = 0;
#pragma unroll
    for (uint32_t d = 16u; d != 0u; d >>= 1)
      if (__shfl_sync(0xFFFFFFFFu, end, src + d - 1u) <= item) src += d;
    const bool act = item < all_more;
    const uint32_t sl = item - __shfl_sync(0xFFFFFFFFu, end - more, src) + 1u;  // the head is slab 0
    const uint32_t n = __shfl_sync(0xFFFFFFFFu, lk, src);
    const uint32_t all = __shfl_sync(0xFFFFFFFFu, total, src);
    const uint32_t* k = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(K), src));
    const uint32_t* v = reinterpret_cast<const uint32_t*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(V), src));
    lane_slabs o;
    o.shard = __shfl_sync(0xFFFFFFFFu, s.shard, src);
    o.lo = __shfl_sync(0xFFFFFFFFu, s.lo, src);
    o.n_stack = __shfl_sync(0xFFFFFFFFu, s.n_stack, src);
    o.bump = __shfl_sync(0xFFFFFFFFu, s.bump, src);
    o.first = __shfl_sync(0xFFFFFFFFu, s.first, src);
    if (act) {
      const uint32_t at = sl * kSufData;
      uint32_t x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t g = r8 + 8u * q, di = at + g;
        x[q] = 0u;
        if (g < kSufData && di < all) x[q] = *(di < n ? k + di : v + (di - n));
      }
      const uint32_t cur = lane_slab(p, o, sl);
      const uint32_t after = at + kSufData < all ? lane_slab(p, o, sl + 1u) : kInvalid;
      if (r8 == SUF_WORD_NEXT % 8) x[3] = after;
      uint32_t* b = p.addr(cur) + r8;
#pragma unroll
      for (int q = 0; q < 4; ++q) b[8 * q] = x[q];
    }
  }
}

// Retire a chain (one lane; as suffix_retire).
MT_DEV void lane_retire_chain(const pool_view& p, uint32_t head) {
  if (!p.valid(head)) return;
  const uint32_t hdr = ld_relaxed_u32(p.addr(head) + SUF_WORD_HDR);
  const uint32_t nn = suf_nodes(hdr & kMaxLen16, hdr >> 16);
  uint32_t c = head;
#pragma unroll 1
  for (uint32_t q = 0; q < nn; ++q) {
    if (!p.valid(c)) break;
    const uint32_t nx = ld_relaxed_u32(p.addr(c) + SUF_WORD_NEXT);
    retire_slab(p, c);
    c = nx;
  }
  if (c != kInvalid) lane_error(p.err, ERR_CORRUPT, MT_AT(SRC_LANE));
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
// Where a full border node is cut: 6 or 7, never between the two entries of
// one slice.  high: the largest slice of the lower half.
MT_DEV uint32_t lane_split_pos(const uint32_t (&w)[32], uint32_t& high) {
  constexpr int h = kMaxEntries / 2;
  const uint32_t k5 = w[2 * (h - 1)], k6 = w[2 * h];
  high = k5;  // where the cut moves up, entry h has the same slice
  return k5 == k6 ? h + 1 : h;
}
// The image of the upper half (entries sp..) as a node of its own.
MT_DEV void lane_upper_half(uint32_t (&w)[32], uint32_t sp) {
  const bool up = sp == (uint32_t)kMaxEntries / 2u + 1u;
  constexpr int h = kMaxEntries / 2;
#pragma unroll
  for (int e = 0; e < kMaxEntries; ++e) {
    // (By value: a conditional over array elements would index the array.)
    const uint32_t ka = e + h < kMaxEntries ? w[2 * (e + h < kMaxEntries ? e + h : 0)] : 0u;
    const uint32_t va = e + h < kMaxEntries ? w[2 * (e + h < kMaxEntries ? e + h : 0) + 1] : 0u;
    const uint32_t kb = e + h + 1 < kMaxEntries ? w[2 * (e + h + 1 < kMaxEntries ? e + h + 1 : 0)] : 0u;
    const uint32_t vb = e + h + 1 < kMaxEntries ? w[2 * (e + h + 1 < kMaxEntries ? e + h + 1 : 0) + 1] : 0u;
    w[2 * e] = up ? kb : ka;
    w[2 * e + 1] = up ? vb : va;
  }
  w[WORD_META] = META_BORDER | (w[WORD_META] & META_SIB) | ((uint32_t)kMaxEntries - sp);
  w[WORD_KS] >>= 2u * sp;
}
// The image of the lower half (entries 0 .. sp-1), with its new sibling.
MT_DEV void lane_lower_half(uint32_t (&w)[32], uint32_t sp, uint32_t high, uint32_t sib) {
#pragma unroll
  for (int e = kMaxEntries / 2; e < kMaxEntries; ++e) {
    lane_set_if((uint32_t)e >= sp, w[2 * e], 0u);
    lane_set_if((uint32_t)e >= sp, w[2 * e + 1], 0u);
  }
  w[WORD_KS] &= (1u << (2u * sp)) - 1u;
  w[WORD_META] = (w[WORD_META] & ~META_COUNT) | META_SIB | sp;
  w[WORD_HIGH] = high;
  w[WORD_SIB] = sib;
}

// What a lane has to do at its border node.
enum lane_job : uint32_t { JOB_NONE = 0, JOB_ADD = 1, JOB_SET = 2, JOB_DEL = 3 };

// The call's logs of sparse nodes and emptied layers (as coop_erase).
MT_DEV void lane_log_erase(const tree_view& tv, const lane_place& at, const uint32_t* key, uint32_t slice,
                           uint32_t meta) {
  const uint32_t left = meta & META_COUNT;
  const bool is_root = (meta & META_ROOT) != 0u;
  if (tv.merge_log != nullptr && !is_root && (left == kMergeAt || left == 0u)) {
    const uint32_t r = atomicAdd(tv.merge_log, 1u);
    if (r < tv.merge_cap) {
      tv.merge_log[2u + 2u * r] = at.root;
      tv.merge_log[3u + 2u * r] = slice;
    }
  }
  if (tv.layer_log != nullptr && at.layer >= 1u && at.layer < kLayerRecWords && left == 0u && !(meta & META_SIB) &&
      (is_root || tv.merge_log != nullptr)) {
    const uint32_t r = atomicAdd(tv.layer_log, 1u);
    if (r < tv.layer_cap) {
      uint32_t* rec = tv.layer_log + 2u + (size_t)kLayerRecWords * r;
      rec[0] = at.layer;
#pragma unroll 1
      for (uint32_t q = 0; q < at.layer; ++q) rec[1u + q] = key[q];
    }
  }
}

// Where a launch that is followed by a tile kernel puts the requests that lanes
// cannot place (room for all of the launch's requests).
struct defer_list {
  uint32_t* list;
  uint32_t* count;
};

// Serve the requests of src, one per lane and round (OP_FIND with CONC false:
// finds that run beside no writer):
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
//      A full border node below a parent with room is split in the same way.
//   4. What does not fit (roots and parents to be split, entries that become new
//      layers, nodes that stay locked) is served by the whole warp as one tile,
//      one request after the other.  Slabs that its lanes took and did not use
//      are the first that the tile takes.  (A tile kernel after this one, fed
//      through a list, costs a small call a second launch and the latency of the
//      slowest warp: 1,000 inserts on 100K keys 30 us instead of 26, 2,000 mixed
//      requests on 200K keys 41 instead of 38.)
//      In a launch of more than one round (TAIL), where the other lanes' next
//      requests would wait, they go to that list and the slabs taken for them are
//      the last resort of the tile kernel's allocations: a 1M mixed batch with
//      300K new keys 0.78 ms with warps serving them, 0.61 with the list; 200K
//      inserts into 1M keys of 1-8 slices 225 and 174 us.
// Measured against tiles of 8 lanes per find and 32 per write: a pair of 1M
// mixed batches on 16M keys 1.18 ms (4.94), insert + update + find + erase of
// 300K keys each on 4M keys 0.46 ms (1.57), 1M finds (half of them misses) on 1M
// keys of 1-8 slices 124 us (357; 70 warp instructions per find instead of 587).
// Finds are bound by the load path (64% busy: every node goes through shared
// memory as one line) and by issue (51%); mixed batches by the latency of up to
// 17 dependent node visits and two fences per round, with about 4 warps per
// scheduler: at 3, 4, 5 and 6 blocks per SM they differ by less than 4%.
template <int OP, bool CONC, bool TAIL = false, class Src>
MT_DEV void lane_serve(const tree_view& tv, const Src& src, const defer_list& dl = defer_list{}) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  constexpr bool kFinds = OP == OP_MIXED || OP == OP_FIND;
  constexpr bool kInserts = OP == OP_MIXED || OP == OP_INSERT || OP == OP_UPSERT;
  constexpr bool kErases = OP == OP_MIXED || OP == OP_ERASE, kUpdates = OP == OP_MIXED || OP == OP_UPDATE;
  constexpr bool kChains = kInserts || kUpdates, kWrites = kChains || kErases;
  const uint32_t slot = lane_slot(lane_id());
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32u;
  const uint32_t warps = (gridDim.x * blockDim.x) / 32u;
  const pool_view& p = tv.pool;
  const uint32_t n = src.size(), maxV = src.max_value_length();
  const uint32_t per = max(1u, min(32u, (n + warps - 1u) / warps));
  slab_cache<32> cache;
  cache.init(p, warp);
  cache.keeps = !TAIL;
#pragma unroll 1
  for (uint32_t base = warp * per; base < n; base += warps * per) {
    if (__any_sync(kAll, slot == 0u && fatal_error(p))) break;
    const uint32_t pos = base + slot;
    lane_request r;
    r.id = r.kind = r.klen = r.vlen = 0;
    r.key = nullptr;
    r.val = nullptr;
    r.out_len = nullptr;
    r.out_ok = nullptr;
    uint32_t have = LANE_SKIP;
    if (slot < per && pos < n) have = src.template fetch<OP>(p, pos, r);
    const bool act = have == LANE_SERVE;
    const uint32_t klen = r.klen, vlen = r.vlen;
    const uint32_t* key = r.key;
    uint32_t* val = r.val;
    const bool find = kFinds && act && r.kind == MT_REQ_FIND;
    const bool insert = kInserts && act && r.kind == MT_REQ_INSERT;
    const bool update = kUpdates && act && r.kind == MT_REQ_UPDATE;
    const bool erase = kErases && act && r.kind == MT_REQ_ERASE;
    if (kChains && (insert || update)) asm volatile("prefetch.global.L2 [%0];" ::"l"(val));
    bool defer = kChains && (insert || update) && (klen == 0u || klen > kMaxLen16 || vlen > kMaxLen16);
    bool go = act && !defer && klen > 0u;

    // 1. To the border node.
    lane_place at;
    at.idx = 0;
    at.full = at.stuck = false;
    lane_locate<CONC>(tv, go, key, klen, at);
    bool chain = go && at.found && (at.state == KS_SUFFIX || (find && at.state == KS_LONGVAL));
    if (chain && !p.valid(at.val)) {
      lane_error(p.err, ERR_CORRUPT, MT_AT(SRC_LANE));
      chain = go = false;
    }

    // 2. Chains: compare and copy, then write.
    const bool more = at.layer + 1u < klen;
    const uint32_t rest = more ? klen - at.layer - 1u : 0u;
    if (chain) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.addr(at.val)));
    bool eq = false;
    uint32_t cv = 0, res = 0, found_len = 0;
    warp_chains<kFinds>(p, chain, at.val, key + at.layer + 1u, rest, find ? val : nullptr, maxV, eq, cv);
    const bool present = go && at.found && (at.state != KS_SUFFIX || eq);
    if (find && present) {
      if (at.state == KS_VALUE) {
        if (val != nullptr && maxV > 0u) val[0] = at.val;
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
      } else if (at.stuck) {
        defer = true;
      } else {
        job = JOB_ADD;
      }
    }
    uint32_t nv = kInvalid, ns = KS_VALUE, spare = kInvalid;
    if (kChains) {
      uint32_t need = 0;
      const bool right_half = kInserts && job == JOB_ADD && at.full && at.parent != kInvalid;
      if (job == JOB_ADD || job == JOB_SET) {
        ns = more ? KS_SUFFIX : (vlen == 1u ? KS_VALUE : KS_LONGVAL);
        if (ns == KS_VALUE) nv = val[0];
        else need = suf_nodes(rest, vlen);
      }
      lane_slabs sl{};
      if (!warp_take_slabs<TAIL>(p, need + (right_half ? 1u : 0u), cache, sl)) {
        job = JOB_NONE;
        defer = true;
        need = 0;
      } else if (right_half) {
        spare = lane_slab(p, sl, need);
      }
      warp_write_chains(p, need != 0u, sl, key + at.layer + 1u, rest, val, vlen, nv);
      __syncwarp();
      fence_release();
    }

    // 3. The border node.
    const uint32_t slice = klen > 0u && act ? key[at.layer] : 0u;
    uint32_t idx = at.idx, tries = 0, old_chain = kInvalid;
#pragma unroll 1
    while (kWrites && __any_sync(kAll, job != JOB_NONE)) {
      uint32_t w[32];
      bool won = false, split = false, parent_ok = false;
      uint32_t e = 0, pslot = 0, pmeta = 0;
      if (job != JOB_NONE && ++tries > kLaneTries) {
        job = JOB_NONE;
        defer = true;
      }
      // Where the node is to be split, its parent must list it and have room;
      // then the node itself.  A torn image counts as a lock that is held.
      if (kInserts && job != JOB_NONE && spare != kInvalid) {
        lane_load_relaxed(p.addr(at.parent), w);
        pmeta = lane_verify(w) ? w[WORD_META] : META_LOCK;
        uint32_t hits = 0;
#pragma unroll
        for (int k = 0; k < kMaxEntries; ++k)
          if ((uint32_t)k < (pmeta & META_COUNT) && w[2 * k + 1] == idx) hits |= 1u << k;
        parent_ok = (pmeta & META_LOCK) ||
                    (hits != 0u && !(pmeta & META_BORDER) && (pmeta & META_COUNT) < (uint32_t)kMaxEntries);
        pslot = (uint32_t)__ffs(hits) - 1u;
      }
      bool read = false;
      if (job != JOB_NONE) {
        lane_load_relaxed(p.addr(idx), w);
        read = lane_verify(w);
      }
      if (read) {
        const uint32_t meta = w[WORD_META];
        if ((meta & META_SIB) && slice > w[WORD_HIGH]) {
          idx = w[WORD_SIB];
          if (!p.valid(idx)) {
            lane_error(p.err, ERR_CORRUPT, MT_AT(SRC_LANE));
            job = JOB_NONE;
          }
        } else if (!(meta & META_BORDER)) {
          job = JOB_NONE;  // a layer root that was split meanwhile
          defer = true;
        } else if (!(meta & META_LOCK)) {
          const uint32_t ks = w[WORD_KS];
          uint32_t k, v;
          e = lane_search(w, slice, more, k, v);
          const bool hit = lane_is_entry(meta, ks, e, k, slice, more);
          const uint32_t st = ks_get(ks, e);
          bool lock = false;
          if (job == JOB_ADD) {
            const bool full = (meta & META_COUNT) >= (uint32_t)kMaxEntries;
            if (hit || (full && ((meta & META_ROOT) || !parent_ok))) {
              job = JOB_NONE;  // the slice was taken meanwhile, or a split that is not this node's alone
              defer = true;
            } else if (!full) {
              lock = true;
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
            if (won && job != JOB_ADD && (st & KS_SLAB)) old_chain = v;  // (not a LINK)
          }
        }
      }
      // Publish: first new right halves (visible before anything leads to
      // them), then the nodes, then the parents of split ones.
      const bool splits = kInserts && __any_sync(kAll, won && split);
      uint32_t high = 0;
      if (splits) {
        if (won && split) {
          const uint32_t sp = lane_split_pos(w, high);
          lane_upper_half(w, sp);
          if (slice > high) lane_insert_entry(w, e - sp, slice, nv, ns);
          lane_seal(w);
          lane_store_weak(p.addr(spare), w);
          lane_load_relaxed(p.addr(idx), w);  // locked by this lane: as read above
          lane_lower_half(w, sp, high, spare);
        }
        __syncwarp();
        fence_release();
      }
      if (won) {
        if (kInserts && job == JOB_ADD && (!split || slice <= high)) lane_insert_entry(w, e, slice, nv, ns);
        if (kChains && job == JOB_SET) {
#pragma unroll
          for (int k = 0; k < kMaxEntries; ++k) lane_set_if((uint32_t)k == e, w[2 * k + 1], nv);
          w[WORD_KS] = (w[WORD_KS] & ~(3u << (2u * e))) | (ns << (2u * e));
        }
        if (kErases && job == JOB_DEL) lane_remove_entry(w, e);
        w[WORD_META] = (w[WORD_META] | META_LOCK) + META_VERSION_ONE;
        lane_seal(w);
        lane_store_weak(p.addr(idx), w);
      }
      if (splits && won && split) {
        lane_load_relaxed(p.addr(at.parent), w);  // locked by this lane: as read above
        lane_insert_entry(w, pslot, high, idx, 0u);
#pragma unroll
        for (int k = 1; k < kMaxEntries; ++k) lane_set_if((uint32_t)k == pslot + 1u, w[2 * k + 1], spare);
        w[WORD_META] = (w[WORD_META] | META_LOCK) + META_VERSION_ONE;
        lane_seal(w);
        lane_store_weak(p.addr(at.parent), w);
      }
      if (__any_sync(kAll, won)) fence_release();
      if (won) {
        red_and_relaxed(p.addr(idx) + WORD_META, ~META_LOCK);
        if (kInserts && split) {
          red_and_relaxed(p.addr(at.parent) + WORD_META, ~META_LOCK);
          spare = kInvalid;
        }
        if (kErases && job == JOB_DEL) lane_log_erase(tv, at, key, slice, w[WORD_META]);
        nv = kInvalid;  // in the tree now
        res = 1u;
        job = JOB_NONE;
      }
    }
    // Chains replaced or erased, and slabs taken in vain.
    if (kWrites && old_chain != kInvalid) lane_retire_chain(p, old_chain);
    if (kChains && (ns & KS_SLAB) && nv != kInvalid) lane_keep_slabs<TAIL>(p, nv, suf_nodes(rest, vlen), cache);
    if (kInserts && spare != kInvalid) lane_keep_slabs<TAIL>(p, spare, 1u, cache);

    // 4. What is left: to the list, or by the whole warp as one tile, one request
    // after the other.
    if (kWrites && TAIL) {
      const uint32_t m = __ballot_sync(kAll, defer);
      if (m) {
        uint32_t at0 = 0;
        if (lane_id() == 0u) at0 = atomicAdd(dl.count, (uint32_t)__popc(m));
        at0 = __shfl_sync(kAll, at0, 0);
        if (defer) dl.list[at0 + __popc(m & ((1u << lane_id()) - 1u))] = r.id;
      }
    }
    if constexpr (kWrites && !TAIL) {
      uint32_t left = __ballot_sync(kAll, defer);
      const tile<32> t;
#pragma unroll 1
      while (left) {
        const int l = __ffs(left) - 1;
        left &= left - 1u;
        const uint32_t* k = reinterpret_cast<const uint32_t*>(t.shfl64(reinterpret_cast<uint64_t>(key), l));
        const uint32_t* v = reinterpret_cast<const uint32_t*>(t.shfl64(reinterpret_cast<uint64_t>(val), l));
        const uint32_t kl = t.shfl(klen, l), vl = t.shfl(vlen, l), kind = t.shfl(r.kind, l);
        int done = RES_FAIL;
        if (kInserts && kind == MT_REQ_INSERT) done = coop_insert<32, OP == OP_UPSERT>(t, tv, cache, k, kl, v, vl);
        else if (kUpdates && kind == MT_REQ_UPDATE) done = coop_update<32>(t, tv, cache, k, kl, v, vl);
        else if (kErases && kind == MT_REQ_ERASE) done = coop_erase<32>(t, tv, k, kl);
        if ((int)t.rank == l) res = done == RES_OK;
      }
    }
    if (have != LANE_SKIP && !(TAIL && defer)) {
      if (kFinds && r.kind == MT_REQ_FIND) src.found(pos, r, present, found_len);
      else src.result(pos, r, res != 0u);
    }
  }
  if (kWrites && !TAIL) cache.release(tile<32>(), p);
}

}  // namespace mtb
