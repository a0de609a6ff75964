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

// Bits 2e of the entries e < n of a border node whose key continues past its
// slice (more) or ends at it (!more).
MT_DEV uint32_t lane_eligible(uint32_t meta, uint32_t ks, bool more) {
  const uint32_t n = meta & META_COUNT;
  return (more ? ks : ~ks) & 0x01555555u & ((1u << (2u * n)) - 1u);
}

// Where a request's key belongs: the border node of its last layer and, when
// the node has an entry for (slice, continues), that entry.
struct lane_place {
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
    if (!hit) return true;
    const uint32_t state = (more ? KS_MORE : 0u) | ((w[WORD_KS] & (hit << 1)) ? KS_SLAB : 0u);
    if (state != KS_LINK) {
      at.found = true;
      at.state = state;
      at.val = val;
      return true;
    }
    idx = val;
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

}  // namespace mtb
