// Range scans of the host API: 16 lanes per query, one lane per entry of the
// border node at hand.
//
// At 16 lanes a node image puts entry e's slice and value into lane e
// (mt_node.cuh), so the results of a border node are written side by side: each
// lane reads its own entry's chain line and writes its own output row.  (With
// one entry after the other, as coop_scan does, a query waits for 13 chain
// lines per node in turn.)  400K queries of 100 results on 32M keys: 2.01 ms,
// from 5.25 ms with one entry after the other on 4 lanes; bound by random
// 128-byte lines, of which a result uses a few words.  (Before the bulk build
// laid neighbours' chains side by side: 2.30 ms at 8 blocks per SM, 2.54 at 6 and
// 2.77 at 10, and no change from asking L2 for the next node's chains.  Asking
// for child layers' roots ahead: 30K bounded scans over layers 124 -> 141 us.)
#pragma once
#include "mt_internal.cuh"

namespace mtb {

// Output rows of up to this many slices (key and value together) are written by
// one lane each; longer ones by the whole tile, one row after the other.  30K
// queries of 20 results with rows of 40 + 30 slices: 290 us by lanes, 377 by the
// tile; 3K queries of one result with rows of 100 + 60 slices: 45 and 28 us.
#ifndef MT_SCAN_LANE_ROW
#define MT_SCAN_LANE_ROW 96
#endif
constexpr uint32_t kScanLaneRow = MT_SCAN_LANE_ROW;

// Write the results of entries [start, start + m) of border node nd (none of
// them a LINK) as results c0, c0 + 1, ...  False after a recorded error; then
// `m` is the number written.
template <ld_order OS>
MT_DEV bool scan_emit_node(const tile<16>& t, const pool_view& p, const scan_frames<16>& frames, uint32_t layer,
                           const node<16>& nd, uint32_t start, uint32_t& m, const scan_out& o, uint32_t c0) {
  const uint32_t e = t.rank;
  const uint32_t st = ks_get(nd.ks, min(e, (uint32_t)kMaxEntries - 1u));
  const uint32_t key = nd.w[0], v = nd.w[1];
  bool mine = e >= start && e < start + m;
  const uint32_t bad = t.ballot(mine && (st & KS_SLAB) && !p.valid(v));
  if (bad) {
    if (t.leader()) record_error(p, ERR_CORRUPT, MT_AT(SRC_SCAN));
    m = (uint32_t)__ffs(bad) - 1u - start;
    mine = mine && e < start + m;
  }
  if ((o.keys ? o.maxK : 0u) + (o.values ? o.maxV : 0u) > kScanLaneRow) {
    // The chains are read one after the other: all of them asked for first.
    if (mine && (st & KS_SLAB)) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.addr(v)));
    for (uint32_t k = start; k < start + m; ++k) {
      const uint32_t ks = t.shfl(st, (int)k), kv = t.shfl(v, (int)k), slice = t.shfl(key, (int)k);
      suffix_head<16> h;
      if (ks & KS_SLAB) h.template load<OS>(t, p, kv);
      scan_emit<16, OS>(t, p, frames, layer, slice, ks, kv, (ks & KS_SLAB) ? &h : nullptr, o, c0 + k - start);
    }
    return bad == 0u;
  }
  if (mine) {
    const uint32_t c = c0 + e - start;
    uint32_t d[8];
    uint32_t rest = 0, vlen = 1;
    const uint32_t* a = p.addr((st & KS_SLAB) ? v : 0u);
    if (st & KS_SLAB) {
      load_words<8, OS>(a, d);
      const uint32_t hdr = ld_word<OS>(a + SUF_WORD_HDR);
      rest = hdr & kMaxLen16;
      vlen = hdr >> 16;
    } else {
      d[0] = v;
#pragma unroll
      for (int i = 1; i < 8; ++i) d[i] = 0u;
    }
    if (o.key_lengths) o.key_lengths[c] = layer + 1u + rest;
    if (o.value_lengths) o.value_lengths[c] = vlen;
    // Data words [0, nk) go to the key row, [rest, rest + nv) to the value row.
    uint32_t nk = 0, nv = 0;
    uint32_t* krow = nullptr;
    uint32_t* vrow = nullptr;
    if (o.keys) {
      krow = o.keys + (size_t)c * o.maxK;
      for (uint32_t i = 0; i < layer && i < o.maxK; ++i) krow[i] = frames.slice_at(p, i);
      if (layer < o.maxK) krow[layer] = key;
      nk = min(rest, o.maxK > layer + 1u ? o.maxK - layer - 1u : 0u);
      krow += layer + 1u;
    }
    if (o.values) {
      vrow = o.values + (size_t)c * o.maxV;
      nv = min(vlen, o.maxV);
    }
#pragma unroll
    for (uint32_t i = 0; i < 8u; ++i) {
      if (i < nk) krow[i] = d[i];
      if (i >= rest && i - rest < nv) vrow[i - rest] = d[i];
    }
    const uint32_t last = nv ? rest + nv : nk;
    uint32_t base = 0;
    for (uint32_t i = 8u; i < last; ++i) {
      if (i - base >= kSufData) {
        const uint32_t nx = ld_word<OS>(a + SUF_WORD_NEXT);
        if (!p.valid(nx)) break;
        a = p.addr(nx);
        base += kSufData;
      }
      if (i >= nk && i < rest) continue;
      const uint32_t x = ld_word<OS>(a + (i - base));
      if (i < nk) krow[i] = x;
      else vrow[i - rest] = x;
    }
  }
  t.sync();
  return bad == 0u;
}

// Sign of the key rest of the chain at v against K[0..lk).
template <ld_order OS>
MT_DEV int scan_compare(const tile<16>& t, const pool_view& p, uint32_t v, const uint32_t* K, uint32_t lk) {
  suffix_head<16> h;
  h.template load<OS>(t, p, v);
  return suffix_compare<16, OS>(t, p, h, K, lk).sign;
}

// The walk of coop_scan_walk (mt_tree.cuh), a border node at a time.
template <bool CONCURRENT>
MT_DEV uint32_t scan_query(const tile<16>& t, const tree_view& tv, const uint32_t* lower, uint32_t llen, bool use_upper,
                           const uint32_t* upper, uint32_t ulen, uint32_t max_count, const scan_out& o,
                           scan_frames<16>& frames) {
  constexpr ld_order O = CONCURRENT ? kConc : ld_order::NC;
  constexpr ld_order OS = CONCURRENT ? kConcSuffix : ld_order::NC;
  const pool_view& p = tv.pool;
  if (max_count == 0u) return 0u;
  if (use_upper && ulen == 0u) return 0u;
  uint32_t count = 0, hops = 0, layer = 0;
  const uint32_t hop_limit = kMaxHops + 8u * max_count;
  bool ltight = llen > 0u;  // still on the lower bound's path
  bool utight = use_upper;  // still on the upper bound's path
  node<16> nd;
  uint32_t start;
  {
    const uint32_t s0 = ltight ? lower[0] : 0u;
    if (!descend<16, O>(t, p, tv.root, s0, nd, hops, hop_limit)) return 0u;
    start = ltight ? nd.lower_pos(t, s0, llen > 1u) : 0u;
  }
  while (true) {
    const uint32_t n = nd.count();
    const uint32_t e = t.rank;
    const uint32_t key = nd.w[0], val = nd.w[1];
    const uint32_t st = ks_get(nd.ks, min(e, (uint32_t)kMaxEntries - 1u));
    const bool more = ks_more(st);
    const bool live = e < n;
    if (t.leader() && nd.has_sib() && p.valid(nd.sib))
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.addr(nd.sib)));
    bool child_ltight = false, child_utight = false, done = false;
    if (ltight) {
      // Entries before the lower bound are passed over; the one at its
      // position decides by its key rest.
      const uint32_t ls = lower[layer];
      const bool lm = layer + 1u < llen;
      start = max(start, (uint32_t)__popc(t.ballot(live && pos_less(key, more, ls, lm))));
      const uint32_t eq = t.ballot(live && e >= start && key == ls && more == lm);
      if (eq) {
        const int at = __ffs(eq) - 1;
        const uint32_t es = t.shfl(st, at), ev = t.shfl(val, at);
        if (es == KS_SUFFIX) {
          if (!p.valid(ev)) {
            if (t.leader()) record_error(p, ERR_CORRUPT, MT_AT(SRC_SCAN));
            return count;
          }
          if (scan_compare<OS>(t, p, ev, lower + layer + 1u, llen - layer - 1u) < 0) start = (uint32_t)at + 1u;
        } else if (es == KS_LINK) {
          child_ltight = true;
        }
      }
      ltight = false;
    }
    uint32_t stop = n;
    const uint32_t lower_at = child_ltight ? start : 0xFFFFFFFFu;
    uint32_t upper_at = 0xFFFFFFFFu;
    if (utight) {
      const uint32_t us = upper[layer];
      const bool um = layer + 1u < ulen;
      const uint32_t beyond = t.ballot(live && pos_less(us, um, key, more));
      if (beyond) {
        stop = (uint32_t)__ffs(beyond) - 1u;
        done = true;
      }
      const uint32_t eq = t.ballot(live && e >= start && key == us && more == um);
      if (eq) {
        const uint32_t at = (uint32_t)__ffs(eq) - 1u;
        const uint32_t es = t.shfl(st, (int)at), ev = t.shfl(val, (int)at);
        if (es == KS_LINK) {
          upper_at = at;
        } else {
          int sign = 0;
          if (es == KS_SUFFIX) {
            if (!p.valid(ev)) {
              if (t.leader()) record_error(p, ERR_CORRUPT, MT_AT(SRC_SCAN));
              return count;
            }
            sign = scan_compare<OS>(t, p, ev, upper + layer + 1u, ulen - layer - 1u);
          }
          stop = at + (sign > 0 ? 0u : 1u);
          done = true;
        }
      }
    }
    const uint32_t links = t.ballot(live && e >= start && e < stop && st == KS_LINK);
    const uint32_t lend = links ? (uint32_t)__ffs(links) - 1u : max(start, stop);
    uint32_t m = min(lend - start, max_count - count);
    if (m) {
      const bool fine = scan_emit_node<OS>(t, p, frames, layer, nd, start, m, o, count);
      count += m;
      if (!fine || count >= max_count) return count;
    }
    if (links) {
      child_ltight = lower_at == lend;
      child_utight = upper_at == lend;
      const uint32_t s = t.shfl(key, (int)lend), v = t.shfl(val, (int)lend);
      scan_frame f;
      f.node = nd.idx;
      f.slice = s;
      f.upper_tight = utight ? 1u : 0u;
      f.pad = 0u;
      if (!frames.push(t, p, layer, f)) return count;
      ++layer;
      ltight = child_ltight;
      utight = child_utight;
      const uint32_t s0 = ltight ? lower[layer] : 0u;
      if (!descend<16, O>(t, p, v, s0, nd, hops, hop_limit)) return count;
      start = ltight ? nd.lower_pos(t, s0, layer + 1u < llen) : 0u;
      continue;
    }
    if (done) return count;
    // Next border node of this layer.
    if (nd.has_sib()) {
      if (utight && nd.high >= upper[layer]) return count;
      const uint32_t sib = nd.sib;
      if (!p.valid(sib) || ++hops > hop_limit) {
        if (t.leader()) record_error(p, ERR_CORRUPT, MT_AT(SRC_SCAN));
        return count;
      }
      if (!nd.template load_verified<O>(t, p, sib)) return count;
      start = 0;
      continue;
    }
    // End of this layer: resume the parent layer after the LINK slice.
    scan_frame f;
    do {
      if (layer == 0u) return count;
      t.sync();
      --layer;
      f = frames.pop_to(t, p, layer);
      utight = f.upper_tight != 0u;
      if (utight && f.slice == upper[layer]) return count;  // the LINK was upper's own path
      if (!p.valid(f.node)) {
        if (t.leader()) record_error(p, ERR_CORRUPT, MT_AT(SRC_SCAN));
        return count;
      }
    } while (f.slice == 0xFFFFFFFFu);  // nothing can follow that slice in its layer
    if (!nd.template load_verified<O>(t, p, f.node)) return count;
    while (nd.must_move_right(f.slice)) {
      if (!p.valid(nd.sib) || ++hops > hop_limit) {
        if (t.leader()) record_error(p, ERR_CORRUPT, MT_AT(SRC_SCAN));
        return count;
      }
      if (!nd.template load_verified<O>(t, p, nd.sib)) return count;
    }
    start = __popc(nd.entry_mask(t, [&](uint32_t k, uint32_t) { return k <= f.slice; }));
  }
}

}  // namespace mtb
