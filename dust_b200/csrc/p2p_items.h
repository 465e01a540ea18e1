// p2p_items.h -- how the near field of a leaf is cut into items (k_p2p_split).
//
// A leaf of nt targets with S sources: blocks of 32 targets, each with the
// sources in pieces of `it`, and a last block of the remaining targets, whose
// lanes share the sources, in pieces of it (32 / remainder).  Counts are 64-bit
// (nt S / 2,048 items pass 2^32 at 3 million particles in one leaf), and a leaf
// that would take more than an eighth of the list gets longer pieces (an eighth
// and an item per block then), so that one large leaf leaves room for the others.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define P2P_HD __host__ __device__ __forceinline__
#else
#define P2P_HD inline
#endif

struct P2PCut {
  uint32_t nb;            // whole blocks
  uint32_t it, seg_r;     // sources of an item of a whole block and of the last one
  uint64_t ni_b, ni;      // items of a block, of the leaf
};

P2P_HD P2PCut p2p_cut(uint32_t nt, uint32_t S, uint32_t it, uint64_t cap) {
  P2PCut c;
  c.nb = nt / 32;
  const uint32_t rem = nt % 32;
  for (int q = 0; q < 2; ++q) {
    const uint64_t sr = rem ? (uint64_t)it * (32u / rem) : 1u;
    c.it = it;
    c.seg_r = sr < S ? (uint32_t)sr : S;
    c.ni_b = ((uint64_t)S + it - 1) / it;
    c.ni = c.nb * c.ni_b + (rem ? ((uint64_t)S + c.seg_r - 1) / c.seg_r : 0);
    if (c.ni <= cap / 8) break;
    // (rounded up; a piece of S sources at most)
    const uint64_t longer = it * ((c.ni + cap / 8) / (cap / 8) + 1);
    it = longer < S ? (uint32_t)longer : S;
  }
  return c;
}

// item e of a leaf: its first target and its sources [lo, hi)
P2P_HD void p2p_item(const P2PCut &c, uint32_t S, uint64_t e, uint32_t &tb, uint32_t &lo,
                     uint32_t &hi) {
  const uint64_t b = e / c.ni_b < c.nb ? e / c.ni_b : c.nb, s = e - b * c.ni_b;
  const uint64_t seg = b < c.nb ? c.it : c.seg_r, end = (s + 1) * seg;
  tb = 32u * (uint32_t)b;
  lo = (uint32_t)(s * seg);
  hi = end < S ? (uint32_t)end : S;
}
