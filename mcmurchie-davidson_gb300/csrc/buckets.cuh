// buckets.cuh -- how the quartets of an unscreened class are counted and numbered: host
// and device arithmetic without CUDA types, so that a host compiler takes it too.
//
// A bucket's quartets are counted in 64 bits: the pairs of one molecule's class reach
// 72,828 ((ps) of 51 waters 6-31G**), so a class has more than 2^32 quartets and one
// triangle's a (a + 1) passes 2^32 from a = 65,536 on.
#pragma once

#ifdef __CUDACC__
#define MMDG_HD __host__ __device__ __forceinline__
#else
#include <math.h>
#define MMDG_HD inline
#endif

namespace mmdg {

constexpr int kMaxKeys = 256;
constexpr int kMaxGroups = 16;  // primitive-count groups per pair-class list (kMaxGroups^2 <= kMaxKeys)

// The buckets of an unscreened class of one molecule: its class lists are sorted by
// primitive count, so group g of the bra list is the slots bstart[g] .. bstart[g + 1),
// each of at most bw[g] primitive pairs; bucket k = gb * nkg + gk is the rectangle of two
// groups (the triangle for a group with itself, nothing for gk > gb, when the lists are
// the same).
struct TensorBuckets {
  int nbg, nkg;
  int bstart[kMaxGroups + 1], kstart[kMaxGroups + 1];
  int bw[kMaxGroups], kw[kMaxGroups];
};

// quartets of bucket k
MMDG_HD unsigned long long bucket_quartets(const TensorBuckets& tb, int same, int k) {
  const int gb = k / tb.nkg, gk = k - gb * tb.nkg;
  const unsigned long long a = tb.bstart[gb + 1] - tb.bstart[gb], b = tb.kstart[gk + 1] - tb.kstart[gk];
  return !same || gk < gb ? a * b : (gk == gb ? a * (a + 1) / 2 : 0ull);
}

// bra and ket list slot of a bucket's quartet
MMDG_HD void bucket_slot(const TensorBuckets& tb, int same, int key, unsigned long long slot, int& ib, int& jk) {
  const int gb = key / tb.nkg, gk = key - gb * tb.nkg;
  if (same && gb == gk) {  // slot = ib (ib + 1) / 2 + jk
    ib = (int)((sqrtf(8.0f * float(slot) + 1.0f) - 1.0f) * 0.5f);
    while ((long long)ib * (ib + 1) / 2 > (long long)slot) --ib;
    while ((long long)(ib + 1) * (ib + 2) / 2 <= (long long)slot) ++ib;
    jk = (int)((long long)slot - (long long)ib * (ib + 1) / 2);
  } else {
    const unsigned b = (unsigned)(tb.kstart[gk + 1] - tb.kstart[gk]);
    ib = slot >> 32 ? (int)(slot / b) : (int)((unsigned)slot / b);  // (a 64-bit division is ten times the work)
    jk = (int)(slot - (unsigned long long)ib * b);
  }
  ib += tb.bstart[gb];
  jk += tb.kstart[gk];
}

// Work items of a bucket of c quartets with 2^lg lanes each: whole warps
template <typename Index>
MMDG_HD Index bucket_items(Index c, int lg) {
  return ((c << lg) + 31) & ~Index(31);
}

}  // namespace mmdg
