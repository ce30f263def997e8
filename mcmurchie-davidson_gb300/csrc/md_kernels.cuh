// md_kernels.cuh -- the shell-quartet kernels (one instantiation per angular class).
//
// Fock builds (formPT semantics): k_screen walks the candidates (bra shell pair, ket
// shell pair) of all angular classes and appends the survivors of the Schwarz x density bound to bucketed quartet lists (buckets
// keyed by the primitive-count groups of the two pairs, FP64 and FP32 lists); then per
// class k_fock, a persistent kernel, evaluates the list, 1 to 32 lanes per (quartet, ket
// chunk) (the lanes share the quartet's primitive pairs, see plan_buckets),
// chunk-major, so a warp shares its code path and, inside a bucket, its primitive
// trip counts.  FP32 lists are split by grid stride; FP64 lists are claimed 32 lanes per
// warp from an atomic counter, so the SMs finish together.  The classes above L = 4 have
// a warp-cooperative Fock kernel of their own (md_warp.cuh).  The ERI tensor enumerates the same buckets without a list (nothing
// is screened), the Schwarz table runs a warp-wide group per heavy pair; listed
// quartets use one thread per shell quartet.
#pragma once
#include "buckets.cuh"
#include "md_device.cuh"
#include "md_gen.cuh"

namespace mmdg {

constexpr int kThreads = 128;     // threads per block (shared-memory R tables are sized for it)
constexpr int kMaxFockBlock = 256; // largest block a k_fock launch may use (autotuned tile)

struct ClassLaunch {
  const int* bra;   // shell-pair indices of the bra class list
  const int* ket;   // shell-pair indices of the ket class list
  int nbra, nket;
  int same;         // bra class == ket class: only ket slot <= bra slot
};

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }

template <class MD, typename Real>
__device__ __forceinline__ Ctx<Real> make_ctx(const Geometry& g, int bp, int kp, Real* rs) {
  Ctx<Real> c;
  c.g = &g;
  c.chunk = -1;
  c.nasym = 0;
  c.bra_begin = __ldg(g.pr_begin + bp);
  c.bra_end = c.bra_begin + __ldg(g.pr_count + bp);
  c.ket_begin = __ldg(g.pr_begin + kp);
  c.ket_end = c.ket_begin + __ldg(g.pr_count + kp);
  c.ebra = __ldg(g.e_off + bp);
  c.eket = __ldg(g.e_off + kp);
  c.nnz_ab = MD::NNZ_AB;
  c.nnz_cd = MD::NNZ_CD;
  c.rs = rs;
  c.rstr = kThreads;
  return c;
}

// Screening pass of all classes: every candidate (bra slot, ket slot) is tested against
// the shell-level bound Q_ab Q_cd max(4D_ab, 4D_cd, D_ac, D_ad, D_bc, D_bd) (an upper
// bound of the function-level test, fock.pyx:46-57) and appended to the FP64 or the FP32
// list of its class.  Each list is split into buckets keyed by (bra primitive-count
// group, ket primitive-count group), so that the 32 quartets a warp evaluates together
// have the same primitive loop trip counts.
struct ScreenClass {
  const int *bra, *ket;       // class lists
  const int* kmoff;           // ket list: slot offset of every molecule (lists are molecule-major)
  const int *gbra, *gket;     // slot -> primitive-count group
  const float* qtile;         // largest Q of every kThreads ket slots
  const long long* key_off;   // bucket offsets within the class region
  long long region;           // first entry of the class in the quartet lists
  int key0, nkg;              // first bucket, groups of the ket list
  int same;                   // bra class == ket class: only ket slot <= bra slot
  int first;                  // its first block
};

__device__ __forceinline__ void bucket_append(bool keep, int key, int2 v, int2* out, unsigned* n,
                                              const long long* key_off) {
  const unsigned act = __activemask();
  const unsigned peers = __match_any_sync(act, keep ? key : -1);
  if (!keep) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(n + key, (unsigned)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  out[key_off[key] + base + __popc(peers & ((1u << lane) - 1u))] = v;
}

// One block per (class, bra slot); its threads walk the ket slots of the same molecule (the
// lists are molecule-major), so a batch of molecules never forms cross-molecule
// candidates.  Tiles of kThreads kets whose largest Q cannot reach the threshold even with
// the molecule's largest density element are passed over unread (most of a big molecule's:
// the lists are sorted by Q inside a primitive-count group).  (H2O)16 6-31G**, all 21
// classes: 0.6 ms; one launch per class, every candidate read, took 1.7.
static __global__ void __launch_bounds__(kThreads) k_screen(Geometry g, FockArgs f, const ScreenClass* classes, int nclass,
                                                            int2* q64, int2* q32, unsigned* n64, unsigned* n32,
                                                            float split, const float* dmax) {
  __shared__ unsigned s_tiles[kThreads / 32];
  int lo = 0, hi = nclass - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (classes[mid].first <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const ScreenClass c = classes[lo];
  const int ib = (int)blockIdx.x - c.first;
  const int bp = __ldg(c.bra + ib);
  const int sa = __ldg(g.pa + bp), sb = __ldg(g.pb + bp);
  const int mol = __ldg(g.sh_mol + sa);
  const float qb = __ldg(g.Q + bp);
  const int gb = __ldg(c.gbra + ib);
  const float* D = f.Dsh + g.mol_sbase[mol];
  const int S = g.mol_ns[mol];
  const int a = __ldg(g.sh_local + sa), b = __ldg(g.sh_local + sb);
  const float dab = 4.0f * __ldg(D + a * S + b);
  const float most = 4.0f * dmax[mol];
  const int k0 = __ldg(c.kmoff + mol);
  int k1 = __ldg(c.kmoff + mol + 1);
  if (c.same) k1 = min(k1, ib + 1);
  n64 += c.key0;
  n32 += c.key0;
  q64 += c.region;
  q32 += c.region;
  const int t1 = (k1 + kThreads - 1) / kThreads;
  for (int t0 = k0 / kThreads; t0 < t1; t0 += kThreads) {
    const int mine = t0 + threadIdx.x;
    const bool open = mine < t1 && !((qb * __ldg(c.qtile + mine)) * most < f.tolf_lo);
    const unsigned bits = __ballot_sync(0xffffffffu, open);
    if ((threadIdx.x & 31) == 0) s_tiles[threadIdx.x >> 5] = bits;
    __syncthreads();
    for (int w = 0; w < kThreads / 32; ++w) {
      for (unsigned left = s_tiles[w]; left; left &= left - 1) {
        const int jk = (t0 + 32 * w + __ffs(left) - 1) * kThreads + threadIdx.x;
        bool keep = jk >= k0 && jk < k1;
        float qq = 0.f;
        int key = 0;
        if (keep) {
          const int kp = __ldg(c.ket + jk);
          const int sc = __ldg(g.pa + kp), sd = __ldg(g.pb + kp);
          qq = qb * __ldg(g.Q + kp);
          const int cc = __ldg(g.sh_local + sc), d = __ldg(g.sh_local + sd);
          const float dm = fmaxf(fmaxf(dab, 4.0f * __ldg(D + cc * S + d)),
                                 fmaxf(fmaxf(__ldg(D + a * S + cc), __ldg(D + a * S + d)),
                                       fmaxf(__ldg(D + b * S + cc), __ldg(D + b * S + d))));
          keep = qq * dm >= f.tolf_lo;
          if (f.pair_owner) {
            const int own = __ldg(f.pair_canon + bp) >= __ldg(f.pair_canon + kp) ? __ldg(f.pair_owner + bp)
                                                                                  : __ldg(f.pair_owner + kp);
            keep = keep && own == f.part;
          }
          key = gb * c.nkg + __ldg(c.gket + jk);
        }
        const bool low = qq < split;  // 0: no FP32 list
        const int2 v = make_int2(ib, jk);
        bucket_append(keep && !low, key, v, q64, n64, c.key_off);
        if (split > 0.f) bucket_append(keep && low, key, v, q32, n32, c.key_off);
      }
    }
    __syncthreads();
  }
}

// largest Q of every kThreads slots of the pair-class lists (blockIdx.y)
constexpr int kPairClasses = 6;
struct TileArgs {
  const int* list[kPairClasses];
  int n[kPairClasses];
  float* qtile[kPairClasses];
};
static __global__ void __launch_bounds__(kThreads) k_tile_q(TileArgs a, const float* Q) {
  __shared__ int s_q[kThreads / 32];
  const int c = blockIdx.y, x = blockIdx.x * kThreads + threadIdx.x;
  if ((int)blockIdx.x * kThreads >= a.n[c]) return;
  const int q = x < a.n[c] ? __float_as_int(Q[a.list[c][x]]) : 0;  // Q >= 0: ordered as integers
  const int m = __reduce_max_sync(0xffffffffu, q);
  if ((threadIdx.x & 31) == 0) s_q[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    int v = s_q[0];
    for (int w = 1; w < kThreads / 32; ++w) v = max(v, s_q[w]);
    a.qtile[c][blockIdx.x] = __int_as_float(v);
  }
}

// One bucketed list of a class: bucket k holds count[k] quartets from key_off[k] on, each
// of about key_w[k] primitive quartets.
struct BucketList {
  const int2* list;
  const unsigned* count;
  const long long* key_off;
  const int* key_w;
  int nkeys;
};

// How a launch walks its buckets: position x (heaviest bucket, stored last, first) covers
// the work items pre[x] .. pre[x + 1), a multiple of 32, of bucket nkeys - 1 - x, with
// 2^lg[x] lanes per quartet.  Index: unsigned for the Fock lists, whose lengths are 32-bit
// counters, 64 bits for the unscreened classes (buckets.cuh).
template <typename Index>
struct BucketPlan {
  Index pre[kMaxKeys + 1];
  unsigned char lg[kMaxKeys];
};

// Lanes per quartet.  A quartet of w primitive quartets on one thread is a serial chain of
// w x ~1.1 us, whatever the rest of the GPU does: an oxygen-core (ss|ss) quartet (1296)
// took 1.4 ms, which alone was the length of that class's launch on (H2O)4 and of most
// classes on one molecule.  So a bucket's quartets get the smallest power of two of lanes
// (up to 32) that brings a lane below twice the launch's average work per thread (never
// below kLanePrims primitive quartets: a shorter share costs more in digestion and sums
// over the lanes than it saves).  Long lists thus keep one lane per quartet except for
// the few heavy buckets that would run on after the others.  Measured (ms per build, 8
// streams; share of 1/4, 1/2, 1, 2 averages, sums over the lanes): (H2O)4 6-31G** 1.87,
// 1.52, 1.44, 1.30; (H2O)16 with FP32 below 1e-5 24.4, 23.3, 22.6, 22.3; kLanePrims 2, 4,
// 8 on (H2O)4: 2.45, 1.44, 1.33, 4 the better on one stream.  One thread per quartet: 2.74.
constexpr float kLanePrims = 4.0f;

template <typename Index, class CountF, class WeightF>
__device__ __forceinline__ void plan_buckets(BucketPlan<Index>& p, int nkeys, int nchunk, long long nthreads, CountF count,
                                             WeightF weight, int most = 5) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    float W = 0.f;
    for (int x = lane; x < nkeys; x += 32) W += float(count(nkeys - 1 - x)) * float(weight(nkeys - 1 - x));
    for (int o = 16; o > 0; o >>= 1) W += __shfl_xor_sync(0xffffffffu, W, o);
    const float share = fmaxf(kLanePrims, 2.0f * W * float(nchunk) / float(nthreads));
    Index acc = 0;
    for (int x0 = 0; x0 < nkeys; x0 += 32) {
      const int x = x0 + lane;
      Index len = 0;
      int lg = 0;
      if (x < nkeys) {
        const Index c = count(nkeys - 1 - x);
        const float w = float(weight(nkeys - 1 - x));
        while (lg < most && w > share * float(1 << lg)) ++lg;
        len = bucket_items(c, lg);
      }
      Index end = len;
      for (int d = 1; d < 32; d <<= 1) {
        const Index t = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += t;
      }
      if (x < nkeys) {
        p.pre[x] = acc + end - len;
        p.lg[x] = (unsigned char)lg;
      }
      acc += __shfl_sync(0xffffffffu, end, 31);
    }
    if (lane == 0) p.pre[nkeys] = acc;
  }
  __syncthreads();
}

// The share of lane `sub` of a 2^lg-lane group: the bra primitive pairs are split first
// (their transform runs once per bra pair), the ket ones among the remaining lanes.
template <class C>
__device__ __forceinline__ void split_primitives(C& c, int lg, int sub) {
  if (lg == 0) return;
  const int nb = c.bra_end - c.bra_begin, nk = c.ket_end - c.ket_begin;
  const int lb = min(lg, 31 - __clz(nb)), lk = lg - lb;
  const int sb = sub & ((1 << lb) - 1), sk = sub >> lb;
  const int b0 = (sb * nb) >> lb, b1 = ((sb + 1) * nb) >> lb;
  const int k0 = (sk * nk) >> lk, k1 = ((sk + 1) * nk) >> lk;
  c.bra_end = c.bra_begin + (k1 > k0 ? b1 : b0);  // no ket pair left for this lane: nothing to do
  c.bra_begin += b0;
  c.ebra += (long long)b0 * c.nnz_ab;
  c.ket_end = c.ket_begin + k1;
  c.ket_begin += k0;
  c.eket += (long long)k0 * c.nnz_cd;
}

// A digest behind a group of 2^lg lanes: every value is summed over the group, and the
// lanes take turns in digesting the sums.
template <class Digest>
struct GroupDigest {
  Digest& d;
  int lanes, sub;
  unsigned mask;
  int turn;
  __device__ __forceinline__ GroupDigest(Digest& d_, int lg, int lane)
      : d(d_), lanes(1 << lg), sub(lane & ((1 << lg) - 1)),
        mask((lg == 5 ? 0xffffffffu : ((1u << (1 << lg)) - 1u)) << (lane & ~((1 << lg) - 1))), turn(0) {}
  template <typename Real>
  __device__ __forceinline__ void put(int ca, int cb, int cc, int cd, Real v) {
    for (int o = 1; o < lanes; o <<= 1) v += __shfl_xor_sync(mask, v, o);
    if ((turn++ & (lanes - 1)) == sub) d.put(ca, cb, cc, cd, v);
  }
};

// Evaluation of a bucketed quartet list: persistent loop over (chunk, bucket, quartet),
// chunk-major, so that a warp shares its chunk (code path) and its primitive trip
// counts; heaviest buckets first.  The lanes of an FP64 quartet sum their integrals with
// shuffles and take turns in digesting the sums (digesting every lane's partial integrals
// instead, G being linear in them, rounds once per lane: the error of G against 64 bits
// went from 5.6e-15 to 8.0e-15 on (H2O)4).  The one-lane path stays separate: the group's
// bookkeeping in every digestion cost it 3-7 % on (H2O)16.  The lanes of an FP32 quartet
// do digest partial integrals, which spares that kernel up to 40 registers.
//
// FP64 lists claim their work: each warp takes the next 32 items from the launch's
// counter.  With a static grid-stride split the average SM sat idle for 20 % of a
// (ps|ss) launch while the slowest finished (ncu: sm__cycles_active avg 9.9M, max 12.4M
// cycles of 12.4M), and on several streams a block that starts late holds its share
// back.  (Claiming one item ahead hid nothing more on long lists, and on short ones
// left warps idle beside claimed work: mixed (H2O)16 26.7 -> 25.4 ms without.)  Claims of 128 or 256 items were 1.8-2.7x slower (the warps'
// working set of pairs and E' rows spreads over that many more quartets).  The
// memory-latency-bound FP32 lists keep the static split, neighbouring warps on
// neighbouring quartets.
template <class MD, typename Real>
__global__ void __launch_bounds__(kMaxFockBlock) k_fock(Geometry g, FockArgs f, ClassLaunch cl, BucketList bl) {
  __shared__ BucketPlan<unsigned> plan;
  // block size: kThreads for classes with shared-memory R tables, else 64..256 (tile),
  // a multiple of 32 either way, so every warp is full
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  plan_buckets(plan, bl.nkeys, MD::NCHUNK, nthreads, [&](int k) { return __ldg(bl.count + k); },
               [&](int k) { return __ldg(bl.key_w + k); });
  __shared__ unsigned s_count[kMaxKeys];
  __shared__ long long s_off[kMaxKeys];
  for (int x = threadIdx.x; x < bl.nkeys; x += blockDim.x) {  // by plan position
    s_count[x] = __ldg(bl.count + bl.nkeys - 1 - x);
    s_off[x] = __ldg(bl.key_off + bl.nkeys - 1 - x);
  }
  __syncthreads();
  const unsigned n = plan.pre[bl.nkeys];
  const long long total = (long long)n * MD::NCHUNK;
  extern __shared__ double smem_d[];
  Real* rs = reinterpret_cast<Real*>(smem_d) + threadIdx.x;
  unsigned nfq = 0, nsq = 0, npq = 0, nbp = 0, nas = 0;
  int x = 0;
  constexpr bool kClaim = sizeof(Real) == 8;
  const unsigned lane = threadIdx.x & 31u;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;; idx += nthreads) {
    if (kClaim) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(f.work, 32ull);
      idx = (long long)__shfl_sync(0xffffffffu, base, 0) + lane;
    }
    if (idx >= total) break;  // warp-uniform: total is a multiple of 32
    const int chunk = (int)(idx / n);
    const unsigned r = (unsigned)(idx - (long long)chunk * n);
    if (r < plan.pre[x]) x = 0;
    while (r >= plan.pre[x + 1]) ++x;
    const int lg = plan.lg[x];
    const unsigned slot = (r - plan.pre[x]) >> lg;
    if (slot < s_count[x]) {
      const int2 e = bl.list[s_off[x] + (s_count[x] - 1u - slot)];
      const int bp = __ldg(cl.bra + e.x), kp = __ldg(cl.ket + e.y);
      const int sa = __ldg(g.pa + bp), sb = __ldg(g.pb + bp), sc = __ldg(g.pa + kp), sd = __ldg(g.pb + kp);
      Ctx<Real> c = make_ctx<MD, Real>(g, bp, kp, rs);
      c.chunk = MD::NCHUNK > 1 ? chunk : -1;
      QuartetInfo q{sa, sb, sc, sd, sa == sb, sc == sd, bp == kp, __ldg(g.sh_mol + sa)};
      FockDigest<ncart(MD::LB), ncart(MD::LD)> dg(g, f, q);
      const int sub = (int)lane & ((1 << lg) - 1);
      split_primitives(c, lg, sub);
      if (kClaim && lg > 0) {  // warp-uniform: a bucket fills whole warps
        GroupDigest<FockDigest<ncart(MD::LB), ncart(MD::LD)>> gd(dg, lg, (int)lane);
        MD::run(c, gd);
        nfq += dg.nfq;
      } else {
        MD::run(c, dg);
        if (sub == 0) nfq += dg.nfq;
      }
      if (chunk == 0) {
        if (sub == 0) ++nsq;
        npq += unsigned((c.bra_end - c.bra_begin) * (c.ket_end - c.ket_begin));
        nbp += unsigned(c.bra_end - c.bra_begin);
        nas += c.nasym;
      }
    }
  }
  if (f.counters) {
    const unsigned mask = __activemask();
    const unsigned s0 = __reduce_add_sync(mask, nfq), s1 = __reduce_add_sync(mask, nsq),
                   s2 = __reduce_add_sync(mask, npq), s3 = __reduce_add_sync(mask, nbp),
                   s4 = __reduce_add_sync(mask, nas);
    if ((threadIdx.x & 31) == __ffs(mask) - 1 && (s0 | s1 | s2)) {
      atomicAdd(f.counters + 0, (unsigned long long)s0);
      atomicAdd(f.counters + 1, (unsigned long long)s1);
      atomicAdd(f.counters + 2, (unsigned long long)s2);
      atomicAdd(f.counters + 3, (unsigned long long)s3);
      atomicAdd(f.counters + 4, (unsigned long long)s4);
    }
  }
}

// Every ERI of the class into the tensor, 1 to 32 lanes per (quartet, ket chunk) as in
// k_fock, persistent over the buckets.  (One thread per quartet: N = 75 10.6 ms, its 21
// launches each as long as their heaviest quartet; with groups 2.2 ms one after another, the
// classes on eight streams 1.15.)
template <class MD>
__global__ void __launch_bounds__(kThreads) k_tensor(Geometry g, TensorArgs t, ClassLaunch cl, TensorBuckets tb) {
  __shared__ BucketPlan<unsigned long long> plan;
  const int nkeys = tb.nbg * tb.nkg;
  plan_buckets(plan, nkeys, MD::NCHUNK, (long long)gridDim.x * kThreads,
               [&](int k) { return bucket_quartets(tb, cl.same, k); },
               [&](int k) { return tb.bw[k / tb.nkg] * tb.kw[k % tb.nkg]; });
  // (64-bit totals kept in registers would cost the larger classes spills: read where needed)
  const int stride = gridDim.x * kThreads;
  const unsigned lane = threadIdx.x & 31u;
  extern __shared__ double smem_d[];
  double* rs = smem_d + threadIdx.x;
  int x = 0;
  for (long long idx = ((long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + lane;
       idx < (long long)plan.pre[nkeys] * MD::NCHUNK; idx += stride) {
    const int chunk = MD::NCHUNK > 1 ? (int)(idx / (long long)plan.pre[nkeys]) : 0;
    const unsigned long long r = (unsigned long long)idx - chunk * plan.pre[nkeys];
    if (r < plan.pre[x]) x = 0;
    while (r >= plan.pre[x + 1]) ++x;
    const int lg = plan.lg[x], key = nkeys - 1 - x;
    const unsigned long long slot = (r - plan.pre[x]) >> lg;
    if (slot >= bucket_quartets(tb, cl.same, key)) continue;
    int ib, jk;
    bucket_slot(tb, cl.same, key, slot, ib, jk);
    const int bp = __ldg(cl.bra + ib), kp = __ldg(cl.ket + jk);
    const int sa = __ldg(g.pa + bp), sb = __ldg(g.pb + bp), sc = __ldg(g.pa + kp), sd = __ldg(g.pb + kp);
    Ctx<double> c = make_ctx<MD, double>(g, bp, kp, rs);
    c.chunk = MD::NCHUNK > 1 ? chunk : -1;
    QuartetInfo q{sa, sb, sc, sd, sa == sb, sc == sd, bp == kp, __ldg(g.sh_mol + sa)};
    TensorDigest<ncart(MD::LB), ncart(MD::LD)> dg(g, t, q);
    GroupDigest<TensorDigest<ncart(MD::LB), ncart(MD::LD)>> gd(dg, lg, (int)lane);
    split_primitives(c, lg, gd.sub);
    MD::run(c, gd);
  }
}

// listed shell quartets of one class (mmdg_eri_quartets): one thread per (item, ket
// chunk), chunk-major
template <class MD, typename Real>
__global__ void __launch_bounds__(kThreads) k_quartets(Geometry g, QuartetArgs a, const QuartetItem* items, int n) {
  const long long idx = blockIdx.x * (long long)kThreads + threadIdx.x;
  if (idx >= (long long)n * MD::NCHUNK) return;
  const int chunk = (int)(idx / n);
  const QuartetItem it = items[idx - (long long)chunk * n];
  extern __shared__ double smem_d[];
  Real* rs = reinterpret_cast<Real*>(smem_d) + threadIdx.x;
  Ctx<Real> c = make_ctx<MD, Real>(g, it.bra, it.ket, rs);
  c.chunk = MD::NCHUNK > 1 ? chunk : -1;
  QuartetDigest<ncart(MD::LB), ncart(MD::LD)> dg(a, it.slot, it.flags);
  MD::run(c, dg);
}

// diagonal quartets (ab|ab) of one pair class: the Schwarz table.  2^lg lanes per (pair,
// ket chunk), chunk-major; whole groups leave together
template <class MD>
__global__ void __launch_bounds__(kThreads) k_schwarz(Geometry g, SchwarzArgs s, const int* list, int n, int lg) {
  const long long idx = (blockIdx.x * (long long)kThreads + threadIdx.x) >> lg;
  if (idx >= (long long)n * MD::NCHUNK) return;
  const int chunk = (int)(idx / n);
  const int bp = __ldg(list + (idx - (long long)chunk * n));
  const int sa = __ldg(g.pa + bp), sb = __ldg(g.pb + bp);
  extern __shared__ double smem_d[];
  double* rs = smem_d + threadIdx.x;
  Ctx<double> c = make_ctx<MD, double>(g, bp, bp, rs);
  c.chunk = MD::NCHUNK > 1 ? chunk : -1;
  QuartetInfo q{sa, sb, sa, sb, sa == sb, sa == sb, true, __ldg(g.sh_mol + sa)};
  SchwarzDigest<ncart(MD::LB), ncart(MD::LD)> dg(g, s, q, bp);
  GroupDigest<SchwarzDigest<ncart(MD::LB), ncart(MD::LD)>> gd(dg, lg, (int)(threadIdx.x & 31));
  split_primitives(c, lg, gd.sub);
  MD::run(c, gd);
}

template <class MD, typename Real>
constexpr size_t smem_bytes() {
  return MD::RSMEM ? size_t(MD::HL) * kThreads * sizeof(Real) : 0;
}

}  // namespace mmdg

namespace mmdg {
// blocks of a persistent launch: every SM filled to the kernel's occupancy
// (grid > 0: an autotuned grid, capped at that occupancy)
template <typename K>
inline int persistent_blocks(K kernel, size_t smem, int grid = 0, int block = kThreads) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, block, smem);
  const int full = sms * (per > 0 ? per : 1);
  return grid > 0 && grid < full ? grid : full;
}
}  // namespace mmdg
