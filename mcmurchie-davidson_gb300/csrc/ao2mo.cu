// ao2mo.cu -- the AO -> MO four-index transform of the ERI tensor (mmd/postscf.py:26-27:
// four einsums with the MO coefficients, one index at a time).
//
// One quarter transform contracts the last index with C and writes the new index
// first:
//     out[S, p, q, r] = sum_s in[p, q, r, s] C[s, S]
// so four calls of the same kernel turn (pq|rs) into (PQ|RS) in the original index
// order: pqrs -> Spqr -> RSpq -> QRSp -> PQRS.  Each call is a GEMM
// out (N x N^3) = C^T (N x N) . in^T (N x N^3) in FP64: 64 x 64 output tiles per
// 256-thread block, 4 x 4 outputs per thread, the K dimension staged through shared
// memory 16 at a time (k_quarter; N > 128).  An FP64 warp instruction holds the FP64 pipe of its
// sub-partition for ~64 cycles on this GPU, so the eight shared-memory loads around
// a thread's 16 independent FMAs per k step cost nothing; the 16 accumulators keep
// the pipe fed.
//
// Up to N = 128 the product runs on the tensor cores instead (k_quarter_tc): every row of
// the tensor and every column of C is scaled by a power of two and cut into eight signed
// 8-bit digits (62 bits), digits are exact BF16 numbers, and the digit products with
// i + j = d, d = 0..7 (36 of 64), are summed by tcgen05.mma in one FP32 accumulator per d:
// at most 8 x 128 products of at most 2^14, so every sum is an integer of at most 2^24 and
// exact.  The eight integers are put together in fixed point and rounded once.  (Split-
// operand products after K. Ozaki, T. Ogita, S. Oishi and S. M. Rump, Numer. Algorithms 59,
// 95-118, 2012.)
//
// Left out are the bits below a row's and a column's 62 and the digit products with i + j >
// 7, together at most 9.03 units of 2^62 per k in the fixed-point product, whose unit is
// 2^(er + ec - 2168) with er, ec the exponent fields of the row's and the column's largest
// element: at most 9.03 N 2^(er + ec - 2106) (rms 2^-57 of their product at N = 76).  An FP64
// sum may be off by N 2^-53 S, S = sum_k |a_k| |c_k|.  The first is the smaller bound where S
// is at least 2^(er + ec - 2049), an eighth of the product of the two largest elements' powers
// of two: 0.57 N 2^-53 S.  So an output is kept if it is that large itself, or if one of the
// largest elements meets a partner that makes the product so; every other one (a weak one: the
// largest elements meet small ones, as a localised or symmetry-adapted C over decaying rows) is
// looked at along its row and column and, with no such product, summed in FP64.  No element is
// less exact than an FP64 sum may be.
#include <cuda_runtime.h>

#include <stdint.h>

#include "../../include/mmdg.h"

int mmdg_internal_fail(int code, const char* msg);

namespace {

constexpr int TS = 64;  // output rows (new index S) per block
constexpr int TMv = 64; // output columns (old flattened pqr) per block
constexpr int TK = 16;  // contracted index s per stage

__global__ void __launch_bounds__(256) k_quarter(const double* __restrict__ in, const double* __restrict__ C,
                                                 double* __restrict__ out, int N, long long M) {
  __shared__ double Cs[TK][TS + 1];    // C[s0 + k, S0 + j]
  __shared__ double Is[TK][TMv + 1];   // in[m0 + j, s0 + k] (transposed)
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int S0 = blockIdx.y * TS;
  const long long m0 = (long long)blockIdx.x * TMv;
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  for (int s0 = 0; s0 < N; s0 += TK) {
    for (int e = threadIdx.x; e < TK * TS; e += 256) {
      const int k = e / TS, j = e - k * TS;
      const int s = s0 + k, S = S0 + j;
      Cs[k][j] = (s < N && S < N) ? C[(long long)s * N + S] : 0.0;
    }
    for (int e = threadIdx.x; e < TK * TMv; e += 256) {
      const int j = e / TK, k = e - j * TK;  // k fastest: coalesced along s
      const int s = s0 + k;
      const long long m = m0 + j;
      Is[k][j] = (s < N && m < M) ? in[m * N + s] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      double cv[4], iv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) cv[a] = Cs[k][ty * 4 + a];
#pragma unroll
      for (int b = 0; b < 4; ++b) iv[b] = Is[k][tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fma(cv[a], iv[b], acc[a][b]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int S = S0 + ty * 4 + a;
    if (S >= N) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const long long m = m0 + tx + 16 * b;
      if (m < M) out[(long long)S * M + m] = acc[a][b];
    }
  }
}


// ------------------------------------------------------------------ tensor-core form
constexpr int kTcThreads = 256;
constexpr int kTcRows = 128;                        // rows m of the tensor per tile (MMA M)
constexpr int kTcCols = 32;                         // new indices S per block (MMA N)
constexpr int kTcDigits = 8;
constexpr int kTcStage = kTcRows * 16 * 2;          // bytes of one digit of a 16-wide k step
constexpr int kTcTmem = kTcDigits * kTcCols;        // accumulator columns
constexpr int kTcRawStride = 17;                    // doubles per row of the raw stage (16 + 1: no bank conflict)
constexpr int kTcQueue = 256;                       // weak outputs looked at together
constexpr int kTcMany = 512;                        // of a tile: from here on they are summed at once
constexpr int kTcWide = 2 * kTcDigits - 1;          // digit slots of C per k octet: seven of zeros, then the digits

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major operand without swizzle: 8 x 16-byte core matrices of 128 contiguous bytes, `lbo`
// bytes apart along k and 128 bytes apart along the rows
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3fff) | (uint64_t)((lbo >> 4) & 0x3fff) << 16 | (uint64_t)(128 >> 4) << 32 |
         (uint64_t)1 << 46;
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(add)
      : "memory");
}
// waits for the barrier's phase; false when it did not come (never expected: then the
// block's outputs become NaN instead of the kernel spinning on)
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t phase) {
  for (int i = 0; i < (1 << 22); ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void tmem_load8(uint32_t addr, uint32_t* v) {
  // (the wait in the same statement: nothing that uses the registers can move before it)
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               "tcgen05.wait::ld.sync.aligned;\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}

// x 2^(1084 - emax) as a fixed-point number (|.| < 2^62, truncated), plus 128 in every byte:
// byte 7 - i minus 128 is then its signed digit i.  emax: the largest exponent field of the
// row (at least 1).
__device__ __forceinline__ uint64_t fixed_digits(double x, int emax) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff, ee = e > 1 ? e : 1;
  const uint64_t m = (b & 0xfffffffffffffULL) | (e ? 1ULL << 52 : 0ULL);
  uint64_t v = (m << 9) >> min(emax - ee, 63);
  if ((int64_t)b < 0) v = 0ULL - v;
  return v + 0x8080808080808080ULL;
}
// digit i of two fixed-point numbers as a pair of BF16 (the first in the low half): the byte
// placed into 2^23's mantissa, 2^23 + 128 subtracted (exact), the upper halves packed
__device__ __forceinline__ uint32_t digit_pair(uint64_t u, uint64_t v, int i) {
  const int byte = 7 - i;
  const uint32_t us = byte >= 4 ? (uint32_t)(u >> 32) : (uint32_t)u, vs = byte >= 4 ? (uint32_t)(v >> 32) : (uint32_t)v;
  const uint32_t sel = 0x7440u | (uint32_t)(byte & 3);
  const float f = __uint_as_float(__byte_perm(us, 0x4B000000u, sel)) - 8388736.0f;
  const float g = __uint_as_float(__byte_perm(vs, 0x4B000000u, sel)) - 8388736.0f;
  return __byte_perm(__float_as_uint(f), __float_as_uint(g), 0x7632u);
}
// eight consecutive k of one row: their digits as one 16-byte core-matrix row per digit
__device__ __forceinline__ void store_digits(const double* x, int emax, unsigned char* at) {
  uint32_t w[kTcDigits][4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uint64_t u = fixed_digits(x[2 * p], emax), v = fixed_digits(x[2 * p + 1], emax);
#pragma unroll
    for (int i = 0; i < kTcDigits; ++i) w[i][p] = digit_pair(u, v, i);
  }
#pragma unroll
  for (int i = 0; i < kTcDigits; ++i)
    *reinterpret_cast<uint4*>(at + i * kTcStage) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// An element's size and place: the upper half of its magnitude with k (below 128) in the lowest
// bits, so that a maximum over a row or column brings its exponent field and where it is
__device__ __forceinline__ unsigned size_at(int hi, int k) { return ((unsigned)hi & 0x7fffff80u) | (unsigned)k; }
__device__ __forceinline__ int field_of(unsigned size) { return (int)(size >> 20); }
__device__ __forceinline__ unsigned at_least_one(unsigned size) { return field_of(size) ? size : size | 1u << 20; }

// the rare case, kept out of line: a result outside the normal doubles
__device__ __noinline__ double scaled(uint64_t mant, int e) { return ldexp((double)mant, e); }

// sum_d acc_d 256^(7-d) 2^(top - 2112) as a double, rounded to nearest, without a branch (eight
// of them interleave); outside the normal doubles `far` is set, and the value is (-1)^neg mant
// 2^e.  `low`: below 2^63 units, 2^(top - 2049).
__device__ __forceinline__ double assemble(const uint32_t (*acc)[8], int col, int top_field, bool& far, bool& low, bool& neg,
                                           uint64_t& mant, int& e) {
  int a[kTcDigits];
#pragma unroll
  for (int d = 0; d < kTcDigits; ++d) a[d] = __float2int_rn(__uint_as_float(acc[d][col]));
  long long hi = (long long)a[0] * (1 << 24) + ((long long)a[1] * (1 << 16) + ((long long)a[2] * (1 << 8) + a[3]));
  const long long lo = (long long)a[4] * (1 << 24) + ((long long)a[5] * (1 << 16) + ((long long)a[6] * (1 << 8) + a[7]));
  hi += lo >> 32;  // value = hi 2^32 + (low 32 bits of lo)
  neg = hi < 0;  // magnitude of the 96-bit two's complement number
  const uint32_t tail = neg ? 0u - (uint32_t)lo : (uint32_t)lo;
  hi = neg ? ~hi + (tail == 0u) : hi;
  low = (hi >> 31) == 0;
  const bool small = hi == 0;
  const uint64_t h = small ? (uint64_t)tail : (uint64_t)hi, rest = small ? 0ULL : (uint64_t)tail << 32;
  const int lead = __clzll((long long)h);  // 64 for zero
  const uint64_t top = (h << (lead & 63)) | ((rest >> 1) >> (63 - (lead & 63)));  // leading one at bit 63
  mant = (top >> 11) + ((top >> 10) & 1);                                         // 2^52 .. 2^53
  e = (small ? 0 : 32) - lead + 11 + top_field - 2112;                            // value = mant 2^e
  const int field = e + 1075;
  far = h != 0 && (field <= 0 || field >= 2046);
  const uint64_t bits = ((uint64_t)(uint32_t)(field - 1) << 52) + mant;
  return __longlong_as_double((long long)(h == 0 ? 0ULL : (bits | (uint64_t)neg << 63)));
}

// columns with an infinity or NaN (all lanes of a warp)
__device__ __forceinline__ unsigned special_columns(const unsigned* s_col) {
  return __ballot_sync(0xffffffffu, field_of(s_col[threadIdx.x & 31]) == 0x7ff);
}

// upper half of the magnitude of C's fixed-point number (k, n), to a unit: below 2^30, 2^26 is
// an eighth of the power of two of the column's largest
__device__ __forceinline__ unsigned upper_half(const uint64_t* Cf, int NT, int k, int n) {
  const unsigned* const at = reinterpret_cast<const unsigned*>(Cf) + 1;
  return (unsigned)abs((int)(at[2 * (((k >> 3) * NT + n) * 8 + (k & 7))] - 0x80808080u));
}

// The first n outputs of the queue (row << 5 | column), eight lanes each: whether two partners
// are large enough for the digits, else the FP64 sum.  (These two stand out of line: inlined,
// their registers cost the loop around them 10 %.)
__device__ __noinline__ void settle(const double* __restrict__ in, const double* __restrict__ C, double* __restrict__ out,
                                    int N, long long M, const unsigned* queue, int n, const uint64_t* Cf, int NT,
                                    const unsigned* s_col) {
  const int sub = threadIdx.x & 7;
  const unsigned special = special_columns(s_col);
  const unsigned mates = 0xffu << (threadIdx.x & 24);
  for (int q = threadIdx.x >> 3; q < n; q += kTcThreads / 8) {
    const unsigned w = queue[q];
    const int c = (int)(w & 31u);
    const double* __restrict__ a = in + (long long)(w >> 5) * N;
    // the row's upper halves, their loads in flight together
    int up[16];
#pragma unroll
    for (int x = 0; x < 16; ++x) up[x] = sub + 8 * x < N ? __ldg(reinterpret_cast<const int*>(a + sub + 8 * x) + 1) : 0;
    int most = 0, er = 1;  // largest field less its partner's leading zeros, the row's largest field
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      if (sub + 8 * x >= N) break;
      const int f = field_of(size_at(up[x], 0));
      most = max(most, f > 0 ? f - __clz((int)upper_half(Cf, NT, 8 * x + sub, c)) : 0);
      er = max(er, f);
    }
    for (int o = 1; o < 8; o <<= 1) {
      most = max(most, __shfl_xor_sync(mates, most, o));
      er = max(er, __shfl_xor_sync(mates, er, o));
    }
    if (!(special >> c & 1) && er < 0x7ff && most >= max(er - 5, 1)) continue;
    double v = 0.0;
    for (int k = sub; k < N; k += 8) v = fma(__ldg(a + k), __ldg(C + (long long)k * N + c), v);
    for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(mates, v, o);
    if (sub == 0) out[(long long)c * M + (w >> 5)] = v;
  }
}

// A tile's `total` outputs marked in `weak`, summed in FP64, neighbours along a row.  All threads.
__device__ __noinline__ void sum_many(const double* __restrict__ rows, const double* __restrict__ C, double* __restrict__ out,
                                      int N, long long M, const unsigned* weak, int* before, int total) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int n[4], end = 0;
#pragma unroll
    for (int x = 0; x < 4; ++x) end += n[x] = __popc(weak[4 * lane + x]);
    int at = end;
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, end, d);
      if (lane >= d) end += t;
    }
    at = end - at;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      before[4 * lane + x] = at;
      at += n[x];
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < total; q += kTcThreads) {
    int lo = 0, hi = kTcRows - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (before[mid] <= q) lo = mid;
      else hi = mid - 1;
    }
    unsigned w = weak[lo];
    for (int x = before[lo]; x < q; ++x) w &= w - 1;
    const int c = __ffs((int)w) - 1;
    const double* __restrict__ a = rows + (long long)lo * N;
    double v = 0.0;
    for (int k = 0; k < N; ++k) v = fma(__ldg(a + k), __ldg(C + (long long)k * N + c), v);
    out[(long long)c * M + lo] = v;
  }
}

// One quarter transform.  Block (x, y): the S tile y (its part of C stays in shared memory as
// 62-bit numbers: as digits it would take twice the room, one block per SM from N = 97 on) of
// the row tiles x, x + gridDim.x, ...  Per 16-wide k step the block stages the raw rows, cuts
// them and C's share into digits and one thread issues the digit products; two blocks per SM
// (256 of the 512 TMEM columns each) overlap one's products with the other's digits.
// Bound by the integer work around the products: of a tile's ~41,000 cycles at N = 76 (two
// blocks per SM) about 6,600 cut the rows' digits, 7,400 put results together, 7,500 find the
// row exponents, 6,000 stage rows, 3,000 cut C's digits and make the products eight accumulators
// wide, 4,000 look for weak outputs and 3,400 settle them (0.8 % of all).
// One product of N = 8 NT columns per row digit, instead of one per digit pair, took issuing
// them from 2,400 to 150 cycles a step.  us per transform of a dense tensor, k_quarter -> this
// (without the look at weak outputs): N = 7 86 -> 47 (34), 13 86 -> 52 (41), 32 537 -> 100 (81),
// 64 6,930 -> 1,240 (1,020), 76 28,980 -> 3,630 (2,980), 100 91,700 -> 14,200 (11,500), 128
// 219,500 -> 30,700 (25,600); N = 76 with C in four blocks 7,040, C = 1 (everything weak but
// the diagonal) 18,400.  FP64 arithmetic alone is 16,000 at N = 76, memory 320.  Weak outputs
// settled tile by tile: 4,070 (one lane each), 4,550 (eight); one of the row's largest elements
// looked at instead of two: 4,000.  C kept as digits: 76 -2 %, 100 +36 %, 128 +48 %.
// Prefetching the next tile into L2 was slower up to N = 76.
__global__ void __launch_bounds__(kTcThreads, 2)
    k_quarter_tc(const double* __restrict__ in, const double* __restrict__ C, double* __restrict__ out, int N,
                 long long M) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_tmem;
  // largest size_at of every row, this tile's and the next one's, and the largest of the other
  // half of its k; the largest of every column
  __shared__ unsigned s_rows[2][kTcRows], s_other[2][kTcRows];
  __shared__ unsigned s_col[kTcCols];
  // outputs that the digits may not hold: this tile's columns of every row, how many before a row
  // and in all (of two tiles in turn), and those kept until they fill the block (row << 5 | column)
  __shared__ unsigned s_weak[kTcRows];
  __shared__ int s_before[kTcRows], s_total[2], s_queued;
  __shared__ unsigned s_queue[kTcQueue + kTcMany];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int steps = (N + 15) / 16, Kp = steps * 16;
  const int S0 = blockIdx.y * kTcCols, cols = min(kTcCols, N - S0), NT = (cols + 15) & ~15;
  unsigned char* const As = sm;                                          // [digit][k octet][row][16 B]
  double* const raw = reinterpret_cast<double*>(sm + kTcDigits * kTcStage);
  unsigned char* const Bs = sm + kTcDigits * kTcStage + sizeof(double) * kTcRawStride * kTcRows;  // [k octet][slot][S][16 B]
  uint64_t* const Cf = reinterpret_cast<uint64_t*>(Bs + 2 * kTcWide * kTcCols * 16);              // [k octet][S][8]
  const uint32_t bar = smem_addr(&s_bar);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)),
                 "r"(kTcTmem)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // ---- C's fixed-point numbers, and the zeros before its digits
  for (int n = warp; n < kTcCols; n += kTcThreads / 32) {
    unsigned top = 0;
    if (n < cols)
      for (int k = lane; k < N; k += 32)
        top = max(top, size_at(__double2hiint(__ldg(C + (long long)k * N + S0 + n)), k));
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) s_col[n] = at_least_one(top);
  }
  if (tid < kTcRows) s_weak[tid] = 0u;
  if (tid < 2) s_total[tid] = 0;
  if (tid == 2) s_queued = 0;
  __syncthreads();
  const uint32_t tmem = s_tmem;
  for (int u = tid; u < NT * (Kp / 8); u += kTcThreads) {
    const int n = u % NT, oct = u / NT;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = oct * 8 + j;
      Cf[u * 8 + j] = fixed_digits(n < cols && k < N ? __ldg(C + (long long)k * N + S0 + n) : 0.0, field_of(s_col[n]));
    }
  }
  for (int u = tid; u < 2 * (kTcDigits - 1) * NT; u += kTcThreads) {
    const int o = u / ((kTcDigits - 1) * NT);
    *reinterpret_cast<uint4*>(Bs + (u + o * kTcDigits * NT) * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  // instruction descriptor: D FP32, A and B BF16, both K-major, N = 8 NT, M = 128
  const uint32_t idesc = 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(kTcDigits * NT >> 3) << 17 | (uint32_t)(kTcRows >> 4) << 24;
  uint32_t phase = 0;
  bool good = true;
  // largest size_at of every row of the tile at m: a warp per 16 rows, their loads in flight
  // together (row by row this took 25,000 of a tile's 54,000 cycles)
  auto row_exponents = [&](long long m, int to) {
    constexpr int R = kTcRows / 8;
    const int rows = (int)min((long long)kTcRows, M - m) - warp * R;
    const int* __restrict__ src = reinterpret_cast<const int*>(in + (m + warp * R) * N) + 1;  // high words
    unsigned top[R];
#pragma unroll
    for (int r = 0; r < R; ++r) top[r] = 0u;
    for (int k = lane; k < N; k += 64) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int* __restrict__ h = src + 2 * (r * N + k);
        const unsigned u = r < rows ? size_at(__ldg(h), k) : 0u;
        const unsigned w = r < rows && k + 32 < N ? size_at(__ldg(h + 64), k + 32) : 0u;
        top[r] = max(top[r], max(u, w));
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned even = __reduce_max_sync(0xffffffffu, lane & 1 ? 0u : top[r]);
      const unsigned odd = __reduce_max_sync(0xffffffffu, lane & 1 ? top[r] : 0u);
      if (lane == 0) {
        s_rows[to][warp * R + r] = at_least_one(max(even, odd));
        s_other[to][warp * R + r] = min(even, odd);
      }
    }
  };
  const long long mstep = (long long)gridDim.x * kTcRows;
  int buf = 0;
  if ((long long)blockIdx.x * kTcRows < M) row_exponents((long long)blockIdx.x * kTcRows, 0);
  const int lr = tid >> 4, lk = tid & 15;  // raw staging: row lr + 16 x, k lk
  const int row = tid & (kTcRows - 1), oct = tid >> 7;
  for (long long m0 = (long long)blockIdx.x * kTcRows; m0 < M; m0 += mstep, buf ^= 1) {
    const int rows = (int)min((long long)kTcRows, M - m0);
    const double* __restrict__ src = in + m0 * N;
    double nxt[8];
#pragma unroll
    for (int x = 0; x < 8; ++x)
      nxt[x] = lr + 16 * x < rows && lk < N ? __ldg(src + (long long)(lr + 16 * x) * N + lk) : 0.0;
    const unsigned* const s_row = s_rows[buf];
    for (int st = 0; st < steps; ++st) {
#pragma unroll
      for (int x = 0; x < 8; ++x) raw[(lr + 16 * x) * kTcRawStride + lk] = nxt[x];
      if (st + 1 < steps) {
        const int k = (st + 1) * 16 + lk;
#pragma unroll
        for (int x = 0; x < 8; ++x)
          nxt[x] = lr + 16 * x < rows && k < N ? __ldg(src + (long long)(lr + 16 * x) * N + k) : 0.0;
      }
      __syncthreads();  // raw rows and exponents are in place
      if (st > 0) {     // the products of the previous step have read the digits
        good = good && wait_phase(bar, phase);
        phase ^= 1;
      }
      {
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = raw[row * kTcRawStride + oct * 8 + j];
        store_digits(x, field_of(s_row[row]), As + (oct * kTcRows + row) * 16);
        // C's digits of the step: a pair of k per thread
        for (int u = tid; u < 8 * NT; u += kTcThreads) {
          const ulonglong2 f = reinterpret_cast<const ulonglong2*>(Cf + (size_t)st * 16 * NT)[u];
          const int o = u / (4 * NT);
          unsigned char* const at = Bs + (o * kTcWide + kTcDigits - 1) * NT * 16 + (u - o * 4 * NT) * 4;
#pragma unroll
          for (int i = 0; i < kTcDigits; ++i) *reinterpret_cast<uint32_t*>(at + i * NT * 16) = digit_pair(f.x, f.y, i);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        if (st == 0) s_total[buf ^ 1] = 0;  // (read before this tile's first barrier)
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // the digits of C lie one after another along N, the accumulators one after another in
        // TMEM: digit i of the rows meets digits 0 .. 7 - i of C, added into accumulators i .. 7.
        // Every product spans all eight accumulators (its first i meet zeros): the ISA keeps
        // tcgen05.mma of one thread in order for the same accumulator and shape only, and these
        // all add into the same columns.
        const uint32_t a0 = smem_addr(As), b0 = smem_addr(Bs);
#pragma unroll
        for (int i = 0; i < kTcDigits; ++i)
          mma_bf16(tmem, operand(a0 + i * kTcStage, kTcRows * 16),
                   operand(b0 + (uint32_t)((kTcDigits - 1 - i) * NT * 16), (uint32_t)(kTcWide * NT * 16)), idesc,
                   st > 0 || i > 0 ? 1u : 0u);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                     : "memory");
      }
    }
    if (m0 + mstep < M) row_exponents(m0 + mstep, buf ^ 1);  // beside the last products
    good = good && wait_phase(bar, phase);
    phase ^= 1;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    // ---- outputs: lane = row of the warp's quarter, the two warps of a quarter share the columns
    const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * (NT / 2);
    const unsigned big = s_row[r], big2 = s_other[buf][r];
    const int er = field_of(big);
    const unsigned special = special_columns(s_col);
    const int widest = __reduce_max_sync(0xffffffffu, field_of(s_col[lane])), gap = er - field_of(big2);
    const unsigned need = big >= 1u << 20 ? 1u << 26 : ~0u, need2 = big2 >= 1u << 20 && gap <= 3 ? 1u << (26 + gap) : ~0u;
    unsigned mine = 0;
    for (int c = c0; c < c0 + NT / 2; c += 8) {
      uint32_t acc[kTcDigits][8];
#pragma unroll
      for (int d = 0; d < kTcDigits; ++d)
        tmem_load8(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(d * NT + c), acc[d]);
      double v[8];
      unsigned out_of = 0, weak = 0;  // columns outside the normal doubles; the digits may not hold them
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        bool far, low, neg;
        uint64_t mant;
        int e;
        v[x] = assemble(acc, x, er + field_of(s_col[c + x]), far, low, neg, mant, e);
        out_of |= (far ? 1u : 0u) << x;
        weak |= (low ? 1u : 0u) << x;
      }
      const int left = cols - c;
      const unsigned real = r < rows && left > 0 ? (left >= 8 ? 0xffu : (1u << left) - 1u) : 0u;
      // (all er + ec up to 1027: what is left out is below half a unit of the subnormals per k)
      weak &= er + widest <= 1027 ? 0u : real;
      // one of the row's two largest elements meets a partner that makes the product large enough:
      // nine in ten end here
      out_of &= real;
      for (unsigned todo = weak; todo; todo &= todo - 1) {
        const int x = __ffs((int)todo) - 1;
        if (upper_half(Cf, NT, big & 127, c + x) >= need || upper_half(Cf, NT, big2 & 127, c + x) >= need2) weak &= ~(1u << x);
      }
      weak |= er == 0x7ff ? real : special >> c & real;
      if (out_of) {
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          if (!(out_of >> x & 1)) continue;
          bool far, low, neg;
          uint64_t mant;
          int e;
          assemble(acc, x, er + field_of(s_col[c + x]), far, low, neg, mant, e);
          v[x] = neg ? -scaled(mant, e) : scaled(mant, e);
        }
      }
      reinterpret_cast<unsigned char*>(s_weak + r)[c >> 3] = (unsigned char)weak;
      mine |= weak << (c - c0);
#pragma unroll
      for (int x = 0; x < 8; ++x)
        if (real >> x & 1)
          out[(long long)(S0 + c + x) * M + m0 + r] = good ? v[x] : __longlong_as_double(0x7ff8000000000000LL);
    }
    const int some = __reduce_add_sync(0xffffffffu, __popc(mine)), queued = s_queued;
    if (lane == 0 && some) atomicAdd(&s_total[buf], some);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();  // accumulators, exponents and raw rows are free again
    const int total = s_total[buf];
    if (total == 0) continue;
    // ---- the weak outputs: a few wait for those of the next tiles, as many as fill the block
    // (eight warps waiting for one cost 40 % at N = 76); many are summed at once, without a look at
    // their partners, neighbours along a row
    if (total <= kTcMany) {
      if (queued >= kTcQueue) {
        settle(in, C + S0, out + (long long)S0 * M, N, M, s_queue, queued, Cf, NT, s_col);
        __syncthreads();
        if (tid == 0) s_queued = 0;
        __syncthreads();
      }
      if (mine) {
        int at = atomicAdd(&s_queued, __popc(mine));
        for (unsigned todo = mine; todo; todo &= todo - 1)
          s_queue[at++] = (unsigned)(m0 + r) << 5 | (unsigned)(c0 + __ffs((int)todo) - 1);
      }
      continue;
    }
    sum_many(src, C + S0, out + (long long)S0 * M + m0, N, M, s_weak, s_before, total);
  }
  __syncthreads();
  settle(in, C + S0, out + (long long)S0 * M, N, M, s_queue, s_queued, Cf, NT, s_col);
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTcTmem));
}

// at least a third of an SM's shared memory, so that two blocks (2 x 256 TMEM columns), never
// three, share an SM
inline size_t tc_smem(int N) {
  const int Kp = (N + 15) / 16 * 16, NT = N < kTcCols ? (N + 15) / 16 * 16 : kTcCols;
  const size_t need = (size_t)kTcDigits * kTcStage + sizeof(double) * kTcRawStride * kTcRows + 2 * kTcWide * kTcCols * 16 +
                      sizeof(uint64_t) * Kp * NT;
  return need < 80 * 1024 ? 80 * 1024 : need;
}

}  // namespace

// largest N of the tensor-core form: its sums are exact up to here
static const long long kTcMax = 128;

extern "C" int mmdg_ao2mo(long long N, const double* C, const double* eri_in, double* eri_out, double* work,
                          void* stream) {
  if (N <= 0 || !C || !eri_in || !eri_out || !work)
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_ao2mo: bad argument");
  if (N > 1290) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_ao2mo: N^3 exceeds the grid (N <= 1290)");
  if (eri_out == eri_in || work == eri_in || work == eri_out)
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_ao2mo: eri_in, eri_out and work must be distinct");
  cudaStream_t st = (cudaStream_t)stream;
  const long long M = N * N * N;
  const dim3 grid((unsigned)((M + TMv - 1) / TMv), (unsigned)((N + TS - 1) / TS));
  const double* src[4] = {eri_in, work, eri_out, work};
  double* dst[4] = {work, eri_out, work, eri_out};
  const bool tc = N <= kTcMax;
  const size_t smem = tc ? tc_smem((int)N) : 0;
  dim3 tgrid;
  if (tc) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // (the kernel's limit belongs to the device, not to the call: always that of the largest N,
    // so that no thread lowers it under another's launch)
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_quarter_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_smem((int)kTcMax));
    if (e != cudaSuccess) return mmdg_internal_fail(MMDG_E_CUDA, cudaGetErrorString(e));
    const long long tiles = (M + kTcRows - 1) / kTcRows;
    tgrid.y = (unsigned)((N + kTcCols - 1) / kTcCols);
    const long long want = 2LL * sms / tgrid.y;
    tgrid.x = (unsigned)(want < 1 ? 1 : (want < tiles ? want : tiles));
  }
  for (int q = 0; q < 4; ++q) {
    if (tc) k_quarter_tc<<<tgrid, kTcThreads, smem, st>>>(src[q], C, dst[q], (int)N, M);
    else k_quarter<<<grid, 256, 0, st>>>(src[q], C, dst[q], (int)N, M);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return mmdg_internal_fail(MMDG_E_CUDA, cudaGetErrorString(e));
  }
  return MMDG_OK;
}
