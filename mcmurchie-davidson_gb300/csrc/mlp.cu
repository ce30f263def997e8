// mlp.cu -- kernels of the learned initial-guess network: a 3-layer MLP with BF16
// weights and FP32 accumulation, trained and served on the GPU.
//
// The network maps atom-pair features to density-matrix blocks (the SCF's initial
// guess; the reference starts from P = 0, mmd/scf.py:15,23-24).  Sizes are tiny
// (~100 k parameters, ~1 M training pairs), so the GEMMs are shared-memory tiled
// FP32 FMA kernels reading BF16 weights (activations and sums stay FP32, as the tensor
// cores' FP32 sums truncate), with the layers' elementwise work in their epilogues.
//
//   gemm:   C[M,N] (+)= op(A)[M,K] op(B)[K,N], A/B in FP32 or BF16, C in FP32
//   act:    Y = silu(Z + b) (stores Z + b for the backward), or identity
//   loss:   dY = 2 (Y - T) * mask / count, and the loss value
//   adam:   FP32 master weights, BF16 copies refreshed in the same pass
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/mmdg.h"
#include "pairs.cuh"

namespace {

constexpr int TM = 128, TN = 64, TK = 16;
constexpr int TT = TM * TN / 32;  // threads of a GEMM block, 8 x 4 outputs each

template <typename T>
__device__ __forceinline__ float ld(const T* p, long long i);
template <>
__device__ __forceinline__ float ld<float>(const float* p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(p[i]);
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);  // (a BF16 is the upper half of a float)
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                     __uint_as_float(u.y & 0xffff0000u));
}

// What a GEMM does with its sums.
enum Epilogue {
  kStore,   // C (+)= sums (atomics when K is split over blockIdx.z)
  kLinear,  // C = Z = sums + bias (row broadcast), Y = silu(Z) or Z
  kActGrad  // C = sums * silu'(Zp), db[n] += its column sums (db zeroed by the launcher)
};
struct EpilogueArgs {
  const float* bias = nullptr;
  float* Y = nullptr;
  const float* Zp = nullptr;
  float* db = nullptr;
  int silu = 0;
};

// two FP32 FMAs in one instruction, each rounded as an FMA of its own
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long both(float x) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
  return d;
}
__device__ __forceinline__ float2 halves(unsigned long long x) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(x));
  return d;
}

__device__ __forceinline__ float silu_of(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = 1.f / (1.f + expf(-z));
  return s * (1.f + z * (1.f - s));
}

// op(A) op(B);  op(A): ta ? A^T (A stored K x M) : A (M x K), likewise B.  128 x 64 tiles, 8 x 4
// outputs per thread read as float4 from shared memory (three 16-byte loads per 32 FMAs, issued
// as 16 packed pairs of rows), the next K stage in registers meanwhile.  VEC: rows of a
// multiple of four elements at aligned addresses are fetched and written four at a time (78
// registers against 128).  At the network's sizes it waits on latencies (ncu, 256 x 256 layer of
// 8192 rows: FMA pipe 48 % busy, 3.3 warps per scheduler, stalls on the FMA chain, shared loads
// and the fetch about equal) and on the last wave: 256 tiles on 152 SMs.  The eight GEMMs of a
// training step of 8192 rows: 840 us with 64 x 64 tiles, 4 x 4 outputs and scalar shared loads,
// 300 with these tiles, 290 with packed FMAs, 265 with fours (a 256 x 256 layer 45 -> 41 -> 37 us,
// 29 TFLOP/s).  No better per step (320 us): 8 x 8 outputs per thread 332, two stages ahead in
// registers 332, 64 x 64 tiles 334, both 429, K stages of 8 or 32 (before the fours) 393 / 439.
template <typename TA, typename TB, int EPI, bool VEC>
__global__ void __launch_bounds__(TT) k_gemm(int M, int N, int K, const TA* __restrict__ A, int lda, int ta,
                                              const TB* __restrict__ B, int ldb, int tb, float* __restrict__ C, int ldc,
                                              float beta, EpilogueArgs ep) {
  __shared__ __align__(16) float As[2][TK][TM + 4];
  __shared__ __align__(16) float Bs[2][TK][TN + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  // split K over blockIdx.z (the weight gradients: M x N small, K = batch rows)
  const int kspan = ((K + gridDim.z - 1) / gridDim.z + TK - 1) / TK * TK;
  const int kbeg = blockIdx.z * kspan, kend = min(K, kbeg + kspan);
  // element x of this thread's share of a stage: consecutive threads along the stored row
  auto a_at = [&](int x, int& kk, int& mm) {
    const int e = tid + x * TT;
    kk = ta ? e / TM : e % TK;
    mm = ta ? e % TM : e / TK;
  };
  auto b_at = [&](int x, int& kk, int& nn) {
    const int e = tid + x * TT;
    kk = tb ? e % TK : e / TN;
    nn = tb ? e / TK : e % TN;
  };
  float ra[TK * TM / TT], rb[TK * TN / TT];
  auto fetch = [&](int k0) {
    if (VEC) {  // four neighbours along the stored row at a time
#pragma unroll
      for (int x = 0; x < TK * TM / TT / 4; ++x) {
        const int e = tid + x * TT;
        const int m = m0 + (ta ? e % (TM / 4) * 4 : e / (TK / 4)), k = k0 + (ta ? e / (TM / 4) : e % (TK / 4) * 4);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M && k < kend) v = ld4(ta ? A + (long long)k * lda + m : A + (long long)m * lda + k);
        ra[4 * x] = v.x, ra[4 * x + 1] = v.y, ra[4 * x + 2] = v.z, ra[4 * x + 3] = v.w;
      }
#pragma unroll
      for (int x = 0; x < TK * TN / TT / 4; ++x) {
        const int e = tid + x * TT;
        const int n = n0 + (tb ? e / (TK / 4) : e % (TN / 4) * 4), k = k0 + (tb ? e % (TK / 4) * 4 : e / (TN / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < N && k < kend) v = ld4(tb ? B + (long long)n * ldb + k : B + (long long)k * ldb + n);
        rb[4 * x] = v.x, rb[4 * x + 1] = v.y, rb[4 * x + 2] = v.z, rb[4 * x + 3] = v.w;
      }
      return;
    }
#pragma unroll
    for (int x = 0; x < TK * TM / TT; ++x) {
      int kk, mm;
      a_at(x, kk, mm);
      const int m = m0 + mm, k = k0 + kk;
      ra[x] = m < M && k < kend ? (ta ? ld(A, (long long)k * lda + m) : ld(A, (long long)m * lda + k)) : 0.f;
    }
#pragma unroll
    for (int x = 0; x < TK * TN / TT; ++x) {
      int kk, nn;
      b_at(x, kk, nn);
      const int n = n0 + nn, k = k0 + kk;
      rb[x] = n < N && k < kend ? (tb ? ld(B, (long long)n * ldb + k) : ld(B, (long long)k * ldb + n)) : 0.f;
    }
  };
  auto stage = [&](int s) {
    if (VEC) {
#pragma unroll
      for (int x = 0; x < TK * TM / TT / 4; ++x) {
        const int e = tid + x * TT;
        if (ta) {
          *reinterpret_cast<float4*>(&As[s][e / (TM / 4)][e % (TM / 4) * 4]) =
              make_float4(ra[4 * x], ra[4 * x + 1], ra[4 * x + 2], ra[4 * x + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) As[s][e % (TK / 4) * 4 + i][e / (TK / 4)] = ra[4 * x + i];
        }
      }
#pragma unroll
      for (int x = 0; x < TK * TN / TT / 4; ++x) {
        const int e = tid + x * TT;
        if (!tb) {
          *reinterpret_cast<float4*>(&Bs[s][e / (TN / 4)][e % (TN / 4) * 4]) =
              make_float4(rb[4 * x], rb[4 * x + 1], rb[4 * x + 2], rb[4 * x + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) Bs[s][e % (TK / 4) * 4 + i][e / (TK / 4)] = rb[4 * x + i];
        }
      }
      return;
    }
#pragma unroll
    for (int x = 0; x < TK * TM / TT; ++x) {
      int kk, mm;
      a_at(x, kk, mm);
      As[s][kk][mm] = ra[x];
    }
#pragma unroll
    for (int x = 0; x < TK * TN / TT; ++x) {
      int kk, nn;
      b_at(x, kk, nn);
      Bs[s][kk][nn] = rb[x];
    }
  };
  unsigned long long acc2[4][4] = {};  // two rows each
  if (kbeg < kend) {
    fetch(kbeg);
    stage(0);
  }
  __syncthreads();
  int s = 0;
  for (int k0 = kbeg; k0 < kend; k0 += TK, s ^= 1) {
    const bool more = k0 + TK < kend;
    if (more) fetch(k0 + TK);
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(&As[s][kk][ty * 4]);
      const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(&As[s][kk][TM / 2 + ty * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&Bs[s][kk][tx * 4]);
      const unsigned long long a[4] = {a0.x, a0.y, a1.x, a1.y}, b[4] = {both(b0.x), both(b0.y), both(b0.z), both(b0.w)};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc2[i][j] = fma2(a[i], b[j], acc2[i][j]);
    }
    if (more) stage(s ^ 1);
    __syncthreads();
  }
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = halves(acc2[i][j]);
      acc[2 * i][j] = v.x;
      acc[2 * i + 1][j] = v.y;
    }
  float col[4] = {0.f, 0.f, 0.f, 0.f};
  const int n = n0 + tx * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + (i < 4 ? 0 : TM / 2) + ty * 4 + (i & 3);
    if (m >= M || n >= N) continue;
    const long long at = (long long)m * ldc + n;
    if (VEC && (EPI != kStore || (gridDim.z == 1 && beta == 0.f))) {  // N a multiple of 4
      float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      if (EPI == kLinear) {
        const float4 q = ld4(ep.bias + n);
        v = make_float4(v.x + q.x, v.y + q.y, v.z + q.z, v.w + q.w);
        *reinterpret_cast<float4*>(ep.Y + at) =
            ep.silu ? make_float4(silu_of(v.x), silu_of(v.y), silu_of(v.z), silu_of(v.w)) : v;
      } else if (EPI == kActGrad) {
        if (ep.silu) {
          const float4 q = ld4(ep.Zp + at);
          v = make_float4(v.x * silu_grad(q.x), v.y * silu_grad(q.y), v.z * silu_grad(q.z), v.w * silu_grad(q.w));
        }
        col[0] += v.x, col[1] += v.y, col[2] += v.z, col[3] += v.w;
      }
      *reinterpret_cast<float4*>(C + at) = v;
      continue;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (n + j >= N) continue;
      if (EPI == kLinear) {
        const float z = acc[i][j] + __ldg(ep.bias + n + j);
        C[at + j] = z;
        ep.Y[at + j] = ep.silu ? silu_of(z) : z;
      } else if (EPI == kActGrad) {
        const float d = ep.silu ? acc[i][j] * silu_grad(__ldg(ep.Zp + at + j)) : acc[i][j];
        C[at + j] = d;
        col[j] += d;
      } else if (gridDim.z > 1) {
        atomicAdd(C + at + j, acc[i][j]);  // C zeroed by the launcher
      } else {
        C[at + j] = beta != 0.f ? fmaf(beta, C[at + j], acc[i][j]) : acc[i][j];
      }
    }
  }
  if (EPI == kActGrad) {
    float* part = &As[0][0][0];  // [warp][column]: the K loop ended with a barrier
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      col[j] += __shfl_xor_sync(0xffffffffu, col[j], 16);
      if ((tid & 16) == 0) part[(tid >> 5) * TN + tx * 4 + j] = col[j];
    }
    __syncthreads();
    if (tid < TN && n0 + tid < N) {
      float v = 0.f;
      for (int w = 0; w < TT / 32; ++w) v += part[w * TN + tid];
      atomicAdd(ep.db + n0 + tid, v);
    }
  }
}

// Z = X + b (row broadcast), Y = silu(Z) (or Y = Z); Z kept for the backward
__global__ void k_bias_act(float* Z, float* Y, const float* b, long long rows, int cols, int silu) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  const float z = Z[i] + b[i % cols];
  Z[i] = z;
  Y[i] = silu ? silu_of(z) : z;
}

// dZ = dY * silu'(Z)
__global__ void k_act_grad(const float* Z, const float* dY, float* dZ, long long n, int silu) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (!silu) {
    dZ[i] = dY[i];
    return;
  }
  dZ[i] = dY[i] * silu_grad(Z[i]);
}

// column sums: db[c] = sum_r dZ[r, c] (32 columns x 256 rows per block, FP32 atomics; db
// zeroed first).  One thread per column over 1024 rows: 60 us per layer of 8192 rows, 16
// blocks; now 4
constexpr int kSumRows = 256;
__global__ void __launch_bounds__(256) k_colsum(const float* __restrict__ dZ, float* __restrict__ db, long long rows,
                                                int cols) {
  __shared__ float part[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c = blockIdx.x * 32 + x;
  const long long r0 = (long long)blockIdx.y * kSumRows, r1 = min(rows, r0 + kSumRows);
  float s = 0.f;
  if (c < cols)
    for (long long r = r0 + y; r < r1; r += 8) s += dZ[r * cols + c];
  part[y][x] = s;
  __syncthreads();
  if (y == 0 && c < cols) {
    for (int w = 1; w < 8; ++w) s += part[w][x];
    atomicAdd(db + c, s);
  }
}

// sum of the mask (a double: exact for 0/1 masks), for k_mse
__global__ void __launch_bounds__(256) k_mask_sum(const float* __restrict__ mask, double* __restrict__ count, long long n) {
  __shared__ double part[8];
  double s = 0.0;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) s += (double)mask[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) s += part[w];
    atomicAdd(count, s);
  }
}

// count non-null: 1/count is taken from the device (the mask's sum, at least 1), else inv_count.
// One FP64 atomic per block of the grid-stride loop (one per warp of a thread per element
// took 88 us for 8192 x 225, all on one address).
__global__ void __launch_bounds__(256) k_mse(const float* __restrict__ Y, const float* __restrict__ T,
                                             const float* __restrict__ mask, float* __restrict__ dY,
                                             double* __restrict__ loss, long long n, float inv_count,
                                             const double* __restrict__ count) {
  __shared__ double part[8];
  if (count) inv_count = (float)(1.0 / fmax((double)(float)*count, 1.0));
  // 32 neighbours are summed in FP32, the rest in FP64: the loss's rounding does not depend on
  // the grid
  double l = 0.0;
  for (long long w = blockIdx.x * 256LL + (threadIdx.x & ~31); w < n; w += gridDim.x * 256LL) {
    const long long i = w + (threadIdx.x & 31);
    float q = 0.f;
    if (i < n) {
      const float d = (Y[i] - T[i]) * mask[i];
      dY[i] = 2.f * d * inv_count;
      q = d * d * inv_count;
    }
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    l += (double)q;
  }
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) l += part[w];
    atomicAdd(loss, l);
  }
}

// one Adam step of up to kAdamMax tensors (blockIdx.y)
constexpr int kAdamMax = 8;
struct AdamTensors {
  float* w[kAdamMax];
  __nv_bfloat16* wb[kAdamMax];
  const float* g[kAdamMax];
  float* m[kAdamMax];
  float* v[kAdamMax];
  long long n[kAdamMax];
};
__global__ void k_adam(AdamTensors t, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int y = blockIdx.y;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= t.n[y]) return;
  const float gi = t.g[y][i];
  const float mi = b1 * t.m[y][i] + (1.f - b1) * gi;
  const float vi = b2 * t.v[y][i] + (1.f - b2) * gi * gi;
  t.m[y][i] = mi;
  t.v[y][i] = vi;
  const float wi = t.w[y][i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  t.w[y][i] = wi;
  if (t.wb[y]) t.wb[y][i] = __float2bfloat16(wi);
}

__global__ void k_to_bf16(const float* w, __nv_bfloat16* wb, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) wb[i] = __float2bfloat16(w[i]);
}

unsigned nb(long long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

int launch_fail(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return MMDG_OK;
  return mmdg_internal_fail(MMDG_E_CUDA, what);
}

}  // namespace

// whether every row of an operand can be read or written four elements at a time (else one by
// one: 41 us against 37 for the layer above, whose sums are the same in the same order)
template <typename T>
static bool fours(const T* p, int ld, int inner) {
  return p == nullptr || (ld % 4 == 0 && inner % 4 == 0 && reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T)) == 0);
}
template <typename TA, typename TB, int EPI>
static void gemm(dim3 grid, cudaStream_t st, int M, int N, int K, const TA* A, int lda, int ta, const TB* B, int ldb,
                 int tb, float* C, int ldc, float beta, const EpilogueArgs& ep) {
  if (fours(A, lda, ta ? M : K) && fours(B, ldb, tb ? K : N) && fours(C, ldc, N) && fours(ep.bias, 4, N) &&
      fours(ep.Y, ldc, N) && fours(ep.Zp, ldc, N))
    k_gemm<TA, TB, EPI, true><<<grid, TT, 0, st>>>(M, N, K, A, lda, ta, B, ldb, tb, C, ldc, beta, ep);
  else
    k_gemm<TA, TB, EPI, false><<<grid, TT, 0, st>>>(M, N, K, A, lda, ta, B, ldb, tb, C, ldc, beta, ep);
}

static const long long kFill = 304;  // blocks that fill the GPU: two per SM

// C = op(A) op(B) (+ beta C): a_bf16 / b_bf16 select BF16 operands (weights)
extern "C" int mmdg_mlp_gemm(int M, int N, int K, const void* A, int lda, int ta, int a_bf16, const void* B, int ldb,
                             int tb, int b_bf16, float* C, int ldc, float beta, void* stream) {
  if (M < 0 || N < 0 || K < 0 || !A || !B || !C) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_gemm: bad argument");
  if (!M || !N) return MMDG_OK;
  dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
  cudaStream_t st = (cudaStream_t)stream;
  // few output tiles and a long K (weight gradients over a batch): split K over
  // enough blocks to fill the GPU, partial tiles added with atomics into a zeroed C
  const long long tiles = (long long)grid.x * grid.y;
  if (beta == 0.f && tiles < 152 && K >= 256) {
    const int split = (int)std::min<long long>((K + 127) / 128, (kFill + tiles - 1) / tiles);
    if (split > 1) {
      grid.z = split;
      // the N columns alone: what lies between them and ldc is the caller's
      if (cudaMemset2DAsync(C, sizeof(float) * std::max(ldc, N), 0, sizeof(float) * N, M, st) != cudaSuccess)
        return mmdg_internal_fail(MMDG_E_CUDA, "mmdg_mlp_gemm: memset");
    }
  }
  const EpilogueArgs ep;
  if (a_bf16 && !b_bf16)
    gemm<__nv_bfloat16, float, kStore>(grid, st, M, N, K, (const __nv_bfloat16*)A, lda, ta, (const float*)B, ldb, tb, C,
                                       ldc, beta, ep);
  else if (!a_bf16 && b_bf16)
    gemm<float, __nv_bfloat16, kStore>(grid, st, M, N, K, (const float*)A, lda, ta, (const __nv_bfloat16*)B, ldb, tb, C,
                                       ldc, beta, ep);
  else if (!a_bf16 && !b_bf16)
    gemm<float, float, kStore>(grid, st, M, N, K, (const float*)A, lda, ta, (const float*)B, ldb, tb, C, ldc, beta, ep);
  else
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_gemm: at most one BF16 operand");
  return launch_fail("mmdg_mlp_gemm: launch");
}

// Z = X W^T + b, Y = silu(Z) or Z: X (rows x in), W BF16 (out x in)
extern "C" int mmdg_mlp_linear(long long rows, int out, int in, const float* X, const void* W, const float* b, float* Z,
                               float* Y, int silu, void* stream) {
  if (!X || !W || !b || !Z || !Y || rows < 0 || rows > 0x7fffffffLL || out <= 0 || in <= 0)
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_linear: bad argument");
  if (!rows) return MMDG_OK;
  EpilogueArgs ep;
  ep.bias = b;
  ep.Y = Y;
  ep.silu = silu;
  const dim3 grid((out + TN - 1) / TN, (unsigned)((rows + TM - 1) / TM));
  gemm<float, __nv_bfloat16, kLinear>(grid, (cudaStream_t)stream, (int)rows, out, in, X, in, 0, (const __nv_bfloat16*)W,
                                      in, 1, Z, out, 0.f, ep);
  return launch_fail("mmdg_mlp_linear: launch");
}

// The step from one layer's dZ (rows x out) to the layer before: dZp = (dZ W) silu'(Zp) (or dZ W),
// db = column sums of dZp; W BF16 (out x in), Zp, dZp (rows x in)
extern "C" int mmdg_mlp_back(long long rows, int out, int in, const float* dZ, const void* W, const float* Zp, float* dZp,
                             float* db, int silu, void* stream) {
  if (!dZ || !W || !Zp || !dZp || !db || rows < 0 || rows > 0x7fffffffLL || out <= 0 || in <= 0)
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_back: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(db, 0, sizeof(float) * in, st) != cudaSuccess)
    return mmdg_internal_fail(MMDG_E_CUDA, "mmdg_mlp_back: memset");
  if (!rows) return MMDG_OK;
  EpilogueArgs ep;
  ep.Zp = Zp;
  ep.db = db;
  ep.silu = silu;
  const dim3 grid((in + TN - 1) / TN, (unsigned)((rows + TM - 1) / TM));
  gemm<float, __nv_bfloat16, kActGrad>(grid, st, (int)rows, in, out, dZ, out, 0, (const __nv_bfloat16*)W, in, 0, dZp, in,
                                       0.f, ep);
  return launch_fail("mmdg_mlp_back: launch");
}

extern "C" int mmdg_mlp_bias_act(float* Z, float* Y, const float* b, long long rows, int cols, int silu, void* stream) {
  if (!Z || !Y || !b || rows < 0 || cols <= 0) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_bias_act: bad argument");
  if (!rows) return MMDG_OK;
  k_bias_act<<<nb(rows * cols), 256, 0, (cudaStream_t)stream>>>(Z, Y, b, rows, cols, silu);
  return launch_fail("mmdg_mlp_bias_act: launch");
}

extern "C" int mmdg_mlp_act_grad(const float* Z, const float* dY, float* dZ, long long n, int silu, void* stream) {
  if (!Z || !dY || !dZ || n < 0) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_act_grad: bad argument");
  if (!n) return MMDG_OK;
  k_act_grad<<<nb(n), 256, 0, (cudaStream_t)stream>>>(Z, dY, dZ, n, silu);
  return launch_fail("mmdg_mlp_act_grad: launch");
}

extern "C" int mmdg_mlp_colsum(const float* dZ, float* db, long long rows, int cols, void* stream) {
  if (!dZ || !db || rows < 0 || cols <= 0) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_colsum: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(db, 0, sizeof(float) * cols, st) != cudaSuccess)
    return mmdg_internal_fail(MMDG_E_CUDA, "mmdg_mlp_colsum: memset");
  if (!rows) return MMDG_OK;
  // (long batches in several launches: at most 65535 blocks along the rows)
  const long long step = 65535LL * kSumRows;
  for (long long r = 0; r < rows; r += step) {
    const long long part = std::min(step, rows - r);
    const dim3 grid(nb(cols, 32), (unsigned)((part + kSumRows - 1) / kSumRows));
    k_colsum<<<grid, 256, 0, st>>>(dZ + r * cols, db, part, cols);
  }
  return launch_fail("mmdg_mlp_colsum: launch");
}

extern "C" int mmdg_mlp_mse(const float* Y, const float* T, const float* mask, float* dY, double* loss, long long n,
                            float inv_count, void* stream) {
  if (!Y || !T || !mask || !dY || !loss || n < 0) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_mse: bad argument");
  if (!n) return MMDG_OK;
  k_mse<<<std::min(nb(n), 608u), 256, 0, (cudaStream_t)stream>>>(Y, T, mask, dY, loss, n, inv_count, nullptr);
  return launch_fail("mmdg_mlp_mse: launch");
}

// mmdg_mlp_mse with count = max(sum of the mask, 1) taken on the device (count: a device double)
extern "C" int mmdg_mlp_mse_masked(const float* Y, const float* T, const float* mask, float* dY, double* loss,
                                   double* count, long long n, void* stream) {
  if (!Y || !T || !mask || !dY || !loss || !count || n < 0)
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_mse_masked: bad argument");
  if (!n) return MMDG_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(count, 0, sizeof(double), st) != cudaSuccess)
    return mmdg_internal_fail(MMDG_E_CUDA, "mmdg_mlp_mse_masked: memset");
  const unsigned blocks = std::min(nb(n), 608u);
  k_mask_sum<<<blocks, 256, 0, st>>>(mask, count, n);
  k_mse<<<blocks, 256, 0, st>>>(Y, T, mask, dY, loss, n, 0.f, count);
  return launch_fail("mmdg_mlp_mse_masked: launch");
}

extern "C" int mmdg_mlp_adam_many(int count, float* const* w, void* const* w_bf16, const float* const* g,
                                  float* const* m, float* const* v, const long long* n, float lr, float b1, float b2,
                                  float eps, int step, void* stream) {
  if (count < 0 || (count && (!w || !g || !m || !v || !n)) || step < 1)
    return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_adam: bad argument");
  const float c1 = 1.f / (1.f - powf(b1, (float)step)), c2 = 1.f / (1.f - powf(b2, (float)step));
  for (int first = 0; first < count; first += kAdamMax) {
    const int k = std::min(count - first, kAdamMax);
    AdamTensors t;
    long long most = 0;
    for (int x = 0; x < k; ++x) {
      const int y = first + x;
      if (!w[y] || !g[y] || !m[y] || !v[y] || n[y] < 0) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_adam: bad argument");
      t.w[x] = w[y];
      t.wb[x] = w_bf16 ? (__nv_bfloat16*)w_bf16[y] : nullptr;
      t.g[x] = g[y];
      t.m[x] = m[y];
      t.v[x] = v[y];
      t.n[x] = n[y];
      most = std::max(most, n[y]);
    }
    if (most) k_adam<<<dim3(nb(most), k), 256, 0, (cudaStream_t)stream>>>(t, lr, b1, b2, eps, c1, c2);
  }
  return launch_fail("mmdg_mlp_adam: launch");
}

extern "C" int mmdg_mlp_adam(float* w, void* w_bf16, const float* g, float* m, float* v, long long n, float lr,
                             float b1, float b2, float eps, int step, void* stream) {
  return mmdg_mlp_adam_many(1, &w, &w_bf16, &g, &m, &v, &n, lr, b1, b2, eps, step, stream);
}

extern "C" int mmdg_mlp_to_bf16(const float* w, void* w_bf16, long long n, void* stream) {
  if (!w || !w_bf16 || n < 0) return mmdg_internal_fail(MMDG_E_ARG, "mmdg_mlp_to_bf16: bad argument");
  if (!n) return MMDG_OK;
  k_to_bf16<<<nb(n), 256, 0, (cudaStream_t)stream>>>(w, (__nv_bfloat16*)w_bf16, n);
  return launch_fail("mmdg_mlp_to_bf16: launch");
}
