// No-pivot leaf of the random-butterfly-transformed factors, up to 128 columns
// in two launches:
//
//   1. genp_top_kernel, one CTA: LU without interchanges of the leaf's top
//      128 x 128 block in shared memory, 32 columns at a time; it leaves the
//      packed factors and the reciprocals of U's diagonal in the work area.
//   2. genp_below_kernel: every 32 rows below the block solve l U = a by
//      blocks (product with the columns before, then substitution in the
//      diagonal block); sixteen more CTAs compute the inverse of L11, which the TRSMs
//      to the right of the leaf apply.
//
// What bounds a factorization of a few thousand columns is the chain of dependent
// launches, not the work in them.  A 32-column leaf (13 us, with every CTA
// repeating the top block's factorization) needs four panels, three TRSMs and
// three updates where this needs two launches: FP16 factor and refined solve of
// n = 6002, two right-hand sides, 9.57 -> 6.86 ms.  Both kernels are substitution
// with correctly rounded reciprocals: without pivoting nothing bounds the
// condition of U's diagonal blocks, and a product with the inverse of one leaves
// an error of its condition times u in the rows below (8 w u |L||U| exceeded 400
// times where the condition is 1.6^31).  With FP32 operands the factors have the
// bits of 32-column leaves with their TRSMs and updates (n = 64 .. 3000).  A leaf
// of n = 4096 takes the rows below 12.0 us in place of 9.8 (ncu, cold caches), and
// the top block as much less without the inverses to form.
//
// An exactly zero pivot sets info and leaves its column unscaled, as getf2.
#include <cuda_runtime.h>

#include <algorithm>

#include "device_util.cuh"
#include "gblu_internal.h"
#include "objects.h"
#include "profile.h"

namespace gblu {

namespace {

constexpr int kB = 32;                   // sub-block
constexpr int kGenpLd = kGenpW + 4;      // column stride in shared memory (16-byte columns, no bank conflicts)
constexpr int kGenpTopThreads = 512;
constexpr int kGenpRows = 32;            // rows of a CTA below the block
constexpr int kGenpThreads = 256;
constexpr int kInvColsPerCta = kGenpThreads / 32;
constexpr int kInvCtas = kGenpW / kInvColsPerCta;
constexpr int kXLd = kGenpRows + 4;

// Work area: the factored top block (ld 128), then the reciprocals of U's diagonal.
constexpr size_t kGenpWork = (size_t)(kGenpW * kGenpW + kGenpW) * sizeof(float);

__device__ __forceinline__ float part_of(const float4& v, int i) {
  return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }

__device__ __forceinline__ void copy16(float* dst, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// C(32 rows at r0, 8 columns at c0) -= L(:, k .. k + 31) U(k .. k + 31, :) by one
// warp; lane: rows 4 (lane % 8) .., columns lane / 8 and lane / 8 + 4.
__device__ __forceinline__ void update_tile(float* S, int r0, int c0, int k) {
  const int lane = threadIdx.x & 31;
  float* c = S + (c0 + (lane >> 3)) * kGenpLd;
  r0 += 4 * (lane & 7);
  float4 acc[2];
#pragma unroll
  for (int jj = 0; jj < 2; ++jj) acc[jj] = ld4(c + 4 * jj * kGenpLd + r0);
#pragma unroll 4
  for (int k4 = k; k4 < k + kB; k4 += 4) {
    float4 u[2];
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) u[jj] = ld4(c + 4 * jj * kGenpLd + k4);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const float4 l = ld4(S + (k4 + kk) * kGenpLd + r0);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const float uk = part_of(u[jj], kk);
        acc[jj].x = fmaf(-l.x, uk, acc[jj].x);
        acc[jj].y = fmaf(-l.y, uk, acc[jj].y);
        acc[jj].z = fmaf(-l.z, uk, acc[jj].z);
        acc[jj].w = fmaf(-l.w, uk, acc[jj].w);
      }
    }
  }
#pragma unroll
  for (int jj = 0; jj < 2; ++jj) st4(c + 4 * jj * kGenpLd + r0, acc[jj]);
}

// Bound by the column chain (a broadcast, a reciprocal and an update a column),
// so everything else runs beside it.  Per 32 columns: warps 0-3 update the
// diagonal block with the 32 columns before; warp 0 then factors it in
// registers (lane = row) and publishes it eight columns at a time to warps 1-3
// (a row below it a thread, l U = a) and 4-6 (a column right of it a thread,
// L u = a), which follow eight columns behind, after the rows and columns they
// solve have had their update; warps 7-15 update the rest.  Against the same steps one after the other:
// 52,000 -> 45,000 cycles a 128 x 128 block.  Columns and rows past w are those
// of the identity.
__global__ void __launch_bounds__(kGenpTopThreads)
genp_top_kernel(float* __restrict__ A, int64_t lda, int64_t c0, int w, int64_t* __restrict__ ipiv,
                int64_t* __restrict__ info, float* __restrict__ work) {
  extern __shared__ __align__(16) float S[];  // S[c * kGenpLd + r]
  __shared__ __align__(16) float UT[kB][kB + 4];  // the current diagonal block by rows
  __shared__ float rd[kB];                        // reciprocals of its pivots
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = (w + kB - 1) / kB, end = kB * nb;
  float* rdiag = work + kGenpW * kGenpW;
  float* Ac = A + c0 + c0 * lda;
#pragma unroll 16
  for (int e = 0; e < kGenpW * kGenpW / kGenpTopThreads; ++e) {
    const int idx = e * kGenpTopThreads + tid, c = idx / kGenpW, r = idx % kGenpW;
    S[c * kGenpLd + r] = (r < w && c < w) ? Ac[r + c * lda] : (r == c ? 1.f : 0.f);
  }
  int zc = -1;  // warp 0: the first zero pivot's column
  __syncthreads();
#pragma unroll 1
  for (int b = 0; b < nb; ++b) {
    const int o = kB * b, kp = o - kB;
    const int nrem = (end - o) / kB - 1;  // blocks below and right of the diagonal one
    if (b > 0) {
      if (warp < 4) {
        update_tile(S, o, o + 8 * warp, kp);
        named_bar_sync(5, 128);
      }
      if (warp > 0) {
        for (int q = warp - 1; q < 8 * nrem; q += 15) {
          if (q < 4 * nrem) update_tile(S, o + kB + kB * (q / 4), o + 8 * (q % 4), kp);
          else update_tile(S, o, o + kB + 8 * (q - 4 * nrem), kp);
        }
        named_bar_sync(6, kGenpTopThreads - 32);
      }
    }
    if (warp == 0) {
      float r[kB];
#pragma unroll
      for (int j = 0; j < kB; ++j) r[j] = S[(o + j) * kGenpLd + o + lane];
      float own = 1.f;
      float u = __shfl_sync(0xffffffffu, r[0], 0);
      float rp = u != 0.f ? recip_rn(u) : 1.0f;
#pragma unroll
      for (int k = 0; k < kB; ++k) {
        zc = (u == 0.f && zc < 0) ? o + k : zc;
        own = lane == k ? rp : own;
        const bool below = lane > k;
        const float l = r[k] * rp;
        r[k] = below ? l : r[k];
        // the next column first: its reciprocal is formed beside the others' updates
        if (k + 1 < kB) {
          const float un = __shfl_sync(0xffffffffu, r[k + 1 < kB ? k + 1 : 0], k);
          if (below) r[k + 1 < kB ? k + 1 : 0] = fmaf(-l, un, r[k + 1 < kB ? k + 1 : 0]);
          u = __shfl_sync(0xffffffffu, r[k + 1 < kB ? k + 1 : 0], k + 1);
          rp = u != 0.f ? recip_rn(u) : 1.0f;
        }
#pragma unroll
        for (int j = 0; j < kB; ++j) {
          if (j <= k + 1) continue;
          const float uj = __shfl_sync(0xffffffffu, r[j], k);
          if (below) r[j] = fmaf(-l, uj, r[j]);
        }
        if ((k & 7) == 7) {  // columns k - 7 .. k are final
#pragma unroll
          for (int j = 0; j < kB; ++j)
            if (j / 8 == k / 8) S[(o + j) * kGenpLd + o + lane] = r[j];
          if (lane / 8 == k / 8) {
            rd[lane] = own;
            rdiag[o + lane] = own;
#pragma unroll
            for (int j = 0; j < kB; j += 4)
              if (j / 8 >= k / 8) st4(&UT[lane][j], make_float4(r[j], r[j + 1], r[j + 2], r[j + 3]));
          }
          named_bar_arrive(1 + k / 8, 7 * 32);
        }
      }
    } else if (warp < 4) {  // row t: x U_bb = a
      const int t = o + kB * warp + lane;
      const bool on = t < end;  // the same for the warp
      float x[kB];
      if (on) {
#pragma unroll
        for (int j = 0; j < kB; ++j) x[j] = S[(o + j) * kGenpLd + t];
      }
#pragma unroll
      for (int i = 0; i < kB; ++i) {
        if ((i & 7) == 0) named_bar_sync(1 + i / 8, 7 * 32);
        if (!on) continue;
        x[i] *= rd[i];
#pragma unroll
        for (int j4 = 0; j4 < kB / 4; ++j4) {
          if (4 * j4 + 3 <= i) continue;
          const float4 u = ld4(&UT[i][4 * j4]);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (4 * j4 + q > i) x[4 * j4 + q] = fmaf(-x[i], part_of(u, q), x[4 * j4 + q]);
        }
      }
      if (on) {
#pragma unroll
        for (int j = 0; j < kB; ++j) S[(o + j) * kGenpLd + t] = x[j];
      }
    } else if (warp < 7) {  // column t: L_bb x = a
      const int t = o + kB * (warp - 3) + lane;
      const bool on = t < end;
      float x[kB];
      if (on) {
#pragma unroll
        for (int j = 0; j < kB; j += 4) {
          const float4 v = ld4(&S[t * kGenpLd + o + j]);
          x[j] = v.x; x[j + 1] = v.y; x[j + 2] = v.z; x[j + 3] = v.w;
        }
      }
#pragma unroll
      for (int k = 0; k < kB; ++k) {
        if ((k & 7) == 0) named_bar_sync(1 + k / 8, 7 * 32);
        if (!on) continue;
#pragma unroll
        for (int i4 = 0; i4 < kB / 4; ++i4) {
          if (4 * i4 + 3 <= k) continue;
          const float4 l = ld4(&S[(o + k) * kGenpLd + o + 4 * i4]);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (4 * i4 + q > k) x[4 * i4 + q] = fmaf(-part_of(l, q), x[k], x[4 * i4 + q]);
        }
      }
      if (on) {
#pragma unroll
        for (int j = 0; j < kB; j += 4) st4(&S[t * kGenpLd + o + j], make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]));
      }
    } else if (b > 0) {
      for (int q = warp - 7; q < 4 * nrem * nrem; q += 9)
        update_tile(S, o + kB + kB * (q % nrem), o + kB + 8 * (q / nrem), kp);
    }
    __syncthreads();
  }
#pragma unroll 8
  for (int e = 0; e < kGenpW * kGenpW / kGenpTopThreads; ++e) {
    const int idx = e * kGenpTopThreads + tid, c = idx / kGenpW, r = idx % kGenpW;
    const float v = S[c * kGenpLd + r];
    work[idx] = v;
    if (r < w && c < w) Ac[r + c * lda] = v;
  }
  if (tid < w) ipiv[c0 + tid] = c0 + tid + 1;
  if (tid == 0 && zc >= 0)
    atomicCAS(reinterpret_cast<unsigned long long*>(info), 0ull, (unsigned long long)(c0 + zc + 1));
}

constexpr size_t kGenpTopSmem = (size_t)kGenpW * kGenpLd * sizeof(float);
constexpr size_t kGenpBelowSmem =
    ((size_t)kGenpW * kGenpLd + kGenpW + (size_t)kGenpW * kXLd) * sizeof(float);

// CTAs 0 .. row_ctas - 1: 32 rows below the block each.  Warp: 4 rows, lane: a
// column of the current 32, so after the copies no warp waits for another.
// 32 rows a CTA put a 6000-row leaf on all SMs; the chain of one warp (48
// steps of five 16-byte loads and 16 FMAs, and 128 of a product, a shuffle and
// an FMA for each of the four rows) is then what it takes.
// The other CTAs: the inverse of L11 by the TRSM chain, one column a warp.
__global__ void __launch_bounds__(kGenpThreads)
genp_below_kernel(float* __restrict__ A, int64_t lda, int64_t m, int64_t c0, int w, const float* __restrict__ work,
                  int row_ctas, float* __restrict__ linv) {
  extern __shared__ __align__(16) float smem[];
  float* sU = smem;                              // the top block, by columns
  float* sR = sU + kGenpW * kGenpLd;             // reciprocals of U's diagonal
  float* sX = sR + kGenpW;                       // sX[column * 36 + row]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((int)blockIdx.x >= row_ctas) {
    const int j0 = ((int)blockIdx.x - row_ctas) * kInvColsPerCta;
    for (int i = tid + j0 * (kGenpW / 4); i < kGenpW * (kGenpW / 4); i += kGenpThreads) {
      const int c = i / (kGenpW / 4), r = 4 * (i % (kGenpW / 4));
      if (r + 3 > c) copy16(sU + c * kGenpLd + r, work + c * kGenpW + r);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int j = j0 + warp;
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = lane + 32 * q == j ? 1.f : 0.f;
#pragma unroll
    for (int qk = 0; qk < 4; ++qk) {
      if (32 * qk + 31 < j) continue;
#pragma unroll 4
      for (int kk = max(j, 32 * qk); kk < 32 * qk + 32; ++kk) {
        const float xk = __shfl_sync(0xffffffffu, v[qk], kk & 31);
#pragma unroll
        for (int q = qk; q < 4; ++q) {
          const int r = lane + 32 * q;
          if (r > kk) v[q] = fmaf(-sU[kk * kGenpLd + r], xk, v[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) linv[lane + 32 * q + j * kGenpW] = v[q];
    return;
  }
  const int nb = (w + kB - 1) / kB;
  const int64_t r0 = c0 + w + (int64_t)blockIdx.x * kGenpRows;
  const int nr = (int)min((int64_t)kGenpRows, m - r0);
  for (int b = 0; b < nb; ++b)  // U's blocks, the diagonal ones included
    for (int i = tid; i < kB * 8 * (b + 1); i += kGenpThreads) {
      const int c = kB * b + i / (8 * (b + 1)), k = 4 * (i % (8 * (b + 1)));
      copy16(sU + c * kGenpLd + k, work + c * kGenpW + k);
    }
  for (int i = tid; i < nb * kB / 4; i += kGenpThreads) copy16(sR + 4 * i, work + kGenpW * kGenpW + 4 * i);
  {
    float x[kGenpW / 8];
#pragma unroll
    for (int e = 0; e < kGenpW / 8; ++e) {
      const int c = warp + 8 * e;
      x[e] = (c < w && lane < nr) ? A[r0 + lane + (c0 + c) * lda] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < kGenpW / 8; ++e) sX[(warp + 8 * e) * kXLd + lane] = x[e];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* xr = sX + 4 * warp;  // this warp's rows
#pragma unroll 1
  for (int b = 0; b < nb; ++b) {
    const int c = kB * b + lane;
    float4 acc = ld4(xr + c * kXLd);
    const float* u = sU + c * kGenpLd;
#pragma unroll 4
    for (int k = 0; k < kB * b; k += 4) {
      const float4 u4 = ld4(u + k);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const float4 x = ld4(xr + (k + kk) * kXLd);
        const float uk = part_of(u4, kk);
        acc.x = fmaf(-x.x, uk, acc.x);
        acc.y = fmaf(-x.y, uk, acc.y);
        acc.z = fmaf(-x.z, uk, acc.z);
        acc.w = fmaf(-x.w, uk, acc.w);
      }
    }
    // substitution: step k's value goes from lane k to the columns after it
    const float r = sR[c];
    float ud[kB];
#pragma unroll
    for (int k = 0; k < kB; k += 4) {
      const float4 u4 = ld4(u + kB * b + k);
      ud[k] = u4.x; ud[k + 1] = u4.y; ud[k + 2] = u4.z; ud[k + 3] = u4.w;
    }
#pragma unroll
    for (int k = 0; k < kB - 1; ++k) {
      const float x0 = __shfl_sync(0xffffffffu, acc.x * r, k), x1 = __shfl_sync(0xffffffffu, acc.y * r, k);
      const float x2 = __shfl_sync(0xffffffffu, acc.z * r, k), x3 = __shfl_sync(0xffffffffu, acc.w * r, k);
      if (lane > k) {
        acc.x = fmaf(-x0, ud[k], acc.x);
        acc.y = fmaf(-x1, ud[k], acc.y);
        acc.z = fmaf(-x2, ud[k], acc.z);
        acc.w = fmaf(-x3, ud[k], acc.w);
      }
    }
    st4(xr + c * kXLd, make_float4(acc.x * r, acc.y * r, acc.z * r, acc.w * r));
    __syncwarp();
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kGenpW / 8; ++e) {
    const int c = warp + 8 * e;
    if (c < w && lane < nr) A[r0 + lane + (c0 + c) * lda] = sX[c * kXLd + lane];
  }
}

}  // namespace

size_t genp_work_bytes() { return kGenpWork; }

void genp_configure(int /*device*/) {
  cudaFuncSetAttribute(genp_top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGenpTopSmem);
  cudaFuncSetAttribute(genp_below_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGenpBelowSmem);
}

cudaError_t genp_panel_launch(float* A, int64_t lda, int64_t m, int64_t c0, int w, int64_t* ipiv,
                              int64_t* info, void* work, float* linv, cudaStream_t s) {
  if (w <= 0 || w > kGenpW || m - c0 < w || (linv && w != kGenpW)) return cudaErrorInvalidValue;
  float* wk = reinterpret_cast<float*>(work);
  const int64_t below = m - c0 - w;
  {
    LaunchScope ls(K_PANEL, 2.0 / 3.0 * w * w * w, 2.0 * w * w * sizeof(float), s);
    genp_top_kernel<<<1, kGenpTopThreads, kGenpTopSmem, s>>>(A, lda, c0, w, ipiv, info, wk);
  }
  cudaError_t e = cudaGetLastError();
  const int64_t row_ctas = (below + kGenpRows - 1) / kGenpRows;
  const int64_t ctas = row_ctas + (linv ? kInvCtas : 0);
  if (e != cudaSuccess || ctas == 0) return e;
  LaunchScope ls(K_PANEL, (double)below * w * w, 2.0 * below * w * sizeof(float), s);
  genp_below_kernel<<<(unsigned)ctas, kGenpThreads, kGenpBelowSmem, s>>>(A, lda, m, c0, w, wk, (int)row_ctas, linv);
  return cudaGetLastError();
}

}  // namespace gblu
