// getrf on the device: recursive right-looking LU with partial pivoting.
//
// Structure (the LAPACK getrf structure the reference states in
// src/blocked_lufact.jl:658-679, arranged recursively as in
// RFLUFactorization's RecursiveFactorization, ext/LinearSolveRecursiveFactorizationExt.jl:15-42):
//
//   rec(c0, w):  if w <= panel width:  panel_kernel   (getf2 on the leaf,
//                                       blocked_lufact.jl:93-122)
//                                       laswp_kernel   (interchanges on every
//                                       other column, :126-141)
//                else  rec(c0, w1)
//                      trsm  U12 := L11 \ A12       (:146-178)
//                      gemm  A22 -= L21 * U12       (:186-656)
//                      rec(c0 + w1, w - w1)
//
// Floating point: each element A[i,j] receives fma(-l_ik, u_kj, a_ij) for
// k ascending, exactly as the reference's muladd loops, and the multipliers
// are a_ik * (1 / u_kk).  Every kernel below keeps that per-element order
// (C is loaded first, then updated k = 0, 1, ...), so the factors and ipiv
// are bit-identical to the reference's blocked LU for any blocking.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "device_util.cuh"
#include "waits.cuh"
#include "gblu_internal.h"
#include "profile.h"

namespace gblu {

constexpr int kPanelThreads = 256;
constexpr int kPanelMaxW = 32;
constexpr int kPanelRowsTarget = 64;

// ---------------------------------------------------------------------------
// Pivot-candidate ordering: larger |a| wins; ties go to the smaller row;
// row -1 means "no candidate" (|a| == 0 or NaN everywhere, blocked_lufact.jl:38-54).
template <typename T>
__device__ __forceinline__ bool cand_better(T v, int64_t g, T bv, int64_t bg) {
  if (g < 0) return false;
  if (bg < 0) return true;
  return (v > bv) || (v == bv && g < bg);
}


// ---------------------------------------------------------------------------
// Cooperative panel kernel: getf2 on rows [c0, m) x columns [c0, c0+w).
// Each CTA holds a contiguous slice of R rows of the panel in shared memory;
// one grid barrier per column exchanges the pivot candidates.
template <typename T>
__global__ void __launch_bounds__(kPanelThreads)
panel_kernel(T* __restrict__ A, int64_t lda, int64_t m, int64_t c0, int w,
             int64_t* __restrict__ ipiv, int64_t* __restrict__ info_out,
             DevScratch* __restrict__ scr, PanelSlots<T> slots, int R) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // column j at tile + j*R
  __shared__ T pivrow[kPanelMaxW];
  __shared__ T diagrow[kPanelMaxW];
  using K = typename PivKey<T>::K;  // pivot candidates compared as integer keys of |a|
  __shared__ K red_v[kPanelThreads / 32];
  __shared__ int64_t red_g[kPanelThreads / 32];
  __shared__ int red_c[kPanelThreads / 32];
  K* cand_key = reinterpret_cast<K*>(slots.cand_val);
  __shared__ int64_t s_best_g;
  __shared__ int s_best_c;

  const int G = gridDim.x;
  const int cta = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = c0 + (int64_t)cta * R;
  const int nloc = (int)max((int64_t)0, min((int64_t)R, m - base));

  for (int j = 0; j < w; ++j)
    for (int i = tid; i < R; i += blockDim.x)
      tile[(size_t)j * R + i] = (i < nloc) ? A[(base + i) + (c0 + j) * lda] : T(0);
  int64_t info_local = 0;
  __syncthreads();

  for (int k = 0; k < w; ++k) {
    const int64_t d = c0 + k;
    const int buf = k & 1;
    const T* colk = tile + (size_t)k * R;

    // 1. local candidate: first row of max |a| among rows >= d (NaN ignored)
    K bv = 0;
    int64_t bg = -1;
    for (int i = tid; i < nloc; i += blockDim.x) {
      int64_t g = base + i;
      K v = PivKey<T>::of(colk[i]);
      if (g >= d && v > bv) { bv = v; bg = g; }
    }
    for (int off = 16; off; off >>= 1) {
      K ov = __shfl_down_sync(0xffffffffu, bv, off);
      int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
      if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; }
    }
    if (lane == 0) { red_v[warp] = bv; red_g[warp] = bg; }
    __syncthreads();
    if (warp == 0) {
      bv = lane < (kPanelThreads / 32) ? red_v[lane] : K(0);
      bg = lane < (kPanelThreads / 32) ? red_g[lane] : -1;
      for (int off = 16; off; off >>= 1) {
        K ov = __shfl_down_sync(0xffffffffu, bv, off);
        int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
        if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; }
      }
      if (lane == 0) {
        stcg(&cand_key[buf * G + cta], bv);
        stcg(&slots.cand_row[buf * G + cta], bg);
        s_best_g = bg;
      }
    }
    __syncthreads();
    // 2. publish the candidate's panel row and, if owned here, the diagonal row
    if (tid < w) {
      if (s_best_g >= 0)
        stcg(&slots.cand_rowvals[((size_t)buf * G + cta) * kPanelMaxW + tid],
             tile[(size_t)tid * R + (s_best_g - base)]);
      if (d >= base && d < base + nloc)
        stcg(&slots.diag_rowvals[buf * kPanelMaxW + tid], tile[(size_t)tid * R + (d - base)]);
    }
    if (!grid_barrier(scr, (unsigned)(k + 1) * (unsigned)G)) return;

    // 3. global winner over the G candidates (same reduction on every CTA)
    bv = 0;
    bg = -1;
    int bc = -1;
    for (int c = tid; c < G; c += blockDim.x) {
      K v = ldcg(&cand_key[buf * G + c]);
      int64_t g = ldcg(&slots.cand_row[buf * G + c]);
      if (cand_better(v, g, bv, bg)) { bv = v; bg = g; bc = c; }
    }
    for (int off = 16; off; off >>= 1) {
      K ov = __shfl_down_sync(0xffffffffu, bv, off);
      int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
      int oc = __shfl_down_sync(0xffffffffu, bc, off);
      if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; bc = oc; }
    }
    if (lane == 0) { red_v[warp] = bv; red_g[warp] = bg; red_c[warp] = bc; }
    __syncthreads();
    if (warp == 0) {
      bv = lane < (kPanelThreads / 32) ? red_v[lane] : K(0);
      bg = lane < (kPanelThreads / 32) ? red_g[lane] : -1;
      bc = lane < (kPanelThreads / 32) ? red_c[lane] : -1;
      for (int off = 16; off; off >>= 1) {
        K ov = __shfl_down_sync(0xffffffffu, bv, off);
        int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
        int oc = __shfl_down_sync(0xffffffffu, bc, off);
        if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; bc = oc; }
      }
      if (lane == 0) { s_best_g = bg; s_best_c = bc; }
    }
    __syncthreads();
    const int64_t p = s_best_g < 0 ? d : s_best_g;  // kp = k when amax == 0
    const int pc = s_best_c;
    if (tid < w) {
      T dv = ldcg(&slots.diag_rowvals[buf * kPanelMaxW + tid]);
      diagrow[tid] = dv;
      pivrow[tid] = (p == d) ? dv : ldcg(&slots.cand_rowvals[((size_t)buf * G + pc) * kPanelMaxW + tid]);
    }
    if (cta == 0 && tid == 0) ipiv[d] = p + 1;
    __syncthreads();
    const T piv = pivrow[k];

    // 4. interchange (only when the pivot is nonzero), scale, rank-1 update
    if (piv != T(0)) {
      if (p != d) {
        if (tid < w) {
          if (d >= base && d < base + nloc) tile[(size_t)tid * R + (d - base)] = pivrow[tid];
          if (p >= base && p < base + nloc) tile[(size_t)tid * R + (p - base)] = diagrow[tid];
        }
        __syncthreads();
      }
      const T inv = T(1) / piv;
      for (int i = tid; i < nloc; i += blockDim.x)
        if (base + i > d) tile[(size_t)k * R + i] *= inv;
    } else if (info_local == 0) {
      info_local = d + 1;
    }
    __syncthreads();
    // rank-1 update of this CTA's rows below the diagonal: one row per thread,
    // columns k+1..w-1 in order (per element: one fma, k ascending)
    for (int i = tid; i < nloc; i += blockDim.x) {
      if (base + i <= d) continue;
      const T l = tile[(size_t)k * R + i];
      for (int j = k + 1; j < w; ++j)
        tile[(size_t)j * R + i] = fma(-l, pivrow[j], tile[(size_t)j * R + i]);
    }
    __syncthreads();
  }

  for (int j = 0; j < w; ++j)
    for (int i = tid; i < nloc; i += blockDim.x) A[(base + i) + (c0 + j) * lda] = tile[(size_t)j * R + i];
  if (cta == 0 && tid == 0 && info_local != 0 && *info_out == 0) *info_out = info_local;
}

// ---------------------------------------------------------------------------
// Cluster panel kernel: the same getf2 on rows [c0, m) x columns [c0, c0+w),
// for panels that fit in the shared memory of one thread-block cluster (up to
// 16 CTAs).  Pivot candidates, the candidate rows and the diagonal row live in
// each CTA's shared memory; after the hardware cluster barrier every CTA reads
// the others' slots through distributed shared memory, so a column costs one
// cluster barrier and one round of DSMEM loads instead of a grid barrier and
// two L2 round trips.  The arithmetic per element is the grid kernel's.
template <typename T>
__global__ void __launch_bounds__(kPanelThreads)
panel_cluster_kernel(T* __restrict__ A, int64_t lda, int64_t m, int64_t c0, int w,
                     int64_t* __restrict__ ipiv, int64_t* __restrict__ info_out, int R) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);  // column j at tile + j*R
  __shared__ typename PivKey<T>::K s_cval[2];
  __shared__ int64_t s_crow[2];
  __shared__ T s_crowv[2][kPanelMaxW];
  __shared__ T s_diagv[2][kPanelMaxW];
  __shared__ T pivrow[kPanelMaxW];
  __shared__ T diagrow[kPanelMaxW];
  using K = typename PivKey<T>::K;  // pivot candidates compared as integer keys of |a|
  __shared__ K red_v[kPanelThreads / 32];
  __shared__ int64_t red_g[kPanelThreads / 32];
  __shared__ int64_t s_best_g;
  __shared__ int s_best_c;

  const int G = (int)cluster.num_blocks();
  const int cta = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = c0 + (int64_t)cta * R;
  const int nloc = (int)max((int64_t)0, min((int64_t)R, m - base));

  for (int j = 0; j < w; ++j)
    for (int i = tid; i < R; i += blockDim.x)
      tile[(size_t)j * R + i] = (i < nloc) ? A[(base + i) + (c0 + j) * lda] : T(0);
  int64_t info_local = 0;
  __syncthreads();

  for (int k = 0; k < w; ++k) {
    const int64_t d = c0 + k;
    const int buf = k & 1;
    const T* colk = tile + (size_t)k * R;
    K bv = 0;
    int64_t bg = -1;
    for (int i = tid; i < nloc; i += blockDim.x) {
      int64_t g = base + i;
      K v = PivKey<T>::of(colk[i]);
      if (g >= d && v > bv) { bv = v; bg = g; }
    }
    for (int off = 16; off; off >>= 1) {
      K ov = __shfl_down_sync(0xffffffffu, bv, off);
      int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
      if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; }
    }
    if (lane == 0) { red_v[warp] = bv; red_g[warp] = bg; }
    __syncthreads();
    if (warp == 0) {
      bv = lane < (kPanelThreads / 32) ? red_v[lane] : K(0);
      bg = lane < (kPanelThreads / 32) ? red_g[lane] : -1;
      for (int off = 16; off; off >>= 1) {
        K ov = __shfl_down_sync(0xffffffffu, bv, off);
        int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
        if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; }
      }
      if (lane == 0) { s_cval[buf] = bv; s_crow[buf] = bg; s_best_g = bg; }
    }
    __syncthreads();
    if (tid < w) {
      if (s_best_g >= 0) s_crowv[buf][tid] = tile[(size_t)tid * R + (s_best_g - base)];
      if (d >= base && d < base + nloc) s_diagv[buf][tid] = tile[(size_t)tid * R + (d - base)];
    }
    cluster.sync();  // publishes the slots of step k (release/acquire across the cluster)

    // winner over the G candidates, read through distributed shared memory
    bv = 0;
    bg = -1;
    int bc = -1;
    if (tid < G) {
      const K* rv = cluster.map_shared_rank(&s_cval[buf], tid);
      const int64_t* rr = cluster.map_shared_rank(&s_crow[buf], tid);
      bv = *rv;
      bg = *rr;
      bc = bg >= 0 ? tid : -1;
    }
    if (warp == 0) {
      for (int off = 16; off; off >>= 1) {
        K ov = __shfl_down_sync(0xffffffffu, bv, off);
        int64_t og = __shfl_down_sync(0xffffffffu, bg, off);
        int oc = __shfl_down_sync(0xffffffffu, bc, off);
        if (cand_better(ov, og, bv, bg)) { bv = ov; bg = og; bc = oc; }
      }
      if (lane == 0) { s_best_g = bg; s_best_c = bc; }
    }
    __syncthreads();
    const int64_t p = s_best_g < 0 ? d : s_best_g;
    const int pc = s_best_c;
    const int downer = (int)((d - c0) / R);
    if (tid < w) {
      const T dv = *cluster.map_shared_rank(&s_diagv[buf][tid], downer);
      diagrow[tid] = dv;
      pivrow[tid] = (p == d) ? dv : *cluster.map_shared_rank(&s_crowv[buf][tid], pc);
    }
    if (cta == 0 && tid == 0) ipiv[d] = p + 1;
    __syncthreads();
    const T piv = pivrow[k];
    if (piv != T(0)) {
      if (p != d) {
        if (tid < w) {
          if (d >= base && d < base + nloc) tile[(size_t)tid * R + (d - base)] = pivrow[tid];
          if (p >= base && p < base + nloc) tile[(size_t)tid * R + (p - base)] = diagrow[tid];
        }
        __syncthreads();
      }
      const T inv = T(1) / piv;
      for (int i = tid; i < nloc; i += blockDim.x)
        if (base + i > d) tile[(size_t)k * R + i] *= inv;
    } else if (info_local == 0) {
      info_local = d + 1;
    }
    __syncthreads();
    // rank-1 update of this CTA's rows below the diagonal: one row per thread,
    // columns k+1..w-1 in order (per element: one fma, k ascending)
    for (int i = tid; i < nloc; i += blockDim.x) {
      if (base + i <= d) continue;
      const T l = tile[(size_t)k * R + i];
      for (int j = k + 1; j < w; ++j)
        tile[(size_t)j * R + i] = fma(-l, pivrow[j], tile[(size_t)j * R + i]);
    }
    __syncthreads();
  }
  for (int j = 0; j < w; ++j)
    for (int i = tid; i < nloc; i += blockDim.x) A[(base + i) + (c0 + j) * lda] = tile[(size_t)j * R + i];
  if (cta == 0 && tid == 0 && info_local != 0 && *info_out == 0) *info_out = info_local;
  cluster.sync();  // no CTA leaves while another may still read its shared memory
}

// ---------------------------------------------------------------------------
// laswp for one leaf: interchanges ipiv[c0, c0+w) applied to every column
// outside [c0, c0+w) (blocked_lufact.jl:126-141 applies them to [1, j0) and
// (j1, n]).  Warp 0 of every CTA composes the w swaps into at most 2w moves
// "row r receives old row src(r)"; then each warp moves one column at a time.
template <typename T>
__global__ void __launch_bounds__(256)
laswp_leaf_kernel(T* __restrict__ A, int64_t lda, int64_t m, int64_t ncols_total,
                  int64_t c0, int w, const int64_t* __restrict__ ipiv,
                  DevScratch* __restrict__ scr, int32_t* __restrict__ perm) {
  __shared__ int64_t mv_dst[2 * kPanelMaxW];
  __shared__ int64_t mv_src[2 * kPanelMaxW];
  __shared__ int s_nmv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    // entry 0 of lane k tracks row c0+k; entry 1 tracks target t_k when it lies
    // below the leaf and no earlier lane already tracks it.
    int64_t t = (lane < w) ? ipiv[c0 + lane] - 1 : -1;
    if (lane < w && (t < c0 + lane || t >= m)) atomicCAS(&scr->error, 0, (int)DEV_BAD_PIVOT_INDEX);
    int64_t row0 = (lane < w) ? c0 + lane : -1;
    int64_t src0 = row0;
    bool dup = false;
    for (int j = 0; j < 32; ++j) {
      int64_t tj = __shfl_sync(0xffffffffu, t, j);
      if (j < lane && tj == t) dup = true;
    }
    int64_t row1 = (lane < w && t >= c0 + w && t < m && !dup) ? t : -1;
    int64_t src1 = row1;
    for (int k = 0; k < w; ++k) {
      int64_t a = c0 + k;
      int64_t b = __shfl_sync(0xffffffffu, t, k);
      if (b == a || b < 0) continue;
      unsigned ha0 = __ballot_sync(0xffffffffu, row0 == a), ha1 = __ballot_sync(0xffffffffu, row1 == a);
      unsigned hb0 = __ballot_sync(0xffffffffu, row0 == b), hb1 = __ballot_sync(0xffffffffu, row1 == b);
      if ((ha0 | ha1) == 0 || (hb0 | hb1) == 0) continue;  // corrupt ipiv: flagged above
      int la = ha0 ? __ffs(ha0) - 1 : __ffs(ha1) - 1;
      int lb = hb0 ? __ffs(hb0) - 1 : __ffs(hb1) - 1;
      int64_t sa = ha0 ? __shfl_sync(0xffffffffu, src0, la) : __shfl_sync(0xffffffffu, src1, la);
      int64_t sb = hb0 ? __shfl_sync(0xffffffffu, src0, lb) : __shfl_sync(0xffffffffu, src1, lb);
      if (ha0) { if (lane == la) src0 = sb; } else { if (lane == la) src1 = sb; }
      if (hb0) { if (lane == lb) src0 = sa; } else { if (lane == lb) src1 = sa; }
    }
    bool m0 = row0 >= 0 && src0 != row0, m1 = row1 >= 0 && src1 != row1;
    unsigned b0 = __ballot_sync(0xffffffffu, m0), b1 = __ballot_sync(0xffffffffu, m1);
    int n0 = __popc(b0);
    if (m0) { int pos = __popc(b0 & ((1u << lane) - 1)); mv_dst[pos] = row0; mv_src[pos] = src0; }
    if (m1) { int pos = n0 + __popc(b1 & ((1u << lane) - 1)); mv_dst[pos] = row1; mv_src[pos] = src1; }
    if (lane == 0) s_nmv = n0 + __popc(b1);
  }
  __syncthreads();
  const int nmv = s_nmv;
  if (nmv == 0) return;
  if (perm != nullptr && blockIdx.x == 0 && warp == 0) {
    // the row permutation (original row of each row) moves like one more column
    int32_t p0 = 0, p1 = 0;
    if (lane < nmv) p0 = perm[mv_src[lane]];
    if (lane + 32 < nmv) p1 = perm[mv_src[lane + 32]];
    __syncwarp();
    if (lane < nmv) perm[mv_dst[lane]] = p0;
    if (lane + 32 < nmv) perm[mv_dst[lane + 32]] = p1;
  }
  const int64_t nother = ncols_total - w;
  const int warps = blockDim.x >> 5;
  const int64_t stride = (int64_t)gridDim.x * warps;
  // two columns per pass: all four loads in flight before the stores
  for (int64_t q = (int64_t)blockIdx.x * warps + warp; q < nother; q += 2 * stride) {
    const int64_t q2 = q + stride;
    T* a = A + (q < c0 ? q : q + w) * lda;
    T* b2 = q2 < nother ? A + (q2 < c0 ? q2 : q2 + w) * lda : nullptr;
    T v0 = T(0), v1 = T(0), u0 = T(0), u1 = T(0);
    if (lane < nmv) v0 = a[mv_src[lane]];
    if (lane + 32 < nmv) v1 = a[mv_src[lane + 32]];
    if (b2 && lane < nmv) u0 = b2[mv_src[lane]];
    if (b2 && lane + 32 < nmv) u1 = b2[mv_src[lane + 32]];
    __syncwarp();
    if (lane < nmv) a[mv_dst[lane]] = v0;
    if (lane + 32 < nmv) a[mv_dst[lane + 32]] = v1;
    if (b2 && lane < nmv) b2[mv_dst[lane]] = u0;
    if (b2 && lane + 32 < nmv) b2[mv_dst[lane + 32]] = u1;
  }
}

// The same from composed moves (the sub-panel kernel's output): every warp
// carries two columns per pass through up to 256 moves, all loads in flight
// before the stores.
template <typename T>
__global__ void __launch_bounds__(256)
laswp_moves_kernel(T* __restrict__ A, int64_t lda, int64_t ncols_total, int64_t c0, int w,
                   const LeafMoves* __restrict__ mv, int32_t* __restrict__ perm) {
  constexpr int MPL = 2 * kLeafMaxW / 32;  // moves per lane, at most
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nmv = min(mv->count, 2 * kLeafMaxW);  // no more, unless the panel gave up
  if (nmv == 0) return;
  int dst[MPL], src[MPL];
#pragma unroll
  for (int i = 0; i < MPL; ++i) {
    const int e = lane + 32 * i;
    const int2 x = e < nmv ? mv->mv[e] : make_int2(-1, 0);
    dst[i] = x.x;
    src[i] = x.y;
  }
  const int nl = (nmv + 31) >> 5;
  if (perm != nullptr && blockIdx.x == 0 && warp == 0) {
    // the row permutation (original row of each row) moves like one more column
    int32_t p[MPL];
#pragma unroll
    for (int i = 0; i < MPL; ++i)
      if (i < nl && dst[i] >= 0) p[i] = perm[src[i]];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < MPL; ++i)
      if (i < nl && dst[i] >= 0) perm[dst[i]] = p[i];
  }
  const int64_t nother = ncols_total - w;
  const int64_t stride = (int64_t)gridDim.x * 8;
  for (int64_t q = (int64_t)blockIdx.x * 8 + warp; q < nother; q += 2 * stride) {
    const int64_t q2 = q + stride;
    T* a = A + (q < c0 ? q : q + w) * lda;
    T* b = q2 < nother ? A + (q2 < c0 ? q2 : q2 + w) * lda : nullptr;
    T v[MPL], u[MPL];
#pragma unroll
    for (int i = 0; i < MPL; ++i) {
      if (i >= nl) break;
      v[i] = u[i] = T(0);
      if (dst[i] >= 0) {
        v[i] = a[src[i]];
        if (b) u[i] = b[src[i]];
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < MPL; ++i) {
      if (i >= nl) break;
      if (dst[i] >= 0) {
        a[dst[i]] = v[i];
        if (b) b[dst[i]] = u[i];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Unit-lower TRSM base case: B[0:k, cols] := L \ B with L = k x k (k <= KM,
// KM = 64 or 128) held in shared memory.  One warp per right-hand-side
// column: lane l holds rows l, l + 32, ... in registers; x_kk is broadcast
// with a shuffle and every row block from kk's on is updated, kk ascending
// (blocked_lufact.jl:146-178 order).  Nothing is masked: a row's value is
// kept aside when it is final (`own`), what its register goes through after
// that, and rows past k, are not used.
//
// Bound: FP64, the FP64 pipe for many columns (k = 128: 320 instructions a
// column, 16.5 cycles each on an SM) and the chain (a shuffle and an FP64
// instruction a step, 108 cycles) for few; FP32, the chain and the issue of 16
// warps.  All of a factorization's TRSM launches (events, ~5 us each of it
// launch), against one masked step at a time and 8-byte copies by as few as one
// warp: FP64 n = 1000 0.67 -> 0.40 ms, n = 8192 14.2 -> 9.2 ms, FP32 n = 3001
// 1.26 -> 0.87 ms.
constexpr int kTrsmMax = 128;
template <typename T>
__host__ __device__ constexpr int trsm_warps_max() { return sizeof(T) == 4 ? 16 : 8; }

template <typename T, int KM>
__global__ void __launch_bounds__(trsm_warps_max<T>() * 32)
trsm_lunit_kernel(const T* __restrict__ L, int64_t ldl, int k, T* __restrict__ B,
                  int64_t ldb, int64_t ncols) {
  constexpr int RPL = KM / 32;  // rows per lane
  constexpr int V = 16 / (int)sizeof(T);
  const int nw = (int)(blockDim.x >> 5);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T(*sL)[KM] = reinterpret_cast<T(*)[KM]>(smem_raw);  // sL[c][r] = L[r, c], r > c
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t stride = (int64_t)gridDim.x * nw;
  int64_t col = (int64_t)blockIdx.x * nw + warp;
  T v[RPL];
  auto load = [&](int64_t c) {
#pragma unroll
    for (int q = 0; q < RPL; ++q) v[q] = lane + 32 * q < k ? B[lane + 32 * q + c * ldb] : T(0);
  };
  // the columns below the diagonal, all copies in flight at once; in 16-byte
  // words where the block is aligned and no word reaches past row k - 1
  const bool vec = ((reinterpret_cast<uintptr_t>(L) | (uintptr_t)(ldl * (int64_t)sizeof(T))) & 15) == 0 && k % V == 0;
  if (vec) {
    constexpr int CPC = KM / V;  // words per column
    for (int idx = threadIdx.x; idx < k * CPC; idx += blockDim.x) {
      const int c = idx / CPC, r = (idx % CPC) * V;
      if (r + V > c + 1 && r < k) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(&sL[c][r]);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(L + r + (int64_t)c * ldl) : "memory");
      }
    }
  } else {
    for (int idx = threadIdx.x; idx < k * KM; idx += blockDim.x) {
      const int c = idx / KM, r = idx % KM;
      if (r > c && r < k) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(&sL[c][r]);
        if constexpr (sizeof(T) == 8)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(L + r + (int64_t)c * ldl) : "memory");
        else
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(L + r + (int64_t)c * ldl) : "memory");
      }
    }
  }
  if (col < ncols) load(col);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (; col < ncols; col += stride) {
#pragma unroll
    for (int b = 0; b < RPL; ++b) {
      if (32 * b >= k) break;
      T own = T(0);
      const int kend = min(32, k - 32 * b);
#pragma unroll 8
      for (int i = 0; i < 32; ++i) {
        if (i >= kend) break;
        const T x = __shfl_sync(0xffffffffu, v[b], i);
        own = lane == i ? x : own;
        const T* l = sL[32 * b + i] + lane;
#pragma unroll
        for (int q = b; q < RPL; ++q) {
          if (q > b && 32 * q >= k) break;
          v[q] = fma(-l[32 * q], x, v[q]);
        }
      }
      v[b] = own;
    }
    T* bc = B + col * ldb;
#pragma unroll
    for (int q = 0; q < RPL; ++q)
      if (lane + 32 * q < k) bc[lane + 32 * q] = v[q];
    if (col + stride < ncols) load(col + stride);
  }
}

template <typename T, int KM>
constexpr size_t trsm_smem() { return (size_t)KM * KM * sizeof(T); }

// ---------------------------------------------------------------------------
// TRSM base blocks of the 16-bit-operand factors (FP32 working matrix; the
// factors are refinement's preconditioner, not the reference's bit pattern):
// X = L^-1 of a unit-lower k x k diagonal block (k <= 128) once per getrf, then
// products with B, with no dependent chain of columns.
constexpr int kTinvLd = 128;       // leading dimension of a cached inverse

// Warp w of CTA b solves L x = e_j, j = 8 b + w (the TRSM chain, starting at row
// j: the inverse is lower triangular); column j of X, ld 128.  A CTA copies only
// the columns of L from its first on.  k a multiple of 4, L on 16 bytes.
constexpr int kTinvCols = 8;       // columns of the inverse per CTA
constexpr int kTinvLds = kTinvLd + 4;
__global__ void __launch_bounds__(32 * kTinvCols)
trsm_inv_kernel(const float* __restrict__ L, int64_t ldl, int k, float* __restrict__ X) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sL = reinterpret_cast<float*>(smem_raw);  // sL[c * kTinvLds + r] = L[r, c]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j0 = (int)blockIdx.x * kTinvCols;
  for (int i = threadIdx.x; i < (k - j0) * (kTinvLd / 4); i += 32 * kTinvCols) {
    const int c = j0 + i / (kTinvLd / 4), r = 4 * (i % (kTinvLd / 4));
    if (r + 3 > c && r < k) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(sL + c * kTinvLds + r);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(L + r + (int64_t)c * ldl) : "memory");
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int j = j0 + warp;
  if (j >= k) return;
  float v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = lane + 32 * q == j ? 1.f : 0.f;
#pragma unroll
  for (int qk = 0; qk < 4; ++qk) {
    if (32 * qk + 31 < j) continue;
    const int end = min(32 * qk + 32, k - 1);
#pragma unroll 4
    for (int kk = max(j, 32 * qk); kk < end; ++kk) {
      const float xk = __shfl_sync(0xffffffffu, v[qk], kk & 31);
#pragma unroll
      for (int q = qk; q < 4; ++q) {
        const int r = lane + 32 * q;
        if (r > kk && r < k) v[q] = fmaf(-sL[kk * kTinvLds + r], xk, v[q]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) X[lane + 32 * q + (int64_t)j * kTinvLd] = lane + 32 * q < k ? v[q] : 0.f;
}

// B (k x ncols, ldb) := L^-1 B for a unit-lower L of up to four 128-row blocks
// whose inverses are cached (the last may be shorter; k a multiple of 4): block
// after block, B_i - sum_j L_ij X_j, then its product with block i's inverse.
// The columns of B are independent, so a CTA keeps NC of them whole in shared
// memory and nothing crosses CTAs; 64-column tiles of L and of the inverses
// stream through a ring of three (32-column ones, twice the barriers: 4 % slower).  Thread (ty, tx): 4 rows x NC / 8 columns with
// 16-byte loads of both operands.
// In one launch for a triangle of 512 rows this replaces four products with
// inverses, two short SIMT updates and a tensor-core update with its operand
// conversions: BF16 n = 16384 48.1 -> 45.5 ms, FP16 without pivoting n = 6002
// 6.86 -> 6.11 ms.  Chains of 256 rows: 45.5 and 6.44 ms; of 1024, where the FP32
// products cost more than the tensor-core update's launches: 47.5 and 6.23 ms.
constexpr int kTrsmChain = 512;    // rows of a chain
constexpr int kChainK = 64;        // columns of a tile
constexpr int kChainStages = 3;
struct TrsmSlots { const float* p[kTrsmChain / kTinvLd]; };

template <int NC>
__global__ void __launch_bounds__(256)
trsm_chain_kernel(const float* __restrict__ L, int64_t ldl, int k, const __grid_constant__ TrsmSlots inv,
                  float* __restrict__ B, int64_t ldb, int64_t ncols) {
  constexpr int CPT = NC / 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sT = reinterpret_cast<float*>(smem_raw);        // [stage][column][128]
  float* sB = sT + kChainStages * kChainK * kTinvLd;     // sB[c * ldB + row]
  const int ldB = (k + 31) / 32 * 32 + 4;                // columns on different banks
  const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
  const int64_t cb = (int64_t)blockIdx.x * NC;
  const int nc = (int)min((int64_t)NC, ncols - cb);
  const int nblk = (k + kTinvLd - 1) / kTinvLd;
  auto cp = [](float* dst, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  };
  // tiles in order: block row i: L_i0 .. L_i,i-1, then the inverse; (i, j, q) is
  // the next one to copy
  int ii = 0, ij = 0, iq = 0, islot = 0;
  auto issue = [&]() {
    if (ii < nblk) {
      const int kb = min(kTinvLd, k - ii * kTinvLd), kc = ij < ii ? kTinvLd : kb;  // rows; columns of this block
      const int c0 = iq * kChainK, n = min(kChainK, kc - c0);
      float* dst = sT + islot * kChainK * kTinvLd;
      if (ij < ii) {
        const float* src = L + ii * kTinvLd + (int64_t)(ij * kTinvLd + c0) * ldl;
        for (int e = tid; e < n * (kTinvLd / 4); e += 256) {
          const int c = e / (kTinvLd / 4), r = 4 * (e % (kTinvLd / 4));
          if (r < kb) cp(dst + 4 * e, src + r + c * ldl);
        }
      } else {
        const float* src = inv.p[ii] + c0 * kTinvLd;
        for (int e = tid; e < n * (kTinvLd / 4); e += 256) {
          const int r = 4 * (e % (kTinvLd / 4));
          if (r + 3 >= c0) cp(dst + 4 * e, src + 4 * e);  // the rows above are zero
        }
      }
      islot = (islot + 1) % kChainStages;
      if (c0 + kChainK < kc) ++iq;
      else { iq = 0; if (ij < ii) ++ij; else { ij = 0; ++ii; } }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int e = tid; e < nc * (k / 4); e += 256) {
    const int c = e / (k / 4), r = 4 * (e % (k / 4));
    cp(sB + c * ldB + r, B + r + (cb + c) * ldb);
  }
#pragma unroll
  for (int t = 0; t < kChainStages - 1; ++t) issue();
  float acc[4][CPT];
  int slot = 0;
  // acc += sign * tile (columns 0 .. n - 1) * sB rows kbase ..
  auto product = [&](const float* tile, int kbase, int n, float sign) {
    const float* bp = sB + tx * ldB + kbase;
#pragma unroll (NC == 32 ? 2 : 4)
    for (int kk = 0; kk < n; kk += 4) {
      float4 b[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) b[c] = *reinterpret_cast<const float4*>(bp + 8 * c * ldB + kk);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 l = *reinterpret_cast<const float4*>(tile + (kk + q) * kTinvLd + 4 * ty);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const float x = sign * (q == 0 ? b[c].x : q == 1 ? b[c].y : q == 2 ? b[c].z : b[c].w);
          acc[0][c] = fmaf(l.x, x, acc[0][c]);
          acc[1][c] = fmaf(l.y, x, acc[1][c]);
          acc[2][c] = fmaf(l.z, x, acc[2][c]);
          acc[3][c] = fmaf(l.w, x, acc[3][c]);
        }
      }
    }
  };
  auto next_tile = [&]() -> const float* {
    asm volatile("cp.async.wait_group %0;" ::"n"(kChainStages - 2) : "memory");
    __syncthreads();  // this tile everywhere, the slot before it free
    issue();
    const float* t = sT + slot * kChainK * kTinvLd;
    slot = (slot + 1) % kChainStages;
    return t;
  };
  for (int i = 0; i < nblk; ++i) {
    const int kb = min(kTinvLd, k - i * kTinvLd);
    float* own = sB + tx * ldB + i * kTinvLd + 4 * ty;
    const bool on = 4 * ty < kb;  // kb is a multiple of 4
    if (i > 0) {
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        if (!on) break;
        const float4 v = *reinterpret_cast<const float4*>(own + 8 * c * ldB);
        acc[0][c] = v.x; acc[1][c] = v.y; acc[2][c] = v.z; acc[3][c] = v.w;
      }
      for (int j = 0; j < i * (kTinvLd / kChainK); ++j) {
        const float* t = next_tile();
        if (on) product(t, j * kChainK, kChainK, -1.f);
      }
      if (on)  // read by the others after the next tile's barrier
#pragma unroll
        for (int c = 0; c < CPT; ++c)
          *reinterpret_cast<float4*>(own + 8 * c * ldB) = make_float4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < CPT; ++c) acc[q][c] = 0.f;
    for (int c0 = 0; c0 < kb; c0 += kChainK) {
      const float* t = next_tile();
      // lower triangular: no columns past the thread's last row
      if (on) product(t, i * kTinvLd + c0, min(kChainK, 4 * ty + 4 - c0), 1.f);
    }
    __syncthreads();  // every thread has read block i's right-hand side
    if (on)
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        *reinterpret_cast<float4*>(own + 8 * c * ldB) = make_float4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
  }
  __syncthreads();
  for (int e = tid; e < nc * k; e += 256) {
    const int c = e / k, r = e % k;
    B[r + (cb + c) * ldb] = sB[c * ldB + r];
  }
}

constexpr size_t trsm_inv_smem() { return (size_t)kTinvLd * kTinvLds * sizeof(float); }
constexpr size_t trsm_chain_smem(int k, int nc) {
  return ((size_t)kChainStages * kChainK * kTinvLd + (size_t)nc * ((k + 31) / 32 * 32 + 4)) * sizeof(float);
}

// ---------------------------------------------------------------------------
// SIMT GEMM update C -= A * B (column-major), every C element updated by
// fma(-a_k, b_k, c) for k ascending.  BM x BN tile (64 x 64, 32 x 32 or
// 16 x 16), 16-deep k slices (FP32's small tiles: 32, fetched a slice ahead,
// FP32 n = 3001 5.84 -> 5.70 ms), 256 threads with a (BM/16) x (BN/16) register
// tile each.  The smaller tiles spread short updates over more SMs: one SM
// of this GPU retires two FP64 FMA lanes per cycle, so an update covered by
// a few 64 x 64 tiles would run on a few SMs.
constexpr int kGBK = 16;

template <typename T, int BM, int BN>
__global__ void __launch_bounds__(256, BM == 64 ? 2 : 4)
gemm_sub_kernel(int64_t M, int64_t N, int64_t K, const T* __restrict__ A, int64_t lda,
                const T* __restrict__ B, int64_t ldb, T* __restrict__ C, int64_t ldc) {
  constexpr int TM = BM / 16, TN = BN / 16;
  constexpr int BK = sizeof(T) == 4 && BM < 64 ? 2 * kGBK : kGBK;  // depth of a slice
  __shared__ T sA[BK][BM];
  __shared__ T sB[BK][BN + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
  T c[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int64_t r = m0 + tx + 16 * i, cc = n0 + ty + 16 * j;
      c[i][j] = (r < M && cc < N) ? C[r + cc * ldc] : T(0);
    }
  // this thread's share of a k slice, fetched into registers (FP32: while the
  // slice before it is used: short updates wait for their loads; in FP64 the
  // other CTAs' turns at the pipe hide them)
  constexpr int QA = (BK * BM) / 256, QB = (BK * BN) / 256;
  constexpr bool kAhead = sizeof(T) == 4;
  T pa[QA], pb[QB];
  auto fetch = [&](int64_t k0) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int idx = tid + 256 * q, kk = idx / BM, i = idx % BM;
      const int64_t r = m0 + i, kc = k0 + kk;
      pa[q] = (r < M && kc < K) ? A[r + kc * lda] : T(0);
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int idx = tid + 256 * q, kb = idx % BK, j = idx / BK;
      const int64_t kr = k0 + kb, cc = n0 + j;
      pb[q] = (kr < K && cc < N) ? B[kr + cc * ldb] : T(0);
    }
  };
  if (kAhead) fetch(0);
  for (int64_t k0 = 0; k0 < K; k0 += BK) {
    if (!kAhead) fetch(k0);
#pragma unroll
    for (int q = 0; q < QA; ++q) sA[(tid + 256 * q) / BM][(tid + 256 * q) % BM] = pa[q];
#pragma unroll
    for (int q = 0; q < QB; ++q) sB[(tid + 256 * q) % BK][(tid + 256 * q) / BK] = pb[q];
    __syncthreads();
    if (kAhead && k0 + BK < K) fetch(k0 + BK);
    const int kmax = (int)min((int64_t)BK, K - k0);
#pragma unroll (kAhead ? 4 : 1)
    for (int kk = 0; kk < kmax; ++kk) {
      T a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = sA[kk][tx + 16 * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = sB[kk][ty + 16 * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) c[i][j] = fma(-a[i], b[j], c[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int64_t r = m0 + tx + 16 * i, cc = n0 + ty + 16 * j;
      if (r < M && cc < N) C[r + cc * ldc] = c[i][j];
    }
}

// FP32 update with a 128 x 128 tile and an 8 x 8 register block per thread
// (rows tx*4 .. tx*4+3 and 64+tx*4 .. 64+tx*4+3, the same for columns), so
// each k step reads four float4 from shared memory for 64 FMAs; the next
// 8-deep k slice is fetched into registers while the current one is used.
// Every C element is loaded first and updated by fma(-a_k, b_k, c) for k
// ascending, as in gemm_sub_kernel.
constexpr int kRbK = 8;

__global__ void __launch_bounds__(256, 2)
gemm_sub_f32_rb_kernel(int64_t M, int64_t N, int64_t K, const float* __restrict__ A, int64_t lda,
                       const float* __restrict__ B, int64_t ldb, float* __restrict__ C, int64_t ldc) {
  constexpr int BM = 128, BN = 128, BK = kRbK;
  __shared__ __align__(16) float sA[BK][BM];      // sA[k][i] = A[m0 + i, k0 + k]
  __shared__ __align__(16) float sB[BK][BN + 4];  // sB[k][j] = B[k0 + k, n0 + j] (padded: conflict-free stores)
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
  float c[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t r = m0 + tx * 4 + (i & 3) + (i >> 2) * 64, cc = n0 + ty * 4 + (j & 3) + (j >> 2) * 64;
      c[i][j] = (r < M && cc < N) ? C[r + cc * ldc] : 0.f;
    }
  // this thread's share of a k slice: A elements (kk = idx / 128, i = idx % 128)
  // and B elements (kb = idx % 8, j = idx / 8) for idx = tid + 256 q, q < 4
  float pa[4], pb[4];
  auto fetch = [&](int64_t k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + 256 * q;
      const int kk = idx >> 7, i = idx & 127;
      const int64_t r = m0 + i, kc = k0 + kk;
      pa[q] = (r < M && kc < K) ? A[r + kc * lda] : 0.f;
      const int kb = idx & 7, j = idx >> 3;
      const int64_t kr = k0 + kb, cc = n0 + j;
      pb[q] = (kr < K && cc < N) ? B[kr + cc * ldb] : 0.f;
    }
  };
  auto stash = [&]() {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + 256 * q;
      sA[idx >> 7][idx & 127] = pa[q];
      sB[idx & 7][idx >> 3] = pb[q];
    }
  };
  fetch(0);
  stash();
  __syncthreads();
  for (int64_t k0 = 0; k0 < K; k0 += BK) {
    const bool more = k0 + BK < K;
    if (more) fetch(k0 + BK);  // in flight while this slice is used
    const int kmax = (int)min((int64_t)BK, K - k0);
    for (int kk = 0; kk < kmax; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(&sA[kk][tx * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&sA[kk][64 + tx * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&sB[kk][ty * 4]);
      const float4 b1 = *reinterpret_cast<const float4*>(&sB[kk][64 + ty * 4]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) c[i][j] = fmaf(-a[i], b[j], c[i][j]);
    }
    __syncthreads();
    if (more) {
      stash();
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t r = m0 + tx * 4 + (i & 3) + (i >> 2) * 64, cc = n0 + ty * 4 + (j & 3) + (j >> 2) * 64;
      if (r < M && cc < N) C[r + cc * ldc] = c[i][j];
    }
}

// The tile for an M x N update.  FP64: the least work on the busiest SM,
// ceil(tiles / SMs) x BM x BN, ties to the larger tile (the FP64 pipe is the
// bound: timing every update shape of the n = 8192 and 16384 recursions with
// each tile, this rule came within 0.1 % of the best tile per shape, and the
// smaller tiles' extra loads cost nothing measurable).  FP32: the largest of
// 128 x 128 (register-blocked kernel), 64 x 64, 32 x 32 whose tiles cover the
// SMs, else 16 x 16.
inline int gemm_tile_choice(int64_t M, int64_t N, int sms, int elem_size) {
  auto tiles = [&](int b) { return ((M + b - 1) / b) * ((N + b - 1) / b); };
  if (elem_size == 4) {
    if (tiles(128) >= sms) return 128;
    if (tiles(64) >= sms) return 64;
    if (tiles(32) >= sms) return 32;
    return 16;
  }
  const int bm[3] = {64, 32, 16};
  int best = 64;
  int64_t bt = 0;
  for (int q = 0; q < 3; ++q) {
    const int64_t t = (tiles(bm[q]) + sms - 1) / sms * bm[q] * bm[q];
    if (q == 0 || t < bt) { bt = t; best = bm[q]; }
  }
  return best;
}

// GBLU_GEMM_TILE=128|64|32|16 forces the SIMT update's tile (128: FP32 only,
// 64 for FP64; the tiles give
// identical results), so each variant can be tested on small matrices.
int forced_gemm_tile() {
  const char* e = getenv("GBLU_GEMM_TILE");
  if (!e) return 0;
  const int t = atoi(e);
  return (t == 128 || t == 64 || t == 32 || t == 16) ? t : 0;
}

// forced: 0 = gemm_tile_choice, else the tile edge (64, 32 or 16)
template <typename T>
void gemm_sub_launch(int64_t M, int64_t N, int64_t K, const T* A, int64_t lda, const T* B, int64_t ldb,
                     T* C, int64_t ldc, int sms, int forced, cudaStream_t s) {
  int t = forced ? forced : gemm_tile_choice(M, N, sms, (int)sizeof(T));
  if (t == 128 && sizeof(T) != 4) t = 64;
  dim3 grid((unsigned)((M + t - 1) / t), (unsigned)((N + t - 1) / t));
  if constexpr (std::is_same<T, float>::value) {
    if (t == 128) {
      gemm_sub_f32_rb_kernel<<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, ldc);
      return;
    }
  }
  if (t == 64) gemm_sub_kernel<T, 64, 64><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, ldc);
  else if (t == 32) gemm_sub_kernel<T, 32, 32><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, ldc);
  else gemm_sub_kernel<T, 16, 16><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, ldc);
}

// ---------------------------------------------------------------------------
// perm from ipiv: (P A)[i] = A[perm[i]].  One CTA; the interchanges are
// inherently sequential, the rest is parallel.
constexpr int kPermSmemMax = 48 * 1024;  // rows held in shared memory
constexpr int kPermChunk = 4096;         // pivots staged in shared memory at a time

__global__ void __launch_bounds__(1024)
perm_from_ipiv_kernel(const int64_t* __restrict__ ipiv, int64_t kmax, int64_t m,
                      int32_t* __restrict__ perm, DevScratch* __restrict__ scr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const bool in_smem = m <= kPermSmemMax;
  int32_t* st = reinterpret_cast<int32_t*>(smem_raw);  // kPermChunk pivot targets
  int32_t* sp = st + kPermChunk;
  int32_t* p = in_smem ? sp : perm;
  __shared__ int s_bad;
  for (int64_t i = threadIdx.x; i < m; i += blockDim.x) p[i] = (int32_t)i;
  if (threadIdx.x == 0) s_bad = 0;
  for (int64_t k0 = 0; k0 < kmax; k0 += kPermChunk) {
    const int kc = (int)min((int64_t)kPermChunk, kmax - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < kc; i += blockDim.x) {
      const int64_t t = ipiv[k0 + i] - 1;
      st[i] = (t < k0 + i || t >= m) ? -1 : (int32_t)t;
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_bad == 0) {
      for (int k = 0; k < kc; ++k) {  // the swaps in order, in shared memory only
        const int t = st[k];
        if (t < 0) { s_bad = 1; atomicCAS(&scr->error, 0, (int)DEV_BAD_PIVOT_INDEX); break; }
        const int64_t r = k0 + k;
        const int32_t x = p[r];
        p[r] = p[t];
        p[t] = x;
      }
    }
  }
  __syncthreads();
  if (in_smem)
    for (int64_t i = threadIdx.x; i < m; i += blockDim.x) perm[i] = sp[i];
}

__global__ void iota_kernel(int32_t* __restrict__ perm, int64_t m) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    perm[i] = (int32_t)i;
}

// ---------------------------------------------------------------------------
// Host driver

size_t getrf_scratch_bytes(int64_t m, int64_t n, int elem_size, int panel_width,
                           int device) {
  const DeviceInfo& di = device_info(device);
  size_t G = (size_t)di.num_sms * 8;  // upper bound on panel CTAs
  size_t b = 256;                     // DevScratch, aligned
  b += 2 * G * elem_size + 2 * G * sizeof(int64_t);
  b += 2 * G * kPanelMaxW * elem_size + 2 * kPanelMaxW * elem_size;
  b += sizeof(LeafMoves);
  return b + 2048;
}

template <typename T>
void getrf_carve(GetrfPlan<T>& p, void* base, size_t bytes, int device) {
  const DeviceInfo& di = device_info(device);
  size_t G = (size_t)di.num_sms * 8;
  char* c = reinterpret_cast<char*>(base);
  auto take = [&](size_t n) { char* r = c; c += (n + 255) & ~size_t(255); return r; };
  p.scratch = reinterpret_cast<DevScratch*>(take(sizeof(DevScratch)));
  p.slots.cand_val = reinterpret_cast<T*>(take(2 * G * sizeof(T)));
  p.slots.cand_row = reinterpret_cast<int64_t*>(take(2 * G * sizeof(int64_t)));
  p.slots.cand_rowvals = reinterpret_cast<T*>(take(2 * G * kPanelMaxW * sizeof(T)));
  p.slots.diag_rowvals = reinterpret_cast<T*>(take(2 * kPanelMaxW * sizeof(T)));
  p.moves = reinterpret_cast<LeafMoves*>(take(sizeof(LeafMoves)));
  (void)bytes;
}

namespace {

template <typename T>
int panel_max_blocks(size_t smem, int /*device*/) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, panel_kernel<T>, kPanelThreads, smem) !=
      cudaSuccess)
    return 0;
  return nb;
}

template <typename T>
struct Driver {
  const GetrfPlan<T>& p;
  cudaStream_t s;
  int device;
  cudaError_t err = cudaSuccess;
  int forced = 0;  // forced_panel_kind()
  int forced_tile = 0;  // forced_gemm_tile()
  // the TRSM inverse cache of this getrf: slot and order of the inverse kept
  // for the diagonal block starting at row 32 i (-1: none yet)
  std::vector<int> inv_slot, inv_k;
  int inv_next = 0;

  T* at(int64_t r, int64_t c) const { return p.A + r + c * p.lda; }

  void check(cudaError_t e) {
    if (err == cudaSuccess && e != cudaSuccess) err = e;
  }

  // Cluster panel when the whole panel fits in one cluster's shared memory and
  // each CTA's share of the rank-1 updates stays small; 0 if not launchable.
  bool panel_cluster(int64_t c0, int w) {
    const int64_t M = p.m - c0;
    const int64_t rmax = sizeof(T) == 4 ? 1536 : 192;  // rows per CTA
    int cs = (int)std::min<int64_t>(16, std::max<int64_t>(1, (M + 255) / 256));
    int64_t R = (M + cs - 1) / cs;
    if (R > rmax) return false;
    const size_t smem = (size_t)R * w * sizeof(T);
    if (!cluster_ok(cs, smem)) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(kPanelThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    double fl = 0;
    for (int k = 0; k < w; ++k) fl += (double)(M - k - 1) * (1.0 + 2.0 * (w - k - 1));
    LaunchScope ls(K_PANEL, fl, 2.0 * M * w * sizeof(T), s);
    check(cudaLaunchKernelEx(&cfg, panel_cluster_kernel<T>, p.A, p.lda, p.m, c0, w, p.ipiv, p.info,
                             (int)R));
    return true;
  }

  static bool cluster_ok(int cs, size_t smem) {
    static std::mutex mu;
    static int cache[17][2] = {};  // [cs][T] : 0 unknown, 1 ok, -1 no (per process, one device family)
    std::lock_guard<std::mutex> g(mu);
    int& c = cache[cs][sizeof(T) == 4 ? 0 : 1];
    if (c == 0) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(cs);
      cfg.blockDim = dim3(kPanelThreads);
      cfg.dynamicSmemBytes = (sizeof(T) == 4 ? 1536 : 192) * kPanelMaxW * sizeof(T);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = cs;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int nclusters = 0;
      cudaError_t e = cudaOccupancyMaxActiveClusters(&nclusters, panel_cluster_kernel<T>, &cfg);
      c = (e == cudaSuccess && nclusters >= 1) ? 1 : -1;
      cudaGetLastError();
    }
    (void)smem;
    return c == 1;
  }

  // Leaf width at row c0: the sub-panel kernel's where it takes the leaf
  // (0 in sub_width: it does not), else panel_width.
  int sub_width(int64_t c0) const {
    if (forced == 1 || forced == 2 || !p.use_sub_panel || !p.moves) return 0;
    if (std::is_same<T, float>::value && ((p.nopivot && p.tslu_work) || (p.tslu && p.tslu_work && p.m - c0 > 512))) return 0;
    return panel_sub_width<T>(device, p.m - c0);
  }
  int leaf_width(int64_t c0) const {
    if (std::is_same<T, float>::value && p.nopivot && p.tslu_work) return kGenpW;
    const int w = sub_width(c0);
    return w > 0 ? w : p.panel_width;
  }

  void panel(int64_t c0, int w) {
    const int64_t M = p.m - c0;
    const DeviceInfo& di = device_info(device);
    if constexpr (std::is_same<T, float>::value) {
      // random-butterfly-transformed factors: no pivot search, no interchanges
      if (p.nopivot && p.tslu_work) {
        // the leaf's kernels leave inverse_slot's inverse of L11 on the way
        float* linv = nullptr;
        if (p.trsm_inv && w == kGenpW && c0 + w < p.n && inv_next < p.trsm_inv_slots) {
          reserve_slots();
          inv_slot[(size_t)(c0 / 32)] = inv_next;
          inv_k[(size_t)(c0 / 32)] = kGenpW;
          linv = p.trsm_inv + (size_t)inv_next++ * kTinvLd * kTinvLd;
        }
        check(genp_panel_launch(p.A, p.lda, p.m, c0, w, p.ipiv, p.info, p.tslu_work, linv, s));
        return;
      }
      // low-precision factors: tournament pivoting for the tall leaves
      if (p.tslu && p.tslu_work && M > 512 && tslu_fits(M, w)) {
        check(tslu_panel_launch(p.A, p.lda, p.m, c0, w, p.ipiv, p.info, p.tslu_work, p.scratch, s));
        laswp(c0, w);
        return;
      }
    }
    // forced: 0 automatic, 1 grid kernel only, 2 shared-memory cluster kernel
    // where it fits, 3 sub-panel kernel where it fits (falling back in order)
    if (sub_width(c0) >= w) {
      check(panel_sub_launch<T>(p.A, p.lda, p.m, c0, w, p.ipiv, p.info, p.moves, p.scratch, s));
      laswp(c0, w, true);
      return;
    }
    if (forced != 1 && p.use_cluster_panel && panel_cluster(c0, w)) {
      laswp(c0, w);
      return;
    }
    int G = p.panel_ctas > 0 ? p.panel_ctas
                             : (int)std::max<int64_t>(1, (M + kPanelRowsTarget - 1) / kPanelRowsTarget);
    int R = (int)((M + G - 1) / G);
    size_t smem = (size_t)R * w * sizeof(T);
    const size_t smem_cap = std::min<size_t>(di.smem_optin, 200 * 1024);
    if (smem > smem_cap) {  // need more CTAs for this height
      int64_t rmax = (int64_t)(smem_cap / ((size_t)w * sizeof(T)));
      G = (int)((M + rmax - 1) / rmax);
      R = (int)((M + G - 1) / G);
      smem = (size_t)R * w * sizeof(T);
    }
    int per_sm = panel_max_blocks<T>(smem, device);
    int gmax = std::min(per_sm * di.num_sms, di.num_sms * 8);
    if (G > gmax) {
      G = gmax;
      R = (int)((M + G - 1) / G);
      smem = (size_t)R * w * sizeof(T);
      if (smem > smem_cap || G <= 0) { check(cudaErrorInvalidConfiguration); return; }
    }
    check(cudaMemsetAsync(&p.scratch->barrier, 0, sizeof(unsigned), s));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(kPanelThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    {
      double fl = 0;  // getf2 flops of the leaf: scale + rank-1 updates
      for (int k = 0; k < w; ++k) fl += (double)(M - k - 1) * (1.0 + 2.0 * (w - k - 1));
      LaunchScope ls(K_PANEL, fl, 2.0 * M * w * sizeof(T), s);
      check(cudaLaunchKernelEx(&cfg, panel_kernel<T>, p.A, p.lda, p.m, c0, w, p.ipiv, p.info,
                               p.scratch, p.slots, R));
    }
    laswp(c0, w);
  }

  // interchanges of the leaf on every other column
  // The leaf's interchanges on every other column, and on the row permutation
  // (so getrs can gather through it without replaying ipiv).
  // composed: by the moves the sub-panel kernel left, else from ipiv.
  void laswp(int64_t c0, int w, bool composed = false) {
    const DeviceInfo& di = device_info(device);
    const int64_t nother = p.n - w;
    // CTAs per SM (GBLU_LASWP_CTAS_PER_SM overrides).  Without composed moves
    // every CTA first turns the leaf's pivots into its row moves, so fewer CTAs
    // walking more columns each pay that once per SM rather than once per 8
    // columns.  With them 1, 2 and 4 are alike and 8 is a little slower (BF16,
    // n = 16384: 44.11, 44.13, 44.15 and 44.26 ms; FP64 n = 1000 and 8192 and
    // FP32 n = 3001 within 0.1 %).
    static const int64_t per_sm = [] {
      const char* e = getenv("GBLU_LASWP_CTAS_PER_SM");
      return e ? std::max<int64_t>(1, atoll(e)) : int64_t(4);
    }();
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((nother + 7) / 8, (int64_t)di.num_sms * per_sm));
    LaunchScope ls(K_LASWP, 0.0, 4.0 * w * std::max<int64_t>(nother, 0) * sizeof(T), s);
    if (composed) laswp_moves_kernel<T><<<blocks, 256, 0, s>>>(p.A, p.lda, p.n, c0, w, p.moves, p.perm);
    else laswp_leaf_kernel<T><<<blocks, 256, 0, s>>>(p.A, p.lda, p.m, p.n, c0, w, p.ipiv, p.scratch, p.perm);
    check(cudaGetLastError());
  }

  void gemm(int64_t M, int64_t N, int64_t K, const T* A, int64_t lda, const T* B, int64_t ldb,
            T* C, int64_t ldc) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    if constexpr (std::is_same<T, float>::value) {
      // the tensor-core path costs a conversion launch besides the GEMM:
      // updates with fewer than 256 rows or 128 columns stay on the SIMT
      // kernel (GBLU_TC_MIN_N overrides the column threshold; 64, 128, 256 and
      // 512 columns: BF16 n = 16384 44.25, 44.15, 44.61 and 45.87 ms, FP16
      // without pivoting n = 6002 5.35, 5.34, 5.42 and 5.69 ms)
      static const int64_t tc_min_n = [] {
        const char* e = getenv("GBLU_TC_MIN_N");
        return e ? std::max<int64_t>(1, atoll(e)) : int64_t(128);
      }();
      if (p.tc_mode != 0 && M >= 256 && N >= tc_min_n && K >= 64 &&
          tc_work_bytes(M, N, K) <= p.tc_work_bytes) {
        check(tc_gemm_sub(p.tc_mode, M, N, K, A, lda, B, ldb, C, ldc, p.tc_work, &p.scratch->error, s));
        return;
      }
    }
    LaunchScope ls(K_GEMM, 2.0 * M * N * K, (2.0 * M * N + (double)M * K + (double)K * N) * sizeof(T), s);
    gemm_sub_launch<T>(M, N, K, A, lda, B, ldb, C, ldc, device_info(device).num_sms, forced_tile, s);
    check(cudaGetLastError());
  }

  void reserve_slots() {
    if (!inv_slot.empty()) return;
    inv_slot.assign((size_t)(p.m / 32 + 2), -1);
    inv_k.assign(inv_slot.size(), 0);
  }

  // The cached inverse of the k x k diagonal block of L at row r0 (r0 a
  // multiple of 32): computed on first use in this getrf (the block is final
  // once the leaves covering it are done; a later getrf starts a new cache),
  // reused for any order up to k (the leading block of an inverse is the
  // inverse of the leading block).  Returns the slot, or -1 when full.
  int inverse_slot(int64_t r0, int64_t k) {
    reserve_slots();
    const size_t key = (size_t)(r0 / 32);
    if (key >= inv_slot.size()) return -1;
    if (inv_slot[key] >= 0 && inv_k[key] >= k) return inv_slot[key];
    int slot = inv_slot[key];
    if (slot < 0) {
      if (inv_next >= p.trsm_inv_slots) return -1;
      slot = inv_next++;
    }
    float* X = p.trsm_inv + (size_t)slot * kTinvLd * kTinvLd;
    LaunchScope ls(K_TRSM, (double)k * k * k / 3.0, ((double)k * k / 2 + (double)k * kTinvLd) * 4.0, s);
    trsm_inv_kernel<<<(unsigned)((k + kTinvCols - 1) / kTinvCols), 32 * kTinvCols, trsm_inv_smem(), s>>>(
        reinterpret_cast<const float*>(at(r0, r0)), p.lda, (int)k, X);
    check(cudaGetLastError());
    inv_slot[key] = slot;
    inv_k[key] = (int)k;
    return slot;
  }

  // The chain of inverses for a triangle of up to kTrsmChain rows; false when
  // the matrix is not aligned or the inverse cache is full.  Columns a CTA: more
  // read the tiles of L less often, fewer leave no SM idle; the widest that
  // gives half the SMs a CTA (32 only from one CTA an SM on: 2 % slower).
  bool trsm_chain(int64_t r0, int k, int64_t bc0, int64_t ncols) {
    if (((reinterpret_cast<uintptr_t>(at(r0, r0)) | reinterpret_cast<uintptr_t>(at(r0, bc0)) | (uintptr_t)(p.lda * 4)) & 15) != 0)
      return false;  // its copies are of 16 bytes
    TrsmSlots sl{};
    for (int i = 0; i * kTinvLd < k; ++i) {
      const int slot = inverse_slot(r0 + i * kTinvLd, std::min(kTinvLd, k - i * kTinvLd));
      if (slot < 0) return false;
      sl.p[i] = p.trsm_inv + (size_t)slot * kTinvLd * kTinvLd;
    }
    const int sms = device_info(device).num_sms;
    const int nc = ncols >= 16 * (int64_t)sms ? 32 : ncols >= 8 * (int64_t)sms ? 16 : 8;
    const unsigned grid = (unsigned)((ncols + nc - 1) / nc);
    LaunchScope ls(K_TRSM, (double)k * k * ncols, (2.0 * k * ncols + (double)k * k) * 4.0, s);
    auto* kern = nc == 32 ? trsm_chain_kernel<32> : nc == 16 ? trsm_chain_kernel<16> : trsm_chain_kernel<8>;
    kern<<<grid, 256, trsm_chain_smem(k, nc), s>>>(reinterpret_cast<const float*>(at(r0, r0)), p.lda, k, sl,
                                                   reinterpret_cast<float*>(at(r0, bc0)), p.lda, ncols);
    check(cudaGetLastError());
    return true;
  }

  // B (k x ncols at (r0, bc0)) := L \ B, L unit lower at (r0, r0) of size k.
  void trsm(int64_t r0, int64_t k, int64_t bc0, int64_t ncols) {
    if (k <= 0 || ncols <= 0) return;
    if constexpr (std::is_same<T, float>::value) {
      if (p.trsm_inv && k > 64 && k <= kTrsmChain && k % 4 == 0 && r0 % 32 == 0 && trsm_chain(r0, (int)k, bc0, ncols))
        return;
    }
    if (k <= p.trsm_base && k <= kTrsmMax) {
      const DeviceInfo& di = device_info(device);
      // One column per warp.  FP64: four warps saturate an SM's FP64 pipe while
      // they all issue; eight when the columns fill the SMs more than once
      // (their chains then overlap).  FP32: 16 where there are columns enough.
      const int64_t per_sm = (ncols + di.num_sms - 1) / di.num_sms;
      const int warps = sizeof(T) == 4 ? (per_sm > 8 ? 16 : 8) : (per_sm > 4 ? 8 : 4);
      unsigned blocks = (unsigned)std::min<int64_t>((ncols + warps - 1) / warps, (int64_t)di.num_sms * (k <= 64 ? 4 : 1));
      LaunchScope ls(K_TRSM, (double)k * (k - 1) * ncols, (2.0 * k * ncols + (double)k * k) * sizeof(T), s);
      if (k <= 64)
        trsm_lunit_kernel<T, 64><<<blocks, warps * 32, trsm_smem<T, 64>(), s>>>(
            at(r0, r0), p.lda, (int)k, at(r0, bc0), p.lda, ncols);
      else
        trsm_lunit_kernel<T, 128><<<blocks, warps * 32, trsm_smem<T, 128>(), s>>>(
            at(r0, r0), p.lda, (int)k, at(r0, bc0), p.lda, ncols);
      check(cudaGetLastError());
      return;
    }
    int64_t k1 = k / 2;
    // halves of whole blocks, so the cached inverses recur; of 32 rows where a
    // chain found no slots
    if (p.trsm_inv) {
      const int64_t g = k > kTrsmChain ? kTinvLd : 32;
      const int64_t a = (k1 + g - 1) / g * g;
      if (a < k) k1 = a;
    }
    trsm(r0, k1, bc0, ncols);
    gemm(k - k1, ncols, k1, at(r0 + k1, r0), p.lda, at(r0, bc0), p.lda, at(r0 + k1, bc0), p.lda);
    trsm(r0 + k1, k - k1, bc0, ncols);
  }

  void rec(int64_t c0, int64_t w) {
    const int wb = leaf_width(c0);
    if (w <= wb) {
      panel(c0, (int)w);
      return;
    }
    int64_t w1 = ((w / 2 + wb - 1) / wb) * wb;
    // whole blocks of the TRSM inverse cache (the leaf widths divide them), so
    // every triangle's blocks are the same ones
    if (p.trsm_inv && w1 > kTinvLd) w1 = (w1 + kTinvLd - 1) / kTinvLd * kTinvLd;
    if (w1 >= w) w1 = w - wb;
    rec(c0, w1);
    const int64_t c1 = c0 + w1, w2 = w - w1;
    trsm(c0, w1, c1, w2);
    gemm(p.m - c1, w2, w1, at(c1, c0), p.lda, at(c0, c1), p.lda, at(c1, c1), p.lda);
    rec(c1, w2);
  }
};

}  // namespace

cudaError_t simt_gemm_sub_f32(int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
                              const float* B, int64_t ldb, float* C, int64_t ldc, cudaStream_t s) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
  int device = 0;
  cudaGetDevice(&device);
  LaunchScope ls(K_GEMM, 2.0 * M * N * K, (2.0 * M * N + (double)M * K + (double)K * N) * 4.0, s);
  gemm_sub_launch<float>(M, N, K, A, lda, B, ldb, C, ldc, device_info(device).num_sms, forced_gemm_tile(), s);
  return cudaGetLastError();
}

cudaError_t perm_build_launch(const int64_t* ipiv, int64_t kmax, int64_t m, int32_t* perm,
                              DevScratch* scr, cudaStream_t s) {
  size_t smem = (size_t)kPermChunk * sizeof(int32_t) + (m <= kPermSmemMax ? (size_t)m * sizeof(int32_t) : 0);
  LaunchScope ls(K_PERM, 0.0, 8.0 * kmax + 4.0 * m, s);
  perm_from_ipiv_kernel<<<1, 1024, smem, s>>>(ipiv, kmax, m, perm, scr);
  return cudaGetLastError();
}

int trsm_inv_slot_count(int64_t n) { return (int)(n / 64 + 8); }
size_t trsm_inv_bytes(int64_t n) {
  return (size_t)trsm_inv_slot_count(n) * kTinvLd * kTinvLd * sizeof(float);
}

void getrf_configure(int device) {
  cudaFuncSetAttribute(trsm_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)trsm_inv_smem());
  cudaFuncSetAttribute(trsm_chain_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_chain_smem(kTrsmChain, 32));
  cudaFuncSetAttribute(trsm_chain_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_chain_smem(kTrsmChain, 16));
  cudaFuncSetAttribute(trsm_chain_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_chain_smem(kTrsmChain, 8));
  const DeviceInfo& di = device_info(device);
  const int cap = (int)std::min<size_t>(di.smem_optin, 200 * 1024);
  cudaFuncSetAttribute(panel_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(panel_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(panel_cluster_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(panel_cluster_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
  cudaFuncSetAttribute(panel_cluster_kernel<double>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaFuncSetAttribute(panel_cluster_kernel<float>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  panel_sub_configure<double>(device);
  panel_sub_configure<float>(device);
  cudaFuncSetAttribute(trsm_lunit_kernel<double, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_smem<double, 128>());
  cudaFuncSetAttribute(trsm_lunit_kernel<float, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_smem<float, 128>());
  cudaFuncSetAttribute(trsm_lunit_kernel<double, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)trsm_smem<double, 64>());
  cudaFuncSetAttribute(perm_from_ipiv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (kPermSmemMax + kPermChunk) * (int)sizeof(int32_t));
  getrs_configure(device);
  tc_configure(device);
  tslu_configure(device);
  genp_configure(device);
}

// GBLU_PANEL=grid|cluster|reg forces one panel kernel (reg: the sub-panel kernel) (where the panel fits
// it; the kernels give identical results), so every variant can be tested on
// small matrices.  Read at each factorization.
int forced_panel_kind() {
  const char* e = getenv("GBLU_PANEL");
  if (!e) return 0;
  if (!strcmp(e, "grid")) return 1;
  if (!strcmp(e, "cluster")) return 2;
  if (!strcmp(e, "reg")) return 3;
  return 0;
}

template <typename T>
cudaError_t getrf_launch(const GetrfPlan<T>& p, cudaStream_t stream) {
  int device = 0;
  cudaGetDevice(&device);
  Driver<T> d{p, stream, device};
  d.forced = forced_panel_kind();
  d.forced_tile = forced_gemm_tile();
  const int64_t minmn = std::min(p.m, p.n);
  d.check(cudaMemsetAsync(p.info, 0, sizeof(int64_t), stream));
  if (minmn > 0) {
    {
      LaunchScope ls(K_PERM, 0.0, 4.0 * p.m, stream);
      iota_kernel<<<(unsigned)std::min<int64_t>((p.m + 255) / 256, 1024), 256, 0, stream>>>(p.perm, p.m);
      d.check(cudaGetLastError());
    }
    d.rec(0, minmn);  // each leaf's laswp also permutes p.perm
    if (p.n > p.m) d.trsm(0, p.m, p.m, p.n - p.m);  // wide: U12 := L11 \ A12
  }
  return d.err;
}

template cudaError_t getrf_launch<double>(const GetrfPlan<double>&, cudaStream_t);
template cudaError_t getrf_launch<float>(const GetrfPlan<float>&, cudaStream_t);
template void getrf_carve<double>(GetrfPlan<double>&, void*, size_t, int);
template void getrf_carve<float>(GetrfPlan<float>&, void*, size_t, int);

}  // namespace gblu
