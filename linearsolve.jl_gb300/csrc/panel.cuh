// Sub-panel cluster kernel: getf2 of one leaf (rows [c0, m) x columns
// [c0, c0 + w)), the leaf in the shared memory of one thread-block cluster
// and eight columns at a time in registers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "device_util.cuh"
#include "waits.cuh"
#include "gblu_internal.h"

namespace gblu {

constexpr int kSubW = 8;          // columns of a sub-panel
constexpr int kSubMaxCtas = 16;
constexpr unsigned long long kPushLandNs = 100000;  // a push takes about a microsecond

// The value whose bit pattern is the key (|a| for a key of a)
template <typename T>
__device__ __forceinline__ T key_magnitude(typename PivKey<T>::K key) {
  if constexpr (sizeof(T) == 4) return __uint_as_float(key);
  else return __longlong_as_double((long long)key);
}

// RN(1 / x) of a positive normal x whose reciprocal is normal, in integer
// arithmetic without a branch.  The library division is a chain of dependent
// FP64 instructions (about 70 cycles each here, 600 in place) behind a branch
// the scheduler cannot move a warp reduction across; this takes about 230 and
// interleaves.  The quotient's last unit and its rounding are settled by the
// exact remainder modulo 2^64 (it is smaller than four divisors).  A tie
// cannot occur: 2^k = m (2 q + 1) only for m = 1.
__device__ __forceinline__ double recip_normal(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int e = (int)(b >> 52);
  unsigned long long q = recip_word(m) >> 11;       // ~ 2^105 / m
  long long rem = -(long long)(q * m);              // 2^105 - q m
  const long long ms = (long long)m;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const bool neg = rem < 0, big = rem >= ms;
    q += big ? 1ull : (neg ? ~0ull : 0ull);
    rem += big ? -ms : (neg ? ms : 0ll);
  }
  q += 2 * rem > ms ? 1ull : 0ull;
  // 1 / x = q 2^-105 2^(1075 - e) with q in [2^52, 2^53]: biased exponent 2045 - e, + 1 at q = 2^53
  return __longlong_as_double((long long)(((unsigned long long)(unsigned)(2045 - e) << 52) + (q - (1ull << 52))));
}
__device__ __forceinline__ float recip_normal(float x) {
  const unsigned b = __float_as_uint(x);
  const int m = (int)((b & 0x7FFFFFu) | 0x800000u);
  const unsigned e = b >> 23;
  float y;                                          // ~ 1 / (m 2^-23), in [1/2, 1], within 2^-23 of it
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3F800000u | (b & 0x7FFFFFu))));
  const unsigned q = __float_as_uint(y) - (125u << 23);  // y 2^24 ~ 2^47 / m
  const int r2 = -2 * (int)(q * (unsigned)m);       // 2 (2^47 - q m): at most three units off
  int d = 0;                                        // round(rem / m)
  d += r2 > m;
  d += r2 > 3 * m;
  d += r2 > 5 * m;
  d -= r2 < -m;
  d -= r2 < -3 * m;
  d -= r2 < -5 * m;
  return __uint_as_float(((253u - e) << 23) + (q + (unsigned)d - 0x800000u));  // as above
}
// the biased exponents recip_normal takes: x and 1 / x normal
template <typename T>
__device__ __forceinline__ bool recip_in_range(T x) {
  if constexpr (sizeof(T) == 4) return (__float_as_uint(x) >> 23) - 1u < 251u;
  else return ((unsigned)((unsigned long long)__double_as_longlong(x) >> 52)) - 1u < 2043u;
}

// x with the sign of s (bit operations only)
template <typename T>
__device__ __forceinline__ T with_sign_of(T x, T s) {
  if constexpr (sizeof(T) == 4)
    return __uint_as_float(__float_as_uint(x) ^ (__float_as_uint(s) & 0x80000000u));
  else
    return __longlong_as_double(__double_as_longlong(x) ^
                                (__double_as_longlong(s) & (long long)0x8000000000000000ull));
}

// 16-byte words of T
template <typename T>
struct Word {
  static constexpr int N = 16 / (int)sizeof(T);
  static __device__ __forceinline__ int4 pack(const T* x) {
    if constexpr (sizeof(T) == 4)
      return make_int4(__float_as_int(x[0]), __float_as_int(x[1]), __float_as_int(x[2]), __float_as_int(x[3]));
    else
      return make_int4(__double2loint(x[0]), __double2hiint(x[0]), __double2loint(x[1]), __double2hiint(x[1]));
  }
  static __device__ __forceinline__ void unpack(T* x, const int4& v) {
    if constexpr (sizeof(T) == 4) {
      x[0] = __int_as_float(v.x); x[1] = __int_as_float(v.y); x[2] = __int_as_float(v.z); x[3] = __int_as_float(v.w);
    } else {
      x[0] = __hiloint2double(v.y, v.x); x[1] = __hiloint2double(v.w, v.z);
    }
  }
};
template <typename T, int L>
__device__ __forceinline__ void words_store(T* dst, const T (&src)[L]) {
#pragma unroll
  for (int q = 0; q < L / Word<T>::N; ++q) reinterpret_cast<int4*>(dst)[q] = Word<T>::pack(&src[q * Word<T>::N]);
}
template <typename T, int L>
__device__ __forceinline__ void words_load(T (&dst)[L], const T* src) {
#pragma unroll
  for (int q = 0; q < L / Word<T>::N; ++q)
    Word<T>::unpack(&dst[q * Word<T>::N], reinterpret_cast<const int4*>(src)[q]);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// f(integral_constant r) for the r in [LO, HI) equal to the warp-uniform rr: a
// tree of uniform branches, so registers indexed by r stay registers.
template <int LO, int HI, typename F>
__device__ __forceinline__ void with_slot(int rr, F&& f) {
  if constexpr (HI - LO == 1) {
    f(std::integral_constant<int, LO>{});
  } else {
    constexpr int MID = (LO + HI) / 2;
    if (rr < MID) with_slot<LO, MID>(rr, f);
    else with_slot<MID, HI>(rr, f);
  }
}

// Pivot choice over a warp: every lane holds a candidate (key v, 0 = none; row
// g >= 0); on return every lane holds the largest key and the smallest row
// with it (g meaningless when v == 0).
template <typename K>
__device__ __forceinline__ void warp_max_row(K& v, unsigned& g) {
  constexpr unsigned kAll = 0xffffffffu;
  if constexpr (sizeof(K) == 4) {
    const unsigned mk = __reduce_max_sync(kAll, (unsigned)v);
    g = __reduce_min_sync(kAll, (unsigned)v == mk ? g : 0xffffffffu);
    v = mk;
  } else {
    const unsigned hi = (unsigned)((unsigned long long)v >> 32), lo = (unsigned)v;
    const unsigned mh = __reduce_max_sync(kAll, hi);
    const unsigned ml = __reduce_max_sync(kAll, hi == mh ? lo : 0u);
    g = __reduce_min_sync(kAll, (hi == mh && lo == ml) ? g : 0xffffffffu);
    v = (K)(((unsigned long long)mh << 32) | ml);
  }
}

template <typename T, int W>
__host__ __device__ constexpr int panel_sub_ld() { return W + 16 / (int)sizeof(T); }

// getf2 of rows [c0, m) x columns [c0, c0 + w), w <= W, by one cluster of G
// CTAs; CTA c holds rows c R .. c R + R - 1 of the leaf in shared memory,
// row-major (16-byte words of a row move as units; the padding word makes a
// column of words conflict-free).  Per sub-panel of eight columns:
//   * NWC chain warps hold the eight columns in registers (RPT rows a thread).
//     Per column: each warp reduces its candidate; warp 0 pushes the CTA's
//     candidate, its row and (its owner) the diagonal row into every CTA's
//     receive slots with st.async, counted by that column's mbarrier; every
//     chain warp waits for them, picks the winner itself and scales and
//     updates its rows.  Receive slots are double-buffered by column parity: a
//     CTA pushes column k + 2 only after it received every column k + 1, and a
//     CTA pushes column k + 1 only after its chain warps finished column k.
//   * boundary: the CTAs that hold moved rows push their other columns' words
//     to where they end (counted by a third mbarrier, so no cluster barrier);
//     every CTA solves U12 for itself, all warps update the next sub-panel's
//     columns, and the helper warps (NW - NWC) the rest beside its chain.
// Every element receives its updates for k ascending, multipliers are
// a * RN(1 / pivot): bit-identical to panel_kernel.
//
// What bounds it is the chain of dependent steps of a column, not arithmetic
// or memory (cycles in place, FP32, 16 CTAs, 1000 rows: candidate and
// reduction 90, packet 120, push and exchange 600, winner and its row 300,
// update 100; FP64 adds the reciprocal and 68 cycles an FP64 instruction), then
// the boundaries (about 3000 cycles each).  Eight columns and not the whole
// leaf in registers: a column's exchange carries 8 values of a row instead of
// 32, its update is short, and the bulk of the update leaves the chain.
// Measured per leaf of 32 columns, launch included, against the kernel this
// replaced (whole rows in registers, one exchange of whole rows a column, a
// CTA barrier and a separate reciprocal warp): FP64 96 rows 75 -> 47 us, 512
// 77 -> 47, 1000 77 -> 53, 2000 78 -> 61, 4000 88 -> 80, 8000 121 -> 118; FP32
// 128 rows 46 -> 24, 1000 46 -> 32, 3000 47 -> 37, 8000 55 -> 44, 16000 61 -> 55.
template <typename T, int NT, int NWC, int RPT, int W>
__global__ void __launch_bounds__(NT, 1)
panel_sub_kernel(T* __restrict__ A, int64_t lda, int64_t m, int64_t c0, int w, int64_t* __restrict__ ipiv,
                 int64_t* __restrict__ info_out, int R, unsigned rmagic, LeafMoves* __restrict__ moves,
                 DevScratch* __restrict__ scr) {
  using K = typename PivKey<T>::K;
  using WD = Word<T>;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NW = NT / 32, NC = 32 * NWC, NB = kSubW, LD = panel_sub_ld<T, W>();
  constexpr int RB = NB / WD::N;                 // 16-byte words of a sub-panel row
  // a candidate's packet: key, row | its row | FP64: 1 / |key|
  constexpr int PW = sizeof(T) == 4 ? 1 + RB : 2 + RB;
  constexpr int NMV = 2 * NB;                    // rows a sub-panel's interchanges touch, at most
  constexpr int NU = (NB * (W - NB) + NT - 1) / NT;  // U12 elements per thread
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // row i at tile + i * LD: the leaf's columns, then a word with the row the
  // content came from
  T* tile = reinterpret_cast<T*>(smem_raw);
  __shared__ __align__(16) int4 r_pkt[2][kSubMaxCtas][PW];  // received: CTA c's candidate
  __shared__ __align__(16) T r_diag[2][NB];               // received: the diagonal row
  __shared__ __align__(16) T r_mv[NMV][LD];               // received: moved rows
  // received: A12; then U12 (leaf columns).  Two, by sub-panel parity: the next
  // A12 may arrive while the helper warps still read this U12
  __shared__ __align__(16) T s_Ub[2][NB][W];
  __shared__ __align__(8) unsigned long long r_bar[3];    // count the received bytes: a column's (two), a boundary's
  __shared__ __align__(16) int4 s_pkt[2][NWC][PW];        // each chain warp's candidate
  __shared__ __align__(16) T s_diag[2][NB];               // the diagonal row, in its owner CTA
  __shared__ __align__(16) T s_prow[NB][NB];              // the sub-panel's rows: L11 \ U11
  __shared__ int s_mrow[NMV], s_mfrom[NMV];               // moved rows and their sources (-1: none)

  uint32_t nctas, rank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(nctas));
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int G = (int)nctas, cta = (int)rank;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = (int)(m - c0);
  const int lo = cta * R;                          // this CTA's rows: lo .. lo + nloc - 1 of the leaf
  const int nloc = max(0, min(R, M - lo));
  T* Ab = A + c0 + c0 * lda;                       // the leaf's first element
  const uint32_t rx_bytes = (uint32_t)(G * 16 * PW + 16 * RB);
  int* const err = &scr->error;
  // set once a wait gave up: stop waiting, finish without hanging
  int me = threadIdx.x;  // -1 then
  auto owner = [&](int row) { return (int)__umulhi((unsigned)row, rmagic); };  // row / R

  // the leaf into the tile: units of 32 rows x one 16-byte word of columns
  const int nrg = (nloc + 31) >> 5, nwd = (w + WD::N - 1) / WD::N;
#pragma unroll 4
  for (int t = warp; t < nrg * nwd; t += NW) {
    const int wd = t / nrg, i = (t - wd * nrg) * 32 + lane;
    if (i < nloc) {
      T x[WD::N];
#pragma unroll
      for (int q = 0; q < WD::N; ++q) {
        const int c = wd * WD::N + q;
        x[q] = c < w ? Ab[lo + i + (int64_t)c * lda] : T(0);
      }
      *reinterpret_cast<int4*>(tile + i * LD + wd * WD::N) = WD::pack(x);
    }
  }
  for (int i = tid; i < nloc; i += NT) *reinterpret_cast<int*>(tile + i * LD + W) = lo + i;
  if (cta == 0 && tid == 0) moves->count = 0;
  if (G > 1) {
    if (tid == 0) {
      for (int q = 0; q < 3; ++q) pan_bar_init(pan_saddr(&r_bar[q]));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      pan_bar_arm(pan_saddr(&r_bar[0]), rx_bytes);  // column 0
      pan_bar_arm(pan_saddr(&r_bar[1]), rx_bytes);  // column 1
    }
    __syncwarp();
    cluster_arrive();  // every CTA's mbarriers exist before the first push
    cluster_wait();
  }
  __syncthreads();
  int64_t info_local = 0;
  // lanes c and c + 16 of warp 0 push to CTA c
  const int pc = lane & 15, ph = lane >> 4;
  uint32_t p_bar = 0, p_pkt = 0, p_diag = 0;
  if (pc < G) {
    p_bar = pan_mapa(pan_saddr(&r_bar[0]), pc);
    p_pkt = pan_mapa(pan_saddr(&r_pkt[0][cta][0]), pc);
    p_diag = pan_mapa(pan_saddr(&r_diag[0][0]), pc);
  }

  for (int s0 = 0; s0 < w; s0 += NB) {
    const int kb = min(NB, w - s0);
    const int c1 = s0 + kb;
    T(*s_U)[W] = s_Ub[(s0 / NB) & 1];
    if (warp < NWC) {
      T pr[RPT][NB];
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int i = tid + NC * r;
        if (i < nloc) words_load<T, NB>(pr[r], tile + i * LD + s0);
        else
#pragma unroll
          for (int j = 0; j < NB; ++j) pr[r][j] = T(0);
      }
      // the interchanges of this sub-panel, composed as they come: lane e < 16
      // holds a touched row and the row its value comes from
      int mrow = lane < kb ? s0 + lane : -1, mfrom = mrow;
      int piv_row = 0;    // lane j: the pivot row of column s0 + j
      auto compose = [&](int j) {  // column s0 + j's interchange
        const int p = __shfl_sync(kAll, piv_row, j);
        const unsigned hm = __ballot_sync(kAll, mrow == p);
        if (hm == 0u && lane == NB + j) mrow = mfrom = p;
        const int hb = hm ? __ffs(hm) - 1 : NB + j;
        mfrom = __shfl_sync(kAll, mfrom, lane == j ? hb : (lane == hb ? j : lane));
      };
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        if (j >= kb) break;
        const int k = s0 + j, b = k & 1;
        // 1. candidates of column k: each warp's first row of max |a|.  Rows
        // above the diagonal are among the leaf's first W (the other slots
        // need no test); slots past the last row hold zeros or NaN, which are
        // never candidates.
        K v = 0;
        unsigned g = 0;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
          const int gi = lo + tid + NC * r;
          K kv = PivKey<T>::of(pr[r][j]);
          if (NC * r < W && gi < k) kv = 0;
          if (r == 0 || kv > v) { v = kv; g = (unsigned)gi; }
        }
        const unsigned mine = g;
        // FP64: 1 / |candidate| of every lane, beside the reduction and the rest
        // of the previous column's update
        T rinv = T(0);
        if (sizeof(T) == 8) rinv = recip_normal(key_magnitude<T>(v));
        warp_max_row(v, g);
        const int ld = k - lo;  // the diagonal row here
        const bool own_diag = ld >= 0 && ld < nloc;
        with_slot<0, RPT>(RPT > 1 ? ((int)g - lo) / NC : 0, [&](auto r) {
          if (mine == g) {
            int4* sp = s_pkt[b][warp];
            if constexpr (sizeof(T) == 4) {
              sp[0] = make_int4((int)v, (int)g, 0, 0);
            } else {
              sp[0] = make_int4((int)(unsigned)v, (int)(unsigned)(v >> 32), (int)g, 0);
              sp[1 + RB] = make_int4(__double2loint(rinv), __double2hiint(rinv), 0, 0);
            }
            words_store<T, NB>(reinterpret_cast<T*>(sp + 1), pr[decltype(r)::value]);
          }
        });
        if (own_diag) {
#pragma unroll
          for (int r = 0; r < RPT; ++r)
            if (NC * r < W && tid + NC * r == ld) words_store<T, NB>(s_diag[b], pr[r]);
        }
        if constexpr (NWC > 1) named_bar_sync(1, NC);
        else __syncwarp();
        const int4* pk = s_pkt[b][0];
        // the best of the n <= 16 candidates c[l * PW] (n a power of two or
        // lanes clamped): key, row, where; FP32: its reciprocal
        auto choose = [&](const int4* c, int l) {
          const int4 w0 = c[l * PW];
          int gr;
          if constexpr (sizeof(T) == 4) { v = (K)(unsigned)w0.x; gr = w0.y; }
          else { v = ((K)(unsigned)w0.y << 32) | (K)(unsigned)w0.x; gr = w0.z; }
          T lr = T(0);
          if (sizeof(T) == 4) lr = recip_normal(key_magnitude<T>(v));
          g = (unsigned)gr * 16u + (unsigned)l;
          warp_max_row(v, g);
          pk = c + (g & 15u) * PW;
          if (sizeof(T) == 4) rinv = __shfl_sync(kAll, lr, g & 15u);
          g >>= 4;
        };
        if (NWC > 1 && (G == 1 || warp == 0)) choose(s_pkt[b][0], lane & (NWC - 1));  // the CTA's candidate
        else if (sizeof(T) == 4 && G == 1) rinv = recip_normal(key_magnitude<T>(v));
        const T* drow = s_diag[b];
        if (G > 1) {
          // 2. warp 0 pushes the CTA's candidate and the diagonal row to every CTA
          if (warp == 0) {
            if (pc < G) {
              const uint32_t bar = p_bar + 8u * b, dst = p_pkt + (uint32_t)(b * sizeof(r_pkt[0]));
#pragma unroll
              for (int q = 0; q < PW; q += 2)
                if (q + 1 < PW || ph == 0) pan_st_async(dst + 16u * (q + ph), pk[q + ph], bar);
              if (own_diag) {
                const uint32_t dd = p_diag + (uint32_t)(b * sizeof(r_diag[0]));
                const int4* ds = reinterpret_cast<const int4*>(s_diag[b]);
#pragma unroll
                for (int q = 0; q < RB; q += 2) pan_st_async(dd + 16u * (q + ph), ds[q + ph], bar);
              }
            }
            if (j > 0) compose(j - 1);  // while the candidates travel
          }
          // 3. the winner over the CTAs
          if (me >= 0 && !pan_bar_wait(pan_saddr(&r_bar[b]), (uint32_t)(k >> 1) & 1u, err)) me = -1;
          choose(r_pkt[b][0], pc < G ? pc : 0);
          drow = r_diag[b];
          if (me == 0 && k + 2 < w) pan_bar_arm(pan_saddr(&r_bar[b]), rx_bytes);  // column k + 2
        } else if (j > 0 && warp == 0) {
          compose(j - 1);
        }
        T pv[NB], dv[NB];       // the pivot row, the diagonal row
        words_load<T, NB>(dv, drow);
        words_load<T, NB>(pv, reinterpret_cast<const T*>(pk + 1));
        if constexpr (sizeof(T) == 8) rinv = __hiloint2double(pk[1 + RB].y, pk[1 + RB].x);
        const bool none = v == 0;  // zero or NaN from the diagonal down: kp = k
        const int p = none ? k : (int)g;
        T inv;
        bool nz = true;
        if (none || !recip_in_range(key_magnitude<T>(v))) {
          if (none) {  // the pivot is the diagonal entry, zero or NaN
#pragma unroll
            for (int q = 0; q < NB; ++q) pv[q] = dv[q];
            nz = PivKey<T>::nonzero(pv[j]);
            if (!nz && info_local == 0) info_local = c0 + k + 1;
          }
          inv = T(1) / (nz ? pv[j] : T(1));
        } else {
          inv = with_sign_of(rinv, pv[j]);
        }
        piv_row = lane == j ? p : piv_row;
        if (warp == 0) words_store<T, NB>(s_prow[j], pv);  // final; every lane the same words
        // 4. interchange (p != k implies a nonzero pivot): row p receives the
        // diagonal row.  Row k is final (s_prow); the registers of finished
        // rows are updated too and not used again, so nothing is masked.
        if (RPT == 1) {
          const bool isp = lo + tid == p && tid < nloc;
#pragma unroll
          for (int q = 0; q < NB; ++q) pr[0][q] = isp ? dv[q] : pr[0][q];
        } else {
          const int lp = p - lo;
          if (lp >= 0 && lp < nloc && ((lp & (NC - 1)) >> 5) == warp)
            with_slot<0, RPT>(lp / NC, [&](auto r) {
              const bool isp = (lp & 31) == lane;
#pragma unroll
              for (int q = 0; q < NB; ++q)
                pr[decltype(r)::value][q] = isp ? dv[q] : pr[decltype(r)::value][q];
            });
        }
        // scale, update (the next column first)
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
          // FP64: slots without rows below the diagonal stay off the FP64 pipe
          const int wr = warp * 32 + NC * r;
          if (sizeof(T) == 8 && (RPT > 1 || NWC > 1) && (wr >= nloc || lo + wr + 31 <= k)) continue;
          const T l = nz ? pr[r][j] * inv : pr[r][j];
          pr[r][j] = l;
#pragma unroll
          for (int q = j + 1; q < NB; ++q) pr[r][q] = fma(-l, pv[q], pr[r][q]);
        }
      }
      // the rows below the sub-panel back to the tile, and the moves
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int i = tid + NC * r;
        if (i < nloc && lo + i >= c1) words_store<T, NB>(tile + i * LD + s0, pr[r]);
      }
      if (warp == 0) {
        compose(kb - 1);  // the last column's interchange
        if (lane < NMV) {
          // rows of the leaf, also where a wait gave up and a packet was none
          s_mrow[lane] = min(mrow, M - 1);
          s_mfrom[lane] = min(mfrom, M - 1);
        }
      }
      if (warp == NWC - 1 && cta == 0 && lane < kb) ipiv[c0 + s0 + lane] = c0 + min(piv_row, M - 1) + 1;
    }
    __syncthreads();  // the sub-panel, its moves and the helpers' updates are in shared memory
    // 5. the interchanges on the leaf's other columns, a 16-byte word a thread.
    // The CTA that holds a moved row pushes its words to the CTA where it ends;
    // rows that become rows of the sub-panel go, right of it, to every CTA
    // (A12: each CTA computes U12 for itself).
    const int nright = w - c1, nleftw = s0 / WD::N, nrw = (nright + WD::N - 1) / WD::N;
    constexpr int MW = (W - NB) / WD::N + 1;      // words of a row outside the sub-panel and the id's, at most
    constexpr int MWP = MW <= 8 ? 8 : MW <= 16 ? 16 : 32;
    constexpr int MI = (NMV * MWP + NT - 1) / NT;  // moved words a thread
    // word 0: the id; then the words left of the sub-panel, then right of it
    auto moved_word = [&](int q) { return q == 0 ? W / WD::N : (q <= nleftw ? q - 1 : q - 1 + RB); };
    if (G > 1 && warp == 0) {
      // the words this CTA receives
      int words = 0;
      if (lane < NMV) {
        const int row = s_mrow[lane];
        if (row >= lo && row < lo + nloc && row != s_mfrom[lane]) words = 1 + nleftw + (lane < NB ? 0 : nrw);
      }
      words = __reduce_add_sync(kAll, words) + NB * nrw;
      if (me == 0) pan_bar_arm(pan_saddr(&r_bar[2]), 16u * (uint32_t)words);
    }
    if (nrw > 0) {
      const int e = (tid >> 4) & (NB - 1), src = s_mfrom[e];
      if (src >= lo && src < lo + nloc) {
        const int4* from = reinterpret_cast<const int4*>(tile + (src - lo) * LD + c1);
        if (G == 1) {
          for (int q = pc + 16 * (tid >> 7); q < nrw; q += 16 * (NT >> 7)) reinterpret_cast<int4*>(&s_U[e][c1])[q] = from[q];
        } else if (pc < G) {
          const uint32_t ua = pan_mapa(pan_saddr(&s_U[e][c1]), pc);
          for (int q = tid >> 7; q < nrw; q += NT >> 7) pan_st_async(ua + 16u * q, from[q], p_bar + 16u);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < MI; ++t) {
      const int idx = tid + NT * t, e = idx / MWP, q = idx & (MWP - 1);
      if (e >= NMV) break;
      const int row = s_mrow[e], src = s_mfrom[e];
      const int cw = moved_word(q);
      if (row >= 0 && row != src && q <= nleftw + (e < NB ? 0 : nrw) && src >= lo && src < lo + nloc) {
        const int4 x = reinterpret_cast<const int4*>(tile + (src - lo) * LD)[cw];
        if (G == 1) {
          reinterpret_cast<int4*>(r_mv[e])[cw] = x;
        } else {
          const int o = owner(row);
          pan_st_async(pan_mapa(pan_saddr(&r_mv[e][0]), o) + 16u * cw, x, pan_mapa(pan_saddr(&r_bar[2]), o));
        }
      }
    }
    if (G == 1) __syncthreads();
    else if (me >= 0 && !pan_bar_wait(pan_saddr(&r_bar[2]), (uint32_t)(s0 / NB) & 1u, err)) me = -1;
    // U12 := L11 \ A12.  FP32: a thread a column; FP64: eight lanes a column
    // (a warp's FP64 instructions issue 68 cycles apart, so 28 of them in one
    // warp cost more than seven with a shuffle each)
    const int ui = tid & (NB - 1);
    if (nright > 0) {
      if constexpr (sizeof(T) == 4) {
        if (tid < nright) {
          T u[NB];
#pragma unroll
          for (int i = 0; i < NB; ++i) u[i] = s_U[i][c1 + tid];
#pragma unroll
          for (int i = 1; i < NB; ++i) {
            T l[NB];
            words_load<T, NB>(l, s_prow[i]);
#pragma unroll
            for (int j = 0; j < i; ++j) u[i] = fma(-l[j], u[j], u[i]);
            s_U[i][c1 + tid] = u[i];
          }
        }
      } else {
        T l[NB], u[NU];
        words_load<T, NB>(l, s_prow[ui]);
#pragma unroll
        for (int q = 0; q < NU; ++q) {
          const int c = tid / NB + (NT / NB) * q;
          u[q] = c < nright ? s_U[ui][c1 + c] : T(0);
        }
#pragma unroll
        for (int j = 0; j < NB - 1; ++j) {
#pragma unroll
          for (int q = 0; q < NU; ++q) {
            if (warp * (32 / NB) + (NT / NB) * q >= nright) break;  // no column in this warp
            const T uj = __shfl_sync(kAll, u[q], (lane & ~(NB - 1)) | j);
            if (ui > j) u[q] = fma(-l[j], uj, u[q]);
          }
        }
#pragma unroll
        for (int q = 0; q < NU; ++q) {
          const int c = tid / NB + (NT / NB) * q;
          if (c < nright) s_U[ui][c1 + c] = u[q];
        }
      }
    }
    __syncthreads();  // the rows that leave have been read
#pragma unroll
    for (int t = 0; t < MI; ++t) {
      const int idx = tid + NT * t, e = idx / MWP, q = idx & (MWP - 1);
      if (e >= NMV) break;
      const int row = s_mrow[e];
      const int cw = moved_word(q);
      if (row >= lo && row < lo + nloc && row != s_mfrom[e] && q <= nleftw + (e < NB ? 0 : nrw))
        reinterpret_cast<int4*>(tile + (row - lo) * LD)[cw] = reinterpret_cast<const int4*>(r_mv[e])[cw];
    }
    {  // the sub-panel's own rows: L11 \ U11 and U12
      const int e = (tid >> 4) & (NB - 1), row = s0 + e - lo;
      if (tid < 16 * NB && e < kb && row >= 0 && row < nloc) {
        int4* to = reinterpret_cast<int4*>(tile + row * LD + s0);
        for (int q = tid & 15; q < RB + nrw; q += 16)
          to[q] = q < RB ? reinterpret_cast<const int4*>(s_prow[e])[q] : reinterpret_cast<const int4*>(&s_U[e][c1])[q - RB];
      }
    }
    if (nright <= 0) break;
    __syncthreads();
    // 6. A22 -= L21 U12 on the rows below the sub-panel: the next sub-panel's
    // columns by every warp, the rest by the helper warps beside the next
    // sub-panel's chain
    const int i0 = max(0, c1 - lo);
    const int ngr = i0 < nloc ? (nloc - i0 + 31) / 32 : 0;  // groups of 32 rows
    const unsigned gmagic = ngr > 0 ? ((1u << 20) + ngr - 1) / ngr : 0;  // t / ngr for t * ngr < 2^20
    auto update = [&](int cbeg, int cend, int w0, int nw) {
      const int ncw = (cend - cbeg + WD::N - 1) / WD::N;  // a word of columns per work unit
      for (int t = warp - w0; t < ngr * ncw; t += nw) {
        const int cw = (int)(((unsigned)t * gmagic) >> 20), i = i0 + (t - cw * ngr) * 32 + lane;
        const int col = cbeg + cw * WD::N;
        if (i < nloc) {
          T l[NB], a[WD::N];
          words_load<T, NB>(l, tile + i * LD + s0);
          int4* pa = reinterpret_cast<int4*>(tile + i * LD + col);
          WD::unpack(a, *pa);
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            T uu[WD::N];
            WD::unpack(uu, *reinterpret_cast<const int4*>(&s_U[j][col]));
#pragma unroll
            for (int q = 0; q < WD::N; ++q) a[q] = fma(-l[j], uu[q], a[q]);
          }
          *pa = WD::pack(a);
        }
      }
    };
    const int cn = NW > NWC ? min(c1 + NB, w) : w;
    update(c1, cn, 0, NW);
    __syncthreads();
    if (NW > NWC && warp >= NWC) update(cn, w, NWC, NW - NWC);
  }
  __syncthreads();
  int failed = me < 0;
  if (G > 1 && tid == 0) failed |= ld_volatile_i32(err);  // used below, behind the stores
#pragma unroll 4
  for (int t = warp; t < nrg * nwd; t += NW) {
    const int wd = t / nrg, i = (t - wd * nrg) * 32 + lane;
    if (i < nloc) {
      T x[WD::N];
      WD::unpack(x, *reinterpret_cast<const int4*>(tile + i * LD + wd * WD::N));
#pragma unroll
      for (int q = 0; q < WD::N; ++q) {
        const int c = wd * WD::N + q;
        if (c < w) Ab[lo + i + (int64_t)c * lda] = x[q];
      }
    }
  }
  // the leaf's interchanges as row moves, for the other columns of the matrix
  for (int i = tid; i < nloc; i += NT) {
    const int id = *reinterpret_cast<const int*>(tile + i * LD + W);
    if (id != lo + i && (unsigned)id < (unsigned)M) {  // always a row, unless a wait gave up
      const int at = atomicAdd(&moves->count, 1);
      if (at < 2 * kLeafMaxW) moves->mv[at] = make_int2((int)c0 + lo + i, (int)c0 + id);
    }
  }
  if (cta == 0 && tid == 0 && info_local != 0 && *info_out == 0) *info_out = info_local;
  // No CTA leaves while another may still push to it.  Every push was waited for
  // unless a wait gave up somewhere: then a CTA stays until the others have left
  // or are here too, and until their last pushes have landed.
  if (G > 1 && __syncthreads_or(failed)) {
    cluster_arrive();
    cluster_wait();
    if (tid == 0) {
      const unsigned long long t0 = global_ns();
      while (global_ns() - t0 < kPushLandNs) {}
    }
  }
}

}  // namespace gblu
