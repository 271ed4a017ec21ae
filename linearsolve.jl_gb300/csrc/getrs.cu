// getrs on the device: P, L and U solves as two wavefront kernels.
//
// Order of operations follows the reference's back-solve
// _naive_lu_ldiv! (src/factorization.jl:433-457), applied per RHS column:
//   b[i] <-> b[ipiv[i]] for i ascending           (here: one gather through perm)
//   for j ascending:   b[i] = fma(-L[i,j], b[j], b[i])   (i > j)
//   for j descending:  b[j] /= U[j,j];  b[i] = fma(-U[i,j], b[j], b[i])  (i < j)
// Each row's value is updated in exactly that sequence, so the result is
// bit-identical to the reference's vector back-solve.  The transposed solve
// (trans = 'T') is U^T y = b, L^T z = y, x = P^T z as LAPACK dgetrs 'T'.
//
// Parallel structure: the matrix is cut into 64-row block rows.  Each CTA takes
// one block row of one right-hand side (fast FP32: two) by ticket (handed out in
// launch order, so every CTA waits only for CTAs already running), streams its
// off-diagonal tiles in order, polling the published solution values right
// before a tile needs them, then solves its diagonal block and publishes its
// rows.  All waits are bounded (DEV_TIMEOUT_SOLVE).
//
// A right-hand side a CTA, not several: a warp issues one FP64 instruction per
// 68 cycles however independent they are, so right-hand sides in one warp add
// up along the chain.  Five right-hand sides, both sweeps, one CTA per block
// row for all of them -> one CTA each: exact n = 2000 5.18 -> 0.61 ms,
// n = 6001 15.5 -> 1.9 ms; fast n = 6001 'N' 3.27 -> 0.82 ms, 'T' 7.55 -> 0.99 ms.
#include <algorithm>

#include "device_util.cuh"
#include "waits.cuh"
#include "gblu_internal.h"
#include "profile.h"

namespace gblu {

constexpr int kTS = kGetrsTile;  // block-row height == tile width
// fast-solve matrices per 64-row block b, each 64 x 64 column-major:
// InvL_bb, InvU_bb, InvL_bb L_{b,b-1}, InvU_bb U_{b,b+1}
constexpr int kInvSlots = 4;

constexpr int kSweepThreads = 128;  // exact sweeps: all issue copies; threads 0..63 own one row each
// Threads per row of the fast sweeps, each taking its share of a tile's columns:
// FP32 products are bound by their instructions' latency, FP64 ones by the SM's
// FP64 pipe, where more threads gain nothing.
template <typename T>
constexpr int kFastSplit = sizeof(T) == 4 ? 4 : 2;
constexpr int kStages = 3;          // tiles in flight per CTA

template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int sz = valid ? (int)sizeof(T) : 0;  // 0: zero-fill, nothing read
  if (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Row stride of a staged tile: 16 bytes of padding keep every column of
// t[c][r] 16-byte aligned (for 16-byte copies) and its reads conflict-free.
template <typename T>
__host__ __device__ constexpr int tile_ld() { return kTS + 16 / (int)sizeof(T); }

// Issue the copies of tile element (r, c) = op(LU)[r0 + r, c0 + c] into t[c][r];
// 'N': LU[r0+r + (c0+c)*lda] (contiguous in r), 'T': LU[c0+c + (r0+r)*lda]
// (contiguous in c).  Elements outside nr x nc are zero-filled, not read.  An
// 'N' tile of a 16-byte-aligned matrix (vec16) moves in 16-byte copies, each
// thread walking a fixed row slice across every (THREADS / 16-byte copies per
// column)-th column; a ragged tile's copies take fewer source bytes.  (With
// element copies for those, the last block row, which has the most tiles, came
// 15 us after the others at n = 3000.)
template <typename T, bool TRANS, int THREADS = kSweepThreads>
__device__ __forceinline__ void issue_tile(T (*t)[tile_ld<T>()], const T* __restrict__ LU, int64_t lda,
                                           int64_t r0, int64_t c0, int nr, int nc, bool vec16) {
  if (!TRANS && vec16) {
    constexpr int V = 16 / (int)sizeof(T);    // elements per copy
    constexpr int CPC = kTS / V;              // copies per column
    constexpr int CSTEP = THREADS / CPC;  // columns per pass
    const int cl = (int)threadIdx.x / CPC, rv = ((int)threadIdx.x % CPC) * V;
    const T* src = LU + (r0 + rv) + (c0 + cl) * lda;
    const int sz = min(V, max(nr - rv, 0)) * (int)sizeof(T);
#pragma unroll
    for (int c = cl; c < kTS; c += CSTEP, src += CSTEP * lda) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(&t[c][rv]);
      const int n = c < nc ? sz : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(n ? src : LU), "r"(n) : "memory");
    }
    return;
  }
#pragma unroll 8
  for (int idx = threadIdx.x; idx < kTS * kTS; idx += THREADS) {
    const int a = idx >> 6, b = idx & 63;  // b runs along the contiguous direction
    const int r = TRANS ? a : b, c = TRANS ? b : a;
    const bool ok = r < nr && c < nc;
    const T* src = ok ? (TRANS ? LU + (c0 + c) + (r0 + r) * lda : LU + (r0 + r) + (c0 + c) * lda) : LU;
    cp_async_elem(&t[c][r], src, ok);
  }
}

// The IEEE division, out of line (inlined, its instructions are scheduled into
// the chain although the branch to it is not taken).
template <typename T>
__device__ __noinline__ T divide_ieee(T a, T b) { return a / b; }

// One lane's store without a branch (a divergent one costs the warp 50 cycles
// of the chain).
__device__ __forceinline__ void store_if(bool on, double* p, double v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.global.f64 [%1], %2;\n\t}" ::"r"((int)on), "l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void store_if(bool on, float* p, float v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.global.f32 [%1], %2;\n\t}" ::"r"((int)on), "l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void store_shared_if(bool on, double* p, double v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.volatile.shared.f64 [%1], %2;\n\t}" ::"r"((int)on), "r"((unsigned)__cvta_generic_to_shared(p)), "d"(v) : "memory");
}
__device__ __forceinline__ void store_shared_if(bool on, float* p, float v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.volatile.shared.f32 [%1], %2;\n\t}" ::"r"((int)on), "r"((unsigned)__cvta_generic_to_shared(p)), "f"(v) : "memory");
}

// A value another warp of the CTA leaves in shared memory (the sentinel until
// then).  Bounded like every wait; zero once any CTA failed.
template <typename T>
__device__ __forceinline__ T smem_value(const T* p, DevScratch* scr) {
  using U = typename SweepBits<T>::U;
  const volatile U* q = reinterpret_cast<const volatile U*>(p);
  unsigned long long t0 = 0;
  for (unsigned it = 0;; ++it) {
    const U v = *q;
    if (v != SweepBits<T>::kSentinel) return SweepBits<T>::as_t(v);
    if ((it & 1023u) == 1023u) {
      if (ld_volatile_i32(&scr->error) != 0) return T(0);
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kSpinTimeoutNs) {
        atomicCAS(&scr->error, 0, (int)DEV_TIMEOUT_SOLVE);
        return T(0);
      }
    }
  }
}

// One exact triangular sweep over 64-row block rows, one right-hand side per CTA.
//   FWD  : block rows first-to-last, columns ascending; 'N' unit-lower L with
//          the right-hand side gathered through perm, 'T' non-unit U^T.
//   !FWD : block rows last-to-first, columns descending; 'N' non-unit U,
//          'T' unit L^T; results scattered to Out (through perm for 'T').
// Each row accumulates its updates in exactly the reference's order.  Warps 0
// and 1 own the block's 32-row halves (a row a lane); warps 2 and 3 help with
// the copies and poll the values of the block row just before this one, which
// the row warps apply one by one as they arrive (published as soon as final).
// Then the first half's 32-step chain, its coefficients in registers, the
// second half applying the first's solutions as they come, and its chain.
//
// Bound: the chain of n dependent steps, each a shuffle and an FP64
// instruction (35 + 68 cycles), and three more of those for the division by a
// non-unit diagonal entry.  In place: 123 cycles a step (unit) and 425
// (non-unit), against 203 and 500 when a step waited for a shared-memory load
// of its coefficient and for a branch to publish; n = 2000, one right-hand
// side, both sweeps: 0.76 -> 0.61 ms.
template <typename T, bool TRANS, bool FWD>
__global__ void __launch_bounds__(kSweepThreads)
solve_sweep_kernel(int64_t n, const T* __restrict__ LU, int64_t lda, const int32_t* __restrict__ perm,
                   const T* __restrict__ In, int64_t ldi, T* __restrict__ Y, int64_t ldy,
                   T* __restrict__ Out, int64_t ldo, int nrhs, DevScratch* __restrict__ scr) {
  using SB = SweepBits<T>;
  using UB = typename SB::U;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T(*tiles)[kTS][tile_ld<T>()] = reinterpret_cast<T(*)[kTS][tile_ld<T>()]>(smem_raw);
  // 16-byte copies need a 16-byte-aligned matrix and column stride
  const bool vec16 = ((reinterpret_cast<uintptr_t>(LU) | (uintptr_t)(lda * (int64_t)sizeof(T))) & 15) == 0;
  __shared__ T sx[kTS];   // solution values of the current off-diagonal tile
  __shared__ T s_lx[kTS]; // of the last one, as they arrive (sentinel until then)
  __shared__ T s_dx[kTS]; // the first half's own solutions, as they become final
  __shared__ int s_ticket;
  constexpr bool kUnit = FWD != TRANS;  // fwd 'N' (L) and bwd 'T' (L^T) have unit diagonals
  const int nblk = (int)((n + kTS - 1) / kTS);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_ticket = (int)atomicAdd(&scr->ticket, 1u);
  if (tid < kTS) s_lx[tid] = s_dx[tid] = SB::as_t(SB::kSentinel);
  __syncthreads();
  const int ord = s_ticket / nrhs, rhs = s_ticket - ord * nrhs;
  const int blk = FWD ? ord : nblk - 1 - ord;
  if (In) In += rhs * ldi;
  Y += rhs * ldy;
  if (Out) Out += rhs * ldo;
  const int64_t r0 = (int64_t)blk * kTS;
  const int nr = (int)min((int64_t)kTS, n - r0);
  const int r = tid;  // row within the block (threads 0..63)
  const bool valid = r < nr;
  T acc = T(0);
  T* dst = nullptr;   // where this row's solution is published
  if (valid) {
    const int64_t prow = (FWD != TRANS) ? (int64_t)perm[r0 + r] : r0 + r;
    acc = SB::canon(FWD ? In[TRANS ? r0 + r : prow] : Y[r0 + r]);
    dst = FWD ? Y + r0 + r : Out + (TRANS ? prow : r0 + r);
  }
  const int noff = FWD ? blk : nblk - 1 - blk;  // off-diagonal tiles of this block row
  const int ntiles = noff + 1;                  // + the diagonal tile
  auto col_block = [&](int t) -> int { return t < noff ? (FWD ? t : nblk - 1 - t) : blk; };
  auto issue = [&](int t) {
    const int64_t c0 = (int64_t)col_block(t) * kTS;
    issue_tile<T, TRANS>(tiles[t % kStages], LU, lda, r0, c0, nr, (int)min((int64_t)kTS, n - c0), vec16);
  };
#pragma unroll
  for (int t = 0; t < kStages - 1; ++t) {
    if (t < ntiles) issue(t);
    cp_async_commit();
  }
  auto src_of = [&](int cb, int c) -> const T* {
    const int64_t c0 = (int64_t)cb * kTS;
    return FWD ? &Y[c0 + c] : &Out[TRANS ? (int64_t)perm[c0 + c] : c0 + c];
  };
  // Solution values of the next off-diagonal tile are fetched one tile ahead
  // (most are published long before they are needed); a value still equal to
  // the sentinel is polled until it arrives.
  UB pre = 0;
  auto prefetch = [&](int t) {
    const int cb = col_block(t);
    const int nc = (int)min((int64_t)kTS, n - (int64_t)cb * kTS);
    if (tid < nc) pre = SB::load(src_of(cb, tid));
  };
  if (noff > 1) prefetch(0);
  for (int t = 0; t < noff - 1; ++t) {
    cp_async_wait<kStages - 2>();  // tile t has landed
    __syncthreads();               // everywhere, and the slot of tile t - 1 is free
    if (t + kStages - 1 < ntiles) issue(t + kStages - 1);
    cp_async_commit();
    T(*tile)[tile_ld<T>()] = tiles[t % kStages];
    const int cb = col_block(t);
    const int nc = (int)min((int64_t)kTS, n - (int64_t)cb * kTS);
    int ok = 1;
    if (tid < kTS) {
      T v = T(0);
      if (tid < nc) {
        if (pre != SB::kSentinel) v = SB::as_t(pre);
        else if (!poll_value(src_of(cb, tid), scr, &v)) ok = 0;
      }
      sx[tid] = v;
    }
    if (!__syncthreads_and(ok)) {
      cp_async_wait<0>();  // no copy may land after the CTA has left
      return;
    }
    if (t + 1 < noff - 1) prefetch(t + 1);
    if (tid < kTS) {
      if (FWD) {
#pragma unroll 8
        for (int c = 0; c < kTS; ++c) acc = fma(-tile[c][r], sx[c], acc);
      } else if (nc == kTS) {
#pragma unroll 8
        for (int c = kTS - 1; c >= 0; --c) acc = fma(-tile[c][r], sx[c], acc);
      } else {
        for (int c = nc - 1; c >= 0; --c) acc = fma(-tile[c][r], sx[c], acc);
      }
    }
  }
  cp_async_wait<0>();  // the last off-diagonal tile and the diagonal one
  __syncthreads();
  if (warp >= 2) {
    if (noff > 0) {
      const int cb = col_block(noff - 1);
      const int nc = (int)min((int64_t)kTS, n - (int64_t)cb * kTS);
      const int c = tid - 64;
      const T* p = src_of(cb, c < nc ? c : 0);
      bool pend = c < nc;
      unsigned long long t0 = 0;
      for (unsigned it = 0; __any_sync(kAll, pend); ++it) {
        if (pend) {
          const UB v = SB::load(p);
          if (v != SB::kSentinel) {
            *reinterpret_cast<volatile UB*>(&s_lx[c]) = v;
            pend = false;
          }
        }
        if ((it & 63u) == 63u) {
          bool give_up = ld_volatile_i32(&scr->error) != 0;
          const unsigned long long now = global_ns();
          if (t0 == 0) t0 = now;
          else if (now - t0 > kSpinTimeoutNs) {
            atomicCAS(&scr->error, 0, (int)DEV_TIMEOUT_SOLVE);
            give_up = true;
          }
          if (__any_sync(kAll, give_up)) break;  // the whole warp; the row warps see the error word
        }
      }
    }
    return;
  }
  // The row warps.  Coefficients of the own half's diagonal block in registers.
  T(*dt)[tile_ld<T>()] = tiles[noff % kStages];
  T a[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) a[i] = dt[32 * warp + i][r];
  const T dg = (!kUnit && valid) ? dt[r][r] : T(1);
  const T y = T(1) / dg;
  const bool y_ok = DivRange<T>::in_range(y);
  if (noff > 0) {
    T(*tile)[tile_ld<T>()] = tiles[(noff - 1) % kStages];
    if (FWD) {
#pragma unroll 4
      for (int c = 0; c < kTS; ++c) acc = fma(-tile[c][r], smem_value(&s_lx[c], scr), acc);
    } else {
      const int nc = (int)min((int64_t)kTS, n - (int64_t)col_block(noff - 1) * kTS);
      if (nc == kTS) {
#pragma unroll 4
        for (int c = kTS - 1; c >= 0; --c) acc = fma(-tile[c][r], smem_value(&s_lx[c], scr), acc);
      } else {
        for (int c = nc - 1; c >= 0; --c) acc = fma(-tile[c][r], smem_value(&s_lx[c], scr), acc);
      }
    }
  }
  const bool first = warp == (FWD ? 0 : 1);
  if (!first) {  // the first half's columns, in sweep order
    if (FWD) {
      if (nr > 32)
#pragma unroll 4
        for (int c = 0; c < 32; ++c) acc = fma(-dt[c][r], smem_value(&s_dx[c], scr), acc);
    } else {
      for (int c = nr - 1; c >= 32; --c) acc = fma(-dt[c][r], smem_value(&s_dx[c], scr), acc);
    }
  }
  // The chain: in each step the owner's value is final, goes to every lane, is
  // published, and updates the rows after it.  The finished rows' registers are
  // updated too and not used again, so nothing is predicated.
  if constexpr (kUnit) {
#pragma unroll
    for (int st = 0; st < 32; ++st) {
      const int i = FWD ? st : 31 - st;
      const int c = 32 * warp + i;
      if (c >= nr) continue;  // uniform
      const T x = __shfl_sync(kAll, acc, i);
      acc = fma(-a[i], x, acc);
      store_if(lane == i, dst, x);
      if (first) store_shared_if(lane == i, &s_dx[c], x);
    }
  } else {
    // First divided by the diagonal entry (Markstein's division, every lane by
    // its own).  Where Markstein's quotient may not be the correctly rounded
    // one the IEEE division is taken; the branch to it costs 120 cycles of the
    // chain, so it is tested once per four columns, which then start over.
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const T before = acc;
      T own = T(0);
      int ok = 1;
#pragma unroll
      for (int st = 4 * g; st < 4 * g + 4; ++st) {
        const int i = FWD ? st : 31 - st;
        if (32 * warp + i >= nr) continue;  // uniform
        const T q = acc * y;
        const T e = fma(-dg, q, acc);
        const T d = fma(e, y, q);
        const bool zero = !PivKey<T>::nonzero(acc);  // q is the signed zero
        const T x = __shfl_sync(kAll, zero ? q : d, i);
        ok &= __shfl_sync(kAll, (int)(y_ok && (zero || DivRange<T>::in_range(q))), i);
        own = lane == i ? x : own;
        acc = fma(-a[i], x, acc);
      }
      if (!ok) {
        acc = before;
#pragma unroll 1
        for (int st = 4 * g; st < 4 * g + 4; ++st) {
          const int i = FWD ? st : 31 - st;
          if (32 * warp + i >= nr) continue;
          const T x = SB::canon(__shfl_sync(kAll, divide_ieee(acc, dg), i));
          own = lane == i ? x : own;
          acc = fma(-dt[32 * warp + i][r], x, acc);
        }
      }
      const bool mine = (FWD ? lane : 31 - lane) / 4 == g && valid;
      store_if(mine, dst, own);
      if (first) store_shared_if(mine, &s_dx[r], own);
    }
  }
}

__device__ __forceinline__ unsigned cluster_ctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_nctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ int ld_cluster(uint32_t a) {
  int v;
  asm volatile("ld.relaxed.cluster.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t a, float v) {
  asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(__float_as_int(v)) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v) {
  asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(__double_as_longlong(v)) : "memory");
}

// Fast sweeps.  'N': block row i's solution is x_i = d_i - M_i x_p, where x_p
// is the block row just before it in the sweep, M_i its coupling (fold_kernel)
// and d_i = Inv_ii (b_i - the products with every earlier block row but x_p):
// d_i is computed while x_p is still being solved, so only the 64 x 64
// product M_i x_p lies on the wavefront's critical path.  'T' has no coupling:
// x_i = op(Inv_ii) (b_i - every product).  H threads per
// row, each taking its share of every tile's columns with four independent
// partial sums, combined through shared memory.  Tile order per block row:
// the earlier off-diagonal blocks (but the last, in sweep order, for 'N'),
// Inv_ii, then M_i, whose share each thread holds in registers before x_p comes.
// NR right-hand sides per CTA: one in FP64 (a warp issues an FP64 instruction per
// 68 cycles, so more would add up along the chain), up to two in FP32, more going
// to CTAs of their own.
// The CTAs of a cluster are consecutive block rows of the same right-hand sides:
// a solution goes straight to the shared memory of the next two, which poll it
// there like the published values (sentinel until then) without the trip through
// L2 (a store and a load, 1100 cycles).  A block row then takes 0.8 us, of which
// d_i after x_{i-2} is most (1250 cycles: two products and their sums).
// FP32 factors, n = 3000, four right-hand sides, one sweep: 79 us with four
// right-hand sides and two threads a row in a CTA and no clusters, 64 with two
// right-hand sides a CTA, 58 with four threads a row, 54 with one neighbour
// pushed to, 46 with two and ragged tiles in 16-byte copies.
// Backward-error accurate, not bit-exact.
template <typename T, int NR, bool TRANS, bool FWD>
__global__ void __launch_bounds__(kTS* kFastSplit<T>)
fast_sweep_kernel(int64_t n, const T* __restrict__ LU, int64_t lda, const int32_t* __restrict__ perm,
                  const T* __restrict__ In, int64_t ldi, T* __restrict__ Y, int64_t ldy,
                  T* __restrict__ Out, int64_t ldo, int nrhs, DevScratch* __restrict__ scr,
                  const T* __restrict__ inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T(*tiles)[kTS][tile_ld<T>()] = reinterpret_cast<T(*)[kTS][tile_ld<T>()]>(smem_raw);
  __shared__ T sx[kTS][NR];
  constexpr int H = kFastSplit<T>, Q = kTS / H, kThreads = kTS * H;
  static_assert(NR <= H, "thread (r, q) finishes row r of right-hand side q");
  __shared__ T part[H][kTS][NR];
  __shared__ T s_lx[2][kTS][NR];  // the block rows one and two before this one, pushed by their CTAs
  __shared__ int s_ticket;
  const int rank = (int)cluster_ctarank(), cs = (int)cluster_nctarank();
  const bool vec16 = ((reinterpret_cast<uintptr_t>(LU) | (uintptr_t)(lda * (int64_t)sizeof(T))) & 15) == 0;
  const int nblk = (int)((n + kTS - 1) / kTS);
  constexpr bool kCouple = !TRANS;
  constexpr bool kUnit = FWD != TRANS;
  if (threadIdx.x == 0 && rank == 0) s_ticket = (int)atomicAdd(&scr->ticket, 1u);  // one a cluster
  for (int e = threadIdx.x; e < 2 * kTS * NR; e += kThreads)
    (&s_lx[0][0][0])[e] = SweepBits<T>::as_t(SweepBits<T>::kSentinel);
  cluster_sync_all();  // every CTA of the cluster runs and has its s_lx
  const int ticket = ld_cluster(pan_mapa(pan_saddr(&s_ticket), 0));
  const int groups = (nrhs + NR - 1) / NR;  // clusters per cs block rows
  const int ord = ticket / groups * cs + rank, q0 = ticket % groups * NR;
  if (ord >= nblk) {  // the last cluster's spare CTAs
    cluster_sync_all();
    return;
  }
  const int blk = FWD ? ord : nblk - 1 - ord;
  nrhs = min(NR, nrhs - q0);
  if (In) In += q0 * ldi;
  Y += q0 * ldy;
  if (Out) Out += q0 * ldo;
  const int64_t r0 = (int64_t)blk * kTS;
  const int nr = (int)min((int64_t)kTS, n - r0);
  const int tid = threadIdx.x, r = tid & 63, h = tid >> 6;
  const bool valid = r < nr;
  const int noff = FWD ? blk : nblk - 1 - blk;  // block rows before this one in the sweep
  const int nlead = kCouple ? max(noff - 1, 0) : noff;  // off-diagonal tiles before the coupling
  const int ntiles = nlead + 1 + (kCouple && noff > 0 ? 1 : 0);
  const int pcb = FWD ? blk - 1 : blk + 1;      // the coupled block row (noff > 0)
  const int pnc = noff > 0 ? (int)min((int64_t)kTS, n - (int64_t)pcb * kTS) : 0;
  auto col_block = [&](int t) -> int { return FWD ? t : nblk - 1 - t; };
  auto issue = [&](int t) {
    if (t < nlead) {
      const int64_t c0 = (int64_t)col_block(t) * kTS;
      issue_tile<T, TRANS, kThreads>(tiles[t % kStages], LU, lda, r0, c0, nr, (int)min((int64_t)kTS, n - c0), vec16);
    } else {
      const bool coupling = t > nlead;
      const int slot = (coupling ? 2 : 0) + (kUnit ? 0 : 1);  // L's, U's
      issue_tile<T, TRANS, kThreads>(tiles[t % kStages], inv + ((int64_t)blk * kInvSlots + slot) * (kTS * kTS), kTS, 0, 0,
                           nr, coupling ? pnc : nr, true);
    }
  };
  T a[4][NR];  // partial sums; thread h = 0 starts from the right-hand side
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int q = 0; q < NR; ++q) a[j][q] = T(0);
  if (h == 0 && valid)
#pragma unroll
    for (int q = 0; q < NR; ++q)
      if (q < nrhs) a[0][q] = FWD ? In[(TRANS ? r0 + r : (int64_t)perm[r0 + r]) + q * ldi] : Y[(r0 + r) + q * ldy];
  T d = T(0);  // thread (r, q): row r of right-hand side q
#pragma unroll
  for (int t = 0; t < kStages - 1; ++t) {
    if (t < ntiles) issue(t);
    cp_async_commit();
  }
  // solution values of the next block needed, fetched one step ahead
  using UB = typename SweepBits<T>::U;
  constexpr int KP = (kTS * NR + kThreads - 1) / kThreads;
  UB pre[KP];
  auto src_of = [&](int cb, int c, int q) -> const T* {
    const int64_t c0 = (int64_t)cb * kTS;
    return FWD ? &Y[(c0 + c) + q * ldy] : &Out[(TRANS ? (int64_t)perm[c0 + c] : c0 + c) + q * ldo];
  };
  auto prefetch = [&](int cb) {
    const int nc = (int)min((int64_t)kTS, n - (int64_t)cb * kTS);
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int idx = tid + k * kThreads;
      const int c = idx / NR, q = idx - c * NR;
      pre[k] = (idx < kTS * NR && q < nrhs && c < nc) ? SweepBits<T>::load(src_of(cb, c, q)) : UB(0);
    }
  };
  auto fill_sx = [&](int cb) -> int {
    const int nc = (int)min((int64_t)kTS, n - (int64_t)cb * kTS);
    const int back = abs(pcb - cb);  // 0: the block row just before
    const bool pushed = back < 2 && rank > back;
    int ok = 1;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int idx = tid + k * kThreads;
      if (idx >= kTS * NR) continue;
      const int c = idx / NR, q = idx - c * NR;
      T v = T(0);
      if (q < nrhs && c < nc) {
        if (pushed) v = smem_value(&s_lx[back][c][q], scr);
        else if (pre[k] != SweepBits<T>::kSentinel) v = SweepBits<T>::as_t(pre[k]);
        else if (!poll_value(src_of(cb, c, q), scr, &v)) ok = 0;
      }
      sx[c][q] = v;
    }
    return ok;
  };
  // this thread's share of a tile's columns times sx, added to (sign -1) or
  // into fresh sums (sign +1)
  auto share_product = [&](T(*tile)[tile_ld<T>()], T(&y)[4][NR], T sign) {
#pragma unroll 4
    for (int c = Q * h; c < Q * h + Q; c += 4)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const T m = sign * tile[c + j][r];
#pragma unroll
        for (int q = 0; q < NR; ++q) y[j][q] = fma(m, sx[c + j][q], y[j][q]);
      }
  };
  // this thread's sums over its share to `part`; then row r's whole sum of
  // right-hand side h
  auto put_part = [&](T(&y)[4][NR]) {
#pragma unroll
    for (int q = 0; q < NR; ++q) part[h][r][q] = (y[0][q] + y[1][q]) + (y[2][q] + y[3][q]);
  };
  auto total = [&]() {
    T t = part[0][r][h];
#pragma unroll
    for (int k = 1; k < H; ++k) t += part[k][r][h];
    return t;
  };
  if (nlead > 0) prefetch(col_block(0));
  else if (kCouple && noff > 0) prefetch(pcb);
  for (int t = 0; t < ntiles; ++t) {
    cp_async_wait<kStages - 2>();  // tile t has landed
    __syncthreads();               // everywhere, and the slot of tile t - 1 is free
    if (t + kStages - 1 < ntiles) issue(t + kStages - 1);
    cp_async_commit();
    T(*tile)[tile_ld<T>()] = tiles[t % kStages];
    if (t < nlead) {  // an earlier off-diagonal block: b -= L_ij x_j
      const int ok = fill_sx(col_block(t));
      if (!__syncthreads_and(ok)) break;  // the error word is set
      if (t + 1 < nlead) prefetch(col_block(t + 1));
      else if (kCouple) prefetch(pcb);
      share_product(tile, a, T(-1));
      continue;
    }
    T y[4][NR];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < NR; ++q) y[j][q] = T(0);
    if (t == nlead) {  // d = Inv_ii (right-hand side so far)
      put_part(a);
      __syncthreads();
      if (h < NR) sx[r][h] = valid ? total() : T(0);
      __syncthreads();
      share_product(tile, y, T(1));
      put_part(y);
      __syncthreads();
      if (h < NR) d = total();
      continue;
    }
    // the coupling: x = d - M_i x_p
    T m[Q];
#pragma unroll
    for (int c = 0; c < Q; ++c) m[c] = tile[Q * h + c][r];
    const int ok = fill_sx(pcb);
    if (!__syncthreads_and(ok)) break;
#pragma unroll
    for (int c = 0; c < Q; ++c)
#pragma unroll
      for (int q = 0; q < NR; ++q) y[c & 3][q] = fma(m[c], sx[Q * h + c][q], y[c & 3][q]);
    put_part(y);
    __syncthreads();
    if (h < NR) d -= total();
  }
  cp_async_wait<0>();  // no copy may land after the CTA has left
  if (h < nrhs && valid) {  // nrhs <= NR
    const T v = SweepBits<T>::canon(d);
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (rank + 1 + b < cs && ord + 1 + b < nblk) st_cluster(pan_mapa(pan_saddr(&s_lx[b][r][h]), rank + 1 + b), v);
    if (FWD) Y[(r0 + r) + h * ldy] = v;
    else Out[(TRANS ? (int64_t)perm[r0 + r] : r0 + r) + h * ldo] = v;
  }
  cluster_sync_all();  // a CTA stays until nothing more can be pushed to it
}

template <typename T>
constexpr size_t sweep_smem() { return (size_t)kStages * kTS * tile_ld<T>() * sizeof(T); }

// Inverses of the 64 x 64 diagonal blocks for the fast sweeps: CTA (b, 0)
// inverts the unit-lower L_bb, CTA (b, 1) the upper U_bb; thread j computes
// column j of the inverse in registers (substitution against e_j, the block
// in shared memory).  A ragged last block is padded with the identity.
// Output: inv[(b * kInvSlots + which) * 4096 + i + 64 j] = Inv(i, j).
template <typename T>
__global__ void __launch_bounds__(kTS)
diag_inverse_kernel(int64_t n, const T* __restrict__ LU, int64_t lda, T* __restrict__ inv) {
  __shared__ T s[kTS][kTS + 1];  // s[c][r] = block(r, c)
  const int b = blockIdx.x, which = blockIdx.y;
  const int64_t r0 = (int64_t)b * kTS;
  const int nb = (int)min((int64_t)kTS, n - r0);
  const int j = threadIdx.x;
  for (int idx = j; idx < kTS * kTS; idx += kTS) {
    const int c = idx >> 6, r = idx & 63;
    T v = (r < nb && c < nb) ? LU[(r0 + r) + (r0 + c) * lda] : T(0);
    if (r == c && r >= nb) v = T(1);
    s[c][r] = v;
  }
  __syncthreads();
  T x[kTS];
#pragma unroll
  for (int i = 0; i < kTS; ++i) x[i] = (i == j) ? T(1) : T(0);
  if (which == 0) {  // L_bb unit lower: forward substitution
#pragma unroll
    for (int k = 0; k < kTS; ++k)
#pragma unroll
      for (int i = k + 1; i < kTS; ++i) x[i] = fma(-s[k][i], x[k], x[i]);
  } else {  // U_bb upper: backward substitution
#pragma unroll
    for (int k = kTS - 1; k >= 0; --k) {
      x[k] = x[k] / s[k][k];
#pragma unroll
      for (int i = 0; i < k; ++i) x[i] = fma(-s[k][i], x[k], x[i]);
    }
  }
  T* out = inv + ((int64_t)b * kInvSlots + which) * (kTS * kTS) + (int64_t)j * kTS;
#pragma unroll
  for (int i = 0; i < kTS; ++i) out[i] = x[i];
}

// The couplings of the fast 'N' sweeps: slot 2 of block b = InvL_bb L_{b,b-1}
// (b >= 1), slot 3 = InvU_bb U_{b,b+1} (b <= nblk - 2); zero where there is
// no such block and outside ragged edges.  Thread (r, g): row r, columns
// 16 g .. 16 g + 15 of the product.
template <typename T>
__global__ void __launch_bounds__(256)
fold_kernel(int64_t n, const T* __restrict__ LU, int64_t lda, T* __restrict__ inv) {
  __shared__ T sO[kTS][kTS + 1];  // sO[c][k] = O(k, c), O the off-diagonal block
  const int b = blockIdx.x, which = blockIdx.y;
  const int64_t nblk = (n + kTS - 1) / kTS;
  T* out = inv + ((int64_t)b * kInvSlots + 2 + which) * (kTS * kTS);
  const int64_t ob = which == 0 ? (int64_t)b - 1 : (int64_t)b + 1;
  const int tid = threadIdx.x;
  if (ob < 0 || ob >= nblk) {
    for (int idx = tid; idx < kTS * kTS; idx += 256) out[idx] = T(0);
    return;
  }
  const int64_t r0 = (int64_t)b * kTS, c0 = ob * kTS;
  const int nb = (int)min((int64_t)kTS, n - r0), nc = (int)min((int64_t)kTS, n - c0);
  const T* I = inv + ((int64_t)b * kInvSlots + which) * (kTS * kTS);
  for (int idx = tid; idx < kTS * kTS; idx += 256) {
    const int c = idx >> 6, k = idx & 63;
    sO[c][k] = (k < nb && c < nc) ? LU[(r0 + k) + (c0 + c) * lda] : T(0);
  }
  __syncthreads();
  const int r = tid & 63, g = tid >> 6;
  T acc[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] = T(0);
  for (int k = 0; k < kTS; ++k) {
    const T a = I[r + k * kTS];  // Inv(r, k), coalesced over r
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = fma(a, sO[16 * g + j][k], acc[j]);
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) out[r + (int64_t)(16 * g + j) * kTS] = r < nb ? acc[j] : T(0);
}

size_t getrs_inverse_bytes(int64_t n, int elem_size) {
  const int64_t nblk = (n + kTS - 1) / kTS;
  return (size_t)std::max<int64_t>(nblk, 1) * kInvSlots * kTS * kTS * elem_size;
}

template <typename T>
cudaError_t getrs_invert_launch(const GetrsPlan<T>& p, cudaStream_t s) {
  if (p.n <= 0) return cudaSuccess;
  if (!p.inv) return cudaErrorInvalidValue;
  const int64_t nblk = (p.n + kTS - 1) / kTS;
  LaunchScope ls(K_SOLVE, (double)nblk * 2.0 * kTS * kTS * kTS / 3.0,
                 (double)nblk * 3.0 * kTS * kTS * sizeof(T), s);
  diag_inverse_kernel<T><<<dim3((unsigned)nblk, 2), kTS, 0, s>>>(p.n, p.LU, p.lda, p.inv);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  LaunchScope ls2(K_SOLVE, (double)nblk * 4.0 * kTS * kTS * kTS, (double)nblk * 6.0 * kTS * kTS * sizeof(T), s);
  fold_kernel<T><<<dim3((unsigned)nblk, 2), 256, 0, s>>>(p.n, p.LU, p.lda, p.inv);
  return cudaGetLastError();
}

size_t getrs_scratch_bytes(int64_t n, int elem_size, int64_t work_cols) {
  int64_t nblk = (n + kTS - 1) / kTS;
  size_t b = 256 + ((2 * nblk * sizeof(int32_t) + 255) & ~size_t(255));
  b += ((size_t)n * work_cols * elem_size + 255) & ~size_t(255);
  return b + 256;
}

template <typename T>
void getrs_carve(GetrsPlan<T>& p, void* base, size_t bytes, int64_t work_cols) {
  char* c = reinterpret_cast<char*>(base);
  auto take = [&](size_t nb) { char* r = c; c += (nb + 255) & ~size_t(255); return r; };
  int64_t nblk = (p.n + kTS - 1) / kTS;
  p.scratch = reinterpret_cast<DevScratch*>(take(sizeof(DevScratch)));
  p.flags = reinterpret_cast<int32_t*>(take(2 * nblk * sizeof(int32_t)));
  p.work = reinterpret_cast<T*>(take((size_t)p.n * work_cols * sizeof(T)));
  p.work_cols = work_cols;
  (void)bytes;
}

namespace {
// Columns x[:, 0 .. gridDim.y - 1] filled with the sentinel, and the ticket of
// the sweep that follows reset.  (A byte fill cannot write a signalling NaN.)
template <typename T>
__global__ void __launch_bounds__(256)
sentinel_kernel(int64_t n, T* __restrict__ x, int64_t ldx, unsigned* __restrict__ ticket) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *ticket = 0u;
  typename SweepBits<T>::U* c = reinterpret_cast<typename SweepBits<T>::U*>(x + blockIdx.y * ldx);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c[i] = SweepBits<T>::kSentinel;
}

template <typename T>
cudaError_t sentinel_launch(const GetrsPlan<T>& p, int nr, T* x, int64_t ldx, cudaStream_t s) {
  LaunchScope ls(K_OTHER, 0.0, (double)p.n * nr * sizeof(T), s);
  const unsigned ctas = (unsigned)std::min<int64_t>((p.n + 255) / 256, 1024);
  sentinel_kernel<T><<<dim3(ctas, (unsigned)nr), 256, 0, s>>>(p.n, x, ldx, &p.scratch->ticket);
  return cudaGetLastError();
}

template <typename T, int NR, bool TRANS, bool FWD>
cudaError_t launch_sweep(const GetrsPlan<T>& p, int nr, T* B, int64_t ldb, cudaStream_t s) {
  const int64_t nblk = (p.n + kTS - 1) / kTS;
  const T* In = FWD ? B : nullptr;
  T* Out = FWD ? nullptr : B;
  // algorithmic work of one sweep: the triangle (n^2/2 elements) read once,
  // n^2 flops per right-hand side
  LaunchScope ls(K_SOLVE, (double)p.n * (double)p.n * nr,
                 0.5 * (double)p.n * (double)p.n * sizeof(T) + 2.0 * p.n * nr * sizeof(T), s);
  if (p.fast && p.inv) {
    // clusters of eight block rows (of fewer for fewer)
    const int cs = nblk >= 8 ? 8 : nblk >= 4 ? 4 : nblk >= 2 ? 2 : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((nblk + cs - 1) / cs * cs * ((nr + NR - 1) / NR)));
    cfg.blockDim = dim3(kTS * kFastSplit<T>);
    cfg.dynamicSmemBytes = sweep_smem<T>();
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fast_sweep_kernel<T, NR, TRANS, FWD>, p.n, p.LU, p.lda, p.perm, In, ldb, p.work,
                              p.n, Out, ldb, nr, p.scratch, p.inv);
  }
  solve_sweep_kernel<T, TRANS, FWD><<<(unsigned)(nblk * nr), kSweepThreads, sweep_smem<T>(), s>>>(
      p.n, p.LU, p.lda, p.perm, In, ldb, p.work, p.n, Out, ldb, nr, p.scratch);
  return cudaGetLastError();
}

template <typename T, int NR>
cudaError_t run_chunk(const GetrsPlan<T>& p, char trans, int nr, T* B, int64_t ldb, cudaStream_t s) {
  const bool tr = trans == 'T' || trans == 't' || trans == 'C' || trans == 'c';
  // dependents poll Y (forward) and B (backward): fill both with the sentinel
  cudaError_t e = sentinel_launch(p, nr, p.work, p.n, s);
  if (e != cudaSuccess) return e;
  e = tr ? launch_sweep<T, NR, true, true>(p, nr, B, ldb, s) : launch_sweep<T, NR, false, true>(p, nr, B, ldb, s);
  if (e != cudaSuccess) return e;
  e = sentinel_launch(p, nr, B, ldb, s);
  if (e != cudaSuccess) return e;
  return tr ? launch_sweep<T, NR, true, false>(p, nr, B, ldb, s) : launch_sweep<T, NR, false, false>(p, nr, B, ldb, s);
}

template <typename T, int NR>
void configure_fast() {
  const int b = (int)sweep_smem<T>();
  cudaFuncSetAttribute(fast_sweep_kernel<T, NR, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(fast_sweep_kernel<T, NR, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(fast_sweep_kernel<T, NR, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(fast_sweep_kernel<T, NR, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
}

template <typename T>
void configure_exact() {
  const int b = (int)sweep_smem<T>();
  cudaFuncSetAttribute(solve_sweep_kernel<T, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(solve_sweep_kernel<T, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(solve_sweep_kernel<T, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(solve_sweep_kernel<T, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
}
}  // namespace

void getrs_configure(int /*device*/) {
  configure_exact<double>();
  configure_exact<float>();
  configure_fast<double, 1>();
  configure_fast<float, 1>();
  configure_fast<float, 2>();
}

template <typename T>
cudaError_t getrs_launch(const GetrsPlan<T>& p, char trans, int64_t nrhs, T* B, int64_t ldb,
                         uint32_t* /*epoch*/, cudaStream_t s) {
  if (p.n <= 0 || nrhs <= 0) return cudaSuccess;
  const int64_t chunk = std::min<int64_t>(p.work_cols, 8);
  for (int64_t c = 0; c < nrhs; c += chunk) {
    int nr = (int)std::min<int64_t>(chunk, nrhs - c);
    T* Bc = B + c * ldb;
    cudaError_t e;
    if (sizeof(T) == 8 || nr == 1) e = run_chunk<T, 1>(p, trans, nr, Bc, ldb, s);
    else e = run_chunk<T, sizeof(T) == 8 ? 1 : 2>(p, trans, nr, Bc, ldb, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template cudaError_t getrs_launch<double>(const GetrsPlan<double>&, char, int64_t, double*, int64_t,
                                          uint32_t*, cudaStream_t);
template cudaError_t getrs_launch<float>(const GetrsPlan<float>&, char, int64_t, float*, int64_t,
                                         uint32_t*, cudaStream_t);
template void getrs_carve<double>(GetrsPlan<double>&, void*, size_t, int64_t);
template void getrs_carve<float>(GetrsPlan<float>&, void*, size_t, int64_t);
template cudaError_t getrs_invert_launch<double>(const GetrsPlan<double>&, cudaStream_t);
template cudaError_t getrs_invert_launch<float>(const GetrsPlan<float>&, cudaStream_t);

}  // namespace gblu
