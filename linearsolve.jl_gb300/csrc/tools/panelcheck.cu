// Self-test of the sub-panel kernel's bounded waits: one CTA of the cluster is
// late with one push, by far more than the wait limit this file is compiled
// with, so the waits of the others run out.  Whatever they go on with, every
// index they use is checked against the leaf (panel.cuh), every wait ends, and
// no CTA leaves before the pushes to it are done.  The caller checks the error
// word, the interchanges and the moves.
#define gblu gblu_panelcheck  // apart from the library's instances of the same kernels
#define GBLU_SPIN_TIMEOUT_NS 1000000ull  // 1 ms

#include <cuda_runtime.h>
#include <stdint.h>

#include "../waits.cuh"

namespace {
constexpr unsigned long long kLateNs = 50000000ull;  // 50 ms

// Pushes CTA 1 has begun, and the one it is late with.
__device__ int late_count, late_at;

__device__ __forceinline__ void late_st_async(uint32_t raddr, int4 v, uint32_t rbar) {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  if (rank == 1 && atomicAdd(&late_count, 1) == late_at) {
    const unsigned long long t0 = gblu::global_ns();
    while (gblu::global_ns() - t0 < kLateNs) {}
  }
  gblu::pan_st_async(raddr, v, rbar);
}
}  // namespace

#define pan_st_async late_st_async
#include "../panel.cuh"
#undef pan_st_async

namespace {

template <typename T, int NT, int NWC, int RPT, int W>
int32_t run(T* A, int64_t m, int32_t ctas, int64_t* ipiv, int64_t* info, gblu::LeafMoves* moves, gblu::DevScratch* scr) {
  auto* kern = gblu::panel_sub_kernel<T, NT, NWC, RPT, W>;
  const int64_t R = (m + ctas - 1) / ctas;
  if (R > 32 * NWC * RPT || W > m) return 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = (size_t)R * gblu::panel_sub_ld<T, W>() * sizeof(T);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return 2;
  const unsigned rmagic = (unsigned)(((1ull << 32) + R - 1) / R);
  if (cudaLaunchKernelEx(&cfg, kern, A, m, m, (int64_t)0, W, ipiv, info, (int)R, rmagic, moves, scr) != cudaSuccess) return 3;
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 4;
}

}  // namespace

// Factors the m x W panel A (host, leading dimension m; FP64: m of 64 .. 512, W =
// 64; FP32: m of 513 .. 1024, W = 128) with CTA 1 late at its push number `at`
// (-1: never).  ipiv: W entries; moves: 2 * 256 entries, count of them.
extern "C" int32_t gblu_tool_panelcheck(int32_t fp64, int64_t m, void* A, int32_t at, int64_t* ipiv, int32_t* moves,
                                        int32_t* count, int32_t* code) {
  const int W = fp64 ? 64 : 128;
  if (m < (fp64 ? 64 : 513) || m > (fp64 ? 512 : 1024) || !A || !ipiv || !moves || !count || !code) return 1;
  const size_t bytes = (size_t)m * W * (fp64 ? 8 : 4);
  unsigned char* d = nullptr;
  const size_t o_ipiv = (bytes + 255) & ~size_t(255), o_info = o_ipiv + 1024, o_scr = o_info + 256, o_mv = o_scr + 256;
  if (cudaMalloc(&d, o_mv + sizeof(gblu::LeafMoves)) != cudaSuccess) return 2;
  cudaMemset(d, 0, o_mv + sizeof(gblu::LeafMoves));
  cudaMemcpy(d, A, bytes, cudaMemcpyHostToDevice);
  const int zero = 0;
  cudaMemcpyToSymbol(late_count, &zero, sizeof(int));
  cudaMemcpyToSymbol(late_at, &at, sizeof(int));
  int64_t* di = reinterpret_cast<int64_t*>(d + o_ipiv);
  int64_t* dn = reinterpret_cast<int64_t*>(d + o_info);
  auto* scr = reinterpret_cast<gblu::DevScratch*>(d + o_scr);
  auto* mv = reinterpret_cast<gblu::LeafMoves*>(d + o_mv);
  int32_t rc = fp64 ? run<double, 256, 1, 1, 64>(reinterpret_cast<double*>(d), m, (int32_t)((m + 31) / 32), di, dn, mv, scr)
                    : run<float, 256, 2, 1, 128>(reinterpret_cast<float*>(d), m, 16, di, dn, mv, scr);
  gblu::DevScratch hs{};
  static gblu::LeafMoves hm;
  if (rc == 0 && (cudaMemcpy(A, d, bytes, cudaMemcpyDeviceToHost) != cudaSuccess ||
                  cudaMemcpy(ipiv, di, W * sizeof(int64_t), cudaMemcpyDeviceToHost) != cudaSuccess ||
                  cudaMemcpy(&hs, scr, sizeof(hs), cudaMemcpyDeviceToHost) != cudaSuccess ||
                  cudaMemcpy(&hm, mv, sizeof(hm), cudaMemcpyDeviceToHost) != cudaSuccess))
    rc = 5;
  cudaFree(d);
  if (rc) return rc;
  *code = hs.error;
  *count = hm.count;
  for (int i = 0; i < 2 * gblu::kLeafMaxW; ++i) moves[2 * i] = hm.mv[i].x, moves[2 * i + 1] = hm.mv[i].y;
  return 0;
}
