// Launch of the sub-panel cluster kernel (panel.cuh): which leaves it takes,
// its leaf width, and the CTAs, warps and rows per thread by height.
#include <cuda_runtime.h>

#include <algorithm>

#include "gblu_internal.h"
#include "panel.cuh"
#include "profile.h"

namespace gblu {

namespace {

// CTAs of a leaf of M rows.  FP64: 32 rows a CTA up to the 16 of a cluster (a
// warp issues one FP64 instruction in 68 cycles however many of its lanes are
// active, so rows are spread as thin as a warp).  FP32: one CTA up to 256 rows
// (a column then costs a CTA barrier instead of an exchange across the
// cluster: 24-26 us a 32-column leaf against 30 at 16 CTAs), else all 16.
template <typename T>
int sub_ctas(int64_t M) {
  if (sizeof(T) == 8) return (int)std::min<int64_t>(kSubMaxCtas, std::max<int64_t>(1, (M + 31) / 32));
  return M <= 256 ? 1 : kSubMaxCtas;
}

template <typename T, int NT, int NWC, int RPT, int W>
cudaError_t sub_launch(T* A, int64_t lda, int64_t m, int64_t c0, int w, int64_t* ipiv, int64_t* info,
                       LeafMoves* moves, DevScratch* scr, int ctas, bool query, cudaStream_t s) {
  const int64_t M = m - c0;
  const int64_t R = (M + ctas - 1) / ctas;
  auto* kern = panel_sub_kernel<T, NT, NWC, RPT, W>;
  constexpr int kRowsMax = 32 * NWC * RPT;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = (size_t)(query ? kRowsMax : R) * panel_sub_ld<T, W>() * sizeof(T);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (query) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    int clusters = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    if (e == cudaSuccess && clusters < 1) e = cudaErrorInvalidConfiguration;
    return e;
  }
  if (R > kRowsMax || w > W || w > M) return cudaErrorInvalidValue;
  double fl = 0;
  for (int k = 0; k < w; ++k) fl += (double)(M - k - 1) * (1.0 + 2.0 * (w - k - 1));
  LaunchScope ls(K_PANEL, fl, 2.0 * M * w * sizeof(T), s);
  const unsigned rmagic = (unsigned)(((1ull << 32) + R - 1) / R);  // row / R for row * R < 2^32
  return cudaLaunchKernelEx(&cfg, kern, A, lda, m, c0, w, ipiv, info, (int)R, rmagic, moves, scr);
}

// The variant for M rows (0: none); FP64 up to 8192 rows, FP32 up to 16384.
template <typename T>
int sub_variant(int64_t M) {
  if (M < 1) return 0;
  if (sizeof(T) == 8) return M <= 512 ? 1 : M <= 1024 ? 2 : M <= 2048 ? 3 : M <= 4096 ? 4 : M <= 8192 ? 5 : 0;
  return M <= 32 ? 1 : M <= 128 ? 2 : M <= 256 ? 3 : M <= 512 ? 1 : M <= 1024 ? 4 : M <= 2048 ? 2 : M <= 4096 ? 3
         : M <= 8192 ? 5 : M <= 16384 ? 6 : 0;
}

// Rows per thread and chain warps so that a CTA's rows fill its chain warps
// once or twice; the leaf as wide as its rows leave room in shared memory.
// A wider leaf saves the interchange, TRSM and update launches of the levels
// below it; its rank-8 updates run in the helper warps beside the column chain.
template <typename T>
cudaError_t sub_dispatch(int v, T* A, int64_t lda, int64_t m, int64_t c0, int w, int64_t* ipiv, int64_t* info,
                         LeafMoves* mv, DevScratch* scr, int ctas, bool query, cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    switch (v) {
      case 1: return sub_launch<T, 256, 1, 1, 64>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 2: return sub_launch<T, 256, 2, 1, 64>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 3: return sub_launch<T, 256, 4, 1, 64>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 4: return sub_launch<T, 512, 8, 1, 64>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 5: return sub_launch<T, 512, 8, 2, 32>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
    }
  } else {
    switch (v) {
      case 1: return sub_launch<T, 256, 1, 1, 128>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 2: return sub_launch<T, 256, 4, 1, 128>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 3: return sub_launch<T, 512, 8, 1, 128>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 4: return sub_launch<T, 256, 2, 1, 128>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 5: return sub_launch<T, 512, 8, 2, 64>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
      case 6: return sub_launch<T, 512, 8, 4, 32>(A, lda, m, c0, w, ipiv, info, mv, scr, ctas, query, s);
    }
  }
  return cudaErrorInvalidValue;
}

}  // namespace

namespace {

// Per device, as the kernels' attributes are (cudaFuncSetAttribute changes them
// for the current device only).
template <typename T>
bool& sub_ready(int device) {
  static bool ready[64] = {false};
  return ready[device];
}

}  // namespace

template <typename T>
void panel_sub_configure(int device) {
  if (device < 0 || device >= 64) return;
  bool ok = true;
  for (int v = 1; v <= (sizeof(T) == 8 ? 5 : 6); ++v)
    ok = ok && sub_dispatch<T>(v, nullptr, 0, 0, 0, 0, nullptr, nullptr, nullptr, nullptr, kSubMaxCtas, true,
                               nullptr) == cudaSuccess;
  cudaGetLastError();
  sub_ready<T>(device) = ok;
}

template <typename T>
int panel_sub_width(int device, int64_t M) {
  if (device < 0 || device >= 64 || sub_variant<T>(M) == 0 || !sub_ready<T>(device)) return 0;
  if (sizeof(T) == 8) return M <= 4096 ? 64 : 32;
  return M <= 4096 ? 128 : M <= 8192 ? 64 : 32;
}

template <typename T>
cudaError_t panel_sub_launch(T* A, int64_t lda, int64_t m, int64_t c0, int w, int64_t* ipiv, int64_t* info,
                             LeafMoves* moves, DevScratch* scr, cudaStream_t s) {
  const int64_t M = m - c0;
  return sub_dispatch<T>(sub_variant<T>(M), A, lda, m, c0, w, ipiv, info, moves, scr, sub_ctas<T>(M), false, s);
}

template void panel_sub_configure<double>(int);
template void panel_sub_configure<float>(int);
template int panel_sub_width<double>(int, int64_t);
template int panel_sub_width<float>(int, int64_t);
template cudaError_t panel_sub_launch<double>(double*, int64_t, int64_t, int64_t, int, int64_t*, int64_t*, LeafMoves*,
                                              DevScratch*, cudaStream_t);
template cudaError_t panel_sub_launch<float>(float*, int64_t, int64_t, int64_t, int, int64_t*, int64_t*, LeafMoves*,
                                             DevScratch*, cudaStream_t);

}  // namespace gblu
