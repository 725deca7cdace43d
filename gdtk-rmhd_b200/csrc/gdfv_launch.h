// gdfv_launch.h -- interface between the host runtime and the two kernel
// translation units (FP64 flux and FP32 flux, compiled with different flags).
#pragma once
#include <cuda_runtime.h>

#include "gdfv_stage.cuh"

namespace gdfv {

// Rows of cells per column tile (the tile is 32 x TJ columns) of each flux precision.
#ifndef GDFV_TJ_FP64
#define GDFV_TJ_FP64 6
#endif
#ifndef GDFV_TJ_FP32
#define GDFV_TJ_FP32 8
#endif
// rows of the float-flux MHD kernels (their ten variables need more shared memory per row)
#ifndef GDFV_TJ_FP32_MHD
#define GDFV_TJ_FP32_MHD 7
#endif
// rows of the float-flux Euler corrector: with 7 rows its CTAs of 256 threads get 80
// registers (fewer spills) at the same 3 CTAs per SM
#ifndef GDFV_TJ_FP32_CORR
#define GDFV_TJ_FP32_CORR 7
#endif
// rows of the FP64 MHD kernels (one CTA per SM: their shared memory allows no second)
#ifndef GDFV_TJ_FP64_MHD
#define GDFV_TJ_FP64_MHD 7
#endif
// rows of the FP64 Euler corrector (by default those of the FP64 kernels)
#ifndef GDFV_TJ_FP64_CORR
#define GDFV_TJ_FP64_CORR GDFV_TJ_FP64
#endif
// rows of the float-flux MHD corrector (by default those of the float MHD kernels)
#ifndef GDFV_TJ_FP32_MHD_CORR
#define GDFV_TJ_FP32_MHD_CORR GDFV_TJ_FP32_MHD
#endif
constexpr int TJ_FP64 = GDFV_TJ_FP64;
constexpr int TJ_FP32_MHD_CORR = GDFV_TJ_FP32_MHD_CORR;
constexpr int TJ_FP64_CORR = GDFV_TJ_FP64_CORR;
constexpr int TJ_FP64_MHD = GDFV_TJ_FP64_MHD;
constexpr int TJ_FP32_CORR = GDFV_TJ_FP32_CORR;
constexpr int TJ_FP32 = GDFV_TJ_FP32;
constexpr int TJ_FP32_MHD = GDFV_TJ_FP32_MHD;

// Rows per column tile of the kernels a run launches.
inline int tile_rows(int precision, bool mhd) {
    return precision == 0 ? (mhd ? TJ_FP64_MHD : TJ_FP64) : (mhd ? TJ_FP32_MHD : TJ_FP32);
}
// Rows per column tile of the corrector (stage 2) of a run.
inline int tile_rows_corrector(int precision, bool mhd) {
    return precision == 0 ? (mhd ? TJ_FP64_MHD : TJ_FP64_CORR) : (mhd ? TJ_FP32_MHD_CORR : TJ_FP32_CORR);
}

// CTAs of the stage kernels resident on one SM (their launch bounds; FP64 MHD: their shared memory).
inline int tile_ctas_per_sm(int precision, bool mhd) {
    return precision == 0 ? (mhd ? 1 : GDFV_MINB_FP64) : (mhd ? GDFV_MINB_MHD_FP32 : GDFV_MINB_FP32);
}

// CTAs per SM the FP64 line sweeps are compiled for: 128 registers (Euler), 255 (MHD, no spills;
// 3 and 4 CTAs spill 0.2 and 0.4 KB: Orszag-Tang 512x512x4 both stages 776 / 830 / 901 us with 2 /
// 3 / 4, 256x256x4 240 / 268 / 263 us)
#ifndef GDFV_MARCH_MINB
#define GDFV_MARCH_MINB 4
#endif
#ifndef GDFV_MARCH_MINB_MHD
#define GDFV_MARCH_MINB_MHD 2
#endif
inline int sweep_ctas_per_sm(bool mhd) { return mhd ? GDFV_MARCH_MINB_MHD : GDFV_MARCH_MINB; }

// Options under which the float-flux Euler stages run the kernel on decoded primitives
// (gdfv_stage_prim.cuh) when the arguments carry primitive buffers (the FP64 form keeps
// stage_kernel, which ran faster than an FP64 build of the primitive kernel): the
// defaults (limiter and extrema clipping on, e4 epsilon), no outflow boundary with a
// flux or ghost rule of its own, no graded block, no exchange with an Rmatrix, 3D.
inline bool prim_path(const NumParams& P) {
    return !P.mhd && P.apply_limiter && P.extrema_clipping && !P.lmr_epsilon && !P.outflow_bcs && !P.graded &&
           !P.rotating && P.dims == 3;
}

// Launch one stage (0 = residual only, 1 = predictor, 2 = corrector) over A.n_tiles tiles.
cudaError_t launch_stage_fp64(int stage, int flux, bool mhd, const StageArgs& A, cudaStream_t s);
cudaError_t launch_stage_fp32(int stage, int flux, bool mhd, const StageArgs& A, cudaStream_t s);
// Primitives (rho, vel, u, a; SoA [6][total], float or double) of the state U, for the
// kernels on decoded primitives, enqueued on stream s.
void prims_fp32(const double* U, long long total, const NumParams& P, void* Pout, cudaStream_t s);
// One stage (0, 1 or 2) as FP64 line sweeps (A.sweep_off set; gdfv_sweep.cuh), their tiles of
// one direction of a block, and the FP64 primitives (6 or, MHD, 10 per cell) of the state U.
cudaError_t launch_sweeps(int stage, int flux, bool mhd, const StageArgs& A, cudaStream_t s);
long long sweep_tile_count(const int* n, int D, int cells);
void prims_fp64(const double* U, long long total, const NumParams& P, bool mhd, void* Pout, cudaStream_t s);
// Raise the dynamic shared-memory limit of every instantiation (once per device).
cudaError_t configure_stage_fp64();
cudaError_t configure_stage_fp32();

}  // namespace gdfv
