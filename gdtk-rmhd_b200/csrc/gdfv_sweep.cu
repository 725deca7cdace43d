// gdfv_sweep.cu -- instantiations and launch of the FP64 line sweeps (compiled without FMA
// contraction, as gdfv_stage_fp64.cu).
#include "gdfv_launch.h"
#include "gdfv_sweep.cuh"

namespace gdfv {

namespace {
template <bool MHD, int FLUX, int OPT, int D, bool LAST>
cudaError_t sweep_one(const StageArgs& A, int stage, cudaStream_t s) {
    if (A.sweep_tiles[D] <= 0) return cudaSuccess;
    constexpr size_t bytes = D == 0 ? 0 : march_bytes<MHD, LAST>();
    static_assert(bytes <= 48 * 1024, "above the default limit");
    sweep_kernel<MHD, FLUX, OPT, D, LAST><<<A.sweep_tiles[D], SWEEP_LINES, bytes, s>>>(A, stage);
    return cudaGetLastError();
}

template <bool MHD, int FLUX, int OPT>
cudaError_t sweeps(const StageArgs& A, int stage, cudaStream_t s) {
    cudaError_t e = sweep_one<MHD, FLUX, OPT, 0, false>(A, stage, s);
    if (e != cudaSuccess) return e;
    if (A.P.dims == 2) return sweep_one<MHD, FLUX, OPT, 1, true>(A, stage, s);
    e = sweep_one<MHD, FLUX, OPT, 1, false>(A, stage, s);
    return e == cudaSuccess ? sweep_one<MHD, FLUX, OPT, 2, true>(A, stage, s) : e;
}

// OPT as in launch_rows: the defaults, or every option
template <bool MHD, int FLUX>
cudaError_t sweeps_opt(const StageArgs& A, int stage, cudaStream_t s) {
    if (A.P.apply_limiter && A.P.extrema_clipping && !A.P.lmr_epsilon && !A.P.outflow_bcs && !A.P.graded)
        return sweeps<MHD, FLUX, 1>(A, stage, s);
    return sweeps<MHD, FLUX, 0>(A, stage, s);
}

}  // namespace

cudaError_t launch_sweeps(int stage, int flux, bool mhd, const StageArgs& A, cudaStream_t s) {
    if (mhd) return flux == FLUX_HLLE ? sweeps_opt<true, FLUX_HLLE>(A, stage, s) : cudaErrorInvalidValue;
    if (flux == FLUX_AUSMDV) return sweeps_opt<false, FLUX_AUSMDV>(A, stage, s);
    if (flux == FLUX_HLLC) return sweeps_opt<false, FLUX_HLLC>(A, stage, s);
    return cudaErrorInvalidValue;
}

void prims_fp64(const double* U, long long total, const NumParams& P, bool mhd, void* Pout, cudaStream_t s) {
    const unsigned nb = (unsigned)((total + 255) / 256);
    if (mhd) sweep_prims_kernel<true><<<nb, 256, 0, s>>>(U, total, P, static_cast<double*>(Pout));
    else sweep_prims_kernel<false><<<nb, 256, 0, s>>>(U, total, P, static_cast<double*>(Pout));
}

long long sweep_tile_count(const int* n, int D, int cells) { return sweep_tiles(n, D, cells); }

}  // namespace gdfv
