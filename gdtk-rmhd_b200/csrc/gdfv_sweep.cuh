// gdfv_sweep.cuh -- FP64 stages as line sweeps: one launch per grid direction, each adding its
// two faces' fluxes to the residual sums of the cells, the last one finishing the stage.
//
// Why beside stage_kernel: the FP64 fluxes and limiters are chains of dependent FP64
// operations (latency 8.5 cycles, one warp instruction per 2 cycles and scheduler), and the
// fused kernel holds the planes of three directions in shared memory between barriers: 14
// warps per SM (MHD: 8) that wait on each other, 35% of the FP64 pipe.  A sweep along one
// direction needs no barrier and hardly any exchange: along j and k a thread walks a stretch
// of one grid line (i runs over the lanes, so every access is coalesced) with its window of
// three cells, the last plus-face state and the last flux in registers, and a cell's loads are
// under way (cp.async into the thread's own shared memory) while the cell before it is
// computed; along i the lanes of a warp are neighbouring cells of a row and exchange states and
// fluxes by shuffles.  830 to 1,270 thread instructions per cell and sweep, 57 to 63% issue
// active at 14 warps (16 fit), and no re-evaluation but at the ends of stretches.  It pays with
// memory traffic -- the primitives are read in every sweep and the sums go through memory twice,
// 400 to 440 B per cell and stage for Euler against 120 -- which stays below the arithmetic.
//
// Measured (both stages, one B200, stage_kernel at its best tiles / sweeps): 256^3 ausmdv 6.38
// / 4.18 ms, 128x128x64 506 / 367 us, graded hllc 121x85x61 449 / 324 us, Orszag-Tang
// 256x256x4 271 / 240 us, 512x512x4 1,112 / 784 us.  Tried and slower: the sweeps with one
// thread per cell of a tile, passing states and fluxes in shared memory between barriers
// (5.07 ms at 256^3 at 24 warps and 80 registers, the same at 16 and 32 warps); the residual
// sums and U staged in shared memory there (6.3 ms); the walk with its loads in registers
// (5.0 ms) and at 5 or 6 CTAs per SM (spills; 5.3 ms).
//
// Bit for bit stage_kernel's FP64 results: the same functions per cell and face
// (recon_cell, face_flux) and the reference's order of the residual sum, W, E, S, N, B, T
// (time_derivatives, e4/fvcell.d:824-856), whose partial sums the sweeps hand on.
//
// The stages read decoded primitives (rho, vel, u, a and for MHD B, psi; SoA), which each
// stage stores of the state it produces, as the float kernel on decoded primitives does.
#pragma once
#include "gdfv_launch.h"

namespace gdfv {

constexpr int SWEEP_LINES = 128;   // threads per CTA
constexpr int SWEEP_WINDOWS = 8;   // windows of 32 slots per warp of the i sweep
// Tiles of direction D of a block; cells: those a tile updates along j and k.
inline long long sweep_tiles(const int* n, int D, int cells) {
    if (D == 0) {   // CTAs of four warps
        const long long slots = (long long)(n[0] + 2) * n[1] * n[2], per = 32 * SWEEP_WINDOWS - 2;
        return ((slots - 2 + per - 1) / per + SWEEP_LINES / 32 - 1) / (SWEEP_LINES / 32);
    }
    const long long lines = (long long)n[0] * (D == 1 ? n[2] : n[1]);
    return (lines + SWEEP_LINES - 1) / SWEEP_LINES * ((n[D] + cells - 1) / cells);
}

template <bool MHD>
__device__ __forceinline__ Prim<double> load_prim(const double* __restrict__ P, long long total, long long g) {
    Prim<double> s;
    s.rho = __ldg(P + g);
    s.v[0] = __ldg(P + total + g);
    s.v[1] = __ldg(P + 2 * total + g);
    s.v[2] = __ldg(P + 3 * total + g);
    s.u = __ldg(P + 4 * total + g);
    s.a = __ldg(P + 5 * total + g);
    if (MHD) {
        s.B[0] = __ldg(P + 6 * total + g);
        s.B[1] = __ldg(P + 7 * total + g);
        s.B[2] = __ldg(P + 8 * total + g);
        s.psi = __ldg(P + 9 * total + g);
    }
    return s;
}
template <bool MHD>
__device__ __forceinline__ void store_prim(double* __restrict__ P, long long total, long long g, const Prim<double>& s) {
    P[g] = s.rho;
    P[total + g] = s.v[0];
    P[2 * total + g] = s.v[1];
    P[3 * total + g] = s.v[2];
    P[4 * total + g] = s.u;
    P[5 * total + g] = s.a;
    if (MHD) {
        P[6 * total + g] = s.B[0];
        P[7 * total + g] = s.B[1];
        P[8 * total + g] = s.B[2];
        P[9 * total + g] = s.psi;
    }
}

// The ghost (i, j, k) of block B from the primitives of its source cells: finish_cell's
// rules (the source's decoded state is what P holds).
template <bool MHD>
__device__ __noinline__ Prim<double> sweep_ghost(const StageArgs& A, const double* Pin, const BlockDesc& B, int i, int j,
                                                 int k) {
    const CellSrc s = resolve<true, true>(A, B, i, j, k);
    Prim<double> out;
    if (s.kind == SRC_INFLOW) {
        const InflowState& in = A.inflow[s.inflow];
        out.rho = in.rho; out.u = in.u; out.a = in.a; out.psi = in.psi;
        for (int m = 0; m < 3; ++m) { out.v[m] = in.vel[m]; out.B[m] = in.B[m]; }
        return out;
    }
    out = load_prim<MHD>(Pin, A.total, s.blk->offset + s.c0);
    if (s.kind == SRC_MIRROR) {
        out.v[s.axis] = -out.v[s.axis];
        if (MHD) {
            const double x = B.x0 + ((double)i + 0.5) * B.len[0], y = B.y0 + ((double)j + 0.5) * B.len[1];
            if (x > -0.4136 && x < 0.4136) dipole_field(x, y, out.B[0], out.B[1]);
        }
    } else if (s.kind == SRC_ROTATE) {
        out = rotate_vectors<MHD>(A.rot + 9 * s.inflow, out);
    } else if (s.kind == SRC_FIXEDP || s.kind == SRC_FIXEDPT) {
        const InflowState& o = A.inflow[s.inflow];
        out = fixed_ghost(out, s.kind == SRC_FIXEDP, o.p, o.rho, o.u, A.P.gas.Cvinv, A.P.gas.Cv, A.P.gas.R);
    } else if (s.kind == SRC_EXTRAP1_G0 || s.kind == SRC_EXTRAP1_G1) {
        const Prim<double> f1 = load_prim<MHD>(Pin, A.total, s.blk->offset + s.c1);
        Prim<double> g0;
        extrapolate<MHD>(f1, out, out, g0);
        if (s.kind == SRC_EXTRAP1_G0) return g0;
        Prim<double> g1;
        extrapolate<MHD>(out, g0, out, g1);
        return g1;
    }
    return out;
}

// Where the ghost (i, j, k) of block B comes from when it is a copy of a cell: g >= 0 its global
// index, neg the primitive to negate (0: none); g < 0: sweep_ghost forms it.
struct GhostCopy {
    long long g;
    int neg;
};
template <bool MHD>
__device__ __noinline__ GhostCopy ghost_copy(const StageArgs& A, const BlockDesc& B, int i, int j, int k) {
    const CellSrc s = resolve<true, true>(A, B, i, j, k);
    if (s.kind == SRC_CELL) return GhostCopy{s.blk->offset + s.c0, 0};
    if (!MHD && s.kind == SRC_MIRROR) return GhostCopy{s.blk->offset + s.c0, 1 + s.axis};
    return GhostCopy{-1, 0};
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Shared memory of a thread of the j and k sweeps: what the end of its current cell reads (the
// primitives of the cell after next, the residual sums and, in the last sweep, U and dU0),
// brought there asynchronously from the cell's start on: [MARCH_SLOTS][128].
template <bool MHD, bool LAST>
constexpr int march_slots() { return (MHD ? 10 : 6) + (LAST ? 3 : 1) * (MHD ? 10 : 5); }
template <bool MHD, bool LAST>
constexpr size_t march_bytes() { return sizeof(double) * (size_t)march_slots<MHD, LAST>() * SWEEP_LINES; }

// What a sweep hands to each cell: place, face area along D, volume, own lengths.
template <int D, int OPT>
__device__ __forceinline__ double face_area(const StageArgs& A, const BlockDesc& B, int i, int j, int k) {
    if (OPT == 0 && B.graded) {
        double L[3];
        cell_lengths(B, i, j, k, L);
        if (A.P.dims == 3) return D == 0 ? d_mul(L[1], L[2]) : (D == 1 ? d_mul(L[2], L[0]) : d_mul(L[0], L[1]));
        return D == 0 ? L[1] : L[0];
    }
    return B.area[D];
}

// The end of a stage for one cell whose residual sum si is complete: dU = si / volume, then
// R(U) (stage 0), the predictor (1) or the corrector (2) with decode, checks, primitives of
// the new state and signal frequency, as stage_kernel's phase D.  SU: the thread's U and dU0 in
// shared memory.
template <bool MHD, int OPT>
__device__ __forceinline__ void sweep_finish(const StageArgs& A, int stage, const BlockDesc& B, int blk, int i, int j,
                                             int k, long long g, int parity, double dt, double damp, const double* si,
                                             const double* SU, double& sig_max) {
    constexpr int NQ = MHD ? 10 : 5;
    const NumParams& P = A.P;
    const long long total = A.total;
    double vol_inv = B.vol_inv;
    double clen[3] = {B.len[0], B.len[1], B.len[2]};
    if (OPT == 0 && B.graded) {
        cell_lengths(B, i, j, k, clen);
        vol_inv = P.dims == 3 ? 1.0 / d_mul(d_mul(clen[0], clen[1]), clen[2]) : 1.0 / d_mul(clen[0], clen[1]);
    }
    if (stage == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) A.R_out[(long long)q * total + g] = d_add(d_mul(vol_inv, si[q]), 0.0);
        return;
    }
    constexpr int LN = SWEEP_LINES;
    double U[NQ];
    if (stage == 1) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double dU = d_add(d_mul(vol_inv, si[q]), 0.0);
            A.dU0[(long long)q * total + g] = dU;
            U[q] = d_add(SU[q * LN], d_mul(dt, dU));
        }
        if (A.R_out) {   // U1 before the psi damping
#pragma unroll
            for (int q = 0; q < NQ; ++q) A.R_out[(long long)q * total + g] = U[q];
        }
        if (MHD && P.divergence_cleaning) U[PSI] = d_mul(U[PSI], damp);
    } else {
        double* Uout = A.Ubuf[parity ^ 1];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double dU = d_add(d_mul(vol_inv, si[q]), 0.0);
            const double d0 = SU[(NQ + q) * LN];
            U[q] = d_add(SU[q * LN], d_mul(dt, d_add(d_mul(0.5, d0), d_mul(0.5, dU))));
            if (MHD && q == PSI && P.divergence_cleaning) U[PSI] = d_mul(U[PSI], damp);
            Uout[(long long)q * total + g] = U[q];
        }
    }
    Prim<double> s;
    double p, T;
    if (decode(P, U, s, p, T) != 0) {
        atomicAdd(&A.ctl->n_fail, 1);
        atomicMin(reinterpret_cast<unsigned long long*>(&A.ctl->first_bad_cell), (unsigned long long)g);
        return;
    }
    store_prim<MHD>(static_cast<double*>(stage == 1 ? A.prim1 : A.prim[parity ^ 1]), total, g, s);
    if (!check_data(P, s, p, T)) {
        atomicAdd(stage == 1 ? &A.ctl->n_invalid1 : &A.ctl->n_invalid2, 1);
        atomicMin(reinterpret_cast<unsigned long long*>(&A.ctl->first_bad_cell), (unsigned long long)g);
    }
    if (stage == 2) {
        const double sig = signal_frequency(P, clen, s);
        sig_max = fmax(sig_max, sig);
        if (i == B.n[0] - 1 && j == B.n[1] - 1 && k == B.n[2] - 1) A.last_signal[blk] = sig;
    }
}

// The reconstruction of a cell (values before, at and after it) whose limiters are out of the
// branch-free quotients' range: minus- and plus-face values.
template <int N>
struct Values { double q[N]; };
template <int NRS, bool MHD, int OPT, int D>
__device__ __noinline__ Values<2 * NRS> recon_out_of_range(const NumParams& P, const BlockDesc& B, int c,
                                                           Values<NRS> q1, Values<NRS> q0, Values<NRS> q2) {
    Values<2 * NRS> r;
    if (OPT == 0 && B.graded)
        recon_cell_graded_of<double, NRS, MHD, false>(B.gw[D] + (long long)(c + 1) * GW_N, P, q1.q, q0.q, q2.q, r.q,
                                                      r.q + NRS);
    else
        recon_cell_of<double, NRS, MHD, OPT, false>(B.w[D], P, q1.q, q0.q, q2.q, r.q, r.q + NRS);
    return r;
}

// D: direction; LAST: the sweep that finishes the stage (k, or j in 2D).  A.sweep_part holds the
// residual sums between sweeps; stage 0 reads the primitives of its state from A.prim1.
template <bool MHD, int FLUX, int OPT, int D, bool LAST>
__global__ void __launch_bounds__(SWEEP_LINES, MHD ? GDFV_MARCH_MINB_MHD : GDFV_MARCH_MINB)
    sweep_kernel(const __grid_constant__ StageArgs A, int stage) {
    constexpr int NPV = MHD ? 10 : 6, NRS = MHD ? 9 : 5, NQ = MHD ? 10 : 5;
    __shared__ double s_red[SWEEP_LINES / 32];

    const Control* ctl = A.ctl;
    int parity = 0;
    double dt = 0.0;
    if (stage != 0) {
        if (ctl->halted || ctl->status != ST_OK) return;
        if (stage == 2 && (ctl->n_fail > 0 || ctl->n_invalid1 > A.max_invalid_cells)) return;
        parity = ctl->step & 1;
        dt = ctl->dt_global;
    }
    const double c_h = ctl->c_h;
    double damp = 1.0;
    if (LAST && MHD && A.P.divergence_cleaning && stage != 0) {
        // e4/fvcell.d:1068-1074 divergence_damping_factor
        const double c_h2 = c_h * c_h;
        const double c_p2 = 0.18 * A.P.divB_damping_length * c_h;
        damp = exp(-(c_h2 / c_p2) * dt);
    }
    const NumParams& P = A.P;
    const long long total = A.total;
    const double* __restrict__ Pin = static_cast<const double*>(stage == 1 ? A.prim[parity] : A.prim1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long* off = A.sweep_off + D * (A.sweep_blocks + 1);

    // reconstruction of cell c from the primitives of the cells before, at and after it, and the
    // flux of the face between cell c - 1 (lo) and cell c (at)
    auto recon = [&](const BlockDesc& B, int c, const double* lo, const double* at, const double* hi, double* qm,
                     double* qp) {
        double q1[NRS], q0[NRS], q2[NRS];
        gather<double, NRS, D>(lo, 1, 0, q1);
        gather<double, NRS, D>(at, 1, 0, q0);
        gather<double, NRS, D>(hi, 1, 0, q2);
        bool done;
        if (OPT == 0 && B.graded)
            done = recon_cell_graded<double, NRS, MHD>(B.gw[D] + (long long)(c + 1) * GW_N, P, q1, q0, q2, qm, qp);
        else
            done = recon_cell<double, NRS, MHD, OPT>(B.w[D], nullptr, P, q1, q0, q2, qm, qp);
        if (!done) {
            Values<NRS> v1, v0, v2;
#pragma unroll
            for (int s = 0; s < NRS; ++s) { v1.q[s] = q1[s]; v0.q[s] = q0[s]; v2.q[s] = q2[s]; }
            const Values<2 * NRS> r = recon_out_of_range<NRS, MHD, OPT, D>(P, B, c, v1, v0, v2);
#pragma unroll
            for (int s = 0; s < NRS; ++s) { qm[s] = r.q[s]; qp[s] = r.q[NRS + s]; }
        }
    };
    auto flux = [&](const BlockDesc& B, int c, const double* lo, const double* at, const double* qL,
                    const double* qR, double* F) {
        face_flux<double, MHD, FLUX, D, NPV>(P, c_h, qL, qR, lo, 0, at, 0, 1, F);
        if constexpr (OPT == 0 && !MHD) {
            // OutFlowBC_SimpleFlux: the boundary face's flux is the interior cell's (boundary_flux_effect.d:504-645)
            if (c == 0 && B.bc_type[2 * D] == BC_SIMPLE_FLUX) simple_outflow_flux<double, D>(P, at, 0, 1, -1, F);
            if (c == B.n[D] && B.bc_type[2 * D + 1] == BC_SIMPLE_FLUX)
                simple_outflow_flux<double, D>(P, lo, 0, 1, 1, F);
        }
    };

    // primitives of cell c of the line through (i, j, k), g the global index they would have
    auto load = [&](const BlockDesc& B, int c, int i, int j, int k, long long g, double* p) {
        if (c < 0 || c >= B.n[D]) {
            const GhostCopy s = ghost_copy<MHD>(A, B, D == 0 ? c : i, D == 1 ? c : j, D == 2 ? c : k);
            if (s.g < 0) {
                const Prim<double> t = sweep_ghost<MHD>(A, Pin, B, D == 0 ? c : i, D == 1 ? c : j, D == 2 ? c : k);
                put_prim<double, NPV>(p, 1, 0, t);
                return;
            }
#pragma unroll
            for (int v = 0; v < NPV; ++v) p[v] = __ldg(Pin + (long long)v * total + s.g);
            if (s.neg) p[1 + D] = -p[1 + D];   // a mirror negates the normal velocity
            return;
        }
#pragma unroll
        for (int v = 0; v < NPV; ++v) p[v] = __ldg(Pin + (long long)v * total + g);
    };

    if constexpr (D == 0) {
        // a warp's stretch of the stream of slots (rows of n0 + 2: cells -1 .. n0), 32 at a time
        const unsigned full = 0xffffffffu;
        const int b = block_of_tile(off, A.sweep_blocks, blockIdx.x);
        const BlockDesc& B = A.blocks[b];
        const int n0 = B.n[0], n1 = B.n[1];
        const unsigned n2 = (unsigned)n0 + 2;
        const unsigned long long slots = (unsigned long long)n2 * ((unsigned long long)n1 * B.n[2]);
        const unsigned long long x0 = ((unsigned long long)(blockIdx.x - off[b]) * (SWEEP_LINES / 32) + warp) *
                                      (32 * SWEEP_WINDOWS - 2);
        double qp_end[NRS], F_end[NQ];   // of the last slot of the window before
#pragma unroll
        for (int v = 0; v < NRS; ++v) qp_end[v] = 0.0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) F_end[q] = 0.0;
        for (int w = 0; w < SWEEP_WINDOWS; ++w) {
            const unsigned long long x = x0 + (unsigned)(32 * w + lane);
            if (x0 + 32u * w >= slots) break;   // (the same for the whole warp)
            const bool valid = x < slots;
            const unsigned xs = valid ? (unsigned)x : 0u, l = xs / n2;
            const int c = (int)(xs - l * n2) - 1;
            const int k = (int)(l / (unsigned)n1), j = (int)(l - (unsigned)k * (unsigned)n1);
            const long long g = B.offset + (long long)n0 * l + c;
            double pm[NPV], p0[NPV], qm[NRS], qp[NRS], qL[NRS], F[NQ];
            {
                double pp[NPV];
                load(B, c - 1, 0, j, k, g - 1, pm);
                load(B, c, 0, j, k, g, p0);
                load(B, c + 1, 0, j, k, g + 1, pp);
                recon(B, c, pm, p0, pp, qm, qp);
            }
#pragma unroll
            for (int v = 0; v < NRS; ++v) {
                const double t = __shfl_up_sync(full, qp[v], 1);
                qL[v] = lane == 0 ? qp_end[v] : t;
                qp_end[v] = __shfl_sync(full, qp[v], 31);
            }
            const bool has_face = valid && c >= 0 && (w > 0 || lane > 0);
            if (has_face) {
                flux(B, c, pm, p0, qL, qm, F);
            } else {
#pragma unroll
                for (int q = 0; q < NQ; ++q) F[q] = 0.0;
            }
            const bool update = valid && c >= 1 && (w > 0 || lane > 1);   // cell c - 1
            const double Af = face_area<D, OPT>(A, B, update ? c - 1 : 0, j, k);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const double t = __shfl_up_sync(full, F[q], 1);
                const double FW = lane == 0 ? F_end[q] : t;
                F_end[q] = __shfl_sync(full, F[q], 31);
                const double si = __dsub_rn(__dsub_rn(0.0, d_mul(FW, -Af)), d_mul(F[q], Af));
                if (update) A.sweep_part[(long long)q * total + g - 1] = si;
            }
        }
    } else {
        double sig_max = 0.0;
        const int blk = block_of_tile(off, A.sweep_blocks, blockIdx.x);
        const BlockDesc& B = A.blocks[blk];
        const unsigned lt = (unsigned)((long long)blockIdx.x - off[blk]);
        const int n0 = B.n[0], n1 = B.n[1], nD = B.n[D];
        const unsigned lines = (unsigned)n0 * (unsigned)(D == 1 ? B.n[2] : n1);
        const unsigned groups = (lines + SWEEP_LINES - 1) / SWEEP_LINES;
        const unsigned m = lt / groups, l = (lt - m * groups) * SWEEP_LINES + tid;
        if (l < lines) {
            const int q_ = (int)(l / (unsigned)n0), i = (int)(l - (unsigned)q_ * (unsigned)n0);
            const int cells = A.sweep_cells[D];
            const int c0 = (int)m * cells, c1 = min(c0 + cells, nD);   // the cells this tile updates
            const long long sD = D == 1 ? n0 : (long long)n0 * n1;
            const long long g0 = B.offset + (long long)(i + n0 * (D == 1 ? n1 * q_ : q_));   // cell 0 of the line
            const int j0 = D == 1 ? 0 : q_, k0 = D == 1 ? q_ : 0;
            double pm[NPV], p0[NPV], pp[NPV], qp_prev[NRS], F_prev[NQ];
            load(B, c0 - 2, i, j0, k0, g0 + sD * (c0 - 2), pm);
            load(B, c0 - 1, i, j0, k0, g0 + sD * (c0 - 1), p0);
            load(B, c0, i, j0, k0, g0 + sD * c0, pp);
            extern __shared__ __align__(16) unsigned char smem_raw[];
            constexpr int T = SWEEP_LINES;
            double* SP = reinterpret_cast<double*>(smem_raw) + tid;   // [NPV], then [NQ] sums, U, dU0
            double* SS = SP + NPV * T;
            const double* Uin = A.Ubuf[parity];
            for (int c = c0 - 1; c <= c1; ++c) {
                int neg = 0;
                if (c < c1) {   // cell c + 2
                    long long g = g0 + sD * (c + 2);
                    if (c + 2 >= nD) {
                        const int j_ = D == 1 ? c + 2 : q_, k_ = D == 1 ? q_ : c + 2;
                        const GhostCopy s = ghost_copy<MHD>(A, B, i, j_, k_);
                        g = s.g;
                        neg = s.neg;
                        if (g < 0) put_prim<double, NPV>(SP, T, 0, sweep_ghost<MHD>(A, Pin, B, i, j_, k_));
                    }
                    if (g >= 0) {
#pragma unroll
                        for (int v = 0; v < NPV; ++v) cp_async8(SP + v * T, Pin + (long long)v * total + g);
                    }
                }
                if (c > c0) {   // the residual sums of cell c - 1, and what its update reads
                    const long long g = g0 + sD * (c - 1);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        cp_async8(SS + q * T, A.sweep_part + (long long)q * total + g);
                        if (LAST && stage != 0) cp_async8(SS + (NQ + q) * T, Uin + (long long)q * total + g);
                        if (LAST && stage == 2) cp_async8(SS + (2 * NQ + q) * T, A.dU0 + (long long)q * total + g);
                    }
                }
                cp_commit();
                double qm[NRS], qp[NRS], F[NQ];
                recon(B, c, pm, p0, pp, qm, qp);
                if (c >= c0) flux(B, c, pm, p0, qp_prev, qm, F);
                cp_wait<0>();
                if (c > c0) {   // cell c - 1
                    const int jj = D == 1 ? c - 1 : q_, kk = D == 1 ? q_ : c - 1;
                    const double Af = face_area<D, OPT>(A, B, i, jj, kk);
                    const long long g = g0 + sD * (c - 1);
                    double si[NQ];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        si[q] = SS[q * T];
                        si[q] = __dsub_rn(si[q], d_mul(F_prev[q], -Af));
                        si[q] = __dsub_rn(si[q], d_mul(F[q], Af));
                    }
                    if constexpr (LAST) {
                        sweep_finish<MHD, OPT>(A, stage, B, blk, i, jj, kk, g, parity, dt, damp, si, SS + NQ * T,
                                               sig_max);
                    } else {
#pragma unroll
                        for (int q = 0; q < NQ; ++q) A.sweep_part[(long long)q * total + g] = si[q];
                    }
                }
#pragma unroll
                for (int v = 0; v < NPV; ++v) { pm[v] = p0[v]; p0[v] = pp[v]; pp[v] = SP[v * T]; }
                if (neg) pp[1 + D] = -pp[1 + D];   // a mirror negates the normal velocity
#pragma unroll
                for (int v = 0; v < NRS; ++v) qp_prev[v] = qp[v];
#pragma unroll
                for (int q = 0; q < NQ; ++q) F_prev[q] = F[q];
            }
        }
        if (LAST && stage == 2) {
            for (int o = 16; o > 0; o >>= 1) sig_max = fmax(sig_max, __shfl_xor_sync(0xffffffffu, sig_max, o));
            if (lane == 0) s_red[warp] = sig_max;
            __syncthreads();
            if (tid == 0) {
                double v = s_red[0];
                for (int wv = 1; wv < SWEEP_LINES / 32; ++wv) v = fmax(v, s_red[wv]);
                atomicMax(&A.max_signal[blk], (unsigned long long)__double_as_longlong(v));
            }
        }
    }
}

// Primitives of the state U (the stencil loader's decode), for the sweeps.
template <bool MHD>
__global__ void sweep_prims_kernel(const double* __restrict__ U, long long total, NumParams P, double* __restrict__ Pout) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= total) return;
    double u[10];
#pragma unroll
    for (int q = 0; q < (MHD ? 10 : 5); ++q) u[q] = U[q * total + g];
    Prim<double> s;
    decode_prim<false, MHD>(P, u, s);
    store_prim<MHD>(Pout, total, g, s);
}

}  // namespace gdfv
