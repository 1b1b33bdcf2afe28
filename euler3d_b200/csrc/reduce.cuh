// Reductions of a run, each by one block: the density RMS with the stop tests, and the force
// coefficients.  Used by their own kernels (solver.cu) and by the control block of the resident kernel
// (stage_resident.cuh), so every sum has a fixed shape that does not depend on the block's size.
#pragma once
#include <cuda_runtime.h>

#include "forces.cuh"
#include "ordered_sum.cuh"
#include "stage.cuh"

namespace e3d {

constexpr int kReduceThreads = 256;   // lanes of the sum of the RMS partials

// Arguments of the RMS / stop-test kernel of one solver.
struct FinalizeArgs {
    const double *partials;  // per-tile (per-block) sums of R_rho^2
    int n_part;
    double n_domain;         // interior cells
    double *hist;            // RMS history
    Control *ctl;
    const double *rsq;       // FP64_EXACT: R_rho^2 per cell in reference order, summed sequentially
    int n_cells;
};

// Shared memory of the reductions.
union ControlScratch {
    double terms[6][kCoeffThreads];
    double lanes[kReduceThreads];
    OrderedScratch ord;
};

// ------------------------------------------------------------------------------ RMS and stop tests
// Sum of the per-block partials in a fixed order, RMS, and the stop tests of
// EulerSolver::Run (src/solver/EulerSolver.cpp:96-112).  One block of NT threads per solver; the sum is
// that of kReduceThreads lanes whatever NT is.
// partials: the block partials, in global or (resident kernel) shared memory; ctl: the run control, in
// global memory or the block's copy; stage: as for ordered_sum.
template <int NT, bool SHARED = false>
__device__ __forceinline__ void finalize_body(const FinalizeArgs &f, Control *ctl, const double *partials,
                                              ControlScratch &sh, double *stage = nullptr) {
    if (ctl->done) return;
    if (ctl->fault) {  // a stage kernel's bounded wait gave up: its cells kept their old state, so stop
        if (threadIdx.x == 0) {
            ctl->done = 1;
            ctl->stop_reason = E3D_STOP_MAX_ITER;
        }
        return;
    }
    double sum;
    if (f.rsq) {
        sum = ordered_sum<NT>(f.rsq, f.n_cells, sh.ord, stage);
    } else {
        for (int lane = threadIdx.x; lane < kReduceThreads; lane += NT) {
            double v = 0.0;
            for (int i = lane; i < f.n_part; i += kReduceThreads) v += SHARED ? partials[i] : __ldcg(partials + i);
            sh.lanes[lane] = v;
        }
        __syncthreads();
        for (int s = kReduceThreads / 2; s >= 32; s >>= 1) {
            for (int lane = threadIdx.x; lane < s; lane += NT) sh.lanes[lane] += sh.lanes[lane + s];
            __syncthreads();
        }
        sum = threadIdx.x < 32 ? sh.lanes[threadIdx.x] : 0.0;  // the tree's last levels in one warp
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, s);
    }
    if (threadIdx.x != 0) return;
    double rms = sqrt(sum / f.n_domain);
    if (ctl->n_rms < ctl->hist_cap) f.hist[ctl->n_rms] = rms;
    if (ctl->n_rms == 0) ctl->rms0 = rms;
    ctl->n_rms += 1;
    ctl->last_rms = rms;
    ctl->minit_valid = 0;
    ctl->sample_now = 0;
    if (!isfinite(rms)) {  // the reference would spin to MAX_ITER on a NaN; stop and report it
        ctl->nonfinite = 1;
        ctl->done = 1;
        ctl->stop_reason = E3D_STOP_MAX_ITER;
        return;
    }
    if (rms < ctl->min_res || (ctl->min_drop > 0.0 && rms < ctl->min_drop * ctl->rms0)) {
        ctl->done = 1;
        ctl->stop_reason = E3D_STOP_RESIDUAL;
        return;
    }
    if (ctl->stall_window > 0 && (ctl->stall_below <= 0.0 || rms < ctl->stall_below * ctl->rms0)) {
        // the residual has stopped falling (a precision floor)
        if (ctl->best_rms == 0.0 || rms < ctl->best_rms) {
            ctl->best_rms = rms;
            ctl->since_best = 0;
        } else if (++ctl->since_best >= ctl->stall_window) {
            ctl->done = 1;
            ctl->stop_reason = E3D_STOP_STALL;
            return;
        }
    }
    ctl->it += 1;
    const bool sample = ctl->it % ctl->sampling == 0;
    if (sample) ctl->sample_now = 1;
    // with a sample pending that may stop the run on its coefficients, its kernel looks at the count
    if ((!sample || ctl->defer) && ctl->it >= ctl->max_iter) {
        ctl->done = 1;
        ctl->stop_reason = E3D_STOP_MAX_ITER;
    }
}

// ------------------------------------------------------------------------------ force coefficients
// AeroCoefficients::Update (src/solver/AeroCoefficients.cpp:38-52): face terms in parallel; in exact
// mode each of the six sums by one thread in the reference's wall order, so the sums are the
// reference's, otherwise a fixed-shape tree of kCoeffThreads lanes.  One block of NT threads per solver.
template <int NT>
__device__ __forceinline__ void coeff_body(const CoeffArgs &a, Control *ctl, ControlScratch &sh) {
    if (a.run_mode && !forces_due(ctl)) return;
    double (*terms)[kCoeffThreads] = sh.terms;
    if (a.sequential) {
        // the reference's order: one running sum over the wall list, thread k's the k-th
        double acc = 0.0;
        for (int base = 0; base < a.n_wall; base += kCoeffThreads) {
            const int n = min(kCoeffThreads, a.n_wall - base);
            force_terms<NT>(a, base, n, terms);
            __syncthreads();
            if (threadIdx.x < 6)
                for (int j = 0; j < n; j++) acc += terms[threadIdx.x][j];
            __syncthreads();
        }
        if (threadIdx.x < 6) terms[threadIdx.x][0] = acc;
        __syncthreads();
    } else {
        for (int lane = threadIdx.x; lane < kCoeffThreads; lane += NT) {
            double acc[6];
            force_lane(a, lane, acc);
#pragma unroll
            for (int k = 0; k < 6; k++) terms[k][lane] = acc[k];
        }
        __syncthreads();
        for (int st = kCoeffThreads / 2; st > 0; st >>= 1) {
            for (int lane = threadIdx.x; lane < st; lane += NT)
#pragma unroll
                for (int k = 0; k < 6; k++) terms[k][lane] += terms[k][lane + st];
            __syncthreads();
        }
    }
    if (threadIdx.x != 0) return;
    const double F[3] = {terms[0][0], terms[1][0], terms[2][0]}, CP[3] = {terms[3][0], terms[4][0], terms[5][0]};
    force_finish(a, ctl, F, CP);
}

}  // namespace e3d
