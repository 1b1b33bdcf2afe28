// Run control, and the force coefficients of the wall faces.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "euler3d_b200.h"

namespace e3d {

// Run control shared by the kernels of e3d_solver_run; lives in device memory.
struct Control {
    int done;          // nonzero: every later kernel returns at once
    int stop_reason;   // E3D_STOP_*
    int it;            // EulerSolver::_nbInteration
    int n_rms;         // iterations whose RMS has been computed
    int counter;       // consecutive stagnated coefficient samples (src/solver/EulerSolver.cpp:142-147)
    int sample_now;    // this iteration's force coefficients are to be sampled (cleared when they are)
    int defer;         // they cannot stop the run: the next iteration's first stage integrates them
    int minit_valid;   // interior Mach of the loaded state still holds (no stage has run since)
    int nonfinite;     // the RMS became NaN/Inf
    int max_iter, sampling, hist_cap;
    int fault;         // a bounded wait in a kernel gave up
    double min_res, min_aero, last_rms, cl, cd, cm;
    double min_drop;   // > 0: also stop once the RMS is below min_drop x the run's first RMS
    double rms0;       // RMS of the run's first iteration
    int n_samples;     // coefficient samples taken (residuals.dat rows)
    int sample_cap;    // capacity of the sample record
    int stall_window;  // > 0: stop once the RMS has set no new minimum for this many iterations
    int since_best;    // iterations since the RMS last set a new minimum
    double best_rms;   // smallest RMS of the run so far
    double stall_below;  // the stall test counts only once RMS < stall_below x the first RMS (0: always)
    double force[3], moment[3];
};

constexpr int kCoeffThreads = 512;    // lanes of the force sums

struct CoeffArgs {
    int n_wall;
    const int *__restrict__ cell;       // device cell of each wall face, reference wall order
    const double *__restrict__ svec;    // 3 per wall face: full face normal
    const double *__restrict__ center;  // 3 per wall face: face centre
    const double2 *__restrict__ q;
    const double *__restrict__ w0;      // FP32_FLUX mode: pressure from the double conservative state
    int w0_stride;
    double gamma;
    double p_inf, cp_factor, cref, sref, ref[3];
    int axis[3], sign[3];
    Control *ctl;
    int run_mode;                       // 1: sampled inside e3d_solver_run, apply the stop test
    int sequential;                     // 1: sum in the reference's wall order (FP64_EXACT)
    double *__restrict__ out;           // 6 doubles (force, moment) when not in run mode
    double *__restrict__ cp_out;        // [n_wall] Cp of every wall face (AeroCoefficients::_cp), or null
    double *terms;                      // [6][n_wall] terms of the force blocks, and how many blocks have
    unsigned *arrivals;                 // written theirs (zero between uses)
    double *__restrict__ samples;       // run mode: 7 doubles (iteration, force, moment) per sample, or null
};

__device__ __forceinline__ double wall_pressure(const CoeffArgs &a, int c) {
    if (!a.w0) return __ldcg(&a.q[3 * c + 2].x);
    const size_t st = (size_t)a.w0_stride;
    const double rho = __ldcg(a.w0 + c), mu = __ldcg(a.w0 + st + c), mv = __ldcg(a.w0 + 2 * st + c);
    const double mw = __ldcg(a.w0 + 3 * st + c);
    return (a.gamma - 1.0) * (__ldcg(a.w0 + 4 * st + c) - 0.5 * (mu * mu + mv * mv + mw * mw) / rho);
}

// Lane `lane` of the force sums: wall faces lane, lane + T, lane + 2T, ... (T = kCoeffThreads) in that
// order, their loads issued four faces at a time.
__device__ __forceinline__ void force_lane(const CoeffArgs &a, int lane, double acc[6]) {
    constexpr int U = 4;
#pragma unroll
    for (int k = 0; k < 6; k++) acc[k] = 0.0;
    for (int base = lane; base < a.n_wall; base += U * kCoeffThreads) {
        double p[U], sv[U][3], ce[U][3];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = base + u * kCoeffThreads;
            if (i < a.n_wall) {
                p[u] = wall_pressure(a, a.cell[i]);
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    sv[u][k] = a.svec[3 * i + k];
                    ce[u][k] = a.center[3 * i + k];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (base + u * kCoeffThreads >= a.n_wall) break;
            const double cp = a.cp_factor * (p[u] - a.p_inf);
            if (a.cp_out) a.cp_out[base + u * kCoeffThreads] = cp;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double coeff = sv[u][k] * cp * a.cref / a.sref;
                acc[k] += coeff;
                acc[3 + k] += coeff * ce[u][k];
            }
        }
    }
}

// Force terms of wall faces base .. base + n - 1 (threads tid, tid + NT, ...) into terms[6][.].
template <int NT>
__device__ __forceinline__ void force_terms(const CoeffArgs &a, int base, int n, double (*terms)[kCoeffThreads]) {
    for (int j = threadIdx.x; j < n; j += NT) {
        const int i = base + j;
        double p = wall_pressure(a, a.cell[i]);
        double cp = a.cp_factor * (p - a.p_inf);
        if (a.cp_out) a.cp_out[i] = cp;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            double coeff = a.svec[3 * i + k] * cp * a.cref / a.sref;
            terms[k][j] = coeff;
            terms[3 + k][j] = coeff * a.center[3 * i + k];
        }
    }
}

// One thread: force and moment from the summed terms, then (run mode) EulerSolver::ConvergenceCriteria
// and the CL/CD/CM selection (src/solver/EulerSolver.cpp:132-152, :253-279).
__device__ __forceinline__ void force_finish(const CoeffArgs &a, Control *ctl, const double F[3], const double CP[3]) {
    const double lever[3] = {a.ref[0] - CP[0], a.ref[1] - CP[1], a.ref[2] - CP[2]};
    const double M[3] = {(F[1] * lever[2] - F[2] * lever[1]) / a.cref, (F[2] * lever[0] - F[0] * lever[2]) / a.cref,
                   (F[0] * lever[1] - F[1] * lever[0]) / a.cref};
    if (!a.run_mode) {
        for (int k = 0; k < 3; k++) {
            a.out[k] = F[k];
            a.out[3 + k] = M[k];
        }
        return;
    }
    double cl = F[a.axis[0]] * a.sign[0], cd = F[a.axis[1]] * a.sign[1], cm = M[a.axis[2]] * a.sign[2];
    double tol = ctl->min_aero;
    bool ok = fabs(ctl->cl - cl) < tol && fabs(ctl->cd - cd) < tol && fabs(ctl->cm - cm) < tol;
    ctl->counter = ok ? ctl->counter + 1 : 0;
    if (a.samples && ctl->n_samples < ctl->sample_cap) {  // a residuals.dat row (EulerSolver::PrintInfo)
        double *s = a.samples + 7 * (size_t)ctl->n_samples;
        s[0] = ctl->it;
        for (int k = 0; k < 3; k++) {
            s[1 + k] = F[k];
            s[4 + k] = M[k];
        }
    }
    ctl->n_samples += 1;
    ctl->cl = cl;
    ctl->cd = cd;
    ctl->cm = cm;
    for (int k = 0; k < 3; k++) {
        ctl->force[k] = F[k];
        ctl->moment[k] = M[k];
    }
    if (ctl->counter >= 2) {
        ctl->done = 1;
        ctl->stop_reason = E3D_STOP_COEFFICIENTS;
    } else if (ctl->it >= ctl->max_iter) {
        ctl->done = 1;
        ctl->stop_reason = E3D_STOP_MAX_ITER;
    }
    ctl->sample_now = 0;
}

// Are force coefficients due?  Deferred ones also when the run has stopped on its iteration count.
__device__ __forceinline__ bool forces_due(const Control *ctl) { return ctl->sample_now && (ctl->defer || !ctl->done); }

// Deferred forces: `parts` blocks of kForceThreads threads at the front of an iteration's first stage
// integrate the forces of the state that the stage reads, while its other blocks work (a kernel of its
// own between the iterations took 5 to 30 us).  Every thread forms the six terms of a few faces; the
// block that arrives last adds them in coeff_body's order: its lanes and tree, or in exact mode the
// reference's sequential sums.
constexpr int kForceThreads = 128, kMaxForceBlocks = 64, kBatchForceBlocks = 4;
constexpr size_t kForceSmem = sizeof(double) * 6 * kCoeffThreads;

static __device__ __noinline__ void force_block(const CoeffArgs &a, int part, int parts, unsigned char *smem) {
    Control *ctl = a.ctl;
    if (!forces_due(ctl) || !ctl->defer) return;  // uniform: cleared when every block has arrived
    double (*sums)[kCoeffThreads] = reinterpret_cast<double (*)[kCoeffThreads]>(smem);
    __shared__ unsigned order;
    const int tid = threadIdx.x, n = a.n_wall;
    for (int i = part * kForceThreads + tid; i < n; i += parts * kForceThreads) {
        const double cp = a.cp_factor * (wall_pressure(a, a.cell[i]) - a.p_inf);
        if (a.cp_out) a.cp_out[i] = cp;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double coeff = a.svec[3 * i + k] * cp * a.cref / a.sref;
            __stcg(a.terms + (size_t)k * n + i, coeff);
            __stcg(a.terms + (size_t)(3 + k) * n + i, coeff * a.center[3 * i + k]);
        }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) order = atomicAdd(a.arrivals, 1u);
    __syncthreads();
    if (order != (unsigned)parts - 1) return;
    __threadfence();
    if (a.sequential) {
        double acc = 0.0;
        for (int base = 0; base < n; base += kCoeffThreads) {
            const int m = min(kCoeffThreads, n - base);
            for (int j = tid; j < 6 * kCoeffThreads; j += kForceThreads) {
                const int k = j / kCoeffThreads, i = j % kCoeffThreads;
                if (i < m) sums[k][i] = __ldcg(a.terms + (size_t)k * n + base + i);
            }
            __syncthreads();
            if (tid < 6)
                for (int i = 0; i < m; i++) acc += sums[tid][i];
            __syncthreads();
        }
        if (tid < 6) sums[tid][0] = acc;
        __syncthreads();
    } else {
        for (int lane = tid; lane < kCoeffThreads; lane += kForceThreads) {
            double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
            for (int i = lane; i < n; i += kCoeffThreads)
#pragma unroll
                for (int k = 0; k < 6; k++) acc[k] += __ldcg(a.terms + (size_t)k * n + i);
#pragma unroll
            for (int k = 0; k < 6; k++) sums[k][lane] = acc[k];
        }
        __syncthreads();
        for (int st = kCoeffThreads / 2; st > 0; st >>= 1) {
            for (int l = tid; l < st; l += kForceThreads)
#pragma unroll
                for (int k = 0; k < 6; k++) sums[k][l] += sums[k][l + st];
            __syncthreads();
        }
    }
    if (tid) return;
    *a.arrivals = 0u;
    const double F[3] = {sums[0][0], sums[1][0], sums[2][0]}, CP[3] = {sums[3][0], sums[4][0], sums[5][0]};
    force_finish(a, ctl, F, CP);
}

}  // namespace e3d
