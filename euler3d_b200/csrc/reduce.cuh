// Reductions of a run, each by one block: the density RMS with the stop tests, and the force
// coefficients.  Used by their own kernels (solver.cu) and by the control block of the resident kernel
// (stage_resident.cuh), so every sum has a fixed shape that does not depend on the block's size.
#pragma once
#include <cuda_runtime.h>

#include "forces.cuh"
#include "stage.cuh"

namespace e3d {

constexpr int kReduceThreads = 256;   // lanes of the sum of the RMS partials
constexpr int kOrderedThreads = 1024;  // block of FP64_EXACT's RMS kernel

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

// ------------------------------------------------------------------------------ ordered sum
// FP64_EXACT sums R_rho^2 in the reference's cell order, one rounding per cell
// (EulerSolver::computeRMS, src/solver/EulerSolver.cpp:382-389).  The same bits in parallel: while the
// running sum s stays in one binade, with unit u = its last place, adding x >= 0 rounds x to a whole
// number of units whatever s is, except where x lies exactly half-way between two (then the parity of s
// decides).  So between the few special elements -- those at which the sum enters another binade, the
// half-way cases (about one of either per binade) and the first ones -- the sum is a sum of integers, in
// any order; the special elements are added one after another by one thread, each preceded by the
// integers before it.  Where the sum changes binade is predicted from ordinary prefix sums, and the
// prediction is checked against the exact sum at every special element; a failed check (a prefix within
// rounding of a power of two), more special elements than the list holds, or an element that is not a
// finite number >= 0 falls back to the serial loop.
// One thread adding 16,770 numbers from memory took 400 us, which was the exact mode's iteration.
constexpr int kSpecials = 512, kFirstSpecial = 32;

union ControlScratch {
    double terms[6][kCoeffThreads];
    double lanes[kReduceThreads];
    struct {
        double begin[kOrderedThreads + 1];  // ordinary prefix sum before each thread's elements
        double warp_sum[32];
        long long warp_units[32];
        int warp_count[32];
        long long prefix[kSpecials];  // whole units before a special element
        double value[kSpecials];
        int expo[kSpecials];          // binade of the sum before it
        long long units;              // whole units of all elements
        double sum;
        int fail;
    } ord;
};

__device__ __forceinline__ int biased_exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ double pow2_biased(int e) { return __hiloint2double(e << 20, 0); }

// Exclusive scan over the block of each thread's v; total: the sum.
template <int NT, typename V>
__device__ __forceinline__ V block_scan(V v, V *warp_tot, V &total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    V inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const V y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    V off = 0, all = 0;
    for (int w = 0; w < NT / 32; w++) {
        if (w == wid) off = all;
        all += warp_tot[w];
    }
    total = all;
    const V prev = __shfl_up_sync(0xffffffffu, inc, 1);
    return lane ? off + prev : off;
}

// s = 0; for i in 0..n-1: s += x[i], every addition rounded; returned to thread 0.  x is global memory
// on a 32-byte boundary, or, with stage, copied there first (shared memory for n doubles): each thread's
// elements are contiguous, a whole sector at a time.
template <int NT>
__device__ double ordered_sum(const double *x, int n, ControlScratch &scratch, double *stage) {
    auto &sh = scratch.ord;
    const int tid = threadIdx.x, per = stage ? (n + NT - 1) / NT | 1 : ((n + NT - 1) / NT + 3) & ~3;
    const int i0 = min(tid * per, n), i1 = min(i0 + per, n);
    if (stage) {  // an odd stride per thread: no bank conflicts
        constexpr int U = 8;
        for (int i = tid; i < n; i += U * NT) {
            double v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = i + u * NT < n ? __ldcg(x + i + u * NT) : 0.0;
#pragma unroll
            for (int u = 0; u < U; u++)
                if (i + u * NT < n) stage[i + u * NT] = v[u];
        }
        __syncthreads();
    }
    // this thread's elements in order
    auto each = [&](auto &&f) {
        if (stage) {
            for (int i = i0; i < i1; i++) f(i, stage[i]);
        } else {
            for (int i = i0; i < i1; i += 4) {
                const int m = min(4, i1 - i);
                double v[4] = {0.0, 0.0, 0.0, 0.0};
                if (m == 4) {
                    const double2 lo = __ldcg(reinterpret_cast<const double2 *>(x + i));
                    const double2 hi = __ldcg(reinterpret_cast<const double2 *>(x + i) + 1);
                    v[0] = lo.x, v[1] = lo.y, v[2] = hi.x, v[3] = hi.y;
                } else {
                    for (int k = 0; k < m; k++) v[k] = __ldcg(x + i + k);
                }
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < m) f(i + k, v[k]);
            }
        }
    };
    double p = 0.0;
    bool bad = false;
    each([&](int, double v) {
        bad |= !(v >= 0.0 && v < 1e300);
        p += v;
    });
    double all;
    const double before = block_scan<NT>(p, sh.warp_sum, all);
    sh.begin[tid] = before;
    if (tid == NT - 1) sh.begin[NT] = all;
    if (__syncthreads_or(bad || !(all < 1e300))) {
        double s = 0.0;
        if (tid == 0)
            for (int i = 0; i < n; i++) s += __ldcg(x + i);
        return s;
    }
    // walk over this thread's elements: whole units summed, `special(v, units so far, binade)` called
    auto walk = [&](auto &&special) {
        double q = before, part = 0.0;  // part: whole units since the last special element, below 2^53
        long long units = 0;
        each([&](int i, double v) {
            if (v == 0.0) return;
            const int e = biased_exponent(q);
            const double next = q + v;
            bool sp = i < kFirstSpecial || q < 1e-280 || biased_exponent(next) != e;
            if (!sp) {
                // in units of 2^(e - 1075), rounded to a whole number by adding and taking off 2^52
                const double t = v * pow2_biased(2098 - e), r = (t + 0x1p52) - 0x1p52;
                if (fabs(t - r) == 0.5 || t >= 0x1p52) sp = true;
                else part += r;
            }
            if (sp) {
                units += (long long)part;
                part = 0.0;
                special(v, units, e);
            }
            q = next;
        });
        units += (long long)part;
        // the next thread starts from its own prefix: the same binade, or the check below gives up
        if (i0 < i1 && biased_exponent(q) != biased_exponent(sh.begin[tid + 1])) bad = true;
        return units;
    };
    int count = 0;
    const long long units = walk([&](double, long long, int) { count++; });
    int n_special;
    const int slot = block_scan<NT>(count, sh.warp_count, n_special);
    long long all_units;
    const long long units_before = block_scan<NT>(units, sh.warp_units, all_units);
    if (tid == 0) sh.fail = 0;
    bad = __syncthreads_or(bad) || n_special > kSpecials;
    if (!bad && count) {
        int k = slot;
        walk([&](double v, long long u, int e) {
            sh.prefix[k] = units_before + u;
            sh.value[k] = v;
            sh.expo[k++] = e;
        });
    }
    __syncthreads();
    double s = 0.0;
    if (tid == 0) {
        long long done = 0;
        // adds whole units to s, which must be in binade e before and after
        auto add_units = [&](long long u, int e) {
            if (!u) return;
            if (e < 60 || biased_exponent(s) != e) {
                bad = true;
                return;
            }
            const long long m = (long long)(s * pow2_biased(2098 - e)) + u;
            if (m >= 1ll << 53) bad = true;
            else s = (double)m * pow2_biased(e - 52);
        };
        for (int k = 0; k < n_special && !bad; k++) {
            add_units(sh.prefix[k] - done, sh.expo[k]);
            s += sh.value[k];
            done = sh.prefix[k];
        }
        if (!bad) add_units(all_units - done, biased_exponent(sh.begin[NT]));
        if (bad) {
            s = 0.0;
            for (int i = 0; i < n; i++) s += __ldcg(x + i);
        }
    }
    return s;
}

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
        sum = ordered_sum<NT>(f.rsq, f.n_cells, sh, stage);
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
