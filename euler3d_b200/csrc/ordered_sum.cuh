// Sum of numbers one after another, every addition rounded, by one block.
#pragma once
#include <cuda_runtime.h>

namespace e3d {

constexpr int kOrderedThreads = 1024;  // block of FP64_EXACT's RMS kernel

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

struct OrderedScratch {
    double begin[kOrderedThreads + 1];  // ordinary prefix sum before each thread's elements
    double warp_sum[32];
    long long warp_units[32];
    int warp_count[32];
    long long prefix[kSpecials];  // whole units before a special element
    double value[kSpecials];
    int expo[kSpecials];          // binade of the sum before it
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
__device__ double ordered_sum(const double *x, int n, OrderedScratch &sh, double *stage) {
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
        // adds whole units to s, which must be in binade e before and after: also where there are none,
        // since they were counted in that binade's unit (elements below half of it are none, but may be
        // one of the binade below).  Elements before e = 60 are all special.
        auto add_units = [&](long long u, int e) {
            if (e < 60 ? u != 0 : biased_exponent(s) != e) {
                bad = true;
                return;
            }
            if (!u) return;
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

}  // namespace e3d
