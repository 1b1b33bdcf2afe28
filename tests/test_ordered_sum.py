"""FP64_EXACT's sum over the cells (euler3d_b200/csrc/ordered_sum.cuh), compiled for the CPU: the block's
threads run as fibres that meet at every barrier and shuffle.

The sum promises the bits of the plain running sum for every input.  Inputs: ordinary ones, and running
sums that stop a few units short of a power of two, which the block's prefix sums, rounded in another
order, may have passed: elements behind it that are more than half a unit of the lower binade and less
than half a unit of the upper one then decide whether the prediction was checked."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = r"""
#include <cuda_runtime.h>
#include <ucontext.h>
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>
using std::min;
struct Index { int x; } static threadIdx;
static ucontext_t scheduler, fibre[1024];
static int n_threads, finished;
static double slot[1024];
static void meet() { const int me = threadIdx.x; swapcontext(&fibre[me], &scheduler); }
static void __syncthreads() { meet(); }
static int __syncthreads_or(int p) {
    slot[threadIdx.x] = p != 0;
    meet();
    int any = 0;
    for (int t = 0; t < n_threads; t++) any |= slot[t] != 0.0;
    meet();
    return any;
}
template <typename V> static V __shfl_up_sync(unsigned, V v, int o) {
    static_assert(sizeof(V) <= 8, "");
    const int t = threadIdx.x;
    std::memcpy(&slot[t], &v, sizeof v);
    meet();
    V r = v;
    if ((t & 31) >= o) std::memcpy(&r, &slot[t - o], sizeof r);
    meet();
    return r;
}
static int __double2hiint(double x) { uint64_t b; std::memcpy(&b, &x, 8); return (int)(b >> 32); }
static double __hiloint2double(int hi, int lo) {
    const uint64_t b = (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}
template <typename V> static V __ldcg(const V *p) { return *p; }
#include "ordered_sum.cuh"

static e3d::OrderedScratch scratch;
static std::vector<double> room;
static const double *input;
static int count;
static double *stage, result;
template <int NT> static void body() {
    const double s = e3d::ordered_sum<NT>(input, count, scratch, stage);
    if (threadIdx.x == 0) result = s;
    finished++;
}
template <int NT> static double run(const double *x, int n, bool staged) {
    static std::vector<char> stacks((size_t)NT * 16384);
    input = x, count = n, n_threads = NT, finished = 0;
    room.assign(n, -1.0);
    stage = staged ? room.data() : nullptr;
    for (int t = 0; t < NT; t++) {
        getcontext(&fibre[t]);
        fibre[t].uc_stack.ss_sp = &stacks[(size_t)t * 16384];
        fibre[t].uc_stack.ss_size = 16384;
        fibre[t].uc_link = &scheduler;
        makecontext(&fibre[t], body<NT>, 0);
    }
    while (finished < NT)
        for (int t = 0; t < NT; t++) {
            threadIdx.x = t;
            swapcontext(&scheduler, &fibre[t]);
        }
    return result;
}
extern "C" double ordered_sum(const double *x, int n, int threads, int staged) {
    return threads == 1024 ? run<1024>(x, n, staged) : threads == 512 ? run<512>(x, n, staged) : run<128>(x, n, staged);
}
extern "C" double running_sum(const double *x, int n) {
    double s = 0.0;
    for (int i = 0; i < n; i++) s += x[i];
    return s;
}
"""


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    from euler3d_b200 import build

    d = tmp_path_factory.mktemp("ordered")
    (d / "sum.cpp").write_text(SOURCE)
    csrc = os.path.join(os.path.dirname(HERE), "euler3d_b200", "csrc")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", f"-I{csrc}", f"-I{cuda}",
                    "-o", str(d / "sum.so"), str(d / "sum.cpp")], check=True)
    lib = C.CDLL(str(d / "sum.so"))
    lib.ordered_sum.restype = lib.running_sum.restype = C.c_double

    def call(x, threads, staged):
        buf = np.empty(x.size + 4)  # the kernel's vector loads want 32-byte boundaries
        at = buf[(-buf.ctypes.data // 8) % 4:][: x.size]
        at[:] = x
        p = at.ctypes.data_as(C.c_void_p)
        return lib.ordered_sum(p, x.size, threads, int(staged)), lib.running_sum(p, x.size)

    return call


def short_of_power_of_two(seed, lead=3000, tail=5, power=11):
    """`lead` random numbers whose running sum ends a few units below 2^power, then `tail` elements of
    0.55 to 0.95 of the lower binade's unit."""
    rng = np.random.default_rng(seed)
    top, unit = 2.0 ** power, 2.0 ** (power - 53)
    x = rng.uniform(0.1, 1.0, lead)
    x *= (top - 1.0) / x.sum()
    for _ in range(8):  # the last element takes up what is missing
        s = np.add.accumulate(x)[-1]
        x[-1] += (top - rng.integers(1, 31) * unit) - s
        if top - 31 * unit < np.add.accumulate(x)[-1] < top:
            break
    return np.concatenate([x, rng.uniform(0.55, 0.95, tail) * unit])


@pytest.mark.parametrize("threads,staged", [(1024, False), (512, True)])
def test_prediction_past_a_power_of_two(sums, threads, staged):
    for seed in range(60):
        got, want = sums(short_of_power_of_two(seed), threads, staged)
        assert got == want, seed


@pytest.mark.parametrize("threads,staged", [(1024, False), (512, True), (128, False), (128, True)])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 1500, 4099])
def test_is_the_running_sum(sums, n, threads, staged):
    rng = np.random.default_rng(n)
    for x in (rng.uniform(0, 1, n), 10.0 ** rng.uniform(-40, 3, n), np.where(rng.uniform(size=n) < 0.3, 0.0, 0.1),
              np.full(n, 2.0 ** -30), 2.0 ** rng.integers(-60, 4, n).astype(float), np.zeros(n),
              10.0 ** rng.uniform(-320, -290, n)):
        got, want = sums(x, threads, staged)
        assert got == want
