// Resident kernel: whole iterations of a run in one launch, for meshes whose face tiles all fit on the
// GPU at once.
//
// A stage of a small mesh takes the stage kernels about 10 us whatever its size: launch, the chain of
// loads behind the tile's copies, then the arithmetic of a few faces per thread.  Here every tile has a
// block of its own for the whole run.  Its face records, contribution lists, geometry and cell states
// stay in shared memory and W0 in registers; a stage reads only the halo, and tiles wait for each other
// instead of for the kernel boundary:
//   - Cells with a neighbour in another tile are published after every stage, in 16-byte words of three
//     data words and a tag, the number of the state's version.  A word is written and read whole
//     (st / ld .b128), so the data is there when the tag is: one trip through L2, no fence and no flag.
//     Version v sits in slot v & 1.  Tiles that share a face read each other, so when a tile overwrites
//     version v - 1 with v + 1 it has seen every reader's version v and those reads are done.  Tags go on
//     counting from launch to launch, so a slot never holds an old word with a new tag.
//   - One more block, the control block, waits for every tile's RMS partial of an iteration (a tagged
//     word too; in exact mode for the flags below), applies the stop tests, posts the number of
//     iterations decided (with a stop bit), then integrates the wall forces and posts that too.  For
//     them it reads the state that the tiles wrote to the state buffer at the end of the iteration, once
//     their flags (released after those writes) say so.
//   - The tiles do not wait for the decision: they go on with the next iteration and look at it before
//     that iteration's last stage, the first one whose results leave the block (final states, W0, ghost
//     records, the RMS partial).  Until then the farfield ghosts, which carry state from stage to stage,
//     live in shared memory.  A stop leaves everything as the decided iteration left it.
// The arithmetic is that of the stage kernels (the same functions), so states, RMS history and
// coefficients have the same bits.
//
// What bounds it is the chain of a stage in one tile, 3.55 us on a channel of 4,096 FP64 cells: 1.2 us
// for the halo (0.6 its words' trip through L2, the rest waiting for slower neighbours; 1.7 before an
// iteration's last stage, with the decision and the forces), 0.9 us for the fluxes and 1.2 us for the
// update (FP64 latency and instruction issue of the few warps of one tile; the issue slots are 21 % used).
// Measured on B200, us per RK5 iteration with force
// sampling every iteration, CUDA graphs of stage kernels against this kernel:
//   channel 4,096 cells FP64          55.8   17.1      O-grid 20,200 cells, AUSM, FP64      50.5   21.2
//   channel 37,442 cells FP32_FLUX    52.2   20.5      channel 16,770 cells FP64_EXACT       506   42.7
// (the last with the sequential RMS sum of ordered_sum, which the graphs' RMS kernel uses now too)
//
// The launch is cooperative (all blocks resident), every wait is bounded, and a wait that gives up
// raises the run's fault word and an abort word that the other waits watch.
#pragma once
#include <stddef.h>

#include <algorithm>

#include "common.hpp"
#include "reduce.cuh"
#include "stage.cuh"
#include "stage_f32.cuh"

namespace e3d {

constexpr int kFlagStride = 8;          // words between two tiles' flags: a 32-byte sector each
constexpr int kResidentIterations = 256;  // per launch, unless the caller asks for more frequent checks
constexpr unsigned kStopBit = 1u << 31;

// flags[t]: iterations whose final state tile t has written.  After the tile flags: abort, iterations
// decided (| kStopBit), iterations whose forces are done.
enum : int { WORD_ABORT = 0, WORD_DECIDED = 1, WORD_FORCES = 2, kControlWords = 3 };

struct ResidentArgs {
    unsigned *flags;       // [n_tiles * kFlagStride] then the control words, kFlagStride apart
    double2 *q[2];         // state buffers (FP64 modes)
    float4 *q32[2];        // state buffers (FP32_FLUX)
    uint4 *words;          // [2][n_tiles * kTileCells][words per cell] published cells
    uint4 *partials;       // [n_tiles] RMS partials: value, -, tag
    unsigned tag;          // of version 0
    int iterations;        // at most this many in this launch
    int max_far;           // farfield ghosts of a tile, at most
    int stage_rsq;         // exact mode: R_rho^2 of every cell fits the control block's shared memory
    int stages;            // per iteration: 5 (RK5) or 1 (explicit Euler)
    FinalizeArgs fin;
    CoeffArgs coeff[2];    // for the state in buffer 0 / 1
};

struct LoopStep {
    const StageArgs &a;
    double *far;     // farfield ghost records of the tile, in shared memory
    int first_far;   // the tile's first boundary face
    double al;
    bool first, last, minit;
    double2 *qo;
    float4 *q32o;
    __device__ __forceinline__ double alpha() const { return al; }
    __device__ __forceinline__ bool first_stage() const { return first; }
    __device__ __forceinline__ bool last_stage() const { return last; }
    __device__ __forceinline__ bool ghost_store() const { return last; }
    __device__ __forceinline__ bool minit_valid() const { return minit; }
    __device__ __forceinline__ double *ghost(int j, int slot, int tag) const {
        return tag >= TAG_FAR ? far + 8 * (j - first_far) : a.ghost + 8 * (size_t)slot;
    }
    __device__ __forceinline__ bool stores_state() const { return last; }
    __device__ __forceinline__ double2 *qout() const { return qo; }
    __device__ __forceinline__ float4 *q32out() const { return q32o; }
};

__device__ __forceinline__ unsigned load_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// A 16-byte word in one access.
__device__ __forceinline__ uint4 load_word(const uint4 *p) {
    unsigned __int128 v;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(v) : "l"(p) : "memory");
    const unsigned long long lo = (unsigned long long)v, hi = (unsigned long long)(v >> 64);
    return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}

__device__ __forceinline__ void store_word(uint4 *p, uint4 w) {
    const unsigned long long lo = (unsigned long long)w.y << 32 | w.x, hi = (unsigned long long)w.w << 32 | w.z;
    const unsigned __int128 v = (unsigned __int128)hi << 64 | lo;
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(v) : "memory");
}

__device__ __forceinline__ void store_release(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait (one look, then `polls` more of about 0.5 us, StageArgs::wait_polls) until the word (without
// its stop bit) reaches v; false when it gives up or the run was aborted.  got: the word seen.  The limit
// is not looked at before the first look, which mostly succeeds: a channel of 4,096 cells takes 3.67 ms for
// 200 iterations with the check in front and 3.55 ms with it behind.
__device__ __forceinline__ bool wait_word(const unsigned *word, unsigned v, const unsigned *abort, int polls,
                                          unsigned &got) {
    for (int n = 0;; n++) {
        got = load_acquire(word);
        if ((got & ~kStopBit) >= v) return true;
        if (n >= polls || ((n & 31) == 31 && load_acquire(abort))) return false;
    }
}

// Bounded wait until all K words at p carry the tag.
template <int K>
__device__ __forceinline__ bool wait_words(const uint4 *p, unsigned tag, const unsigned *abort, int polls, uint4 w[K]) {
    for (int n = 0;; n++) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < K; k++) w[k] = load_word(p + k);
#pragma unroll
        for (int k = 0; k < K; k++) all &= w[k].w == tag;
        if (all) return true;
        if (n >= polls || ((n & 31) == 31 && load_acquire(abort))) return false;
    }
}

// Bytes of a cell record and of a face record (and of a face's fluxes); published words per cell.
template <int PREC>
struct ResidentLayout {
    static constexpr uint32_t kState = PREC == PREC_F32 ? 32 : 48, kRec = PREC == PREC_F32 ? 24 : 40;
    static constexpr int kWords = PREC == PREC_F32 ? 3 : 4;
};

// Dynamic shared memory of a tile's block: cell records, face records, fluxes, contribution lists,
// farfield ghosts (a tile's farfield and unclassified faces come first of its boundary faces), an
// mbarrier.  The control block uses the same space: its scratch, its copy of the run control, and the
// tiles' RMS partials (or, in exact mode, R_rho^2 of every cell where that fits).
constexpr size_t kControlHead = ((sizeof(ControlScratch) + 15) & ~(size_t)15) + ((sizeof(Control) + 15) & ~(size_t)15);

inline size_t resident_smem_bytes(int prec, int LC, int FC, int MC, int max_far, int n_tiles) {
    const size_t st = prec == PREC_F32 ? 32 : 48, rec = ((prec == PREC_F32 ? 24 : 40) * (size_t)FC + 15) & ~(size_t)15;
    const size_t tile = (size_t)LC * st + 2 * rec + (size_t)MC * kTileCells * 2 + 64 * (size_t)max_far;
    return std::max(tile + 16, kControlHead + 8 * (size_t)n_tiles);
}

// The control block (see above): RMS, stop tests and forces of every iteration.
// Not inlined: it would take registers from the tiles' code.
template <int NT>
__device__ __noinline__ void resident_control(const StageArgs &a, const ResidentArgs &r, unsigned char *smem) {
    const int tid = threadIdx.x;
    ControlScratch &sh = *reinterpret_cast<ControlScratch *>(smem);
    Control *ctl = reinterpret_cast<Control *>(smem + ((sizeof(ControlScratch) + 15) & ~(size_t)15));
    double *room = reinterpret_cast<double *>(smem + kControlHead);
    // the run control stays here for the launch; every word but the fault word, which any block sets, is
    // written back on every exit
    constexpr int kWords = (int)(sizeof(Control) / 4), kFault = (int)(offsetof(Control, fault) / 4);
    for (int i = tid; i < kWords; i += NT) reinterpret_cast<int *>(ctl)[i] = reinterpret_cast<const int *>(a.ctl)[i];
    __syncthreads();
    auto write_back = [&] {
        __syncthreads();
        for (int i = tid; i < kWords; i += NT)
            if (i != kFault) reinterpret_cast<int *>(a.ctl)[i] = reinterpret_cast<const int *>(ctl)[i];
    };
    unsigned *words = r.flags + (size_t)a.n_tiles * kFlagStride;
    const unsigned *abort = words + WORD_ABORT * kFlagStride;
    int buf = 0;  // buffer of the iteration's final state
    for (int it = 1; it <= r.iterations; it++) {
        buf ^= r.stages & 1;
        // every tile's final state of the iteration is in the state buffer
        auto states_written = [&] {
            unsigned got;
            bool ok = true;
            for (int t = tid; t < a.n_tiles && ok; t += NT)
                ok = wait_word(r.flags + (size_t)t * kFlagStride, (unsigned)it, abort, a.wait_polls, got);
            return ok;
        };
        bool ok = true;
        if (r.fin.rsq) {
            ok = states_written();
        } else {
            for (int t = tid; t < a.n_tiles && ok; t += NT) {
                uint4 w[1];
                ok = wait_words<1>(r.partials + t, r.tag + (unsigned)(it * r.stages), abort, a.wait_polls, w);
                room[t] = __hiloint2double((int)w[0].y, (int)w[0].x);
            }
        }
        auto gave_up = [&] {  // a wait, here or in a tile: the run stops
            if (!__syncthreads_or(!ok)) return false;
            if (tid == 0) {
                atomicExch(a.fault, 1);
                atomicExch(words + WORD_ABORT * kFlagStride, 1u);
                ctl->done = 1;
                ctl->stop_reason = E3D_STOP_MAX_ITER;
            }
            return true;
        };
        if (gave_up()) break;
        finalize_body<NT, true>(r.fin, ctl, room, sh, r.stage_rsq ? room : nullptr);
        __syncthreads();  // thread 0's stop tests are written, the scratch is free
        // the forces first when they can stop the run; otherwise only the iteration count can
        const bool sample = !ctl->done && ctl->sample_now, forces_decide = sample && ctl->min_aero > 0.0;
        bool stop = ctl->done || (sample && !forces_decide && ctl->it >= ctl->max_iter);
        if (tid == 0 && !forces_decide)
            store_release(words + WORD_DECIDED * kFlagStride, (unsigned)it | (stop ? kStopBit : 0u));
        if (sample) {
            ok = states_written();
            if (gave_up()) break;
            coeff_body<NT>(r.coeff[buf], ctl, sh);
        }
        __syncthreads();
        stop = ctl->done;
        if (tid == 0) {
            if (forces_decide) store_release(words + WORD_DECIDED * kFlagStride, (unsigned)it | (stop ? kStopBit : 0u));
            store_release(words + WORD_FORCES * kFlagStride, (unsigned)it);
        }
        __syncthreads();
        if (stop) break;
    }
    write_back();
}

template <int PREC, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) resident_kernel(const __grid_constant__ StageArgs a,
                                                            const __grid_constant__ ResidentArgs r) {
    constexpr bool F32 = PREC == PREC_F32, EXACT = PREC == PREC_EXACT;
    constexpr uint32_t kState = ResidentLayout<PREC>::kState, kRec = ResidentLayout<PREC>::kRec;
    constexpr int kWords = ResidentLayout<PREC>::kWords;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_word;
    if (a.ctl->done) return;  // the run stopped in an earlier launch
    if ((int)blockIdx.x == a.n_tiles) {
        resident_control<NT>(a, r, smem_raw);
        return;
    }
    const int tile = blockIdx.x, tid = threadIdx.x, T = kTileCells, MC = a.max_contrib;
    const int c0 = tile * T, nloc = min(T, a.n_cells - c0);
    const int nf = a.tile_face_ptr[tile + 1] - a.tile_face_ptr[tile];
    unsigned *words = r.flags + (size_t)a.n_tiles * kFlagStride;
    const unsigned *abort = words + WORD_ABORT * kFlagStride;
    bool minit = a.ctl->minit_valid;

    // shared memory
    unsigned char *st_p = smem_raw, *rec_p = st_p + (size_t)a.smem_cells * kState;
    unsigned char *fs_p = rec_p + round16(kRec * a.smem_faces), *ct_p = fs_p + round16(kRec * a.smem_faces);
    double *far = reinterpret_cast<double *>(ct_p + (size_t)MC * T * 2);
    uint64_t *bar = reinterpret_cast<uint64_t *>(far + 8 * (size_t)r.max_far);
    TileBuf b;
    b.st = reinterpret_cast<double2 *>(st_p);
    b.rec = reinterpret_cast<FaceRec *>(rec_p);
    b.ct = reinterpret_cast<unsigned short *>(ct_p);
    Tile32 b32;
    b32.st = reinterpret_cast<float4 *>(st_p);
    b32.rec = reinterpret_cast<FaceRec32 *>(rec_p);
    b32.ct = b.ct;
    double *fs = reinterpret_cast<double *>(fs_p);
    float *fs32 = reinterpret_cast<float *>(fs_p);

    // the tile's own data, once
    if (tid == 0) mbar_init(bar, 1);
    __syncthreads();
    if (tid == 0) {
        const uint32_t b_state = (uint32_t)nloc * kState, b_rec = round16(kRec * (uint32_t)nf), b_ct = (uint32_t)MC * T * 2u;
        mbar_expect_tx(bar, b_state + b_rec + b_ct);
        bulk_g2s(st_p, F32 ? (const void *)(r.q32[0] + 2 * (size_t)c0) : (const void *)(r.q[0] + 3 * (size_t)c0), b_state, bar);
        bulk_g2s(rec_p, F32 ? a.tile_rec32 + a.tile_rec32_off[tile] : a.tile_rec + a.tile_rec_off[tile], b_rec, bar);
        bulk_g2s(ct_p, a.tile_contrib + (size_t)tile * MC * T, b_ct, bar);
    }
    const int *hrow = a.tile_halo + (size_t)tile * a.halo_stride;
    const int h0 = tid < a.halo_stride ? hrow[tid] : -1;
    const int h1 = tid + NT < a.halo_stride ? hrow[tid + NT] : -1;
    // version v of halo cell i (cell h) into its place: version 0 from the state buffer, later ones from
    // the words its tile publishes; false when the wait for them gives up
    const size_t slot = (size_t)a.n_tiles * T * kWords;
    auto load_halo = [&](int i, int h, unsigned v) {
        if (v == 0) {
            if (F32) {
                for (int k = 0; k < 2; k++) b32.st[2 * (nloc + i) + k] = __ldcg(r.q32[0] + 2 * (size_t)h + k);
            } else {
                for (int k = 0; k < 3; k++) b.st[3 * (nloc + i) + k] = __ldcg(r.q[0] + 3 * (size_t)h + k);
            }
            return true;
        }
        uint4 w[kWords];
        if (!wait_words<kWords>(r.words + (v & 1) * slot + (size_t)h * kWords, r.tag + v, abort, a.wait_polls, w)) return false;
        uint4 *dst = reinterpret_cast<uint4 *>(st_p + (size_t)(nloc + i) * kState);
        dst[0] = make_uint4(w[0].x, w[0].y, w[0].z, w[1].x);
        dst[1] = make_uint4(w[1].y, w[1].z, w[2].x, w[2].y);
        if (!F32) dst[2] = make_uint4(w[2].z, w[kWords - 1].x, w[kWords - 1].y, w[kWords - 1].z);
        return true;
    };
    // this thread's cell as version v, for the tiles that read it: its record w[] as 32-bit words
    auto publish = [&](const unsigned *w, unsigned v) {
        uint4 *dst = r.words + (v & 1) * slot + (size_t)(c0 + tid) * kWords;
#pragma unroll
        for (int k = 0; k < kWords; k++)
            store_word(dst + k, make_uint4(w[3 * k], w[3 * k + 1], F32 && k == 2 ? 0u : w[3 * k + 2], r.tag + v));
    };
    // the halo's version v; with `it`, thread 0 also waits for that iteration's decision and forces
    // (s_word).  False when a wait gave up.
    auto gather = [&](unsigned v, unsigned it) {
        bool ok = true;
        if (h0 >= 0) ok = load_halo(tid, h0, v);
        if (h1 >= 0) ok = load_halo(tid + NT, h1, v) && ok;
        for (int i = tid + 2 * NT; i < a.halo_stride; i += NT) {
            const int h = hrow[i];
            if (h >= 0) ok = load_halo(i, h, v) && ok;
        }
        if (it && tid == 0) {
            unsigned decided = 0, forces;
            ok = wait_word(words + WORD_DECIDED * kFlagStride, it, abort, a.wait_polls, decided) && ok;
            if (ok && !(decided & kStopBit)) ok = wait_word(words + WORD_FORCES * kFlagStride, it, abort, a.wait_polls, forces);
            s_word = decided;
        }
        return !__syncthreads_or(!ok);
    };
    auto give_up = [&] {  // uniform across the block
        if (tid == 0) {
            atomicExch(a.fault, 1);
            atomicExch(words + WORD_ABORT * kFlagStride, 1u);
        }
    };
    double W0[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    double4 cg = make_double4(0.0, 0.0, 0.0, 0.0);
    float4 cg32 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < nloc) {
        if (F32) tile_load_cell_f32(a, c0 + tid, W0, cg32);
        else tile_load_cell(a, c0, tid, W0, cg);
    }
    if (!tile_wait(a, bar, 0)) {
        give_up();
        tile_drain(bar, 0);
        return;
    }
    gather(0, 0);
    // interior faces come first in the records
    int nfi = 0;
    for (int j = 0; j < nf; j += NT) {
        const int code = j + tid < nf ? (F32 ? b32.rec[j + tid].code : b.rec[j + tid].code) : -1;
        nfi += __syncthreads_count(code >= 0 && (code >> (2 * kTileLocalBits)) == TAG_LEFT);
    }
    int n_far = 0;  // farfield and unclassified faces, the first of the boundary faces
    for (int j = nfi; j < nf; j += NT) {
        const int code = j + tid < nf ? (F32 ? b32.rec[j + tid].code : b.rec[j + tid].code) : 0;
        n_far += __syncthreads_count((code >> (2 * kTileLocalBits)) >= TAG_FAR);
    }
    auto ghost_slot = [&](int k) { return F32 ? b32.rec[nfi + k].ghost : b.rec[nfi + k].ghost; };
    for (int k = tid; k < 8 * n_far; k += NT) far[k] = a.ghost[8 * (size_t)ghost_slot(k >> 3) + (k & 7)];
    // does another tile read this thread's cell?
    bool shared_cell = false;
    if (tid < nloc) {
        for (int k = 0; k < MC; k++) {
            const unsigned e = b.ct[k * T + tid];
            if (e == kNoContrib) break;
            const int code = F32 ? b32.rec[e >> 1].code : b.rec[e >> 1].code, mask = (1 << kTileLocalBits) - 1;
            shared_cell |= (code >> (2 * kTileLocalBits)) == TAG_LEFT &&
                           ((code & mask) >= nloc || ((code >> kTileLocalBits) & mask) >= nloc);
        }
    }
    __syncthreads();  // the farfield ghosts are here

    unsigned ver = 0;
    for (int it = 0; it < r.iterations; it++) {
        for (int s = 0; s < r.stages; s++) {
            const bool first = s == 0, last = s == r.stages - 1;
            if (ver) {
                if (!gather(ver, last ? it : 0)) {
                    give_up();
                    return;
                }
                if (last && it && (s_word & kStopBit)) return;  // iteration `it` was the last
            }
            const double alpha = r.stages == 1 ? 1.0
                                 : s == 0      ? 0.0533
                                 : s == 1      ? 0.1263
                                 : s == 2      ? 0.2375
                                 : s == 3      ? 0.4414
                                               : 1.0;
            // only an iteration's final state goes to the state buffers
            const int out = (ver + 1) & 1;
            const LoopStep sp{a, far, nfi, alpha, first, last, minit, r.q[out], r.q32[out]};
            if constexpr (F32) tile_fluxes_f32<NT>(a, sp, b32, fs32, tid, nf, c0);
            else tile_fluxes<EXACT, NT>(a, sp, b, fs, tid, nf, c0);
            __syncthreads();
            if (last)
                for (int k = tid; k < 8 * n_far; k += NT) a.ghost[8 * (size_t)ghost_slot(k >> 3) + (k & 7)] = far[k];
            double r2 = 0.0;
            ver++;
            if (tid < nloc) {
                if constexpr (F32) {
                    PrimF o;
                    r2 = tile_update_f32(a, sp, b32, fs32, c0, tid, W0, cg32, o);
                    b32.st[2 * tid] = make_float4(o.rho, o.u, o.v, o.w);
                    b32.st[2 * tid + 1] = make_float4(o.p, o.H, o.s, o.r);
                    const float v[9] = {o.rho, o.u, o.v, o.w, o.p, o.H, o.s, o.r, 0.f};
                    unsigned w[9];
#pragma unroll
                    for (int k = 0; k < 9; k++) w[k] = __float_as_uint(v[k]);
                    if (shared_cell) publish(w, ver);
                } else {
                    Prim o;
                    r2 = tile_update<EXACT>(a, sp, b, fs, c0, tid, W0, cg, o);
                    store_prim(b.st, tid, o);
                    const double v[6] = {o.rho, o.u, o.v, o.w, o.p, o.H};
                    unsigned w[12];
#pragma unroll
                    for (int k = 0; k < 6; k++) {
                        w[2 * k] = (unsigned)__double2loint(v[k]);
                        w[2 * k + 1] = (unsigned)__double2hiint(v[k]);
                    }
                    if (shared_cell) publish(w, ver);
                }
            }
            if (last) {
                const double sum = block_sum<NT>(r2);  // ends with a barrier after every thread's stores
                if (tid == 0)
                    store_word(r.partials + tile, make_uint4((unsigned)__double2loint(sum), (unsigned)__double2hiint(sum),
                                                             0u, r.tag + ver));
                if (tid == NT - 1) store_release(r.flags + (size_t)tile * kFlagStride, (unsigned)(it + 1));
            }
        }
        minit = false;
    }
}

// The block sizes, largest first: threads, and the blocks per SM that the registers are budgeted for.
// More threads shorten a tile's flux phase (one face per thread at 512); a tighter budget spills (the
// update of 256 threads takes 1.7 us at three blocks' registers and 0.9 us at two's), so each count of
// blocks per SM has its own.
struct ResidentShape {
    int threads, blocks;
};
constexpr ResidentShape kResidentShapes[] = {{512, 1}, {256, 2}, {256, 3}, {128, 4}, {128, 6}};
constexpr int kResidentShapeCount = 5;

// The more tiles share an SM, the less the stage kernels' fixed costs weigh.  us per RK5 iteration, forces
// sampled every iteration, autotuned stage kernels against this kernel (B200):
//   tiles        channel, 2 layers       O-grid, 4 layers        box of tetrahedra
//   FP64         436  45.0  31.6         436  43.7  34.9         435  42.8  35.6
//                587  46.6  41.5         587  44.8  49.2         571  44.0  48.4      648  55.1  62.6
//   FP32_FLUX    587  47.4  36.4         587  43.8  37.4         571  42.2  43.9      648  42.2  48.4
//                704  47.3  47.7         781  44.4  57.6         824  43.8  57.5
//   FP64_EXACT   291   126   111         313   152   207         289   127   118      375   143   225
// Up to three tiles per SM (two in exact mode, whose RMS and forces are the control block's sequential
// sums) it is the faster one everywhere; with more, the shapes of 128 threads, that depends on the mesh, and
// the creation of a tuned solver times both ways.
constexpr int kTimedShape = 3;

template <int PREC>
struct ResidentLaunch {
    static const void *kernel(int shape) {
        switch (shape) {
            case 0: return (const void *)resident_kernel<PREC, 512, 1>;
            case 1: return (const void *)resident_kernel<PREC, 256, 2>;
            case 2: return PREC == PREC_EXACT ? nullptr : (const void *)resident_kernel<PREC, PREC == PREC_EXACT ? 128 : 256, PREC == PREC_EXACT ? 4 : 3>;
            case 3: return (const void *)resident_kernel<PREC, 128, 4>;
            default: return PREC == PREC_EXACT ? nullptr : (const void *)resident_kernel<PREC, 128, PREC == PREC_EXACT ? 4 : 6>;
        }
    }
    // Blocks of the shape that fit on an SM (0: not built for this precision).
    static int max_blocks(int shape, size_t smem) {
        if (!kernel(shape)) return 0;
        raise_smem_limit(kernel(shape), smem);
        int n = 0;
        E3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel(shape), kResidentShapes[shape].threads, smem));
        return n;
    }
    // False: the GPU, or the part of it that the stream may use, does not hold the grid at once.
    static bool launch(const StageArgs &a, const ResidentArgs &r, int shape, size_t smem, cudaStream_t s) {
        void *args[] = {const_cast<StageArgs *>(&a), const_cast<ResidentArgs *>(&r)};
        const cudaError_t e = cudaLaunchCooperativeKernel(kernel(shape), dim3(a.n_tiles + 1),
                                                          dim3(kResidentShapes[shape].threads), args, smem, s);
        if (e == cudaErrorCooperativeLaunchTooLarge) {
            cudaGetLastError();
            return false;
        }
        E3D_CUDA(e);
        return true;
    }
};

}  // namespace e3d
