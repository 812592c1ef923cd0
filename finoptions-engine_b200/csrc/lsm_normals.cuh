// lsm_normals.cuh - a path's standard normals: Philox words through bounded ZIGNOR over 256 layers
// (crates/finoptions-sim/src/random/normal.rs:33-109), one path per thread.
//
// What bounds it is instruction issue, so the lanes of a warp stay together although their
// rejections differ: every lane runs the words of its stream through the sampler four at a time, in
// counter order, and what a word means (a fresh draw, the uniform of a wedge test, a half of a
// tail draw) is a state of the lane. Accepted normals wait in a ring of eight in shared memory
// (the thread's own column, so no bank conflicts) and leave four at a time at a warp-uniform slot.
//   * A rejection costs its lane one word or two and nothing else: no lane generates a block of its
//     own, no redraw runs apart, and the next draws do not move. A path of more than eight normals
//     starts four words ahead, which covers the 1.25 words that 52 normals lose on average; the
//     few lanes that lose more run one more block.
//   * A wedge test compares the uniform with the density's parabola through the layer's ends and
//     middle. The two differ by at most Wedge::gap, so further apart the parabola decides and exp is
//     not evaluated; closer (about one test in 140) the exact test runs.
// Words leave the generator in counter order and every decision is the exact test's, so a path's
// normals do not depend on any of this.
// Warp instructions per normal at 52 normals a path, 2^20 paths: 140 with a queue of words per lane and
// redraws in line, 91 so, of which Philox takes 22.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "lsm_device.cuh"

namespace fo {

// In global memory: a warp reads 32 consecutive entries (constant memory serves one a cycle).
static __device__ const uint64_t g_zig_x[257] = FO_ZIG_NORM_X_BITS;
static __device__ const uint64_t g_zig_f[257] = FO_ZIG_NORM_F_BITS;
static __device__ const uint64_t g_zig_wedge[256][4] = FO_ZIG_WEDGE_BITS;

constexpr uint32_t kRing = 8;            // normals a thread holds
constexpr uint32_t kChunkNormals = kChunkSteps;  // normals taken together: two blocks
constexpr uint32_t kReserveNormals = 8;  // paths of more normals than this start four words ahead

// A layer's wedge between its edges a < b, with t the position from a to b and h(t) the density's
// position from f(a) to f(b): |h(t) - (t + bend t (1 - t))| <= gap (gen_zignor_tables.py).
struct alignas(16) Wedge {
    double inverse_width, bend, gap, pad;
};

// Shared memory of a CTA of T sampling threads.
template <int T>
struct NormalSmem {
    double2 edge[256];  // x[i], x[i + 1]: a layer's width and the width its inner part accepts
    Wedge wedge[256];   // layers from 1
    double f[257];
    double ring[kRing][T];
    double parked[kChunkNormals][T];  // the caller's: what it keeps of a chunk
};

template <int T>
__device__ __forceinline__ void load_normal_tables(NormalSmem<T>& sm) {
    for (int i = threadIdx.x; i < 257; i += blockDim.x) {
        sm.f[i] = bits_to_double(g_zig_f[i]);
        if (i == 256) break;
        sm.edge[i] = make_double2(bits_to_double(g_zig_x[i]), bits_to_double(g_zig_x[i + 1]));
        sm.wedge[i] = Wedge{bits_to_double(g_zig_wedge[i][0]), bits_to_double(g_zig_wedge[i][1]),
                            bits_to_double(g_zig_wedge[i][2]), 0.0};
    }
    __syncthreads();
}

// One path's stream. The caller takes its normals in chunks of four, in order, with next.
// Invariant between chunks: at most four normals wait in the ring. Everything is in line and there is one
// copy of it: a call in the path loop, even one never taken, costs the caller's registers.
template <int T>
struct NormalStream {
    const NormalSmem<T>* tables;
    double* ring;        // this thread's column
    uint32_t path, domain;
    uint32_t tail;       // normals accepted so far (modulo 2^32: used for ring slots and differences)
    uint32_t state;      // what the next word is: kFresh, kWedge, kTailX / kTailY (plus kNegative)
    uint64_t held;       // the rejected draw's word (kWedge) or the tail's first word (kTailY)
    uint64_t blocks;     // blocks generated

    static constexpr uint32_t kFresh = 0, kWedge = 1, kTailX = 2, kTailY = 4, kNegative = 8;

    __device__ __forceinline__ void init(NormalSmem<T>& sm, uint32_t domain_, uint32_t path_) {
        tables = &sm;
        ring = &sm.ring[0][threadIdx.x];
        path = path_;
        domain = domain_;
        tail = 0;
        state = kFresh;
        held = 0;
        blocks = 0;
    }

    // Normals k .. k + C - 1 of a path of n (k a multiple of C; those past n are undefined). False when the
    // sampler gave up on one of them. C is kChunkNormals, or 2 for paths of at most two normals.
    template <int C>
    __device__ __forceinline__ bool next(const PhiloxKeys& keys, uint32_t k, uint32_t n, double (&z)[C]) {
        const uint32_t left = n - k;
        const uint32_t want = left < C ? left : C;
        // C words a round: one round, two at the start of a path that keeps a reserve, and more for
        // the lanes still short of the chunk (k normals have left the ring). The ring has room: at
        // most four normals wait when a chunk starts, fewer than four in a lane that is short. The
        // reference gives up on a normal after 2^20 rejections (random/normal.rs:66); here the
        // chunk does.
        int rounds = k == 0 && n > kReserveNormals ? -1 : 0;
        do {
            if (rounds >= kMaxRejectionIterations) return false;
            run<C / 2>(keys);
            rounds += 1;
        } while (rounds <= 0 || tail - k < want);
#pragma unroll
        for (uint32_t j = 0; j < C; ++j) z[j] = ring[((k + j) % kRing) * T];
        return true;
    }
    // Normal k of the chunk that next handed out last.
    __device__ __forceinline__ double normal(uint32_t k) const { return ring[(k % kRing) * T]; }

    // N blocks through the sampler.
    template <int N>
    __device__ __forceinline__ void run(const PhiloxKeys& keys) {
        uint64_t words[2 * N];
        philox_blocks<N>(blocks, path, domain, keys, words);
        blocks += N;
        const uint32_t tail0 = tail, state0 = state;
        const uint64_t held0 = held;
        bool hard = state > kWedge;  // the tail, or a wedge test too close for the parabola
#pragma unroll
        for (int i = 0; i < 2 * N; ++i) {
            const uint32_t layer = uint32_t(words[i]) & 0xffu;
            const double2 edge = tables->edge[layer];
            double value = zig_symmetric_unit(words[i]) * edge.x;
            bool accepted = fabs(value) < edge.y;
            if (!accepted || state != kFresh) {
                if (state == kFresh) {
                    held = words[i];
                    state = kWedge;
                    hard = hard || layer == 0;
                } else {
                    state = kFresh;
                    const uint32_t drawn = uint32_t(held) & 0xffu;
                    const double2 sides = tables->edge[drawn];
                    const Wedge& wedge = tables->wedge[drawn];
                    value = zig_symmetric_unit(held) * sides.x;
                    const double t = (fabs(value) - sides.y) * wedge.inverse_width;
                    // The uniform less at most 2^-53.
                    const double u = bits_to_double((words[i] >> 12) | kExponent0) - 1.0;
                    const double apart = u - fo_fma(wedge.bend, fo_fma(-t, t, t), t);
                    hard = hard || !(fabs(apart) > wedge.gap);
                    accepted = apart > 0.0;
                }
            }
            ring[(tail % kRing) * T] = value;  // overwritten by the next accepted draw unless accepted
            tail += accepted ? 1u : 0u;
        }
        if (hard) {
            // Again, word by word through every state (one lane's words in 300).
            tail = tail0;
            state = state0;
            held = held0;
#pragma unroll 1
            for (int i = 0; i < 2 * N; ++i) {
                const uint64_t low = (i & 1) ? words[1] : words[0];
                const uint64_t high = (i & 1) ? words[2 * N - 1] : words[2 * N - 2];
                word_by_word((i & 2) ? high : low);
            }
        }
    }

    __device__ __forceinline__ void word_by_word(uint64_t word) {
        double value = 0.0;
        bool done = false;
        if (state == kFresh) {
            const uint32_t layer = uint32_t(word) & 0xffu;
            value = zig_symmetric_unit(word) * tables->edge[layer].x;
            done = fabs(value) < tables->edge[layer].y;
            if (!done) {
                held = word;
                state = layer != 0 ? kWedge : kTailX | (zig_symmetric_unit(word) < 0.0 ? kNegative : 0u);
            }
        } else if (state == kWedge) {
            // The wedge test itself (random/normal.rs:72-79).
            const uint32_t layer = uint32_t(held) & 0xffu;
            value = zig_symmetric_unit(held) * tables->edge[layer].x;
            const double u = double(word >> 11) * (1.0 / 9007199254740992.0);
            const double inner = tables->f[layer + 1], outer = tables->f[layer];
            done = inner + (outer - inner) * u < fo_exp(-0.5 * value * value);
            state = kFresh;
        } else if (state & kTailX) {
            held = word;
            state ^= kTailX | kTailY;
        } else {
            // One draw of the tail beyond r (random/normal.rs:50-63).
            const double r = bits_to_double(FO_ZIG_NORM_R_BITS);
            const double ox = bits_to_double((held >> 12) | kExponent0) - (1.0 - 1.1102230246251565e-16);
            const double oy = bits_to_double((word >> 12) | kExponent0) - (1.0 - 1.1102230246251565e-16);
            const double x = fo_log(ox) / r, y = fo_log(oy);
            done = -2.0 * y >= x * x;
            value = (state & kNegative) ? x - r : r - x;
            state = done ? kFresh : state ^ (kTailX | kTailY);
        }
        if (done) {
            ring[(tail % kRing) * T] = value;
            tail += 1;
        }
    }
};

}  // namespace fo
