// lsm_persistent.cuh - grouped, row-addressed and ragged LSM batches as one persistent launch per
// wave (crates/finoptions-lsm/src/batch/pricing.rs:452-589 for the work of one group).
//
// A wave's work is a queue of items (lsm_batch.cuh): the training simulation of a group's path
// blocks, the backward fit of one (group, strike) problem, the evaluation of a group's path blocks
// for a chunk of its strikes. The host orders it topologically and largest work first: every
// group's simulation, then every problem's fit (largest training paths x rows first), then the
// evaluations in the order their groups' fits were queued. Resident CTAs take items from the queue
// in order; a fit waits until its group's training paths are stored, an evaluation until its
// group's fits are done, each wait bounded in time. The CTA that finishes a group's last
// evaluation item writes that group's summaries, so the launch ends with every result written.
//
// Work items run the same arithmetic, in the same order, as pricing a group alone: a problem's fit
// is one CTA over its paths in a fixed thread-to-path assignment, and evaluation partials are
// kept per 256-path block. The results therefore do not depend on the queue order, the paths per
// item or the grid size the autotuner picks.
//
// Data written by one CTA and read by another inside the launch (stored paths, fitted records,
// partials, status words) is read through L2 (ld.global.cg): L1 is not coherent across SMs.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <type_traits>

#include "lsm_adjoint.cuh"
#include "lsm_batch.cuh"
#include "lsm_batch_kernels.h"
#include "lsm_common.cuh"
#include "lsm_fit_warp.cuh"
#include "lsm_kernels.h"
#include "lsm_sync.cuh"

namespace fo {

namespace {

constexpr int kPersistentThreads = 256;
using BatchNormals = NormalSmem<kPersistentThreads>;
constexpr int kPersistentLoads = 1;  // paths a backward thread of the persistent launch loads together
constexpr int kFitKernelLoads = 4;     // ... and one of the fit kernel
// A dependency wait gives up after this long: one problem's fit on one CTA can take seconds for
// populations of millions of paths, so the limit is well above any fit's duration.
constexpr unsigned long long kDependencyTimeoutNs = 20000000000ull;

__device__ __forceinline__ unsigned long long ld_l2_u64(const unsigned long long* p) { return __ldcg(p); }

__device__ __forceinline__ bool status_failed(const unsigned long long* word) { return ld_l2_u64(word) != kNone; }

// Thread 0 waits (time-bounded) until *counter reaches target; every thread returns whether it did.
// The pause between polls doubles from 64 ns up to max_pause: dependency waits keep their polls of
// L2 rare, a team's per-row exchange polls often.
__device__ bool wait_for(const unsigned* counter, unsigned target, unsigned* timeout, int* flag,
                         unsigned max_pause = 4096) {
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned pause = 64;
        unsigned long long start = 0;
        while (ld_relaxed_gpu(counter) < target) {
            if (ld_volatile_u32(timeout) != 0) {
                ok = 0;
                break;
            }
            const unsigned long long now = global_timer_ns();
            if (start == 0) {
                start = now;
            } else if (now - start > kDependencyTimeoutNs) {
                atomicExch(timeout, 1u);
                ok = 0;
                break;
            }
            __nanosleep(pause);
            pause = pause < max_pause ? 2 * pause : pause;
        }
        __threadfence();  // acquire: the items counted are visible to this CTA's reads below
        *flag = ok;
    }
    __syncthreads();
    return *flag != 0;
}

// Every thread's writes of the item are made visible device-wide, then thread 0 adds n.
// Returns (in thread 0) the counter's value before the addition.
__device__ __forceinline__ unsigned signal_done(unsigned* counter, unsigned n) {
    __threadfence();
    __syncthreads();
    unsigned before = 0;
    if (threadIdx.x == 0) before = atomicAdd(counter, n);
    return before;
}

// A row's rule as the evaluation stages it. Rules written by other CTAs of the same launch are read
// through L2; kReadOnly (a later kernel) may use the read-only path.
template <bool kReadOnly>
__device__ __forceinline__ void load_rule(const ExerciseRule* rule, ExerciseRule* out) {
    static_assert(sizeof(ExerciseRule) == 4 * sizeof(double2), "a rule loads as four 16-byte words");
    const double2* src = reinterpret_cast<const double2*>(rule);
    double2* dst = reinterpret_cast<double2*>(out);
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = kReadOnly ? __ldg(src + i) : __ldcg(src + i);
}

// A row that its ExerciseRule does not decide (an unsupported row, an extreme market): the record's kind and, for a regression, its model. An in-the-money
// path at a row without training support is counted.
template <int D>
__device__ __forceinline__ int decide_record(const BatchArgs& a, uint32_t record, double spot, double strike) {
    const FitRecord& rec = a.records[record];
    const int32_t kind = __ldcg(&rec.kind);
    if (kind == kRuleNoSupport) atomicAdd(&a.itm_counts[record], 1u);
    if (kind != kRuleRegression) return kDecideContinue;
    FitModel model;
    const double2* src = reinterpret_cast<const double2*>(&rec.model);
    double2* dst = reinterpret_cast<double2*>(&model);
    for (int i = 0; i < int(sizeof(FitModel) / sizeof(double2)); ++i) dst[i] = __ldcg(src + i);
    return decide_general<D>(&model, spot, strike, a.tie_rule);
}

__device__ __forceinline__ uint32_t blocks_of(uint64_t paths) {
    return uint32_t((paths + kPersistentThreads - 1) / kPersistentThreads);
}

// ---- training simulation ------------------------------------------------------------------------

__device__ void simulate_item(const BatchArgs& a, uint32_t gi, uint32_t first, uint32_t count,
                              BatchNormals& normals, const PhiloxKeys& keys) {
    const BatchGroup& g = a.groups[gi];
    const DevicePlan plan = g.plan;  // a local copy: its fields stay in registers (no reloads across stores)
    const uint64_t P = plan.train_paths;
    const uint32_t fsr = plan.first_stored_row;
    double* out = a.slab + g.slab_offset;
    const bool escrowed = plan.escrowed != 0;
    for (uint32_t b = first; b < first + count; ++b) {
        const uint64_t p = uint64_t(b) * kPersistentThreads + threadIdx.x;
        if (p >= P) continue;
        double* at = out + p;  // rows come in order, the unstored origin row first
        auto store = [&](int row, double value) {
            if (uint32_t(row) < fsr) return;
            // Escrowed observations: origin -> S0; otherwise prepaid forward + prepaid cash.
            if (escrowed) value = plan.row_node[row] == 0 ? plan.initial_spot : value + plan.escrow_cash[row];
            *at = value;
            at += P;
        };
        const SimResult r = simulate_path(plan, normals, keys, plan.train_domain, uint32_t(p), store);
        if (r.code != 0) atomicMin(&a.group_status[gi].train_sim_fail, (unsigned long long)p);
    }
}

// ---- backward fit of one problem ----------------------------------------------------------------

// The CTAs that fit one problem together. Member m owns the contiguous paths [lo, hi).
struct Team {
    uint32_t member, members;
    double2* slots;    // [2][members][kSlots]
    unsigned* arrive;  // arrivals at this problem's exchanges
    unsigned round;    // exchanges this member has made
    unsigned* timeout;
    int* flag;
};

// Every member publishes its CTA totals of a reduction (S double-double slots) and sums all members'
// in member order, so each member ends with the same totals. Consecutive exchanges alternate between
// two buffers: a member overwrites one only after every member has arrived at the exchange in
// between, that is, has finished reading it. False when a wait gave up (the timeout flag is set).
static_assert(kTeamSlots == kSlots, "a member's exchange holds one row reduction");

template <int S, bool kTeam>
__device__ bool team_exchange(Team& t, dd* total /* shared [S] */) {
    if constexpr (!kTeam) return true;
    if (t.members == 1) return true;
    const unsigned parity = t.round & 1u;
    if (threadIdx.x < S)
        t.slots[(size_t(parity) * t.members + t.member) * kSlots + threadIdx.x] =
            make_double2(total[threadIdx.x].hi, total[threadIdx.x].lo);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(t.arrive, 1u);
    t.round += 1;
    if (!wait_for(t.arrive, t.members * t.round, t.timeout, t.flag, 256)) return false;
    if (threadIdx.x < S) {
        const double2* column = t.slots + size_t(parity) * t.members * kSlots + threadIdx.x;
        dd acc = dd_make(0.0);
        for (uint32_t m = 0; m < t.members; ++m) {
            const double2 v = __ldcg(column + size_t(m) * kSlots);
            acc = dd_add(acc, dd{v.x, v.y});
        }
        total[threadIdx.x] = acc;
    }
    __syncthreads();
    return true;
}

struct BackwardItemSmem {
    double red[32 * kSlots];
    dd total[kSlots];
    FitModel model;
    ExerciseRule rule;
    double new_pivot;  // the row's own mean, when its sums are taken again about it
    int kind;
    int recenter;
    int beyond[2];     // by order parity: a staged spot or value is beyond kRuleSpotLimit, or not a number
};

// A stored training state. The persistent launch reads rows that other CTAs of the same launch wrote,
// so through L2 (the SM's L1 is not coherent with other SMs' writes); the fit kernel of the phase
// executor runs after the simulation kernel has finished, so its reads may use the read-only path.
template <bool kReadOnly>
__device__ __forceinline__ double load_slab(const double* p) {
    if constexpr (kReadOnly) return __ldg(p);
    else return __ldcg(p);
}

// Backward induction of one problem over the group's stored rows (policy.rs:215-296, 471-601): per row
// one deterministic reduction of in-the-money power sums and the regression solve by one warp. A
// problem of up to kTeamPaths paths is one CTA's; a larger one is split over a team of CTAs (this one
// is member `member` of `members`), each owning a contiguous range of paths, whose CTA sums are
// exchanged in member order before every decision, so that every member fits the same model; member
// 0 writes the records. Thread t owns paths t + 256 m of the range (round m = 0, 1, ...). The values
// of the first chip_rounds rounds live in shared memory (`chip`), the others in HBM; neither where a
// value lives nor how many paths a thread loads together (kU) changes the order of a sum.
// False when a team exchange gave up.
//
// What bounds it: a path-row is 36 FP64 operations (72 cycles a warp and scheduler) beside 24 to 32 bytes
// of L2 traffic, and between two rows' passes stands a serial part (reduce, decide, fit, rule) of 13,000
// cycles that only the SM's other CTA can fill. At 4,096 states x 8 strikes x 32,768 paths the fits took
// 271 ms with four CTAs per SM, one path at a time and every value in HBM, its paths decided in a branch of
// their own. They take 167 ms so: two CTAs (128 registers a thread, 176 bytes of spill stores in the kernel; with three or
// four the pass spills, 197 and 274 ms), values on chip where they fit, kU = 4 paths side by side without a branch (kU = 2 179 ms,
// 3 167 ms) and the next four loaded ahead (170 ms without). A row takes 75,000 cycles, 58,000 the pass.
template <int D, bool kReadOnlySlab, bool kTeam, int kU>
__device__ bool backward_item(const BatchArgs& a, uint32_t pi, uint32_t member, uint32_t members, unsigned* timeout,
                              int* flag, BackwardItemSmem& sm, double* chip, uint32_t chip_rounds) {
    const BatchProblem pr = a.problems[pi];
    if (pr.skip_fit) return true;
    if (status_failed(&a.group_status[pr.group].train_sim_fail)) return true;
    const BatchGroup& g = a.groups[pr.group];
    const DevicePlan plan = g.plan;  // a local copy: its fields stay in registers (no reloads across stores)
    ProblemStatus* st = a.problem_status + pi;
    FitRecord* records = a.records + pr.records;
    constexpr uint32_t T = kPersistentThreads;
    const uint64_t P = plan.train_paths;
    // This member's paths [lo, hi): contiguous ranges of a multiple of 256 paths, in member order.
    const uint64_t span = members == 1 ? P : ((P + members - 1) / members + 255) / 256 * 256;
    const uint64_t lo = members == 1 ? 0 : (uint64_t(member) * span < P ? uint64_t(member) * span : P);
    const uint64_t hi = members == 1 ? P : (lo + span < P ? lo + span : P);
    const uint32_t n = uint32_t(hi - lo);
    const uint32_t full = n / T, rest = n % T;  // rounds in which every thread has a path, and the last one's paths
    const uint32_t rounds = full + (threadIdx.x < rest ? 1u : 0u);  // this thread's
    // Restrict-qualified: this problem's values are its own, and the slab is only read here, so the
    // loads of several paths may be issued together, ahead of the stores.
    double* __restrict__ values = a.values + pr.values + lo + threadIdx.x;
    const double* __restrict__ slab = a.slab + g.slab_offset + lo + threadIdx.x;
    chip += threadIdx.x;
    Team team{member, members, a.team_slots + pr.team_base, a.team_arrive + pi, 0u, timeout, flag};
    const bool writer = member == 0;
    const double K = pr.strike;
    const Divisor Kd = make_divisor(K);
    const int degree = a.degree;
    const bool strict = a.tie_rule == 0;
    const uint32_t E = plan.rows - 1;
    const uint32_t fsr = plan.first_stored_row;
    const int lowest = plan.origin_row ? 1 : 0;
    auto row_ptr = [&](uint32_t row) { return slab + uint64_t(row - fsr) * P; };
    auto load_value = [&](uint32_t m) { return m < chip_rounds ? chip[m * T] : values[m * T]; };
    auto store_value = [&](uint32_t m, double v) {
        if (m < chip_rounds) chip[m * T] = v;
        else values[m * T] = v;
    };
    auto key = [&](uint32_t order, uint32_t m) {
        return ((unsigned long long)order << 32) | (lo + threadIdx.x + uint64_t(m) * T);
    };
    // Moneyness of an in-the-money state: the correctly rounded quotient by the strike.
    const auto moneyness = [&](double spot) {
        const double x = Kd.inv != 0.0 ? divide_above(spot, Kd) : spot / K;
        return finite_nonnegative(x) ? x : spot / K;
    };
    if (threadIdx.x < 2) sm.beyond[threadIdx.x] = 0;
    __syncthreads();
    uint32_t order = 0;
    int row = int(E) - 1;
    double pivot = 1.0;
    RowSums sums;
    uint32_t itm_paths = 0;  // in-the-money paths in the sums (sums.acc[0], counted in integers)
    auto clear_sums = [&] {
#pragma unroll
        for (int k = 0; k < kSlots; ++k) sums.acc[k] = 0.0;
        itm_paths = 0;
    };
    // The sums of a row whose discounted values are stored, path by path with every check.
    auto sum_row = [&](int at, bool report) {
        clear_sums();
        const double* spots = row_ptr(uint32_t(at));
        for (uint32_t m = 0; m < rounds; ++m) {
            const double v = load_value(m), sp = load_slab<kReadOnlySlab>(&spots[m * T]);
            const bool finite = fo_isfinite(v);
            if (report && !finite) atomicMin(&st->fit_payoff_fail, key(order, m));
            if (!(sp > K)) continue;
            const double x = moneyness(sp);
            if (!within_rule(sp)) sm.beyond[order & 1] = 1;
            if (!finite_nonnegative(x) || !finite) {
                sums.acc[kBadSlot] += 1.0;
                if (report) atomicMin(&st->fit_nonfinite, key(order, m));
            } else {
                itm_paths += 1;
                accumulate_moments(sums, x, v, pivot);
            }
        }
    };
    clear_sums();
    {
        // The terminal payoffs, discounted into the first fitted row where there is one.
        const double* terminal = row_ptr(E);
        const double disc = row >= lowest ? plan.disc_from_later[row] : 1.0;
#pragma unroll 4
        for (uint32_t m = 0; m < rounds; ++m) {
            const double d = load_slab<kReadOnlySlab>(&terminal[m * T]) - K;
            store_value(m, (d > 0.0 ? d : 0.0) * disc);
        }
    }
    if (row >= lowest) {
        // The in-the-money mean of the first fitted row is its moment pivot.
        const double* srow = row_ptr(uint32_t(row));
        double loc[2] = {0.0, 0.0};
#pragma unroll 4
        for (uint32_t m = 0; m < rounds; ++m) {
            const double sp = load_slab<kReadOnlySlab>(&srow[m * T]);
            if (!(sp > K)) continue;
            const double x = moneyness(sp);
            if (fo_isfinite(x)) {
                loc[0] += 1.0;
                loc[1] += x;
            }
        }
        cta_reduce_dd<2>(loc, sm.red, sm.total);
        if (!team_exchange<2, kTeam>(team, sm.total)) return false;
        if (sm.total[0].hi > 0.0) pivot = dd_round(dd_div(sm.total[1], sm.total[0]));
        sum_row(row, true);
    }
    for (; row >= lowest; --row, ++order) {
        sums.acc[0] = double(itm_paths);
        cta_reduce_dd<kSlots>(sums.acc, sm.red, sm.total);
        if (sm.beyond[order & 1] != 0 && order > 0) {
            // The pass that staged the row formed its sums without looking at what lies beyond the limit.
            sum_row(row, true);
            sums.acc[0] = double(itm_paths);
            cta_reduce_dd<kSlots>(sums.acc, sm.red, sm.total);
        }
        if (!team_exchange<kSlots, kTeam>(team, sm.total)) return false;
        if (threadIdx.x == 0) {
            const uint64_t itm = uint64_t(sm.total[0].hi);
            double mean = pivot;
            sm.recenter = degree > 0 && itm >= uint64_t(degree + 1) && sm.total[kBadSlot].hi == 0.0 &&
                                  pivot_too_far(sm.total, pivot, itm, &mean)
                              ? 1
                              : 0;
            sm.new_pivot = mean;
        }
        __syncthreads();
        if (sm.recenter) {
            // The pivot lay more than a standard deviation from the row's in-the-money mean: take
            // the row's sums again about that mean.
            pivot = sm.new_pivot;
            sum_row(row, false);
            sums.acc[0] = double(itm_paths);
            cta_reduce_dd<kSlots>(sums.acc, sm.red, sm.total);
            if (!team_exchange<kSlots, kTeam>(team, sm.total)) return false;
        }
        if (threadIdx.x < 32) {
            // Warp 0 decides the row and fits it (the lane-parallel solve, bit-identical to the
            // one-thread one), then writes the row's record, the model as 16-byte words by lanes.
            const uint64_t itm = uint64_t(sm.total[0].hi);
            const uint64_t bad = uint64_t(sm.total[kBadSlot].hi);
            const uint64_t population = itm + bad;
            const uint32_t required = uint32_t(degree + 1);
            int kind;
            if (population == 0) {
                kind = a.support == 1 ? kRuleContinue : kRuleNoSupport;
            } else if (population < required && a.support == 1) {
                kind = kRuleContinue;
            } else if (population < required || bad > 0) {
                kind = kRuleFitFailed;  // InsufficientObservations / non-finite population
            } else {
                fit_continuation_warp(sm.total, pivot, itm, degree, a.rank_tolerance, plan.rank_limit, &sm.model);
                kind = sm.model.status == kFitOk ? kRuleRegression : kRuleFitFailed;
            }
            FitRecord& rec = records[row];
            constexpr int kModelWords = int(sizeof(FitModel) / sizeof(double2));
            static_assert(sizeof(FitModel) % sizeof(double2) == 0, "FitModel is 16-byte aligned");
            if (writer && threadIdx.x < kModelWords)
                reinterpret_cast<double2*>(&rec.model)[threadIdx.x] =
                    reinterpret_cast<const double2*>(&sm.model)[threadIdx.x];
            if (threadIdx.x == 0) {
                sm.rule = kind == kRuleRegression ? make_exercise_rule(sm.model, D, K) : never_exercise();
                sm.kind = kind;
                sm.beyond[(order + 1) & 1] = 0;
            }
            if (writer && threadIdx.x == 0) {
                rec.kind = kind;
                rec.itm = population;
                rec.pivot = pivot;
                rec.origin_exercise = 0;
                rec.origin_continuation = 0.0;
                rec.diag_status = -1;
            }
        }
        __syncthreads();
        const int kind = sm.kind;
        if (kind == kRuleFitFailed) return true;  // the problem's fit raised; the host reports it
        if (kind == kRuleRegression) pivot = sm.model.mean;
        const bool stage_next = row - 1 >= lowest;
        const bool plain = sm.rule.general == 0 && sm.beyond[order & 1] == 0;
        const double disc = stage_next ? plan.disc_from_later[row - 1] : 1.0;
        const double* cur = row_ptr(uint32_t(row));
        const double* nxt = stage_next ? row_ptr(uint32_t(row - 1)) : cur;
        clear_sums();
        if (plain && stage_next && Kd.inv != 0.0) {
            // The pass proper: decide, discount, add to the next row's sums. Spots and values beyond the
            // rule's limit are only noticed (their high words' maximum) and looked at after it.
            const ExerciseRule rule = sm.rule;
            uint32_t highest = 0;
            // N paths side by side, without a branch of their own: a path out of the money adds t = 0 and
            // y = 0, which changes no sum. Groups with none in the money skip the part.
            const auto group = [&](auto strict_rule, auto& v, auto& sc, auto& sn) {
                constexpr int N = int(sizeof(v) / sizeof(v[0]));
                bool decides = false, adds = false;
                double t[N];
                bool in[N];
#pragma unroll
                for (int u = 0; u < N; ++u) {
                    sc[u] -= K;
                    decides = decides || sc[u] > 0.0;
                    in[u] = sn[u] > K;
                    adds = adds || in[u];
                }
                if (decides) {
#pragma unroll
                    for (int u = 0; u < N; ++u) {
                        const double c = rule_continuation<D>(rule, sc[u]);
                        v[u] = sc[u] > 0.0 && (decltype(strict_rule)::value ? sc[u] > c : sc[u] >= c) ? sc[u] : v[u];
                    }
                }
#pragma unroll
                for (int u = 0; u < N; ++u) {
                    v[u] *= disc;
                    highest = max(highest, max(uint32_t(__double2hiint(v[u])), uint32_t(__double2hiint(sn[u]))));
                }
                if (adds) {
                    double y[N];
#pragma unroll
                    for (int u = 0; u < N; ++u) {
                        t[u] = in[u] ? divide_above(sn[u], Kd) - pivot : 0.0;
                        y[u] = in[u] ? v[u] : 0.0;
                        itm_paths += in[u] ? 1u : 0u;
                    }
#pragma unroll
                    for (int u = 0; u < N; ++u) accumulate_centred(sums, t[u], y[u]);
                }
            };
            const auto pass = [&](auto strict_rule, auto on_chip, uint32_t from, uint32_t to) {
                double* const held = decltype(on_chip)::value ? chip : values;
                uint32_t m = from;
                if (from + kU <= to) {
                    // The next kU paths' loads are issued ahead of the current ones' arithmetic; two sets of
                    // registers take turns.
                    double v0[kU], c0[kU], n0[kU], v1[kU], c1[kU], n1[kU];
                    const uint32_t end = to - kU;  // the last whole group's first round
                    const auto fetch = [&](uint32_t at, auto& v, auto& sc, auto& sn) {
                        at = min(at, end);
#pragma unroll
                        for (int u = 0; u < kU; ++u) {
                            v[u] = held[(at + u) * T];
                            sc[u] = load_slab<kReadOnlySlab>(&cur[(at + u) * T]);
                            sn[u] = load_slab<kReadOnlySlab>(&nxt[(at + u) * T]);
                        }
                    };
                    const auto finish = [&](auto& v, auto& sc, auto& sn) {
                        group(strict_rule, v, sc, sn);
#pragma unroll
                        for (int u = 0; u < kU; ++u) held[(m + u) * T] = v[u];
                        m += kU;
                    };
                    fetch(m, v0, c0, n0);
                    for (;;) {
                        fetch(m + kU, v1, c1, n1);
                        finish(v0, c0, n0);
                        if (m > end) break;
                        fetch(m + kU, v0, c0, n0);
                        finish(v1, c1, n1);
                        if (m > end) break;
                    }
                }
                for (; m < to; ++m) {
                    double v[1] = {held[m * T]}, sc[1] = {load_slab<kReadOnlySlab>(&cur[m * T])},
                           sn[1] = {load_slab<kReadOnlySlab>(&nxt[m * T])};
                    group(strict_rule, v, sc, sn);
                    held[m * T] = v[0];
                }
            };
            const auto run = [&](auto strict_rule) {
                const uint32_t split = min(chip_rounds, rounds);
                pass(strict_rule, std::true_type{}, 0, split);
                pass(strict_rule, std::false_type{}, split, rounds);
            };
            if (strict) run(std::true_type{});
            else run(std::false_type{});
            if (highest >= kRuleLimitHigh) sm.beyond[(order + 1) & 1] = 1;
            continue;
        }
        // The lowest row, and rows whose spots or rule need the model itself.
        for (uint32_t m = 0; m < rounds; ++m) {
            double v = load_value(m);
            const double sc = load_slab<kReadOnlySlab>(&cur[m * T]);
            const double excess = sc - K;
            if (kind == kRuleRegression && excess > 0.0) {
                if (plain) {
                    if (exercise_rule(a.tie_rule, excess, rule_continuation<D>(sm.rule, excess))) v = excess;
                } else {
                    const int decision = within_rule(sc) && sm.rule.general == 0
                                             ? (exercise_rule(a.tie_rule, excess, rule_continuation<D>(sm.rule, excess))
                                                    ? kDecideExercise
                                                    : kDecideContinue)
                                             : decide_general<D>(&sm.model, sc, K, a.tie_rule);
                    if (decision == kDecideNonFinite) atomicMin(&st->fit_predict_fail, key(order, m));
                    else if (decision == kDecideExercise) v = excess;
                }
            }
            store_value(m, stage_next ? v * disc : v);
        }
        if (stage_next) {
            order += 1;
            sum_row(row - 1, true);
            order -= 1;
        }
    }
    // Common origin decision (policy.rs:265-281): mean of the values discounted to the origin.
    if (plan.origin_row) {
        double acc[2] = {0.0, 0.0};
        for (uint32_t m = 0; m < rounds; ++m) {
            const double w = load_value(m) * plan.origin_discount;
            if (!fo_isfinite(w)) atomicMin(&st->fit_payoff_fail, key(order, m));
            acc[0] += 1.0;
            acc[1] += w;
        }
        cta_reduce_dd<2>(acc, sm.red, sm.total);
        if (!team_exchange<2, kTeam>(team, sm.total)) return false;
        if (writer && threadIdx.x == 0) {
            const double mean = dd_round(dd_div(sm.total[1], sm.total[0]));
            const double intrinsic = plan.initial_spot - K > 0.0 ? plan.initial_spot - K : 0.0;
            FitRecord& rec = records[0];
            rec.kind = kRuleOrigin;
            rec.origin_exercise = exercise_rule(a.tie_rule, intrinsic, mean) ? 1 : 0;
            rec.origin_continuation = mean;
            rec.itm = 0;
            rec.diag_status = -1;
        }
    }
    return true;
}

// Rank / condition diagnostic of every regression row of problem pi (regression.rs:540-577), and every
// row's rule for the evaluation; the records were written by this CTA.
template <int D>
__device__ __noinline__ void diagnose_problem(const BatchArgs& a, uint32_t pi) {
    const BatchProblem pr = a.problems[pi];
    const uint32_t rows = a.groups[pr.group].plan.rows;
    for (uint32_t r = threadIdx.x; r + 1 < rows; r += blockDim.x) {
        FitRecord& rec = a.records[pr.records + r];
        ExerciseRule rule = rec.kind == kRuleRegression ? make_exercise_rule(rec.model, a.degree, pr.strike)
                                                        : never_exercise();
        if (rec.kind == kRuleNoSupport) rule.general = 1;
        a.rules[pr.records + r] = rule;
        if (rec.kind != kRuleRegression) continue;
        int rank = 0, aux = 0;
        double condition = 0.0;
        rec.diag_status =
            diagnose_design_d<D>(rec.model, a.rank_tolerance, a.condition_limit, &rank, &condition, &aux);
        rec.diag_rank = rank;
        rec.diag_condition = condition;
        rec.diag_aux = aux;
    }
}

// ---- evaluation -----------------------------------------------------------------------------------

// CTA sums of S (payoff, squared payoff) pairs as double-double totals: every pair is summed across
// its warp by the same two-value transpose whatever S is, then over the warps in a fixed order, so a
// strike's block totals do not depend on how many strikes an item evaluates together.
template <int S>
__device__ void cta_reduce_pairs(double (&acc)[2 * S], double* red /* [32 * 2S] */, dd* out /* [2S] */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < S; ++k) {
        double pair[2] = {acc[2 * k], acc[2 * k + 1]};
        const double total = warp_transpose_reduce<2>(pair);
        if (lane < 2) red[warp * 2 * S + 2 * k + lane] = total;
    }
    __syncthreads();
    combine_warps<2 * S>(red, [&](int slot, dd v) { out[slot] = v; });
    __syncthreads();
}

// A row's rule for one strike, as an evaluation item stages it: the rule's polynomial and the strike in the
// place of its flag (a flagged rule is staged as one that never exercises, its strike noted in by_record).
struct alignas(16) StrikeRule {
    double slope, shift;
    double c[kMaxColumns];
    double strike;
};
static_assert(sizeof(StrikeRule) == sizeof(ExerciseRule), "the rules' shared memory is counted in either");

// Shared memory of one evaluation item: S strikes evaluated together by every thread.
template <int S>
struct EvalSmem {
    double red[kPersistentThreads / 32 * 2 * S];
    dd tot[2 * S];
    unsigned cnt[2 * S];
    double strikes[S];
    uint32_t rbase[S];
    uint32_t pbase[S];
    uint32_t problem[S];
};

// Evaluation blocks [first, first + count) of group gi for strike chunk z: each thread re-simulates one
// evaluation path per block and applies up to S fitted policies on the fly (policy.rs:642-834); per
// (problem, block) double-double partials and stopping counts.
// kStaged: the rules were staged in shared memory, a row's S rules and strikes side by side; a row is
// decided for all S strikes without a branch, and those of them that need their records (an unsupported row,
// a rule beyond its range) one by one. Otherwise each strike reads its rule from global memory. Either way
// a strike's decisions are the same arithmetic, whatever strikes are priced beside it.
// Issue-bound, its warps too few to hide every latency: at 4,096 states x 8 strikes x 32,768 paths the
// phase took 186 ms with the basis recurrence and a branch per strike (1,240 warp instructions a
// path-step), 87 ms with staged rules (486), 72 ms with the strike in the rule, the payoff's sign for the
// strikes still running and the signs of differences for the comparisons (346), at two CTAs per SM (73.6 at
// three: their spills leave the little L1 beside 3 x 71 KB of shared memory). With one strike the chunk's
// steps are unrolled (34.3 -> 31.4 ms for 1,024 ragged contracts); with eight that is slower (78 ms).
template <int S, int D, bool kStaged, bool kReadOnly>
__device__ void evaluate_item(const BatchArgs& a, uint32_t gi, uint32_t first, uint32_t count, uint32_t z,
                              BatchNormals& normals, const PhiloxKeys& keys, EvalSmem<S>& sm, StrikeRule* staged,
                              uint32_t rule_rows) {
    const BatchGroup& g = a.groups[gi];
    const uint32_t p0 = g.first_problem + z * S;
    const int ns = min(S, int(g.problems) - int(z) * S);
    if (ns <= 0 || status_failed(&a.group_status[gi].train_sim_fail)) return;  // uniform over the CTA
    const DevicePlan plan = g.plan;  // a local copy: its fields stay in registers (no reloads across stores)
    const uint32_t rows = plan.rows;
    unsigned* by_record = reinterpret_cast<unsigned*>(staged + size_t(S) * rule_rows);  // [rows] strikes decided by their records
    if (threadIdx.x < S) {
        const bool live = int(threadIdx.x) < ns;
        const BatchProblem pr = a.problems[live ? p0 + threadIdx.x : p0];
        sm.strikes[threadIdx.x] = live ? pr.strike : 1.0;
        sm.rbase[threadIdx.x] = live ? pr.records : 0u;
        sm.pbase[threadIdx.x] = live ? pr.partial_base : 0u;
        sm.problem[threadIdx.x] = live ? p0 + threadIdx.x : p0;
    }
    if constexpr (kStaged)
        for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) by_record[r] = plan.disc_to_origin[r] < 0x1p100 ? 0u : ~0u;
    __syncthreads();
    if constexpr (kStaged) {
        for (uint32_t i = threadIdx.x; i < S * rows; i += blockDim.x) {
            const uint32_t k = i / rows, r = i % rows;
            ExerciseRule rule = never_exercise();
            if (int(k) < ns && r + 1 < rows) load_rule<kReadOnly>(&a.rules[sm.rbase[k] + r], &rule);
            if (rule.general) {
                atomicOr(&by_record[r], 1u << k);
                rule = never_exercise();
            }
            StrikeRule& to = staged[r * S + k];
            to.slope = rule.slope;
            to.shift = rule.shift;
#pragma unroll
            for (int i = 0; i < kMaxColumns; ++i) to.c[i] = rule.c[i];
            to.strike = sm.strikes[k];
        }
        __syncthreads();
    }
    const uint64_t P = plan.eval_paths;
    const uint32_t last = rows - 1;
    for (uint32_t b = first; b < first + count; ++b) {
        if (threadIdx.x < 2 * S) sm.cnt[threadIdx.x] = 0;
        __syncthreads();
        const uint64_t p = uint64_t(b) * kPersistentThreads + threadIdx.x;
        // A strike's payoff is -1 until its policy stops the path: its sign is what says that it still runs.
        double payoff[S];
#pragma unroll
        for (int k = 0; k < S; ++k) payoff[k] = -1.0;
        const auto running = [&](int k) { return __double2hiint(payoff[k]) < 0; };
        unsigned expired = 0;  // strikes whose policy reached expiry
        auto observe = [&](int row, double spot) {
            if (plan.escrowed) spot = plan.row_node[row] == 0 ? plan.initial_spot : spot + plan.escrow_cash[row];
            const double disc = plan.disc_to_origin[row];
            if (uint32_t(row) == last) {
#pragma unroll
                for (int k = 0; k < S; ++k) {
                    if (k >= ns || !running(k)) continue;
                    const double d = spot - sm.strikes[k];
                    payoff[k] = (d > 0.0 ? d : 0.0) * disc;
                    expired |= 1u << k;
                    if (!finite_nonnegative(payoff[k]))
                        atomicMin(&a.problem_status[sm.problem[k]].eval_terminal_fail, (unsigned long long)p);
                }
                return;
            }
            // The strikes of `apart` that still run, one by one: those without a staged rule, and every strike at a
            // state or a discount beyond what the rules cover.
            const auto decide_apart = [&](unsigned apart) {
#pragma unroll
                for (int k = 0; k < S; ++k) apart &= running(k) ? ~0u : ~(1u << k);
#pragma unroll 1
                for (int k = 0; k < ns; ++k) {
                    const double d = spot - sm.strikes[k];
                    if (!((apart >> k) & 1u) || !(d > 0.0)) continue;
                    int decision = kDecideContinue;
                    const volatile ExerciseRule& rule = a.rules[sm.rbase[k] + row];  // read through L2
                    if (!kStaged && rule.general == 0 && within_rule(spot) && disc < 0x1p100) {
                        if (exercise_rule(a.tie_rule, d, rule_continuation<D>(rule, d))) decision = kDecideExercise;
                    } else {
                        decision = decide_record<D>(a, sm.rbase[k] + row, spot, sm.strikes[k]);
                    }
                    ProblemStatus& st = a.problem_status[sm.problem[k]];
                    if (decision == kDecideNonFinite)
                        atomicMin(&st.eval_fail, ((unsigned long long)row << 33) | (p << 1));
                    if (decision != kDecideExercise) continue;
                    const double paid = d * disc;
                    if (!fo_isfinite(paid)) atomicMin(&st.eval_fail, ((unsigned long long)row << 33) | (p << 1) | 1ull);
#pragma unroll
                    for (int m = 0; m < S; ++m) payoff[m] = m == k ? fo_fabs(paid) : payoff[m];
                }
            };
            if (!kStaged || by_record[row] != 0 || !within_rule(spot)) {
                const unsigned apart = kStaged && within_rule(spot) ? by_record[row] : ~0u;
                decide_apart(apart);
                if (S == 1 || apart == ~0u) return;
            }
            // The others by the signs of K - spot, of the continuation less the excess and of the payoff so far: a
            // strike without a rule never exercises. (A difference of finite doubles is zero, and then
            // positive, only where they are equal.)
            const StrikeRule* rules = staged + row * S;
            const auto decide = [&](auto strict) {
#pragma unroll
                for (int k = 0; k < S; ++k) {
                    const StrikeRule rule = rules[k];
                    const double below = rule.strike - spot;
                    const double c = rule_continuation<D>(rule, -below);
                    const int kept = decltype(strict)::value ? __double2hiint(c + below) : ~__double2hiint(-below - c);
                    if ((__double2hiint(below) & kept & __double2hiint(payoff[k])) < 0) payoff[k] = -below * disc;
                }
            };
            if (a.tie_rule == 0) decide(std::true_type{});
            else decide(std::false_type{});
        };
        if (p < P) {
            const SimResult r =
                simulate_path<(S == 1)>(plan, normals, keys, plan.eval_domain, uint32_t(p), observe);
            if (r.code != 0) atomicMin(&a.group_status[gi].eval_sim_fail, (unsigned long long)p);
        }
        // Paths that stopped early and that reached expiry, per strike.
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const bool at_expiry = ((expired >> k) & 1u) != 0, stopped = !running(k);
            const unsigned late = __popc(__ballot_sync(0xffffffffu, at_expiry));
            const unsigned early = __popc(__ballot_sync(0xffffffffu, stopped && !at_expiry));
            if ((threadIdx.x & 31) == 0) {
                if (early) atomicAdd(&sm.cnt[2 * k], early);
                if (late) atomicAdd(&sm.cnt[2 * k + 1], late);
            }
            payoff[k] = stopped || at_expiry ? payoff[k] : 0.0;
        }
        double acc[2 * S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            acc[2 * k] = payoff[k];
            acc[2 * k + 1] = payoff[k] * payoff[k];
        }
        cta_reduce_pairs<S>(acc, sm.red, sm.tot);
        if (int(threadIdx.x) < 2 * ns) {
            const uint32_t k = threadIdx.x >> 1, which = threadIdx.x & 1u;
            a.eval_partials[(size_t(sm.pbase[k]) + b) * 2 + which] = make_double2(sm.tot[threadIdx.x].hi,
                                                                                  sm.tot[threadIdx.x].lo);
            if (sm.cnt[threadIdx.x]) atomicAdd(&a.counts[size_t(sm.problem[k]) * 2 + which], sm.cnt[threadIdx.x]);
        }
    }
}

struct GreeksEvalSmem {
    double red[32 * 2];
    dd tot[2];
    double gred[32 * kGreekSlots];
    dd gtot[kGreekSlots];
    unsigned cnt[2];
};

// The adjoint variant: evaluation blocks [first, first + count) of group gi for its strike k alone,
// with the pathwise Greeks (lsm_adjoint.cuh) summed per block in double-double.
template <int D, bool kReadOnly>
__device__ void evaluate_greeks_item(const BatchArgs& a, uint32_t gi, uint32_t first, uint32_t count, uint32_t k,
                                     BatchNormals& normals, const PhiloxKeys& keys, GreeksEvalSmem& sm, ExerciseRule* rules, unsigned* stops) {
    const BatchGroup& g = a.groups[gi];
    if (k >= g.problems || status_failed(&a.group_status[gi].train_sim_fail)) return;  // uniform over the CTA
    const uint32_t problem = g.first_problem + k;
    const BatchProblem pr = a.problems[problem];
    const DevicePlan plan = g.plan;  // a local copy: its fields stay in registers (no reloads across stores)
    const uint32_t rows = plan.rows;
    for (uint32_t r = threadIdx.x; r + 1 < rows; r += blockDim.x) load_rule<kReadOnly>(&a.rules[pr.records + r], &rules[r]);
    const double K = pr.strike;
    const uint64_t P = plan.eval_paths;
    const uint32_t last = rows - 1;
    const double sens_scale = 1.0 / g.sigma;  // (Z diffusion - diffusion^2) / sigma = Z sqrt(dt) - sigma dt
    for (uint32_t b = first; b < first + count; ++b) {
        for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) stops[r] = 0;
        if (threadIdx.x < 2) sm.cnt[threadIdx.x] = 0;
        __syncthreads();
        const uint64_t p = uint64_t(b) * kPersistentThreads + threadIdx.x;
        double payoff = 0.0, held = 0.0;  // the payoff and the state it was taken at
        uint32_t stop_row = 0;
        bool active = p < P;
        PathAdjoint adj;
        adj.reset();
        auto observe = [&](int row, double spot) {
            if (!active) return;
            const double disc = plan.disc_to_origin[row];
            if (uint32_t(row) == last) {
                const double d = spot - K;
                payoff = (d > 0.0 ? d : 0.0) * disc;
                if (!fo_isfinite(payoff)) atomicMin(&a.problem_status[problem].eval_terminal_fail, (unsigned long long)p);
                held = spot;
                stop_row = last;
                active = false;
                return;
            }
            const ExerciseRule& rule = rules[row];
            const double excess = spot - K;
            if (!(excess > 0.0)) return;
            bool exercised;
            if (rule.general == 0 && within_rule(spot)) {
                exercised = exercise_rule(a.tie_rule, excess, rule_continuation<D>(rule, excess));
            } else {
                const int decision = decide_record<D>(a, pr.records + row, spot, K);
                if (decision == kDecideNonFinite)
                    atomicMin(&a.problem_status[problem].eval_fail, ((unsigned long long)row << 33) | (p << 1));
                exercised = decision == kDecideExercise;
            }
            if (exercised) {
                payoff = excess * disc;
                if (!fo_isfinite(payoff))
                    atomicMin(&a.problem_status[problem].eval_fail, ((unsigned long long)row << 33) | (p << 1) | 1ull);
                held = spot;
                stop_row = uint32_t(row);
                active = false;
            }
        };
        if (p < P) {
            const auto step = [&](uint32_t, const StepCoef& c, double z, double growth) {
                if (active) adj.step(growth, z * c.diffusion - c.diffusion * c.diffusion);
            };
            const auto cash = [&](uint32_t at, double before, double amount) {
                if (active) adj.cash(at, before, amount);
            };
            const SimResult r =
                simulate_path<false>(plan, normals, keys, plan.eval_domain, uint32_t(p), observe, step, cash);
            if (r.code != 0) atomicMin(&a.group_status[gi].eval_sim_fail, (unsigned long long)p);
        }
        // The backward recurrence after the path, where its sums are not live through the path's loop.
        GreekSums gs;
        gs.reset();
        if (p < P && !active) {
            const bool expired = stop_row == last;
            atomicAdd(&sm.cnt[expired ? 1 : 0], 1u);
            if (!expired) atomicAdd(&stops[stop_row], 1u);
            adj.stop(gs, plan.row_node[stop_row], held, payoff, plan.disc_to_origin[stop_row], expired, plan.policy,
                     sens_scale);
        }
        double acc[2] = {payoff, payoff * payoff};
        cta_reduce_pairs<1>(acc, sm.red, sm.tot);
        if (threadIdx.x < 2) {
            a.eval_partials[(size_t(pr.partial_base) + b) * 2 + threadIdx.x] =
                make_double2(sm.tot[threadIdx.x].hi, sm.tot[threadIdx.x].lo);
            if (sm.cnt[threadIdx.x]) atomicAdd(&a.counts[size_t(problem) * 2 + threadIdx.x], sm.cnt[threadIdx.x]);
        }
        for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x)
            if (stops[r]) atomicAdd(&a.stop_counts[pr.records + r], stops[r]);
        double gacc[kGreekSlots];
        gs.to_slots(gacc);
        cta_reduce_dd<kGreekSlots>(gacc, sm.gred, sm.gtot);
        if (threadIdx.x < kGreekSlots)
            a.greek_partials[(size_t(pr.partial_base) + b) * kGreekSlots + threadIdx.x] =
                make_double2(sm.gtot[threadIdx.x].hi, sm.gtot[threadIdx.x].lo);
    }
}

// ---- per-problem summary ----------------------------------------------------------------------------

// The summary of problem i (its twelve result columns, try_from_parts pricing.rs:1130-1230, and its
// first failing backward row), written by one warp once its group's evaluation is complete: lanes
// 0 / 1 sum the price partials over the blocks in block order, with the Greeks lane s sums Greek
// slot s the same way, and lane 0 scans the records.
__device__ void summarize_problem(const BatchArgs& a, uint32_t i, int lane) {
    const BatchProblem pr = a.problems[i];
    const BatchGroup& g = a.groups[pr.group];
    const uint64_t n = g.plan.eval_paths;
    const uint32_t blocks = blocks_of(n);
    const double2* part = a.eval_partials + size_t(pr.partial_base) * 2;
    // Price partial sums: lane 0 the payoffs, lane 1 their squares, each in block order.
    dd slot_sum = dd_make(0.0);
    if (lane < 2)
        for (uint32_t b = 0; b < blocks; ++b) {
            const double2 v = __ldcg(&part[2 * b + lane]);
            slot_sum = dd_add(slot_sum, dd{v.x, v.y});
        }
    dd sum, sumsq;
    sum.hi = __shfl_sync(0xffffffffu, slot_sum.hi, 0);
    sum.lo = __shfl_sync(0xffffffffu, slot_sum.lo, 0);
    sumsq.hi = __shfl_sync(0xffffffffu, slot_sum.hi, 1);
    sumsq.lo = __shfl_sync(0xffffffffu, slot_sum.lo, 1);
    if (a.greek_partials && lane < kGreekSlots) {
        const double2* gp = a.greek_partials + size_t(pr.partial_base) * kGreekSlots;
        dd acc = dd_make(0.0);
        for (uint32_t b = 0; b < blocks; ++b) {
            const double2 v = __ldcg(&gp[size_t(b) * kGreekSlots + lane]);
            acc = dd_add(acc, dd{v.x, v.y});
        }
        a.greek_sums[size_t(i) * kGreekSlots + lane] = dd_round(acc);
    }
    if (lane != 0) return;
    const uint32_t rows = g.plan.rows;
    const uint32_t E = rows - 1;
    const uint32_t lowest = g.plan.origin_row ? 1u : 0u;
    const FitRecord* rec = a.records + pr.records;
    ProblemStatus st;
    st.fit_payoff_fail = ld_l2_u64(&a.problem_status[i].fit_payoff_fail);
    st.fit_predict_fail = ld_l2_u64(&a.problem_status[i].fit_predict_fail);
    st.fit_nonfinite = ld_l2_u64(&a.problem_status[i].fit_nonfinite);
    st.eval_fail = ld_l2_u64(&a.problem_status[i].eval_fail);
    st.eval_terminal_fail = ld_l2_u64(&a.problem_status[i].eval_terminal_fail);
    ProblemSummary s{};
    // First failure of the backward pass in the reference's order: the discount into the row,
    // then its population, regression, diagnostic and update (policy.rs:215-296).
    s.fit_fail_order = 0xffffffffu;
    s.fit_fail_kind = kFitFailNone;
    if (!pr.skip_fit) {
        const uint32_t fitted = E > lowest ? E - lowest : 0u;
        for (uint32_t order = 0; order <= fitted; ++order) {
            const unsigned long long lo = (unsigned long long)order << 32, hi = lo | 0xffffffffull;
            int kind = kFitFailNone;
            if (st.fit_payoff_fail >= lo && st.fit_payoff_fail <= hi) {
                kind = kFitFailPayoff;
            } else if (order < fitted) {
                const FitRecord& r = rec[E - 1 - order];
                const int rkind = __ldcg(&r.kind);
                if (st.fit_nonfinite >= lo && st.fit_nonfinite <= hi) kind = kFitFailNonFinite;
                else if (rkind == kRuleFitFailed) kind = kFitFailFit;
                else if (rkind == kRuleRegression && __ldcg(&r.diag_status) != kDiagOk) kind = kFitFailDiagnostic;
                else if (st.fit_predict_fail >= lo && st.fit_predict_fail <= hi) kind = kFitFailPredict;
            }
            if (kind != kFitFailNone) {
                s.fit_fail_order = order;
                s.fit_fail_kind = kind;
                break;
            }
        }
    }
    uint32_t min_itm = 0xffffffffu;
    double max_condition = 0.0;
    s.nosupport_row = 0xffffffffu;
    for (uint32_t r = 0; r < E; ++r) {
        const int kind = __ldcg(&rec[r].kind);
        switch (kind) {
            case kRuleOrigin:
                s.origin_fitted = 1;
                s.origin_exercised = uint32_t(__ldcg(&rec[r].origin_exercise));
                break;
            case kRuleNoSupport: {
                s.no_support_nodes += 1;
                const unsigned itm = __ldcg(&a.itm_counts[pr.records + r]);
                if (s.nosupport_row == 0xffffffffu && itm > 0) {
                    s.nosupport_row = r;
                    s.nosupport_count = itm;
                }
                break;
            }
            case kRuleContinue: s.insufficient_nodes += 1; break;
            case kRuleRegression: {
                s.regression_nodes += 1;
                const uint32_t itm = uint32_t(__ldcg(reinterpret_cast<const unsigned long long*>(&rec[r].itm)));
                min_itm = itm < min_itm ? itm : min_itm;
                max_condition = fmax(max_condition, __ldcg(&rec[r].diag_condition));
                break;
            }
            default: break;
        }
    }
    s.minimum_itm = s.regression_nodes == 0 ? 0u : min_itm;
    s.maximum_condition = max_condition;
    if (s.origin_exercised) {
        // LsmEvaluation::deterministic (policy.rs:657-669): every path stops at the origin.
        const double d = g.plan.initial_spot - pr.strike;
        s.price = d > 0.0 ? d : 0.0;
        s.sample_standard_deviation = 0.0;
        s.standard_error = 0.0;
        s.early_paths = uint32_t(n);
        s.expiry_paths = 0;
    } else {
        const dd mean = dd_div(sum, dd_make(double(n)));
        dd m2 = dd_sub(sumsq, dd_mul(sum, mean));
        if (m2.hi < 0.0) m2 = dd_make(0.0);
        s.price = dd_round(mean);
        const double sd = n > 1 ? dd_round(dd_sqrt(dd_div(m2, dd_make(double(n - 1))))) : 0.0;
        s.sample_standard_deviation = sd;
        s.standard_error = n > 1 ? sd / sqrt(double(n)) : 0.0;
        s.early_paths = __ldcg(&a.counts[size_t(i) * 2]);
        s.expiry_paths = __ldcg(&a.counts[size_t(i) * 2 + 1]);
    }
    a.summaries[i] = s;
}

}  // namespace

// ---- the persistent kernel ------------------------------------------------------------------------

// Executors of the work items. kPhaseAll is the persistent launch: one kernel drains the whole queue,
// items of every kind waiting on the counters. The other phases run the items of one kind as a
// queue-draining kernel of their own, launched in stream order (simulation, fits, evaluation), so
// that each kind gets the register budget and CTAs per SM that suit it; their dependency waits are
// then already met. Both run the same item functions, so they give the same results, bit for bit.
enum BatchPhase : int { kPhaseAll = 0, kPhaseSimulate = 1, kPhaseFit = 2, kPhaseEvaluate = 3 };

// Shared memory of the items a kernel runs: all kinds for the persistent launch, one kind each for
// the phase kernels (less static shared memory leaves more of the SM's L1).
template <int S>
union AllItemsSmem {
    BackwardItemSmem bwd;
    EvalSmem<S> eval;
    GreeksEvalSmem greeks;
};
struct NoItemSmem {};
struct FitItemSmem {
    BackwardItemSmem bwd;
};
template <int S>
struct EvalItemSmem {
    EvalSmem<S> eval;
};
struct GreeksItemSmem {
    GreeksEvalSmem greeks;
};
template <int kPhase, int S, bool kGreeks>
struct PhaseSmem {
    using type = AllItemsSmem<S>;
};
template <int S, bool kGreeks>
struct PhaseSmem<1, S, kGreeks> {
    using type = NoItemSmem;
};
template <int S, bool kGreeks>
struct PhaseSmem<2, S, kGreeks> {
    using type = FitItemSmem;
};
template <int S>
struct PhaseSmem<3, S, false> {
    using type = EvalItemSmem<S>;
};
template <int S>
struct PhaseSmem<3, S, true> {
    using type = GreeksItemSmem;
};

constexpr int kFitCtasPerSm = 2;

template <int kPhase, int S, bool kGreeks>
struct PhaseOccupancy {
    // Resident CTAs per SM the register budget is cut for. The adjoint's at four took 58.1 ms for 1,024
    // ragged contracts, its state spilled; at three 48.7, at two 52.3. The one-strike evaluation spills 424
    // bytes at its four.
    static constexpr int value = kPhase == kPhaseSimulate               ? 4
                                 : kPhase == kPhaseFit                  ? kFitCtasPerSm
                                 : kPhase == kPhaseEvaluate && kGreeks  ? 3
                                 : kPhase == kPhaseEvaluate             ? (S == 1 ? 4 : 2)
                                                                        : 3;
};

__device__ __forceinline__ uint32_t dynamic_smem_bytes() {
    uint32_t bytes;
    asm("mov.u32 %0, %dynamic_smem_size;" : "=r"(bytes));
    return bytes;
}

// S: strikes an evaluation item applies together (kGreeks: one, with the adjoint). The dynamic
// shared memory holds the staged rules (rule_rows x S ExerciseRules, plus one word per row: the strikes
// that need their records, or its stopping count with the Greeks) when stage_rules is set; the fit kernel's
// holds path values. kUnstaged: the evaluation kernel of the phase executor for launches that do not stage
// (the staged form's steps keep the registers that this one's would take).
template <int kPhase, int S, bool kGreeks, int D, bool kUnstaged>
__global__ void __launch_bounds__(kPersistentThreads, (PhaseOccupancy<kPhase, S, kGreeks>::value))
    batch_persistent_kernel(BatchArgs a, BatchQueue q, uint32_t rule_rows, int stage_rules) {
    constexpr bool kSim = kPhase == kPhaseAll || kPhase == kPhaseSimulate;
    constexpr bool kFit = kPhase == kPhaseAll || kPhase == kPhaseFit;
    constexpr bool kEval = kPhase == kPhaseAll || kPhase == kPhaseEvaluate;
    __shared__ std::conditional_t<kSim || kEval, BatchNormals, NoItemSmem> normals;
    __shared__ PhiloxKeys keys[2];  // of the training and the evaluation seed (one of each per request)
    __shared__ BatchItem item;
    __shared__ int flag;
    __shared__ typename PhaseSmem<kPhase, S, kGreeks>::type sm;
    extern __shared__ __align__(16) unsigned char persistent_dyn[];
    ExerciseRule* staged = reinterpret_cast<ExerciseRule*>(persistent_dyn);
    if constexpr (kSim || kEval) {
        if (threadIdx.x == 0) {
            keys[0] = philox_keys(a.groups[0].plan.train_seed);
            keys[1] = philox_keys(a.groups[0].plan.eval_seed);
        }
        load_normal_tables(normals);
    }
    for (;;) {
        __syncthreads();  // the previous item is done with the shared memory
        if (threadIdx.x == 0) {
            const unsigned i = atomicAdd(q.next, 1u);
            if (i < q.n_items) {
                item = q.items[i];
            } else {
                item.kind = kItemNone;
            }
        }
        __syncthreads();
        const BatchItem it = item;
        if (it.kind == kItemNone) return;
        if (it.kind == kItemSimulate) {
            if constexpr (kSim) {
                simulate_item(a, it.index, it.first, it.count, normals, keys[0]);
                signal_done(&q.sim_done[it.index], it.count);
            }
        } else if (it.kind == kItemBackward) {
            if constexpr (kFit) {
                const uint32_t gi = a.problems[it.index].group;
                const uint32_t sim_blocks = blocks_of(a.groups[gi].plan.train_paths);
                // The fit kernel runs after the simulation kernel: its dependencies are met.
                if (kPhase == kPhaseFit || wait_for(&q.sim_done[gi], sim_blocks, q.timeout, &flag)) {
                    // Lone CTAs run a copy of the fit without the team exchanges (fewer live registers).
                    constexpr bool kOwn = kPhase == kPhaseFit;
                    constexpr int kU = kOwn ? kFitKernelLoads : kPersistentLoads;
                    double* const chip = reinterpret_cast<double*>(persistent_dyn);
                    const uint32_t chip_rounds =
                        kOwn ? dynamic_smem_bytes() / (kPersistentThreads * uint32_t(sizeof(double))) : 0u;
                    const bool done =
                        it.count == 1 ? backward_item<D, kOwn, false, kU>(a, it.index, 0, 1, q.timeout, &flag, sm.bwd,
                                                                          chip, chip_rounds)
                                      : backward_item<D, kOwn, true, kU>(a, it.index, it.first, it.count, q.timeout,
                                                                         &flag, sm.bwd, chip, chip_rounds);
                    __syncthreads();
                    // Member 0 wrote the records; after the fit kernel a kernel of its own diagnoses them.
                    if (!kOwn && done && it.first == 0) diagnose_problem<D>(a, it.index);
                }
                signal_done(&q.bwd_done[gi], 1u);
            }
        } else if constexpr (kEval) {
            const uint32_t gi = it.index;
            const BatchGroup& g = a.groups[gi];
            if (kPhase == kPhaseEvaluate || wait_for(&q.bwd_done[gi], g.fit_items, q.timeout, &flag)) {
                if constexpr (kGreeks) {
                    unsigned* stops = reinterpret_cast<unsigned*>(staged + rule_rows);
                    evaluate_greeks_item<D, kPhase == kPhaseEvaluate>(a, gi, it.first, it.count, it.chunk, normals, keys[1],
                                                                      sm.greeks, staged, stops);
                } else {
                    constexpr bool kRO = kPhase == kPhaseEvaluate;
                    StrikeRule* rules = reinterpret_cast<StrikeRule*>(persistent_dyn);
                    constexpr bool kBoth = kPhase == kPhaseAll;
                    if constexpr (kBoth || !kUnstaged)
                        if (!kBoth || stage_rules)
                            evaluate_item<S, D, true, kRO>(a, gi, it.first, it.count, it.chunk, normals, keys[1], sm.eval,
                                                           rules, rule_rows);
                    if constexpr (kBoth || kUnstaged)
                        if (!kBoth || !stage_rules)
                            evaluate_item<S, D, false, kRO>(a, gi, it.first, it.count, it.chunk, normals, keys[1], sm.eval,
                                                            rules, rule_rows);
                }
            }
            // The item that completes the group's evaluation writes the group's summaries (in the
            // phase executor a summary kernel follows the evaluation kernel instead).
            if constexpr (kPhase == kPhaseEvaluate) continue;
            const uint32_t chunks = kGreeks ? g.problems : (g.problems + S - 1) / S;
            const unsigned units = blocks_of(g.plan.eval_paths) * chunks;
            const unsigned before = signal_done(&q.eval_done[gi], it.count);
            if (threadIdx.x == 0) flag = before + it.count == units;
            __syncthreads();
            if (flag) {
                __threadfence();
                const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
                for (uint32_t k = warp; k < g.problems; k += blockDim.x >> 5)
                    summarize_problem(a, g.first_problem + k, lane);
            }
        }
    }
}

// ---- launcher ---------------------------------------------------------------------------------------

template <int kPhase, int S, bool kGreeks, int D, bool kUnstaged = false>
static cudaError_t prepare_persistent_d(const BatchQueue& q, uint32_t rule_rows, bool stage, int ctas_per_sm,
                                        PersistentLaunch* out) {
    if constexpr (kPhase == kPhaseEvaluate && !kGreeks && !kUnstaged)
        if (!stage) return prepare_persistent_d<kPhase, S, kGreeks, D, true>(q, rule_rows, stage, ctas_per_sm, out);
    auto kernel = batch_persistent_kernel<kPhase, S, kGreeks, D, kUnstaged>;
    const bool rules = stage && (kPhase == kPhaseAll || kPhase == kPhaseEvaluate);
    size_t smem = rules ? persistent_rule_bytes(S, kGreeks, rule_rows) : 0;
    if (kPhase == kPhaseFit) {
        // What its resident CTAs leave of the SM's shared memory, in whole rounds of path values.
        cudaFuncAttributes attr{};
        cudaError_t fe = cudaFuncGetAttributes(&attr, kernel);
        if (fe != cudaSuccess) return fe;
        constexpr size_t kSmBytes = 228 * 1024, kReservedPerCta = 1024, kRound = kPersistentThreads * sizeof(double);
        smem = (kSmBytes / kFitCtasPerSm - kReservedPerCta - attr.sharedSizeBytes) / kRound * kRound;
    }
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPersistentThreads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    int device = 0, sms = 0;
    e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    const int cap = kPhase == kPhaseAll && ctas_per_sm > 0 && ctas_per_sm < per_sm ? ctas_per_sm : per_sm;
    const int resident = cap * sms;
    out->kernel = reinterpret_cast<const void*>(kernel);
    out->grid = int(q.n_items) < resident ? int(q.n_items) : resident;
    out->smem = smem;
    out->threads = kPersistentThreads;
    return cudaSuccess;
}

// The phase executor's kernel between the fits and the evaluation: every problem's rules and diagnostics, a
// CTA per problem. In the fit kernel their registers slowed every pass (over 390 ms against 176 at 4,096
// states x 8 strikes).
constexpr int kDiagnoseThreads = 64;
template <int D>
__global__ void __launch_bounds__(kDiagnoseThreads) batch_diagnose_kernel(BatchArgs a, BatchQueue, uint32_t, int) {
    if (blockIdx.x < a.n_problems) diagnose_problem<D>(a, blockIdx.x);
}

// The kernel instances of one degree: the persistent launch (phase kPhaseAll) or one phase's kernel.
// Each degree is compiled in a translation unit of its own (lsm_batch_d0.cu .. lsm_batch_d4.cu).
template <int D>
cudaError_t prepare_batch_degree(int phase, bool greeks, int strikes, const BatchQueue& q, uint32_t rule_rows,
                                 bool stage, int ctas_per_sm, PersistentLaunch* out);

template <int D>
const void* batch_diagnose_entry();

#ifdef FO_BATCH_DEGREE
template <>
const void* batch_diagnose_entry<FO_BATCH_DEGREE>() {
    return reinterpret_cast<const void*>(batch_diagnose_kernel<FO_BATCH_DEGREE>);
}

template <int kPhase, int D>
static cudaError_t prepare_phase_degree(bool greeks, int strikes, const BatchQueue& q, uint32_t rule_rows, bool stage,
                                        int ctas_per_sm, PersistentLaunch* out) {
    if constexpr (kPhase == kPhaseSimulate || kPhase == kPhaseFit) {
        // No evaluation code: one instance serves every evaluation width.
        return prepare_persistent_d<kPhase, 1, false, D>(q, rule_rows, stage, ctas_per_sm, out);
    } else {
        if (greeks) return prepare_persistent_d<kPhase, 1, true, D>(q, rule_rows, stage, ctas_per_sm, out);
        switch (strikes) {
            case 1: return prepare_persistent_d<kPhase, 1, false, D>(q, rule_rows, stage, ctas_per_sm, out);
            case 2: return prepare_persistent_d<kPhase, 2, false, D>(q, rule_rows, stage, ctas_per_sm, out);
            case 4: return prepare_persistent_d<kPhase, 4, false, D>(q, rule_rows, stage, ctas_per_sm, out);
            default: return prepare_persistent_d<kPhase, kEvalStrikes, false, D>(q, rule_rows, stage, ctas_per_sm, out);
        }
    }
}

template <>
cudaError_t prepare_batch_degree<FO_BATCH_DEGREE>(int phase, bool greeks, int strikes, const BatchQueue& q,
                                                  uint32_t rule_rows, bool stage, int ctas_per_sm,
                                                  PersistentLaunch* out) {
    constexpr int D = FO_BATCH_DEGREE;
    switch (phase) {
        case kPhaseSimulate:
            return prepare_phase_degree<kPhaseSimulate, D>(greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        case kPhaseFit: return prepare_phase_degree<kPhaseFit, D>(greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        case kPhaseEvaluate:
            return prepare_phase_degree<kPhaseEvaluate, D>(greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
        default: return prepare_phase_degree<kPhaseAll, D>(greeks, strikes, q, rule_rows, stage, ctas_per_sm, out);
    }
}
#endif  // FO_BATCH_DEGREE

}  // namespace fo
