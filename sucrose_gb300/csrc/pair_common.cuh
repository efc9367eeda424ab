// Pair-parallel driver shared by every pair-potential kernel.
//
// The half list is flattened into (pair_i, pair_j) with rows in particle
// order, so the pairs of one particle i are contiguous. Each warp takes 32
// consecutive pairs; each lane evaluates one pair in the reference's
// orientation (I = pair_i < J = pair_j), then
//   * the J-side force and torque go out as one float4 atomic each,
//   * the I-side terms are summed across lanes with a segmented shuffle scan
//     (segments = runs of equal i), and the last lane of each run issues one
//     float4 atomic,
//   * PE and the pair virial r_ij . F_ij are summed per thread and per warp
//     in double-float (FP32 two-sums), then per block in FP64, and added up in
//     a fixed order by the last block or, in a captured step, by the final
//     half step (pair_sums_finish), so the
//     totals do not depend on which pairs a thread happened to evaluate.
// The grid is persistent (a multiple of the SM count); the pair count is read
// from device memory so the launch needs no host synchronisation.
#pragma once
#include <type_traits>

#include "sg_internal.cuh"

// An optional trait of a potential, with its default:
//   kExactFilter (true): in_range decides exactly as eval would. When false,
//     in_range is a superset test and eval makes the decision (and counts it).
template <class P, class = void>
struct ExactFilter : std::true_type {};
template <class P>
struct ExactFilter<P, std::void_t<decltype(P::kExactFilter)>> : std::integral_constant<bool, P::kExactFilter> {};

struct PairOut {
    float3 f;    // force on I (FXIJ)
    float3 ti;   // torque on I (TXI)
    float3 tj;   // torque on J (TXJ)
    float pe;
    float vir;
    int act;     // the pair was inside the potential's range (counted for LJ / GB)
};

struct PairLaunch {
    const int* __restrict__ pair_i;
    const int* __restrict__ pair_j;
    const int* npairs;           // device: end of the (row-order) range
    const int* begin;            // device: start of the range, or nullptr for 0
    // Replica contexts keep each replica's pairs in a section of their own:
    // the pair at row-order index v of replica r sits at
    // sec[r] + v - row_off[rep_off[r]]. sec == nullptr: storage is row order.
    const int* row_off;
    const int* rep_off;
    const long long* sec;
    const int* chunk_rep;        // replica holding pair index 32 c, for every chunk c
    int nrep;
    float4* force;
    float4* torque;
    double* partials;
    unsigned int* done;
    double* acc;                 // per-call sums: acc[0] += PE, acc[1] += virial
    double* acc_total;           // running sums since the last zero_forces
    // solver statistics (ECP) or listed / in-range counts (LJ, GB); nullptr: not
    // counted (a fused step, whose counts nothing reads)
    unsigned long long* stats;
};

// Storage index and particles of lane `lane`'s pair in the 32-pair chunk that
// starts at row-order index `base`; pairs outside [b0, np) are invalid.
SG_DEV void pair_fetch(const PairLaunch& L, int base, int lane, int np, int b0, int& t, int& i, int& j,
                       bool& valid) {
    const int v = base + lane;
    valid = v < np && v >= b0;
    t = v;
    i = -1;
    j = 0;
    if (valid) {
        if (L.sec) {
            int r = L.chunk_rep[base >> 5];
            while (r + 1 < L.nrep && L.row_off[L.rep_off[r + 1]] <= v) ++r;
            t = (int)(L.sec[r] + (long long)(v - L.row_off[L.rep_off[r]]));
        }
        i = L.pair_i[t];
        j = L.pair_j[t];
    }
}

// Where a warp is in the list: chunks of at most 64 pairs of one replica (a
// single system is one).
struct PairWalk {
    int base, stop, rend, r;   // stop: end of the warp's span; rend: of the replica's pairs
    long long shift;           // storage index - list position
    SG_DEV int end() const { return min(base + 64, min(stop, rend)); }
    SG_DEV void enter(const PairLaunch& L) {   // the replica that holds base
        while (r + 1 < L.nrep && L.row_off[L.rep_off[r + 1]] <= base) ++r;
        const int o = L.row_off[L.rep_off[r]];
        rend = L.row_off[L.rep_off[r + 1]];
        shift = L.sec[r] - o;
    }
    SG_DEV void next(const PairLaunch& L) {
        base = end();
        if (base >= rend && base < stop) enter(L);
    }
};

struct PairChunk {   // two listed pairs per lane
    int i0, j0, i1, j1, n, r;
    SG_DEV void load(const PairLaunch& L, const PairWalk& w, int lane) {
        n = w.end() - w.base;
        r = w.r;
        const long long t = w.base + w.shift + lane;
        i0 = lane < n ? L.pair_i[t] : 0;
        j0 = lane < n ? L.pair_j[t] : 0;
        i1 = lane + 32 < n ? L.pair_i[t + 32] : 0;
        j1 = lane + 32 < n ? L.pair_j[t + 32] : 0;
    }
};

SG_DEV void atomic_add_f3(float4* p, float3 v) {
    atomicAdd(p, make_float4(v.x, v.y, v.z, 0.f));
}

template <bool TORQUE>
SG_DEV void segmented_scatter_i(const PairLaunch& L, int i, float3 f, float3 t) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int io = __shfl_up_sync(0xffffffffu, i, o);
        float fx = __shfl_up_sync(0xffffffffu, f.x, o);
        float fy = __shfl_up_sync(0xffffffffu, f.y, o);
        float fz = __shfl_up_sync(0xffffffffu, f.z, o);
        float tx = 0.f, ty = 0.f, tz = 0.f;
        if (TORQUE) {
            tx = __shfl_up_sync(0xffffffffu, t.x, o);
            ty = __shfl_up_sync(0xffffffffu, t.y, o);
            tz = __shfl_up_sync(0xffffffffu, t.z, o);
        }
        if (lane >= o && io == i) {
            f.x += fx; f.y += fy; f.z += fz;
            if (TORQUE) { t.x += tx; t.y += ty; t.z += tz; }
        }
    }
    int inext = __shfl_down_sync(0xffffffffu, i, 1);
    bool last = (lane == 31) || (inext != i);
    // a run of pairs that all lay out of range sums to exact zeros: no atomic
    const bool zero = f.x == 0.f && f.y == 0.f && f.z == 0.f && (!TORQUE || (t.x == 0.f && t.y == 0.f && t.z == 0.f));
    if (last && i >= 0 && !zero) {
        atomic_add_f3(&L.force[i], f);
        if (TORQUE) atomic_add_f3(&L.torque[i], t);
    }
}

#define SG_NSTATS 32
#define SG_PAIR_MAX_BLOCK 256

// Per-thread double-float sums of the pair energy and virial.
struct EnergySums {
    float pe = 0.f, pe_lo = 0.f, vir = 0.f, vir_lo = 0.f;
    SG_DEV void add(float p, float v) {
        float s = pe + p, bb = s - pe;
        pe_lo += (pe - (s - bb)) + (p - bb);
        pe = s;
        s = vir + v;
        bb = s - vir;
        vir_lo += (vir - (s - bb)) + (v - bb);
        vir = s;
    }
};

// One pair per lane, evaluated and scattered (all 32 lanes call it).
// i, j: the pair's particles (loaded by the caller; ignored when !valid).
// COUNT: listed and in-range pairs are counted here.
template <class Pot, bool COUNT>
SG_DEV void pair_process(const PairLaunch& L, const Pot& pot, int t, int i, int j, bool valid, EnergySums& es,
                         unsigned long long* sh_stats) {
    const int lane = threadIdx.x & 31;
    PairOut o;
    o.f = make_float3(0.f, 0.f, 0.f);
    o.ti = o.f;
    o.tj = o.f;
    o.pe = 0.f;
    o.vir = 0.f;
    o.act = 0;
    if (!valid) {
        i = -1;
        j = 0;
    }
    // called by every lane (warp-cooperative potentials need all 32)
    pot.eval(valid, valid ? i : 0, j, t, o, sh_stats);
    if (COUNT) {
        // stats[0] listed pairs, stats[1] pairs inside the range
        const unsigned va = __ballot_sync(0xffffffffu, valid), ac = __ballot_sync(0xffffffffu, o.act != 0);
        if (lane == 0) {
            atomicAdd(&sh_stats[0], (unsigned long long)__popc(va));
            if (ac) atomicAdd(&sh_stats[1], (unsigned long long)__popc(ac));
        }
    }
    if (valid && (!Pot::kCountActive || o.act)) {   // out-of-range pairs add nothing
        atomic_add_f3(&L.force[j], make_float3(-o.f.x, -o.f.y, -o.f.z));
        if (Pot::kTorque) atomic_add_f3(&L.torque[j], o.tj);
    }
    es.add(o.pe, o.vir);
    segmented_scatter_i<Pot::kTorque>(L, i, o.f, o.ti);
}

// Per-warp queue of in-range pairs for the filtered kernels: a cheap range
// test runs on every listed pair first; the pairs in range queue up (in list
// order, so rows stay contiguous) and are evaluated 32 at a time, so no lane
// idles on an out-of-range pair. Slots: storage index, i, j; 64 a warp.
template <class Pot>
struct PairQueues {
    static_assert(!Pot::kCountActive || ExactFilter<Pot>::value, "in_range counts for eval");
    static constexpr int kWords = 64 * 3;   // shared words per warp
    int* q;   // this warp's queue: t at +0, i at +64, j at +128
    int qn;
    int lane;

    SG_DEV void init(int* warp_words) {
        q = warp_words;
        qn = 0;
        lane = threadIdx.x & 31;
    }
    // append this lane's pair when keep (list order kept)
    SG_DEV void push(bool keep, int t, int i, int j) {
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int slot = qn + __popc(km & ((1u << lane) - 1u));
            q[slot] = t;
            q[64 + slot] = i;
            q[128 + slot] = j;
        }
        qn += __popc(km);
        __syncwarp();
    }
    // evaluate the first 32 pairs (or the last n < 32) and shift the rest down
    SG_DEV void drain(int n, const PairLaunch& L, const Pot& pot, EnergySums& es, unsigned long long* sh_stats) {
        const bool ok = lane < n;
        const int tq = ok ? q[lane] : 0, iq = ok ? q[64 + lane] : 0, jq = ok ? q[128 + lane] : 0;
        __syncwarp();
        if (n == 32 && lane < qn - 32) {
            q[lane] = q[32 + lane];
            q[64 + lane] = q[96 + lane];
            q[128 + lane] = q[160 + lane];
        }
        __syncwarp();
        qn -= n;
        pair_process<Pot, false>(L, pot, tq, iq, jq, ok, es, sh_stats);
    }
    // one listed pair per lane: range test, counters, queue, evaluate full batches
    SG_DEV void feed(const PairLaunch& L, const Pot& pot, int t, int i, int j, bool valid, EnergySums& es,
                     unsigned long long* sh_stats) {
        const bool in = valid && pot.in_range(i, j);
        const unsigned vm = __ballot_sync(0xffffffffu, valid), km = __ballot_sync(0xffffffffu, in);
        if (Pot::kCountActive && lane == 0) {
            atomicAdd(&sh_stats[0], (unsigned long long)__popc(vm));
            if (km) atomicAdd(&sh_stats[1], (unsigned long long)__popc(km));
        }
        if constexpr (Pot::kStats) {
            // solver statistics (ECP): a pair turned away counts as listed with
            // no solve (iteration bin 0), and the potential is told of it
            const unsigned rm = vm & ~km;
            if (lane == 0 && rm) {
                atomicAdd(&sh_stats[0], (unsigned long long)__popc(rm));
                atomicAdd(&sh_stats[4], (unsigned long long)__popc(rm));
            }
            if (valid && !in) pot.filtered_out(t);
        }
        push(in, t, i, j);
        if (qn >= 32) drain(32, L, pot, es, sh_stats);
    }
    // the queue's last pairs (qn is warp-uniform)
    SG_DEV void flush(const PairLaunch& L, const Pot& pot, EnergySums& es, unsigned long long* sh_stats) {
        if (qn > 0) drain(qn, L, pot, es, sh_stats);
    }
};

template <class Pot, bool FILTER>
constexpr int pair_min_blocks() {
    if constexpr (FILTER) return Pot::kMinBlocksFiltered;
    else return Pot::kMinBlocks;
}

// FILTER: the range test and per-warp queues of PairQueues.
template <class Pot, bool FILTER>
__global__ void __launch_bounds__(SG_PAIR_MAX_BLOCK, (pair_min_blocks<Pot, FILTER>())) k_pair(PairLaunch L, Pot pot) {
    using Q = PairQueues<Pot>;
    __shared__ unsigned long long sh_stats[SG_NSTATS];
    __shared__ int sh_queue[FILTER ? (SG_PAIR_MAX_BLOCK / 32) * Q::kWords : 1];
    constexpr bool kSh = Pot::kStats || Pot::kCountActive;
    if (kSh) {
        for (int k = threadIdx.x; k < SG_NSTATS; k += blockDim.x) sh_stats[k] = 0ull;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int np = *L.npairs;
    const int b0 = L.begin ? *L.begin : 0;
    EnergySums es;
    Q q;
    q.init(sh_queue + (FILTER ? (threadIdx.x >> 5) * Q::kWords : 0));
    // replica sections: warps walk whole 32-pair chunks, whose first replica is tabulated
    const int bstart = L.sec ? (b0 & ~31) : b0;
    const int stride = nwarps * 32;
    int tn, in_, jn;
    bool vn;
    pair_fetch(L, bstart + gwarp * 32, lane, np, b0, tn, in_, jn, vn);
    for (int base = bstart + gwarp * 32; base < np; base += stride) {
        const int t = tn, i = in_, j = jn;
        const bool valid = vn;
        if (base + stride < np) pair_fetch(L, base + stride, lane, np, b0, tn, in_, jn, vn);   // next indices in flight
        if constexpr (!FILTER)
            pair_process<Pot, Pot::kCountActive>(L, pot, t, i, j, valid, es, sh_stats);
        else
            q.feed(L, pot, t, i, j, valid, es, sh_stats);
    }
    if constexpr (FILTER) q.flush(L, pot, es, sh_stats);
    // the pairs are done: a kernel launched after this one with programmatic
    // serialisation (the final half step) may start loading what this one
    // does not write
    pdl_trigger();
    if (kSh && L.stats) {
        __syncthreads();
        for (int k = threadIdx.x; k < SG_NSTATS; k += blockDim.x)
            if (sh_stats[k]) atomicAdd(&L.stats[k], sh_stats[k]);
    }
    const float e[2] = {es.pe, es.vir}, elo[2] = {es.pe_lo, es.vir_lo};
    pair_sums_finish(e, elo, L.partials, L.done, L.acc, L.acc_total);
}

// The tested launch of a potential whose evaluation costs far more than its
// superset range test (an ECP contact solve, some twelve microseconds by itself,
// for one listed pair in eight): a block tests its span of the list, P pairs a
// thread at a time with their index loads and gathers in flight together, puts
// those that pass into shared memory in list order, and evaluates them in full
// batches of 32 consecutive ones, so that rows stay together for the segmented
// sums and no lane idles. Equal spans, one a block. Pairs turned away are
// counted as listed with no solve (stats[0], stats[4]) and handed to the
// potential's filtered_out.
// Bound: the latency of one test and one evaluation; BLOCKS, the resident blocks
// an SM, sets the registers of the evaluation, and its caller says by size and kind.
// Measured, us, the test in a kernel of its own that wrote the pairs that pass to
// memory, and a second kernel on those, / this: 528 000 listed pairs of 65 536
// repulsive ECP 22.9 / 18.5, 132 000 19.0 / 14.4, 16 500 19.3 / 14.1, 2.1 million
// 41.8 / 37.6; attractive kind 284 000 29.6 / 24.6, 1.7 million 85.3 / 85.4, 3.4
// million 160.7 / 162.5. Phases of a batch a warp, with the barriers between
// them, took 97 us for the 1.7 million, of six 85.4.
#define SG_TEST_P 4
#define SG_TEST_PHASE 6   // batches a warp, on average, before the block tests on
template <class Pot, int BLOCKS>
__global__ void __launch_bounds__(SG_PAIR_MAX_BLOCK, BLOCKS) k_pair_tested(PairLaunch L, Pot pot) {
    constexpr int P = SG_TEST_P, PHASE = SG_TEST_PHASE, CAP = SG_PAIR_MAX_BLOCK * (P + PHASE);
    static_assert(SG_PAIR_MAX_BLOCK / 32 * P <= 32, "one warp scans the round's counts");
    __shared__ int qt[CAP], qi[CAP], qj[CAP];   // less than PHASE pairs a thread, and one round
    __shared__ int sh_next;
    __shared__ int sh_n[SG_PAIR_MAX_BLOCK / 32 * P], sh_total;
    __shared__ unsigned long long sh_stats[SG_NSTATS];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = threadIdx.x; k < SG_NSTATS; k += blockDim.x) sh_stats[k] = 0ull;
    const int np = *L.npairs;
    const int span = max((int)blockDim.x, (int)(((np + gridDim.x - 1) / gridDim.x + 31) & ~31u));
    const long long start = (long long)blockIdx.x * span;
    const int hi = (int)min((long long)np, start + span);
    int base = (int)min((long long)np, start), have = 0;   // block-uniform
    unsigned away = 0;
    EnergySums es;
    for (;;) {
        if (threadIdx.x == 0) sh_next = nw;   // (a round's barriers, or the ones below, come before its use)
        while (base < hi && have < PHASE * (int)blockDim.x) {
            int t[P], i[P], j[P];
            bool keep[P];
            unsigned km[P];
#pragma unroll
            for (int k = 0; k < P; ++k) pair_fetch(L, base + (warp * P + k) * 32, lane, hi, 0, t[k], i[k], j[k], keep[k]);
            // the P range tests first, with no vote or store between them
            unsigned listed[P];
#pragma unroll
            for (int k = 0; k < P; ++k) {
                listed[k] = keep[k];
                keep[k] = keep[k] && pot.in_range(i[k], j[k]);
            }
#pragma unroll
            for (int k = 0; k < P; ++k) {
                km[k] = __ballot_sync(full, keep[k]);
                const unsigned vm = __ballot_sync(full, listed[k]);
                if (listed[k] && !keep[k]) pot.filtered_out(t[k]);
                away += __popc(vm & ~km[k]);
                if (lane == 0) sh_n[warp * P + k] = __popc(km[k]);
            }
            __syncthreads();
            if (warp == 0) {
                const int c = lane < nw * P ? sh_n[lane] : 0;
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(full, incl, o);
                    if (lane >= o) incl += y;
                }
                if (lane < nw * P) sh_n[lane] = incl - c;
                if (lane == 31) sh_total = incl;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < P; ++k) {
                if (keep[k]) {
                    const int slot = have + sh_n[warp * P + k] + __popc(km[k] & ((1u << lane) - 1u));
                    qt[slot] = t[k];
                    qi[slot] = i[k];
                    qj[slot] = j[k];
                }
            }
            have += sh_total;
            base += (int)blockDim.x * P;
            __syncthreads();   // written, and the counts read
        }
        // all of them at the end, else the full batches; a warp takes its next one
        // when it is done (the solves' iterations differ)
        const bool last = base >= hi;
        const int n = last ? have : have & ~31, batches = (n + 31) >> 5;
        for (int b = warp; b < batches;) {
            const bool ok = 32 * b + lane < n;
            const int s = ok ? 32 * b + lane : 0;
            if (lane == 0) b = atomicAdd(&sh_next, 1);
            pair_process<Pot, false>(L, pot, qt[s], qi[s], qj[s], ok, es, sh_stats);
            b = __shfl_sync(full, b, 0);
        }
        if (last) break;
        __syncthreads();
        if (threadIdx.x < 32) {   // fewer than a batch are left
            const bool rest = n + lane < have;
            const int s = rest ? n + lane : 0;
            const int rt = qt[s], ri = qi[s], rj = qj[s];
            __syncwarp();
            if (rest) {
                qt[lane] = rt;
                qi[lane] = ri;
                qj[lane] = rj;
            }
        }
        have -= n;
        // (the next round writes beyond them, and its barriers come before any read)
    }
    pdl_trigger();   // the pairs are done (see k_pair)
    if (L.stats) {
        if (lane == 0 && away) {
            atomicAdd(&sh_stats[0], (unsigned long long)away);
            atomicAdd(&sh_stats[4], (unsigned long long)away);
        }
        __syncthreads();
        for (int k = threadIdx.x; k < SG_NSTATS; k += blockDim.x)
            if (sh_stats[k]) atomicAdd(&L.stats[k], sh_stats[k]);
    }
    const float e[2] = {es.pe, es.vir}, elo[2] = {es.pe_lo, es.vir_lo};
    pair_sums_finish(e, elo, L.partials, L.done, L.acc, L.acc_total);
}

// Launch shape of the pair kernels: block size and the range filter. The
// autotuner (sg_pair_autotune) times the variants on the live list and
// stores the fastest per (kind, size bucket); untuned kinds use defaults.
PairTune sg_pair_tune_for(sg_ctx* ctx, int kind, bool filterable);

template <class Pot, bool FILTER>
int launch_pair_v(sg_ctx* ctx, PairLaunch L, Pot pot, int block) {
    if constexpr (Pot::kFilterable) pot.prefiltered = (FILTER && ExactFilter<Pot>::value) ? 1 : 0;
    const void* fn = (const void*)k_pair<Pot, FILTER>;
    int grid = sg_grid_for(ctx, fn, block, 0);
    int64_t max_useful = (ctx->nl.pair_capacity + block - 1) / block;
    if (grid > max_useful) grid = (int)std::max<int64_t>(1, max_useful);
    if (int rc = sg_pair_slots(ctx, grid, &L.partials, &L.done)) return rc;
    k_pair<Pot, FILTER><<<grid, block, 0, ctx->stream>>>(L, pot);
    SG_LAUNCH_CHECK(ctx, "k_pair");
    return SG_OK;
}

// The list walk of this context's pair kernels: the whole list, or in a
// replica context the rows of the launch family's replicas.
inline PairLaunch make_pair_launch(sg_ctx* ctx) {
    PairLaunch L;
    L.pair_i = ctx->nl.pair_i;
    L.pair_j = ctx->nl.pair_j;
    L.npairs = ctx->nl.dev_flags + 2;
    L.begin = nullptr;
    L.row_off = ctx->nl.row_off;
    L.rep_off = ctx->rep.off;
    L.sec = nullptr;
    L.chunk_rep = nullptr;
    L.nrep = ctx->nrep;
    if (ctx->nrep) {
        // pairs of one potential family: rows of the family's replicas
        const int f = ctx->launch_family;
        L.begin = ctx->nl.row_off + ctx->fam_pstart[f];
        L.npairs = ctx->nl.row_off + ctx->fam_pstart[f + 1];
        L.sec = ctx->nl.rep_pad_off;
        L.chunk_rep = ctx->nl.chunk_rep;
    }
    L.force = ctx->force;
    L.torque = ctx->torque;
    L.done = nullptr;
    L.acc = ctx->acc + 4;
    L.acc_total = ctx->acc;
    L.stats = ctx->step_fused ? nullptr : ctx->stats;
    L.partials = nullptr;
    return L;
}

// The tested launch (single systems).
template <int BLOCKS, class Pot>
int launch_pair_tested(sg_ctx* ctx, Pot pot, int block) {
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "pair forces need sg_nlist_init first");
    PairLaunch L = make_pair_launch(ctx);
    pot.prefiltered = 0;
    int grid = sg_grid_for(ctx, (const void*)k_pair_tested<Pot, BLOCKS>, block, 0);
    const int64_t useful = (ctx->nl.pair_capacity + block - 1) / block;
    grid = (int)std::max<int64_t>(1, std::min<int64_t>(grid, useful));
    if (int rc = sg_pair_slots(ctx, grid, &L.partials, &L.done)) return rc;
    k_pair_tested<Pot, BLOCKS><<<grid, block, 0, ctx->stream>>>(L, pot);
    SG_LAUNCH_CHECK(ctx, "k_pair_tested");
    return SG_OK;
}

// Launch helper: persistent grid sized from occupancy.
template <class Pot>
int launch_pair(sg_ctx* ctx, Pot pot, int kind) {
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "pair forces need sg_nlist_init first");
    if (int rc = sg_need_half_list(ctx, true)) return rc;
    PairLaunch L = make_pair_launch(ctx);
    const PairTune tune = sg_pair_tune_for(ctx, kind, Pot::kFilterable);
    if (Pot::kFilterable && tune.filter) return launch_pair_v<Pot, Pot::kFilterable>(ctx, L, pot, tune.block);
    return launch_pair_v<Pot, false>(ctx, L, pot, tune.block);
}

struct BoxF {
    float3 box, inv_box;
    float3 box_lo;              // box - (float)box: with box, the FP64 box to ~1e-15
    int periodic;
    const int* rep_of;          // batched replicas: per-particle replica, else nullptr
    const float4* rbox;
    const float4* rinv;
    const float4* rbox_lo;
};

inline BoxF make_boxf(const sg_ctx* ctx) {
    BoxF b;
    b.rep_of = ctx->rep.rep_of;
    b.rbox = ctx->rep.box;
    b.rinv = ctx->rep.inv_box;
    b.rbox_lo = ctx->rep.box_lo;
    b.box_lo = make_float3((float)(ctx->box[0] - (double)(float)ctx->box[0]),
                           (float)(ctx->box[1] - (double)(float)ctx->box[1]),
                           (float)(ctx->box[2] - (double)(float)ctx->box[2]));
    b.box = make_float3((float)ctx->box[0], (float)ctx->box[1], (float)ctx->box[2]);
    b.inv_box = make_float3((float)(1.0 / ctx->box[0]), (float)(1.0 / ctx->box[1]), (float)(1.0 / ctx->box[2]));
    b.periodic = ctx->periodic;
    return b;
}

// r_ij = a - c by the minimum image of the box of i (BoxF).
SG_DEV float3 pair_rij_of(float3 a, float3 c, int i, const BoxF& b) {
    if (b.rep_of) {
        const int r = b.rep_of[i];
        const float4 bx = b.rbox[r], ib = b.rinv[r];
        return min_image(make_float3(a.x - c.x, a.y - c.y, a.z - c.z), make_float3(bx.x, bx.y, bx.z),
                         make_float3(ib.x, ib.y, ib.z), 1);
    }
    return min_image(make_float3(a.x - c.x, a.y - c.y, a.z - c.z), b.box, b.inv_box, b.periodic);
}

// Two float4 from one 32-byte aligned address in a single 256-bit load
// (read-only path): a gather of 32 bytes per lane in one request.
SG_DEV void ld_f4x2(const float4* __restrict__ p, float4& a, float4& c) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w)
        : "l"(p));
}

SG_DEV float3 pair_rij(const float4* __restrict__ pos, int i, int j, const BoxF& b) {
    float4 a = pos[i], c = pos[j];
    if (b.rep_of) {
        // pairs never cross replicas: the replica of i gives the box
        const int r = b.rep_of[i];
        const float4 bx = b.rbox[r], ib = b.rinv[r];
        return min_image(make_float3(a.x - c.x, a.y - c.y, a.z - c.z), make_float3(bx.x, bx.y, bx.z),
                         make_float3(ib.x, ib.y, ib.z), 1);
    }
    return min_image(make_float3(a.x - c.x, a.y - c.y, a.z - c.z), b.box, b.inv_box, b.periodic);
}

// pair_rij that also returns the product of the two charges (pos.w).
SG_DEV float3 pair_rij_q(const float4* __restrict__ pos, int i, int j, const BoxF& b, float& qq) {
    const float4 a = pos[i], c = pos[j];
    qq = a.w * c.w;
    const float3 d = make_float3(a.x - c.x, a.y - c.y, a.z - c.z);
    if (b.rep_of) {
        const int r = b.rep_of[i];
        const float4 bx = b.rbox[r], ib = b.rinv[r];
        return min_image(d, make_float3(bx.x, bx.y, bx.z), make_float3(ib.x, ib.y, ib.z), 1);
    }
    return min_image(d, b.box, b.inv_box, b.periodic);
}

// One component of the minimum image, to about 1e-12 absolute: the FP32
// difference a - c with its exact rounding error (two-sum), the image shift
// n * (box_hi + box_lo) applied to each part (for n = +-1 the difference is
// within a factor two of box_hi, so d - n box_hi is exact). Without it, pairs
// across the boundary carry the rounding of a - c (~ulp(box)/2) and of the
// FP32 box.
SG_DEV float min_image_precise(float a, float c, float L, float iL, float Llo, int periodic) {
    const float d = a - c;
    const float bb = d - a;
    const float e = (a - (d - bb)) + (-c - bb);
    if (!periodic) return d + e;
    const float n = roundf(d * iL);
    return __fsub_rn(d, n * L) + (e - n * Llo);
}

// r_ij = a - c by the minimum image of the box of i, to ~1e-12 absolute
// (min_image_precise), from positions already loaded.
SG_DEV float3 pair_rij_of_precise(float3 a, float3 c, int i, const BoxF& b) {
    float3 L = b.box, iL = b.inv_box, lo = b.box_lo;
    int per = b.periodic;
    if (b.rep_of) {
        const int r = b.rep_of[i];
        const float4 bx = b.rbox[r], ib = b.rinv[r], bl = b.rbox_lo[r];
        L = make_float3(bx.x, bx.y, bx.z);
        iL = make_float3(ib.x, ib.y, ib.z);
        lo = make_float3(bl.x, bl.y, bl.z);
        per = 1;
    }
    return make_float3(min_image_precise(a.x, c.x, L.x, iL.x, lo.x, per),
                       min_image_precise(a.y, c.y, L.y, iL.y, lo.y, per),
                       min_image_precise(a.z, c.z, L.z, iL.z, lo.z, per));
}

// pair_rij for the contact-distance potentials (ECP): see min_image_precise.
SG_DEV float3 pair_rij_precise(const float4* __restrict__ pos, int i, int j, const BoxF& b) {
    const float4 a = pos[i], c = pos[j];
    float3 L = b.box, iL = b.inv_box, lo = b.box_lo;
    int per = b.periodic;
    if (b.rep_of) {
        const int r = b.rep_of[i];
        const float4 bx = b.rbox[r], ib = b.rinv[r], bl = b.rbox_lo[r];
        L = make_float3(bx.x, bx.y, bx.z);
        iL = make_float3(ib.x, ib.y, ib.z);
        lo = make_float3(bl.x, bl.y, bl.z);
        per = 1;
    }
    return make_float3(min_image_precise(a.x, c.x, L.x, iL.x, lo.x, per),
                       min_image_precise(a.y, c.y, L.y, iL.y, lo.y, per),
                       min_image_precise(a.z, c.z, L.z, iL.z, lo.z, per));
}

// Reciprocal by the approximate instruction (at most 1 ulp from 1/x for
// normal x, PTX rcp.approx.ftz.f32): a division costs a dozen instructions,
// this one. Used where a 1-ulp quotient is far inside the force tolerance.
SG_DEV float fast_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x^n by repeated multiplication, left to right (the rounding of a loop of
// products); n is uniform across the warp. Up to n = 4 the products are
// selected instead of looped.
SG_DEV float ipowf(float x, int n) {
    const float x2 = x * x, x3 = x2 * x, x4 = x3 * x;
    if (n <= 4) return n <= 0 ? 1.f : n == 1 ? x : n == 2 ? x2 : n == 3 ? x3 : x4;
    float r = x4;
    for (int k = 4; k < n; ++k) r *= x;
    return r;
}

// 1/sqrt(x) by the approximate instruction (PTX rsqrt.approx.ftz.f32): for
// superset range tests that carry a slack far above its error.
SG_DEV float fast_rsqrt(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
