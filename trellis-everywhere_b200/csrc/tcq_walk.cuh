// The walk back over the metric rows of the cluster step kernel (tcq_forward_cluster.cuh), and what a tile's states become.
#pragma once

#include <cuda/std/bit>
#include <type_traits>

#include "tcq_forward.cuh"
#include "tcq_handoff.cuh"
#include "tcq_mbarrier.cuh"

namespace tcq {

// Outputs of one tile over the steps that were walked, by NT threads, from the states in shared memory.
template <int K, int NT>
__device__ __forceinline__ void emit_outputs(const TracebackArgs& a, long long tile, const uint16_t* st, int t_off, int t_end, int tid) {
    constexpr uint32_t Q = Geo<K>::Q;
    if (a.states != nullptr)
        for (int t = t_off + tid; t < t_end; t += NT) a.states[tile * kT + t] = (long long)st[t];
    if (a.bits != nullptr)
        for (int t = t_off + tid; t < t_end; t += NT) a.bits[tile * kT + t] = (long long)(st[t] & (Q - 1));
    if (a.dq != nullptr)
        for (int t = t_off + tid; t < t_end; t += NT) a.dq[tile * kT + t] = cb_value_rt(a.codebook, st[t]);
    if (a.wq != nullptr) {
        // LDLQ row-block layout (src/trellis/ldlq.py:142-143): weight t of this tile is element
        // [t & 15][16 * tile + (t >> 4)] of a 16-row block; j walks along the matrix rows so that a
        // half-warp writes 64 contiguous bytes.  err = src - reconstruction is the block error the
        // recursion feeds back (ldlq.py:90,97), formed here instead of by a separate pass over the block.
        for (int j = tid; j < kT; j += NT) {
            const int t = ((j & 15) << 4) | (j >> 4);
            if (t < t_off || t >= t_end) continue;
            const float v = cb_value_rt(a.codebook, st[t]);
            const long long off = (long long)(j >> 4) * a.ld + tile * 16 + (j & 15);
            a.wq[off] = v;
            if (a.err != nullptr) a.err[off] = __fsub_rn(a.src[off], v);
        }
    }
    if (a.packed != nullptr) {
        // (whole words: a part of a pass is a multiple of 64 steps)
        // word j holds stream bits 32j .. 32j+31; stream bit p is bit (p % K) of symbol 255 - p / K
        for (uint32_t j = uint32_t(kT - t_end) * K / 32 + tid; j < uint32_t(kT - t_off) * K / 32; j += NT) {
            uint32_t word = 0;
#pragma unroll 8
            for (uint32_t b = 0; b < 32; ++b) {
                const uint32_t p = 32 * j + b;
                const uint32_t t = (kT - 1) - p / K;
                word |= ((uint32_t(st[t]) >> (p % K)) & 1u) << b;
            }
            a.packed[tile * a.packed_stride + j] = word;
        }
    }
}

// Walk over metric rows (MetricRows, left by the cluster step kernel): one CTA of W warps per tile.
//
// Per trip the walk takes D steps back.  It reads the NA = Q^D metrics, contiguous in the row, that the current edge can
// have come from, forms the candidates of the first of the D steps for the Q^(D-1) nodes above them exactly as the step
// kernel does (same operations, same order, lowest q among equals), and so on up the tree to the current edge; each node
// carries the q's chosen below it, so the root holds the whole path.  Candidates per step and tile, those that warps and lanes form
// more than once included: 1/100, 1/180, 1/450 of the step kernel's (K = 2, 3, 4).
//
// What bounds it is the latency of one trip, whose address the trip before decides.  So the first level is spread over
// the CTA (one barrier per trip, two buffers); the other levels are small and every warp does them for itself; and the
// emission costs of all levels, which depend on the edge only, are formed while the metrics are on their way.
template <int K> struct WalkShape {
    static constexpr int W = K == 2 ? 4 : K == 3 ? 2 : 1;      // warps
    static constexpr int SPLIT = K == 4 ? 2 : 1;               // lanes that share a first-level node
};

// Lowest q whose candidate is the minimum (Q-1 if no candidate compares equal: not-a-number weights), as the step kernels choose.
template <int N>
__device__ __forceinline__ uint32_t first_minimum(const float (&c)[N], float best) {
    uint32_t qb = N - 1;
#pragma unroll
    for (int q = N - 2; q >= 0; --q) qb = c[q] == best ? uint32_t(q) : qb;
    return qb;
}

// Metrics of fused candidates (StepForm::kFused).  Let u = 2^-24 and let a path's cost after t steps be R in real numbers, F summed as defined,
// with the difference, the square and every sum rounded, and A with the square and the sum as one operation.  The difference is
// the same, all terms are positive, and a sum below 2 H, H a power of two, is rounded by u H at most; so |F - R| <= (t + 2) u H and
// |A - R| <= t u H, and both minima over paths obey the same bounds.  Hence: if a candidate's A is above the smallest candidate's
// A by more than (4 t + 4) u H, its F is above that one's F as well (and no tie).  H is taken from the smallest candidate, a little
// enlarged so that no sum in question reaches 2 H; twelve more u H cover the rounding of the limit itself, and 1e-30 what underflows (512
// operations, 2^-150 each).  Above 1e37 sums may overflow: such tiles are swept again.
// (Plain operators, which the build does not contract: the host computes the same, tests/fused_limit.cu.)
__host__ __device__ __forceinline__ float fused_limit(float best, int t) {
    const float h = cuda::std::bit_cast<float>(cuda::std::bit_cast<uint32_t>(best * 1.0005f) & 0x7f800000u);
    return fmaf(h, float(4 * t + 16) * 0x1p-24f, best) + 1e-30f;
}
constexpr float kFusedMax = 1e37f;
constexpr long long kWalkWaitCycles = 500000000LL;        // of the second group for the first, a quarter of a second where microseconds are due

// A tile's rows lie one after another whatever the path, so where few tiles walk, each on an SM of its own, their CTAs fetch whole rows ahead
// (32 KiB at K = 3) and find a trip's metrics in shared memory: the latency of L2 or HBM leaves the chain of trips.  16 times as many bytes
// are read, 2.8 MB a tile and walk, so it is for few tiles only.
template <int K> struct Ring {
    static constexpr int E = Geo<K>::E, kRows = 192 * 1024 / (E * 4);
    static constexpr size_t kBytes = size_t(kRows) * E * 4 + 16 * 8;       // rows, then an mbarrier each and the waits' flag
    static_assert(kRows <= 14, "the flag is the sixteenth word");
};

template <int K, bool FUSED>
struct WalkShared {
    static constexpr int D = MetricRows<K>::D, W = WalkShape<K>::W, N1 = MetricRows<K>::NA >> K, N2 = D >= 3 ? N1 >> K : 1;
    // (kMaxTrips along other paths: of 100 000 Gaussian tiles one that was settled took more, and tiles of zeros at K = 4 take four times as many in vain)
    static constexpr int kMaxMarks = 16, kMaxTodo = 8, kMaxTrips = 128;
    struct Walker {
        uint16_t st[kT];
        float val1[2][N1];                         // first level: minima and their q, double buffered over trips
        uint32_t path1[2][N1];
        float val[W][D > 2 ? D - 2 : 1][N2];       // levels 2 .. D-1, one copy per warp
        uint32_t path[W][D > 2 ? D - 2 : 1][N2];
        unsigned char mark[FUSED ? 128 : 1];       // by trip: another path comes within the limit
    };
    Walker walker[FUSED ? 2 : 1];
    float wv_pad[kT + 8];                          // by step; the first trip may also look (in vain) at the steps before 0
    // FUSED only
    alignas(16) float cost[FUSED ? kT + 4 : 1];    // rounded cost of the path before each step
    uint16_t other[FUSED ? kT : 1];                // states of another path
    uint32_t todo[FUSED ? kMaxTodo : 1][3];        // such paths: the last step that they do not share, the state there, q's of the trip before it
    int go_on;                                     // the second group's orders
    int trips;                                     // taken by the first group (kAllTrips: the walk is over and `cost` complete), published (tcq_handoff.cuh)
    int verdict;                                   // of the second group on the marks: kOther | kApart
    static constexpr int kAllTrips = 1 << 20, kTold = 4, kOther = 1, kApart = 2;      // (told of every trip, a walk takes 4 to 7 us longer)
};

// The walk over one tile, by WalkShape<K>::W whole warps (threads 0 .. 32 W - 1 of the CTA), from the rows and partial minima of `slot`.
// OTHER: the rows' ancestors lie as in MetricRows::other_pos.  COHERENT: the rows were written by this kernel.
//
// FUSED: the metrics are those of fused candidates.  A node on the path where a second candidate is within fused_limit of the smallest marks
// its trip; nothing else is done on the way.  Without a mark (99 Gaussian tiles of 100) the path is the defined one.  With marks every such
// candidate's own path is walked back until it meets the path found.  In the pass that looks for the overlap that is all as long as
// they meet before the middle of the tile: the overlap is the same either way.  Otherwise, and in the other pass, the two are compared by
// their rounded sums from where they meet (one tile in 800 of the first pass is walked back to its beginning for that).
// Other paths cost as long as they are to walk, so a second group of warps walks them at the same time: where the pass may end with one
// of two edges (one tile in 36 to 75 of the first pass) it walks from the second edge; otherwise it goes behind the first group and takes up
// the trips that get marked.  Its waits for the first group are bounded by the clock; a tile whose wait runs out is listed.
// What this does not settle (marks on the other path too, another winner, more than a few marks, costs above 1e37 or not a
// number) lists the tile in a.again: one Gaussian tile in 10 000, and some tiles of ties, such as one of zeros in the second pass.
//
// RING: rows come to shared memory ahead of the walk; `ring` is Ring<K>::kBytes of it.
template <int K, int CB, bool OTHER, bool FUSED, bool COHERENT, bool RING = false>
__device__ __forceinline__ void walk_tile(const TracebackArgs& a, long long tile, long long slot, WalkShared<K, FUSED>& sh, float* ring = nullptr) {
    static_assert(!RING || !FUSED, "the second group would need rows of its own");
    using GE = Geo<K>;
    using MR = MetricRows<K>;
    constexpr uint32_t Q = GE::Q, E = GE::E;
    constexpr int SH = kL - K, D = MR::D, LB = MR::LB, NA = MR::NA;
    constexpr int W = WalkShape<K>::W, NT = W * 32, SPLIT = WalkShape<K>::SPLIT;
    constexpr int N1 = NA / int(Q);                // first-level nodes
    constexpr int NPT = N1 * SPLIT / NT;           // ... per thread
    constexpr int QS = int(Q) / SPLIT;             // candidates of a node that one thread forms
    constexpr int N2 = D >= 3 ? N1 / int(Q) : 1;   // second-level nodes
    constexpr int NP2 = N2 > 32 ? N2 / 32 : 1;     // ... per lane
    static_assert(NPT * NT == N1 * SPLIT && (SPLIT == 1 || (W == 1 && N1 * SPLIT == 32)), "first-level nodes must divide over the threads");
    const int who = FUSED && threadIdx.x >= NT ? 1 : 0;            // which walker
    auto& mine = sh.walker[who];
    uint16_t* const st = mine.st;
    float* const wv = sh.wv_pad + 8;
    auto& val1 = mine.val1;
    auto& path1 = mine.path1;
    auto& val = mine.val;
    auto& path = mine.path;
    auto sync = [who] {                            // the walker's warps
        // (a barrier number in a register would reserve all sixteen, of which an SM has enough for four CTAs only)
        if constexpr (W == 1) __syncwarp();
        else if (who == 0) asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        else asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
    };
    auto both = [] { asm volatile("bar.sync 3, %0;" ::"n"(2 * NT) : "memory"); };
    auto load = [](const auto* p) {
        if constexpr (COHERENT) return __ldcg(p);
        else return __ldg(p);
    };
    const int tid = FUSED ? int(threadIdx.x) % NT : int(threadIdx.x), lane = tid & 31, wrp = tid >> 5;

    ForwardArgs fw{};
    fw.w = a.w;
    fw.w_add = a.w_add;
    fw.ld = a.ld;
    for (int i = tid; i < kT; i += NT) {
        int t;
        const float x = load_weight(fw, tile, i, t);
        wv[(t - a.roll) & (kT - 1)] = x;
    }
    if (tid < 8) sh.wv_pad[tid] = 0.0f;
    if constexpr (FUSED)
        for (int i = tid; i < 128; i += NT) mine.mark[i] = 0;
    if (FUSED && threadIdx.x == 0) sh.trips = 0;
    uint32_t e, e_end, e_second = ~0u;
    float end_metric = 0.0f;
    unsigned long long key = ~0ull;
    uint32_t rivals = 0;                // lanes whose key is that of another edge that the pass may end with
    if (a.keys != nullptr) {            // argmin of the final metrics, left as per-CTA partial minima by the step kernel (32 at most)
        if (lane < a.nkeys) key = load(a.keys + slot * a.nkeys + lane);
        unsigned long long k = key;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, k, off);
            k = o < k ? o : k;
        }
        e_end = uint32_t(k) & (E - 1);
        end_metric = __uint_as_float(uint32_t(k >> 32));
        if constexpr (FUSED) {
            rivals = __ballot_sync(0xffffffffu, key < kTooMany && key != k && !(__uint_as_float(uint32_t(key >> 32)) > fused_limit(end_metric, kT)));
            if (rivals != 0) e_second = uint32_t(__shfl_sync(0xffffffffu, key, __ffs(int(rivals)) - 1)) & (E - 1);
        }
    } else {
        e_end = uint32_t(a.e_start[tile]) & (E - 1);
    }
    // two: both groups walk.  behind: the second group takes up the marks of the first.
    const bool pair = FUSED && blockDim.x > NT, two = pair && rivals != 0, behind = pair && !two;
    e = who == 1 ? e_second : e_end;
    const uint32_t ov = a.overlap != nullptr ? uint32_t(a.overlap[tile]) & (E - 1) : ~0u;
    // metric of edge x before step 0
    auto start_metric = [&](uint32_t x) { return a.overlap == nullptr ? 0.0f : x == ov ? 0.0f : __uint_as_float(kInfBits); };
    const int t_off = a.t_end - a.bp_steps;
    const float* const rows = a.rows + size_t(slot) * a.nrows * E;
    if (pair) both();
    else sync();

    // emission cost of state (q, y) at weight w (FUSED: its root), and the candidate that it makes of a metric
    auto emission = [](float w, uint32_t q, uint32_t y) {
        const float d = __fsub_rn(w, cb_value<CB>((q << SH) | y));
        return FUSED ? d : __fmul_rn(d, d);
    };
    auto candidate = [](float em, float metric) { return FUSED ? __fmaf_rn(em, em, metric) : __fadd_rn(em, metric); };
    // FUSED: bit 31 of a node's path says that on it a second candidate came within the limit
    constexpr uint32_t kNear = 0x80000000u;
    auto within = [](const auto& c, float limit) {
        int n = 0;
        for (float x : c) n += !(x > limit);
        return n;
    };
    // One trip, from edge e after step tau + D - 1 to the first of its D steps, tau: returns the path, q of step tau + i at bits i*K.
    // metric(q * N1, p): the metric of ancestor q * N1 + p before step tau.  kFirst: the trip that holds step 0; nodes before step 0 have the start
    // metric of their edge.
    // kNow (FUSED): nodes carry kNear.  Otherwise the trip's candidates are kept, and looked at under the loads of the next one.
    float kept1[NPT][QS] = {}, best1[NPT] = {}, kept[D > 2 ? D - 2 : 1][NP2][Q] = {}, bests[D > 2 ? D - 2 : 1][NP2] = {}, kept_root = 0.0f, best_root = 0.0f;
    uint32_t kept_path = 0;
    int kept_tau = -2 * D, kept_j = 0;
    auto look = [&]() __attribute__((always_inline)) {
        // (each level by the one warp that holds, or of those that hold, the path's node)
        bool near = kept_tau + D > 0 && __popc(__ballot_sync(0xffffffffu, !(kept_root > fused_limit(best_root, kept_tau + D)))) > 32 / int(Q);
        uint32_t p = kept_path >> ((D - 1) * K);           // the path's node one level down
#pragma unroll
        for (int d = D - 1; d >= 2; --d) {
            const uint32_t M = 1u << ((D - d) * K);
            if (wrp == 0 && kept_tau + d > 0) {
#pragma unroll
                for (int i = 0; i < (M > 32 ? int(M) / 32 : 1); ++i)
                    if (((lane + 32 * i) & (M - 1)) == p) near = near || within(kept[d - 2][i], fused_limit(bests[d - 2][i], kept_tau + d)) > 1;
            }
            p += ((kept_path >> ((d - 1) * K)) & (Q - 1)) * M;
        }
        if (kept_tau >= 0) {
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
                if (W > 1 && (p ^ uint32_t(tid + i * NT)) % N1 >= 32) continue;         // (warp-uniform)
                int n = within(kept1[i], fused_limit(best1[i], kept_tau + 1));
                if constexpr (SPLIT == 2) n += __shfl_xor_sync(0xffffffffu, n, N1);
                near = near || (uint32_t(tid + i * NT) % N1 == p && n > 1);
            }
        }
        if (near) mine.mark[kept_j] = 1;
    };
    auto trip = [&](int buf, auto first_c, auto now_c, int tau, uint32_t e, auto metric) __attribute__((always_inline)) -> uint32_t {
        constexpr bool kFirst = decltype(first_c)::value, kNow = decltype(now_c)::value;
        float c1[NPT][QS];
#pragma unroll
        for (int i = 0; i < NPT; ++i)
#pragma unroll
            for (int k = 0; k < QS; ++k) {
                const uint32_t q = uint32_t(k + (SPLIT > 1 ? lane / N1 * QS : 0));
                c1[i][k] = metric(q * N1, uint32_t(tid + i * NT) % N1);
            }
        // the emissions of every level, under the loads
        float em1[NPT][QS], em[D - 1][NP2][Q], em_root;
#pragma unroll
        for (int i = 0; i < NPT; ++i)
#pragma unroll
            for (int k = 0; k < QS; ++k) {
                const uint32_t q = uint32_t(k + (SPLIT > 1 ? lane / N1 * QS : 0)), p = uint32_t(tid + i * NT) % N1;
                em1[i][k] = emission(wv[tau], q, (p << (LB + K)) | (e >> ((D - 1) * K)));
            }
#pragma unroll
        for (int d = 2; d < D; ++d) {
            const int M = 1 << ((D - d) * K);      // nodes of this level
#pragma unroll
            for (int i = 0; i < (M > 32 ? M / 32 : 1); ++i)
#pragma unroll
                for (uint32_t q = 0; q < Q; ++q)
                    em[d - 2][i][q] = emission(wv[tau + d - 1], q, (uint32_t((lane + 32 * i) & (M - 1)) << (LB + d * K)) | (e >> ((D - d) * K)));
        }
        em_root = emission(wv[tau + D - 1], uint32_t(lane) & (Q - 1), e);
        if constexpr (FUSED && !kNow) look();

        // first level
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
#pragma unroll
            for (int k = 0; k < QS; ++k) c1[i][k] = candidate(em1[i][k], c1[i][k]);
            float best = min_of<QS>(c1[i]);
            uint32_t qb = first_minimum<QS>(c1[i], best);
            if constexpr (SPLIT == 2) {
                const float bo = __shfl_xor_sync(0xffffffffu, best, N1);
                const uint32_t qo = __shfl_xor_sync(0xffffffffu, qb, N1);
                const bool upper = lane >= N1;
                const float b0 = upper ? bo : best, b1 = upper ? best : bo;
                const uint32_t q0 = upper ? qo : qb, q1 = (upper ? qb : qo) + QS;
                best = fminf(b0, b1);
                qb = b0 == best ? q0 : b1 == best ? q1 : Q - 1;
            }
            const int p = (tid + i * NT) % N1;
            if constexpr (FUSED && kNow) {
                int n = within(c1[i], fused_limit(best, tau + 1));
                if constexpr (SPLIT == 2) n += __shfl_xor_sync(0xffffffffu, n, N1);
                if (n > 1 && (!kFirst || tau >= 0)) qb |= kNear;
            } else if constexpr (FUSED) {
#pragma unroll
                for (int k = 0; k < QS; ++k) kept1[i][k] = c1[i][k];
                best1[i] = best;
            }
            if constexpr (kFirst)
                if (tau < 0) best = start_metric((uint32_t(p) << (LB + K)) | (e >> ((D - 1) * K)));
            val1[buf][p] = best;
            path1[buf][p] = qb;
        }
        sync();
        const float* vin = val1[buf];
        const uint32_t* pin = path1[buf];
#pragma unroll
        for (int d = 2; d < D; ++d) {
            const int M = 1 << ((D - d) * K);
#pragma unroll
            for (int i = 0; i < (M > 32 ? M / 32 : 1); ++i) {
                const uint32_t p = uint32_t((lane + 32 * i) & (M - 1));
                float c[Q];
#pragma unroll
                for (uint32_t q = 0; q < Q; ++q) c[q] = candidate(em[d - 2][i][q], vin[q * uint32_t(M) + p]);
                float best = min_of<int(Q)>(c);
                const uint32_t qb = first_minimum<int(Q)>(c, best);
                uint32_t mark = 0;
                if constexpr (FUSED && kNow) {
                    if (within(c, fused_limit(best, tau + d)) > 1 && (!kFirst || tau + d - 1 >= 0)) mark = kNear;
                } else if constexpr (FUSED) {
#pragma unroll
                    for (uint32_t q = 0; q < Q; ++q) kept[d - 2][i][q] = c[q];
                    bests[d - 2][i] = best;
                }
                if constexpr (kFirst)
                    if (tau + d - 1 < 0) best = start_metric((p << (LB + d * K)) | (e >> ((D - d) * K)));
                val[wrp][d - 2][p] = best;
                path[wrp][d - 2][p] = pin[qb * uint32_t(M) + p] | (qb << ((d - 1) * K)) | mark;
            }
            __syncwarp();
            vin = val[wrp][d - 2];
            pin = path[wrp][d - 2];
        }
        // the root: one candidate per lane.  Candidates are non-negative (or not a number), so their bits order like the values.
        const float c = candidate(em_root, vin[uint32_t(lane) & (Q - 1)]);
        const float best = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(c)));
        const uint32_t eq = __ballot_sync(0xffffffffu, c == best);
        const uint32_t qb = eq != 0 ? uint32_t(__ffs(int(eq)) - 1) : Q - 1;
        const uint32_t whole = pin[qb] | (qb << ((D - 1) * K));
        if constexpr (FUSED && kNow) {
            return __popc(__ballot_sync(0xffffffffu, !(c > fused_limit(best, tau + D)))) > 32 / int(Q) ? whole | kNear : whole;
        } else if constexpr (FUSED) {
            kept_root = c;
            best_root = best;
            kept_path = whole;
            kept_tau = tau;
            kept_j = (a.t_end - D - tau) / D;
        }
        return whole;
    };
    // ... where its metrics are: rows, or before step 0
    auto row_of = [&](uint32_t e, int j) { return rows + size_t(j) * E + (e >> (K * D)) * uint32_t(NA); };    // the ancestors share the edge's bits above K*D
    [[maybe_unused]] unsigned long long* const full = reinterpret_cast<unsigned long long*>(ring + (RING ? Ring<K>::kRows * int(E) : 0));
    [[maybe_unused]] bool lost = RING && a.hurry;  // RING: a row did not come; the walk goes on from global memory
    [[maybe_unused]] int lost_at = 0;              // ... this row
    [[maybe_unused]] int ring_rows = 0;            // rows that the walk reads
    [[maybe_unused]] auto fetch = [&](int j) {
        const uint32_t bar = smem_u32(full + j % Ring<K>::kRows);
        mbar_expect(bar, E * 4);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(ring + j % Ring<K>::kRows * int(E))), "l"(rows + size_t(j) * E), "r"(uint32_t(E) * 4), "r"(bar) : "memory");
    };
    if constexpr (RING) {
        while (a.t_end - D * (ring_rows + 1) > 0 && a.t_end - D * ring_rows > t_off) ++ring_rows;
        if (tid == 0) {
            for (int i = 0; i < Ring<K>::kRows; ++i) mbar_init(smem_u32(full + i), 1);
            *reinterpret_cast<unsigned int*>(full + 15) = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            for (int i = 0; i < Ring<K>::kRows && i < ring_rows; ++i) fetch(i);
        }
        sync();
    }
    auto row_trip = [&](int buf, auto now_c, int tau, uint32_t e, int j) __attribute__((always_inline)) {
        if constexpr (RING) {
            if (!lost) {
                const bool came = mbar_wait(smem_u32(full + j % Ring<K>::kRows), uint32_t(j / Ring<K>::kRows) & 1u, reinterpret_cast<volatile unsigned int*>(full + 15));
                lost = __any_sync(0xffffffffu, !came);
                lost_at = j;
            }
            if (!lost) {
                const float* const row = ring + j % Ring<K>::kRows * int(E) + (e >> (K * D)) * uint32_t(NA);
                const uint32_t whole = trip(buf, std::false_type{}, now_c, tau, e, [&](uint32_t pq, uint32_t p) { return row[OTHER ? MR::order(pq) | MR::order(p) : pq | p]; });
                // every thread has its metrics: the trip's barrier lies behind it
                if (tid == 0 && j + Ring<K>::kRows < ring_rows) fetch(j + Ring<K>::kRows);
                return whole;
            }
        }
        const float* const row = row_of(e, j);
        return trip(buf, std::false_type{}, now_c, tau, e, [&](uint32_t pq, uint32_t p) { return load(row + (OTHER ? MR::order(pq) | MR::order(p) : pq | p)); });
    };
    auto first_trip = [&](int buf, auto now_c, int tau, uint32_t e) __attribute__((always_inline)) {
        const uint32_t g = e >> (K * D);
        return trip(buf, std::true_type{}, now_c, tau, e, [&](uint32_t pq, uint32_t p) { return start_metric(((pq + p) << LB) | g); });
    };

    int tau = a.t_end - D, j = 0, lo = t_off;
    auto take = [&](uint32_t whole, bool first) __attribute__((always_inline)) {       // a trip's states become the path's
#pragma unroll
        for (int i = D - 1; i >= 0; --i) {
            const uint32_t s = (((whole >> (i * K)) & (Q - 1)) << SH) | e;
            if (tid == 0 && (!first || tau + i >= 0)) st[tau + i] = uint16_t(s);
            e = s >> K;
        }
        if (FUSED && behind && tid == 0 && j % sh.kTold == sh.kTold - 1) handoff_publish(sh.trips, j + 1);
    };
    auto walk = [&]() __attribute__((always_inline)) {     // back to step `lo`, or a little further
        for (; tau > 0 && tau + D > lo; ++j, tau -= D) take(row_trip(j & 1, std::false_type{}, tau, e, j), false);
        if (tau + D > lo) {                        // tau <= 0
            take(first_trip(j & 1, std::false_type{}, tau, e), true);
            tau -= D;
        }
        if constexpr (FUSED) {
            look();
            kept_tau = -2 * D;
        }
        sync();
    };
    bool again = false;                            // FUSED: sweep the tile again
    if constexpr (!FUSED) {
        walk();
    } else {
        const uint16_t* const found = sh.walker[0].st;     // the path found
        const bool tied = a.overlap != nullptr;    // the start edge is given; otherwise all are as good
        bool sums = tied;                          // the path is known from its beginning, and its cost by the defined sums
        auto sum_up = [&]() {
            for (int t = tid; t < kT; t += NT) {
                const float d = __fsub_rn(wv[t], cb_value<CB>(found[t]));
                sh.cost[t] = __fmul_rn(d, d);
            }
            sync();
            if (tid == 0) {                        // a chain of 256 sums: about a microsecond
                float m = 0.0f;
#pragma unroll 1
                for (int t = 0; t < kT; t += 16) {
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = sh.cost[t + i];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        sh.cost[t + i] = m;
                        m = __fadd_rn(v[i], m);
                    }
                }
                sh.cost[kT] = m;
            }
            sync();
        };
        // The cost of steps `from` to `to` of a path on top of f, by the defined sums (each lane forms one step's square).
        auto add_up = [&](const uint16_t* states, int from, int to, float f) -> float {
            for (int k = from; k <= to; k += 32) {
                float d = 0.0f;
                if (k + lane <= to) d = __fsub_rn(wv[k + lane], cb_value<CB>(states[k + lane]));
                d = __fmul_rn(d, d);
                const int n = to - k + 1 < 32 ? to - k + 1 : 32;
#pragma unroll 8
                for (int i = 0; i < n; ++i) f = __fadd_rn(__shfl_sync(0xffffffffu, d, i), f);
            }
            return f;
        };
        // Whether the first group has taken so many trips, which it need not have at once where the second one is behind it.
        struct Follower {
            __device__ static long long clock() { return clock64(); }
            __device__ static void pause() { __nanosleep(200); }
            __device__ static bool all(bool x) {           // of the second group
                x = __all_sync(0xffffffffu, x);
                if constexpr (W == 1) return x;
                uint32_t every;
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred p, 2, %2, p;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(every) : "r"(uint32_t(x)), "n"(NT) : "memory");
                return every != 0;
            }
        } follower;
        // (The group waits for the next count that is told and remembers it: a barrier for that many trips.)
        int seen = 0;
        auto taken = [&](int trips) -> bool {
            if (who == 0 || trips <= seen) return true;
            const int told = (trips + sh.kTold - 1) / sh.kTold * sh.kTold;
            if (!handoff_wait(follower, sh.trips, told, a.hurry ? 0 : kWalkWaitCycles)) return false;
            seen = told;
            return true;
        };
        bool apart = false;                        // another path does not meet the one found as far as that is known
        int trips = 0;
        auto any_trip = [&](int tau, uint32_t e) -> uint32_t {
            sync();                                // what the warps still read of the trip before
            return tau > 0 ? row_trip(0, std::true_type{}, tau, e, (a.t_end - D - tau) / D) : first_trip(0, std::true_type{}, tau, e);
        };
        // Another path, from `e` before step t, the first of a trip: back to where it meets the path found, or to a beginning as good.
        // Returns the step before which they meet, or -1.
        auto follow = [&](uint32_t e, int t) -> int {
            while (t > lo && ++trips <= sh.kMaxTrips) {
                t -= D;
                const uint32_t whole = any_trip(t, e);
                if ((whole & kNear) || !taken((a.t_end - t + D - 1) / D)) return -1;
                for (int i = D - 1; i >= 0 && t + i >= 0; --i) {
                    const uint32_t s = (((whole >> (i * K)) & (Q - 1)) << SH) | e;
                    if (tid == 0) sh.other[t + i] = uint16_t(s);
                    e = s >> K;
                    if (t + i >= lo && e == uint32_t(found[t + i]) >> K) return t + i;
                }
            }
            if (lo > 0 && t <= lo) apart = true;
            return t <= 0 && !tied ? 0 : -1;
        };
        // Is the path found the defined one, against the other that meets it before step `met` and parts from it with step t?  first: the path
        // found is the one to take among equals.
        auto ahead = [&](const uint16_t* other, int met, int t, bool first) -> bool {
            if (!taken(sh.kAllTrips)) return false;
            sync();
            const float f = add_up(other, met, t, sh.cost[met]);
            sync();
            return f > sh.cost[t + 1] || (f == sh.cost[t + 1] && first);
        };
        // The same where they have not met down to step t0, the first of a trip.  What they start from is known within the bounds of A, and
        // rounded sums are monotonic: the path found is ahead if it is from its upper bound on against the other's lower one.
        auto surely_ahead = [&](const uint16_t* other, int t0, int t) -> bool {
            if (t0 <= 0) return false;
            sync();
            const float* const row = rows + size_t((a.t_end - D - t0) / D) * E;
            auto from = [&](const uint16_t* states, float sign) {
                const uint32_t x = uint32_t(states[t0]) >> K;
                const float m = load(row + (OTHER ? MR::other_pos(x) : MR::pos(x)));
                return add_up(states, t0, t, __fmaf_rn(sign * 0.5f, __fsub_rn(fused_limit(m, t0), m), m));     // (half of the limit: one side's bound)
            };
            const bool ahead = from(found, 1.0f) < from(other, -1.0f);
            sync();
            return ahead;
        };
        // The marked trips: every candidate within the limit on a node of the path, and its own path.
        auto settle_marks = [&]() -> bool {
            int left = sh.kMaxMarks;
            for (int m = 0; a.t_end - D * m > lo; ++m) {
                if (!taken(m + 2 < (a.t_end - lo + D - 1) / D ? m + 2 : sh.kAllTrips)) return false;      // (a trip is looked at during the next)
                if (*reinterpret_cast<volatile unsigned char*>(&sh.walker[0].mark[m]) == 0) continue;
                if (--left < 0) return false;
                const int first = a.t_end - D * (m + 1);
                const uint32_t root = first + D == a.t_end ? e_end : uint32_t(found[first + D]) >> K;
                const uint32_t whole = any_trip(first, root);
                const float* const row = first > 0 ? row_of(root, m) : nullptr;
                uint32_t p = 0;                    // the path's nodes of this trip, from the root down
                int n = 0;
                for (int d = D; d >= 1 && first + d - 1 >= lo; --d) {
                    const int t = first + d - 1;
                    const uint32_t M = 1u << ((D - d) * K), y = (p << (LB + d * K)) | (root >> ((D - d) * K));
                    auto child = [&](uint32_t q) {
                        const uint32_t x = q * M + p;
                        if (d >= 3) return val[wrp][d >= 3 ? d - 3 : 0][x];
                        if (d == 2) return val1[0][x];
                        return row != nullptr ? load(row + (OTHER ? MR::order(x) : x)) : start_metric((x << LB) | (root >> (K * D)));
                    };
                    auto value = [&](uint32_t q) { return candidate(emission(wv[t], q, y), child(q)); };
                    const uint32_t qp = (whole >> ((d - 1) * K)) & (Q - 1);
                    const float limit = fused_limit(value(qp), t + 1);
                    for (uint32_t q = 0; q < Q; ++q)
                        if (q != qp && !(value(q) > limit)) {
                            if (tid == 0 && n < sh.kMaxTodo) {
                                sh.todo[n][0] = uint32_t(t);
                                sh.todo[n][1] = (q << SH) | y;
                                sh.todo[n][2] = d >= 3 ? path[wrp][d >= 3 ? d - 3 : 0][q * M + p] : d == 2 ? path1[0][q * M + p] : 0u;
                            }
                            ++n;
                        }
                    p += qp * M;
                }
                sync();
                if (n > sh.kMaxTodo) return false;
                for (int i = 0; i < n; ++i) {
                    const int t = int(sh.todo[i][0]);
                    const uint32_t s0 = sh.todo[i][1], qs = sh.todo[i][2];
                    uint32_t x = s0 >> K;
                    int met = -1;
                    if (tid == 0) sh.other[t] = uint16_t(s0);
                    for (int k = t - first - 1; k >= 0 && met < 0 && first + k >= 0; --k) {
                        const uint32_t s = (((qs >> (k * K)) & (Q - 1)) << SH) | x;
                        if (tid == 0) sh.other[first + k] = uint16_t(s);
                        x = s >> K;
                        if (first + k >= lo && x == uint32_t(found[first + k]) >> K) met = first + k;
                    }
                    if (qs & kNear) return false;
                    const bool apart_before = apart;
                    if (met < 0) met = follow(x, first);
                    if (met < 0 && apart && !sums && surely_ahead(sh.other, a.t_end - D * ((a.t_end - lo + D - 1) / D), t)) {
                        apart = apart_before;
                        continue;
                    }
                    if (met < 0 || (sums && !ahead(sh.other, met, t, uint32_t(found[t]) >> SH < s0 >> SH))) return false;
                    sync();
                }
            }
            return true;
        };
        // The second walker's path, from the second edge that the pass may end with.
        auto settle_second = [&]() -> bool {
            const auto& its = sh.walker[FUSED ? 1 : 0];
            int met = lo > 0 ? -1 : 0;
            for (int t = kT - 32; t >= 0 && t + 31 >= lo; t -= 32) {
                const uint32_t same = __ballot_sync(0xffffffffu, t + lane >= lo && its.st[t + lane] >> K == found[t + lane] >> K);
                if (same != 0) {
                    met = t + 31 - __clz(int(same));
                    break;
                }
            }
            const int alone = (a.t_end - (met < 0 ? lo : met) + D - 1) / D;        // trips before they meet
            bool marked = false;
#pragma unroll
            for (int i = 0; i < 4; ++i) marked = marked || __ballot_sync(0xffffffffu, lane + 32 * i < alone && its.mark[lane + 32 * i] != 0) != 0;
            if (marked) return false;
            if (met >= 0) return !sums || ahead(its.st, met, kT - 1, e_end < e_second);
            if (surely_ahead(its.st, a.t_end - D * alone, kT - 1)) return true;
            apart = true;
            return false;
        };
        for (bool deep = false;; deep = true) {
            if (who == 0 || two) walk();
            if (two) both();                       // both have come as far
            if (two && who == 1) {
                both();
                if (sh.go_on == 0) return;
                lo = 0;
                continue;
            }
            const bool alone = !behind || deep;
            if (who == 0) {
                if (sums) sum_up();
                if (behind && !deep && tid == 0) handoff_publish(sh.trips, sh.kAllTrips);
                again = sums && !(sh.cost[kT] < kFusedMax);
                if (tied) again = again || uint32_t(found[0]) >> K != ov;
                else again = again || !(end_metric < kFusedMax) || __ballot_sync(0xffffffffu, key == kTooMany) != 0;
            }
            if (alone || who == 1) {
                if (two && !again) again = !settle_second();
                for (uint32_t left = two ? rivals & (rivals - 1) : rivals; left != 0 && !again; left &= left - 1) {    // more edges that the pass may end with
                    const uint32_t x = uint32_t(__shfl_sync(0xffffffffu, key, __ffs(int(left)) - 1)) & (E - 1);
                    const int met = follow(x, a.t_end);
                    again = met < 0 || (sums && !ahead(sh.other, met, kT - 1, e_end < x));
                }
                again = again || !settle_marks();
            }
            if (who == 1) {
                if (tid == 0) sh.verdict = (again ? sh.kOther : 0) | (apart ? sh.kApart : 0);
                both();
                return;
            }
            if (!alone) {
                both();
                again = again || (sh.verdict & sh.kOther);
                apart = apart || (sh.verdict & sh.kApart);
            }
            if (!again || !apart || sums) break;
            lo = 0;                                // walk on to the beginning and look again
            sums = true;
            apart = false;
            if (tid == 0) sh.go_on = 1;
            if (two) both();
            else sync();
        }
        if (two) {
            if (tid == 0) sh.go_on = 0;
            both();
        }
        if (again) {                               // no outputs: they may lie over the weights, which the sweep to come reads again
            if (tid == 0) a.again[atomicAdd(a.again_count, 1)] = a.first_tile + int(tile);
            return;
        }
        if (tied && tid == 0 && a.sse != nullptr) a.sse[tile] = sh.cost[kT];
    }
    if (tid == 0 && a.e_out != nullptr) a.e_out[tile] = int(st[t_off] >> K);     // a trip may have gone past step t_off
    emit_outputs<K, NT>(a, tile, st, t_off, a.t_end, tid);
    if constexpr (RING)
        if (lost) {
            if (lane == 0 && a.status != nullptr) atomicOr(a.status, 1u);
            // The copies that are still on their way: the next CTA on this SM must not find them in its shared memory.
            const long long t0 = clock64();
            for (int i = lost_at; tid == 0 && i < ring_rows && i < lost_at + Ring<K>::kRows; ++i)
                while (!mbar_try_wait(smem_u32(full + i % Ring<K>::kRows), uint32_t(i / Ring<K>::kRows) & 1u) && clock64() - t0 < kMbarWaitCycles) {}
        }
}

}  // namespace tcq
