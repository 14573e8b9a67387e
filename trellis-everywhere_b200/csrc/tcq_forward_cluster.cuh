// Viterbi step kernel, thread-block-cluster form: the whole codebook lives in registers, and the
// step keeps only the minima.
//
// The plain step kernel (tcq_forward.cuh) re-evaluates each of the 65536 codebook values on
// every step and records the argmin of every edge.  Here a cluster of C CTAs (C SMs) owns a group
// of tiles together and the 65536 states are divided among its C * NT threads, so each thread
// keeps its 65536 / (C * NT) codebook values in registers for the whole launch, and no argmin is
// formed at all: one edge of 2^(16-K) per step lies on the path that the traceback walks, so the
// argmin is worth having for that one only.  Every D-th step's path metrics go to HBM instead of every
// step's argmins, and the traceback re-derives the D argmins between two such rows from the
// Q^D metrics its edge can have come from (tcq_walk.cuh), with the same operations in the same
// order, so that the codes are those of the recorded argmins bit for bit.
//
// Three forms (StepForm).  What bounds a large batch is the fp32 pipe: subtract, square, add for each of 65536 states, tile and
// step, 29.3 clocks per eight candidates and warp in registers alone.  kFused makes the square and the sum one operation, 21.7
// clocks, and leaves it to the walk to find the path of the rounded sums (sweeps of 296 / 370 / 444 tiles: K = 3 566 / 697 / 806 -> 468 / 562 / 671 us,
// K = 4 559 / 696 / 817 -> 477 / 569 / 674; what limits it then is operands of packed instructions as well as issue: fewer
// instructions with the same operands are no faster).  kListed is the rounded form for the tiles that walks have listed, one at a time
// on two SMs or, where there are more than clusters, two, with the walks behind it in the same launch: 3 us when there is none.
//
//   * CTA r owns the butterflies h in [r * HN/C, (r+1) * HN/C): it needs the path metrics
//     old[q * HN + h] for all q (E/C values per tile, in ITS shared memory, layout [Q][HN/C])
//     and produces new[h * Q + l], a contiguous E/C slice of the next metric vector;
//   * every produced metric is consumed, one step later, by exactly one CTA of the cluster
//     (the owner of h' = (h * Q + l) mod HN), so each result is stored once, straight into the
//     consumer's shared memory: a local store or a distributed-shared-memory store
//     (cluster.map_shared_rank), never both;
//   * the stores are asynchronous (st.async) and each one reports its bytes to an mbarrier
//     in the consumer CTA; a CTA starts a step when the mbarrier of its input buffer has
//     counted the whole buffer.  No thread ever executes a memory fence, which matters because
//     a release fence on this chip waits for every outstanding store of the SM, including the
//     metric rows on their way to HBM;
//   * the only other synchronisation is write-after-read: nobody may store into a buffer that
//     a neighbour is still reading.  The hardware cluster barrier handles that with relaxed
//     arrives at the end of every step and a wait just before the next step's first store;
//   * the group's tiles form two sets that alternate, so both kinds of wait normally find
//     their condition already true: the other set's step has run in between.
//
// A metric row goes to HBM straight from the registers that hold the step's results, in the order
// that makes the ancestors of one edge contiguous (MetricRows::pos): a warp's store instruction
// covers whole 32-byte sectors.  Nothing in this kernel waits on memory written by another CTA except
// through the mbarriers and the cluster barrier, and every CTA of a cluster executes the same number of
// barrier phases.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "tcq_walk.cuh"

namespace tcq {

namespace cg = cooperative_groups;

// Hardware cluster barrier, split phase, no memory ordering: used only to keep stores away from
// buffers that are still being read.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_relaxed() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// ---- asynchronous distributed-shared-memory stores ----
// shared::cta address -> the same location in CTA `rank` of the cluster (shared::cluster address)
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// Stores of N = 1, 2 or 4 results, with the buffer's offset OFF as an immediate: to this CTA's shared memory, or
// asynchronously to another CTA's, reporting to its mbarrier at bar + BOFF.
template <int OFF, int N>
__device__ __forceinline__ void st_local(uint32_t dst, const float* v) {
    if constexpr (N == 4)
        asm volatile("st.shared.v4.f32 [%0+%5], {%1, %2, %3, %4};" ::"r"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "n"(OFF) : "memory");
    else if constexpr (N == 2)
        asm volatile("st.shared.v2.f32 [%0+%3], {%1, %2};" ::"r"(dst), "f"(v[0]), "f"(v[1]), "n"(OFF) : "memory");
    else
        asm volatile("st.shared.f32 [%0+%2], %1;" ::"r"(dst), "f"(v[0]), "n"(OFF) : "memory");
}
template <int OFF, int BOFF, int N>
__device__ __forceinline__ void st_remote(uint32_t dst, const float* v, uint32_t bar) {
    if constexpr (N == 4)
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0+%6], {%1, %2, %3, %4}, [%5+%7];"
                     ::"r"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar), "n"(OFF), "n"(BOFF) : "memory");
    else if constexpr (N == 2)
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0+%4], {%1, %2}, [%3+%5];"
                     ::"r"(dst), "f"(v[0]), "f"(v[1]), "r"(bar), "n"(OFF), "n"(BOFF) : "memory");
    else
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0+%3], %1, [%2+%4];"
                     ::"r"(dst), "f"(v[0]), "r"(bar), "n"(OFF), "n"(BOFF) : "memory");
}
// One predecessor's metrics of HB neighbouring butterflies, OFF bytes from src.
template <int HB>
__device__ __forceinline__ void ld_metrics(const float* src, float (&v)[HB]) {
    if constexpr (HB == 4) {
        const float4 x = *reinterpret_cast<const float4*>(src);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else if constexpr (HB == 2) {
        const float2 x = *reinterpret_cast<const float2*>(src);
        v[0] = x.x; v[1] = x.y;
    } else {
        v[0] = *src;
    }
}

// f(0), ..., f(N-1), each with its number as a compile-time constant.
template <int N, int I = 0, typename F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<N, I + 1>(f);
    }
}

// Work of one thread and step: NI items of HB neighbouring butterflies x LU of their successors, i.e. of runs of R = HB * LU
// consecutive edges.  LU = Q unless that would be more than the thread's 65536 / (C * NT) states.
template <int K, int C, int NT>
struct ClusterItem {
    static constexpr int STATES = kStates / (C * NT);
    static constexpr int Q = Geo<K>::Q;
    static constexpr int NB = STATES >= Q * Q ? STATES / (Q * Q) : 1;      // butterflies of a thread
    static constexpr int HB = NB > 2 ? 2 : NB;
    static constexpr int NI = NB / HB;
    static constexpr int LU = STATES >= Q * Q ? Q : STATES / Q;
    static constexpr int R = HB * LU;
    static constexpr int SV = R < 4 ? R : 4;               // successors per store (one float, float2 or float4)
    static constexpr int NWD = R / SV;                     // stores ("words") per item, tile and step
    static_assert(NI * HB * LU * Q == STATES, "a thread's states must form whole successors");
};

// Which CTA owns a butterfly, where in its rows of metrics the butterfly lies, and which run of edges a thread takes.
//
// In general CTA r owns butterflies [r * HN/C, (r+1) * HN/C).  The successors h*Q + l of butterfly h become butterflies
// (h*Q + l) mod HN, i.e. the bits of h move up by K, and the owner's bits are others every step: all but 1/C of the metrics cross
// between SMs.
template <int K, int C, int NT>
struct ClusterPlace {
    using IT = ClusterItem<K, C, NT>;
    static constexpr int Q = Geo<K>::Q, HN = Geo<K>::HN, HNC = HN / C, R = IT::R, NWD = IT::NWD;
    static constexpr int NCHUNK = Q / IT::LU;
    // Item i's butterflies lie HI * i after item 0's, and its successors are the predecessors DQ * i later of the same butterflies.
    static constexpr int HI = HNC / IT::NI, DQ = HI * Q / HN;
    static_assert(IT::NI == 1 || (HI * Q % HN == 0 && HI % (32 * R) == 0 && HI * Q % 16 == 0), "items must differ by constants");
    static constexpr int ITEM_EDGE = HI * Q, ITEM_SLOT = HI, ITEM_ROW = HI * Q >> MetricRows<K>::LB;
    // Address of word w of item i: one of NBASE held in registers, and a constant number of floats.
    static constexpr int NBASE = NWD, BASE_EDGE = IT::SV;  // base b is where edge b * BASE_EDGE after the thread's first goes
    __host__ __device__ static constexpr int base(int, int w) { return w; }
    __host__ __device__ static constexpr int offset(int i, int) { return i * DQ * HNC; }
    __device__ static uint32_t row_pos(uint32_t e) { return MetricRows<K>::pos(e); }
    static constexpr int kSwap = 0;                        // value k of an odd word lies at k ^ kSwap
    // Bytes of a tile's metrics that a CTA receives from others.  The owner of edge e = h*Q + l is bits of h that
    // start K below the rank's own: with C <= Q they are all bits of hl, and each CTA keeps 1/C of what it produces.  A larger
    // cluster's upper owner bits are the rank's lowest ones: a CTA keeps 1/Q if those agree with its uppermost bits, else nothing.
    __device__ static uint32_t remote_bytes(int rank) {
        constexpr int kUp = C > Q ? C / Q : 1;
        constexpr uint32_t all = uint32_t(Q * HNC) * 4;
        return all - (kUp == 1 || rank / (C / kUp) == rank % kUp ? all / (C / kUp) : 0u);
    }
    __device__ static int owner(int h) { return h / HNC; }
    // Slot of a butterfly in a row of metrics.  A thread's run of 8 or 16 edges is stored as 16-byte words; the warp's words
    // w of all lanes lie together, so that each store instruction writes contiguous memory (the network between SMs takes
    // half as long for it as for words 32 bytes apart), and the lane bits are flipped per w so that the loads of the next
    // step, which walk along the edges, still touch every bank once.
    __device__ static int slot(int h) {
        const int hl = h % HNC;
        if constexpr (R <= 4) {
            return hl;
        } else {
            const int word = hl >> 2, w = word % NWD, ln = (word / NWD) & 31;
            return (hl & ~(32 * R - 1)) | (w * 128 + ((ln ^ (w * (8 / NWD))) << 2)) | (hl & 3);
        }
    }
    __device__ static int butterfly(int rank, int sl) {    // the butterfly of a slot
        if constexpr (R <= 4) {
            return rank * HNC + sl;
        } else {
            const int word = (sl >> 2) & (32 * NWD - 1), w = word >> 5, ln = (word & 31) ^ (w * (8 / NWD));
            return rank * HNC + ((sl & ~(32 * R - 1)) | ((ln * NWD + w) << 2) | (sl & 3));
        }
    }
    // first edge of a thread's first run (chunk index fastest: a butterfly's items are neighbours)
    __device__ static int first_edge(int rank, int tid) { return (rank * HNC + tid / NCHUNK * IT::HB) * Q + tid % NCHUNK * IT::LU; }
};

// Two CTAs at K = 3: the owner is the majority of h9 h6 h3.  A step moves these bits up by one place and brings in one new one, so
// most majorities stay: 1/4 of the metrics cross between the SMs, where 1/2 do with an owner that is a bit of its own (or any sum of
// bits modulo two).  Sweep of 74 / 148 / 222 / 296 / 370 / 444 tiles: 230 / 363 / 469 / 596 / 727 / 828 -> 207 / 339 / 449 / 566 / 697 / 806 us;
// with nothing sent at all 183 / 330 / 433 / 556 / 688 / 801.  (At K = 2, majority of h11 h9 h7: 564 -> 568 us for 222 tiles, 561 with
// nothing sent: there the network does not bind.)
//   slot, from the top: number of the pattern h9 h6 h3 among those with its majority, h2, h8 h7 h5 h4, h1, h0 flipped by h2.
//   thread: the warp is the pattern's number, h8 and h0, so that a warp's stores all stay or all cross; the lanes are h7 h5 h4 h2 h1.
//   Loads of a warp then touch every bank once; its store instructions write two runs of 256 bytes, and whole sectors of a metric row
//   (MetricRows::other_pos).
template <> struct ClusterPlace<3, 2, 512> {
    using IT = ClusterItem<3, 2, 512>;
    static constexpr int ITEM_EDGE = 0, ITEM_SLOT = 0, ITEM_ROW = 0;          // one item
    static constexpr int NBASE = 1, BASE_EDGE = 0;
    __host__ __device__ static constexpr int base(int, int) { return 0; }
    __host__ __device__ static constexpr int offset(int, int w) { return w * 64; }
    __device__ static uint32_t row_pos(uint32_t e) { return MetricRows<3>::other_pos(e); }
    static constexpr int kSwap = 1;
    __device__ static uint32_t remote_bytes(int) { return uint32_t(Geo<3>::E) / 2 * 4 / 4; }
    __device__ static int pattern(int h) { return (h >> 3 & 1) | (h >> 5 & 2) | (h >> 7 & 4); }
    // 0 1 2 4 have one set bit at most, 3 5 6 7 two at least
    __device__ static int number(int p) { return 0x32130210 >> (4 * p) & 3; }
    __device__ static int numbered(int rank, int n) {      // a pattern's bits at their places in h
        const int p = (rank != 0 ? 0x7653 : 0x4210) >> (4 * n) & 7;
        return (p & 1) << 3 | (p & 2) << 5 | (p & 4) << 7;
    }
    __device__ static int owner(int h) { return 0xe8 >> pattern(h) & 1; }
    __device__ static int slot(int h) {
        return number(pattern(h)) << 7 | (h >> 2 & 1) << 6 | (h >> 7 & 3) << 4 | (h >> 4 & 3) << 2 | ((h & 3) ^ (h >> 2 & 1));
    }
    __device__ static int butterfly(int rank, int sl) {
        return numbered(rank, sl >> 7) | (sl >> 6 & 1) << 2 | (sl >> 4 & 3) << 7 | (sl >> 2 & 3) << 4 | ((sl & 3) ^ (sl >> 6 & 1));
    }
    __device__ static int first_edge(int rank, int tid) {
        const int ln = tid & 31, wp = tid >> 5;
        return (numbered(rank, wp >> 2) | (wp & 2) << 7 | (wp & 1) | (ln & 3) << 1 | (ln & 12) << 2 | (ln & 16) << 3) * 8;
    }
};

template <int K, int C, int GA, int GB>
constexpr size_t cluster_smem_bytes() {
    // per CTA: metrics [GA+GB tiles][2 buffers][E/C] fp32, weights [GA+GB][256] (twice each), reduction scratch and mbarriers
    return size_t(GA + GB) * 2 * (Geo<K>::E / C) * 4 + size_t(GA + GB) * kT * 8 + 64 * 8;
}

// GA, GB: tiles of the two sets that alternate (GB = 0: one set, for the smallest batches).
template <int K, int CB, int C, int GA, int GB, int NT, StepForm F>
__global__ void __launch_bounds__(NT, 1) tcq_forward_cluster_kernel(const ClusterArgs ca) {
    static_assert(F != StepForm::kListed || (GA == 1 && GB == 1 && C == 2), "each CTA walks a listed tile");
    using GE = Geo<K>;
    using MR = MetricRows<K>;
    using IT = ClusterItem<K, C, NT>;
    constexpr int Q = GE::Q, E = GE::E, HN = GE::HN;
    using PL = ClusterPlace<K, C, NT>;
    constexpr int NI = IT::NI, HB = IT::HB, LU = IT::LU, R = IT::R, SV = IT::SV, NBASE = PL::NBASE;
    constexpr int G = GA + GB;                     // tiles per cluster group
    constexpr int HNC = HN / C;                    // butterflies per CTA
    constexpr int EC = E / C;                      // metrics per tile held by a CTA
    static_assert(HNC / HB * (Q / LU) == NI * NT, "items must divide evenly over the threads");
    constexpr uint32_t MUL = CbLcg<CB>::MUL, ADD = CbLcg<CB>::ADD;
    const ForwardArgs& a = ca.f;

    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());

    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* const cost = reinterpret_cast<float*>(smem_raw);                          // [G][2][EC]
    float2* const wv = reinterpret_cast<float2*>(cost + size_t(G) * 2 * EC);         // [G][256], each weight twice (a packed operand)
    unsigned long long* const red = reinterpret_cast<unsigned long long*>(wv + G * kT);   // [32] reduction scratch
    unsigned long long* const mbar = red + 32;     // [2 sets][2 buffers] mbarriers counting the bytes of each metric buffer
    volatile unsigned int* const gave_up = reinterpret_cast<volatile unsigned int*>(red + 40);   // set by the first wait that runs out

    const int tid = threadIdx.x, lane = tid & 31;
    const bool constrained = a.overlap != nullptr;
    const float kInf = __uint_as_float(kInfBits);
    const f32x2 one2 = pack2(a.one, a.one);

    // ---- this thread's items: codebook values and destinations, fixed for the whole launch ----
    const int e0 = PL::first_edge(rank, tid);                    // first successor edge
    const int qn = e0 / HN;                                      // its role in the next step: predecessor qn of butterfly e0 % HN
    bool local[NBASE];                                           // which this CTA owns itself, or another
    uint32_t dst[NBASE];                                         // where the words go (tile 0, buffer 0)
#pragma unroll
    for (int b = 0; b < NBASE; ++b) {
        const int hn = (e0 + b * PL::BASE_EDGE) % HN;
        local[b] = PL::owner(hn) == rank;
        dst[b] = smem_u32(cost + qn * HNC + PL::slot(hn));
        if (!local[b]) dst[b] = map_to_rank(dst[b], PL::owner(hn));
    }
    const uint32_t dst_bar = map_to_rank(smem_u32(mbar), PL::owner(e0 % HN));     // the consumer's mbarriers (one CTA consumes all of a run)
    const float* const src = cost + PL::slot(e0 / Q);
    const uint32_t row_off = PL::row_pos(uint32_t(e0));            // in a metric row; a run's next edges follow NA apart
    f32x2 cbv[NI * R][Q / 2];                                    // codebook values of (q = 2j, 2j+1) into each run's edges
#pragma unroll
    for (int i = 0; i < NI * R; ++i) {
        const uint32_t xb = uint32_t(e0 + i / R * PL::ITEM_EDGE + i % R) * MUL + ADD;
#pragma unroll
        for (int j = 0; j < Q / 2; ++j)
            cbv[i][j] = pack2(cb_from_x<CB>(xb + uint32_t((2 * j) * E) * MUL), cb_from_x<CB>(xb + uint32_t((2 * j + 1) * E) * MUL));
    }

    // (a.n and not n in the rounded form, here and in `live` below, and the key loop once more for it: written as one for all forms the compiler orders
    // the rounded step at K = 2 differently and it takes 2 % longer, 222 / 444 tiles 574 / 1141 us instead of 554 / 1101)
    const long long n = F == StepForm::kListed ? (long long)*ca.list_count : a.n;
    const long long nclusters = gridDim.x / C;
    const long long cluster_id = blockIdx.x / C;
    const int per = F == StepForm::kListed && n <= nclusters ? 1 : G;      // tiles of a group: while each cluster has one at most, one alone
    const long long ngroups = ((F == StepForm::kRounded ? a.n : n) + per - 1) / per;

    float* row_tile0 = nullptr;                    // metric rows of the group's first tile
    int live = 0;                                  // tiles of the group that exist

    const uint32_t tile_bytes = PL::remote_bytes(rank);      // a tile's metrics that OTHER CTAs send each step
    bool timed_out = false;

    // All bytes of buffer b of set s have landed; then re-arm its mbarrier for the next use.
    // A wait that runs out is recorded (the launch's results are then invalid) and the thread
    // carries on; it never arrives at an mbarrier again, because an arrive on an mbarrier whose phase
    // cannot complete would underflow its arrival count, which is a hardware error.  The byte
    // counts do not depend on the data, so a wait can only run out through a programming error,
    // which the tests would show on every run; the limit exists so that even then nothing hangs.
    // (`last`: the re-arm for the phase that the end-of-group wait checks; the wait self-test
    // inflates exactly that one, so that its timeouts happen after the last store has landed.)
    auto wait_buffer = [&](int s, int b, uint32_t parity, bool last) __attribute__((always_inline)) {
        const uint32_t m = smem_u32(mbar + (2 * s + b));
        if (!mbar_wait(m, parity, gave_up)) timed_out = true;
        if (tid == 0 && !timed_out) mbar_expect(m, tile_bytes * uint32_t(s == 0 ? GA : GB) + (last ? uint32_t(a.inject_extra_bytes) : 0u));
    };

    // One add-compare-select step of tile set S (tiles T0 .. T0+GS-1 of the group), reading buffer CUR.
    // row >= 0: the results are that metric row.  first: nothing to wait for (the pass's first step).
    auto step_set = [&](auto set_c, auto cur_c, int t, uint32_t parity, int row, bool first, bool open_phase) __attribute__((always_inline)) {
        constexpr int S = decltype(set_c)::value, CUR = decltype(cur_c)::value;
        constexpr int T0 = S == 0 ? 0 : GA, GS = S == 0 ? GA : GB;
        if (!first) wait_buffer(S, CUR, parity, t == a.steps - 2);
        f32x2 w2[GS];
#pragma unroll
        for (int g = 0; g < GS; ++g) w2[g] = *reinterpret_cast<const f32x2*>(wv + (T0 + g) * kT + ((t + a.roll) & (kT - 1)));
        bool pending = open_phase;        // the barrier phase entered during the PREVIOUS step_set has not been closed yet
        // The codebook is in registers, so tiles need not share anything: they go one at a time.  The next one's metrics are
        // loaded ahead of this one's last store (which the compiler cannot move a load across): 3 % faster than at the
        // tile's own beginning.  How far ahead is a matter of registers: from the start where the item is a part of a
        // butterfly (K = 4), in the tile's second half with two tiles a set at K = 3 (558 us for 256 tiles, 577 from the
        // end), at the end otherwise (804 us for 444 tiles with three a set; 847 and spills in the second half).
        // With fused candidates at K = 3: in the second half for the shapes with three a set (444 tiles 672 us, from the start 704, from the
        // end 722), early with two (296 tiles 469 us, in the second half 488).
        // Alone on its two SMs a tile at K = 2 has them one edge earlier (74 tiles 264 us, 273 at the end; more tiles: no difference).
        constexpr int kAhead = LU < Q                                ? 0
                               : F == StepForm::kFused && K == 3     ? (GA == 3 ? 5 : 2)
                               : F == StepForm::kRounded && GS == 2 && K == 3 ? R * 5 / 8
                               : F == StepForm::kRounded && G == 1 && C == 2 && K == 2 ? R - 2
                                                                     : R - 1;
        float cin[2][Q][HB];
#pragma unroll
        for (int q = 0; q < Q; ++q) ld_metrics<HB>(src + (T0 * 2 + CUR) * EC + q * HNC, cin[0][q]);
        static_for<GS * NI>([&](auto gc) __attribute__((always_inline)) {
            constexpr int gi = decltype(gc)::value, g = gi / NI, it = gi % NI, NX = gi + 1;
            constexpr int OUT = ((T0 + g) * 2 + (CUR ^ 1)) * EC;
            float outv[R];
            static_for<R>([&](auto ic) __attribute__((always_inline)) {
                constexpr int i = decltype(ic)::value;
                float c[Q];
#pragma unroll
                for (int j = 0; j < Q / 2; ++j) {
                    if constexpr (F == StepForm::kFused) {
                        const f32x2 from = pack2(cin[gi & 1][2 * j][i / LU], cin[gi & 1][2 * j + 1][i / LU]);
                        unpack2(fused_cost2(w2[g], cbv[it * R + i][j], from), c[2 * j], c[2 * j + 1]);
                    } else {
                        unpack2(cand_cost2(w2[g], cbv[it * R + i][j], pack2(cin[gi & 1][2 * j][i / LU], cin[gi & 1][2 * j + 1][i / LU]), one2), c[2 * j], c[2 * j + 1]);
                    }
                }
                if constexpr (i == kAhead && NX < GS * NI) {
#pragma unroll
                    for (int q = 0; q < Q; ++q) ld_metrics<HB>(src + ((T0 + NX / NI) * 2 + CUR) * EC + NX % NI * PL::ITEM_SLOT + q * HNC, cin[NX & 1][q]);
                }
                outv[i] = min_tree<Q>(c);
                if constexpr (gi == GS * NI - 1 && i == R - LU) {
                    // Every input of this step has been loaded AND used (the first successor of the
                    // last tile's last butterfly consumed all of its predecessors' metrics), so this
                    // thread no longer reads the input buffers: tell the cluster, well before anyone
                    // needs to know.  (The barrier's phases are sequential: close the previous one first.)
                    if (pending) cluster_wait_relaxed();
                    pending = false;
                    cluster_arrive_relaxed();
                }
                if constexpr (i % SV == SV - 1) {
                    // Results leave as soon as a store's worth is ready.
                    // Write-after-read: the buffer written now was read by every CTA one step of this
                    // set ago; the barrier phase that every thread entered during the previous
                    // step_set proves it, and it is closed before the first store.
                    if (pending) cluster_wait_relaxed();
                    pending = false;
                    constexpr int wd = i / SV, b = PL::base(it, wd), AT = (OUT + PL::offset(it, wd)) * 4;
                    const float* v = outv + (i + 1 - SV);
                    float swapped[SV];
                    if constexpr (PL::kSwap != 0 && wd % 2 != 0) {
#pragma unroll
                        for (int k = 0; k < SV; ++k) swapped[k] = v[k ^ PL::kSwap];
                        v = swapped;
                    }
                    if (local[b]) st_local<AT, SV>(dst[b], v);
                    else st_remote<AT, (2 * S + (CUR ^ 1)) * 8, SV>(dst[b], v, dst_bar);
                }
            });
            if (row >= 0 && T0 + g < live) {
                float* const rp = row_tile0 + (size_t(T0 + g) * ca.nrows + row) * E + row_off + it * PL::ITEM_ROW;
#pragma unroll
                for (int i = 0; i < R; ++i) rp[i * MR::NA] = outv[i];
            }
        });
        __syncwarp();                 // this warp's local stores, then its arrival (which releases them to the CTA)
        if (lane == 0 && !timed_out) mbar_arrive(smem_u32(mbar + 2 * S + (CUR ^ 1)));
    };

    if ((a.flags & kFwdResetStatus) && blockIdx.x == 0 && tid == 0 && a.status != nullptr) atomicExch(a.status, 0u);
    if (F == StepForm::kFused && (a.flags & kFwdResetCounts) && blockIdx.x == 0 && tid < 2) ca.counts[tid] = 0;

    // ---- mbarriers: the arrivals of the re-arming thread and of every warp (its local stores) plus the bytes of the remote
    //      stores, per phase ----
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mbar_init(smem_u32(mbar + i), 1 + NT / 32);
        mbar_fence_init();
        *gave_up = 0u;
    }
    cluster.sync();                      // every CTA's mbarriers exist before anyone can signal them
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < (GB > 0 ? 4 : 2); ++i) mbar_expect(smem_u32(mbar + i), tile_bytes * uint32_t(i < 2 ? GA : GB));
    }

    for (long long grp = cluster_id; grp < ngroups; grp += nclusters) {
        const long long tile0 = grp * per;
        const long long slot0 = F == StepForm::kListed ? cluster_id * G : tile0;       // whose rows and keys
        live = F != StepForm::kRounded ? int(n - tile0 < per ? n - tile0 : per) : int(a.n - tile0 < G ? a.n - tile0 : G);
        const bool second = F != StepForm::kListed || live > 1;        // whether set 1 has a tile
        auto tile_at = [&](int g) -> long long {
            if constexpr (F == StepForm::kListed) return ca.list[tile0 + g];
            else return tile0 + g;
        };
        row_tile0 = ca.rows + size_t(slot0) * ca.nrows * E;
        // ---- weights and initial metrics (src/trellis/qtip.py:161-165) ----
        for (int i = tid; i < G * kT; i += NT) {
            int t = i & 255;
            const float x = (i >> 8) < live ? load_weight(a, tile_at(i >> 8), i & 255, t) : 0.0f;
            wv[(i & ~255) | t] = make_float2(x, x);
            if ((a.flags & kFwdCheckFinite) && !isfinite(x) && rank == 0 && a.status != nullptr) atomicOr(a.status, 2u);   // reported, never trapped on
        }
        {
            const float init = constrained ? kInf : 0.0f;
            for (int i = tid; i < G * EC; i += NT) cost[(size_t(i / EC) * 2) * EC + (i % EC)] = init;
        }
        __syncthreads();
        if (constrained && tid < G) {
            const int ov = (tid < live ? a.overlap[tile_at(tid)] : 0) & (E - 1);
            const int qo = ov / HN, ho = ov % HN;                 // metric of edge ov is predecessor qo of butterfly ho
            if (PL::owner(ho) == rank) cost[(size_t(tid) * 2) * EC + qo * HNC + PL::slot(ho)] = 0.0f;
        }
        cluster.sync();   // every CTA's buffers are initialised before anyone stores into them

        // The two tile sets alternate; every step_set waits for its input buffer's bytes, computes,
        // waits for the previous step_set's barrier phase before its first store, stores, arrives.
        // (two steps per trip, so that the buffer index is a constant in every instance of step_set)
        // A group's waits on each buffer are an even number (steps / 2), so the phase parities start every group at 0 and
        // alternate from trip to trip.
        using C0 = std::integral_constant<int, 0>;
        using C1 = std::integral_constant<int, 1>;
        step_set(C0{}, C0{}, 0, 0u, MR::row_after(0, a.steps, ca.nrows), true, false);
        uint32_t ph = 0;                                  // parity of the waits on buffer 1 of this trip
#pragma unroll 1
        for (int t = 0; t < a.steps; t += 2) {
            const int row1 = MR::row_after(t + 1, a.steps, ca.nrows);
            if constexpr (GB > 0) if (second) step_set(C1{}, C0{}, t, ph ^ 1u, MR::row_after(t, a.steps, ca.nrows), t == 0, true);
            step_set(C0{}, C1{}, t + 1, ph, row1, false, true);
            if constexpr (GB > 0) if (second) step_set(C1{}, C1{}, t + 1, ph, row1, false, true);
            if (t + 2 < a.steps) step_set(C0{}, C0{}, t + 2, ph, MR::row_after(t + 2, a.steps, ca.nrows), false, true);
            ph ^= 1u;
        }
        cluster_wait_relaxed();             // closes the phase opened by the last step_set
        wait_buffer(0, 0, 1u, false);       // the last step wrote the final metrics into buffer 0
        if constexpr (GB > 0) if (second) wait_buffer(1, 0, 1u, false);
        __syncthreads();

        // ---- final metrics live in buffer 0 (an even number of steps), layout [Q][HNC] = edges q*HN + rank*HNC + hl ----
        if (ca.keys != nullptr) {
            for (int g = 0; g < G; ++g) {
                const float* fv = cost + (size_t(g) * 2) * EC;
                unsigned long long key = ~0ull;
                if constexpr (F == StepForm::kFused) {     // (unrolled, it takes registers from the step: 370 tiles at K = 3 586 us instead of 567)
                    auto take = [&](int i) {
                        const unsigned edge = unsigned(i / HNC) * HN + PL::butterfly(rank, i % HNC);
                        const unsigned long long k2 = (static_cast<unsigned long long>(__float_as_uint(fv[i])) << 32) | edge;
                        key = k2 < key ? k2 : key;
                    };
#pragma unroll 1
                    for (int i = tid; i < EC; i += NT) take(i);
                } else {
                    for (int i = tid; i < EC; i += NT) {
                        const unsigned edge = unsigned(i / HNC) * HN + PL::butterfly(rank, i % HNC);
                        const unsigned long long k2 = (static_cast<unsigned long long>(__float_as_uint(fv[i])) << 32) | edge;
                        key = k2 < key ? k2 : key;
                    }
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
                    key = o < key ? o : key;
                }
                if (lane == 0) red[tid >> 5] = key;
                __syncthreads();
                if (tid < 32) {
                    unsigned long long k2 = tid < NT / 32 ? red[tid] : ~0ull;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) {
                        const unsigned long long o = __shfl_xor_sync(0xffffffffu, k2, off);
                        k2 = o < k2 ? o : k2;
                    }
                    if (F != StepForm::kFused && tid == 0 && g < live) ca.keys[(slot0 + g) * C + rank] = k2;
                    if (F == StepForm::kFused && tid < kFusedKeys) red[48 + tid] = tid == 0 ? k2 : ~0ull;
                    if (F == StepForm::kFused && tid == 0) red[56] = 0;
                }
                __syncthreads();
                if constexpr (F == StepForm::kFused) {     // and who may be below it by the defined sums
                    const float limit = fused_limit(__uint_as_float(unsigned(red[48] >> 32)), kT);
#pragma unroll 1
                    for (int i = tid; i < EC; i += NT)
                        if (!(fv[i] > limit)) {
                            const unsigned edge = unsigned(i / HNC) * HN + PL::butterfly(rank, i % HNC);
                            if (edge == unsigned(red[48])) continue;
                            const unsigned at = atomicAdd(reinterpret_cast<unsigned*>(red + 56), 1u) + 1;
                            if (at < kFusedKeys) red[48 + at] = (static_cast<unsigned long long>(__float_as_uint(fv[i])) << 32) | edge;
                        }
                    __syncthreads();
                    if (tid < kFusedKeys && g < live)
                        ca.keys[((slot0 + g) * C + rank) * kFusedKeys + tid] = tid == kFusedKeys - 1 && *reinterpret_cast<unsigned*>(red + 56) >= kFusedKeys ? kTooMany : red[48 + tid];
                    __syncthreads();
                }
            }
        }
        if (a.final_cost != nullptr && constrained && tid < live) {
            const int ov = a.overlap[tile_at(tid)] & (E - 1);
            const int qo = ov / HN, ho = ov % HN;
            if (PL::owner(ho) == rank) a.final_cost[tile_at(tid)] = cost[(size_t(tid) * 2) * EC + qo * HNC + PL::slot(ho)];
        }
        if constexpr (F == StepForm::kListed) {
            __shared__ WalkShared<K, false> walk_shared;
            __threadfence();                        // the rows and keys of every CTA, before one of them walks
            cluster.sync();
            if (rank < live && tid < WalkShape<K>::W * 32) walk_tile<K, CB, K == 3 && C == 2, false, true>(ca.walk, tile_at(rank), slot0 + rank, walk_shared);
            __syncwarp();
        }
        cluster.sync();   // nobody may start re-initialising while a neighbour still reads or is written to
    }
    if (timed_out && a.status != nullptr) atomicOr(a.status, 1u);
}

}  // namespace tcq
