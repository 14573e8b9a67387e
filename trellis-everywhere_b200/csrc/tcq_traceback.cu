// Traceback kernel: walks the packed backpointers written by the Viterbi step
// kernel from the last step to the first and emits, per tile, the state path and
// everything derived from it (symbols, packed code words, reconstruction).
//
// Replaces the host loops of src/trellis/qtip.py:189-196 and
// src/trellis/viterbi_triton.py:112-116 (256 tiny launches per pass) and fuses the
// exporter's bit packing (scripts/export_packed_8b.py:52-62).
//
// One warp per tile.  The walk itself is a chain of dependent loads:
//   q_t = bp[t][e_t],  s_t = (q_t << (16-K)) | e_t,  e_{t-1} = s_t >> K .
// Whatever q_t turns out to be, e_{t-1} is one of only Q edges that share the low
// bits e_t >> K, so lane j < Q fetches row t-1's entry for candidate q = j while
// the row-t load is still in flight, and the pick is a shuffle; one row further
// back there are Q*Q possible edges, which can be fetched the same way.  The
// dependent chain is thus one memory round trip per two (or three) steps.
// Afterwards the 32 lanes turn the 256 states held in shared memory into coalesced
// outputs.
#include <type_traits>

#include "tcq_traceback.cuh"

namespace tcq {

namespace {

constexpr int kWarpsPerCta = 4;

template <int K>
__device__ __forceinline__ uint32_t bp_entry(const unsigned char* row, uint32_t e) {
    // Edge e's K-bit argmin sits at bit e*K of the row (little endian).  Two byte
    // loads cover a field that straddles a byte; the second index is clamped so the
    // last entry of a row never reads past it.
    constexpr uint32_t Q = Geo<K>::Q, ROWB = Geo<K>::ROWB;
    const uint32_t bit = e * K;
    const uint32_t b0 = bit >> 3;
    const uint32_t b1 = b0 + 1 < ROWB ? b0 + 1 : b0;
    const uint32_t v = uint32_t(row[b0]) | (uint32_t(row[b1]) << 8);
    return (v >> (bit & 7)) & (Q - 1);
}

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

template <int K, int DEPTH>
__global__ void __launch_bounds__(kWarpsPerCta * 32) tcq_traceback_kernel(const TracebackArgs a) {
    using GE = Geo<K>;
    constexpr uint32_t Q = GE::Q, E = GE::E, ROWB = GE::ROWB;
    constexpr int SH = kL - K;                     // q sits above the edge bits
    constexpr int HB = kL - 2 * K;                 // predecessor edge = (q << HB) | (e >> K)

    __shared__ uint16_t st_all[kWarpsPerCta][kT];
    const int lane = threadIdx.x & 31;
    const int wrp = threadIdx.x >> 5;
    uint16_t* const st = st_all[wrp];
    const long long tile = (long long)blockIdx.x * kWarpsPerCta + wrp;
    if (tile >= a.n) return;                       // whole warp leaves together; no block-wide barrier below

    const unsigned char* const bp = a.bp + size_t(tile) * a.bp_steps * ROWB;
    uint32_t e;
    if (a.keys != nullptr) {            // argmin of the final metrics, left as per-CTA partial minima by the cluster kernel
        unsigned long long k = a.keys[tile * a.nkeys];
        for (int i = 1; i < a.nkeys; ++i) {
            const unsigned long long o = a.keys[tile * a.nkeys + i];
            k = o < k ? o : k;
        }
        e = uint32_t(k) & (E - 1);
    } else {
        e = uint32_t(a.e_start[tile]) & (E - 1);
    }
    const int t_off = kT - a.bp_steps;             // row r holds step t = r + t_off

    // ---- the walk: DEPTH rows per memory round trip ----
    // Row r's entry is one broadcast load.  Row r-1's entry can only sit at one of Q edges ((j1 << HB) | (e >> K)),
    // row r-2's at one of Q*Q ((j2 << HB) | (j1 << (HB-K)) | (e >> 2K)); lanes fetch all of them at once and the
    // picks are shuffles.  DEPTH = 3 shortens the dependent chain by a third but every trip then waits for the
    // slowest of 1 + Q + Q*Q scattered sectors instead of 1 + Q; measured, it pays only at K = 2 (16 candidates)
    // and only for small batches, where the walk is bound by latency rather than by sector traffic.
    static_assert(DEPTH == 2 || DEPTH == 3, "two or three rows per trip");
    constexpr int PER = 32 / int(Q) > 0 ? 32 / int(Q) : 1;      // level-2 candidates j2 covered by one load per lane
    constexpr int NL2 = (int(Q) + PER - 1) / PER;              // level-2 loads per lane
    int r = a.bp_steps - 1;
    for (; r >= DEPTH - 1; r -= DEPTH) {
        const uint32_t q1 = bp_entry<K>(bp + size_t(r) * ROWB, e);
        const uint32_t j1 = uint32_t(lane) & (Q - 1);
        const uint32_t e1c = (j1 << HB) | (e >> K);
        const uint32_t c1 = bp_entry<K>(bp + size_t(r - 1) * ROWB, e1c);          // lanes >= Q repeat lanes < Q
        uint32_t c2[NL2];
        if constexpr (DEPTH == 3) {
#pragma unroll
            for (int i = 0; i < NL2; ++i) {
                const uint32_t j2 = (uint32_t(lane) / Q + uint32_t(i * PER)) & (Q - 1);
                c2[i] = bp_entry<K>(bp + size_t(r - 2) * ROWB, (j2 << HB) | (e1c >> K));
            }
        }
        const uint32_t s1 = (q1 << SH) | e;
        const uint32_t e1 = s1 >> K;                                              // == candidate edge of lane q1
        const uint32_t q0 = __shfl_sync(0xffffffffu, c1, int(q1));
        const uint32_t s0 = (q0 << SH) | e1;
        e = s0 >> K;
        if (lane == 0) {
            st[r + t_off] = uint16_t(s1);
            st[r - 1 + t_off] = uint16_t(s0);
        }
        if constexpr (DEPTH == 3) {
            uint32_t pick = c2[0];                                                // q0 is the same in every lane
#pragma unroll
            for (int i = 1; i < NL2; ++i) pick = (q0 / PER == uint32_t(i)) ? c2[i] : pick;
            const uint32_t qm = __shfl_sync(0xffffffffu, pick, int(q1 + Q * (q0 % PER)));
            const uint32_t sm = (qm << SH) | e;
            if (lane == 0) st[r - 2 + t_off] = uint16_t(sm);
            e = sm >> K;
        }
    }
    for (; r >= 0; --r) {                          // the rows left over: one round trip each
        const uint32_t q = bp_entry<K>(bp + size_t(r) * ROWB, e);
        const uint32_t s = (q << SH) | e;
        if (lane == 0) st[r + t_off] = uint16_t(s);
        e = s >> K;
    }
    if (lane == 0 && a.e_out != nullptr) a.e_out[tile] = int(e);
    __syncwarp();
    emit_outputs<K, 32>(a, tile, st, t_off, kT, lane);
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

// OTHER: the rows' ancestors lie as in MetricRows::other_pos.
template <int K, int CB, bool OTHER>
__global__ void __launch_bounds__(WalkShape<K>::W * 32) tcq_walk_kernel(const TracebackArgs a) {
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
    __shared__ uint16_t st[kT];
    __shared__ float wv_pad[kT + 8];               // by step; the first trip may also look (in vain) at the steps before 0
    float* const wv = wv_pad + 8;
    __shared__ float val1[2][N1];                  // first level: minima and their q, double buffered over trips
    __shared__ uint32_t path1[2][N1];
    __shared__ float val[W][D > 2 ? D - 2 : 1][N2];       // levels 2 .. D-1, one copy per warp
    __shared__ uint32_t path[W][D > 2 ? D - 2 : 1][N2];
    const int tid = threadIdx.x, lane = tid & 31, wrp = tid >> 5;
    const long long tile = blockIdx.x;

    ForwardArgs fw{};
    fw.w = a.w;
    fw.w_add = a.w_add;
    fw.ld = a.ld;
    for (int i = tid; i < kT; i += NT) {
        int t;
        const float x = load_weight(fw, tile, i, t);
        wv[(t - a.roll) & (kT - 1)] = x;
    }
    if (tid < 8) wv_pad[tid] = 0.0f;
    uint32_t e;
    if (a.keys != nullptr) {            // argmin of the final metrics, left as per-CTA partial minima by the step kernel
        unsigned long long k = a.keys[tile * a.nkeys];
        for (int i = 1; i < a.nkeys; ++i) {
            const unsigned long long o = a.keys[tile * a.nkeys + i];
            k = o < k ? o : k;
        }
        e = uint32_t(k) & (E - 1);
    } else {
        e = uint32_t(a.e_start[tile]) & (E - 1);
    }
    const uint32_t ov = a.overlap != nullptr ? uint32_t(a.overlap[tile]) & (E - 1) : ~0u;
    // metric of edge x before step 0
    auto start_metric = [&](uint32_t x) { return a.overlap == nullptr ? 0.0f : x == ov ? 0.0f : __uint_as_float(kInfBits); };
    const int t_off = a.t_end - a.bp_steps;
    const float* const rows = a.rows + size_t(tile) * a.nrows * E;
    __syncthreads();

    // emission cost of state (q, y) at weight w
    auto emission = [](float w, uint32_t q, uint32_t y) {
        const float d = __fsub_rn(w, cb_value<CB>((q << SH) | y));
        return __fmul_rn(d, d);
    };
    int tau = a.t_end - D;                              // first of the trip's D steps
    // metric(q * N1, p): the metric of ancestor q * N1 + p before step tau.  kFirst: the trip that holds step 0; nodes before step 0 have the start
    // metric of their edge.
    auto trip = [&](int buf, auto first_c, auto metric) {
        constexpr bool kFirst = decltype(first_c)::value;
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

        // first level
#pragma unroll
        for (int i = 0; i < NPT; ++i) {
#pragma unroll
            for (int k = 0; k < QS; ++k) c1[i][k] = __fadd_rn(em1[i][k], c1[i][k]);
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
            if constexpr (kFirst)
                if (tau < 0) best = start_metric((uint32_t(p) << (LB + K)) | (e >> ((D - 1) * K)));
            val1[buf][p] = best;
            path1[buf][p] = qb;
        }
        if constexpr (W > 1) __syncthreads();
        else __syncwarp();
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
                for (uint32_t q = 0; q < Q; ++q) c[q] = __fadd_rn(em[d - 2][i][q], vin[q * uint32_t(M) + p]);
                float best = min_of<int(Q)>(c);
                const uint32_t qb = first_minimum<int(Q)>(c, best);
                if constexpr (kFirst)
                    if (tau + d - 1 < 0) best = start_metric((p << (LB + d * K)) | (e >> ((D - d) * K)));
                val[wrp][d - 2][p] = best;
                path[wrp][d - 2][p] = pin[qb * uint32_t(M) + p] | (qb << ((d - 1) * K));
            }
            __syncwarp();
            vin = val[wrp][d - 2];
            pin = path[wrp][d - 2];
        }
        // the root: one candidate per lane.  Candidates are non-negative (or not a number), so their bits order like the values.
        const float c = __fadd_rn(em_root, vin[uint32_t(lane) & (Q - 1)]);
        const float best = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(c)));
        const uint32_t eq = __ballot_sync(0xffffffffu, c == best);
        const uint32_t qb = eq != 0 ? uint32_t(__ffs(int(eq)) - 1) : Q - 1;
        const uint32_t whole = pin[qb] | (qb << ((D - 1) * K));       // q of step tau + i at bits i*K
#pragma unroll
        for (int i = D - 1; i >= 0; --i) {
            const uint32_t s = (((whole >> (i * K)) & (Q - 1)) << SH) | e;
            if (tid == 0 && (!kFirst || tau + i >= 0)) st[tau + i] = uint16_t(s);
            e = s >> K;
        }
    };
    int j = 0;
    for (; tau > 0 && tau + D > t_off; ++j, tau -= D) {
        const float* const row = rows + size_t(j) * E + (e >> (K * D)) * uint32_t(NA);     // the ancestors share the edge's bits above K*D
        trip(j & 1, std::false_type{}, [&](uint32_t pq, uint32_t p) { return __ldg(row + (OTHER ? MR::order(pq) | MR::order(p) : pq | p)); });
    }
    if (tau + D > t_off) {                         // tau <= 0
        const uint32_t g = e >> (K * D);
        trip(j & 1, std::true_type{}, [&](uint32_t pq, uint32_t p) { return start_metric(((pq + p) << LB) | g); });
    }
    __syncthreads();
    if (tid == 0 && a.e_out != nullptr) a.e_out[tile] = int(st[t_off] >> K);     // a trip may have gone past step t_off
    emit_outputs<K, NT>(a, tile, st, t_off, a.t_end, tid);
}

template <int K, bool OTHER>
cudaError_t launch_walk(const TracebackArgs& a, cudaStream_t stream) {
    const unsigned grid = unsigned(a.n), block = WalkShape<K>::W * 32;
    switch (a.codebook) {
        case kCb1Mad:  tcq_walk_kernel<K, kCb1Mad, OTHER><<<grid, block, 0, stream>>>(a); break;
        case kCb3Inst: tcq_walk_kernel<K, kCb3Inst, OTHER><<<grid, block, 0, stream>>>(a); break;
        case kCbMcg:   tcq_walk_kernel<K, kCbMcg, OTHER><<<grid, block, 0, stream>>>(a); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_traceback(int K, const TracebackArgs& a, cudaStream_t stream) {
    if (a.n <= 0) return cudaSuccess;
    const unsigned grid = unsigned((a.n + kWarpsPerCta - 1) / kWarpsPerCta);
    if (a.rows != nullptr) {
        switch (K) {
            case 2: return launch_walk<2, false>(a, stream);
            case 3: return a.other_order ? launch_walk<3, true>(a, stream) : launch_walk<3, false>(a, stream);
            case 4: return launch_walk<4, false>(a, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (K) {
        case 2:
            if (a.n <= 1024) tcq_traceback_kernel<2, 3><<<grid, kWarpsPerCta * 32, 0, stream>>>(a);
            else tcq_traceback_kernel<2, 2><<<grid, kWarpsPerCta * 32, 0, stream>>>(a);
            break;
        case 3: tcq_traceback_kernel<3, 2><<<grid, kWarpsPerCta * 32, 0, stream>>>(a); break;
        case 4: tcq_traceback_kernel<4, 2><<<grid, kWarpsPerCta * 32, 0, stream>>>(a); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace tcq
