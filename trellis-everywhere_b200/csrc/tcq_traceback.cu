// Traceback kernels.  tcq_walk_kernel is the walk over the metric rows of the cluster step kernel (tcq_walk.cuh);
// tcq_traceback_kernel walks the packed backpointers written by the single-CTA Viterbi step
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
#include "tcq_walk.cuh"

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

// One CTA of WalkShape<K>::W warps per tile, twice as many after fused sweeps (tcq_walk.cuh).
// (six CTAs on an SM: 888 tiles walk at once)
template <int K, int CB, bool OTHER, bool FUSED>
__global__ void __launch_bounds__(WalkShape<K>::W * (FUSED ? 64 : 32), FUSED ? 6 : 1) tcq_walk_kernel(const TracebackArgs a) {
    __shared__ WalkShared<K, FUSED> sh;
    walk_tile<K, CB, OTHER, FUSED, false>(a, blockIdx.x, blockIdx.x, sh);
}

// The same with rows fetched ahead (Ring): from three tiles on, whose rows are far enough away for it (one or two: 270 us a call at K = 3 without, 276
// with it; 3 / 8 / 24 / 74 tiles 288 / 289 / 391 / 506 without, 278 / 274 / 381 / 480 with it), until the bytes of all tiles bind: at K = 4 one tile
// per SM still gains (148 tiles 819 -> 791), at K = 3, whose rows are twice as long, it loses (771 -> 781), at K = 2 from 96 on (881 -> 893; 64 tiles 602 -> 594).
constexpr bool in_ring(int K, long long n) { return n >= 3 && n <= (K == 2 ? 74 : K == 3 ? 96 : 148); }
template <int K, int CB, bool OTHER>
__global__ void __launch_bounds__(WalkShape<K>::W * 32) tcq_walk_ring_kernel(const TracebackArgs a) {
    extern __shared__ __align__(128) float walk_ring[];
    __shared__ WalkShared<K, false> sh;
    walk_tile<K, CB, OTHER, false, false, true>(a, blockIdx.x, blockIdx.x, sh, walk_ring);
}

template <int K, int CB, bool OTHER>
cudaError_t launch_ring(const TracebackArgs& a, cudaStream_t stream) {
    static bool optin[64] = {};                    // per device ordinal: the shared-memory opt-in has been made
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64 || !optin[dev]) {
        if ((err = cudaFuncSetAttribute(tcq_walk_ring_kernel<K, CB, OTHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Ring<K>::kBytes))) != cudaSuccess) return err;
        if (dev >= 0 && dev < 64) optin[dev] = true;
    }
    tcq_walk_ring_kernel<K, CB, OTHER><<<unsigned(a.n), WalkShape<K>::W * 32, Ring<K>::kBytes, stream>>>(a);
    return cudaGetLastError();
}

template <int K, bool OTHER, bool FUSED>
cudaError_t launch_walk(const TracebackArgs& a, cudaStream_t stream) {
    if constexpr (!FUSED)
        if (in_ring(K, a.n)) switch (a.codebook) {
            case kCb1Mad:  return launch_ring<K, kCb1Mad, OTHER>(a, stream);
            case kCb3Inst: return launch_ring<K, kCb3Inst, OTHER>(a, stream);
            case kCbMcg:   return launch_ring<K, kCbMcg, OTHER>(a, stream);
            default: return cudaErrorInvalidValue;
        }
    const unsigned grid = unsigned(a.n), block = WalkShape<K>::W * (FUSED ? 64 : 32);
    switch (a.codebook) {
        case kCb1Mad:  tcq_walk_kernel<K, kCb1Mad, OTHER, FUSED><<<grid, block, 0, stream>>>(a); break;
        case kCb3Inst: tcq_walk_kernel<K, kCb3Inst, OTHER, FUSED><<<grid, block, 0, stream>>>(a); break;
        case kCbMcg:   tcq_walk_kernel<K, kCbMcg, OTHER, FUSED><<<grid, block, 0, stream>>>(a); break;
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
            case 2: return launch_walk<2, false, false>(a, stream);
            case 3: return a.fused ? launch_walk<3, true, true>(a, stream) : a.other_order ? launch_walk<3, true, false>(a, stream) : launch_walk<3, false, false>(a, stream);
            case 4: return a.fused ? launch_walk<4, false, true>(a, stream) : launch_walk<4, false, false>(a, stream);
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
