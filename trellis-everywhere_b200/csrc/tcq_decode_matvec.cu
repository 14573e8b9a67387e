// Decode-matvec: y = Zq x straight from packed trellis codes, Zq never materialised.
//
// The consumer side of the packed format: what the reference's runtime does in its
// DECODE_MATMUL shader (web/kernels.js:105-128), where one thread walks a whole output
// row and decodes every weight with wz() (window at stream bit (255-t)*K of tile
// (row/16)*tiles_in + col/16, t = (row%16)*16 + col%16).  The incoherence-processing
// fold around it (web/packed.js:163-182) stays with the caller.
//
// Work split here: one CTA per tile row (16 output rows; two for several right-hand sides, see launch_m), eight warps striding over
// the column tiles.  A half-warp owns one tile per iteration, lane i its row i: the 16
// weights of that row sit in 15K+16 consecutive stream bits, fetched as two or three
// words, and every window is a compile-time cut of those.  Weights and x meet as pairs of neighbouring columns in packed
// multiply-adds.  Partial sums (of even and odd columns) stay in registers; the two half-warps meet in one shuffle and the eight
// warps in shared memory, in a fixed order, so results are reproducible run to run.
//
// Bound: instruction issue (83 % of the slots at one right-hand side), not HBM.  A weight costs about seven instructions to decode
// (window, multiply, and/xor, two conversions, addition) and half a packed multiply-add per
// right-hand side.  151936 x 4096, before -> now: one right-hand side K = 2 191 -> 177 us, K = 3 203 -> 193, K = 4 192 -> 170; two
// 217 -> 205, 233 -> 221, 225 -> 205; four 322 -> 291, 318 -> 314, 327 -> 320.  Largest relative error against fp64 on a 4096 x 4096
// matrix 2.9e-7 -> 2.1e-7 (two partial sums).  Fetching the next trip's words ahead and x in shared memory gave nothing (four right-hand sides,
// K = 4: 342 and 314 us).
#include "tcq_traceback.cuh"

namespace tcq {

namespace {

constexpr int kMvWarps = 8;

// The 16 weights of a tile row from its 15K+16 stream bits (v, normalised to start at bit 0), as pairs of neighbouring columns.
// A window is cut out of a word as two bytes, in one instruction, where its offset is a whole number of bytes; words are shifted to make it
// so, one shift for the (at most three) windows of a word that are a byte apart.  At K = 3 no two windows of a word are.
template <int K, int CB, int WN>
__device__ __forceinline__ void decode_row(const uint32_t (&v)[WN], f32x2 (&val)[8]) {
    auto word_at = [&](int s) { return (s & 31) == 0 ? v[s >> 5] : __funnelshift_r(v[s >> 5], (s >> 5) + 1 < WN ? v[(s >> 5) + 1] : 0u, s & 31); };
    uint32_t win[16];
    if constexpr (K == 3) {
#pragma unroll
        for (int col = 0; col < 16; ++col) {
            const int off = (15 - col) * K, s = off & 31;
            win[col] = (s + 16 <= 32 ? v[off >> 5] >> s : word_at(off)) & 0xFFFFu;
        }
    } else {
#pragma unroll
        for (int ph = 0; ph < 8 / K; ++ph)                     // windows ph, ph + 8/K, ...: eight bits apart
#pragma unroll
            for (int a = 0; a < 2 * K; a += 3) {
                const uint32_t u = word_at(K * ph + 8 * a);
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    if (a + b < 2 * K) win[15 - (ph + (a + b) * (8 / K))] = __byte_perm(u, 0u, 0x4400 | (b + 1) << 4 | b);
            }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) val[c] = pack2(cb_value<CB>(win[2 * c]), cb_value<CB>(win[2 * c + 1]));
}

// RT: tile rows per CTA.  Two share the loads of x, which for several right-hand sides are as many instructions as the products.
template <int K, int CB, int M, int RT>
__global__ void __launch_bounds__(kMvWarps * 32)
tcq_decode_matvec_kernel(const uint32_t* __restrict__ packed, int tiles_out, int tiles_in, const float* __restrict__ x, long long ldx,
                         int m, float* __restrict__ y, long long ldy) {
    constexpr int NW = Geo<K>::NWORDS;
    constexpr int WN = (K == 2) ? 2 : 3;                    // words that hold one tile row's 15K+16 bits
    __shared__ float red[kMvWarps][M * RT][16];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = lane & 15, half = lane >> 4;
    const uint32_t sb = uint32_t(240 - 16 * i) * K;          // stream bit of this row's last weight (t = 16i + 15)
    const uint32_t word0 = sb >> 5, sh = sb & 31;            // sh is 0, or 16 for even rows at K = 3
    const int row0 = int(blockIdx.x) * RT;
    const uint32_t* row_base[RT];
#pragma unroll
    for (int t = 0; t < RT; ++t) row_base[t] = packed + (long long)(row0 + t < tiles_out ? row0 + t : row0) * tiles_in * NW;

    f32x2 acc[RT][M];                                        // even and odd columns
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
        for (int j = 0; j < M; ++j) acc[t][j] = 0ull;

    for (int c = 2 * warp + half; c < tiles_in; c += 2 * kMvWarps) {
        uint32_t v[RT][WN];
#pragma unroll
        for (int t = 0; t < RT; ++t) {
            const uint32_t* const p = row_base[t] + (long long)c * NW;
#pragma unroll
            for (int j = 0; j < WN; ++j) {
                const uint32_t wi = word0 + j;
                v[t][j] = __ldg(p + (wi >= uint32_t(NW) ? wi - NW : wi));       // the first row's window wraps to word 0
            }
        }
        f32x2 val[RT][8];
#pragma unroll
        for (int t = 0; t < RT; ++t) {
            if constexpr (K == 3) {
#pragma unroll
                for (int j = 0; j + 1 < WN; ++j) v[t][j] = __funnelshift_r(v[t][j], v[t][j + 1], sh);
                v[t][WN - 1] >>= sh;
            }
            decode_row<K, CB>(v[t], val[t]);
        }
#pragma unroll
        for (int j = 0; j < M; ++j) {
            const ulonglong2* const xp = reinterpret_cast<const ulonglong2*>(x + (long long)(j < m ? j : 0) * ldx + 16 * c);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2 x4 = __ldg(xp + q);
#pragma unroll
                for (int t = 0; t < RT; ++t) {
                    acc[t][j] = fma2(val[t][2 * q], x4.x, acc[t][j]);
                    acc[t][j] = fma2(val[t][2 * q + 1], x4.y, acc[t][j]);
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
        for (int j = 0; j < M; ++j) {
            float a, b;
            unpack2(acc[t][j], a, b);
            a += b;
            a += __shfl_xor_sync(0xFFFFFFFFu, a, 16);
            if (half == 0) red[warp][t * M + j][i] = a;
        }
    __syncthreads();
    if (threadIdx.x < 16 * M * RT) {
        const int tj = threadIdx.x >> 4, r = threadIdx.x & 15, t = tj / M, j = tj % M;
        float s = red[0][tj][r];
#pragma unroll
        for (int w = 1; w < kMvWarps; ++w) s += red[w][tj][r];
        if (j < m && row0 + t < tiles_out) y[(long long)j * ldy + 16ll * (row0 + t) + r] = s;
    }
}

template <int K, int CB, int M, int RT>
void launch_mv(const uint32_t* packed, int tiles_out, int tiles_in, const float* x, long long ldx, int m, float* y, long long ldy,
               cudaStream_t stream) {
    tcq_decode_matvec_kernel<K, CB, M, RT><<<(tiles_out + RT - 1) / RT, kMvWarps * 32, 0, stream>>>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy);
}

// Two tile rows per CTA for four right-hand sides, where the loads of x (16 of 128 bits a tile, four passes through L1 each)
// were the bound: from two CTAs per SM on, and at K = 2, whose decode is shortest, always.  151936 x 4096, one row -> two:
// K = 2 318 -> 291 us, K = 3 345 -> 314, K = 4 339 -> 320; 12288 x 4096: 43 -> 27, 34 -> 39, 33 -> 36 (768 tile rows: one row there
// at K = 3 and 4); 4096 x 4096: 18.6 -> 12.5, 16.5 -> 20.4, 16.5 -> 17.6.
// One and two right-hand sides are bound by instruction issue and gain nothing (K = 3: 193 -> 194, 221 -> 232 us).
template <int K, int CB>
cudaError_t launch_m(const uint32_t* packed, int tiles_out, int tiles_in, const float* x, long long ldx, int m, float* y,
                     long long ldy, cudaStream_t stream) {
    if (m == 1)                            launch_mv<K, CB, 1, 1>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
    else if (m == 2)                       launch_mv<K, CB, 2, 1>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
    else if (K == 2 || tiles_out >= 2048)  launch_mv<K, CB, 4, 2>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
    else                                   launch_mv<K, CB, 4, 1>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
    return cudaGetLastError();
}

template <int K>
cudaError_t launch_cb(int codebook, const uint32_t* packed, int tiles_out, int tiles_in, const float* x, long long ldx, int m,
                      float* y, long long ldy, cudaStream_t stream) {
    switch (codebook) {
        case kCb1Mad:  return launch_m<K, kCb1Mad>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
        case kCb3Inst: return launch_m<K, kCb3Inst>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
        case kCbMcg:   return launch_m<K, kCbMcg>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream);
        default:       return cudaErrorInvalidValue;
    }
}

}  // namespace

// y[j][row] = sum_col Zq[row][col] * x[j][col] for j < m; right-hand sides go four at a time.
cudaError_t launch_decode_matvec(const uint32_t* packed, long long n_out, long long k_in, int K, int codebook, const float* x,
                                 long long ldx, int m, float* y, long long ldy, cudaStream_t stream) {
    if (n_out <= 0 || k_in <= 0 || m <= 0) return cudaSuccess;
    const int tiles_out = int(n_out / 16), tiles_in = int(k_in / 16);
    for (int j0 = 0; j0 < m; j0 += 4) {
        const int mj = m - j0 < 4 ? m - j0 : 4;
        cudaError_t err;
        switch (K) {
            case 2: err = launch_cb<2>(codebook, packed, tiles_out, tiles_in, x + j0 * ldx, ldx, mj, y + j0 * ldy, ldy, stream); break;
            case 3: err = launch_cb<3>(codebook, packed, tiles_out, tiles_in, x + j0 * ldx, ldx, mj, y + j0 * ldy, ldy, stream); break;
            case 4: err = launch_cb<4>(codebook, packed, tiles_out, tiles_in, x + j0 * ldx, ldx, mj, y + j0 * ldy, ldy, stream); break;
            default: return cudaErrorInvalidValue;
        }
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

}  // namespace tcq
