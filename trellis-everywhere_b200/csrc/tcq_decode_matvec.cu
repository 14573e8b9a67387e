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
// Bound: with many tile rows instruction issue (83 % of the slots at one right-hand side), not HBM; a weight costs about seven
// instructions to decode (window, multiply, and/xor, two conversions, addition) and half a packed multiply-add per right-hand side.  With
// few, the latency of a trip: words, x, products.  How the two are held is a matter of registers, which launch_m chooses by size.
// Largest relative error against fp64 on a 4096 x 4096 matrix 2.1e-7.
#include "tcq_traceback.cuh"

namespace tcq {

namespace {

constexpr int kMvWarps = 8;

// The 16-bit window of column col, out of a tile row's 15K+16 stream bits (v, normalised to start at bit 0).  Where windows of a word
// are whole bytes apart (K = 2, 4), three of them are cut out of one shifted word, as two bytes each in one instruction.
template <int K, int WN>
__device__ __forceinline__ uint32_t window(const uint32_t (&v)[WN], int col) {
    auto word_at = [&](int s) { return (s & 31) == 0 ? v[s >> 5] : __funnelshift_r(v[s >> 5], (s >> 5) + 1 < WN ? v[(s >> 5) + 1] : 0u, s & 31); };
    if constexpr (K == 3) {
        const int off = (15 - col) * K, s = off & 31;
        return (s + 16 <= 32 ? v[off >> 5] >> s : word_at(off)) & 0xFFFFu;
    } else {
        const int ph = (15 - col) % (8 / K), byte = (15 - col) / (8 / K), b = byte % 3;
        return __byte_perm(word_at(K * ph + 8 * (byte - b)), 0u, 0x4400 | (b + 1) << 4 | b);
    }
}

// RT: tile rows per CTA; two share the loads of x, which for several right-hand sides are as many instructions as the products.
// MB: CTAs that an SM must hold, i.e. the registers; x is then loaded ahead and a pair of weights lives from its decode to its products.
// MB = 0: the compiler's choice, weights decoded first.
template <int K, int CB, int M, int RT, int MB>
__global__ void __launch_bounds__(kMvWarps * 32, MB)
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
        auto x4 = [&](int j, int q) { return __ldg(reinterpret_cast<const ulonglong2*>(x + (long long)(j < m ? j : 0) * ldx + 16 * c) + q); };
        ulonglong2 xr[MB > 0 ? M : 1][4];
        if constexpr (MB > 0) {
#pragma unroll
            for (int j = 0; j < M; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) xr[j][q] = x4(j, q);
        }
        if constexpr (K == 3) {
#pragma unroll
            for (int t = 0; t < RT; ++t) {
#pragma unroll
                for (int j = 0; j + 1 < WN; ++j) v[t][j] = __funnelshift_r(v[t][j], v[t][j + 1], sh);
                v[t][WN - 1] >>= sh;
            }
        }
        auto pair = [&](int t, int p) {                      // columns 2p and 2p + 1 of tile row t
            return pack2(cb_value<CB>(window<K, WN>(v[t], 2 * p)), cb_value<CB>(window<K, WN>(v[t], 2 * p + 1)));
        };
        auto products = [&](int t, int j, f32x2 lo, f32x2 hi, const ulonglong2& xq) {
            acc[t][j] = fma2(lo, xq.x, acc[t][j]);
            acc[t][j] = fma2(hi, xq.y, acc[t][j]);
        };
        if constexpr (MB > 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                f32x2 val[RT][2];
#pragma unroll
                for (int t = 0; t < RT; ++t) { val[t][0] = pair(t, 2 * q); val[t][1] = pair(t, 2 * q + 1); }
#pragma unroll
                for (int j = 0; j < M; ++j)
#pragma unroll
                    for (int t = 0; t < RT; ++t) products(t, j, val[t][0], val[t][1], xr[j][q]);
            }
        } else {
            f32x2 val[RT][8];
#pragma unroll
            for (int t = 0; t < RT; ++t) {
                uint32_t win[16];                            // in stream order, word by word
#pragma unroll
                for (int p = 0; p < 16; ++p) {
                    const int col = K == 3 ? p : 15 - (p / (2 * K) + p % (2 * K) * (8 / K));
                    win[col] = window<K, WN>(v[t], col);
                }
#pragma unroll
                for (int p = 0; p < 8; ++p) val[t][p] = pack2(cb_value<CB>(win[2 * p]), cb_value<CB>(win[2 * p + 1]));
            }
#pragma unroll
            for (int j = 0; j < M; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const ulonglong2 xq = x4(j, q);
#pragma unroll
                    for (int t = 0; t < RT; ++t) products(t, j, val[t][2 * q], val[t][2 * q + 1], xq);
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

template <int K, int CB, int M, int RT, int MB>
void launch_mv(const uint32_t* packed, int tiles_out, int tiles_in, const float* x, long long ldx, int m, float* y, long long ldy,
               cudaStream_t stream) {
    tcq_decode_matvec_kernel<K, CB, M, RT, MB><<<(tiles_out + RT - 1) / RT, kMvWarps * 32, 0, stream>>>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy);
}

// Which form, by tile rows per SM, column tiles and rate; measured at 4 to 9496 tile rows of 4 to 768 tiles, MCG.  us for rows of 256 tiles,
// the compiler's choice of registers -> this one:
//   one right-hand side: loads ahead (47 registers) up to two rows an SM, where the latency of a trip is the bound (K = 3, 64 rows 10.3 -> 8.3), and
//     at K = 2, whose decode is shortest, always (9496 rows 174 -> 171).  With more rows other warps hide it, and need the registers (31; K = 4, 9496
//     rows 168, with loads ahead 178), and so do rows too narrow to give every warp a tile (K = 2, 9496 rows of 4 tiles 10.4, 12.4).
//   two: the compiler's choice (48; 64 are 10 to 19 % faster up to 148 rows and up to 7 % slower beyond); narrow rows, which are one trip or less, want more CTAs (K = 3, 9496 rows of 4 tiles 14.4 -> 12.3).
//   three and four: one row per CTA while all run at once, three CTAs per SM (K = 3, 64 rows 14.4 -> 10.3, 256 rows 16.4 -> 14.4), two rows from
//     there on (K = 4, 592 rows 32.8 -> 19.2; 9496 rows K = 2 / 3 / 4 294 / 318 / 331 -> 263 / 290 / 267).  At K = 2 between one and two rows
//     an SM two rows in one CTA, decoded first, are faster (256 rows 12.3, 13.1 with one).
template <int K, int CB>
cudaError_t launch_m(const uint32_t* packed, int tiles_out, int tiles_in, const float* x, long long ldx, int m, float* y,
                     long long ldy, cudaStream_t stream) {
    constexpr int kSms = 148;
    const bool narrow = tiles_in <= 2 * kMvWarps;
#define TCQ_MV(M, RT, MB) launch_mv<K, CB, M, RT, MB>(packed, tiles_out, tiles_in, x, ldx, m, y, ldy, stream)
    if (m == 1) {
        if ((K == 2 || tiles_out <= 2 * kSms) && !narrow) TCQ_MV(1, 1, 5);
        else TCQ_MV(1, 1, 0);
    } else if (m == 2) {
        if (narrow) TCQ_MV(2, 1, 6);
        else TCQ_MV(2, 1, 0);
    } else if (tiles_out > 3 * kSms) {
        TCQ_MV(4, 2, 3);
    } else if (K == 2 && tiles_out > kSms && tiles_out <= 2 * kSms) {
        if constexpr (K == 2) TCQ_MV(4, 2, 0);
    } else {
        TCQ_MV(4, 1, 3);
    }
#undef TCQ_MV
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
