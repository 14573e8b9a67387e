// Incoherence processing around the codec on the device (src/trellis/qtip.py:199-268).
//
// Forward (IPContext.__init__, qtip.py:238-260):
//   z = w * sv[:,None] * su[None,:]
//   out_s = rms over each row, clamped at 1e-8, divided by its mean;   z = Hb_rows(z / out_s[:,None])
//   in_s  = rms over each column, same treatment;                      z = Hb_cols(z / in_s[None,:])
//   scale = rms(z) / cb_rms;                                           z = z / scale
// Restore (qtip.py:262-268) undoes the steps in reverse order.  Hb is the block-diagonal
// orthonormal Sylvester-Hadamard transform with blocks of the largest power of two, at most
// 128, that divides the axis (qtip.py:208-223).  The reference multiplies by the dense
// [128,128] matrix; here a CTA takes a 128 x 128 block of the matrix through fast Walsh-Hadamard
// transforms on both axes at once, 64 values per thread in registers, so that each direction
// reads its matrix once and writes it once.  Transformed weights go straight to and come straight from the encoder's
// tile order (tile = (row/16)*(k/16) + col/16, t = (row%16)*16 + col%16, qtip.py:288).
//
// Forward is three reads and one write of 4 bytes per weight: row sums, column sums after the transform down the rows (which is done again
// in the blocks rather than written and read back; the second read starts at the matrix' end, where the first left it in L2), blocks.  Restore is one
// read and one write.  12288 x 4096 (201 MB): forward 220 us (rows 35, their mean 8, columns 53 + 4 + 8, blocks 102), restore 87 us; with a kernel
// per transform and an intermediate matrix 240 and 167.
//
// Every product and sum is rounded where the recipe has it (but divisions by the scale vectors are multiplications by their reciprocals,
// one rounding more than the reference's division), every stage of a transform in natural order, and every reduction runs in an order of
// its own definition, whatever the launch, without atomics.  A weight that moves by an ulp may fall to another code, and the packed bytes
// of a matrix with it, so all of that is part of the result (tests/test_gpu_ip_blocks.py states it bit for bit).  Column sums taken from w itself, which an orthonormal
// transform allows, one factor for two and another order of stages would save 29 + 10 us, at the price of other codes in one matrix of three.
#include <cmath>

#include <cooperative_groups.h>

#include "tcq_traceback.cuh"

namespace tcq {

namespace {

constexpr int kIpThreads = 256;
// Rows up to which every CTA of the column sums takes the mean for itself: a launch less (512 x 512 30.8 -> 27.6 us), and no more than eight loads a
// thread; beyond that the CTAs together would read the row sums as often as the matrix.
constexpr long long kRowsForOwnMean = 1024;
// Rows from which a warp each is enough, eight per SM; fewer get a CTA each (64 x 65536: 110 -> 63 us forward).
constexpr long long kRowsForWarps = 1184;

int ilog2(int v) { int l = 0; while ((1 << l) < v) ++l; return l; }

__host__ __device__ inline int pow2_block(long long d, int cap) {
    int b = 1;
    while (b < cap && d % (2 * b) == 0) b *= 2;
    return b;
}

// The order of the sums: 256 partial sums of a row (column mod 256) and 1024 of a scale vector (index mod 1024), each in index order, halves
// added to halves; a column's squares block by block.

// r[row] = max(rms of the row, 1e-8).  One warp per row (partial sums lane + 32 j), or, where rows are few, one CTA.
template <bool WARP>
__global__ void __launch_bounds__(kIpThreads) ip_row_rms_kernel(const float* __restrict__ w, long long n, long long k, float* __restrict__ r) {
    __shared__ float red[kIpThreads];
    constexpr int NS = WARP ? 8 : 1, STEP = WARP ? 32 : kIpThreads;            // partial sums of a thread, distance of its columns
    const int lane = threadIdx.x & 31;
    const long long row = WARP ? (long long)blockIdx.x * (kIpThreads / 32) + (threadIdx.x >> 5) : (long long)blockIdx.x;
    if (row >= n) return;                                     // whole warps (CTAs) leave together
    const float* const p = w + row * k;
    float s[NS] = {};
    long long c = WARP ? lane : threadIdx.x;
    for (; c + 15 * STEP < k; c += 16 * STEP) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __ldg(p + c + STEP * j);
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j % NS] = __fmaf_rn(v[j], v[j], s[j % NS]);
    }
#pragma unroll
    for (int j = 0; j < 15; ++j)
        if (c + STEP * j < k) {
            const float v = __ldg(p + c + STEP * j);
            s[j % NS] = __fmaf_rn(v, v, s[j % NS]);
        }
    float t = s[0];
    if constexpr (WARP) {
        t = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
    } else {
        red[threadIdx.x] = t;
        __syncthreads();
        for (int h = kIpThreads / 2; h >= 32; h >>= 1) {
            if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
            __syncthreads();
        }
        if (threadIdx.x >= 32) return;
        t = red[lane];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, off);
    if (lane == 0) r[row] = fmaxf(sqrtf(t / float(k)), 1e-8f);
}

// Sum over the CTA's threads, halves added to halves, the same value in every thread.
template <int NT>
__device__ __forceinline__ float cta_sum(float x, float (&red)[NT]) {
    __syncthreads();
    red[threadIdx.x] = x;
    __syncthreads();
    for (int h = NT / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    return red[0];
}

// Partial sum of x over the indices below d that are i mod 1024, in index order.
__device__ __forceinline__ float sum_mod1024(const float* x, long long d, long long i) {
    float t = 0.0f;
    for (; i + 7 * 1024 < d; i += 8 * 1024) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __ldcg(x + i + 1024 * j);
#pragma unroll
        for (int j = 0; j < 8; ++j) t += v[j];
    }
    for (; i < d; i += 1024) t += __ldcg(x + i);
    return t;
}

// Row scales: out_s = r / mean(r) and its reciprocal.  One CTA, for matrices of more than kRowsForOwnMean rows.
__global__ void __launch_bounds__(1024) ip_finish_rows_kernel(const float* __restrict__ r, long long n, float* __restrict__ out_s,
                                                             float* __restrict__ inv_out_s) {
    __shared__ float red[1024];
    const float mean = cta_sum<1024>(sum_mod1024(r, n, threadIdx.x), red) / float(n);
    for (long long i = threadIdx.x; i < n; i += 1024) {
        const float o = r[i] / mean;
        out_s[i] = o;
        inv_out_s[i] = 1.0f / o;
    }
}

__device__ __forceinline__ void mul4(float* v, const float4& f) {
    v[0] = __fmul_rn(v[0], f.x);
    v[1] = __fmul_rn(v[1], f.y);
    v[2] = __fmul_rn(v[2], f.z);
    v[3] = __fmul_rn(v[3], f.w);
}

// One butterfly stage over the register bit H of v.
template <int N, int H>
__device__ __forceinline__ void had_stage(float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (!(i & H)) {
            const float a = v[i], b = v[i + H];
            v[i] = a + b;
            v[i + H] = a - b;
        }
}

// part[b][c] = sum of the squares of column c of block b (of B rows) after the transform down the rows, in row order.  A column's
// values stay in the registers of one thread, 128 of them in those of two lanes 16 apart (with 162 registers three CTAs of four warps are all that fits an
// SM, 59 us for 12288 x 4096).  Nothing but the sums is written, the matrix is transformed again by ip_block_kernel (a third read instead of
// an intermediate that is written and read back).  Column signs do not change a square and are left out.  Blocks from the last to
// the first: the row sums have just read the matrix in the other direction, and what of it L2 still holds is read from there.
// OWN: the row scales are not there yet; every CTA takes the mean of r for itself, under its loads of w (a launch and a round of latency
// less), and the first of each block writes the block's.
constexpr int kColThreads = 128;
template <int B> constexpr int kColumnsPerCta = B == 128 ? kColThreads / 2 : kColThreads;
template <int B, bool OWN>
__global__ void __launch_bounds__(kColThreads) ip_col_sumsq_kernel(const float* __restrict__ w, long long n, long long k, float norm, const float* __restrict__ sv,
                                                                  const float* __restrict__ r, float* __restrict__ out_s,
                                                                  float* __restrict__ inv_out_s, float* __restrict__ part) {
    constexpr int V = B == 128 ? 64 : B;                       // rows of a thread
    __shared__ __align__(16) float rowf[B + 4];                // read four at a time (the upper lanes' rows four banks further)
    auto slot = [](int i) { return i + (i >> 6) * 4; };
    __shared__ float red[kColThreads];
    const int lane = threadIdx.x & 31;
    const int col = B == 128 ? (threadIdx.x >> 5) * 16 + (lane & 15) : threadIdx.x, row = B == 128 ? (lane >> 4) * 64 : 0;
    const long long b = gridDim.y - 1 - blockIdx.y, r0 = b * B, c = (long long)blockIdx.x * kColumnsPerCta<B> + col;
    const float* const p = w + (r0 + row) * k + c;
    float v[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = c < k ? __ldg(p + i * k) : 0.0f;
    if constexpr (OWN) {
        float s[1024 / kColThreads];                           // partial sums tid, tid + 128, ...
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] = sum_mod1024(r, n, threadIdx.x + j * kColThreads);
        const float mean = cta_sum<kColThreads>(((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7])), red) / float(n);
        if (threadIdx.x < B) {
            const float o = r[r0 + threadIdx.x] / mean, inv = 1.0f / o;
            rowf[slot(threadIdx.x)] = __fmul_rn(sv[r0 + threadIdx.x], inv);
            if (blockIdx.x == 0) {
                out_s[r0 + threadIdx.x] = o;
                inv_out_s[r0 + threadIdx.x] = inv;
            }
        }
    } else {
        if (threadIdx.x < B) rowf[slot(threadIdx.x)] = __fmul_rn(sv[r0 + threadIdx.x], inv_out_s[r0 + threadIdx.x]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; i += 4) mul4(v + i, *reinterpret_cast<const float4*>(rowf + slot(row) + i));
    had_stage<V, 1>(v);
    had_stage<V, 2>(v);
    had_stage<V, 4>(v);
    had_stage<V, 8>(v);
    if constexpr (V > 16) had_stage<V, 16>(v);
    if constexpr (V > 32) had_stage<V, 32>(v);
    float s = 0.0f;
    auto add_squares = [&] {
#pragma unroll
        for (int i = 0; i < V; ++i) s = __fmaf_rn(v[i], v[i], s);
    };
    if constexpr (B == 128) {
        const float sign = lane >= 16 ? -1.0f : 1.0f;
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] = __fmul_rn(__fmaf_rn(v[i], sign, __shfl_xor_sync(0xFFFFFFFFu, v[i], 16)), norm);
        add_squares();
        s = __shfl_sync(0xFFFFFFFFu, s, lane & 15);            // of rows 0 .. 63; the upper lane goes on from there
        add_squares();
        if (lane >= 16 && c < k) part[b * k + c] = s;
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] = __fmul_rn(v[i], norm);
        add_squares();
        if (c < k) part[b * k + c] = s;
    }
}

// part[0][c] = sum over the parts of column c, in order, where they are many: a CTA fetches 32 columns of 256 parts at a time into
// shared memory, from which one warp adds them up while the next are on their way.
constexpr int kSumThreads = 512, kSumParts = 256;
__global__ void __launch_bounds__(kSumThreads) ip_sum_parts_kernel(float* part, long long parts, long long k) {
    __shared__ float buf[kSumParts][32];
    constexpr int ROWS = kSumThreads / 32, NL = kSumParts / ROWS;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const long long c = (long long)blockIdx.x * 32 + lane;
    float v[NL];
    auto fetch = [&](long long p0) {
#pragma unroll
        for (int j = 0; j < NL; ++j) {
            const long long p = p0 + row + j * ROWS;
            v[j] = c < k && p < parts ? __ldcg(part + p * k + c) : 0.0f;
        }
    };
    float t = 0.0f;
    fetch(0);
    for (long long p0 = 0; p0 < parts; p0 += kSumParts) {
#pragma unroll
        for (int j = 0; j < NL; ++j) buf[row + j * ROWS][lane] = v[j];
        __syncthreads();
        fetch(p0 + kSumParts);
        if (row == 0) {
            const int live = int(parts - p0 < kSumParts ? parts - p0 : kSumParts);
#pragma unroll 8
            for (int i = 0; i < live; ++i) t += buf[i][lane];
        }
        __syncthreads();
    }
    if (row == 0 && c < k) part[c] = t;
}

// One cluster: column scales from the parts (summed in order), c[i] = max(sqrt(sum_p part[p][i] / n), 1e-8), in_s = c / mean(c),
// inv_in_s = 1 / in_s, and scale = sqrt(sum_i sum_p part[p][i] / in_s[i]^2 / (n k)) / cb_rms.
constexpr int kFinishCtas = 8, kFinishThreads = 512;
constexpr int kFinishParts = 16;                               // more are added up before, by the whole chip
__global__ void __cluster_dims__(kFinishCtas, 1, 1) __launch_bounds__(kFinishThreads)
ip_finish_cols_kernel(float* part, long long parts, long long n, long long k, float* in_s, float* inv_in_s, float cb_rms, float* __restrict__ scale_out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float red[kFinishThreads];
    const int rank = int(cluster.block_rank());
    const long long first = (long long)rank * kFinishThreads + threadIdx.x, stride = kFinishCtas * kFinishThreads;
    for (long long i = first; i < k; i += stride) {
        float t = 0.0f;
        long long p = 0;
        for (; p < parts; p += kFinishParts) {
            float v[kFinishParts];
#pragma unroll
            for (int j = 0; j < kFinishParts; ++j)
                if (p + j < parts) v[j] = __ldcg(part + (p + j) * k + i);
#pragma unroll
            for (int j = 0; j < kFinishParts; ++j)
                if (p + j < parts) t += v[j];
        }
        in_s[i] = fmaxf(sqrtf(t / float(n)), 1e-8f);
        inv_in_s[i] = t;
    }
    cluster.sync();                                            // in_s holds the c of every column
    // every CTA for itself; a thread has the partial sums tid and tid + 512
    const float mean = cta_sum<kFinishThreads>(sum_mod1024(in_s, k, threadIdx.x) + sum_mod1024(in_s, k, threadIdx.x + 512), red) / float(k);
    cluster.sync();                                            // and has been read by every CTA
    for (long long i = first; i < k; i += stride) {
        const float t = inv_in_s[i], s = in_s[i] / mean;
        in_s[i] = s;
        inv_in_s[i] = 1.0f / s;
        part[i] = t / (s * s);                                 // part 0 of this column, which nobody else reads
    }
    cluster.sync();
    if (rank != 0) return;
    const float tot = cta_sum<kFinishThreads>(sum_mod1024(part, k, threadIdx.x) + sum_mod1024(part, k, threadIdx.x + 512), red);
    if (threadIdx.x == 0) *scale_out = sqrtf(tot / (float(n) * float(k))) / cb_rms;
}

// Both transforms of a 128 x 128 block, 256 threads with 64 values each.  Its 14 index bits (rows r0..r6, columns c0..c6) are held two
// ways, of which X is r6 forward and r0 back, the row bit whose stage comes last (first) in order:
//   "column": a thread has the 64 rows without X of one column; lanes c0..c4, warps c5 c6 X.  A warp reads or writes
//             128 contiguous bytes of a row-major matrix.
//   "tile":   a thread has four columns (c0 c1: one 16-byte word) x (c4 c5 c6) x X; lanes c2 c3 and the three lowest other row bits,
//             warps the three highest.  A warp writes half a tile of the encoder, 512 contiguous bytes, or reads eight of its 16 rows.
// So with one pass through shared memory between the two every stage but two (c2 and c3, by shuffle) is done in registers, in
// natural order on both axes.  The column bits are flipped by the tile form's lowest lane bit of the row (16 banks), which makes all
// accesses conflict-free.  64 KiB of
// loads in flight per CTA, two CTAs per SM (three need 80 registers and spill).  Bound by HBM and, half as much, by instruction
// issue: whole blocks have a path of their own without bounds checks, and a shuffle stage is one fused +-v + other.
//   forward: in = w (row-major), out = ((Hb_cols(((Hb_rows(w * sv * rs * su)) * cs)) / scale, in tile order or row-major; rs = 1/out_s, cs = 1/in_s
//   inverse: in = zq (tile order or row-major), out = Hb_rows(Hb_cols(zq * scale) * cs) * rs * sv * su; rs = out_s, cs = in_s
// A block smaller than 128 takes fewer stages; rows and columns beyond the matrix are zero and are not stored.
constexpr int kBlockThreads = 256;
constexpr size_t kBlockSmem = size_t(128) * 128 * 4 + 128 * 4;

template <bool INV, bool TILED, bool FULL>
__device__ __forceinline__ void ip_block(const float* __restrict__ in, int n_live, int k_live, long long k, int logB0, int logB1, float norm0, float norm1,
                                        const float* __restrict__ su, const float* __restrict__ cs, float scale, float* __restrict__ out,
                                        float* blk, const float* rowf) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int RS = INV ? 2 : 1, X = INV ? 1 : 64;          // row step of a thread's 64 rows, value of bit X
    // "column" form: v[row bits without X]; in / out of this form start at the block's row-major origin
    const int cc = (warp & 3) * 32 + lane, rc = (warp >> 2) * X;
    const bool c_live = FULL || cc < k_live;
    auto row_of = [&](int i) { return i * RS + rc; };
    auto at = [](int r, int c) { return r * 128 + (c ^ ((r & RS) != 0 ? 16 : 0)); };
    auto column_stages = [&](float (&v)[64]) {                 // r0 .. r5 forward, r1 .. r6 back
        had_stage<64, 1>(v);
        had_stage<64, 2>(v);
        had_stage<64, 4>(v);
        if (!INV || logB0 > 4) had_stage<64, 8>(v);
        if (logB0 > (INV ? 5 : 4)) had_stage<64, 16>(v);
        if (logB0 > (INV ? 6 : 5)) had_stage<64, 32>(v);
    };
    // "tile" form: v[4 * (8 * X + c456) + c01]; in / out of this form start at the block's origin in their layout
    const int tr = ((lane >> 2) | (warp << 3)) * RS, tc = (lane & 3) * 4;
    auto offset = [&](int j) {
        const int r = tr + (j >> 3) * X;
        return TILED ? (long long)(r >> 4) * (k >> 4) * 256 + (j & 7) * 256 + ((r & 15) << 4) + tc : r * k + tc + 16 * (j & 7);
    };
    auto live = [&](int j) { return FULL || (tr + (j >> 3) * X < n_live && tc + 16 * (j & 7) < k_live); };
    auto tile_stages = [&](float (&v)[64]) {                   // c0 .. c6
        had_stage<64, 1>(v);
        had_stage<64, 2>(v);
#pragma unroll
        for (int m = 1; m <= 2; m <<= 1) {
            const float sign = (lane & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
            for (int i = 0; i < 64; ++i) v[i] = __fmaf_rn(v[i], sign, __shfl_xor_sync(0xFFFFFFFFu, v[i], m));
        }
        if (logB1 > 4) had_stage<64, 4>(v);
        if (logB1 > 5) had_stage<64, 8>(v);
        if (logB1 > 6) had_stage<64, 16>(v);
    };
    auto scale_columns = [&](float (&v)[64], float f) {        // v = (v * f) * cs
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = tc + 16 * j;
            const float4 s4 = FULL || c < k_live ? *reinterpret_cast<const float4*>(cs + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float s[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                v[4 * j + b] = __fmul_rn(__fmul_rn(v[4 * j + b], f), s[b]);
                v[32 + 4 * j + b] = __fmul_rn(__fmul_rn(v[32 + 4 * j + b], f), s[b]);
            }
        }
    };

    float v[64];
    if constexpr (!INV) {
        const float* p = in + rc * k + cc;
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = FULL || (c_live && row_of(i) < n_live) ? __ldg(p + (i * RS) * k) : 0.0f;
        const float suc = c_live ? su[cc] : 0.0f;
        __syncthreads();                                       // rowf
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __fmul_rn(v[i], __fmul_rn(rowf[row_of(i)], suc));
        column_stages(v);
#pragma unroll
        for (int i = 0; i < 64; ++i) blk[at(row_of(i), cc)] = v[i];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<float4*>(v + 4 * j) = *reinterpret_cast<const float4*>(blk + at(tr + (j >> 3) * X, tc + 16 * (j & 7)));
        if (logB0 > 6) had_stage<64, 32>(v);                   // r6
        scale_columns(v, norm0);
        tile_stages(v);
        const float f = 1.0f / scale;
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], norm1), f);
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (live(j)) *reinterpret_cast<float4*>(out + offset(j)) = *reinterpret_cast<const float4*>(v + 4 * j);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            *reinterpret_cast<float4*>(v + 4 * j) = live(j) ? __ldg(reinterpret_cast<const float4*>(in + offset(j))) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __fmul_rn(v[i], scale);
        tile_stages(v);
        scale_columns(v, norm1);
        had_stage<64, 32>(v);                                  // r0
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<float4*>(blk + at(tr + (j >> 3) * X, tc + 16 * (j & 7))) = *reinterpret_cast<const float4*>(v + 4 * j);
        __syncthreads();                                       // and rowf
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = blk[at(row_of(i), cc)];
        column_stages(v);
        const float f = __fmul_rn(norm0, c_live ? su[cc] : 0.0f);            // a sign makes no difference to a rounding
        float* p = out + rc * k + cc;
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
            mul4(v + i, make_float4(f, f, f, f));
            mul4(v + i, *reinterpret_cast<const float4*>(rowf + (warp >> 2) * 64 + i));
#pragma unroll
            for (int j = i; j < i + 4; ++j)
                if (FULL || (c_live && row_of(j) < n_live)) p[(j * RS) * k] = v[j];
        }
    }
}

template <bool INV, bool TILED>
__global__ void __launch_bounds__(kBlockThreads, 2)
ip_block_kernel(const float* __restrict__ in, long long n, long long k, int logB0, int logB1, float norm0, float norm1, const float* __restrict__ sv,
                const float* __restrict__ su, const float* __restrict__ rs, const float* __restrict__ cs,
                const float* __restrict__ scale, float* __restrict__ out) {
    extern __shared__ __align__(16) float ip_smem[];
    float* const blk = ip_smem;                                // [128][128]
    float* const rowf = ip_smem + 128 * 128;                   // [128] factors of the rows, back in the order in which a thread of the column form has them
    const long long r0 = (long long)blockIdx.y * 128, c0 = (long long)blockIdx.x * 128;
    const int n_live = int(n - r0 < 128 ? n - r0 : 128), k_live = int(k - c0 < 128 ? k - c0 : 128);
    if (threadIdx.x < 128) {
        const int row = INV ? (threadIdx.x & 63) * 2 + (threadIdx.x >> 6) : threadIdx.x;
        rowf[threadIdx.x] = row < n_live ? __fmul_rn(sv[r0 + row], rs[r0 + row]) : 0.0f;
    }
    const long long rowmajor = r0 * k + c0, tile = r0 * k + c0 * 16;          // the block's origin: tile (r0/16)*(k/16) + c0/16, 256 values each
    const float* const src = in + (INV && TILED ? tile : rowmajor);
    float* const dst = out + (!INV && TILED ? tile : rowmajor);
    if (n_live == 128 && k_live == 128) ip_block<INV, TILED, true>(src, n_live, k_live, k, logB0, logB1, norm0, norm1, su + c0, cs + c0, *scale, dst, blk, rowf);
    else ip_block<INV, TILED, false>(src, n_live, k_live, k, logB0, logB1, norm0, norm1, su + c0, cs + c0, *scale, dst, blk, rowf);
}

// `spare` [n*k]: takes the result first where `out` overlaps `in` in another layout, whose blocks are not the same memory.
template <bool INV, bool TILED>
cudaError_t launch_block(const float* in, long long n, long long k, const float* sv, const float* su, const float* rs, const float* cs,
                         const float* scale, float* out, float* spare, cudaStream_t stream) {
    static bool optin[64] = {false};                           // per device ordinal: the shared-memory opt-in has been made
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= 64 || !optin[dev]) {
        if ((err = cudaFuncSetAttribute(ip_block_kernel<INV, TILED>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBlockSmem))) != cudaSuccess) return err;
        if (dev >= 0 && dev < 64) optin[dev] = true;
    }
    const int B0 = pow2_block(n, 128), B1 = pow2_block(k, 128);
    const dim3 grid(unsigned((k + 127) / 128), unsigned((n + 127) / 128));
    const uintptr_t bytes = uintptr_t(n) * uintptr_t(k) * 4, a = reinterpret_cast<uintptr_t>(in), b = reinterpret_cast<uintptr_t>(out);
    const bool via_spare = a < b + bytes && b < a + bytes && (TILED || a != b);
    ip_block_kernel<INV, TILED><<<grid, kBlockThreads, kBlockSmem, stream>>>(in, n, k, ilog2(B0), ilog2(B1), float(1.0 / sqrt(double(B0))),
                                                                      float(1.0 / sqrt(double(B1))), sv, su, rs, cs, scale, via_spare ? spare : out);
    err = cudaGetLastError();
    if (err == cudaSuccess && via_spare) err = cudaMemcpyAsync(out, spare, bytes, cudaMemcpyDeviceToDevice, stream);
    return err;
}


size_t up256(size_t v) { return (v + 255) / 256 * 256; }
// z [n*k]: the column sums' parts (at most a sixteenth of it), and later the spare matrix of launch_block.
struct IpWs { float* z; float* r; float* inv_out_s; float* inv_in_s; };
IpWs carve_ip(void* ws, long long n, long long k) {
    unsigned char* p = static_cast<unsigned char*>(ws);
    auto take = [&](size_t floats) { unsigned char* q = p; p += up256(floats * 4); return reinterpret_cast<float*>(q); };
    IpWs o;
    o.z = take(size_t(n) * size_t(k));
    o.r = take(size_t(n));
    o.inv_out_s = take(size_t(n));
    o.inv_in_s = take(size_t(k));
    return o;
}

template <int B>
cudaError_t launch_col_sumsq(const float* w, long long n, long long k, const float* sv, const float* r, float* out_s, float* inv_out_s, float* part,
                             cudaStream_t stream) {
    const dim3 grid(unsigned((k + kColumnsPerCta<B> - 1) / kColumnsPerCta<B>), unsigned(n / B));
    const float norm = float(1.0 / sqrt(double(B)));
    if (n <= kRowsForOwnMean) {
        ip_col_sumsq_kernel<B, true><<<grid, kColThreads, 0, stream>>>(w, n, k, norm, sv, r, out_s, inv_out_s, part);
    } else {
        ip_finish_rows_kernel<<<1, 1024, 0, stream>>>(r, n, out_s, inv_out_s);
        ip_col_sumsq_kernel<B, false><<<grid, kColThreads, 0, stream>>>(w, n, k, norm, sv, r, out_s, inv_out_s, part);
    }
    return cudaGetLastError();
}

}  // namespace

size_t ip_workspace_bytes(long long n, long long k) {
    return up256(size_t(n) * size_t(k) * 4) + 2 * up256(size_t(n) * 4) + up256(size_t(k) * 4);
}

cudaError_t launch_ip_forward(const float* w, long long n, long long k, const float* sv, const float* su, float cb_rms,
                              int tiled, float* z_out, float* out_s, float* in_s, float* scale, void* ws, cudaStream_t stream) {
    const IpWs wk = carve_ip(ws, n, k);
    const int B0 = pow2_block(n, 128);
    if (n >= kRowsForWarps) ip_row_rms_kernel<true><<<unsigned((n + kIpThreads / 32 - 1) / (kIpThreads / 32)), kIpThreads, 0, stream>>>(w, n, k, wk.r);
    else ip_row_rms_kernel<false><<<unsigned(n), kIpThreads, 0, stream>>>(w, n, k, wk.r);
    cudaError_t err = B0 == 128  ? launch_col_sumsq<128>(w, n, k, sv, wk.r, out_s, wk.inv_out_s, wk.z, stream)
                      : B0 == 64 ? launch_col_sumsq<64>(w, n, k, sv, wk.r, out_s, wk.inv_out_s, wk.z, stream)
                      : B0 == 32 ? launch_col_sumsq<32>(w, n, k, sv, wk.r, out_s, wk.inv_out_s, wk.z, stream)
                                 : launch_col_sumsq<16>(w, n, k, sv, wk.r, out_s, wk.inv_out_s, wk.z, stream);
    if (err != cudaSuccess) return err;
    long long parts = n / B0;
    if (parts > kFinishParts) {
        ip_sum_parts_kernel<<<unsigned((k + 31) / 32), kSumThreads, 0, stream>>>(wk.z, parts, k);
        parts = 1;
    }
    ip_finish_cols_kernel<<<kFinishCtas, kFinishThreads, 0, stream>>>(wk.z, parts, n, k, in_s, wk.inv_in_s, cb_rms, scale);
    if ((err = cudaGetLastError()) != cudaSuccess) return err;
    return tiled ? launch_block<false, true>(w, n, k, sv, su, wk.inv_out_s, wk.inv_in_s, scale, z_out, wk.z, stream)
                 : launch_block<false, false>(w, n, k, sv, su, wk.inv_out_s, wk.inv_in_s, scale, z_out, wk.z, stream);
}

cudaError_t launch_ip_restore(const float* zq, int tiled, long long n, long long k, const float* sv, const float* su,
                              const float* out_s, const float* in_s, const float* scale, float* w_hat, void* ws,
                              cudaStream_t stream) {
    float* const spare = carve_ip(ws, n, k).z;
    return tiled ? launch_block<true, true>(zq, n, k, sv, su, out_s, in_s, scale, w_hat, spare, stream)
                 : launch_block<true, false>(zq, n, k, sv, su, out_s, in_s, scale, w_hat, spare, stream);
}

}  // namespace tcq
