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
// The scales need no transform: Hb is orthonormal, so the sum of squares of a column of Hb_rows(z) is that of z, and
// rms(z) is the same before and after the last transform.  Both statistics are plain sums over w: one read each, and the second
// walks the matrix from its end, where the first left it in L2.  So forward is three reads and one write of 4 bytes per
// weight (a third read instead of an intermediate that is written and read back), restore one read and one write.
//
// On a 12288 x 4096 matrix (201 MB): forward 240 -> 191 us (row sums 37, column sums 41, column scales, blocks), restore
// 167 -> 78 us = 5.2 TB/s.  (Before: a transform per axis and kernel, with an intermediate matrix between them.)
// Four launches forward instead of six: 39 -> 34 us on a 1024 x 4096 matrix, which is launches and latency.
//
// Every reduction runs in a fixed order (no atomics), so results are reproducible run to run.  Divisions by the scale
// vectors are multiplications by their reciprocals (one rounding more than the reference's division).
#include <cmath>

#include <cooperative_groups.h>

#include "tcq_traceback.cuh"

namespace tcq {

namespace {

constexpr int kIpThreads = 256;

int ilog2(int v) { int l = 0; while ((1 << l) < v) ++l; return l; }

__host__ __device__ inline int pow2_block(long long d, int cap) {
    int b = 1;
    while (b < cap && d % (2 * b) == 0) b *= 2;
    return b;
}

// r[i] = max(rms of row i, 1e-8) and inv_r[i] = 1 / r[i]; one warp per row, fixed order.
__global__ void __launch_bounds__(kIpThreads) ip_row_rms_kernel(const float* __restrict__ w, long long n, long long k,
                                                               float* __restrict__ r, float* __restrict__ inv_r) {
    const long long row = (long long)blockIdx.x * (kIpThreads / 32) + (threadIdx.x >> 5);
    if (row >= n) return;                                     // whole warps leave together
    const float* const p = w + row * k;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    long long c = threadIdx.x & 31;
    for (; c + 15 * 32 < k; c += 16 * 32) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __ldg(p + c + 32 * j);
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j & 3] = __fmaf_rn(v[j], v[j], s[j & 3]);
    }
    for (; c < k; c += 32) {
        const float v = __ldg(p + c);
        s[0] = __fmaf_rn(v, v, s[0]);
    }
    float t = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, off);
    if ((threadIdx.x & 31) == 0) {
        t = fmaxf(sqrtf(t / float(k)), 1e-8f);
        r[row] = t;
        inv_r[row] = 1.0f / t;
    }
}

// Sum over the CTA's threads in a fixed order, the same value in every thread.
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

// part[p][c] = sum over row part p of (w[r][c] / r[r])^2.  Parts and rows from the last to the first: the row sums have just
// read the matrix in the other direction, and what of it L2 still holds is read from there.
// The first CTA, beside that, normalises the row scales: mean = mean(r), out_s = r / mean.  (The column sums do without the mean, a common factor.)
__global__ void __launch_bounds__(kIpThreads) ip_col_sumsq_kernel(const float* __restrict__ w, long long n, long long k,
                                                                 long long rows_per_part, const float* __restrict__ r,
                                                                 const float* __restrict__ inv_r, float* __restrict__ part,
                                                                 float* __restrict__ out_s, float* __restrict__ inv_out_s,
                                                                 float* __restrict__ mean_out) {
    __shared__ float red[kIpThreads];
    if (blockIdx.x == 0) {
        if (blockIdx.y != 0) return;
        float acc = 0.0f;
        for (long long i = threadIdx.x; i < n; i += kIpThreads) acc += r[i];
        const float mean = cta_sum<kIpThreads>(acc, red) / float(n);
        for (long long i = threadIdx.x; i < n; i += kIpThreads) {
            const float o = r[i] / mean;
            out_s[i] = o;
            inv_out_s[i] = 1.0f / o;
        }
        if (threadIdx.x == 0) *mean_out = mean;
        return;
    }
    const long long c = (long long)(blockIdx.x - 1) * kIpThreads + threadIdx.x;
    const long long p = gridDim.y - 1 - blockIdx.y;
    if (c >= k) return;
    const long long r0 = p * rows_per_part;
    long long i = r0 + rows_per_part < n ? r0 + rows_per_part : n;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (; i - 16 >= r0; i -= 16) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __ldg(w + (i - 1 - j) * k + c);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float x = __fmul_rn(v[j], __ldg(inv_r + i - 1 - j));
            s[j & 3] = __fmaf_rn(x, x, s[j & 3]);
        }
    }
    for (; i > r0; --i) {
        const float x = __fmul_rn(__ldg(w + (i - 1) * k + c), __ldg(inv_r + i - 1));
        s[0] = __fmaf_rn(x, x, s[0]);
    }
    part[p * k + c] = (s[0] + s[1]) + (s[2] + s[3]);
}

// One cluster: column scales from the parts (summed in order), c[i] = max(sqrt(mean^2 * sum_p part[p][i] / n), 1e-8),
// in_s = c / mean(c), inv_in_s = 1 / in_s, and scale = sqrt(sum_i (mean^2 * sum_p part[p][i]) / in_s[i]^2 / (n k)) / cb_rms.
constexpr int kFinishCtas = 8, kFinishThreads = 512;
__global__ void __cluster_dims__(kFinishCtas, 1, 1) __launch_bounds__(kFinishThreads)
ip_finish_cols_kernel(const float* __restrict__ part, int parts, long long n, long long k, const float* __restrict__ mean_in,
                      float* __restrict__ in_s, float* __restrict__ inv_in_s, float cb_rms, float* __restrict__ scale_out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float red[kFinishThreads];
    __shared__ float share[2];
    const int rank = int(cluster.block_rank());
    const float m2 = *mean_in * *mean_in;
    const long long first = (long long)rank * kFinishThreads + threadIdx.x, stride = kFinishCtas * kFinishThreads;
    auto cluster_sum = [&](float x, int slot) {                // every CTA adds the CTAs' sums in rank order
        const float own = cta_sum<kFinishThreads>(x, red);
        if (threadIdx.x == 0) share[slot] = own;
        cluster.sync();
        float t = 0.0f;
        for (int i = 0; i < kFinishCtas; ++i) t += *cluster.map_shared_rank(&share[slot], i);
        return t;
    };
    auto column = [&](long long i) {
        float t = 0.0f;
        int p = 0;
        for (; p + 8 <= parts; p += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __ldg(part + (p + j) * k + i);
#pragma unroll
            for (int j = 0; j < 8; ++j) t += v[j];
        }
        for (; p < parts; ++p) t += __ldg(part + p * k + i);
        return t * m2;
    };
    float acc = 0.0f;
    for (long long i = first; i < k; i += stride) {
        const float t = column(i), c = fmaxf(sqrtf(t / float(n)), 1e-8f);
        in_s[i] = c;
        inv_in_s[i] = t;
        acc += c;
    }
    const float mean = cluster_sum(acc, 0) / float(k);
    float tot = 0.0f;
    for (long long i = first; i < k; i += stride) {
        const float t = inv_in_s[i], s = in_s[i] / mean;
        in_s[i] = s;
        inv_in_s[i] = 1.0f / s;
        tot += t / (s * s);
    }
    tot = cluster_sum(tot, 1);
    if (rank == 0 && threadIdx.x == 0) *scale_out = sqrtf(tot / (float(n) * float(k))) / cb_rms;
    cluster.sync();                                            // nobody leaves while its sums are still being read
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

// Both transforms of a 128 x 128 block, 256 threads with 64 values each.  Its 14 index bits (rows r0..r6, columns c0..c6) are held two ways:
//   "column": a thread has 64 rows (r0 r1 r2 r4 r5 r6) of one column; lanes c0..c4, warps c5 c6 r3.  A warp reads or writes
//             128 contiguous bytes of a row-major matrix.
//   "tile":   a thread has four columns (c0 c1: one 16-byte word) x (c4 c5 c6) x r3; lanes c2 c3 r0 r1 r2, warps r4 r5 r6.  A warp
//             reads or writes half a tile of the encoder, 512 contiguous bytes.
// So with one pass through shared memory between the two every stage but two (c2 and c3, by shuffle) is done in registers.
// The column bits are flipped by the row's lowest bit (16 banks), which makes all accesses to it conflict-free.  64 KiB of
// loads in flight per CTA, two CTAs per SM (three need 80 registers and spill).  Bound by HBM and, half as much, by instruction
// issue: whole blocks have a path of their own without bounds checks, and a shuffle stage is one fused +-v + other.
//   forward: in = w (row-major), out = Hb_cols((Hb_rows(w * sv * rs * su)) * cs) / scale with rs = 1/out_s, cs = 1/in_s, in tile order or row-major
//   inverse: in = zq (tile order or row-major), out = Hb_rows(Hb_cols(zq * scale) * cs) * rs * sv * su with rs = out_s, cs = in_s
// A block smaller than 128 takes fewer stages; rows and columns beyond the matrix are zero and are not stored.
constexpr int kBlockThreads = 256;
constexpr size_t kBlockSmem = size_t(128) * 128 * 4 + 128 * 4;

template <bool INV, bool TILED, bool FULL>
__device__ __forceinline__ void ip_block(const float* __restrict__ in, int n_live, int k_live, long long k, int logB0, int logB1, float norm,
                                        const float* __restrict__ su, const float* __restrict__ cs, float scale, float* __restrict__ out,
                                        float* blk, const float* rowf) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // "column" form: v[r0 r1 r2 r4 r5 r6]; in / out of this form start at the block's row-major origin
    const int cc = (warp & 3) * 32 + lane, rc = (warp >> 2) << 3;
    const bool c_live = FULL || cc < k_live;
    auto row_of = [&](int i) { return (i & 7) | rc | ((i >> 3) << 4); };
    auto at = [](int r, int c) { return r * 128 + (c ^ ((r & 1) << 4)); };
    auto column_stages = [&](float (&v)[64]) {
        had_stage<64, 1>(v);
        had_stage<64, 2>(v);
        had_stage<64, 4>(v);
        if (logB0 > 4) had_stage<64, 8>(v);
        if (logB0 > 5) had_stage<64, 16>(v);
        if (logB0 > 6) had_stage<64, 32>(v);
    };
    // "tile" form: v[4 * (8 * r3 + c456) + c01]; in / out of this form start at the block's origin in their layout
    const int tr = (lane >> 2) | (warp << 4), tc = (lane & 3) * 4;
    const long long tile_base = TILED ? (long long)warp * (k >> 4) * 256 + ((lane >> 2) << 4) + tc : tr * k + tc;
    auto offset = [&](int j) { return tile_base + (TILED ? (j & 7) * 256 + (j >> 3) * 128 : (j & 7) * 16 + (j >> 3) * 8 * k); };
    auto live = [&](int j) { return FULL || (tr + (j >> 3) * 8 < n_live && tc + 16 * (j & 7) < k_live); };
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
    auto scale_columns = [&](float (&v)[64], float f) {        // v *= cs * f
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = tc + 16 * j;
            const float4 s4 = FULL || c < k_live ? *reinterpret_cast<const float4*>(cs + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float s[4] = {__fmul_rn(s4.x, f), __fmul_rn(s4.y, f), __fmul_rn(s4.z, f), __fmul_rn(s4.w, f)};
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                v[4 * j + b] = __fmul_rn(v[4 * j + b], s[b]);
                v[32 + 4 * j + b] = __fmul_rn(v[32 + 4 * j + b], s[b]);
            }
        }
    };

    float v[64];
    if constexpr (!INV) {
        const float* p = in + rc * k + cc;
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = FULL || (c_live && row_of(i) < n_live) ? __ldg(p + ((i & 7) | ((i >> 3) << 4)) * k) : 0.0f;
        const float suc = c_live ? su[cc] : 0.0f;
        __syncthreads();                                       // rowf
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = __fmul_rn(v[i], __fmul_rn(rowf[row_of(i)], suc));
        column_stages(v);
#pragma unroll
        for (int i = 0; i < 64; ++i) blk[at(row_of(i), cc)] = v[i];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<float4*>(v + 4 * j) = *reinterpret_cast<const float4*>(blk + at(tr | ((j >> 3) << 3), tc + 16 * (j & 7)));
        had_stage<64, 32>(v);                                  // r3
        scale_columns(v, norm / scale);
        tile_stages(v);
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (live(j)) *reinterpret_cast<float4*>(out + offset(j)) = *reinterpret_cast<const float4*>(v + 4 * j);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            *reinterpret_cast<float4*>(v + 4 * j) = live(j) ? __ldg(reinterpret_cast<const float4*>(in + offset(j))) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        tile_stages(v);
        scale_columns(v, norm * scale);
        had_stage<64, 32>(v);                                  // r3
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<float4*>(blk + at(tr | ((j >> 3) << 3), tc + 16 * (j & 7))) = *reinterpret_cast<const float4*>(v + 4 * j);
        __syncthreads();                                       // and rowf
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = blk[at(row_of(i), cc)];
        column_stages(v);
        const float suc = c_live ? su[cc] : 0.0f;
        float* p = out + rc * k + cc;
#pragma unroll
        for (int i = 0; i < 64; ++i)
            if (FULL || (c_live && row_of(i) < n_live)) p[((i & 7) | ((i >> 3) << 4)) * k] = __fmul_rn(v[i], __fmul_rn(rowf[row_of(i)], suc));
    }
}

template <bool INV, bool TILED>
__global__ void __launch_bounds__(kBlockThreads, 2)
ip_block_kernel(const float* __restrict__ in, long long n, long long k, int logB0, int logB1, float norm, const float* __restrict__ sv,
                const float* __restrict__ su, const float* __restrict__ rs, const float* __restrict__ cs,
                const float* __restrict__ scale, float* __restrict__ out) {
    extern __shared__ __align__(16) float ip_smem[];
    float* const blk = ip_smem;                                // [128][128]
    float* const rowf = ip_smem + 128 * 128;                   // [128] factors of the rows
    const long long r0 = (long long)blockIdx.y * 128, c0 = (long long)blockIdx.x * 128;
    const int n_live = int(n - r0 < 128 ? n - r0 : 128), k_live = int(k - c0 < 128 ? k - c0 : 128);
    if (threadIdx.x < 128) rowf[threadIdx.x] = int(threadIdx.x) < n_live ? __fmul_rn(sv[r0 + threadIdx.x], rs[r0 + threadIdx.x]) : 0.0f;
    const long long rowmajor = r0 * k + c0, tile = r0 * k + c0 * 16;          // the block's origin: tile (r0/16)*(k/16) + c0/16, 256 values each
    const float* const src = in + (INV && TILED ? tile : rowmajor);
    float* const dst = out + (!INV && TILED ? tile : rowmajor);
    if (n_live == 128 && k_live == 128) ip_block<INV, TILED, true>(src, n_live, k_live, k, logB0, logB1, norm, su + c0, cs + c0, *scale, dst, blk, rowf);
    else ip_block<INV, TILED, false>(src, n_live, k_live, k, logB0, logB1, norm, su + c0, cs + c0, *scale, dst, blk, rowf);
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
    ip_block_kernel<INV, TILED><<<grid, kBlockThreads, kBlockSmem, stream>>>(in, n, k, ilog2(B0), ilog2(B1), float(1.0 / sqrt(double(B0) * B1)), sv, su, rs,
                                                                      cs, scale, via_spare ? spare : out);
    err = cudaGetLastError();
    if (err == cudaSuccess && via_spare) err = cudaMemcpyAsync(out, spare, bytes, cudaMemcpyDeviceToDevice, stream);
    return err;
}


size_t up256(size_t v) { return (v + 255) / 256 * 256; }
// Row parts of the column sums: enough CTAs to fill the chip a few times over.
long long col_parts(long long n, long long k) {
    const long long blocks = n / pow2_block(n, 128), chunks = (k + kIpThreads - 1) / kIpThreads;
    const long long want = (148 * 8 + chunks - 1) / chunks;
    return want < blocks ? want : blocks;
}
struct IpWs { float* z; float* colpart; float* r; float* inv_r; float* inv_out_s; float* inv_in_s; float* mean; };
IpWs carve_ip(void* ws, long long n, long long k) {
    unsigned char* p = static_cast<unsigned char*>(ws);
    auto take = [&](size_t floats) { unsigned char* q = p; p += up256(floats * 4); return reinterpret_cast<float*>(q); };
    IpWs o;
    o.z = take(size_t(n) * size_t(k));
    o.colpart = take(size_t(col_parts(n, k)) * size_t(k));
    o.r = take(size_t(n));
    o.inv_r = take(size_t(n));
    o.inv_out_s = take(size_t(n));
    o.inv_in_s = take(size_t(k));
    o.mean = take(1);
    return o;
}

}  // namespace

size_t ip_workspace_bytes(long long n, long long k) {
    return up256(size_t(n) * size_t(k) * 4) + up256(size_t(col_parts(n, k)) * size_t(k) * 4) + 3 * up256(size_t(n) * 4) + up256(size_t(k) * 4) + 256;
}

cudaError_t launch_ip_forward(const float* w, long long n, long long k, const float* sv, const float* su, float cb_rms,
                              int tiled, float* z_out, float* out_s, float* in_s, float* scale, void* ws, cudaStream_t stream) {
    const IpWs wk = carve_ip(ws, n, k);
    const long long parts = col_parts(n, k), rows_per_part = (n + parts - 1) / parts;
    ip_row_rms_kernel<<<unsigned((n + kIpThreads / 32 - 1) / (kIpThreads / 32)), kIpThreads, 0, stream>>>(w, n, k, wk.r, wk.inv_r);
    const dim3 g0(unsigned((k + kIpThreads - 1) / kIpThreads) + 1, unsigned(parts));
    ip_col_sumsq_kernel<<<g0, kIpThreads, 0, stream>>>(w, n, k, rows_per_part, wk.r, wk.inv_r, wk.colpart, out_s, wk.inv_out_s, wk.mean);
    ip_finish_cols_kernel<<<kFinishCtas, kFinishThreads, 0, stream>>>(wk.colpart, int(parts), n, k, wk.mean, in_s, wk.inv_in_s, cb_rms, scale);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
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
