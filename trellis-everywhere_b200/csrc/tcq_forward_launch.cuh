// Host-side dispatch of the Viterbi step kernel for one K; included by
// tcq_forward_k2.cu / _k3.cu / _k4.cu, which are separate translation units only
// so that the large kernels compile in parallel.
#pragma once


#include "tcq_forward_cluster.cuh"

namespace tcq {

constexpr int kMaxDeviceOrdinals = 64;

// Current device ordinal, or -1 if it does not fit the per-device caches below (then nothing is cached).
static inline cudaError_t device_slot(int* slot) {
    int dev = 0;
    const cudaError_t err = cudaGetDevice(&dev);
    *slot = (err == cudaSuccess && dev >= 0 && dev < kMaxDeviceOrdinals) ? dev : -1;
    return err;
}

// Per kernel instantiation and device, once: opt in to the kernel's dynamic shared memory.  Small
// encoder calls (an LDLQ block is a few hundred tiles) would otherwise pay for the attribute call
// on every launch.  (Racing first calls from two host threads both set the same value.)
template <typename Kern>
static cudaError_t ensure_smem_optin(Kern kern, size_t smem, bool (&done)[kMaxDeviceOrdinals], int slot) {
    if (slot >= 0 && done[slot]) return cudaSuccess;
    const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (err == cudaSuccess && slot >= 0) done[slot] = true;
    return err;
}

template <int K, int CB, int G, int NT, int LU>
static cudaError_t launch_variant(const ForwardArgs& a, int num_sms, cudaStream_t stream) {
    auto kern = tcq_forward_kernel<K, CB, G, NT, LU>;
    constexpr size_t smem = forward_smem_bytes<K, G>();
    static bool optin[kMaxDeviceOrdinals] = {false};
    int slot = -1;
    cudaError_t err = device_slot(&slot);
    if (err != cudaSuccess) return err;
    if ((err = ensure_smem_optin(kern, smem, optin, slot)) != cudaSuccess) return err;
    const long long ngroups = (a.n + G - 1) / G;
    const int grid = int(ngroups < num_sms ? ngroups : num_sms);
    kern<<<grid, NT, smem, stream>>>(a);
    return cudaGetLastError();
}

constexpr size_t kOneCtaPerSm = 116 * 1024;        // dynamic shared memory of which an SM (228 KiB) holds one

// Cluster form with clusters of C CTAs and tile sets of GA and GB.  A launch uses at most as many clusters as the device runs at
// once, which depends on C only (one CTA fills an SM in every instantiation) and is asked for in a call of its own.
template <int K, int CB, int C, int GA, int GB, int NT, StepForm F = StepForm::kRounded>
static cudaError_t launch_cluster_variant(const ClusterArgs& ca, cudaStream_t stream) {
    auto kern = tcq_forward_cluster_kernel<K, CB, C, GA, GB, NT, F>;
    // Never less than half of what an SM has: two small CTAs on one SM leave another SM idle, and a step takes as long as
    // the slowest CTA of its cluster.
    constexpr size_t need = cluster_smem_bytes<K, C, GA, GB>(), smem = need < kOneCtaPerSm ? kOneCtaPerSm : need;
    static bool optin[kMaxDeviceOrdinals] = {false};
    int dev = -1;
    cudaError_t err = device_slot(&dev);
    if (err != cudaSuccess) return err;
    if (C > 8 && (dev < 0 || !optin[dev])) {
        if ((err = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return err;
    }
    if ((err = ensure_smem_optin(kern, smem, optin, dev)) != cudaSuccess) return err;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(NT);
    cfg.gridDim = dim3(C);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (ca.f.n <= 0) return cudaOccupancyMaxActiveClusters(ca.query, kern, &cfg);
    constexpr int G = GA + GB;
    const long long ngroups = (ca.f.n + G - 1) / G;
    const long long ncl = ngroups < ca.at_once ? ngroups : ca.at_once;
    cfg.gridDim = dim3(unsigned(ncl * C));
    return cudaLaunchKernelEx(&cfg, kern, ca);
}

// Relative time of one group of G tiles: G tiles of add-compare-select work plus
// one set of codebook evaluations shared by the group (about 0.85 of a tile's work).
static inline double group_cost(int G) { return double(G) + 0.85; }

// Picks the group size that finishes n tiles soonest on num_sms persistent CTAs.
template <int GMAX>
static int pick_group(long long n, int num_sms) {
    int best = 1;
    double best_t = 1e300;
    for (int G = 1; G <= GMAX; ++G) {
        const long long groups = (n + G - 1) / G;
        const long long rounds = (groups + num_sms - 1) / num_sms;
        const double t = double(rounds) * group_cost(G);
        if (t < best_t - 1e-9) { best_t = t; best = G; }
    }
    return best;
}

}  // namespace tcq
