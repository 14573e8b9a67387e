// The traceback kernels' launcher (tcq_traceback.cu) and those of the decode, packing and incoherence-processing kernels.
#pragma once

#include "tcq_forward.cuh"

namespace tcq {

// Smallest workspace that takes n tiles in one chunk (tcq_capi.cu).
size_t backpointer_workspace_bytes(long long n, int K);

cudaError_t launch_traceback(int K, const TracebackArgs& args, cudaStream_t stream);

// Decode / packing kernels (tcq_decode.cu).
cudaError_t launch_decode_packed(const uint32_t* packed, long long n, int K, int codebook, float* dq, cudaStream_t stream);
cudaError_t launch_decode_matvec(const uint32_t* packed, long long n_out, long long k_in, int K, int codebook, const float* x,
                                 long long ldx, int m, float* y, long long ldy, cudaStream_t stream);
cudaError_t launch_decode_symbols(const long long* bits, long long n, long long T, int K, int codebook,
                                  const long long* s0, float* out, cudaStream_t stream);
cudaError_t launch_pack_symbols(const long long* bits, long long n, int K, uint32_t* packed, cudaStream_t stream);
cudaError_t launch_codebook_lut(int codebook, float* lut, cudaStream_t stream);

// Incoherence processing (tcq_ip.cu).
size_t ip_workspace_bytes(long long n, long long k);
cudaError_t launch_ip_forward(const float* w, long long n, long long k, const float* sv, const float* su, float cb_rms,
                              int tiled, float* z_out, float* out_s, float* in_s, float* scale, void* ws, cudaStream_t stream);
cudaError_t launch_ip_restore(const float* zq, int tiled, long long n, long long k, const float* sv, const float* su,
                              const float* out_s, const float* in_s, const float* scale, float* w_hat, void* ws,
                              cudaStream_t stream);

}  // namespace tcq
