// Viterbi step kernel instantiations for K = 2 bits per weight.
#include "tcq_forward_launch.cuh"

namespace tcq {

namespace {
template <int CB>
cudaError_t launch_cluster_cb(const ClusterArgs& ca, int C, int G, cudaStream_t stream) {
    // The shapes of pick_cluster.  Clusters of eight have 512 threads here (16 states each) and 256 at K = 3 and 4 (32 states):
    // 9 to 30 tiles 8 % faster at K = 2 (24 tiles 421 -> 388 us a call), 7-20 % slower for one tile at K = 3 and 4.
    if (ca.form != StepForm::kRounded) return cudaErrorInvalidValue;
    switch (100 * C + G) {
        case 1601: return launch_cluster_variant<2, CB, 16, 1, 0, 256>(ca, stream);
        case 801: return launch_cluster_variant<2, CB, 8, 1, 0, 512>(ca, stream);
        case 802: return launch_cluster_variant<2, CB, 8, 1, 1, 512>(ca, stream);
        case 401: return launch_cluster_variant<2, CB, 4, 1, 0, 512>(ca, stream);
        case 201: return launch_cluster_variant<2, CB, 2, 1, 0, 512>(ca, stream);
        case 202: return launch_cluster_variant<2, CB, 2, 1, 1, 512>(ca, stream);
        case 203: return launch_cluster_variant<2, CB, 2, 2, 1, 512>(ca, stream);
        default: return cudaErrorInvalidValue;
    }
}

template <int CB>
cudaError_t launch_cta_cb(const ForwardArgs& a, int num_sms, cudaStream_t stream) {
    constexpr int NT = 512, LU = 4;
    switch (pick_group<1>(a.n, num_sms)) {
        case 1: return launch_variant<2, CB, 1, NT, LU>(a, num_sms, stream);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace

template <>
cudaError_t launch_forward_cluster<2>(int codebook, const ClusterArgs& ca, int C, int G, cudaStream_t stream) {
    switch (codebook) {
        case kCb1Mad:  return launch_cluster_cb<kCb1Mad>(ca, C, G, stream);
        case kCb3Inst: return launch_cluster_cb<kCb3Inst>(ca, C, G, stream);
        case kCbMcg:   return launch_cluster_cb<kCbMcg>(ca, C, G, stream);
        default:       return cudaErrorInvalidValue;
    }
}

template <>
cudaError_t launch_forward_cta<2>(int codebook, const ForwardArgs& a, int num_sms, cudaStream_t stream) {
    switch (codebook) {
        case kCb1Mad:  return launch_cta_cb<kCb1Mad>(a, num_sms, stream);
        case kCb3Inst: return launch_cta_cb<kCb3Inst>(a, num_sms, stream);
        case kCbMcg:   return launch_cta_cb<kCbMcg>(a, num_sms, stream);
        default:       return cudaErrorInvalidValue;
    }
}

}  // namespace tcq
