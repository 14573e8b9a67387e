// Viterbi step kernel instantiations for K = 4 bits per weight.
#include "tcq_forward_launch.cuh"

namespace tcq {

namespace {
template <int CB>
cudaError_t launch_cluster_cb(const ClusterArgs& ca, int C, int G, cudaStream_t stream) {
    if (ca.form == StepForm::kListed) return launch_cluster_variant<4, CB, 2, 1, 1, 512, StepForm::kListed>(ca, stream);
    if (ca.form == StepForm::kFused)
        switch (G) {
            case 1: return launch_cluster_variant<4, CB, 2, 1, 0, 512, StepForm::kFused>(ca, stream);
            case 2: return launch_cluster_variant<4, CB, 2, 1, 1, 512, StepForm::kFused>(ca, stream);
            case 3: return launch_cluster_variant<4, CB, 2, 2, 1, 512, StepForm::kFused>(ca, stream);
            case 4: return launch_cluster_variant<4, CB, 2, 2, 2, 512, StepForm::kFused>(ca, stream);
            case 5: return launch_cluster_variant<4, CB, 2, 3, 2, 512, StepForm::kFused>(ca, stream);
            case 6: return launch_cluster_variant<4, CB, 2, 3, 3, 512, StepForm::kFused>(ca, stream);
            default: return cudaErrorInvalidValue;
        }
    switch (100 * C + G) {                       // the shapes of pick_cluster
        case 801: return launch_cluster_variant<4, CB, 8, 1, 0, 256>(ca, stream);
        case 401: return launch_cluster_variant<4, CB, 4, 1, 0, 512>(ca, stream);
        case 201: return launch_cluster_variant<4, CB, 2, 1, 0, 512>(ca, stream);
        case 202: return launch_cluster_variant<4, CB, 2, 1, 1, 512>(ca, stream);
        case 203: return launch_cluster_variant<4, CB, 2, 2, 1, 512>(ca, stream);
        case 204: return launch_cluster_variant<4, CB, 2, 2, 2, 512>(ca, stream);
        case 205: return launch_cluster_variant<4, CB, 2, 3, 2, 512>(ca, stream);
        case 206: return launch_cluster_variant<4, CB, 2, 3, 3, 512>(ca, stream);
        default: return cudaErrorInvalidValue;
    }
}

template <int CB>
cudaError_t launch_cta_cb(const ForwardArgs& a, int num_sms, cudaStream_t stream) {
    constexpr int NT = 512, LU = 4;
    switch (pick_group<3>(a.n, num_sms)) {
        case 1: return launch_variant<4, CB, 1, NT, LU>(a, num_sms, stream);
        case 2: return launch_variant<4, CB, 2, NT, LU>(a, num_sms, stream);
        case 3: return launch_variant<4, CB, 3, NT, LU>(a, num_sms, stream);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace

template <>
cudaError_t launch_forward_cluster<4>(int codebook, const ClusterArgs& ca, int C, int G, cudaStream_t stream) {
    switch (codebook) {
        case kCb1Mad:  return launch_cluster_cb<kCb1Mad>(ca, C, G, stream);
        case kCb3Inst: return launch_cluster_cb<kCb3Inst>(ca, C, G, stream);
        case kCbMcg:   return launch_cluster_cb<kCbMcg>(ca, C, G, stream);
        default:       return cudaErrorInvalidValue;
    }
}

template <>
cudaError_t launch_forward_cta<4>(int codebook, const ForwardArgs& a, int num_sms, cudaStream_t stream) {
    switch (codebook) {
        case kCb1Mad:  return launch_cta_cb<kCb1Mad>(a, num_sms, stream);
        case kCb3Inst: return launch_cta_cb<kCb3Inst>(a, num_sms, stream);
        case kCbMcg:   return launch_cta_cb<kCbMcg>(a, num_sms, stream);
        default:       return cudaErrorInvalidValue;
    }
}

}  // namespace tcq
