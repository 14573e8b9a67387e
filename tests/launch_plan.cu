// The encoder's host side on a made-up CUDA runtime, so that what it launches can be looked at without a GPU: the real argument
// checks, scratch plans and cluster queries (tcq_capi.cu, tcq_forward_launch.cuh) over the entry points of
// launch_plan_runtime.cpp.  Built and run by test_launch_plan.py.  Arguments, in order:
//   fail N             the next N occupancy queries fail
//   encode K N BYTES   tcq_encode_tb of N tiles with BYTES of scratch (0: what tcq_workspace_bytes says)
//   pass K N BYTES     tcq_viterbi_pass, unconstrained, likewise
//   size K N 0         what tcq_workspace_bytes says
//   shapes K           the shapes that a launch may have
//   forms K            the same by form
// Each launch, each call's status and each shape is printed on a line.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../trellis-everywhere_b200/csrc/tcq_forward_launch.cuh"
#include "../trellis-everywhere_b200/csrc/tcq_traceback.cuh"

extern int g_failing_queries;

// What a call puts where in its scratch: complaints about bytes outside, and about bytes that another buffer holds.
constexpr uintptr_t kScratch = 1 << 22;
static size_t g_scratch_bytes = 0;
static long long g_span = 0;           // tiles whose walks have shared a list so far
struct Use { std::string what; uintptr_t begin, end; };
static std::vector<Use> g_uses;
static void use(const std::string& what, const void* p, size_t bytes) {
    const Use u{what, reinterpret_cast<uintptr_t>(p), reinterpret_cast<uintptr_t>(p) + bytes};
    if (u.begin < kScratch + 4 || u.end > kScratch + g_scratch_bytes) std::printf("outside: %s\n", what.c_str());     // (the status word comes first)
    for (const Use& o : g_uses)
        if (o.what != what && !(o.what == "edges" && what == "overlap") && !(o.what == "overlap" && what == "edges") && u.begin < o.end && o.begin < u.end)
            std::printf("shared: %s, %s\n", what.c_str(), o.what.c_str());
    g_uses.push_back(u);
}

namespace tcq {

static cudaError_t cluster(int K, const ClusterArgs& ca, int C, int G) {
    // queries go through the real launcher (of the size with the smallest kernel for all but one)
    if (ca.f.n <= 0) return C == 16 ? launch_cluster_variant<2, kCbMcg, 16, 1, 0, 256>(ca, nullptr) : C == 8 ? launch_cluster_variant<2, kCbMcg, 8, 1, 0, 512>(ca, nullptr)
                          : C == 4 ? launch_cluster_variant<2, kCbMcg, 4, 1, 0, 512>(ca, nullptr) : launch_cluster_variant<2, kCbMcg, 2, 1, 0, 512>(ca, nullptr);
    const char* const form = ca.form == StepForm::kFused ? "fused" : ca.form == StepForm::kListed ? "listed" : "rounded";
    std::printf("cluster K=%d C=%d G=%d n=%lld steps=%d %s\n", K, C, G, ca.f.n, ca.f.steps, form);
    const bool fused = ca.form == StepForm::kFused, listed = ca.form == StepForm::kListed;
    if (listed && (C * ca.at_once > 148 || ca.f.n > G * ca.at_once)) std::printf("outside: more listed tiles than clusters\n");
    use("rows", ca.rows, ca.f.n * ca.nrows * (size_t(4) << (16 - K)));
    if (ca.keys != nullptr) use("keys", ca.keys, ca.f.n * C * 8 * (fused ? kFusedKeys : 1));
    // (a listed tile's overlap lies anywhere in the span, whose walks have said how large it is)
    if (ca.f.overlap != nullptr) use("overlap", ca.f.overlap, listed ? g_span * 4 : ca.f.n * 4);
    if (fused) use("counts", ca.counts, 2 * sizeof(int));
    if (listed) use("list", ca.list, g_span * 4), use("counts", ca.list_count, sizeof(int));
    if (listed && ca.walk.keys != ca.keys) std::printf("outside: keys of the listed walk\n");
    if (listed && ca.walk.e_out != nullptr) use("edges", ca.walk.e_out, g_span * 4);
    return cudaSuccess;
}
static cudaError_t cta(int K, const ForwardArgs& a) {
    std::printf("cta K=%d n=%lld\n", K, a.n);
    return cudaSuccess;
}
template <> cudaError_t launch_forward_cluster<2>(int, const ClusterArgs& ca, int C, int G, cudaStream_t) { return cluster(2, ca, C, G); }
template <> cudaError_t launch_forward_cluster<3>(int, const ClusterArgs& ca, int C, int G, cudaStream_t) { return cluster(3, ca, C, G); }
template <> cudaError_t launch_forward_cluster<4>(int, const ClusterArgs& ca, int C, int G, cudaStream_t) { return cluster(4, ca, C, G); }
template <> cudaError_t launch_forward_cta<2>(int, const ForwardArgs& a, int, cudaStream_t) { return cta(2, a); }
template <> cudaError_t launch_forward_cta<3>(int, const ForwardArgs& a, int, cudaStream_t) { return cta(3, a); }
template <> cudaError_t launch_forward_cta<4>(int, const ForwardArgs& a, int, cudaStream_t) { return cta(4, a); }
cudaError_t launch_traceback(int, const TracebackArgs& a, cudaStream_t) {
    std::printf("walk %s n=%lld keys=%d\n", a.rows != nullptr ? "rows" : "backpointers", a.n, a.keys != nullptr ? a.nkeys : 0);
    if (a.e_out != nullptr) use("edges", a.e_out, a.n * 4);
    if (a.keys != nullptr) use("keys", a.keys, a.n * a.nkeys * 8);
    if (a.fused) {
        if (a.first_tile == 0) g_span = 0;
        g_span = a.first_tile + a.n > g_span ? a.first_tile + a.n : g_span;
        use("list", a.again, g_span * 4), use("counts", a.again_count, sizeof(int));
    }
    return cudaSuccess;
}
cudaError_t launch_decode_packed(const uint32_t*, long long, int, int, float*, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t launch_decode_matvec(const uint32_t*, long long, long long, int, int, const float*, long long, int, float*, long long, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t launch_decode_symbols(const long long*, long long, long long, int, int, const long long*, float*, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t launch_pack_symbols(const long long*, long long, int, uint32_t*, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t launch_codebook_lut(int, float*, cudaStream_t) { return cudaErrorUnknown; }
size_t ip_workspace_bytes(long long, long long) { return 0; }
cudaError_t launch_ip_forward(const float*, long long, long long, const float*, const float*, float, int, float*, float*, float*, float*, void*, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t launch_ip_restore(const float*, int, long long, long long, const float*, const float*, const float*, const float*, const float*, float*, void*, cudaStream_t) { return cudaErrorUnknown; }

}  // namespace tcq

#include "../trellis-everywhere_b200/csrc/tcq_capi.cu"

int main(int argc, char** argv) {
    auto address = [](uintptr_t a) { return reinterpret_cast<void*>(a); };          // aligned and never read
    for (int i = 1; i < argc;) {
        if (!std::strcmp(argv[i], "fail")) {
            g_failing_queries = std::atoi(argv[i + 1]);
            i += 2;
        } else if (!std::strcmp(argv[i], "shapes")) {
            const auto [s, n] = shapes(std::atoi(argv[i + 1]));
            for (int j = 0; j < n; ++j) std::printf("C=%d G=%d\n", s[j].C, s[j].G);
            i += 2;
        } else if (!std::strcmp(argv[i], "forms")) {
            const int K = std::atoi(argv[i + 1]);
            for (bool fused : {false, true}) {
                const auto [s, n] = shapes(K, fused);
                for (int j = 0; j < n && (!fused || K > 2); ++j) std::printf("C=%d G=%d %s\n", s[j].C, s[j].G, fused ? "fused" : "rounded");
            }
            i += 2;
        } else if (!std::strcmp(argv[i], "size")) {
            std::printf("%zu\n", tcq_workspace_bytes(std::atoll(argv[i + 2]), std::atoi(argv[i + 1])));
            i += 4;
        } else {
            const int K = std::atoi(argv[i + 1]);
            const long long n = std::atoll(argv[i + 2]), bytes = std::atoll(argv[i + 3]);
            g_scratch_bytes = bytes > 0 ? size_t(bytes) : tcq_workspace_bytes(n, K);
            g_uses.clear();
            g_span = 0;
            const float* const w = static_cast<float*>(address(1 << 20));
            std::printf("status %d\n", !std::strcmp(argv[i], "pass")
                                           ? tcq_viterbi_pass(w, n, K, 2, nullptr, 0, static_cast<int64_t*>(address(1 << 21)), address(kScratch), g_scratch_bytes, nullptr)
                                           : tcq_encode_tb(w, n, K, 2, static_cast<uint32_t*>(address(1 << 21)), nullptr, nullptr, nullptr, address(kScratch), g_scratch_bytes, nullptr));
            i += 4;
        }
    }
    return 0;
}
