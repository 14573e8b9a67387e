// C ABI of the B200 trellis codec (declared in include/tcq_b200.h): argument
// checking, workspace carving, chunking and the launch sequence.  No device
// memory is allocated or freed here and nothing synchronises with the host.
#include "../../include/tcq_b200.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <iterator>

#include "tcq_forward.cuh"
#include "tcq_traceback.cuh"

namespace {

using namespace tcq;

thread_local char g_last_cuda_error[256] = "";

int cuda_fail(cudaError_t err, const char* where) {
    std::snprintf(g_last_cuda_error, sizeof(g_last_cuda_error), "%s: %s", where, cudaGetErrorString(err));
    return TCQ_E_CUDA;
}

// SM count of the current device (cached per device ordinal).
int current_num_sms(int* out) {
    static int cache[64] = {0};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return cuda_fail(err, "cudaGetDevice");
    if (dev >= 0 && dev < 64 && cache[dev] > 0) { *out = cache[dev]; return TCQ_OK; }
    int sms = 0;
    err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return cuda_fail(err, "cudaDeviceGetAttribute");
    if (dev >= 0 && dev < 64) cache[dev] = sms;
    *out = sms;
    return TCQ_OK;
}

// How many clusters of C CTAs of the step kernel the current device runs at once (one CTA per SM); 0: none.
int clusters_at_once(int C) {
    static int cache[64][17] = {};                 // per device ordinal and C: 0 not known yet, -1 none
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || C < 2 || C > 16) return 0;
    const bool cached = dev >= 0 && dev < 64;
    int n = cached ? cache[dev][C] : 0;
    if (n == 0) {
        ClusterArgs ca{};                          // no tiles: a query.  One CTA fits an SM whatever K and the tiles per group are.
        ca.query = &n;
        if (launch_forward_cluster<2>(kCbMcg, ca, C, 1, nullptr) != cudaSuccess) {
            (void)cudaGetLastError();              // a failed query says nothing about the device: the next call asks again
            return 0;
        }
        if (n < 1) n = -1;
        if (cached) cache[dev][C] = n;
    }
    return n > 0 ? n : 0;
}

// TCQ_FORWARD_KERNEL = cta | cluster2 | cluster4 | cluster8 | cluster16, for comparison runs: the cluster size it asks for, 1 for the
// single-CTA kernel, 0 if it is not set or names none of them.
int kernel_asked_for() {
    const char* v = std::getenv("TCQ_FORWARD_KERNEL");
    if (v == nullptr) return 0;
    if (std::strcmp(v, "cta") == 0) return 1;
    for (const char* name : {"cluster2", "cluster4", "cluster8", "cluster16"})
        if (std::strcmp(v, name) == 0) return std::atoi(name + 7);
    return 0;
}

// Whether the cluster step kernel runs on the current device.
bool cluster_available() { return kernel_asked_for() != 1 && clusters_at_once(2) > 0; }

// How a batch is spread over the chip: clusters of C CTAs, G tiles each, and the time of one round of a 256-step sweep with
// all SMs of a B200 at work, measured.  A larger cluster divides a tile's step over more SMs, which shortens the step for
// the few tiles that then fit, no further than the exchange of metrics between SMs allows (0.4 us a step); more tiles per
// cluster share the step's fixed cost (0.35 us with two SMs; 0.45 us a tile beyond that at K = 3).
// (A shape that another beats in time and tiles at once is not listed: 4 x 2 everywhere, 8 x 2 at K = 4.)
struct ClusterShape { int C, G; double us; };
constexpr ClusterShape kShapes2[] = {{16, 1, 100}, {8, 1, 120}, {8, 2, 156}, {4, 1, 181}, {2, 1, 240}, {2, 2, 398}, {2, 3, 532}};
constexpr ClusterShape kShapes3[] = {{8, 1, 107}, {8, 2, 150}, {4, 1, 152}, {2, 1, 203}, {2, 2, 325}, {2, 3, 440}, {2, 4, 540}, {2, 5, 665}, {2, 6, 786}};
constexpr ClusterShape kShapes4[] = {{8, 1, 105}, {4, 1, 142}, {2, 1, 205}, {2, 2, 338}, {2, 3, 447}, {2, 4, 548}, {2, 5, 680}, {2, 6, 804}};

// With fused candidates (two SMs per cluster only).
constexpr ClusterShape kFusedShapes3[] = {{2, 1, 172}, {2, 2, 285}, {2, 3, 362}, {2, 4, 457}, {2, 5, 553}, {2, 6, 660}};
constexpr ClusterShape kFusedShapes4[] = {{2, 1, 172}, {2, 2, 299}, {2, 3, 370}, {2, 4, 461}, {2, 5, 590}, {2, 6, 661}};

struct ShapeList { const ClusterShape* s; int n; };
ShapeList shapes(int K, bool fused = false) {
    if (fused) return K == 3 ? ShapeList{kFusedShapes3, int(std::size(kFusedShapes3))} : ShapeList{kFusedShapes4, int(std::size(kFusedShapes4))};
    return K == 2 ? ShapeList{kShapes2, int(std::size(kShapes2))} : K == 3 ? ShapeList{kShapes3, int(std::size(kShapes3))} : ShapeList{kShapes4, int(std::size(kShapes4))};
}
bool has_cluster_size(int K, int C) {
    const ShapeList l = shapes(K);
    return std::any_of(l.s, l.s + l.n, [C](const ClusterShape& x) { return x.C == C; });
}

// The shape that finishes n tiles soonest, counting whole rounds.  (Clusters of 4, 8 and 16 leave SMs of
// some GPCs over: 33, 15 and 7 of them run at once on a B200's 148 SMs.)  only: this cluster size (0: any).
constexpr long long kTilesOf16 = 16;              // clusters of sixteen are for the smallest batches, no larger than this (key_words)
struct Sweep { ClusterShape shape; double us; };
Sweep pick_cluster(long long n, int K, int only, bool fused) {
    const auto [s, ns] = shapes(K, fused);
    Sweep best{{2, 2, 0}, 1e300};
    for (int i = 0; i < ns; ++i) {
        if (only != 0 ? s[i].C != only : s[i].C > 8 && n > kTilesOf16) continue;
        const long long at_once = clusters_at_once(s[i].C);
        if (at_once < 1) continue;
        const long long groups = (n + s[i].G - 1) / s[i].G, rounds = (groups + at_once - 1) / at_once;
        if (double(rounds) * s[i].us < best.us) best = Sweep{s[i], double(rounds) * s[i].us};
    }
    return best;
}

// A sweep as one launch, or as two: whole rounds of one shape and what is left in another, both with two SMs per cluster (the
// walk reads as many partial minima for every tile).  One shape for all of 768 tiles takes two rounds of six tiles, the second
// three quarters empty: 3394 us a call at K = 3, 3203 with a round of six and one of five; 500 tiles 2466 -> 2222 us, 300 at K = 2
// 2282 -> 1991.  5 us: a launch.  Only where it promises 4 %: the table is not better than that (256 tiles at K = 2, where it
// promises 2 %, took 3 % longer).
struct SweepPlan { ClusterShape first, second; long long n_first; double us; };
SweepPlan plan_sweep(long long n, int K, bool fused = false) {
    const int asked = kernel_asked_for(), only = asked > 1 ? asked : 0;
    const Sweep one = pick_cluster(n, K, only, fused);
    const SweepPlan whole{one.shape, one.shape, n, one.us};
    if (only != 0 && only != 2) return whole;
    SweepPlan best = whole;
    best.us *= 0.96;
    const auto [s, ns] = shapes(K, fused);
    for (int i = 0; i < ns; ++i) {
        const long long round = s[i].C == 2 ? (long long)clusters_at_once(2) * s[i].G : 0;
        if (round < 1 || n <= round || n % round == 0) continue;
        const Sweep rest = pick_cluster(n % round, K, 2, fused);
        const double us = double(n / round) * s[i].us + rest.us + 5.0;
        if (us < best.us) best = SweepPlan{s[i], rest.shape, n / round * round, us};
    }
    return best.n_first < n ? best : whole;
}

size_t rowb(int K) { return (size_t(1) << (kL - K)) * size_t(K) / 8; }
size_t bp_bytes_per_tile(int K) { return size_t(kT) * rowb(K); }
constexpr size_t kAlign = 256;
size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }

// Scratch comes in two forms.  The cluster step kernel leaves metric rows (MetricRows), the single-CTA kernel packed
// argmins of every step ("backpointers"), which are a quarter of the size.  The status word lies at the front in both.
int rows_for(int K, int steps) {
    return K == 2 ? MetricRows<2>::rows_for(steps) : K == 3 ? MetricRows<3>::rows_for(steps) : MetricRows<4>::rows_for(steps);
}

size_t rows_bytes_per_tile(int K, int part) { return size_t(rows_for(K, part)) * (size_t(1) << (kL - K)) * 4; }

// Partial minima left by the cluster kernel, one per tile and CTA of its cluster: eight a tile, sixteen for the tiles that clusters of
// sixteen may take.  (Sixteen for all took two thirds more beside the rows than there is beside the argmins, so that in the scratch of
// the argmins of n tiles the rows of half a path fitted n/2 - 1 of them: 64 tiles at K = 4 went in three chunks, 1376 us instead of 934.)
size_t key_words(long long chunk, int K) {
    if (kernel_asked_for() == 16) return 16 * size_t(chunk);
    return 8 * size_t(chunk) + (K == 2 ? 8 * size_t(chunk < kTilesOf16 ? chunk : kTilesOf16) : 0);
}
size_t beside_rows_bytes(long long chunk, int K) {             // status word, partial minima, overlaps, edges
    return align_up(64 + key_words(chunk, K) * sizeof(unsigned long long) + 2 * sizeof(int) * size_t(chunk));
}

// Bytes for `chunk` tiles with backpointers: those of one whole pass and two int32 hand-off arrays (and a part that is no longer used:
// what callers were told to bring stays the same).
size_t bp_ws_bytes(long long chunk, int K) {
    return align_up(size_t(chunk) * bp_bytes_per_tile(K)) + 2 * align_up(size_t(chunk) * sizeof(int)) +
           align_up(size_t(chunk) * 4 * sizeof(unsigned long long)) + kAlign /* status word */;
}
// ... with metric rows for walks over `part` steps at a time, the overlaps, the edges handed from part to part and the partial
// minima of the final metrics.
size_t rows_ws_bytes(long long chunk, int K, int part) {
    return beside_rows_bytes(chunk, K) + size_t(chunk) * rows_bytes_per_tile(K, part);
}

// Tiles per chunk at full speed.  Backpointers: eight rounds of the largest tile group on every SM.  Metric rows: two
// rounds of the largest group on every cluster, which takes no more memory.
long long bp_chunk(int num_sms) { return 8LL * 3 * num_sms; }
long long rows_chunk(int num_sms) { return 6LL * num_sms; }

struct Workspace {
    bool clustered;             // metric rows and the cluster step kernel; else backpointers and the single-CTA kernel
    int part;                   // steps whose metric rows the workspace holds for a chunk (256, or 128 or 64: see plan_rows)
    unsigned char* bp;
    float* rows;
    int* e_final;
    int* overlap;
    int* edge;
    unsigned long long* keys;
    unsigned int* status;
    long long chunk;
    // Sweeps with fused candidates (see plan_fused)
    bool fused;
    long long span;             // tiles that go through pass 1 before any goes through pass 2 (their overlaps are kept)
    int* list;                  // [span] tiles to sweep again
    int* counts;                // their numbers after the walks of pass 1 and of pass 2
};

// Batches from here on are swept with fused candidates, and the tiles whose path that does not settle again (one Gaussian tile in 10 000, by a
// kernel of its own after the walks of each pass).  Smaller ones are bound by the exchange between SMs and not by arithmetic, and there a
// tile swept again, 0.25 ms, is a larger part of a call: 148 tiles at K = 3 would gain 4 %.  At K = 2 a sweep gains less (444
// tiles 1115 -> 1022 us), and the longer walk takes most of it: 150 tiles 1220 -> 1230 us a call, 1000 tiles 5431 -> 5372.
constexpr int kFusedFrom = 149;
constexpr int kListedC = 2, kListedG = 2;          // (with four SMs a tile, a few tiles take 0.17 ms instead of 0.25, and a batch of nothing but such tiles longer)
constexpr long long kSpan = 1 << 18;               // the full-speed size holds the overlaps of so many tiles
bool plan_fused(long long n, int K, const Workspace& wk) {
    return K >= 3 && n >= kFusedFrom && wk.part == kT && kernel_asked_for() == 0 && wk.chunk >= (n < 2 * kFusedFrom ? n : 2 * kFusedFrom) && clusters_at_once(kListedC) > 0;
}
// Tiles of a chunk: whole rounds of the largest shape (six tiles a cluster), which has the most tiles per time.
long long fused_chunk() { return 12LL * clusters_at_once(2); }

// Largest chunk of at most `want` tiles; `need(chunk)` bytes, about per_tile each.
template <typename Need>
long long largest_chunk(long long want, size_t ws_bytes, size_t per_tile, long long wave, Need need) {
    if (need(want) <= ws_bytes) return want;
    // solve conservatively, then step down
    long long chunk = (long long)((ws_bytes > 5 * kAlign ? ws_bytes - 5 * kAlign : 0) / per_tile) + 1;
    if (chunk > want) chunk = want;
    while (chunk > 0 && need(chunk) > ws_bytes) --chunk;
    // whole rounds of full groups avoid a ragged last wave inside every chunk
    if (chunk > wave) chunk = chunk / wave * wave;
    return chunk;
}

long long bp_chunk_for(long long n, size_t ws_bytes, int K, int num_sms) {
    return largest_chunk(n < bp_chunk(num_sms) ? n : bp_chunk(num_sms), ws_bytes, bp_bytes_per_tile(K), 3LL * num_sms,
                         [K](long long c) { return bp_ws_bytes(c, K); });
}

// Sweeps of a pass whose path is walked in parts of `part` steps, last part first: the whole pass, then again up to each
// earlier part.  In steps, for the two passes of an encode (the first needs the second half of its path only).
int swept_steps(int part) { return part == 256 ? 512 : part == 128 ? 256 + 256 + 128 : (256 + 192) + (256 + 192 + 128 + 64); }

// Chunk and part for metric rows in ws_bytes: the whole path at once if that many tiles fit; a workspace too small for it holds
// half or a quarter of a path for two or four times the tiles, which pays (and for one tile may be all that fits) although
// the sweep is repeated for each part.  The walks and launches of a chunk: 86 us at 30 tiles, about 120 from 70 on and in halves, 200 in quarters.
void plan_rows(long long n, size_t ws_bytes, int K, int num_sms, long long* chunk, int* part) {
    *chunk = 0;
    *part = 256;
    double best = 1e300;
    for (int p = 256; p >= 64; p /= 2) {
        const long long want = n < rows_chunk(num_sms) ? n : rows_chunk(num_sms);
        long long c = largest_chunk(want, ws_bytes, rows_bytes_per_tile(K, p), 3LL * num_sms,
                                    [K, p](long long m) { return rows_ws_bytes(m, K, p); });
        if (c < 1) continue;
        const bool all = c >= want;
        const long long chunks = (n + c - 1) / c;
        // as many chunks as that takes, or one more, of equal size: a smaller one may fit a round of a faster shape
        for (long long m = chunks; m <= chunks + (all ? 0 : 1); ++m) {
            if (!all) c = (n + m - 1) / m;
            const double us = plan_sweep(c, K).us, rest = n % c != 0 ? plan_sweep(n % c, K).us : 0.0;
            const double total = (double(n / c) * us + rest) * swept_steps(p) / 256.0 + double((n + c - 1) / c) * (p == 256 ? 60.0 + (c < 67 ? 0.9 * double(c) : 60.0) : p == 128 ? 120.0 : 200.0);
            if (total < best) {
                best = total;
                *chunk = c;
                *part = p;
            }
        }
        if (all) break;                            // smaller parts gain nothing
    }
}

// fusible: whether the caller can do with sweeps with fused candidates.
int carve(void* ws, size_t ws_bytes, long long n, int K, int num_sms, Workspace* out, bool fusible) {
    if (ws == nullptr) return TCQ_E_NULL_POINTER;
    if (reinterpret_cast<uintptr_t>(ws) % kAlign) return TCQ_E_MISALIGNED;
    if (kernel_asked_for() > 1 && !has_cluster_size(K, kernel_asked_for())) return TCQ_E_BAD_ARGUMENT;
    *out = Workspace{};
    out->chunk = bp_chunk_for(n, ws_bytes, K, num_sms);
    if (out->chunk < 1) return TCQ_E_WORKSPACE;
    out->part = kT;
    unsigned char* const base = static_cast<unsigned char*>(ws);
    out->status = reinterpret_cast<unsigned int*>(base);
    if (cluster_available()) {
        long long chunk = 0;
        plan_rows(n, ws_bytes, K, num_sms, &chunk, &out->part);
        if (chunk >= 1) {
            out->clustered = true;
            out->chunk = chunk;
            out->keys = reinterpret_cast<unsigned long long*>(base + 64);
            out->overlap = reinterpret_cast<int*>(out->keys + key_words(chunk, K));
            out->edge = out->overlap + chunk;
            out->rows = reinterpret_cast<float*>(base + beside_rows_bytes(chunk, K));
            if (fusible && plan_fused(n, K, *out)) {
                // as above, with the overlaps and the list of a span in all that the rows of a chunk leave over
                const long long c = n <= chunk ? n : fused_chunk() < chunk ? fused_chunk() : chunk;
                const size_t rows = size_t(c) * rows_bytes_per_tile(K, kT), keys = 64 + size_t(c) * 2 * kFusedKeys * sizeof(unsigned long long);
                const size_t left = (ws_bytes - rows) / kAlign * kAlign;
                const long long span = left < keys ? 0 : (long long)((left - keys) / (2 * sizeof(int)));
                if (span >= c) {
                    out->fused = true;
                    out->chunk = c;
                    out->span = n < span ? n : span / c * c;
                    out->counts = reinterpret_cast<int*>(base + 16);
                    out->overlap = reinterpret_cast<int*>(base + keys);
                    out->list = out->overlap + out->span;
                    out->rows = reinterpret_cast<float*>(base + align_up(keys + size_t(out->span) * 2 * sizeof(int)));
                }
            }
            return TCQ_OK;
        }
    }
    const size_t ints = align_up(size_t(out->chunk) * sizeof(int));
    out->overlap = reinterpret_cast<int*>(base + kAlign);
    out->e_final = reinterpret_cast<int*>(base + kAlign + ints);
    out->bp = base + kAlign + 2 * ints;
    return TCQ_OK;
}

// One sweep of the step kernel over a chunk: a.steps steps, of whose path the last a.bp_steps will be walked.
// Fills in what the traceback needs to know of it.
cudaError_t forward(int K, int codebook, const ForwardArgs& a, const Workspace& wk, int num_sms, cudaStream_t s, TracebackArgs* t) {
    t->n = a.n;
    t->bp_steps = a.bp_steps;
    t->t_end = a.steps;
    t->codebook = codebook;
    t->w = a.w;
    t->w_add = a.w_add;
    t->ld = a.ld;
    t->roll = a.roll;
    t->status = a.status;
    t->overlap = a.overlap;
    t->e_start = a.overlap != nullptr ? a.overlap : wk.e_final;
    t->keys = nullptr;
    if (wk.clustered) {
        const SweepPlan plan = plan_sweep(a.n, K, wk.fused);
        ClusterArgs ca{a, wk.rows, rows_for(K, wk.fused ? kT : a.bp_steps), a.overlap == nullptr && a.steps == kT ? wk.keys : nullptr};
        ca.form = wk.fused ? StepForm::kFused : StepForm::kRounded;
        ca.counts = wk.counts;
        t->rows = wk.rows;
        t->nrows = ca.nrows;
        t->other_order = K == 3 && plan.first.C == 2;      // (both launches of a sweep have as many CTAs per cluster)
        t->keys = ca.keys;
        t->nkeys = plan.first.C * (wk.fused ? kFusedKeys : 1);
        t->fused = wk.fused;
        auto launch = [&](const ClusterShape& shape) -> cudaError_t {
            ca.at_once = clusters_at_once(shape.C);
            if (ca.at_once < 1) return cudaErrorNotSupported;
            switch (K) {
                case 2: return launch_forward_cluster<2>(codebook, ca, shape.C, shape.G, s);
                case 3: return launch_forward_cluster<3>(codebook, ca, shape.C, shape.G, s);
                case 4: return launch_forward_cluster<4>(codebook, ca, shape.C, shape.G, s);
                default: return cudaErrorInvalidValue;
            }
        };
        ca.f.n = plan.n_first;
        cudaError_t err = launch(plan.first);
        if (err != cudaSuccess || plan.n_first == a.n) return err;
        const long long at = plan.n_first, tile_step = a.ld > 0 ? 16 : kT;
        ca.f.n = a.n - at;
        ca.f.w += at * tile_step;
        if (ca.f.w_add != nullptr) ca.f.w_add += at * tile_step;
        if (ca.f.overlap != nullptr) ca.f.overlap += at;
        if (ca.f.final_cost != nullptr) ca.f.final_cost += at;
        ca.f.flags &= ~(kFwdResetStatus | kFwdResetCounts);      // the first launch has cleared them
        ca.rows += size_t(at) * ca.nrows * (size_t(1) << (kL - K));
        if (ca.keys != nullptr) ca.keys += at * t->nkeys;
        return launch(plan.second);
    }
    t->bp = wk.bp;
    switch (K) {
        case 2: return launch_forward_cta<2>(codebook, a, num_sms, s);
        case 3: return launch_forward_cta<3>(codebook, a, num_sms, s);
        case 4: return launch_forward_cta<4>(codebook, a, num_sms, s);
        default: return cudaErrorInvalidValue;
    }
}

// One pass over a chunk and the walk back over its last `walk` steps (256 or 128), in parts if the workspace holds the rows of
// a part only.  `out`: the walk's outputs; its e_out gets the edge before the first walked step.
int pass(int K, int codebook, ForwardArgs f, int walk, TracebackArgs out, const Workspace& wk, int num_sms, cudaStream_t s, const char* what) {
    int* const e_out = out.e_out;
    const int first = kT - walk;
    for (int end = kT; end > first;) {
        const int begin = end - wk.part > first ? end - wk.part : first;
        f.steps = end;
        f.bp_steps = end - begin;
        cudaError_t err = forward(K, codebook, f, wk, num_sms, s, &out);
        if (err != cudaSuccess) return cuda_fail(err, what);
        if (end < kT) out.e_start = wk.edge;       // where the later part's walk arrived
        out.e_out = begin == first ? e_out : wk.edge;
        if ((err = launch_traceback(K, out, s)) != cudaSuccess) return cuda_fail(err, what);
        f.final_cost = nullptr;                    // the first sweep is the whole pass: it reported
        f.e_final = nullptr;
        f.flags = 0;
        end = begin;
    }
    return TCQ_OK;
}

// The tiles of a span that the walks of a pass have listed, swept and walked again with every operation rounded: one kernel, which ends
// at once if there are none.  f, t: the pass and its outputs from the span's first tile on.
int listed(int K, int codebook, ForwardArgs f, int walk, TracebackArgs t, const Workspace& wk, const int* count, cudaStream_t s, const char* what) {
    f.steps = kT;
    f.bp_steps = walk;
    ClusterArgs ca{f, wk.rows, rows_for(K, walk), f.overlap == nullptr ? wk.keys : nullptr};
    ca.at_once = clusters_at_once(kListedC);
    if (ca.at_once > wk.chunk / kListedG) ca.at_once = int(wk.chunk / kListedG);         // rows of two tiles per cluster
    ca.f.n = kListedG * (f.n < ca.at_once ? f.n : ca.at_once);
    ca.form = StepForm::kListed;
    ca.list = wk.list;
    ca.list_count = count;
    t.rows = wk.rows;
    t.nrows = ca.nrows;
    t.w = f.w;
    t.w_add = f.w_add;
    t.ld = f.ld;
    t.roll = f.roll;
    t.overlap = t.e_start = f.overlap;
    t.keys = ca.keys;
    t.nkeys = kListedC;
    t.other_order = K == 3;
    t.bp_steps = walk;
    t.t_end = kT;
    t.codebook = codebook;
    ca.walk = t;
    const cudaError_t err = K == 3 ? launch_forward_cluster<3>(codebook, ca, kListedC, kListedG, s) : launch_forward_cluster<4>(codebook, ca, kListedC, kListedG, s);
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, what);
}

// Launches of an encode for a chunk of n tiles: a sweep (of one or two launches) and a walk for each part of the two passes.
int launches_of_chunk(long long n, int K, const Workspace& wk) {
    const int parts = (wk.part >= 128 ? 1 : 2) + 256 / wk.part;
    return parts * (wk.clustered && plan_sweep(n, K, wk.fused).n_first < n ? 3 : 2);
}

int check_common(int K, int codebook, long long n) {
    if (K < 2 || K > 4) return TCQ_E_BAD_K;
    if (codebook < 0 || codebook > 2) return TCQ_E_BAD_CODEBOOK;
    if (n < 0) return TCQ_E_BAD_COUNT;
    return TCQ_OK;
}

bool misaligned(const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a != 0; }

// What one tail-biting encode reads and writes; tiles (ld == 0) or an LDLQ row block (ld > 0).
struct EncodeIO {
    const float* w;
    const float* w_add;
    long long ld;
    long long n;               // tiles
    uint32_t* packed;
    long long packed_stride;
    int64_t* bits;
    float* dq;
    float* sse;
    float* wq;
    float* err;
    bool hurry;                // see TracebackArgs
};

// The launch sequence of the tail-biting encoder (src/trellis/qtip.py:135-144) per workspace chunk:
// step kernel on the rotated tile -> traceback to the overlap -> step kernel tied to the overlap -> traceback.
// The first step kernel of the call clears the workspace's status word itself (no separate memset node).
int encode_core(const EncodeIO& io, int K, int codebook, void* ws, size_t ws_bytes, cudaStream_t s) {
    int rc, num_sms = 0;
    if ((rc = current_num_sms(&num_sms)) != TCQ_OK) return rc;
    Workspace wk;
    if ((rc = carve(ws, ws_bytes, io.n, K, num_sms, &wk, true)) != TCQ_OK) return rc;
    // start of tile c0 inside w / w_add / wq / err: whole tiles (1 KiB each) or 16 columns of the row block per tile
    const long long tile_step = io.ld > 0 ? 16 : kT;
    // pass 1 over cn tiles from c0 on: tile rotated by half its length, free start; only the second half of the path is needed, to
    // reach the state at rotated position 128 (qtip.py:138-141)
    auto forward_1 = [&](long long c0, long long cn) {
        return ForwardArgs{io.w + c0 * tile_step, io.w_add ? io.w_add + c0 * tile_step : nullptr, io.ld, cn, nullptr, kT / 2, 0, 0, wk.bp, wk.e_final, nullptr, 1.0f, 0,
                           wk.status, c0 == 0 ? kFwdResetStatus : 0};
    };
    // pass 2: true order, start and end tied to the overlap (qtip.py:142)
    auto forward_2 = [&](long long c0, long long cn, const int* overlap) {
        return ForwardArgs{io.w + c0 * tile_step, io.w_add ? io.w_add + c0 * tile_step : nullptr, io.ld, cn, overlap, 0, 0, 0, wk.bp, nullptr, io.sse ? io.sse + c0 : nullptr, 1.0f, 0,
                           wk.status, kFwdCheckFinite};
    };
    auto outputs = [&](long long c0) {
        TracebackArgs t{};
        t.bits = io.bits ? reinterpret_cast<long long*>(io.bits) + c0 * kT : nullptr;
        t.dq = io.dq ? io.dq + c0 * kT : nullptr;
        t.packed = io.packed ? io.packed + c0 * io.packed_stride : nullptr;
        t.packed_stride = io.packed_stride;
        t.wq = io.wq ? io.wq + c0 * tile_step : nullptr;
        t.err = io.err ? io.err + c0 * tile_step : nullptr;
        t.src = io.w + c0 * tile_step;
        t.hurry = io.hurry;
        return t;
    };
    if (!wk.fused) {
        for (long long c0 = 0; c0 < io.n; c0 += wk.chunk) {
            const long long cn = io.n - c0 < wk.chunk ? io.n - c0 : wk.chunk;
            TracebackArgs t1{};
            t1.e_out = wk.overlap;
            t1.hurry = io.hurry;
            if ((rc = pass(K, codebook, forward_1(c0, cn), kT / 2, t1, wk, num_sms, s, "pass 1")) != TCQ_OK) return rc;
            if ((rc = pass(K, codebook, forward_2(c0, cn, wk.overlap), kT, outputs(c0), wk, num_sms, s, "pass 2")) != TCQ_OK) return rc;
        }
        return TCQ_OK;
    }
    // Both passes of a whole span one after the other, so that the tiles that a pass has to sweep again, few and anywhere, go together.
    for (long long s0 = 0; s0 < io.n; s0 += wk.span) {
        const long long sn = io.n - s0 < wk.span ? io.n - s0 : wk.span;
        for (int second = 0; second < 2; ++second) {
            for (long long c0 = 0; c0 < sn; c0 += wk.chunk) {
                const long long cn = sn - c0 < wk.chunk ? sn - c0 : wk.chunk;
                ForwardArgs f = second ? forward_2(s0 + c0, cn, wk.overlap + c0) : forward_1(s0 + c0, cn);
                if (!second && c0 == 0) f.flags |= kFwdResetCounts;
                f.final_cost = nullptr;            // the walk sums it up by the defined operations
                TracebackArgs t{};
                if (second) {
                    t = outputs(s0 + c0);
                    t.sse = io.sse ? io.sse + s0 + c0 : nullptr;
                } else {
                    t.e_out = wk.overlap + c0;
                }
                t.again = wk.list;
                t.again_count = wk.counts + second;
                t.first_tile = int(c0);
                t.hurry = io.hurry;
                if ((rc = pass(K, codebook, f, second ? kT : kT / 2, t, wk, num_sms, s, second ? "pass 2" : "pass 1")) != TCQ_OK) return rc;
            }
            ForwardArgs f = second ? forward_2(s0, sn, wk.overlap) : forward_1(s0, sn);
            f.flags = 0;
            TracebackArgs t{};
            if (second) t = outputs(s0);
            else t.e_out = wk.overlap;
            if ((rc = listed(K, codebook, f, second ? kT : kT / 2, t, wk, wk.counts + second, s, second ? "pass 2, listed tiles" : "pass 1, listed tiles")) != TCQ_OK) return rc;
        }
    }
    return TCQ_OK;
}

}  // namespace

size_t tcq::backpointer_workspace_bytes(long long n, int K) { return bp_ws_bytes(n, K); }

extern "C" {

int tcq_abi_version(void) { return 4; }

const char* tcq_strerror(int code) {
    switch (code) {
        case TCQ_OK: return "ok";
        case TCQ_E_BAD_K: return "K must be 2, 3 or 4";
        case TCQ_E_BAD_CODEBOOK: return "unknown codebook id (0 = 1mad, 1 = 3inst, 2 = mcg)";
        case TCQ_E_BAD_COUNT: return "negative tile or element count";
        case TCQ_E_NULL_POINTER: return "a required pointer is NULL";
        case TCQ_E_MISALIGNED: return "pointer is not aligned as the interface requires";
        case TCQ_E_WORKSPACE: return "workspace is smaller than tcq_workspace_min_bytes(K)";
        case TCQ_E_CUDA: return "CUDA runtime error (see tcq_last_cuda_error)";
        case TCQ_E_BAD_ARGUMENT: return "invalid argument";
        case TCQ_E_NONFINITE_INPUT: return "a weight was NaN or infinite; the codes of its tile are meaningless";
        case TCQ_E_DEVICE_TIMEOUT: return "a bounded wait inside a kernel gave up; the outputs of that call are invalid";
        case TCQ_E_TOO_MANY_TILES: return "more tiles than the static scratch holds (see tcq_encode_tb_static_max_tiles)";
        default: return "unknown error code";
    }
}

const char* tcq_last_cuda_error(void) { return g_last_cuda_error; }

size_t tcq_workspace_min_bytes(int K) {
    if (K < 2 || K > 4) return 0;
    return bp_ws_bytes(1, K);
}

size_t tcq_workspace_bytes(int64_t n_tiles, int K) {
    if (K < 2 || K > 4 || n_tiles < 0) return 0;
    int num_sms = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0) num_sms = sms;
    } else {
        (void)cudaGetLastError();
    }
    const long long n = n_tiles < 1 ? 1 : n_tiles;
    const size_t bp = bp_ws_bytes(n < bp_chunk(num_sms) ? n : bp_chunk(num_sms), K);
    size_t rows = rows_ws_bytes(n < rows_chunk(num_sms) ? n : rows_chunk(num_sms), K, kT);
    if (n > rows_chunk(num_sms)) rows += align_up(2 * sizeof(int) * size_t((n < kSpan ? n : kSpan) - rows_chunk(num_sms)));
    return rows > bp ? rows : bp;
}

int tcq_encode_tb(const float* w, int64_t n_tiles, int K, int codebook, uint32_t* packed, int64_t* bits, float* dq,
                  float* sse, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_common(K, codebook, n_tiles);
    if (rc != TCQ_OK) return rc;
    if (n_tiles == 0) return TCQ_OK;
    if (w == nullptr || packed == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(w, 16) || misaligned(packed, 4) || (dq && misaligned(dq, 4)) || (bits && misaligned(bits, 8)) ||
        (sse && misaligned(sse, 4)))
        return TCQ_E_MISALIGNED;
    EncodeIO io{};
    io.w = w;
    io.n = n_tiles;
    io.packed = packed;
    io.packed_stride = kT * K / 32;
    io.bits = bits;
    io.dq = dq;
    io.sse = sse;
    return encode_core(io, K, codebook, ws, ws_bytes, static_cast<cudaStream_t>(stream));
}

int tcq_encode_tb_rows(const float* src, const float* comp, int64_t ld, int64_t n_out, int K, int codebook,
                       uint32_t* packed, int64_t packed_stride, float* wq, float* err, float* sse, void* ws,
                       size_t ws_bytes, void* stream) {
    int rc = check_common(K, codebook, n_out);
    if (rc != TCQ_OK) return rc;
    if (n_out % 16 || ld < n_out) return TCQ_E_BAD_ARGUMENT;
    if (packed != nullptr && packed_stride < kT * K / 32) return TCQ_E_BAD_ARGUMENT;
    if (n_out == 0) return TCQ_OK;
    if (src == nullptr || wq == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(src, 4) || (comp && misaligned(comp, 4)) || misaligned(wq, 4) || (err && misaligned(err, 4)) ||
        (packed && misaligned(packed, 4)) || (sse && misaligned(sse, 4)))
        return TCQ_E_MISALIGNED;
    EncodeIO io{};
    io.w = src;
    io.w_add = comp;
    io.ld = ld;
    io.n = n_out / 16;
    io.packed = packed;
    io.packed_stride = packed_stride;
    io.sse = sse;
    io.wq = wq;
    io.err = err;
    return encode_core(io, K, codebook, ws, ws_bytes, static_cast<cudaStream_t>(stream));
}

int tcq_viterbi_pass(const float* w, int64_t n_tiles, int K, int codebook, const int32_t* overlap, int roll,
                     int64_t* states, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_common(K, codebook, n_tiles);
    if (rc != TCQ_OK) return rc;
    if (roll != 0 && roll != kT / 2) return TCQ_E_BAD_ARGUMENT;
    if (n_tiles == 0) return TCQ_OK;
    if (w == nullptr || states == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(w, 16) || misaligned(states, 8) || (overlap && misaligned(overlap, 4))) return TCQ_E_MISALIGNED;
    int num_sms = 0;
    if ((rc = current_num_sms(&num_sms)) != TCQ_OK) return rc;
    Workspace wk;
    if ((rc = carve(ws, ws_bytes, n_tiles, K, num_sms, &wk, false)) != TCQ_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(wk.status, 0, sizeof(unsigned int), s) != cudaSuccess) return cuda_fail(cudaGetLastError(), "status reset");

    for (long long c0 = 0; c0 < n_tiles; c0 += wk.chunk) {
        const long long cn = n_tiles - c0 < wk.chunk ? n_tiles - c0 : wk.chunk;
        ForwardArgs f{w + c0 * kT, nullptr, 0, cn, overlap ? overlap + c0 : nullptr, roll, 0, 0, wk.bp,
                      overlap ? nullptr : wk.e_final, nullptr, 1.0f, 0, wk.status, kFwdCheckFinite};
        TracebackArgs t{};
        t.states = reinterpret_cast<long long*>(states) + c0 * kT;
        if ((rc = pass(K, codebook, f, kT, t, wk, num_sms, s, "viterbi pass")) != TCQ_OK) return rc;
    }
    return TCQ_OK;
}

int tcq_forward_pass(const float* w, int64_t n_tiles, int K, int codebook, const int32_t* overlap, int roll,
                     int bp_steps, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_common(K, codebook, n_tiles);
    if (rc != TCQ_OK) return rc;
    if ((roll != 0 && roll != kT / 2) || (bp_steps != kT && bp_steps != kT / 2)) return TCQ_E_BAD_ARGUMENT;
    if (n_tiles == 0) return TCQ_OK;
    if (w == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(w, 16) || (overlap && misaligned(overlap, 4))) return TCQ_E_MISALIGNED;
    int num_sms = 0;
    if ((rc = current_num_sms(&num_sms)) != TCQ_OK) return rc;
    Workspace wk;
    if ((rc = carve(ws, ws_bytes, n_tiles, K, num_sms, &wk, true)) != TCQ_OK) return rc;
    if (bp_chunk_for(n_tiles, ws_bytes, K, num_sms) < n_tiles) return TCQ_E_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(wk.status, 0, sizeof(unsigned int), s) != cudaSuccess) return cuda_fail(cudaGetLastError(), "status reset");
    for (long long c0 = 0; c0 < n_tiles; c0 += wk.chunk) {
        const long long cn = n_tiles - c0 < wk.chunk ? n_tiles - c0 : wk.chunk;
        ForwardArgs f{w + c0 * kT, nullptr, 0, cn, overlap ? overlap + c0 : nullptr, roll, bp_steps < wk.part ? bp_steps : wk.part, kT,
                      wk.bp, overlap ? nullptr : wk.e_final, nullptr, 1.0f, 0, wk.status, kFwdCheckFinite};
        if (!wk.clustered) f.bp_steps = bp_steps;
        TracebackArgs t{};
        const cudaError_t err = forward(K, codebook, f, wk, num_sms, s, &t);
        if (err != cudaSuccess) return cuda_fail(err, "forward");
    }
    return TCQ_OK;
}

int tcq_workspace_status(const void* ws, size_t ws_bytes, int64_t n_tiles, int K, void* stream) {
    if (K < 2 || K > 4) return TCQ_E_BAD_K;
    if (n_tiles <= 0) return n_tiles == 0 ? TCQ_OK : TCQ_E_BAD_COUNT;
    int num_sms = 0;
    int rc = current_num_sms(&num_sms);
    if (rc != TCQ_OK) return rc;
    Workspace wk;
    if ((rc = carve(const_cast<void*>(ws), ws_bytes, n_tiles, K, num_sms, &wk, true)) != TCQ_OK) return rc;
    unsigned int host = 0;
    cudaError_t err = cudaMemcpyAsync(&host, wk.status, sizeof(host), cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream));
    if (err == cudaSuccess) err = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if (err != cudaSuccess) return cuda_fail(err, "status read");
    if (host & 1u) return TCQ_E_DEVICE_TIMEOUT;
    return (host & 2u) ? TCQ_E_NONFINITE_INPUT : TCQ_OK;
}

int tcq_selftest_wait_timeout(const float* w, int64_t n_tiles, int K, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_common(K, 0, n_tiles);
    if (rc != TCQ_OK) return rc;
    if (n_tiles < 1 || n_tiles > 8) return TCQ_E_BAD_COUNT;
    if (w == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(w, 16)) return TCQ_E_MISALIGNED;
    int num_sms = 0;
    if ((rc = current_num_sms(&num_sms)) != TCQ_OK) return rc;
    Workspace wk;
    if ((rc = carve(ws, ws_bytes, n_tiles, K, num_sms, &wk, false)) != TCQ_OK) return rc;
    if (bp_ws_bytes(n_tiles, K) > ws_bytes) return TCQ_E_WORKSPACE;
    if (!cluster_available()) return TCQ_E_BAD_ARGUMENT;   // the single-CTA kernel has no bounded waits to test
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(wk.status, 0, sizeof(unsigned int), s) != cudaSuccess) return cuda_fail(cudaGetLastError(), "status reset");
    // the buffers of the final metrics are told to expect 16 bytes more than the cluster will ever send
    ForwardArgs f{w, nullptr, 0, n_tiles, nullptr, 0, 0, kT, nullptr, nullptr, nullptr, 1.0f, 16, wk.status, 0};
    ClusterArgs ca{f, nullptr, 0, nullptr, clusters_at_once(2)};
    cudaError_t err = K == 2   ? launch_forward_cluster<2>(kCbMcg, ca, 2, 2, s)
                      : K == 3 ? launch_forward_cluster<3>(kCbMcg, ca, 2, 2, s)
                               : launch_forward_cluster<4>(kCbMcg, ca, 2, 2, s);
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "forward (self-test)");
}

int tcq_selftest_walk_waits(const float* w, int64_t n_tiles, int K, uint32_t* packed, void* ws, size_t ws_bytes, void* stream) {
    const int rc = check_common(K, kCbMcg, n_tiles);
    if (rc != TCQ_OK) return rc;
    if (n_tiles < 1 || n_tiles > 2000) return TCQ_E_BAD_COUNT;
    if (w == nullptr || packed == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(w, 16) || misaligned(packed, 4)) return TCQ_E_MISALIGNED;
    EncodeIO io{};
    io.w = w;
    io.n = n_tiles;
    io.packed = packed;
    io.packed_stride = kT * K / 32;
    io.hurry = true;
    return encode_core(io, K, kCbMcg, ws, ws_bytes, static_cast<cudaStream_t>(stream));
}

int64_t tcq_encode_launches(int64_t n_tiles, int K, size_t ws_bytes) {
    if (K < 2 || K > 4) return TCQ_E_BAD_K;
    if (n_tiles < 0) return TCQ_E_BAD_COUNT;
    if (n_tiles == 0) return 0;
    int num_sms = 0;
    int rc = current_num_sms(&num_sms);
    if (rc != TCQ_OK) return rc;
    Workspace wk;
    alignas(256) static unsigned char dummy[256];          // carve() only does pointer arithmetic on it
    if ((rc = carve(dummy, ws_bytes, n_tiles, K, num_sms, &wk, true)) != TCQ_OK) return rc;
    auto of_span = [&](int64_t n) {
        const int64_t whole = n / wk.chunk, rest = n % wk.chunk;
        return whole * launches_of_chunk(wk.chunk, K, wk) + (rest > 0 ? launches_of_chunk(rest, K, wk) : 0) + (wk.fused ? 2 : 0);
    };
    if (!wk.fused) return of_span(n_tiles);
    return n_tiles / wk.span * of_span(wk.span) + (n_tiles % wk.span > 0 ? of_span(n_tiles % wk.span) : 0);
}

int tcq_decode_packed(const uint32_t* packed, int64_t n_tiles, int K, int codebook, float* dq, void* stream) {
    int rc = check_common(K, codebook, n_tiles);
    if (rc != TCQ_OK) return rc;
    if (n_tiles == 0) return TCQ_OK;
    if (packed == nullptr || dq == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(packed, 4) || misaligned(dq, 16)) return TCQ_E_MISALIGNED;
    cudaError_t err = launch_decode_packed(packed, n_tiles, K, codebook, dq, static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "decode_packed");
}

int tcq_decode_matvec(const uint32_t* packed, int64_t n_out, int64_t k_in, int K, int codebook, const float* x, int64_t ldx,
                      int m, float* y, int64_t ldy, void* stream) {
    int rc = check_common(K, codebook, n_out);
    if (rc != TCQ_OK) return rc;
    if (k_in < 0 || m < 0) return TCQ_E_BAD_COUNT;
    if (n_out % 16 || k_in % 16 || n_out / 16 > 0x7FFFFFFF || k_in / 16 > 0x7FFFFFFF) return TCQ_E_BAD_ARGUMENT;
    if (n_out == 0 || k_in == 0 || m == 0) return TCQ_OK;
    if (ldx < k_in || ldx % 4 || ldy < n_out) return TCQ_E_BAD_ARGUMENT;
    if (packed == nullptr || x == nullptr || y == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(packed, 4) || misaligned(x, 16) || misaligned(y, 4)) return TCQ_E_MISALIGNED;
    cudaError_t err = launch_decode_matvec(packed, n_out, k_in, K, codebook, x, ldx, m, y, ldy,
                                           static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "decode_matvec");
}

int tcq_decode_symbols(const int64_t* bits, int64_t n, int64_t T, int K, int codebook, const int64_t* s0, float* out,
                       void* stream) {
    int rc = check_common(K, codebook, n);
    if (rc != TCQ_OK) return rc;
    if (T < 0) return TCQ_E_BAD_COUNT;
    if (n == 0 || T == 0) return TCQ_OK;
    if (bits == nullptr || out == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(bits, 8) || misaligned(out, 4) || (s0 && misaligned(s0, 8))) return TCQ_E_MISALIGNED;
    cudaError_t err = launch_decode_symbols(reinterpret_cast<const long long*>(bits), n, T, K, codebook,
                                            reinterpret_cast<const long long*>(s0), out,
                                            static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "decode_symbols");
}

int tcq_pack_symbols(const int64_t* bits, int64_t n_tiles, int K, uint32_t* packed, void* stream) {
    if (K < 2 || K > 4) return TCQ_E_BAD_K;
    if (n_tiles < 0) return TCQ_E_BAD_COUNT;
    if (n_tiles == 0) return TCQ_OK;
    if (bits == nullptr || packed == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(bits, 8) || misaligned(packed, 4)) return TCQ_E_MISALIGNED;
    cudaError_t err = launch_pack_symbols(reinterpret_cast<const long long*>(bits), n_tiles, K, packed,
                                          static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "pack_symbols");
}

namespace {
int check_ip_shape(int64_t n, int64_t k) {
    if (n < 0 || k < 0) return TCQ_E_BAD_COUNT;
    if (n % 16 || k % 16 || n / 16 > 65535) return TCQ_E_BAD_ARGUMENT;
    return TCQ_OK;
}
}  // namespace

size_t tcq_ip_workspace_bytes(int64_t n, int64_t k) {
    if (check_ip_shape(n, k) != TCQ_OK || n == 0 || k == 0) return 0;
    return ip_workspace_bytes(n, k);
}

int tcq_ip_forward(const float* w, int64_t n, int64_t k, const float* sv, const float* su, float cb_rms, int tiled,
                   float* z, float* out_s, float* in_s, float* scale, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_ip_shape(n, k);
    if (rc != TCQ_OK) return rc;
    if (!(cb_rms > 0.0f)) return TCQ_E_BAD_ARGUMENT;
    if (n == 0 || k == 0) return TCQ_OK;
    if (!w || !sv || !su || !z || !out_s || !in_s || !scale || !ws) return TCQ_E_NULL_POINTER;
    if (misaligned(w, 4) || misaligned(z, 16) || misaligned(sv, 4) || misaligned(su, 4) || misaligned(out_s, 4) ||
        misaligned(in_s, 16) || misaligned(scale, 4) || misaligned(ws, 256))
        return TCQ_E_MISALIGNED;
    if (ws_bytes < ip_workspace_bytes(n, k)) return TCQ_E_WORKSPACE;
    cudaError_t err = launch_ip_forward(w, n, k, sv, su, cb_rms, tiled != 0, z, out_s, in_s, scale, ws,
                                        static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "ip_forward");
}

int tcq_ip_restore(const float* zq, int tiled, int64_t n, int64_t k, const float* sv, const float* su, const float* out_s,
                   const float* in_s, const float* scale, float* w_hat, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_ip_shape(n, k);
    if (rc != TCQ_OK) return rc;
    if (n == 0 || k == 0) return TCQ_OK;
    if (!zq || !sv || !su || !out_s || !in_s || !scale || !w_hat || !ws) return TCQ_E_NULL_POINTER;
    if (misaligned(zq, 16) || misaligned(w_hat, 4) || misaligned(sv, 4) || misaligned(su, 4) || misaligned(out_s, 4) ||
        misaligned(in_s, 16) || misaligned(scale, 4) || misaligned(ws, 256))
        return TCQ_E_MISALIGNED;
    if (ws_bytes < ip_workspace_bytes(n, k)) return TCQ_E_WORKSPACE;
    cudaError_t err = launch_ip_restore(zq, tiled != 0, n, k, sv, su, out_s, in_s, scale, w_hat, ws,
                                        static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "ip_restore");
}

int tcq_codebook_lut(int codebook, float* lut, void* stream) {
    if (codebook < 0 || codebook > 2) return TCQ_E_BAD_CODEBOOK;
    if (lut == nullptr) return TCQ_E_NULL_POINTER;
    if (misaligned(lut, 4)) return TCQ_E_MISALIGNED;
    cudaError_t err = launch_codebook_lut(codebook, lut, static_cast<cudaStream_t>(stream));
    return err == cudaSuccess ? TCQ_OK : cuda_fail(err, "codebook_lut");
}

}  // extern "C"
