// The walk's limit on candidates of fused sweeps, on the host: reads pairs of a float (the smallest candidate) and an int (its steps), writes the limits.
// Built and run by test_gpu_fused_sweep.py.
#include <cstdio>

#include "../trellis-everywhere_b200/csrc/tcq_walk.cuh"

int main() {
    struct { float best; int t; } in;
    while (std::fread(&in, sizeof in, 1, stdin) == 1) {
        const float limit = tcq::fused_limit(in.best, in.t);
        std::fwrite(&limit, sizeof limit, 1, stdout);
    }
    return 0;
}
