// The index steps of the read-ahead walks (csrc/hsmu_steps.cuh) over ranges that end at or near INT_MAX:
// every position is visited once, and (built with -fsanitize=signed-integer-overflow) nothing overflows.
#include <climits>
#include <cstdio>
#include <vector>

#include "hsmu_steps.cuh"

using namespace hsmu;

static int fails = 0;

// one walk: `lanes` lanes, `ahead` strides of `lanes` per round; the first lane starts at `first`
static void walk(int first, int end, int lanes, int ahead) {
    const int n = end - first;
    std::vector<int> seen((size_t)n, 0);
    for (StepPos base = first; step_in(base, 0, end); base += lanes * ahead)
        for (int u = 0; u < ahead; u++)
            for (int lane = 0; lane < lanes; lane++)
                if (step_in(base, u * lanes + lane, end)) seen[base + u * lanes + lane - first]++;
    for (int x : seen) fails += x != 1;
}

// the lane-by-lane form
static void walk_rel(int len, int lanes, int ahead) {
    long long visits = 0;
    for (int lane = 0; lane < lanes; lane++)
        for (StepPos p = lane; step_in(p, 0, len); p += lanes * ahead)
            for (int u = 0; u < ahead; u++) visits += step_in(p, u * lanes, len);
    fails += visits != len;
}

int main() {
    const int ends[] = {INT_MAX, INT_MAX - 1, INT_MAX - 31, INT_MAX - 127, INT_MAX - 255, INT_MAX - 1023, 100000, 4096};
    for (int end : ends)
        for (int n : {0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1000, 2048})
            for (int ahead : {1, 4, 8}) walk(end - n, end, 32, ahead);
    for (int len : {0, 1, 3, 4, 5, 15, 16, 17, 255, 256, 257, 1023, 1024, 1025, 70001})
        for (int lanes : {4, 8, 16, 32, 256}) walk_rel(len, lanes, 4);
    walk_rel(INT_MAX, 256, 4);  // the longest row
    if (fails) return std::printf("FAIL %d\n", fails), 1;
    std::printf("ok\n");
    return 0;
}
