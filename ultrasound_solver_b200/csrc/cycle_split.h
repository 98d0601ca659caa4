// How the CTAs of a cycle launch (cycle.cu) are shared out over the right-hand
// sides, and which kernel instance holds every division a launch can see.
// Plain C++: the kernel, its launcher and a host test use the same functions.
#pragma once

#ifdef __CUDACC__
#define USV_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define USV_HOST_DEVICE inline
#endif

namespace usv {

constexpr int kCycThreads = 512;
constexpr int kCycMaxCtas = 512;  // size of the partial-sum rows in the workspace

// Every active right-hand side gets one CTA, the other ctas - active go by size.
// First CTA of the one that follows `seen` active right-hand sides of `before`
// units, of `total` (nodes; 1 for each right-hand side of a single scene).
USV_HOST_DEVICE unsigned cycle_first_cta(unsigned ctas, unsigned active, unsigned seen, unsigned before,
                                         unsigned total) {
    return seen + unsigned((unsigned long long)(ctas - active) * before / total);
}

// Nodes of one of `share` CTAs for n nodes: whole 64-node groups (a vector's padding).
USV_HOST_DEVICE int cycle_cta_nodes(int n, int share) { return ((n + 63) / 64 + share - 1) / share * 64; }

// The dots of a step are (vector group, segment of the CTA's nodes) tasks, a warp
// each. A segment holds at most 4096 nodes: 128 per lane, the longest fp32 sum
// of a bfloat16 basis.
constexpr int kCycTasks = 64;  // tasks that further segments may fill
USV_HOST_DEVICE constexpr int cycle_least_segments(int nodes) { return (nodes + 4095) / 4096; }

// Segments that balance the tasks of `groups` vector groups over the warps:
// fewest vector slices per warp, then fewest segments.
USV_HOST_DEVICE int cycle_segments(int groups, int nodes) {
    constexpr int warps = kCycThreads / 32;
    int best = cycle_least_segments(nodes), rounds = (groups * best + warps - 1) / warps;  // rounds / best: slices per warp
#pragma unroll 1
    for (int sg = best + 1; groups * sg <= kCycTasks; ++sg) {
        const int r = (groups * sg + warps - 1) / warps;
        if (r * best < rounds * sg) best = sg, rounds = r;
    }
    return best;
}

// Tasks whose sums need room in an instance of `capacity` nodes with at most
// `groups` vector groups: the least segments of a long basis exceed kCycTasks.
USV_HOST_DEVICE constexpr int cycle_task_room(int groups, int capacity) {
    return groups * cycle_least_segments(capacity) > kCycTasks ? groups * cycle_least_segments(capacity) : kCycTasks;
}

// Instances by bytes per stored value: nodes a CTA of instance i has room for.
// (scenes: right-hand sides of several scenes in one launch)
constexpr int cycle_instances(int bytes, bool scenes) { return bytes == 16 ? 2 : scenes ? 4 : 3; }
constexpr int cycle_units(int bytes, int i) { return (bytes == 16 ? 2 : 1) << i; }  // 16-byte loads per thread
constexpr int cycle_capacity(int bytes, int i) { return kCycThreads * (16 / bytes) * cycle_units(bytes, i); }

// Most nodes per CTA for which the cycle kernel is taken. Alone, per Arnoldi
// step of GMRES(30), cycle kernel / one launch per pass (us; nodes over all
// right-hand sides):
//   bfloat16   22.7 / 36.0 at 593 k, 34.0 / 46.5 at 1.00 M, 61.9 / 63.8 at 1.40 M, 71.8 / 73.1 at 1.73 M,
//              72.7 / 72.5 at 1.82 M, 78.6 / 76.4 at 1.91 M, 84.3 / 78.7 at 2.10 M
//   complex64  32.6 / 46.0 at 512 k, 60.4 / 65.1 at 729 k, 77.4 / 78.3 at 1.00 M, 72.8 / 72.8 at 1.05 M (4 x 64^3),
//              84.3 / 80.0 at 1.12 M, 81.9 / 76.6 at 1.19 M
//   complex128 29.2 / 47.1 at 262 k, 32.3 / 49.3 at 287 k, 59.2 / 55.9 at 314 k, 61.7 / 58.6 at 365 k (4 x 45^3)
// The basis is then far larger than L2 and both read it from DRAM. But the
// kernel's launches hold the shared memory of their SMs, so those of solves on
// other streams wait, while per-pass kernels overlap. Solves at once, each on
// its own stream, ms (2 / 8 solves):
//   bfloat16   104^3 22.4 / 88 against 23.1 / 93, 112^3 34.6 / 141 against 28.7 / 123 (GMRES(30)),
//              104^3 40.2 / 161 against 40.4 / 163, 112^3 62.6 / 253 against 49.6 / 198 (GCRO-DR(36,8))
//   complex64  84^3 22.8 / 90 against 23.0 / 97, 88^3 32.6 / 129 against 27.3 / 119
//   complex128 66^3 19.5 / 77 against 23.8 / 86, 68^3 34.0 / 137 against 27.0 / 108
// So one scene goes as far as it wins both ways: 8192, 4096 and 2048 nodes. A
// batch of scenes is itself the overlap; two batches at once (100 iterations)
// took 25.4 ms against 25.1 (bfloat16, 1.59 M nodes), 17.4 against 20.4
// (complex64, 948 k), and 13.3 against 11.9 (complex128, 337 k), so the first
// two go on to where the kernels meet alone.
constexpr int cycle_line(int bytes, bool scenes) {
    return bytes == 4 ? (scenes ? 12288 : 8192) : bytes == 8 ? (scenes ? 7104 : 4096) : 2048;
}

struct CycleShape {
    int ctas = 0;       // 0: one launch per Arnoldi pass
    int instance = -1;
};

// Shape for right-hand sides of sizes[b] nodes on `sms` SMs: the smallest
// instance that has room in every launch of the solve. Right-hand sides leave
// as they finish. One that is still active then has at least the share
// 1 + floor(spare n / total) formed here with all of them: `spare` only grows,
// the active total only shrinks, and its real share is a difference of two
// floors, at least the floor of the difference. (Its share in a particular
// launch is no bound: a right-hand side rounded up there can be rounded down
// once another has left. bfloat16 scenes of 12^3, 42^3, 64^3, 64^3 on 148 SMs:
// 4096 nodes for the 42^3 one with all active, 4160 without the smallest.)
inline CycleShape cycle_shape(int bytes, bool scenes, const long long* sizes, int nrhs, int sms) {
    const int line = cycle_line(bytes, scenes);
    CycleShape shape;
    int ctas = sms < kCycMaxCtas ? sms : kCycMaxCtas;
    if (nrhs > ctas) return shape;
    long long total = 0, most = 0;
    for (int b = 0; b < nrhs; ++b) total += sizes[b];
    if (total > (long long)ctas * line) return shape;
    // at least 256 nodes per CTA: with fewer the meetings of the extra CTAs cost
    // more than their share of the work saves (24^3, 148 -> 54 CTAs: complex64
    // 12.6 -> 12.2 us per step, bfloat16 11.8 -> 11.4, complex128 14.2 -> 13.1)
    if (total / 256 < ctas) ctas = total / 256 > nrhs ? int(total / 256) : nrhs;
    for (int b = 0; b < nrhs; ++b) {
        const int per = cycle_cta_nodes(int(sizes[b]), 1 + int((long long)(ctas - nrhs) * sizes[b] / total));
        most = per > most ? per : most;
    }
    if (most > line) return shape;
    for (int i = 0; i < cycle_instances(bytes, scenes); ++i)
        if (most <= cycle_capacity(bytes, i)) {
            shape.ctas = ctas;
            shape.instance = i;
            break;
        }
    return shape;
}

}  // namespace usv
