// Launch shapes of the dataflow kernels that run a batch with one CTA per
// instance (lu_kernels.cu, lu_complex.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace nsg {

// What the launches depend on: instances, the batch's largest LU column and
// order, the mean number of rows in a level of its triangular sweeps and of
// entries in a row of one, and whether any plan has wide levels (wide_levels).
struct FlowBatch {
    int count = 0, max_col = 0, max_n = 0;
    double level_rows = 0.0, row_entries = 0.0;
    bool wide = false;
};

// One CTA of 16 warps with the SM's registers to itself, two such CTAs, or four
// of 8 warps.  (The sweeps need no more than 64 registers a thread: one
// kernel serves the first two.)
enum FlowShape { kShapeAlone, kShapePair, kShapeMany };

inline int flow_sm_count() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    return sms;
}

// CTAs that an SM's 228 KB hold with smem bytes of dynamic shared memory each:
// a CTA also takes 1 KB for the system and its static part.
inline int ctas_per_sm(size_t smem) {
    return static_cast<int>((size_t{228} * 1024) / (smem + 2 * 1024));
}

// Passes of the SMs over the batch with per_sm CTAs of it on each.
inline int flow_waves(const FlowBatch& b, int per_sm) {
    return (b.count + per_sm * flow_sm_count() - 1) / (per_sm * flow_sm_count());
}

// Levels of fewer rows than this on average: a chain or a band, whose rows wait
// for one another one by one whatever the number of warps.
constexpr double kChainRows = 2.0;

// The shape of a launch: up to two instances per SM run on 16 warps each.  Beyond
// that, four CTAs of 8 warps keep as many warps busy and more instances under way
// -- if at least `need` of them, with many_smem bytes each, fit the SM; with fewer,
// and less left of L1, 16 warps an instance are faster, but for chains.
// Measured, two CTAs of 16 warps -> four of 8 or as many as fit, ms for 592
// instances (B200, 1965 MHz):
//   refactor of meshes: 1601 unknowns 1.44 -> 1.48 (297 instances 1.36 -> 1.20),
//     8101 (three fit) 15.4 -> 25.7 (297 instances 13.3
//     -> 13.6), 16,385 (two) 117 -> 201
//   solve: 1601 0.81 -> 0.63, 5777 (three) 3.06 -> 3.71 (297 instances 2.61 ->
//     2.11), 8101 (two) 4.55 -> 5.51, 16,385 (one) 11.8 -> 20.2
//   complex refactor: 37 0.047 -> 0.035, 1601 (eight) 1.92 -> 1.93, 3137 (five)
//     4.52 -> 4.79; complex solve: 1601 1.25 -> 1.01, 3137 (three) 2.39 -> 3.09
//   chains: a band of 9000 12.2 -> 6.9, solve 19.0 -> 16.3, complex 19.4 -> 10.7
//     and 36.4 -> 34.5; of 300, complex, 0.64 -> 0.33 and 0.62 -> 0.33
inline FlowShape flow_shape(const FlowBatch& b, size_t many_smem, int need) {
    if (b.count <= flow_sm_count()) return kShapeAlone;
    if (b.count <= 2 * flow_sm_count()) return kShapePair;
    return ctas_per_sm(many_smem) >= need || b.level_rows < kChainRows ? kShapeMany : kShapePair;
}

// CTAs per SM of the solves that run level after level in global memory (256
// threads; 48 registers a thread).
constexpr int kLevelBlocks = 5;

// Whether a transposed or complex solve runs level after level with the vector in
// a workspace, although the dataflow sweeps, of this shape and with smem bytes a
// CTA, could keep it in shared memory.  One instance takes R times as long
// that way, but every SM holds five of them, where shared memory may hold one or
// two.  R grows with the entries of a row: 1.2 to 1.7 measured for chains and trees
// (one entry), 2 to 2.5 for a band (6), 4 for a mesh of 577 unknowns (9), 7 of 3137
// (15), 11 of 16,385 (24).  592 instances, sweeps and levels: chains of 10,000
// transposed 31.2 and 12.2 ms, complex 32.2 and 14.4; of 3000 complex 5.1 and 3.9;
// trees of short branches, 10,000 unknowns, 4.6 and 2.5, complex 5.8 and 3.2; meshes
// of 7057 4.0 and 12.2.  Plans with wide levels keep theirs in shared memory.
inline bool levels_pay(const FlowBatch& b, FlowShape shape, size_t smem) {
    if (b.wide) return false;
    const int fit = ctas_per_sm(smem), most = shape == kShapeMany ? 4 : 2;
    const int sweeps = flow_waves(b, fit < 1 ? 1 : fit < most ? fit : most);
    return sweeps > flow_waves(b, kLevelBlocks) * (1.3 + 0.4 * b.row_entries);
}

}  // namespace nsg
