// bin_common.cuh -- pieces shared by the binning kernels (bin.cu, bin_segment.cu).
#pragma once

#include "ljcell_internal.cuh"

namespace ljc {

// ---------------------------------------------------------------- within-cell sort
// Keys: LJ_ORDER_INDEX sorts by original index; LJ_ORDER_X by x, then index.
// Indices are unique, so keys are unique and the result is a pure function of
// the input.
template <int ORDER>
__device__ __forceinline__ bool key_less(float xa, int ia, float xb, int ib) {
    if (ORDER == LJ_ORDER_X) return (xa < xb) || (xa == xb && ia < ib);
    return ia < ib;
}

constexpr int kRankMax = 512;  // cells up to this size are ranked record by record, larger ones are sorted

struct SortOut {
    float4* out4;
    int* out_cell;
    float* sx;
    float* sy;
    float* sz;
    int* sidx;
};

// Segment path of the cell-grid build (bin_segment.cu).
struct SegPlan {
    int shift;  // cells per segment = 1 << shift
    int nseg;   // 0: the path does not take this grid
};
SegPlan segment_plan(const lj_ctx* ctx, int n, long long nc);
bool segment_scratch(lj_ctx* ctx, const SegPlan& plan);
// Enqueues the build in the plan's scratch; *gate (device) is nonzero afterwards when a segment was too large for it and the
// ticket kernels have to run instead.
lj_status launch_segment_bin(lj_ctx* ctx, const SegPlan& plan, long long nc, int n, const float* x, const float* y,
                             const float* z, int stride, lj_order order, int* counts, int* offsets,
                             lj_cell_desc* cells, const SortOut& so, const GridDev& g, const unsigned** gate);

// Sets what the build's kernels need on the current device; lj_create calls it.
lj_status bin_shared_limits();
bool large_sort_shared_limit();  // bin.cu's part of it

// A small system binned by one block in one launch.
bool small_bin_takes(const lj_ctx* ctx, int n, long long nc);
lj_status launch_small_bin(lj_ctx* ctx, long long nc, int n, const float* x, const float* y, const float* z, int stride,
                           lj_order order, int* counts, int* offsets, lj_cell_desc* cells, const SortOut& so,
                           const GridDev& g);

}  // namespace ljc
