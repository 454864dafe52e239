// pair_cluster.cu -- single-system kernel of the cluster walk (pair_cluster.cuh).
#include <algorithm>

#include "pair_cluster.cuh"

namespace ljc {

namespace {
constexpr int kCluWarps = 4;
}  // namespace

// Block i of the launch evaluates the groups of targets that start in [a0 + i * stretch, a0 + (i + 1) * stretch),
// its warps in turn; SPLIT: two warps to a group, one for each cluster.
template <bool XWIN, bool SPLIT>
__global__ void __launch_bounds__(32 * kCluWarps, kCluWarpsPerSm / kCluWarps)
    k_pair_cluster(GridDev g, PairParams pp, const float4* p, const int* cs,
                   const int* off, int n, int kb, int ke, int a0, int stretch,
                   float* __restrict__ energy, float* __restrict__ force, Partial* part, unsigned* counter,
                   lj_totals* totals, unsigned* status) {
    __shared__ __align__(16) CluSmem sm[kCluWarps];
    chain_wait();
    if (pp.gate && *pp.gate != pp.want) return;
    const int w = (int)(threadIdx.x >> 5);
    const long long first = a0 + (long long)blockIdx.x * stretch;
    double te = 0.0, tw = 0.0;
    unsigned long long tp = 0;
    if (first < ke) {
        const int a = (int)first, b = (int)min(first + stretch, (long long)ke);
        cluster_stretch<XWIN>(g, pp, p, cs, 0, off, 0, n, a, b, kb, ke, SPLIT ? w / 2 : w, SPLIT ? kCluWarps / 2 : kCluWarps,
                              SPLIT ? w & 1 : -1, sm[w], status,
                              [&](int k, int s, bool valid, float v, float wv, unsigned np, int id) {
                                  if (!valid || k < kb || k >= ke) return;
                                  tw += (double)wv;
                                  tp += np;
                                  if (s == 0) te += (double)v;
                                  int o = k;
                                  if (pp.by_index) {
                                      o = id;
                                      if (o < 0 || o >= n) {
                                          atomicOr(status, kFlagRange);
                                          return;
                                      }
                                  }
                                  if (s == 0) {
                                      if (energy) energy[o] = pp.e4 * v;
                                  } else if (force) {
                                      force[3 * (size_t)o + (s - 1)] = -pp.fscale * v;
                                  }
                              });
    }
    __syncthreads();
    chain_next();  // every walk of the grid has ended when this counts: what follows may share the totals' time
    reduce_totals<32 * kCluWarps>(0.5 * (double)pp.e4 * te, 0.5 * (double)pp.e24 * tw, tp, part, counter, totals);
}

lj_status launch_pair_cluster(lj_ctx* ctx, const lj_grid* g, const PairParams& pp, int n, const float* xyzi,
                              const int* cs, const int* off, bool xwin, float* energy, float* force,
                              lj_totals* totals, int kb, int ke) {
    const int a0 = std::max(kb - (kCluGroup - 1), 0);  // a group that holds kb starts here at the earliest
    const long long nk = ke - a0;
    // a group's clusters to two warps while all of them run at once (1,000 particles at 12 per cell 18.4
    // against 24.5 us, 30,000 25.4 against 30.7, but 60,000 38.9 against 36.9: each of the two warps finds
    // the group's ranges); then more groups per warp with the size of the launch
    const long long wave = (long long)ctx->sm_count * kCluWarpsPerSm * kCluGroup;
    const bool split = 2 * nk <= wave;
    const int stretch = split ? kCluWarps / 2 * kCluGroup
                              : kCluWarps * kCluGroup * clu_groups_per_warp((double)nk / (double)wave);
    const int blocks = (int)((nk + stretch - 1) / stretch);
    const size_t need = 256 + clu_most_blocks(nk, (double)nk / (double)wave, (double)wave / (kCluWarps * kCluGroup)) * sizeof(Partial);
    if (need > ctx->red_bytes) {
        lj_status s = grow(&ctx->red, &ctx->red_bytes, need);
        if (s != LJ_OK) return s;
        if (cudaMemsetAsync(ctx->red, 0, 256, ctx->stream) != cudaSuccess) return LJ_ECUDA;
    }
    unsigned* counter = static_cast<unsigned*>(ctx->red);
    Partial* part = reinterpret_cast<Partial*>(static_cast<char*>(ctx->red) + 256);
    const float4* p4 = reinterpret_cast<const float4*>(xyzi);
    const auto kernel = xwin ? (split ? k_pair_cluster<true, true> : k_pair_cluster<true, false>)
                             : (split ? k_pair_cluster<false, true> : k_pair_cluster<false, false>);
    chain_launch(kernel, blocks, 32 * kCluWarps, 0, ctx->stream, to_dev(*g), pp, p4, cs, off, n, kb, ke, a0, stretch,
                 energy, force, part, counter, totals, ctx->d_status);
    return last_launch_status();
}

}  // namespace ljc
