// bin_segment.cu -- the cell-grid build by segments of cells, for large systems.
//
// Same results as the ticket path (bin.cu), with the particles partitioned first by segments of
// consecutive cells, a thousand or so particles each, and every segment then binned by one block in
// shared memory:
//
//   k_seg_count    per-block histogram of segments; each block reserves its share of every segment, the
//                  last one to finish writes the segments' starts and the list of those too large for
//                  the small sort kernel
//   k_seg_scatter  records to their segment, each block to the slots it reserved
//   k_seg_sort     per segment: cell counts, their prefix, the records grouped by cell and ranked by
//                  key, all in shared memory; counts, offsets and every sorted output leave in order
//
// The ticket path does one global atomic, a gather of its cell's offset and a 16-byte write to a random
// place per particle (in passes over cell ranges that fit L2, each reading all tickets again), and ranks
// each record against its cell through L1.  Here the atomics and the gathers stay in shared memory and
// the dense counts and offsets are written once, without being zeroed or read.  Measured on B200, whole
// build, ticket path -> segments: 10M at 10 per cell 548 -> 456 us, at 80 per cell 787 -> 556, sorted already
// 337 -> 273; 4M on a sphere shell of 64M cells 423 -> 330; 4.2M at 16 per cell 228 -> 198; behind the open
// gate (10M, 100,000 of them in one cell) 3791 -> 3913; but 3M at 14 per cell 172 -> 193 and 1M at 10 per cell
// 71 -> 85, hence kSegMinParticles.  At 10M: count 62 us, scatter 3 x 73 (bound by
// 16-byte writes to random sectors, about 65 per ns; the time does not depend on the instructions,
// the loads in flight or the occupancy), sort 132 (instructions and shared-memory wavefronts, 70% of
// the issue slots).
#include <algorithm>

#include "bin_common.cuh"

namespace ljc {

namespace {
constexpr int kSegMax = 16384;          // segments: a block's histogram is at most 64 KiB of shared memory
constexpr int kSegCells = 8192;         // cells of a segment: its counters take at most 32 KiB
constexpr int kSegAim = 768;            // particles per segment to aim for (up to twice that by the power of two)
constexpr int kSegThreads = 1024;       // count and scatter
constexpr int kSegSmall = 2048;         // records of a segment in the small sort kernel ...
constexpr int kSegLarge = 10240;        // ... and in the large one; a segment above opens the gate
constexpr int kSmallParticles = 4096;  // a system that one block bins (of at most kSegCells cells)
constexpr int kSegMinParticles = 4000000;
constexpr long long kSegRegion = 56LL << 20;  // bytes of records one scatter pass writes (L2 holds 126 MB)

struct SegScratch {
    unsigned* gate;    // [0] gate, [1] number of large segments, [2] blocks that have counted, [3] warp rounds of
                       // particles of several segments, [4] set when those are few: scatter in one pass
    int* total;        // [nseg] particles per segment while counting, then unused
    int* start;        // [nseg + 1]
    int* large;        // [nseg] segments above kSegSmall
    unsigned short* id;  // [n] each particle's segment
    int* base;         // [blocks * nseg] a block's first slot in each segment, from the segment's start
};
}  // namespace

__device__ __forceinline__ int seg_clamped(int cell, int shift, int nseg) { return min(cell >> shift, nseg - 1); }

// Adds one to h[s] for every valid lane and returns the old value a lane would have seen one after the
// other; a warp whose lanes all go to one segment (particles nearly sorted already) adds once, any other
// is counted in mixed.
__device__ __forceinline__ int seg_take(int* h, int s, bool valid, unsigned& mixed) {
    const unsigned m = __ballot_sync(0xffffffffu, valid);
    if (!m) return 0;
    const int leader = __ffs(m) - 1;
    const int s0 = __shfl_sync(0xffffffffu, s, leader);
    const bool one = __all_sync(0xffffffffu, !valid || s == s0);
    mixed += one ? 0u : 1u;
    if (one) {
        int v = 0;
        if ((int)lane_id() == leader) v = atomicAdd(&h[s0], __popc(m));
        return __shfl_sync(0xffffffffu, v, leader) + __popc(m & lanemask_lt());
    }
    return valid ? atomicAdd(&h[s], 1) : 0;
}

// One block: exclusive prefix of the segments' totals, the large segments, the gate.
__device__ __forceinline__ void seg_scan(int nseg, int n, const SegScratch& sc) {
    __shared__ int s_warp[kSegThreads / 32];
    __shared__ int s_large;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = kSegMax / kSegThreads;
    const int first = tid * PER;
    if (tid == 0) s_large = 0;
    int sum = 0;
#pragma unroll
    for (int k = 0; k < PER; k += 4) {  // total has room for a multiple of 64 entries, zeroed
        if (first + k >= nseg) break;
        const int4 q = __ldcg(reinterpret_cast<const int4*>(sc.total + first + k));
        sum += q.x + q.y + q.z + q.w;
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    int run = (warp ? s_warp[warp - 1] : 0) + inc - sum;
    for (int k = 0; k < PER && first + k < nseg; ++k) {
        const int v = __ldcg(sc.total + first + k);
        sc.start[first + k] = run;
        if (v > kSegSmall) sc.large[atomicAdd(&s_large, 1)] = first + k;
        if (v > kSegLarge) sc.gate[0] = 1u;
        run += v;
    }
    __syncthreads();
    if (tid == 0) {
        sc.start[nseg] = n;
        sc.gate[1] = (unsigned)s_large;
        sc.gate[4] = __ldcg(&sc.gate[3]) <= (unsigned)n / 128u ? 1u : 0u;  // a quarter of the warps' rounds
    }
}

// Block b counts particles [n b / blocks, n (b + 1) / blocks); the last block to finish scans the totals.
__global__ void __launch_bounds__(kSegThreads) k_seg_count(GridDev g, const float* __restrict__ x,
                                                           const float* __restrict__ y, const float* __restrict__ z,
                                                           int stride, int n, int shift, int nseg, SegScratch sc,
                                                           unsigned* status) {
    extern __shared__ int s_hist[];
    chain_next();
    for (int i = threadIdx.x; i < nseg; i += kSegThreads) s_hist[i] = 0;
    __syncthreads();
    const long long lo = (long long)n * blockIdx.x / gridDim.x, hi = (long long)n * (blockIdx.x + 1) / gridDim.x;
    constexpr int U = 4;  // particles per thread and round: all loads in flight before the first use
    bool bad = false;
    unsigned mixed = 0;
    for (long long i0 = lo; i0 < hi; i0 += U * kSegThreads) {
        float px[U], py[U], pz[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * kSegThreads + threadIdx.x;
            px[u] = i < hi ? __ldg(&x[i * stride]) : 0.f;
            py[u] = i < hi ? __ldg(&y[i * stride]) : 0.f;
            pz[u] = i < hi ? __ldg(&z[i * stride]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * kSegThreads + threadIdx.x;
            const bool valid = i < hi;
            bad |= !(isfinite(px[u]) && isfinite(py[u]) && isfinite(pz[u]));
            const int seg = seg_clamped(cell_of(g, px[u], py[u], pz[u]), shift, nseg);
            if (valid) sc.id[i] = (unsigned short)seg;
            seg_take(s_hist, seg, valid, mixed);
        }
    }
    if (bad) atomicOr(status, kFlagNonFinite);
    if (mixed && lane_id() == 0) atomicAdd(&sc.gate[3], mixed);
    __syncthreads();
    int* base = sc.base + (size_t)blockIdx.x * nseg;
    for (int i = threadIdx.x; i < nseg; i += kSegThreads) {
        const int c = s_hist[i];
        if (c) base[i] = atomicAdd(&sc.total[i], c);
    }
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&sc.gate[2], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    seg_scan(nseg, n, sc);
}

// Block b moves the particles it counted to the slots it reserved, as (x, y, z, index bits): those of
// segments [seg_lo, seg_hi) only (see launch_segment_bin).
__global__ void __launch_bounds__(kSegThreads) k_seg_scatter(const float* __restrict__ x,
                                                             const float* __restrict__ y, const float* __restrict__ z,
                                                             int stride, int n, int nseg, SegScratch sc,
                                                             float4* __restrict__ tmp, unsigned* status, int seg_lo,
                                                             int seg_hi) {
    extern __shared__ int s_next[];
    chain_wait();
    chain_next();
    if (sc.gate[0]) return;
    if (sc.gate[4]) {  // nearly sorted particles: the writes of all segments are in order anyway
        if (seg_lo > 0) return;
        seg_hi = nseg;
    }
    const int* base = sc.base + (size_t)blockIdx.x * nseg;
    for (int i = seg_lo + threadIdx.x; i < seg_hi; i += kSegThreads) s_next[i - seg_lo] = sc.start[i] + base[i];
    __syncthreads();
    const long long lo = (long long)n * blockIdx.x / gridDim.x, hi = (long long)n * (blockIdx.x + 1) / gridDim.x;
    constexpr int U = 4;
    unsigned mixed = 0;
    for (long long i0 = lo; i0 < hi; i0 += U * kSegThreads) {
        int seg[U];
        float px[U], py[U], pz[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * kSegThreads + threadIdx.x;
            seg[u] = i < hi ? (int)sc.id[i] - seg_lo : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * kSegThreads + threadIdx.x;
            px[u] = i < hi ? __ldg(&x[i * stride]) : 0.f;
            py[u] = i < hi ? __ldg(&y[i * stride]) : 0.f;
            pz[u] = i < hi ? __ldg(&z[i * stride]) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * kSegThreads + threadIdx.x;
            const bool mine = seg[u] >= 0 && seg[u] < seg_hi - seg_lo;
            const int slot = seg_take(s_next, seg[u], mine, mixed);
            if (!mine) continue;
            if (slot >= 0 && slot < n)
                tmp[slot] = make_float4(px[u], py[u], pz[u], __int_as_float((int)i));
            else
                atomicOr(status, kFlagRange);
        }
    }
}

// A record in shared memory: (y, z, twice the original index plus one where x is -0, x as an unsigned integer
// of the same order, -0 as +0), so that its last two words are the sort key of LJ_ORDER_X as one 64-bit
// integer and hold every bit of x and of the index.
__device__ __forceinline__ uint4 pack_record(const float4& r) {
    const unsigned bits = __float_as_uint(r.x), u = r.x == 0.0f ? 0u : bits;
    return make_uint4(__float_as_uint(r.y), __float_as_uint(r.z),
                      2u * __float_as_uint(r.w) + (bits == 0x80000000u ? 1u : 0u),
                      u ^ ((unsigned)((int)u >> 31) | 0x80000000u));
}
__device__ __forceinline__ float4 unpack_record(const uint4& k) {
    const unsigned u = (k.w ^ ((unsigned)((int)~k.w >> 31) | 0x80000000u)) | (k.z << 31);  // k.z odd: u is 0
    return make_float4(__uint_as_float(u), __uint_as_float(k.x), __uint_as_float(k.y), __uint_as_float(k.z >> 1));
}

// Sorts the m records of one crowded cell by key, the whole block: a bitonic network over any number of records.
// Each run of k starts with the mirrored comparison, so every comparison is ascending and the places past the
// end, which count as greater, are never exchanged with.
template <int ORDER, int THREADS>
__device__ __noinline__ void cell_sort(uint4* rec, int m) {
    const auto exchange = [&](int lo, int hi) {
        if (hi >= m) return;
        const uint4 a = rec[lo], b = rec[hi];
        const bool less = ORDER == LJ_ORDER_X ? (b.w < a.w || (b.w == a.w && b.z < a.z)) : b.z < a.z;
        if (less) {
            rec[lo] = b;
            rec[hi] = a;
        }
    };
    for (int lk = 1; (1 << (lk - 1)) < m; ++lk) {
        const int pairs = ((m + (1 << lk) - 1) >> lk) << (lk - 1);
        for (int q = threadIdx.x; q < pairs; q += THREADS) {
            const int run = (q >> (lk - 1)) << lk, at = q & ((1 << (lk - 1)) - 1);
            exchange(run + at, run + (1 << lk) - 1 - at);
        }
        __syncthreads();
        for (int lj = lk - 2; lj >= 0; --lj) {
            for (int q = threadIdx.x; q < pairs; q += THREADS) {
                const int lo = ((q >> lj) << (lj + 1)) + (q & ((1 << lj) - 1));
                exchange(lo, lo + (1 << lj));
            }
            __syncthreads();
        }
    }
}

// One segment: its m records (at most CAP), load(i) the i-th, sorted to s0 on; its W cells from c0 on.
// The records are read twice (the second time from L2) rather than held in registers, which would halve
// the blocks per SM.
template <int ORDER, int THREADS, int CAP, class Load>
__device__ __forceinline__ void seg_sort(const GridDev& g, int c0, int W, int s0, int m, Load load,
                                         int* __restrict__ counts, int* __restrict__ offsets, bool vec,
                                         lj_cell_desc* __restrict__ cells, const SortOut& so, uint4* s_rec,
                                         int* s_cnt, unsigned short* s_cell) {
    constexpr int PER = (CAP + THREADS - 1) / THREADS;
    __shared__ int s_sum[THREADS / 32];
    __shared__ int s_crowded, s_list[CAP / (kRankMax + 1)];  // cells of more than kRankMax records
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    vec = vec && (W & 3) == 0;
    if (m == 0) {
        if (vec) {
            for (int c = 4 * tid; c < W; c += 4 * THREADS) {
                *reinterpret_cast<int4*>(counts + c0 + c) = make_int4(0, 0, 0, 0);
                *reinterpret_cast<int4*>(offsets + c0 + c) = make_int4(s0, s0, s0, s0);
            }
        } else {
            for (int c = tid; c < W; c += THREADS) {
                counts[c0 + c] = 0;
                offsets[c0 + c] = s0;
            }
        }
        if (cells)
            for (int c = tid; c < W; c += THREADS) cells[c0 + c] = lj_cell_desc{0, s0};
        return;
    }
    for (int c = 4 * tid; c < W; c += 4 * THREADS) *reinterpret_cast<int4*>(s_cnt + c) = make_int4(0, 0, 0, 0);
    if (tid == 0) s_crowded = 0;
    __syncthreads();
    int where[PER];  // cell << 16 | ticket
#pragma unroll
    for (int u = 0; u < PER; ++u)
        if (u * THREADS + tid < m) {
            const float4 r = load(u * THREADS + tid);
            const int c = min(max(cell_of(g, r.x, r.y, r.z) - c0, 0), W - 1);
            const int ticket = atomicAdd(&s_cnt[c], 1);
            if (ticket == kRankMax) s_list[atomicAdd(&s_crowded, 1)] = c;
            where[u] = (c << 16) | ticket;
        }
    __syncthreads();
    // exclusive prefix of the cell counts in place: each warp takes a run of cells, 128 at a time
    const int run = ((W + 4 * THREADS - 1) / (4 * THREADS)) * 128;
    const int a = min(warp * run, W), b = min(a + run, W);
    int sum = 0;
    for (int c = a + 4 * lane; c < b; c += 128) {
        const int4 v = *reinterpret_cast<const int4*>(s_cnt + c);
        sum += v.x + v.y + v.z + v.w;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    int carry = lane < warp ? s_sum[lane] : 0;
    carry = __reduce_add_sync(0xffffffffu, carry);
    for (int cb = a; cb < b; cb += 128) {
        const int c = cb + 4 * lane;
        const int4 v = c < b ? *reinterpret_cast<const int4*>(s_cnt + c) : make_int4(0, 0, 0, 0);
        const int t = v.x + v.y + v.z + v.w;
        int inc = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += q;
        }
        int4 ex;
        ex.x = carry + inc - t;
        ex.y = ex.x + v.x;
        ex.z = ex.y + v.y;
        ex.w = ex.z + v.z;
        if (c < b) {
            *reinterpret_cast<int4*>(s_cnt + c) = ex;
            if (vec) {
                *reinterpret_cast<int4*>(counts + c0 + c) = v;
                *reinterpret_cast<int4*>(offsets + c0 + c) = make_int4(s0 + ex.x, s0 + ex.y, s0 + ex.z, s0 + ex.w);
            } else {
                const int vv[4] = {v.x, v.y, v.z, v.w}, ee[4] = {ex.x, ex.y, ex.z, ex.w};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (c + k < W) {
                        counts[c0 + c + k] = vv[k];
                        offsets[c0 + c + k] = s0 + ee[k];
                    }
            }
            if (cells) {
                const int vv[4] = {v.x, v.y, v.z, v.w}, ee[4] = {ex.x, ex.y, ex.z, ex.w};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (c + k < W) cells[c0 + c + k] = lj_cell_desc{vv[k], s0 + ee[k]};
            }
        }
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PER; ++u)
        if (u * THREADS + tid < m) {
            const int c = where[u] >> 16, at = s_cnt[c] + (where[u] & 0xffff);
            const float4 r = load(u * THREADS + tid);
            s_rec[at] = pack_record(r);
            s_cell[at] = (unsigned short)c;
        }
    __syncthreads();
    for (int l = 0; l < s_crowded; ++l) {
        const int c = s_list[l], e0 = s_cnt[c];
        cell_sort<ORDER, THREADS>(s_rec + e0, (c + 1 < W ? s_cnt[c + 1] : m) - e0);
    }
    // a record's rank is the number of its cell's records with a smaller key, its place in a sorted cell
    for (int i = tid; i < m; i += THREADS) {
        const uint4 k = s_rec[i];
        const int c = s_cell[i];
        const int e0 = s_cnt[c], e1 = c + 1 < W ? s_cnt[c + 1] : m;
        int rank = 0;
        if (e1 - e0 > kRankMax) {
            rank = i - e0;
        } else if (ORDER == LJ_ORDER_X) {
            const unsigned long long key = ((unsigned long long)k.w << 32) | k.z;
            const unsigned long long* kj = reinterpret_cast<const unsigned long long*>(s_rec + e0) + 1;
#pragma unroll 4
            for (int j = e1 - e0; j > 0; --j, kj += 2) rank += *kj < key ? 1 : 0;
        } else {
#pragma unroll 4
            for (int j = e0; j < e1; ++j) rank += s_rec[j].z < k.z ? 1 : 0;
        }
        const float4 q = unpack_record(k);
        const int slot = s0 + e0 + rank;
        so.out4[slot] = q;
        so.out_cell[s0 + i] = c0 + c;  // every slot of a cell holds its id, whatever the order inside the cell
        if (so.sx) so.sx[slot] = q.x;
        if (so.sy) so.sy[slot] = q.y;
        if (so.sz) so.sz[slot] = q.z;
        if (so.sidx) so.sidx[slot] = __float_as_int(q.w);
    }
}

// SMALL: one block per segment of at most CAP records; else the blocks take the larger ones from the list.
template <int ORDER, int THREADS, int CAP, bool SMALL>
__global__ void __launch_bounds__(THREADS, SMALL ? 6 : 1) k_seg_sort(GridDev g, int ncell, int n, int shift, int nseg, SegScratch sc,
                                                      const float4* tmp, int* __restrict__ counts,
                                                      int* __restrict__ offsets, int vec, lj_cell_desc* __restrict__ cells,
                                                      SortOut so) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint4* s_rec = reinterpret_cast<uint4*>(s_raw);
    int* s_cnt = reinterpret_cast<int*>(s_raw + (size_t)CAP * 18);
    unsigned short* s_cell = reinterpret_cast<unsigned short*>(s_raw + (size_t)CAP * 16);
    chain_wait();
    chain_next();
    if (sc.gate[0]) return;
    if (SMALL && blockIdx.x == 0 && threadIdx.x == 0) offsets[ncell] = n;
    const int items = SMALL ? nseg : min((int)sc.gate[1], nseg);
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = SMALL ? it : sc.large[it];
        const int s0 = sc.start[b], m = sc.start[b + 1] - s0;
        if (m < 0 || m > CAP || s0 < 0 || s0 + m > n) continue;
        const int c0 = b << shift, W = min(1 << shift, ncell - c0);
        seg_sort<ORDER, THREADS, CAP>(
            g, c0, W, s0, m, [&](int i) { return __ldcg(&tmp[s0 + i]); }, counts, offsets, vec != 0, cells, so, s_rec,
            s_cnt, s_cell);
        if (!SMALL) __syncthreads();
    }
}

// A whole small system as one segment: one launch instead of the ticket path's six kernels and three
// memsets, which its smallest systems spend their time on.
template <int ORDER>
__global__ void __launch_bounds__(kSegThreads) k_bin_small(GridDev g, int ncell, const float* __restrict__ x,
                                                           const float* __restrict__ y, const float* __restrict__ z,
                                                           int stride, int n, int* __restrict__ counts,
                                                           int* __restrict__ offsets, int vec,
                                                           lj_cell_desc* __restrict__ cells, SortOut so,
                                                           unsigned* status) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint4* s_rec = reinterpret_cast<uint4*>(s_raw);
    unsigned short* s_cell = reinterpret_cast<unsigned short*>(s_raw + (size_t)kSmallParticles * 16);
    int* s_cnt = reinterpret_cast<int*>(s_raw + (size_t)kSmallParticles * 18);
    if (threadIdx.x == 0) offsets[ncell] = n;
    bool bad = false;
    seg_sort<ORDER, kSegThreads, kSmallParticles>(
        g, 0, ncell, 0, n,
        [&](int i) {
            const float4 r = make_float4(__ldg(&x[(long long)i * stride]), __ldg(&y[(long long)i * stride]),
                                         __ldg(&z[(long long)i * stride]), __int_as_float(i));
            bad |= !(isfinite(r.x) && isfinite(r.y) && isfinite(r.z));
            return r;
        },
        counts, offsets, vec != 0, cells, so, s_rec, s_cnt, s_cell);
    if (bad) atomicOr(status, kFlagNonFinite);
}

// The limits of the kernels' dynamic shared memory on the current device, at the most that any build asks
// for.  The limit belongs to the kernel on the device, not to a context: set per call to what that call
// needs, one thread's smaller grid would make another thread's launch fail.
lj_status bin_shared_limits() {
    const auto raise = [](auto kernel, size_t bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
    };
    const size_t hist = kSegMax * sizeof(int), cells = kSegCells * sizeof(int);
    static_assert(kSegMax * sizeof(int) <= kOneBlockPerSm, "k_seg_scatter's slots");
    const bool ok = raise(k_bin_small<LJ_ORDER_X>, (size_t)kSmallParticles * 18 + cells) &&
                    raise(k_bin_small<LJ_ORDER_INDEX>, (size_t)kSmallParticles * 18 + cells) &&
                    raise(k_seg_sort<LJ_ORDER_X, 256, kSegSmall, true>, (size_t)kSegSmall * 18 + cells) &&
                    raise(k_seg_sort<LJ_ORDER_INDEX, 256, kSegSmall, true>, (size_t)kSegSmall * 18 + cells) &&
                    raise(k_seg_sort<LJ_ORDER_X, 1024, kSegLarge, false>, (size_t)kSegLarge * 18 + cells) &&
                    raise(k_seg_sort<LJ_ORDER_INDEX, 1024, kSegLarge, false>, (size_t)kSegLarge * 18 + cells) &&
                    raise(k_seg_count, hist) && raise(k_seg_scatter, kOneBlockPerSm) && large_sort_shared_limit();
    if (!ok) cudaGetLastError();
    return ok ? LJ_OK : LJ_ECUDA;
}

bool small_bin_takes(const lj_ctx* ctx, int n, long long nc) {
    return n >= 1 && n <= kSmallParticles && nc <= kSegCells && ctx->tuning.scatter_passes == 0;
}

lj_status launch_small_bin(lj_ctx* ctx, long long nc, int n, const float* x, const float* y, const float* z, int stride,
                           lj_order order, int* counts, int* offsets, lj_cell_desc* cells, const SortOut& so,
                           const GridDev& g) {
    const auto kernel = order == LJ_ORDER_X ? k_bin_small<LJ_ORDER_X> : k_bin_small<LJ_ORDER_INDEX>;
    const size_t bytes = (size_t)kSmallParticles * 18 + (((size_t)nc * sizeof(int) + 15) & ~(size_t)15);
    const int vec = ((reinterpret_cast<uintptr_t>(counts) | reinterpret_cast<uintptr_t>(offsets)) & 15) == 0;
    kernel<<<1, kSegThreads, bytes, ctx->stream>>>(g, (int)nc, x, y, z, stride, n, counts, offsets, vec, cells, so,
                                                   ctx->d_status);
    return last_launch_status();
}

// Segments of a power of two of cells, kSegAim to twice as many particles on average.  Taken from
// kSegMinParticles particles up (below, its launches and those behind the gate cost what it saves: see
// the figures above), for grids of at most kSegMax * kSegCells cells and at most 256 particles per cell,
// and not where the caller sets the number of scatter passes.
SegPlan segment_plan(const lj_ctx* ctx, int n, long long nc) {
    SegPlan p{0, 0};
    if (n < kSegMinParticles || ctx->tuning.scatter_passes > 0 || (long long)n > 256 * nc) return p;
    const long long want = std::max(1LL, std::min((long long)kSegMax, (long long)n / kSegAim));
    int shift = 0;
    while (((nc + (1LL << shift) - 1) >> shift) > want && (1 << shift) < kSegCells) ++shift;
    const long long nseg = (nc + (1LL << shift) - 1) >> shift;
    if (nseg > kSegMax) return p;
    p.shift = shift;
    p.nseg = (int)nseg;
    return p;
}

template <int ORDER>
static lj_status launch_seg_sorts(lj_ctx* ctx, const SegPlan& plan, long long nc, int n, const SegScratch& sc,
                                  int* counts, int* offsets, lj_cell_desc* cells, const SortOut& so,
                                  const GridDev& g) {
    const auto small = k_seg_sort<ORDER, 256, kSegSmall, true>;
    const auto large = k_seg_sort<ORDER, 1024, kSegLarge, false>;
    const size_t cnt = std::max((size_t)16, sizeof(int) << plan.shift);
    const int vec = ((reinterpret_cast<uintptr_t>(counts) | reinterpret_cast<uintptr_t>(offsets)) & 15) == 0;
    const size_t b_small = (size_t)kSegSmall * 18 + cnt, b_large = (size_t)kSegLarge * 18 + cnt;
    chain_launch(small, plan.nseg, 256, b_small, ctx->stream, g, (int)nc, n, plan.shift, plan.nseg, sc, ctx->tmp4,
                 counts, offsets, vec, cells, so);
    lj_status s;
    if ((s = last_launch_status()) != LJ_OK) return s;
    chain_launch(large, std::min(ctx->sm_count, plan.nseg), 1024, b_large, ctx->stream, g, (int)nc, n, plan.shift,
                 plan.nseg, sc, ctx->tmp4, counts, offsets, vec, cells, so);
    return last_launch_status();
}

// Bytes of an array of one word per segment.
static size_t seg_array(const SegPlan& plan) { return ((size_t)plan.nseg * sizeof(int) + 255) & ~(size_t)255; }

// Makes room for the plan's scratch; false where there is none (no memory, or the stream is being captured, when
// nothing may be allocated): the caller takes the ticket path, which needs less and which an earlier, larger
// build of any grid has made room for.
bool segment_scratch(lj_ctx* ctx, const SegPlan& plan) {
    const size_t need = 256 + 3 * seg_array(plan) + 256 + (size_t)ctx->sm_count * plan.nseg * sizeof(int);
    if (ctx->seg && need <= ctx->seg_bytes) return true;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &capturing) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return capturing == cudaStreamCaptureStatusNone && grow(&ctx->seg, &ctx->seg_bytes, need) == LJ_OK;
}

lj_status launch_segment_bin(lj_ctx* ctx, const SegPlan& plan, long long nc, int n, const float* x, const float* y,
                             const float* z, int stride, lj_order order, int* counts, int* offsets,
                             lj_cell_desc* cells, const SortOut& so, const GridDev& g, const unsigned** gate) {
    const int blocks = ctx->sm_count;
    const size_t seg = seg_array(plan);
    lj_status s;
    char* p = static_cast<char*>(ctx->seg);
    SegScratch sc;
    sc.gate = reinterpret_cast<unsigned*>(p);
    sc.total = reinterpret_cast<int*>(p + 256);
    sc.large = reinterpret_cast<int*>(p + 256 + seg);
    sc.start = reinterpret_cast<int*>(p + 256 + 2 * seg);  // nseg + 1 entries
    sc.base = reinterpret_cast<int*>(p + 256 + 3 * seg + 256);
    sc.id = reinterpret_cast<unsigned short*>(ctx->cell_ticket);  // the tickets' place: used behind the gate only
    *gate = sc.gate;
    cudaStream_t st = ctx->stream;
    if (cudaMemsetAsync(p, 0, 256 + seg, st) != cudaSuccess) return LJ_ECUDA;
    const size_t hist = (size_t)plan.nseg * sizeof(int);
    k_seg_count<<<blocks, kSegThreads, hist, st>>>(g, x, y, z, stride, n, plan.shift, plan.nseg, sc, ctx->d_status);
    if ((s = last_launch_status()) != LJ_OK) return s;
    // In passes of at most kSegRegion bytes of records, so that a run's 16-byte writes meet in L2 before
    // the line leaves it
    const long long passes = std::max(1LL, std::min(8LL, ((long long)n * 16 + kSegRegion - 1) / kSegRegion));
    for (long long q = 0; q < passes; ++q) {
        const int s_lo = (int)(plan.nseg * q / passes), s_hi = (int)(plan.nseg * (q + 1) / passes);
        chain_launch(k_seg_scatter, blocks, kSegThreads, kOneBlockPerSm, st, x, y, z, stride, n, plan.nseg, sc, ctx->tmp4,
                     ctx->d_status, s_lo, s_hi);
        if ((s = last_launch_status()) != LJ_OK) return s;
    }
    return order == LJ_ORDER_X ? launch_seg_sorts<LJ_ORDER_X>(ctx, plan, nc, n, sc, counts, offsets, cells, so, g)
                               : launch_seg_sorts<LJ_ORDER_INDEX>(ctx, plan, nc, n, sc, counts, offsets, cells, so, g);
}

}  // namespace ljc
