// pair_compat.cu -- the reference law on filled grids: one warp per cell.
//
// Every particle of a cell has the same partners, the particles of the clamped 27-cell stencil but
// itself (no cutoff), so a warp takes a cell: it copies the stencil's particles outside the cell to
// shared memory, x, y and z apart, and its targets walk that one list without a mask, in the paired
// FP32 instructions.  Lane l holds targets l % 4, l % 4 + 4, ... (up to 4, so 16 per round) and the
// eight lane groups take two candidates each per step; the 4 lanes of a group read the same 8 bytes per
// coordinate, and what a step loads serves 16 targets.  The cell's own particles are evaluated apart,
// where the mask j != k belongs.
//
// A warp takes at most a chunk of its cell's targets, 64 or, on few cells, 16; the rest of a crowded cell goes to
// other warps, so that the time follows the number of targets and not the fullest cell.  Measured on B200, one
// warp for all of a cell's targets -> chunks (two targets per lane, k_pair_compat): 10,000 particles in one cell
// 155 ms -> 0.26 (1.22), 100,000 on 27 cells 216 -> 2.55 (15.7), 1,000,000 with 20,000 in one cell 634 -> 2.0
// (2.9); and on evenly filled cells, where the search for crowded ones costs, 1M at 8 per cell 168 -> 171 us,
// 4.2M at 16 902 -> 918.  In a launch of its own that search costs 6 us there, but the crowded cells' first
// chunks then run alone (droplets up to twice as long).
//
// What bounds it: 11 paired operations and two reciprocal square roots per two evaluations, about 25
// cycles per 64 evaluations by register reads and by the FMA pipe (22); at 16 per cell that is two
// thirds of the 0.92 ms that 4.2M particles take on B200 (1.52 ms with two targets per lane; 6 blocks per SM and
// 76 registers instead of 8 and 64 take 6% longer).  k_pair_compat (pair.cu), two targets of possibly different cells
// per lane, masks every candidate against both targets' cells and ranges and duplicates each coordinate
// for them.
#include <algorithm>
#include <climits>

#include "pair_common.cuh"

namespace ljc {

namespace {
constexpr int kCellWarps = 4;
constexpr int kCellList = 512;   // candidates a warp holds
constexpr int kCellLanes = 4;    // lanes across the targets
constexpr int kCellDeep = 4;     // targets per lane and round

struct CellSmem {
    float x[kCellList], y[kCellList], z[kCellList];
    int4 range[10];  // first pair of candidates, index of its first candidate minus twice that, end
};
}  // namespace

__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Adds r^-12 - r^-6 of two candidates at differences d, r^2 = d.d + 1e-5, to pot.  As r^-6 (r^-6 - 1):
// one rounding less than the two powers' difference.
__device__ __forceinline__ void compat_law(float2 dx, float2 dy, float2 dz, float2& pot, bool m0 = true,
                                           bool m1 = true) {
    float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, make_float2(1e-5f, 1e-5f))));
    const float inf = __int_as_float(0x7f800000);
    const float2 sdr = make_float2(rsqrt_ftz(m0 ? r2.x : inf), rsqrt_ftz(m1 ? r2.y : inf));
    const float2 s2 = __fmul2_rn(sdr, sdr);
    const float2 s4 = __fmul2_rn(s2, s2);
    const float2 r6 = __fmul2_rn(s4, s2);
    pot = __ffma2_rn(r6, __fadd2_rn(r6, make_float2(-1.0f, -1.0f)), pot);
}

template <int NT>
__device__ __forceinline__ void cell_walk(const CellSmem& sm, int cnt, int group, const float2 (&nx)[kCellDeep],
                                          const float2 (&ny)[kCellDeep], const float2 (&nz)[kCellDeep],
                                          float2 (&pot)[kCellDeep]) {
#pragma unroll 2
    for (int v = 2 * group; v < cnt; v += 16) {
        const float2 X = *reinterpret_cast<const float2*>(&sm.x[v]);
        const float2 Y = *reinterpret_cast<const float2*>(&sm.y[v]);
        const float2 Z = *reinterpret_cast<const float2*>(&sm.z[v]);
#pragma unroll
        for (int q = 0; q < NT; ++q)
            compat_law(__fadd2_rn(X, nx[q]), __fadd2_rn(Y, ny[q]), __fadd2_rn(Z, nz[q]), pot[q]);
    }
}

// Evaluates the targets [t0, t1) of cell c, which holds [cs, ce) (one warp, all lanes).
__device__ __forceinline__ void cell_targets(const GridDev& g, const float4* p, const int* off,
                                             int n, int c, int cs, int ce, int t0, int t1, CellSmem& sm,
                                             float* __restrict__ v) {
    const int lane = (int)(threadIdx.x & 31u), t = lane % kCellLanes, group = lane / kCellLanes;
    const unsigned below = lanemask_lt();
    // the stencil's ranges: lane r < 9 reads row r; the own row's parts before and after the cell
    int T, nr;
    {
        int cx, cy, cz;
        decode_cell(g, c, cx, cy, cz);
        int s = 0, e = 0;
        if (lane < 9) {
            const int z = cz + lane / 3 - 1, y = cy + lane % 3 - 1;
            if (z >= 0 && z < g.gz && y >= 0 && y < g.gy) {
                const int rb = (z * g.gy + y) * g.gx;
                s = min(max(off[rb + max(cx - 1, 0)], 0), n);
                e = min(max(off[rb + min(cx + 1, g.gx - 1) + 1], s), n);
            }
        }
        const int src = lane == 9 ? 4 : min(lane, 8);
        s = __shfl_sync(0xffffffffu, s, src);
        e = __shfl_sync(0xffffffffu, e, src);
        if (lane == 4) e = min(e, cs);
        if (lane == 9) s = max(s, ce);
        const int pairs = lane < 10 ? (max(e - s, 0) + 1) >> 1 : 0;  // an odd range's last pair holds one
        int inc = pairs;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += q;
        }
        T = __shfl_sync(0xffffffffu, inc, 9);
        const unsigned full = __ballot_sync(0xffffffffu, pairs > 0);
        nr = __popc(full);
        if (pairs > 0) sm.range[__popc(full & below)] = make_int4(inc - pairs, s - 2 * (inc - pairs), e, 0);
        __syncwarp();
    }
    const int4 rng = lane < nr ? sm.range[lane] : make_int4(INT_MAX, 0, 0, 0);
    bool staged = false;  // the whole list is in shared memory already
    for (int k0 = t0; k0 < t1; k0 += kCellLanes * kCellDeep) {
        const int m = min(t1 - k0, kCellLanes * kCellDeep), deep = (m + kCellLanes - 1) / kCellLanes;
        float2 nx[kCellDeep], ny[kCellDeep], nz[kCellDeep], pot[kCellDeep];
#pragma unroll
        for (int q = 0; q < kCellDeep; ++q) {
            const float4 r = p[k0 + min(t + kCellLanes * q, m - 1)];
            nx[q] = make_float2(-r.x, -r.x);
            ny[q] = make_float2(-r.y, -r.y);
            nz[q] = make_float2(-r.z, -r.z);
            pot[q] = make_float2(0.f, 0.f);
        }
        // own cell: two particles per lane group and step, never a target itself
        for (int j0 = cs; j0 < ce; j0 += 16) {
            const int j = j0 + 2 * group;
            const float4 a = p[min(j, ce - 1)], b = p[min(j + 1, ce - 1)];
            const float2 X = make_float2(a.x, b.x), Y = make_float2(a.y, b.y), Z = make_float2(a.z, b.z);
#pragma unroll
            for (int q = 0; q < kCellDeep; ++q) {
                const int k = k0 + t + kCellLanes * q;
                if (q < deep)
                    compat_law(__fadd2_rn(X, nx[q]), __fadd2_rn(Y, ny[q]), __fadd2_rn(Z, nz[q]), pot[q],
                               j < ce && j != k, j + 1 < ce && j + 1 != k);
            }
        }
        int base = 0, before = -1;  // before: index of the last range that starts below base
        do {
            int cnt = 0;
            if (staged) {
                cnt = (T * 2 + 15) & ~15;
                base = T;
            } else {
                // up to kCellList candidates, 64 a step; an odd range's missing candidate is a far one
                for (; base < T && cnt + 64 <= kCellList; base += 32, cnt += 64) {
                    const unsigned rel = (unsigned)(rng.x - base);
                    const unsigned starts = __reduce_or_sync(0xffffffffu, rel < 32u ? 1u << rel : 0u);
                    const int ri = before + __popc(starts & (below * 2u + 1u));
                    before += __popc(starts);
                    const int j = 2 * (base + lane) + __shfl_sync(0xffffffffu, rng.y, ri);
                    const int je = __shfl_sync(0xffffffffu, rng.z, ri);
                    float4 a = make_float4(kFarPlace, kFarPlace, kFarPlace, 0.f), b = a;  // its term is an exact 0
                    if (j < je) a = p[j];
                    if (j + 1 < je) b = p[j + 1];
                    const int w = cnt + 2 * lane;
                    *reinterpret_cast<float2*>(&sm.x[w]) = make_float2(a.x, b.x);
                    *reinterpret_cast<float2*>(&sm.y[w]) = make_float2(a.y, b.y);
                    *reinterpret_cast<float2*>(&sm.z[w]) = make_float2(a.z, b.z);
                }
                staged = base >= T && 2 * T <= kCellList;
                if (base > T) cnt -= 2 * (base - T) / 16 * 16;  // without the whole runs of 16 past the end
            }
            __syncwarp();
            switch (deep) {
                case 1: cell_walk<1>(sm, cnt, group, nx, ny, nz, pot); break;
                case 2: cell_walk<2>(sm, cnt, group, nx, ny, nz, pot); break;
                case 3: cell_walk<3>(sm, cnt, group, nx, ny, nz, pot); break;
                default: cell_walk<4>(sm, cnt, group, nx, ny, nz, pot);
            }
            __syncwarp();
        } while (base < T);
#pragma unroll
        for (int q = 0; q < kCellDeep; ++q) {
            float s = pot[q].x + pot[q].y;
#pragma unroll
            for (int o = kCellLanes; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const int k = k0 + t + kCellLanes * q;
            if (group == 0 && k < t1) v[k] = 4.0f * s;
        }
    }
}

// Work items: the first `chunk` targets of every cell, one warp each, and the chunks beyond them of cells that
// hold more, which the launch's first `finders` warps look for.  Window q of the sorted targets, [q chunk,
// (q + 1) chunk), holds the start of at most one such chunk, and one of the cell that holds the window's first
// target; a finder takes every finders-th window, so the chunks of one crowded cell go to different warps.  The
// finders also look at every target's cell id: one outside the grid is reported.
__global__ void __launch_bounds__(32 * kCellWarps, 8) k_compat_cells(GridDev g, const float4* p,
                                                                     const int* cell_id,
                                                                     const int* off, int n, int chunk,
                                                                     int windows, int finders, float* __restrict__ v,
                                                                     unsigned* status) {
    __shared__ __align__(16) CellSmem smem[kCellWarps];
    chain_wait();
    const int lane = (int)(threadIdx.x & 31u);
    const int ncell = g.gx * g.gy * g.gz;
    const long long warp = (long long)blockIdx.x * kCellWarps + (threadIdx.x >> 5);
    int c = 0, cs = 0, ce = 0, t0 = 0;
    if (warp < finders) {
        const long long q = warp + (long long)lane * finders;
        if (q < windows) {
            const int k = (int)(q * chunk);
            c = cell_id[k];
            if (c >= 0 && c < ncell) {
                cs = min(max(off[c], 0), k);
                ce = min(off[c + 1], n);
                const long long start = cs + (long long)(k - cs + chunk - 1) / chunk * chunk;
                t0 = start > cs ? (int)min(start, (long long)INT_MAX) : ce;
            }
        }
        const int hi = (int)((long long)n * (warp + 1) / finders);
        bool bad = false;
#pragma unroll 4
        for (int k = (int)((long long)n * warp / finders) + lane; k < hi; k += 32) {
            const int id = cell_id[k];
            bad |= id < 0 || id >= ncell;
        }
        if (bad) atomicOr(status, kFlagRange);
    } else if (warp - finders < ncell && lane == 0) {
        c = (int)(warp - finders);
        t0 = cs = min(max(off[c], 0), n);
        ce = min(off[c + 1], n);
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, t0 < ce); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1, start = __shfl_sync(0xffffffffu, t0, src), end = __shfl_sync(0xffffffffu, ce, src);
        cell_targets(g, p, off, n, __shfl_sync(0xffffffffu, c, src), __shfl_sync(0xffffffffu, cs, src), end, start,
                     end - start < chunk ? end : start + chunk, smem[threadIdx.x >> 5], v);
    }
}

lj_status launch_compat_cells(lj_ctx* ctx, const lj_grid* g, int n, const float* xyzi, const int* cell_id,
                              const int* off, float* v) {
    const long long nc = (long long)g->dim[0] * g->dim[1] * g->dim[2];
    // A chunk of four rounds where the cells alone fill the GPU, of one round where they do not; as many finders as
    // run at once, each with at most a window per lane.
    const long long warps = (long long)ctx->sm_count * kCompatWarpsPerSm;
    const int chunk = kCellLanes * kCellDeep * (nc >= warps ? 4 : 1);
    const long long windows = ((long long)n + chunk - 1) / chunk;
    const long long per = std::min(32LL, std::max(1LL, windows / warps));
    const long long finders = (windows + per - 1) / per;
    chain_launch(k_compat_cells, (unsigned)((nc + finders + kCellWarps - 1) / kCellWarps), 32 * kCellWarps, 0,
                 ctx->stream, to_dev(*g), reinterpret_cast<const float4*>(xyzi), cell_id, off, n, chunk, (int)windows,
                 (int)finders, v, ctx->d_status);
    return last_launch_status();
}

}  // namespace ljc
