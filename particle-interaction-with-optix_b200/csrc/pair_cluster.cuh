// pair_cluster.cuh -- the cluster walk of the truncated law: per-warp routine shared by the
// single-system kernel (pair_cluster.cu) and the batched kernel (batch.cu).
//
// A cluster is 8 consecutive sorted targets of one (y, z) row of cells, counted from the start of an
// aligned run of kCluSegment cells of the row.  A warp holds one cluster at a time (lane l: target
// l & 7) and
//
//   1. finds the 9 stencil rows' candidate ranges for 16 targets (two clusters) at once, lanes 0-8 the
//      starts and lanes 9-17 the ends, so the dependent loads of the searches are paid once per 16 targets;
//   2. scans the ranges, laid end to end, 64 candidates a step, and keeps those within the cutoff of
//      the cluster's bounding box in a list in shared memory (x, y and z apart);
//   3. walks the list: the warp's four lane groups take 4 candidates each, every lane evaluates its
//      target against two candidates at a time in the paired FP32 instructions.  All lanes of a group
//      read the same 16 bytes (one shared-memory wavefront), no lane has a window of its own, nothing
//      is masked (the list is filled up to a multiple of 16 with far candidates) and the own targets
//      are never in the list (they are evaluated apart, where the mask belongs).
//
// Which cells a cluster spans, what it scans and in which order depends on the grid and the row's
// particles only, so a target's sums carry the same bits whatever range of targets, system of a batch
// or slab of layers it is evaluated in.
//
// What bounds it: the paired FP32 instructions read two registers per operand and the register file
// delivers about two per cycle, so a walk step (64 evaluations, 17 paired operations) takes 45 cycles,
// against 34 by the FMA pipe alone (timed apart); the scan takes about as many instructions as the walk
// at 10 particles per cell.  Smaller clusters scan more, larger ones walk more (list lengths on uniform
// particles at 10 per cell: 100, 144 and 205 candidates for 4, 8 and 16 targets, 226 scanned for 8).
// Measured on B200 against the row passes of two targets per lane (kernel 10), pair stage alone, 2M
// uniform particles: 484 against 514 us at 10 per cell, 828 against 1013 at 30, 1805 against 2378 at
// 80, but 401 against 367 at 5 and 379 against 285 at 2 (rows too thin to fill the lanes); at 12 per
// cell 18 against 40 us for 1,000 particles and 47 against 79 for 100,000, where a warp's 16 targets
// instead of 64 leave fewer SMs idle; 10M at 10 per cell 2.14 against 2.33 ms.
#pragma once

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "pair_common.cuh"

namespace ljc {

constexpr int kCluTargets = 8;       // targets of a cluster
constexpr int kCluGroup = 16;        // targets that share their candidate ranges
constexpr int kCluList = 256;        // accepted candidates a warp holds in shared memory
constexpr int kCluSegment = 64;      // cells of a row from whose start clusters are counted (far targets stay apart;
                                     // a segment's last group is half empty: 10M at 10 per cell loses 1% at 16 cells)
constexpr int kCluWarpsPerSm = 28;   // 72 registers per thread (64 spill: a 10M step takes 4% longer)

// A warp's shared memory: the accepted candidates by coordinate, and the candidate ranges.
struct CluSmem {
    float x[kCluList], y[kCluList], z[kCluList];
    int4 range[9];  // first pair of candidates, index of its first candidate minus twice that, end
};

struct CluAcc {
    float2 s12, ns6, fx, fy, fz;  // sums over the even and odd candidates: s^12, -s^6, minus the force sums
    unsigned np;
};

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// r^-2 of an interacting candidate (counted in np), an exact 0 of any other: the reciprocal and the
// count run under the test's predicate (46.1 cycles per 64 evaluations in a timing of the walk alone,
// 47.7 with a select in front of the reciprocal).
__device__ __forceinline__ float rcp_count(float r2, float rc2, unsigned& np) {
    float r;
    asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %2, %3;\n\tmov.f32 %0, 0f00000000;\n\t@p rcp.approx.ftz.f32 %0, %2;\n\t"
        "@p add.u32 %1, %1, 1;\n\t}"
        : "=&f"(r), "+r"(np)
        : "f"(r2), "f"(rc2));
    return r;
}

// The law of two candidates at differences d with r^-2 in ir2 (the same operations, in the same
// order, as the other kernels of the truncated law).
__device__ __forceinline__ void clu_law(float2 dx, float2 dy, float2 dz, float2 ir2, float2 nsig2, CluAcc& a) {
    const float2 s2n = __fmul2_rn(nsig2, ir2);
    const float2 s4 = __fmul2_rn(s2n, s2n);
    const float2 ns6 = __fmul2_rn(s4, s2n);
    const float2 s12 = __fmul2_rn(ns6, ns6);
    a.s12 = __fadd2_rn(a.s12, s12);
    a.ns6 = __fadd2_rn(a.ns6, ns6);
    const float2 t = __ffma2_rn(make_float2(2.0f, 2.0f), s12, ns6);
    const float2 fsn = __fmul2_rn(t, s2n);
    a.fx = __ffma2_rn(fsn, dx, a.fx);
    a.fy = __ffma2_rn(fsn, dy, a.fy);
    a.fz = __ffma2_rn(fsn, dz, a.fz);
}

__device__ __forceinline__ void clu_eval(float2 qx, float2 qy, float2 qz, float2 nx, float2 ny, float2 nz, float rc2,
                                         float2 nsig2, CluAcc& a) {
    const float2 dx = __fadd2_rn(qx, nx);
    const float2 dy = __fadd2_rn(qy, ny);
    const float2 dz = __fadd2_rn(qz, nz);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    float2 ir2;
    ir2.x = rcp_count(r2.x, rc2, a.np);
    ir2.y = rcp_count(r2.y, rc2, a.np);
    clu_law(dx, dy, dz, ir2, nsig2, a);
}

// The list's first cnt candidates (a multiple of 16): lane group s = lane / 8 takes every fourth run of 4.
__device__ __forceinline__ void clu_walk(const CluSmem& sm, int cnt, int s, float2 nx, float2 ny, float2 nz,
                                         float rc2, float2 nsig2, CluAcc& a) {
#pragma unroll 2
    for (int v = 4 * s; v < cnt; v += 16) {
        const float4 X = *reinterpret_cast<const float4*>(&sm.x[v]);
        const float4 Y = *reinterpret_cast<const float4*>(&sm.y[v]);
        const float4 Z = *reinterpret_cast<const float4*>(&sm.z[v]);
        clu_eval(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), nx, ny, nz, rc2, nsig2, a);
        clu_eval(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), nx, ny, nz, rc2, nsig2, a);
    }
}

// Groups per warp for a launch of `waves` waves of one-group warps: the square root balances what a warp
// pays once (its segment, the block's totals) against the last, partly empty wave.  Measured, pair stage at
// 10 per cell, best of 1 to 16 groups: 1 at 1.5 waves (100,000 particles), 3 at 6, 4 at 15 and 25, 6 to 8
// at 45, 8 at 90; 10M (150 waves) 2.22 ms at 4 groups, 2.14 at 12 and 16, 2.15 at 8 and 24.
inline int clu_groups_per_warp(double waves) { return std::max(1, (int)(std::sqrt(waves) + 0.5)); }

// Blocks to make room for in a launch over nk targets of `waves` waves, of which each is one_wave blocks without
// grouping: the most that any smaller launch has (the number itself falls where a warp takes a group more), and
// those of the other walks, so that a smaller launch, or one on a sparser grid, finds its room made.
inline size_t clu_most_blocks(long long nk, double waves, double one_wave) {
    const double most = one_wave * std::max(std::min(2.0 * waves, 1.0), waves / std::max(1.0, std::sqrt(waves) - 0.5));
    return std::max((size_t)most + 2, (size_t)(nk / kPairThreads + 1));
}

// Evaluates the groups that start in [a, b), one warp (all 32 lanes must call): of consecutive groups
// every turns-th from the turn-th on, so that a block's warps share their candidates in L1; of a group
// both clusters, or (only >= 0) the only-th.  p, cs, off:
// the system's sorted records, cell ids (minus cbase) and offsets (minus obase); n particles; groups
// without a target of [kb, ke) are skipped.  emit(k, s, valid, v, w, np, id) is called by all
// lanes for each cluster: valid: k is a target of the lane; v: the target's sum of s^12 - s^6 in lane
// group s = 0, minus its force sums' components x, y, z in groups 1-3; w, np: this lane's share of the
// target's sum of 2 s^12 - s^6 and of its interacting pairs; id: the record's fourth word.
template <bool XWIN, class Emit>
__device__ __forceinline__ void cluster_stretch(const GridDev& g, const PairParams& pp, const float4* p,
                                                const int* cs, int cbase, const int* off,
                                                int obase, int n, int a, int b, int kb, int ke, int turn, int turns,
                                                int only, CluSmem& sm, unsigned* status, Emit emit) {
    const int lane = (int)(threadIdx.x & 31u), t = lane & 7, s = lane >> 3;
    const unsigned below = lanemask_lt();
    const int ncell = g.gx * g.gy * g.gz;
    const float rc2 = pp.rc2;
    const float2 nsig2 = make_float2(-pp.sig2, -pp.sig2);
    int gs = a, se = a, row0 = 0, cy = 0, cz = 0;  // gs: start of the group; se: end of its segment; row0: first cell of its row
    bool entered = false;
    while (gs < b) {
        if (gs >= se) {  // a new segment of cells
            int c = cs[gs] - cbase;
            if (c < 0 || c >= ncell) {
                if (lane == 0) atomicOr(status, kFlagRange);
                c = 0;
            }
            const int row = c / g.gx, cx = c - row * g.gx;
            cz = row / g.gy;
            cy = row - cz * g.gy;
            row0 = row * g.gx;
            const int c0 = row0 + cx / kCluSegment * kCluSegment, c1 = min(c0 + kCluSegment, row0 + g.gx);
            const int ss = min(max(off[c0] - obase, 0), gs);
            se = min(max(off[c1] - obase, gs + 1), n);
            if (!entered) {  // [a, b) may begin inside a group, which then is the previous stretch's
                entered = true;
                gs = min(ss + (gs - ss + kCluGroup - 1) / kCluGroup * kCluGroup, se);
                if (gs >= se) continue;
                if (gs >= b) break;
            }
        }
        const int ge = min(gs + kCluGroup, se);
        if (turn != 0 || ge <= kb || gs >= ke) {
            turn = turn == 0 ? turns - 1 : turn - 1;
            gs = ge;
            continue;
        }
        turn = turns - 1;
        // candidate ranges of the group's box: lanes 0-8 find the start, lanes 9-17 the end of stencil row r
        int T, nr;
        {
            const int k = min(gs + (lane & (kCluGroup - 1)), ge - 1);
            const float4 pi = chain_load(&p[k]);
            const int ck = cs[k] - cbase - row0;
            const int cxa = min(max(__shfl_sync(0xffffffffu, ck, 0), 0), g.gx - 1);
            const int cxb = min(max(__shfl_sync(0xffffffffu, ck, kCluGroup - 1), cxa), g.gx - 1);
            const float bx0 = warp_min(pi.x), bx1 = warp_max(pi.x), by0 = warp_min(pi.y), by1 = warp_max(pi.y),
                        bz0 = warp_min(pi.z), bz1 = warp_max(pi.z);
            int pos = 0;
            const bool second = lane >= 9;
            const int r = second ? lane - 9 : lane;
            if (r < 9) {
                const int rz = r / 3, dz = rz - 1, dy = r - 3 * rz - 1;
                const int z = cz + dz, y = cy + dy;
                if (z >= 0 && z < g.gz && y >= 0 && y < g.gy) {
                    const float m = fmaxf(fmaxf(fmaxf(fabsf(bx0), fabsf(bx1)), fmaxf(fabsf(by0), fabsf(by1))),
                                          fmaxf(fabsf(bz0), fabsf(bz1)));
                    const float slack = pp.slack + 8.0f * FLT_EPSILON * m;
                    float dzm = 0.f, dym = 0.f;
                    if (dz < 0) dzm = bz0 - fmaf((float)cz, g.w, g.oz);
                    if (dz > 0) dzm = fmaf((float)(cz + 1), g.w, g.oz) - bz1;
                    if (dy < 0) dym = by0 - fmaf((float)cy, g.w, g.oy);
                    if (dy > 0) dym = fmaf((float)(cy + 1), g.w, g.oy) - by1;
                    dzm = fmaxf(dzm - slack, 0.f);
                    dym = fmaxf(dym - slack, 0.f);
                    const float d2 = fmaf(dym, dym, dzm * dzm);
                    if (d2 < pp.rc2w) {
                        const int rb = (z * g.gy + y) * g.gx;
                        int lo = min(max(off[rb + max(cxa - 1, 0)] - obase, 0), n);
                        int hi = min(max(off[rb + min(cxb + 1, g.gx - 1) + 1] - obase, lo), n);
                        if (XWIN) {
                            const float h = sqrtf(pp.rc2w - d2) + slack;
                            const float v = second ? bx1 + h : bx0 - h;
                            while (lo < hi) {  // first x >= v (starts) or x > v (ends)
                                const int mid = (lo + hi) >> 1;
                                const float x = p[mid].x;
                                if (x < v || (second && x == v))
                                    lo = mid + 1;
                                else
                                    hi = mid;
                            }
                            pos = lo;
                        } else {
                            pos = second ? hi : lo;
                        }
                    }
                }
            }
            // the ranges end to end as pairs of candidates (an odd range's last pair holds one), empty ones dropped
            const int re = __shfl_down_sync(0xffffffffu, pos, 9);
            const int pairs = lane < 9 ? (max(re - pos, 0) + 1) >> 1 : 0;
            int inc = pairs;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            T = __shfl_sync(0xffffffffu, inc, 8);
            const unsigned full = __ballot_sync(0xffffffffu, pairs > 0);
            nr = __popc(full);
            if (pairs > 0) sm.range[__popc(full & below)] = make_int4(inc - pairs, pos - 2 * (inc - pairs), re, 0);
            __syncwarp();
        }
        const int4 rng = lane < nr ? sm.range[lane] : make_int4(INT_MAX, 0, 0, 0);
        __syncwarp();
        for (int cl = only < 0 ? gs : gs + only * kCluTargets; cl < ge; cl += only < 0 ? kCluTargets : kCluGroup) {
            const int nt = min(kCluTargets, ge - cl);
            const int k = cl + min(t, nt - 1);  // lanes past the end repeat the last target
            const float4 pi = chain_load(&p[k]);
            const float bx0 = warp_min(pi.x), bx1 = warp_max(pi.x), by0 = warp_min(pi.y), by1 = warp_max(pi.y),
                        bz0 = warp_min(pi.z), bz1 = warp_max(pi.z);
            const float2 nx = make_float2(-pi.x, -pi.x), ny = make_float2(-pi.y, -pi.y), nz = make_float2(-pi.z, -pi.z);
            CluAcc acc;
            acc.s12 = acc.ns6 = acc.fx = acc.fy = acc.fz = make_float2(0.f, 0.f);
            acc.np = 0;
            {  // the cluster's own targets: lane group s takes targets 2s and 2s + 1
                const int c0 = 2 * s, c1 = c0 + 1;
                const float2 dx = __fadd2_rn(make_float2(__shfl_sync(0xffffffffu, pi.x, c0),
                                                         __shfl_sync(0xffffffffu, pi.x, c1)), nx);
                const float2 dy = __fadd2_rn(make_float2(__shfl_sync(0xffffffffu, pi.y, c0),
                                                         __shfl_sync(0xffffffffu, pi.y, c1)), ny);
                const float2 dz = __fadd2_rn(make_float2(__shfl_sync(0xffffffffu, pi.z, c0),
                                                         __shfl_sync(0xffffffffu, pi.z, c1)), nz);
                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                const float inf = __int_as_float(0x7f800000);
                float2 ir2;
                ir2.x = rcp_count(c0 != t && c0 < nt ? r2.x : inf, rc2, acc.np);
                ir2.y = rcp_count(c1 != t && c1 < nt ? r2.y : inf, rc2, acc.np);
                clu_law(dx, dy, dz, ir2, nsig2, acc);
            }
            // scan: 64 candidates a step, those within the cutoff of the cluster's box go to the list.  The
            // box test rounds as the distance test does, operation by operation on smaller magnitudes, so
            // it never drops a candidate that the distance test of any target accepts.
            int cnt = 0, before = -1;  // before: index of the last range that starts below base
            for (int base = 0; base < T; base += 32) {
                const unsigned rel = (unsigned)(rng.x - base);
                const unsigned starts = __reduce_or_sync(0xffffffffu, rel < 32u ? 1u << rel : 0u);
                const int ri = before + __popc(starts & (below * 2u + 1u));
                before += __popc(starts);
                const int j = 2 * (base + lane) + __shfl_sync(0xffffffffu, rng.y, ri);
                const int je = __shfl_sync(0xffffffffu, rng.z, ri);
                const bool ok0 = j < je, ok1 = j + 1 < je;
                const float4 q0 = chain_load(&p[ok0 ? j : cl]);
                const float4 q1 = chain_load(&p[ok1 ? j + 1 : cl]);
                const float dx0 = fmaxf(fmaxf(bx0 - q0.x, q0.x - bx1), 0.f), dx1 = fmaxf(fmaxf(bx0 - q1.x, q1.x - bx1), 0.f);
                const float dy0 = fmaxf(fmaxf(by0 - q0.y, q0.y - by1), 0.f), dy1 = fmaxf(fmaxf(by0 - q1.y, q1.y - by1), 0.f);
                const float dz0 = fmaxf(fmaxf(bz0 - q0.z, q0.z - bz1), 0.f), dz1 = fmaxf(fmaxf(bz0 - q1.z, q1.z - bz1), 0.f);
                const float d0 = fmaf(dz0, dz0, fmaf(dy0, dy0, dx0 * dx0));
                const float d1 = fmaf(dz1, dz1, fmaf(dy1, dy1, dx1 * dx1));
                const unsigned own = (unsigned)(j - cl);
                const bool keep0 = ok0 && d0 < rc2 && own >= (unsigned)nt, keep1 = ok1 && d1 < rc2 && own + 1u >= (unsigned)nt;
                const unsigned kept0 = __ballot_sync(0xffffffffu, keep0), kept1 = __ballot_sync(0xffffffffu, keep1);
                const int mid = cnt + __popc(kept0);
                if (keep0) {
                    const int w = cnt + __popc(kept0 & below);
                    sm.x[w] = q0.x;
                    sm.y[w] = q0.y;
                    sm.z[w] = q0.z;
                }
                if (keep1) {
                    const int w = mid + __popc(kept1 & below);
                    sm.x[w] = q1.x;
                    sm.y[w] = q1.y;
                    sm.z[w] = q1.z;
                }
                cnt = mid + __popc(kept1);
                if (cnt > kCluList - 64 && base + 32 < T) {  // no room for another step: walk the whole runs, keep the rest
                    __syncwarp();
                    const int whole = cnt & ~15;
                    clu_walk(sm, whole, s, nx, ny, nz, rc2, nsig2, acc);
                    __syncwarp();
                    const int rest = cnt - whole;
                    if (lane < rest) {
                        sm.x[lane] = sm.x[whole + lane];
                        sm.y[lane] = sm.y[whole + lane];
                        sm.z[lane] = sm.z[whole + lane];
                    }
                    cnt = rest;
                }
            }
            // fill the last run with candidates that no target accepts (kFarPlace)
            if (lane < ((16 - cnt) & 15)) sm.x[cnt + lane] = sm.y[cnt + lane] = sm.z[cnt + lane] = kFarPlace;
            __syncwarp();
            clu_walk(sm, (cnt + 15) & ~15, s, nx, ny, nz, rc2, nsig2, acc);
            __syncwarp();
            // the 4 lane groups' sums: halves of (e, fx, fy, fz) exchanged twice, one value left per group
            const float s12 = acc.s12.x + acc.s12.y, ns6 = acc.ns6.x + acc.ns6.y;
            const float e = s12 + ns6, fx = acc.fx.x + acc.fx.y, fy = acc.fy.x + acc.fy.y, fz = acc.fz.x + acc.fz.y;
            const bool hi2 = (s & 2) != 0, hi1 = (s & 1) != 0;
            const float u0 = (hi2 ? fy : e) + __shfl_xor_sync(0xffffffffu, hi2 ? e : fy, 16);
            const float u1 = (hi2 ? fz : fx) + __shfl_xor_sync(0xffffffffu, hi2 ? fx : fz, 16);
            const float v = (hi1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, hi1 ? u0 : u1, 8);
            emit(k, s, t < nt, v, fmaf(2.0f, s12, ns6), acc.np, __float_as_int(pi.w));
        }
        gs = ge;
    }
}

}  // namespace ljc
