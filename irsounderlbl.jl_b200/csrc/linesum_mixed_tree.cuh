// linesum_mixed_tree.cuh -- the FP32 forward line sum (IRS_MIXED: Weideman and FullFaddeeva)
// with its far lines on the block tree of linesum_tree32.cuh.
//
//  fw_tree_kernel  node values of every (segment, leaf of 128 points): one CTA per (strip of
//                  4096 points, segment)
//  fw_leaf_kernel  one warp per leaf: the lines near it (and those whose cutoff falls among
//                  its points) point by point, the interpolated far field, the clamp, the sum
//                  over the segments
//
// Near lines of a leaf, by class (a line is staged once per leaf, tiles of 32):
//   fast     wing at every point, inside the cutoff: two points per reciprocal, packed
//   edge     wing, the cutoff falls among the points: packed, masked by the cutoff test
//   core     inside the cutoff and the Faddeeva core (|x| <= x_far) reaches some points: the
//            pairs of 32-point rows that it reaches take the real part of the two-level
//            continued fraction and the wing as one quotient
//              H = K n / (m q),  m = x^2 + y^2,  K = y/sqrt(pi),
//              n = m^2 - 3/2 x^2 + 5/2 y^2 + 3/2,  q = m^2 - 3 x^2 + 3 y^2 + 9/4
//            (wing: n = q = 1), packed, one reciprocal for two points; the points with
//            |x| + y < 15 come from a buffer evaluated lane-parallel
//   general  core and cutoff edge, or a cutoff within 8 times the core's reach (where H and
//            the pedestal nearly cancel): per-pair tests, the continued fraction inline.  (With
//            the rule at 8 times the reach and half a leaf, every core of a step of 0.05 to 0.1
//            cm^-1 was general: 5,000 lines x 2,000 points 0.81 / 1.06 ms, now 0.72 / 0.88; with m^3
//            of the quotient in range up to |x| = 1.4e3 only, x_far = 3000 took 0.70 ms for
//            34,801 points, now 0.50.)
// Pedestals of fast and core lines are quadratics in the point index, summed per lane.
//
// Bound by issue (78 to 82 % of the slots in both kernels).  Measured on a B200 (far + near lines),
// against a 2048-point strip pre-pass, each warp's 8 far nodes from 320 points, window searches
// and per-row core evaluation: six IASI profiles, 400,000 lines 10.3 + 95.2 -> 15.0 + 61.1 ms;
// two CrIS long-wave profiles with VP_Y 0.64 + 4.19 -> 0.87 + 1.97 ms; one scene of the
// 5,000-line list 30 + 236 -> 67 + 124 us.  Of the 61 ms the cores take 30 (half of it the points
// with |x| + y < 15; 1.1 the core rows' own offsets and the floor of their quotient), the cutoff
// edges 7, the interpolation 2, staging and the segments' fixed work the rest.  64 registers at
// four CTAs per SM; three CTAs (80 registers, no spills) 62.8 ms against 60.0.
#pragma once
#include "linesum_tree32.cuh"

namespace irs {

constexpr int kFwWarps = 8;

__host__ __device__ constexpr int fw_sums(bool lm) { return lm ? 2 : 1; }

// idx[seg][j] of every segment's kept lines (CellIndex): thread t owns the cells after line
// t - 1's up to line t's; long gaps are filled by the warp.
__global__ void __launch_bounds__(256) cell_fill_kernel(const SegDev* __restrict__ segs, const int* __restrict__ seg_count,
                                                        const double* __restrict__ V, int n, double inv_cell, double off,
                                                        int* __restrict__ idx) {
    const int s = blockIdx.y, cnt = seg_count[s], lane = threadIdx.x & 31;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t - lane > cnt) return;  // whole warps
    const double* v = V + segs[s].off;
    int* row = idx + (size_t)s * n;
    // first cell boundary j with (V + 0.5 + off) / cell < j, clamped: cells j are those at or
    // below a line's key when row[j] <= its index
    auto after = [&](int i) -> int {  // boundaries at or before line i's key: j <= (V + .5 + off)/cell
        const double c = floor((v[i] + 0.5 + off) * inv_cell);
        return c < 0.0 ? 0 : c >= (double)(n - 1) ? n : (int)c + 1;
    };
    int a = 0, b = 0;
    if (t <= cnt) {
        a = t == 0 ? 0 : after(t - 1);
        b = t == cnt ? n : after(t);
    }
    const bool big = b - a > 64;
    if (!big)
        for (int j = a; j < b; ++j) row[j] = t;
    unsigned m = __ballot_sync(kFull, big);
    while (m) {
        const int l = __ffs(m) - 1;
        m &= m - 1;
        const int a2 = __shfl_sync(kFull, a, l), b2 = __shfl_sync(kFull, b, l), t2 = __shfl_sync(kFull, t, l);
        for (int j = a2 + lane; j < b2; j += 32) row[j] = t2;
    }
}

// ------------------------------------------------------------------ far lines
// one warp's share of a block's far lines at its 16 nodes: (value, dispersive) of node
// lane % 16 in every lane
template <bool LM>
__device__ __forceinline__ float2 fw_block(const LpOutMixed& lp, long long off, const TreeList& TL, int first, int step,
                                           float cb, float h, int lane, float4* __restrict__ T, float* __restrict__ Tg) {
    const float2 xp = make_float2(h * tree_node_f(lane & 7), h * tree_node_f((lane & 7) + 8));
    const float2 xs = make_float2(xp.y, xp.x);
    float2 vs = make_float2(0.f, 0.f), vc = vs, ds = vs, dc = vs;
    float PA = 0.f, PAc = 0.f, PB = 0.f, PBc = 0.f, PC = 0.f, PCc = 0.f;
    for (int t0 = 32 * first; t0 < TL.n; t0 += 32 * step) {
        const int nt = min(32, TL.n - t0);
        __syncwarp();
        if (lane < nt) {
            const long long q = off + tree_line(TL, t0 + lane);
            const float2 uf = lp.U[q];
            const float4 a0 = lp.p0[q];
            const float uh = (uf.x - cb) - (h - 0.5f);  // exact: see split_hi_lo
            T[lane] = make_float4(uh, uf.y, a0.x, a0.y);
            if (LM) Tg[lane] = lp.p2[q].x;
            // c1 (x - u)^2 + c0 = c1 x^2 - 2 c1 u x + (c1 u^2 + c0)
            const float u = uh + uf.y, pb = a0.z * u;
            kahan_add(PA, PAc, a0.z);
            kahan_add(PB, PBc, pb);
            kahan_add(PC, PCc, fmaf(pb, u, a0.w));
        }
        __syncwarp();
        float2 v = make_float2(0.f, 0.f), d = v;
        for (int k = lane >> 3; k < nt; k += 4) {  // lane: nodes lane % 8 and + 8, every fourth line
            const float4 f = T[k];
            const float2 nu_ = make_float2(-f.x, -f.x), nl = make_float2(-f.y, -f.y);
            const float2 dsw = __fadd2_rn(__fadd2_rn(xs, nu_), nl);
            const float2 es = __ffma2_rn(dsw, dsw, make_float2(f.z, f.z));
            const float R = rcp_fast(es.x * es.y);
            const float2 r = __fmul2_rn(es, make_float2(R, R));
            v = __ffma2_rn(make_float2(f.w, f.w), r, v);
            if (LM) {
                const float g = Tg[k];
                d = __ffma2_rn(__fmul2_rn(make_float2(g, g), make_float2(dsw.y, dsw.x)), r, d);
            }
        }
        kahan_add(vs.x, vc.x, v.x);
        kahan_add(vs.y, vc.y, v.y);
        if (LM) {
            kahan_add(ds.x, dc.x, d.x);
            kahan_add(ds.y, dc.y, d.y);
        }
    }
    auto groups = [&](float2 x) {  // the four line groups; node lane % 16
        x.x += __shfl_xor_sync(kFull, x.x, 8);
        x.y += __shfl_xor_sync(kFull, x.y, 8);
        x.x += __shfl_xor_sync(kFull, x.x, 16);
        x.y += __shfl_xor_sync(kFull, x.y, 16);
        return (lane & 8) ? x.y : x.x;
    };
    const float A = warp_sum(PA - PAc), B = warp_sum(PB - PBc), C = warp_sum(PC - PCc);
    const float xk = (lane & 8) ? xp.y : xp.x;
    return make_float2(groups(vs) + fmaf(xk, fmaf(xk, A, -2.f * B), C), LM ? groups(ds) : 0.f);
}

// the ranges of the level's blocks, one lane each (lane b: block b), inside their parents'
__device__ __forceinline__ int4 fw_level_ranges(const CellIndex& ci, const int* row, int l, long long sb, float cut, float m,
                                                float reach, int4 up, int lane) {
    const int nb = 1 << l;
    if (lane >= nb) return make_int4(0, 0, 0, 0);
    const float h = (float)(kTrStrip >> (l + 1));
    return tree_inside(tree_ranges(ci, row, (float)(sb + (long long)lane * (kTrStrip >> l)), h, cut, m, reach), up);
}
__device__ __forceinline__ int4 shfl_int4(int4 v, int src) {
    return make_int4(__shfl_sync(kFull, v.x, src), __shfl_sync(kFull, v.y, src), __shfl_sync(kFull, v.z, src),
                     __shfl_sync(kFull, v.w, src));
}

// A whole (strip, segment) by one warp, for launches with enough of them: the levels' blocks
// one after the other, no block-wide barriers, the node values of a level in place of their
// parents' (children 2b, 2b + 1 written from the last block down).  Against eight warps per
// (strip, segment), whose bounds, epilogues and barriers are per warp, 20.5 -> 15.0 ms on six
// IASI profiles (370,440 strips) and 1.33 -> 0.87 ms on the two CrIS ones.
template <bool ANY_LM, bool LM>
__device__ __forceinline__ void fw_tree_warp(const LpOutMixed& lp, long long off, const CellIndex& ci, const int* row,
                                             long long sb, float cut, float m, float reach, long long n_nu,
                                             const TreeTables* __restrict__ tab, float* __restrict__ far,
                                             int4* __restrict__ ranges, int lane, float4* __restrict__ T,
                                             float* __restrict__ Tg, double (*__restrict__ F)[fw_sums(ANY_LM)][kTrNodes],
                                             unsigned& work) {
    int4 up = make_int4(0, 0, 0, 0);  // lane b: block b's parent's ranges
    const int j = lane & (kTrNodes - 1);
#pragma unroll 1
    for (int l = 0; l < kTrLevels; ++l) {
        const int nb = 1 << l, size = kTrStrip >> l;
        const float h = (float)(size >> 1);
        const int4 own = fw_level_ranges(ci, row, l, sb, cut, m, reach, up, lane);
        if (l + 1 == kTrLevels) ranges[lane] = own;
        for (int b = l ? nb - 2 : 0; b >= 0; b -= 2) {  // a pair of blocks: lanes 0..15 the left one's nodes
            const long long cb = sb + (long long)b * size;
            if (cb >= n_nu) continue;  // warp-uniform
            float2 v = make_float2(0.f, 0.f);
            for (int s = 0; s < (l ? 2 : 1); ++s) {
                const int4 u = shfl_int4(up, b + s), o = shfl_int4(own, b + s);
                const TreeList TL = tree_list(o, u);
                if (lane == 0) work += (unsigned)TL.n * kTrNodes;
                const float2 x = fw_block<LM>(lp, off, TL, 0, 1, (float)(cb + s * size), h, lane, T, Tg);
                if ((lane >> 4) == s) v = x;
            }
            const int bl = b + (l ? lane >> 4 : 0);
            double d0 = (double)v.x, d1 = (double)v.y;
            if (l) {
                const double(*fp)[kTrNodes] = F[b >> 1];
#pragma unroll
                for (int k = 0; k < kTrNodes; ++k) {
                    const double w = tab->M[lane >> 4][k][j];
                    d0 = fma(fp[0][k], w, d0);
                    if (LM) d1 = fma(fp[fw_sums(ANY_LM) - 1][k], w, d1);
                }
            }
            __syncwarp();  // the parent is read (block 0's is overwritten here)
            if (l + 1 < kTrLevels) {
                if (l || lane < kTrNodes) {
                    F[bl][0][j] = d0;
                    if (LM) F[bl][fw_sums(ANY_LM) - 1][j] = d1;
                }
            } else {
                far[(bl * fw_sums(ANY_LM)) * kTrNodes + j] = (float)d0;
                if (LM) far[(bl * fw_sums(ANY_LM) + 1) * kTrNodes + j] = (float)d1;
            }
            __syncwarp();
        }
        // lane b of the next level: block b >> 1 of this one
        up = shfl_int4(own, lane >> 1);
    }
}

template <bool ANY_LM, bool LM>
__device__ __forceinline__ void fw_tree_segment(const LpOutMixed& lp, long long off, const CellIndex& ci, const int* row,
                                                float cut, float m, float reach, long long n_nu,
                                                const TreeTables* __restrict__ tab, float* __restrict__ far,
                                                int4* __restrict__ ranges, unsigned long long* __restrict__ evald) {
    constexpr int NC = fw_sums(ANY_LM);
    __shared__ float4 tiles[kFwWarps][32];
    __shared__ float tiles_g[ANY_LM ? kFwWarps : 1][32];
    __shared__ float part[kTrLeaves][NC][kTrNodes];
    __shared__ double F[2][kTrLeaves / 2][NC][kTrNodes];
    __shared__ int4 rg[2][kTrLeaves / 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long sb = (long long)blockIdx.x * kTrStrip;
    unsigned work = 0;
#pragma unroll 1
    for (int l = 0; l < kTrLevels; ++l) {
        const int nb = 1 << l, wpb = l < 3 ? kFwWarps >> l : 1, bpw = l < 3 ? 1 : nb / kFwWarps;
        const float h = (float)(kTrStrip >> (l + 1));
        for (int i = 0; i < bpw; ++i) {
            const int b = l < 3 ? warp / wpb : warp * bpw + i;
            const long long cb = sb + (long long)b * (kTrStrip >> l);
            if (cb >= n_nu) break;  // warp-uniform
            const int4 u = l ? rg[(l + 1) & 1][b >> 1] : make_int4(0, 0, 0, 0);
            const int4 own = tree_inside(tree_ranges(ci, row, (float)cb, h, cut, m, reach), u);
            const TreeList TL = tree_list(own, u);
            const float2 v = fw_block<LM>(lp, off, TL, l < 3 ? warp % wpb : 0, wpb, (float)cb, h, lane, tiles[warp],
                                          tiles_g[ANY_LM ? warp : 0]);
            if (lane < kTrNodes) {
                part[l < 3 ? warp : b][0][lane] = v.x;
                if (LM) part[l < 3 ? warp : b][NC - 1][lane] = v.y;
            }
            if (lane == 0 && (l >= 3 || warp % wpb == 0)) {
                if (l + 1 < kTrLevels) rg[l & 1][b] = own;
                else ranges[b] = own;
                work += (unsigned)TL.n * kTrNodes;
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nb * NC * kTrNodes; i += kFwWarps * 32) {
            const int j = i % kTrNodes, c = (i / kTrNodes) % NC, b = i / (kTrNodes * NC);
            if ((c && !LM) || sb + (long long)b * (kTrStrip >> l) >= n_nu) continue;
            double v = 0.0;
            for (int w = 0; w < wpb; ++w) v += (double)part[b * wpb + w][c][j];
            if (l) {
                const double* fp = F[(l + 1) & 1][b >> 1][c];
#pragma unroll
                for (int k = 0; k < kTrNodes; ++k) v = fma(fp[k], tab->M[b & 1][k][j], v);
            }
            if (l + 1 < kTrLevels) F[l & 1][b][c][j] = v;
            else far[(b * NC + c) * kTrNodes + j] = (float)v;
        }
        __syncthreads();
    }
    if (evald && lane == 0 && work) atomicAdd(evald, (unsigned long long)work);
}

template <bool ANY_LM>
__global__ void __launch_bounds__(kFwWarps * 32, 5) fw_tree_kernel(
    const SegDev* __restrict__ segs, const unsigned* __restrict__ core_reach, CellIndex ci, LpOutMixed lp, float cut_g,
    long long n_nu, int n_leaves, const TreeTables* __restrict__ tab, float* __restrict__ far, int4* __restrict__ ranges,
    int seg0, unsigned long long* __restrict__ evald) {
    const int s = seg0 + (int)blockIdx.y;
    const SegDev sg = segs[s];
    const size_t cell = (size_t)blockIdx.y * n_leaves + (size_t)blockIdx.x * kTrLeaves;
    float* fo = far + cell * fw_sums(ANY_LM) * kTrNodes;
    const int* row = ci.idx + (size_t)s * ci.n;
    const float m = (float)sg.margin_g, reach = __uint_as_float(core_reach[s]);
    if (ANY_LM && (sg.flags & SEG_LM))  // block-uniform
        fw_tree_segment<ANY_LM, ANY_LM>(lp, sg.off, ci, row, cut_g, m, reach, n_nu, tab, fo, ranges + cell, evald);
    else
        fw_tree_segment<ANY_LM, false>(lp, sg.off, ci, row, cut_g, m, reach, n_nu, tab, fo, ranges + cell, evald);
}

// one warp per (strip, segment)
constexpr int kFwTreeWarps = 4;
template <bool ANY_LM>
__global__ void __launch_bounds__(kFwTreeWarps * 32, ANY_LM ? 6 : 10) fw_tree_warp_kernel(
    const SegDev* __restrict__ segs, const unsigned* __restrict__ core_reach, CellIndex ci, LpOutMixed lp, float cut_g,
    long long n_nu, int n_leaves, const TreeTables* __restrict__ tab, float* __restrict__ far, int4* __restrict__ ranges,
    int seg0, unsigned long long* __restrict__ evald) {
    __shared__ float4 tiles[kFwTreeWarps][32];
    __shared__ float tiles_g[ANY_LM ? kFwTreeWarps : 1][32];
    __shared__ double F[kFwTreeWarps][kTrLeaves / 2][fw_sums(ANY_LM)][kTrNodes];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int strip = (int)blockIdx.x * kFwTreeWarps + warp, s = seg0 + (int)blockIdx.y;
    const long long sb = (long long)strip * kTrStrip;
    if (sb >= n_nu) return;
    const SegDev sg = segs[s];
    const size_t cell = (size_t)blockIdx.y * n_leaves + (size_t)strip * kTrLeaves;
    float* fo = far + cell * fw_sums(ANY_LM) * kTrNodes;
    const int* row = ci.idx + (size_t)s * ci.n;
    const float m = (float)sg.margin_g, reach = __uint_as_float(core_reach[s]);
    unsigned work = 0;
    if (ANY_LM && (sg.flags & SEG_LM))
        fw_tree_warp<ANY_LM, ANY_LM>(lp, sg.off, ci, row, sb, cut_g, m, reach, n_nu, tab, fo, ranges + cell, lane, tiles[warp],
                                     tiles_g[ANY_LM ? warp : 0], F[warp], work);
    else
        fw_tree_warp<ANY_LM, false>(lp, sg.off, ci, row, sb, cut_g, m, reach, n_nu, tab, fo, ranges + cell, lane, tiles[warp],
                                    tiles_g[ANY_LM ? warp : 0], F[warp], work);
    if (evald && lane == 0 && work) atomicAdd(evald, (unsigned long long)work);
}

// ------------------------------------------------------------------ near lines
// The core's quotient in units of s = 2^-14 (m s, q s^2, n s^2, K s: the same roundings), so that m^3
// of two points is in range up to |x| = 1.8e5 instead of 1.4e3
constexpr float kFwScale = 6.103515625e-05f;
constexpr int kFwBuf = 160;  // 512 (1.1 KB more a warp) measured slower, 61.1 against 60.0 ms on the IASI case
template <bool LM>
struct FwTile {
    float4 fu[32];   // uh, ul, b2, a
    float4 p0[32];   // edge: c1, c0, g, -; core: s fx^2, s y^2, s K (K = a fx^2), dfar^2; general: c1, c0, dfar^2, An
    float4 p1[32];   // core, general: fx, y, An, Yw
    float fg[LM ? 32 : 1];
    int4 cr[32];     // core: inner points [x, y], offset in cw (-1: not held), rows lo | hi << 8
    float cw[kFwBuf];
    float cwi[LM ? kFwBuf : 1];
};

template <int METHOD, bool LM>
__device__ __forceinline__ void fw_segment(const SegDev& sg, const LpOutMixed& lp, long long wb, int4 own, int wlo,
                                           int whi, float cut, float x_far2, int lane, FwTile<LM>& T,
                                           const float (*__restrict__ Lw)[kTrLeaf], const float* __restrict__ gfar,
                                           unsigned& work, float sig[4]) {
    constexpr float kCentre = 0.5f * (kTrLeaf - 1);
    constexpr float kHalf = 0.5f * kTrLeaf + 0.5f;
    const float cut2 = cut * cut, pl0 = (float)lane;
    const unsigned lt = (1u << lane) - 1u;
    float2 S[2], C[2], SD[2], CD[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) S[h] = C[h] = SD[h] = CD[h] = make_float2(0.f, 0.f);
    float PA = 0.f, PAc = 0.f, PB = 0.f, PBc = 0.f, PC = 0.f, PCc = 0.f;
    // the lines not taken by the far field: [wlo, own.x), [own.y, own.z), [own.w, whi)
    const int n1 = max(own.x - wlo, 0), n2 = n1 + (own.z - own.y), n = n2 + max(whi - own.w, 0);
    for (int t0 = 0; t0 < n; t0 += 32) {
        const int nt = min(32, n - t0), t = t0 + lane;
        int cls = 0;
        float uh = 0.f, ul = 0.f, df = 0.f;
        float4 a0, a1;
        float2 a2 = make_float2(0.f, 0.f);
        if (lane < nt) {
            const long long q = sg.off + (t < n1 ? wlo + t : t < n2 ? own.y + (t - n1) : own.w + (t - n2));
            const float2 uf = lp.U[q];
            uh = uf.x - (float)wb;  // exact: see split_hi_lo
            ul = uf.y;
            df = lp.df[q];
            const float dist = fabsf(uh - kCentre);
            const bool wing = dist > df + kHalf, in = dist + kHalf <= cut;
            cls = dist > cut + kHalf ? 0 : wing ? (in ? 1 : 2) : (in && cut >= 8.f * (df + 0.5f) ? 3 : 4);
            if (cls) {
                a0 = lp.p0[q];
                if (cls >= 3) a1 = lp.p1[q];
                if (LM) a2 = lp.p2[q];
                // the quotient's (m s)^3 for two points stays in range
                if (cls == 3 && (METHOD != 3 || x_far2 + a1.w * a1.w > 2.0e6f / kFwScale)) cls = 4;
            }
        }
        const unsigned m1 = __ballot_sync(kFull, cls == 1), m2 = __ballot_sync(kFull, cls == 2);
        const unsigned m3 = __ballot_sync(kFull, cls == 3), m4 = __ballot_sync(kFull, cls == 4);
        const int e1 = __popc(m1), e2 = e1 + __popc(m2), e3 = e2 + __popc(m3), e4 = e3 + __popc(m4);
        // inner points of the core lines (one to spare on each side), held in cw when they are
        // few (a wide zone fills its rows and is evaluated there)
        int nin = 0, plo = 1, coff = 0, cfit = 0;
        if (METHOD == 3 && m3) {  // warp-uniform
            if (cls == 3 && a1.w < 15.f) {
                const float hw = (15.f - a1.w) / a1.z + 1.f, c = uh + ul;
                const float lo = fmaxf(c - hw, 0.f), hi = fminf(c + hw, (float)(kTrLeaf - 1));
                if (lo <= hi) {
                    plo = (int)ceilf(lo);
                    nin = max((int)floorf(hi) - plo + 1, 0);
                }
            }
            int inc = nin <= 32 ? nin : 0;
            const int own_n = inc;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(kFull, inc, d);
                if (lane >= d) inc += v;
            }
            coff = inc - own_n;
            const unsigned ov = __ballot_sync(kFull, inc > kFwBuf && own_n > 0);
            cfit = ov ? __shfl_sync(kFull, coff, __ffs(ov) - 1) : __shfl_sync(kFull, inc, 31);
            if (own_n == 0 || inc > kFwBuf) coff = -1 - coff;  // not held (the offsets stay monotone)
        }
        __syncwarp();
        if (cls) {
            const int pos = cls == 1 ? __popc(m1 & lt) : cls == 2 ? e1 + __popc(m2 & lt)
                          : cls == 3 ? e2 + __popc(m3 & lt) : e3 + __popc(m4 & lt);
            T.fu[pos] = make_float4(uh, ul, a0.x, a0.y);
            if (LM) T.fg[pos] = a2.x;
            if (cls & 1) {  // pedestal: sum over points p of c1 (p - u)^2 + c0
                const float u = uh + ul, pb = a0.z * u;
                kahan_add(PA, PAc, a0.z);
                kahan_add(PB, PBc, pb);
                kahan_add(PC, PCc, fmaf(pb, u, a0.w));
            }
            if (cls == 2) T.p0[pos] = make_float4(a0.z, a0.w, 0.f, 0.f);
            else if (cls == 3) {
                const float fx2 = a1.z * a1.z;
                T.p0[pos] = make_float4(kFwScale * fx2, kFwScale * (a1.w * a1.w), kFwScale * (a1.y * a1.w * (float)kInvSqrtPi),
                                        df * df);
                T.p1[pos] = make_float4(a1.z, a1.w, a1.y, a2.y);
                const float c = uh + ul;
                const int rl = (int)fminf(fmaxf((c - df) * (1.f / 32.f) - 0.1f, 0.f), 4.f);  // rows the core reaches
                const int rh = (int)fminf(fmaxf((c + df) * (1.f / 32.f) + 0.1f, -1.f), 3.f);
                T.cr[pos] = make_int4(plo, plo + nin - 1, coff, rl | (rh << 8));
            } else if (cls == 4) {
                T.p0[pos] = make_float4(a0.z, a0.w, a1.x, a1.y);
                T.p1[pos] = make_float4(a1.z, a1.w, a1.y, a2.y);
            }
        }
        __syncwarp();
        if (e4 == 0) continue;
        work += (unsigned)e4 * kTrLeaf;
        if (cfit > 0) {
            for (int e = lane; e < cfit; e += 32) {  // the held line owning element e: the last with offset <= e
                int lo = e2, hi = e3 - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    const int z = T.cr[mid].z;  // lines not held own no elements: their offset is the next one's
                    if ((z < 0 ? -1 - z : z) <= e) lo = mid; else hi = mid - 1;
                }
                const int4 r = T.cr[lo];
                const float4 u = T.fu[lo], p = T.p1[lo];
                const float d = ((float)(r.x + (e - r.z)) - u.x) - u.y;
                const float2 w = faddeeva32_inline(d * p.x, p.y);
                T.cw[e] = w.x;
                if (LM) T.cwi[e] = w.y;
            }
            __syncwarp();
        }
        float2 acc[2], dsp[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) acc[h] = dsp[h] = make_float2(0.f, 0.f);
        for (int k = 0; k < e1; ++k) {
            const float4 f = T.fu[k];
            const float d0 = (pl0 - f.x) - f.y, g = LM ? T.fg[k] : 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 ds = __fadd2_rn(make_float2(d0, d0), make_float2(64.f * h + 32.f, 64.f * h));  // swapped
                const float2 es = __ffma2_rn(ds, ds, make_float2(f.z, f.z));
                const float R = rcp_fast(es.x * es.y);
                const float2 r = __fmul2_rn(es, make_float2(R, R));
                acc[h] = __ffma2_rn(make_float2(f.w, f.w), r, acc[h]);
                if (LM) dsp[h] = __ffma2_rn(__fmul2_rn(make_float2(g, g), make_float2(ds.y, ds.x)), r, dsp[h]);
            }
        }
        for (int k = e1; k < e2; ++k) {  // cutoff-edge lines
            const float4 f = T.fu[k], p = T.p0[k];
            const float d0 = (pl0 - f.x) - f.y, g = LM ? T.fg[k] : 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 ds = __fadd2_rn(make_float2(d0, d0), make_float2(64.f * h + 32.f, 64.f * h));
                const float2 es = __ffma2_rn(ds, ds, make_float2(f.z, f.z));
                const float R = rcp_fast(es.x * es.y);
                const float2 r = __fmul2_rn(es, make_float2(R, R));
                const float2 dn = make_float2(ds.y, ds.x), d2 = __fmul2_rn(dn, dn);
                const float2 v = __ffma2_rn(make_float2(f.w, f.w), r, __ffma2_rn(make_float2(p.x, p.x), d2, make_float2(p.y, p.y)));
                const bool ix = d2.x <= cut2, iy = d2.y <= cut2;
                acc[h].x += ix ? v.x : 0.f;
                acc[h].y += iy ? v.y : 0.f;
                if (LM) {
                    const float2 vd = __fmul2_rn(__fmul2_rn(make_float2(g, g), dn), r);
                    dsp[h].x += ix ? vd.x : 0.f;
                    dsp[h].y += iy ? vd.y : 0.f;
                }
            }
        }
        if (METHOD == 3) {
            for (int k = e2; k < e3; ++k) {  // core lines
                const float4 f = T.fu[k], p = T.p0[k], p1 = T.p1[k];
                const int4 cr = T.cr[k];
                const int rl = cr.w & 255, rh = cr.w >> 8;  // rh = -1: none (arithmetic shift)
                const float g = LM ? T.fg[k] : 0.f;
                constexpr float s1 = kFwScale, s2 = kFwScale * kFwScale;  // X, m times s; n, q times s^2
                const float c1 = fmaf(2.5f * s1, p.y, 1.5f * s2), c2 = fmaf(3.f * s1, p.y, 2.25f * s2);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // from each point's own position: the first subtraction is exact, and the second
                    // rounds at the size of d (an offset from the lane's first point would round at
                    // up to 128 steps: 2e-5 of the value half a step from a centre)
                    const float2 dn = __fadd2_rn(__fadd2_rn(make_float2(pl0 + 64.f * h, pl0 + 64.f * h + 32.f), make_float2(-f.x, -f.x)),
                                                 make_float2(-f.y, -f.y));
                    if (rh < 2 * h || rl > 2 * h + 1) {  // warp-uniform: no core point in these rows
                        const float2 ds = make_float2(dn.y, dn.x);
                        const float2 es = __ffma2_rn(ds, ds, make_float2(f.z, f.z));
                        const float R = rcp_fast(es.x * es.y);
                        const float2 r = __fmul2_rn(es, make_float2(R, R));
                        acc[h] = __ffma2_rn(make_float2(f.w, f.w), r, acc[h]);
                        if (LM) dsp[h] = __ffma2_rn(__fmul2_rn(make_float2(g, g), dn), r, dsp[h]);
                        continue;
                    }
                    const float2 d2 = __fmul2_rn(dn, dn);
                    const float2 X = __fmul2_rn(d2, make_float2(p.x, p.x));
                    const float2 m = __fadd2_rn(X, make_float2(p.y, p.y));
                    float2 nn = __ffma2_rn(m, m, __ffma2_rn(X, make_float2(-1.5f * s1, -1.5f * s1), make_float2(c1, c1)));
                    float2 q = __ffma2_rn(m, m, __ffma2_rn(X, make_float2(-3.f * s1, -3.f * s1), make_float2(c2, c2)));
                    const bool cx = d2.x <= p.w, cy = d2.y <= p.w;
                    nn.x = cx ? nn.x : 1.f;
                    nn.y = cy ? nn.y : 1.f;
                    q.x = cx ? q.x : 1.f;
                    q.y = cy ? q.y : 1.f;
                    // m q is zero where y is lost beside x = 0 or x^2 = 3/2: points that the buffer
                    // replaces below, but the reciprocal is their neighbours' too.  Any other
                    // point's is far above the floor (3e-7 at |x| + y = 15)
                    float2 den = __fmul2_rn(m, q);
                    den.x = fmaxf(den.x, 1e-18f);
                    den.y = fmaxf(den.y, 1e-18f);
                    const float R = rcp_fast(den.x * den.y);
                    const float2 r = __fmul2_rn(make_float2(den.y, den.x), make_float2(R, R));
                    float2 v = __fmul2_rn(__fmul2_rn(nn, make_float2(p.z, p.z)), r), vd = make_float2(0.f, 0.f);
                    if (LM) {  // Im w = (x/sqrt(pi)) (m^2 - 5/2 x^2 + 3/2 y^2 + 3/2) / (m q); wing: x / (sqrt(pi) m)
                        const float c3 = fmaf(1.5f * s1, p.y, 1.5f * s2), kd = s1 * (p1.w * (float)kInvSqrtPi * p1.x);
                        float2 ni = __ffma2_rn(m, m, __ffma2_rn(X, make_float2(-2.5f * s1, -2.5f * s1), make_float2(c3, c3)));
                        ni.x = cx ? ni.x : 1.f;
                        ni.y = cy ? ni.y : 1.f;
                        vd = __fmul2_rn(__fmul2_rn(__fmul2_rn(ni, make_float2(kd, kd)), dn), r);
                    }
                    if (cr.y >= 64 * h && cr.x < 64 * h + 64 && cr.y >= cr.x) {  // warp-uniform: inner points in these rows
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const float d = s ? dn.y : dn.x, x = d * p1.x;
                            const int pt = lane + 32 * (2 * h + s);
                            const bool core = s ? cy : cx;
                            if (!(core && fabsf(x) + p1.y < 15.f)) continue;
                            float2 w;
                            if (cr.z >= 0 && pt >= cr.x && pt <= cr.y) {
                                w.x = T.cw[cr.z + pt - cr.x];
                                if (LM) w.y = T.cwi[cr.z + pt - cr.x];
                            } else {
                                w = faddeeva32(x, p1.y);
                            }
                            if (s) {
                                v.y = p1.z * w.x;
                                if (LM) vd.y = p1.w * w.y;
                            } else {
                                v.x = p1.z * w.x;
                                if (LM) vd.x = p1.w * w.y;
                            }
                        }
                    }
                    acc[h] = __fadd2_rn(acc[h], v);
                    if (LM) dsp[h] = __fadd2_rn(dsp[h], vd);
                }
            }
        }
        for (int k = e3; k < e4; ++k) {  // general lines
            const float4 f = T.fu[k], p = T.p0[k], p1 = T.p1[k];
            const float g = LM ? T.fg[k] : 0.f, y2 = p1.y * p1.y;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float d = ((pl0 + 32.f * q) - f.x) - f.y, d2 = d * d;
                const float ped = fmaf(p.x, d2, p.y);
                const bool core = d2 <= p.z;  // |x| <= x_far
                float v, vd = 0.f;
                if (METHOD == 3) {
                    // the wing at every lane; rows holding a core point (warp-uniform) the two-level
                    // continued fraction too, the points nearer through the shared routine
                    const float r = rcp_fast(d2 + f.z);
                    v = fmaf(f.w, r, ped);
                    if (LM) vd = g * d * r;
                    if (__any_sync(kFull, core)) {
                        const float x = d * p1.x;
                        float2 w = faddeeva_cf2(x, p1.y, y2);
                        if (core && fabsf(x) + p1.y < 15.f) w = faddeeva32(x, p1.y);
                        if (core) {
                            v = fmaf(p.w, w.x, ped);
                            if (LM) vd = p1.w * w.y;
                        }
                    }
                    if (d2 > cut2) v = vd = 0.f;
                } else {
                    if (d2 > cut2) continue;
                    v = core ? fmaf(p.w, weideman24_32(d * p1.x, p1.y), ped) : fmaf(f.w, rcp_fast(d2 + f.z), ped);
                }
                if (q & 1) {
                    acc[q >> 1].y += v;
                    if (LM) dsp[q >> 1].y += vd;
                } else {
                    acc[q >> 1].x += v;
                    if (LM) dsp[q >> 1].x += vd;
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // tile sums into the compensated sums
            kahan_add(S[h].x, C[h].x, acc[h].x);
            kahan_add(S[h].y, C[h].y, acc[h].y);
            if (LM) {
                kahan_add(SD[h].x, CD[h].x, dsp[h].x);
                kahan_add(SD[h].y, CD[h].y, dsp[h].y);
            }
        }
    }
    // pedestals, and the far field's interpolant about the value of a middle node (so that the
    // weights' rounding acts on its variation over the leaf only)
    const float A = warp_sum(PA - PAc), B = warp_sum(PB - PBc), Cq = warp_sum(PC - PCc);
    float2 it[2], id[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float x0 = pl0 + 64.f * h, x1 = x0 + 32.f;
        it[h] = make_float2(fmaf(x0, fmaf(x0, A, -2.f * B), Cq), fmaf(x1, fmaf(x1, A, -2.f * B), Cq));
        id[h] = make_float2(0.f, 0.f);
    }
    if (gfar) {
        float nd = gfar[lane & (kTrNodes - 1)], dd = LM ? gfar[kTrNodes + (lane & (kTrNodes - 1))] : 0.f;
        const float mid = __shfl_sync(kFull, nd, kTrNodes / 2);
        nd -= mid;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            kahan_add(S[h].x, C[h].x, mid);
            kahan_add(S[h].y, C[h].y, mid);
        }
#pragma unroll
        for (int k = 0; k < kTrNodes; ++k) {
            const float F = __shfl_sync(kFull, nd, k), FD = LM ? __shfl_sync(kFull, dd, k) : 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 w = make_float2(Lw[k][64 * h + lane], Lw[k][64 * h + 32 + lane]);
                it[h] = __ffma2_rn(make_float2(F, F), w, it[h]);
                if (LM) id[h] = __ffma2_rn(make_float2(FD, FD), w, id[h]);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        kahan_add(S[h].x, C[h].x, it[h].x);
        kahan_add(S[h].y, C[h].y, it[h].y);
        sig[2 * h] = fmaxf(S[h].x, 0.f);
        sig[2 * h + 1] = fmaxf(S[h].y, 0.f);
        if (LM) {
            kahan_add(SD[h].x, CD[h].x, id[h].x);
            kahan_add(SD[h].y, CD[h].y, id[h].y);
            sig[2 * h] = fmaxf(sig[2 * h] + SD[h].x, 0.f);
            sig[2 * h + 1] = fmaxf(sig[2 * h + 1] + SD[h].y, 0.f);
        }
    }
}

// The segments with (LM) or without line mixing, one launch each: the first stores the optical
// depths, the second adds its own (one kernel for both ran out of instruction cache).
// PERT: segments flagged SEG_RELMAT write their clamped sums to pert[(profile, layer)][pstride]
// for relmat_finish_kernel.
template <int METHOD, bool LM>
__global__ void __launch_bounds__(kFwWarps * 32, LM ? 3 : 4) fw_leaf_kernel(
    const SegDev* __restrict__ segs, const int2* __restrict__ pl_segs, CellIndex ci, LpOutMixed lp, long long n_nu,
    float cut_g, float x_far, int store, int far_sums, float* __restrict__ tau, double* __restrict__ pert,
    long long pstride, const TreeTables* __restrict__ tab, const float* __restrict__ far, const int4* __restrict__ ranges,
    int n_leaves, int pl0, int seg0, unsigned long long* __restrict__ evald) {
    __shared__ float Lw[kTrNodes][kTrLeaf];
    __shared__ FwTile<LM> tiles[kFwWarps];
    for (int i = threadIdx.x; i < kTrNodes * kTrLeaf; i += kFwWarps * 32) (&Lw[0][0])[i] = ((const float*)tab->L)[i];
    __syncthreads();  // the only block-wide barrier: before any warp leaves
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pl = pl0 + (int)blockIdx.y, leaf = (int)blockIdx.x * kFwWarps + warp;
    const long long wb = (long long)leaf * kTrLeaf;
    if (wb >= n_nu) return;
    float tsum[4] = {0.f, 0.f, 0.f, 0.f};
    unsigned work = 0;
    bool any = false;
    const int2 rng = pl_segs[pl];
    for (int s = rng.x; s < rng.x + rng.y; ++s) {
        const SegDev sg = segs[s];
        if (((sg.flags & SEG_LM) != 0) != LM) continue;
        const int* row = ci.idx + (size_t)s * ci.n;
        const float m = (float)sg.margin_g;
        const int wlo = cell_floor(ci, row, (float)wb - cut_g - m);
        const int whi = cell_ceil(ci, row, (float)(wb + kTrLeaf) + cut_g + m);
        int4 own = make_int4(wlo, wlo, whi, whi);  // no far field: every line direct
        const float* gf = nullptr;
        if (far) {
            const size_t cell = (size_t)(s - seg0) * n_leaves + leaf;
            own = ranges[cell];
            gf = far + cell * far_sums * kTrNodes;
        }
        float sig[4];
        fw_segment<METHOD, LM>(sg, lp, wb, own, wlo, whi, cut_g, x_far * x_far, lane, tiles[warp], Lw, gf, work, sig);
        any = true;
        const bool rel = pert && (sg.flags & SEG_RELMAT);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (rel) pert[(size_t)pl * pstride + wb + 32 * q + lane] = (double)sig[q];
            else tsum[q] += sig[q];
        }
        __syncwarp();
    }
    float* out = tau + (size_t)pl * n_nu + wb;
    if (store || any) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = 32 * q + lane;
            if (wb + i < n_nu) out[i] = store ? tsum[q] : out[i] + tsum[q];
        }
    }
    if (evald && lane == 0 && work) atomicAdd(evald, (unsigned long long)work);
}

}  // namespace irs
