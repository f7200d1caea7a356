// linesum_tree64.cuh -- the FP64 line sum on a uniform grid, with the wings of distant
// lines summed through Chebyshev interpolation.
//
// The same sum as linesum_f64_kernel (linesum.cuh; src/CrossSections/voigt.jl:243-313,
// line_mixing.jl:1166-1186) over the same lines and per-point windows, all in FP64.  A
// line far from a block of points is a smooth function there (its Lorentz wing has its
// poles at |nu - nu0| from the block's centre), so the far lines of a block are
// evaluated at 32 Chebyshev nodes of the block instead of at its points and
// interpolated.  With the nodes of a block of half-width h and lines from 1.85 h of its
// centre, the interpolation error of one line's term is below 6e-16 of its largest value
// on the block (checked with 40-digit arithmetic), i.e. the rounding of the direct sum.
// Three levels of blocks, each a quarter of the one above (strip, group, leaf = one
// warp's points): a line is summed at the widest block that it is far from, and a
// block's node values are carried to its four quarters by fixed 32 x 32 matrices.  What
// is left to a leaf's points one by one are the lines within 1.85 half-widths (or
// within the Faddeeva core's reach, |x| <= x_far, of the leaf) and the lines whose
// cutoff falls among its points.
//
// Pedestals are quadratics in nu: summed exactly as three moments per block.
//
// What bounds it: on the 5,000-line list the leaf kernel uses 37 % of the FP64 pipe and 35 % of
// the issue slots; it waits for instructions (the branches of w(z) against the instruction cache)
// and on dependent operations, at 14 warps per SM.  Per 128-point leaf and segment of the 5,000-line CO2
// list at 0.0025 cm^-1 (4,545 lines in the cutoff) about 190 evaluations per point take
// the place of 4,545; most of what remains are the core rows.
// Measured on a B200 against linesum_f64_kernel (one thread per point, every line of its
// window): 5,000 CO2 lines x 34,801 points x 49 layers 10.65 -> 0.67 ms (far 0.09, leaf
// 0.58), 66,667 lines x 846,001 points 3.89 -> 0.27 ms, 5,000 lines x 5,501 points 1.17 ->
// 0.077 ms, 9,000 lines of three species in 1210-1290 cm^-1 x 44,801 points x 49 layers
// 17.5 -> 1.82 ms.  Error against 64-bit torch on the two cross sections: 1.7e-15 / 3.2e-15 of
// the spectrum's norm before, 6.2e-16 / 5.7e-16 after.
#pragma once
#include "linesum.cuh"
#include "rte_ils.cuh"  // rcp64_fast

namespace irs {

constexpr int kT64Nodes = 32;
constexpr double kT64Ratio = 1.85;  // far: |nu0 - c| >= 1.85 h
constexpr int kT64Warps = 8;        // warps of tree64_far_kernel
constexpr int kT64LeafWarps = 4;    // leaves (warps) per CTA of tree64_leaf_kernel: one group

// node positions, the quarter-block matrices and the leaf interpolation weights, built on
// the host in extended precision (t64_tables, irs_host.cpp)
struct T64Tables {
    double x[kT64Nodes];                        // nodes on [-1, 1]
    double M[4][kT64Nodes][kT64Nodes];          // [quarter][k][j]: L_k at node j of the quarter
    double L4[kT64Nodes][128], L1[kT64Nodes][32];  // [k][i]: L_k at point i of a 128- / 32-point leaf
};

// four reciprocals from one (Montgomery's trick); products of the far-wing denominators
// (between about 1e-4 and 1e3 cm^-2 squared) stay normal
__device__ __forceinline__ void rcp64_quad(const double e[4], double r[4]) {
    const double p01 = e[0] * e[1], p23 = e[2] * e[3];
    const double R = rcp64_fast(p01 * p23);
    const double r01 = R * p23, r23 = R * p01;
    r[0] = r01 * e[1];
    r[1] = r01 * e[0];
    r[2] = r23 * e[3];
    r[3] = r23 * e[2];
}

// The far lines of a block [c - h, c + h] as index ranges [x, y) and [z, w): shifted centre
// in [c + h - cut + m, c - R) and [c + R, c - h + cut - m), R the far distance including
// the core's reach, m covering the disorder of the shifted centres (the array is sorted by
// the unshifted ones).  Empty ranges (x == y, z == w) at the centre when there are none.
__device__ __forceinline__ double t64_bound(int b, double c, double h, double cut, double m, double reach) {
    const double R = fmax(kT64Ratio * h, reach + h) + m;
    if (!(cut - h - m > R)) return c;
    return b == 0 ? c + h - cut + m : b == 1 ? c - R : b == 2 ? c + R : c - h + cut - m;
}
__device__ __forceinline__ int4 t64_order(int a, int b, int c, int d) {
    b = max(a, b);
    c = max(b, c);
    return make_int4(a, b, c, max(c, d));
}
// a block inside one whose ranges are `up`: its own contain them (up empty: unchanged)
__device__ __forceinline__ int4 t64_inside(int4 s, int4 up) {
    if (up.y > up.x) { s.x = min(s.x, up.x); s.y = max(s.y, up.y); }
    if (up.w > up.z) { s.z = min(s.z, up.z); s.w = max(s.w, up.w); }
    return t64_order(s.x, s.y, s.z, s.w);
}
// margin of a segment: four times the largest pressure shift (twice it bounds the disorder
// at either end of a range), and grid steps to spare
__device__ __forceinline__ double t64_margin(const SegDev& sg, double dnu) { return 4.0 * sg.margin_g * dnu; }

struct T64Tile {
    double2 ub[kT64Nodes], ag[kT64Nodes];  // (u, b^2), (a, g): a/(d^2 + b^2), g d/(d^2 + b^2)
};

// A block's centre is held as its strip's centre cs plus an offset o: cs + o rounded to one
// double is an ulp of nu off (1e-13 cm^-1), which is 1e-12 of the distances within a strip
// of 0.0002 cm^-1 steps and would show at every level, since the quarters' matrices hold
// for the exact geometry.

// One warp: the far lines [j0, j1) of the block at cs + o, lane k at node t (relative to it),
// tiles first, first + step, ...  A tile's lines are staged once (coalesced) and read as
// broadcasts, four at a time with one reciprocal.  mom: the lane's own lines' pedestal
// moments sum P, P u, P u^2 (P = Sn Hc, u = nu0 - centre).
template <bool LM>
__device__ __forceinline__ void t64_nodes(const LpOutF64& lp, long long off, int j0, int j1, int first, int step,
                                          double cs, double o, double t, int lane, T64Tile& T, double& acc,
                                          double& accD, double mom[3]) {
    for (int k0 = j0 + 32 * first; k0 < j1; k0 += 32 * step) {
        __syncwarp();
        double u = 0.0, b = 1.0, k = 0.0, g = 0.0;
        if (k0 + lane < j1) {
            const long long q = off + k0 + lane;
            u = (lp.nu0[q] - cs) - o;
            b = lp.b[q];
            k = lp.k0[q];
            if (LM) g = lp.g[q];
            const double P = lp.Sn[q] * lp.Hc[q];
            mom[0] += P;
            mom[1] = fma(P, u, mom[1]);
            mom[2] = fma(P * u, u, mom[2]);
        }
        T.ub[lane] = make_double2(u, b * b);
        T.ag[lane] = make_double2(k * b, g);
        __syncwarp();
        const int n = min(32, j1 - k0);
        for (int i = 0; i < n; i += 4) {  // lines beyond n: a = g = 0, b^2 = 1
            double d[4], e[4], r[4], a[4], gg[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const double2 ub = T.ub[i + v], ag = T.ag[i + v];
                d[v] = t - ub.x;
                e[v] = fma(d[v], d[v], ub.y);
                a[v] = ag.x;
                gg[v] = ag.y;
            }
            rcp64_quad(e, r);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                acc = fma(a[v], r[v], acc);
                if (LM) accD = fma(gg[v] * d[v], r[v], accD);
            }
        }
    }
}
// [a, b) without [p, q): the two pieces [a, min(b, p)) and [max(a, q), b)
template <bool LM>
__device__ __forceinline__ void t64_nodes_except(const LpOutF64& lp, long long off, int a, int b, int p, int q,
                                                 int first, int step, double cs, double o, double t, int lane,
                                                 T64Tile& T, double& acc, double& accD, double mom[3]) {
    if (p >= q) { p = b; q = b; }
    t64_nodes<LM>(lp, off, a, min(b, p), first, step, cs, o, t, lane, T, acc, accD, mom);
    t64_nodes<LM>(lp, off, max(a, q), b, first, step, cs, o, t, lane, T, acc, accD, mom);
}

__device__ __forceinline__ double warp_sum64(double v) {
#pragma unroll
    for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
    return v;
}

// One CTA per (strip of 16 leaves, segment): the strip's far lines at its nodes, shared by
// the warps; then two warps per group (4 leaves): the strip's node values at the group's
// nodes plus the group's own far lines.  far[cell][k] (and farD with line mixing) with
// cell = (segment, group), pedestals of the lines taken so far included, and the group's
// ranges.  Split over (strip, segment) and over the warps because the strips are few:
// 17 strips for the 34,801 points of the 5,000-line list.
template <bool ANY_LM>
__global__ void __launch_bounds__(32 * kT64Warps, 3) tree64_far_kernel(
    const SegDev* __restrict__ segs, const int* __restrict__ seg_count, const unsigned* __restrict__ core_reach,
    LpOutF64 lp, double g0, double dnu, double cutoff, int leaf_pts, const T64Tables* __restrict__ tab,
    double* __restrict__ far, double* __restrict__ farD, int4* __restrict__ ranges, int seg0,
    const int* __restrict__ uniform, unsigned long long* __restrict__ evald) {
    if (uniform && !*uniform) return;
    __shared__ T64Tile tiles[kT64Warps];
    __shared__ double part[kT64Warps][kT64Nodes], partD[ANY_LM ? kT64Warps : 1][kT64Nodes], pm[kT64Warps][3];
    __shared__ double F[kT64Nodes], FD[ANY_LM ? kT64Nodes : 1];
    __shared__ int sj[5][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int strip = blockIdx.x, s = seg0 + (int)blockIdx.y, n_groups = 4 * gridDim.x;
    const SegDev sg = segs[s];
    const bool lm = ANY_LM && (sg.flags & SEG_LM);
    const long long cnt = seg_count[s];
    const double reach = (double)__uint_as_float(core_reach[s]), m = t64_margin(sg, dnu), rc2 = 1.0 / (cutoff * cutoff);
    const double hs = 8.0 * leaf_pts * dnu, hg = 2.0 * leaf_pts * dnu;  // half-widths
    const double cs = g0 + dnu * ((double)strip * 16 * leaf_pts + 8.0 * leaf_pts - 0.5);
    for (int i = warp; i < 20; i += kT64Warps) {  // 4 bounds of the strip and of each group
        const int blk = i / 4;
        const double c = blk ? cs + (2 * blk - 5) * hg : cs, h = blk ? hg : hs;
        const int j = (int)warp_lower_bound(lp.nu0 + sg.off, t64_bound(i % 4, c, h, cutoff, m, reach), cnt, lane);
        if (lane == 0) sj[blk][i % 4] = j;
    }
    __syncthreads();
    const int4 S = t64_order(sj[0][0], sj[0][1], sj[0][2], sj[0][3]);
    const double xk = tab->x[lane];
    double acc = 0.0, accD = 0.0, mom[3] = {0.0, 0.0, 0.0};
    if (lm) {
        t64_nodes<true>(lp, sg.off, S.x, S.y, warp, kT64Warps, cs, 0.0, hs * xk, lane, tiles[warp], acc, accD, mom);
        t64_nodes<true>(lp, sg.off, S.z, S.w, warp, kT64Warps, cs, 0.0, hs * xk, lane, tiles[warp], acc, accD, mom);
    } else {
        t64_nodes<false>(lp, sg.off, S.x, S.y, warp, kT64Warps, cs, 0.0, hs * xk, lane, tiles[warp], acc, accD, mom);
        t64_nodes<false>(lp, sg.off, S.z, S.w, warp, kT64Warps, cs, 0.0, hs * xk, lane, tiles[warp], acc, accD, mom);
    }
    part[warp][lane] = acc;
    if (lm) partD[warp][lane] = accD;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double v = warp_sum64(mom[i]);
        if (lane == 0) pm[warp][i] = v;
    }
    __syncthreads();
    if (warp == 0) {
        double v = 0.0, A = 0.0, B = 0.0, C = 0.0, vD = 0.0;
        for (int w = 0; w < kT64Warps; ++w) {
            v += part[w][lane];
            A += pm[w][0];
            B += pm[w][1];
            C += pm[w][2];
            if (lm) vD += partD[w][lane];
        }
        const double t = hs * xk;  // pedestals: sum P (2 - (t - u)^2 / cut^2)
        F[lane] = v - (2.0 * A - rc2 * fma(t, fma(t, A, -2.0 * B), C));
        if (ANY_LM) FD[lane] = vD;
    }
    __syncthreads();
    // two warps per group: even lists of tiles and odd ones
    const int grp = warp >> 1, half = warp & 1;
    const double og = (2 * grp - 3) * hg, tg = hg * xk;
    const int4 G = t64_inside(t64_order(sj[1 + grp][0], sj[1 + grp][1], sj[1 + grp][2], sj[1 + grp][3]), S);
    acc = accD = 0.0;
    mom[0] = mom[1] = mom[2] = 0.0;
    if (lm) {
        t64_nodes_except<true>(lp, sg.off, G.x, G.y, S.x, S.y, half, 2, cs, og, tg, lane, tiles[warp], acc, accD, mom);
        t64_nodes_except<true>(lp, sg.off, G.z, G.w, S.z, S.w, half, 2, cs, og, tg, lane, tiles[warp], acc, accD, mom);
    } else {
        t64_nodes_except<false>(lp, sg.off, G.x, G.y, S.x, S.y, half, 2, cs, og, tg, lane, tiles[warp], acc, accD, mom);
        t64_nodes_except<false>(lp, sg.off, G.z, G.w, S.z, S.w, half, 2, cs, og, tg, lane, tiles[warp], acc, accD, mom);
    }
    {
        const double A = warp_sum64(mom[0]), B = warp_sum64(mom[1]), C = warp_sum64(mom[2]);
        acc -= 2.0 * A - rc2 * fma(tg, fma(tg, A, -2.0 * B), C);
    }
    // each warp carries half of the strip's nodes down
    for (int k = 16 * half; k < 16 * half + 16; ++k) {
        const double w = tab->M[grp][k][lane];
        acc = fma(F[k], w, acc);
        if (lm) accD = fma(FD[k], w, accD);
    }
    part[warp][lane] = acc;
    if (lm) partD[warp][lane] = accD;
    __syncthreads();
    if (half == 0) {
        const size_t cell = (size_t)(s - seg0) * n_groups + 4 * strip + grp;
        far[cell * kT64Nodes + lane] = part[warp][lane] + part[warp + 1][lane];
        if (ANY_LM && farD) farD[cell * kT64Nodes + lane] = lm ? partD[warp][lane] + partD[warp + 1][lane] : 0.0;
        if (lane == 0) {
            ranges[cell] = G;
            int n = (G.y - G.x) + (G.w - G.z) - (S.y - S.x) - (S.w - S.z);  // S's lines lie inside G's
            if (grp == 0) n += (S.y - S.x) + (S.w - S.z);
            if (evald) atomicAdd(evald, (unsigned long long)max(n, 0) * kT64Nodes);
        }
    }
}

// Core points within |x| + y < 8 (Weideman's 40-term series, four times the cost of the
// outer forms): a few points of one or two 32-point rows per line, evaluated lane-parallel
// per tile into cw and read back by the rows, as in the mixed kernel.
template <int Q, bool LM>
struct T64Leaf {
    static constexpr int kBuf = Q == 4 ? 256 : 96;
    T64Tile far;                        // far lines; wing lines: (nu0, b^2), (a, g or P)
    double2 c0[32], c1[32], c2[32];     // core lines: (nu0, f), (b, k0), (y, Sn)
    double cP[32], cg[LM ? 32 : 1], cY[LM ? 32 : 1];
    int4 cr[32];                        // inner points [x, y], offset in cw
    int jx[32], cj[32];                 // line indices (edge tests)
    double nd[kT64Nodes], ndD[LM ? kT64Nodes : 1];
    double cw[kBuf], cwi[LM ? kBuf : 1];
};

// One tile (nt <= 32 lines from j0) evaluated at the leaf's points.  EDGE: per-point
// windows [jlo, jhi) and per-point pedestals; otherwise every line covers every point and
// its pedestal goes into the moments.  Wing lines (core off the leaf) first, then core lines.
template <int METHOD, int Q, bool LM, bool EDGE>
__device__ __forceinline__ void t64_tile(const LpOutF64& lp, long long off, int j0, int nt, double cs, double o, double hp,
                                         double dnu, const double* __restrict__ grid, long long wb, long long n_nu,
                                         double rc2, double x_far, int lane, const double nu[Q], const int jlo[Q],
                                         const int jhi[Q], T64Leaf<Q, LM>& T, double acc[Q], double accD[Q],
                                         double mom[3]) {
    constexpr int P = 32 * Q;
    __syncwarp();
    double u = 0.0, nu0 = 0.0, f = 1.0, b = 1.0, k0 = 0.0, y = 0.0, Sn = 0.0, Pd = 0.0, g = 0.0, Y = 0.0;
    bool core = false;
    if (lane < nt) {
        const long long q = off + j0 + lane;
        nu0 = lp.nu0[q];
        u = (nu0 - cs) - o;
        f = lp.f[q];
        b = lp.b[q];
        k0 = lp.k0[q];
        y = lp.y[q];
        Sn = lp.Sn[q];
        Pd = Sn * lp.Hc[q];
        if (LM) {
            g = lp.g[q];
            Y = lp.YSn[q];
        }
        core = (fabs(u) - hp) * f <= x_far;  // hp: the points' half-extent, rounded up
        if (!EDGE) {
            mom[0] += Pd;
            mom[1] = fma(Pd, u, mom[1]);
            mom[2] = fma(Pd * u, u, mom[2]);
        }
    }
    const unsigned cm = __ballot_sync(kFull, lane < nt && core), wm = __ballot_sync(kFull, lane < nt && !core);
    const unsigned lt = (1u << lane) - 1u;
    const int nc = __popc(cm), nw = __popc(wm);
    int nin = 0, plo = 1, coff = 0, cfit = 0;
    if (METHOD == 3 && cm) {
        if (core && y < 8.0) {  // inner points, one to spare on each side
            const double hw = (8.0 - y) / (f * dnu) + 1.0, pc = u / dnu + 0.5 * (P - 1);
            const double lo = fmax(pc - hw, 0.0), hi = fmin(pc + hw, (double)(P - 1));
            if (lo <= hi) {
                plo = (int)ceil(lo);
                nin = max((int)floor(hi) - plo + 1, 0);
            }
        }
        int inc = nin;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(kFull, inc, d);
            if (lane >= d) inc += v;
        }
        coff = inc - nin;
        const unsigned ov = __ballot_sync(kFull, inc > T.kBuf && nin > 0);
        cfit = ov ? __shfl_sync(kFull, coff, __ffs(ov) - 1) : __shfl_sync(kFull, inc, 31);
        if (inc > T.kBuf) nin = 0;  // beyond the buffer: per point
    }
    if (lane < nt && !core) {
        const int pos = __popc(wm & lt);
        T.far.ub[pos] = make_double2(nu0, b * b);
        T.far.ag[pos] = make_double2(k0 * b, EDGE ? Pd : g);
        if (EDGE) {
            T.jx[pos] = j0 + lane;
            if (LM) T.cg[pos] = g;  // wing lines from the bottom; core lines use the top below
        }
    } else if (lane < nt) {
        const int pos = __popc(cm & lt);
        T.c0[pos] = make_double2(nu0, f);
        T.c1[pos] = make_double2(b, k0);
        T.c2[pos] = make_double2(y, Sn);
        if (EDGE) {
            T.cP[pos] = Pd;
            T.cj[pos] = j0 + lane;
        }
        if (LM) {
            T.cg[31 - pos] = g;
            T.cY[pos] = Y;
        }
        if (METHOD == 3) T.cr[pos] = make_int4(plo, plo + nin - 1, coff, 0);
    }
    if (!EDGE && lane >= nw && lane < ((nw + 3) & ~3)) {  // pad the last group of four
        T.far.ub[lane] = make_double2(0.0, 1.0);
        T.far.ag[lane] = make_double2(0.0, 0.0);
    }
    __syncwarp();
    if (METHOD == 3 && cfit > 0) {
        for (int e = lane; e < cfit; e += 32) {  // the line owning element e: the last with offset <= e
            int lo = 0, hi = nc - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (T.cr[mid].z <= e) lo = mid; else hi = mid - 1;
            }
            const int4 r = T.cr[lo];
            const double2 uf = T.c0[lo];
            const long long ip = min(wb + r.x + (e - r.z), n_nu - 1);
            const double d = grid[ip] - uf.x;
            const double2 w = faddeeva64(d * uf.y, T.c2[lo].x);
            T.cw[e] = w.x;
            if (LM) T.cwi[e] = w.y;
        }
        __syncwarp();
    }
    // wing lines
    if (!EDGE) {
        if (Q == 4) {
            for (int i = 0; i < nw; ++i) {
                const double2 ub = T.far.ub[i], ag = T.far.ag[i];
                double d[4], e[4], r[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    d[q] = nu[q % Q] - ub.x;
                    e[q] = fma(d[q], d[q], ub.y);
                }
                rcp64_quad(e, r);
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    acc[q] = fma(ag.x, r[q], acc[q]);
                    if (LM) accD[q] = fma(ag.y * d[q], r[q], accD[q]);
                }
            }
        } else {
            for (int i = 0; i < nw; i += 4) {
                double d[4], e[4], r[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const double2 ub = T.far.ub[i + v];
                    d[v] = nu[0] - ub.x;
                    e[v] = fma(d[v], d[v], ub.y);
                }
                rcp64_quad(e, r);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const double2 ag = T.far.ag[i + v];
                    acc[0] = fma(ag.x, r[v], acc[0]);
                    if (LM) accD[0] = fma(ag.y * d[v], r[v], accD[0]);
                }
            }
        }
    } else {
        for (int i = 0; i < nw; ++i) {
            const double2 ub = T.far.ub[i], ag = T.far.ag[i];
            const int j = T.jx[i];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const double d = nu[q] - ub.x, d2 = d * d;
                const double r = rcp64_fast(d2 + ub.y);
                const bool in = j >= jlo[q] && j < jhi[q];
                acc[q] += in ? fma(ag.x, r, -ag.y * fma(-d2, rc2, 2.0)) : 0.0;
                if (LM) accD[q] += in ? T.cg[i] * d * r : 0.0;
            }
        }
    }
    // core lines
    for (int i = 0; i < nc; ++i) {
        const double2 uf = T.c0[i], bk = T.c1[i], ys = T.c2[i];
        const double if2 = METHOD == 3 ? rcp64_fast(uf.y * uf.y) : 0.0;
        const double gi = LM ? T.cg[31 - i] : 0.0, Yi = LM ? T.cY[i] : 0.0;
        const int4 cr = METHOD == 3 ? T.cr[i] : make_int4(1, 0, 0, 0);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double d = nu[q] - uf.x, x = d * uf.y;
            const double r = rcp64_fast(fma(d, d, bk.x * bk.x));
            double v = bk.y * bk.x * r, vD = LM ? gi * d * r : 0.0;
            const bool cr_in = !(fabs(x) > x_far);
            if (__any_sync(kFull, cr_in)) {
                if (METHOD == 1) {
                    if (cr_in) v = ys.y * weideman24_64(x, ys.x);
                } else {
                    const int pt = lane + 32 * q;
                    const bool held = pt >= cr.x && pt <= cr.y;
                    const bool inner = cr_in && !held && fabs(x) + ys.x < 8.0;
                    const bool ratio = cr_in && !held && !inner && fma(x, x, ys.x * ys.x) < kWofzSeries2;
                    // 1/z = (d - i b) r / f
                    const double dr = d * r, br = bk.x * r;
                    double2 S;
                    if (__any_sync(kFull, ratio)) {
                        S = wofz_ratio64(fma(x, x, -ys.x * ys.x), 2.0 * x * ys.x);
                        if (!ratio) {
                            const double2 S2 = wofz_series64(fma(dr, dr, -br * br) * if2, -2.0 * dr * br * if2);
                            S = S2;
                        }
                    } else {
                        S = wofz_series64(fma(dr, dr, -br * br) * if2, -2.0 * dr * br * if2);
                    }
                    if (cr_in) {
                        if (held) {
                            v = ys.y * T.cw[cr.z + pt - cr.x];
                            if (LM) vD = Yi * T.cwi[cr.z + pt - cr.x];
                        } else if (inner) {
                            const double2 w = faddeeva64(x, ys.x);
                            v = ys.y * w.x;
                            if (LM) vD = Yi * w.y;
                        } else {
                            v = bk.y * fma(br, S.x, -dr * S.y);
                            if (LM) vD = gi * fma(dr, S.x, br * S.y);
                        }
                    }
                }
            }
            if (EDGE) {
                const int j = T.cj[i];
                const bool in = j >= jlo[q] && j < jhi[q];
                acc[q] += in ? fma(-T.cP[i], fma(-d * d, rc2, 2.0), v) : 0.0;
                if (LM) accD[q] += in ? vD : 0.0;
            } else {
                acc[q] += v;
                if (LM) accD[q] += vD;
            }
        }
    }
}

// the index window of each point, [jlo, jhi): the same binary searches on the shifted
// centres as linesum_f64_kernel makes (lower_bound1, upper_bound1), their common first
// steps taken once for the leaf, so that lines out of order are taken the same way
template <int Q>
__device__ __forceinline__ void t64_windows(const double* __restrict__ a, long long n, const double nu[Q], double nmin,
                                            double nmax, double cutoff, int jlo[Q], int jhi[Q]) {
    {
        int lo = 1, hi = (int)n + 1;
        const double vmin = nmin - cutoff, vmax = nmax - cutoff;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const double x = a[mid - 1];
            if (x < vmin) lo = mid + 1;
            else if (!(x < vmax)) hi = mid;
            else break;
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double v = nu[q] - cutoff;
            int l = lo, h = hi;
            while (l < h) {
                const int mid = (l + h) >> 1;
                if (a[mid - 1] < v) l = mid + 1; else h = mid;
            }
            jlo[q] = l - 1;
        }
    }
    {
        int lo = 0, hi = (int)n;
        const double vmin = nmin + cutoff, vmax = nmax + cutoff;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const double x = a[mid - 1];
            if (x > vmax) hi = mid - 1;
            else if (!(x > vmin)) lo = mid;
            else break;
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double v = nu[q] + cutoff;
            int l = lo, h = hi;
            while (l < h) {
                const int mid = (l + h + 1) >> 1;
                if (a[mid - 1] > v) h = mid - 1; else l = mid;
            }
            jhi[q] = l;
        }
    }
}

template <int METHOD, int Q, bool LM>
__device__ __forceinline__ void t64_segment(const SegDev& sg, long long cnt, const LpOutF64& lp, double reach,
                                            double cs, double o, double dnu, double cutoff, double x_far,
                                            const double* __restrict__ grid, long long wb, long long n_nu,
                                            const double nu[Q], double nmin, double nmax, int lane, int quarter,
                                            const T64Tables* __restrict__ tab, const double* __restrict__ far,
                                            const double* __restrict__ farD, int4 up, T64Leaf<Q, LM>& T, double sig[Q],
                                            unsigned long long& work) {
    constexpr int P = 32 * Q;
    const double h = 0.5 * P * dnu, m = t64_margin(sg, dnu), rc2 = 1.0 / (cutoff * cutoff);
    const double* a = lp.nu0 + sg.off;
    const double c = cs + o;
    int jlo[Q], jhi[Q];
    t64_windows<Q>(a, cnt, nu, nmin, nmax, cutoff, jlo, jhi);
    int jmin = jlo[0], jmax = jhi[0];
#pragma unroll
    for (int q = 1; q < Q; ++q) {
        jmin = min(jmin, jlo[q]);
        jmax = max(jmax, jhi[q]);
    }
    jmin = __reduce_min_sync(kFull, jmin);
    jmax = __reduce_max_sync(kFull, jmax);
    const double R = fmax(kT64Ratio * h, reach + h) + m;
    const bool full = cutoff - h - m > R;  // lines nearer than the far ones cover every point
    int bd[4];
#pragma unroll
    for (int b = 0; b < 4; ++b)
        bd[b] = jmin + (int)warp_lower_bound(a + jmin, t64_bound(b, c, h, cutoff, m, reach), max(jmax - jmin, 0), lane);
    const int4 own = t64_inside(t64_order(bd[0], bd[1], bd[2], bd[3]), up);
    double t[Q], acc[Q], accD[Q], mom[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        t[q] = (nu[q] - cs) - o;
        acc[q] = accD[q] = 0.0;
    }
    const double hp = fmax(nmax - c, c - nmin) + 1e-9 * dnu;
    {
        const int nf = (own.y - own.x) + (own.w - own.z);
        work += (unsigned long long)(jmax - jmin - nf) * P + (unsigned long long)(nf - (up.y - up.x) - (up.w - up.z)) * kT64Nodes;
    }
    // far lines of the leaf, at its nodes, and the group's node values
    const double tn = h * tab->x[lane];
    double nd = 0.0, ndD = 0.0;
    t64_nodes_except<LM>(lp, sg.off, own.x, own.y, up.x, up.y, 0, 1, cs, o, tn, lane, T.far, nd, ndD, mom);
    t64_nodes_except<LM>(lp, sg.off, own.z, own.w, up.z, up.w, 0, 1, cs, o, tn, lane, T.far, nd, ndD, mom);
    if (far) {
        __syncwarp();
        T.nd[lane] = far[lane];
        if (LM) T.ndD[lane] = farD[lane];
        __syncwarp();
#pragma unroll 8
        for (int k = 0; k < kT64Nodes; ++k) {
            const double w = tab->M[quarter][k][lane];
            nd = fma(T.nd[k], w, nd);
            if (LM) ndD = fma(T.ndD[k], w, ndD);
        }
    }
    // direct lines: [jmin, own.x) and [own.w, jmax) with their cutoffs among the points,
    // [own.y, own.z) near ones
#define IRS_T64_RANGE(A, B, EDGE)                                                                                     \
    for (int j0 = (A); j0 < (B); j0 += 32)                                                                            \
        t64_tile<METHOD, Q, LM, EDGE>(lp, sg.off, j0, min(32, (B) - j0), cs, o, hp, dnu, grid, wb, n_nu, rc2, x_far,   \
                                      lane, nu, jlo, jhi, T, acc, accD, mom)
    if (full) {
        IRS_T64_RANGE(own.y, own.z, false);
        IRS_T64_RANGE(jmin, own.x, true);
        IRS_T64_RANGE(own.w, jmax, true);
    } else {  // no far lines at this leaf (the cutoff is narrow or the core wide)
        IRS_T64_RANGE(jmin, jmax, true);
    }
#undef IRS_T64_RANGE
    // the interpolant at the points, corrected for their offset from the uniform grid
    __syncwarp();
    T.nd[lane] = nd;
    if (LM) T.ndD[lane] = ndD;
    __syncwarp();
    double v[Q], vD[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = vD[q] = 0.0;
#pragma unroll 4
    for (int k = 0; k < kT64Nodes; ++k) {
        const double F = T.nd[k], FD = LM ? T.ndD[k] : 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const double w = Q == 4 ? tab->L4[k][32 * q + lane] : tab->L1[k][lane];
            v[q] = fma(F, w, v[q]);
            if (LM) vD[q] = fma(FD, w, vD[q]);
        }
    }
    const double A = warp_sum64(mom[0]), B = warp_sum64(mom[1]), C = warp_sum64(mom[2]);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const double dl = t[q] / dnu - ((double)(lane + 32 * q) - 0.5 * (P - 1));  // grid steps off the ideal point
        const double up1 = __shfl_down_sync(kFull, v[q], 1), dn1 = __shfl_up_sync(kFull, v[q], 1);
        const double slope = lane == 0 ? up1 - v[q] : lane == 31 ? v[q] - dn1 : 0.5 * (up1 - dn1);
        double sv = acc[q] + fma(slope, dl, v[q]) - (2.0 * A - rc2 * fma(t[q], fma(t[q], A, -2.0 * B), C));
        sv = fmax(sv, 0.0);
        if (LM) {
            const double u1 = __shfl_down_sync(kFull, vD[q], 1), d1 = __shfl_up_sync(kFull, vD[q], 1);
            const double sl = lane == 0 ? u1 - vD[q] : lane == 31 ? vD[q] - d1 : 0.5 * (u1 - d1);
            sv = fmax(sv + accD[q] + fma(sl, dl, vD[q]), 0.0);
        }
        sig[q] = sv;
    }
}

// One warp per leaf of 32 Q points, the four leaves of a group per CTA; grid (groups,
// profile-layers).
template <int METHOD, int Q, bool ANY_LM>
__global__ void __launch_bounds__(32 * kT64LeafWarps, 4) tree64_leaf_kernel(
    const SegDev* __restrict__ segs, const int* __restrict__ seg_count, const unsigned* __restrict__ core_reach,
    const int2* __restrict__ pl_segs, LpOutF64 lp, const double* __restrict__ grid, long long n_nu, double g0,
    double dnu, double cutoff, double x_far, const T64Tables* __restrict__ tab, const double* __restrict__ far,
    const double* __restrict__ farD, const int4* __restrict__ ranges, int n_groups, int pl0, int seg0,
    double* __restrict__ tau, double* __restrict__ pert, long long pstride, const int* __restrict__ uniform,
    unsigned long long* __restrict__ evald) {
    if (uniform && !*uniform) return;
    constexpr int P = 32 * Q;
    extern __shared__ __align__(16) unsigned char t64_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T64Leaf<Q, ANY_LM>& T = reinterpret_cast<T64Leaf<Q, ANY_LM>*>(t64_smem)[warp];
    const int pl = pl0 + (int)blockIdx.y;
    const long long wb = ((long long)blockIdx.x * kT64LeafWarps + warp) * P;
    if (wb >= n_nu) return;  // no block-wide barriers
    const int strip = (int)blockIdx.x >> 2, in_strip = ((int)blockIdx.x & 3) * kT64LeafWarps + warp;
    const double cs = g0 + dnu * ((double)strip * 16 * P + 8.0 * P - 0.5), o = (in_strip - 7.5) * P * dnu;
    double nu[Q], tsum[Q];
    double nmin = 1e300, nmax = -1e300;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        nu[q] = grid[min(wb + 32 * q + lane, n_nu - 1)];
        nmin = fmin(nmin, nu[q]);
        nmax = fmax(nmax, nu[q]);
        tsum[q] = 0.0;
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        nmin = fmin(nmin, __shfl_xor_sync(kFull, nmin, d));
        nmax = fmax(nmax, __shfl_xor_sync(kFull, nmax, d));
    }
    unsigned long long work = 0;
    const int2 rng = pl_segs[pl];
    for (int s = rng.x; s < rng.x + rng.y; ++s) {
        const SegDev sg = segs[s];
        const long long cnt = seg_count[s];
        const double reach = (double)__uint_as_float(core_reach[s]);
        const size_t cell = (size_t)(s - seg0) * n_groups + blockIdx.x;
        const int4 up = far ? ranges[cell] : make_int4(0, 0, 0, 0);
        const double* fr = far ? far + cell * kT64Nodes : nullptr;
        double sig[Q];
        if (ANY_LM && (sg.flags & SEG_LM))
            t64_segment<METHOD, Q, ANY_LM>(sg, cnt, lp, reach, cs, o, dnu, cutoff, x_far, grid, wb, n_nu, nu, nmin, nmax,
                                           lane, warp, tab, fr, far ? farD + cell * kT64Nodes : nullptr, up, T, sig, work);
        else
            t64_segment<METHOD, Q, false>(sg, cnt, lp, reach, cs, o, dnu, cutoff, x_far, grid, wb, n_nu, nu, nmin, nmax,
                                          lane, warp, tab, fr, nullptr, up,
                                          reinterpret_cast<T64Leaf<Q, false>&>(T), sig, work);
        const bool rel = pert && (sg.flags & SEG_RELMAT);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const long long i = wb + 32 * q + lane;
            if (rel) {
                if (i < n_nu) pert[(size_t)pl * pstride + i] = sig[q];
            } else {
                tsum[q] = fma(sig[q], sg.coef, tsum[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const long long i = wb + 32 * q + lane;
        if (i < n_nu) tau[(size_t)pl * n_nu + i] = tsum[q];
    }
    if (evald && lane == 0) atomicAdd(evald, work);
}

// *out stays 1 when every grid point lies within 1e-7 steps of the uniform grid of its ends
// (rounding of the points is about 1e-10 steps), which the interpolation's first-order
// correction covers to 1e-15
__global__ void __launch_bounds__(256) grid_uniform_kernel(const double* __restrict__ grid, long long n, double g0,
                                                           double dnu, int* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(fabs(grid[i] - fma((double)i, dnu, g0)) <= 1e-7 * dnu)) *out = 0;
}

}  // namespace irs
