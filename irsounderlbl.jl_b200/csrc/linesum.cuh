// linesum.cuh -- the line-by-line sum: sigma(nu_i) = max(sum_j Sn_j [H(x, y) - ped_j(nu_i)], 0)
// over lines within the cutoff (src/CrossSections/voigt.jl:243-313), times the layer
// column coef and summed over species into the layer optical depth
// (src/Sensor/sounder.jl:283-307); with VP_Y line mixing the CO2 term is
// max(sigma_V + sum_j YSn_j Im w, 0) (line_mixing.jl:1166-1186, :1351-1369).
//
// Two kernels here, and linesum_tree64.cuh:
//  * linesum_f64_kernel -- the plain FP64 GPU kernel: one thread per grid point,
//    a binary search per point and species for the window on the shifted centres,
//    FP64 arithmetic and IEEE division, exactly the reference kernel's structure.  It
//    serves PseudoVoigt, cross sections of short lists and grids that are not uniform; the
//    FP64 sum of the other methods on a uniform grid is tree64_leaf_kernel's.
//  * linesum_mixed_kernel -- FP32 + Kahan, every line of the window evaluated at every
//    point (IRS_MIXED_DIRECT), and PseudoVoigt.  IRS_MIXED's sum is fw_leaf_kernel's
//    (linesum_mixed_tree.cuh).
#pragma once
#include "faddeeva.cuh"
#include "irs_internal.h"
#include "lineparams.cuh"

namespace irs {

// voigt.jl:220-236, 1-based
__device__ __forceinline__ long long lower_bound1(const double* a, double v, long long n) {
    long long lo = 1, hi = n + 1;
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (a[mid - 1] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ long long upper_bound1(const double* a, double v, long long n) {
    long long lo = 0, hi = n;
    while (lo < hi) {
        const long long mid = (lo + hi + 1) >> 1;
        if (a[mid - 1] > v) hi = mid - 1; else lo = mid;
    }
    return lo;
}

// ------------------------------------------------------------------ FP64
template <int METHOD>
__global__ void __launch_bounds__(256) linesum_f64_kernel(
    const SegDev* __restrict__ segs, const int* __restrict__ seg_count, const int2* __restrict__ pl_segs,
    LpOutF64 lp, const double* __restrict__ grid, long long n_nu, double cutoff, double x_far,
    double* __restrict__ tau, double* __restrict__ pert, long long pstride, const int* __restrict__ uniform) {
    if (uniform && *uniform) return;  // taken by tree64_leaf_kernel
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int pl = blockIdx.y;
    if (i >= n_nu) return;
    const double nu = grid[i];
    const int2 rng = pl_segs[pl];
    double tsum = 0.0;
    const double rc = 1.0 / cutoff;
    for (int s = rng.x; s < rng.x + rng.y; ++s) {
        const SegDev sg = segs[s];
        const long long cnt = seg_count[s];
        const double* nu0 = lp.nu0 + sg.off;
        const long long jlo = lower_bound1(nu0, nu - cutoff, cnt);
        const long long jhi = upper_bound1(nu0, nu + cutoff, cnt);
        double acc = 0.0, accD = 0.0;
        const bool lm = (sg.flags & 2) != 0;
        for (long long j = jlo; j <= jhi; ++j) {
            const long long q = sg.off + j - 1;
            const double d = nu - lp.nu0[q];
            if (METHOD == 2) {  // PseudoVoigt, voigt.jl:301-311 (f = gV, y = eta, Sn = S, Hc = base)
                const double gV = lp.f[q], eta = lp.y[q];
                const double G = 0.46971863934982566 / gV * exp(-0.69314718055994531 * d * d / (gV * gV));
                const double Lz = gV * 0.31830988618379067 / (d * d + gV * gV);
                const double zr = d * rc;
                acc += lp.Sn[q] * (eta * Lz + (1.0 - eta) * G) - (2.0 - zr * zr) * lp.Hc[q];
            } else {            // voigt.jl:264-275
                const double x = d * lp.f[q];
                const double y = lp.y[q];
                const double zr = d * rc;
                const double ped = (2.0 - zr * zr) * lp.Hc[q];
                const double H = (fabs(x) > x_far ? y * kInvSqrtPi / (x * x + y * y) : hcore64<METHOD>(x, y)) - ped;
                acc += lp.Sn[q] * H;
            }
            if (lm) {  // line_mixing.jl:1177-1184
                const double x = d * lp.f[q];
                const double y = lp.y[q];
                const double imw = fabs(x) > x_far ? x * kInvSqrtPi / (x * x + y * y) : faddeeva64(x, y).y;
                accD += lp.YSn[q] * imw;
            }
        }
        double sig = fmax(acc, 0.0);
        if (lm) sig = fmax(sig + accD, 0.0);
        if (pert && (sg.flags & SEG_RELMAT)) {  // relmat line mixing: finished by relmat_finish_kernel
            pert[(size_t)pl * pstride + i] = sig;
            continue;
        }
        tsum += sig * sg.coef;
    }
    tau[(size_t)pl * n_nu + i] = tsum;
}

// ----------------------------------------------------------------- mixed
// Each warp owns 128 consecutive grid points (4 per lane, point = 32 q + lane)
// and walks its own window of lines in tiles of 32 staged in warp-private shared
// memory (no block-wide barriers).  The staging lane of each line precomputes,
// once per (warp, line): the FP32 position split u = uh + ul relative to the
// warp, the class of the line for this warp (outside the cutoff / fast / slow),
// and, for fast lines, the line's pedestal as a quadratic in the point index, so
// the 32 pedestals of a tile reduce to three numbers.
//   fast: inside the cutoff and in the Lorentz far wing (|x| > x_far) for all 128
//         points: d by one FADD from a per-line origin, one MUFU reciprocal per
//         two pairs, one FMA into the tile sum;
//   slow: Faddeeva core or cutoff edge: per-pair tests.
// Tile sums go into a Kahan-compensated FP32 accumulator per point.
constexpr int kMxWarps = 16;
constexpr int kMxThreads = 32 * kMxWarps;
constexpr int kMxQ = 4;                               // points per lane
constexpr int kMxWarpPts = 32 * kMxQ;                 // 128 points per warp
constexpr int kMxStrip = kMxWarps * kMxWarpPts;       // 2048 points per CTA
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ long long lower_bound0(const double* a, double v, long long n) {
    long long lo = 0, hi = n;
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// 1/x with the MUFU approximation (max 1 ulp); x > 0 and finite here
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
    return v;
}

// Inner points of a slow line: |x| + y < 15 (plus one point each side), where
// faddeeva32 takes its CF4 or Weideman branch.  They span a few points of one or two
// 32-point rows, so evaluating them inside the per-point loop leaves most lanes of
// those rows idle; instead each tile evaluates the inner points of all its slow lines
// lane-parallel into cw (up to kCoreBuf per tile; lines beyond it keep the per-point
// evaluation) and the per-point loop reads them back.
constexpr int kCoreBuf = 128;

struct WarpTile {
    float4 fu[32];  // fast lines: uh, ul, b2, a               (PV: uh, ul, -, class)
    float4 su[32];  // slow lines: uh, ul, b2, a               (PV: gV2, aPV, c1, c0)
    float4 sp[32];  // slow lines: c1, c0, dfar2, An           (PV: kPV, gPV, -, -)
    float4 sq[32];  // slow lines: fx, y, g, Yw
    float fg[32];   // fast lines: g (dispersive line mixing)
    int4 sr[32];    // slow lines (FullFaddeeva): inner points [x, y] of the block, their offset z in cw
    float2 cw[kCoreBuf];  // w(x + i y) at the inner points of the tile's slow lines, line after line
};

// First index i in [0, n) with a[i] >= v (n if none), found by the whole warp: each
// round probes 32 evenly spaced positions and keeps the interval between the last
// probe below v and the first one at or above it (32-ary search: 4 dependent loads
// for 66 k lines instead of 17).  All lanes return the same value.
__device__ __forceinline__ long long warp_lower_bound(const double* a, double v, long long n, int lane) {
    long long lo = 0, hi = n;  // the answer lies in [lo, hi]
    while (hi - lo > 32) {
        const long long step = (hi - lo + 31) / 32;
        const long long p = min(lo + (long long)(lane + 1) * step - 1, hi - 1);
        const unsigned below = __ballot_sync(kFull, a[p] < v);  // a prefix of the lanes
        const int c = __popc(below);
        const long long nlo = lo + (long long)c * step;
        hi = min(hi, lo + (long long)(c + 1) * step);
        lo = min(nlo, hi);
    }
    const long long p = lo + lane;
    const unsigned below = __ballot_sync(kFull, p < hi && a[p] < v);
    return lo + __popc(below);
}

// window [jlo, jhi) of the lines that can reach this warp's points [wb, wb + kMxWarpPts - 1]
__device__ __forceinline__ void warp_window(const LpOutMixed& lp, const SegDev& sg, long long cnt,
                                            long long wb, float cut, int lane, long long& jlo, long long& jhi) {
    const double* V = lp.V + sg.off;
    jlo = warp_lower_bound(V, (double)wb - cut - sg.margin_g, cnt, lane);
    jhi = warp_lower_bound(V, (double)(wb + kMxWarpPts - 1) + cut + sg.margin_g + 1e-9, cnt, lane);
}

// Fast line, two points q and q+1 with packed FP32x2 arithmetic.  The squared
// distances are formed in swapped order es = (e[q+1], e[q]) so one reciprocal of
// their product gives both reciprocals with a single packed multiply:
//   r = es * (1/(e[q] e[q+1])) = (1/e[q], 1/e[q+1]).
__device__ __forceinline__ void fast_pair(float2 d0s, float2 offs, float2 b2, float2 a, float2& acc) {
    const float2 dds = __fadd2_rn(d0s, offs);       // (d[q+1], d[q])
    const float2 es = __ffma2_rn(dds, dds, b2);     // (e[q+1], e[q])
    const float R = rcp_fast(es.x * es.y);
    const float2 r = __fmul2_rn(es, make_float2(R, R));
    acc = __ffma2_rn(a, r, acc);
}

// The optical-depth row of a warp's 128 points.  Each segment's clamped sums are
// added to it in segment order (the first one stores), so no per-point total stays
// in registers from one segment to the next.
struct OutRow {
    float* p;    // tau at the warp's first point
    int n;       // the warp's points inside the grid
    bool wrote;  // a segment has stored
};
__device__ __forceinline__ void out_add(OutRow& o, int q, int lane, float sig) {
    const int i = 32 * q + lane;
    if (i < o.n) o.p[i] = o.wrote ? o.p[i] + sig : sig;
}

template <int METHOD, bool LM>
__device__ __forceinline__ void warp_segment(const SegDev& sg, long long cnt, const LpOutMixed& lp, long long wb,
                                             float cut, float cut2, int lane, WarpTile& T, OutRow& orow,
                                             unsigned long long& work, double* __restrict__ prow) {
    constexpr float kCentre = 0.5f * (kMxWarpPts - 1);
    constexpr float kHalf = 0.5f * kMxWarpPts + 0.5f;
    long long jlo, jhi;
    warp_window(lp, sg, cnt, wb, cut, lane, jlo, jhi);
    const float pl0 = (float)lane;
    // per-lane constant offsets of the point pairs, swapped: (32(q+1), 32q)
    float2 offs[kMxQ / 2];
#pragma unroll
    for (int h = 0; h < kMxQ / 2; ++h) offs[h] = make_float2(32.f * (2 * h + 1), 32.f * (2 * h));
    float sum[kMxQ], comp[kMxQ], sumD[kMxQ], compD[kMxQ];
#pragma unroll
    for (int q = 0; q < kMxQ; ++q) sum[q] = comp[q] = sumD[q] = compD[q] = 0.f;
    const unsigned lt = (1u << lane) - 1u;
    const int ilo = (int)jlo, ihi = (int)jhi;  // indices within a segment fit in int: seg_count is an int
    for (int t0 = ilo; t0 < ihi; t0 += 32) {
        const int nt = min(32, ihi - t0);
        float pa = 0.f, pb = 0.f, pc = 0.f;  // this line's pedestal quadratic (fast lines)
        int cls = 0;
        float4 a0, a1;
        float2 a2 = make_float2(0.f, 0.f);
        float uh = 0.f, ul = 0.f;
        if (lane < nt) {
            const long long q = sg.off + t0 + lane;
            const float2 uf = lp.U[q];
            uh = uf.x - (float)wb;  // exact: see split_hi_lo
            ul = uf.y;
            a0 = lp.p0[q];
            if (LM) a2 = lp.p2[q];
            const float dist = fabsf(uh - kCentre);
            if (dist > cut + kHalf) cls = 0;
            else if (dist + kHalf <= cut && dist > lp.df[q] + kHalf) {
                cls = 1;
                // sum over points p of c1 (p - u)^2 + c0 = p^2 c1 - 2 p c1 u + (c1 u^2 + c0)
                const float u = uh + ul;
                pa = a0.z;
                pb = a0.z * u;
                pc = fmaf(pb, u, a0.w);
            } else {
                cls = 2;
                a1 = lp.p1[q];
            }
        }
        // FullFaddeeva slow lines: the inner points of the block, [plo, plo + nin - 1],
        // and their offsets in cw by a warp scan; cfit = the points that fit (warp-uniform)
        int nin = 0, plo = 1, coff = 0, cfit = 0;
        const unsigned sm = __ballot_sync(kFull, cls == 2);
        if (METHOD == 3 && sm) {  // (warp-uniform)
            if (cls == 2 && a1.w < 15.f) {
                const float hw = (15.f - a1.w) / a1.z + 1.f;
                const float c = uh + ul;
                const float lo = fmaxf(c - hw, 0.f), hi = fminf(c + hw, (float)(kMxWarpPts - 1));
                if (lo <= hi) {
                    plo = (int)ceilf(lo);
                    nin = max((int)floorf(hi) - plo + 1, 0);
                }
            }
            int inc = nin;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(kFull, inc, d);
                if (lane >= d) inc += t;
            }
            coff = inc - nin;
            const unsigned ov = __ballot_sync(kFull, inc > kCoreBuf && nin > 0);
            cfit = ov ? __shfl_sync(kFull, coff, __ffs(ov) - 1) : __shfl_sync(kFull, inc, 31);
            if (inc > kCoreBuf) nin = 0;  // beyond the buffer: evaluated per point
        }
        const unsigned fm = __ballot_sync(kFull, cls == 1);
        __syncwarp();
        if (cls == 1) {
            const int pos = __popc(fm & lt);
            T.fu[pos] = make_float4(uh, ul, a0.x, a0.y);
            if (LM) T.fg[pos] = a2.x;
        } else if (cls == 2) {
            const int pos = __popc(sm & lt);
            T.su[pos] = make_float4(uh, ul, a0.x, a0.y);
            T.sp[pos] = make_float4(a0.z, a0.w, a1.x, a1.y);
            T.sq[pos] = make_float4(a1.z, a1.w, a2.x, a2.y);
            if (METHOD == 3) T.sr[pos] = make_int4(plo, plo + nin - 1, coff, 0);
        }
        const float A = warp_sum(pa), B = warp_sum(pb), Cc = warp_sum(pc);
        __syncwarp();
        const int nf = __popc(fm), ns = __popc(sm);
        if (lane == 0) work += (unsigned long long)(nf + ns) * kMxWarpPts;
        if (METHOD == 3 && cfit > 0) {  // the inner points, one per lane: the slow line owning
                                        // element e is the last one whose offset is <= e
            for (int e = lane; e < cfit; e += 32) {
                int lo = 0, hi = ns - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (T.sr[mid].z <= e) lo = mid;
                    else hi = mid - 1;
                }
                const int4 r = T.sr[lo];
                const float4 u = T.su[lo], w = T.sq[lo];
                const float d = ((float)(r.x + (e - r.z)) - u.x) - u.y;  // as in the per-point loop
                T.cw[e] = faddeeva32_inline(d * w.x, w.y);
            }
            __syncwarp();
        }
        float2 acc2[kMxQ / 2];
        float tdsp[kMxQ];
#pragma unroll
        for (int h = 0; h < kMxQ / 2; ++h) acc2[h] = make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < kMxQ; ++q) tdsp[q] = 0.f;
        for (int k = 0; k < nf; ++k) {
            const float4 f = T.fu[k];
            const float d0 = (pl0 - f.x) - f.y;
            const float2 d0s = make_float2(d0, d0), b2 = make_float2(f.z, f.z), a = make_float2(f.w, f.w);
#pragma unroll
            for (int h = 0; h < kMxQ / 2; ++h) fast_pair(d0s, offs[h], b2, a, acc2[h]);
            if (LM) {
                const float g = T.fg[k];
#pragma unroll
                for (int q = 0; q < kMxQ; ++q) {
                    const float d = d0 + 32.f * q;
                    tdsp[q] = fmaf(g * d, rcp_fast(fmaf(d, d, f.z)), tdsp[q]);
                }
            }
        }
        float tacc[kMxQ];
#pragma unroll
        for (int h = 0; h < kMxQ / 2; ++h) {
            tacc[2 * h] = acc2[h].x;
            tacc[2 * h + 1] = acc2[h].y;
        }
        for (int k = 0; k < ns; ++k) {
            const float4 u = T.su[k];
            const float4 p = T.sp[k];
            const float4 w = T.sq[k];
            if (METHOD == 3) {
                // every row: the far wing; rows holding a core point (warp-uniform): the
                // two-level continued fraction (one reciprocal) at every lane, the inner
                // points from cw, and an inner point beyond cw through faddeeva32
                const int4 r4 = T.sr[k];
                const int rlo = r4.x, rhi = r4.y, rb = r4.z - r4.x;  // inner points held in cw: [rlo, rhi] at rb + point
                const float y2 = w.y * w.y;
#pragma unroll
                for (int q = 0; q < kMxQ; ++q) {
                    const float d = ((pl0 + 32.f * q) - u.x) - u.y;
                    const float d2 = d * d;
                    const float ped = fmaf(p.x, d2, p.y);
                    const float r = rcp_fast(d2 + u.z);
                    float v = fmaf(u.w, r, ped), vd = w.z * d * r;
                    const bool core = d2 <= p.z;  // |x| <= x_far
                    if (__any_sync(kFull, core)) {
                        const float x = d * w.x;
                        const int pt = lane + 32 * q;
                        float2 fw = faddeeva_cf2(x, w.y, y2);
                        if (pt >= rlo && pt <= rhi) fw = T.cw[rb + pt];
                        else if (core && fabsf(x) + w.y < 15.f) fw = faddeeva32(x, w.y);
                        if (core) {
                            v = fmaf(p.w, fw.x, ped);
                            vd = w.w * fw.y;
                        }
                    }
                    if (d2 > cut2) v = vd = 0.f;
                    tacc[q] += v;
                    if (LM) tdsp[q] += vd;
                }
                continue;
            }
#pragma unroll
            for (int q = 0; q < kMxQ; ++q) {
                const float d = ((pl0 + 32.f * q) - u.x) - u.y;
                const float d2 = d * d;
                if (d2 > cut2) continue;
                const float ped = fmaf(p.x, d2, p.y);
                float v, vd;
                if (d2 <= p.z) {  // |x| <= x_far: Faddeeva core (Weideman-24)
                    v = fmaf(p.w, weideman24_32(d * w.x, w.y), ped);
                    vd = 0.f;
                } else {
                    const float r = rcp_fast(d2 + u.z);
                    v = fmaf(u.w, r, ped);
                    vd = w.z * d * r;
                }
                tacc[q] += v;
                if (LM) tdsp[q] += vd;
            }
        }
#pragma unroll
        for (int q = 0; q < kMxQ; ++q) {
            const float pp = pl0 + 32.f * q;
            kahan_add(sum[q], comp[q], tacc[q] + fmaf(pp, fmaf(pp, A, -2.f * B), Cc));
            if (LM) kahan_add(sumD[q], compD[q], tdsp[q]);
        }
    }
    // relmat line mixing: this species' clamped sum goes to its own row, and
    // relmat_finish_kernel adds max(sum + d_sigma, 0) once the perturbation is known
    const bool rel = prow && (sg.flags & SEG_RELMAT);
#pragma unroll
    for (int q = 0; q < kMxQ; ++q) {
        float sig = fmaxf(sum[q], 0.f);
        if (LM) sig = fmaxf(sig + sumD[q], 0.f);
        if (rel) prow[wb + 32 * q + lane] = (double)sig;
        else out_add(orow, q, lane, sig);
    }
    if (!rel) orow.wrote = true;
}

// PseudoVoigt (voigt.jl:281-313): no far-wing shortcut; p0 = (gV2, aPV, c1, c0),
// p1 = (kPV, gPV, -, -): value = aPV/(d^2 + gV2) + gPV 2^(-kPV d^2) + c1 d^2 + c0.
__device__ __forceinline__ void warp_segment_pv(const SegDev& sg, long long cnt, const LpOutMixed& lp, long long wb,
                                                float cut, float cut2, int lane, WarpTile& T, OutRow& orow) {
    constexpr float kCentre = 0.5f * (kMxWarpPts - 1);
    constexpr float kHalf = 0.5f * kMxWarpPts + 0.5f;
    long long jlo, jhi;
    warp_window(lp, sg, cnt, wb, cut, lane, jlo, jhi);
    const float pl0 = (float)lane;
    float sum[kMxQ], comp[kMxQ];
#pragma unroll
    for (int q = 0; q < kMxQ; ++q) sum[q] = comp[q] = 0.f;
    for (long long t0 = jlo; t0 < jhi; t0 += 32) {
        const int nt = (int)min(32LL, jhi - t0);
        __syncwarp();
        if (lane < nt) {
            const long long q = sg.off + t0 + lane;
            const float2 uf = lp.U[q];
            const float uh = uf.x - (float)wb;  // exact: see split_hi_lo
            const float dist = fabsf(uh - kCentre);
            const float cls = dist > cut + kHalf ? 0.f : (dist + kHalf <= cut ? 1.f : 2.f);
            T.fu[lane] = make_float4(uh, uf.y, 0.f, cls);
            T.su[lane] = lp.p0[q];
            T.sp[lane] = lp.p1[q];
        }
        __syncwarp();
        float tacc[kMxQ];
#pragma unroll
        for (int q = 0; q < kMxQ; ++q) tacc[q] = 0.f;
        for (int k = 0; k < nt; ++k) {
            const float4 u = T.fu[k];
            if (u.w == 0.f) continue;
            const float4 a0 = T.su[k];
            const float4 a1 = T.sp[k];
#pragma unroll
            for (int q = 0; q < kMxQ; ++q) {
                const float d = ((pl0 + 32.f * q) - u.x) - u.y;
                const float d2 = d * d;
                if (u.w == 2.f && d2 > cut2) continue;
                tacc[q] += fmaf(a0.y, rcp_fast(d2 + a0.x), fmaf(a1.y, exp2f(-a1.x * d2), fmaf(a0.z, d2, a0.w)));
            }
        }
#pragma unroll
        for (int q = 0; q < kMxQ; ++q) kahan_add(sum[q], comp[q], tacc[q]);
    }
#pragma unroll
    for (int q = 0; q < kMxQ; ++q) out_add(orow, q, lane, fmaxf(sum[q], 0.f));
    orow.wrote = true;
}

// PERT: segments flagged SEG_RELMAT write their clamped sums to the rows
// pert[(profile, layer)][pstride] instead of the optical depth, for
// relmat_finish_kernel (a separate instantiation, so the kernels without it are
// unchanged).
// dynamic shared memory of linesum_mixed_kernel: the warps' tiles
constexpr size_t kMxSmem = sizeof(WarpTile) * kMxWarps;

template <int METHOD, bool ANY_LM, bool PERT = false>
__global__ void __launch_bounds__(kMxThreads, ANY_LM ? 1 : 2) linesum_mixed_kernel(
    const SegDev* __restrict__ segs, const int* __restrict__ seg_count, const int2* __restrict__ pl_segs,
    LpOutMixed lp, long long n_nu, float cut_g, float* __restrict__ tau, unsigned long long* __restrict__ evald,
    double* __restrict__ pert, long long pstride) {
    extern __shared__ __align__(16) unsigned char mx_smem[];
    WarpTile* tiles = reinterpret_cast<WarpTile*>(mx_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pl = (int)blockIdx.y;
    const long long wb = (long long)blockIdx.x * kMxStrip + (long long)warp * kMxWarpPts;
    if (wb >= n_nu) return;  // no block-wide barriers below: whole warps may leave
    unsigned long long work = 0;
    const float cut2 = cut_g * cut_g;
    WarpTile& T = tiles[warp];
    OutRow orow{tau + (size_t)pl * n_nu + wb, (int)min((long long)kMxWarpPts, n_nu - wb), false};
    const int2 rng = pl_segs[pl];
    for (int s = rng.x; s < rng.x + rng.y; ++s) {
        const SegDev sg = segs[s];
        const long long cnt = seg_count[s];
        if (METHOD == 2)
            warp_segment_pv(sg, cnt, lp, wb, cut_g, cut2, lane, T, orow);
        else if (ANY_LM && (sg.flags & SEG_LM))
            warp_segment<METHOD, true>(sg, cnt, lp, wb, cut_g, cut2, lane, T, orow, work, nullptr);
        else
            warp_segment<METHOD, false>(sg, cnt, lp, wb, cut_g, cut2, lane, T, orow, work,
                                        PERT ? pert + (size_t)pl * pstride : nullptr);
    }
    if (evald && lane == 0 && work) atomicAdd(evald, work);
    if (!orow.wrote) {  // no segment stored: zero optical depth
#pragma unroll
        for (int q = 0; q < kMxQ; ++q) out_add(orow, q, lane, 0.f);
    }
}

}  // namespace irs
