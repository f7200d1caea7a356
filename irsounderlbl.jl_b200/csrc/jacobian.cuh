// jacobian.cuh -- the analytic Jacobian of forward_model on the GPU.
//
// Restates vmr_jacobian.jl:152-505 with its atoms:
//   cross-section derivatives (sigma, d/dT, d/dp, d/dvmr_self) in one pass
//                                cross_section_jacobian.jl:68-240 (jg_params_kernel,
//                                jg_linesum_kernel); VP_Y dispersive term with its
//                                analytic derivatives (the reference central-
//                                differences it, :255-322)
//   RTE Jacobian                 schwarzschild_jacobian.jl:66-266 (jg_rte_kernel)
//   channel tail K = dBT/dR . resample . ILS . dI/dx      vmr_jacobian.jl:359-503
//                                (jg_channel_kernel)
// The line sum is FP32 (the tile sums of the values Kahan-compensated, those of the derivatives
// plain), and so is the channel contraction (plain sums); the optical-depth sums,
// transmittances and radiance derivatives are FP64.
#pragma once
#include <type_traits>

#include "faddeeva.cuh"
#include "lineparams.cuh"
#include "linesum.cuh"
#include "linesum_tree32.cuh"
#include "linesum_tree64.cuh"
#include "rte_ils.cuh"

namespace irs {

constexpr int kJgMaxOut = 11;  // tau, T_lo, T_hi, and (lo, hi) for up to 4 retrieved species

// Per-line primitives (FP64 physics, stored FP32 except the sorted key), grid units.  q2
// and q3 are written only for segments that need them (SEG_NEED_P, SEG_NEED_V), q4 with
// line mixing.
struct JgOut {
    double* V;              // sorted key
    float2* U;              // shifted centre as hi + lo (split_hi_lo)
    float* df;              // core half-width x_far / fx
    float4 *q0;             // An, fx, y, Hc
    float4 *q1;             // An_T, fx_T, y_T, Hc_T
    float4 *q2;             // y_p, u_p, Hc_p, -
    float4 *q3;             // y_v, u_v, Hc_v, -
    float4 *q4;             // Yw, Yw_T, Yw_p, -
};
constexpr size_t kJgLineBytes = 8 + 8 + 4 + 5 * 16;

// cross_section_jacobian.jl:43-56 in FP64 (H and its x, y gradient)
__device__ __forceinline__ void h_and_grad64(double x, double y, double x_far, double& H, double& Hx, double& Hy) {
    if (fabs(x) > x_far) {
        const double d = x * x + y * y, d2 = d * d;
        H = y * kInvSqrtPi / d;
        Hx = -2.0 * x * y * kInvSqrtPi / d2;
        Hy = kInvSqrtPi * (x * x - y * y) / d2;
        return;
    }
    const double2 w = faddeeva64(x, y);
    H = w.x;
    Hx = -2.0 * x * w.x + 2.0 * y * w.y;
    Hy = 2.0 * (x * w.y + y * w.x) - 2.0 * kInvSqrtPi;
}

// partition.jl:52-66
__device__ __forceinline__ double tips_slope(const TipsDev& t, int idx, double T) {
    const double* q = t.q + (size_t)idx * t.stride;
    const int lo = (int)floor(T) - t.tmin[idx] + 1, hi = lo + 1;
    if (lo < 1 || hi > t.n[idx]) return 0.0;
    return q[hi - 1] - q[lo - 1];
}

// One thread per (line, segment); no DPTMIN (the Jacobian freezes the line set,
// vmr_jacobian.jl:188-201).  cross_section_jacobian.jl:198-236.
__global__ void __launch_bounds__(256) jg_params_kernel(const SegDev* __restrict__ segs,
                                                        const ListDev* __restrict__ lists, TipsDev tp,
                                                        LpConfig cfg, JgOut o, unsigned* __restrict__ core_reach) {
    const SegDev sg = segs[blockIdx.y];
    const ListDev L = lists[sg.list];
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= L.n) return;
    const long long slot = sg.off + j;
    const int mol = L.mol;
    const double T = sg.T, p = sg.p_atm, vs = sg.vs, c = cfg.cutoff, dg = cfg.dnu_g, co = sg.coef;
    const double nu = L.nu[j], n_air = L.nair[j];
    const double n_self = mol == 1 ? 0.95 : (mol == 2 ? 0.75 : n_air);
    const double d_air = L.delta[j], d_self = mol == 1 ? 0.002 : (mol == 2 ? -0.003 : 0.0);
    const double nu0 = nu + (d_air * (1.0 - vs) + d_self * vs) * p;
    const double dn0p = d_air * (1.0 - vs) + d_self * vs, dn0v = (d_self - d_air) * p;
    // temperature_scaled_intensity_deriv, broadening.jl:112-128
    const int ti = L.tips[j];
    const double c2 = 1.4387752;
    double Qr, dlnQ;
    if (ti >= 0) {
        const double QT = tips_lookup(tp, ti, T);
        Qr = tips_lookup(tp, ti, 296.0) / QT;
        dlnQ = tips_slope(tp, ti, T) / QT;
    } else {
        Qr = 296.0 / T;
        dlnQ = (1.0 / 296.0) / (T / 296.0);
    }
    const double stim = (1.0 - exp(-c2 * nu / T)) / (1.0 - exp(-c2 * nu / 296.0));
    const double S = L.S296[j] * Qr * exp(-c2 * L.E[j] * (1.0 / T - 1.0 / 296.0)) * stim;
    const double a = c2 * nu;
    const double dS = S * (-dlnQ + c2 * L.E[j] / (T * T) - (a / (T * T)) / (exp(a / T) - 1.0));
    // pressure_broadened_width_deriv, broadening.jl:62-78
    const double tr = 296.0 / T;
    const double ac = pow(tr, n_air) * L.gair[j], bc = pow(tr, n_self) * L.gself[j];
    const double A = ac * (1.0 - vs) * p, B = bc * vs * p;
    const double gl = A + B, dglT = -(n_air * A + n_self * B) / T;
    const double gd0 = nu * 3.58126e-7 * sqrt(T / mol_mass(mol)), dgd = gd0 / (2.0 * T);
    const double gd = fmax(gd0, 1e-10);
    const double f = kSqrtLn2 / gd, df = -f * (dgd / gd);
    const double dglp = p > 0.0 ? gl / p : ac * (1.0 - vs) + bc * vs, dglv = (bc - ac) * p;
    const double y = gl * f, dyT = dglT * f + gl * df, dyp = dglp * f, dyv = dglv * f;
    const double Sn = S * f * kInvSqrtPi, dSnT = (dS * f + S * df) * kInvSqrtPi;
    double Hc, Hcx, Hcy;
    h_and_grad64(c * f, y, cfg.x_far, Hc, Hcx, Hcy);
    const double dHcT = Hcx * (c * df) + Hcy * dyT, dHcp = Hcy * dyp, dHcv = Hcy * dyv;
    double Yw = 0.0, YwT = 0.0, Ywp = 0.0;
    if ((sg.flags & SEG_LM) && L.has_y0) {  // line_mixing.jl:1193-1220 with Y(T) = y0 (296/T)^0.75
        const double Y = L.y0[j] * pow(296.0 / T, 0.75);
        if (Y != 0.0 && S > 0.0) {
            const double YT = -0.75 * Y / T;
            Yw = Y * p * Sn * co;
            YwT = (YT * Sn + Y * dSnT) * p * co;
            Ywp = Y * Sn * co;
        }
    }
    o.V[slot] = (nu - cfg.grid0) / dg;
    o.U[slot] = split_hi_lo((nu0 - cfg.grid0) / dg, cfg.u_gran, 1.0 / cfg.u_gran);
    o.df[slot] = (float)fmin(cfg.x_far / (f * dg), 1.0e30);
    o.q0[slot] = make_float4((float)(Sn * co), (float)(f * dg), (float)y, (float)Hc);
    o.q1[slot] = make_float4((float)(dSnT * co), (float)(df * dg), (float)dyT, (float)dHcT);
    if (sg.flags & (SEG_NEED_P | SEG_NEED_V)) {
        o.q2[slot] = make_float4((float)dyp, (float)(dn0p / dg), (float)dHcp, 0.f);
        o.q3[slot] = make_float4((float)dyv, (float)(dn0v / dg), (float)dHcv, 0.f);
    }
    if (sg.flags & SEG_LM) o.q4[slot] = make_float4((float)Yw, (float)YwT, (float)Ywp, 0.f);
    if (core_reach) {  // the segment's largest core half-width (non-negative floats order as their bits)
        const unsigned mask = __activemask();
        const unsigned r = __reduce_max_sync(mask, __float_as_uint((float)fmin(cfg.x_far / (f * dg), 1.0e30)));
        if ((int)(threadIdx.x & 31) == __ffs(mask) - 1) atomicMax(&core_reach[blockIdx.y], r);
    }
}

// ------------------------------------------------------------------ line sum
constexpr int kJgQ = 4;                        // points per lane
constexpr int kJgWarpPts = 32 * kJgQ;          // 128 points per warp: a leaf of the tree
constexpr int kJgWarps = 8;
static_assert(kJgWarpPts == kTrLeaf, "one warp per leaf");

// Segment weights onto the layer channels: channel o += w[0] s + w[1] s_T + w[2] s_p + w[3]
// s_v, for channels 0..2 (tau, T_lo, T_hi) and, for a retrieved species, its two (lo, hi) at
// 3 + 2 r for the bits r of retr.
struct SegW {
    float base[3][4], pair[2][4];
    unsigned retr;
};

// The sums of a segment: NS of (value, d/dT, d/dp, d/dv_self), and with line mixing the
// dispersive value, d/dT and (NS >= 3) d/dp.  Only the channels of a retrieved species read
// d/dp, and only those of water d/dv (SegW): the other segments sum two terms a pair
// instead of four (SEG_NEED_P, SEG_NEED_V).
//
// Per pair of the general form: H-ped and its derivatives; x = d fx, y; P = An Hc.
// Far wing: H = y/(sqrt(pi)(x^2+y^2)); core: FP32 Faddeeva and its gradient (H_x, H_y).
template <bool LM, int NS>
__device__ __forceinline__ void jg_core_terms(float d, float2 w, float2 gr, const float4& q0, const float4& q1, const float4& q2,
                                              const float4& q3, const float4& q4, float t[7]) {
    const float An = q0.x, fx = q0.y, xT = d * q1.y, Hx = gr.x, Hy = gr.y;
    t[0] = An * w.x;
    t[1] = q1.x * w.x + An * (Hx * xT + Hy * q1.z);
    if (NS >= 3) t[2] = An * (Hy * q2.x - Hx * (fx * q2.y));
    if (NS >= 4) t[3] = An * (Hy * q3.x - Hx * (fx * q3.y));
    if (LM) {  // L = Im w: L_x = -H_y, L_y = H_x
        t[4] = q4.x * w.y;
        t[5] = q4.y * w.y + q4.x * (Hx * q1.z - Hy * xT);
        if (NS >= 3) t[6] = q4.z * w.y + q4.x * (Hy * (fx * q2.y) + Hx * q2.x);
    }
}

// The general form of a pair, pedestal included: (H - pf Hc) and its derivatives, the wing
// from x and y themselves, so that where H and the pedestal nearly cancel (narrow cutoffs)
// they carry the same roundings.
template <bool LM, int NS>
__device__ __forceinline__ void jg_pair(float d, bool core, const float4& q0, const float4& q1, const float4& q2,
                                        const float4& q3, const float4& q4, float icut2, float t[7]) {
    const float An = q0.x, fx = q0.y, y = q0.z, Hc = q0.w, x = d * fx, xT = d * q1.y;
    float2 w, gr;
    if (core) {
        w = faddeeva32_grad(x, y, gr);
    } else {
        constexpr float k = (float)kInvSqrtPi;
        const float r = rcp_approx32(fmaf(x, x, y * y)), r2 = r * r;
        w = make_float2(y * k * r, x * k * r);
        gr = make_float2(-2.f * x * y * k * r2, k * (x * x - y * y) * r2);
    }
    // pedestal (2 - (d/cut)^2) Hc and its derivatives; the factor moves with the centre
    const float pf = 2.f - d * d * icut2, Hm = w.x - pf * Hc;
    t[0] = An * Hm;
    t[1] = q1.x * Hm + An * (gr.x * xT + gr.y * q1.z - pf * q1.w);
    if (NS >= 3) t[2] = An * (gr.y * q2.x - gr.x * (fx * q2.y) - (2.f * d * q2.y * icut2 * Hc + pf * q2.z));
    if (NS >= 4) t[3] = An * (gr.y * q3.x - gr.x * (fx * q3.y) - (2.f * d * q3.y * icut2 * Hc + pf * q3.z));
    if (LM) {
        t[4] = q4.x * w.y;
        t[5] = q4.y * w.y + q4.x * (gr.x * q1.z - gr.y * xT);
        if (NS >= 3) t[6] = q4.z * w.y + q4.x * (gr.y * (fx * q2.y) + gr.x * q2.x);
    }
}

// The far wing of a line in rho = 1/(d^2 + b2), d the offset in grid units and b2 = (y/fx)^2:
//   s  = a_s rho
//   sT = aT1 rho + aT2 rho^2
//   sp = ap1 rho + ap2 rho^2 + ap3 d rho^2        (sv likewise)
//   D  = cD d rho,  DT = cT1 d rho + cT2 d rho^2,
//   Dp = cp1 d rho + cp2 rho + cp3 rho^2 + cp4 d rho^2          (line mixing)
// which follow from H = y/(sqrt(pi)(x^2+y^2)), its x and y derivatives and x = d fx
// (x_T = d fx_T, x_p = -fx u_p).  f0 = (-, -, b2, a_s), f1 = (aT1, aT2, ap1, ap2),
// f2 = (ap3, av1, av2, av3), l0 = (cD, cT1, cT2, cp1), l1 = (cp2, cp3, cp4, -), and the
// pedestal scales P[o] of -P pf, pf = 2 - (i - u)^2 / c^2 (pf also moves with the centre for
// d/dp and d/dv).  1/fx by the MUFU reciprocal (about 1 ulp).
template <bool LM, int NS>
__device__ __forceinline__ void jg_wing_coeffs(const float4& a0, const float4& a1, const float4& a2,
                                               const float4& a3, const float4& a4, float4& f0, float4& f1,
                                               float4& f2, float4& l0, float4& l1, float P[4]) {
    constexpr float k = (float)kInvSqrtPi;
    const float An = a0.x, fx = a0.y, y = a0.z, Hc = a0.w;
    const float AnT = a1.x, fxT = a1.y, yT = a1.z, HcT = a1.w;
    const float ifx = rcp_fast(fx);
    const float gg = ifx * ifx, b2 = y * y * gg, Aky = An * k * y, Akg = An * k * gg;
    const float r_fx = fxT * ifx;
    // floored: at a centre on a grid point an unbroadened line's d^2 + b2 would be 0, and the
    // reciprocal is shared with another point (jg_offsets)
    f0 = make_float4(0.f, 0.f, fmaxf(b2, 1e-18f), Aky * gg);
    f1 = make_float4(gg * k * (AnT * y + An * yT) - 2.f * Aky * r_fx * gg, 2.f * Aky * b2 * r_fx * gg - 2.f * Akg * yT * b2,
                     0.f, 0.f);
    P[0] = An * Hc;
    P[1] = AnT * Hc + An * HcT;
    if (NS >= 3) {
        f1.z = Akg * a2.x;
        f1.w = -2.f * Akg * a2.x * b2;
        f2.x = 2.f * Aky * a2.y * gg;
        P[2] = An * a2.z;
    }
    if (NS >= 4) {
        f2.y = Akg * a3.x;
        f2.z = -2.f * Akg * a3.x * b2;
        f2.w = 2.f * Aky * a3.y * gg;
        P[3] = An * a3.z;
    }
    if (LM) {
        const float Yw = a4.x, YwT = a4.y, Ywp = a4.z;
        l0 = make_float4(Yw * k * ifx, YwT * k * ifx - Yw * k * gg * fxT,
                         2.f * Yw * k * gg * fxT * b2 - 2.f * Yw * k * y * fx * yT * gg * gg, Ywp * k * ifx);
        if (NS >= 3)
            l1 = make_float4(Yw * k * a2.y * ifx, -2.f * Yw * k * a2.y * b2 * ifx, -2.f * Yw * k * y * fx * a2.x * gg * gg, 0.f);
    }
}

// A line's pedestals as quadratics in the point index i (value A + B i + C i^2, the
// centre u in the same coordinates as i)
template <int NS>
__device__ __forceinline__ void jg_pedestal_quadratics(const float P[4], const float4& a0, const float4& a2,
                                                       const float4& a3, float u, float icut2, float pA[NS],
                                                       float pB[NS], float pC[NS]) {
    const float e0 = 2.f - u * u * icut2, e1 = 2.f * u * icut2;
#pragma unroll
    for (int o = 0; o < NS; ++o) {
        pA[o] = -P[o] * e0;
        pB[o] = -P[o] * e1;
        pC[o] = P[o] * icut2;
    }
    const float shp = 2.f * a0.x * a0.w * icut2;  // pf_p = 2 (i - u) u_p / c^2
    if (NS >= 3) {
        pA[2] += shp * a2.y * u;
        pB[2] -= shp * a2.y;
    }
    if (NS >= 4) {
        pA[3] += shp * a3.y * u;
        pB[3] -= shp * a3.y;
    }
}

// adds the wing's terms of two points (packed): dn their offsets, rho their reciprocals
template <bool LM, int NS>
__device__ __forceinline__ void jg_wing_add(float2 dn, float2 rho, const float4& f0, const float4& f1, const float4& f2,
                                            const float4& l0, const float4& l1, float2 v[7]) {
    const float2 rho2 = __fmul2_rn(rho, rho);
    v[0] = __ffma2_rn(make_float2(f0.w, f0.w), rho, v[0]);
    v[1] = __ffma2_rn(make_float2(f1.x, f1.x), rho, __ffma2_rn(make_float2(f1.y, f1.y), rho2, v[1]));
    if (NS >= 3 || LM) {
        const float2 drho2 = __fmul2_rn(dn, rho2);
        if (NS >= 3)
            v[2] = __ffma2_rn(make_float2(f1.z, f1.z), rho,
                              __ffma2_rn(make_float2(f1.w, f1.w), rho2, __ffma2_rn(make_float2(f2.x, f2.x), drho2, v[2])));
        if (NS >= 4)
            v[3] = __ffma2_rn(make_float2(f2.y, f2.y), rho,
                              __ffma2_rn(make_float2(f2.z, f2.z), rho2, __ffma2_rn(make_float2(f2.w, f2.w), drho2, v[3])));
        if (LM) {
            const float2 drho = __fmul2_rn(dn, rho);
            v[4] = __ffma2_rn(make_float2(l0.x, l0.x), drho, v[4]);
            v[5] = __ffma2_rn(make_float2(l0.y, l0.y), drho, __ffma2_rn(make_float2(l0.z, l0.z), drho2, v[5]));
            if (NS >= 3)
                v[6] = __ffma2_rn(make_float2(l0.w, l0.w), drho,
                                  __ffma2_rn(make_float2(l1.x, l1.x), rho,
                                             __ffma2_rn(make_float2(l1.y, l1.y), rho2,
                                                        __ffma2_rn(make_float2(l1.z, l1.z), drho2, v[6]))));
        }
    }
}
// offsets and reciprocals of two points: xn their positions (natural), xs swapped; one MUFU
// reciprocal of the product of the swapped denominators serves both
__device__ __forceinline__ void jg_offsets(float2 xn, float2 xs, float uh, float ul, float b2, float2& dn, float2& rho) {
    const float2 nu_ = make_float2(-uh, -uh), nl = make_float2(-ul, -ul);
    dn = __fadd2_rn(__fadd2_rn(xn, nu_), nl);
    const float2 ds = __fadd2_rn(__fadd2_rn(xs, nu_), nl);
    const float2 es = __ffma2_rn(ds, ds, make_float2(b2, b2));
    const float R = rcp_fast(es.x * es.y);
    rho = __fmul2_rn(es, make_float2(R, R));
}

// The kinds of segments by their sums.  Line mixing is CO2's and d/dv_self water's, so they
// do not meet.
enum { kJg2, kJg3, kJg4, kJgLm2, kJgLm3, kJgModes };
__host__ __device__ inline int jg_mode(int flags) {
    if (flags & SEG_LM) return flags & (SEG_NEED_P | SEG_NEED_V) ? kJgLm3 : kJgLm2;
    return flags & SEG_NEED_V ? kJg4 : flags & SEG_NEED_P ? kJg3 : kJg2;
}

// sums in use: value, d/dT, [d/dp], [d/dv], then with line mixing D, D_T, [D_p]
template <bool LM, int NS>
__device__ __forceinline__ constexpr bool jg_used(int c) {
    return c < NS || (LM && c >= 4 && c < (NS >= 3 ? 7 : 6));
}

// ------------------------------------------------------------------ far lines
// One CTA per (strip of 4096 points, segment): the tree's levels from the strip down to the
// 32 leaves, each level's own far lines (tree_list) spread over the warps, then the parents'
// node values through M (FP64) and the next level.  Leaves far[(segment, leaf)][sum][node]
// and the leaf's ranges.  Against the two levels it replaces (1024-point strips from 1024
// points, then every warp's 8 nodes from 320 points): see the figures at jg_linesum_kernel.
struct JgStage {
    float4 f0[32], f1[32], f2[32];
};
struct JgStageLm {
    float4 l0[32], l1[32];
};
__host__ __device__ constexpr int jg_sums(bool lm) { return lm ? 7 : 4; }
constexpr size_t jg_tree_smem(bool lm) {
    return (sizeof(JgStage) + (lm ? sizeof(JgStageLm) : 0)) * kJgWarps +
           (size_t)2 * (kTrLeaves / 2) * jg_sums(lm) * kTrNodes * sizeof(double) +
           (size_t)kTrLeaves * jg_sums(lm) * kTrNodes * sizeof(float) + 2 * (kTrLeaves / 2) * sizeof(int4);
}

// one warp's share of a block's far lines at its nodes, written to part[sum][node]
template <bool LM, int NS>
__device__ __forceinline__ void jg_block(const JgOut& g, long long off, const TreeList& TL, int first, int step, float cb,
                                         float h, float icut2, int lane, JgStage& T, JgStageLm* TLm,
                                         float (*__restrict__ part)[kTrNodes]) {
    const float2 xp = make_float2(h * tree_node_f(lane & 7), h * tree_node_f((lane & 7) + 8));
    const float2 xps = make_float2(xp.y, xp.x);
    float2 v[7], vs[2], vc[2];  // the value (c = 0) and D (c = 4) compensated over tiles
#pragma unroll
    for (int c = 0; c < 7; ++c) v[c] = make_float2(0.f, 0.f);
    vs[0] = vs[1] = vc[0] = vc[1] = make_float2(0.f, 0.f);
    float QA[NS], QB[NS], QC[NS], QAc = 0.f, QBc = 0.f, QCc = 0.f;
#pragma unroll
    for (int o = 0; o < NS; ++o) QA[o] = QB[o] = QC[o] = 0.f;
    for (int t0 = 32 * first; t0 < TL.n; t0 += 32 * step) {
        const int nt = min(32, TL.n - t0);
        __syncwarp();
        if (lane < nt) {
            const long long q = off + tree_line(TL, t0 + lane);
            const float2 uf = g.U[q];
            const float uh = (uf.x - cb) - (h - 0.5f), ul = uf.y;  // exact: see split_hi_lo
            const float4 a0 = g.q0[q], a1 = g.q1[q];
            float4 a2, a3, a4, f0, f1, f2, l0, l1;
            if (NS >= 3) { a2 = g.q2[q]; a3 = g.q3[q]; }
            if (LM) a4 = g.q4[q];
            float P[4], pA[NS], pB[NS], pC[NS];
            jg_wing_coeffs<LM, NS>(a0, a1, a2, a3, a4, f0, f1, f2, l0, l1, P);
            T.f0[lane] = make_float4(uh, ul, f0.z, f0.w);
            T.f1[lane] = f1;
            if (NS >= 3) T.f2[lane] = f2;
            if (LM) {
                TLm->l0[lane] = l0;
                if (NS >= 3) TLm->l1[lane] = l1;
            }
            jg_pedestal_quadratics<NS>(P, a0, a2, a3, uh + ul, icut2, pA, pB, pC);
            kahan_add(QA[0], QAc, pA[0]);
            kahan_add(QB[0], QBc, pB[0]);
            kahan_add(QC[0], QCc, pC[0]);
#pragma unroll
            for (int o = 1; o < NS; ++o) {
                QA[o] += pA[o];
                QB[o] += pB[o];
                QC[o] += pC[o];
            }
        }
        __syncwarp();
        for (int k = lane >> 3; k < nt; k += 4) {  // lane: nodes lane % 8 and + 8, every fourth line
            const float4 f0 = T.f0[k], f1 = T.f1[k];
            float4 f2, l0, l1;
            if (NS >= 3) f2 = T.f2[k];
            if (LM) {
                l0 = TLm->l0[k];
                if (NS >= 3) l1 = TLm->l1[k];
            }
            float2 dn, rho;
            jg_offsets(xp, xps, f0.x, f0.y, f0.z, dn, rho);
            jg_wing_add<LM, NS>(dn, rho, f0, f1, f2, l0, l1, v);
        }
#pragma unroll
        for (int c = 0; c < (LM ? 2 : 1); ++c) {
            kahan_add(vs[c].x, vc[c].x, v[4 * c].x);
            kahan_add(vs[c].y, vc[c].y, v[4 * c].y);
            v[4 * c] = make_float2(0.f, 0.f);
        }
    }
    v[0] = vs[0];
    if (LM) v[4] = vs[1];
    const float xk = (lane & 8) ? xp.y : xp.x;  // node lane % 16
#pragma unroll
    for (int c = 0; c < 7; ++c) {
        if (!jg_used<LM, NS>(c)) continue;
        float2 x = v[c];
        x.x += __shfl_xor_sync(kFull, x.x, 8);
        x.y += __shfl_xor_sync(kFull, x.y, 8);
        x.x += __shfl_xor_sync(kFull, x.x, 16);
        x.y += __shfl_xor_sync(kFull, x.y, 16);
        float val = (lane & 8) ? x.y : x.x;
        if (c < NS) {
            const float A = warp_sum(c == 0 ? QA[0] - QAc : QA[c]), B = warp_sum(c == 0 ? QB[0] - QBc : QB[c]);
            const float C = warp_sum(c == 0 ? QC[0] - QCc : QC[c]);
            val += fmaf(xk, fmaf(xk, C, B), A);
        }
        if (lane < kTrNodes) part[c][lane] = val;
    }
}

template <bool ANY_LM, bool LM, int NS>
__device__ __forceinline__ void jg_tree_segment(const JgOut& g, long long off, const CellIndex& ci, const int* row,
                                                float cut, float m, float reach, long long n_nu,
                                                const TreeTables* __restrict__ tab, float* __restrict__ far,
                                                int4* __restrict__ ranges, unsigned char* smem) {
    constexpr int NC = jg_sums(ANY_LM);
    JgStage* tiles = (JgStage*)smem;
    JgStageLm* tiles_lm = (JgStageLm*)(tiles + kJgWarps);
    double* F = (double*)(ANY_LM ? (void*)(tiles_lm + kJgWarps) : (void*)tiles_lm);  // [2][16][NC][16]
    float(*part)[NC][kTrNodes] = (float(*)[NC][kTrNodes])(F + 2 * (kTrLeaves / 2) * NC * kTrNodes);  // [32]
    int4* rg = (int4*)(part + kTrLeaves);  // [2][16]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long sb = (long long)blockIdx.x * kTrStrip;
    const float icut2 = 1.f / (cut * cut);
#pragma unroll 1
    for (int l = 0; l < kTrLevels; ++l) {
        const int nb = 1 << l, wpb = l < 3 ? kJgWarps >> l : 1, bpw = l < 3 ? 1 : nb / kJgWarps;
        const float h = (float)(kTrStrip >> (l + 1));
        int4* up = rg + ((l + 1) & 1) * (kTrLeaves / 2);
        for (int i = 0; i < bpw; ++i) {
            const int b = l < 3 ? warp / wpb : warp * bpw + i;
            const long long cb = sb + (long long)b * (kTrStrip >> l);
            if (cb >= n_nu) break;  // warp-uniform
            const int4 u = l ? up[b >> 1] : make_int4(0, 0, 0, 0);
            const int4 own = tree_inside(tree_ranges(ci, row, (float)cb, h, cut, m, reach), u);
            jg_block<LM, NS>(g, off, tree_list(own, u), l < 3 ? warp % wpb : 0, wpb, (float)cb, h, icut2, lane,
                             tiles[warp], tiles_lm + warp, part[l < 3 ? warp : b]);
            if (lane == 0 && (l >= 3 || warp % wpb == 0)) {
                if (l + 1 < kTrLevels) rg[(l & 1) * (kTrLeaves / 2) + b] = own;
                else ranges[b] = own;
            }
        }
        __syncthreads();
        double* Fo = F + (size_t)(l & 1) * (kTrLeaves / 2) * NC * kTrNodes;
        const double* Fp = F + (size_t)((l + 1) & 1) * (kTrLeaves / 2) * NC * kTrNodes;
        for (int i = threadIdx.x; i < nb * NC * kTrNodes; i += kJgWarps * 32) {
            const int j = i % kTrNodes, c = (i / kTrNodes) % NC, b = i / (kTrNodes * NC);
            if (!jg_used<LM, NS>(c) || sb + (long long)b * (kTrStrip >> l) >= n_nu) continue;
            double v = 0.0;
            for (int w = 0; w < wpb; ++w) v += (double)part[b * wpb + w][c][j];
            if (l) {
                const double* fp = Fp + ((b >> 1) * NC + c) * kTrNodes;
#pragma unroll
                for (int k = 0; k < kTrNodes; ++k) v = fma(fp[k], tab->M[b & 1][k][j], v);
            }
            if (l + 1 < kTrLevels) Fo[(b * NC + c) * kTrNodes + j] = v;
            else far[(b * NC + c) * kTrNodes + j] = (float)v;
        }
        __syncthreads();
    }
}

template <bool ANY_LM>
__global__ void __launch_bounds__(kJgWarps * 32, 3) jg_tree_kernel(
    const SegDev* __restrict__ segs, const unsigned* __restrict__ core_reach, CellIndex ci, JgOut g, float cut_g,
    long long n_nu, int n_leaves, const TreeTables* __restrict__ tab, float* __restrict__ far,
    int4* __restrict__ ranges, int seg0) {
    extern __shared__ __align__(16) unsigned char jg_tree_sh[];
    const int s = seg0 + (int)blockIdx.y;
    const SegDev sg = segs[s];
    const size_t cell = (size_t)blockIdx.y * n_leaves + (size_t)blockIdx.x * kTrLeaves;
    float* fo = far + cell * jg_sums(ANY_LM) * kTrNodes;
    int4* ro = ranges + cell;
    const int* row = ci.idx + (size_t)sg.list * ci.n;
    const float m = (float)sg.margin_g, reach = __uint_as_float(core_reach[s]);
    const int mode = jg_mode(sg.flags);
#define IRS_JT(LMX, NS) jg_tree_segment<ANY_LM, LMX, NS>(g, sg.off, ci, row, cut_g, m, reach, n_nu, tab, fo, ro, jg_tree_sh)
    if (ANY_LM && mode == kJgLm2) IRS_JT(ANY_LM, 2);  // block-uniform
    else if (ANY_LM && mode == kJgLm3) IRS_JT(ANY_LM, 3);
    else if (mode == kJg4) IRS_JT(false, 4);
    else if (mode == kJg3) IRS_JT(false, 3);
    else IRS_JT(false, 2);
#undef IRS_JT
}

// ------------------------------------------------------------------ near lines
// Warp-private staging of one tile (32 lines), ordered by class: fast lines (wing at every
// point, inside the cutoff: packed pairs of points, pedestals as quadratics), cutoff-edge
// lines (wing, the cutoff falls among the points), core lines (inside the cutoff, the
// Faddeeva core reaches some points: only the 32-point rows that it reaches take it; their
// pedestals are quadratics too, so the cutoff has to be 8 times their reach, where the
// pedestal is under 1/64 of the line's value at any point and cancels nothing), and general
// ones (core and cutoff edge, or a narrow cutoff: H - pedestal per pair).  The inner points of core lines
// (|x| + y < 15, the CF4 and Weideman branches) are evaluated lane-parallel per tile into
// cw, as in the forward line sum.
constexpr int kJgBuf = 128;
template <bool LM>
struct JgTile {
    float4 f0[32], f1[32], f2[32];  // uh, ul, b2, a_s; wing coefficients
    float4 q0[32], q1[32];          // core, general: primitives; edge: pedestals, their centre terms
    float4 q2[32], q3[32];
    float4 l0[LM ? 32 : 1], l1[LM ? 32 : 1], q4[LM ? 32 : 1];
    int4 cr[32];                    // core lines: inner points [x, y], offset in cw, core rows (lo | hi << 8)
    float df2[32];
    float2 cw[kJgBuf];
};

template <bool LM, int NS>
__device__ __forceinline__ void jg_segment(const SegDev& sg, const JgOut& g, long long wb, int4 own, int wlo, int whi,
                                           float cut, int lane, JgTile<LM>& T, const float (*__restrict__ Lw)[kTrLeaf],
                                           const float* __restrict__ gfar, const SegW& W,
                                           const double* __restrict__ prow, long long pstride,
                                           float* __restrict__ acc) {
    constexpr float kCentre = 0.5f * (kJgWarpPts - 1);
    constexpr float kHalf = 0.5f * kJgWarpPts + 0.5f;
    const float cut2 = cut * cut, icut2 = 1.f / cut2;
    const float pl0 = (float)lane;
    const unsigned lt = (1u << lane) - 1u;
    float2 S[2], C[2], SD[2], CD[2], V[2][7];  // value (compensated), dispersive value, the derivatives
    float2 xn[2], xs[2];                       // the lane's points of rows (2h, 2h + 1), natural and swapped
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        S[h] = C[h] = SD[h] = CD[h] = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 7; ++c) V[h][c] = make_float2(0.f, 0.f);
        xn[h] = make_float2(pl0 + 64.f * h, pl0 + 64.f * h + 32.f);
        xs[h] = make_float2(xn[h].y, xn[h].x);
    }
    float QA[NS], QB[NS], QC[NS], QAc = 0.f, QBc = 0.f, QCc = 0.f;
#pragma unroll
    for (int o = 0; o < NS; ++o) QA[o] = QB[o] = QC[o] = 0.f;
    // the lines not taken by the far field: [wlo, own.x), [own.y, own.z), [own.w, whi)
    const int n1 = max(own.x - wlo, 0), n2 = n1 + (own.z - own.y), n = n2 + max(whi - own.w, 0);
    for (int t0 = 0; t0 < n; t0 += 32) {
        const int nt = min(32, n - t0), t = t0 + lane;
        int cls = 0;
        float uh = 0.f, ul = 0.f, df = 0.f;
        float4 a0, a1, a2, a3, a4;
        if (lane < nt) {
            const long long q = sg.off + (t < n1 ? wlo + t : t < n2 ? own.y + (t - n1) : own.w + (t - n2));
            const float2 uf = g.U[q];
            uh = uf.x - (float)wb;  // exact: see split_hi_lo
            ul = uf.y;
            df = g.df[q];
            const float dist = fabsf(uh - kCentre);
            const bool wing = dist > df + kHalf, in = dist + kHalf <= cut;
            cls = dist > cut + kHalf ? 0 : wing ? (in ? 1 : 2) : (in && cut >= 8.f * (df + kHalf) ? 3 : 4);
            if (cls) {
                a0 = g.q0[q];
                a1 = g.q1[q];
                if (NS >= 3) { a2 = g.q2[q]; a3 = g.q3[q]; }
                if (LM) a4 = g.q4[q];
            }
        }
        const unsigned m1 = __ballot_sync(kFull, cls == 1), m2 = __ballot_sync(kFull, cls == 2);
        const unsigned m3 = __ballot_sync(kFull, cls == 3), m4 = __ballot_sync(kFull, cls == 4);
        const int e1 = __popc(m1), e2 = e1 + __popc(m2), e3 = e2 + __popc(m3), e4 = e3 + __popc(m4);
        // inner points of the core lines and their offsets in cw (a warp scan)
        int nin = 0, plo = 1, coff = 0, cfit = 0;
        if (m3) {  // warp-uniform
            if (cls == 3 && a0.z < 15.f) {
                const float hw = (15.f - a0.z) / a0.y + 1.f, c = uh + ul;
                const float lo = fmaxf(c - hw, 0.f), hi = fminf(c + hw, (float)(kJgWarpPts - 1));
                if (lo <= hi) {
                    plo = (int)ceilf(lo);
                    nin = max((int)floorf(hi) - plo + 1, 0);
                }
            }
            int inc = nin;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(kFull, inc, d);
                if (lane >= d) inc += v;
            }
            coff = inc - nin;
            const unsigned ov = __ballot_sync(kFull, inc > kJgBuf && nin > 0);
            cfit = ov ? __shfl_sync(kFull, coff, __ffs(ov) - 1) : __shfl_sync(kFull, inc, 31);
            if (inc > kJgBuf) nin = 0;  // beyond the buffer: per point
        }
        __syncwarp();
        if (cls) {
            const int pos = cls == 1 ? __popc(m1 & lt) : cls == 2 ? e1 + __popc(m2 & lt)
                          : cls == 3 ? e2 + __popc(m3 & lt) : e3 + __popc(m4 & lt);
            float4 f0, f1, f2, l0, l1;
            float P[4];
            jg_wing_coeffs<LM, NS>(a0, a1, a2, a3, a4, f0, f1, f2, l0, l1, P);
            T.f0[pos] = make_float4(uh, ul, f0.z, f0.w);
            T.f1[pos] = f1;
            if (NS >= 3) T.f2[pos] = f2;
            if (LM) {
                T.l0[pos] = l0;
                if (NS >= 3) T.l1[pos] = l1;
            }
            if (cls & 1) {  // inside the cutoff at every point
                float pA[NS], pB[NS], pC[NS];
                jg_pedestal_quadratics<NS>(P, a0, a2, a3, uh + ul, icut2, pA, pB, pC);
                kahan_add(QA[0], QAc, pA[0]);
                kahan_add(QB[0], QBc, pB[0]);
                kahan_add(QC[0], QCc, pC[0]);
#pragma unroll
                for (int o = 1; o < NS; ++o) {
                    QA[o] += pA[o];
                    QB[o] += pB[o];
                    QC[o] += pC[o];
                }
            }
            if (cls == 2) {
                T.q0[pos] = make_float4(P[0], P[1], NS >= 3 ? P[2] : 0.f, NS >= 4 ? P[3] : 0.f);
                if (NS >= 3)
                    T.q1[pos] = make_float4(2.f * a2.y * icut2 * P[0], 2.f * a3.y * icut2 * P[0], 0.f, 0.f);
            } else if (cls >= 3) {
                T.q0[pos] = a0;
                T.q1[pos] = a1;
                if (NS >= 3) {
                    T.q2[pos] = a2;
                    T.q3[pos] = a3;
                }
                if (LM) T.q4[pos] = a4;
                T.df2[pos] = df * df;
                const float c = uh + ul;
                const int rl = (int)fminf(fmaxf((c - df) * (1.f / 32.f) - 0.1f, 0.f), 4.f);  // rows the core reaches
                const int rh = (int)fminf(fmaxf((c + df) * (1.f / 32.f) + 0.1f, -1.f), 3.f);
                T.cr[pos] = make_int4(plo, plo + nin - 1, coff, rl | (rh << 8));
            }
        }
        __syncwarp();
        if (e4 == 0) continue;
        if (cfit > 0) {
            for (int e = lane; e < cfit; e += 32) {  // the line owning element e: the last with offset <= e
                int lo = e2, hi = e3 - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (T.cr[mid].z <= e) lo = mid; else hi = mid - 1;
                }
                const int4 r = T.cr[lo];
                const float4 u = T.f0[lo], p = T.q0[lo];
                const float d = ((float)(r.x + (e - r.z)) - u.x) - u.y;
                T.cw[e] = faddeeva32_inline(d * p.y, p.z);
            }
            __syncwarp();
        }
        float2 v[2][7];  // this tile's sums of the value terms; the derivatives go to V directly
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            v[h][0] = v[h][4] = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < 7; ++c)
                if (c != 0 && c != 4) v[h][c] = V[h][c];
        }
        for (int k = 0; k < e1; ++k) {
            const float4 f0 = T.f0[k], f1 = T.f1[k];
            float4 f2, l0, l1;
            if (NS >= 3) f2 = T.f2[k];
            if (LM) {
                l0 = T.l0[k];
                if (NS >= 3) l1 = T.l1[k];
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float2 dn, rho;
                jg_offsets(xn[h], xs[h], f0.x, f0.y, f0.z, dn, rho);
                jg_wing_add<LM, NS>(dn, rho, f0, f1, f2, l0, l1, v[h]);
            }
        }
        // cutoff-edge lines: the wing and the pedestals of every point, masked by the cutoff
        for (int k = e1; k < e2; ++k) {
            const float4 f0 = T.f0[k], f1 = T.f1[k], P = T.q0[k];
            float4 f2, l0, l1, pc;
            if (NS >= 3) { f2 = T.f2[k]; pc = T.q1[k]; }
            if (LM) {
                l0 = T.l0[k];
                if (NS >= 3) l1 = T.l1[k];
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float2 dn, rho, e[7];
                jg_offsets(xn[h], xs[h], f0.x, f0.y, f0.z, dn, rho);
                const float2 d2 = __fmul2_rn(dn, dn);
                const float2 pf = __ffma2_rn(d2, make_float2(icut2, icut2), make_float2(-2.f, -2.f));  // -(2 - d^2/c^2)
                e[0] = __fmul2_rn(make_float2(P.x, P.x), pf);
                e[1] = __fmul2_rn(make_float2(P.y, P.y), pf);
                if (NS >= 3) e[2] = __ffma2_rn(make_float2(P.z, P.z), pf, __fmul2_rn(make_float2(-pc.x, -pc.x), dn));
                if (NS >= 4) e[3] = __ffma2_rn(make_float2(P.w, P.w), pf, __fmul2_rn(make_float2(-pc.y, -pc.y), dn));
                e[4] = e[5] = e[6] = make_float2(0.f, 0.f);
                jg_wing_add<LM, NS>(dn, rho, f0, f1, f2, l0, l1, e);
                const bool ix = d2.x <= cut2, iy = d2.y <= cut2;
#pragma unroll
                for (int c = 0; c < 7; ++c)
                    if (jg_used<LM, NS>(c)) {
                        v[h][c].x += ix ? e[c].x : 0.f;
                        v[h][c].y += iy ? e[c].y : 0.f;
                    }
            }
        }
        // core lines
        for (int k = e2; k < e3; ++k) {
            const float4 f0 = T.f0[k], f1 = T.f1[k];
            float4 f2, l0, l1;
            if (NS >= 3) f2 = T.f2[k];
            if (LM) {
                l0 = T.l0[k];
                if (NS >= 3) l1 = T.l1[k];
            }
            const int4 cr = T.cr[k];
            const int rl = cr.w & 255, rh = cr.w >> 8;  // rh = -1: none (arithmetic shift)
            const float df2 = T.df2[k];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float2 dn, rho;
                jg_offsets(xn[h], xs[h], f0.x, f0.y, f0.z, dn, rho);
                if (rh < 2 * h || rl > 2 * h + 1) {  // warp-uniform: no core point in these rows
                    jg_wing_add<LM, NS>(dn, rho, f0, f1, f2, l0, l1, v[h]);
                    continue;
                }
                float2 e[7];
#pragma unroll
                for (int c = 0; c < 7; ++c) e[c] = make_float2(0.f, 0.f);
                jg_wing_add<LM, NS>(dn, rho, f0, f1, f2, l0, l1, e);
                const float4 q0 = T.q0[k], q1 = T.q1[k];
                float4 q2, q3, q4;
                if (NS >= 3) { q2 = T.q2[k]; q3 = T.q3[k]; }
                if (LM) q4 = T.q4[k];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float d = r ? dn.y : dn.x;
                    const bool core = d * d <= df2;
                    if (!__any_sync(kFull, core)) continue;
                    const float x = d * q0.y, y = q0.z;
                    const int pt = lane + 32 * (2 * h + r);
                    float2 gr;
                    float2 w = faddeeva_cf2_grad(x, y, y * y, gr);
                    if (core && fabsf(x) + y < 15.f) {
                        w = pt >= cr.x && pt <= cr.y ? T.cw[cr.z + pt - cr.x] : faddeeva32(x, y);
                        gr = wofz_grad32(x, y, w);
                    }
                    float t7[7];
                    jg_core_terms<LM, NS>(d, w, gr, q0, q1, q2, q3, q4, t7);
                    if (core) {
#pragma unroll
                        for (int c = 0; c < 7; ++c)
                            if (jg_used<LM, NS>(c)) {
                                if (r) e[c].y = t7[c];
                                else e[c].x = t7[c];
                            }
                    }
                }
#pragma unroll
                for (int c = 0; c < 7; ++c)
                    if (jg_used<LM, NS>(c)) v[h][c] = __fadd2_rn(v[h][c], e[c]);
            }
        }
        // general lines: the core and the cutoff edge among the points, H - pedestal per pair
        for (int k = e3; k < e4; ++k) {
            const float4 f0 = T.f0[k], q0 = T.q0[k], q1 = T.q1[k];
            float4 q2 = make_float4(0.f, 0.f, 0.f, 0.f), q3 = q2, q4 = q2;
            if (NS >= 3) { q2 = T.q2[k]; q3 = T.q3[k]; }
            if (LM) q4 = T.q4[k];
            const float df2 = T.df2[k];
#pragma unroll
            for (int q = 0; q < kJgQ; ++q) {
                const float d = ((pl0 + 32.f * q) - f0.x) - f0.y, d2 = d * d;
                if (d2 > cut2) continue;
                float t7[7];
                jg_pair<LM, NS>(d, d2 <= df2, q0, q1, q2, q3, q4, icut2, t7);
                const int h = q >> 1;
#pragma unroll
                for (int c = 0; c < 7; ++c)
                    if (jg_used<LM, NS>(c)) {
                        if (q & 1) v[h][c].y += t7[c];
                        else v[h][c].x += t7[c];
                    }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // the compensated tile sums
            kahan_add(S[h].x, C[h].x, v[h][0].x);
            kahan_add(S[h].y, C[h].y, v[h][0].y);
            if (LM) {
                kahan_add(SD[h].x, CD[h].x, v[h][4].x);
                kahan_add(SD[h].y, CD[h].y, v[h][4].y);
            }
#pragma unroll
            for (int c = 0; c < 7; ++c)
                if (c != 0 && c != 4) V[h][c] = v[h][c];
        }
    }
    // pedestals, and the far field's interpolants, per sum
#pragma unroll
    for (int c = 0; c < 7; ++c) {
        if (!jg_used<LM, NS>(c)) continue;
        float2 it[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        if (c < NS) {
            const float A = warp_sum(c == 0 ? QA[0] - QAc : QA[c]), B = warp_sum(c == 0 ? QB[0] - QBc : QB[c]);
            const float Cq = warp_sum(c == 0 ? QC[0] - QCc : QC[c]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                it[h].x = fmaf(xn[h].x, fmaf(xn[h].x, Cq, B), A);
                it[h].y = fmaf(xn[h].y, fmaf(xn[h].y, Cq, B), A);
            }
        }
        if (gfar) {
            // about the value of a middle node, so that the weights' rounding acts on the
            // field's variation over the leaf only
            float nd = gfar[c * kTrNodes + (lane & (kTrNodes - 1))];
            const float mid = __shfl_sync(kFull, nd, kTrNodes / 2);
            nd -= mid;
            float2 f[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int k = 0; k < kTrNodes; ++k) {
                const float F = __shfl_sync(kFull, nd, k);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    f[h] = __ffma2_rn(make_float2(F, F), make_float2(Lw[k][64 * h + lane], Lw[k][64 * h + 32 + lane]), f[h]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (c == 0) {
                    kahan_add(S[h].x, C[h].x, mid);
                    kahan_add(S[h].y, C[h].y, mid);
                } else {
                    f[h] = __fadd2_rn(f[h], make_float2(mid, mid));
                }
                it[h] = __fadd2_rn(it[h], f[h]);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (c == 0) {
                kahan_add(S[h].x, C[h].x, it[h].x);
                kahan_add(S[h].y, C[h].y, it[h].y);
                V[h][0] = S[h];
            } else if (c == 4) {
                kahan_add(SD[h].x, CD[h].x, it[h].x);
                kahan_add(SD[h].y, CD[h].y, it[h].y);
                V[h][4] = SD[h];
            } else {
                V[h][c] = __fadd2_rn(V[h][c], it[h]);
            }
        }
    }
    // clamps (voigt.jl:276, line_mixing.jl:1368, cross_section_jacobian.jl:107-113, :312-319)
    // and the segment's weights onto the layer channels
#pragma unroll
    for (int q = 0; q < kJgQ; ++q) {
        float s[7];
#pragma unroll
        for (int c = 0; c < 7; ++c) s[c] = jg_used<LM, NS>(c) ? ((q & 1) ? V[q >> 1][c].y : V[q >> 1][c].x) : 0.f;
        float v = s[0], vT = s[1], vp = s[2], vv = s[3];
        if (!(v > 0.f)) v = vT = vp = vv = 0.f;
        if (LM) {
            v += s[4];
            vT += s[5];
            vp += s[6];
            if (!(v > 0.f)) v = vT = vp = 0.f;
        }
        if (prow) {  // relaxation-matrix line mixing: rows (perturbation, d/dT, d/dp) x column amount
            v += (float)prow[32 * q];
            vT += (float)prow[pstride + 32 * q];
            if (NS >= 3) vp += (float)prow[2 * pstride + 32 * q];
            if (!(v > 0.f)) v = vT = vp = 0.f;
        }
        auto add = [&](const float w[4], int o) {
            float a = w[0] * v + w[1] * vT;
            if (NS >= 3) a += w[2] * vp;
            if (NS >= 4) a += w[3] * vv;
            acc[o * kJgWarpPts + 32 * q + lane] += a;
        };
        for (int o = 0; o < 3; ++o) add(W.base[o], o);
        for (unsigned r = W.retr; r; r &= r - 1)  // warp-uniform
            for (int o = 0; o < 2; ++o) add(W.pair[o], 3 + 2 * (__ffs(r) - 1) + o);
    }
}

// dynamic shared memory of jg_linesum_kernel<LM, NS>: the warps' tiles, the leaf weights and
// the warps' per-point output accumulators
constexpr size_t jg_smem_bytes(bool lm, int n_out) {
    return (lm ? sizeof(JgTile<true>) : sizeof(JgTile<false>)) * kJgWarps + sizeof(float) * kTrNodes * kTrLeaf +
           sizeof(float) * kJgWarps * n_out * kJgWarpPts;
}

// One warp per leaf, the segments of one kind (MODE); one launch per kind, the first stores
// the layer channels and the others add to theirs.  A kernel holding every kind ran out of
// instruction cache (warps in different kinds at a time: 6.5 of 9 stall cycles per
// instruction were for instructions).
// Bound by issue.  Measured on a B200, against two-level far fields (1024-point strips, then
// each warp's 8 nodes from 320 points), four sums (seven) for every segment and the cores per
// pair: 16 scenes of the 5,000-line list 1.53 + 7.50 -> 1.10 + 2.89 ms (far + near lines), one
// IASI spectrum with VP_Y 9.78 + 91.9 -> 7.7 + 35.3 ms, two 645-1000 cm^-1 profiles of six
// species 2.74 + 12.9 -> 2.5 + 8.5 ms.  K of three species against the FP64 oracle: 1.2e-6 ->
// 1.6e-7 of its norm at 700 cm^-1, 9.3e-7 -> 8.2e-7 at 2200; single monochromatic entries
// 1.7e-4 -> 2.7e-7 of the largest (the gradient of w in closed form).
template <int MODE>
__global__ void __launch_bounds__(kJgWarps * 32, MODE == kJg2 ? 3 : 2) jg_linesum_kernel(
    const SegDev* __restrict__ segs, const SegW* __restrict__ wts, const int2* __restrict__ pl_segs, CellIndex ci,
    JgOut g, long long n_nu, float cut_g, int n_out, int store, int far_sums, float* __restrict__ out,
    const double* __restrict__ pert, long long pstride, const TreeTables* __restrict__ tab,
    const float* __restrict__ far, const int4* __restrict__ ranges, int n_leaves, int pl0, int seg0) {
    constexpr bool LM = MODE == kJgLm2 || MODE == kJgLm3;
    constexpr int NS = MODE == kJg2 || MODE == kJgLm2 ? 2 : MODE == kJg4 ? 4 : 3;
    extern __shared__ __align__(16) unsigned char jg_sh[];
    JgTile<LM>* tiles = (JgTile<LM>*)jg_sh;
    float(*Lw)[kTrLeaf] = (float(*)[kTrLeaf])(tiles + kJgWarps);
    for (int i = threadIdx.x; i < kTrNodes * kTrLeaf; i += kJgWarps * 32) ((float*)Lw)[i] = ((const float*)tab->L)[i];
    __syncthreads();  // the only block-wide barrier: before any warp leaves
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* acc = (float*)(Lw + kTrNodes) + (size_t)warp * n_out * kJgWarpPts;  // [n_out][128], warp-private
    const int pl = pl0 + (int)blockIdx.y, leaf = (int)blockIdx.x * kJgWarps + warp;
    const long long wb = (long long)leaf * kJgWarpPts;
    if (wb >= n_nu) return;
    for (int i = lane; i < n_out * kJgWarpPts; i += 32) acc[i] = 0.f;
    unsigned touched = 0;  // layer channels with a contribution (warp-uniform)
    const int2 rng = pl_segs[pl];
    for (int si = rng.x; si < rng.x + rng.y; ++si) {
        const SegDev sg = segs[si];
        if (jg_mode(sg.flags) != MODE) continue;
        const int* row = ci.idx + (size_t)sg.list * ci.n;
        const float m = (float)sg.margin_g;
        const int wlo = cell_floor(ci, row, (float)wb - cut_g - m);
        const int whi = cell_ceil(ci, row, (float)(wb + kJgWarpPts) + cut_g + m);
        int4 own = make_int4(wlo, wlo, whi, whi);  // no far field: every line direct
        const float* gf = nullptr;
        if (far) {
            const size_t cell = (size_t)(si - seg0) * n_leaves + leaf;
            own = ranges[cell];
            gf = far + cell * far_sums * kTrNodes;
        }
        const double* prow = pert && (sg.flags & SEG_RELMAT) ? pert + (size_t)pl * 3 * pstride + wb + lane : nullptr;
        const SegW& W = wts[si];
        touched |= 7u;
        for (unsigned r = W.retr; r; r &= r - 1) touched |= 3u << (3 + 2 * (__ffs(r) - 1));
        jg_segment<LM, NS>(sg, g, wb, own, wlo, whi, cut_g, lane, tiles[warp], Lw, gf, W, prow, pstride, acc);
    }
    float* base = out + (size_t)pl * n_out * n_nu;
    for (int o = 0; o < n_out; ++o) {
        if (!store && !(touched >> o & 1u)) continue;
#pragma unroll
        for (int q = 0; q < kJgQ; ++q) {
            const long long i = wb + 32 * q + lane;
            const float v = acc[o * kJgWarpPts + 32 * q + lane];
            if (i < n_nu) base[(size_t)o * n_nu + i] = store ? v : base[(size_t)o * n_nu + i] + v;
        }
    }
}

// ------------------------------------------------------------------ RTE Jacobian
struct JgLayer {       // per (profile, layer), beyond LayerRT
    double frac;       // _cg_mass_frac (T_ave weight on the upper level)
    double wM;         // log-p weight of p_mid on the upper level
    double dp;         // layer thickness, hPa
};
struct JgProfile {     // per profile
    int n_retr;
    int retr_h2o, retr_co2;  // retrieved index of H2O / CO2 whose continuum VMR derivative is used, or -1
    int include_T, include_tsfc, include_eps, log_vmr;
    int n_state;
};

// exp(a) for small arguments (a^7/5040 < 1e-17)
__device__ __forceinline__ double exp_small(double a) {
    if (fabs(a) > 0.01) return exp(a);
    return fma(a, fma(a, fma(a, fma(a, fma(a, fma(a, 1.0 / 720.0, 1.0 / 120.0), 1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0), 1.0);
}

// exp(a) - 1 for the steps of a central difference: below 2^-8 the series' next term is
// a^5/120 of a, under 1e-11 of the difference it goes into
__device__ __forceinline__ double expm1_tiny(double a) {
    if (fabs(a) > 0.00390625) return expm1(a);
    return a * fma(a, fma(a, fma(a, fma(a, 1.0 / 120.0, 1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0);
}

constexpr int kJgRteThreads = 128, kJgRteFine = 16;
constexpr int kJgRteChunk = 64;  // layers of JgRteBase in shared memory at a time
// Constants of one layer for jg_rte_kernel, formed once per (profile, layer): the MT-CKD
// continua's column factor and exponents at T_mid and, as ratios, at T_mid +- 0.05 K (the
// reference's central difference, vmr_jacobian.jl:322-344); c2/T and 1/T of the Planck terms.
// Per (point, layer) the continua then take three exponentials for their value and all their
// derivatives; evaluated from scratch at every perturbed argument (two pow, one exp and
// several divisions each, eight times) they were most of the kernel.
struct JgRteLayer {
    double c2m, l296, l246, G, vh, vc;  // c2/T_mid, ln(296/T_mid), ln(T_mid/246), column factor, VMRs
    double rp, rm, dp, dm;              // T/(T + h), T/(T - h) and their logs
    double c2a, ia, c2t, it, c2b, ib;   // c2/T and 1/T at T_ave, T_top, T_bot
    double frac, wM;
    // exp(-c2/T j d), d the grid step, at T_mid, T_ave, T_top: the factors of exp(-c2 nu/T)
    // within 16 grid points (JgRteBase has the other factor)
    double step[3][kJgRteFine];
};
// Per CTA and layer: exp(-c2 nu/T) at T_mid, T_ave, T_top on every 16th of its points, and
// the self continuum's (296/T)^te at the first.
struct JgRteBase {
    double q[3][kJgRteThreads / kJgRteFine];
    double E;
};
constexpr double kJgRteDT = 0.05;
__global__ void __launch_bounds__(128) jg_rte_layers_kernel(const LayerRT* __restrict__ lrt, const JgLayer* __restrict__ jl,
                                                            int n, double dnu, JgRteLayer* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / kJgRteFine, j = t % kJgRteFine;
    if (i >= n) return;
    const LayerRT r = lrt[i];
    JgRteLayer& o = out[i];
    const double T = r.T_mid, p = r.p_mid;
    const double c2m = 1.4387769 / T, c2a = 1.4387769 / r.T_ave, c2t = 1.4387769 / r.T_top;
    o.step[0][j] = exp(-c2m * (j * dnu));
    o.step[1][j] = exp(-c2a * (j * dnu));
    o.step[2][j] = exp(-c2t * (j * dnu));
    if (j) return;
    const JgLayer y = jl[i];
    o.c2m = c2m;
    o.l296 = log(296.0 / T);
    o.l246 = log(T / 246.0);
    const double rho = (p / 1013.0) * (296.0 / T), n1 = p * 100.0 / (1.380649e-23 * T) * 1e-6;
    o.G = rho * n1 * (8.314462 * T / (0.028964 * 9.80665) * y.dp / p * 100.0);
    o.vh = r.vmr_h2o;
    o.vc = r.vmr_co2;
    o.rp = T / (T + kJgRteDT);
    o.rm = T / (T - kJgRteDT);
    o.dp = -log1p(kJgRteDT / T);
    o.dm = -log1p(-kJgRteDT / T);
    o.c2a = c2a;
    o.ia = 1.0 / r.T_ave;
    o.c2t = c2t;
    o.it = 1.0 / r.T_top;
    o.c2b = 1.4387769 / r.T_bot;
    o.ib = 1.0 / r.T_bot;
    o.frac = y.frac;
    o.wM = y.wM;
}

// planck_radiance and dB/dT (planck.jl:22-24, :67-71) from one expm1 and one reciprocal:
// B = c1 nu^3 / (e^x - 1), dB/dT = B (x/T) e^x / (e^x - 1), x = c2 nu / T
__device__ __forceinline__ void planck_grad64(double c1nu3, double nu, double c2T, double iT, double& B, double& dB) {
    const double x = nu * c2T, r = rcp64(expm1(x));
    B = c1nu3 * r;
    dB = B * (x * iT) * (1.0 + r);
}
// the same with q = exp(-x) given: 1/(e^x - 1) = q/(1 - q); where 1 - q would lose more than
// two bits, from x
__device__ __forceinline__ void planck_grad64_q(double c1nu3, double nu, double c2T, double iT, double q, double& B, double& dB) {
    if (q > 0.75) return planck_grad64(c1nu3, nu, c2T, iT, B, dB);
    const double r = q * rcp64_fast(1.0 - q);
    B = c1nu3 * r;
    dB = B * (nu * c2T * iT) * (1.0 + r);
}
// _cim_correction and its derivative (schwarzschild.jl:59-63, schwarzschild_jacobian.jl) with
// w = exp(-s)
__device__ __forceinline__ void cim_both(double s, double w, double& f, double& fp) {
    f = s / 6.0;
    fp = 1.0 / 6.0;
    if (!(s < 0.06)) {
        const double a = w - 1.0, r = rcp64(s * a), is = a * r, iw = s * r;  // 1/s, 1/(w - 1)
        f = 1.0 - 2.0 * fma(w, iw, is);
        fp = 2.0 * (is * is) - 2.0 * w * (iw * iw);
    }
}
// _lit_correction and its derivative
__device__ __forceinline__ void lit_both(double s, double w, double& f, double& fp) {
    f = s * (0.5 - s * (1.0 / 3.0 - s * 0.125));
    fp = 0.5 - s * (2.0 / 3.0 - s * 0.375);
    if (!(s < 1e-4)) {
        const double is = rcp64(s);
        f = (1.0 - w) * is - w;
        fp = (w * (s + 1.0) - 1.0) * (is * is) + w;
    }
}

// One thread per (profile, grid point): the monochromatic Jacobian columns
// D[x][nu] = dI/dx (FP32) for every state element, and I (FP64).
// schwarzschild_jacobian.jl:66-266 with the state chains of vmr_jacobian.jl:383-503.
// Transmittances come from the FP64 cumulative optical depth: the top-of-layer
// transmittance of layer m is exp(-(OD_total - OD_below_and_m)).
//
// MODE selects what the sweep leaves behind:
//   0  D (forward mode, the columns of the monochromatic Jacobian) and I;
//   1  I only (the derivative terms are not formed);
//   2  the adjoint: with Ibar[profile][nu] = the radiance cotangent on the grid (the ILS
//      and channel resampling transposed, applied to dy dBT/dR), each term D[x][nu] is
//      multiplied by Ibar[nu] as it is formed and summed over the grid on the device
//      (warp shuffles, then FP64 shared-memory and global atomics) into xbar[profile][x]
//      = sum_nu Ibar D[x] = (K^T dy)[x].  D is never stored.  Dynamic shared memory:
//      n_state doubles.
//
// Bound by latency and issue (some 970 instructions a point and layer, 290 of them FP64; the
// bytes, 0.9 GB for 16 scenes, take 0.14 ms), so registers are given up for warps: eight CTAs
// per SM in forward mode (64 registers, some spills; 1.28 ms, seven 1.39, six 1.44), six in
// the adjoint (1.04 ms, eight 1.19).  exp(-c2 nu/T) is the product of a factor per 16th point
// and one per step, both from tables, and the continuum exponent's change across a CTA a short
// series; the next layer's sums are prefetched.  16 scenes of the 5,000-line list 1.59 -> 1.28
// ms (3.69 with every continuum evaluated from scratch), one IASI profile 2.42 -> 2.15, the
// adjoint of two 645-1000 cm^-1 profiles 0.55 + 1.25 -> 0.47 + 1.04.
template <bool CIA = false, int MODE = 0>
__global__ void __launch_bounds__(kJgRteThreads, CIA ? 1 : MODE == 0 ? 8 : 6) jg_rte_kernel(
    const float* __restrict__ jl, int n_out, const LayerRT* __restrict__ lrt, const JgRteLayer* __restrict__ jlay,
    const ProfileRT* __restrict__ prt, const JgProfile* __restrict__ jprof, const double* __restrict__ vlev,
    int L, const double* __restrict__ grid, long long n_nu, int src, ContDev cont, double* __restrict__ I,
    float* __restrict__ D, const double* __restrict__ Ibar = nullptr, double* __restrict__ xbar = nullptr) {
    extern __shared__ double jg_xsh[];
    __shared__ JgRteBase base[kJgRteChunk];
    const long long i0 = (long long)blockIdx.x * kJgRteThreads, i_raw = i0 + threadIdx.x;
    const int p = blockIdx.y;
    const bool valid = i_raw < n_nu;
    // every lane stays to the end (the layers' base, the adjoint's reductions), clamped
    const long long i = valid ? i_raw : n_nu - 1;
    if (MODE == 2) {
        for (int x = threadIdx.x; x < jprof[p].n_state; x += blockDim.x) jg_xsh[x] = 0.0;
        __syncthreads();
    }
    const double ib = MODE == 2 && valid ? Ibar[(size_t)p * n_nu + i] : 0.0;
    const double nu = grid[i], c1nu3 = 1.191042953e-5 * (nu * nu * nu);
    const ProfileRT pr = prt[p];
    const JgProfile jp = jprof[p];
    const LayerRT* lr = lrt + (size_t)p * L;
    const JgRteLayer* jy = jlay + (size_t)p * L;
    const float* out = jl + (size_t)p * L * n_out * n_nu;
    const double* vl = vlev + (size_t)p * 4 * (L + 1);  // level VMR of the retrieved species
    double Cs = 0, Cf = 0, te = 0, Se = 0, td = 0;
    if (cont.mask & 1) {
        const Lerp l = lerp_at(cont.h2o, cont.n_h2o, nu);
        Cs = lerp_val(cont.h2o + cont.n_h2o, l);
        Cf = lerp_val(cont.h2o + 2 * cont.n_h2o, l);
        te = lerp_val(cont.h2o + 3 * cont.n_h2o, l);
    }
    if (cont.mask & 2) {
        const Lerp l = lerp_at(cont.co2, cont.n_co2, nu);
        Se = 1e-20 * lerp_val(cont.co2 + cont.n_co2, l);
        td = lerp_val(cont.co2 + 2 * cont.n_co2, l);
    }
    __shared__ double te_first;
    if (threadIdx.x == 0) te_first = te;
    auto fill = [&](int k0) {  // the base of the layers k0 ..
        __syncthreads();
        constexpr int Q = kJgRteThreads / kJgRteFine;
        const int nl = min(kJgRteChunk, L - k0);
        for (int e = threadIdx.x; e < nl * 3 * Q; e += kJgRteThreads) {
            const int k = e / (3 * Q), x = e / Q % 3, a = e % Q;
            const JgRteLayer& r = jy[k0 + k];
            base[k].q[x][a] = exp(-grid[min(i0 + a * kJgRteFine, n_nu - 1)] * (x == 0 ? r.c2m : x == 1 ? r.c2a : r.c2t));
        }
        if (cont.mask & 1)
            for (int k = threadIdx.x; k < nl; k += kJgRteThreads) base[k].E = exp(te_first * jy[k0 + k].l296);
        __syncthreads();
    };
    // exp(-c2 nu/T) of layer k, x as in JgRteBase
    auto q_at = [&](int k, const JgRteLayer& r, int x) {
        return base[k % kJgRteChunk].q[x][threadIdx.x / kJgRteFine] * __ldg(&r.step[x][threadIdx.x % kJgRteFine]);
    };
    CiaPoint cp;
    if (CIA) cia_prepare(cont.cia, cont.mask, nu, cp);
    const double invmu = 1.0 / pr.mu, eps = pr.eps;
    // MT-CKD continua of layer k, continuum.jl:183-250 (with the dz(T) of
    // optical_depth.jl:123-130 inside G): tau = G rad [vh (Cs E vh + Cf (1 - vh)) + Se Q vc]
    struct Cont {
        double x, e, E, Q;  // c2 nu / T, exp(-x), (296/T)^te, (T/246)^td
    };
    const bool mt = (cont.mask & 3) != 0;
    auto cont_at = [&](int k, const JgRteLayer& r) {
        Cont c{0.0, 0.0, 0.0, 1.0};
        c.x = nu * r.c2m;
        c.e = q_at(k, r, 0);
        if (cont.mask & 1) c.E = base[k % kJgRteChunk].E * exp_small((te - te_first) * r.l296);
        if ((cont.mask & 2) && td != 0.0) c.Q = exp(td * r.l246);
        return c;
    };
    auto cont_sum = [&](const JgRteLayer& r, double E, double Q) {
        return fma(r.vh, fma(Cs * E, r.vh, Cf * (1.0 - r.vh)), Se * Q * r.vc);
    };
    auto cia_at = [&](const LayerRT& r, const JgRteLayer& y, double vh, double vc, double T) {
        // y.G = rho n1 dz(T_mid): dz(T) = dz(T_mid) T / T_mid
        const double rho = (r.p_mid / 1013.0) * (296.0 / r.T_mid), n1 = r.p_mid * 100.0 / (1.380649e-23 * r.T_mid) * 1e-6;
        return cia_tau(cont, cp, nu, vh, vc, r.p_mid, T, y.G / (rho * n1) * (T / r.T_mid));
    };
    auto layer_s = [&](int k, const JgRteLayer& r, const Cont& c) {
        double t = (double)out[((size_t)k * n_out) * n_nu + i];
        if (mt) t = fma(r.G * radfn_e(nu, c.x, c.e), cont_sum(r, c.E, c.Q), t);
        if (CIA) t += cia_at(lr[k], r, r.vh, r.vc, lr[k].T_mid);
        return t * invmu;
    };
    // pass 1: total optical depth and the downwelling radiance at the surface
    double OD = 0.0, Id = 0.0, gk = 1.0;
    double Bb, dBb;  // at the layer's bottom level: the top of the layer below
    planck_grad64(c1nu3, nu, jy[0].c2b, jy[0].ib, Bb, dBb);
    const double B0 = Bb, dB0 = dBb;
    for (int k = 0; k < L; ++k) {
        if (k % kJgRteChunk == 0) fill(k);
        if (k + 2 < L) asm volatile("prefetch.global.L1 [%0];" ::"l"(out + (size_t)(k + 2) * n_out * n_nu + i));
        const JgRteLayer& r = jy[k];
        Cont c{};
        if (mt) c = cont_at(k, r);
        const double s = layer_s(k, r, c);
        OD += s;
        if (eps < 1.0) {  // schwarzschild_jacobian.jl:221-243
            const double w = exp(-s), u = 1.0 - w;
            double Ba, Bt, f, fp, d;
            planck_grad64_q(c1nu3, nu, r.c2t, r.it, q_at(k, r, 2), Bt, d);
            if (src == 0) {
                planck_grad64_q(c1nu3, nu, r.c2a, r.ia, q_at(k, r, 1), Ba, d);
                cim_both(s, w, f, fp);
                Id += gk * (u * fma(Bb - Ba, f, Ba));
            } else {
                lit_both(s, w, f, fp);
                Id += gk * fma(Bt - Bb, f, Bb * u);
            }
            gk *= w;
            Bb = Bt;
        }
    }
    const double Tr0 = exp(-OD), refl = 1.0 - eps;
    double Bs, dBs;
    planck_grad64(c1nu3, nu, 1.4387769 / pr.T_sfc, 1.0 / pr.T_sfc, Bs, dBs);
    double Iv = eps * Bs * Tr0, Ib = eps * Bs * Tr0;
    const double dIde = Bs * Tr0 - (eps < 1.0 ? Id * Tr0 : 0.0);
    const double dIdTs = eps * dBs * Tr0;
    // pass 2, surface to top
    const int nT = jp.include_T ? L + 1 : 0;
    double cum = 0.0, gdn = 1.0, Id_below = 0.0;
    double carryT = 0.0, carryV[4] = {0, 0, 0, 0};
    const size_t nn = (size_t)n_nu;
    float* Dp = MODE == 0 ? D + (size_t)p * jp.n_state * nn : nullptr;
    auto emit = [&](size_t x, double val) {  // D[x][nu] = val
        if (MODE == 0) {
            if (valid) Dp[x * nn + i] = (float)val;
        } else if (MODE == 2) {
            double v = valid ? val * ib : 0.0;
#pragma unroll
            for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if ((threadIdx.x & 31) == 0) atomicAdd(&jg_xsh[x], v);
        }
    };
    constexpr bool DERIV = MODE != 1;
    Bb = B0;
    dBb = dB0;
    for (int m = 0; m < L; ++m) {
        if (L > kJgRteChunk && m % kJgRteChunk == 0) fill(m);
        if (m + 1 < L) {  // the loads are a layer's longest wait
            const float* nx = out + (size_t)(m + 1) * n_out * nn + i;
            for (int q = 0; q < (DERIV ? n_out : 1); ++q) asm volatile("prefetch.global.L1 [%0];" ::"l"(nx + q * nn));
        }
        const JgRteLayer& r = jy[m];
        Cont c{};
        if (mt) c = cont_at(m, r);
        const double s = layer_s(m, r, c);
        cum += s;
        const double Tt = exp(-(OD - cum));  // transmittance from the top of layer m to space
        const double w = exp(-s), u = 1.0 - w;
        double e, dea, dTl_lo, dTl_hi, Ba = 0.0, dBa = 0.0, Bt, dBt, f, fp;
        planck_grad64_q(c1nu3, nu, r.c2t, r.it, q_at(m, r, 2), Bt, dBt);
        if (src == 0) {
            planck_grad64_q(c1nu3, nu, r.c2a, r.ia, q_at(m, r, 1), Ba, dBa);
            cim_both(s, w, f, fp);
            const double core = Ba + (Bt - Ba) * f;
            e = u * core;
            dea = w * core + u * (Bt - Ba) * fp;
            const double cavg = Tt * u * (1.0 - f) * dBa;
            dTl_lo = cavg * (1.0 - r.frac);
            dTl_hi = cavg * r.frac + Tt * u * f * dBt;
        } else {
            lit_both(s, w, f, fp);
            e = Bt * u + (Bb - Bt) * f;
            dea = Bt * w + (Bb - Bt) * fp;
            dTl_lo = Tt * f * dBb;
            dTl_hi = Tt * (u - f) * dBt;
        }
        double dIdtau = invmu * (-Ib + Tt * dea);
        if (eps < 1.0) {  // reflected downwelling, schwarzschild_jacobian.jl:210-264
            double em, dem;
            if (src == 0) {
                const double core = Ba + (Bb - Ba) * f;
                em = u * core;
                dem = w * core + u * (Bb - Ba) * fp;
            } else {
                em = Bb * u + (Bt - Bb) * f;
                dem = Bb * w + (Bt - Bb) * fp;
            }
            const double above = Id - Id_below - gdn * em;  // emitted above layer m
            dIdtau += refl * invmu * Tr0 * (-above + gdn * dem - Id);
            const double rg = refl * Tr0 * gdn;
            if (src == 0) {
                const double cavg = rg * u * (1.0 - f) * dBa;
                dTl_lo += cavg * (1.0 - r.frac) + rg * u * f * dBb;
                dTl_hi += cavg * r.frac;
            } else {
                dTl_lo += rg * (u - f) * dBb;
                dTl_hi += rg * f * dBt;
            }
            Id_below += gdn * em;
            gdn *= w;
        }
        Iv += Tt * e;
        Ib += Tt * e;
        Bb = Bt;
        dBb = dBt;
        // continuum derivatives: d/dT by the reference's central difference
        // (vmr_jacobian.jl:322-344), the VMR ones of the quadratic in closed form, which its
        // central differences give
        const float* om = out + (size_t)m * n_out * nn;
        double cT = 0.0, cvh = 0.0, cvc = 0.0;
        if (DERIV && mt) {
            const double Gr = r.G * radfn_e(nu, c.x, c.e);
            if (jp.include_T) {
                const double xp = c.x * r.rp, xm = c.x * r.rm;  // -x(T +- h) = -x + x - x r
                const double ep = fma(c.e, expm1_tiny(c.x - xp), c.e), em = fma(c.e, expm1_tiny(c.x - xm), c.e);
                const double Ep = fma(c.E, expm1_tiny(te * r.dp), c.E), Em = fma(c.E, expm1_tiny(te * r.dm), c.E);
                double Qp = c.Q, Qm = c.Q;
                if ((cont.mask & 2) && td != 0.0) {
                    Qp = fma(Qp, expm1_tiny(-td * r.dp), Qp);
                    Qm = fma(Qm, expm1_tiny(-td * r.dm), Qm);
                }
                cT = (r.G * r.rp * radfn_e(nu, xp, ep) * cont_sum(r, Ep, Qp) -
                      r.G * r.rm * radfn_e(nu, xm, em) * cont_sum(r, Em, Qm)) * (1.0 / (2 * kJgRteDT));
            }
            cvh = Gr * (2.0 * r.vh * (Cs * c.E) + Cf * (1.0 - 2.0 * r.vh));
            cvc = Gr * (Se * c.Q);
        }
        if (DERIV && CIA) {
            const LayerRT lm = lr[m];
            const double vh = r.vh, vc = r.vc, Tm = lm.T_mid;
            if (jp.include_T)
                cT += (cia_at(lm, r, vh, vc, Tm + kJgRteDT) - cia_at(lm, r, vh, vc, Tm - kJgRteDT)) / (2 * kJgRteDT);
            if (jp.retr_h2o >= 0) {
                const double h = fmax(fabs(vh), 1e-30) * 1e-6;
                cvh += (cia_at(lm, r, vh + h, vc, Tm) - cia_at(lm, r, vh - h, vc, Tm)) / (2 * h);
            }
            if (jp.retr_co2 >= 0) {
                const double h = fmax(fabs(vc), 1e-30) * 1e-6;
                cvc += (cia_at(lm, r, vh, vc + h, Tm) - cia_at(lm, r, vh, vc - h, Tm)) / (2 * h);
            }
        }
        if (DERIV && jp.include_T) {
            const double tlo = (double)om[1 * nn + i] + cT * (1.0 - r.wM);
            const double thi = (double)om[2 * nn + i] + cT * r.wM;
            emit((size_t)m, carryT + dTl_lo + dIdtau * tlo);
            carryT = dTl_hi + dIdtau * thi;
        }
#pragma unroll
        for (int rr = 0; rr < (DERIV ? 4 : 0); ++rr) {
            if (rr >= jp.n_retr) break;
            const double cv = rr == jp.retr_h2o ? cvh : (rr == jp.retr_co2 ? cvc : 0.0);
            const double vlo = (double)om[(size_t)(3 + 2 * rr) * nn + i] + cv * (1.0 - r.wM);
            const double vhi = (double)om[(size_t)(4 + 2 * rr) * nn + i] + cv * r.wM;
            const double sc = jp.log_vmr ? vl[rr * (L + 1) + m] : 1.0;
            emit((size_t)(nT + rr * (L + 1) + m), sc * (carryV[rr] + dIdtau * vlo));
            carryV[rr] = dIdtau * vhi;
        }
    }
    if (DERIV && jp.include_T) emit((size_t)L, carryT);
#pragma unroll
    for (int rr = 0; rr < (DERIV ? 4 : 0); ++rr) {
        if (rr >= jp.n_retr) break;
        const double sc = jp.log_vmr ? vl[rr * (L + 1) + L] : 1.0;
        emit((size_t)(nT + rr * (L + 1) + L), sc * carryV[rr]);
    }
    int col = nT + jp.n_retr * (L + 1);
    if (DERIV && jp.include_tsfc) emit((size_t)(col++), dIdTs);
    if (DERIV && jp.include_eps) emit((size_t)(col++), dIde);
    if (eps < 1.0) Iv += refl * Id * Tr0;
    if (MODE != 2 && valid) I[(size_t)p * nn + i] = Iv;
    if (MODE == 2) {
        __syncthreads();
        for (int x = threadIdx.x; x < jp.n_state; x += blockDim.x) atomicAdd(&xbar[(size_t)p * jp.n_state + x], jg_xsh[x]);
    }
}

// ------------------------------------------------------------------ channel tail
__device__ __forceinline__ double dbt_dr(double nu, double R) {  // vmr_jacobian.jl:120-125
    if (R <= 0.0) return 0.0;
    const double A = 1.191042953e-5 * (nu * nu * nu), Lg = log1p(A / R);
    return 1.4387769 * nu * A / ((Lg * Lg) * R * (R + A));
}

// K[x][c] = dBT/dR_c * resample(ILS(D[x]))_c (strides k_state, k_chan), vmr_jacobian.jl:359-380.  One warp per
// (state element, channel); the ILS taps (kernf: the normalised FP64 taps rounded to
// FP32) run over lanes (FP32 products, FP32 sums).  A window that lies inside the grid,
// as it does for every channel away from the padded ends, needs no per-tap bounds test.
__global__ void __launch_bounds__(256) jg_channel_kernel(const float* __restrict__ D, long long n_nu, int n_state,
                                                         const float* __restrict__ kernf, long long n_taps,
                                                         double dnu_hi, GridDev g, GridDev ch, int with_ils,
                                                         const double* __restrict__ R, int observable,
                                                         float* __restrict__ K, long long k_state, long long k_chan) {
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int x = blockIdx.y, p = blockIdx.z;
    if (wid >= ch.n) return;
    const double nu = ch.at(wid);
    const float* Dx = D + ((size_t)p * n_state + x) * n_nu;
    auto value = [&](long long i) -> double {
        if (!with_ils) return (double)Dx[i];
        const long long half = (n_taps - 1) / 2, j0 = i - half;
        const int nt = (int)n_taps;
        float acc = 0.f;
        if (j0 >= 0 && j0 + n_taps <= n_nu) {
            const float* Dw = Dx + j0;
#pragma unroll 4
            for (int k = lane; k < nt; k += 32) acc = fmaf(Dw[k], kernf[k], acc);
        } else {
            for (int k = lane; k < nt; k += 32) {
                const long long j = j0 + k;
                if (j >= 0 && j < n_nu) acc = fmaf(Dx[j], kernf[k], acc);
            }
        }
        for (int d = 16; d; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
        return (double)acc * dnu_hi;
    };
    double v;
    const double g0 = g.at(0), gl = g.at(n_nu - 1);
    if (nu <= g0) v = value(0);
    else if (nu >= gl) v = value(n_nu - 1);
    else {
        long long i = (long long)floor((nu - g0) / dnu_hi);
        i = max(0LL, min(i, n_nu - 2));
        while (i > 0 && g.at(i) > nu) --i;
        while (i + 2 < n_nu && g.at(i + 1) <= nu) ++i;
        const double a = g.at(i), b = g.at(i + 1), w = (nu - a) / (b - a);
        const double r0 = value(i);
        v = w == 0.0 ? r0 : r0 * (1.0 - w) + value(i + 1) * w;
    }
    if (lane == 0) {
        double scale = 1.0;
        if (observable == 0) scale = dbt_dr(nu, R[(size_t)p * ch.n + wid]);
        K[(size_t)p * n_state * ch.n + x * k_state + wid * k_chan] = (float)(v * scale);
    }
}

// The same for channels on grid nodes: 16 channels of two state elements per CTA, FP32 products
// and sums as above.  The ring of chan_sums with both elements' points as packed pairs: a row
// costs three loads (through shared memory, 8 to 16 rows ahead) and 16 packed FMAs for 32
// products, so that the FP32 pipe is the bound (the 4.6 G products of 16 scenes x 101 states
// take 0.13 ms at full rate, rows past the ends 0.16; a third of the rest is the reduction).
// Phases and splits lie flat over the threads (step 100: 200 of 256, the last warp leaves at
// once), a split's rows end at a multiple of 8, and the 32 sums of a lane are transposed while
// they are reduced (31 shuffles for 160).  16 scenes 0.59 -> 0.34 ms, one IASI profile's 151
// columns 2.08 -> 1.16 ms; loads into registers eight rows ahead 0.51 / 1.74, and with bounds
// tests on every row 0.48 / 1.67.
constexpr int kJgChan = 16;
// zeros on either side of the FP32 taps: the ring starts C rows before the first tap, and the
// last split ends at most C + 8 (256 / step) rows past the last (steps of 16 to 256 points)
constexpr int kJgcPad = kJgChan * 256, kJgcBack = 3 * kJgcPad;
constexpr int kJgChanSmem = kJgChan * 3 * kChanThreads * 4;
// four bytes to shared memory, or zeros
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 4 : 0)
                 : "memory");
}
__global__ void __launch_bounds__(kChanThreads, 3) jg_channel_nodes_kernel(
    const float* __restrict__ D, int n_nu, int n_state, const float* __restrict__ kernf, int n_taps, double dnu_hi,
    GridDev ch, ChanNodes nodes, const double* __restrict__ R, int observable, float* __restrict__ K, long long k_state,
    long long k_chan) {
    constexpr int C = kJgChan;
    extern __shared__ float jgc_smem[];
    float(*slot)[3][kChanThreads] = reinterpret_cast<float(*)[3][kChanThreads]>(jgc_smem);
    float(*part)[2 * C] = reinterpret_cast<float(*)[2 * C]>(jgc_smem);  // after the sums
    const int c0 = blockIdx.x * C, x0 = blockIdx.y * 2, x1 = min(x0 + 1, n_state - 1), p = blockIdx.z;
    const int step = nodes.step, base = nodes.first + c0 * step - (n_taps - 1) / 2;
    const float* __restrict__ X0 = D + ((size_t)p * n_state + x0) * n_nu;
    const float* __restrict__ X1 = D + ((size_t)p * n_state + x1) * n_nu;
    const int splits = kChanThreads / step, sp = (int)threadIdx.x / step, r = (int)threadIdx.x - sp * step;
    const int M = (n_taps + step - 1) / step + C - 1;  // rows in which some tap is met
    const int per = ((M + splits - 1) / splits + 7) & ~7;
    float2 acc[C], ring[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = ring[c] = make_float2(0.f, 0.f);
    if (sp < splits) {
        const int m0 = sp * per, m1 = min(M, m0 + per);
#pragma unroll
        for (int u = 1; u < C; ++u) ring[u].x = ring[u].y = kernf[kJgcPad + r + (m0 - C + u) * step];  // the rows before
        auto sums = [&](auto edge) {
            int jf = base + r + m0 * step;  // next point to fetch
            const float *p0 = X0 + jf, *p1 = X1 + jf, *pk = kernf + kJgcPad + r + m0 * step;
            auto fetch = [&](int h) {               // eight rows to the slots h .. h + 7
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const bool in = !decltype(edge)::value || (unsigned)jf < (unsigned)n_nu;
                    cp_async4(&slot[h + u][0][threadIdx.x], in ? p0 : X0, in);
                    cp_async4(&slot[h + u][1][threadIdx.x], in ? p1 : X0, in);
                    cp_async4(&slot[h + u][2][threadIdx.x], pk, true);
                    p0 += step;
                    p1 += step;
                    pk += step;
                    jf += step;
                }
            };
            fetch(0);
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (m0 + 8 < m1) fetch(8);
            asm volatile("cp.async.commit_group;" ::: "memory");
            for (int mb = m0; mb < m1; mb += C) {
#pragma unroll
                for (int h = 0; h < C; h += 8) {
                    if (mb + h < m1) {
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float2 x = make_float2(slot[h + u][0][threadIdx.x], slot[h + u][1][threadIdx.x]);
                            const float t = slot[h + u][2][threadIdx.x];
                            ring[h + u] = make_float2(t, t);
#pragma unroll
                            for (int c = 0; c < C; ++c) acc[c] = __ffma2_rn(x, ring[(h + u - c + C) % C], acc[c]);
                        }
                        if (mb + h + C < m1) fetch(h);
                        asm volatile("cp.async.commit_group;" ::: "memory");
                    }
                }
            }
        };
        // a row past the last tap meets zeros of the pad, so only points outside the grid matter
        if (base >= 0 && base + (long long)(M + 8 * splits) * step <= n_nu) sums(std::false_type{});
        else sums(std::true_type{});
    }
    // lane l ends with the warp's sum of element l & 1, channel l >> 1: halving exchanges
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[2 * C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        v[2 * c] = acc[c].x;
        v[2 * c + 1] = acc[c].y;
    }
#pragma unroll
    for (int d = C; d; d >>= 1) {
        const bool up = lane & d;
#pragma unroll
        for (int q = 0; q < d; ++q) {
            const float keep = up ? v[q + d] : v[q], give = up ? v[q] : v[q + d];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, give, d);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    part[warp][lane] = v[0];
    __syncthreads();
    const int c = c0 + (int)(threadIdx.x >> 1), x = x0 + (int)(threadIdx.x & 1);
    if (threadIdx.x < 2 * C && c < ch.n && x < n_state) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kChanThreads / 32; ++w) s += part[w][threadIdx.x];
        double scale = 1.0;
        if (observable == 0) scale = dbt_dr(ch.at(c), R[(size_t)p * ch.n + c]);
        K[(size_t)p * n_state * ch.n + x * k_state + c * k_chan] = (float)((double)s * dnu_hi * scale);
    }
}

// ------------------------------------------------------------------ adjoint tail
// The transpose of the channel tail for the pullback: per (profile, channel) the
// cotangent of R, rbar = dy dBT/dR (vmr_jacobian.jl:120-125; dy itself for the radiance
// observable), split onto the two grid nodes the linear resampling reads
// (sounder.jl:372-377): a0 at node ci, a1 at node ci + 1.
struct ChanAdj {
    long long ci;
    double a0, a1;
};
__global__ void __launch_bounds__(256) vjp_channel_kernel(const double* __restrict__ R, const double* __restrict__ dy,
                                                          long long n_nu, double dnu_hi, GridDev g, GridDev ch,
                                                          int observable, ChanAdj* __restrict__ out) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int p = blockIdx.y;
    if (c >= ch.n) return;
    const double nu = ch.at(c);
    const size_t pc = (size_t)p * ch.n + c;
    const double scale = observable == 0 ? dbt_dr(nu, R[pc]) : 1.0;
    const double rb = dy[pc] * scale;
    ChanAdj a{0, 0.0, 0.0};
    const double g0 = g.at(0), gl = g.at(n_nu - 1);
    if (nu <= g0) { a.ci = 0; a.a0 = rb; }
    else if (nu >= gl) { a.ci = n_nu - 1; a.a0 = rb; }
    else {  // the node search of ils_bt_kernel
        long long i = (long long)floor((nu - g0) / dnu_hi);
        i = max(0LL, min(i, n_nu - 2));
        while (i > 0 && g.at(i) > nu) --i;
        while (i + 2 < n_nu && g.at(i + 1) <= nu) ++i;
        const double lo = g.at(i), hi = g.at(i + 1), w = (nu - lo) / (hi - lo);
        a.ci = i;
        a.a0 = w == 0.0 ? rb : rb * (1.0 - w);
        a.a1 = w == 0.0 ? 0.0 : rb * w;
    }
    out[pc] = a;
}

// Ibar[profile][j] = sum over channels of a0 K(j - ci) + a1 K(j - ci - 1), with K(k) =
// dnu_hi kern[k + half] inside the taps (apply_ils, ils.jl:131-153, transposed; zero
// outside the grid as the forward convolution) or the unit impulse without the ILS.
// One thread per grid point; the channels reaching it are found by a binary search on
// their (ascending) nodes.
__global__ void __launch_bounds__(256) ils_adjoint_kernel(const ChanAdj* __restrict__ ca, long long n_ch,
                                                          const double* __restrict__ kern, long long n_taps,
                                                          double dnu_hi, int with_ils, long long n_nu,
                                                          double* __restrict__ Ibar) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int p = blockIdx.y;
    if (j >= n_nu) return;
    const ChanAdj* c = ca + (size_t)p * n_ch;
    const long long half = with_ils ? (n_taps - 1) / 2 : 0;
    long long lo = 0, hi = n_ch;  // first channel with ci >= j - half - 1
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (c[mid].ci < j - half - 1) lo = mid + 1; else hi = mid;
    }
    double acc = 0.0;
    for (long long k = lo; k < n_ch && c[k].ci <= j + half; ++k) {
        const ChanAdj a = c[k];
        const long long d0 = j - a.ci, d1 = d0 - 1;
        if (with_ils) {
            if (d0 >= -half && d0 <= half) acc = fma(a.a0, kern[d0 + half], acc);
            if (d1 >= -half && d1 <= half) acc = fma(a.a1, kern[d1 + half], acc);
        } else {
            if (d0 == 0) acc += a.a0;
            if (d1 == 0) acc += a.a1;
        }
    }
    Ibar[(size_t)p * n_nu + j] = with_ils ? acc * dnu_hi : acc;
}

}  // namespace irs
