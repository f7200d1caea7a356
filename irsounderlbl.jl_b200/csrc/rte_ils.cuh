// rte_ils.cuh -- continuum + Schwarzschild RTE per grid point, then the ILS and
// brightness temperature at the channel nodes only.
//
//  rte_kernel (one thread per grid point and profile) restates
//    continua added to the layer optical depth   src/Sensor/sounder.jl:310-322,
//      h2o_continuum / co2_continuum              src/CrossSections/continuum.jl:169-250
//    level_transmittances (FP64 product)          src/Solver/transmittance.jl:26-43
//    schwarzschild_rte, :cim and :toon sources    src/Solver/schwarzschild.jl:130-209
//    add_reflected_downwelling! when eps < 1      schwarzschild.jl:228-274
//    planck_radiance                              src/Solver/planck.jl:22-24
//  for the plain FP64 path: FP64 throughout.
//  rte_mixed_kernel is the same for the FP32 optical depths of the mixed path: FP64
//  only in the cumulative optical depth and the transmittances, FP32 (Kahan-summed
//  radiance) elsewhere.
//
//  ils_bt_kernel (one warp per channel and profile; ils_nodes_kernel where the channels
//  are grid nodes at a constant step) restates apply_ils
//  (src/Sensor/ils.jl:131-153) evaluated at the grid nodes that the linear channel
//  resampling reads (sounder.jl:372-377), then brightness_temperature
//  (planck.jl:53-57).  Channel nodes are grid nodes for every sounder, so this is the
//  full convolution sampled where it is used, not an approximation.
#pragma once
#include "irs_internal.h"

namespace irs {

struct GridDev {
    long long n, den;
    double a_n, s_n, start, step;
    __host__ __device__ double at(long long i) const {
        return den ? (a_n + double(i) * s_n) / double(den) : start + double(i) * step;
    }
};
inline GridDev to_dev(const GridSpec& g) {
    GridDev d;
    d.n = g.n; d.den = g.den; d.a_n = g.a_n; d.s_n = g.s_n; d.start = g.start; d.step = g.step;
    return d;
}

// HITRAN CIA tables on the device (continuum.jl:104-160): tables t = 0 CO2-CO2,
// 1 N2-N2, 2 O2-O2 hold blocks [b0[t], b0[t+1]) in file order, each described by
// (T, nu_min, nu_max, first knot, knot count) with ascending knots nu/sg.
struct CiaDev {
    const double* blk;
    const double* nu;
    const double* sg;
    int b0[4];
};
constexpr int kCiaMax = 16;  // applicable blocks of one table cached per grid point
// The blocks that contain one grid point, their temperatures and sigma(nu), in file
// order (the temperature bracket of each layer is then a scan of these).
struct CiaPoint {
    double T[3][kCiaMax], s[3][kCiaMax];
    int n[3];
};

struct ContDev {
    const double* h2o;  // nu[n], cs[n], cf[n], te[n]
    const double* co2;  // nu[n], seff[n], tdep[n]
    int n_h2o, n_co2;
    int mask;           // 1 h2o, 2 co2, 4 co2_cia, 8 n2, 16 o2 (only when apply_continuum)
    CiaDev cia;
};
constexpr int kCiaMask = 4 | 8 | 16;

// linear interpolation on the block's knots (Interpolations.jl linear_interpolation)
__device__ __forceinline__ double cia_block_value(const CiaDev& c, int b, double nu) {
    const double* d = c.blk + 5 * (size_t)b;
    const double* x = c.nu + (long long)d[3];
    const double* y = c.sg + (long long)d[3];
    const int n = (int)d[4];
    if (n == 1) return y[0];
    int lo = 0, hi = n;  // upper_bound
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (x[mid] <= nu) lo = mid + 1; else hi = mid; }
    const int i = min(max(lo - 1, 0), n - 2);
    const double w = (nu - x[i]) / (x[i + 1] - x[i]);
    return y[i] * (1.0 - w) + y[i + 1] * w;
}
__device__ __forceinline__ void cia_prepare(const CiaDev& c, int mask, double nu, CiaPoint& cp) {
    for (int t = 0; t < 3; ++t) {
        cp.n[t] = 0;
        if (!(mask & (4 << t))) continue;
        for (int b = c.b0[t]; b < c.b0[t + 1]; ++b) {
            const double* d = c.blk + 5 * (size_t)b;
            if (nu < d[1] || nu > d[2]) continue;
            const int k = cp.n[t]++;
            if (k < kCiaMax) {
                cp.T[t][k] = d[0];
                cp.s[t][k] = cia_block_value(c, b, nu);
            }
        }
    }
}
// _cia_sigma (continuum.jl:333-362): the applicable blocks bracketing T (first in file
// order among equal temperatures), linear in T, the nearest one outside the range
__device__ __forceinline__ double cia_sigma_at(const CiaDev& c, const CiaPoint& cp, int t, double nu, double T) {
    const int na = cp.n[t];
    if (na == 0) return 0.0;
    bool hl = false, hh = false;
    double T_lo = 0, s_lo = 0, T_hi = 0, s_hi = 0;
    auto take = [&](double bt, double s) {
        if (bt <= T && (!hl || bt > T_lo)) { hl = true; T_lo = bt; s_lo = s; }
        if (bt >= T && (!hh || bt < T_hi)) { hh = true; T_hi = bt; s_hi = s; }
    };
    if (na <= kCiaMax) {
        for (int k = 0; k < na; ++k) take(cp.T[t][k], cp.s[t][k]);
    } else {  // more applicable blocks than cached: scan the table
        for (int b = c.b0[t]; b < c.b0[t + 1]; ++b) {
            const double* d = c.blk + 5 * (size_t)b;
            if (nu < d[1] || nu > d[2]) continue;
            take(d[0], cia_block_value(c, b, nu));
        }
    }
    if (!hl) return s_hi;
    if (!hh) return s_lo;
    if (T_lo == T_hi) return s_lo;
    const double w = (T - T_lo) / (T_hi - T_lo);
    return (1.0 - w) * s_lo + w * s_hi;
}
// co2_cia, n2_cia, o2_cia (continuum.jl:252-331) times dz: sigma x pair densities
__device__ __forceinline__ double cia_tau(const ContDev& c, const CiaPoint& cp, double nu, double vh, double vc,
                                          double p, double T, double dz) {
    const double nair = p * 100.0 / (1.380649e-23 * T) * 1e-6;
    const double vdry = 1.0 - vh;
    double k = 0.0;
    if (c.mask & 4) k += cia_sigma_at(c.cia, cp, 0, nu, T) * (vc * nair) * nair;
    if (c.mask & 8) {
        const double n2 = 0.78084 * vdry * nair;
        k += cia_sigma_at(c.cia, cp, 1, nu, T) * n2 * n2;
    }
    if (c.mask & 16) {
        const double o2 = 0.20946 * vdry * nair;
        k += cia_sigma_at(c.cia, cp, 2, nu, T) * o2 * o2;
    }
    return k * dz;
}

// compensated FP32 sum: the value is s - c
__device__ __forceinline__ void kahan_add32(float& s, float& c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

__global__ void grid_values_kernel(GridDev g, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g.n) out[i] = g.at(i);
}

// 1/x for positive normal x: MUFU's 20-bit estimate and one third-order step
// y (1 + e + e^2), e = 1 - x y (error e^3 = 2^-60 before rounding)
__device__ __forceinline__ double rcp64_fast(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
// the same for any x: IEEE division outside the range where it holds
__device__ __forceinline__ double rcp64(double x) {
    const double a = fabs(x);
    return a > 1e-290 && a < 1e290 ? rcp64_fast(x) : 1.0 / x;
}
// planck_radiance (planck.jl:22-24) with c1 nu^3 and c2/T given
__device__ __forceinline__ double planck64(double c1nu3, double nu, double c2T) { return c1nu3 * rcp64(expm1(nu * c2T)); }
// _cim_correction (schwarzschild.jl:59-63) and _lit_correction (:43-47) with w = exp(-s)
__device__ __forceinline__ double cim_w(double s, double w) {
    if (s < 0.06) return s / 6.0;
    if (s > 1e17) return 1.0;  // 2/s is rounded away (s * r would be inf * 0 at s = inf)
    const double a = w - 1.0, r = rcp64(s * a);  // 1/s = a r, 1/(w - 1) = s r
    return 1.0 - 2.0 * fma(w, s * r, a * r);
}
__device__ __forceinline__ double lit_w(double s, double w) {
    if (s < 1e-4) return s * (0.5 - s * (1.0 / 3.0 - s * 0.125));
    return (1.0 - w) * rcp64(s) - w;
}
// radfn (continuum.jl:169-174) with x = c2 nu / T and e = exp(-x)
__device__ __forceinline__ double radfn_e(double nu, double x, double e) {
    return x <= 0.01 ? 0.5 * x * nu : x <= 10.0 ? nu * (1.0 - e) * rcp64_fast(1.0 + e) : nu;
}
// Interpolations.jl linear interpolation, Flat() extrapolation
struct Lerp {
    int i;
    double w;
    int edge;  // -1 below, +1 above, 0 inside
};
__device__ __forceinline__ Lerp lerp_at(const double* k, int n, double x) {
    Lerp r{0, 0.0, 0};
    if (x <= k[0]) { r.edge = -1; return r; }
    if (x >= k[n - 1]) { r.edge = 1; r.i = n - 1; return r; }
    int lo = 0, hi = n;  // upper_bound
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (k[mid] <= x) lo = mid + 1; else hi = mid; }
    r.i = min(max(lo - 1, 0), n - 2);
    r.w = (x - k[r.i]) / (k[r.i + 1] - k[r.i]);
    return r;
}
__device__ __forceinline__ double lerp_val(const double* v, const Lerp& l) {
    if (l.edge) return v[l.i];
    return v[l.i] * (1.0 - l.w) + v[l.i + 1] * l.w;
}

// Constants of one layer for rte_kernel: c2/T at its temperatures and the MT-CKD continua's
// column factors and exponents, formed once per (profile, layer).
struct RteLayer64 {
    double c2a, c2t, c2b;               // c2/T at T_ave, T_top, T_bot
    double c2m, l296, l246, G, vh, vc;  // c2/T_mid, ln(296/T_mid), ln(T_mid/246), rho n1 dz, VMRs
};
__global__ void __launch_bounds__(128) rte_layers_kernel(const LayerRT* __restrict__ lrt, int n, int cont,
                                                         RteLayer64* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const LayerRT r = lrt[i];
    RteLayer64 o{};
    o.c2a = 1.4387769 / r.T_ave;
    o.c2t = 1.4387769 / r.T_top;
    o.c2b = 1.4387769 / r.T_bot;
    if (cont) {
        const double T = r.T_mid, p = r.p_mid;
        o.c2m = 1.4387769 / T;
        o.l296 = log(296.0 / T);
        o.l246 = log(T / 246.0);
        o.G = (p / 1013.0) * (296.0 / T) * (p * 100.0 / (1.380649e-23 * T) * 1e-6) * r.dz_cm;
        o.vh = r.vmr_h2o;
        o.vc = r.vmr_co2;
    }
    out[i] = o;
}

// A point's layers are cut into G runs, one thread each: within a run the recursion from its
// top (transmittance 1), and the runs are joined by the products of their transmittances,
//   I = sum_g T_above(g) I_g,      D <- D T_g + D_g   (downwelling at the run's bottom),
// so that the serial chain of a point is a G-th as long and G times the warps hide it: one
// scene's 34,801 points were 136 CTAs, one wave of one CTA per SM, each thread 49 layers in a
// row.  G = 4 for grids under kRteWide points (FP32, 34,801 points: 52 us at G = 1, 26 at 4),
// else 1, where the points alone fill the chip and a point's set-up and join are made once
// (4.2 M points: 2.07 ms at G = 1, 2.9 at 4).  The rule reads the grid only, so that a batch
// equals its profiles one by one.  Threads of one run hold consecutive points.
constexpr int kRteThreads = 256;
constexpr long long kRteWide = 148LL * 1024;
template <int G>
struct RteShape {
    static constexpr int points = kRteThreads / G;
};

// MT-CKD coefficients at a point, by the threads of the first two runs for all of its runs
template <int G>
struct RteCont {
    double v[5][RteShape<G>::points];  // h2o self, foreign, exponent; co2 strength, exponent
};
template <int G>
__device__ __forceinline__ void rte_cont_load(const ContDev& cont, double nu, int pt, int g, RteCont<G>& c) {
    if ((cont.mask & 1) && g == 0) {
        const Lerp l = lerp_at(cont.h2o, cont.n_h2o, nu);
        c.v[0][pt] = lerp_val(cont.h2o + cont.n_h2o, l);
        c.v[1][pt] = lerp_val(cont.h2o + 2 * cont.n_h2o, l);
        c.v[2][pt] = lerp_val(cont.h2o + 3 * cont.n_h2o, l);
    }
    if ((cont.mask & 2) && g == (G > 1 ? 1 : 0)) {
        const Lerp l = lerp_at(cont.co2, cont.n_co2, nu);
        c.v[3][pt] = lerp_val(cont.co2 + cont.n_co2, l);
        c.v[4][pt] = lerp_val(cont.co2 + 2 * cont.n_co2, l);
    }
    if (G > 1) __syncthreads();
}

// CIA: a CIA table is in use (a separate instantiation keeps the per-point CIA cache
// out of the common kernel).  Bound by latency (37 % of the FP64 pipe, 57 % of the issue slots;
// waits on dependences and loads).  One exponential per continuum
// term and per transmittance, one expm1 per Planck radiance (the level between two layers
// once), reciprocals in place of divisions.  One scene (34,801 points x 49 layers) 116 -> 44
// us; with a reflecting surface, Toon source and 44,801 points 246 -> 38 us.
template <typename TT, int G, bool CIA = false>
__global__ void __launch_bounds__(kRteThreads) rte_kernel(const TT* __restrict__ tau, const LayerRT* __restrict__ lrt,
                                                  const RteLayer64* __restrict__ lay, const ProfileRT* __restrict__ prt,
                                                  int L, const double* __restrict__ grid, long long n_nu, int src,
                                                  ContDev cont, double* __restrict__ I) {
    constexpr int P = RteShape<G>::points;
    __shared__ double sT[G][P], sI[G][P], sD[G][P];
    __shared__ RteCont<G> sC;
    const int pt = threadIdx.x % P, g = threadIdx.x / P;
    const long long i_raw = (long long)blockIdx.x * P + pt;
    const int p = blockIdx.y;
    const long long i = min(i_raw, n_nu - 1);
    const double nu = grid[i], c1nu3 = 1.191042953e-5 * (nu * nu * nu);
    rte_cont_load<G>(cont, nu, pt, g, sC);
    double Cs = 0, Cf = 0, te = 0, Se = 0, td = 0;
    if (cont.mask & 1) {
        Cs = sC.v[0][pt];
        Cf = sC.v[1][pt];
        te = sC.v[2][pt];
    }
    if (cont.mask & 2) {
        Se = 1e-20 * sC.v[3][pt];
        td = sC.v[4][pt];
    }
    CiaPoint cp;
    if (CIA) cia_prepare(cont.cia, cont.mask, nu, cp);
    const ProfileRT pr = prt[p];
    const double invmu = 1.0 / pr.mu;
    const bool refl = pr.eps < 1.0, mt = (cont.mask & 3) != 0;
    const LayerRT* lr = lrt + (size_t)p * L;
    const RteLayer64* ly = lay + (size_t)p * L;
    const TT* tp = tau + (size_t)p * L * n_nu + i;
    // this run: layers k1 - 1 down to k0 (group 0 at the top)
    const int k1 = (int)((long long)L * (G - g) / G), k0 = (int)((long long)L * (G - 1 - g) / G);
    double T = 1.0, Iv = 0.0, D = 0.0;
    double Bt = k1 > k0 ? planck64(c1nu3, nu, ly[k1 - 1].c2t) : 0.0;  // at the top of the current layer
    for (int k = k1 - 1; k >= k0; --k) {
        const RteLayer64& r = ly[k];
        double t = (double)tp[(size_t)k * n_nu];
        if (mt) {  // continuum.jl:169-250
            const double x = nu * r.c2m;
            double E = 0.0, Q = 1.0;
            if (cont.mask & 1) E = exp(te * r.l296);
            if ((cont.mask & 2) && td != 0.0) Q = exp(td * r.l246);
            t = fma(r.G * radfn_e(nu, x, exp(-x)), fma(r.vh, fma(Cs * E, r.vh, Cf * (1.0 - r.vh)), Se * Q * r.vc), t);
        }
        if (CIA) t += cia_tau(cont, cp, nu, lr[k].vmr_h2o, lr[k].vmr_co2, lr[k].p_mid, lr[k].T_mid, lr[k].dz_cm);
        const double s = t * invmu, w = exp(-s), u = 1.0 - w;
        const double Tk = T * w, dT = T - Tk;
        const double Bb = src != 0 || refl ? planck64(c1nu3, nu, r.c2b) : 0.0;
        double f;
        if (src == 0) {
            const double Ba = planck64(c1nu3, nu, r.c2a);
            f = cim_w(s, w);
            Iv += Ba * dT + (Bt - Ba) * (dT * f);
            if (refl) D = fma(D, w, u * (Ba + (Bb - Ba) * f));  // add_reflected_downwelling!, schwarzschild.jl:228-274
            Bt = refl ? Bb : k > k0 ? planck64(c1nu3, nu, ly[k - 1].c2t) : 0.0;
        } else {
            f = lit_w(s, w);
            Iv += Bt * dT + (Bb - Bt) * (T * f);
            if (refl) D = fma(D, w, Bb * u + (Bt - Bb) * f);
            Bt = Bb;
        }
        T = Tk;
    }
    sT[g][pt] = T;
    sI[g][pt] = Iv;
    sD[g][pt] = D;
    __syncthreads();
    if (g == 0 && i_raw < n_nu) {
        double Tt = 1.0, It = 0.0, Dt = 0.0;
#pragma unroll
        for (int q = 0; q < G; ++q) {
            It = fma(Tt, sI[q][pt], It);
            Dt = fma(Dt, sT[q][pt], sD[q][pt]);
            Tt *= sT[q][pt];
        }
        It += pr.eps * planck64(c1nu3, nu, 1.4387769 / pr.T_sfc) * Tt;
        if (refl) It += (1.0 - pr.eps) * Dt * Tt;
        I[(size_t)p * n_nu + i] = It;
    }
}

// ------------------------------------------------------- RTE, mixed precision
// rte_mixed_kernel: the same radiative transfer as rte_kernel for the FP32 optical
// depths of the mixed path, with FP64 kept only where the result needs it: the
// cumulative layer-to-space optical depth and the transmittances exp(-OD) (and the
// surface-to-layer transmittance of the reflected term).  Planck radiances, the CIM /
// Toon corrections and the MT-CKD continua are FP32, and the radiance is summed in
// FP32 with Kahan compensation.  Per (grid point, layer) it reads the FP32 tau once.
//
// Per-layer FP32 constants, computed once per CTA from LayerRT into shared memory:
struct RteLayerF {
    float2 c2_ave, c2_top, c2_bot;         // c2 / T as hi + lo
    float c2_mid;
    float h2o_self, h2o_for, l2_296, co2;  // continuum column factors, log2(296/T_mid)
    float l2_246;                          // log2(T_mid / 246)
};
__device__ __forceinline__ float2 split_f(double x) {
    const float h = (float)x;
    return make_float2(h, (float)(x - (double)h));
}
// planck_radiance (planck.jl:22-24) with c1 nu^3, nu and c2/T given: c1 nu^3 / expm1(c2 nu / T);
// above x = 0.5 exp(x) - 1 loses under one bit, so the cheaper expf serves there.  x carries
// its rounding error xl (an FP32 x alone is 1e-7 x of B off, the largest error of the mixed
// spectra): e^(x + xl) - 1 = E + xl (E + 1).
__device__ __forceinline__ float planck32(float c1nu3, float2 nu, float2 c2T) {
    const float x = nu.x * c2T.x;
    const float xl = fmaf(nu.x, c2T.x, -x) + fmaf(nu.x, c2T.y, nu.y * c2T.x);
    const float E = x > 0.5f ? expf(x) - 1.0f : expm1f(x);
    return c1nu3 * __frcp_rn(fmaf(xl, E + 1.0f, E));
}
// _cim_correction (schwarzschild.jl:59-63): s/6 below 0.06 as the reference, then the
// series 1 - 2 (1/s - 1/(e^s - 1)) = s/6 - s^3/360 + s^5/15120 - ... (next term below
// 2e-7 of the value for s < 0.5, where the direct form loses digits in FP32), then the
// direct form
__device__ __forceinline__ float cim_corr32(float s) {
    if (s < 0.06f) return s * (1.0f / 6.0f);
    if (s < 0.5f) {
        const float s2 = s * s;
        return s * fmaf(s2, fmaf(s2, 1.0f / 15120.0f, -1.0f / 360.0f), 1.0f / 6.0f);
    }
    return 1.0f - 2.0f * (1.0f / s - 1.0f / expm1f(s));
}
// _lit_correction (schwarzschild.jl:43-47): (1 - e^-s)/s - e^-s; the reference's series
// below 1e-4, continued to s^5 below 0.1 (next term s^6/840), then the direct form
__device__ __forceinline__ float lit_corr32(float s) {
    if (s < 1e-4f) return s * (0.5f - s * (1.0f / 3.0f - s * 0.125f));
    if (s < 0.1f)
        return s * fmaf(s, fmaf(s, fmaf(s, fmaf(s, 1.0f / 144.0f, -1.0f / 30.0f), 0.125f), -1.0f / 3.0f), 0.5f);
    const float e = __expf(-s);
    return -expm1f(-s) / s - e;
}
// radfn (continuum.jl:169-174) with c2/T given
__device__ __forceinline__ float radfn32(float nu, float c2T) {
    const float x = nu * c2T;
    if (x <= 0.01f) return 0.5f * x * nu;
    if (x <= 10.0f) {
        const float e = __expf(-x);
        return nu * (1.0f - e) / (1.0f + e);
    }
    return nu;
}

// Runs of layers as in rte_kernel (G threads per point).  Within a run the
// transmittance is exp(-od) of the run's FP64 cumulative optical depth.  One scene's 34,801
// points 51 -> 26 us, 160,001 points with a reflecting surface 325 -> 232 us; 4.2 M points
// 1.91 -> 2.07 ms (of 84), the price of the compensated Planck argument: BT of the 5,000-line
// scenes against FP64 3.5e-6 -> 1.7e-6 K RMS.
template <int G, bool CIA>
__global__ void __launch_bounds__(kRteThreads) rte_mixed_kernel(const float* __restrict__ tau, const LayerRT* __restrict__ lrt,
                                                        const ProfileRT* __restrict__ prt, int L,
                                                        const double* __restrict__ grid, long long n_nu, int src,
                                                        ContDev cont, double* __restrict__ I) {
    extern __shared__ __align__(16) unsigned char rte_smem[];
    RteLayerF* lc = reinterpret_cast<RteLayerF*>(rte_smem);
    constexpr int P = RteShape<G>::points;
    __shared__ double sO[G][P], sI[G][P], sD[G][P];
    __shared__ RteCont<G> sC;
    const int p = blockIdx.y;
    const LayerRT* lr = lrt + (size_t)p * L;
    for (int k = threadIdx.x; k < L; k += blockDim.x) {  // layer constants (FP64 -> FP32)
        const LayerRT r = lr[k];
        RteLayerF c;
        c.c2_ave = split_f(1.4387769 / r.T_ave);
        c.c2_top = split_f(1.4387769 / r.T_top);
        c.c2_bot = split_f(1.4387769 / r.T_bot);
        c.c2_mid = (float)(1.4387769 / r.T_mid);
        const double rho = (r.p_mid / 1013.0) * (296.0 / r.T_mid);
        const double nh = r.vmr_h2o * r.p_mid * 100.0 / (1.380649e-23 * r.T_mid) * 1e-6;
        const double nc = r.vmr_co2 * r.p_mid * 100.0 / (1.380649e-23 * r.T_mid) * 1e-6;
        c.h2o_self = (float)(r.vmr_h2o * rho * nh * r.dz_cm);
        c.h2o_for = (float)((1.0 - r.vmr_h2o) * rho * nh * r.dz_cm);
        c.l2_296 = (float)log2(296.0 / r.T_mid);
        c.co2 = (float)(1e-20 * nc * rho * r.dz_cm);
        c.l2_246 = (float)log2(r.T_mid / 246.0);
        lc[k] = c;
    }
    __syncthreads();
    const int pt = threadIdx.x % P, g = threadIdx.x / P;
    const ProfileRT pr = prt[p];
    const float imu = (float)(1.0 / pr.mu);
    const bool refl = pr.eps < 1.0;
    const long long i_raw = (long long)blockIdx.x * P + pt;
    const long long i = min(i_raw, n_nu - 1);
    const double nud = grid[i];
    const float2 nu2 = split_f(nud);
    const float nu = nu2.x;
    const float c1nu3 = (float)(1.191042953e-5 * (nud * nud * nud));
    rte_cont_load<G>(cont, nud, pt, g, sC);
    float Cs = 0.f, Cf = 0.f, te = 0.f, Se = 0.f, td = 0.f;
    if (cont.mask & 1) {
        Cs = (float)sC.v[0][pt];
        Cf = (float)sC.v[1][pt];
        te = (float)sC.v[2][pt];
    }
    if (cont.mask & 2) {
        Se = (float)sC.v[3][pt];
        td = (float)sC.v[4][pt];
    }
    CiaPoint cp;
    if (CIA) cia_prepare(cont.cia, cont.mask, nud, cp);
    const float* tp = tau + (size_t)p * L * n_nu + i;
    // the layer's optical depth along the path (FP32)
    auto slant = [&](int k) -> float {
        const RteLayerF& c = lc[k];
        float t = tp[(size_t)k * n_nu];
        if (CIA) {
            const LayerRT r = lr[k];
            t += (float)cia_tau(cont, cp, nud, r.vmr_h2o, r.vmr_co2, r.p_mid, r.T_mid, r.dz_cm);
        }
        if (cont.mask & 3) {
            const float rad = radfn32(nu, c.c2_mid);
            float k_c = 0.f;
            if (cont.mask & 1) k_c = fmaf(Cs * exp2f(te * c.l2_296), c.h2o_self, Cf * c.h2o_for);
            if (cont.mask & 2) k_c = fmaf(Se * (td == 0.f ? 1.f : exp2f(td * c.l2_246)), c.co2, k_c);
            t = fmaf(k_c, rad, t);
        }
        return t * imu;
    };
    const int k1 = (int)((long long)L * (G - g) / G), k0 = (int)((long long)L * (G - 1 - g) / G);
    double od = 0.0;        // cumulative optical depth from the top of the run
    double Tr_up = 1.0;     // transmittance of the level above
    double D = 0.0;         // downwelling radiance at the current bottom (reflecting surface)
    float Is = 0.f, Ic = 0.f;  // radiance, Kahan-compensated
    float B_up = k1 > k0 ? planck32(c1nu3, nu2, lc[k1 - 1].c2_top) : 0.f;  // B at the top level of the current layer
    for (int k = k1 - 1; k >= k0; --k) {
        const RteLayerF& c = lc[k];
        const float s = slant(k);
        od += (double)s;
        const double Tr_k = exp(-od);
        const float dT = (float)(Tr_up - Tr_k);
        const float B_bot = planck32(c1nu3, nu2, c.c2_bot);
        float v, em = 0.f;
        if (src == 0) {
            const float Ba = planck32(c1nu3, nu2, c.c2_ave), f = cim_corr32(s);
            v = fmaf(Ba, dT, (B_up - Ba) * (dT * f));
            if (refl) em = -expm1f(-s) * fmaf(B_bot - Ba, f, Ba);
        } else {
            const float f = lit_corr32(s);
            v = fmaf(B_up, dT, (B_bot - B_up) * ((float)Tr_up * f));
            if (refl) em = fmaf(B_bot, -expm1f(-s), (B_up - B_bot) * f);
        }
        if (refl) D = fma(D, exp(-(double)s), (double)em);  // add_reflected_downwelling!
        kahan_add32(Is, Ic, v);
        B_up = B_bot;
        Tr_up = Tr_k;
    }
    sO[g][pt] = od;
    sI[g][pt] = (double)Is - (double)Ic;
    sD[g][pt] = D;
    __syncthreads();
    if (g == 0 && i_raw < n_nu) {
        double ot = 0.0, Tt = 1.0, It = 0.0, Dt = 0.0;
#pragma unroll
        for (int q = 0; q < G; ++q) {
            It = fma(Tt, sI[q][pt], It);
            if (refl) Dt = fma(Dt, exp(-sO[q][pt]), sD[q][pt]);
            ot += sO[q][pt];
            Tt = exp(-ot);
        }
        It += pr.eps * (double)planck32(c1nu3, nu2, split_f(1.4387769 / pr.T_sfc)) * Tt;
        if (refl) It += (1.0 - pr.eps) * Dt * Tt;
        I[(size_t)p * n_nu + i] = It;
    }
}

// ---------------------------------------------------------------- ILS
// ils.jl:80-114: raw taps, then area normalisation
__global__ void ils_taps_kernel(double dnu, double opd_max, double fwhm, int apod, long long n_half,
                                double* __restrict__ kern) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k > 2 * n_half) return;
    const int n_pts = 2048;
    const double dL = opd_max / (n_pts - 1);
    const double dv = double(k - n_half) * dnu;
    const double sg = fwhm / (2.0 * sqrt(2.0 * log(2.0)));
    const double nb[3][3] = {{0.384093, 0.087577, 0.528330},
                             {0.152442, 0.136176, 0.711382},
                             {0.045335, 0.554883, 0.399782}};
    double s = 0.0;
    for (int j = 0; j < n_pts; ++j) {
        const double L = (double(j) / double(n_pts - 1)) * opd_max;
        double A;
        if (apod == 0) A = exp(-(2.0 * (M_PI * M_PI)) * (sg * sg) * (L * L));
        else {
            const double x = L / opd_max;
            const double t = 1.0 - x * x;
            A = fabs(x) > 1.0 ? 0.0 : nb[apod - 1][0] + nb[apod - 1][1] * t * t + nb[apod - 1][2] * (t * t) * (t * t);
        }
        s += A * cos(2.0 * M_PI * L * dv);
    }
    kern[k] = 2.0 * s * dL;
}
__global__ void ils_normalise_kernel(double* kern, long long n, double dnu) {
    __shared__ double part[1024];
    double s = 0.0;
    for (long long k = threadIdx.x; k < n; k += blockDim.x) s += kern[k];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int d = blockDim.x / 2; d; d >>= 1) {
        if ((int)threadIdx.x < d) part[threadIdx.x] += part[threadIdx.x + d];
        __syncthreads();
    }
    const double tot = part[0] * dnu;
    __syncthreads();
    for (long long k = threadIdx.x; k < n; k += blockDim.x) kern[k] /= tot;
}

// Channels on grid nodes at a constant step: channel c reads the convolution at node
// first + c step, and the linear resampling (sounder.jl:372-377) has weight 0.  Found on
// the host from the grids' exact rational forms; step 0 where it does not hold (or the
// step is outside 16..256, where apod_at serves).
struct ChanNodes {
    int first, step;
};
constexpr int kChanThreads = 256;

// The convolution at C consecutive channels, one CTA: sum[c] = sum_k X[base + c step + k]
// kern[k], X zero outside [0, n_nu).  A thread takes one phase r of the step (of the
// kChanThreads / T splits of the rows m) and walks the points r + m step; the taps that a
// point meets in the C channels are C rows of the same phase, so a ring of C registers holds
// them and each point costs two coalesced loads for C products.  One warp per channel and
// two loads per product, as apod_at does it, left 221 channels of one scene waiting on 400
// dependent loads (94 us, now 13).  jg_channel_nodes_kernel does the same for the Jacobian.
// Returns the sum of channel threadIdx.x to the first C threads.
template <typename T, int C>
__device__ __forceinline__ T chan_sums(const T* __restrict__ X, int n_nu, const T* __restrict__ kern, int n_taps,
                                       int base, int step) {
    __shared__ T part[kChanThreads / 32][C];
    const int lanes = (step + 31) & ~31;            // threads per split
    const int splits = kChanThreads / lanes;
    const int r = threadIdx.x % lanes, sp = threadIdx.x / lanes;
    const int M = (n_taps + step - 1) / step + C - 1;  // rows m in which some tap is met
    const int per = ((M + splits - 1) / splits + C - 1) / C * C;
    T acc[C], ring[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = ring[c] = T(0);
    if (r < step && sp < splits) {
        const int m0 = sp * per, m1 = min(M, m0 + per);
#pragma unroll
        for (int u = 1; u < C; ++u) {  // the rows before this split's
            const int m = m0 - C + u, k = r + m * step;
            if (m >= 0 && k < n_taps) ring[u] = kern[k];
        }
        for (int mb = m0; mb < m1; mb += C) {
            T x[C];
#pragma unroll
            for (int u = 0; u < C; ++u) {
                const int j = base + r + (mb + u) * step;
                x[u] = (mb + u < m1 && (unsigned)j < (unsigned)n_nu) ? X[j] : T(0);
            }
#pragma unroll
            for (int u = 0; u < C; ++u) {
                const int k = r + (mb + u) * step;
                ring[u] = k < n_taps ? kern[k] : T(0);
#pragma unroll
                for (int c = 0; c < C; ++c) acc[c] = fma(x[u], ring[(u - c + C) % C], acc[c]);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        T v = acc[c];
#pragma unroll
        for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        if (lane == 0) part[warp][c] = v;
    }
    __syncthreads();
    T tot = T(0);
    if (threadIdx.x < C) {
#pragma unroll
        for (int w = 0; w < kChanThreads / 32; ++w) tot += part[w][threadIdx.x];
    }
    return tot;
}

__device__ __forceinline__ double brightness_t(double nu, double R) {  // planck.jl:53-57
    return R <= 0.0 ? 0.0 : 1.4387769 * nu / log1p(1.191042953e-5 * (nu * nu * nu) / R);
}

// R and BT of 8 channels per CTA (channels on grid nodes, with the ILS)
constexpr int kIlsChan = 8;
__global__ void __launch_bounds__(kChanThreads) ils_nodes_kernel(const double* __restrict__ I, int n_nu,
                                                                 const double* __restrict__ kern, int n_taps,
                                                                 double dnu_hi, GridDev ch, ChanNodes nodes,
                                                                 double* __restrict__ R, double* __restrict__ BT) {
    const int c0 = blockIdx.x * kIlsChan, p = blockIdx.y;
    const double v = chan_sums<double, kIlsChan>(I + (size_t)p * n_nu, n_nu, kern, n_taps,
                                                 nodes.first + c0 * nodes.step - (n_taps - 1) / 2, nodes.step);
    const int c = c0 + (int)threadIdx.x;
    if (threadIdx.x < kIlsChan && c < ch.n) {
        const double Rv = v * dnu_hi;
        R[(size_t)p * ch.n + c] = Rv;
        BT[(size_t)p * ch.n + c] = brightness_t(ch.at(c), Rv);
    }
}

__device__ double apod_at(const double* __restrict__ Ip, long long n_nu, const double* __restrict__ kern,
                          long long n_taps, long long i, int lane) {
    const long long half = (n_taps - 1) / 2;
    double acc = 0.0;
    for (long long k = lane; k < n_taps; k += 32) {
        const long long j = i + k - half;
        if (j >= 0 && j < n_nu) acc = fma(Ip[j], kern[k], acc);
    }
    for (int d = 16; d; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    return acc;
}

__global__ void __launch_bounds__(256) ils_bt_kernel(const double* __restrict__ I, long long n_nu,
                                                     const double* __restrict__ kern, long long n_taps,
                                                     double dnu_hi, GridDev g, GridDev ch, int with_ils,
                                                     double* __restrict__ R, double* __restrict__ BT) {
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int p = blockIdx.y;
    if (wid >= ch.n) return;
    const double nu = ch.at(wid);
    const double* Ip = I + (size_t)p * n_nu;
    auto value = [&](long long i) -> double {
        if (!with_ils) return Ip[i];
        return apod_at(Ip, n_nu, kern, n_taps, i, lane) * dnu_hi;
    };
    double Rv;
    const double g0 = g.at(0), gl = g.at(n_nu - 1);
    if (nu <= g0) Rv = value(0);
    else if (nu >= gl) Rv = value(n_nu - 1);
    else {
        long long i = (long long)floor((nu - g0) / dnu_hi);
        i = max(0LL, min(i, n_nu - 2));
        while (i > 0 && g.at(i) > nu) --i;
        while (i + 2 < n_nu && g.at(i + 1) <= nu) ++i;
        const double a = g.at(i), b = g.at(i + 1);
        const double w = (nu - a) / (b - a);
        const double r0 = value(i);
        Rv = w == 0.0 ? r0 : r0 * (1.0 - w) + value(i + 1) * w;
    }
    if (lane == 0) {
        R[(size_t)p * ch.n + wid] = Rv;
        BT[(size_t)p * ch.n + wid] = brightness_t(nu, Rv);
    }
}

}  // namespace irs
