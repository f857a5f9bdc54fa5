// Per-cell kernels of the sampling path:
//   yields_kernel         FSSW::calculate_dN_dxtdy_for_one_particle_species
//                         + calculate_dN_analytic (src/FSSW.cpp:565-848) for every
//                           (cell, species) pair
//   cdf kernels           RandomVariable1DArray (src/RandomVariable1DArray.cpp:25-74):
//                         per-species fixed-point prefix sums of the cell yields
#include <cuda_runtime.h>

#include <algorithm>

#include "device_common.cuh"
#include "kernels.h"

namespace iss {

namespace {

constexpr float kHbarCf = 0.197327053f;

// ------------------------------------------------------------------------
// special functions off the table (x < 0.5 or x > 399.95): direct
// evaluation of K_n from its integral representation (trapezoidal rule)
__device__ double bessel_k_direct(int n, double x) {
    if (x > 700.0) return 0.0;
    const double h = fmin(0.02, 0.5 / sqrt(x));
    double acc = 0.5;
    for (int k = 1; k < 20000; k++) {
        const double t = k * h;
        const double lg = n * t - x * (cosh(t) - 1.0);
        acc += 0.5 * exp(lg) * (1.0 + exp(-2.0 * n * t));
        if (lg < -70.0) break;
    }
    return acc * h * exp(-x);
}

__device__ double expint_direct(int n, double x) {
    if (x > 1.0) {
        double b = x + n, c = 1e300, d = 1.0 / b, h = d;
        for (int i = 1; i < 10000; i++) {
            const double a = -static_cast<double>(i) * (n - 1 + i);
            b += 2.0;
            d = 1.0 / (a * d + b);
            c = b + a / c;
            const double del = c * d;
            h *= del;
            if (fabs(del - 1.0) < 1e-16) break;
        }
        return h * exp(-x);
    }
    const double ge = 0.57721566490153286061;
    double psi = -ge;
    for (int k = 1; k < n; k++) psi += 1.0 / k;
    double sum = (n == 1) ? (-log(x) - ge) : 1.0 / (n - 1);
    double term = 1.0;
    for (int m = 1; m < 500; m++) {
        term *= -x / m;
        const double del = (m != n - 1) ? -term / (m - n + 1) : term * (psi - log(x));
        sum += del;
        if (fabs(del) < 1e-17 * fabs(sum)) break;
    }
    return sum;
}

// Position of a float-float argument on the special-function grid.
struct GridPos {
    int idx;
    float frac;
    bool on_table;
};

__device__ __forceinline__ GridPos grid_pos(float xh, float xl) {
    GridPos g;
    g.on_table = (xh >= 0.5f) && (xh <= 399.95f);
    float s, se;
    two_sum(xh, -0.5f, s, se);
    se += xl;
    float ph, pe;
    two_prod(s, 20.0f, ph, pe);
    const float pl = fmaf(20.0f, se, pe);
    int idx = static_cast<int>(floorf(ph));
    float f = (ph - static_cast<float>(idx)) + pl;
    const bool below = f < 0.0f, above = f >= 1.0f;
    idx += static_cast<int>(above) - static_cast<int>(below);
    f = below ? f + 1.0f : (above ? f - 1.0f : f);
    g.idx = min(max(idx, 0), 7989);
    g.frac = f;
    return g;
}

// ------------------------------------------------------------------------
constexpr int kYieldThreads = 128;
constexpr int64_t kTwoCellsFrom = 2500;
constexpr int kYieldGroups = 4;   // species groups per cell (grid y)

// Surface of cell l in a batch: the last b with surf[b].c0 <= l.
__device__ __forceinline__ int surface_of(const SurfSeg* __restrict__ surf, int n_surf, int64_t l) {
    int lo = 0, hi = n_surf - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (surf[mid].c0 <= l) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Form of the bulk correction of the yields (include_deltaf_bulk): none (also
// for the kinds without a yield term), Chapman-Enskog (kinds 1 and 21), the
// 14-moment form (kind 11)
constexpr int kNoBulk = 0, kBulkCe = 1, kBulk14 = 2;

// Per-cell quantities shared by every species' yield in cell l.
struct CellYieldIn {
    float T, b_hi, b_lo;
    bool warm;
    float da0, bulkPi, dsq, pref_q, inv_kappa, unit_pref;
    float4 th, th2, cf;
};

// Sums of the thermal series (calculate_dN_analytic, src/FSSW.cpp:719-848) of
// one species in one cell: they depend on the species only through its
// float-float mass, statistics, number of terms and chemical potential mu.
struct SeriesSums {
    float Neq, b1, b2, b3, q1, q2;
};

// Term nn of the series, with what the terms share: x1 = m beta and
// bm = beta mu as float-float numbers.  kFirst: nn = 1, where n x and the
// divisions by n drop out (nine species in ten have this term only).  A
// division by n = 2, 4, 8 is a multiplication by the exact 1 / n: the same
// correctly rounded quotient.  kTable: an argument off the special-function
// table only sets off; without it, it is evaluated directly as well.
template <int kBulk, bool kDiff, bool kFirst, bool kTable>
__device__ __forceinline__ void series_term(const DevConfig& cfg, const CellYieldIn& c, int nn, float theta,
                                            float x1_h, float x1_l, float bm_h, float bm_l, bool no_mu,
                                            float mbeta, SeriesSums& s, bool& off) {
    const float fn = kFirst ? 1.0f : static_cast<float>(nn);
    // x_n = n m beta
    float xh = x1_h, xl = x1_l;
    if (!kFirst) {
        float xe;
        two_prod(fn, x1_h, xh, xe);
        xl = fmaf(fn, x1_l, xe);
    }
    // lambda^n = exp(n beta mu)
    float fug = 1.0f;
    if (!no_mu) {
        float ah = bm_h, al = bm_l;
        if (!kFirst) {
            float ae;
            two_prod(fn, bm_h, ah, ae);
            al = fmaf(fn, bm_l, ae);
        }
        fug = expf(ah) * (1.0f + al);
    }
    const GridPos g = grid_pos(xh, xl);
    if (!g.on_table) off = true;
    float K1, K2, K3;
    if (kTable || g.on_table) {
        const float4 ka = __ldg(cfg.tab.sfK + g.idx);
        const float4 kb = __ldg(cfg.tab.sfK + g.idx + 1);
        K1 = fmaf(g.frac, kb.x - ka.x, ka.x);
        K2 = fmaf(g.frac, kb.y - ka.y, ka.y);
        K3 = fmaf(g.frac, kb.z - ka.z, ka.z);
    } else {
        const double xd = static_cast<double>(xh) + static_cast<double>(xl);
        K2 = static_cast<float>(bessel_k_direct(2, xd));
        K1 = kBulk != kNoBulk ? static_cast<float>(bessel_k_direct(1, xd)) : 0.0f;
        K3 = kBulk == kBulk14 ? static_cast<float>(bessel_k_direct(3, xd)) : 0.0f;
    }
    const float tf = theta * fug;
    float tf_n = tf, k2_n = 3.0f * K2, k3_n = 3.0f * K3;
    if (!kFirst) {
        if ((nn & (nn - 1)) == 0) {
            const float r = 1.0f / fn;
            tf_n *= r;
            k2_n *= r;
            k3_n *= r;
        } else {
            tf_n = tf_n / fn;
            if (kBulk != kNoBulk) k2_n = k2_n / fn;
            if (kBulk == kBulk14) k3_n = k3_n / fn;
        }
    }
    s.Neq = fmaf(tf_n, K2, s.Neq);
    if (kBulk == kBulkCe) {
        s.b1 = fmaf(tf, fmaf(mbeta, K1, k2_n), s.b1);
        s.b2 = fmaf(tf, K1, s.b2);
    } else if (kBulk == kBulk14) {
        s.b1 = fmaf(tf, K2, s.b1);
        s.b2 = fmaf(tf, fmaf(mbeta, K1, k2_n), s.b2);
        s.b3 = fmaf(tf, fmaf(mbeta, K2, k3_n), s.b3);
    }
    if (kDiff) {
        s.q1 = fmaf(tf_n, K2, s.q1);
        float En[9];
        if (kTable || g.on_table) {
            // rows of 12 floats: three 16-byte reads each
            const float4* ea = cfg.tab.sfE + 3 * g.idx;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const float4 a = __ldg(ea + i), b = __ldg(ea + 3 + i);
                En[4 * i] = fmaf(g.frac, b.x - a.x, a.x);
                if (i < 2) {
                    En[4 * i + 1] = fmaf(g.frac, b.y - a.y, a.y);
                    En[4 * i + 2] = fmaf(g.frac, b.z - a.z, a.z);
                    En[4 * i + 3] = fmaf(g.frac, b.w - a.w, a.w);
                }
            }
        } else {
            const double xd = static_cast<double>(xh) + static_cast<double>(xl);
            En[0] = static_cast<float>(expint_direct(2, xd));
            for (int i = 1; i < 9; i++) En[i] = static_cast<float>(expint_direct(2 * i + 2, xd));
        }
        const float arg = xh;
        const float em = expf(-xh) * (1.0f - xl);
        float I = fmaf(0.375f, En[0], __fmul_rn(em / arg, 2.0f / __fmul_rn(arg, arg) + 2.0f / arg - 0.5f));
        // 3 (2k-5)!! / (2^k k!) for k = 3..10
        const float ck[8] = {0.0625f, 0.0234375f, 0.01171875f, 0.0068359375f,
                             0.00439453125f, 0.0030212402343750f,
                             0.0021820068359375f, 0.0016365051269531f};
#pragma unroll
        for (int k2 = 0; k2 < 8; k2++) I = fmaf(ck[k2], En[k2 + 1], I);
        I = -(mbeta * mbeta * mbeta) * I;
        s.q2 = fmaf(fn * tf, I, s.q2);
    }
}

template <int kBulk, bool kDiff, bool kTable>
__device__ __forceinline__ SeriesSums thermal_series(const DevConfig& cfg, const CellYieldIn& c,
                                                     const YieldGroup& gr, float mu, bool& off) {
    const float b_hi = c.b_hi, b_lo = c.b_lo;
    // beta*mu and m*beta as float-float numbers
    float bm_h, bm_e;
    two_prod(mu, b_hi, bm_h, bm_e);
    const float bm_l = fmaf(mu, b_lo, bm_e);
    float x1_h, x1_e;
    two_prod(gr.m_hi, b_hi, x1_h, x1_e);
    const float x1_l = x1_e + fmaf(gr.m_hi, b_lo, gr.m_lo * b_hi);
    const bool no_mu = mu == 0.0f;   // exp(0) = 1
    const float mbeta = x1_h + x1_l;
    SeriesSums s{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    series_term<kBulk, kDiff, true, kTable>(cfg, c, 1, 1.0f, x1_h, x1_l, bm_h, bm_l, no_mu, mbeta, s, off);
    if (gr.light && c.warm) {
        for (int nn = 2; nn <= 10; nn++) {
            float theta = 1.0f;
            if (gr.sign == 1 && (nn % 2 == 0)) theta = -1.0f;
            if (gr.sign == 0) theta = 0.0f;
            series_term<kBulk, kDiff, false, kTable>(cfg, c, nn, theta, x1_h, x1_l, bm_h, bm_l, no_mu, mbeta, s, off);
        }
    }
    return s;
}

// The yield of calculate_dN_dxtdy_for_one_particle_species
// (src/FSSW.cpp:565-715) is, for a species of degeneracy g and baryon number
// B, g (X + B Y): X and Y hold the prefactor, the equilibrium sum and the
// bulk and diffusion terms, and depend on the species only through the
// quantities its group shares (mass and the series sums).  They are formed
// once per series; each member then costs one multiply-add.
template <int kBulk, bool kDiff>
__device__ __forceinline__ float2 yield_coefs(const CellYieldIn& c, const YieldGroup& gr,
                                              const SeriesSums& ss) {
    const float T = c.T;
    const float4 cf = c.cf;
    const float mass = gr.m_hi + gr.m_lo;
    const float m2 = mass * mass;
    // (the products and fused multiply-adds are spelled out: the yields feed the
    // integer CDF, so every build has to round them alike)
    float x = __fmul_rn(m2 * T, ss.Neq);
    float y = 0.0f;
    if (kBulk == kBulkCe) {
        const float r1 = __fmul_rn(m2 * T, ss.b1);
        x = fmaf(__fmul_rn(-c.bulkPi, cf.x), fmaf(m2 * mass / 3.0f, ss.b2, -__fmul_rn(cf.y, r1)), x);
    } else if (kBulk == kBulk14) {
        const float r1 = __fmul_rn(m2 * T, ss.b1);
        const float r2 = __fmul_rn(m2 * T * T, ss.b2);
        const float r3 = __fmul_rn(m2 * mass * T * T, ss.b3);
        x = fmaf(c.bulkPi, fmaf(__fmul_rn(r1, m2), cf.x, __fmul_rn(r3, cf.z)), x);
        y = __fmul_rn(__fmul_rn(c.bulkPi, r2), cf.y);
    }
    if (kDiff) {
        const float r4 = __fmul_rn(m2 * T * T, ss.q1);
        const float r5 = __fmul_rn(T * T * T / 3.0f, ss.q2);
        const float dq = __fmul_rn(c.dsq, c.inv_kappa);
        x = fmaf(x, c.da0, -__fmul_rn(__fmul_rn(dq, c.pref_q), r4));
        y = fmaf(y, c.da0, -__fmul_rn(dq, r5));
    } else {
        x = __fmul_rn(x, c.da0);
        y = __fmul_rn(y, c.da0);
    }
    return make_float2(c.unit_pref * x, c.unit_pref * y);
}

// negative -> 0 (FSSW::calculate_dN_dxtdy_for_one_particle_species,
// src/FSSW.cpp:707); NaN -> 0; +inf -> FLT_MAX so the cell CDF stays
// finite; -0 -> +0 so the bits order as the values
__device__ __forceinline__ float member_yield(const float4& q, float2 xy) {
    const float total = q.w * fmaf(q.x, xy.y, xy.x);
    return __uint_as_float(__float_as_uint(fminf(fmaxf(total, 0.0f), 3.40282347e38f)) & 0x7FFFFFFFu);
}

// Per-cell quantities of cell l (not dropped: u.dsigma >= 0)
template <int kBulk, bool kDiff>
__device__ __forceinline__ CellYieldIn cell_yield_in(const DevConfig& cfg, const CellArrays& cells,
                                                     int64_t l, const float4& da) {
    CellYieldIn c;
    c.th = cells.th[l];
    c.th2 = cells.th2[l];
    c.cf = cells.coef[l];
    const float T = c.th.x;
    const float2 beta = cells.beta[l];
    c.T = T;
    c.da0 = da.x;
    c.b_hi = beta.x;
    c.b_lo = beta.y;
    c.warm = T >= 0.05f;   // as double: T > 0.05 (0.05f is the first float above it)
    c.bulkPi = 0.0f;
    if (kBulk != kNoBulk) c.bulkPi = cfg.bulk_kind == 1 ? c.th2.w / kHbarCf : c.th2.w;
    c.dsq = c.pref_q = c.inv_kappa = 0.0f;
    if (kDiff) {
        const float4 p2 = cells.pi2[l];
        c.dsq = fmaf(p2.w, da.w, fmaf(p2.y, da.y, __fmul_rn(p2.z, da.z)));
        c.pref_q = c.th2.z / (c.th2.x + c.th2.y);
        c.inv_kappa = 1.0f / c.cf.w;
    }
    // formed once: without this the compiler repeats the FP64 and FP32
    // divisions in every term rather than hold their results
    asm volatile("" : "+f"(c.b_hi), "+f"(c.b_lo), "+f"(c.bulkPi));
    if (kDiff) asm volatile("" : "+f"(c.dsq), "+f"(c.pref_q), "+f"(c.inv_kappa));
    // (1/hbarc^3) / (2 pi^2)
    c.unit_pref = (1.0f / (0.197327053f * 0.197327053f * 0.197327053f)) / (2.0f * 9.8696044010893586f);
    return c;
}

// The yields of cell l (a lane's; past the last cell the lane only takes part)
// for the groups of row blockIdx.y, whatever the chemical potentials and the
// surfaces of the warp's cells: b is the block's surface, or -1 where it has
// several.
template <int kBulk, bool kDiff>
__device__ __forceinline__ void yields_any(const DevConfig& cfg, const CellArrays& cells, float* __restrict__ yields,
                                        uint32_t* __restrict__ ymax, uint32_t* __restrict__ off_table, int64_t l,
                                        int b, const YieldGroup* s_g, const int32_t* s_gst,
                                        const float4* s_q, const int32_t* s_rst, const int32_t* s_mem,
                                        uint32_t* s_rmax, uint32_t* s_max) {
    const int nsp = cfg.n_species, G = cfg.n_ygroups;
    const int64_t n = cfg.n_cells;
    const bool one_surface = b >= 0;
    const bool valid = l < n;
    const int64_t lc = valid ? l : 0;   // lanes past the last cell read cell 0 and store nothing
    const float4 da = cells.da[lc];
    const bool live = valid && !(da.x < 0.0f);
    const CellYieldIn c = cell_yield_in<kBulk, kDiff>(cfg, cells, lc, da);
    uint32_t* ymax_row = ymax + static_cast<int64_t>(
        one_surface ? b : surface_of(cfg.surf, cfg.n_surfaces, valid ? l : n - 1)) * nsp;
    float* out = yields + l;
    const bool by_run = __all_sync(0xffffffffu, c.th.z == 0.0f && c.th.w == 0.0f);
    for (int g = blockIdx.y; g < G; g += gridDim.y) {
        const YieldGroup gr = s_g[g];
        const int r0 = s_gst[g], r1 = s_gst[g + 1];
        float2 xy = make_float2(0.0f, 0.0f);
        float mu_of = __int_as_float(0x7fc00000);   // mu of xy: none yet
        for (int r = r0; r < r1; r++) {
            const int t0 = s_rst[r], t1 = s_rst[r + 1];
            for (int t = t0; t < t1; t++) {
                const float4 q = s_q[t];    // baryon number, strangeness, charge, degeneracy
                float yv = 0.0f;
                if (live) {
                    const float mu = q.x * c.th.y + q.y * c.th.z + q.z * c.th.w;
                    if (mu != mu_of) {
                        bool off = false;
                        xy = yield_coefs<kBulk, kDiff>(c, gr, thermal_series<kBulk, kDiff, true>(cfg, c, gr, mu, off));
                        mu_of = mu;
                        if (off) {   // yields_off_table_kernel
                            xy = make_float2(0.0f, 0.0f);
                            *off_table = 1u;
                        }
                    }
                    yv = member_yield(q, xy);
                }
                if (one_surface) {
                    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(yv));
                    if ((threadIdx.x & 31) == 0 && m) atomicMax(by_run ? s_rmax + r : s_max + t, m);
                }
                if (by_run) {
                    if (!one_surface && yv > 0.0f)
                        for (int u = t0; u < t1; u++) atomicMax(ymax_row + s_mem[u], __float_as_uint(yv));
                    if (valid)
                        for (int u = t0; u < t1; u++) out[static_cast<int64_t>(s_mem[u]) * n] = yv;
                    break;
                }
                if (!one_surface && yv > 0.0f) atomicMax(ymax_row + s_mem[t], __float_as_uint(yv));
                if (valid) out[static_cast<int64_t>(s_mem[t]) * n] = yv;
            }
        }
    }
}

// Yields of every (cell, species) pair, kCells cells per thread.  A group's
// series runs for its first run and is reused by the next ones while their
// chemical potential is the same in the warp's cells.  In a warp whose cells
// have no strangeness and charge potential (and lie, with the block's others, on
// one surface) mu and with it the yield is the same for a whole run: a run costs
// one multiply-add and one maximum, a member only its store.  Other warps take
// yields_any, where each member forms its mu.
//
// Besides the yields, the kernel raises ymax[b S + k] to the largest yield of
// species k on surface b (its float bits: yields are >= +0, so the unsigned
// order of the bits is the order of the values; ymax starts at 0): through a
// per-block maximum in shared memory when the block's cells lie on one surface,
// else lane by lane.
//
// Series with an argument off the special-function tables (x < 0.5: pions
// above 0.27 GeV; x > 399.95) are left at zero and flagged, for
// yields_off_table_kernel: the FP64 evaluation, inlined here, had its set-up
// run for every term of every cell.
//
// Bound by instruction issue (75 % of the issue slots; 64 M of 136 M warp
// instructions are the series of 200,000 cells): some 100 one-term and 5
// ten-term series per cell, and 319 stores.  Two cells per thread share a run's
// look-up, maximum and addresses; with 1/T from the prologue (its FP64 division
// ran once per row of groups) and the runs as one 16-byte record each, 200,000
// cells with 319 species and 14-moment bulk take 168 us (228 with a look-up per
// member, 345 with the FP64 set-up in the loop).  Three cells measure the same,
// four 4 us more, one cell 12 to 30 us more.  With diffusion, whose longer
// series leave less to share, two cells gain nothing at 100,000 cells (231 us
// either way; 246 and 590 before) and lose below (6,000 cells: 40 us, 34 with
// one), so there is no such variant.  Where every cell has a strangeness and
// charge potential 100,000 cells take 212 us, with diffusion 456 us.  7 blocks
// per SM, 5 with diffusion: 6 and 5 take 172 and 182 us, 6 and 7 with
// diffusion 237 us.
// kDiff: include_deltaf_diffusion (a separate instantiation, so the common
// case carries none of the diffusion series' registers).
template <int kBulk, bool kDiff, int kCells>
__global__ void __launch_bounds__(kYieldThreads, kDiff ? 5 : 7)
yields_kernel(DevConfig cfg, CellArrays cells, float* __restrict__ yields, uint32_t* __restrict__ ymax,
              uint32_t* __restrict__ off_table) {
    extern __shared__ float4 s_dyn[];
    __shared__ int s_b[2];
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int kBlockCells = kYieldThreads * kCells;
    const int nsp = cfg.n_species;
    const int G = cfg.n_ygroups, R = cfg.n_yruns;
    // the yield list as it is, then the runs' and members' maxima; the members'
    // own entries (s_q, s_rst, s_mem) are staged only in blocks that read them
    const int words4 = yield_list_float4(nsp, G, R);
    const YieldGroup* s_g = reinterpret_cast<const YieldGroup*>(s_dyn);
    const float4* s_run = s_dyn + G;   // YieldRun
    const float4* s_q = s_run + R;
    const int32_t* s_gst = reinterpret_cast<const int32_t*>(s_q + nsp);
    const int32_t* s_rst = s_gst + G + 1;
    const int32_t* s_mem = s_rst + R + 1;
    const int32_t* rst = reinterpret_cast<const int32_t*>(cfg.ylist + G + R + nsp) + G + 1;
    const int32_t* mem = rst + R + 1;
    uint32_t* s_rmax = reinterpret_cast<uint32_t*>(s_dyn + words4);
    uint32_t* s_max = s_rmax + R;
    const int64_t n = cfg.n_cells;
    const int64_t first = static_cast<int64_t>(blockIdx.x) * kBlockCells;
    const int gst4 = G + R + nsp;      // the float4 of s_gst
    for (int k = threadIdx.x; k < G + R; k += kYieldThreads) s_dyn[k] = cfg.ylist[k];
    for (int k = gst4 + threadIdx.x; k < gst4 + (G + 4) / 4; k += kYieldThreads) s_dyn[k] = cfg.ylist[k];
    for (int k = threadIdx.x; k < nsp + R; k += kYieldThreads) s_rmax[k] = 0u;
    if (threadIdx.x < 2) {
        const int64_t lb = threadIdx.x == 0 ? first : min(first + kBlockCells, n) - 1;
        s_b[threadIdx.x] = surface_of(cfg.surf, cfg.n_surfaces, lb);
    }
    __syncthreads();
    const bool one_surface = s_b[0] == s_b[1];
    // a warp's cells are consecutive, a lane's 32 apart
    const int64_t l0 = first + (threadIdx.x >> 5) * (32 * kCells) + (threadIdx.x & 31);
    CellYieldIn c[kCells];
    bool live[kCells];
    bool usual = one_surface && first + kBlockCells <= n && n < (int64_t(1) << 30) && nsp <= kMaxRunSpecies;
#pragma unroll
    for (int j = 0; j < kCells; j++) {
        const int64_t l = min(l0 + 32 * j, n - 1);
        const float4 da = cells.da[l];
        live[j] = !(da.x < 0.0f);
        c[j] = cell_yield_in<kBulk, kDiff>(cfg, cells, l, da);
        usual = usual && c[j].th.z == 0.0f && c[j].th.w == 0.0f;
    }
    if (__syncthreads_or(!usual)) {
        for (int k = G + R + threadIdx.x; k < words4; k += kYieldThreads) s_dyn[k] = cfg.ylist[k];
        __syncthreads();
    }
    // blockIdx.y picks every gridDim.y-th species group: the groups come in
    // decreasing order of work, so interleaving keeps the rows' work equal,
    // and the grid has several waves of blocks
    if (__all_sync(FULL, usual)) {
        // the usual warp: mu is B muB for all its cells, so the loop over the
        // runs has no branch that lanes take apart
        const uint32_t row_bytes = static_cast<uint32_t>(n) * 4u;
        char* const out_bytes = reinterpret_cast<char*>(yields + l0);
        for (int g = blockIdx.y; g < G; g += gridDim.y) {
            const YieldGroup gr = s_g[g];
            const int r1 = s_gst[g + 1];
            float2 xy[kCells];
            float mu_of[kCells];   // mu of xy: none yet
#pragma unroll
            for (int j = 0; j < kCells; j++) mu_of[j] = __int_as_float(0x7fc00000);
#pragma unroll 1
            for (int r = s_gst[g]; r < r1; r++) {
                const float4 run = s_run[r];   // YieldRun
                bool other_mu = false;
#pragma unroll
                for (int j = 0; j < kCells; j++) other_mu = other_mu || run.x * c[j].th.y != mu_of[j];
                if (__any_sync(FULL, other_mu)) {
#pragma unroll
                    for (int j = 0; j < kCells; j++) {
                        bool off = false;
                        mu_of[j] = run.x * c[j].th.y;
                        xy[j] = yield_coefs<kBulk, kDiff>(
                            c[j], gr, thermal_series<kBulk, kDiff, true>(cfg, c[j], gr, mu_of[j], off));
                        if (off) {   // yields_off_table_kernel
                            xy[j] = make_float2(0.0f, 0.0f);
                            if (live[j]) *off_table = 1u;
                        }
                    }
                }
                const float4 q = make_float4(run.x, 0.0f, 0.0f, run.y);
                float yv[kCells];
                uint32_t m = 0u;
#pragma unroll
                for (int j = 0; j < kCells; j++) {
                    yv[j] = live[j] ? member_yield(q, xy[j]) : 0.0f;
                    m = max(m, __float_as_uint(yv[j]));
                }
                m = __reduce_max_sync(FULL, m);
                if ((threadIdx.x & 31) == 0) atomicMax(s_rmax + r, m);
                const uint32_t m01 = __float_as_uint(run.z), m23 = __float_as_uint(run.w);
                const uint32_t id[kRunMembers] = {m01 & 0xFFFFu, m01 >> 16, m23 & 0xFFFFu, m23 >> 16};
#pragma unroll
                for (int i = 0; i < kRunMembers; i++) {
                    if (i > 0 && id[i] == 0xFFFFu) continue;
                    char* const at = out_bytes + static_cast<uint64_t>(id[i]) * row_bytes;
#pragma unroll
                    for (int j = 0; j < kCells; j++) reinterpret_cast<float*>(at)[32 * j] = yv[j];
                }
            }
        }
    } else {
#pragma unroll 1
        for (int j = 0; j < kCells; j++) {
            const int64_t l = l0 + 32 * j;
            yields_any<kBulk, kDiff>(cfg, cells, yields, ymax, off_table, l, one_surface ? s_b[0] : -1, s_g, s_gst,
                                     s_q, s_rst, s_mem, s_rmax, s_max);
        }
    }
    if (one_surface) {
        __syncthreads();
        for (int r = threadIdx.x; r < R; r += kYieldThreads)
            for (int t = rst[r]; t < rst[r + 1]; t++) {
                const uint32_t m = max(s_max[t], s_rmax[r]);
                if (m) atomicMax(ymax + static_cast<int64_t>(s_b[0]) * nsp + mem[t], m);
            }
    }
}

// Whether a term of the group's series has an argument off the special-function
// tables in this cell (thermal_series: n x_1 grows with n, so the first and the
// last term tell) and the direct evaluation gives other than the zero that
// yields_kernel left (K_n is zero above 700, in every term above x_1)
__device__ __forceinline__ bool off_series(const CellYieldIn& c, const YieldGroup& gr) {
    const float x1 = __fmul_rn(gr.m_hi, c.b_hi);
    const float xn = __fmul_rn(gr.light && c.warm ? 10.0f : 1.0f, x1);
    return !(x1 >= 0.5f && xn <= 399.95f) && !(x1 > 701.0f);
}

// The yields that yields_kernel left out, where it left out any: the series
// with an argument off the tables, evaluated directly, by blocks of a warp in
// turns of 32 cells and every kOffRows-th group.  32 hot cells cost a thousand
// times what others do and the FP64 pipe of their SM bounds them, so what counts
// is that the dear turns (those of the first rows: the groups come in decreasing
// order of work) are spread over the SMs: the first turn goes by the place of the
// block, the next ones to the warps that come free.  (A grid over the cells, whose
// blocks take one turn or two, waits for those with two; first turns by arrival
// leave SMs without; 4, 5, 6 and 8 blocks per SM: 20,000 cells at 0.3 GeV 6.0, 5.0,
// 5.0 and 5.8 ms, with diffusion 4.5, 2.9, 3.2 and 4.2.)
// Calls of one event, ms, with the evaluation inlined in the yields kernel, in a
// grid of 304 blocks over the cells and so: 1,000 cells at 0.3 GeV 2.24, 2.17, 1.97;
// 20,000 5.88, 7.77, 5.03; 50,000 11.55, 15.59, 11.07; 100,000, one in 40 of them hot
// 19.2, 18.4, 15.6; 20,000 with diffusion 4.41, 4.43, 2.87; 50,000 at 5 MeV 1.46, 2.13,
// 1.26; 20,000 at 0.5 MeV, where all is zero, 0.28, 0.37, 0.15.
constexpr int kOffRows = 16;
constexpr int kOffBlocks = 5;   // per SM

template <int kBulk, bool kDiff>
__global__ void __launch_bounds__(32)
yields_off_table_kernel(DevConfig cfg, CellArrays cells, float* __restrict__ yields, uint32_t* __restrict__ ymax,
                        uint32_t* __restrict__ off_table) {
    if (*off_table == 0u) return;
    extern __shared__ float4 s_dyn[];
    constexpr unsigned FULL = 0xffffffffu;
    const int nsp = cfg.n_species;
    const int G = cfg.n_ygroups;
    const int words4 = yield_list_float4(nsp, G, cfg.n_yruns);
    for (int k = threadIdx.x; k < words4; k += 32) s_dyn[k] = cfg.ylist[k];
    __syncwarp();
    const YieldGroup* groups = reinterpret_cast<const YieldGroup*>(s_dyn);
    const float4* list = s_dyn + G + cfg.n_yruns;
    const int32_t* gst = reinterpret_cast<const int32_t*>(list + nsp);
    const int32_t* rst = gst + G + 1;
    const int32_t* mem = rst + cfg.n_yruns + 1;
    const int64_t n = cfg.n_cells;
    const int lane = threadIdx.x;
    // the first turns by the place of the block, which spreads the dear ones over
    // the SMs, the others as warps come free
    const int64_t chunks = (n + 31) / 32;
    for (int64_t turn = blockIdx.x; turn < chunks * kOffRows;
         turn = gridDim.x + static_cast<int64_t>(__shfl_sync(FULL, lane == 0 ? atomicAdd(off_table + 1, 1u) : 0u, 0))) {
        const int row = static_cast<int>(turn / chunks);
        const int64_t l0 = (turn - row * chunks) * 32;
        const int64_t l = min(l0 + lane, n - 1);
        const float4 da = cells.da[l];
        const bool live = l0 + lane < n && !(da.x < 0.0f);
        const CellYieldIn c = cell_yield_in<kBulk, kDiff>(cfg, cells, l, da);
        const int64_t row0 = static_cast<int64_t>(surface_of(cfg.surf, cfg.n_surfaces, l)) * nsp;
        for (int g = row; g < G; g += kOffRows) {
            const YieldGroup gr = groups[g];
            if (!(live && off_series(c, gr))) continue;
            float2 xy = make_float2(0.0f, 0.0f);
            float mu_of = __int_as_float(0x7fc00000);
            bool off = false;
            for (int t = rst[gst[g]]; t < rst[gst[g + 1]]; t++) {
                const float4 q = list[t];
                const float mu = q.x * c.th.y + q.y * c.th.z + q.z * c.th.w;
                if (mu != mu_of) {
                    off = false;
                    xy = yield_coefs<kBulk, kDiff>(c, gr, thermal_series<kBulk, kDiff, false>(cfg, c, gr, mu, off));
                    mu_of = mu;
                }
                if (!off) continue;
                const float yv = member_yield(q, xy);
                yields[static_cast<int64_t>(mem[t]) * n + l] = yv;
                if (yv > 0.0f) atomicMax(ymax + row0 + mem[t], __float_as_uint(yv));
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------
// per-species fixed-point prefix sums over cells (cdf_quantize): tile sums,
// tile offsets and totals, tile scan with the guide-table scatter

constexpr int kScanThreads = 256;
constexpr int kScanPer = 8;
constexpr int kScanTile = kScanThreads * kScanPer;
static_assert(kScanTile == kCdfTile && kCdfSub % kScanPer == 0, "runs are whole threads of the scan");
// tiles per block of the scan, whose blocks leave at once where the row is
// sparse: 4 (31,262 tiles, all rows but a few sparse: 18 us), 1 where the
// blocks fit the chip in a wave or two anyway (319 tiles: 8 us, 16 us with 4)
constexpr int kScanTilesPerBlock = 4;
constexpr int64_t kScanFewTiles = 4096;

__device__ __forceinline__ unsigned long long warp_incl_scan_u64(unsigned long long v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// exclusive block scan of one value per thread; returns the block total
__device__ unsigned long long block_excl_scan_u64(unsigned long long v, unsigned long long* s_warp,
                                                  unsigned long long* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned long long inc = warp_incl_scan_u64(v);
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        const unsigned long long w = lane < nw ? s_warp[lane] : 0ull;
        const unsigned long long wi = warp_incl_scan_u64(w);
        if (lane < nw) s_warp[lane] = wi - w;
        if (lane == nw - 1) s_warp[32] = wi;
    }
    __syncthreads();
    const unsigned long long out = s_warp[wid] + inc - v;
    *total = s_warp[32];
    __syncthreads();
    return out;
}

// Scan tiles are numbered over all rows (b, k) of the batch: surface b owns
// tiles [tile_base, tile_base + S nt) -- species k's row is its k-th run of
// nt tiles.  A block finds its surface by binary search over tile_base.
struct TileRef {
    const SurfSeg* sg;
    int b, k;
    int64_t tile;             // tile index inside the row
};

__device__ __forceinline__ TileRef tile_ref(const SurfSeg* __restrict__ surf, int n_surf, int S,
                                            int64_t t) {
    int lo = 0, hi = n_surf - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (surf[mid].tile_base <= t) lo = mid; else hi = mid - 1;
    }
    TileRef r;
    r.sg = surf + lo;
    r.b = lo;
    const int64_t local = t - r.sg->tile_base;   // below 2^31: a tile is a block of a grid
    r.k = static_cast<int>(static_cast<uint32_t>(local) / static_cast<uint32_t>(r.sg->nt));
    r.tile = local - static_cast<int64_t>(r.k) * r.sg->nt;
    if (r.k >= S) r.k = S - 1;   // not reached: the grid has exactly the batch's tiles
    return r;
}

// The yields of a tile, read coalesced, to a thread's kScanPer consecutive
// cells (padded: element e of the tile sits at (e / 8) * 9 + e % 8)
__device__ __forceinline__ void load_tile(const uint32_t* __restrict__ row, int64_t t0, int64_t n,
                                          uint32_t* s_in) {
    uint32_t v[kScanPer];
#pragma unroll
    for (int k = 0; k < kScanPer; k++) {
        const int64_t i = t0 + k * kScanThreads + threadIdx.x;
        v[k] = i < n ? __ldg(row + i) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kScanPer; k++) {
        const int e = k * kScanThreads + threadIdx.x;
        s_in[(e / kScanPer) * (kScanPer + 1) + e % kScanPer] = v[k];
    }
}

constexpr int kSumThreads = 128;
constexpr int kSumRuns = kCdfTile / kSumThreads;   // runs of a warp

// Sums over the warp of the quantised yields of kSumRuns runs (32 cells each,
// one per lane): the sum of run `lane`, of the last run in the lanes past it.
// q = floor(y 2^s) (cdf_quantize) with s = 188 - L - exponent(ymax), in limbs of
// 23 bits: y times 2^s less the low limbs is exact (what a denormal loses is
// below 1); adding 2^23 rounded down leaves the floor in the mantissa, and the
// rest goes on to the next limb.  q < 2^(62 - L), so two limbs hold it from
// L = 16 on and three always.  The float bits are summed as they are, modulo
// 2^32: 32 limbs add up below 2^28, 32 exponents of 2^23 to kExp.
template <int kLimbs>
__device__ __forceinline__ unsigned long long warp_runs(float* y, int s) {
    constexpr float kTwo23 = 8388608.0f;
    constexpr uint32_t kExp = 0x60000000u;   // 32 * 0x4B000000
    int e = s - 23 * (kLimbs - 1);
    if (e < -126 || e > 127) {
        const int e1 = e / 2;
        const float f1 = __uint_as_float(static_cast<uint32_t>(127 + e1) << 23);
#pragma unroll
        for (int k = 0; k < kSumRuns; k++) y[k] *= f1;
        e -= e1;
    }
    const float f = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
    const int lane = threadIdx.x & 31;
    uint32_t mine[kLimbs];
#pragma unroll
    for (int k = 0; k < kSumRuns; k++) {
        const float t = y[k] * f;
        float a = __fadd_rz(t, kTwo23), r = t - (a - kTwo23);
#pragma unroll
        for (int j = kLimbs - 1; j >= 0; j--) {
            const uint32_t sum = __reduce_add_sync(0xffffffffu, __float_as_uint(a));
            mine[j] = lane >= k ? sum : mine[j];
            if (j == 0) break;
            a = __fmaf_rz(r, kTwo23, kTwo23);
            if (j > 1) r = fmaf(r, kTwo23, kTwo23 - a);
        }
    }
    unsigned long long q = mine[kLimbs - 1] - kExp;
#pragma unroll
    for (int j = kLimbs - 2; j >= 0; j--) q = (q << 23) + (mine[j] - kExp);
    return q;
}

// Sum of every tile, and inside it the prefix sums of its runs of kCdfSub
// cells, which are what the cell draws of sparse rows search.  A warp reads
// kSumRuns runs, a cell per lane, and only the first warp goes on to the prefix
// sums of the tile.  Bound by memory (64 M yields of 200,000 cells: 255 MB, 48 us)
// once the integer work is out of the way: quantising each yield by shifts of
// 64 bits and scanning them in shared memory, eight cells per thread, took 91 us;
// warps of eight runs instead of sixteen, which repeat the tile's look-up twice
// as often, 55 us.  16 surfaces of 225,000 cells together: 126 -> 71 us.
__global__ void __launch_bounds__(kSumThreads)
cdf_tile_sum_kernel(const float* __restrict__ yields, int64_t N, const SurfSeg* __restrict__ surf,
                    int n_surf, int S, const uint32_t* __restrict__ ymax,
                    unsigned long long* __restrict__ tile_sum, unsigned long long* __restrict__ sub) {
    static_assert(kCdfSub == 32 && kCdfSubs == 64 && kSumRuns * kSumThreads == kCdfTile, "a run per warp load");
    __shared__ __align__(16) unsigned long long s_run[kCdfSubs];
    const TileRef tr = tile_ref(surf, n_surf, S, blockIdx.x);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t i0 = tr.tile * kScanTile + wid * (kSumRuns * 32) + lane;
    const int64_t left = tr.sg->n - i0;
    const float* row = yields + static_cast<int64_t>(tr.k) * N + tr.sg->c0 + i0;
    float y[kSumRuns];
    if (left > (kSumRuns - 1) * 32) {
#pragma unroll
        for (int k = 0; k < kSumRuns; k++) y[k] = __ldg(row + k * 32);
    } else {
#pragma unroll
        for (int k = 0; k < kSumRuns; k++) y[k] = k * 32 < left ? __ldg(row + k * 32) : 0.0f;
    }
    const int L = tr.sg->L;
    const int s = 150 + cdf_quant_base(ymax[tr.b * S + tr.k], L);
    const unsigned long long q = L >= 16 ? warp_runs<2>(y, s) : warp_runs<3>(y, s);
    if (lane < kSumRuns) s_run[wid * kSumRuns + lane] = q;
    __syncthreads();
    if (wid != 0) return;
    const unsigned long long a = s_run[2 * lane], b = s_run[2 * lane + 1];
    const unsigned long long inc = warp_incl_scan_u64(a + b);
    ulonglong2 out;
    out.x = inc - (a + b);
    out.y = out.x + a;
    reinterpret_cast<ulonglong2*>(sub + static_cast<int64_t>(blockIdx.x) * kCdfSubs)[lane] = out;
    if (lane == 31) tile_sum[blockIdx.x] = inc;
}

// one block per row (b, k): exclusive scan of the row's tile sums, the row
// total Q, the FP64 yield Q 2^-E, whether the row is sparse, C[n] = Q and the
// guide sentinel
__global__ void __launch_bounds__(kScanThreads)
cdf_tile_offset_kernel(const SurfSeg* __restrict__ surf, int S,
                       const unsigned long long* __restrict__ tile_sum,
                       const uint32_t* __restrict__ ymax, double ymult, bool allow_sparse,
                       unsigned long long* __restrict__ tile_off,
                       unsigned long long* __restrict__ qtot, int32_t* __restrict__ sparse,
                       double* __restrict__ totals, unsigned long long* __restrict__ cdf,
                       int32_t* __restrict__ guide) {
    __shared__ unsigned long long s_warp[33];
    const int r = blockIdx.x;
    const int b = r / S, k = r - b * S;
    const SurfSeg sg = surf[b];
    const int64_t first = sg.tile_base + static_cast<int64_t>(k) * sg.nt;
    unsigned long long carry = 0;
    for (int i0 = 0; i0 < sg.nt; i0 += kScanThreads) {
        const int i = i0 + threadIdx.x;
        const unsigned long long v = i < sg.nt ? tile_sum[first + i] : 0ull;
        unsigned long long tot;
        const unsigned long long ex = block_excl_scan_u64(v, s_warp, &tot);
        if (i < sg.nt) tile_off[first + i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) {
        const int base = cdf_quant_base(ymax[r], sg.L);
        qtot[r] = carry;
        const double total = carry ? ldexp(static_cast<double>(carry), -(150 + base)) : 0.0;
        totals[r] = total;
        // a row whose CDF would be written for few draws is left unwritten
        sparse[r] = allow_sparse && total * ymult * sg.ne * kSparseDraws < static_cast<double>(sg.n);
        cdf[sg.cdf_base + static_cast<int64_t>(k) * (sg.n + 1) + sg.n] = carry;
        const int64_t G = int64_t(1) << sg.g;
        guide[sg.guide_base + static_cast<int64_t>(k) * (G + 1) + G] = static_cast<int32_t>(sg.n - 1);
    }
}

// f(j) = floor(j * Q / 2^g): the smallest v of guide bucket j (r >> (64 - g) == j)
__device__ __forceinline__ unsigned long long bucket_start(unsigned long long j, int g,
                                                           unsigned long long Q) {
    return __umul64hi(j << (64 - g), Q);
}

// Writes tile tile_id of the dense row (b, k) of the cell CDF, C[i] = sum of q over cells < i, and
// scatters the guide table (indexed search, Chen & Asau 1974): guide[j] is
// the cell whose interval [C[i], C[i+1]) holds f(j).  The intervals partition
// [0, Q), so every bucket j < 2^g gets exactly one writer; the cell of any v
// drawn in bucket j lies in [guide[j], guide[j+1]].
__device__ __forceinline__ void scan_tile(
    const float* __restrict__ yields, int64_t N, const SurfSeg* __restrict__ surf, int n_surf, int S,
    const uint32_t* __restrict__ ymax, int64_t tile_id, const unsigned long long* __restrict__ tile_off,
    const unsigned long long* __restrict__ qtot, const int32_t* __restrict__ sparse,
    unsigned long long* __restrict__ cdf, int32_t* __restrict__ guide, uint32_t* s_in, unsigned long long* s_c,
    unsigned long long* s_warp) {
    const TileRef tr = tile_ref(surf, n_surf, S, tile_id);
    const int64_t n = tr.sg->n;
    const int r = tr.b * S + tr.k;
    if (sparse[r]) return;   // the whole block: one row per tile
    const int64_t t0 = tr.tile * kScanTile;
    const uint32_t* row =
        reinterpret_cast<const uint32_t*>(yields + static_cast<int64_t>(tr.k) * N + tr.sg->c0);
    unsigned long long* out = cdf + tr.sg->cdf_base + static_cast<int64_t>(tr.k) * (n + 1);
    const int g = tr.sg->g;
    const int64_t G = int64_t(1) << g;
    int32_t* gd = guide + tr.sg->guide_base + static_cast<int64_t>(tr.k) * (G + 1);
    const int base = cdf_quant_base(ymax[r], tr.sg->L);
    const unsigned long long Q = qtot[r];
    __syncthreads();   // the buffers are free of the block's tile before
    load_tile(row, t0, n, s_in);
    __syncthreads();
    const uint32_t* mine = s_in + threadIdx.x * (kScanPer + 1);
    unsigned long long* mine_c = s_c + threadIdx.x * (kScanPer + 1);
    unsigned long long acc = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; k++) {
        const unsigned long long q = cdf_quantize(mine[k], base);
        mine_c[k] = q;
        acc += q;
    }
    unsigned long long tot;
    const unsigned long long ex = block_excl_scan_u64(acc, s_warp, &tot);
    const unsigned long long start = tile_off[tile_id] + ex;
    const int64_t e0 = t0 + static_cast<int64_t>(threadIdx.x) * kScanPer;
    // q -> exclusive prefix C, in place
    unsigned long long run = start;
#pragma unroll
    for (int k = 0; k < kScanPer; k++) {
        const unsigned long long q = mine_c[k];
        mine_c[k] = run;
        run += q;
    }
    __syncthreads();
    // coalesced store of C[t0 .. t0 + tile)
    for (int k = 0; k < kScanPer; k++) {
        const int e = k * kScanThreads + threadIdx.x;
        const int64_t i = t0 + e;
        if (i < n) out[i] = s_c[(e / kScanPer) * (kScanPer + 1) + e % kScanPer];
    }
    if (Q == 0 || e0 >= n || run == start) return;
    // Guide scatter.  Bucket j starts at f(j) = floor(j Q / G) = j qd + floor(j qr / G)
    // with Q = qd G + qr; f is stepped exactly: f(j+1) = f(j) + qd + carry.
    // First bucket at or after this thread's first cell: a float estimate of
    // ceil(start G / Q), then exact steps.
    // (the top 24 significant bits of Q and start, converted exactly from
    // 32-bit integers: within a bucket of the answer for g <= 22)
    const int qsh = max(0, 40 - __clzll(static_cast<long long>(Q)));
    int64_t j = static_cast<int64_t>(
        static_cast<float>(static_cast<uint32_t>(start >> qsh)) *
        __fdividef(static_cast<float>(G), static_cast<float>(static_cast<uint32_t>(Q >> qsh))));
    j = j < 0 ? 0 : (j > G ? G : j);
    while (j > 0 && bucket_start(static_cast<unsigned long long>(j - 1), g, Q) >= start) --j;
    while (j < G && bucket_start(static_cast<unsigned long long>(j), g, Q) < start) ++j;
    const unsigned long long qd = Q >> g, qr = Q & static_cast<unsigned long long>(G - 1);
    unsigned long long rem = (static_cast<unsigned long long>(j) * qr) & static_cast<unsigned long long>(G - 1);
    unsigned long long f = j < G ? bucket_start(static_cast<unsigned long long>(j), g, Q) : Q;
#pragma unroll
    for (int k = 0; k < kScanPer; k++) {
        const unsigned long long hi = (k + 1 < kScanPer) ? mine_c[k + 1] : run;
        while (j < G && f < hi) {
            gd[j] = static_cast<int32_t>(e0 + k);
            ++j;
            rem += qr;
            f += qd + (rem >> g);
            rem &= static_cast<unsigned long long>(G - 1);
        }
    }
}

__global__ void __launch_bounds__(kScanThreads, 6)
cdf_tile_scan_kernel(const float* __restrict__ yields, int64_t N, const SurfSeg* __restrict__ surf,
                     int n_surf, int S, const uint32_t* __restrict__ ymax, int64_t n_tiles,
                     int tiles_per_block,
                     const unsigned long long* __restrict__ tile_off,
                     const unsigned long long* __restrict__ qtot, const int32_t* __restrict__ sparse,
                     unsigned long long* __restrict__ cdf, int32_t* __restrict__ guide) {
    // s_in holds the FP32 yield bits (load_tile), s_c the CDF values on the
    // way out, in the same padded places
    __shared__ uint32_t s_in[kScanThreads * (kScanPer + 1)];
    __shared__ unsigned long long s_c[kScanThreads * (kScanPer + 1)];
    __shared__ unsigned long long s_warp[33];
    const int64_t first_tile = static_cast<int64_t>(blockIdx.x) * tiles_per_block;
    const int64_t last_tile = min(first_tile + tiles_per_block, n_tiles);
    for (int64_t tile = first_tile; tile < last_tile; tile++)
        scan_tile(yields, N, surf, n_surf, S, ymax, tile, tile_off, qtot, sparse, cdf, guide, s_in, s_c, s_warp);
}

}  // namespace

// ------------------------------------------------------------------------
// launch wrappers

cudaError_t launch_yields(const DevConfig& cfg, const CellArrays& cells, float* yields, uint32_t* ymax,
                          int num_sms, cudaStream_t stream) {
    // ymax and, behind it, the flag of arguments off the tables and the turns of
    // the kernel that evaluates them
    const size_t rows = static_cast<size_t>(cfg.n_surfaces) * cfg.n_species;
    uint32_t* off_table = ymax + rows;
    cudaError_t e0 = cudaMemsetAsync(ymax, 0, sizeof(uint32_t) * (rows + kYieldFlags), stream);
    if (e0 != cudaSuccess) return e0;
    if (cfg.n_cells <= 0) return cudaSuccess;
    // two cells per thread once a row of blocks is more than the groups can
    // spread over the chip (3,000 cells: 22 us, 24 with one; 1,245 cells: 22 and 18)
    const int per_thread = !cfg.include_diff && cfg.n_cells >= kTwoCellsFrom ? 2 : 1;
    const int64_t block_cells = kYieldThreads * per_thread;
    const unsigned blocks = static_cast<unsigned>((cfg.n_cells + block_cells - 1) / block_cells);
    const size_t smem = sizeof(float4) * static_cast<size_t>(yield_list_float4(cfg.n_species, cfg.n_ygroups,
                                                                               cfg.n_yruns)) +
                        sizeof(uint32_t) * static_cast<size_t>(cfg.n_species + cfg.n_yruns);
    const int bulk = !cfg.include_bulk ? kNoBulk
                     : (cfg.bulk_kind == 1 || cfg.bulk_kind == 21) ? kBulkCe
                     : cfg.bulk_kind == 11 ? kBulk14 : kNoBulk;
    using Kernel = void (*)(DevConfig, CellArrays, float*, uint32_t*, uint32_t*);
    const Kernel kernels[3][3] = {
        {yields_kernel<kNoBulk, false, 1>, yields_kernel<kNoBulk, false, 2>, yields_kernel<kNoBulk, true, 1>},
        {yields_kernel<kBulkCe, false, 1>, yields_kernel<kBulkCe, false, 2>, yields_kernel<kBulkCe, true, 1>},
        {yields_kernel<kBulk14, false, 1>, yields_kernel<kBulk14, false, 2>, yields_kernel<kBulk14, true, 1>}};
    using OffKernel = void (*)(DevConfig, CellArrays, float*, uint32_t*, uint32_t*);
    const OffKernel off_kernels[3][2] = {
        {yields_off_table_kernel<kNoBulk, false>, yields_off_table_kernel<kNoBulk, true>},
        {yields_off_table_kernel<kBulkCe, false>, yields_off_table_kernel<kBulkCe, true>},
        {yields_off_table_kernel<kBulk14, false>, yields_off_table_kernel<kBulk14, true>}};
    const Kernel kernel = kernels[bulk][cfg.include_diff ? 2 : per_thread - 1];
    const OffKernel off_kernel = off_kernels[bulk][cfg.include_diff ? 1 : 0];
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(smem));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(off_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    // rows of species groups: as tuned (per 128 cells), more where that leaves
    // fewer than three waves of blocks (16 per SM of two cells per thread, 21 of
    // one): a call of 1.1 waves runs two, and more waves repeat the cells' set-up
    // too often (45,000 cells in 12, 16, 26 and 40 blocks per SM: 63, 59, 61 and
    // 63 us; 12,000 cells 30, 30, 36 and 38 us).
    int want = per_thread * (cfg.yield_groups > 0 ? cfg.yield_groups : kYieldGroups);
    want = std::max(want, static_cast<int>((static_cast<int64_t>(num_sms) * (per_thread == 2 ? 16 : 21) + blocks - 1) / blocks));
    const unsigned groups = static_cast<unsigned>(std::max(1, std::min(want, cfg.n_ygroups)));
    kernel<<<dim3(blocks, groups), kYieldThreads, smem, stream>>>(cfg, cells, yields, ymax, off_table);
    const int64_t turns = (cfg.n_cells + 31) / 32 * kOffRows;
    const unsigned off_blocks = static_cast<unsigned>(std::min<int64_t>(turns, static_cast<int64_t>(num_sms) * kOffBlocks));
    off_kernel<<<off_blocks, 32, smem, stream>>>(cfg, cells, yields, ymax, off_table);
    return cudaGetLastError();
}

int cdf_num_tiles(int64_t n) { return static_cast<int>((n + kScanTile - 1) / kScanTile); }

cudaError_t launch_cdf_head(const float* yields, int64_t N, const SurfSeg* surf, int n_surf,
                            int64_t n_tiles, int S, const uint32_t* ymax, double ymult, bool allow_sparse,
                            const CdfBuffers& b, cudaStream_t stream) {
    if (n_tiles <= 0 || S <= 0 || n_surf <= 0) return cudaSuccess;
    const int rows = n_surf * S;
    const unsigned grid = static_cast<unsigned>(n_tiles);
    cdf_tile_sum_kernel<<<grid, kSumThreads, 0, stream>>>(yields, N, surf, n_surf, S, ymax, b.tile_sum, b.sub);
    cdf_tile_offset_kernel<<<rows, kScanThreads, 0, stream>>>(
        surf, S, b.tile_sum, ymax, ymult, allow_sparse && n_tiles >= kSparseTiles, b.tile_off, b.qtot, b.sparse,
        b.totals, b.cdf, b.guide);
    return cudaGetLastError();
}

cudaError_t launch_cdf_scan(const float* yields, int64_t N, const SurfSeg* surf, int n_surf,
                            int64_t n_tiles, int S, const uint32_t* ymax, const CdfBuffers& b,
                            cudaStream_t stream) {
    if (n_tiles <= 0 || S <= 0 || n_surf <= 0) return cudaSuccess;
    const int per_block = n_tiles > kScanFewTiles ? kScanTilesPerBlock : 1;
    const unsigned grid = static_cast<unsigned>((n_tiles + per_block - 1) / per_block);
    cdf_tile_scan_kernel<<<grid, kScanThreads, 0, stream>>>(yields, N, surf, n_surf, S, ymax, n_tiles, per_block,
                                                           b.tile_off, b.qtot, b.sparse, b.cdf, b.guide);
    return cudaGetLastError();
}

}  // namespace iss
