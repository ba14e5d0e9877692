// kernels_fp64.cu -- FP64 plain form of Wflow's SBM + kinematic-wave step (the drop-in).
//
// Compiled with --fmad=false: every multiply and add rounds separately, as in the reference's
// scalar Julia Float64 code. All elementary functions come from wf_math.cuh.
//
// Kernels of one model step (update_model!, Wflow/src/sbm_model.jl:60-92):
//   vertical  : storage_prev! of the land balance, interception, snow, open-water runoff,
//               soil fraction, soil boundary conditions, update_soil_water_flow!  (per cell)
//   ssf       : lateral subsurface kinematic wave (wavefront), fused with
//               update_soil_water_storage! and the overland lateral inflow      (per chain)
//   overland  : overland kinematic wave with fixed sub-steps (wavefront)
//   river     : river lateral inflow + river kinematic wave (wavefront)
//   balance   : update_total_water_storage! and compute_mass_balance!           (per cell)
#include <cuda_runtime.h>

#include "wf_fields.cuh"
#include "wf_li_couple.cuh"
#include "wf_kernels.h"
#include "wf_launch.cuh"
#include "wf_math.cuh"
#include "wf_reservoir.cuh"
#include "snow_scheme.cuh"
#include "wf_ff.cuh"
#include "wf_walker.cuh"
#include "wf_wave64.cuh"

using wfm::div_;
using wfm::div_by_;
using wfm::gt0_;
using wfm::gt_;
using wfm::jclamp;
using wfm::jmax;
using wfm::jmin;
using wfm::le0_;
using wfm::lt_;

namespace {

constexpr double KIN_WAVE_MIN_FLOW = 1e-30;                       // routing/utils.jl:1
constexpr double MM_PER_DAY = (1.0 / 86400.0) * 1e-3;             // units.jl MM_PER_DAY factor
constexpr double NANV = __builtin_nan("");

// ------------------------------------------------------------------ process functions ----
// Divisors that a cell divides by several times (the step, the porosity, a layer's saturated
// depth) come with their reciprocal (rdt, r...): such a quotient costs 3 FP64 instructions
// (wf_math.cuh div_by_), and each FP64 instruction of a warp 64 cycles.

// vegetation/rainfall_interception.jl:9-70
__device__ void interception_gash(double cmax, double e_r, double gap, double P, double max_evap, double dt,
                                  double rdt, double& tf, double& ic, double& sf) {
    if (gt0_(cmax)) {
        double fs, fi, psat;
        if (lt_(gap, 1.0 / 1.1)) {
            fs = 0.1 * gap;
            fi = 1.0 - 1.1 * gap;
            psat = gt_(e_r, fi) ? 0.0 : div_(-cmax, e_r * dt) * wfm::log(1.0 - div_(e_r, fi));
        } else {
            fs = 1.0 - gap;
            fi = 0.0;
            psat = 0.0;
        }
        if (gt_(P, psat)) {
            const double cmax_dt = div_by_(cmax, dt, rdt);
            ic = (fi * psat - cmax_dt) + e_r * (P - psat) + cmax_dt;
        } else {
            ic = fi * P;
        }
        sf = fs * P;
        tf = P - ic - sf;
        if (gt_(ic, max_evap)) {
            const double drain = ic - max_evap;
            ic = max_evap;
            tf += drain;
        }
    } else {
        tf = P;
        ic = 0.0;
        sf = 0.0;
    }
}

// vegetation/rainfall_interception.jl:78-130
__device__ void interception_modrut(double P, double pet, double& cs, double gap, double cmax, double dt,
                                    double rdt, double& tf, double& ce, double& sf) {
    double fs, pc;
    if (lt_(gap, 1.0 / 1.1)) {
        fs = 0.1 * gap;
        pc = (1.0 - gap - fs) * P;
    } else {
        fs = 1.0 - gap;
        pc = 0.0;
    }
    sf = fs * P;
    tf = gap * P;
    if (gt_(cs, cmax)) {
        const double d = cs - cmax;
        cs = cmax;
        tf += div_by_(d, dt, rdt);
    }
    cs += pc * dt;
    const double max_evap = div_by_(cs, dt, rdt);
    if (gt_(pet, max_evap)) {
        ce = max_evap;
        cs = 0.0;
    } else {
        ce = pet;
        cs -= ce * dt;
    }
    if (gt_(cs, cmax)) {
        const double d = cs - cmax;
        cs = cmax;
        tf += div_by_(d, dt, rdt);
    }
}

// utils.jl:27-30
__device__ __forceinline__ double scurve(double x, double a, double b, double c) {
    return div_(1.0, b + wfm::exp(-c * (x - a)));
}

// utils.jl:1070-1076 with Wflow's pow
__device__ __forceinline__ double bounded_power(double base, double p) { return gt_(base, 1.0) ? 1.0 : wfm::pow(base, p); }

// soil/soil_process.jl:51-92. The iteration is the longest serial chain of the column (a daily step
// takes hundreds): its quotients by l_sat and dt use the reciprocals, and `st < usd / dt` is decided
// from st dt, which the update needs anyway, unless the two are within 16 ulps. 55 FP64
// instructions per iteration (119 with plain divisions, comparisons and the generic exp and log).
__device__ void unsatzone_flow_layer(double usd, double kv_z, double l_sat, double c, double dt, double rdt,
                                     double& usd_out, double& flow) {
    if (le0_(usd)) {
        usd_out = 0.0;
        flow = 0.0;
        return;
    }
    const double r_sat = div_(1.0, l_sat);
    const double st_sat = jmax(0.0, usd - l_sat);
    double st = kv_z * bounded_power(div_by_(usd, l_sat, r_sat), c);
    double sum_ast = jmin(st, div_by_(st_sat, dt, rdt));
    usd -= sum_ast * dt;
    const double remainder = jmin((st - sum_ast) * dt, usd);
    const long its = (long)wfm::cld(remainder, 2e-4);
    const double kv_it = its > 0 ? div_(kv_z, (double)its) : 0.0;
    for (long i = 0; i < its; ++i) {
        st = kv_it * bounded_power(div_by_(usd, l_sat, r_sat), c);
        const double taken = st * dt;
        bool below = gt0_(taken) && gt0_(usd) && wfm::to_bits(taken) + 16 < wfm::to_bits(usd);
        double st_max = 0.0;
        if (!below) {
            st_max = div_by_(usd, dt, rdt);
            below = lt_(st, st_max);
        }
        if (below) {
            usd -= taken;
            sum_ast += st;
        } else {
            usd = 0.0;
            sum_ast += st_max;
            break;
        }
    }
    usd_out = usd;
    flow = sum_ast;
}

// soil/soil_process.jl:113-130
__device__ __forceinline__ double head_brooks_corey(double vwc, double ts, double tr, double c, double psi) {
    const double lam = div_(2.0, c - 3.0);
    return gt0_(lam) ? div_(psi, wfm::pow(div_(vwc, ts - tr), div_(1.0, lam))) : psi;
}

// soil/soil_process.jl:166-176
__device__ __forceinline__ double feddes_h3(double h3h, double h3l, double tpot) {
    const double td = div_by_(tpot, MM_PER_DAY, 1.0 / MM_PER_DAY);
    if (wfm::le_(td, 1.0)) return h3l;
    if (lt_(td, 5.0)) return h3l + (h3h - h3l) * (td - 1.0) / (5.0 - 1.0);
    return h3h;
}

// soil/soil_process.jl:183-200
__device__ __forceinline__ double rwu_feddes(double h, double h1, double h2, double h3, double h4, double a1) {
    if (lt_(h, h4)) return 0.0;
    if (lt_(h, h3)) return div_(h - h4, h3 - h4);
    if (wfm::is_zero_(a1)) {
        if (lt_(h, h2)) return 1.0;
        if (lt_(h, h1)) return div_(h1 - h, h1 - h2);
        return 0.0;
    }
    return 1.0;
}

// rwu_feddes of a layer's Brooks-Corey head. The reduction is 0 below h4 and, for a1 != 0, 1 from h3
// up: an FP32 head decides those cases when it is more than 0.1 % away from both heads, and only the
// heads between them pay the power and three divisions (80 FP64 instructions). The porosity range is
// subtracted in FP64, so that the saturation x is within 4e-7 also where the two porosities are close. The
// head is then within 1e-4 over the range that the FP32 path takes: (c - 3) / 2 < 29 times the error of
// log2 x, below 3e-6, and half the error of c, 2e-6, times |log2 x| < 20.
__device__ __forceinline__ double rwu_layer(double vwc, double ts, double tr, double c, double psi, double h1, double h2,
                                            double h3, double h4, double a1) {
    const float x = wfm::f32_of(vwc) / wfm::f32_of(ts - tr);
    const float p32 = wfm::f32_of(psi), c32 = wfm::f32_of(c), lo = wfm::f32_of(h4), hi = wfm::f32_of(h3);
    // (f32_of gives an infinity for a NaN: the FP64 path takes those)
    if (c32 > 3.01f && c32 < 60.0f && p32 < 0.0f && p32 > -1e30f && lo < hi && hi < 0.0f && x > 1e-6f && x < 1e6f) {
        const float head = p32 * exp2f(-0.5f * (c32 - 3.0f) * log2f(x));
        if (head > hi * 0.999f && !wfm::is_zero_(a1)) return 1.0;
        if (head < lo * 1.001f) return 0.0;
    }
    return rwu_feddes(head_brooks_corey(vwc, ts, tr, c, psi), h1, h2, h3, h4, a1);
}

__device__ __forceinline__ double lb_drainable(double ts, double tfc) { return jmax(ts - tfc, 0.02); }

// ------------------------------------------------------------------ soil column ---------

template <int MAXN>
struct Column {
    int N, nl, nu;
    double act[MAXN], cum[MAXN + 1], thick[MAXN], usld[MAXN];
    double ts, tr, tfc, d, kv0, f, zexp;
    int profile;

    __device__ void load_static(const WfDevFields& F, int64_t slot) {
        N = F.N;
        nl = F.nlayers[slot];
        ts = F.L[THETA_S][slot];
        tr = F.L[THETA_R][slot];
        tfc = F.L[THETA_FC][slot];
        d = F.L[SOIL_THICKNESS][slot];
        zexp = F.L[Z_EXP][slot];
        profile = F.kv_profile;
        cum[0] = 0.0;
#pragma unroll
        for (int k = 0; k < MAXN; ++k) {
            act[k] = k < N ? F.LY[LY_ACT_THICK][k][slot] : NANV;
            cum[k + 1] = cum[k] + act[k];
        }
    }
    // utils.jl:390-409
    __device__ void set_thickness(double ref) {
        nu = N;
#pragma unroll
        for (int k = 0; k < MAXN; ++k) {
            if (k >= N) break;
            double t = NANV;
            if (gt_(ref, cum[k + 1])) {
                t = act[k];
            } else {
                const double above = ref - cum[k];
                if (gt0_(above)) t = above;
            }
            thick[k] = t;
            if (wfm::isnan_(t)) nu -= 1;
        }
    }
    // utils.jl:727-761 (n is 1-based)
    __device__ __forceinline__ double kv_at(const double* kvf, double z, int n) const {
        double zz = z;
        if (profile == WF_KV_EXPONENTIAL_CONSTANT && !lt_(z, zexp)) zz = zexp;
        return kvf[n - 1] * kv0 * wfm::exp(-f * zz);
    }
    // soil.jl:1213-1259
    __device__ void update_ustorelayerdepth(double zi_prev, double zi) {
        const int n_prev = nu;
        double tprev[MAXN];
#pragma unroll
        for (int k = 0; k < MAXN; ++k) tprev[k] = thick[k];
        set_thickness(zi);
        const int n_new = nu;
        if (lt_(zi, zi_prev)) {
#pragma unroll
            for (int k = 1; k <= MAXN; ++k) {
                if (k < n_new || k > n_prev) continue;
                if (wfm::isnan_(thick[k - 1])) {
                    usld[k - 1] = 0.0;
                } else {
                    const double sc = div_(thick[k - 1], tprev[k - 1]);
                    usld[k - 1] = sc * usld[k - 1];
                }
            }
        } else {
#pragma unroll
            for (int k = 1; k <= MAXN; ++k) {
                if (k < n_prev || k > n_new) continue;
                const double tp = wfm::isnan_(tprev[k - 1]) ? 0.0 : tprev[k - 1];
                const double delta = thick[k - 1] - tp;
                usld[k - 1] = usld[k - 1] + delta * (tfc - tr);
            }
        }
    }
    // utils.jl:1090-1131
    __device__ void water_table_change(double net_flux, double sy, double dt, double& dh, double& exfilt) const {
        const double te = ts - tr;
        if (le0_(net_flux)) {
            dh = div_(net_flux * dt, sy);
        } else {
            dh = 0.0;
#pragma unroll
            for (int k = MAXN; k >= 1; --k) {
                if (k > nu) continue;
                const double cap = div_(jmax(thick[k - 1] * te - usld[k - 1], 0.0), dt);
                const double fl = jmin(net_flux, cap);
                if (wfm::le_(cap, net_flux)) {
                    dh += thick[k - 1];
                } else {
                    const double syk = te - div_(usld[k - 1], thick[k - 1]);
                    dh += div_(fl * dt, syk);
                }
                net_flux -= fl;
                if (wfm::is_zero_(net_flux)) break;
            }
        }
        exfilt = jmax(net_flux, 0.0);
    }
};

// routing/subsurface/subsurface_process.jl:6-41
__device__ __forceinline__ double ssf_celerity(double zi, double slope, double sy, double kh0, double f, int profile,
                                               double zexp) {
    double z = zi;
    if (profile == WF_KV_EXPONENTIAL_CONSTANT) z = zi < zexp ? zi : zexp;
    return div_(kh0 * wfm::exp(-f * z) * slope, sy);
}

// routing/subsurface/subsurface_process.jl:57-78, with dt_dx = dt / dx, cinv = 1 / celerity, df their
// sum and rdf = 1 / df
__device__ __forceinline__ double kw_ssf_newton(double q, double cterm, double dt_dx, double cinv, double df, double rdf) {
    int count = 0;
    while (true) {
        const double fq = dt_dx * q + cinv * q - cterm;
        const double q_old = q;
        q -= div_by_(fq, df, rdf);
        if (wfm::isnan_(q)) q = 0.0;
        q = jmax(q, KIN_WAVE_MIN_FLOW);
        if (wfz::converged(fq) || (count >= 3000)) break;
        if (wfm::to_bits(q) == wfm::to_bits(q_old)) break;  // fixed point: the remaining iterations repeat this one
        count += 1;
    }
    return q;
}

// (a + b) / 2
__device__ __forceinline__ double mean2(double a, double b) {
    const double t = a + b;
    const unsigned hx = (unsigned)__double2hiint(t) & 0x7fffffffu;
    return hx - 0x00200000u < 0x7fd00000u ? wfm::from_bits(wfm::to_bits(t) - 0x0010000000000000ULL) : t / 2.0;
}

// Largest change of the water table of a sub-step that needs no sub-iterations: the reference takes
// ceil(round(|dz| / 0.1, 12 digits)) of them, one or none up to 0.1 m.
__device__ __forceinline__ bool one_iteration(double dz) { return lt_(wfm::fabs_(dz), 0.0999); }

// routing/subsurface/subsurface_process.jl:89-172
template <int MAXN>
__device__ void kinematic_wave_ssf(double q_in, double q_prev, double zi_prev, double q_net, double slope, double sy,
                                   double d, double dt, double dx, double dw, double q_max, double kh0,
                                   Column<MAXN>& col, double& q_out, double& zi_out, double& exfilt_out,
                                   double& netflux_out) {
    if (q_in + q_prev == 0.0 && q_net <= 0.0) {
        q_out = 0.0;
        zi_out = d;
        exfilt_out = 0.0;
        netflux_out = 0.0;
        return;
    }
    const double f = col.f;
    double cel = ssf_celerity(zi_prev, slope, sy, kh0, f, col.profile, col.zexp);
    double dt_dx = div_(dt, dx), cinv = div_(1.0, cel);
    double df = dt_dx + cinv;
    double cterm = dt_dx * (q_in + q_net) + div_by_(q_prev, cel, cinv);
    double q = kw_ssf_newton(mean2(q_prev, q_in), cterm, dt_dx, cinv, df, div_(1.0, df));
    q = jmin(q, (q_max * dw));
    double net_flux = div_(q_in + q_net - q, dw * dx);
    double dh, exfilt;
    col.water_table_change(net_flux, sy, dt, dh, exfilt);
    double zi = zi_prev - dh;
    if (gt_(zi, d)) {
        const double q_excess = div_((dw * dx) * sy * (zi - d), dt);
        q = jmax(q - q_excess, KIN_WAVE_MIN_FLOW);
    }
    zi = jclamp(zi, 0.0, d);
    const long its = one_iteration(zi - zi_prev)
                         ? 1
                         : (long)wfm::ceil_(wfm::round_sigdigits(wfm::fabs_(zi - zi_prev) / 0.1, 12));
    if (its > 1) {
        const double dt_s = dt / (double)its;
        double q_sum = 0.0, exfilt_sum = 0.0, net_flux_sum = 0.0;
        for (long i = 0; i < its; ++i) {
            cel = ssf_celerity(zi_prev, slope, sy, kh0, f, col.profile, col.zexp);
            dt_dx = div_(dt_s, dx);
            cinv = div_(1.0, cel);
            df = dt_dx + cinv;
            cterm = dt_dx * q_in + div_by_(q_prev, cel, cinv) + q_net * dt_dx;
            q = kw_ssf_newton(q_prev, cterm, dt_dx, cinv, df, div_(1.0, df));
            q = jmin(q, (q_max * dw));
            net_flux = div_(q_in + q_net - q, dw * dx);
            col.water_table_change(net_flux, sy, dt_s, dh, exfilt);
            zi = zi_prev - dh;
            if (gt_(zi, d)) {
                const double q_excess = div_((dw * dx) * sy * (zi - d), dt_s);
                q = jmax(q - q_excess, KIN_WAVE_MIN_FLOW);
            }
            zi = jclamp(zi, 0.0, d);
            col.update_ustorelayerdepth(zi_prev, zi);
            exfilt_sum += exfilt;
            net_flux_sum += net_flux;
            q_sum += q;
            q_prev = q;
            zi_prev = zi;
        }
        q = q_sum / (double)its;
        exfilt = exfilt_sum / (double)its;
        net_flux = net_flux_sum / (double)its;
    } else {
        col.update_ustorelayerdepth(zi_prev, zi);
    }
    q_out = q;
    zi_out = zi;
    exfilt_out = exfilt;
    netflux_out = net_flux;
}

// ----------------------------------------------------------------- vertical kernel ------

// glacier_store * glacier_fraction of a cell (compute_total_storage, mass_balance.jl:96-113); the
// reference's zero term without a glacier
__device__ __forceinline__ double glacier_storage(const WfDevFields& F, int64_t e, int64_t slot) {
    return F.glacier ? F.GM[GM_STORE][e] * F.G[G_FRAC][slot] : 0.0 * 0.0;
}

// update_glacier_model! (glacier.jl:122-154) of one cell: glacier_hbv (snow_scheme.cuh) on its
// snow storage and glacier store. Returns the melt rate.
__device__ __forceinline__ double glacier_update(const WfDevFields& F, int64_t e, int64_t slot, double T, double dt,
                                                 double& snow) {
    double store, melt;
    wfsn::glacier_hbv(F.G[G_FRAC][slot], F.GM[GM_STORE][e], snow, T, F.G[G_TTM][slot], F.G[G_DDF][slot],
                      F.G[G_SIFRAC][slot], F.g_max_rate, dt, &snow, &store, &melt);
    F.GM[GM_STORE][e] = store;
    F.GM[GM_MELT][e] = melt;
    return melt;
}

// Parts of the per-cell update. VERT_ALL: the whole update_land_hydrology_model! (sbm.jl:82-132).
// With gravitational snow transport the transport sweep runs between VERT_SNOW (interception and
// snow, sbm.jl:92-96, and the transport capacities) and VERT_SOIL (glacier, open-water runoff and
// soil, sbm.jl:102-131).
enum VertPhase { VERT_ALL = 0, VERT_SNOW = 1, VERT_SOIL = 2 };

template <int MAXN, int PHASE>
__global__ void __launch_bounds__(256) vertical_kernel(WfDevFields F) {
    const int M = F.M;
    const int64_t E = F.land_slots * M;
    const double dt = F.dt, rdt = div_(1.0, F.dt);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if (F.land_node_of_slot[slot] < 0) continue;
        const int m = (int)(e - slot * M);
        double* const* Mf = F.Mf;
        double* const* L = F.L;
        const double Pr = Mf[PRECIP][e], PET = Mf[POTEVAP][e], T = Mf[TEMP][e];
        double canopy = Mf[CANOPY][e];
        double snow = Mf[SNOW][e], snow_water = Mf[SNOW_WATER][e];
        const double gap = L[GAP][slot], cmax = L[CMAX][slot];
        const double potevap = L[KC][slot] * PET * (1.0 - gap);
        double tf = 0.0, ic, sf = 0.0, srunoff = 0.0;
        if (PHASE != VERT_SOIL) {
        // storage_prev! of the land balance (mass_balance.jl:95-125, Wflow.jl:315)
        if (F.mass_balance)
            Mf[BL_PREV][e] = Mf[TSWS][e] + canopy + (snow + snow_water) + glacier_storage(F, e, slot) + 0.0;
        // ---- interception (canopy.jl:213-226 Gash, :259-271 Rutter)
        if (F.gash) {
            interception_gash(cmax, L[E_R][slot], gap, Pr, potevap, dt, rdt, tf, ic, sf);
        } else {
            interception_modrut(Pr, potevap, canopy, gap, cmax, dt, rdt, tf, ic, sf);
        }
        // ---- snow (snow.jl:238-293, snow_process.jl:26-116)
        if (F.snow) {
            const double eff = tf + sf;
            const double tti = L[TTI][slot], tt = L[TT][slot];
            double rainfrac;
            if (wfm::is_zero_(tti)) {
                rainfrac = gt_(T, tt) ? 1.0 : 0.0;
            } else {
                rainfrac = jclamp(div_(T - (tt - tti * 0.5), tti), 0.0, 1.0);
            }
            const double snowfrac = 1.0 - rainfrac;
            const double sp = snowfrac * 1.0 * eff, lp = rainfrac * 1.0 * eff;
            const double ttm = L[TTM][slot], ddf = L[DDF][slot], whc = L[WHC][slot];
            double melt;
            if (gt_(T, ttm)) {
                melt = jmin(ddf * (T - ttm), div_by_(snow, dt, rdt));
                snow -= melt * dt;
                snow_water += melt * dt;
            } else {
                melt = 0.0;
                const double refr = jmin(ddf * 0.05 * (ttm - T) * dt, snow_water);
                snow += refr;
                snow_water -= refr;
            }
            snow = jmax(snow, 0.0);
            snow_water = jmax(snow_water, 0.0);
            snow += sp * dt;
            snow_water += lp * dt;
            const double maxsw = snow * whc;
            if (gt_(snow_water, maxsw)) {
                srunoff = div_by_(snow_water - maxsw, dt, rdt);
                snow_water = maxsw;
            } else {
                srunoff = 0.0;
            }
            Mf[SWE][e] = snow_water + snow;
        }
        if (PHASE == VERT_SNOW) {
            // lateral_snow_transport! capacities from the updated states (surface_process.jl:9-19)
            Mf[CANOPY][e] = canopy;
            Mf[SNOW][e] = snow;
            Mf[SNOW_WATER][e] = snow_water;
            F.GM[GM_SRUNOFF][e] = srunoff;
            F.GM[GM_IC][e] = ic;
            const double frac = jmin(0.5, div_(L[SLOPE][slot], 5.67)) * jmin(1.0, div_(snow, 10.0));
            F.GM[GM_CAP][e] = div_by_(frac * snow, dt, rdt);
            F.GM[GM_CAPW][e] = div_by_(snow_water * frac, dt, rdt);
            continue;
        }
        } else {
            // after the transport sweep: the moved snow states, the interception and snow runoff
            // of VERT_SNOW
            ic = F.GM[GM_IC][e];
            srunoff = F.GM[GM_SRUNOFF][e];
        }
        // ---- glacier (glacier.jl:122-154) and the water flux at the surface (runoff.jl:37-58)
        double wfs, gfrac = 0.0;
        if (F.snow) {
            if (F.glacier) {
                gfrac = F.G[G_FRAC][slot];
                const double gmelt = glacier_update(F, e, slot, T, dt, snow);
                wfs = srunoff + gmelt * gfrac;
            } else {
                wfs = srunoff + 0.0 * 0.0;
            }
        } else {
            wfs = tf + sf;
        }
        // ---- open water runoff (runoff.jl:61-111)
        const double rfrac = L[RIVER_FRACTION][slot], wfrac = L[WATER_FRACTION][slot];
        const double wd_land = Mf[OL_H][e];
        const int64_t rs = F.land_river_slot[slot];
        const double wd_river = rs >= 0 ? F.RM[RV_H][rs * M + m] : 0.0;
        const double runoff_river = jmin(1.0, rfrac) * wfs;
        const double runoff_land = jmin(1.0, wfrac) * wfs;
        const double ae_river = rfrac * jmin(div_by_(wd_river, dt, rdt), PET);
        const double ae_land = wfrac * jmin(div_by_(wd_land, dt, rdt), PET);
        // ---- soil (soil.jl:643-682, 1150-1211)
        const double soil_fraction = jmax(gap - wfrac - rfrac - gfrac, 0.0);
        const double pot_trans = jmax(0.0, potevap - ic);
        double pot_soilevap = soil_fraction * PET;
        pot_soilevap -= 0.0;
        const double wfs_soil = jmax(wfs + 0.0 - runoff_river - runoff_land + 0.0, 0.0);

        Column<MAXN> col;
        col.load_static(F, slot);
        col.kv0 = Mf[KV0][e];
        col.f = Mf[FSCALE][e];
        const double ts = col.ts, tr = col.tr;
        const double swc = L[SWC][slot];
        double sat = Mf[SAT][e];
#pragma unroll
        for (int k = 0; k < MAXN; ++k) col.usld[k] = k < col.N ? F.LY[LY_USLD][k][e] : 0.0;
        double kvf[MAXN], cexp[MAXN], rfr[MAXN];
#pragma unroll
        for (int k = 0; k < MAXN; ++k) {
            kvf[k] = k < col.N ? F.LY[LY_KVFRAC][k][slot] : 0.0;
            cexp[k] = k < col.N ? F.LY[LY_C][k][slot] : 0.0;
            rfr[k] = k < col.N ? F.LY[LY_ROOTFRAC][k][slot] : 0.0;
        }
        // update_diagnostic_vars! (soil.jl:1400-1436)
        double usd = 0.0;
#pragma unroll
        for (int k = 0; k < MAXN; ++k)
            if (k < col.nl) usd += col.usld[k];
        const double te = ts - tr, rte = div_(1.0, te);
        double zi = jmax(0.0, col.d - div_by_(sat, te, rte));
        double drain = (col.d - zi) * lb_drainable(ts, col.tfc);
        double ucap = swc - sat - usd;
        col.set_thickness(zi);
        // soil temperature and infiltration reduction (soil.jl:684-729)
        double tsoil = Mf[TSOIL][e];
        if (F.snow) tsoil = tsoil + L[W_SOIL][slot] * (T - tsoil);
        double fred = 1.0;
        if (F.snow && F.infilt_reduction) {
            const double cf = L[CF_SOIL][slot];
            fred = scurve(tsoil, 273.15, 1.0 / (1.0 - cf), 8.0) + cf;
        }
        // infiltration (soil_process.jl:16-41)
        const double cfrac = L[COMPACT_FRAC][slot];
        const double cap_soil = col.kv0 * kvf[0];
        const double cap_comp = L[CAP_COMP][slot];
        const double soilinf = wfs_soil * (1.0 - cfrac);
        const double pathinf = wfs_soil * cfrac;
        const double mis = jmin(cap_soil * fred, soilinf);
        const double mip = jmin(cap_comp * fred, pathinf);
        const double infiltration = jmin(mip + mis, jmax(0.0, div_by_(ucap, dt, rdt)));
        const double infex = (soilinf - mis) + (pathinf - mip);
        // unsaturated_zone_flow! (soil.jl:764-804)
        double transfer = 0.0;
        if (col.nu > 0) {
            double z = 0.0, flow = 0.0;
#pragma unroll
            for (int k = 0; k < MAXN; ++k) {
                if (k >= col.nu) break;
                z = z + col.thick[k];
                const double l_sat = col.thick[k] * (ts - tr);
                const double kv_z = col.kv_at(kvf, z, k + 1);
                const double u = k == 0 ? col.usld[k] + infiltration * dt : col.usld[k] + flow * dt;
                double uo;
                unsatzone_flow_layer(u, kv_z, l_sat, cexp[k], dt, rdt, uo, flow);
                col.usld[k] = uo;
            }
            transfer = flow;
        }
        // soil_evaporation! (soil.jl:814-856)
        double soilevap, esat;
        {
            double pot = pot_soilevap;
            double se;
            if (col.nu == 0) {
                se = 0.0;
            } else if (col.nu == 1) {
                se = pot * jmin(1.0, div_(col.usld[0], zi * (ts - tr)));
            } else {
                se = pot * jmin(1.0, div_(col.usld[0], col.thick[0] * (ts - tr)));
            }
            se = jmin(se, div_by_(col.usld[0], dt, rdt));
            pot -= se;
            col.usld[0] = col.usld[0] - se * dt;
            const double thd = lb_drainable(ts, col.tfc);
            if (col.nu == 0 || col.nu == 1) {
                esat = pot * jmin(1.0, div_(col.act[0] - zi, col.act[0]));
                esat = jmin(esat, div_by_((col.act[0] - zi) * thd, dt, rdt));
            } else {
                esat = 0.0;
            }
            soilevap = se + esat;
            drain -= esat * dt;
        }
        // transpiration! (soil.jl:865-975)
        double actevapustore = 0.0, act_sat, transpiration;
        {
            const double rd = L[ROOTING_DEPTH][slot];
            const double h1 = L[H1][slot], h2 = L[H2][slot], h4 = L[H4][slot], a1 = L[ALPHA_H1][slot];
            const double psi = L[PSI_B][slot];
            const double h3 = feddes_h3(L[H3_HIGH][slot], L[H3_LOW][slot], pot_trans);
            double sum_rf = 0.0, rf_low = 0.0;
#pragma unroll
            for (int k = 1; k <= MAXN; ++k) {
                if (k > col.nu) break;
                double r;
                if (k == col.nu && lt_(zi, rd)) {
                    const double rl = jmin(col.act[k - 1], rd - col.cum[k - 1]);
                    r = rfr[k - 1] * div_(col.thick[k - 1], rl);
                } else {
                    r = rfr[k - 1];
                }
                sum_rf += r;
                rf_low = r;
            }
            const double root_scale = jmax(div_(1.0, sum_rf), 1.0);
#pragma unroll
            for (int k = 1; k <= MAXN; ++k) {
                if (k > col.nu) break;
                const double r = k < col.nu ? rfr[k - 1] : rf_low;
                const double rs_ = gt0_(rd) ? root_scale * r : 0.0;
                const double r_thick = div_(1.0, col.thick[k - 1]);
                const double vwc = jmax(div_by_(col.usld[k - 1], col.thick[k - 1], r_thick), 1e-7);
                const double alpha = rwu_layer(vwc, ts, tr, cexp[k - 1], psi, h1, h2, h3, h4, a1);
                const double availcap =
                    jmin(1.0, jmax(0.0, div_by_(rd - col.cum[k - 1], col.thick[k - 1], r_thick)));
                const double maxextr = div_by_(col.usld[k - 1] * availcap, dt, rdt);
                const double a = jmin(alpha * rs_ * pot_trans, maxextr);
                col.usld[k - 1] = col.usld[k - 1] - a * dt;
                actevapustore += a;
            }
            const double wetroots = scurve(zi, rd, 1.0, L[ROOTDISTPAR][slot]);
            const double alpha0 = rwu_feddes(0.0, h1, h2, h3, h4, a1);
            const double rest = pot_trans - actevapustore;
            act_sat = jmin(rest * wetroots * alpha0, div_by_(drain, dt, rdt));
            drain -= act_sat * dt;
            transpiration = actevapustore + act_sat;
        }
        // actual_infiltration! (soil.jl:987-1017)
        double excess = 0.0;
#pragma unroll
        for (int k = MAXN; k >= 1; --k) {
            if (k > col.nu) continue;
            excess = jmax(0.0, col.usld[k - 1] - col.thick[k - 1] * (ts - tr));
            col.usld[k - 1] = col.usld[k - 1] - excess;
            if (k > 1) col.usld[k - 2] = col.usld[k - 2] + excess;
        }
        const double act_infilt = infiltration - div_by_(excess, dt, rdt);
        const double satex = (wfs_soil - act_infilt) - infex;
        // unsaturated store and capacity for the capillary flux (soil.jl:1193-1196)
        usd = 0.0;
#pragma unroll
        for (int k = 0; k < MAXN; ++k)
            if (k < col.nl) usd += col.usld[k];
        ucap = swc - sat - usd;
        // capillary_flux! (soil.jl:1050-1111)
        double capflux_act = 0.0;
        if (col.nu > 0) {
            const double ksat = col.kv_at(kvf, zi, col.nu);
            const double maxcap = jmax(0.0, jmin(jmin(jmin(ksat, actevapustore), div_by_(ucap, dt, rdt)), div_by_(drain, dt, rdt)));
            const double rd = L[ROOTING_DEPTH][slot];
            const double chmax = L[CAP_HMAX][slot];
            double capflux = gt_(zi, rd) ? maxcap * wfm::pow(1.0 - div_(jmin(zi, chmax), chmax), L[CAP_N][slot]) : 0.0;
#pragma unroll
            for (int k = MAXN; k >= 1; --k) {
                if (k > col.nu) continue;
                const double toadd =
                    jmin(capflux, jmax(div_by_(col.thick[k - 1] * (ts - tr) - col.usld[k - 1], dt, rdt), 0.0));
                col.usld[k - 1] = col.usld[k - 1] + toadd * dt;
                capflux -= toadd;
                capflux_act += toadd;
            }
        }
        // leakage! (soil.jl:1118-1136)
        const double deepksat = col.kv_at(kvf, col.d, col.nl);
        const double leak = jmax(0.0, jmin(L[MAX_LEAKAGE][slot], jmin(div_by_(drain, dt, rdt), deepksat)));
        const double recharge = (transfer - capflux_act - leak - act_sat - esat);
        double aet = soilevap + transpiration + ae_river + ae_land + 0.0;
        aet += ic;  // sbm.jl:130
        // ---- write back
        Mf[CANOPY][e] = canopy;
        Mf[SNOW][e] = snow;
        Mf[SNOW_WATER][e] = snow_water;
        Mf[TSOIL][e] = tsoil;
#pragma unroll
        for (int k = 0; k < MAXN; ++k)
            if (k < col.N) F.LY[LY_USLD][k][e] = col.usld[k];
        Mf[ZI][e] = zi;
        Mf[SSF_ZI][e] = zi;  // sbm_model.jl:80-81
        Mf[RECHARGE][e] = recharge;
        Mf[NET_RUNOFF_RIVER][e] = runoff_river - ae_river;
        Mf[AET][e] = aet;
        Mf[LEAKAGE][e] = leak;
        Mf[SATEX][e] = satex;
        Mf[INFEX][e] = infex;
        Mf[RUNOFF_LAND][e] = runoff_land;
        Mf[AE_LAND][e] = ae_land;
        Mf[INTERCEPTION][e] = ic;
        Mf[TRANSPIRATION][e] = transpiration;
        Mf[SOIL_EVAP][e] = soilevap;
        Mf[ACT_INFILT][e] = act_infilt;
    }
}

// ------------------------------------------------------------------ subsurface ----------

// Recharge flux of a cell (boundary_conditions.jl:219-236, check_flux :12-21)
__device__ __forceinline__ double ssf_flux(const WfDevFields& F, int64_t e, double area, double zi_ssf, double d) {
    const double flux = F.Mf[RECHARGE][e] * area;
    return wfm::le_(d, zi_ssf) ? jmax(0.0, flux) : flux;
}

// The soil column of a cell as the subsurface update finds it
template <int MAXN>
__device__ __forceinline__ void ssf_column(const WfDevFields& F, int64_t slot, int64_t e, Column<MAXN>& col) {
    col.load_static(F, slot);
    col.kv0 = F.Mf[KV0][e];
    col.f = F.Mf[FSCALE][e];
#pragma unroll
    for (int k = 0; k < MAXN; ++k) col.usld[k] = k < col.N ? F.LY[LY_USLD][k][e] : 0.0;
}

// One sub-step of a cell for the upstream inflow qin (tr: what of the upstream discharge goes to the
// river): discharge, water table, storages and cumulative fluxes, after the model step's last sub-step
// the averages and update_soil_water_storage!. Returns the discharge.
template <int MAXN>
__device__ double ssf_cell(const WfDevFields& F, int64_t slot, int64_t e, double qin, double tr, double dt_s, bool first,
                           bool last, double dt) {
    double* const* Mf = F.Mf;
    double* const* L = F.L;
    const double area = L[AREA][slot];
    const double d = L[SOIL_THICKNESS][slot];
    const double zi_ssf = Mf[SSF_ZI][e];
    const double flux = ssf_flux(F, e, area, zi_ssf, d);
    const double q_net = 0.0 + flux;
    Column<MAXN> col;
    ssf_column(F, slot, e, col);
    const double zi_soil = Mf[ZI][e];
    col.set_thickness(zi_soil);
    const double q_prev = Mf[SSF_Q][e];
    const double kh0 = L[KH_RATIO][slot] * col.kv0;
    double q, zi_new, exfilt, netflux;
    kinematic_wave_ssf<MAXN>(qin, q_prev, zi_ssf, q_net, L[SLOPE][slot], L[SY][slot], d, dt_s, L[FLOW_LENGTH][slot],
                             L[FLOW_WIDTH][slot], Mf[Q_MAX][e], kh0, col, q, zi_new, exfilt, netflux);
    const bool early = (qin + q_prev == 0.0 && q_net <= 0.0);
    Mf[SSF_Q][e] = q;
    Mf[SSF_ZI][e] = zi_new;
    Mf[SSF_STORAGE][e] = L[SY][slot] * (d - zi_new) * area;
    // cumulative fluxes (set_flux_vars! zeroes them at the start of the model step)
    double c_tr = (first ? 0.0 : Mf[SSF_TR_CUM][e]) + tr * dt_s;
    double c_rf = (first ? 0.0 : Mf[RCH_FLUX_CUM][e]) + flux * dt_s;
    double c_qin = (first ? 0.0 : Mf[SSF_QIN_CUM][e]) + qin * dt_s;
    double c_q = (first ? 0.0 : Mf[SSF_Q_CUM][e]) + q * dt_s;
    double c_ex = (first ? 0.0 : Mf[SSF_EXF_CUM][e]) + exfilt * dt_s;
    double c_nf = (first ? 0.0 : Mf[SSF_QNET_CUM][e]) + netflux * area * dt_s;
    if (!early) {
#pragma unroll
        for (int k = 0; k < MAXN; ++k)
            if (k < col.N) F.LY[LY_USLD][k][e] = col.usld[k];
        Mf[ZI][e] = zi_new;
    }
    if (!last) {
        Mf[SSF_TR_CUM][e] = c_tr;
        Mf[RCH_FLUX_CUM][e] = c_rf;
        Mf[SSF_QIN_CUM][e] = c_qin;
        Mf[SSF_Q_CUM][e] = c_q;
        Mf[SSF_EXF_CUM][e] = c_ex;
        Mf[SSF_QNET_CUM][e] = c_nf;
        return q;
    }
    // averages (groundwater.jl:622-638, lateral_subsurface_flow.jl:182-196)
    const double rdt = div_(1.0, dt);
    const double exf_avg = div_by_(c_ex, dt, rdt);
    Mf[RCH_FLUX_AVG][e] = div_by_(c_rf, dt, rdt);
    Mf[SSF_QIN_AVG][e] = div_by_(c_qin, dt, rdt);
    Mf[SSF_Q_AVG][e] = div_by_(c_q, dt, rdt);
    Mf[SSF_QNET_AVG][e] = div_by_(c_nf, dt, rdt);
    Mf[SSF_EXF_AVG][e] = exf_avg;
    Mf[SSF_TR_AVG][e] = div_by_(c_tr, dt, rdt);
    // ---- update_soil_water_storage! (soil.jl:1294-1392), soil state after the sweep
    if (early) {
        // the soil column kept its state: reload it
#pragma unroll
        for (int k = 0; k < MAXN; ++k) col.usld[k] = k < col.N ? F.LY[LY_USLD][k][e] : 0.0;
        col.set_thickness(zi_soil);
    }
    const double zi_s = early ? zi_soil : zi_new;
    const double ts = col.ts, tr_ = col.tr;
    double usd = 0.0;
#pragma unroll
    for (int k = 0; k < MAXN; ++k)
        if (k < col.nu) usd += col.usld[k];
    const double runoff =
        jmax(0.0, exf_avg + Mf[SATEX][e] + Mf[RUNOFF_LAND][e] + Mf[INFEX][e]);
    const double sat = (d - zi_s) * (ts - tr_);
    Mf[SAT][e] = sat;
    Mf[USTOREDEPTH][e] = usd;
    Mf[TSWS][e] = sat + usd;
    Mf[EXFILT][e] = exf_avg;
    Mf[RUNOFF][e] = runoff;
    const double net_runoff = runoff - Mf[AE_LAND][e];
    Mf[NET_RUNOFF][e] = net_runoff;
    // overland lateral inflow (surface_kinwave.jl:740-766, :365)
    const double inwater = (net_runoff + 0.0) * area + 0.0;
    Mf[OL_INWATER][e] = inwater;
    Mf[OL_QLAT][e] = div_(inwater, L[FLOW_LENGTH][slot]);
    return q;
}

// Subsurface sweep of several sub-steps (fixed ones shorter than the model step, or adaptive): the
// whole cell update in the wavefront walker, since each sub-step needs the column of the last.
template <int MAXN>
struct SsfPhys {
    WfDevFields F;
    WfDevGraph g;
    WfSweep sw;

    __device__ bool node(int64_t slot, int64_t e, int m, int s, uint32_t ep, int64_t chain, bool is_end,
                         double& hq) {
        double dt_s;
        bool first, last;
        if (!wf_substep(sw, m, s, dt_s, first, last)) return true;
        // upstream inflow (lateral_subsurface_flow.jl:236-242)
        double qin = 0.0, tr = 0.0;
        for (int32_t o = g.up_ptr[slot]; o < g.up_ptr[slot + 1]; ++o) {
            double qu;
            if (!wfw::upstream_q(g, sw, hq, o, m, s, ep, F.status, qu)) return false;
            const double fr = g.up_fr[o];
            qin = qin + qu * (1.0 - fr);
            tr = tr + qu * fr;
        }
        hq = ssf_cell<MAXN>(F, slot, e, qin, tr, dt_s, first, last, sw.dt);
        if (is_end) wfw::publish(g, chain, m, s, ep, hq);
        return true;
    }
};

// ---- one sub-step per model step: terms per cell | slim wavefront | cell update

// The sweep's discharge follows from the inflow alone unless the water table moves by the
// sub-iteration threshold or below the soil bottom. Falling, it moves by |net| dt / (dw dx sy). Rising,
// it fills the unsaturated layers from below: W_RISE is the volume that raises it by 0.0989 m
// (water_table_change's fluxes up to that height), over dt. Both with 1 % in hand of the 0.1 m of
// the reference's threshold, so a net flux below them takes no sub-iteration, whatever the roundings.
template <int MAXN>
__global__ void __launch_bounds__(128) ssf_prep64_kernel(WfDevFields F, WfSweep sw) {
    const int M = F.M;
    const int64_t E = F.land_slots * M;
    double* const* Mf = F.Mf;
    double* const* L = F.L;
    const double dt = sw.dt_s, rdt = div_(1.0, dt);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if (F.land_node_of_slot[slot] < 0) continue;
        const double d = L[SOIL_THICKNESS][slot], zi = Mf[SSF_ZI][e];
        const double dx = L[FLOW_LENGTH][slot], dw = L[FLOW_WIDTH][slot], sy = L[SY][slot];
        const double q_prev = Mf[SSF_Q][e];
        Column<MAXN> col;
        ssf_column(F, slot, e, col);
        col.set_thickness(Mf[ZI][e]);
        const double kh0 = L[KH_RATIO][slot] * col.kv0;
        const double cel = ssf_celerity(zi, L[SLOPE][slot], sy, kh0, col.f, col.profile, col.zexp);
        const double dt_dx = div_(dt, dx), cinv = div_(1.0, cel);
        const double df = dt_dx + cinv;
        F.W[W_SDTDX][e] = dt_dx;
        F.W[W_CINV][e] = cinv;
        F.W[W_SDF][e] = df;
        F.W[W_SRDF][e] = div_(1.0, df);
        F.W[W_QPC][e] = div_by_(q_prev, cel, cinv);
        F.W[W_QNET][e] = 0.0 + ssf_flux(F, e, L[AREA][slot], zi, d);
        F.W[W_QLIM][e] = Mf[Q_MAX][e] * dw;
        const double te = col.ts - col.tr;
        double x = 0.0, h = 0.0;
        bool reached = false;
#pragma unroll
        for (int k = MAXN; k >= 1; --k) {
            if (k > col.nu || reached) continue;
            const double t = col.thick[k - 1], cap = jmax(t * te - col.usld[k - 1], 0.0);
            if (gt_(h + t, 0.0989)) {
                const double need = jmax((0.0989 - h) * (te - div_(col.usld[k - 1], t)), 0.0);
                x += jmin(need, cap);
                reached = true;
            } else {
                x += cap;
                h += t;
            }
        }
        const double per_dt = dw * dx * rdt * (1.0 - 1e-6);
        F.W[W_RISE][e] = reached ? x * per_dt : wfm::from_bits(0x7ff0000000000000ULL);
        F.W[W_FALL][e] = jmin(0.0989, d - zi - 1e-9) * sy * per_dt;
    }
}

template <int MAXN>
struct SsfWave64 {
    static constexpr bool kLand = true, kTr = false;
    WfDevFields F;
    WfDevGraph g;
    WfSweep sw;

    struct In {
        double dt_dx, cinv, df, rdf, qpc, q_net, q_lim, rise, fall, q_prev;
    };
    struct St {
        double q;
    };
    __device__ __forceinline__ void load(int64_t slot, int64_t e, int m, bool fresh, bool resumed, In& x) const {
        double* const* W = F.W;
        x.dt_dx = W[W_SDTDX][e];
        x.cinv = W[W_CINV][e];
        x.df = W[W_SDF][e];
        x.rdf = W[W_SRDF][e];
        x.qpc = W[W_QPC][e];
        x.q_net = W[W_QNET][e];
        x.q_lim = W[W_QLIM][e];
        x.rise = W[W_RISE][e];
        x.fall = W[W_FALL][e];
        x.q_prev = F.Mf[SSF_Q][e];
    }
    __device__ __forceinline__ void start(const In&, St&) const {}
    // The discharge of a cell whose water table moves across the threshold or the soil bottom
    __device__ __noinline__ double full(int64_t slot, int64_t e, double qin, double q_net) const {
        double* const* L = F.L;
        Column<MAXN> col;
        ssf_column(F, slot, e, col);
        col.set_thickness(F.Mf[ZI][e]);
        double q, zi_new, exfilt, netflux;
        kinematic_wave_ssf<MAXN>(qin, F.Mf[SSF_Q][e], F.Mf[SSF_ZI][e], q_net, L[SLOPE][slot], L[SY][slot],
                                 L[SOIL_THICKNESS][slot], sw.dt_s, L[FLOW_LENGTH][slot], L[FLOW_WIDTH][slot],
                                 F.Mf[Q_MAX][e], L[KH_RATIO][slot] * col.kv0, col, q, zi_new, exfilt, netflux);
        return q;
    }
    __device__ __forceinline__ bool active(int, St&) const { return true; }
    __device__ __forceinline__ void sub(const In& x, St& st, const wfz::Rec& r, double qin, double tr, int64_t slot,
                                        int64_t e, int m, int s, int64_t chain, bool is_end, double& hq, bool more) {
        double q;
        // the early-out of kinematic_wave_ssf; its full form decides when a discharge is negative
        const bool none = wfm::is_zero_(qin) && wfm::is_zero_(x.q_prev);
        if (none && le0_(x.q_net)) {
            q = 0.0;
        } else if (lt_(qin, 0.0) || lt_(x.q_prev, 0.0)) {
            q = full(slot, e, qin, x.q_net);
        } else {
            const double in_net = qin + x.q_net;
            q = kw_ssf_newton(mean2(x.q_prev, qin), x.dt_dx * in_net + x.qpc, x.dt_dx, x.cinv, x.df, x.rdf);
            q = jmin(q, x.q_lim);
            const double net = in_net - q;
            if (!(gt0_(net) ? lt_(net, x.rise) : lt_(-net, x.fall))) q = full(slot, e, qin, x.q_net);
        }
        st.q = q;
        hq = q;
        if (is_end) wfz::publish(g, chain, m, s, q);
    }
    __device__ __forceinline__ void finish(const St& st, int64_t e, bool) const { F.W[W_Q][e] = st.q; }
};

// The cell update from the sweep's discharges (ssf_cell repeats the cell's own solve: its water table
// and column need the discharge before the soil-bottom limit).
template <int MAXN>
__global__ void __launch_bounds__(128) ssf_post64_kernel(WfDevFields F, WfDevGraph g, WfSweep sw) {
    const int M = F.M;
    const int64_t E = F.land_slots * M;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if (F.land_node_of_slot[slot] < 0) continue;
        const int m = (int)(e - slot * M);
        double qin = 0.0, tr = 0.0;
        for (int32_t o = g.up_ptr[slot]; o < g.up_ptr[slot + 1]; ++o) {
            const double qu = F.W[W_Q][g.up_slot[o] * M + m], fr = g.up_fr[o];
            qin = qin + qu * (1.0 - fr);
            tr = tr + qu * fr;
        }
        ssf_cell<MAXN>(F, slot, e, qin, tr, sw.dt_s, true, true, sw.dt);
    }
}

// ------------------------------------------- overland and river kinematic waves ---------

// Terms of a sweep launch per cell: storage_prev! at the first sub-step of the model step, the river's
// lateral inflow, and the solve's terms of the state before the launch.
template <bool LAND>
__global__ void __launch_bounds__(128) kw_prep64_kernel(WfDevFields F, WfSweep sw) {
    const int M = F.M;
    const int64_t E = (LAND ? F.land_slots : F.river_slots) * M;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if ((LAND ? F.land_node_of_slot : F.river_node_of_slot)[slot] < 0) continue;
        const int m = (int)(e - slot * M);
        bool first = sw.first == 0;
        double dt_s = sw.dt_s;
        if (sw.aflag) {
            bool last;
            if (!wf_substep(sw, m, 0, dt_s, first, last)) continue;
        }
        double dx, alpha, q_prev, q_lat;
        if (LAND) {
            if (first && F.mass_balance) F.Mf[BO_PREV][e] = F.Mf[OL_STORAGE][e];
            dx = F.L[FLOW_LENGTH][slot];
            alpha = F.L[OL_ALPHA][slot];
            q_prev = F.Mf[OL_Q][e];
            q_lat = F.Mf[OL_QLAT][e];
        } else {
            double* const* RM = F.RM;
            double* const* R = F.R;
            dx = R[R_LENGTH][slot];
            const double rlen = div_(1.0, dx);
            if (first) {
                if (F.mass_balance) RM[BR_PREV][e] = RM[RV_STORAGE][e];
                // update_lateral_inflow! (surface_kinwave.jl:710-734)
                const int64_t le = F.river_land_slot[slot] * M + m;
                const double inw = F.Mf[SSF_TR_AVG][le] + F.Mf[OL_TR_AVG][le] +
                                   F.Mf[NET_RUNOFF_RIVER][le] * R[R_AREA][slot] + 0.0;
                RM[RV_INWATER][e] = inw;
                q_lat = div_by_(inw, dx, rlen);
                RM[RV_QLAT][e] = q_lat;
            } else {
                q_lat = RM[RV_QLAT][e];
            }
            // external inflow (surface_kinwave.jl:523-532); the wavefront adds an abstraction itself
            const double ext = R[R_EXT_INFLOW][slot];
            if (!lt_(ext, 0.0)) q_lat = q_lat + (div_by_(ext, dx, rlen) - 0.0);
            alpha = R[R_ALPHA][slot];
            q_prev = RM[RV_Q][e];
        }
        const double dt_dx = div_(dt_s, dx), c1 = 5.0 * dt_dx, c2 = 3.0 * alpha;
        wfz::KwState k;
        wfz::kw_state(q_prev, dt_dx, alpha, c1, c2, k);
        double* const* W = F.W;
        W[W_U][e] = k.u;
        W[W_A][e] = k.A;
        W[W_P][e] = k.P;
        W[W_DF][e] = k.df;
        W[W_RDF][e] = k.rdf;
        W[W_B][e] = dt_s * q_lat;
        W[W_DTDX][e] = dt_dx;
        W[W_C1][e] = c1;
        W[W_C2][e] = c2;
    }
}

// The wavefront. CUM: the walker sums the discharges, inflows (land: and flows to the river) over the
// launch's sub-steps; a launch of one sub-step leaves the sums to the completion kernel, which finds
// the upstream discharges in the discharge array (not with RES). RES: the model has reservoirs; a
// reservoir cell hands its reservoir's outflow, not its river discharge, to the downstream cell.
template <bool LAND, bool CUM, bool RES>
struct KwWave64 {
    static constexpr bool kLand = LAND, kTr = CUM;
    WfDevFields F;
    WfDevGraph g;
    WfSweep sw;

    struct In {
        wfz::KwState k;
        double b, dt_dx, c1, c2, alpha, q_prev;
        double u;                // river: final iterate of the round before, if there was one
        double c_q, c_qin, c_x;  // cumulative discharge, inflow, flow to the river (abstraction)
    };
    struct St {
        wfz::KwState k;
        double q_prev, u;
        double c_q, c_qin, c_x;
    };
    __device__ __forceinline__ double* q_of() const { return LAND ? F.Mf[OL_Q] : F.RM[RV_Q]; }
    __device__ __forceinline__ double* cq_of() const { return LAND ? F.Mf[OL_Q_CUM] : F.RM[RV_Q_CUM]; }
    __device__ __forceinline__ double* cqin_of() const { return LAND ? F.Mf[OL_QIN_CUM] : F.RM[RV_QIN_CUM]; }
    __device__ __forceinline__ double* cx_of() const { return LAND ? F.Mf[OL_TR_CUM] : F.RM[RV_ABS_CUM]; }

    __device__ __forceinline__ void load(int64_t slot, int64_t e, int m, bool fresh, bool resumed, In& x) const {
        double* const* W = F.W;
        x.k.u = W[W_U][e];
        x.k.A = W[W_A][e];
        x.k.P = W[W_P][e];
        x.k.df = W[W_DF][e];
        x.k.rdf = W[W_RDF][e];
        x.b = W[W_B][e];
        x.dt_dx = W[W_DTDX][e];
        x.c1 = W[W_C1][e];
        x.c2 = W[W_C2][e];
        x.alpha = LAND ? F.L[OL_ALPHA][slot] : F.R[R_ALPHA][slot];
        x.q_prev = q_of()[e];
        x.u = !LAND && resumed ? W[W_UEND][e] : 0.0;
        x.c_q = x.c_qin = x.c_x = 0.0;
        if (CUM) {
            if (sw.aflag) fresh = (sw.aflag[m] & WF_SUB_FIRST) != 0;
            if (!fresh) {
                x.c_q = cq_of()[e];
                x.c_qin = cqin_of()[e];
                x.c_x = cx_of()[e];
            }
        }
    }
    __device__ __forceinline__ void start(const In& x, St& st) const {
        st.k = x.k;
        st.q_prev = x.q_prev;
        st.u = x.u;
        st.c_q = x.c_q;
        st.c_qin = x.c_qin;
        st.c_x = x.c_x;
    }
    // a member that has reached the end of the step takes no further sub-step
    __device__ __forceinline__ bool active(int m, St& st) const {
        if (!sw.aflag || (sw.aflag[m] & WF_SUB_ACTIVE)) return true;
        st.u = -1.0;
        return false;
    }
    __device__ __forceinline__ void sub(const In& x, St& st, const wfz::Rec& r, double qin, double tr, int64_t slot,
                                        int64_t e, int m, int s, int64_t chain, bool is_end, double& hq, bool more) {
        const double dt_s = sw.aflag ? sw.adt[m] : sw.dt_s;
        if (LAND && (r.flags & wfz::REC_NO_INFLOW)) qin = 0.0;
        const float r_dt32 = __frcp_rn(wfm::f32_of(dt_s));
        double b = x.b, q_lat = 0.0, taken = 0.0;
        const bool draws = !LAND && (r.flags & wfz::REC_ABSTRACTION);
        if (draws) {  // abstraction up to 80 % of the storage (surface_kinwave.jl:523-532)
            const double len = F.R[R_LENGTH][slot], ext = F.R[R_EXT_INFLOW][slot];
            // the storage that the previous sub-step left (of this launch: from its final iterate st.u)
            const double storage =
                s > 0 ? len * (wfm::is_zero_(st.q_prev) ? 0.0 : x.alpha * (st.u * st.u * st.u)) : F.RM[RV_STORAGE][e];
            taken = jmin(-ext, div_(storage, dt_s) * 0.80);
            q_lat = F.RM[RV_QLAT][e] + (div_(-taken, len) - 0.0);
            b = dt_s * q_lat;
        }
        double q, u;
        bool zero = false;
        // q_in + q_prev + q_lat == 0: only without a positive previous discharge or with a negative term,
        // and then not where the sum in FP32 is far above what the three terms' roundings leave
        const float in32 = wfm::f32_of(qin), prev32 = wfm::f32_of(st.q_prev), lat32 = wfm::f32_of(b) * r_dt32;
        if (!(gt0_(st.q_prev) && !lt_(b, 0.0) && !lt_(qin, 0.0)) &&
            !(fabsf(in32 + prev32 + lat32) > 1e-4f * (fabsf(in32) + fabsf(prev32) + fabsf(lat32)))) {
            if (!draws)
                q_lat = LAND ? F.Mf[OL_QLAT][e]
                             : F.RM[RV_QLAT][e] + (div_(F.R[R_EXT_INFLOW][slot], F.R[R_LENGTH][slot]) - 0.0);
            zero = wfm::is_zero_(qin + st.q_prev + q_lat);
        }
        if (zero) {
            q = u = 0.0;
        } else {
            q = wfz::kw_solve(st.k, x.dt_dx * qin + st.k.A + b, x.dt_dx, x.alpha, x.c1, x.c2, u);
        }
        double q_down = q;
        if (RES) {
            const int32_t res = F.res_of_rslot[slot];
            if (res >= 0) q_down = wfr::reservoir_node(F, res, m, q, dt_s);
        }
        hq = q_down;
        if (is_end) wfz::publish(g, chain, m, s, q_down);
        if (CUM) {
            st.c_q = st.c_q + q * dt_s;
            st.c_qin = st.c_qin + qin * dt_s;
            if (LAND ? (r.flags & wfz::REC_WEIGHTED) != 0 : draws) st.c_x = st.c_x + (LAND ? tr : taken) * dt_s;
        }
        st.q_prev = q;
        st.u = u;
        if (more) wfz::kw_state(q, x.dt_dx, x.alpha, x.c1, x.c2, st.k);
    }
    __device__ __forceinline__ void finish(const St& st, int64_t e, bool last_round) const {
        if (lt_(st.u, 0.0)) return;  // no sub-step taken
        q_of()[e] = st.q_prev;
        F.W[W_UEND][e] = st.u;
        if (CUM) {
            cq_of()[e] = st.c_q;
            cqin_of()[e] = st.c_qin;
            cx_of()[e] = st.c_x;
        }
        if (!last_round) {
            F.W[W_U][e] = st.k.u;
            F.W[W_A][e] = st.k.A;
            F.W[W_P][e] = st.k.P;
            F.W[W_DF][e] = st.k.df;
            F.W[W_RDF][e] = st.k.rdf;
        }
    }
};

// After a sweep launch: depth and storage of every cell, its sums when the walker has not kept them
// (CUM), and after the model step's last sub-step the averages.
template <bool LAND, bool CUM>
__global__ void __launch_bounds__(128) kw_post64_kernel(WfDevFields F, WfDevGraph g, WfSweep sw) {
    const int M = F.M;
    const int64_t E = (LAND ? F.land_slots : F.river_slots) * M;
    const double dt = sw.dt, rdt = div_(1.0, dt);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if ((LAND ? F.land_node_of_slot : F.river_node_of_slot)[slot] < 0) continue;
        const int m = (int)(e - slot * M);
        bool first = sw.first == 0, last = sw.last_of_step != 0;
        double dt_s = sw.dt_s;
        if (sw.aflag && !wf_substep(sw, m, 0, dt_s, first, last)) continue;
        const double u = F.W[W_UEND][e];
        const double* q_all = LAND ? F.Mf[OL_Q] : F.RM[RV_Q];
        const double q = q_all[e];
        const double area = wfm::is_zero_(q) ? 0.0 : (LAND ? F.L[OL_ALPHA][slot] : F.R[R_ALPHA][slot]) * (u * u * u);
        const int32_t flags = g.up_rec64[slot].z;
        double* cq = LAND ? F.Mf[OL_Q_CUM] : F.RM[RV_Q_CUM];
        double* cqin = LAND ? F.Mf[OL_QIN_CUM] : F.RM[RV_QIN_CUM];
        double* cx = LAND ? F.Mf[OL_TR_CUM] : F.RM[RV_ABS_CUM];
        double c_q, c_qin, c_x;
        if (CUM) {
            c_q = cq[e];
            c_qin = cqin[e];
            c_x = cx[e];
        } else {
            double qin = 0.0, tr = 0.0, taken = 0.0;
            for (int32_t o = g.up_ptr[slot]; o < g.up_ptr[slot + 1]; ++o) {
                const double qu = q_all[g.up_slot[o] * M + m];
                if (LAND) {
                    tr = tr + qu * g.up_fr[o];
                    qin = qin + qu * g.up_w[o];
                } else {
                    qin = qin + qu;
                }
            }
            if (flags & wfz::REC_NO_INFLOW) qin = 0.0;
            // the storage before the sub-step: this kernel overwrites it below
            if (!LAND && (flags & wfz::REC_ABSTRACTION))
                taken = jmin(-F.R[R_EXT_INFLOW][slot], div_(F.RM[RV_STORAGE][e], dt_s) * 0.80);
            c_q = (first ? 0.0 : cq[e]) + q * dt_s;
            c_qin = (first ? 0.0 : cqin[e]) + qin * dt_s;
            c_x = (first ? 0.0 : cx[e]) + (LAND ? tr : taken) * dt_s;
            if (!last) {
                cq[e] = c_q;
                cqin[e] = c_qin;
                cx[e] = c_x;
            }
        }
        if (LAND) {
            const double sfw = F.L[SFW][slot];
            double h = F.Mf[OL_H][e];
            if (gt0_(sfw)) h = div_(area, sfw);
            F.Mf[OL_H][e] = h;
            F.Mf[OL_STORAGE][e] = F.L[FLOW_LENGTH][slot] * sfw * h;
        } else {
            F.RM[RV_H][e] = div_(area, F.R[R_WIDTH][slot]);
            F.RM[RV_STORAGE][e] = F.R[R_LENGTH][slot] * area;
        }
        if (!last) continue;
        (LAND ? F.Mf[OL_Q_AVG] : F.RM[RV_Q_AVG])[e] = div_by_(c_q, dt, rdt);
        (LAND ? F.Mf[OL_TR_AVG] : F.RM[RV_ABS_AVG])[e] = div_by_(c_x, dt, rdt);
        (LAND ? F.Mf[OL_QIN_AVG] : F.RM[RV_QIN_AVG])[e] = div_by_(c_qin, dt, rdt);
    }
}

template <class Phys, bool MULTI>
__global__ void __launch_bounds__(128) wave64_kernel(Phys phys, int64_t p_chunks, int SLp, int SLs, int SLr,
                                                     int batch) {
    wfz::walk<Phys, MULTI>(phys, p_chunks, SLp, SLs, SLr, batch, phys.F.status);
}

// --------------------------------------------------------- gravitational snow transport ----

// One material of lateral_snow_transport! (surface_process.jl:9-19): accucapacityflux! over the
// land graph (routing/utils.jl:82-104, 144-148). A cell's material is its own plus the hand-offs
// of its upstream cells, added in the order of the graph's topological sort (the order in which
// the reference's sweep hands them on); it passes min(material / dt, capacity) on to its
// downstream cell and keeps the rest. MAT 0: snow storage (snow_out = its flux), MAT 1: snow
// water (snow_out += its flux). FP64 in both forms (the split form's double-FP32 states are
// converted on the way in and out). A chain position is bound by its loads in a row: the upstream list
// in the transport's order (snow_up: its chains), then the words of up to four children together.
template <int MAT>
struct SnowPhys {
    WfDevFields F;
    WfDevGraph g;
    WfSweep sw;

    __device__ bool node(int64_t slot, int64_t e, int m, int s, uint32_t ep, int64_t chain, bool is_end,
                         double& hq) {
        const int f = MAT == 0 ? SNOW : SNOW_WATER;
        double material = F.split ? (double)F.Mh[f][e] + (double)F.Ml[f][e] : F.Mf[f][e];
        const double cap = F.GM[MAT == 0 ? GM_CAP : GM_CAPW][e];
        const double before = MAT == 0 ? 0.0 : F.GM[GM_SNOW_OUT][e];
        const int32_t o0 = __ldg(g.up_ptr + slot), o1 = __ldg(g.up_ptr + slot + 1);
        int skip = 0;
        for (int32_t o = o0; o < o1; o += wfv::GROUP) {
            wfv::UpGroup u;
            if (!wfv::gather_group(g, sw, g.snow_up, o, o1, skip, m, s, F.status, u)) return false;
#pragma unroll
            for (int i = 0; i < wfv::GROUP; ++i)
                if (u.chain[i] >= -1) material += u.chain[i] < 0 ? hq : wfm::from_bits(u.word[i]);
        }
        const double dt = sw.dt;
        const double flux = jmin(div_(material, dt), cap);
        const double update = flux * dt;
        material -= update;
        if (F.split) {
            const wff::ff v = wff::from_d(material);
            F.Mh[f][e] = v.hi;
            F.Ml[f][e] = v.lo;
        } else {
            F.Mf[f][e] = material;
        }
        F.GM[GM_SNOW_OUT][e] = MAT == 0 ? flux : before + flux;
        hq = update;
        if (is_end) wfz::publish(g, chain, m, s, update);
        return true;
    }
};

// flux_in! (routing/utils.jl:160-166): snow_in = the snow_out of the upstream cells, summed in
// the upstream lists' (ascending) order.
__global__ void __launch_bounds__(256) snow_in_kernel(WfDevFields F, WfDevGraph g) {
    const int M = F.M;
    const int64_t E = F.land_slots * M;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if (F.land_node_of_slot[slot] < 0) continue;
        const int m = (int)(e - slot * M);
        double acc = 0.0;
        for (int32_t o = g.up_ptr[slot]; o < g.up_ptr[slot + 1]; ++o) acc = acc + F.GM[GM_SNOW_OUT][g.up_slot[o] * M + m];
        F.GM[GM_SNOW_IN][e] = acc;
    }
}

template <class Phys>
__global__ void __launch_bounds__(128) walk_kernel(Phys phys) {
    wfw::walk(phys.g, phys.sw, phys, phys.F.status);
}

// ------------------------------------------------------------------ balance ------------

__device__ __forceinline__ void mb_error(double tin, double tout, double rate, double& err, double& rel) {
    err = tin - tout - rate;
    const double avg = (tin + tout) / 2.0;
    rel = avg == 0.0 ? 0.0 : err / avg;
}

__global__ void __launch_bounds__(256) balance_kernel(WfDevFields F) {
    const int M = F.M;
    const int64_t EL = F.land_slots * M, ER = F.river_slots * M;
    const double dt = F.dt;
    double* const* Mf = F.Mf;
    double* const* L = F.L;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < EL + ER; e += (int64_t)gridDim.x * blockDim.x) {
        if (e >= EL) {
            if (!F.mass_balance || F.li_coupled) continue;
            const int64_t re = e - EL;
            const int64_t rs = re / M;
            if (F.river_node_of_slot[rs] < 0) continue;
            double* const* RM = F.RM;
            // river kinematic wave balance (mass_balance.jl:290-313)
            const double tin = RM[RV_INWATER][re] + RM[RV_QIN_AVG][re] + jmax(0.0, F.R[R_EXT_INFLOW][rs]);
            const double tout = RM[RV_Q_AVG][re] + RM[RV_ABS_AVG][re] + 0.0;
            double err, rel;
            mb_error(tin, tout, (RM[RV_STORAGE][re] - RM[BR_PREV][re]) / dt, err, rel);
            RM[BR_ERR][re] = err;
            RM[BR_REL][re] = rel;
            continue;
        }
        const int64_t slot = e / M;
        if (F.land_node_of_slot[slot] < 0) continue;
        const int m = (int)(e - slot * M);
        // update_total_water_storage! (sbm.jl:143-182)
        const int64_t rs = F.land_river_slot[slot];
        const double area = L[AREA][slot];
        double ts = 0.0;
        if (rs >= 0) ts = ((F.RM[RV_H][rs * M + m] * F.R[R_WIDTH][rs] * F.R[R_LENGTH][rs]) / (area));
        const double snow = Mf[SNOW][e], sw = Mf[SNOW_WATER][e], canopy = Mf[CANOPY][e];
        const double glacier = glacier_storage(F, e, slot);
        ts += snow + sw + glacier + canopy + 0.0;
        const double sub_surface = Mf[USTOREDEPTH][e] + Mf[SAT][e];
        const double lateral = Mf[OL_H][e] * (1.0 - L[RIVER_FRACTION][slot]);
        ts += sub_surface + lateral;
        Mf[TOTAL_STORAGE][e] = ts;
        if (!F.mass_balance) continue;
        double err, rel;
        // land hydrology balance (mass_balance.jl:215-253)
        {
            const double Pv = F.split ? (double)F.Mh[PRECIP][e] : Mf[PRECIP][e];
            const double snow_in = F.snow_transport ? F.GM[GM_SNOW_IN][e] : 0.0;
            const double snow_out = F.snow_transport ? F.GM[GM_SNOW_OUT][e] : 0.0;
            const double tin = Mf[SSF_QIN_AVG][e] / area + (Pv + 0.0) + snow_in + 0.0 / area;
            const double vout = Mf[NET_RUNOFF][e] + Mf[AET][e] + Mf[NET_RUNOFF_RIVER][e] + Mf[LEAKAGE][e] + 0.0;
            const double tout = Mf[SSF_Q_AVG][e] / area + vout + snow_out + 0.0 / area;
            const double storage = Mf[TSWS][e] + canopy + (snow + sw) + glacier + 0.0;
            mb_error(tin, tout, (storage - Mf[BL_PREV][e]) / dt, err, rel);
            Mf[BL_ERR][e] = err;
            Mf[BL_REL][e] = rel;
        }
        // overland balance (mass_balance.jl:382-399); the local-inertial one is written by
        // li_couple_out_kernel
        if (!F.li_coupled) {
            mb_error(Mf[OL_INWATER][e] + Mf[OL_QIN_AVG][e], Mf[OL_Q_AVG][e],
                     (Mf[OL_STORAGE][e] - Mf[BO_PREV][e]) / dt, err, rel);
            Mf[BO_ERR][e] = err;
            Mf[BO_REL][e] = rel;
        }
        // subsurface balance (mass_balance.jl:470-490, groundwater.jl:671-695)
        {
            const double flux = Mf[RCH_FLUX_AVG][e];
            double fin = 0.0, fout = 0.0;
            if (flux > 0.0) fin += flux; else fout -= flux;
            mb_error(Mf[SSF_QIN_AVG][e] + fin, Mf[SSF_Q_AVG][e] + fout, Mf[SSF_QNET_AVG][e], err, rel);
            Mf[BS_ERR][e] = err;
            Mf[BS_REL][e] = rel;
        }
    }
}

// ---------------------------------------------------- local-inertial routing in the step ----
// (wf_li_couple.cuh; one member, FP64 form: element = slot)

// update_bc_overland_flow_model! (surface_staggered_scheme.jl:1080-1097): the land runoff of
// the step into the scheme's input, in its node order; the river's external inflow; the overland
// storage before the step for the balance (storage_prev!, mass_balance.jl:170-183).
__global__ void __launch_bounds__(256) li_couple_in_kernel(WfDevFields F, WfLiCoupleView v) {
    double* const* Mf = F.Mf;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < F.land_slots;
         s += (int64_t)gridDim.x * blockDim.x) {
        const int64_t node = F.land_node_of_slot[s];
        if (node < 0) continue;
        double ro = (Mf[NET_RUNOFF][s] + Mf[NET_RUNOFF_RIVER][s]) * F.L[AREA][s];
        const int64_t rs = F.land_river_slot[s];
        if (rs >= 0) {
            ro += Mf[SSF_TR_AVG][s];  // get_flux_to_river (lateral_subsurface_flow.jl:346-347)
            v.ext[F.river_node_of_slot[rs]] = F.R[R_EXT_INFLOW][rs];
        }
        v.runoff[node] = ro;
        if (F.mass_balance) Mf[BO_PREV][s] = Mf[OL_STORAGE][s];
    }
}

// After the scheme's step: its depths, storages and the discharge of each river cell's outgoing
// edge into the model's overland and river fields, and the overland balance of every land cell
// (compute_flow_balance!, mass_balance.jl:402-461; add_inflow / add_outflow :355-376) with the
// river balance cleared (the reference computes none for this routing).
__global__ void __launch_bounds__(256) li_couple_out_kernel(WfDevFields F, WfLiCoupleView v, int balance) {
    double* const* Mf = F.Mf;
    double* const* RM = F.RM;
    const double dt = F.dt;
    const int64_t EL = F.land_slots, ER = F.river_slots;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < EL + ER;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (i >= EL) {
            const int64_t rs = i - EL;
            const int64_t r = F.river_node_of_slot[rs];
            if (r < 0) continue;
            RM[RV_H][rs] = v.h_river[r];
            RM[RV_STORAGE][rs] = v.storage_river[r];
            const int64_t e = v.out_ptr[r] < v.out_ptr[r + 1] ? v.out_edge[v.out_ptr[r]] : -1;
            RM[RV_Q][rs] = e >= 0 ? v.q[e] : 0.0;
            RM[RV_Q_AVG][rs] = e >= 0 ? v.q_avg[e] : 0.0;
            if (F.mass_balance && balance) {
                RM[BR_ERR][rs] = 0.0;
                RM[BR_REL][rs] = 0.0;
            }
            continue;
        }
        const int64_t s = i;
        const int64_t node = F.land_node_of_slot[s];
        if (node < 0) continue;
        Mf[OL_H][s] = v.h_land[node];
        Mf[OL_STORAGE][s] = v.storage[node];
        Mf[OL_Q][s] = 0.0;
        Mf[OL_Q_AVG][s] = 0.0;
        if (!F.mass_balance || !balance) continue;
        double tin = 0.0, tout = 0.0;
        auto add_in = [&](double q) {
            if (q > 0.0) tin += q;
            else tout -= q;
        };
        auto add_out = [&](double q) {
            if (q > 0.0) tout += q;
            else tin -= q;
        };
        add_in(v.qx_avg[v.ixd[node]]);
        add_in(v.qy_avg[v.iyd[node]]);
        add_in(v.runoff[node]);
        add_out(v.qx_avg[node]);
        add_out(v.qy_avg[node]);
        const int64_t k = v.river_index[node];
        if (k >= 0) {
            double q_src = 0.0, q_dst = 0.0;
            for (int64_t o = v.in_ptr[k]; o < v.in_ptr[k + 1]; ++o) q_src += v.q_avg[v.in_edge[o]];
            add_in(q_src);
            tin += jmax(0.0, v.ext[k]);
            for (int64_t o = v.out_ptr[k]; o < v.out_ptr[k + 1]; ++o) q_dst += v.q_avg[v.out_edge[o]];
            add_out(q_dst);
            tout += v.abstraction_cum[k] / dt + v.abstraction[k];
        }
        double err, rel;
        mb_error(tin, tout, (v.storage[node] - Mf[BO_PREV][s]) / dt, err, rel);
        Mf[BO_ERR][s] = err;
        Mf[BO_REL][s] = rel;
    }
}

// volumetric water content of one layer after a step (soil.jl:1320-1342)
template <int MAXN>
__global__ void vwc_kernel(WfDevFields F, int layer, double* out) {
    const int M = F.M;
    const int64_t E = F.land_slots * M;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t slot = e / M;
        if (F.land_node_of_slot[slot] < 0) continue;
        Column<MAXN> col;
        col.load_static(F, slot);
        col.set_thickness(F.Mf[ZI][e]);
        const int k = layer + 1;
        double v = NANV;
        if (k <= col.nl) {
            if (k <= col.nu) {
                v = (F.LY[LY_USLD][layer][e] + (col.act[layer] - col.thick[layer]) * (col.ts - col.tr)) / col.act[layer] +
                    col.tr;
            } else {
                v = col.ts;
            }
        }
        out[e] = v;
    }
}

int grid_for(int64_t n, int block, int num_sms) {
    int64_t b = (n + block - 1) / block;
    int64_t cap = (int64_t)num_sms * 16;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

template <class Phys>
cudaError_t launch_walk(const Phys& phys, const WfLaunchCfg& c) {
    const int threads = wave_threads(c);
    int blocks;
    Phys p = phys;
    p.sw.SL = p.sw.aflag ? 1 : wave_sub_lanes(p.sw.S, c);
    cudaError_t err = wave_grid(walk_kernel<Phys>, threads, 0, c, p.g, blocks, p.sw.prio_items,
                                wf_items_per_chunk(p.g.G, p.g.M, p.sw.SL));
    if (err != cudaSuccess) return err;
    walk_kernel<Phys><<<blocks, threads, 0, c.stream>>>(p);
    return cudaGetLastError();
}

}  // namespace

template <int PHASE>
cudaError_t launch_vertical(const WfDevFields& F, const WfLaunchCfg& c) {
    const int block = c.vertical_block > 0 ? c.vertical_block : 128;
    const int grid = grid_for(F.land_slots * F.M, block, c.num_sms);
    if (F.N <= 4)
        vertical_kernel<4, PHASE><<<grid, block, 0, c.stream>>>(F);
    else
        vertical_kernel<WF_MAX_LAYERS, PHASE><<<grid, block, 0, c.stream>>>(F);
    return cudaGetLastError();
}

cudaError_t wf_fp64_vertical(const WfDevFields& F, const WfLaunchCfg& c) { return launch_vertical<VERT_ALL>(F, c); }
cudaError_t wf_fp64_vertical_snow(const WfDevFields& F, const WfLaunchCfg& c) {
    return launch_vertical<VERT_SNOW>(F, c);
}
cudaError_t wf_fp64_vertical_soil(const WfDevFields& F, const WfLaunchCfg& c) {
    return launch_vertical<VERT_SOIL>(F, c);
}

cudaError_t wf_fp64_ssf(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, const WfLaunchCfg& c) {
    if (F.N <= 4) return launch_walk(SsfPhys<4>{F, g, sw}, c);
    return launch_walk(SsfPhys<WF_MAX_LAYERS>{F, g, sw}, c);
}

cudaError_t wf_snow_transport_sweep(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, int material,
                                    const WfLaunchCfg& c) {
    if (material == 0) return launch_walk(SnowPhys<0>{F, g, sw}, c);
    return launch_walk(SnowPhys<1>{F, g, sw}, c);
}

cudaError_t wf_snow_in(const WfDevFields& F, const WfDevGraph& g, const WfLaunchCfg& c) {
    snow_in_kernel<<<grid_for(F.land_slots * F.M, 256, c.num_sms), 256, 0, c.stream>>>(F, g);
    return cudaGetLastError();
}

cudaError_t wf_fp64_li_couple_in(const WfDevFields& F, const WfLiCoupleView& v, const WfLaunchCfg& c) {
    li_couple_in_kernel<<<grid_for(F.land_slots, 256, c.num_sms), 256, 0, c.stream>>>(F, v);
    return cudaGetLastError();
}
cudaError_t wf_fp64_li_couple_out(const WfDevFields& F, const WfLiCoupleView& v, int balance, const WfLaunchCfg& c) {
    li_couple_out_kernel<<<grid_for(F.land_slots + F.river_slots, 256, c.num_sms), 256, 0, c.stream>>>(F, v,
                                                                                                     balance);
    return cudaGetLastError();
}

namespace {

// Launch of a slim wavefront. Long chains (as many as half of the resident warps take) go first, each
// in a warp of its own; the lanes beyond a chain's sub-steps stay idle, because one lane's long solve
// (a drained cell that gets water again takes up to 75 iterations) holds up its whole warp. The other
// chains are packed as loosely as their number allows (wave_lanes).
template <class Phys, bool MULTI>
cudaError_t launch_wave64(const Phys& phys, const WfLaunchCfg& c) {
    const int threads = wave_threads(c);
    const size_t smem = wfz::walk_smem(threads);
    const WfDevGraph& g = phys.g;
    int SLr = g.lanes, SLs = SLr;
    if (MULTI) {
        const int cap = c.sub_lanes > 0 ? std::min(c.sub_lanes, 32) : 32;
        int need = 1;
        while (need < phys.sw.S && need < cap) need <<= 1;
        SLr = c.sub_lanes > 0 ? need : std::max(SLr, std::min(need, g.lanes_multi));
        SLs = SLr;
    }
    int per_sm = 0;
    const cudaError_t err =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wave64_kernel<Phys, MULTI>, threads, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    // One or two warps per scheduler: a scheduler issues one FP64 instruction per 64 cycles, which one warp
    // keeps busy, and more warps only slow the long chains down. River flow, whose positions are almost all
    // arithmetic: one (hourly, 301 x 301 cells: 5.25 ms with two, 4.72 with one; 700 x 700: 13.7 and 12.6);
    // the land sweeps, which wait more: two (daily overland flow of 200 x 200 cells: 3.22 and 3.50).
    const int fill = std::min(per_sm, Phys::kLand ? 2 : 1);
    int blocks = c.walk_blocks > 0 ? c.walk_blocks : c.num_sms * fill;
    const int wpb = threads / 32;
    const int64_t resident = (int64_t)std::min(blocks, c.num_sms * per_sm) * wpb;
    const int SLp = first_lanes(g, c);
    const int64_t p_chunks = first_chunks(g, SLp, resident);
    const int64_t items = p_chunks * wf_items_per_chunk(1, g.M, SLp) +
                          (g.n_chunks - p_chunks) * wf_items_per_chunk(g.G, g.M, SLr);
    const int64_t need = std::max<int64_t>((items + wpb - 1) / wpb, 1);
    if (blocks > need) blocks = (int)need;
    // batches of short chains only where there are more items than warps
    const int batch = (int)std::max<int64_t>(1, std::min<int64_t>(wfv::BATCH, items / (4 * resident)));
    wave64_kernel<Phys, MULTI><<<blocks, threads, smem, c.stream>>>(phys, p_chunks, SLp, SLs, SLr, batch);
    return cudaGetLastError();
}

template <int MAXN>
cudaError_t launch_ssf_wave(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, const WfLaunchCfg& c) {
    const int grid = grid_for(F.land_slots * F.M, 128, c.num_sms);
    ssf_prep64_kernel<MAXN><<<grid, 128, 0, c.stream>>>(F, sw);
    const cudaError_t err = launch_wave64<SsfWave64<MAXN>, false>(SsfWave64<MAXN>{F, g, sw}, c);
    if (err != cudaSuccess) return err;
    ssf_post64_kernel<MAXN><<<grid, 128, 0, c.stream>>>(F, g, sw);
    return cudaGetLastError();
}

template <bool LAND, bool CUM, bool RES, bool MULTI>
cudaError_t launch_kw(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, const WfLaunchCfg& c) {
    const int grid = grid_for((LAND ? F.land_slots : F.river_slots) * F.M, 128, c.num_sms);
    kw_prep64_kernel<LAND><<<grid, 128, 0, c.stream>>>(F, sw);
    const cudaError_t err = launch_wave64<KwWave64<LAND, CUM, RES>, MULTI>(KwWave64<LAND, CUM, RES>{F, g, sw}, c);
    if (err != cudaSuccess) return err;
    kw_post64_kernel<LAND, CUM><<<grid, 128, 0, c.stream>>>(F, g, sw);
    return cudaGetLastError();
}

}  // namespace

cudaError_t wf_fp64_ssf_wave(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, const WfLaunchCfg& c) {
    return F.N <= 4 ? launch_ssf_wave<4>(F, g, sw, c) : launch_ssf_wave<WF_MAX_LAYERS>(F, g, sw, c);
}

cudaError_t wf_fp64_overland(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, const WfLaunchCfg& c) {
    return sw.S > 1 ? launch_kw<true, true, false, true>(F, g, sw, c)
                    : launch_kw<true, false, false, false>(F, g, sw, c);
}

cudaError_t wf_fp64_river(const WfDevFields& F, const WfDevGraph& g, const WfSweep& sw, const WfLaunchCfg& c) {
    if (F.n_res > 0)
        return sw.S > 1 ? launch_kw<false, true, true, true>(F, g, sw, c)
                        : launch_kw<false, true, true, false>(F, g, sw, c);
    return sw.S > 1 ? launch_kw<false, true, false, true>(F, g, sw, c)
                    : launch_kw<false, false, false, false>(F, g, sw, c);
}

// ------------------------------------------------------------------ reservoirs -----------
// Kernels of both arithmetic forms (reservoir state is FP64 in both).

// A member field of the land layout as FP64 (double-FP32 pair in the split form).
__device__ __forceinline__ double land_member_d(const WfDevFields& F, int f, int64_t e) {
    return F.split ? (double)F.Mh[f][e] + (double)F.Ml[f][e] : F.Mf[f][e];
}

// Before the river sweep: storage at the start of the step for the water balance
// (mass_balance.jl:156-160), the inflow from the outlet cell's overland and subsurface flow
// (update_inflow!, surface_kinwave.jl:771-802; the overland part excludes what goes to the
// river, which the river's lateral inflow carries) and the reset of the step's cumulatives
// (set_reservoir_vars!, surface_kinwave.jl:227-237).
__global__ void __launch_bounds__(256) reservoir_prep_kernel(WfDevFields F) {
    const int M = F.M;
    const int64_t E = F.n_res * M;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / M;
        const int m = (int)(e - r * M);
        const int64_t le = F.res_land_slot[r] * M + m;
        double* const* RS = F.RS;
        if (F.mass_balance) RS[RS_PREV][e] = RS[RS_STORAGE][e];
        RS[RS_IN_OL][e] = land_member_d(F, OL_Q_AVG, le);
        RS[RS_IN_SSF][e] = land_member_d(F, SSF_Q_AVG, le);
        RS[RS_IN_CUM][e] = 0.0;
        RS[RS_OUT_CUM][e] = 0.0;
        RS[RS_DOWN_CUM][e] = 0.0;
        RS[RS_EVAP_CUM][e] = 0.0;
        RS[RS_ABS_CUM][e] = 0.0;
    }
}

// After the river sweep: step averages (average_reservoir_vars!, surface_kinwave.jl:244-258) and
// the reservoir water balance (compute_flow_balance!, mass_balance.jl:261-284).
__global__ void __launch_bounds__(256) reservoir_post_kernel(WfDevFields F) {
    const int M = F.M;
    const int64_t E = F.n_res * M;
    const double dt = F.dt;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / M;
        double* const* RS = F.RS;
        RS[RS_OUT_AVG][e] = RS[RS_OUT_CUM][e] / dt;
        RS[RS_IN_AVG][e] = RS[RS_IN_CUM][e] / dt;
        RS[RS_ABS_AVG][e] = RS[RS_ABS_CUM][e] / dt;
        if (!F.mass_balance) continue;
        RS[RS_EVAP_AVG][e] = RS[RS_EVAP_CUM][e] / dt;
        const double area = F.RP[RP_AREA][r];
        const double tin = RS[RS_IN_AVG][e] + RS[RS_PRECIP][e] * area;
        const double tout = RS[RS_OUT_AVG][e] + RS[RS_EVAP_AVG][e] * area;
        double err, rel;
        mb_error(tin, tout, (RS[RS_STORAGE][e] - RS[RS_PREV][e]) / dt, err, rel);
        RS[RS_ERR][e] = err;
        RS[RS_REL][e] = rel;
    }
}

cudaError_t wf_reservoir_prep(const WfDevFields& F, const WfLaunchCfg& c) {
    if (F.n_res <= 0) return cudaSuccess;
    reservoir_prep_kernel<<<grid_for(F.n_res * F.M, 256, c.num_sms), 256, 0, c.stream>>>(F);
    return cudaGetLastError();
}

cudaError_t wf_reservoir_post(const WfDevFields& F, const WfLaunchCfg& c) {
    if (F.n_res <= 0) return cudaSuccess;
    reservoir_post_kernel<<<grid_for(F.n_res * F.M, 256, c.num_sms), 256, 0, c.stream>>>(F);
    return cudaGetLastError();
}

cudaError_t wf_fp64_balance(const WfDevFields& F, const WfLaunchCfg& c) {
    const int block = 256;
    const int grid = grid_for((F.land_slots + F.river_slots) * F.M, block, c.num_sms);
    balance_kernel<<<grid, block, 0, c.stream>>>(F);
    return cudaGetLastError();
}

cudaError_t wf_fp64_vwc(const WfDevFields& F, int layer, double* out, const WfLaunchCfg& c) {
    const int block = 256;
    const int grid = grid_for(F.land_slots * F.M, block, c.num_sms);
    if (F.N <= 4)
        vwc_kernel<4><<<grid, block, 0, c.stream>>>(F, layer, out);
    else
        vwc_kernel<WF_MAX_LAYERS><<<grid, block, 0, c.stream>>>(F, layer, out);
    return cudaGetLastError();
}
