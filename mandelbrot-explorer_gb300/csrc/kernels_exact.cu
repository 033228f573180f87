// Exact-form CUDA passes of the perturbation renderer (compiled with
// -fmad=false so that every double operation below is the IEEE operation the
// reference executes, in the reference's order). Each kernel is persistent:
// every warp pulls its next samples from a global work counter (warp_take).
//
// Reference: cbotx/Mandelbrot-Explorer src/engine/mandel_perturbation.cpp
// ("mp.cpp"); the per-pixel semantics are those of its scalar loops.
#include "counts.cuh"
#include "direct_loop.cuh"
#include "kernels.h"
#include "orbit_color.h"
#include "smooth.cuh"

#include <type_traits>

namespace mbx {

static constexpr double kLn2 = 0x1.62e42fefa39efp-1; // log(2.0), correctly rounded

__device__ __forceinline__ int sample_index(const FrameGeom& g, const int* a) { // mp.cpp:4334-4340
    return (a[0] * g.sub + g.sub / 2 + a[2]) * g.W * g.sub + (a[1] * g.sub + g.sub / 2 + a[3]);
}

// Resolve list entry `i` of the pass to its {row, col, subrow, subcol}.
__device__ __forceinline__ void entry_key(const PixelSet& px, int i, int* a) { entry_coords(px, i, a); }

__device__ __forceinline__ bool cancelled(const DeviceFrame& f) { return f.cancel && *f.cancel; }

// The warp's next samples, taken together: the first of `lanes` consecutive
// entries (lane k takes entry + k), or -1 when the work is done or cancelled.
// Called by the warp's low `lanes` lanes, which so start every sample in step:
// lanes that fetch one by one drift apart for good and the warp then executes
// the loop once per drifted group (the 1e-300 frame's exact form cost twice as
// much per sample at 1920x1080, 35 samples a lane, as at 480x270, one a lane).
__device__ __forceinline__ int warp_take(const DeviceFrame& f, int n, int lanes) {
    const unsigned mask = lanes >= 32 ? 0xffffffffu : (1u << lanes) - 1u;
    __syncwarp(mask);
    int base = -1;
    // (plain read first: warps past the end leave without an atomic)
    if ((threadIdx.x & 31u) == 0 && !cancelled(f) && (int)*(volatile unsigned int*)&f.ctr->next < n) {
        base = (int)atomicAdd(&f.ctr->next, (unsigned)lanes);
        if (base >= n) base = -1;
    }
    return __shfl_sync(mask, base, 0);
}

__device__ __noinline__ double smooth_value(int n, double zrad) { return (double)n - log(log(zrad) / 2 / kLn2) / kLn2; }
// (float)smooth_value and the distance as a float: mostly without FP64 (smooth.cuh)
__device__ __forceinline__ float smooth_float(int n, double zrad) {
    float v;
    return smooth_pair(n, zrad, v) ? v : (float)smooth_value(n, zrad);
}
__device__ __noinline__ double distance_value(double zrad, double a, double b) { return sqrt(zrad) * log(zrad) / sqrt(a * a + b * b); }
__device__ __noinline__ float julia_distance(double zrad, double a, double b) {
    const double denom = sqrt((a * a) + (b * b));
    return denom > 0.0 ? (float)(sqrt(zrad) * log(zrad) / denom) : 0.0f;
}
__device__ __forceinline__ float distance_float(double zrad, double a, double b) {
    float v;
    return distance_pair(zrad, a, b, v) ? v : (float)distance_value(zrad, a, b);
}

// High words of a part's magnitude that settle a step's tests without FP64:
// from kFeNearWord (just above 1e-4) on, |z|^2 >= 1e-8; in [kFeWLo, kFeWHi)
// (just above 1e-8, 7e7) the larger part of w keeps |w|^2 within [1e-16, 1e16].
constexpr unsigned kFeNearWord = 0x3f1a36e3u, kFeWLo = 0x3e45798fu, kFeWHi = 0x4190b076u;

// ---------------------------------------------------------------------------
// Double path (mp.cpp:2290-2585, tryBLA mp.cpp:2714-2755).
// zmag2: |dz|^2
__device__ __forceinline__ int bla_try_fp64(const BlaView& b, const double2* Z, int s, double zmag2, double& dzr, double& dzi, double& ddr, double& ddi, double dcr, double dci, bool ede, double ESC2,
                                            int mx_ref_it) {
    int maxp = b.nlev - 1;
    int startp = (s == 1) ? maxp : __ffs(s - 1) - 1;
    if (startp > maxp) startp = maxp;
    if (startp < b.minlevel) return 0;
    for (int p = startp; p >= b.minlevel; --p) {
        int i = (s - 1) >> p;
        if (i >= b.size[p]) continue;
        const double r2 = b.r2[b.off[p] + i];
        if (!d_abs_less(zmag2, r2)) continue; // (r2 >= +0)
        int l = 1 << p;
        int land = s + l;
        if (land >= mx_ref_it - 1) continue;
        double4 bc = b.ab[b.off[p] + i];
        double nzr = bc.x * dzr - bc.y * dzi + bc.z * dcr - bc.w * dci;
        double nzi = bc.x * dzi + bc.y * dzr + bc.z * dci + bc.w * dcr;
        double2 zl = Z[land];
        double fr = zl.x + nzr, fi = zl.y + nzi;
        if (d_abs_less(ESC2, fr * fr + fi * fi)) return 0; // > ESC2
        if (ede) {
            double4 bd = b.ce[b.off[p] + i];
            double nddr = (bd.x * dzr - bd.y * dzi) + (bc.x * ddr - bc.y * ddi) + (bd.z * dcr - bd.w * dci);
            double nddi = (bd.x * dzi + bd.y * dzr) + (bc.x * ddi + bc.y * ddr) + (bd.z * dci + bd.w * dcr);
            ddr = nddr;
            ddi = nddi;
        }
        dzr = nzr;
        dzi = nzi;
        return l;
    }
    return 0;
}

// OC: the orbit colourings (orbit_color.h): their accumulators take every
// iteration's z; a trap turns BLA and the state-repetition detector off
// (mp.cpp:2121, 2388), a BLA skip restarts the stripe window (:2422-2427).
__device__ __forceinline__ void exact_counts(Counters* c, BlockCounts& s, unsigned long long n_steps, unsigned long long n_bla, unsigned long long n_skip, unsigned long long n_eff, unsigned n_int,
                                             unsigned n_fin, int lanes) {
    block_count(s, 0, n_steps, lanes);
    block_count(s, 1, n_bla, lanes);
    block_count(s, 2, n_skip, lanes);
    block_count(s, 3, n_eff, lanes);
    block_count(s, 4, n_int, lanes);
    block_count(s, 5, n_fin, lanes);
    __syncthreads();
    if (threadIdx.x == 0) {
        counts_flush(&c->steps, s.v[0]);
        counts_flush(&c->bla_applies, s.v[1]);
        counts_flush(&c->bla_skipped, s.v[2]);
        counts_flush(&c->effective_iters, s.v[3]);
        counts_flush(&c->interior, s.v[4]);
        counts_flush(&c->finished, s.v[5]);
    }
}

template <int OC>
__global__ void __launch_bounds__(128) k_fp64_pass(DeviceFrame f, Fp64Params p) {
    __shared__ BlockCounts s_counts;
    block_counts_init(s_counts);
    const FrameGeom& g = p.g;
    const double2* Z = f.orbit.Z;
    const double2* D = f.orbit.D;
    const CDivBy by_delta = c_div_by(p.sa_delta);
    const int bla_mask = (1 << f.bla.minlevel) - 1;
    const int tickets = (int)(((unsigned)f.px.n + 31u) >> 5);
    const bool spread = tickets <= p.spread_tickets;
    unsigned long long n_steps = 0, n_bla = 0, n_skip = 0, n_eff = 0;
    unsigned int n_int = 0, n_fin = 0;
    for (;;) {
        const int first = warp_take(f, f.px.n, 32);
        if (first < 0) break;
        const int i = spread ? spread_entry(first >> 5, (int)(threadIdx.x & 31u), tickets) : first + (int)(threadIdx.x & 31u);
        if (i >= f.px.n) continue;
        int arr[4];
        entry_key(f.px, i, arr);
        // Per-pixel dc (mp.cpp:2300-2315) from the host-built mpf spacing tables.
        int xpix = g.sub * (arr[1] - p.ref[1]) + (arr[3] - p.ref[3]);
        int ypix = g.sub * (arr[0] - p.ref[0]) + (arr[2] - p.ref[2]);
        C2 dc = c2(p.dcx[xpix + p.xoff], p.dcy[ypix + p.yoff]);
        if (p.per) dc = c2(dc.re - p.frac_re, dc.im - p.frac_im);
        // Series-approximation seed (mp.cpp:2317-2330).
        C2 dz = c2(0, 0), dd = c2(0, 0);
        for (int x = p.sa_order; x >= 0; --x) {
            dz = c_add(dz, p.A[x]);
            dz = c_mul(dz, dc);
            dz = c_div(dz, by_delta);
        }
        if (g.deriv) {
            for (int x = p.sa_order; x >= 0; --x) {
                dd = c_add(dd, p.B[x]);
                dd = c_mul(dd, dc);
                dd = c_div(dd, by_delta);
            }
        }
        int j = p.sa_it + 1;
        double dzr = dz.re, dzi = dz.im, dcr = dc.re, dci = dc.im, ddr = dd.re, ddi = dd.im;
        double tmp, zr = 0, zi = 0, zrad = 0;
        double q_r = dzr * dzr, q_i = dzi * dzi; // dz's squares, kept with it
        int k = j;
        const int per = p.per;
        int rk = k, rkm1 = k - 1;
        double zsr = 1e30, zsi = 1e30;
        int save_j = j, period_win = 1;
        int conf_P = 0, conf_next = 0, conf_count = 0, conf_giveup = 0;
        double conf_D2 = 0, conf_zr = 0, conf_zi = 0;
        const bool detect = p.use_interior != 0;
        const bool int_rep = p.int_rep && detect && !(OC & kOcTrap);
        OrbitColor<OC> oc;
        oc.init();
        double sdzr = 1e300, sdzi = 1e300;
        int sk = -1, save_j2 = j, twin2 = 1;
        int outcome = 0; // 0 running, 1 escaped, 2 interior, 3 glitch
        double edr = 0, edi = 0; // dz/dc at the escape
        double gscore = -1.0;
        int tick = 0;
        while (j < g.mxit) {
            if (((++tick) & 4095) == 0 && cancelled(f)) {
                outcome = 4;
                break;
            }
            if (int_rep) {
                if (k == sk && d_eq(dzr, sdzr) && d_eq(dzi, sdzi)) {
                    outcome = 2;
                    break;
                }
                if (j - save_j2 >= twin2) {
                    sdzr = dzr;
                    sdzi = dzi;
                    sk = k;
                    save_j2 = j;
                    twin2 += twin2;
                }
            }
            // (a BLA position: the orbit index less one a multiple of the least skip)
            const double q = rkm1 >= 1 && ((rkm1 - 1) & bla_mask) == 0 && f.bla.use && !(OC & kOcTrap) ? q_r + q_i : 1e300;
            if (d_abs_less(q, f.bla.rmax2)) {
                int skip = bla_try_fp64(f.bla, Z, rkm1, q, dzr, dzi, ddr, ddi, dcr, dci, g.deriv, g.ESC2, p.mx_ref_it);
                if (skip > 0) {
                    ++n_bla;
                    n_skip += skip;
                    k += skip;
                    j += skip;
                    rk += skip;
                    if (per && rk >= per) rk -= per;
                    rkm1 = (per && rk == 0) ? per - 1 : rk - 1;
                    q_r = dzr * dzr;
                    q_i = dzi * dzi;
                    oc.skipped();
                    zsr = 1e30;
                    zsi = 1e30;
                    save_j = j;
                    period_win = 1;
                    conf_P = 0;
                    conf_giveup = 0;
                    continue;
                }
            }
            ++n_steps;
            if (g.deriv) {
                if (k == 0) {
                    tmp = d_twice(dzr * (1 + ddr) - dzi * (1 + ddi));
                    ddi = d_twice(dzr * (1 + ddi) + dzi * (1 + ddr));
                } else {
                    double2 zk = Z[k - 1], dk = D[k - 1];
                    tmp = d_twice(ddr * zk.x - ddi * zk.y + dzr * (dk.x + ddr) - dzi * (dk.y + ddi));
                    ddi = d_twice(ddr * zk.y + ddi * zk.x + dzr * (dk.y + ddi) + dzi * (dk.x + ddr));
                }
                ddr = tmp;
            }
            const double m = d_twice(dzr * dzi);
            if (k == 0) {
                tmp = q_r - q_i + dcr;
                dzi = m + dci;
            } else {
                double2 zp = Z[rkm1];
                tmp = d_twice(dzr * zp.x - dzi * zp.y) + q_r - q_i + dcr;
                dzi = d_twice(dzr * zp.y + dzi * zp.x) + m + dci;
            }
            dzr = tmp;
            q_r = dzr * dzr;
            q_i = dzi * dzi;
            double2 zc = Z[rk];
            zr = dzr + zc.x;
            zi = dzi + zc.y;
            const int kd = k; // the derivative shadow's entry of this z
            oc.push(zr, zi);
            ++k;
            rkm1 = rk;
            if (per) {
                if (++rk == per) rk = 0;
            } else
                rk = k;
            // A common iteration, settled on high words: |z| below the bailout and
            // at least twice |dz|'s larger part (so |z|^2 is not below |dz|^2: no
            // rebase), the reference not at its end, no interior test due (as in
            // pixel_fe). 16 FP64 instructions; the tests below formed some 30.
            const unsigned hz = umax_(hi_abs(zr), hi_abs(zi));
            if (hz < p.esc_word && hz >= umax_(hi_abs(dzr), hi_abs(dzi)) + 0x00100000u && (per || k != p.mx_ref_it) &&
                (!detect || (conf_P <= 0 && ((j & 15) != 0 || conf_giveup >= 3 ||
                                             (hz >= kFeNearWord && j - save_j < period_win && umax_(hi_abs(zr - zsr), hi_abs(zi - zsi)) + 0x01b00000u >= hz &&
                                              d_abs_less(p.interior_eps2, 1e-17)))))) {
                ++j;
                continue;
            }
            zrad = zr * zr + zi * zi;
            double dr = 0, di = 0;
            if (g.deriv) {
                const double2 dk1 = D[kd];
                dr = ddr + dk1.x;
                di = ddi + dk1.y;
            }
            if (d_abs_less(g.ESC2, zrad)) { // zrad > ESC2
                edr = dr;
                edi = di;
                outcome = 1;
                break;
            }
            if (detect) {
                if (conf_P > 0) {
                    conf_D2 *= 4 * zrad;
                    if (conf_D2 > 1e18) conf_D2 = 1e18;
                    if (j >= conf_next) {
                        double pr = zr - conf_zr, pi = zi - conf_zi;
                        bool ret = (pr * pr + pi * pi < p.interior_eps2 * zrad);
                        if (ret && conf_D2 < 1.0) {
                            if (++conf_count >= p.interior_confirm) {
                                outcome = 2;
                                break;
                            }
                            conf_zr = zr;
                            conf_zi = zi;
                            conf_D2 = 1;
                            conf_next = j + conf_P;
                        } else {
                            conf_P = 0;
                            ++conf_giveup;
                        }
                    }
                } else if ((j & 15) == 0 && conf_giveup < 3) {
                    double pr = zr - zsr, pi = zi - zsi;
                    if (pr * pr + pi * pi < p.interior_eps2 * zrad) {
                        conf_P = j - save_j;
                        if (conf_P < 1) conf_P = 1;
                        conf_zr = zr;
                        conf_zi = zi;
                        conf_D2 = 1;
                        conf_next = j + conf_P;
                        conf_count = 0;
                    }
                    if (j - save_j >= period_win) {
                        zsr = zr;
                        zsi = zi;
                        save_j = j;
                        period_win += period_win;
                    }
                }
            }
            if (d_abs_less(zrad, q_r + q_i) || (!per && k == p.mx_ref_it)) {
                if ((q_r + q_i) / zrad > 10000000) {
                    gscore = zrad / f.orbit.zm3[per ? j % per : j];
                    outcome = 3;
                    break;
                }
                dzr = zr;
                dzi = zi;
                q_r = dzr * dzr;
                q_i = dzi * dzi;
                if (g.deriv) {
                    ddr = dr - 1;
                    ddi = di;
                }
                k = 0;
                rk = 0;
                rkm1 = per ? per - 1 : -1;
            }
            if (!per && k == p.mx_ref_it) {
                gscore = (double)zrad / f.orbit.zm3[j];
                outcome = 3;
                break;
            }
            ++j;
        }
        if (outcome == 4) continue; // cancelled
        if (outcome == 0 && j >= g.mxit) outcome = 2;
        const int idx = sample_index(g, arr);
        if (outcome == 1) {
            float v;
            if (g.ede) {
                v = (float)(sqrt(zrad) / g.dxf * log(zrad) / sqrt(edr * edr + edi * edi));
            } else {
                v = smooth_float(j + 1, zrad);
                if (g.normal) {
                    // normal angle arg(z) - arg(dz/dc) (mp.cpp:2489-2492)
                    if (f.out.normal) f.out.normal[idx] = (float)(atan2(zi, zr) - atan2(edi, edr));
                } else if (g.deovl) {
                    if (f.out.normal) f.out.normal[idx] = (float)(sqrt(zrad) / g.dxf * log(zrad) / sqrt(edr * edr + edi * edi));
                } else if (OC) { // trap, else stripe average (mp.cpp:2497-2500)
                    v = oc.escaped(smooth_value(j + 1, zrad), zrad, g.ER);
                }
            }
            f.out.iter[idx] = v;
            if (f.out.escN) f.out.escN[idx] = j + 1;
            f.out.done[i] = 1;
            ++n_fin;
            n_eff += (unsigned long long)(j + 1);
        } else if (outcome == 2) {
            f.out.iter[idx] = oc.interior();
            if (f.out.escN) f.out.escN[idx] = -1;
            f.out.done[i] = 1;
            ++n_fin;
            n_eff += (unsigned long long)g.mxit;
            ++n_int;
        } else {
            f.out.glitch[i] = gscore;
            if (gscore >= 0 && gscore < 1e100) atomicMin(&f.ctr->glitch_min_bits, (unsigned long long)__double_as_longlong(gscore));
        }
    }
    exact_counts(f.ctr, s_counts, n_steps, n_bla, n_skip, n_eff, n_int, n_fin, 32);
}

// ---------------------------------------------------------------------------
// Floatexp path helpers (mp.cpp:2770-2970).
__device__ void bla_rerescale_underflow(FE& S, double& wr, double& wi, double nwr, double nwi) { // mp.cpp:2770-2781
    if (nwr == 0.0 && nwi == 0.0) {
        S = fe_make(1.0, 0);
        wr = wi = 0.0;
        return;
    }
    FE wmag = fe_sqrt(fe_add(fe_mul(fe_from(nwr), fe_from(nwr)), fe_mul(fe_from(nwi), fe_from(nwi))));
    S = fe_mul(S, wmag);
    double inv = 1.0 / fe_to_double(wmag);
    wr = nwr * inv;
    wi = nwi * inv;
}

__device__ void fe_step_underflow(FE Xr, FE Xi, FE dcr, FE dci, FE& S, double& wr, double& wi) { // mp.cpp:2794-2835
    const double sm = S.m, sm2 = sm * sm;
    const int64_t se = S.e;
    const int64_t NONE = (int64_t)0x8000000000000000ll;
    int64_t e = NONE;
    const bool has_w = wr != 0.0 || wi != 0.0;
    if (has_w && Xr.m != 0.0) e = max(e, Xr.e + se);
    if (has_w && Xi.m != 0.0) e = max(e, Xi.e + se);
    if (has_w) e = max(e, se + se);
    if (dcr.m != 0.0) e = max(e, dcr.e);
    if (dci.m != 0.0) e = max(e, dci.e);
    if (e == NONE) {
        S = fe_make(1.0, 0);
        wr = wi = 0.0;
        return;
    }
    auto align = [e](double m, int64_t te) -> double {
        int64_t d = te - e;
        if (m == 0.0 || d < -54) return 0.0;
        return m * pow2i((int)d);
    };
    const double xs_r = align(Xr.m * sm, Xr.e + se);
    const double xs_i = align(Xi.m * sm, Xi.e + se);
    const double s2 = align(sm2, se + se);
    const double cr = align(dcr.m, dcr.e);
    const double ci = align(dci.m, dci.e);
    const double nr = 2.0 * (xs_r * wr - xs_i * wi) + s2 * (wr * wr - wi * wi) + cr;
    const double ni = 2.0 * (xs_r * wi + xs_i * wr) + 2.0 * s2 * wr * wi + ci;
    const double mag2 = nr * nr + ni * ni;
    const double mag = mag2 > 0.0 ? sqrt(mag2) : hypot(nr, ni);
    if (mag == 0.0) {
        S = fe_make(1.0, 0);
        wr = wi = 0.0;
        return;
    }
    S = fe_renorm(mag, e);
    wr = nr / mag;
    wi = ni / mag;
}

__device__ void fe_deriv_underflow(FE zr, FE zi, FE& SJ, double& jr, double& ji, double& invSJd) { // mp.cpp:2842-2876
    double im = 0.5 / SJ.m;
    int64_t ie = 1 - SJ.e;
    if (im >= 1.0) {
        im *= 0.5;
        ++ie;
    }
    FE invSJ = fe_make(im, ie);
    int64_t e = invSJ.e;
    if (zr.m != 0.0) e = max(e, zr.e);
    if (zi.m != 0.0) e = max(e, zi.e);
    auto align = [e](FE x) -> double {
        if (x.m == 0.0) return 0.0;
        int64_t d = x.e - e;
        if (d < -54) return 0.0;
        return x.m * pow2i((int)d);
    };
    double azr = align(zr), azi = align(zi);
    double ar = 2.0 * (azr * jr - azi * ji) + align(invSJ);
    double ai = 2.0 * (azr * ji + azi * jr);
    double mag = sqrt(ar * ar + ai * ai);
    if (mag == 0.0) {
        SJ = fe_make(1.0, 0);
        jr = ji = 0.0;
        invSJd = 1.0;
        return;
    }
    SJ = fe_mul(SJ, fe_renorm(mag, e));
    jr = ar / mag;
    ji = ai / mag;
    invSJd = 1.0 / fe_to_double(SJ);
}

// tryBLAfe (mp.cpp:2883-2970).
__device__ int bla_try_fe(const BlaView& b, const double2* Z, bool periodic, int s, FE& S, FE S2, double& wr, double& wi, double dr, double di, double ESC2, int mx_ref_it, double* ab) {
    if (s < 1 || b.nlev == 0) return 0;
    int maxp = b.nlev - 1;
    int startp = (s == 1) ? maxp : __ffs(s - 1) - 1;
    if (startp > maxp) startp = maxp;
    if (startp < b.minlevel) return 0;
    if (d_le_zero(b.rmax2)) return 0;
    const FE rmax = fe_from(b.rmax2);
    {
        // |w|^2 >= (the larger part)^2 >= 2^(2 k), k its binade, so |dz|^2's
        // exponent is at least S2.e + 2 k: above rmax2's, no radius holds
        const unsigned h = umax_(hi_abs(wr), hi_abs(wi));
        const int64_t lo = S2.e + 2 * ((int)(h >> 20) - 1023);
        if (h >= 0x20000000u && h < 0x5fe00000u && !d_is_zero(S2.m) && lo > rmax.e) return 0;
    }
    const FE dz2 = fe_mul(S2, fe_from(wr * wr + wi * wi));
    if (!fe_abs_less(dz2, rmax)) return 0;
    for (int p = startp; p >= b.minlevel; --p) {
        int i = (s - 1) >> p;
        if (i >= b.size[p]) continue;
        const double r2 = b.r2[b.off[p] + i];
        // |dz|^2 < r2, on exponents and mantissa bits (r2 normal) or in floatexp
        const uint64_t rb = dbits(r2);
        const int re = (int)(rb >> 52) - 1022;
        if ((int64_t)rb > 0 && d_normal(rb) ? !(dz2.e < re || (dz2.e == re && (dbits(dz2.m) & 0xfffffffffffffull) < (rb & 0xfffffffffffffull))) && !d_is_zero(dz2.m)
                                            : d_le_zero(r2) || !fe_abs_less(dz2, fe_from(r2)))
            continue;
        int l = 1 << p;
        int land = s + l;
        if (land >= mx_ref_it - 1) continue;
        double4 bc = b.ab[b.off[p] + i];
        double nwr = (bc.x * wr - bc.y * wi) + (bc.z * dr - bc.w * di);
        double nwi = (bc.x * wi + bc.y * wr) + (bc.z * di + bc.w * dr);
        const double BIG = 1e150;
        double2 zl = Z[land];
        if (d_abs_less(nwr, BIG) && d_abs_less(nwi, BIG)) { // (finite, below 1e150)
            // z = Z_land + S n: with each part of Z_land and of S n below 4, |z|^2
            // is below 128, so only a bailout^2 below that needs z itself
            const unsigned hn = umax_(hi_abs(nwr), hi_abs(nwi));
            if (!(umax_(hi_abs(zl.x), hi_abs(zl.y)) < 0x40100000u && (int)(hn >> 20) - 1022 + S.e <= 2 && d_abs_less(200.0, ESC2))) {
                double fr = zl.x + fe_to_double(fe_mul_d(S, nwr));
                double fi = zl.y + fe_to_double(fe_mul_d(S, nwi));
                if (d_abs_less(ESC2, fr * fr + fi * fi)) return 0; // > ESC2
            }
            double wm2 = nwr * nwr + nwi * nwi;
            if (d_is_zero(wm2)) {
                if (periodic)
                    bla_rerescale_underflow(S, wr, wi, nwr, nwi);
                else
                    return 0;
            } else {
                double wmag = int_sqrt(wm2);
                S = fe_mul(S, fe_from(wmag));
                double inv = int_div(1.0, wmag);
                wr = nwr * inv;
                wi = nwi * inv;
            }
        } else {
            FE dzr = fe_mul_d(S, wr), dzi = fe_mul_d(S, wi);
            FE dcrfe = fe_mul_d(S, dr), dcife = fe_mul_d(S, di);
            FE nzr = fe_add(fe_sub(fe_mul_d(dzr, bc.x), fe_mul_d(dzi, bc.y)), fe_sub(fe_mul_d(dcrfe, bc.z), fe_mul_d(dcife, bc.w)));
            FE nzi = fe_add(fe_add(fe_mul_d(dzr, bc.y), fe_mul_d(dzi, bc.x)), fe_add(fe_mul_d(dcrfe, bc.w), fe_mul_d(dcife, bc.z)));
            double fr = zl.x + fe_to_double(nzr), fi = zl.y + fe_to_double(nzi);
            if (fr * fr + fi * fi > ESC2) return 0;
            FE Snew = fe_sqrt<true>(fe_add(fe_mul(nzr, nzr), fe_mul(nzi, nzi)));
            if (Snew.m == 0.0) {
                S = fe_make(1.0, 0);
                wr = wi = 0.0;
            } else {
                S = Snew;
                wr = fe_to_double(fe_div<true>(nzr, S));
                wi = fe_to_double(fe_div<true>(nzi, S));
            }
        }
        if (ab) {
            ab[0] = bc.x;
            ab[1] = bc.y;
            ab[2] = bc.z;
            ab[3] = bc.w;
        }
        return l;
    }
    return 0;
}

struct PixOut {
    float value; // (interior samples, and the orbit colourings' escapes)
    float nrm;
    int n;
    int state; // 1 escaped, 2 interior, 4 cancelled
    // at the escape, for the value (fe_escape_value: formed after the loop, by the
    // warp's samples together)
    double zrad, zr, zi, jr, ji;
    FE SJ;
};

// The plain delta step of pixelRescaled in the fused form, w' = (2 X + s w) w + d,
// with the products sw = s w of the current state.
// On GB300 each FP64 instruction holds its SM quarter's FP64 unit for 64
// cycles, independent operands or not, so the exact form's loops are bound by
// their count of FP64 instructions (compares included), while about thirty
// integer ones fit beside each. A common step therefore forms only what the
// next state needs: the doubling X + X (exact) on the bit pattern, the step,
// s w' once (for z now and for the next step), and z: 14 FP64 instructions. The
// tests of a step are made on high words, exact tests on the bit patterns
// (floatexp.h d_is_zero, d_abs_less, d_eq) only where those leave them open.
__device__ __forceinline__ void fe_plain_step(double Xr, double Xi, double swr, double swi, double wr, double wi, double dr, double di, double& nwr, double& nwi) {
    const double fR = d_twice(Xr) + swr;
    const double fI = d_twice(Xi) + swi;
    nwr = fR * wr - fI * wi + dr;
    nwi = fR * wi + fI * wr + di;
}
// |x| < 2^-1056 (the subnormal 2^18 * 2^-1074): the step's underflow test, on
// the bit pattern
__device__ __forceinline__ bool below_step_floor(double x) { return (dbits(x) & 0x7fffffffffffffffull) < 0x40000ull; }

// pixelRescaled (mp.cpp:3287-3618), smooth / EDE / DE-overlay.
// OC: the orbit colourings, as in k_fp64_pass (mp.cpp:3338-3346, 3389-3397,
// 3503-3504, 3524-3529); a trap turns BLA off.
template <int OC>
__device__ PixOut pixel_fe(const DeviceFrame& f, const FeParams& p, FE dcr, FE dci, unsigned long long& n_steps, unsigned long long& n_bla, unsigned long long& n_skip) {
    const FrameGeom& g = p.g;
    const double2* Z = f.orbit.Z;
    const FE2* Zfe = f.orbit.Zfe;
    const int reflen = p.mx_ref_it + 1;
    const int per = p.per;
    int rm = 0;
    FE S = fe_sqrt<true>(fe_add(fe_mul(dcr, dcr), fe_mul(dci, dci)));
    double wr, wi, dr, di;
    if (d_is_zero(S.m)) {
        S = fe_make(1.0, 0);
        wr = wi = dr = di = 0.0;
    } else {
        wr = fe_to_double(fe_div<true>(dcr, S));
        wi = fe_to_double(fe_div<true>(dci, S));
        dr = wr;
        di = wi;
    }
    double s = fe_to_double(S);
    FE S2 = fe_mul(S, S);
    double swr = s * wr, swi = s * wi; // kept with s and w
    int m = 1, iter = 1;
    double zsr = 1e30, zsi = 1e30;
    int save_iter = 1, period_win = 1;
    int conf_P = 0, conf_next = 0, conf_count = 0, conf_giveup = 0;
    double conf_D2 = 0, conf_zr = 0, conf_zi = 0;
    const bool deriv = g.deriv != 0;
    FE SJ = fe_make(1.0, 0);
    double jr = 1.0, ji = 0.0, invSJd = 1.0;
    const bool detect = p.use_interior != 0;
    const bool int_rep = p.int_rep && detect && !(OC & kOcTrap);
    OrbitColor<OC> oc;
    oc.init();
    double rwr = 1e300, rwi = 1e300;
    FE sS = fe_make(1e300, 0);
    int sm = -1, save_iter2 = 1, twin2r = 1;
    PixOut o;
    o.nrm = 0.0f;
    o.n = -1;
    int tick = 0;
    while (iter < g.mxit) {
        if (((++tick) & 4095) == 0 && cancelled(f)) {
            o.state = 4;
            return o;
        }
        if (int_rep) {
            if (m == sm && d_eq(wr, rwr) && d_eq(wi, rwi) && d_eq(S.m, sS.m) && S.e == sS.e) {
                o.value = -2.0f;
                o.state = 2;
                return o;
            }
            if (iter - save_iter2 >= twin2r) {
                rwr = wr;
                rwi = wi;
                sS = S;
                sm = m;
                save_iter2 = iter;
                twin2r += twin2r;
            }
        }
        if (f.bla.use && !(OC & kOcTrap) && m >= 2) {
            double ab[4];
            int skip = bla_try_fe(f.bla, Z, p.ref_period_gt0, rm, S, S2, wr, wi, dr, di, g.ESC2, per ? per : reflen, deriv ? ab : nullptr);
            if (skip > 0) {
                ++n_bla;
                n_skip += skip;
                oc.skipped();
                if (deriv) {
                    FE Jr = fe_mul_d(SJ, jr), Ji = fe_mul_d(SJ, ji);
                    FE nJr = fe_add(fe_sub(fe_mul_d(Jr, ab[0]), fe_mul_d(Ji, ab[1])), fe_from(ab[2]));
                    FE nJi = fe_add(fe_add(fe_mul_d(Jr, ab[1]), fe_mul_d(Ji, ab[0])), fe_from(ab[3]));
                    SJ = fe_sqrt<true>(fe_add(fe_mul(nJr, nJr), fe_mul(nJi, nJi)));
                    if (d_is_zero(SJ.m)) {
                        SJ = fe_make(1.0, 0);
                        jr = ji = 0.0;
                        invSJd = 1.0;
                    } else {
                        jr = fe_to_double(fe_div<true>(nJr, SJ));
                        ji = fe_to_double(fe_div<true>(nJi, SJ));
                        invSJd = int_div(1.0, fe_to_double(SJ));
                    }
                }
                m += skip;
                iter += skip;
                rm += skip;
                if (per && rm >= per) rm -= per;
                s = fe_to_double(S);
                S2 = fe_mul(S, S);
                dr = fe_to_double(fe_div<true>(dcr, S));
                di = fe_to_double(fe_div<true>(dci, S));
                swr = s * wr;
                swi = s * wi;
                zsr = 1e30;
                zsi = 1e30;
                save_iter = iter;
                period_win = 1;
                conf_P = 0;
                conf_giveup = 0;
                continue;
            }
        }
        ++n_steps;
        double2 X = m ? Z[rm] : make_double2(0.0, 0.0);
        double Xr = X.x, Xi = X.y;
        // the pre-step z (DE colourings only)
        double zmr = 0.0, zmi = 0.0;
        bool deriv_underflow = false;
        if (deriv) {
            zmr = Xr + swr;
            zmi = Xi + swi;
            deriv_underflow = d_is_zero(zmr) && d_is_zero(zmi) && d_is_zero(invSJd);
        }
        FE zmrfe = fe_make(0, 0), zmife = fe_make(0, 0);
        if (deriv_underflow) {
            FE Xrfe = m ? Zfe[rm].re : fe_make(0.0, 0);
            FE Xife = m ? Zfe[rm].im : fe_make(0.0, 0);
            zmrfe = fe_add(Xrfe, fe_mul_d(S, wr));
            zmife = fe_add(Xife, fe_mul_d(S, wi));
        }
        double nwr, nwi;
        fe_plain_step(Xr, Xi, swr, swi, wr, wi, dr, di, nwr, nwi);
        const bool step_underflow = below_step_floor(nwr) && below_step_floor(nwi);
        if (step_underflow && !(d_is_zero(nwr) && d_is_zero(nwi) && d_is_zero(wr) && d_is_zero(wi) && d_is_zero(dcr.m) && d_is_zero(dci.m))) {
            FE Xrfe = m ? Zfe[rm].re : fe_make(0.0, 0);
            FE Xife = m ? Zfe[rm].im : fe_make(0.0, 0);
            fe_step_underflow(Xrfe, Xife, dcr, dci, S, wr, wi);
            s = fe_to_double(S);
            S2 = fe_mul(S, S);
            dr = fe_to_double(fe_div<true>(dcr, S));
            di = fe_to_double(fe_div<true>(dci, S));
        } else {
            wr = nwr;
            wi = nwi;
        }
        ++m;
        ++iter;
        rm++;
        if (per && rm == per) rm = 0;
        if (deriv) {
            if (deriv_underflow) {
                fe_deriv_underflow(zmrfe, zmife, SJ, jr, ji, invSJd);
            } else {
                double a = d_twice(zmr * jr - zmi * ji) + invSJd;
                double b = d_twice(zmr * ji + zmi * jr);
                jr = a;
                ji = b;
                const unsigned hj = umax_(hi_abs(jr), hi_abs(ji));
                double jm2 = 1.0;
                if (hj < kFeWLo || hj >= kFeWHi) jm2 = jr * jr + ji * ji;
                if (d_abs_less(1e16, jm2) || (d_abs_less(jm2, 1e-16) && !d_is_zero(jm2))) {
                    FE jmag = fe_sqrt<true>(fe_from(jm2));
                    SJ = fe_mul(SJ, jmag);
                    double inv = int_div(1.0, fe_to_double(jmag));
                    jr *= inv;
                    ji *= inv;
                    invSJd = int_div(1.0, fe_to_double(SJ));
                }
            }
        }
        X = m ? Z[rm] : make_double2(0.0, 0.0);
        Xr = X.x;
        Xi = X.y;
        swr = s * wr;
        swi = s * wi;
        const double zr = Xr + swr, zi = Xi + swi;
        oc.push(zr, zi);
        // A common iteration: |z| between 1e-4 and the bailout and at least twice
        // |dz|'s larger part (|z|^2 >= 4 max^2 > |dz|^2: no rebase), |w| in its
        // window, the reference not at its end, and no interior test due.
        const unsigned hz = umax_(hi_abs(zr), hi_abs(zi)), hw = umax_(hi_abs(wr), hi_abs(wi)), hs = umax_(hi_abs(swr), hi_abs(swi));
        if (hz >= kFeNearWord && hz < p.esc_word && hz >= hs + 0x00100000u && hw >= kFeWLo && hw < kFeWHi && (per || m < reflen)) {
            if (!detect) continue;
            if (conf_P <= 0) {
                if ((iter & 15) != 0 || conf_giveup >= 3) continue;
                // z against the saved one: with a part 2^-27 of |z|'s larger part
                // apart, |z - zs|^2 >= 5.5e-17 max^2 > 9e-18 2 max^2
                if (iter - save_iter < period_win && umax_(hi_abs(zr - zsr), hi_abs(zi - zsi)) + 0x01b00000u >= hz && d_abs_less(p.interior_eps2, 1e-17)) continue;
            }
        }
        double zrad = zr * zr + zi * zi;
        const double wmag2 = wr * wr + wi * wi;
        bool keep = true;
        if (d_abs_less(g.ESC2, zrad)) { // zrad > ESC2
            o.n = iter;
            o.state = 1;
            o.zrad = zrad;
            o.zr = zr;
            o.zi = zi;
            o.jr = jr;
            o.ji = ji;
            o.SJ = SJ;
            if (OC && !g.ede && !g.normal && !g.deovl) // trap, else stripe average
                o.value = oc.escaped((double)iter - log(log(zrad) / 2.0 / kLn2) / kLn2, zrad, g.ER);
            return o;
        }
        if (detect) {
            if (conf_P > 0) {
                conf_D2 *= 4.0 * zrad;
                if (d_abs_less(1e18, conf_D2)) conf_D2 = 1e18; // conf_D2 >= +0 or NaN
                if (iter >= conf_next) {
                    double pr = zr - conf_zr, pi = zi - conf_zi;
                    if (d_abs_less(pr * pr + pi * pi, p.interior_eps2 * zrad) && d_abs_less(conf_D2, 1.0)) {
                        if (++conf_count >= p.interior_confirm) {
                            o.value = oc.interior();
                            o.state = 2;
                            return o;
                        }
                        conf_zr = zr;
                        conf_zi = zi;
                        conf_D2 = 1;
                        conf_next = iter + conf_P;
                    } else {
                        conf_P = 0;
                        ++conf_giveup;
                    }
                }
            } else if ((iter & 15) == 0 && conf_giveup < 3) {
                double pr = zr - zsr, pi = zi - zsi;
                if (d_abs_less(pr * pr + pi * pi, p.interior_eps2 * zrad)) {
                    conf_P = iter - save_iter;
                    if (conf_P < 1) conf_P = 1;
                    conf_zr = zr;
                    conf_zi = zi;
                    conf_D2 = 1;
                    conf_next = iter + conf_P;
                    conf_count = 0;
                }
                if (iter - save_iter >= period_win) {
                    zsr = zr;
                    zsi = zi;
                    save_iter = iter;
                    period_win += period_win;
                }
            }
        }
        // |w|^2 > 1e16, or 0 < |w|^2 < 1e-16 (|w|^2 >= +0 or NaN)
        if (d_abs_less(1e16, wmag2) || (d_abs_less(wmag2, 1e-16) && !d_is_zero(wmag2))) {
            FE wmag = fe_sqrt<true>(fe_from(wmag2));
            S = fe_mul(S, wmag);
            s = fe_to_double(S);
            S2 = fe_mul(S, S);
            double inv = int_div(1.0, fe_to_double(wmag));
            wr *= inv;
            wi *= inv;
            dr = fe_to_double(fe_div<true>(dcr, S));
            di = fe_to_double(fe_div<true>(dci, S));
            keep = false;
        }
        double dzmag2 = s * s * (keep ? wmag2 : wr * wr + wi * wi);
        if (d_abs_less(zrad, 1e-8) || d_abs_less(zrad, dzmag2) || (!per && m >= reflen)) { // zrad, dzmag2 >= +0 or NaN
            FE Xmr = m ? Zfe[rm].re : fe_make(0.0, 0);
            FE Xmi = m ? Zfe[rm].im : fe_make(0.0, 0);
            FE Swr = fe_mul_d(S, wr), Swi = fe_mul_d(S, wi);
            FE zrfe = fe_add(Xmr, Swr), zife = fe_add(Xmi, Swi);
            FE zradfe = fe_add(fe_mul(zrfe, zrfe), fe_mul(zife, zife));
            FE dzfe = fe_add(fe_mul(Swr, Swr), fe_mul(Swi, Swi));
            if ((!per && m >= reflen) || fe_abs_less(zradfe, dzfe)) {
                FE Snew = fe_sqrt<true>(zradfe);
                if (d_is_zero(Snew.m)) {
                    wr = wi = 0.0;
                } else {
                    S = Snew;
                    s = fe_to_double(S);
                    S2 = fe_mul(S, S);
                    wr = fe_to_double(fe_div<true>(zrfe, S));
                    wi = fe_to_double(fe_div<true>(zife, S));
                    dr = fe_to_double(fe_div<true>(dcr, S));
                    di = fe_to_double(fe_div<true>(dci, S));
                }
                m = 0;
                rm = -1;
                keep = false;
            }
        }
        if (!keep) {
            swr = s * wr;
            swi = s * wi;
        }
    }
    o.value = oc.interior();
    o.state = 2;
    return o;
}

// solveRescaledSimd8NoBla semantics for one lane (mp.cpp:3620-3816).
__device__ PixOut pixel_fe_nobla(const DeviceFrame& f, const FeParams& p, FE dcr, FE dci, unsigned long long& n_steps) {
    const FrameGeom& g = p.g;
    const double2* Z = f.orbit.Z;
    const FE2* Zfe = f.orbit.Zfe;
    const int mx_ref_it = p.mx_ref_it;
    const int referenceLength = mx_ref_it + 1;
    double wr = 0, wi = 0, sd, dr = 0, di = 0;
    FE scale;
    const FE s0 = fe_sqrt(fe_add(fe_mul(dcr, dcr), fe_mul(dci, dci)));
    if (s0.m == 0.0) {
        scale = fe_make(1.0, 0);
    } else {
        scale = s0;
        wr = fe_to_double(fe_div(dcr, s0));
        wi = fe_to_double(fe_div(dci, s0));
        dr = wr;
        di = wi;
    }
    sd = fe_to_double(scale);
    int index = 1, iteration = 1;
    PixOut o;
    o.nrm = 0.0f;
    o.n = -1;
    int tick = 0;
    for (;;) {
        if (iteration >= g.mxit) {
            o.value = -2.0f;
            o.state = 2;
            return o;
        }
        if (((++tick) & 4095) == 0 && cancelled(f)) {
            o.state = 4;
            return o;
        }
        ++n_steps;
        double pr = 0, pi = 0;
        if (index > 0) {
            double2 zp = Z[index - 1];
            pr = zp.x;
            pi = zp.y;
        }
        const int current = index > mx_ref_it ? mx_ref_it : index;
        double2 zc = Z[current];
        double nwr, nwi;
        const double fR = (pr + pr) + (sd * wr);
        const double fI = (pi + pi) + (sd * wi);
        nwr = ((fR * wr) - (fI * wi)) + dr;
        nwi = ((fR * wi) + (fI * wr)) + di;
        const double aR = zc.x + (sd * nwr), aI = zc.y + (sd * nwi);
        double actual = (aR * aR) + (aI * aI);
        double delta = (nwr * nwr) + (nwi * nwi);
        if (delta == 0.0 && (nwr != 0.0 || nwi != 0.0 || wr != 0.0 || wi != 0.0 || dcr.m != 0.0 || dci.m != 0.0)) {
            const FE rR = index ? Zfe[index - 1].re : fe_make(0.0, 0);
            const FE rI = index ? Zfe[index - 1].im : fe_make(0.0, 0);
            fe_step_underflow(rR, rI, dcr, dci, scale, wr, wi);
            sd = fe_to_double(scale);
            dr = fe_to_double(fe_div(dcr, scale));
            di = fe_to_double(fe_div(dci, scale));
            const FE ar = fe_add(Zfe[current].re, fe_mul_d(scale, wr));
            const FE ai = fe_add(Zfe[current].im, fe_mul_d(scale, wi));
            actual = fe_to_double(fe_add(fe_mul(ar, ar), fe_mul(ai, ai)));
            delta = wr * wr + wi * wi;
        } else {
            wr = nwr;
            wi = nwi;
        }
        ++index;
        ++iteration;
        if (actual > g.ESC2) {
            o.n = iteration;
            o.state = 1;
            o.zrad = actual;
            return o;
        }
        if (delta > 1e16 || (delta < 1e-16 && delta > 0.0)) {
            const FE nm = fe_sqrt(fe_from(delta));
            scale = fe_mul(scale, nm);
            sd = fe_to_double(scale);
            const double inverse = 1.0 / fe_to_double(nm);
            wr *= inverse;
            wi *= inverse;
            dr = fe_to_double(fe_div(dcr, scale));
            di = fe_to_double(fe_div(dci, scale));
        }
        const double absd = sd * sd * (wr * wr + wi * wi);
        if (actual < 1e-8 || actual < absd || index >= referenceLength) {
            const FE rR = index ? Zfe[index - 1].re : fe_make(0.0, 0);
            const FE rI = index ? Zfe[index - 1].im : fe_make(0.0, 0);
            const FE sR = fe_mul_d(scale, wr), sI = fe_mul_d(scale, wi);
            const FE aRf = fe_add(rR, sR), aIf = fe_add(rI, sI);
            const FE a2 = fe_add(fe_mul(aRf, aRf), fe_mul(aIf, aIf));
            const FE d2 = fe_add(fe_mul(sR, sR), fe_mul(sI, sI));
            if (index >= referenceLength || fe_abs_less(a2, d2)) {
                const FE ns = fe_sqrt(a2);
                if (ns.m == 0.0) {
                    wr = wi = 0.0;
                } else {
                    scale = ns;
                    sd = fe_to_double(ns);
                    wr = fe_to_double(fe_div(aRf, ns));
                    wi = fe_to_double(fe_div(aIf, ns));
                    dr = fe_to_double(fe_div(dcr, ns));
                    di = fe_to_double(fe_div(dci, ns));
                }
                index = 0;
            }
        }
    }
}

// The escaped sample's value, and its normal angle or overlay distance
// (mp.cpp:3498-3529).
__device__ __noinline__ float fe_distance(FE dxfe, double zrad, FE SJ, double jr, double ji) {
    const double num = sqrt(zrad) * log(zrad);
    const FE Jmag = fe_mul_d(SJ, sqrt(jr * jr + ji * ji));
    return (float)fe_to_double(fe_div(fe_from(num), fe_mul(dxfe, Jmag)));
}
__device__ __forceinline__ void fe_escape_value(const FeParams& p, PixOut& o) {
    const FrameGeom& g = p.g;
    if (g.ede) {
        o.value = fe_distance(p.dxfe, o.zrad, o.SJ, o.jr, o.ji);
        return;
    }
    if (g.normal) // normal angle arg(z) - arg(J); SJ > 0 (mp.cpp:3512-3515)
        o.nrm = (float)(atan2(o.zi, o.zr) - atan2(o.ji, o.jr));
    else if (g.deovl)
        o.nrm = fe_distance(p.dxfe, o.zrad, o.SJ, o.jr, o.ji);
    o.value = smooth_float(o.n, o.zrad);
}

template <int OC>
__global__ void __launch_bounds__(128) k_fe_pass(DeviceFrame f, FeParams p) {
    __shared__ BlockCounts s_counts;
    block_counts_init(s_counts);
    if (p.lanes_per_warp && (int)(threadIdx.x & 31u) >= p.lanes_per_warp) return;
    const FrameGeom& g = p.g;
    unsigned long long n_steps = 0, n_bla = 0, n_skip = 0, n_eff = 0;
    unsigned int n_int = 0, n_fin = 0;
    const int n = f.px.n_dev ? min((int)*f.px.n_dev, f.px.n) : f.px.n;
    const int lanes = p.lanes_per_warp ? p.lanes_per_warp : 32;
    for (;;) {
        const int first = warp_take(f, n, lanes);
        if (first < 0) break;
        const int i = first + (int)(threadIdx.x & 31u);
        if (i >= n) continue;
        int arr[4];
        entry_key(f.px, i, arr);
        // dc in floatexp (mp.cpp:2160-2163).
        double px = arr[1] + (double)arr[3] / g.sub;
        double py = arr[0] + (double)arr[2] / g.sub;
        FE Dcr = fe_mul_d(p.dxfe, px - p.ref_x);
        FE Dci = fe_mul_d(p.dyfe, py - p.ref_y);
        // (the no-BLA lane kernel has no orbit colourings, mp.cpp:2148)
        PixOut o = (OC == 0 && p.no_bla_kernel) ? pixel_fe_nobla(f, p, Dcr, Dci, n_steps) : pixel_fe<OC>(f, p, Dcr, Dci, n_steps, n_bla, n_skip);
        if (o.state == 4) continue; // cancelled
        if (o.state == 1 && (OC == 0 || g.ede || g.normal || g.deovl)) fe_escape_value(p, o);
        const int idx = sample_index(g, arr);
        // mp.cpp:2173-2183: EMPTY or cutoff-sensitive results go to the
        // arbitrary-precision recompute, flagged here for the host.
        const float v = o.value;
        if (v == kEmpty || (p.cutoff_sensitive && (v < 0 || v > g.mxit - 16))) {
            f.out.gmp[i] = 1;
            atomicAdd(&f.ctr->gmp_flags, 1u);
        }
        f.out.iter[idx] = v;
        if ((g.deovl || g.normal) && f.out.normal) f.out.normal[idx] = o.nrm;
        if (f.out.escN) f.out.escN[idx] = o.state == 1 ? o.n : -1;
        f.out.done[i] = 1;
        ++n_fin;
        if (o.state == 1) {
            n_eff += (unsigned long long)o.n;
        } else {
            n_eff += (unsigned long long)g.mxit;
            ++n_int;
        }
    }
    exact_counts(f.ctr, s_counts, n_steps, n_bla, n_skip, n_eff, n_int, n_fin, lanes);
}

// ---------------------------------------------------------------------------
// The direct loops: shallow frames (floatPointCompute, mp.cpp:330-399, and the
// lane-refill kernel's per-lane arithmetic, mp.cpp:416-532) and Julia frames
// (ComputeJulia, mp.cpp:992-1041). The plain loops here, with the interior
// test's derivative in FP64, take only the samples that direct_loop.cuh leaves
// open.
struct DirectEndState {
    double zr, zi, zrad, dcr, dci;
    int n;
};
template <int OC>
__device__ __noinline__ int shallow_scalar_plain(double c_re, double c_im, int mxit, const FrameGeom& g, DirectEndState& s, OrbitColor<OC>& oc) {
    double z_re = c_re, z_im = c_im, d_re = 2, d_im = 0, dc_re = 1, dc_im = 0, tmp;
    const bool deriv = g.ede || g.deovl || g.normal;
    oc.init(); // mp.cpp:347-369
    int i = 1;
    while (i < mxit) {
        tmp = 2.0 * (d_re * z_re - d_im * z_im);
        d_im = 2.0 * (d_re * z_im + d_im * z_re);
        d_re = tmp;
        if (deriv) {
            tmp = 2.0 * (dc_re * z_re - dc_im * z_im) + 1;
            dc_im = 2.0 * (dc_re * z_im + dc_im * z_re);
            dc_re = tmp;
        }
        tmp = z_re * z_re - z_im * z_im + c_re;
        z_im = 2.0 * z_re * z_im + c_im;
        z_re = tmp;
        oc.push(z_re, z_im);
        tmp = z_re * z_re + z_im * z_im;
        if (tmp > g.ESC2) {
            s = DirectEndState{z_re, z_im, tmp, dc_re, dc_im, i + 1};
            return kDirectEscaped;
        }
        tmp = d_re * d_re + d_im * d_im;
        if (tmp < 0.000000001) return kDirectInterior;
        ++i;
    }
    return kDirectInterior;
}

__device__ __noinline__ int shallow_lane_plain(double cr, double ci, int mxit, const FrameGeom& g, DirectEndState& s) {
    double zr = cr, zi = ci, dr = 2, di = 0, dcr = 1, dci = 0;
    for (int n = 1;; ++n) {
        double ndr = 2.0 * ((dr * zr) - (di * zi));
        double ndi = 2.0 * ((dr * zi) + (di * zr));
        double ndcr = (2.0 * ((dcr * zr) - (dci * zi))) + 1.0;
        double ndci = 2.0 * ((dcr * zi) + (dci * zr));
        double nzr = ((zr * zr) - (zi * zi)) + cr;
        double nzi = (2.0 * (zr * zi)) + ci;
        zr = nzr;
        zi = nzi;
        dr = ndr;
        di = ndi;
        dcr = ndcr;
        dci = ndci;
        double zrad = (zr * zr) + (zi * zi);
        double dmag = (dr * dr) + (di * di);
        if (zrad > g.ESC2) {
            s = DirectEndState{zr, zi, zrad, dcr, dci, n + 1};
            return kDirectEscaped;
        }
        if (dmag < 1e-9 || n + 1 >= mxit) return kDirectInterior;
    }
}

// The stripe average of an escaped sample: the terms of its last
// kStripeWindow iterates, from the orbit iterated again from z_k = (zr, zi) (the
// trigonometry of the other iterations, and of every interior sample, is never
// formed; with at most a window of iterations the sums are the reference's).
__device__ __noinline__ float shallow_stripe(double cr, double ci, double zr, double zi, int k, int n, double zrad, double ER) {
    StripeTail tail;
    tail.init();
    double x2 = zr * zr, y2 = zi * zi;
    const int first = n - kStripeWindow;
    for (++k; k < n; ++k) {
        const double nzi = d_twice(zr) * zi + ci;
        zr = (x2 - y2) + cr;
        zi = nzi;
        x2 = zr * zr;
        y2 = zi * zi;
        if (k >= first) tail.push(zr, zi);
    }
    return tail.value(zrad, ER);
}
// Where to start again: the sample keeps its z of the last two multiples of the
// window; the earlier one lies a window or more before the last iterate z_(n-1).
struct StripeMark {
    double zr, zi, nr, ni;
    __device__ void visit(int k, double r, double i) {
        if ((k & (kStripeWindow - 1)) == 0) {
            zr = nr;
            zi = ni;
            nr = r;
            ni = i;
        }
    }
};
__device__ __forceinline__ int stripe_mark(int n) { return ((n - 1) & ~(kStripeWindow - 1)) - kStripeWindow; } // (<= 0: from c)

// Which loop a direct pass runs, and what its samples are.
enum DirectForm { kFormLane, kFormScalar, kFormJulia };

// The sample's c (z0 of a Julia frame) of pass entry i.
__device__ __forceinline__ void direct_c(const DeviceFrame& f, const ShallowParams& p, const int* arr, double& cr, double& ci) {
    if (arr[2] == 0 && arr[3] == 0 && !f.px.keys) {
        ci = p.c0i + p.dy * arr[0];
        cr = p.c0r + p.dx * arr[1];
    } else {
        cr = p.c0r + p.dx * arr[1] + p.dx * arr[3] / p.g.sub;
        ci = p.c0i + p.dy * arr[0] + p.dy * arr[2] / p.g.sub;
    }
}

// A finished sample waiting for its value: the escape iteration (interior: -1),
// z and |z|^2 there, and dz/dc or, under a trap, its minima (a, b, zr), under a
// stripe average its mark (a, b).
struct DirectDone {
    double zrad, a, b, zr, zi;
    int n, i;
};

// The sample's value and outputs (mp.cpp:373-398, 1500-1515; Julia :1019-1041).
template <int FORM, int OC>
__device__ __forceinline__ void direct_write(const DeviceFrame& f, const ShallowParams& p, const DirectDone& d) {
    const FrameGeom& g = p.g;
    int arr[4];
    entry_key(f.px, d.i, arr);
    const int idx = sample_index(g, arr);
    const bool inside = d.n < 0;
    if (FORM == kFormJulia) {
        float v = -2.0f;
        if (!inside) {
            if (g.ede) {
                if (d.n == 0) v = (float)distance_value(d.zrad, 1.0, 0.0);
                else if (!distance_pair(d.zrad, d.a, d.b, v)) v = julia_distance(d.zrad, d.a, d.b);
                if (v >= 0.0f) v /= (float)p.dx;
            } else {
                v = d.n == 0 ? (float)(-log(log(d.zrad) / 2 / kLn2) / kLn2) : smooth_float(d.n, d.zrad);
            }
        }
        f.out.iter[idx] = v;
        if (f.out.escN) f.out.escN[idx] = d.n;
        return;
    }
    double val = -2.0, de = 0.0;
    if (OC & kOcTrap) {
        if (inside || !(g.ede || g.normal || g.deovl)) { // (an escaped DE sample's value is not its trap's)
            OrbitTrap t;
            t.point2 = d.a;
            t.cross = d.b;
            t.circle = d.zr;
            val = inside ? (double)t.value(0.0) : (double)t.value(smooth_value(d.n, d.zrad)); // mp.cpp:383-389
        }
    }
    if (!inside && !((OC & kOcTrap) && !(g.ede || g.normal || g.deovl))) {
        if (g.ede) {
            val = (double)distance_float(d.zrad, d.a, d.b);
        } else {
            if (g.normal) de = atan2(d.zi, d.zr) - atan2(d.b, d.a); // mp.cpp:375-378
            else if (g.deovl) de = distance_value(d.zrad, d.a, d.b);
            if (OC == kOcStripe && !g.normal && !g.deovl) {
                double cr, ci;
                direct_c(f, p, arr, cr, ci);
                const int k = stripe_mark(d.n);
                val = k > 0 ? shallow_stripe(cr, ci, d.a, d.b, k, d.n, d.zrad, g.ER) : shallow_stripe(cr, ci, cr, ci, 0, d.n, d.zrad, g.ER);
            } else {
                val = (double)smooth_float(d.n, d.zrad);
            }
        }
    }
    if (FORM == kFormLane) {
        val = (double)(float)val;
        if (g.ede && val >= 0) val /= p.dx;
        f.out.iter[idx] = (float)val;
    } else if (g.normal) { // mp.cpp:1504-1507 (with EDE also set: the raw distance, angle 0)
        f.out.iter[idx] = (float)val;
        if (f.out.normal) f.out.normal[idx] = (float)de;
    } else if (g.deovl) {
        float v = (float)val;
        f.out.iter[idx] = v;
        if (f.out.normal) f.out.normal[idx] = (v < 0) ? 0.0f : (float)(de / p.dx);
    } else { // the value is stored as float before the EDE division (mp.cpp:1512-1515)
        float v = (float)val;
        if (g.ede && v >= 0) v = (float)((double)v / p.dx);
        f.out.iter[idx] = v;
    }
    if (f.out.escN) f.out.escN[idx] = d.n;
    f.out.done[d.i] = 1;
}

// The direct pass, persistent. Neighbouring samples differ widely in length (the
// whole set at 1280x720: 43 steps a sample, 276 the longest of 32 neighbours), and
// an FP64 warp instruction costs the same with one lane as with 32, so lanes are
// kept full:
//   * while samples are left, a warp steps its lanes in blocks of kDirectBlock
//     and fetches new samples once kDirectRefill lanes are idle;
//   * then the block's threads, few of them still iterating, are packed into as
//     few warps as hold them, every kDirectRound steps (the samples left are
//     the longest: without this they ran 6.6 to a warp);
//   * a value costs over a hundred FP64 instructions (log, sqrt, divisions;
//     atan2 and sin for a stripe average), so finished samples wait in shared
//     memory until a warp has 32 and forms them in full (a stripe average's terms
//     are as many as the orbit is long: short and long orbits wait apart).
// Measured (1280x720 whole set / stripe average 601x399 with 3x3 supersampling /
// 2560x1440 overlay image): one sample after the other per lane 5.7 / 14.9 / 53.7
// ms, with the refill alone 7.1 / 15.8 / 53.6, packed 3.1 / 19.2 / 49.6, with the
// stripe terms from powers of z, their bins and marks, and one branch a step
// 2.3 / 8.8 / 36.8.
constexpr int kDirectBlock = 8, kDirectRefill = 4, kDirectRound = 32;
template <int OC>
constexpr int kDirectBins = OC == kOcStripe ? 2 : 1;
constexpr int kDirectLongOrbit = 32;

template <int FORM, bool DERIV, int OC>
struct DirectSample {
    typename std::conditional<FORM == kFormJulia, JuliaLane<DERIV>, DirectLane<FORM == kFormLane, DERIV>>::type L;
    typename std::conditional<(OC & kOcTrap) != 0, DirectTrap, char>::type trap;
    typename std::conditional<OC == kOcStripe && !DERIV, StripeMark, char>::type mark;
    int entry;
};

template <int FORM, bool DERIV, int OC>
__global__ void __launch_bounds__(512) k_direct(DeviceFrame f, ShallowParams p) {
    using Sample = DirectSample<FORM, DERIV, OC>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_live[16 * kDirectBins<OC>], s_stop;
    __shared__ BlockCounts s_counts;
    block_counts_init(s_counts);
    const FrameGeom& g = p.g;
    const int n_all = f.px.n;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    const int warps = (int)(blockDim.x >> 5);
    constexpr int kBins = kDirectBins<OC>;
    DirectDone* buf = reinterpret_cast<DirectDone*>(smem) + 64 * kBins * warp; // this warp's finished samples
    Sample* pool = reinterpret_cast<Sample*>(smem + sizeof(DirectDone) * 64 * kBins * warps);
    Sample S;
    unsigned long long n_eff = 0, n_steps = 0;
    unsigned int n_int = 0;
    int waiting[kBins] = {}, st = kDirectRuns;
    bool live = false;

    auto run = [&](int steps) {
#pragma unroll 1
        for (int k = 0; k < steps && st == kDirectRuns; ++k) {
            if constexpr (FORM == kFormJulia) {
                st = S.L.step(p.cr, p.ci, g.mxit, g.ESC2, p.esc_word);
            } else {
                st = S.L.step(g.mxit, g.ESC2, p.esc_word, [&](double zr, double zi, double x2, double y2) {
                    if constexpr ((OC & kOcTrap) != 0) S.trap.push(zr, zi, x2, y2);
                    if constexpr (OC == kOcStripe && !DERIV) S.mark.visit(S.L.n, zr, zi); // (n: the iterate's index, before it counts)
                });
            }
        }
    };
    // takes the warp's ended lanes off and forms 32 values when they are there
    auto finish = [&]() {
        __syncwarp();
        const unsigned ended = __ballot_sync(0xffffffffu, live && st != kDirectRuns);
        if (ended == 0) return;
        unsigned in_bin[kBins];
        if constexpr (kBins == 2) {
            in_bin[1] = __ballot_sync(0xffffffffu, live && st == kDirectEscaped && S.L.n > kDirectLongOrbit);
            in_bin[0] = ended & ~in_bin[1];
        } else {
            in_bin[0] = ended;
        }
        if (live && st != kDirectRuns) {
            DirectDone d{S.L.x2 + S.L.y2, S.L.dcr, S.L.dci, S.L.zr, S.L.zi, S.L.n, S.entry};
            if constexpr ((OC & kOcTrap) != 0) {
                if (!(DERIV && st == kDirectEscaped)) {
                    d.a = S.trap.point2;
                    d.b = bitsd(S.trap.cross);
                    d.zr = S.trap.circle;
                }
            }
            if constexpr (OC == kOcStripe && !DERIV) {
                d.a = S.mark.zr;
                d.b = S.mark.zi;
            }
            if constexpr (FORM != kFormJulia) {
                if (st == kDirectOpen) {
                    DirectEndState e;
                    OrbitColor<OC & kOcTrap> oc;
                    st = FORM == kFormLane ? shallow_lane_plain(S.L.cr, S.L.ci, g.mxit, g, e) : shallow_scalar_plain<OC & kOcTrap>(S.L.cr, S.L.ci, g.mxit, g, e, oc);
                    if (st == kDirectEscaped) d = DirectDone{e.zrad, e.dcr, e.dci, e.zr, e.zi, e.n, S.entry};
                    if constexpr (OC == kOcStripe && !DERIV) {
                        if (st == kDirectEscaped && stripe_mark(e.n) > 0) { // the mark, iterated
                            double zr = S.L.cr, zi = S.L.ci;
                            for (int k = 0; k < stripe_mark(e.n); ++k) {
                                const double nzi = d_twice(zr) * zi + S.L.ci;
                                zr = (zr * zr - zi * zi) + S.L.cr;
                                zi = nzi;
                            }
                            d.a = zr;
                            d.b = zi;
                        }
                    }
                    if constexpr ((OC & kOcTrap) != 0) {
                        if (!(DERIV && st == kDirectEscaped)) {
                            d.a = oc.trap.point2;
                            d.b = oc.trap.cross;
                            d.zr = oc.trap.circle;
                        }
                    }
                }
            }
            if (st == kDirectInterior) {
                d.n = -1;
                n_eff += (unsigned long long)g.mxit;
                if (FORM == kFormJulia) n_steps += (unsigned long long)g.mxit;
                ++n_int;
            } else {
                n_eff += (unsigned long long)d.n;
                n_steps += (unsigned long long)d.n;
            }
#pragma unroll
            for (int k = 0; k < kBins; ++k)
                if ((in_bin[k] >> lane) & 1u) buf[64 * k + waiting[k] + __popc(in_bin[k] & below)] = d;
            live = false;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kBins; ++k) {
            waiting[k] += __popc(in_bin[k]);
            if (waiting[k] >= 32) {
                waiting[k] -= 32;
                direct_write<FORM, OC>(f, p, buf[64 * k + waiting[k] + lane]);
                __syncwarp();
            }
        }
    };

    for (int rounds = 0;; ++rounds) {
        const unsigned idle = __ballot_sync(0xffffffffu, !live);
        const int want = __popc(idle);
        if (want >= kDirectRefill || (rounds & 3) == 0) {
            int base = 0;
            if (lane == 0) {
                base = n_all;
                if (!cancelled(f) && (int)*(volatile unsigned int*)&f.ctr->next < n_all) base = want ? (int)atomicAdd(&f.ctr->next, (unsigned)want) : 0;
            }
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= n_all) break;
            const int i = base + __popc(idle & below);
            if (!live && i < n_all) {
                S.entry = i;
                int arr[4];
                entry_key(f.px, i, arr);
                double cr, ci;
                direct_c(f, p, arr, cr, ci);
                if constexpr (FORM == kFormJulia) st = S.L.start(cr, ci, g.ESC2);
                else st = S.L.start(cr, ci, g.mxit, g.ESC2);
                if constexpr ((OC & kOcTrap) != 0) S.trap.init();
                live = true;
            }
        }
        if (live) run(kDirectBlock);
        finish();
    }
    for (;;) {
        const unsigned m = __ballot_sync(0xffffffffu, live);
        if (lane == 0) s_live[warp] = __popc(m);
        if (threadIdx.x == 0) s_stop = cancelled(f) ? 1 : 0;
        __syncthreads();
        int total = 0, before = 0, used = 0;
        for (int w = 0; w < warps; ++w) {
            const int c = s_live[w];
            if (w < (int)warp) before += c;
            total += c;
            used += c ? 1 : 0;
        }
        const bool stop = s_stop != 0;
        if (total == 0 || stop) break;
        const bool pack = (total + 31) / 32 < used;
        if (pack && live) pool[before + __popc(m & below)] = S;
        __syncthreads();
        if (pack) {
            live = (int)threadIdx.x < total;
            if (live) {
                S = pool[threadIdx.x];
                st = kDirectRuns;
            }
        }
        if (live) run(kDirectRound);
        finish();
    }
    // the values still waiting, over the block's warps in full, both bins at once
    // (one after the other, a stripe frame of 120x80 took 262 us at maxiter 50; 213)
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < kBins; ++k) s_live[k * warps + warp] = waiting[k];
    }
    __syncthreads();
    int total = 0;
    for (int v = 0; v < kBins * warps; ++v) total += s_live[v];
    for (int t = (int)threadIdx.x; t < total; t += (int)blockDim.x) {
        int at = t, v = 0;
        for (; at >= s_live[v]; ++v) at -= s_live[v];
        direct_write<FORM, OC>(f, p, reinterpret_cast<DirectDone*>(smem)[64 * (kBins * (v % warps) + v / warps) + at]);
    }
    exact_counts(f.ctr, s_counts, n_steps, 0, 0, n_eff, n_int, 0, 32);
}

// ---------------------------------------------------------------------------
// BLA table construction (mp.cpp:2613-2709): level 0 from the orbit, then one
// launch per merge level; every entry of a level is independent.
__global__ void k_bla_level0(const double2* Z, const double2* D, int reflen, double eps, double dcmax, int ede, double* r2, double4* ab, double4* ce, unsigned long long* rmax2_bits) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int s = t + 1;
    if (s >= reflen) return;
    double2 z = Z[s];
    double zr = z.x, zi = z.y;
    double Zmag = sqrt(zr * zr + zi * zi);
    double ar = 2.0 * zr, ai = 2.0 * zi;
    double Amag = 2.0 * Zmag;
    double R = eps * (Zmag - dcmax) / (Amag + 1.0);
    double rr = R > 0 ? R * R : 0.0;
    r2[t] = rr;
    ab[t] = make_double4(ar, ai, 1.0, 0.0);
    if (ede) {
        double2 d = D[s];
        ce[t] = make_double4(2.0 * d.x, 2.0 * d.y, 0.0, 0.0);
    }
    if (rr > 0) atomicMax(rmax2_bits, (unsigned long long)__double_as_longlong(rr));
}

__global__ void k_bla_merge(double dcmax, int ede, double* r2, double4* ab, double4* ce, int src_off, int dst_off, int dst_size) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= dst_size) return;
    const int xi = src_off + 2 * i, yi = xi + 1;
    double4 xc = ab[xi], yc = ab[yi];
    double4 zc;
    zc.x = yc.x * xc.x - yc.y * xc.y;
    zc.y = yc.x * xc.y + yc.y * xc.x;
    zc.z = yc.x * xc.z - yc.y * xc.w + yc.z;
    zc.w = yc.x * xc.w + yc.y * xc.z + yc.w;
    if (ede) {
        double4 xd = ce[xi], yd = ce[yi];
        double4 zd;
        zd.x = (yd.x * xc.x - yd.y * xc.y) + (yc.x * xd.x - yc.y * xd.y);
        zd.y = (yd.x * xc.y + yd.y * xc.x) + (yc.x * xd.y + yc.y * xd.x);
        zd.z = (yd.x * xc.z - yd.y * xc.w) + (yc.x * xd.z - yc.y * xd.w) + yd.z;
        zd.w = (yd.x * xc.w + yd.y * xc.z) + (yc.x * xd.w + yc.y * xd.z) + yd.w;
        ce[dst_off + i] = zd;
    }
    double Rx = sqrt(r2[xi]), Ry = sqrt(r2[yi]);
    double Axmag = sqrt(xc.x * xc.x + xc.y * xc.y);
    double Bxmag = sqrt(xc.z * xc.z + xc.w * xc.w);
    double cand = Axmag > 0 ? (Ry - Bxmag * dcmax) / Axmag : 0.0;
    double R = (cand < Rx) ? cand : Rx; // std::min(Rx, cand)
    r2[dst_off + i] = R > 0 ? R * R : 0.0;
    ab[dst_off + i] = zc;
}

// ---------------------------------------------------------------------------
// Adaptive-SS flags over the base samples (mp.cpp:1838-1884).
// Adaptive-SS selection (mp.cpp:1796-1879). mode: kSsIterations (the
// iteration difference against thresh), kSsEde (a sign change: the set
// boundary), kSsStripe / kSsTrap (the stripe average and orbit traps store a
// value, not a count: the set boundary, or a colour change of more than
// `steps` palette entries per pixel, `gain` entries per unit of value; the
// stripe average's steps default to 0, the boundary only).
__global__ void k_ss_flags(const float* iter, int W, int H, int sub, int mode, double thresh, double gain, double steps, uint8_t* flags) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= W * H) return;
    int i = q / W, j = q % W;
    auto at = [&](int r, int c) { return iter[(r * sub + sub / 2) * W * sub + (c * sub + sub / 2)]; };
    bool need = false;
    if (mode == kSsEde) {
        float cv = at(i, j);
        for (int xi = -1; xi <= 1 && !need; ++xi)
            for (int yi = -1; yi <= 1; ++yi) {
                if (xi == 0 && yi == 0) continue;
                int ny = i + yi, nx = j + xi;
                if (nx >= 0 && nx < W && ny >= 0 && ny < H && cv * at(ny, nx) < 0) {
                    need = true;
                    break;
                }
            }
    } else {
        float cv = at(i, j);
        float diff = 0;
        bool boundary = false;
        for (int xi = -1; xi <= 1; ++xi)
            for (int yi = -1; yi <= 1; ++yi) {
                if (xi == 0 && yi == 0) continue;
                int ny = i + yi, nx = j + xi;
                if (nx >= 0 && nx < W && ny >= 0 && ny < H) {
                    const float nv = at(ny, nx);
                    diff = fmaxf(diff, fabsf(cv - nv));
                    if (cv * nv < 0) boundary = true; // interior / exterior edge
                }
            }
        if (mode == kSsStripe)
            need = boundary || (steps > 0 && diff * gain > steps);
        else if (mode == kSsTrap)
            need = boundary || (diff * gain > steps);
        else
            need = log((double)diff) > thresh;
    }
    flags[q] = need ? 1 : 0;
}

__global__ void k_fill(float* iter, float* normal, int32_t* escN, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        iter[i] = kEmpty;
        if (normal) normal[i] = 0.0f;
        if (escN) escN[i] = -10;
    }
}

// ---------------------------------------------------------------------------
cudaError_t launch_fill(float* iter, float* normal, int32_t* escN, size_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 152 * 16) blocks = 152 * 16;
    k_fill<<<blocks, 256, 0, st>>>(iter, normal, escN, n);
    return cudaGetLastError();
}
cudaError_t launch_fp64_pass(const DeviceFrame& f, const Fp64Params& fp, int blocks, int threads, cudaStream_t st) {
    Fp64Params p = fp;
    p.esc_word = direct_escape_word(p.g.ESC2);
    switch (p.g.oc) {
    case 0: k_fp64_pass<0><<<blocks, threads, 0, st>>>(f, p); break;
    case kOcStripe: k_fp64_pass<kOcStripe><<<blocks, threads, 0, st>>>(f, p); break;
    case kOcTrap: k_fp64_pass<kOcTrap><<<blocks, threads, 0, st>>>(f, p); break;
    default: k_fp64_pass<kOcStripe | kOcTrap><<<blocks, threads, 0, st>>>(f, p); break;
    }
    return cudaGetLastError();
}
cudaError_t launch_fe_pass(const DeviceFrame& f, const FeParams& fp, int blocks, int threads, cudaStream_t st) {
    FeParams p = fp;
    p.esc_word = direct_escape_word(p.g.ESC2);
    switch (p.g.oc) {
    case 0: k_fe_pass<0><<<blocks, threads, 0, st>>>(f, p); break;
    case kOcStripe: k_fe_pass<kOcStripe><<<blocks, threads, 0, st>>>(f, p); break;
    case kOcTrap: k_fe_pass<kOcTrap><<<blocks, threads, 0, st>>>(f, p); break;
    default: k_fe_pass<kOcStripe | kOcTrap><<<blocks, threads, 0, st>>>(f, p); break;
    }
    return cudaGetLastError();
}
// Blocks of 512 threads, one per SM (four warps a scheduler keep its FP64 unit
// busy, and the larger the block, the better its last samples pack); frames that
// would leave SMs without a block take blocks of 128.
template <int FORM, bool DERIV, int OC>
static cudaError_t launch_direct(const DeviceFrame& f, const ShallowParams& p, int nsm, cudaStream_t st) {
    const int threads = f.px.n >= nsm * 512 ? 512 : 128;
    const int blocks = threads == 512 ? nsm : (f.px.n + 127) / 128;
    const size_t smem = sizeof(DirectDone) * 2 * kDirectBins<OC> * threads + sizeof(DirectSample<FORM, DERIV, OC>) * threads;
    auto kern = k_direct<FORM, DERIV, OC>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<blocks, threads, smem, st>>>(f, p);
    return cudaGetLastError();
}
template <bool DERIV>
static cudaError_t launch_scalar(const DeviceFrame& f, const ShallowParams& p, int nsm, cudaStream_t st) {
    switch (p.g.oc) {
    case 0: return launch_direct<kFormScalar, DERIV, 0>(f, p, nsm, st);
    case kOcStripe: return launch_direct<kFormScalar, DERIV, kOcStripe>(f, p, nsm, st);
    default: return launch_direct<kFormScalar, DERIV, kOcTrap>(f, p, nsm, st); // (a trap's value comes before a stripe average's)
    }
}
cudaError_t launch_julia(const DeviceFrame& f, const ShallowParams& jp, int nsm, cudaStream_t st) {
    ShallowParams p = jp;
    p.esc_word = direct_escape_word(p.g.ESC2);
    return p.g.ede ? launch_direct<kFormJulia, true, 0>(f, p, nsm, st) : launch_direct<kFormJulia, false, 0>(f, p, nsm, st);
}
cudaError_t launch_shallow(const DeviceFrame& f, const ShallowParams& sp, int nsm, cudaStream_t st) {
    ShallowParams p = sp;
    p.esc_word = direct_escape_word(p.g.ESC2);
    if (p.g.oc == 0 && p.simd_semantics) // (no orbit colourings in the lane kernel, mp.cpp:1459)
        return p.g.ede ? launch_direct<kFormLane, true, 0>(f, p, nsm, st) : launch_direct<kFormLane, false, 0>(f, p, nsm, st);
    return (p.g.ede || p.g.deovl || p.g.normal) ? launch_scalar<true>(f, p, nsm, st) : launch_scalar<false>(f, p, nsm, st);
}
cudaError_t launch_bla_build(const double2* Z, const double2* D, int reflen, double eps, double dcmax, bool ede, double* r2, double4* ab, double4* ce, const int* off, const int* size, int nlev, unsigned long long* rmax2_bits, cudaStream_t st) {
    int n0 = reflen - 1;
    if (n0 <= 0) return cudaSuccess;
    k_bla_level0<<<(n0 + 255) / 256, 256, 0, st>>>(Z, D, reflen, eps, dcmax, ede ? 1 : 0, r2, ab, ce, rmax2_bits);
    for (int p = 1; p < nlev; ++p) {
        int n = size[p];
        if (n <= 0) break;
        k_bla_merge<<<(n + 255) / 256, 256, 0, st>>>(dcmax, ede ? 1 : 0, r2, ab, ce, off[p - 1], off[p], n);
    }
    return cudaGetLastError();
}
cudaError_t launch_ss_flags(const float* iter, int W, int H, int sub, int mode, double thresh, double gain, double steps, uint8_t* flags, cudaStream_t st) {
    int n = W * H;
    k_ss_flags<<<(n + 255) / 256, 256, 0, st>>>(iter, W, H, sub, mode, thresh, gain, steps, flags);
    return cudaGetLastError();
}

} // namespace mbx
