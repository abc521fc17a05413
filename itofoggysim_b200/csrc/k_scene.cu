// Scene-level kernels: Mie coefficients, plane-wave right-hand side, layout conversion between
// the reference's flat coefficient vector and the device's ragged scaled layout, and the
// cluster cross-sections.
#include <algorithm>

#include "foggy_kernels.cuh"
#include "k_common.cuh"
#include "k_special.cuh"

namespace foggy {

// ---- Mie coefficients a_n, b_n (lib_mie_ss_helper_functions.f90:628-722; logarithmic
// derivative by downward recurrence 751-924; start n_c from 937-951) -----------------------
__global__ void k_mie_ab(int n_param, const double* size_param, const double* m_re, const double* m_im,
                         const int* p_of_param, int pstride, cplx* an_out, cplx* bn_out) {
    int ip = blockIdx.x * blockDim.x + threadIdx.x;
    if (ip >= n_param) return;
    double x = size_param[ip];
    cplx m = mk(m_re[ip], m_im[ip]);
    int p = p_of_param[ip];
    cplx mx = mk(m.x * x, m.y * x);
    double amx = sqrt(mx.x * mx.x + mx.y * mx.y);
    int n_c = (int)ceil(x + 4.05 * cbrt(x) + 2.0);
    int n_mx = max(n_c, (int)amx) + 15;
    cplx* an = an_out + (size_t)ip * pstride;
    cplx* bn = bn_out + (size_t)ip * pstride;
    // downward: A_{i-1} = i/(mx) - 1/(A_i + i/(mx)); keep A_n for n = 1..p in an[] temporarily
    cplx A = mk(0, 0);
    for (int i = n_mx; i >= 2; --i) {
        cplx ndm = cdiv(mk((double)i, 0), mx);
        A = ndm - cdiv(mk(1, 0), A + ndm);
        if (i - 1 <= p) an[i - 2] = A;
    }
    double jb[kMaxDegree + 2], yb[kMaxDegree + 2];
    dev_sph_jn(x, p, jb);
    dev_sph_yn(x, p, yb);
    for (int n = 1; n <= p; ++n) {
        cplx An = an[n - 1];
        double ndx = (double)n / x;
        cplx jn = mk(jb[n], 0), jnm = mk(jb[n - 1], 0), hn = mk(jb[n], yb[n]), hnm = mk(jb[n - 1], yb[n - 1]);
        cplx bufa = cdiv(An, m) + mk(ndx, 0);
        cplx bufb = m * An + mk(ndx, 0);
        an[n - 1] = cdiv(bufa * jn - jnm, bufa * hn - hnm);
        bn[n - 1] = cdiv(bufb * jn - jnm, bufb * hn - hnm);
    }
}

__global__ void k_gather_an(int n, const int* pidx, int pstride, const cplx* an_p, const cplx* bn_p,
                            cplx* an_s, cplx* bn_s) {
    int j = blockIdx.x;
    int ip = pidx[j];
    for (int t = threadIdx.x; t < pstride; t += blockDim.x) {
        an_s[(size_t)j * pstride + t] = an_p[(size_t)ip * pstride + t];
        bn_s[(size_t)j * pstride + t] = bn_p[(size_t)ip * pstride + t];
    }
}

// ---- scaled pi_nm, tau_nm of each wave (lib_math_legendre.f90:834-982; values divided by
// g_nm = (-1)^m sqrt((n+m)!/(n-m)!), which turns the recurrence into the stable normalised
// one).  Table pt[w][n(n+1)+m] (pi) and tt[...] (tau).  One thread per m >= 0. -------------
__global__ void k_pitau(int nw, const WaveDev* waves, int pmax, double* pi_out, double* tau_out) {
    int w = blockIdx.x;
    int m = threadIdx.x;
    if (m > pmax) return;
    double alpha = waves[w].alpha;
    double x = cos(alpha), s = sin(alpha);
    int S = (pmax + 1) * (pmax + 1);
    double* pi = pi_out + (size_t)w * S;
    double* tau = tau_out + (size_t)w * S;
    double sgm = (m & 1) ? -1.0 : 1.0;
    if (x == 1.0 || x == -1.0) {
        // The reference's pole table (lib_math_legendre.f90:854-920), phase removed, then
        // scaled by 1/g_{n,+-1} = -1/sqrt(n(n+1)), -sqrt(n(n+1)).  At x = -1 it sets
        // tau_n^{+-1} = -pi_n^{+-1} for odd n, which flips the sign of tau_n^{-1} there
        // relative to the limit of the general formula; kept as the reference has it.
        for (int n = max(m, 1); n <= pmax; ++n) {
            pi[n * (n + 1) + m] = 0.0;
            tau[n * (n + 1) + m] = 0.0;
            pi[n * (n + 1) - m] = 0.0;
            tau[n * (n + 1) - m] = 0.0;
        }
        if (m == 1) {
            for (int n = 1; n <= pmax; ++n) {
                double h = (double)(n * (n + 1) / 2);
                double pim = -0.5, pip = -h, taum = 0.5, taup = -h;   // with phase, x = +1
                if (x == -1.0) {
                    if (!(n & 1)) { pim = -pim; pip = -pip; }
                    else { taum = -pim; taup = -pip; }
                }
                double r = sqrt((double)n * (n + 1));
                // phase removed (odd |m|): negate; scaled by 1/g
                pi[n * (n + 1) - 1] = -pim * (-r);
                tau[n * (n + 1) - 1] = -taum * (-r);
                pi[n * (n + 1) + 1] = -pip / (-r);
                tau[n * (n + 1) + 1] = -taup / (-r);
            }
        }
        if (m == 0) { pi[0] = 0.0; tau[0] = 0.0; }
        return;
    }
    if (m == 0) {
        // tau_n^0 = -P_n^1 (no phase) -> scaled: -sqrt(n(n+1)) * Phat_n^1
        // Phat_n^1 by the normalised recurrence from Phat_1^1 = sqrt(1/2) s
        double pm2 = 0.0, pm1 = 0.0;
        for (int n = 1; n <= pmax; ++n) {
            double pn;
            if (n == 1) pn = sqrt(0.5) * s;
            else if (n == 2) pn = sqrt(3.0) * x * pm1;
            else pn = ((2.0 * n - 1.0) * x * pm1 - sqrt((n - 1.0) * (n - 1.0) - 1.0) * pm2) / sqrt((double)n * n - 1.0);
            pm2 = pm1;
            pm1 = pn;
            pi[n * (n + 1)] = 0.0;
            tau[n * (n + 1)] = -sqrt((double)n * (n + 1)) * pn;
        }
        pi[0] = 0.0;
        tau[0] = 0.0;
        return;
    }
    // Qhat_n^m = Phat_n^m / sin(alpha), Phat = sqrt((n-m)!/(n+m)!) P_n^m (no phase)
    double qmm = 1.0;
    for (int k = 1; k <= m; ++k) qmm *= sqrt((2.0 * k - 1.0) / (2.0 * k));
    for (int k = 1; k < m; ++k) qmm *= s;
    double qm2 = 0.0, qm1 = 0.0;   // Qhat_{n-2}, Qhat_{n-1}
    for (int n = m; n <= pmax; ++n) {
        double qn;
        if (n == m) qn = qmm;
        else if (n == m + 1) qn = sqrt(2.0 * m + 1.0) * x * qm1;
        else qn = ((2.0 * n - 1.0) * x * qm1 - sqrt((n - 1.0 - m) * (n - 1.0 + m)) * qm2) / sqrt((double)(n - m) * (n + m));
        double qprev = qm1;
        qm2 = qm1;
        qm1 = qn;
        double pv = m * qn;                                           // pi-hat_n^m
        double tv = n * x * qn - sqrt((double)(n + m) * (n - m)) * qprev;   // tau-hat_n^m
        pi[n * (n + 1) + m] = sgm * pv;
        tau[n * (n + 1) + m] = sgm * tv;
        // negative orders: pi_{n,-m} = -(-1)^m pi_{n,m}, tau_{n,-m} = (-1)^m tau_{n,m} (scaled)
        pi[n * (n + 1) - m] = -sgm * sgm * pv;
        tau[n * (n + 1) - m] = sgm * sgm * tv;
    }
}

// ---- right-hand side b = [a_n p ; b_n q] (lib_mie_ms_solver_interface.f90:230-315) with the
// plane-wave coefficients of lib_mie_illumination.f90:392-478 (several waves, Jones vector,
// TE swaps p and q) and :636-763 (p = tau e^{-i m beta}/(n(n+1)) e^{i(k.d + phase)}).
// One block per sphere; pq keeps the incident coefficients for the cross-sections. --------
namespace {
// p, q of one plane wave W at degree n, order m of a sphere centred at cj (pi_s, tau_s its scaled
// Legendre values there), times W.g, added to pv, qv
__device__ __forceinline__ void add_wave(const WaveDev& W, const double* cj, int m, double rn, double pi_s,
                                         double tau_s, cplx& pv, cplx& qv) {
    double d0 = cj[0] - W.d0[0], d1 = cj[1] - W.d0[1], d2 = cj[2] - W.d0[2];
    double dn = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    double kd = W.kc[0] * d0 + W.kc[1] * d1 + W.kc[2] * d2;
    if (W.alpha == 0.0 && m != 1 && m != -1) { pi_s = 0.0; tau_s = 0.0; }
    double sb, cbv;
    sincos(-m * W.beta, &sb, &cbv);
    cplx base = mk(rn * cbv, rn * sb);
    cplx tp = mk(0, 0), tq = mk(0, 0);
    if (W.ax > 0) {
        cplx e = mk(1, 0);
        if (dn > 0.0 || W.phx != 0.0) { double ss, cc; sincos(kd + W.phx, &ss, &cc); e = mk(cc, ss); }
        tp = tp + W.ax * (e * (tau_s * base));
        tq = tq + W.ax * (e * (pi_s * base));
    }
    if (W.ay > 0) {
        cplx e = mk(1, 0);
        if (dn > 0.0 || W.phy != 0.0) { double ss, cc; sincos(kd + W.phy, &ss, &cc); e = mk(cc, ss); }
        tp = tp + W.ay * (e * (pi_s * base));    // TE: p and q swap
        tq = tq + W.ay * (e * (tau_s * base));
    }
    pv = pv + W.g * tp;
    qv = qv + W.g * tq;
}
}  // namespace

// nw waves shared by all spheres (tables [w][S]) and nl local waves per sphere (waves[j nl + l],
// tables [(j nl + l)][S]), the plane waves that stand in for Gaussian beams at each sphere
__global__ void k_rhs(SceneView sc, int nw, const WaveDev* waves, int pmax, const double* pi_tab,
                      const double* tau_tab, int nl, const WaveDev* lwaves, const double* lpi_tab,
                      const double* ltau_tab, cplx* b, cplx* pq) {
    int j = blockIdx.x;
    int pj = sc.p[j];
    int Pj = pj * (pj + 2);
    int64_t o = sc.off[j];
    int S = (pmax + 1) * (pmax + 1);
    const double* cj = sc.centres + 3 * (size_t)j;
    for (int t = threadIdx.x; t < Pj; t += blockDim.x) {
        int n = (int)sqrt((double)(t + 1));
        if ((n + 1) * (n + 1) <= t + 1) ++n;
        if (n * n > t + 1) --n;
        int m = t + 1 - n * n - n;
        cplx pv = mk(0, 0), qv = mk(0, 0);
        double rn = 1.0 / (double)(n * (n + 1));
        const int e = n * (n + 1) + m;
        for (int w = 0; w < nw; ++w)
            add_wave(waves[w], cj, m, rn, pi_tab[(size_t)w * S + e], tau_tab[(size_t)w * S + e], pv, qv);
        for (int l = 0; l < nl; ++l) {
            const size_t wl = (size_t)j * nl + l;
            add_wave(lwaves[wl], cj, m, rn, lpi_tab[wl * S + e], ltau_tab[wl * S + e], pv, qv);
        }
        pq[o + t] = pv;
        pq[o + Pj + t] = qv;
        b[o + t] = sc.an[(size_t)j * sc.pmax + n - 1] * pv;
        b[o + Pj + t] = sc.bn[(size_t)j * sc.pmax + n - 1] * qv;
    }
}

// ---- Gaussian beams in the plane-wave approximation (lib_mie_illumination.f90:781-918,
// calculation_type 3, and 1022-1050; beam functions of
// FoggySim/src/lib/field/lib_field_gaussian_beam.f90:111-891).  At each sphere the beam is replaced
// by the plane wave with the direction of its phase gradient, its phase (shifted back to the
// beam origin by 2 pi z / lambda_0) and its polarisation projected on the rotated beam axes; the
// local amplitude does not enter the coefficients (lib_mie_illumination.f90:392-478 uses only
// g, the Jones vector and the phase), and the beam's g scales them twice (:864-877). --------
namespace {
// Euler rotation, x-convention (lib_math_get_matrix_rot, lib_math_type_operator.f90:1768-1810), applied to v
__device__ void euler_apply(double phi, double theta, double psi, const double v[3], double o[3]) {
    double sph, cph, sth, cth, sps, cps;
    sincos(phi, &sph, &cph);
    sincos(theta, &sth, &cth);
    sincos(psi, &sps, &cps);
    const double a = v[0], b = v[1], c = v[2];
    o[0] = (cps * cph - cth * sph * sps) * a + (cps * sph + cth * cph * sps) * b + (sps * sth) * c;
    o[1] = (-sps * cph - cth * sph * cps) * a + (-sps * sph + cth * cph * cps) * b + (cps * sth) * c;
    o[2] = (sth * sph) * a + (-sth * cph) * b + cth * c;
}
// physicists' Hermite polynomial by its three-term recurrence
__device__ double hermite_h(int n, double x) {
    double h0 = 1.0, h1 = 2.0 * x;
    if (n == 0) return h0;
    for (int k = 1; k < n; ++k) {
        const double h2 = 2.0 * x * h1 - 2.0 * k * h0;
        h0 = h1;
        h1 = h2;
    }
    return h1;
}
}  // namespace

__global__ void k_gauss_local(SceneView sc, int nb, const GaussDev* beams, double lambda0, double n_medium,
                              WaveDev* out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= sc.n * nb) return;
    const int j = t / nb;
    const GaussDev B = beams[t - j * nb];
    const double PI_ = 3.14159265358979323846;
    const double xw[3] = {sc.centres[3 * (size_t)j] - B.d0[0], sc.centres[3 * (size_t)j + 1] - B.d0[1],
                          sc.centres[3 * (size_t)j + 2] - B.d0[2]};
    const bool rot = B.phi != 0.0 || B.theta != 0.0;
    double x[3] = {xw[0], xw[1], xw[2]};
    if (rot) euler_apply(PI_ / 2.0 + B.phi, B.theta, PI_ / 2.0 + B.phi, xw, x);
    // propagation direction: minus the phase gradient in the beam frame, normalised, rotated back
    // (get_derivative_xy / get_derivative_z, lib_field_gaussian_beam.f90:573-679)
    const double pn2 = (PI_ * n_medium) * (PI_ * n_medium), lz2 = (lambda0 * x[2]) * (lambda0 * x[2]);
    const double wx2 = B.wx0 * B.wx0, wx4 = wx2 * wx2, wy2 = B.wy0 * B.wy0, wy4 = wy2 * wy2;
    auto dxy = [&](double w4, double xy) {
        return (xy == 0.0 || x[2] == 0.0) ? 0.0 : -2.0 * PI_ * lambda0 * xy * x[2] * n_medium / (pn2 * w4 + lz2);
    };
    double dz = (2.0 * B.tem_m * wx2 + 2.0 * x[0] * x[0]) / (pn2 * wx4 + lz2);
    dz += (2.0 * B.tem_n * wy2 + 2.0 * x[1] * x[1]) / (pn2 * wy4 + lz2);
    dz += -4.0 * pn2 * x[0] * x[0] * wx4 / ((pn2 * wx4 + lz2) * (pn2 * wx4 + lz2));
    dz += -4.0 * pn2 * x[1] * x[1] * wy4 / ((pn2 * wy4 + lz2) * (pn2 * wy4 + lz2));
    dz = PI_ * n_medium * (dz * lambda0 * lambda0 / 2.0 - 2.0) / lambda0;
    double kb[3] = {-dxy(wx4, x[0]), -dxy(wy4, x[1]), -dz};
    const double kn = sqrt(kb[0] * kb[0] + kb[1] * kb[1] + kb[2] * kb[2]);
    kb[0] /= kn;
    kb[1] /= kn;
    kb[2] /= kn;
    double kv[3] = {kb[0], kb[1], kb[2]};
    if (rot) euler_apply(-PI_ / 2.0 - B.phi, -B.theta, -PI_ / 2.0 - B.phi, kb, kv);
    const double kr = sqrt(kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2]);
    const double th = (kr == 0.0) ? 0.0 : acos(kv[2] / kr);
    const double ph = (kv[0] == 0.0 && kv[1] == 0.0) ? 0.0 : atan2(kv[1], kv[0]);
    // argument of the beam at the point (get_absolute_value_and_argument, :681-799)
    const double k = 2.0 * PI_ * n_medium / lambda0, two_pi = 2.0 * PI_;
    const double zrx = PI_ * wx2 * n_medium / lambda0, zry = PI_ * wy2 * n_medium / lambda0;
    const double wx = B.wx0 * sqrt(1.0 + (x[2] / zrx) * (x[2] / zrx)), wy = B.wy0 * sqrt(1.0 + (x[2] / zry) * (x[2] / zry));
    const double crx = x[2] / (x[2] * x[2] + zrx * zrx), cry = x[2] / (x[2] * x[2] + zry * zry);
    double arg = -fmod(k * crx * x[0] * x[0] / 2.0, two_pi);
    arg = arg - fmod(k * cry * x[1] * x[1] / 2.0, two_pi);
    arg = arg - fmod(k * x[2], two_pi) + B.phase;
    arg = arg + (B.tem_m + 0.5) * atan2(x[2], zrx);
    arg = arg + (B.tem_n + 0.5) * atan2(x[2], zry);
    const double hx = hermite_h(B.tem_m, x[0] * sqrt(2.0) / wx), hy = hermite_h(B.tem_n, x[1] * sqrt(2.0) / wy);
    if (hx * hy < 0.0) arg = arg - PI_;
    arg = fmod(arg, two_pi);
    if (B.convention == 2) arg = -arg;
    if (arg < 0.0) arg = two_pi + arg;
    double phase = fmod(arg + fmod(two_pi * x[2] / lambda0, two_pi), two_pi);
    if (phase < 0.0) phase = two_pi + phase;
    // polarisation on the rotated beam axes (:329-352)
    double ax[3] = {1.0, 0.0, 0.0}, ay[3] = {0.0, 1.0, 0.0};
    if (ph != 0.0 || th != 0.0) {
        const double ex[3] = {1.0, 0.0, 0.0}, ey[3] = {0.0, 1.0, 0.0};
        euler_apply(PI_ / 2.0 + B.phi, B.theta, PI_ / 2.0 + B.phi, ex, ax);
        euler_apply(PI_ / 2.0 + B.phi, B.theta, PI_ / 2.0 + B.phi, ey, ay);
    }
    const double pxr = B.jxr * fabs(ax[0]) + B.jyr * fabs(ay[0]), pxi = B.jxi * fabs(ax[0]) + B.jyi * fabs(ay[0]);
    const double pyr = B.jyr * fabs(ay[1]) + B.jxr * fabs(ax[1]), pyi = B.jyi * fabs(ay[1]) + B.jxi * fabs(ax[1]);
    const double nrm = sqrt(pxr * pxr + pxi * pxi + pyr * pyr + pyi * pyi);
    // the plane wave as the right-hand side takes it (direction through its cartesian round trip)
    WaveDev W;
    double st_, ct_, sp_, cp_;
    sincos(th, &st_, &ct_);
    sincos(ph, &sp_, &cp_);
    W.kc[0] = k * st_ * cp_;
    W.kc[1] = k * st_ * sp_;
    W.kc[2] = k * ct_;
    const double r2 = sqrt(W.kc[0] * W.kc[0] + W.kc[1] * W.kc[1] + W.kc[2] * W.kc[2]);
    W.alpha = (r2 == 0.0) ? 0.0 : acos(W.kc[2] / r2);
    W.beta = (W.kc[0] == 0.0 && W.kc[1] == 0.0) ? 0.0 : atan2(W.kc[1], W.kc[0]);
    W.ax = hypot(pxr / nrm, pxi / nrm);
    W.phx = atan2(pxi / nrm, pxr / nrm) + phase;
    W.ay = hypot(pyr / nrm, pyi / nrm);
    W.phy = atan2(pyi / nrm, pyr / nrm) + phase;
    W.g = B.g * B.g;
    W.d0[0] = B.d0[0];
    W.d0[1] = B.d0[1];
    W.d0[2] = B.d0[2];
    out[t] = W;
}

// ---- layout conversion ---------------------------------------------------------------------
// reference flat layout (per sphere 2C entries, C = (pg+1)^2 - 1) <-> ragged scaled layout
__global__ void k_unpack(SceneView sc, int pg, const double* g, const cplx* xref, cplx* xdev) {
    int j = blockIdx.x;
    int pj = sc.p[j];
    int Pj = pj * (pj + 2);
    int C = (pg + 1) * (pg + 1) - 1;
    int64_t o = sc.off[j];
    for (int t = threadIdx.x; t < Pj; t += blockDim.x) {
        int n = (int)sqrt((double)(t + 1));
        if ((n + 1) * (n + 1) <= t + 1) ++n;
        if (n * n > t + 1) --n;
        int m = t + 1 - n * n - n;
        double rg = 1.0 / g[n * (n + 1) + m];
        xdev[o + t] = rg * xref[(size_t)2 * C * j + t];
        xdev[o + Pj + t] = rg * xref[(size_t)2 * C * j + C + t];
    }
}

// identity_ref != nullptr: entries above the sphere's own degree are copied from it (the
// identity rows of the reference operator); otherwise they are set to zero.
__global__ void k_pack(SceneView sc, int pg, const double* g, const cplx* ydev, const cplx* identity_ref,
                       cplx* yref) {
    int j = blockIdx.x;
    int pj = sc.p[j];
    int Pj = pj * (pj + 2);
    int C = (pg + 1) * (pg + 1) - 1;
    int64_t o = sc.off[j];
    for (int t = threadIdx.x; t < C; t += blockDim.x) {
        size_t ra = (size_t)2 * C * j + t, rb = ra + C;
        if (t < Pj) {
            int n = (int)sqrt((double)(t + 1));
            if ((n + 1) * (n + 1) <= t + 1) ++n;
            if (n * n > t + 1) --n;
            int m = t + 1 - n * n - n;
            double gv = g[n * (n + 1) + m];
            yref[ra] = gv * ydev[o + t];
            yref[rb] = gv * ydev[o + Pj + t];
        } else if (identity_ref) {
            yref[ra] = identity_ref[ra];
            yref[rb] = identity_ref[rb];
        } else {
            yref[ra] = mk(0, 0);
            yref[rb] = mk(0, 0);
        }
    }
}

// ---- cluster cross-sections, per sphere partial sums {ext, abs} ----------------------------
// In the scaled basis the reference weights n(n+1)(2n+1)(n-m)!/(n+m)! reduce to n(n+1)(2n+1).
__global__ void k_cross_sections(SceneView sc, const cplx* x, const cplx* pq, double* part) {
    int j = blockIdx.x;
    int pj = sc.p[j];
    int Pj = pj * (pj + 2);
    int64_t o = sc.off[j];
    double se = 0.0, sa = 0.0;
    for (int t = threadIdx.x; t < Pj; t += blockDim.x) {
        int n = (int)sqrt((double)(t + 1));
        if ((n + 1) * (n + 1) <= t + 1) ++n;
        if (n * n > t + 1) --n;
        double E = (double)(n * (n + 1) * (2 * n + 1));
        cplx a = x[o + t], bb = x[o + Pj + t];
        cplx p = pq[o + t], q = pq[o + Pj + t];
        cplx an = sc.an[(size_t)j * sc.pmax + n - 1], bn = sc.bn[(size_t)j * sc.pmax + n - 1];
        double ra = (an.x != 0.0 || an.y != 0.0) ? cdiv(mk(1, 0), an).x - 1.0 : 0.0;
        double rb = (bn.x != 0.0 || bn.y != 0.0) ? cdiv(mk(1, 0), bn).x - 1.0 : 0.0;
        se += E * ((conjg(p) * a).x + (conjg(q) * bb).x);
        sa += E * ((a.x * a.x + a.y * a.y) * ra + (bb.x * bb.x + bb.y * bb.y) * rb);
    }
    __shared__ double red[2][256];
    red[0][threadIdx.x] = se;
    red[1][threadIdx.x] = sa;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * j] = red[0][0];
        part[2 * j + 1] = red[1][0];
    }
}

// ---- scattered field at observation points (lib_mie_ms_get_field,
// FoggySim/src/lib/mie_theory/lib_mie_multi_sphere.f90:379-434; per sphere lib_mie_ss_get_field,
// lib_mie_single_sphere.f90:1397-1582; vector spherical wave functions of
// lib_math_vector_spherical_harmonics_components_real_xu,
// libmath/src/math/lib_math_vector_spherical_harmonics.f90:132-419) -------------------------------
//   E += sum_nm E_nm i (a_nm N_nm + b_nm M_nm),  H += n_medium / c0 sum_nm E_nm (b_nm N_nm + a_nm M_nm)
//   E_nm = |E0| (2n+1) (n-m)!/(n+m)! i^n, with h_n^(1) in M, N, per sphere in its own frame,
// converted to cartesian components and summed; zero at a point inside any sphere.
//
// One thread per point, one warp per 32 points and subset of the spheres, the subsets of a CTA's warps added in
// order, and with few points those of several CTAs (field_plan): a warp's lanes share the sphere, so its coefficients are one broadcast load, and the radial functions
// and Legendre rows sit in shared memory, one column per thread.  For each degree the angular sums over m,
//   A_P, A_tau, A_pi = sum_m (P, tau, pi) a'_m e^{i m phi} and B likewise, +m and -m together,
// come first and meet the radial factors once: 18 multiply-adds per coefficient, where forming M and N per (n, m)
// took about 110.  FP64-pipe bound.  46600 points x 71 spheres of order 5: 3.6 -> 0.79 ms (one CTA per point with its
// threads over the spheres before, 71 of 128 at work and the Bessel sequences in local memory).
namespace {
// j_n(x), n = 0..P, into out[n ld] (dev_sph_jn's recurrences with a stride)
__device__ __forceinline__ void sph_jn_column(double x, int P, double* out, int ld) {
    double s, c;
    sincos(x, &s, &c);
    const double rx = 1.0 / x;
    const double j0 = s * rx, j1 = (s * rx - c) * rx;
    if (x > (double)P) {
        double a = j0, b = j1;
        out[0] = j0;
        for (int n = 1; n <= P; ++n) {
            out[n * ld] = b;
            const double t = (2.0 * n + 1.0) * rx * b - a;
            a = b;
            b = t;
        }
        return;
    }
    const int start = P + 16 + (int)x + (int)sqrt(40.0 * (P + x));
    double fnp1 = 0.0, fn = 1e-300;
    for (int n = start; n >= 1; --n) {
        const double fnm1 = (2.0 * n + 1.0) * rx * fn - fnp1;
        if (n - 1 <= P) out[(n - 1) * ld] = fnm1;
        fnp1 = fn;
        fn = fnm1;
        if (fabs(fn) > 1e250) {
            fn *= 1e-250;
            fnp1 *= 1e-250;
            for (int k = n - 1; k <= P; ++k) out[k * ld] *= 1e-250;
        }
    }
    const double scale = (fabs(j0) >= fabs(j1)) ? j0 / out[0] : j1 / out[ld];
    for (int n = 0; n <= P; ++n) out[n * ld] *= scale;
}
// s += r z
__device__ __forceinline__ void axpy(cplx& s, double r, cplx z) {
    s.x = fma(r, z.x, s.x);
    s.y = fma(r, z.y, s.y);
}
}  // namespace

// The coefficients with what depends on (n, m) alone, a and b of one order side by side:
// (n-m)!/(n+m)! for m >= 0, (-1)^m for m < 0 (there it cancels against P_n^{-m}).
__global__ void k_field_coeff(int C, const cplx* x, cplx* ab) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const size_t j = blockIdx.x;
    for (int t = threadIdx.x; t < C; t += blockDim.x) {
        int n, m;
        decode_nm(t, n, m);
        double f = (m & 1) ? -1.0 : 1.0;
        if (m >= 0) {
            f = 1.0;
            for (int q = n - m + 1; q <= n + m; ++q) f *= (double)q;
            f = 1.0 / f;
        }
        ab[2 * (j * C + t)] = f * x[2 * j * C + t];
        ab[2 * (j * C + t) + 1] = f * x[2 * j * C + C + t];
    }
}

// the outputs of a point from its sums v[c ld]: E without its factor i, H without h_factor (real and imaginary parts of
// x, y, z), and the spheres' warps that found it inside
namespace {
__device__ __forceinline__ void field_store(const double* v, int ld, double h_factor, int ip, cplx* E_out, cplx* H_out) {
    const bool in = v[12 * ld] != 0.0;
    for (int c = 0; c < 3; ++c) {
        const cplx E = mk(-v[(2 * c + 1) * ld], v[2 * c * ld]);
        const cplx H = mk(h_factor * v[(6 + 2 * c) * ld], h_factor * v[(7 + 2 * c) * ld]);
        E_out[3 * (size_t)ip + c] = in ? mk(0.0, 0.0) : E;
        H_out[3 * (size_t)ip + c] = in ? mk(0.0, 0.0) : H;
    }
}
}  // namespace

// part given: the sums of this CTA's warps go there, [blockIdx.y][13][point]
__global__ void __launch_bounds__(512) k_field(SceneView sc, const double* radius_s, int pg, int C, const cplx* ab,
                                               int npoints, const double* pts, double e0, double h_factor, cplx* E_out,
                                               cplx* H_out, double* part) {
    extern __shared__ __align__(16) double field_smem[];
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = T >> 5;
    double* jb = field_smem + tid;                  // [pg + 2] j_n
    double* q1 = jb + (size_t)(pg + 2) * T;         // [pg + 1] Q_{n-1}^m (order 0: P_{n-1})
    double* q2 = q1 + (size_t)(pg + 1) * T;         // [pg + 1] of n - 2
    const int ip = blockIdx.x * 32 + lane;
    const int pi_ = ip < npoints ? ip : npoints - 1;
    const double p0 = pts[3 * (size_t)pi_], p1 = pts[3 * (size_t)pi_ + 1], p2 = pts[3 * (size_t)pi_ + 2];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");   // for the coefficients
    bool inside = false;
    double acc[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) acc[c] = 0.0;
    for (int j = blockIdx.y * warps + warp; j < sc.n; j += gridDim.y * warps) {
        const double d0 = p0 - sc.centres[3 * (size_t)j];
        const double d1 = p1 - sc.centres[3 * (size_t)j + 1];
        const double d2 = p2 - sc.centres[3 * (size_t)j + 2];
        const double r = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
        if (!(r > radius_s[j])) {
            inside = true;
            continue;
        }
        if (!(e0 > 1e-200)) continue;
        const double th = acos(d2 / r);
        double st, xc;
        sincos(th, &st, &xc);
        // the reference's pole table (lib_math_legendre.f90:854-920, without the phase): the limits of the general
        // functions, but for tau_{n,-1} of odd n at theta = pi, which has the opposite sign
        const bool pole = xc == 1.0 || xc == -1.0;
        const bool south = xc == -1.0;
        if (pole) st = 0.0;
        double sp = 0.0, cp = 1.0;
        if (d0 != 0.0 || d1 != 0.0) {
            const double m = fmax(fabs(d0), fabs(d1)), a = d0 / m, b = d1 / m, h = sqrt(a * a + b * b);
            cp = a / h;
            sp = b / h;
        }
        const double rho = sc.k * r, rr = 1.0 / rho;
        sph_jn_column(rho, pg + 1, jb, T);
        // y_{n-1}, y_n upwards (dev_sph_yn)
        double sr, cr;
        sincos(rho, &sr, &cr);
        double ym = -cr * rr, y = (-cr * rr - sr) * rr;
        double qmm = 1.0;                               // Q_n^n = (2n-1)!! sin^{n-1}
        q1[0] = 1.0;                                    // P_0
        q2[0] = 0.0;
        cplx es[3] = {mk(0, 0), mk(0, 0), mk(0, 0)}, hs[3] = {mk(0, 0), mk(0, 0), mk(0, 0)};
        const cplx* cj = ab + 2 * (size_t)j * C;
        for (int n = 1; n <= pg; ++n) {
            cplx aP = mk(0, 0), aT = mk(0, 0), aQ = mk(0, 0), bP = mk(0, 0), bT = mk(0, 0), bQ = mk(0, 0);
            const cplx* cn = cj + 2 * (n * n - 1 + n);
            if (n > 1) qmm *= (2.0 * n - 1.0) * st;
            cplx e = mk(cp, sp);
            for (int m = 1; m <= n; ++m) {
                // Q_n^m = P_n^m / sin t by the LPMNS recurrence; pi = m Q, tau = n x Q_n - (n + m) Q_{n-1}
                double q, qp = 0.0;
                if (m == n) {
                    q = qmm;
                } else {
                    qp = q1[m * T];
                    const double qpp = m == n - 1 ? 0.0 : q2[m * T];
                    q = ((2.0 * n - 1.0) * xc * qp - (n + m - 1.0) * qpp) / (double)(n - m);
                    q2[m * T] = qp;
                }
                q1[m * T] = q;
                const double P = q * st, pv = m * q, tv = n * xc * q - (n + m) * qp;
                const cplx ap = cn[2 * m], bp = cn[2 * m + 1], am = cn[-2 * m], bm = cn[-2 * m + 1];
                const cplx ga = e * ap, gb = e * bp, ha = conjg(e) * am, hb = conjg(e) * bm;
                const cplx sa = ga + ha, da = ga - ha, sb = gb + hb, db = gb - hb;
                const bool odd_south = south && m == 1 && (n & 1);
                axpy(aP, P, sa);
                axpy(aT, tv, odd_south ? da : sa);
                axpy(aQ, pv, da);
                axpy(bP, P, sb);
                axpy(bT, tv, odd_south ? db : sb);
                axpy(bQ, pv, db);
                if (m < n) e = e * mk(cp, sp);
                if (m == 1) {
                    // order 0: tau = -P_n^1
                    const cplx a0 = cn[0], b0 = cn[1];
                    const double pm = q1[0], pn = ((2.0 * n - 1.0) * xc * pm - (n - 1.0) * q2[0]) / (double)n;
                    q2[0] = pm;
                    q1[0] = pn;
                    const double P0 = pole ? ((south && (n & 1)) ? -1.0 : 1.0) : pn, t0 = -P;
                    axpy(aP, P0, a0);
                    axpy(aT, t0, a0);
                    axpy(bP, P0, b0);
                    axpy(bT, t0, b0);
                }
            }
            const double yp = (2.0 * n + 1.0) * rr * y - ym;   // y_{n+1}
            const cplx zn = mk(jb[n * T], y), zm = mk(jb[(n - 1) * T], ym), zp = mk(jb[(n + 1) * T], yp);
            ym = y;
            y = yp;
            const double f = e0 * (2.0 * n + 1.0);
            const cplx W = ipow_mul(n, f * zn);
            const cplx V = ipow_mul(n, (f * rr) * (0.5 * (rho * zm + zn - rho * zp)));
            const cplx Wr = ((double)(n * (n + 1)) * rr) * W;
            auto im = [](cplx z) { return mk(-z.y, z.x); };
            es[0] = es[0] + Wr * aP;
            es[1] = es[1] + (V * aT + W * im(bQ));
            es[2] = es[2] + (V * im(aQ) - W * bT);
            hs[0] = hs[0] + Wr * bP;
            hs[1] = hs[1] + (V * bT + W * im(aQ));
            hs[2] = hs[2] + (V * im(bQ) - W * aT);
        }
        // to cartesian components; E carries another i
        auto add = [&](const cplx* v, double* o) {
            const cplx x_ = st * cp * v[0] + xc * cp * v[1] - sp * v[2];
            const cplx y_ = st * sp * v[0] + xc * sp * v[1] + cp * v[2];
            const cplx z_ = xc * v[0] - st * v[1];
            o[0] += x_.x;
            o[1] += x_.y;
            o[2] += y_.x;
            o[3] += y_.y;
            o[4] += z_.x;
            o[5] += z_.y;
        };
        add(es, acc);
        add(hs, acc + 6);
    }
    // the warps' sums in order, through shared memory (one component at a time: one value per thread)
    double* red = field_smem;
    __syncthreads();
    red[tid] = inside ? 1.0 : 0.0;
    __syncthreads();
    bool in = false;
    for (int w = 0; w < warps; ++w) in |= red[w * 32 + lane] != 0.0;
    double sum[13];
    sum[12] = in ? 1.0 : 0.0;
    for (int c = 0; c < 12; ++c) {
        __syncthreads();
        red[tid] = acc[c];
        __syncthreads();
        double v = 0.0;
        for (int w = 0; w < warps; ++w) v += red[w * 32 + lane];
        sum[c] = v;
    }
    if (warp == 0 && ip < npoints) {
        if (!part) field_store(sum, 1, h_factor, ip, E_out, H_out);
        else
            for (int c = 0; c < 13; ++c) part[((size_t)blockIdx.y * 13 + c) * npoints + ip] = sum[c];
    }
}

// The CTAs' sums in order; 32 points per CTA, one warp per component (eight loads in flight: bound by their latency).
__global__ void __launch_bounds__(13 * 32) k_field_sum(int slabs, int npoints, const double* part, double h_factor,
                                                       cplx* E_out, cplx* H_out) {
    __shared__ double tot[13 * 32];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5, ip = blockIdx.x * 32 + lane;
    double v = 0.0;
    if (ip < npoints) {
#pragma unroll 8
        for (int k = 0; k < slabs; ++k) v += part[((size_t)k * 13 + c) * npoints + ip];
    }
    tot[threadIdx.x] = v;
    __syncthreads();
    if (c == 0 && ip < npoints) field_store(tot + lane, 32, h_factor, ip, E_out, H_out);
}

namespace {
size_t field_smem_bytes(int pg, int threads) { return (size_t)threads * (3 * pg + 4) * sizeof(double); }

// Warps per CTA: enough for 16 on every SM, four at least, no more than there are spheres or shared memory for.  Where
// that leaves half of the warps away (few points), CTAs of up to eight warps split the spheres, until the SMs
// are full or every warp has one sphere; slabs = CTAs per 32 points.  All spheres of 32 points in one CTA took 104 us for
// 1 to 100 points among 71 spheres of order 5 and 3.6 ms among 2000 of order 8, one CTA per point (the kernel before)
// 58 us and 1.24 ms, this 48 us and 0.094 ms.
struct FieldPlan {
    int blocks, warps, slabs;
};
FieldPlan field_plan(int n, int pg, int npoints) {
    FieldPlan f{(npoints + 31) / 32, 1, 1};
    const int all = 148 * 16;
    auto fit = [&](int w) {
        while (w > 1 && field_smem_bytes(pg, 32 * w) > ((size_t)200 << 10)) --w;
        return w;
    };
    f.warps = fit(std::max(std::min({16, n, (all + f.blocks - 1) / f.blocks}), std::min(4, n)));
    if ((int64_t)f.blocks * f.warps < all / 2 && f.warps < n) {
        const int w = std::min(f.warps, 8);
        const int64_t slabs = std::min<int64_t>((n + w - 1) / w, (all + (int64_t)f.blocks * w - 1) / (f.blocks * w));
        if (slabs > 1) {
            f.warps = w;
            f.slabs = (int)slabs;
        }
    }
    return f;
}
}  // namespace

size_t field_part(int n, int pg, int npoints) {
    const FieldPlan f = field_plan(n, pg, npoints);
    return f.slabs > 1 ? (size_t)f.slabs * 13 * npoints : 0;
}

void launch_field(const SceneView& sc, const double* radius_s, int pg, int C, const cplx* x, cplx* ab, int npoints,
                  const double* pts, double e0, double h_factor, cplx* E_out, cplx* H_out, double* part, cudaStream_t s) {
    const FieldPlan f = field_plan(sc.n, pg, npoints);
    const size_t smem = field_smem_bytes(pg, 32 * f.warps);
    raise_smem_ceiling(reinterpret_cast<const void*>(k_field), smem);
    k_field_coeff<<<sc.n, 128, 0, s>>>(C, x, ab);
    // each of the next two starts beside the one before and waits for its results
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(f.blocks, f.slabs);
    cfg.blockDim = dim3(32 * f.warps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (f.slabs == 1) part = nullptr;
    cudaLaunchKernelEx(&cfg, k_field, sc, radius_s, pg, C, (const cplx*)ab, npoints, pts, e0, h_factor, E_out, H_out, part);
    if (!part) return;
    cfg.gridDim = dim3(f.blocks);
    cfg.blockDim = dim3(13 * 32);
    cfg.dynamicSmemBytes = 0;
    cudaLaunchKernelEx(&cfg, k_field_sum, f.slabs, npoints, (const double*)part, h_factor, E_out, H_out);
}

}  // namespace foggy
