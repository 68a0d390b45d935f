// GLS vertical-mixing corrector: one thread per rho-interior water column.
//
// Restates the column physics of the reference's GLS pseudo-code (ROMS Fortran kept inside
// nonlinear/gls_corrector_step.py, which does not parse): production and dissipation with the
// buoyancy switch (:397-516), surface and bottom Dirichlet conditions (:526-564) from the wind
// stress and a quadratic bottom drag on the bottom-level velocity (nonlinear/set_vbc.py:19-41),
// the implicit tke and gls solves with their boundary fluxes (:568-656), the length-scale
// limitation, Galperin stability functions and the mixing coefficients (:662-825).  The new
// time level starts from Hz_w*tke(nstp) as the predictor leaves it without advection
// (nonlinear/gls_predictor_step.py:153-154).
#pragma once
#include "sf_internal.h"

namespace sf {

// Galperin et al. (1988) stability-function constants from the Mellor-Yamada A1, A2, B1,
// B2, C1 (published values), in the form the corrector evaluates (:740-748).
constexpr double kMyA1 = 0.92, kMyA2 = 0.74, kMyB1 = 16.6, kMyB2 = 10.1, kMyC1 = 0.08;
constexpr double kSh1 = kMyA2 * (1.0 - 6.0 * kMyA1 / kMyB1);
constexpr double kSh2 = 3.0 * kMyA2 * (6.0 * kMyA1 + kMyB2);
constexpr double kSm2 = 9.0 * kMyA1 * kMyA2;
constexpr double kSm3 = kMyA1 * (1.0 - 3.0 * kMyC1 - 6.0 * kMyA1 / kMyB1);
constexpr double kSm4 = 18.0 * kMyA1 * kMyA1 + 9.0 * kMyA1 * kMyA2;
constexpr double kGh0 = 0.0233, kGhcri = 0.02, kGhmin = -0.28;
constexpr double kVonKar = 0.41, kGlsEps = 1.0e-10;

template <typename R>
__device__ __forceinline__ R qpow(R a, R b) { return pow(a, b); }
template <>
__device__ __forceinline__ float qpow<float>(float a, float b) { return powf(a, b); }

// x^e for the models' exponents.  A multiple of 1/2 up to 8 (every exponent of k-epsilon and k-omega, the
// exponent m of the generic model) is products and one square root; others take pow.  The test is
// the same for every thread.
struct GlsExp {
    int h;       // 2 e, or kGlsPow
    double e;
};
constexpr int kGlsPow = 1 << 20;
inline GlsExp gls_exp(double e) {
    GlsExp x;
    x.e = e;
    x.h = e * 2.0 == floor(e * 2.0) && fabs(e) <= 8.0 ? (int)(2.0 * e) : kGlsPow;
    return x;
}
template <typename R>
__device__ __forceinline__ R gls_pow(R x, GlsExp e) {
    if (e.h == kGlsPow) return qpow(x, (R)e.e);
    const int a = e.h < 0 ? -e.h : e.h, n = a >> 1;
    R r = a & 1 ? sqrt(x) : R(1);
    if (n) {
        R q = x;
        if (n & 1) r *= q;
        if (n > 1) {
            q *= q;
            if (n & 2) r *= q;
            if (n > 3) {
                q *= q;
                if (n & 4) r *= q;
                if (n & 8) r *= q * q;
            }
        }
    }
    return e.h < 0 ? R(1) / r : r;
}

// gls_pow with 2 e known to the compiler (H), or read from e (kGlsPow).
template <int H, typename R>
__device__ __forceinline__ R gls_powc(R x, GlsExp e) {
    if constexpr (H == kGlsPow) {
        return gls_pow(x, e);
    } else {
        constexpr int a = H < 0 ? -H : H, n = a >> 1;
        static_assert(n <= 3, "x, x^2, x^3 and their halves");
        R r = n == 0 ? R(1) : n == 1 ? x : n == 2 ? x * x : x * (x * x);
        if constexpr (a & 1) r = n ? sqrt(x) * r : sqrt(x);
        return H < 0 ? R(1) / r : r;
    }
}

// The model's constants, evaluated once on the host in FP64 (a column evaluated a dozen powers of
// them), and its exponents.
template <typename R>
struct GlsConst {
    R dt, Kmin, Pmin, Akv_bak, Akt_bak, Akk_bak, Akp_bak, c1, c2, c3m, c3p, sigk, sigp, ogls_sigp, rdrag2;
    R cmu0, cmu_fac1, cmu_fac2, cmu_fac3, cmu0p, Zos, Zob, glsN, gls0, fluxt, fluxb;
    GlsExp m, n, in, mi, n1;   // m, n, 1/n, -1/n, n - 1
};
template <typename R>
GlsConst<R> gls_const(const sf_gls_params &P, double dt) {
    GlsConst<R> G;
    const double Zos = fmax(P.Zos, 1.0e-4), Zob = fmax(P.Zob, 1.0e-4), cp = pow(P.cmu0, P.p);
    G.dt = (R)dt;
    G.Kmin = (R)P.Kmin;
    G.Pmin = (R)P.Pmin;
    G.Akv_bak = (R)P.Akv_bak;
    G.Akt_bak = (R)P.Akt_bak;
    G.Akk_bak = (R)P.Akk_bak;
    G.Akp_bak = (R)P.Akp_bak;
    G.c1 = (R)P.c1;
    G.c2 = (R)P.c2;
    G.c3m = (R)P.c3m;
    G.c3p = (R)P.c3p;
    G.sigk = (R)P.sigk;
    G.sigp = (R)P.sigp;
    G.ogls_sigp = (R)(1.0 / P.sigp);
    G.rdrag2 = (R)P.rdrag2;
    G.cmu0 = (R)P.cmu0;
    G.cmu_fac1 = (R)pow(P.cmu0, -P.p / P.n);
    G.cmu_fac2 = (R)pow(P.cmu0, 3.0 + P.p / P.n);
    G.cmu_fac3 = (R)(1.0 / (P.cmu0 * P.cmu0));
    G.cmu0p = (R)cp;
    G.Zos = (R)Zos;
    G.Zob = (R)Zob;
    G.glsN = (R)(cp * pow(kVonKar * Zos, P.n));
    G.gls0 = (R)(cp * pow(kVonKar * Zob, P.n));
    G.fluxt = (R)(dt * cp * P.n * pow(kVonKar, P.n) * 0.5);
    G.fluxb = (R)(dt * cp * P.n * pow(kVonKar, P.n) * 0.5);
    G.m = gls_exp(P.m);
    G.n = gls_exp(P.n);
    G.in = gls_exp(1.0 / P.n);
    G.mi = gls_exp(-1.0 / P.n);
    G.n1 = gls_exp(P.n - 1.0);
    return G;
}

// One thread per column.  Bound: 76 bytes a point and level in FP32 (12 fields read, 7 written: 0.31 ms for
// 1026 x 514 x 50 at the copy bandwidth) and its instructions: the column used to take eight pow a
// level and seven local arrays (1.98 ms; FP64 generic model, 514 x 258 x 32: 0.84 ms).  Three passes:
//   down  production, dissipation and the elimination of both systems.  The gls surface flux needs
//         the solved tke: it enters the top row linearly, so a second right-hand side b (1 in the top
//         row, 0 below) is eliminated beside the first and scaled later.
//   up    tke.
//   up    gls and the coefficients.
// What a pass leaves for the next lies in the column's own outputs, whose old values have been used by
// then: CF and the eliminated tke in Akv and Akt, CF and the two right-hand sides of gls in Akk, gls
// and Akp.  Powers: with psi = cmu0^p k^m l^n, psi / k^m depends on l alone, so each of the dissipation,
// the length scale and the limited psi takes one power of l; the upper limit on l that stratification
// sets (a limit on psi in the reference's text) is compared as a length, without one.
// Blocks per SM: the levels are a chain of divisions and roots, so warps hide the latency, not loads in
// flight (levels in chunks of 4 at 128 registers: 0.97 and 0.41 ms for the two cases above; one at a
// time with 10 blocks at 48 registers in FP32, 7 at 72 in FP64, though these spill 16 and 72 bytes a thread: 0.76
// and 0.31, 0.68 and 0.30 now; 12 blocks 0.88).
template <typename R>
constexpr int gls_blocks() { return sizeof(R) == 4 ? 10 : 7; }
// KEPS: the exponents of k-epsilon, the default model (m = 3/2, n = -1), as constants: the branches on
// each exponent and its cases leave the level loops. 1024x512x50 FP32 0.760 ms -> 0.683, 512x256x32 FP64
// 0.231 -> 0.202; a model with other exponents takes the other variant (gen: 0.800 and 0.303).
template <typename R, typename Off, bool KEPS>
__global__ void __launch_bounds__(128, gls_blocks<R>()) k_gls_corrector(
    Geo<R> g, const GlsConst<R> G, const R *__restrict__ u, const R *__restrict__ v, const R *__restrict__ z_r,
    const R *__restrict__ Hz, const R *__restrict__ bvf, const R *__restrict__ sustr,
    const R *__restrict__ svstr, R *tke, R *gls, R *Akv, R *Akt, R *Akk, R *Akp, R *Lscale,
    const R *__restrict__ tkn0, const R *__restrict__ gln0, const uint8_t *__restrict__ sel,
    const int *__restrict__ list, const int *__restrict__ count) {
    constexpr int kM = KEPS ? 3 : kGlsPow, kN = KEPS ? -2 : kGlsPow, kI = KEPS ? -2 : kGlsPow,
                  kMi = KEPS ? 2 : kGlsPow, kN1 = KEPS ? -4 : kGlsPow;
    int pi = (int)tid_flat();
    if (list) {                    // a compacted list of columns: thread t takes list[t]
        if (pi >= *count) return;
        pi = list[pi];
    }
    if (pi >= g.s2) return;
    const int j = fdiv(pi, g.dI), i = pi - j * g.I;
    if (!rint_(i, j, g.I, g.J)) return;
    if (sel && !sel[pi]) return;   // column not selected: left as it is
    const Off p = (Off)pi, s2 = (Off)g.s2;
    const int I = g.I, N = g.N;
    const R dt = G.dt, Kmin = G.Kmin, Pmin = G.Pmin, eps = (R)kGlsEps;

    // --- down: levels N-1 .. 1
    Off o = p + (Off)(N - 1) * s2;   // W level k, rho level k + 1 in Fortran numbering
    R ut = u[o] , ute = u[o + 1], vt = v[o], vtn = v[o + I], zt = z_r[o], hzt = Hz[o];
    R akk = Akk[o], akp = Akp[o];
    const R akpN = Akp[o + s2] + akp, AkpB = Akp[p] + Akp[p + s2];
    R fk1 = R(0), fp1 = R(0);               // FCK, FCP of the level above
    R cfk = R(0), tk = R(0), cfp = R(0), ga = R(0), gb = R(0), cffp = R(0);   // its eliminated rows
    R top = R(1);
    for (int k = N - 1; k >= 1; --k) {
        const Off b = o - s2;
        const R ub = u[b], ube = u[b + 1], vb = v[b], vbn = v[b + I], zb = z_r[b], hb = Hz[b];
        const R kk = Akk[b], kp = Akp[b], av = Akv[o], at = Akt[o], tko = tke[o], glo = gls[o], strat2 = bvf[o];
        // vertical mixing of the turbulent fields (:401-415), none through the lowest layer
        const bool lowest = k == 1;
        const R fk = lowest ? R(0) : (R(-0.5) * dt) * (akk + kk) / hb;
        const R fp = lowest ? R(0) : (R(-0.5) * dt) * (akp + kp) / hb;
        // production and dissipation (:397-516)
        const R cff = R(0.5) / (zt - zb);
        const R du = (ut - ub) + (ute - ube), dv = (vt - vb) + (vtn - vbn);
        const R sh2 = (cff * du) * (cff * du) + (cff * dv) * (cff * dv);
        const R cffz = R(0.5) * (hb + hzt);
        const R c3 = strat2 > R(0) ? G.c3m : G.c3p;
        const R dAkt = at - G.Akt_bak, dAkv = av - G.Akv_bak, buo = strat2 * dAkt;
        R Kprod = sh2 * dAkv - buo;
        R Pprod = G.c1 * sh2 * dAkv - c3 * buo;
        R sk = R(0), sp = R(0);   // the buoyancy terms taken implicitly
        if (Kprod < R(0)) {
            Kprod = Kprod + buo;
            sk = buo;
        }
        if (Pprod < R(0)) {
            Pprod = Pprod + c3 * buo;
            sp = c3 * buo;
        }
        // the new level starts from tke/gls(nnew) after advection when given, else from
        // Hz_w * tke/gls(nstp) (the predictor's start without the advective terms)
        const R tr = (tkn0 ? tkn0[o] : cffz * tko) + dt * cffz * Kprod;
        const R gr = (gln0 ? gln0[o] : cffz * glo) + dt * cffz * Pprod * glo / fmax(tko, Kmin);
        const R diss = G.cmu_fac2 * gls_powc<kMi>(glo / gls_powc<kM>(tko, G.m), G.mi) * sqrt(tko);
        const R bck = cffz * (R(1) + dt * diss + dt * sk / tko) - fk - fk1;
        const R bcp = cffz * (R(1) + dt * G.c2 * diss + dt * sp / tko) - fp - fp1;
        // tke (:571-604) and gls (:608-656) eliminated
        const R ck = R(1) / (bck - cfk * fk1);
        cfk = ck * fk;
        tk = ck * (tr - fk1 * tk);
        cffp = R(1) / (bcp - cfp * fp1);
        cfp = cffp * fp;
        ga = cffp * (gr - fp1 * ga);
        gb = cffp * (top - fp1 * gb);
        top = R(0);
        Akv[o] = cfk;
        Akt[o] = tk;
        Akk[o] = cfp;
        gls[o] = ga;
        Akp[o] = gb;
        fk1 = fk;
        fp1 = fp;
        akk = kk;
        akp = kp;
        ut = ub;
        ute = ube;
        vt = vb;
        vtn = vbn;
        zt = zb;
        hzt = hb;
        o = b;
    }
    // surface and bottom conditions (:526-564); bottom stress on the bottom-level velocity
    auto bustr = [&](Off q) {
        const R va = R(0.25) * (v[q] + v[q + I] + v[q - 1] + v[q - 1 + I]);
        return G.rdrag2 * u[q] * sqrt(u[q] * u[q] + va * va);
    };
    auto bvstr = [&](Off q) {
        const R ua = R(0.25) * (u[q] + u[q + 1] + u[q - I] + u[q + 1 - I]);
        return G.rdrag2 * v[q] * sqrt(ua * ua + v[q] * v[q]);
    };
    const R su = sustr[p] + sustr[p + 1], sv = svstr[p] + svstr[p + I];
    const R bu = bustr(p) + bustr(p + 1), bv = bvstr(p) + bvstr(p + I);
    const R tkN = fmax(G.cmu_fac3 * R(0.5) * sqrt(su * su + sv * sv), Kmin);
    const R tk0 = fmax(G.cmu_fac3 * R(0.5) * sqrt(bu * bu + bv * bv), Kmin);
    const R glN = fmax(gls_powc<kM>(tkN, G.m) * G.glsN, Pmin);
    const R gl0 = fmax(G.gls0 * gls_powc<kM>(tk0, G.m), Pmin);
    // --- up: tke
    o = p + s2;
    tk = fmax(tk, Kmin);
    const R tk1 = tk;
    Akt[o] = tk;
    auto up = [&](auto nc) {
        constexpr int C = decltype(nc)::value;
        R a[C], f[C];
        Off l = o;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            l += s2;
            a[c] = Akt[l];
            f[c] = Akv[l];
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            o += s2;
            tk = fmax(a[c] - f[c] * tk, Kmin);
            Akt[o] = tk;
        }
    };
    in_chunks<4>(N - 2, up);
    // fluxes of gls through the surface and the bottom (:608-630)
    const R fluxt = G.fluxt * gls_powc<kM>(R(0.5) * (tkN + tk), G.m) *
                    gls_powc<kN1>(G.Zos + R(0.5) * Hz[p + (Off)(N - 1) * s2], G.n1) * akpN;
    const R fluxb = G.fluxb * gls_powc<kM>(R(0.5) * (tk0 + tk1), G.m) * gls_powc<kN1>(R(0.5) * Hz[p] + G.Zob, G.n1) * AkpB;
    // --- up: gls and the mixing coefficients (:662-825); the old values of a level are read before they
    // are written
    const R sqrt2 = sqrt(R(2));
    R gl = cffp * fluxb;   // level 1 takes the bottom flux as the term below it
    o = p + s2;
    for (int k = 1; k < N; ++k) {
        const R a = gls[o], b = Akp[o], f = Akk[o], t = Akt[o], b2 = bvf[o], ls = Lscale[o], to = tke[o];
        gl = (a - fluxt * b) - (k == 1 ? gl : f * gl);
        const R b2p = fmax(R(0), b2);
        const R tkn = fmax(t, Kmin), tm = gls_powc<kM>(tkn, G.m);
        const R Ls_gl = G.cmu_fac1 * gls_powc<kI>(fmax(gl, Pmin) / tm, G.in);
        const R Ls_unlmt = fmax(eps, fmin(Ls_gl, sqrt(R(0.56) * tkn) / (sqrt(b2p) + eps)));
        const R Ls = b2 > R(0) ? fmin(Ls_unlmt, sqrt(R(0.56) * tkn / (b2p + eps))) : Ls_unlmt;
        R Gh = fmin((R)kGh0, -b2 * Ls * Ls / (R(2) * tkn));
        Gh = fmin(Gh, Gh - (Gh - (R)kGhcri) * (Gh - (R)kGhcri) / (Gh + (R)kGh0 - R(2) * (R)kGhcri));
        Gh = fmax(Gh, (R)kGhmin);
        const R Sh = (R)kSh1 / (R(1) - (R)kSh2 * Gh);
        const R Sm = ((R)kSm3 + Sh * Gh * (R)kSm4) / (R(1) - (R)kSm2 * Gh);
        const R ql = sqrt2 * R(0.5) * (Ls * sqrt(tkn) + ls * sqrt(to));
        Akv[o] = G.Akv_bak + Sm * ql;
        Akt[o] = G.Akt_bak + Sh * ql;
        Akk[o] = G.Akk_bak + Sm * ql / G.sigk;
        Akp[o] = G.Akp_bak + Sm * ql * G.ogls_sigp;
        Lscale[o] = Ls;
        tke[o] = tkn;
        gls[o] = fmax(G.cmu0p * tm * gls_powc<kN>(Ls, G.n), Pmin);
        o += s2;
    }
    const R AvN = G.Akv_bak + (R)kVonKar * G.Zos * G.cmu0 * sqrt(tkN);
    const R Av0 = G.Akv_bak + (R)kVonKar * G.Zob * G.cmu0 * sqrt(tk0);
    Akv[o] = AvN;   // o is level N here
    Akv[p] = Av0;
    Akk[o] = G.Akk_bak + AvN / G.sigk;
    Akk[p] = G.Akk_bak + Av0 / G.sigk;
    Akp[o] = G.Akp_bak + AvN * G.ogls_sigp;
    Akp[p] = G.Akp_bak + Av0 / G.sigp;
    Akt[o] = G.Akt_bak;
    Akt[p] = G.Akt_bak;
    tke[o] = tkN;
    tke[p] = tk0;
    gls[o] = glN;
    gls[p] = gl0;
}


// ---------------------------------------------------------------------------------------------
// GLS predictor (nonlinear/gls_predictor_step.py:18-216, ROMS pseudo-code in the reference): the
// auxiliary advective half step of tke and gls at W levels 1..N-1 on the rho-interior points.
// Fourth-order centred horizontal fluxes FX/FE with the edge differences repeated at the domain
// edges (:62-127); the LF step interpolated back half a step with the AM3 weights cff1..cff3
// and the half-step box height Hz_half (:133-157); fourth-order vertical fluxes with the
// one-sided third-order forms at the bottom and surface (:162-208).  Also tke/gls(nnew) =
// Hz_w * tke/gls(nstp), the start of the corrector's update (:153-154).
// ---------------------------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ R vflux_(const R *q, const R *W, long p, long s2, int m, int N) {
    // FC at rho level m (1..N, Fortran numbering) of the W-level field q
#define Q(k) (q[(long)(k) * s2 + p])
    const R cf = R(0.5) * (W[(long)m * s2 + p] + W[(long)(m - 1) * s2 + p]);
    if (m == 1) return cf * (R(1.0 / 3.0) * Q(0) + R(5.0 / 6.0) * Q(1) - R(1.0 / 6.0) * Q(2));
    if (m == N)
        return cf * (R(1.0 / 3.0) * Q(N) + R(5.0 / 6.0) * Q(N - 1) - R(1.0 / 6.0) * Q(N - 2));
    return cf * (R(7.0 / 12.0) * (Q(m - 1) + Q(m)) - R(1.0 / 12.0) * (Q(m - 2) + Q(m + 1)));
#undef Q
}

// One tracer's horizontal flux divergence FX(i+1)-FX(i) + FE(j+1)-FE(j) at (i, j), level k.
template <typename R>
__device__ __forceinline__ R hdiv_(const R *q, const R *XF0, const R *XF1, const R *EF0,
                                   const R *EF1, long p, int i, int j, int I, int J, long s2,
                                   int k) {
    const R *qk = q + (long)k * s2;
    auto gx = [&](int m) -> R {   // grad(m) = q(m) - q(m-1), edges repeated
        m = m < 1 ? 1 : (m > I - 1 ? I - 1 : m);
        return qk[(long)j * I + m] - qk[(long)j * I + m - 1];
    };
    auto gy = [&](int m) -> R {
        m = m < 1 ? 1 : (m > J - 1 ? J - 1 : m);
        return qk[(long)m * I + i] - qk[(long)(m - 1) * I + i];
    };
    auto FX = [&](int a) -> R {   // at U point a of row j
        const long u = (long)j * I + a;
        const R xf = R(0.5) * (XF0[u] + XF1[u]);
        return xf * R(0.5) * (qk[u - 1] + qk[u] - R(1.0 / 6.0) * (gx(a + 1) - gx(a - 1)));
    };
    auto FE = [&](int b) -> R {   // at V point b of column i
        const long v = (long)b * I + i;
        const R ef = R(0.5) * (EF0[v] + EF1[v]);
        return ef * R(0.5) * (qk[v - I] + qk[v] - R(1.0 / 6.0) * (gy(b + 1) - gy(b - 1)));
    };
    (void)p;
    return (FX(i + 1) - FX(i)) + (FE(j + 1) - FE(j));
}

template <typename R>
__global__ void __launch_bounds__(128) k_gls_prestep(Geo<R> g, GlsPre c, const R *__restrict__ Huon,
        const R *__restrict__ Hvom, const R *__restrict__ W, const R *__restrict__ Hz,
        const R *__restrict__ tke0, const R *__restrict__ tkei, R *__restrict__ tke3,
        R *__restrict__ tken, const R *__restrict__ gls0, const R *__restrict__ glsi,
        R *__restrict__ gls3, R *__restrict__ glsn, R *__restrict__ Hz_half) {
    const int pi = (int)tid_flat();
    if (pi >= g.s2) return;
    const int I = g.I, J = g.J, N = g.N;
    const int i = pi % I, j = pi / I;
    if (i < 1 || i > I - 2 || j < 1 || j > J - 2) return;
    const long p = pi, s2 = g.s2;
    const R cff4 = (R)c.c3 * (g.pm[p] * g.pn[p]);
    R FCt = vflux_(tke0, W, p, s2, 1, N), FCg = vflux_(gls0, W, p, s2, 1, N);
    R CFk = R(0.5) * (W[s2 + p] + W[p]);
    for (int k = 1; k < N; ++k) {
        const R *XF0 = Huon + (long)(k - 1) * s2, *XF1 = Huon + (long)k * s2;
        const R *EF0 = Hvom + (long)(k - 1) * s2, *EF1 = Hvom + (long)k * s2;
        const long o = (long)k * s2 + p;
        const R cff = R(0.5) * (Hz[o - s2] + Hz[o]);
        const long u = (long)j * I + i, v = u;
        const R divUV = (R(0.5) * (XF0[u + 1] + XF1[u + 1]) - R(0.5) * (XF0[u] + XF1[u])) +
                        (R(0.5) * (EF0[v + I] + EF1[v + I]) - R(0.5) * (EF0[v] + EF1[v]));
        const R CFk1 = R(0.5) * (W[o + s2] + W[o]);
        R hh = cff - cff4 * divUV;
        hh = hh - cff4 * (CFk1 - CFk);
        const R FCt1 = vflux_(tke0, W, p, s2, k + 1, N), FCg1 = vflux_(gls0, W, p, s2, k + 1, N);
        const R ht = hdiv_(tke0, XF0, XF1, EF0, EF1, p, i, j, I, J, s2, k);
        const R hg = hdiv_(gls0, XF0, XF1, EF0, EF1, p, i, j, I, J, s2, k);
        const R t = (cff * ((R)c.c1 * tke0[o] + (R)c.c2 * tkei[o]) - cff4 * ht) - cff4 * (FCt1 - FCt);
        const R q = (cff * ((R)c.c1 * gls0[o] + (R)c.c2 * glsi[o]) - cff4 * hg) - cff4 * (FCg1 - FCg);
        tke3[o] = t / hh;
        gls3[o] = q / hh;
        tken[o] = cff * tke0[o];
        glsn[o] = cff * gls0[o];
        Hz_half[o] = hh;
        FCt = FCt1;
        FCg = FCg1;
        CFk = CFk1;
    }
    // the auxiliary level's bottom and surface values are the nstp ones (no advective update
    // there); the corrector's vertical fluxes at rho levels 1 and N read them
    tke3[p] = tke0[p];
    gls3[p] = gls0[p];
    tke3[(long)N * s2 + p] = tke0[(long)N * s2 + p];
    gls3[(long)N * s2 + p] = gls0[(long)N * s2 + p];
}

// Zero-gradient lateral condition on the auxiliary level (edges from the adjacent interior
// point, corners from the diagonal one), W levels 1..N-1.
template <typename R>
__global__ void k_gls_aux_bc(Geo<R> g, R *__restrict__ tke3, R *__restrict__ gls3) {
    const int I = g.I, J = g.J;
    const int nb = 2 * I + 2 * (J - 2);
    const long e = tid_flat();
    if (e >= (long)nb * (g.N - 1)) return;
    const int k = 1 + (int)(e / nb), b = (int)(e % nb);
    int i, j;
    if (b < I) { i = b; j = 0; }
    else if (b < 2 * I) { i = b - I; j = J - 1; }
    else if (b < 2 * I + J - 2) { i = 0; j = 1 + (b - 2 * I); }
    else { i = I - 1; j = 1 + (b - 2 * I - (J - 2)); }
    const int si = i == 0 ? 1 : (i == I - 1 ? I - 2 : i);
    const int sj = j == 0 ? 1 : (j == J - 1 ? J - 2 : j);
    const long o = (long)k * g.s2;
    tke3[o + (long)j * I + i] = tke3[o + (long)sj * I + si];
    gls3[o + (long)j * I + i] = gls3[o + (long)sj * I + si];
}

// ---------------------------------------------------------------------------------------------
// GLS corrector, advective terms (nonlinear/gls_corrector_step.py:172-388): tke/gls(nnew), the
// Hz_w-weighted new level the predictor starts, less the horizontal flux divergence of the
// auxiliary level (time level 3) — third-order upstream-biased fluxes whose curvature term
// comes from the upstream side of the W-level U/V flux, weighted by Gadv (:181-298; the
// one-sided differences repeated at the domain edges, :196-212, :253-268) — then floored at
// Kmin/Pmin (:300-317); then less the vertical flux divergence of the auxiliary level
// (fourth-order, with the one-sided third-order forms at the bottom and surface, :329-377) and
// floored again (:378-388).  W levels 1..N-1 on the rho-interior points.
// ---------------------------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ R hdiv_up3_(const R *qk, const R *XF0, const R *XF1, const R *EF0,
                                       const R *EF1, int i, int j, int I, int J, R gadv) {
    auto gx = [&](int m) -> R {   // grad(m) = q(m) - q(m-1), edges repeated
        m = m < 1 ? 1 : (m > I - 1 ? I - 1 : m);
        return qk[(long)j * I + m] - qk[(long)j * I + m - 1];
    };
    auto gy = [&](int m) -> R {
        m = m < 1 ? 1 : (m > J - 1 ? J - 1 : m);
        return qk[(long)m * I + i] - qk[(long)(m - 1) * I + i];
    };
    auto FX = [&](int a) -> R {   // at U point a of row j: curv(a-1) if the flux is eastward
        const long u = (long)j * I + a;
        const R xf = R(0.5) * (XF0[u] + XF1[u]);
        const R curv = xf > R(0) ? gx(a) - gx(a - 1) : gx(a + 1) - gx(a);
        return xf * R(0.5) * (qk[u - 1] + qk[u] - gadv * curv);
    };
    auto FE = [&](int b) -> R {   // at V point b of column i
        const long v = (long)b * I + i;
        const R ef = R(0.5) * (EF0[v] + EF1[v]);
        const R curv = ef > R(0) ? gy(b) - gy(b - 1) : gy(b + 1) - gy(b);
        return ef * R(0.5) * (qk[v - I] + qk[v] - gadv * curv);
    };
    return FX(i + 1) - FX(i) + FE(j + 1) - FE(j);
}

template <typename R>
__global__ void __launch_bounds__(128) k_gls_advect(Geo<R> g, R dt, R gadv, R Kmin, R Pmin,
        const R *__restrict__ Huon, const R *__restrict__ Hvom, const R *__restrict__ W,
        const R *__restrict__ tke3, const R *__restrict__ gls3, R *__restrict__ tken,
        R *__restrict__ glsn) {
    const int pi = (int)tid_flat();
    if (pi >= g.s2) return;
    const int I = g.I, J = g.J, N = g.N;
    const int i = pi % I, j = pi / I;
    if (i < 1 || i > I - 2 || j < 1 || j > J - 2) return;
    const long p = pi, s2 = g.s2;
    const R cff = dt * g.pm[p] * g.pn[p];
    R FCt = vflux_(tke3, W, p, s2, 1, N), FCg = vflux_(gls3, W, p, s2, 1, N);
    for (int k = 1; k < N; ++k) {
        const R *XF0 = Huon + (long)(k - 1) * s2, *XF1 = Huon + (long)k * s2;
        const R *EF0 = Hvom + (long)(k - 1) * s2, *EF1 = Hvom + (long)k * s2;
        const long o = (long)k * s2 + p;
        const R ht = hdiv_up3_(tke3 + (long)k * s2, XF0, XF1, EF0, EF1, i, j, I, J, gadv);
        const R hg = hdiv_up3_(gls3 + (long)k * s2, XF0, XF1, EF0, EF1, i, j, I, J, gadv);
        const R FCt1 = vflux_(tke3, W, p, s2, k + 1, N), FCg1 = vflux_(gls3, W, p, s2, k + 1, N);
        R t = fmax(tken[o] - cff * ht, Kmin);
        R q = fmax(glsn[o] - cff * hg, Pmin);
        t = fmax(t - cff * (FCt1 - FCt), Kmin);
        q = fmax(q - cff * (FCg1 - FCg), Pmin);
        tken[o] = t;
        glsn[o] = q;
        FCt = FCt1;
        FCg = FCg1;
    }
}

template <typename R>
cudaError_t Ops<R>::gls_advect(const sf_ctx *ctx, double dt, double gadv, double Kmin,
                               double Pmin, const R *Huon, const R *Hvom, const R *W,
                               const R *tke3, const R *gls3, R *tken, R *glsn, cudaStream_t s) {
    const Geo<R> g = geo(ctx);
    k_gls_advect<R><<<(unsigned)((g.s2 + 127) / 128), 128, 0, s>>>(
        g, (R)dt, (R)gadv, (R)Kmin, (R)Pmin, Huon, Hvom, W, tke3, gls3, tken, glsn);
    return cudaGetLastError();
}

template <typename R>
cudaError_t Ops<R>::gls_prestep(const sf_ctx *ctx, GlsPre c, const R *Huon, const R *Hvom,
                                const R *W, const R *Hz, const R *tke0, const R *tkei, R *tke3,
                                R *tken, const R *gls0, const R *glsi, R *gls3, R *glsn,
                                R *Hz_half, cudaStream_t s) {
    const Geo<R> g = geo(ctx);
    k_gls_prestep<R><<<(unsigned)((g.s2 + 127) / 128), 128, 0, s>>>(
        g, c, Huon, Hvom, W, Hz, tke0, tkei, tke3, tken, gls0, glsi, gls3, glsn, Hz_half);
    const long nb = (long)(2 * g.I + 2 * (g.J - 2)) * (g.N - 1);
    k_gls_aux_bc<R><<<(unsigned)((nb + 255) / 256), 256, 0, s>>>(g, tke3, gls3);
    return cudaGetLastError();
}

}  // namespace sf
