// fw_models_big.cuh -- the detailed ionic models: ten Tusscher-Panfilov 2006
// (TP06) and Courtemanche 1998, in the interface of fw_models.cuh.
//
// Template parameter T is the type of the potential, the gates, the
// currents and the concentration rates; the ion-concentration state (TP06:
// Ca_i, Ca_SR, Ca_ss, Na_i, K_i; Courtemanche: Na_i, K_i, Ca_i, Ca_up,
// Ca_rel; Luo-Rudy 1991: Ca_i) takes 8 bytes per node in both forms.  Under
// FW_F64 every quantity is float64, and the update comes twice: in a form
// with few divisions and exponentials (fw_math.cuh) for the potentials of a
// simulation, and in the reference's evaluation order, with CUDA's
// exp/log/sqrt/pow, for any other.  Under FW_F32 everything is computed in float32 from the
// concentrations rounded to float, and the accumulation `c += dt * rate`
// -- increments ~1e-6 of the value, below float32's resolution -- is
// compensated (CPair below), so no float64 arithmetic (a small fraction of
// GB300's float32 rate) is left in the per-node work.
//
// Reference quirks kept: TP06 never updates Ca_i (tp06_2d.py:1098 assigns the
// new value and then the old one); Courtemanche's IKr conductance is fixed
// at 0.0294 (courtemanche_2d.py:420-422) and the model's `xs` array is the
// IKr gate, `xr` the IKs gate (its run_ionic_kernel passes xr, xs to the
// kernel's xs, xr arguments, courtemanche_2d.py:152-160 against :581).
#pragma once

#include <math.h>
#include <stdint.h>

#include <initializer_list>

#include "fw_math.cuh"
#include "fw_models.cuh"

namespace fw {

// Host: the |u| below which an in-range update holds for a model's n
// parameters: 300 mV, less where an exponent slope * (|u| + u0) that they
// scale would leave 40, and 0 -- the reference-order update everywhere --
// where one of them is infinite, NaN or above 1e30, or one of `divisors`, by
// which a quotient is taken (dm::rcp needs a finite divisor other than zero,
// and a user may block a pump with a half-saturation of infinity), is not
// within 1e-30 .. 1e30.
inline double range_limit(const double *p, int n, std::initializer_list<int> divisors,
                          double slope, double u0)
{
    for (int i = 0; i < n; ++i)
        if (!(fabs(p[i]) <= 1e30)) return 0.0;
    for (int i : divisors)
        if (!(p[i] >= 1e-30)) return 0.0;
    const double lim = 40.0 / slope - u0;
    return lim < 300.0 ? lim : 300.0;
}

// Transcendentals of the reference-order updates.  float64: CUDA's exp / log / pow
// (the reference's expressions, within a few ulp of the C library).
// float32: the SFU forms (__expf, __logf: a few ulp, growing by about one
// ulp per unit of |x| for exp, CUDA's documented bound) and the integer and
// half-integer powers as products -- the float32 form is compared with
// float64 by tolerance, and these calls are most of its instructions.
__device__ __forceinline__ float mexp(float x) { return __expf(x); }
__device__ __forceinline__ double mexp(double x) { return exp(x); }
__device__ __forceinline__ float mlog(float x) { return __logf(x); }
__device__ __forceinline__ double mlog(double x) { return log(x); }
// x / (e^x - 1), continuous through x = 0 where it is 1.  Several rates are
// written in the reference as a difference quotient such as
// (u - u0) / (exp(k (u - u0)) - 1), which is 0 / 0 at u = u0; in float64
// that point is never met in practice, but in float32 the exponential
// rounds to exactly 1 within ~1e-6 mV of u0 and the quotient becomes
// inf or NaN.  The float32 forms use this function instead (series
// 1 - x / 2 for |x| < 1e-4, where the next term is below 1e-9).
__device__ __forceinline__ float x_expm1(float x)
{
    return fabsf(x) < 1e-4f ? 1.f - 0.5f * x : x / expm1f(x);
}

__device__ __forceinline__ float pow3(float x) { return x * x * x; }
__device__ __forceinline__ double pow3(double x) { return pow(x, 3.0); }
__device__ __forceinline__ float pow15(float x) { return x * sqrtf(x); }
__device__ __forceinline__ double pow15(double x) { return pow(x, 1.5); }

// Instantaneous buffering (Rapid buffer approximation): the free
// concentration c after adding d to the total c + B c / (c + K) solves
// c^2 + (B - T + K) c - K T = 0 with T = c0 + B c0 / (c0 + K) + d
// (tp06_2d.py:793-873).  With c = c0 + delta the constant term becomes
// -(c0 + K) d, so delta solves delta^2 + p delta - (c0 + K) d = 0 with
// p = c0 + K + B K / (c0 + K) - d; its root near zero, in the form without
// cancellation, is 2 (c0 + K) d / (p + sqrt(p^2 + 4 (c0 + K) d)).
__device__ __forceinline__ float buffered_step(float c0, float B, float K,
                                               float d)
{
    const float kc = c0 + K;
    const float p = kc + B * K * dm::rcp(kc) - d;
    const float q = kc * d;
    return 2.f * q * dm::rcp(p + sqrtf(fmaxf(p * p + 4.f * q, 0.f)));
}
// float64: the root's own form (sqrt(b^2 + 4 c) - b) / 2 would cancel four
// digits of the subspace calcium; sqrt as x / sqrt(x).  With p < 0 -- a
// concentration below -K, or one that more than doubles in the step -- the
// root's other form is the one without cancellation.
__device__ __forceinline__ double buffered_step(double c0, double B, double K,
                                                double d)
{
    const double kc = c0 + K;
    const double p = kc + B * K * dm::rcp(kc) - d;
    const double q = kc * d;
    const double s = p * p + 4.0 * q;
    if (__double2hiint(p) < 0 || __double2hiint(s) <= 0x00100000)
        return 0.5 * (sqrt(s) - p);
    return 2.0 * q * dm::rcp(p + s * dm::rsq(s));
}

// ---------------------------------------------------------------- accumulators
// The ion-concentration accumulators.  float64 form: a double.  float32
// form: a compensated pair of floats, the value hi + lo with |lo| at most
// half an ulp of hi (about 48 bits of mantissa), kept in the 8 bytes per
// node a double would take (float2 per node).  An increment d, ~1e-7 of the
// value and below float32's resolution of it, is added with Knuth's
// two-sum error-free transformation -- the rounding error of hi + d is
// recovered exactly and carried in lo -- so the accumulation runs on the
// float32 pipe (GB300's float64 rate is a small fraction of it).  The
// rates see the value rounded to float (hi).
struct CPair {
    float hi, lo;
    __device__ __forceinline__ explicit operator float() const { return hi; }
    __device__ __forceinline__ CPair &operator+=(float d)
    {
        const float s = hi + d;
        const float bp = s - hi;
        const float e = (hi - (s - bp)) + (d - bp);
        const float l = lo + e;
        hi = s + l;
        lo = l - (hi - s);
        return *this;
    }
};

template <class T>
struct ConcOf {
    using type = double;
};
template <>
struct ConcOf<float> {
    using type = CPair;
};
template <class T>
using Conc = typename ConcOf<T>::type;

__device__ __forceinline__ void conc_load(double &c, const void *a, int64_t p)
{
    c = ((const double *)a)[p];
}
__device__ __forceinline__ void conc_load(CPair &c, const void *a, int64_t p)
{
    const float2 v = ((const float2 *)a)[p];
    c.hi = v.x;
    c.lo = v.y;
}
__device__ __forceinline__ void conc_store(void *a, int64_t p, double c)
{
    ((double *)a)[p] = c;
}
__device__ __forceinline__ void conc_store(void *a, int64_t p, const CPair &c)
{
    ((float2 *)a)[p] = make_float2(c.hi, c.lo);
}
__device__ __forceinline__ double conc_probe(double c) { return c; }
__device__ __forceinline__ double conc_probe(const CPair &c)
{
    return (double)c.hi + (double)c.lo;
}

// ---------------------------------------------------------------- TP06
// Parameters in the order of tp06_2d.py's ionic_kernel_2d signature
// (:1003-1012); state in TP062D.state_vars order minus u (:77-79).
struct ModelTP06 {
    static constexpr int NS = 19, NP = 49;
    static constexpr int kMinBlocksF32 = 4;  // 64 registers, no spills
    enum {
        ko, cao, nao, Vc, Vsr, Vss, Bufc, Kbufc, Bufsr, Kbufsr, Bufss, Kbufss,
        Vmaxup, Kup, Vrel, k1_, k2_, k3, k4, EC, maxsr, minsr, Vleak, Vxfer, R,
        F, T_, RTONF, CAPACITANCE, gkr, pKNa, gk1, gna, gbna, KmK, KmNa, knak,
        gcal, gbca, knaca, KmNai, KmCa, ksat, n_, gpca, KpCa, gpk, gto, gks
    };
    enum { s_cai, s_casr, s_cass, s_nai, s_Ki, s_m, s_h, s_j, s_xr1, s_xr2,
           s_xs, s_r, s_s, s_d, s_f, s_f2, s_fcass, s_rr, s_oo };
    static constexpr bool is_conc(int i) { return i <= s_Ki; }

    template <class T>
    struct St {
        Conc<T> cai, casr, cass, nai, Ki;
        T m, h, j, xr1, xr2, xs, r, s, d, f, f2, fcass, rr, oo;
    };
    template <class T>
    __device__ static __forceinline__ St<T> load(void *const *S, int64_t p)
    {
        St<T> x;
        conc_load(x.cai, S[s_cai], p);
        conc_load(x.casr, S[s_casr], p);
        conc_load(x.cass, S[s_cass], p);
        conc_load(x.nai, S[s_nai], p);
        conc_load(x.Ki, S[s_Ki], p);
        x.m = ((const T *)S[s_m])[p];
        x.h = ((const T *)S[s_h])[p];
        x.j = ((const T *)S[s_j])[p];
        x.xr1 = ((const T *)S[s_xr1])[p];
        x.xr2 = ((const T *)S[s_xr2])[p];
        x.xs = ((const T *)S[s_xs])[p];
        x.r = ((const T *)S[s_r])[p];
        x.s = ((const T *)S[s_s])[p];
        x.d = ((const T *)S[s_d])[p];
        x.f = ((const T *)S[s_f])[p];
        x.f2 = ((const T *)S[s_f2])[p];
        x.fcass = ((const T *)S[s_fcass])[p];
        x.rr = ((const T *)S[s_rr])[p];
        x.oo = ((const T *)S[s_oo])[p];
        return x;
    }
    template <class T>
    __device__ static __forceinline__ void store(void *const *S, int64_t p,
                                                 const St<T> &x)
    {
        // Ca_i is not written: the reference never changes it
        conc_store(S[s_casr], p, x.casr);
        conc_store(S[s_cass], p, x.cass);
        conc_store(S[s_nai], p, x.nai);
        conc_store(S[s_Ki], p, x.Ki);
        ((T *)S[s_m])[p] = x.m;
        ((T *)S[s_h])[p] = x.h;
        ((T *)S[s_j])[p] = x.j;
        ((T *)S[s_xr1])[p] = x.xr1;
        ((T *)S[s_xr2])[p] = x.xr2;
        ((T *)S[s_xs])[p] = x.xs;
        ((T *)S[s_r])[p] = x.r;
        ((T *)S[s_s])[p] = x.s;
        ((T *)S[s_d])[p] = x.d;
        ((T *)S[s_f])[p] = x.f;
        ((T *)S[s_f2])[p] = x.f2;
        ((T *)S[s_fcass])[p] = x.fcass;
        ((T *)S[s_rr])[p] = x.rr;
        ((T *)S[s_oo])[p] = x.oo;
    }
    template <class T>
    __device__ static __forceinline__ double probe(const St<T> &x, int i)
    {
        switch (i) {
        case s_cai: return conc_probe(x.cai);
        case s_casr: return conc_probe(x.casr);
        case s_cass: return conc_probe(x.cass);
        case s_nai: return conc_probe(x.nai);
        case s_Ki: return conc_probe(x.Ki);
        case s_m: return x.m;
        case s_h: return x.h;
        case s_j: return x.j;
        case s_xr1: return x.xr1;
        case s_xr2: return x.xr2;
        case s_xs: return x.xs;
        case s_r: return x.r;
        case s_s: return x.s;
        case s_d: return x.d;
        case s_f: return x.f;
        case s_f2: return x.f2;
        case s_fcass: return x.fcass;
        case s_rr: return x.rr;
        default: return x.oo;
        }
    }

    // What depends on the parameters alone, computed on the host in float64
    // and appended to them (a dozen divisions, a logarithm and a square root
    // per node and step otherwise).
    enum {
        d_pkn = NP, d_gkr, d_kz, d_cal, d_kw, d_ncx, d_nao3, d_nak, d_naf, d_icf,
        d_ssf, d_vcss, d_vsrss, d_ec2, d_kup2, d_mec, d_lim, d_end
    };
    static constexpr int ND = d_end - NP;
    static void derive(const double *p, double dt, double *q)
    {
        const double RT = p[R] * p[T_];
        const double nao3 = p[nao] * p[nao] * p[nao];
        const double inverseVcF = 1.0 / (p[Vc] * p[F]);
        q[d_pkn] = p[ko] + p[pKNa] * p[nao];
        q[d_gkr] = p[gkr] * sqrt(p[ko] / 5.4);
        q[d_kz] = 2.0 * p[F] / RT;
        q[d_cal] = 2.0 * p[F] * p[gcal];
        q[d_kw] = p[F] / RT;
        q[d_ncx] = p[knaca] / (p[KmNai] * p[KmNai] * p[KmNai] + nao3) /
                   (p[KmCa] + p[cao]);
        q[d_nao3] = nao3 * 2.5;
        q[d_nak] = p[knak] * (p[ko] / (p[ko] + p[KmK]));
        q[d_naf] = dt * inverseVcF * p[CAPACITANCE];
        q[d_icf] = (double)(1.0f / ((float)p[Vc] * (float)p[F]));
        q[d_ssf] = p[CAPACITANCE] / (2.0 * p[Vss] * p[F]);
        q[d_vcss] = p[Vc] / p[Vss];
        q[d_vsrss] = p[Vsr] / p[Vss];
        q[d_ec2] = p[EC] * p[EC];
        q[d_kup2] = p[Kup] * p[Kup];
        q[d_mec] = p[maxsr] * p[EC] * p[EC];
        // exponents z = (u - 15) d_kz, n u d_kw, (n - 1) u d_kw and u d_kw,
        // d_kw = d_kz / 2
        const double n = fmax(fmax(fabs(p[n_]), fabs(p[n_] - 1.0)), 2.0);
        q[d_lim] = range_limit(p, NP,
                               {Vc, Vss, Kbufsr, Kbufss, Kup, k3, EC, maxsr, minsr, R, F,
                                T_, KmK, KmNa, KmNai, KmCa, KpCa, ko, cao, nao},
                               q[d_kw] * n, 15.0);
    }

    // ionic_kernel_2d and the calc_* helpers (tp06_2d.py:242-1103)
    template <class T>
    __device__ static __forceinline__ T update(T u, T un, St<T> &x,
                                               const Params<T, NP + ND> &P, T dt)
    {
        const T Ek = P.v[RTONF] * dm::lg(dm::quotient(P.v[ko], (T)x.Ki));
        // the range in which no exponential or product of them below leaves
        // T's (the squares (u + 25)^2 / 170 and the like set |u| < 300, which
        // is d_lim for parameters as they come), and states with which no
        // infinity meets a 0 in a product that a quotient would not have
        if (in_range(u, u - Ek, P.v[d_lim]) && regular(x))
            return update_in_range<T>(u, un, x, P, dt, Ek);
        return update_any<T>(u, un, x, P, dt);
    }
    __device__ static __forceinline__ bool in_range(double u, double x, double lim)
    {
        return fabs(u) < lim && x > -400.0 && x < 1000.0;
    }
    __device__ static __forceinline__ bool in_range(float u, float x, float lim)
    {
        return fabsf(u) < fminf(lim, 130.f) && x > -100.f && x < 1000.f;
    }
    __device__ static __forceinline__ bool regular(const St<double> &x)
    {
        return dm::all_normal((double)x.cai, (double)x.nai, (double)x.Ki) &&
               dm::all_finite((double)x.casr, (double)x.cass, x.m, x.h, x.j, x.xr1, x.xr2,
                              x.xs, x.r, x.s, x.d, x.f, x.f2, x.fcass, x.rr, x.oo);
    }
    // (float32: an infinite calcium, whose currents make the potential
    // infinite or NaN in this step in any form, is not looked for: 1 % of a
    // step)
    __device__ static __forceinline__ bool regular(const St<float> &) { return true; }

    // The update with few divisions and exponentials, in either precision:
    // every rate is written as one quotient -- 1 / (1 + e^-y) as e^y / (1 + e^y),
    // sums and products of such terms over their common denominator, rates
    // dt / tau instead of tau -- and in float64 the exponentials of one slope
    // share one evaluation (fw_math.cuh).  Against the form below (update_any,
    // the reference's order) the same mathematics in 918
    // instead of 2306 float64 instructions a warp of nodes and step (192 x 190
    // nodes: 61 against 150 us a step, the float64 pipe 81 and 83 % busy) and
    // 850 instead of 1070 instructions in all in float32 (256 x 256 x 40: 103
    // against 107 us, then bound by the latency of its loads).  Against 113-bit
    // arithmetic, one step from states of a tissue in activity, the rms error of
    // every variable is at most that of the reference's order (float64 m
    // 5.25e-17 of itself against 5.46e-17, oo 1.19e-16 against 1.29e-16, xs
    // 4.7e-17 against 1.5e-16; float32 Ki 9.71e-15 against 9.72e-15); the
    // subspace calcium, whose quadratic loses four digits in the reference's
    // form, is 56 times closer.
    template <class T>
    __device__ static __forceinline__ T update_in_range(T u, T un, St<T> &x,
                                                        const Params<T, NP + ND> &P,
                                                        T dt, T Ek)
    {
        using namespace dm;
        const T c1 = (T)1.0;
        const T ndt = sizeof(T) == 8 ? -dt : -dt * (T)kLog2e;
        const T cass = (T)x.cass, cai = (T)x.cai, casr = (T)x.casr;
        const T nai = (T)x.nai, Ki = (T)x.Ki;
        const T Ena = P.v[RTONF] * lg(quotient(P.v[nao], nai));
        const T Eks = P.v[RTONF] * lg(quotient(P.v[d_pkn], Ki + P.v[pKNa] * nai));
        const T Eca = (T)0.5 * P.v[RTONF] * lg(quotient(P.v[cao], cai));
        const Slope<T> g20 = FW_SLOPE(u, 20.0);
        const Slope<T> g10 = squared(g20), g5 = FW_SLOPE(u, 5.0);
        const Slope<T> g14 = FW_SLOPE(u, 14.0), g7 = squared(g14);
        const Slope<T> g15 = FW_SLOPE(u, 15.0), g75 = squared(g15);
        const Slope<T> g6 = FW_SLOPE(u, 6.0);

        // calc_ina
        T ina;
        {
            // a step is of the size of tau_m, so an error of rate_m is one of
            // m: no exponential common to numerator and denominator here
            const T da = c1 + FW_EX_OF(u + (T)60.0, -1 / 5.0);
            T eb;
            if constexpr (sizeof(T) == 8) eb = FW_AT(g5, -35.0, 5.0, 1096.6331584284585);
            else eb = FW_EX_OF(u + (T)35.0, 1 / 5.0);
            const T db = c1 + eb, dc = c1 + FW_EX_OF(u - (T)50.0, 1 / 200.0);
            const T rate_m = da * (db * dc) * rcp((T)0.1 * (db + dc));
            const T em = c1 + FW_EX(u + (T)56.86, -1 / 9.03);
            T rate_h, rate_j;
            if (u >= (T)(-40.0)) {
                rate_h = (T)(0.77 / 0.13) * rcp(c1 + FW_EX(u + (T)10.66, -1 / 11.1));
                const T q = FW_AT(g10, -32.0, 10.0, 24.53253019710935);
                rate_j = (T)0.6 * FW_EX(u, 0.057) * q * rcp(c1 + q);
            } else {
                rate_h = (T)0.057 * FW_EX(u + (T)80.0, -1 / 6.8) +
                         (T)2.7 * FW_EX(u, 0.079) + (T)310000.0 * FW_EX(u, 0.3485);
                rate_j = ((T)(-25428.0) * FW_EX(u, 0.2444) -
                          (T)6.948e-06 * FW_EX(u, -0.04391)) *
                             (u + (T)37.78) * rcp(c1 + FW_EX(u + (T)79.23, 0.311)) +
                         (T)0.02424 * FW_EX(u, -0.01052) *
                             rcp(c1 + FW_EX(u + (T)40.14, -0.1378));
            }
            const T rh = rcp_near(c1 + FW_EX(u + (T)71.55, 1 / 7.43));
            const T h_inf = rh * rh;
            x.m = gate_fast(x.m, rcp_near(em * em), ndt, rate_m);
            x.h = gate_to(x.h, h_inf, decay(ndt, rate_h));
            x.j = gate_to(x.j, h_inf, decay(ndt, rate_j));
            ina = P.v[gna] * x.m * x.m * x.m * x.h * x.j * (u - Ena);
        }
        // calc_ical
        T ical;
        {
            const T qd = FW_AT(g75, -8.0, 7.5, 2.9056777468820014);
            const T d_inf = qd * rcp(c1 + qd);
            const T a = FW_EX(u + (T)35.0, 1 / 13.0), da = c1 + a;
            const T db = c1 + FW_AT(g5, -5.0, 5.0, 2.718281828459045);
            const T c = FW_AT(g20, 50.0, 20.0, 0.0820849986238988), dc = c1 + c;
            const T rate_d = da * db * dc *
                             rcp(((T)1.65 * a + (T)0.25) * (T)1.4 * dc + c * da * db);
            const T f_inf = rcp(c1 + FW_AT(g7, -20.0, 7.0, 17.41170806332765));
            const T uf = u + (T)27.0;
            const T Af = (T)1102.5 * FW_EX(uf * uf, -1 / 225.0) + (T)20.0;
            const T q13 = FW_AT(g10, 13.0, 10.0, 0.2725317930340126), d13 = c1 + q13;
            const T d30 = c1 + FW_AT(g10, -30.0, 10.0, 20.085536923187668);
            const T rate_f = d13 * d30 *
                             rcp((Af * d13 + (T)200.0 * q13) * d30 + (T)180.0 * d13);
            const T f2_inf = (T)0.67 * rcp(c1 + FW_AT(g7, -35.0, 7.0, 148.4131591025766)) + (T)0.33;
            const T uf2 = u + (T)25.0;
            const T Af2 = (T)600.0 * FW_EX(uf2 * uf2, -1 / 170.0);
            const T q25 = FW_AT(g10, 25.0, 10.0, 0.0820849986238988), d25 = c1 + q25;
            const T rate_f2 = d25 * d30 *
                              rcp((Af2 * d25 + (T)31.0 * q25) * d30 + (T)16.0 * d25);
            const T cs = cass * (T)20.0, q = cs * cs;
            const T fcass_inf = (T)0.6 * rcp(c1 + q) + (T)0.4;
            const T rate_fcass = (c1 + q) * rcp((T)82.0 + (T)2.0 * q);
            x.d = gate_to(x.d, d_inf, decay(ndt, rate_d));
            x.f = gate_to(x.f, f_inf, decay(ndt, rate_f));
            x.f2 = gate_to(x.f2, f2_inf, decay(ndt, rate_f2));
            x.fcass = gate_to(x.fcass, fcass_inf, decay(ndt, rate_fcass));
            // 4 (u - 15) F^2 / RT / (e2 - 1) = 2 F z / (e^z - 1)
            const T z = (u - (T)15.0) * P.v[d_kz];
            const T e2 = ex(z);
            ical = P.v[d_cal] * x.d * x.f * x.f2 * x.fcass * x_over_expm1(z, e2) *
                   ((T)0.25 * e2 * cass - P.v[cao]);
        }
        // calc_ito
        T ito;
        {
            const T qr = FW_AT(g6, 20.0, 6.0, 0.035673993347252395);
            const T r_inf = qr * rcp(c1 + qr);
            const T s_inf = rcp(c1 + FW_AT(g5, -20.0, 5.0, 54.598150033144236));
            const T ur = u + (T)40.0, us = u + (T)45.0;
            const T rate_r = rcp((T)9.5 * FW_EX(ur * ur, -1 / 1800.0) + (T)0.8);
            const T ds = c1 + FW_AT(g5, 20.0, 5.0, 0.01831563888873418);
            const T rate_s =
                ds * rcp(((T)85.0 * FW_EX(us * us, -1 / 320.0) + (T)3.0) * ds + (T)5.0);
            x.s = gate_to(x.s, s_inf, decay(ndt, rate_s));
            x.r = gate_to(x.r, r_inf, decay(ndt, rate_r));
            ito = P.v[gto] * x.r * x.s * (u - Ek);
        }
        // calc_ikr
        T ikr;
        {
            const T q1 = FW_AT(g7, -26.0, 7.0, 41.029269993825565);
            const T xr1_inf = q1 * rcp(c1 + q1);
            const T q45 = FW_AT(g10, -45.0, 10.0, 90.01713130052181);
            const T rate_xr1 = (c1 + q45) * (c1 + FW_EX(u + (T)30.0, 1 / 11.5)) *
                               rcp((T)2700.0 * q45);
            const T xr2_inf = rcp(c1 + FW_EX(u + (T)88.0, 1 / 24.0));
            const T q60 = FW_AT(g20, -60.0, 20.0, 20.085536923187668);
            const T rate_xr2 = (c1 + q60) * (c1 + FW_AT(g20, 60.0, 20.0, 0.049787068367863944)) *
                               rcp((T)3.36 * q60);
            x.xr1 = gate_to(x.xr1, xr1_inf, decay(ndt, rate_xr1));
            x.xr2 = gate_to(x.xr2, xr2_inf, decay(ndt, rate_xr2));
            ikr = P.v[d_gkr] * x.xr1 * x.xr2 * (u - Ek);
        }
        // calc_iks
        T iks;
        {
            const T q = FW_AT(g6, 5.0, 6.0, 0.4345982085070782);   // 1 / sqrt(1 + 1 / q) = q / sqrt(q (1 + q))
            const T Axs = (T)1400.0 * q * rsq(q * (c1 + q));
            const T db = c1 + FW_AT(g15, 35.0, 15.0, 0.09697196786440507);
            const T rate_xs = db * rcp(Axs + (T)80.0 * db);
            const T qx = FW_AT(g14, -5.0, 14.0, 1.4292400324179777);
            x.xs = gate_to(x.xs, qx * rcp(c1 + qx), decay(ndt, rate_xs));
            iks = P.v[gks] * x.xs * x.xs * (u - Eks);
        }
        // calc_ik1: ak1 / (ak1 + bk1) times e^(-0.1 x) above and below
        const T ux = u - Ek;
        T ik1;
        {
            const T ip = FW_EX(ux, -0.1), ip2 = ip * ip;
            const T a = FW_EX(ux - (T)200.0, 0.06);
            const T e1 = FW_EX(ux + (T)100.0, 0.0002);
            // e^(-0.5 x): the fifth power, or on its own where that would
            // carry five times the error
            T ip5 = ip2 * ip2 * ip;
            if constexpr (sizeof(T) == 4) ip5 = FW_EX(ux, -0.5);
            const T g = (T)0.1 * (c1 + ip5) * ip;
            const T b = ((T)3.0 * e1 * ip + (T)0.36787944117144233) * (c1 + a);
            ik1 = P.v[gk1] * g * rcp(g + b) * ux;
        }
        // calc_inaca, calc_inak
        const T w = u * P.v[d_kw];
        const T eg = ex(P.v[n_] * w), em = ex(-w);
        const T rev = eg * em;
        const T inaca = P.v[d_ncx] *
                        (eg * (nai * nai * nai) * P.v[cao] - rev * P.v[d_nao3] * cai) *
                        rcp(c1 + P.v[ksat] * rev);
        const T inak = P.v[d_nak] * nai *
                       rcp((nai + P.v[KmNa]) *
                           (c1 + (T)0.1245 * FW_EX(w, -0.1) + (T)0.0353 * em));
        const T ipca = P.v[gpca] * cai * rcp(P.v[KpCa] + cai);
        const T ipk = P.v[gpk] * ux * rcp(c1 + FW_EX(u - (T)25.0, -1 / 5.98));
        const T ibna = P.v[gbna] * (u - Ena);
        const T ibca = P.v[gbca] * (u - Eca);
        // calc_irel: kCaSR = kr = kn / ks, kn = maxsr ks - (maxsr - minsr) casr^2
        // as a sum
        const T cs2 = casr * casr;
        const T ks = cs2 + P.v[d_ec2];
        const T kn = P.v[minsr] * cs2 + P.v[d_mec];
        const T kr = div_near(kn, ks);
        const T drr = P.v[k4] * (c1 - x.rr) - P.v[k2_] * kr * cass * x.rr;
        x.rr += dt * drr;
        const T kc = P.v[k1_] * cass * cass;
        x.oo = div_near(kc * x.rr, P.v[k3] * kr + kc);
        const T irel = P.v[Vrel] * x.oo * (casr - cass);
        const T ileak = P.v[Vleak] * (casr - cai);
        const T cai2 = cai * cai;
        const T iup = P.v[Vmaxup] * cai2 * rcp(cai2 + P.v[d_kup2]);
        const T ixfer = P.v[Vxfer] * (cass - cai);
        // calc_casr, calc_cass (tp06_2d.py:793-873), calc_nai, calc_ki
        // (:924-966); calc_cai is discarded by the reference
        const T dCaSR = dt * (iup - irel - ileak);
        const T dCaSS = dt * (irel * P.v[d_vsrss] - ixfer * P.v[d_vcss] -
                              ical * P.v[d_ssf]);
        const T dNai = -(ina + ibna + (T)3 * (inak + inaca)) * P.v[d_naf];
        T dKi = -(ik1 + ito + ikr + iks - (T)2 * inak + ipk);
        // float32: the three factors one by one.  A product formed on the host
        // is rounded once, but that rounding is an error of every increment,
        // and adds to those of the parameters where these offset them
        if constexpr (sizeof(T) == 4) dKi = dt * (dKi * P.v[d_icf] * P.v[CAPACITANCE]);
        else dKi *= P.v[d_naf];
        x.casr += buffered_step(casr, P.v[Bufsr], P.v[Kbufsr], dCaSR);
        x.cass += buffered_step(cass, P.v[Bufss], P.v[Kbufss], dCaSS);
        x.nai += dNai;
        x.Ki += dKi;
        return un - dt * (ikr + iks + ik1 + ito + ina + ibna + ical + ibca + inak +
                          inaca + ipca + ipk);
    }

    // The update in the reference's order, for potentials outside the range
    // above (a blown-up simulation).
    // (Copies go into the call, so that x and P keep to registers elsewhere.)
    template <class T>
    __device__ static __forceinline__ T update_any(T u, T un, St<T> &x,
                                                   const Params<T, NP + ND> &P, T dt)
    {
        St<T> y = x;
        Params<T, NP + ND> Q = P;
        un = update_call<T>(u, un, y, Q, dt);
        x = y;
        return un;
    }
    template <class T>
    __device__ static __noinline__ T update_call(T u, T un, St<T> &x,
                                                 const Params<T, NP + ND> &P, T dt)
    {
        return update_ref<T>(u, un, x, P, dt);
    }
    template <class T>
    __device__ static __forceinline__ T update_ref(T u, T un, St<T> &x,
                                                   const Params<T, NP + ND> &P, T dt)
    {
        const T c1 = (T)1.0;
        const T cass = (T)x.cass, cai = (T)x.cai, casr = (T)x.casr;
        const T nai = (T)x.nai, Ki = (T)x.Ki;
        const T inverseVcF = c1 / (P.v[Vc] * P.v[F]);
        const T inversevssF2 = c1 / ((T)2 * P.v[Vss] * P.v[F]);

        const T Ek = P.v[RTONF] * mlog(P.v[ko] / Ki);
        const T Ena = P.v[RTONF] * mlog(P.v[nao] / nai);
        const T Eks = P.v[RTONF] * mlog((P.v[ko] + P.v[pKNa] * P.v[nao]) /
                                          (Ki + P.v[pKNa] * nai));
        const T Eca = (T)0.5 * P.v[RTONF] * mlog(P.v[cao] / cai);

        // calc_ina
        T ina;
        {
            const T am = c1 / (c1 + mexp(((T)(-60.0) - u) / (T)5.0));
            const T beta_m = (T)0.1 / (c1 + mexp((u + (T)35.0) / (T)5.0)) +
                             (T)0.1 / (c1 + mexp((u - (T)50.0) / (T)200.0));
            const T tau_m = am * beta_m;
            const T e_m = mexp(((T)(-56.86) - u) / (T)9.03);
            const T m_inf = c1 / ((c1 + e_m) * (c1 + e_m));
            T alpha_h, beta_h, alpha_j, beta_j;
            if (u >= (T)(-40.0)) {
                alpha_h = (T)0;
                beta_h = (T)0.77 / ((T)0.13 * (c1 + mexp(-(u + (T)10.66) / (T)11.1)));
                alpha_j = (T)0;
                beta_j = (T)0.6 * mexp((T)0.057 * u) /
                         (c1 + mexp((T)(-0.1) * (u + (T)32.0)));
            } else {
                alpha_h = (T)0.057 * mexp(-(u + (T)80.0) / (T)6.8);
                beta_h = (T)2.7 * mexp((T)0.079 * u) +
                         (T)310000.0 * mexp((T)0.3485 * u);
                alpha_j = ((T)(-25428.0) * mexp((T)0.2444 * u) -
                           (T)6.948e-06 * mexp((T)(-0.04391) * u)) *
                          (u + (T)37.78) / (c1 + mexp((T)0.311 * (u + (T)79.23)));
                beta_j = (T)0.02424 * mexp((T)(-0.01052) * u) /
                         (c1 + mexp((T)(-0.1378) * (u + (T)40.14)));
            }
            const T tau_h = c1 / (alpha_h + beta_h);
            const T e_h = mexp((u + (T)71.55) / (T)7.43);
            const T h_inf = c1 / ((c1 + e_h) * (c1 + e_h));
            const T tau_j = c1 / (alpha_j + beta_j);
            const T j_inf = h_inf;
            x.m = m_inf - (m_inf - x.m) * mexp(-dt / tau_m);
            x.h = h_inf - (h_inf - x.h) * mexp(-dt / tau_h);
            x.j = j_inf - (j_inf - x.j) * mexp(-dt / tau_j);
            ina = P.v[gna] * x.m * x.m * x.m * x.h * x.j * (u - Ena);
        }
        // calc_ical
        T ical;
        {
            const T FF = P.v[F], RT = P.v[R] * P.v[T_];
            const T d_inf = c1 / (c1 + mexp(((T)(-8) - u) / (T)7.5));
            const T Ad = (T)1.4 / (c1 + mexp(((T)(-35) - u) / (T)13)) + (T)0.25;
            const T Bd = (T)1.4 / (c1 + mexp((u + (T)5) / (T)5));
            const T Cd = c1 / (c1 + mexp(((T)50 - u) / (T)20));
            const T tau_d = Ad * Bd + Cd;
            const T f_inf = c1 / (c1 + mexp((u + (T)20) / (T)7));
            const T Af = (T)1102.5 * mexp(-(u + (T)27) * (u + (T)27) / (T)225);
            const T Bf = (T)200.0 / (c1 + mexp(((T)13 - u) / (T)10.0));
            const T Cf = (T)180.0 / (c1 + mexp((u + (T)30) / (T)10)) + (T)20;
            const T tau_f = Af + Bf + Cf;
            const T f2_inf = (T)0.67 / (c1 + mexp((u + (T)35) / (T)7)) + (T)0.33;
            const T Af2 = (T)600 * mexp(-(u + (T)25) * (u + (T)25) / (T)170);
            const T Bf2 = (T)31 / (c1 + mexp(((T)25 - u) / (T)10));
            const T Cf2 = (T)16 / (c1 + mexp((u + (T)30) / (T)10));
            const T tau_f2 = Af2 + Bf2 + Cf2;
            const T q = cass / (T)0.05 * (cass / (T)0.05);
            const T fcass_inf = (T)0.6 / (c1 + q) + (T)0.4;
            const T tau_fcass = (T)80.0 / (c1 + q) + (T)2.0;
            x.d = d_inf - (d_inf - x.d) * mexp(-dt / tau_d);
            x.f = f_inf - (f_inf - x.f) * mexp(-dt / tau_f);
            x.f2 = f2_inf - (f2_inf - x.f2) * mexp(-dt / tau_f2);
            x.fcass = fcass_inf - (fcass_inf - x.fcass) * mexp(-dt / tau_fcass);
            const T z = (T)2 * (u - (T)15) * FF / RT;
            const T e2 = mexp(z);
            if constexpr (sizeof(T) == 8) {
                ical = P.v[gcal] * x.d * x.f * x.f2 * x.fcass * (T)4 *
                       (u - (T)15) * (FF * FF / RT) *
                       ((T)0.25 * e2 * cass - P.v[cao]) / (e2 - c1);
            } else {
                // 4 (u - 15) F^2 / RT / (e2 - 1) = 2 F z / (e^z - 1)
                ical = P.v[gcal] * x.d * x.f * x.f2 * x.fcass * (T)2 * FF *
                       x_expm1(z) * ((T)0.25 * e2 * cass - P.v[cao]);
            }
        }
        // calc_ito
        T ito;
        {
            const T r_inf = c1 / (c1 + mexp(((T)20 - u) / (T)6.0));
            const T s_inf = c1 / (c1 + mexp((u + (T)20) / (T)5.0));
            const T tau_r =
                (T)9.5 * mexp(-(u + (T)40.0) * (u + (T)40.0) / (T)1800.0) + (T)0.8;
            const T tau_s =
                (T)85.0 * mexp(-(u + (T)45.0) * (u + (T)45.0) / (T)320.0) +
                (T)5.0 / (c1 + mexp((u - (T)20.0) / (T)5.0)) + (T)3.0;
            x.s = s_inf - (s_inf - x.s) * mexp(-dt / tau_s);
            x.r = r_inf - (r_inf - x.r) * mexp(-dt / tau_r);
            ito = P.v[gto] * x.r * x.s * (u - Ek);
        }
        // calc_ikr
        T ikr;
        {
            const T xr1_inf = c1 / (c1 + mexp(((T)(-26.0) - u) / (T)7.0));
            const T axr1 = (T)450.0 / (c1 + mexp(((T)(-45.0) - u) / (T)10.0));
            const T bxr1 = (T)6.0 / (c1 + mexp((u - (T)(-30.0)) / (T)11.5));
            const T tau_xr1 = axr1 * bxr1;
            const T xr2_inf = c1 / (c1 + mexp((u - (T)(-88.0)) / (T)24.0));
            const T axr2 = (T)3.0 / (c1 + mexp(((T)(-60.0) - u) / (T)20.0));
            const T bxr2 = (T)1.12 / (c1 + mexp((u - (T)60.0) / (T)20.0));
            const T tau_xr2 = axr2 * bxr2;
            x.xr1 = xr1_inf - (xr1_inf - x.xr1) * mexp(-dt / tau_xr1);
            x.xr2 = xr2_inf - (xr2_inf - x.xr2) * mexp(-dt / tau_xr2);
            ikr = P.v[gkr] * fw_sqrt(P.v[ko] / (T)5.4) * x.xr1 * x.xr2 * (u - Ek);
        }
        // calc_iks
        T iks;
        {
            const T Axs = (T)1400.0 / fw_sqrt(c1 + mexp(((T)5.0 - u) / (T)6));
            const T Bxs = c1 / (c1 + mexp((u - (T)35.0) / (T)15.0));
            const T tau_xs = Axs * Bxs + (T)80;
            const T xs_inf = c1 / (c1 + mexp(((T)(-5.0) - u) / (T)14.0));
            x.xs = xs_inf - (xs_inf - x.xs) * mexp(-dt / tau_xs);
            iks = P.v[gks] * x.xs * x.xs * (u - Eks);
        }
        // calc_ik1
        const T ak1 = (T)0.1 / (c1 + mexp((T)0.06 * (u - Ek - (T)200)));
        const T bk1 = ((T)3.0 * mexp((T)0.0002 * (u - Ek + (T)100)) +
                       mexp((T)0.1 * (u - Ek - (T)10))) /
                      (c1 + mexp((T)(-0.5) * (u - Ek)));
        const T ik1 = P.v[gk1] * (ak1 / (ak1 + bk1)) * (u - Ek);
        // calc_inaca, calc_inak
        const T RT = P.v[R] * P.v[T_];
        const T inaca =
            P.v[knaca] *
            (c1 / (P.v[KmNai] * P.v[KmNai] * P.v[KmNai] +
                   P.v[nao] * P.v[nao] * P.v[nao])) *
            (c1 / (P.v[KmCa] + P.v[cao])) *
            (c1 / (c1 + P.v[ksat] * mexp((P.v[n_] - c1) * u * P.v[F] / RT))) *
            (mexp(P.v[n_] * u * P.v[F] / RT) * nai * nai * nai * P.v[cao] -
             mexp((P.v[n_] - c1) * u * P.v[F] / RT) * P.v[nao] * P.v[nao] *
                 P.v[nao] * cai * (T)2.5);
        const T rec_iNaK = c1 / (c1 + (T)0.1245 * mexp((T)(-0.1) * u * P.v[F] / RT) +
                                 (T)0.0353 * mexp(-u * P.v[F] / RT));
        const T inak = P.v[knak] * (P.v[ko] / (P.v[ko] + P.v[KmK])) *
                       (nai / (nai + P.v[KmNa])) * rec_iNaK;
        const T ipca = P.v[gpca] * cai / (P.v[KpCa] + cai);
        const T ipk = P.v[gpk] * (c1 / (c1 + mexp(((T)25 - u) / (T)5.98))) * (u - Ek);
        const T ibna = P.v[gbna] * (u - Ena);
        const T ibca = P.v[gbca] * (u - Eca);
        // calc_irel
        const T kCaSR = P.v[maxsr] - (P.v[maxsr] - P.v[minsr]) /
                                         (c1 + P.v[EC] / casr * (P.v[EC] / casr));
        const T k1 = P.v[k1_] / kCaSR;
        const T k2 = P.v[k2_] * kCaSR;
        const T drr = P.v[k4] * (c1 - x.rr) - k2 * cass * x.rr;
        x.rr += dt * drr;
        x.oo = k1 * cass * cass * x.rr / (P.v[k3] + k1 * cass * cass);
        const T irel = P.v[Vrel] * x.oo * (casr - cass);
        const T ileak = P.v[Vleak] * (casr - cai);
        const T iup = P.v[Vmaxup] / (c1 + P.v[Kup] * P.v[Kup] / (cai * cai));
        const T ixfer = P.v[Vxfer] * (cass - cai);
        // calc_casr, calc_cass (tp06_2d.py:793-873), calc_nai, calc_ki
        // (:924-966); calc_cai is discarded by the reference
        const T dCaSR = dt * (iup - irel - ileak);
        const T dCaSS = dt * (-ixfer * (P.v[Vc] / P.v[Vss]) +
                              irel * (P.v[Vsr] / P.v[Vss]) +
                              -ical * inversevssF2 * P.v[CAPACITANCE]);
        const T dNai = dt * (-(ina + ibna + (T)3 * inak + (T)3 * inaca) *
                             inverseVcF * P.v[CAPACITANCE]);
        const T dKi = dt * (-(ik1 + ito + ikr + iks - (T)2 * inak + ipk) *
                            inverseVcF * P.v[CAPACITANCE]);
        if constexpr (sizeof(T) == 8) {
            // the reference's quadratic for the free SR / subspace calcium
            const T CaCSQN = P.v[Bufsr] * casr / (casr + P.v[Kbufsr]);
            const T bjsr = P.v[Bufsr] - CaCSQN - dCaSR - casr + P.v[Kbufsr];
            const T cjsr = P.v[Kbufsr] * (CaCSQN + dCaSR + casr);
            const T CaSSBuf = P.v[Bufss] * cass / (cass + P.v[Kbufss]);
            const T bcss = P.v[Bufss] - CaSSBuf - dCaSS - cass + P.v[Kbufss];
            const T ccss = P.v[Kbufss] * (CaSSBuf + dCaSS + cass);
            x.casr = (fw_sqrt(bjsr * bjsr + 4 * cjsr) - bjsr) / 2;
            x.cass = (fw_sqrt(bcss * bcss + 4 * ccss) - bcss) / 2;
            x.nai += dNai;
            x.Ki += dKi;
        } else {
            // float32 rates, compensated accumulation: the new free calcium
            // is c0 + delta, delta the root near zero of the same quadratic
            // shifted to c0 (see buffered_step), so only the addition needs
            // the accumulator's precision
            x.casr += buffered_step(casr, P.v[Bufsr], P.v[Kbufsr], dCaSR);
            x.cass += buffered_step(cass, P.v[Bufss], P.v[Kbufss], dCaSS);
            x.nai += dNai;
            x.Ki += dKi;
        }
        return un - dt * (ikr + iks + ik1 + ito + ina + ibna + ical + ibca + inak +
                          inaca + ipca + ipk);
    }
};

// ---------------------------------------------------------------- Courtemanche
// Parameters in the order of courtemanche_2d.py's ionic_kernel_2d signature
// (:569-577); state in Courtemanche2D.state_vars order minus u (:118-120).
struct ModelCRN {
    static constexpr int NS = 21, NP = 39;
    static constexpr int kMinBlocksF32 = 3;  // 4 would spill
    enum {
        gna, gnab, gk1, gkr, gks, gto, gcal, gcab, gkur_coeff, F, T_, R, Vc, Vj,
        Vup, Vrel, ibk, cao, nao, ko, caupmax, kup, kmnai, kmko, kmnancx,
        kmcancx, ksatncx, kmcmdn, kmtrpn, kmcsqn, trpnmax, cmdnmax, csqnmax,
        inacamax, inakmax, ipcamax, krel, iupmax, kq10
    };
    enum { s_nai, s_ki, s_cai, s_caup, s_carel, s_m, s_h, s_j, s_d, s_f, s_oa,
           s_oi, s_ua, s_ui, s_xr, s_xs, s_fca, s_irel, s_vrel, s_urel, s_wrel };
    static constexpr bool is_conc(int i) { return i <= s_carel; }

    template <class T>
    struct St {
        Conc<T> nai, ki, cai, caup, carel;
        T m, h, j, d, f, oa, oi, ua, ui, xr, xs, fca, irel, vrel, urel, wrel;
    };
    template <class T>
    __device__ static __forceinline__ St<T> load(void *const *S, int64_t p)
    {
        St<T> x;
        conc_load(x.nai, S[s_nai], p);
        conc_load(x.ki, S[s_ki], p);
        conc_load(x.cai, S[s_cai], p);
        conc_load(x.caup, S[s_caup], p);
        conc_load(x.carel, S[s_carel], p);
        x.m = ((const T *)S[s_m])[p];
        x.h = ((const T *)S[s_h])[p];
        x.j = ((const T *)S[s_j])[p];
        x.d = ((const T *)S[s_d])[p];
        x.f = ((const T *)S[s_f])[p];
        x.oa = ((const T *)S[s_oa])[p];
        x.oi = ((const T *)S[s_oi])[p];
        x.ua = ((const T *)S[s_ua])[p];
        x.ui = ((const T *)S[s_ui])[p];
        x.xr = ((const T *)S[s_xr])[p];
        x.xs = ((const T *)S[s_xs])[p];
        x.fca = ((const T *)S[s_fca])[p];
        x.irel = ((const T *)S[s_irel])[p];
        x.vrel = ((const T *)S[s_vrel])[p];
        x.urel = ((const T *)S[s_urel])[p];
        x.wrel = ((const T *)S[s_wrel])[p];
        return x;
    }
    template <class T>
    __device__ static __forceinline__ void store(void *const *S, int64_t p,
                                                 const St<T> &x)
    {
        conc_store(S[s_nai], p, x.nai);
        conc_store(S[s_ki], p, x.ki);
        conc_store(S[s_cai], p, x.cai);
        conc_store(S[s_caup], p, x.caup);
        conc_store(S[s_carel], p, x.carel);
        ((T *)S[s_m])[p] = x.m;
        ((T *)S[s_h])[p] = x.h;
        ((T *)S[s_j])[p] = x.j;
        ((T *)S[s_d])[p] = x.d;
        ((T *)S[s_f])[p] = x.f;
        ((T *)S[s_oa])[p] = x.oa;
        ((T *)S[s_oi])[p] = x.oi;
        ((T *)S[s_ua])[p] = x.ua;
        ((T *)S[s_ui])[p] = x.ui;
        ((T *)S[s_xr])[p] = x.xr;
        ((T *)S[s_xs])[p] = x.xs;
        ((T *)S[s_fca])[p] = x.fca;
        ((T *)S[s_irel])[p] = x.irel;
        ((T *)S[s_vrel])[p] = x.vrel;
        ((T *)S[s_urel])[p] = x.urel;
        ((T *)S[s_wrel])[p] = x.wrel;
    }
    template <class T>
    __device__ static __forceinline__ double probe(const St<T> &x, int i)
    {
        switch (i) {
        case s_nai: return conc_probe(x.nai);
        case s_ki: return conc_probe(x.ki);
        case s_cai: return conc_probe(x.cai);
        case s_caup: return conc_probe(x.caup);
        case s_carel: return conc_probe(x.carel);
        case s_m: return x.m;
        case s_h: return x.h;
        case s_j: return x.j;
        case s_d: return x.d;
        case s_f: return x.f;
        case s_oa: return x.oa;
        case s_oi: return x.oi;
        case s_ua: return x.ua;
        case s_ui: return x.ui;
        case s_xr: return x.xr;
        case s_xs: return x.xs;
        case s_fca: return x.fca;
        case s_irel: return x.irel;
        case s_vrel: return x.vrel;
        case s_urel: return x.urel;
        default: return x.wrel;
        }
    }
    template <class T>
    __device__ static __forceinline__ T gate(T x, T x_inf, T tau, T dt)
    {
        return x_inf - (x_inf - x) * mexp(-dt / tau);
    }

    enum {
        d_rtf = NP, d_rtf2, d_kw, d_nak, d_ncx, d_nao3, d_leak, d_rfv, d_vru, d_upj,
        d_relj, d_fnr, d_fni, d_t1, d_t2, d_cs, d_lim, d_end
    };
    static constexpr int ND = d_end - NP;
    static void derive(const double *p, double, double *q)
    {
        const double RT = p[R] * p[T_], FVj = p[F] * p[Vj];
        q[d_rtf] = RT / p[F];
        q[d_rtf2] = RT / (2.0 * p[F]);
        q[d_kw] = p[F] / RT;
        q[d_nak] = p[inakmax] * (p[ko] / (p[ko] + p[kmko]));
        q[d_ncx] = p[inacamax] / ((p[kmnancx] * p[kmnancx] * p[kmnancx] +
                                   p[nao] * p[nao] * p[nao]) *
                                  (p[kmcancx] + p[cao]));
        q[d_nao3] = p[nao] * p[nao] * p[nao];
        q[d_leak] = p[iupmax] / p[caupmax];
        q[d_rfv] = 1.0 / FVj;
        q[d_vru] = p[Vrel] / p[Vup];
        q[d_upj] = p[Vup] / p[Vj];
        q[d_relj] = p[Vrel] / p[Vj];
        // Fn in units of 1.367e-15
        q[d_fnr] = 1e-12 * p[Vrel] / 1.367e-15;
        q[d_fni] = 5e-13 / p[F] / 1.367e-15;
        q[d_t1] = p[trpnmax] * p[kmtrpn];
        q[d_t2] = p[cmdnmax] * p[kmcmdn];
        q[d_cs] = p[csqnmax] * p[kmcsqn];
        // exponents up to u d_kw, and nao / 67.3
        q[d_lim] = range_limit(p, NP,
                               {F, T_, R, Vj, Vup, caupmax, kup, kmnai, kmko, kmnancx,
                                kmcancx, kmcmdn, kmtrpn, kmcsqn, cao, nao, ko},
                               q[d_kw], 0.0);
        if (p[nao] > 40.0 * 67.3) q[d_lim] = 0.0;
    }

    // ionic_kernel_2d and its helpers (courtemanche_2d.py:180-641)
    template <class T>
    __device__ static __forceinline__ T update(T u, T un, St<T> &x,
                                               const Params<T, NP + ND> &P, T dt)
    {
        if constexpr (sizeof(T) == 4) {
            // float32 keeps the reference's order and with it the bits of its
            // results: the rates of h jump by a quarter at u = -40, so a node
            // that meets the branch a step earlier for another rounding
            // differs by 1e-3 there
            return update_ref<T>(u, un, x, P, dt);
        } else {
            if (fabs(u) < P.v[d_lim] && regular(x)) return update_in_range(u, un, x, P, dt);
            return update_any(u, un, x, P, dt);
        }
    }

    __device__ static __forceinline__ bool regular(const St<double> &x)
    {
        return dm::all_normal((double)x.nai, (double)x.ki, (double)x.cai) &&
               dm::all_finite((double)x.caup, (double)x.carel, x.m, x.h, x.j, x.d, x.f,
                              x.oa, x.oi, x.ua, x.ui, x.xr, x.xs, x.fca, x.irel, x.vrel,
                              x.urel, x.wrel);
    }

    // As ModelTP06::update_in_range (float64 only): one quotient per rate.
    // 192 x 190 nodes: 66 against 180 us a step.
    __device__ static __forceinline__ double
    update_in_range(double u, double un, St<double> &x,
                    const Params<double, NP + ND> &P, double dt)
    {
        using namespace dm;
        using T = double;
        const T c1 = (T)1;
        const T ndt = -dt;
        const T cai = (T)x.cai, nai = (T)x.nai, carel = (T)x.carel;
        const T caup = (T)x.caup, ki = (T)x.ki;
        const T rnai = rcp(nai);
        const T ena = P.v[d_rtf] * lg(quotient(P.v[nao], nai));
        const T ek = P.v[d_rtf] * lg(quotient(P.v[ko], ki));
        const T eca = P.v[d_rtf2] * lg(quotient(P.v[cao], cai));
        const Slope<T> g17 = FW_SLOPE(u, 17.0), g85 = squared(g17);
        const T uk = u - ek;
        // calc_gating_m, calc_gating_h, calc_gating_j
        T ina;
        {
            const T z = (T)(-0.1) * (u + (T)47.13);
            T am = (T)3.2 * x_over_expm1(z, ex(z));
            if (u == (T)(-47.13)) am = (T)3.2;
            const T sm = am + (T)0.08 * FW_EX(u, -1 / 11.0);
            x.m = gate_fast(x.m, div_near(am, sm), ndt, sm);
            T h_inf = (T)0, j_inf = (T)0, rate_h, rate_j;
            if (u >= (T)(-40)) {
                rate_h = (T)(1 / 0.13) * rcp(c1 + FW_EX(u + (T)10.66, -1 / 11.1));
                // e^(-2.535e-7 u), |u| < 300: the series to the third power
                const T y = (T)(-2.535e-07) * u;
                const T ey = c1 + y * (c1 + y * ((T)0.5 + y * (T)(1 / 6.0)));
                rate_j = (T)0.3 * ey * rcp(c1 + FW_EX(u + (T)32, -0.1));
            } else {
                const T ah = (T)0.135 * FW_EX((T)80 + u, -1 / 6.8);
                rate_h = ah + (T)3.56 * FW_EX(u, 0.079) + (T)310000 * FW_EX(u, 0.35);
                h_inf = div_near(ah, rate_h);
                const T aj = ((T)(-127140) * FW_EX(u, 0.2444) -
                              (T)3.474e-05 * FW_EX(u, -0.04391)) *
                             (u + (T)37.78) * rcp(c1 + FW_EX(u + (T)79.23, 0.311));
                rate_j = aj + (T)0.1212 * FW_EX(u, -0.01052) *
                                  rcp(c1 + FW_EX(u + (T)40.14, -0.1378));
                j_inf = div_near(aj, rate_j);
            }
            x.h = gate_to(x.h, h_inf, decay(ndt, rate_h));
            x.j = gate_to(x.j, j_inf, decay(ndt, rate_j));
            ina = P.v[gna] * (x.m * x.m * x.m) * x.h * x.j * (u - ena);
        }
        const T ik1 = P.v[gk1] * uk * rcp(c1 + FW_EX(u + (T)80, 0.07));
        T ito, ikur;
        {
            const T q10 = FW_AT(g85, -10.0, 8.5, 3.242908421924544);   // e^-((u + 10) / 8.5) = 1 / q10
            const T da = c1 + q10 * FW_EX(u - (T)30, -1 / 59.0);
            const T db = (T)2.5 + FW_AT(g17, -82.0, 17.0, 124.40338763970256);
            const T rate_o = P.v[kq10] * (T)0.65 * (q10 * db + da) * rcp(da * db);
            const T E_o = decay(ndt, rate_o);
            const T o_inf = rcp(c1 + FW_EX(u + (T)20.47, -1 / 17.54));
            const T di = (T)18.53 + FW_EX(u + (T)113.7, 1 / 10.95);
            const T dj = (T)35.56 + FW_EX(u + (T)1.26, -1 / 7.44);
            const T rate_oi = P.v[kq10] * (di + dj) * rcp(di * dj);
            const T oi_inf = rcp(c1 + FW_EX(u + (T)43.1, 1 / 5.3));
            x.oa = gate_to(x.oa, o_inf, E_o);
            x.oi = gate_to(x.oi, oi_inf, decay(ndt, rate_oi));
            ito = P.v[gto] * (x.oa * x.oa * x.oa) * x.oi * uk;
            const T gkur = (T)0.005 + (T)0.05 * rcp(c1 + FW_EX(u - (T)15, -1 / 13.0));
            const T ua_inf = rcp(c1 + FW_EX(u + (T)30.3, -1 / 9.6));
            const T rate_ui = P.v[kq10] * (rcp((T)21 + FW_EX(u - (T)185, -1 / 28.0)) +
                                           FW_EX(u - (T)158, 1 / 16.0));
            const T ui_inf = rcp(c1 + FW_EX(u - (T)99.45, 1 / 27.48));
            x.ua = gate_to(x.ua, ua_inf, E_o);   // tau_ua is tau_o
            x.ui = gate_to(x.ui, ui_inf, decay(ndt, rate_ui));
            ikur = P.v[gkur_coeff] * gkur * (x.ua * x.ua * x.ua) * x.ui * uk;
        }
        T ikr, iks;
        {
            // the model's xs holds the IKr gate, xr the IKs gate
            const T za = (u + (T)14.1) * (T)(-1 / 5.0);
            const T zb = (u - (T)3.3328) * (T)(1 / 5.1237);
            const T rate_r = (T)(0.0003 * 5) * x_over_expm1(za, ex(za)) +
                             (T)(7.3898e-05 * 5.1237) * x_over_expm1(zb, ex(zb));
            const T xr_inf = rcp(c1 + FW_EX(u + (T)14.1, -1 / 6.5));
            x.xs = gate_to(x.xs, xr_inf, decay(ndt, rate_r));
            ikr = (T)0.0294 * x.xs * uk * rcp(c1 + FW_EX(u + (T)15, 1 / 22.4));
            const T zc = (u - (T)19.9) * (T)(-1 / 17.0);
            const T zd = (u - (T)19.9) * (T)(1 / 9.0);
            const T rate_s = (T)2 * ((T)(4e-05 * 17) * x_over_expm1(zc, ex(zc)) +
                                     (T)(3.5e-05 * 9) * x_over_expm1(zd, ex(zd)));
            const T xs_inf = rsq(c1 + FW_EX(u - (T)19.9, -1 / 12.7));
            x.xr = gate_to(x.xr, xs_inf, decay(ndt, rate_s));
            iks = P.v[gks] * (x.xr * x.xr) * uk;
        }
        T ical;
        {
            // 1 / tau_d = 0.035 (u + 10) (1 + e) / (1 - e), e = e^z
            const T u10 = u + (T)10;
            const T z = u10 * (T)(-1 / 6.24);
            const T e = ex(z);
            const T rate_d = (T)(0.035 * 6.24) * x_over_expm1(z, e) * (c1 + e);
            const T d_inf = rcp(c1 + FW_EX(u10, -1 / 8.0));
            const T rate_f = (T)(0.0197 / 9) * FW_EX(u10 * u10, -(0.0337 * 0.0337)) +
                             (T)(0.02 / 9);
            const T f_inf = rcp(c1 + FW_EX(u + (T)28, 1 / 6.9));
            const T fca_inf = (T)0.00035 * rcp((T)0.00035 + cai);
            x.d = gate_to(x.d, d_inf, decay(ndt, rate_d));
            x.f = gate_to(x.f, f_inf, decay(ndt, rate_f));
            x.fca = gate_to(x.fca, fca_inf, decay(ndt, (T)0.5));
            ical = P.v[gcal] * x.d * x.f * x.fca * (u - (T)65);
        }
        T inak, inaca;
        {
            const T w = u * P.v[d_kw];
            const T em = ex(-w), fwd = FW_EX(w, 0.35), rev = fwd * em;
            const T s = (T)(1 / 7.0) * (ex(P.v[nao] * (T)(1 / 67.3)) - c1);
            const T dn = c1 + (T)0.1245 * FW_EX(w, -0.1) + (T)0.0365 * s * em;
            // (kmnai / nai)^1.5
            const T q = P.v[kmnai] * rnai;
            inak = P.v[d_nak] * rcp(dn * (c1 + q * q * rsq(q)));
            inaca = P.v[d_ncx] *
                    (fwd * (nai * nai * nai) * P.v[cao] - rev * P.v[d_nao3] * cai) *
                    rcp(c1 + P.v[ksatncx] * rev);
        }
        const T ibca = P.v[gcab] * (u - eca);
        const T ibna = P.v[gnab] * (u - ena);
        const T ipca = P.v[ipcamax] * cai * rcp(cai + (T)0.0005);
        {
            // Fn / 1.367e-15; the steps at 3.4175e-13 and 6.835e-14 are 250
            // and 50 of these units
            const T fn = P.v[d_fnr] * x.irel -
                         P.v[d_fni] * ((T)0.5 * ical - (T)0.2 * inaca);
            const T u_inf = rcp(c1 + ex_limited((T)250 - fn));
            const T tau_v = (T)1.91 + (T)2.09 * u_inf;
            const T v_inf = c1 - rcp(c1 + ex_limited((T)50 - fn));
            // 1 / tau_w = (1 + 0.3 e) (u - 7.9) / (6 (1 - e)), e = e^z
            const T z = (u - (T)7.9) * (T)(-1 / 5.0);
            const T e = ex(z);
            const T rate_w = (T)(5.0 / 6.0) * (c1 + (T)0.3 * e) * x_over_expm1(z, e);
            const T w_inf = c1 - rcp(c1 + FW_EX(u - (T)40, -1 / 17.0));
            x.urel = gate_to(x.urel, u_inf, decay(ndt, (T)0.125));
            x.vrel = gate_to(x.vrel, v_inf, decay(ndt, rcp(tau_v)));
            x.wrel = gate_to(x.wrel, w_inf, decay(ndt, rate_w));
            x.irel = P.v[krel] * (x.urel * x.urel) * x.vrel * x.wrel * (carel - cai);
        }
        const T itr = (caup - carel) * (T)(1 / 180.0);
        const T iup = P.v[iupmax] * cai * rcp(cai + P.v[kup]);
        const T iupleak = caup * P.v[d_leak];
        // calc_caup, calc_nai, calc_ki, calc_cai, calc_carel
        // (courtemanche_2d.py:219-253)
        x.caup += dt * (iup - iupleak - itr * P.v[d_vru]);
        x.nai += dt * (((T)(-3) * (inak + inaca) - ibna - ina) * P.v[d_rfv]);
        x.ki += dt * (((T)2 * inak - ik1 - ito - ikur - ikr - iks - P.v[ibk]) *
                      P.v[d_rfv]);
        const T B1 = ((T)2 * inaca - ipca - ical - ibca) * ((T)0.5 * P.v[d_rfv]) +
                     (iupleak - iup) * P.v[d_upj] + x.irel * P.v[d_relj];
        const T k1 = cai + P.v[kmtrpn], k2 = cai + P.v[kmcmdn];
        const T q1 = k1 * k1, q2 = k2 * k2, q12 = q1 * q2;
        x.cai += dt * (B1 * q12 * rcp(q12 + P.v[d_t1] * q2 + P.v[d_t2] * q1));
        const T k3 = carel + P.v[kmcsqn], q3 = k3 * k3;
        x.carel += dt * ((itr - x.irel) * q3 * rcp(q3 + P.v[d_cs]));
        return un - dt * (ina + ik1 + ito + ikur + ikr + iks + ical + ipca + inak +
                          inaca + ibna + ibca);
    }

    // The update in the reference's order, for potentials outside the range
    // above.
    // (Copies go into the call, so that x and P keep to registers elsewhere.)
    __device__ static __forceinline__ double update_any(double u, double un, St<double> &x,
                                                        const Params<double, NP + ND> &P,
                                                        double dt)
    {
        St<double> y = x;
        Params<double, NP + ND> Q = P;
        un = update_call(u, un, y, Q, dt);
        x = y;
        return un;
    }
    __device__ static __noinline__ double update_call(double u, double un, St<double> &x,
                                                      const Params<double, NP + ND> &P,
                                                      double dt)
    {
        return update_ref<double>(u, un, x, P, dt);
    }
    template <class T>
    __device__ static __forceinline__ T update_ref(T u, T un, St<T> &x,
                                                   const Params<T, NP + ND> &P, T dt)
    {
        const T c1 = (T)1;
        const T cai = (T)x.cai, nai = (T)x.nai, carel = (T)x.carel;
        const T caup = (T)x.caup, ki = (T)x.ki;
        const T RTF = P.v[R] * P.v[T_] / P.v[F];
        const T ena = RTF * mlog(P.v[nao] / nai);
        const T ek = RTF * mlog(P.v[ko] / ki);
        const T eca = P.v[R] * P.v[T_] / ((T)2 * P.v[F]) * mlog(P.v[cao] / cai);
        // calc_gating_m, calc_gating_h, calc_gating_j
        {
            T am;
            if constexpr (sizeof(T) == 8) {
                if (u == (T)(-47.13))
                    am = (T)3.2;
                else
                    am = (T)0.32 * (u + (T)47.13) /
                         (c1 - mexp((T)(-0.1) * (u + (T)47.13)));
            } else {
                am = (T)3.2 * x_expm1((T)(-0.1) * (u + (T)47.13));
            }
            const T bm = (T)0.08 * mexp(-u / (T)11);
            x.m = gate(x.m, am / (am + bm), c1 / (am + bm), dt);
            T ah = (T)0.135 * mexp(-((T)80 + u) / (T)6.8);
            T bh = (T)3.56 * mexp((T)0.079 * u) + (T)310000 * mexp((T)0.35 * u);
            T aj = ((T)(-127140) * mexp((T)0.2444 * u) -
                    (T)3.474e-05 * mexp((T)(-0.04391) * u)) *
                   (u + (T)37.78) / (c1 + mexp((T)0.311 * (u + (T)79.23)));
            T bj = (T)0.1212 * mexp((T)(-0.01052) * u) /
                   (c1 + mexp((T)(-0.1378) * (u + (T)40.14)));
            if (u >= (T)(-40)) {
                ah = (T)0;
                bh = c1 / ((T)0.13 * (c1 + mexp(-(u + (T)10.66) / (T)11.1)));
                aj = (T)0;
                bj = (T)0.3 * mexp((T)(-2.535e-07) * u) /
                     (c1 + mexp((T)(-0.1) * (u + (T)32)));
            }
            x.h = gate(x.h, ah / (ah + bh), c1 / (ah + bh), dt);
            const T j_inf = aj / (aj + bj);
            const T tau_j = c1 / (aj + bj);
            x.j = j_inf - (j_inf - x.j) * mexp(-dt / tau_j);
        }
        const T ina = P.v[gna] * pow3(x.m) * x.h * x.j * (u - ena);
        const T ik1 = P.v[gk1] * (u - ek) / (c1 + mexp((T)0.07 * (u + (T)80)));
        T ito, ikur;
        {
            const T ao = (T)0.65 / (mexp(-(u + (T)10) / (T)8.5) +
                                    mexp(-(u - (T)30) / (T)59.0));
            const T bo = (T)0.65 / ((T)2.5 + mexp((u + (T)82) / (T)17.0));
            const T tau_o = c1 / (P.v[kq10] * (ao + bo));
            const T o_inf = c1 / (c1 + mexp(-(u + (T)20.47) / (T)17.54));
            const T aoi = c1 / ((T)18.53 + mexp((u + (T)113.7) / (T)10.95));
            const T boi = c1 / ((T)35.56 + mexp(-(u + (T)1.26) / (T)7.44));
            const T tau_oi = c1 / (P.v[kq10] * (aoi + boi));
            const T oi_inf = c1 / (c1 + mexp((u + (T)43.1) / (T)5.3));
            x.oa = gate(x.oa, o_inf, tau_o, dt);
            x.oi = gate(x.oi, oi_inf, tau_oi, dt);
            ito = P.v[gto] * pow3(x.oa) * x.oi * (u - ek);
            const T gkur = (T)0.005 + (T)0.05 / (c1 + mexp(-(u - (T)15) / (T)13.0));
            const T tau_ua = c1 / (P.v[kq10] * (ao + bo));
            const T ua_inf = c1 / (c1 + mexp(-(u + (T)30.3) / (T)9.6));
            const T aui = c1 / ((T)21 + mexp(-(u - (T)185) / (T)28.0));
            const T bui = mexp((u - (T)158) / (T)16.0);
            const T tau_ui = c1 / (P.v[kq10] * (aui + bui));
            const T ui_inf = c1 / (c1 + mexp((u - (T)99.45) / (T)27.48));
            x.ua = gate(x.ua, ua_inf, tau_ua, dt);
            x.ui = gate(x.ui, ui_inf, tau_ui, dt);
            ikur = P.v[gkur_coeff] * gkur * pow3(x.ua) * x.ui * (u - ek);
        }
        T ikr, iks;
        {
            // the model's xs holds the IKr gate, xr the IKs gate
            T axr, bxr;
            if constexpr (sizeof(T) == 8) {
                axr = (T)0.0003 * (u + (T)14.1) /
                      (c1 - mexp(-(u + (T)14.1) / (T)5));
                bxr = (T)7.3898e-05 * (u - (T)3.3328) /
                      (mexp((u - (T)3.3328) / (T)5.1237) - c1);
            } else {
                axr = (T)(0.0003 * 5) * x_expm1(-(u + (T)14.1) / (T)5);
                bxr = (T)(7.3898e-05 * 5.1237) *
                      x_expm1((u - (T)3.3328) / (T)5.1237);
            }
            const T tau_xr = c1 / (axr + bxr);
            const T xr_inf = c1 / (c1 + mexp(-(u + (T)14.1) / (T)6.5));
            x.xs = gate(x.xs, xr_inf, tau_xr, dt);
            ikr = (T)0.0294 * x.xs * (u - ek) / (c1 + mexp((u + (T)15) / (T)22.4));
            T axs, bxs;
            if constexpr (sizeof(T) == 8) {
                axs = (T)4e-05 * (u - (T)19.9) /
                      (c1 - mexp(-(u - (T)19.9) / (T)17));
                bxs = (T)3.5e-05 * (u - (T)19.9) /
                      (mexp((u - (T)19.9) / (T)9) - c1);
            } else {
                axs = (T)(4e-05 * 17) * x_expm1(-(u - (T)19.9) / (T)17);
                bxs = (T)(3.5e-05 * 9) * x_expm1((u - (T)19.9) / (T)9);
            }
            const T tau_xs = c1 / ((T)2 * (axs + bxs));
            const T xs_inf = c1 / fw_sqrt(c1 + mexp(-(u - (T)19.9) / (T)12.7));
            x.xr = gate(x.xr, xs_inf, tau_xs, dt);
            iks = P.v[gks] * (x.xr * x.xr) * (u - ek);
        }
        T ical;
        {
            const T e = mexp(-(u + (T)10) / (T)6.24);
            T tau_d;
            if constexpr (sizeof(T) == 8) {
                tau_d = (c1 - e) / ((T)0.035 * (u + (T)10) * (c1 + e));
            } else {
                // (1 - e^-v) / v = 1 / x_expm1(-v), v = (u + 10) / 6.24
                tau_d = c1 / ((T)(0.035 * 6.24) *
                              x_expm1(-(u + (T)10) / (T)6.24) * (c1 + e));
            }
            const T d_inf = c1 / (c1 + mexp(-(u + (T)10) / (T)8.0));
            const T tau_f = (T)9 / ((T)0.0197 * mexp(-((T)0.0337 * (T)0.0337) *
                                                      ((u + (T)10) * (u + (T)10))) +
                                    (T)0.02);
            const T f_inf = c1 / (c1 + mexp((u + (T)28) / (T)6.9));
            const T fca_inf = c1 / (c1 + cai / (T)0.00035);
            x.d = gate(x.d, d_inf, tau_d, dt);
            x.f = gate(x.f, f_inf, tau_f, dt);
            x.fca = gate(x.fca, fca_inf, (T)2, dt);
            ical = P.v[gcal] * x.d * x.f * x.fca * (u - (T)65);
        }
        const T RT = P.v[R] * P.v[T_];
        T inak, inaca;
        {
            const T s = c1 / (T)7.0 * (mexp(P.v[nao] / (T)67.3) - c1);
            const T fnak = c1 / (c1 + (T)0.1245 * mexp((T)(-0.1) * (P.v[F] * u) / RT) +
                                 (T)0.0365 * s * mexp(-(P.v[F] * u) / RT));
            inak = P.v[inakmax] * fnak * (c1 / (c1 + pow15(P.v[kmnai] / nai))) *
                   (P.v[ko] / (P.v[ko] + P.v[kmko]));
            const T gamma = (T)0.35;
            const T exp_term = mexp(gamma * (P.v[F] * u) / RT);
            const T exp_rev_term = mexp((gamma - c1) * (P.v[F] * u) / RT);
            const T numerator = P.v[inacamax] *
                                (exp_term * pow3(nai) * P.v[cao] -
                                 exp_rev_term * pow3(P.v[nao]) * cai);
            const T term1 = pow3(P.v[kmnancx]) + pow3(P.v[nao]);
            const T term2 = P.v[kmcancx] + P.v[cao];
            const T term3 = c1 + P.v[ksatncx] * exp_rev_term;
            inaca = numerator / (term1 * term2 * term3);
        }
        const T ibca = P.v[gcab] * (u - eca);
        const T ibna = P.v[gnab] * (u - ena);
        const T ipca = P.v[ipcamax] * cai / (cai + (T)0.0005);
        {
            const T Fn = (T)1e-12 * P.v[Vrel] * x.irel -
                         (T)5 * (T)1e-13 / P.v[F] * ((T)0.5 * ical - (T)0.2 * inaca);
            const T u_inf = c1 / (c1 + mexp(-(Fn - (T)3.4175e-13) / (T)1.367e-15));
            const T tau_v = (T)1.91 + (T)2.09 / (c1 + mexp(-(Fn - (T)3.4175e-13) /
                                                           (T)1.367e-15));
            const T v_inf = c1 - c1 / (c1 + mexp(-(Fn - (T)6.835e-14) / (T)1.367e-15));
            const T ew = mexp(-(u - (T)7.9) / (T)5.0);
            T tau_w;
            if constexpr (sizeof(T) == 8) {
                tau_w = (T)6 * (c1 - ew) / ((c1 + (T)0.3 * ew) * (u - (T)7.9));
            } else {
                tau_w = (T)(6.0 / 5.0) /
                        ((c1 + (T)0.3 * ew) * x_expm1(-(u - (T)7.9) / (T)5.0));
            }
            const T w_inf = c1 - c1 / (c1 + mexp(-(u - (T)40) / (T)17.0));
            x.urel = gate(x.urel, u_inf, (T)8, dt);
            x.vrel = gate(x.vrel, v_inf, tau_v, dt);
            x.wrel = gate(x.wrel, w_inf, tau_w, dt);
            x.irel = P.v[krel] * (x.urel * x.urel) * x.vrel * x.wrel * (carel - cai);
        }
        const T itr = (caup - carel) / (T)180;
        const T iup = P.v[iupmax] / (c1 + P.v[kup] / cai);
        const T iupleak = caup / P.v[caupmax] * P.v[iupmax];
        // calc_caup, calc_nai, calc_ki, calc_cai, calc_carel
        // (courtemanche_2d.py:219-253); under float32 the rates are float32
        // and only the accumulation is float64
        const T FVj = P.v[F] * P.v[Vj];
        const T dCaup = dt * (iup - iupleak - itr * (P.v[Vrel] / P.v[Vup]));
        const T dNai = dt * (((T)(-3) * inak - (T)3 * inaca - ibna - ina) / FVj);
        const T dKi = dt * (((T)2 * inak - ik1 - ito - ikur - ikr - iks -
                             P.v[ibk]) / FVj);
        const T ktr = P.v[kmtrpn], kcm = P.v[kmcmdn];
        const T B1 = ((T)2 * inaca - ipca - ical - ibca) / ((T)2 * FVj) +
                     (P.v[Vup] * (iupleak - iup) + x.irel * P.v[Vrel]) / P.v[Vj];
        const T B2 = c1 + P.v[trpnmax] * ktr / ((cai + ktr) * (cai + ktr)) +
                     P.v[cmdnmax] * kcm / ((cai + kcm) * (cai + kcm));
        const T dCai = dt * (B1 / B2);
        const T kcs = P.v[kmcsqn];
        const T dCarel = dt * ((itr - x.irel) /
                               (c1 + P.v[csqnmax] * kcs /
                                         ((carel + kcs) * (carel + kcs))));
        x.caup += dCaup;
        x.nai += dNai;
        x.ki += dKi;
        x.cai += dCai;
        x.carel += dCarel;
        return un - dt * (ina + ik1 + ito + ikur + ikr + iks + ical + ipca + inak +
                          inaca + ibna + ibca);
    }
};

// ---------------------------------------------------------------- LR91
// Luo-Rudy 1991.  Parameters in the order of luo_rudy91_2d.py's
// ionic_kernel_2d signature: gna, gsi, gk, gk1, gkp, gb, ko, ki, nai, nao,
// cao, R, T, F, PR_NaK; state m, h, j, d, f, x, cai (LuoRudy912D.state_vars
// minus u).  calc_ina uses the updated m, h, j; calc_isk and calc_ik the
// gates before their update, as the reference does.  Under FW_F32 Ca_i is
// stored as float64 and only its accumulation is float64.
struct ModelLR91 {
    static constexpr int NS = 7, NP = 15;
    enum { gna, gsi, gk, gk1, gkp, gb, ko, ki, nai, nao, cao, R, T_, F, PR_NaK };
    enum { s_m, s_h, s_j, s_d, s_f, s_x, s_cai };
    static constexpr bool is_conc(int i) { return i == s_cai; }

    template <class T>
    struct St {
        T m, h, j, d, f, x;
        Conc<T> cai;
    };
    template <class T>
    __device__ static __forceinline__ St<T> load(void *const *S, int64_t p)
    {
        St<T> x;
        x.m = ((const T *)S[s_m])[p];
        x.h = ((const T *)S[s_h])[p];
        x.j = ((const T *)S[s_j])[p];
        x.d = ((const T *)S[s_d])[p];
        x.f = ((const T *)S[s_f])[p];
        x.x = ((const T *)S[s_x])[p];
        conc_load(x.cai, S[s_cai], p);
        return x;
    }
    template <class T>
    __device__ static __forceinline__ void store(void *const *S, int64_t p,
                                                 const St<T> &x)
    {
        ((T *)S[s_m])[p] = x.m;
        ((T *)S[s_h])[p] = x.h;
        ((T *)S[s_j])[p] = x.j;
        ((T *)S[s_d])[p] = x.d;
        ((T *)S[s_f])[p] = x.f;
        ((T *)S[s_x])[p] = x.x;
        conc_store(S[s_cai], p, x.cai);
    }
    template <class T>
    __device__ static __forceinline__ double probe(const St<T> &x, int i)
    {
        switch (i) {
        case s_m: return x.m;
        case s_h: return x.h;
        case s_j: return x.j;
        case s_d: return x.d;
        case s_f: return x.f;
        case s_x: return x.x;
        default: return conc_probe(x.cai);
        }
    }
    // calc_gating_var (luo_rudy91_2d.py): tau = 1 / (a + b),
    // inf = a / (a + b), var += dt (inf - var) / tau
    template <class T>
    __device__ static __forceinline__ T gating(T var, T dt, T a, T b)
    {
        const T tau = (T)1. / (a + b);
        const T inf = a / (a + b);
        return var + dt * (inf - var) / tau;
    }

    enum { d_ena = NP, d_ek, d_ek1, d_gk, d_gk1, d_end };
    static constexpr int ND = d_end - NP;
    static void derive(const double *p, double, double *q)
    {
        const double RTF = p[R] * p[T_] / p[F], gs = sqrt(p[ko] / 5.4);
        q[d_ena] = RTF * log(p[nao] / p[nai]);
        q[d_ek] = RTF * log((p[ko] + p[PR_NaK] * p[nao]) / (p[ki] + p[PR_NaK] * p[nai]));
        q[d_ek1] = RTF * log(p[ko] / p[ki]);
        q[d_gk] = p[gk] * gs;
        q[d_gk1] = p[gk1] * gs;
    }

    template <class T>
    __device__ static __forceinline__ T update(T u, T un, St<T> &x,
                                               const Params<T, NP + ND> &P, T dt)
    {
        if constexpr (sizeof(T) == 4) {
            // float32 keeps the reference's order and with it the bits of its
            // results: the rates of h jump by a quarter at u = -40, so a node
            // that meets the branch a step earlier for another rounding
            // differs by 1e-3 there
            return update_ref<T>(u, un, x, P, dt);
        } else {
            if (in_range(u, u - P.v[d_ek1])) return update_in_range(u, un, x, P, dt);
            return update_any(u, un, x, P, dt);
        }
    }
    __device__ static __forceinline__ bool in_range(double u, double x)
    {
        return fabs(u) < 300.0 && x > -400.0 && x < 1000.0;
    }

    // As ModelTP06::update_in_range; var + dt (inf - var) / tau with
    // tau = 1 / (a + b), inf = a / (a + b) is var + dt (a (1 - var) - b var).
    // 192 x 190 nodes: 33 against 75 us a step (float64 only).
    __device__ static __forceinline__ double
    update_in_range(double u, double un, St<double> &x,
                    const Params<double, NP + ND> &P, double dt)
    {
        using namespace dm;
        using T = double;
        const T c1 = (T)1;
        auto gate = [dt](T v, T a, T b) { return v + dt * (a * ((T)1 - v) - b * v); };
        // calc_ina
        T ina;
        {
            T alpha_h = 0, beta_h, alpha_J = 0, beta_J;
            if (u >= (T)(-40.)) {
                beta_h = (T)(1 / 0.13) * rcp(c1 + FW_EX(u + (T)10.66, -1 / 11.1));
                // e^(-2.535e-7 u), |u| < 300: the series to the third power
                const T y = (T)(-2.535e-07) * u;
                const T ey = c1 + y * (c1 + y * ((T)0.5 + y * (T)(1 / 6.0)));
                beta_J = (T)0.3 * ey * rcp(c1 + FW_EX(u + (T)32, -0.1));
            } else {
                alpha_h = (T)0.135 * FW_EX((T)80 + u, -1 / 6.8);
                beta_h = (T)3.56 * FW_EX(u, 0.079) + (T)3.1e5 * FW_EX(u, 0.35);
                beta_J = (T)0.1212 * FW_EX(u, -0.01052) *
                         rcp(c1 + FW_EX(u + (T)40.14, -0.1378));
                alpha_J = ((T)(-1.2714e5) * FW_EX(u, 0.2444) -
                           (T)3.474e-5 * FW_EX(u, -0.04391)) *
                          (u + (T)37.78) * rcp(c1 + FW_EX(u + (T)79.23, 0.311));
            }
            const T z = (T)(-0.1) * (u + (T)47.13);
            const T alpha_m = (T)3.2 * x_over_expm1(z, ex(z));
            const T beta_m = (T)0.08 * FW_EX(u, -1 / 11.0);
            x.m = gate(x.m, alpha_m, beta_m);
            x.h = gate(x.h, alpha_h, beta_h);
            x.j = gate(x.j, alpha_J, beta_J);
            ina = P.v[gna] * x.m * x.m * x.m * x.h * x.j * (u - P.v[d_ena]);
        }
        // calc_isk (gates before the update)
        T isi;
        {
            const T cai = (T)x.cai;
            const T E_Si = (T)7.7 - (T)13.0287 * lg(cai);
            isi = P.v[gsi] * x.d * x.f * (u - E_Si);
            const T u5 = u - (T)5, u44 = u + (T)44, u28 = u + (T)28, u30 = u + (T)30;
            const T alpha_d = (T)0.095 * FW_EX(u5, -0.01) * rcp(c1 + FW_EX(u5, -0.072));
            const T beta_d = (T)0.07 * FW_EX(u44, -0.017) * rcp(c1 + FW_EX(u44, 0.05));
            const T alpha_f = (T)0.012 * FW_EX(u28, -0.008) * rcp(c1 + FW_EX(u28, 0.15));
            const T beta_f = (T)0.0065 * FW_EX(u30, -0.02) * rcp(c1 + FW_EX(u30, -0.2));
            x.d = gate(x.d, alpha_d, beta_d);
            x.f = gate(x.f, alpha_f, beta_f);
            x.cai += dt * ((T)(-0.0001) * isi + (T)0.07 * ((T)0.0001 - cai));
        }
        // calc_ik (gate before the update)
        T ik;
        {
            T Xi = c1;
            if (u > (T)(-100)) {
                // 2.837 (e^y - 1) / ((u + 77) e^(y - 1.68)), y = 0.04 (u + 77)
                const T z = (T)(-0.04) * (u + (T)77);
                Xi = (T)(2.837 * 0.04 * 5.365555971121975) * rcp(x_over_expm1(z, ex(z)));
            }
            ik = P.v[d_gk] * x.x * Xi * (u - P.v[d_ek]);
            const T u50 = u + (T)50, u20 = u + (T)20;
            x.x = gate(x.x, (T)0.0005 * FW_EX(u50, 0.083) * rcp(c1 + FW_EX(u50, 0.057)),
                       (T)0.0013 * FW_EX(u20, -0.06) * rcp(c1 + FW_EX(u20, -0.04)));
        }
        // calc_ik1: alpha / (alpha + beta) over the common denominator
        const T ux = u - P.v[d_ek1];
        const T da = c1 + FW_EX(ux - (T)59.215, 0.2385);
        const T db = c1 + FW_EX(ux + (T)4.753, -0.5143);
        const T nb = (T)0.49124 * FW_EX(ux + (T)5.476, 0.08032) +
                     FW_EX(ux - (T)594.31, 0.06175);
        const T na = (T)1.02 * db;
        const T ik1 = P.v[d_gk1] * na * rcp(na + nb * da) * ux;
        // calc_ikp, calc_ib
        const T ikp = P.v[gkp] * rcp(c1 + FW_EX(u - (T)7.488, -1 / 5.98)) * ux;
        const T ib = P.v[gb] * (u + (T)59.87);
        return un - dt * (ina + isi + (ik1 + ikp + ib) + ik);
    }

    // The update in the reference's order, for potentials outside the range
    // above.
    // (Copies go into the call, so that x and P keep to registers elsewhere.)
    __device__ static __forceinline__ double update_any(double u, double un, St<double> &x,
                                                        const Params<double, NP + ND> &P,
                                                        double dt)
    {
        St<double> y = x;
        Params<double, NP + ND> Q = P;
        un = update_call(u, un, y, Q, dt);
        x = y;
        return un;
    }
    __device__ static __noinline__ double update_call(double u, double un, St<double> &x,
                                                      const Params<double, NP + ND> &P,
                                                      double dt)
    {
        return update_ref<double>(u, un, x, P, dt);
    }
    template <class T>
    __device__ static __forceinline__ T update_ref(T u, T un, St<T> &x,
                                                   const Params<T, NP + ND> &P, T dt)
    {
        const T c1 = (T)1;
        const T RTF = P.v[R] * P.v[T_] / P.v[F];
        const T E_Na = RTF * mlog(P.v[nao] / P.v[nai]);
        // calc_ina
        T ina;
        {
            T alpha_h = 0, beta_h = 0, beta_J = 0, alpha_J = 0;
            if (u >= (T)(-40.)) {
                beta_h = (T)1. / ((T)0.13 * (c1 + mexp((u + (T)10.66) / (T)(-11.1))));
                beta_J = (T)0.3 * mexp((T)(-2.535) * (T)1e-07 * u) /
                         (c1 + mexp((T)(-0.1) * (u + (T)32)));
            } else {
                alpha_h = (T)0.135 * mexp(((T)80 + u) / (T)(-6.8));
                beta_h = (T)3.56 * mexp((T)0.079 * u) +
                         (T)3.1 * (T)1e5 * mexp((T)0.35 * u);
                beta_J = (T)0.1212 * mexp((T)(-0.01052) * u) /
                         (c1 + mexp((T)(-0.1378) * (u + (T)40.14)));
                alpha_J = ((T)(-1.2714) * (T)1e5 * mexp((T)0.2444 * u) -
                           (T)3.474 * (T)1e-5 * mexp((T)(-0.04391) * u)) *
                          (u + (T)37.78) / (c1 + mexp((T)0.311 * (u + (T)79.23)));
            }
            T alpha_m;
            if constexpr (sizeof(T) == 8)
                alpha_m = (T)0.32 * (u + (T)47.13) /
                          (c1 - mexp((T)(-0.1) * (u + (T)47.13)));
            else
                alpha_m = (T)3.2 * x_expm1((T)(-0.1) * (u + (T)47.13));
            const T beta_m = (T)0.08 * mexp(-u / (T)11);
            x.m = gating(x.m, dt, alpha_m, beta_m);
            x.h = gating(x.h, dt, alpha_h, beta_h);
            x.j = gating(x.j, dt, alpha_J, beta_J);
            ina = P.v[gna] * x.m * x.m * x.m * x.h * x.j * (u - E_Na);
        }
        // calc_isk (gates before the update)
        T isi;
        {
            const T cai = (T)x.cai;
            const T E_Si = (T)7.7 - (T)13.0287 * mlog(cai);
            isi = P.v[gsi] * x.d * x.f * (u - E_Si);
            const T alpha_d = (T)0.095 * mexp((T)(-0.01) * (u - (T)5)) /
                              (c1 + mexp((T)(-0.072) * (u - (T)5)));
            const T beta_d = (T)0.07 * mexp((T)(-0.017) * (u + (T)44)) /
                             (c1 + mexp((T)0.05 * (u + (T)44)));
            const T alpha_f = (T)0.012 * mexp((T)(-0.008) * (u + (T)28)) /
                              (c1 + mexp((T)0.15 * (u + (T)28)));
            const T beta_f = (T)0.0065 * mexp((T)(-0.02) * (u + (T)30)) /
                             (c1 + mexp((T)(-0.2) * (u + (T)30)));
            x.d = gating(x.d, dt, alpha_d, beta_d);
            x.f = gating(x.f, dt, alpha_f, beta_f);
            x.cai += dt * ((T)(-0.0001) * isi + (T)0.07 * ((T)0.0001 - cai));
        }
        // calc_ik (gate before the update)
        T ik;
        {
            const T E_K = RTF * mlog((P.v[ko] + P.v[PR_NaK] * P.v[nao]) /
                                     (P.v[ki] + P.v[PR_NaK] * P.v[nai]));
            const T G_K = P.v[gk] * fw_sqrt(P.v[ko] / (T)5.4);
            T Xi;
            if (u > (T)(-100)) {
                if constexpr (sizeof(T) == 8)
                    Xi = (T)2.837 * (mexp((T)0.04 * (u + (T)77)) - c1) /
                         ((u + (T)77) * mexp((T)0.04 * (u + (T)35)));
                else  // (e^z - 1) / (u + 77) = 0.04 / x_expm1(z)
                    Xi = (T)(2.837 * 0.04) /
                         (x_expm1((T)0.04 * (u + (T)77)) *
                          mexp((T)0.04 * (u + (T)35)));
            } else {
                Xi = c1;
            }
            ik = G_K * x.x * Xi * (u - E_K);
            const T alpha_x = (T)0.0005 * mexp((T)0.083 * (u + (T)50)) /
                              (c1 + mexp((T)0.057 * (u + (T)50)));
            const T beta_x = (T)0.0013 * mexp((T)(-0.06) * (u + (T)20)) /
                             (c1 + mexp((T)(-0.04) * (u + (T)20)));
            x.x = gating(x.x, dt, alpha_x, beta_x);
        }
        const T E_K1 = RTF * mlog(P.v[ko] / P.v[ki]);
        // calc_ik1
        const T alpha_K1 = (T)1.02 / (c1 + mexp((T)0.2385 * (u - E_K1 - (T)59.215)));
        const T beta_K1 = ((T)0.49124 * mexp((T)0.08032 * (u - E_K1 + (T)5.476)) +
                           mexp((T)0.06175 * (u - E_K1 - (T)594.31))) /
                          (c1 + mexp((T)(-0.5143) * (u - E_K1 + (T)4.753)));
        const T K_1x = alpha_K1 / (alpha_K1 + beta_K1);
        const T G_K1 = P.v[gk1] * fw_sqrt(P.v[ko] / (T)5.4);
        const T ik1 = G_K1 * K_1x * (u - E_K1);
        // calc_ikp, calc_ib
        const T K_p = (T)1. / (c1 + mexp(((T)7.488 - u) / (T)5.98));
        const T ikp = P.v[gkp] * K_p * (u - E_K1);
        const T ib = P.v[gb] * (u + (T)59.87);
        const T ik1t = ik1 + ikp + ib;
        return un - dt * (ina + isi + ik1t + ik);
    }
};

}  // namespace fw
