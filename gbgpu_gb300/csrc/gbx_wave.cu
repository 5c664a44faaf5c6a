// FastGB waveform family for GB300 (sm_103a): one CTA builds a tile of
// binaries (P = max(1, 512/N) of them) entirely in shared memory -- slow part,
// N-point FFT, fftshift/heterodyne and TDI combination -- and then either
// writes the reference's output arrays, folds the window into <d|h>, <h|h>
// against the data and PSD, or scatter-adds it into global templates.
//
// Reference: gbgpu/gbgpu.py:108-578 (waveform), gbgpu/thirdbody.py:155-428
// (third body), gbgpu/cutils/gbgpu_utils.cu:54-185 (likelihood / fill loops).
#include <math.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "gbx_common.cuh"
#include "gbx_index.h"
#include "gbx_internal.h"

extern "C" size_t gbx_wave_workspace_bytes(int num_bin);

namespace gbx {

__device__ double2 g_tw_d[kTwN / 2];
__device__ float2 g_tw_f[kTwN / 2];
__device__ float4 g_tw_p[kTwN / 2];   // the same twiddles as float pairs (c.h, c.l, s.h, s.l)
__device__ float4 g_sc_p[256];        // cos, sin of j pi/128 as float pairs (pair form)
__device__ double2 g_sc_d[256];       // cos, sin of j pi/128 (FP64 form)

__global__ void tw_init_kernel()
{
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < kTwN / 2) {
        double s, c;
        sincospi(-2.0 * (double)m / (double)kTwN, &s, &c);
        g_tw_d[m] = make_double2(c, s);
        g_tw_f[m] = make_float2((float)c, (float)s);
        const dfl cp = df_from(c), sp = df_from(s);
        g_tw_p[m] = make_float4(cp.h, cp.l, sp.h, sp.l);
    }
    if (m < 256) {
        double s, c;
        sincospi((double)m / 128.0, &s, &c);
        const dfl cp = df_from(c), sp = df_from(s);
        g_sc_p[m] = make_float4(cp.h, cp.l, sp.h, sp.l);
        g_sc_d[m] = make_double2(c, s);
    }
}

template <typename R> __device__ __forceinline__ typename C2<R>::T tw(int m);
template <> __device__ __forceinline__ float2 tw<float>(int m) { return g_tw_f[m]; }
template <> __device__ __forceinline__ double2 tw<double>(int m) { return g_tw_d[m]; }

// ----------------------------------------------------------------------------
// per-binary constants (shared memory)
// ----------------------------------------------------------------------------
struct __align__(16) Bin {
    double f0, fdot, fddot, phi0;
    double om, om_m_dfa;           // 2 pi f0, 2 pi f0 - 2 pi q/T   (gbgpu.py:462-464)
    double pifdot, pi3fddot;       // pi fdot, pi/3 fddot           (gbgpu.py:495-500)
    double k[3];
    union {
        struct {
            double up[3], vp[3];   // u and v rotated by the polarisation angle (FP64 form)
            double ap4, ci;        // (1 + cos^2 iota)/4, cos iota
            double kh[2], kl[2];   // x and y of k: multiples of 2^-26, and the rest
            double pf2, p3f3;      // 2 pi fdot, pi fddot
        } q;
        struct {
            dfl up[3], vp[3];      // the same as pairs (pair form)
            dfl ap4, ci;
        } pr;
    };
    double2 scale;                 // amp * 0.5 T / N [* tdi2 factor]
    union { double n2; dfl n2d; }; // n2 [rad/s]: FP64 form / float pair (mixed form)
    union { double T2; dfl T2d; }; // T2 [s], likewise
    union {
        struct {
            float kf[3], uf[3], vf[3];   // k, u, v in FP32 (mixed form; r.e+.r = (r.v)^2 - (r.u)^2)
        };
        struct {
            // FP64 form: v_LOS = (ka sin u + kb cos u)/(1 - eD cos u) + kc
            double e2, eD, ka, kb, kc;
        } kep;
    };
    float2 DPf, DCf;
    float f0f, fdotf, fddotf;
    float w0h, w0l, w1, w2;        // f(t)/fstar = (w0h + w0l) + w1 t + w2 t^2 (w0 split hi/lo)
    float w1l;                     // w1 - (float)w1 (the pair form's w1 t term)
    dfl kd[3], omd, omdfad, phi0d, pfd;   // float-pair copies for the mixed carrier phase
    dfl tpfd;                      // 2 pi fdot as a float pair
    dfl p3d, pfddd;                // pi/3 fddot, pi fddot (the mixed form uses the heads)
    float A2f, e2f, varpif, sinvarpif;
    int start;                     // start index - start_freq_ind
    int b;                         // binary index
    int di, ni, gi;                // data / noise / group rows
    int eS, eD;                    // power-of-two scalings of the mixed likelihood
    int valid;
};

static_assert(sizeof(Bin) % 16 == 0, "Bin is copied as int4 vectors");

struct KParams {
    gbx_wave_args a;
    // likelihood
    const double2 *A_data, *E_data;
    const double *A_psd, *E_psd;
    int L, num_data, num_psd;
    const int *data_index, *noise_index;
    double df;
    double2 *d_h, *h_h;
    double *dlogl;                 // swap: one log-likelihood change per (old, new) pair
    // waveform outputs
    double2 *XYZ, *AET;
    int *start_out;
    // fill
    double2 *A_glob, *E_glob;
    const int *group_index;
    int num_groups;
    long long gstride;             // elements between consecutive groups of A_glob / E_glob
    int P;                         // binaries per tile in uniform mode
    double fstar, ifstar;          // c / (2 pi L) and its reciprocal
    dfl stepd[GBX_MAX_LOG2N + 1];  // T / 2^k as float pairs (exact: division by a power of two)
    dfl Locd;                      // L / c as a float pair (pair form)
    double Loc;                    // L / c (FP64 form)
    float T2f;                     // T^2 (FP64 form)
    int maxS;                      // largest tile (samples) the shared memory is sized for
    int maxP;                      // most binaries in a tile of this launch (<= kMaxPack)
};

enum { MODE_WAVE = 0, MODE_LL = 1, MODE_FILL = 2, MODE_SWAP = 4 };

// doubles of the per-tile reduction scratch: 3 per 32-sample chunk, and at
// least 8 per lane group (16 groups) for the swap epilogue
// group partials of the likelihood (up to kMaxPack groups x 3 float pairs) and
// the per-binary FP64 sums (up to kMaxPack x 3) after them, or the swap
// epilogue's group x 8 FP64 partials
__host__ __device__ __forceinline__ int red_doubles(int maxS)
{
    return 3 * (maxS >> 5) > 8 * kMaxPack ? 3 * (maxS >> 5) : 8 * kMaxPack;
}

// sin(x) and cos(x) for moderate |x| (the carrier phase reduced to [-pi, pi],
// omega L, link arguments: |x| < 8).  Cody-Waite reduction r = x - k pi/2
// with pi/2 split into two floats (Cody & Waite, "Software Manual for the
// Elementary Functions", 1980), then the Taylor series of sin and cos on
// |r| <= pi/4 (truncation below 2e-9 and 2e-10), then the quadrant k mod 4.
__device__ __forceinline__ void sincos_mod(float x, float &s, float &c)
{
    constexpr float kTwoOverPi = 0.636619772367581343f;
    constexpr float kPio2Hi = 1.57079637050628662f;       // float(pi/2)
    constexpr float kPio2Lo = -4.37113900018624283e-8f;   // pi/2 - float(pi/2)
    const float k = rintf(x * kTwoOverPi);
    const float r = fmaf(-k, kPio2Lo, fmaf(-k, kPio2Hi, x));
    const float r2 = r * r;
    float ps = fmaf(r2, 1.0f / 362880.0f, -1.0f / 5040.0f);
    ps = fmaf(r2, ps, 1.0f / 120.0f);
    ps = fmaf(r2, ps, -1.0f / 6.0f);
    const float sr = fmaf(r * r2, ps, r);
    float pc = fmaf(r2, -1.0f / 3628800.0f, 1.0f / 40320.0f);
    pc = fmaf(r2, pc, -1.0f / 720.0f);
    pc = fmaf(r2, pc, 1.0f / 24.0f);
    pc = fmaf(r2, pc, -0.5f);
    const float cr = fmaf(r2, pc, 1.0f);
    const int q = (int)k;
    const float a = (q & 1) ? cr : sr, b = (q & 1) ? sr : cr;
    s = (q & 2) ? -a : a;
    c = ((q + 1) & 2) ? -b : b;
}

// sin(a)/a and cos(a) from their Taylor series in x = a^2: 3 and 4 terms for
// |a| < 0.16 (truncation below 4e-9 and 1e-11), 4 and 5 terms for |a| < 0.5
// (below 3e-8 and 3e-10), 8 terms up to |a| = 1.6 (below 2e-10); sincos_mod
// beyond that.
__device__ __forceinline__ void sinc_cos_f(float a, float &S, float &C)
{
    const float x = a * a;
    if (x < 0.0256f) {
        S = fmaf(fmaf(x, 1.0f / 120.0f, -1.0f / 6.0f), x, 1.0f);
        float c = fmaf(x, -1.0f / 720.0f, 1.0f / 24.0f);
        c = fmaf(c, x, -0.5f);
        C = fmaf(c, x, 1.0f);
    } else if (x < 0.25f) {
        float s = fmaf(x, -1.0f / 5040.0f, 1.0f / 120.0f);
        s = fmaf(s, x, -1.0f / 6.0f);
        S = fmaf(s, x, 1.0f);
        float c = fmaf(x, -1.0f / 3628800.0f, 1.0f / 40320.0f);
        c = fmaf(c, x, -1.0f / 720.0f);
        c = fmaf(c, x, 1.0f / 24.0f);
        c = fmaf(c, x, -0.5f);
        C = fmaf(c, x, 1.0f);
    } else if (x < 2.56f) {
        float s = -1.0f / 1307674368000.0f;
        s = fmaf(s, x, 1.0f / 6227020800.0f);
        s = fmaf(s, x, -1.0f / 39916800.0f);
        s = fmaf(s, x, 1.0f / 362880.0f);
        s = fmaf(s, x, -1.0f / 5040.0f);
        s = fmaf(s, x, 1.0f / 120.0f);
        s = fmaf(s, x, -1.0f / 6.0f);
        S = fmaf(s, x, 1.0f);
        float c = -1.0f / 87178291200.0f;
        c = fmaf(c, x, 1.0f / 479001600.0f);
        c = fmaf(c, x, -1.0f / 3628800.0f);
        c = fmaf(c, x, 1.0f / 40320.0f);
        c = fmaf(c, x, -1.0f / 720.0f);
        c = fmaf(c, x, 1.0f / 24.0f);
        c = fmaf(c, x, -0.5f);
        C = fmaf(c, x, 1.0f);
    } else {
        float sn, cs;
        sincos_mod(a, sn, cs);
        S = sn / a;
        C = cs;
    }
}

// sin(a)/a alone: the S half of sinc_cos_f (same series and ranges).
__device__ __forceinline__ float sinc_f(float a)
{
    const float x = a * a;
    if (x < 0.0256f) return fmaf(fmaf(x, 1.0f / 120.0f, -1.0f / 6.0f), x, 1.0f);
    if (x < 0.25f) {
        float s = fmaf(x, -1.0f / 5040.0f, 1.0f / 120.0f);
        s = fmaf(s, x, -1.0f / 6.0f);
        return fmaf(s, x, 1.0f);
    }
    if (x < 2.56f) {
        float s = -1.0f / 1307674368000.0f;
        s = fmaf(s, x, 1.0f / 6227020800.0f);
        s = fmaf(s, x, -1.0f / 39916800.0f);
        s = fmaf(s, x, 1.0f / 362880.0f);
        s = fmaf(s, x, -1.0f / 5040.0f);
        s = fmaf(s, x, 1.0f / 120.0f);
        s = fmaf(s, x, -1.0f / 6.0f);
        return fmaf(s, x, 1.0f);
    }
    float sn, cs;
    sincos_mod(a, sn, cs);
    return sn / a;
}

// Shared-memory position swizzle for one length-2^lg sub-array: the low k
// bits are XOR-ed with the top k bits (k = 4 for lg >= 8).  Bit-reversed reads
// (the FFT output order) then spread over the banks instead of hitting one;
// runs of consecutive positions stay conflict-free.  A bijection, applied to
// every access of the sub-array.
__device__ __forceinline__ int swz(int pos, int lg)
{
    const int k = lg >= 8 ? 4 : (lg >> 1);
    return pos ^ ((pos >> (lg - k)) & ((1 << k) - 1));
}

// 2^e as a double for -1022 <= e <= 1023, built from its bit pattern
__device__ __forceinline__ double exp2_int(int e)
{
    return __longlong_as_double((long long)(1023 + e) << 52);
}

// FP64 -> FP32 with an exact power-of-two scaling, done on the integer pipe.
// Rounds to nearest (ties away), flushes results below FP32's normal range to
// signed zero and saturates to infinity above it.  (hi:lo) << 3 holds the 23
// leading mantissa bits at [22:0] and the exponent's low 9 bits at [31:23];
// subtracting (896 - e) << 23 modulo 2^32 leaves the FP32 biased exponent
// ne = ex - 896 + e there whenever 0 < ne < 255.
__device__ __forceinline__ float d2f_scaled(double x, int e)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int ne = (int)((hi >> 20) & 0x7ffu) - 896 + e;
    unsigned mag = __funnelshift_l(lo, hi, 3) - ((unsigned)(896 - e) << 23) + ((lo >> 28) & 1u);
    mag = ((unsigned)(ne - 1) < 254u) ? mag : (ne >= 255 ? 0x7f800000u : 0u);
    return __uint_as_float((hi & 0x80000000u) | (mag & 0x7fffffffu));
}

// the same with ties to even and no scaling: (float)x for values in FP32's
// normal range, infinities and NaN, zero below it
__device__ __forceinline__ float d2f_rn(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int ne = (int)((hi >> 20) & 0x7ffu) - 896;
    unsigned mag = __funnelshift_l(lo, hi, 3) - (896u << 23) +
                   ((lo >> 28) & ((lo & 0x2fffffffu) != 0u ? 1u : 0u));
    const unsigned top = ne == 1151 && ((hi << 12) | lo) != 0u ? 0x7fffffffu : 0x7f800000u;   // NaN, infinity
    mag = ((unsigned)(ne - 1) < 254u) ? mag : (ne >= 255 ? top : 0u);
    return __uint_as_float((hi & 0x80000000u) | (mag & 0x7fffffffu));
}

// FP32 -> FP64 (exact) on the integer pipe: exponent rebias, mantissa shift;
// FP32 zeros and subnormals give signed zero, infinities stay infinite.
__device__ __forceinline__ double f2d_bits(float f)
{
    const unsigned u = __float_as_uint(f);
    const unsigned ex = (u >> 23) & 0xffu;
    unsigned hi = (u & 0x80000000u) | ((ex + 896u) << 20) | ((u & 0x7fffffu) >> 3);
    hi = ex == 0 ? (u & 0x80000000u) : (ex == 0xffu ? (u & 0x80000000u) | 0x7ff00000u : hi);
    const unsigned lo = ex == 0 || ex == 0xffu ? 0u : (u << 29);
    return __hiloint2double((int)hi, (int)lo);
}

__device__ __forceinline__ double2 f2d(float2 v)
{
    return make_double2(f2d_bits(v.x), f2d_bits(v.y));
}

// ----------------------------------------------------------------------------
// third body: line-of-sight velocity (gbgpu/thirdbody.py:228-380); the FP64
// form's vlos3_fp64 stands with its pre-pass below
// ----------------------------------------------------------------------------
// Kepler's equation in FP32: eccentric anomaly u for a mean
// anomaly l in [0, pi] (Mikkola's starter and a fourth-order Newton step,
// gbgpu/thirdbody.py:243-320).
__device__ __forceinline__ float kepler_solve_f(float l, float e)
{
    float alpha = (1.0f - e) / (4.0f * e + 0.5f);
    float beta = 0.5f * l / (4.0f * e + 0.5f);
    float z = sqrtf(beta * beta + alpha * alpha * alpha);
    z = cbrtf(beta + z);
    float s = z - alpha / z;
    float s2 = s * s;
    float w = s - 0.078f * s2 * s2 * s / (1.0f + e);
    float u0 = l + e * (3.0f * w - 4.0f * w * w * w);
    float su0, cu0;
    sincosf(u0, &su0, &cu0);
    float f = u0 - e * su0 - l;
    float f1 = 1.0f - e * cu0;
    float f2 = 0.5f * (e * su0);
    float f3 = (1.0f / 6.0f) * (e * cu0);
    float f4 = -(1.0f / 24.0f) * (e * su0);
    float u1 = -f / f1;
    float u2 = -f / (f1 + f2 * u1);
    float u3 = -f / (f1 + f2 * u2 + f3 * u2 * u2);
    float u4 = -f / (f1 + f2 * u3 + f3 * u3 * u3 + f4 * u3 * u3 * u3);
    return u0 + u4;
}

// Eccentric anomaly (mod 2 pi) at the delayed time xi (a float pair): the
// mean anomaly M = n2 (xi - T2) and its reduction to [-pi, pi] in float-pair
// arithmetic (~1e-13 rad), then the FP32 solve on |M| with the sign put back
// (only sin/cos of the anomaly are used, so the reduction changes nothing).
// Also returns M itself (unreduced, FP32).
__device__ __forceinline__ float kepler_u_df(dfl xi, const Bin &B, float &Mout)
{
    const dfl M = df_mul(B.n2d, df_add(xi, df_neg(B.T2d)));
    Mout = M.h + M.l;
    const float q = rintf(M.h * (float)kInvTwoPi);
    const dfl r = df_add(M, df_neg(df_mul_f(df_from(kTwoPi), q)));
    const float l = r.h + r.l;
    const float u = kepler_solve_f(fminf(fabsf(l), (float)kPi), B.e2f);
    return l < 0.0f ? -u : u;
}

// v_LOS of the FP32 Kepler solve, A2 (sin(phi + varpi) + e sin varpi) with
// the true anomaly phi from u, and its time derivative
// dv/dt = A2 cos(phi + varpi)
// dphi/dM n2, with dphi/dM = sqrt(1 - e^2) / (1 - e cos u)^2 (1 / (1 - e cos u)
// below e = 1e-6, where the model takes phi = u).
__device__ float vlos_dt_mixed(dfl t, const Bin &B, float &dvdt)
{
    float M;
    const float u = kepler_u_df(t, B, M);
    const float e = B.e2f;
    float su, cu;
    sincosf(u, &su, &cu);
    const float ic = 1.0f / (1.0f - e * cu);
    float phi = u, dphi_dM = ic;
    if (e > 1e-6f) {
        const float sq = sqrtf(1.0f - e * e);
        const float bt = (1.0f - sq) / e;
        phi += 2.0f * atan2f(bt * su, 1.0f - bt * cu);
        dphi_dM = sq * ic * ic;
    }
    float sp, cp;
    sincosf(phi + B.varpif, &sp, &cp);
    dvdt = B.A2f * cp * dphi_dM * B.n2d.h;
    return B.A2f * (sp + e * B.sinvarpif);
}

// v_LOS (as vlos_dt_mixed) and its derivatives dv[0..4] = d/d(A2, varpi, e2,
// P2 [yr], T2 [yr]), dv[5] = d/dt.  With c = 1 - e cos u and M = n2 (t - T2):
// du/dM = 1/c, du/de = sin u / c (Kepler), and for the true anomaly
// dphi/du = sqrt(1-e^2)/c, dphi/de|u = sin u / (sqrt(1-e^2) c); below
// e = 1e-6 the model takes phi = u (gbgpu/thirdbody.py:339-350).
// n2 = 2 pi / (P2 yr) and T2 [s] = T2 yr give dM/dP2 = -M/P2 and
// dM/dT2 = -n2 yr = -2 pi / P2.
__device__ float vlos_grad_mixed(dfl t, const Bin &B, float cosvarpi, float P2yr, float dv[6])
{
    float M;
    const float u = kepler_u_df(t, B, M);
    const float e = B.e2f;
    float su, cu;
    sincosf(u, &su, &cu);
    const float c = 1.0f - e * cu;
    const float ic = 1.0f / c;
    float phi = u, dphi_dM, dphi_de;
    if (e > 1e-6f) {
        const float sq = sqrtf(1.0f - e * e);
        const float bt = (1.0f - sq) / e;
        phi += 2.0f * atan2f(bt * su, 1.0f - bt * cu);
        dphi_dM = sq * ic * ic;
        dphi_de = su * ic * (sq * ic + 1.0f / sq);
    } else {
        dphi_dM = ic;
        dphi_de = su * ic;
    }
    float sp, cp;
    sincosf(phi + B.varpif, &sp, &cp);
    const float A = B.A2f;
    dv[0] = sp + e * B.sinvarpif;
    dv[1] = A * fmaf(e, cosvarpi, cp);
    dv[2] = A * fmaf(cp, dphi_de, B.sinvarpif);
    const float dvdM = A * cp * dphi_dM;
    const float iP2 = 1.0f / P2yr;
    dv[3] = dvdM * M * -iP2;
    dv[4] = dvdM * (float)(-kTwoPi) * iP2;
    dv[5] = dvdM * B.n2d.h;
    return A * dv[0];
}

// ----------------------------------------------------------------------------
// FP64 arithmetic of the set-up and the FP64 form.  One FP64 warp instruction
// occupies its scheduler's FP64 unit for 64 cycles (measured), against one
// cycle for an FP32 one, so the form is bound by the number of FP64
// instructions and everything below is arranged to need few of them: 343 per
// sample for the whole likelihood at N = 128, where every link with its own
// sincos and the library's sin, sincos and divisions took 754 (10,001 binaries
// of uneven N: 7.78 -> 3.92 ms; 2,003 windows of N = 512: 1.53 -> 0.83 ms).
// ----------------------------------------------------------------------------
// sin x and cos x: table of cos, sin at j pi/128 (tab[j & 255]) and the Taylor
// series on the remainder |r| <= pi/256 (next terms below 1e-17 and 2e-20),
// combined by the angle-addition formulas.  pi/128 = C1 + C2 to 106 bits; the
// FMAs form x - j C1 without an intermediate rounding.  17 FP64 instructions.
__device__ __forceinline__ double2 turn_tab(double x, const double2 *__restrict__ tab, double &cm, double &sr)
{
    constexpr double kInv = 40.74366543152520595683;                // 128/pi
    constexpr double C1 = 0.024543692606170258;                    // double(pi/128)
    constexpr double C2 = 9.567553118338697e-19;                    // pi/128 - C1
    constexpr double kRound = 6755399441055744.0;                   // 1.5 2^52: rounds to integer
    const double t = fma(x, kInv, kRound);
    const double jd = t - kRound;
    const double r = fma(-jd, C2, fma(-jd, C1, x));
    const double r2 = r * r;
    sr = fma(r * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), r);                      // sin r
    cm = r2 * fma(r2, fma(r2, -1.0 / 720.0, 1.0 / 24.0), -0.5);                // cos r - 1
    return tab[__double2loint(t) & (kScN - 1)];
}

__device__ __forceinline__ void sincos_tab(double x, const double2 *__restrict__ tab, double &s, double &c)
{
    double cm, sr;
    const double2 cs = turn_tab(x, tab, cm, sr);
    s = cs.y + fma(cs.y, cm, cs.x * sr);
    c = cs.x + fma(cs.x, cm, -(cs.y * sr));
}

// sin(a)/a from its Taylor series in a^2: 5 terms after the first for
// |a| < 0.16, 7 for |a| < 0.5, 11 for |a| < 1.6 (next terms below 5e-20,
// 4e-20, 5e-21), sincos_tab beyond.  The last 2, 3 and 4 of them are summed in
// FP32 (at most 7e-20, 2e-18 and 3e-18 of rounding) and widened on the integer
// pipe, and the ranges are told apart by the high word.  From |a| = 1.1 on the
// rounding of a^2 and of the last two sums is kept (6 more instructions, for links
// above 21 mHz only): relative error below 1.2e-16 up to 1.6, where sin(a) and a
// division give 1.7e-16; without it 2.7e-16 at 1.6.
__device__ __forceinline__ double sinc_fp64(double a, const double2 *__restrict__ tab)
{
    const double x = a * a;
    const int hx = __double2hiint(x);
    const float xf = d2f_scaled(x, 0);
    double p;
    if (hx < 0x3f9a36e2) {                                  // x < 0.0256
        p = f2d_bits(fmaf(xf, -1.0f / 39916800.0f, 1.0f / 362880.0f));
    } else if (hx < 0x3fd00000) {                           // x < 0.25
        float t = fmaf(xf, -1.0f / 1307674368000.0f, 1.0f / 6227020800.0f);
        p = fma(x, f2d_bits(fmaf(t, xf, -1.0f / 39916800.0f)), 1.0 / 362880.0);
    } else if (hx < 0x40047ae1) {                           // x < 2.56
        float t = fmaf(xf, -1.0f / 25852016738884976640000.0f, 1.0f / 51090942171709440000.0f);
        t = fmaf(t, xf, -1.0f / 121645100408832000.0f);
        p = f2d_bits(fmaf(t, xf, 1.0f / 355687428096000.0f));
        p = fma(x, p, -1.0 / 1307674368000.0);
        p = fma(x, p, 1.0 / 6227020800.0);
        p = fma(x, p, -1.0 / 39916800.0);
        p = fma(x, p, 1.0 / 362880.0);
        if (hx >= 0x3ff35c29) {                             // x >= 1.21
            p = fma(x, p, -1.0 / 5040.0);
            p = fma(x, p, 1.0 / 120.0);
            const double c = -1.0 / 6.0, q = fma(x, p, c), ql = fma(x, p, c - q) - 9.251858538542970e-18;
            const double s = fma(x, q, 1.0);
            return s + fma(x, ql, fma(fma(a, a, -x), q, fma(x, q, 1.0 - s)));
        }
    } else {
        double s, c;
        sincos_tab(a, tab, s, c);
        return s / a;
    }
    p = fma(x, p, -1.0 / 5040.0);
    p = fma(x, p, 1.0 / 120.0);
    p = fma(x, p, -1.0 / 6.0);
    return fma(x, p, 1.0);
}

// 1 / x: the hardware's ~20-bit estimate and two Newton-Raphson steps, whose last
// rounding is all that is left (equal to the division for each of 5e8 random x); the
// division for zero, subnormal, huge and non-finite x.
__device__ __forceinline__ double recip_fp64(double x)
{
    const unsigned ex = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
    if (ex - 2u >= 2040u) return 1.0 / x;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(fma(-x, r, 1.0), r, r);
    return fma(fma(-x, r, 1.0), r, r);
}

// df_from with one FP64 instruction instead of four (the casts run on the FP64
// pipe too): parts below FP32's normal range become zero
__device__ __forceinline__ dfl df_split(double x)
{
    if ((__double2hiint(x) & 0x7ff00000) == 0x7ff00000) return df_from(x);
    const float h = d2f_rn(x);
    return {h, d2f_rn(x - f2d_bits(h))};
}

// ----------------------------------------------------------------------------
// per-binary set-up (gbgpu.py:212-266, 296-309)
// ----------------------------------------------------------------------------
struct Trig {
    double st, ct, sp, cp, si, ci, s2p, c2p;    // polar angle, lam, iota, 2 psi
};

// the library's sincos, out of line
__device__ __noinline__ double2 sincos_lib(double x)
{
    double s, c;
    sincos(x, &s, &c);
    return make_double2(s, c);
}

// Bound by its FP64 instructions: with the table's sincos, one-instruction
// splits into pairs and products with reciprocals from the host a warp takes 198
// in the pair form, 280 with the library's sincos, casts and divisions.  The
// mixed and FP64 forms keep the library's sincos and the divisions: in the mixed
// form another last bit moves an FP32 rounding in one window of 10^5, by up to
// 4e-7 of a gradient (its splits alone take a warp from 307 to 265; 50,000
// binaries 40 -> 37 us, gradient 8,191 23 -> 19 us), and in the FP64 form the last
// bit of k, 5e-14 s of k.P, is as large as the form's other rounding errors.
__device__ Trig setup_bin(Bin &B, const KParams &K, int b, int N, int mode)
{
    const gbx_wave_args &a = K.a;
    const int nb = a.num_bin;
    const double *p = a.params;
    double amp = p[b], f0 = p[nb + b], fdot = p[2 * nb + b], fddot = p[3 * nb + b];
    double phi0 = p[4 * nb + b], iota = p[5 * nb + b], psi = p[6 * nb + b];
    double lam = p[7 * nb + b], beta = p[8 * nb + b];
    const double T = a.T;
    B.b = b;
    B.valid = 1;
    B.f0 = f0; B.fdot = fdot; B.fddot = fddot;
    {
        // phi0 mod 2 pi: less rounding in the sums it enters (FP64 form)
        const double k = rint(phi0 * kInvTwoPi);
        B.phi0 = fma(-k, kTwoPiLo, fma(-k, kTwoPi, phi0));
    }
    double q = rint(f0 * T);
    // om - 2 pi q/T cancels about seven digits; the two products are rounded
    // separately (no FMA contraction) so the phase slope carries the same
    // rounding as the reference's (om - df) (gbgpu.py:462-464, 497)
    B.om = __dmul_rn(2.0 * kPi, f0);
    B.om_m_dfa = __dsub_rn(B.om, __dmul_rn(2.0 * kPi, q / T));
    B.pifdot = kPi * fdot;
    B.pi3fddot = (1.0 / 3.0 * kPi) * fddot;
    const bool lib = a.precision != GBX_PAIR;
    auto sc_of = [lib](double x, double &s, double &c) {
        // (the table's reduction is good up to |x| of 1e12)
        if (lib || !(fabs(x) < 1e6)) {
            const double2 r = sincos_lib(x);
            s = r.x;
            c = r.y;
        } else {
            sincos_tab(x, g_sc_d, s, c);
        }
    };
    double si, ci, s1p, c1p;
    sc_of(iota, si, ci);
    sc_of(psi, s1p, c1p);
    const double s2p = 2.0 * s1p * c1p, c2p = fma(-2.0 * s1p, s1p, 1.0);
    double Ap = 1.0 + ci * ci, Ac = -2.0 * ci;
    double theta = kPi / 2.0 - beta;
    double st, ct, sp, cp;
    sc_of(theta, st, ct);
    sc_of(lam, sp, cp);
    double u[3] = {ct * cp, ct * sp, -st};
    double v[3] = {sp, -cp, 0.0};
    B.k[0] = -st * cp; B.k[1] = -st * sp; B.k[2] = -ct;
    // r.e+.r DP + r.ex.r DC = (r.v + i r.u)^2 with its real part times
    // 1 + cos^2 iota and its imaginary part times 2 cos iota after a turn by
    // 2 psi: the turn goes into the basis, v' + i u' = (v + i u) e^{i psi}
    double vp[3], up[3];
    for (int c = 0; c < 3; c++) {
        vp[c] = v[c] * c1p - u[c] * s1p;
        up[c] = v[c] * s1p + u[c] * c1p;
    }
    if (a.precision == GBX_PAIR) {
        for (int c = 0; c < 3; c++) {
            B.pr.up[c] = df_split(up[c]);
            B.pr.vp[c] = df_split(vp[c]);
        }
        B.pr.ap4 = df_split(0.25 * Ap);
        B.pr.ci = df_split(ci);
    } else if (a.precision == GBX_FP64) {
        for (int c = 0; c < 3; c++) {
            B.q.up[c] = up[c];
            B.q.vp[c] = vp[c];
        }
        B.q.ap4 = 0.25 * Ap;
        B.q.ci = ci;
        B.q.pf2 = 2.0 * B.pifdot;
        B.q.p3f3 = 3.0 * B.pi3fddot;
        for (int c = 0; c < 2; c++) {
            B.q.kh[c] = rint(B.k[c] * 67108864.0) * (1.0 / 67108864.0);
            B.q.kl[c] = B.k[c] - B.q.kh[c];
        }
    }
    B.fdotf = d2f_rn(fdot);
    B.fddotf = d2f_rn(fddot);
    if (a.precision != GBX_FP64) {
        for (int c = 0; c < 3; c++) {
            B.kf[c] = d2f_rn(B.k[c]);
            B.uf[c] = d2f_rn(u[c]);
            B.vf[c] = d2f_rn(v[c]);
            B.kd[c] = df_split(B.k[c]);
        }
        B.omd = df_split(B.om);
        B.omdfad = df_split(B.om_m_dfa);
        B.phi0d = df_split(phi0);
        B.pfd = df_split(B.pifdot);
        B.tpfd = dfl{2.0f * B.pfd.h, 2.0f * B.pfd.l};
        B.p3d = df_split(B.pi3fddot);
        B.pfddd = df_split(kPi * fddot);
        B.DPf = make_float2(d2f_rn(Ap * c2p), d2f_rn(-Ac * s2p));
        B.DCf = make_float2(d2f_rn(-Ap * s2p), d2f_rn(-Ac * c2p));
        B.f0f = d2f_rn(f0);
        // f/fstar with the constant term kept as an unevaluated float pair so
        // the FP32 transfer frequency carries no per-binary rounding bias
        const dfl w0 = df_split(lib ? f0 / K.fstar : f0 * K.ifstar);
        const dfl w1 = df_split(lib ? fdot / K.fstar : fdot * K.ifstar);
        B.w0h = w0.h;
        B.w0l = w0.l;
        B.w1 = w1.h;
        B.w1l = w1.l;
        B.w2 = d2f_rn(lib ? 0.5 * fddot / K.fstar : 0.5 * fddot * K.ifstar);
    }
    // start index: round(((q - N/2)/T)/(1/T)) (gbgpu.py:296, 387) is q - N/2, the
    // three roundings moving it by less than 1e-7 of a bin
    B.start = (int)(q - (double)(N >> 1)) - a.start_freq_ind;
    // output scaling (gbgpu.py:298-309): amp * 0.5 T / N [* 2i sin 2wL e^{-2iwL}]
    double fc = 0.5 * T * exp2_int(__clz(N) - 31);           // 0.5 T / N
    double2 sc = make_double2(amp * fc, 0.0);
    if (a.tdi2 == GBX_TDI2_BIT) {
        double omL = 2.0 * kPi * f0 * (a.armlength / kCSI);
        double s2, c2;
        sincos(2.0 * omL, &s2, &c2);
        // 2i s (c - i s) = 2 s^2 + 2i s c
        double2 t2 = make_double2(2.0 * s2 * s2, 2.0 * s2 * c2);
        sc = make_double2(fc * t2.x * amp, fc * t2.y * amp);
    }
    B.scale = sc;
    if (a.nparams >= 14) {
        const double A2 = p[9 * nb + b], varpi = p[10 * nb + b], e2 = p[11 * nb + b];
        double P2 = p[12 * nb + b];
        const double n2 = 2.0 * kPi / (P2 * a.year), T2 = p[13 * nb + b] * a.year;
        if (a.precision == GBX_FP64) {
            B.n2 = n2;
            B.T2 = T2;
            // A2 [sin(phi + varpi) + e sin varpi] with the true anomaly
            // phi = u + 2 arg(1 - bt e^{-iu}), bt = (1 - sqrt(1 - e^2))/e
            // (gbgpu/thirdbody.py:339-380), that is sin phi = sq sin u/(1 - eD cos u),
            // cos phi = (cos u - eD)/(1 - eD cos u) with eD = 2 bt/(1 + bt^2) and
            // sq = (1 - bt^2)/(1 + bt^2): eD is e up to bt's rounding, which
            // reaches 1e-10 for small e and is kept as the model has it.  Below
            // e = 1e-6 the model takes phi = u: bt = 0.
            double sv, cv;
            sc_of(varpi, sv, cv);
            const double bt = e2 > 1e-6 ? (1.0 - sqrt(1.0 - e2 * e2)) / e2 : 0.0;
            const double ib = 1.0 / fma(bt, bt, 1.0), eD = 2.0 * bt * ib, sq = (1.0 - bt) * (1.0 + bt) * ib;
            B.kep.e2 = e2;
            B.kep.eD = eD;
            B.kep.ka = A2 * (sq * cv);
            B.kep.kb = A2 * (sq * sq * sv);                       // 1 - eD^2 = sq^2
            B.kep.kc = A2 * ((e2 - eD) * sv);
        } else {
            B.n2d = df_split(n2);
            B.T2d = df_split(T2);
            B.A2f = (float)A2;
            double vr = varpi - 2.0 * kPi * floor(varpi * kInvTwoPi);
            B.varpif = (float)vr;
            B.sinvarpif = (float)sin(varpi);
        }
        B.e2f = (float)e2;
    }
    B.di = B.ni = B.gi = 0;
    B.eS = B.eD = 0;
    if (mode == MODE_LL || mode == MODE_SWAP) {
        int di = K.data_index ? K.data_index[b] : 0;
        int ni = K.noise_index ? K.noise_index[b] : 0;
        if (di < 0 || di >= K.num_data || ni < 0 || ni >= K.num_psd) {
            flag(a.status, GBX_FLAG_INDEX);
            B.valid = 0;
            di = ni = 0;
        }
        B.di = di; B.ni = ni;
        // power-of-two scalings so that S*2^eS and d*2^eD are O(1) in FP32
        int jm = B.start + N / 2;
        jm = jm < 0 ? 0 : (jm >= K.L ? K.L - 1 : jm);
        double Sm = K.A_psd[(size_t)ni * K.L + jm];
        int lg = (Sm > 0.0 && isfinite(Sm)) ? ilogb(Sm) : 0;
        B.eS = -lg;
        B.eD = -(lg >> 1) - 14;
    } else if (mode == MODE_FILL) {
        int gi = K.group_index[b];
        if (gi < 0 || gi >= K.num_groups) {
            flag(a.status, GBX_FLAG_INDEX);
            B.valid = 0;
            gi = 0;
        }
        B.gi = gi;
        // a zero amplitude adds nothing (the samplers zero rejected proposals)
        if (amp == 0.0) B.valid = 0;
    }
    return Trig{st, ct, sp, cp, si, ci, s2p, c2p};
}

// ----------------------------------------------------------------------------
// Unequal arms (no counterpart in the reference, whose TDI assumes one
// armlength, gbgpu.py:167-170): arm a = 12, 23, 31 has length ell_a L at the
// sample, ell_a = |r_a| with r_a = (P_j - P_i)/L from the orbit table.  Each
// link carries its own arm: transfer argument a = (f/f*)(ell_a +- k.r_a)/2 (the
// reference's (f/f*)(1 +- k.r)/2 times ell_a with r normalised), antenna
// pattern r.e.r / ell_a^2 and amplitude ell_a; the TDI delays are the phase
// factors D_a = exp(-i omL ell_a) at the instantaneous frequency
// (quasi-static: the slow part is not re-sampled at the delayed times):
//   X = -2i omL [(1 - D_31^2)(G21 + D_12 G12) - (1 - D_12^2)(G31 + D_31 G13)]
// with Y, Z cyclic, and TDI-2 multiplies X by (1 - D_12^2 D_31^2) (Y, Z
// cyclic).  With every ell_a = 1 this is the reference's fctr2 [G21 - G31 +
// (G12 - G13) fctr] (gbgpu.py:362-372), since -2i omL (1 - D^2) = 4 omL
// sin(omL) e^{-i omL}, and its TDI-2 factor 1 - D^4 = 2i sin 2wL e^{-2iwL}
// (gbgpu.py:298-309) evaluated at f(t) instead of f0.
// ----------------------------------------------------------------------------
__device__ __forceinline__ double2 one_minus(double2 z) { return make_double2(1.0 - z.x, -z.y); }

__device__ __forceinline__ void slow_unequal_fp64(const Bin &B, double tm, double fstar,
                                               const double (&r)[3][3], const double (&kdotr)[3],
                                               const double (&fonfs)[3], const double (&kp)[3],
                                               const double2 (&A)[3], int tdi, double2 out[3])
{
    double ell[3];
#pragma unroll
    for (int a = 0; a < 3; a++) ell[a] = sqrt(r[a][0] * r[a][0] + r[a][1] * r[a][1] + r[a][2] * r[a][2]);
    double2 G[6];
    const int arm[6] = {0, 1, 2, 0, 1, 2};
    const int sc[6] = {0, 1, 2, 1, 2, 0};
    const double sg[6] = {1.0, 1.0, 1.0, -1.0, -1.0, -1.0};
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const double arg = 0.5 * fonfs[sc[q]] * (ell[arm[q]] + sg[q] * kdotr[arm[q]]);
        double sn, cs;
        sincos(arg + kp[sc[q]], &sn, &cs);
        const double amp = 0.25 * sin(arg) / arg / ell[arm[q]];
        G[q] = cmul(make_double2(amp * cs, -amp * sn), A[arm[q]]);
    }
    const double f = B.f0 + B.fdot * tm + 0.5 * B.fddot * tm * tm;
    const double omL = f / fstar;
    double2 D[3], D2[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        double sn, cs;
        sincos(omL * ell[a], &sn, &cs);
        D[a] = make_double2(cs, -sn);
        D2[a] = cmul(D[a], D[a]);
    }
    double2 X = csub(cmul(one_minus(D2[2]), cadd(G[3], cmul(D[0], G[0]))),
                     cmul(one_minus(D2[0]), cadd(G[2], cmul(D[2], G[5]))));
    double2 Y = csub(cmul(one_minus(D2[0]), cadd(G[4], cmul(D[1], G[1]))),
                     cmul(one_minus(D2[1]), cadd(G[0], cmul(D[0], G[3]))));
    double2 Z = csub(cmul(one_minus(D2[1]), cadd(G[5], cmul(D[2], G[2]))),
                     cmul(one_minus(D2[2]), cadd(G[1], cmul(D[1], G[4]))));
    if (tdi & GBX_TDI2_BIT) {
        X = cmul(one_minus(cmul(D2[0], D2[2])), X);
        Y = cmul(one_minus(cmul(D2[1], D2[0])), Y);
        Z = cmul(one_minus(cmul(D2[2], D2[1])), Z);
    }
    const double2 pre = make_double2(0.0, -2.0 * omL);
    out[0] = cmul(pre, X);
    out[1] = cmul(pre, Y);
    out[2] = cmul(pre, Z);
}

// ----------------------------------------------------------------------------
// FP64 slow part (gbgpu.py:399-540 and 348-375)
// ----------------------------------------------------------------------------
// The general path, used with unequal arms: every link with its own carrier.
__device__ __forceinline__ void slow_links_fp64(const Bin &B, int n, int N, double tm, int tdi,
                                             const double *__restrict__ tab, double fstar,
                                             double2 out[3])
{
    double r[3][3];
#pragma unroll
    for (int s = 0; s < 3; s++)
#pragma unroll
        for (int c = 0; c < 3; c++) r[s][c] = __ldg(tab + (size_t)(9 + 3 * s + c) * N + n);
    double kdotr[3], fonfs[3], kp[3];
    double2 A[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        kdotr[a] = B.k[0] * r[a][0] + B.k[1] * r[a][1] + B.k[2] * r[a][2];
        const double ru = B.q.up[0] * r[a][0] + B.q.up[1] * r[a][1] + B.q.up[2] * r[a][2];
        const double rv = B.q.vp[0] * r[a][0] + B.q.vp[1] * r[a][1] + B.q.vp[2] * r[a][2];
        A[a] = make_double2(4.0 * B.q.ap4 * (rv * rv - ru * ru), 4.0 * B.q.ci * ru * rv);
    }
#pragma unroll
    for (int s = 0; s < 3; s++) {
        double kP = 0.0;
#pragma unroll
        for (int c = 0; c < 3; c++) kP = fma(B.k[c], __ldg(tab + (size_t)(3 * s + c) * N + n), kP);
        const double xi = tm - kP;
        fonfs[s] = (B.f0 + B.fdot * xi + 0.5 * B.fddot * xi * xi) / fstar;
        kp[s] = B.om * kP - (B.phi0 + B.om_m_dfa * tm + B.pifdot * xi * xi + B.pi3fddot * xi * xi * xi);
    }
    slow_unequal_fp64(B, tm, fstar, r, kdotr, fonfs, kp, A, tdi, out);
}

// Equal arms: A and E (AE, formed before the transform) or X, Y, Z at one
// sample, amplitude divided out.
//
// With L/c = 1/(2 pi f*), arm a = 12, 23, 31 from spacecraft a to a + 1 and
// k.P_s/c - k.P_1/c = del_s = (L/c) {0, k.r_12, -k.r_31}, spacecraft s has the
// carrier phase and f/f*
//   phi_s = phi_1 + del_s (W0 - del_s W1),  fo_s = (L/c) (W0 - 2 del_s W1),
//   W0 = 2 pi f(xi_1), W1 = pi fdot(xi_1)
// (exact in fdot; left out are pi/3 fddot del^3 < 600 s^3 fddot radians and
// its share of fo_s).  The two links of an arm carry the angles
// th = a+ + phi_a and th + d with d = -(L/c)^2 W1 k.r_a (the (L/c) k.r W0
// terms cancel exactly), so one sincos per arm is enough.  With h = omL/2,
// S+- = sin(a+-)/a+-, p = S+ + S-, m = S+ - S- and
// z_a = A_a e^{-i (th + d/2 + 3h)}, the TDI combination
// fc2 (G21 - G31 + (G12 - G13) fc) (gbgpu.py:362-372) becomes, with
//   U = [p cos h cos(d/2) + i m cos h sin(d/2)] z,
//   V = [m sin h cos(d/2) + i p sin h sin(d/2)] z,
//   X = 4 omL sin(omL) [(U_1 - i V_1) - (U_3 + i V_3)]  (Y, Z cyclic).
// d is ~1e-13 rad: its part of U and V is added in FP32 and widened on the
// integer pipe (no FP64 instruction), in FP64 from 1e-9 on.
// THIRD: psi_s is taken off phi_s and fo_s grows by the factor 1 + v_s/c, which
// d follows (|d| ~ 1e-5; the sincos of d/2 itself above 1e-4).
template <bool THIRD, bool AE>
__device__ __forceinline__ void slow_fp64(const Bin &B, int n, int N, double tm,
                                          const double *__restrict__ tab, double Loc,
                                          const double2 *__restrict__ sct, bool chirp,
                                          const double *psi, const double *vl, double2 out[3])
{
    double kr[3], ru[3], rv[3];
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const double r0 = __ldg(tab + (size_t)(9 + 3 * a) * N + n);
        const double r1 = __ldg(tab + (size_t)(10 + 3 * a) * N + n);
        const double r2 = __ldg(tab + (size_t)(11 + 3 * a) * N + n);
        kr[a] = fma(B.k[2], r2, fma(B.k[1], r1, B.k[0] * r0));
        ru[a] = fma(B.q.up[2], r2, fma(B.q.up[1], r1, B.q.up[0] * r0));
        rv[a] = fma(B.q.vp[2], r2, fma(B.q.vp[1], r1, B.q.vp[0] * r0));
    }
    // r_31 = -(r_12 + r_23): differences of the same positions
    kr[2] = -(kr[0] + kr[1]);
    ru[2] = -(ru[0] + ru[1]);
    rv[2] = -(rv[0] + rv[1]);
    // k.P_1/c = s + r, s exact: multiples of 2^-43 below 2^10 (2^-26 times 2^-17)
    const double P0 = __ldg(tab + n), P1 = __ldg(tab + (size_t)N + n);
    const double H0 = __ldg(tab + (size_t)36 * N + n), H1 = __ldg(tab + (size_t)37 * N + n);
    const double L0 = __ldg(tab + (size_t)38 * N + n), L1 = __ldg(tab + (size_t)39 * N + n);
    const double s = fma(B.q.kh[1], H1, B.q.kh[0] * H0);
    const double r = fma(B.q.kh[1], L1, fma(B.q.kh[0], L0, fma(B.q.kl[1], P1,
                         fma(B.q.kl[0], P0, B.k[2] * __ldg(tab + (size_t)2 * N + n)))));
    const double xi = tm - (s + r);
    const double fx = B.pi3fddot * xi;
    // The phase of spacecraft 1, om kP - (om - df) tm - phi0 - pf xi^2 with
    // pf = pi fdot + pi/3 fddot xi, is one term of every link's angle, so its
    // rounding does not average out over the links as that of separately
    // formed phases does: the large products keep their rounding errors
    // (lo), and om kP is reduced mod 2 pi before the sum.
    constexpr double kRound = 6755399441055744.0;
    const double pf = B.pifdot + fx, xi2 = xi * xi;
    double big = B.om * s, lo = fma(B.om, r, fma(B.om, s, -big));
    double arg = fma(B.om_m_dfa, tm, B.phi0);
    if (chirp) {
        // pf xi^2 above a fraction of a radian somewhere: with the error of xi,
        // its square and the product, and TwoSum into the large part
        const double g = pf * xi2;
        const double c2 = fma(xi + xi, ((tm - xi) - s) - r, fma(xi, xi, -xi2));
        const double gl = fma(pf, c2, fma(pf, xi2, -g));
        const double S = big - g, bb = S - big;
        lo += ((big - (S - bb)) - (g + bb)) - gl;
        big = S;
    } else {
        arg = fma(pf, xi2, arg);
    }
    const double turns = fma(big, kInvTwoPi, kRound) - kRound;
    double ph[3], fo[3];
    ph[0] = fma(-turns, kTwoPi, big) - arg;
    lo = fma(-turns, kTwoPiLo, lo);
    const double W1 = fma(3.0, fx, B.pifdot);
    const double W0 = fma(xi, W1 + B.pifdot, B.om);
    const double hLoc = 0.5 * Loc;
    const double h = hLoc * fma(tm, fma(B.q.p3f3, tm, B.q.pf2), B.om);        // omL/2
    ph[0] += fma(3.0, h, lo);
    // fo: half of f/f* from here on
    fo[0] = hLoc * W0;
    const double dw = -Loc * W1;
    const double del1 = Loc * kr[0], del2 = -Loc * kr[2];
    fo[1] = fma(dw, del1, fo[0]);
    fo[2] = fma(dw, del2, fo[0]);
    ph[1] = fma(del1, fma(-del1, W1, W0), ph[0]);
    ph[2] = fma(del2, fma(-del2, W1, W0), ph[0]);
    const double dd = hLoc * dw;                                // d/2 = dd k.r
    double dv[3];
    if (THIRD) {
#pragma unroll
        for (int s = 0; s < 3; s++) {
            ph[s] -= psi[s];
            dv[s] = fo[s] * (vl[s] * (1.0 / kCSI));
            fo[s] += dv[s];
        }
    }
    // |d| < 1e-9 everywhere (|k.r| <= 1): high word of dd below that of 5e-10
    const bool tiny = !THIRD && (__double2hiint(dd) & 0x7fffffff) < 0x3e012e0b;
    double sh, ch;
    if ((__double2hiint(h) & 0x7fffffff) < 0x3fc47ae1) {                // |h| < 0.16
        const double x = h * h;
        const float xf = d2f_scaled(x, 0);
        sh = h * sinc_fp64(h, sct);
        // cos h: terms from h^8 on in FP32 (rounding below 1e-18)
        double p = f2d_bits(fmaf(xf, -1.0f / 3628800.0f, 1.0f / 40320.0f));
        p = fma(x, p, -1.0 / 720.0);
        p = fma(x, p, 1.0 / 24.0);
        p = fma(x, p, -0.5);
        ch = fma(x, p, 1.0);
    } else {
        sincos_tab(h, sct, sh, ch);
    }
    double2 U[3], V[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int s2 = a == 2 ? 0 : a + 1;
        const double ap = fma(fo[a], kr[a], fo[a]), am = fma(-fo[s2], kr[a], fo[s2]);
        const double Sp = sinc_fp64(ap, sct), Sm = sinc_fp64(am, sct);
        double d2 = dd * kr[a];
        if (THIRD)
            d2 += 0.5 * ((psi[a] - psi[s2]) + (fma(-dv[s2], kr[a], dv[s2]) - fma(dv[a], kr[a], dv[a])));
        const double Ar = B.q.ap4 * fma(rv[a], rv[a], -(ru[a] * ru[a]));
        const double Ai = B.q.ci * (ru[a] * rv[a]);
        // z = (A e^{-i theta_tab}) e^{-i r}
        double cm, sr;
        const double2 t = turn_tab(ph[a] + (ap + d2), sct, cm, sr);
        const double2 w = make_double2(fma(Ai, t.y, Ar * t.x), fma(Ai, t.x, -(Ar * t.y)));
        const double2 z = make_double2(fma(w.x, cm, fma(w.y, sr, w.x)), fma(w.y, cm, fma(-w.x, sr, w.y)));
        const double p = Sp + Sm, m = Sp - Sm;
        if (tiny) {
            const float d2f = d2f_scaled(d2, 0);
            const float e2 = d2f_scaled(m, 0) * d2f_scaled(ch, 0) * d2f;
            const float e1 = d2f_scaled(p, 0) * d2f_scaled(sh, 0) * d2f;
            const float zx = d2f_scaled(z.x, 0), zy = d2f_scaled(z.y, 0);
            const double pc = p * ch, ms = m * sh;
            U[a] = make_double2(fma(pc, z.x, f2d_bits(-e2 * zy)), fma(pc, z.y, f2d_bits(e2 * zx)));
            V[a] = make_double2(fma(ms, z.x, f2d_bits(-e1 * zy)), fma(ms, z.y, f2d_bits(e1 * zx)));
        } else {
            double sd, cd;
            if (fabs(d2) < 0.5e-4) {
                const double e = -0.5 * d2 * d2;
                cd = 1.0 + e;
                sd = d2 * fma(1.0 / 3.0, e, 1.0);
            } else {
                sincos_tab(d2, sct, sd, cd);
            }
            const double pc = p * ch * cd, ms = m * sh * cd, e2 = m * ch * sd, e1 = p * sh * sd;
            U[a] = make_double2(fma(pc, z.x, -(e2 * z.y)), fma(pc, z.y, e2 * z.x));
            V[a] = make_double2(fma(ms, z.x, -(e1 * z.y)), fma(ms, z.y, e1 * z.x));
        }
    }
    const double g4 = 16.0 * h * sh * ch;                       // 4 omL sin(omL)
    if constexpr (AE) {
        // Z - X = 2 U_3 - (U_1 + U_2) + i (V_1 - V_2),
        // X - 2Y + Z = 3 (U_1 - U_2) + i (V_1 + V_2 - 2 V_3)
        const double gA = 0.70710678118654752440 * g4, gE = 0.40824829046386301637 * g4;
        const double2 us = cadd(U[0], U[1]), ud = csub(U[0], U[1]);
        const double2 vs = cadd(V[0], V[1]), vd = csub(V[0], V[1]);
        out[0] = make_double2(gA * (fma(2.0, U[2].x, -us.x) - vd.y), gA * (fma(2.0, U[2].y, -us.y) + vd.x));
        out[1] = make_double2(gE * fma(3.0, ud.x, -fma(-2.0, V[2].y, vs.y)),
                              gE * fma(3.0, ud.y, fma(-2.0, V[2].x, vs.x)));
    } else {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int e = c == 0 ? 2 : c - 1;                   // X: 1, 3; Y: 2, 1; Z: 3, 2
            out[c] = make_double2(g4 * ((U[c].x - U[e].x) + (V[c].y + V[e].y)),
                                  g4 * ((U[c].y - U[e].y) - (V[c].x + V[e].x)));
        }
    }
}

// Spacecraft 1's delay k . P_1 / c at sample n as a float pair, from the
// orbit table's hi/lo rows: exact products (FMA), TwoSum accumulation.
__device__ __forceinline__ dfl kP1_pair(const Bin &B, const float *tabf, int N, int n)
{
    dfl P[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
        P[c] = {__ldg(tabf + (size_t)(9 + c) * N + n), __ldg(tabf + (size_t)(18 + c) * N + n)};
    float p0 = B.kd[0].h * P[0].h, p1 = B.kd[1].h * P[1].h, p2 = B.kd[2].h * P[2].h;
    float e = fmaf(B.kd[0].h, P[0].h, -p0);
    e += fmaf(B.kd[1].h, P[1].h, -p1);
    e += fmaf(B.kd[2].h, P[2].h, -p2);
#pragma unroll
    for (int c = 0; c < 3; c++) e = fmaf(B.kd[c].h, P[c].l, fmaf(B.kd[c].l, P[c].h, e));
    const dfl s01 = df_two_sum(p0, p1);
    const dfl s012 = df_two_sum(s01.h, p2);
    return df_fast(s012.h, (s01.l + s012.l) + e);
}

// Mixed form: the carrier phase om k.P - argS (gbgpu.py:495-505), the delays
// k.P/c and the delayed times are evaluated in float-pair arithmetic (about
// 48 bits, so ~1e-12 rad at 100 rad) and reduced modulo 2 pi; everything else
// is FP32.
template <bool THIRD, bool STORE_E = false>
__device__ __forceinline__ void slow_mixed(const Bin &B, int n, int N, dfl step, float Loc,
                                           const double *__restrict__ tab,
                                           const dfl *psi, const float *vl, float2 out[3],
                                           float2 *Eout = nullptr)
{
    const float *tabf = reinterpret_cast<const float *>(tab + (size_t)18 * N);
    const dfl twopi = df_from(kTwoPi);
    const float inv2pi = (float)kInvTwoPi;
    // arm vectors r_12, r_23 from the table; r_31 = -(r_12 + r_23) closes the
    // triangle, so arm 3's projections are minus the sum of the other two
    float r[2][3];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int c = 0; c < 3; c++) r[a][c] = __ldg(tabf + (size_t)(3 * a + c) * N + n);
    float kdotr[3], fonfs[3], phh[3], phl[3], dlt[3], sml[3];
#pragma unroll
    for (int a = 0; a < 2; a++)
        kdotr[a] = fmaf(B.kf[0], r[a][0], fmaf(B.kf[1], r[a][1], B.kf[2] * r[a][2]));
    kdotr[2] = -(kdotr[0] + kdotr[1]);
    const dfl tm = df_mul_f(step, (float)n);                 // n T/N
    // With xi = tm - kP the carrier phase om kP - argS (gbgpu.py:495-505)
    // expands exactly into a spacecraft-independent part and powers of kP:
    //   om kP - phi0 - (om - df) tm - pi fdot xi^2 - pi/3 fddot xi^3
    //   = Phi0(tm) + kP w(tm) - pi kP^2 fd(tm) + pi/3 fddot kP^3
    // Phi0 = -phi0 - (om - df) tm - pi fdot tm^2 - pi/3 fddot tm^3,
    // w = 2 pi (f0 + fdot tm + fddot tm^2 / 2), fd = fdot + fddot tm.
    // Phi0 and w are float pairs evaluated once per sample; the kP^2 and kP^3
    // terms are below 1e-8 rad and need only FP32.
    const float tf = tm.h;
    dfl Phi0 = df_add(df_mul(B.omdfad, tm), B.phi0d);
    const dfl tm2 = df_mul(tm, tm);
    Phi0 = df_add(Phi0, df_mul(tm2, df_fast(B.pfd.h, fmaf(B.p3d.h, tf, B.pfd.l))));
    Phi0 = df_neg(Phi0);
    const dfl wt = df_add(B.omd, df_add(df_mul(B.tpfd, tm), dfl{B.pfddd.h * tf * tf, 0.0f}));
    const float fdt = fmaf(B.fddotf, tf, B.fdotf);
    const dfl kP0 = kP1_pair(B, tabf, N, n);
    // its phase, reduced mod 2 pi
    dfl ph0 = df_add(Phi0, df_mul(kP0, wt));
    if (!THIRD) {
        const float q = rintf(ph0.h * inv2pi);
        ph0 = df_add(ph0, df_neg(df_mul_f(twopi, q)));
    }
    // spacecraft 2 and 3 differ by k.(P_s - P_1)/c = (L/c) k.r (r_12 and -r_31,
    // |.| <= L/c = 8.3 s): the carrier phase moves by that times w (<= 1.3 rad
    // below 25 mHz), added in FP32 to the float pair of spacecraft 1
    const float dk[3] = {0.0f, Loc * kdotr[0], -Loc * kdotr[2]};
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const float kPf = kP0.h + dk[s];
        const float small = kPf * kPf * fmaf(kPf, (1.0f / 3.0f) * B.pfddd.h, -(float)kPi * fdt);
        dfl ph = ph0;
        if (s > 0) {
            const dfl d = df_two_sum(ph0.h, dk[s] * wt.h);
            ph = dfl{d.h, d.l + ph0.l};
        }
        ph.l += small;
        if (THIRD) {
            ph = df_add(ph, df_neg(psi[s]));
            const float q = rintf(ph.h * inv2pi);
            ph = df_add(ph, df_neg(df_mul_f(twopi, q)));
        }
        phh[s] = ph.h;
        phl[s] = ph.l;
        // FP32: instantaneous frequency over the transfer frequency, and
        // f(t)/f* - f(xi)/f* = kP (w1 + w2 (t + xi)) formed directly (tiny)
        const float xf = tf - kPf;
        float fo = B.w0h + fmaf(fmaf(B.w2, xf, B.w1), xf, B.w0l);
        if (THIRD) fo *= 1.0f + vl[s] * (float)(1.0 / kCSI);
        fonfs[s] = fo;
        dlt[s] = kPf * fmaf(B.w2, tf + xf, B.w1);
        sml[s] = small;
    }
    // r.e+.r = (r.v)^2 - (r.u)^2, r.ex.r = 2 (r.u)(r.v)  (v has no z component)
    float ru[3], rv[3];
#pragma unroll
    for (int a = 0; a < 2; a++) {
        ru[a] = fmaf(B.uf[0], r[a][0], fmaf(B.uf[1], r[a][1], B.uf[2] * r[a][2]));
        rv[a] = fmaf(B.vf[0], r[a][0], B.vf[1] * r[a][1]);
    }
    ru[2] = -(ru[0] + ru[1]);
    rv[2] = -(rv[0] + rv[1]);
    float2 A[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float pp = fmaf(rv[a], rv[a], -ru[a] * ru[a]);
        const float cc = 2.0f * ru[a] * rv[a];
        A[a] = make_float2(fmaf(pp, B.DPf.x, cc * B.DCf.x), fmaf(pp, B.DPf.y, cc * B.DCf.y));
    }
    // links 12, 23, 31, 21, 32, 13: G = 1/4 sinc(a) exp(-i a) exp(-i phase_s)
    // A_arm (gbgpu.py:509-525)
    float2 G[6];
    if constexpr (THIRD) {
        // exp(-i phase_s) per spacecraft (the Doppler phases differ between
        // spacecraft), the pair's low part applied to first order
        float Er[3], Ei[3];
#pragma unroll
        for (int s = 0; s < 3; s++) {
            float sn, cs;
            sincos_mod(phh[s], sn, cs);
            Er[s] = fmaf(sn, -phl[s], cs);
            Ei[s] = -fmaf(cs, phl[s], sn);
            if (STORE_E) Eout[s] = make_float2(Er[s], Ei[s]);
        }
        const int arm[6] = {0, 1, 2, 0, 1, 2};
        const int sc[6] = {0, 1, 2, 1, 2, 0};
        const float sg[6] = {1.f, 1.f, 1.f, -1.f, -1.f, -1.f};
#pragma unroll
        for (int q = 0; q < 6; q++) {
            const int s = sc[q];
            float a = 0.5f * fonfs[s] * fmaf(sg[q], kdotr[arm[q]], 1.0f);
            float S, C;
            sinc_cos_f(a, S, C);
            const float aS = a * S;          // sin(a)
            const float t = 0.25f * S;
            // (C - i aS)(Er + i Ei)
            float2 e = make_float2(t * fmaf(C, Er[s], aS * Ei[s]), t * fmaf(C, Ei[s], -aS * Er[s]));
            G[q] = cmul(e, A[arm[q]]);
        }
    } else {
        // Each link carries its spacecraft's carrier in one exponential of the
        // summed angle a + phase_s (the angle's FP32 rounding and the phase's
        // low part applied to first order).  The two links of arm 12 -> (a+1)
        // carry angles a+ + phase_a and a- + phase_(a+1) whose difference is
        //   d = [dlt_a (1 + k.r) - dlt_(a+1) (1 - k.r)] / 2 + (kP^2 terms),
        // with dlt_s = f(t)/f* - f(xi_s)/f* (the phases differ by (L/c) k.r
        // w(t) = k.r f(t)/f*), |d| < 1e-7 rad: the second exponential is the
        // first one times (1 - i d), d formed from its small parts.
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int s2 = a == 2 ? 0 : a + 1;
            const float ap = 0.5f * fonfs[a] * (1.0f + kdotr[a]);
            const float am = 0.5f * fonfs[s2] * (1.0f - kdotr[a]);
            const dfl th = df_two_sum(phh[a], ap);
            const float thl = th.l + phl[a];
            float sn, cs;
            sincos_mod(th.h, sn, cs);
            const float2 eA = cmul(make_float2(fmaf(sn, -thl, cs), -fmaf(cs, thl, sn)), A[a]);
            const float tp = 0.25f * sinc_f(ap), tq = 0.25f * sinc_f(am);
            G[a] = make_float2(tp * eA.x, tp * eA.y);
            const float d = fmaf(0.5f * dlt[a], 1.0f + kdotr[a], -0.5f * dlt[s2] * (1.0f - kdotr[a])) +
                            (sml[s2] - sml[a]);
            G[a + 3] = make_float2(tq * fmaf(d, eA.y, eA.x), tq * fmaf(-d, eA.x, eA.y));
        }
        if (STORE_E) {
#pragma unroll
            for (int s = 0; s < 3; s++) {
                float sn, cs;
                sincos_mod(phh[s], sn, cs);
                Eout[s] = make_float2(fmaf(sn, -phl[s], cs), -fmaf(cs, phl[s], sn));
            }
        }
    }
    float omL = B.w0h + fmaf(fmaf(B.w2, tf, B.w1), tf, B.w0l);
    float so, co;
    sincos_mod(omL, so, co);
    float2 fc = make_float2(co, -so);
    float g4 = 4.0f * omL * so;
    float2 fc2 = make_float2(g4 * co, -g4 * so);
    float2 X = cadd(csub(G[3], G[2]), cmul(csub(G[0], G[5]), fc));
    float2 Y = cadd(csub(G[4], G[0]), cmul(csub(G[1], G[3]), fc));
    float2 Z = cadd(csub(G[5], G[1]), cmul(csub(G[2], G[4]), fc));
    out[0] = cmul(fc2, X);
    out[1] = cmul(fc2, Y);
    out[2] = cmul(fc2, Z);
}

// ----------------------------------------------------------------------------
// In-place decimation-in-frequency FFT over `nsub` contiguous sub-arrays of
// length N = 2^lg in shared memory; the output is in bit-reversed order.
//
// Stage `hl` (half-span h = 2^hl) maps (x_i, x_{i+h}) -> (x_i + x_{i+h},
// (x_i - x_{i+h}) W_{2h}^{i mod h}).  Stages hl >= 5 run in register passes of
// up to three stages (radix-8 groups of elements 2^q apart, q >= 5, so a warp
// touches 32 consecutive addresses: no bank conflicts); the last five stages
// (h = 16 ... 1) run inside a warp on 32 consecutive elements with shuffles.
// One __syncthreads per pass: ceil((lg - 5)/3) + 1 barriers instead of lg.
// ----------------------------------------------------------------------------
template <typename R, int RB>
__device__ __forceinline__ void fft_reg_pass(typename C2<R>::T *buf, int nsub, int lg, int hl)
{
    using V = typename C2<R>::T;
    constexpr int M = 1 << RB;
    const int q = hl - RB + 1;                 // log2 of the in-group stride
    const int groups = nsub << (lg - RB);      // N / 2^RB groups per sub-array
    for (int g = threadIdx.x; g < groups; g += kBlock) {
        const int a = g >> (lg - RB);
        const int rem = g & ((1 << (lg - RB)) - 1);
        const int blk = rem >> q;
        const int r = rem & ((1 << q) - 1);
        V *sub = buf + ((size_t)a << lg);
        const int p0 = (blk << (hl + 1)) + r;
        V x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = sub[swz(p0 + (m << q), lg)];
#pragma unroll
        for (int j = 0; j < RB; j++) {
            const int dm = M >> (j + 1);             // register distance of the pair
            const int hh = hl - j;                   // log2 half-span of this stage
            const int ts = kTwN >> (hh + 1);
#pragma unroll
            for (int m = 0; m < M; m++) {
                if (m & dm) continue;
                const int rp = r + ((m & (dm - 1)) << q);
                V u = x[m], v = x[m + dm];
                x[m] = cadd(u, v);
                x[m + dm] = cmul(csub(u, v), tw<R>(rp * ts));
            }
        }
#pragma unroll
        for (int m = 0; m < M; m++) sub[swz(p0 + (m << q), lg)] = x[m];
    }
}

template <typename R>
__device__ __forceinline__ typename C2<R>::T shfl_c(typename C2<R>::T v, int o)
{
    v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    return v;
}

template <typename R>
__device__ __forceinline__ void fft_dif(typename C2<R>::T *buf, int nsub, int lg)
{
    using V = typename C2<R>::T;
    // register passes for the stages with half-span >= 32
    int hl = lg - 1;
    while (hl >= 5) {
        const int rb = (hl - 4) >= 3 ? 3 : (hl - 4);
        if (rb == 3) fft_reg_pass<R, 3>(buf, nsub, lg, hl);
        else if (rb == 2) fft_reg_pass<R, 2>(buf, nsub, lg, hl);
        else fft_reg_pass<R, 1>(buf, nsub, lg, hl);
        hl -= rb;
        __syncthreads();
    }
    // the last five stages inside a warp: lane l holds element 32c + l.  The
    // lower lane of a pair keeps x + y, the upper one (y - x) W: both are
    // (sg x + y) w' with sg = +-1 and w' = 1 on lower lanes (and in the last
    // stage, whose twiddles are all 1), so the stage is branch-free.
    // Half-span 2 takes W^0 = 1 and W^(kTwN/4) = -i (sincospi is exact
    // there): a swap and a sign on the upper odd lanes instead of a product.
    const int lane = threadIdx.x & 31;
    V w[3];
    R sg[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const int hh = 4 - k;                       // half-span 2^hh = 16 >> k
        const bool up = (lane & (16 >> k)) != 0;
        sg[k] = up ? (R)-1 : (R)1;
        if (k < 3) {
            const int rp = lane & ((1 << hh) - 1);
            w[k] = up ? tw<R>(rp * (kTwN >> (hh + 1))) : V{(R)1, (R)0};
        }
    }
    const bool mi = (lane & 3) == 3;                // upper lane of half-span 2, W = -i
    const int chunks = (nsub << lg) >> 5;
    for (int c = threadIdx.x >> 5; c < chunks; c += kBlock >> 5) {
        const int e = (c << 5) + lane;
        const int idx = ((e >> lg) << lg) + swz(e & ((1 << lg) - 1), lg);
        V x = buf[idx];
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const V y = shfl_c<R>(x, 16 >> k);
            const V d = {fma(sg[k], x.x, y.x), fma(sg[k], x.y, y.y)};
            if (k < 3) x = cmul(d, w[k]);
            else if (k == 3) x = mi ? V{d.y, -d.x} : d;
            else x = d;
        }
        buf[idx] = x;
    }
    __syncthreads();
}

// FP64: the same transform with fewer FP64 instructions (each costs 64 cycles
// of its scheduler, so nothing else matters).  A register pass takes its 2, 4
// or 8 elements as one small DFT whose inner factors are 1, -i and
// (+-1 - i)/sqrt2, and multiplies output k once by W^(r k): 84 instructions
// per 8 elements instead of 96, 28 per 4 instead of 32.
template <int RB>
__device__ __forceinline__ void dft_small_d(double2 (&x)[1 << RB])
{
    constexpr int M = 1 << RB;
#pragma unroll
    for (int j = 0; j < RB; j++) {
        const int dm = M >> (j + 1);
#pragma unroll
        for (int m = 0; m < M; m++) {
            if (m & dm) continue;
            const double2 u = x[m], t = csub(u, x[m + dm]);
            x[m] = cadd(u, x[m + dm]);
            // times exp(-i pi e / 4)
            const int e = (m & (dm - 1)) * (4 / dm);
            constexpr double h = 0.70710678118654752440;
            if (e == 0) x[m + dm] = t;
            else if (e == 2) x[m + dm] = make_double2(t.y, -t.x);
            else if (e == 1) x[m + dm] = make_double2((t.x + t.y) * h, (t.y - t.x) * h);
            else x[m + dm] = make_double2((t.y - t.x) * h, -(t.x + t.y) * h);
        }
    }
}
// register m of dft_small_d holds output k = bitrev(m); its factor W^(r k), the
// table's half period continued by its sign
template <int RB>
__device__ __forceinline__ double2 twiddle_d(int r, int m, int ts)
{
    const int k = RB == 1 ? 1 : RB == 2 ? ((m & 1) << 1) | (m >> 1) : ((m & 1) << 2) | (m & 2) | (m >> 2);
    const int idx = r * k * ts;
    const double2 w = tw<double>(idx & (kTwN / 2 - 1));
    return (idx & (kTwN / 2)) ? make_double2(-w.x, -w.y) : w;
}

template <int RB>
__device__ __forceinline__ void fft_reg_pass_d(double2 *buf, int nsub, int lg, int hl)
{
    constexpr int M = 1 << RB;
    const int q = hl - RB + 1;
    const int groups = nsub << (lg - RB);
    const int ts = kTwN >> (hl + 1);
    for (int g = threadIdx.x; g < groups; g += kBlock) {
        const int a = g >> (lg - RB);
        const int rem = g & ((1 << (lg - RB)) - 1);
        const int blk = rem >> q;
        const int r = rem & ((1 << q) - 1);
        double2 *sub = buf + ((size_t)a << lg);
        const int p0 = (blk << (hl + 1)) + r;
        double2 x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = sub[swz(p0 + (m << q), lg)];
        dft_small_d<RB>(x);
        sub[swz(p0, lg)] = x[0];
#pragma unroll
        for (int m = 1; m < M; m++) sub[swz(p0 + (m << q), lg)] = cmul(x[m], twiddle_d<RB>(r, m, ts));
    }
}

// last five stages on 32-element blocks, one block per half-warp with two
// elements per lane (as fft_dif_pair: the lane trades one element with lane
// l ^ h before each stage, so no butterfly is computed twice): 16 FP64
// instructions per element instead of 22
__device__ __forceinline__ void fft_dif_d(double2 *buf, int nsub, int lg)
{
    int hl = lg - 1;
    while (hl >= 5) {
        const int rb = (hl - 4) >= 3 ? 3 : (hl - 4);
        if (rb == 3) fft_reg_pass_d<3>(buf, nsub, lg, hl);
        else if (rb == 2) fft_reg_pass_d<2>(buf, nsub, lg, hl);
        else fft_reg_pass_d<1>(buf, nsub, lg, hl);
        hl -= rb;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int l = lane & 15;
    double2 w[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int hh = 4 - k;
        w[k] = tw<double>((l & ((1 << hh) - 1)) * (kTwN >> (hh + 1)));
    }
    const int blocks = (nsub << lg) >> 5;
    const int npairs = (blocks + 1) >> 1;
    for (int c = threadIdx.x >> 5; c < npairs; c += kBlock >> 5) {
        const int blk = 2 * c + (lane >> 4);
        const bool live = blk < blocks;
        const int e0 = (live ? blk : blocks - 1) << 5;   // a spare half-warp repeats the last block
        double2 *sub = buf + ((e0 >> lg) << lg);
        const int off = e0 & ((1 << lg) - 1);
        double2 u = sub[swz(off + l, lg)], v = sub[swz(off + l + 16, lg)];
        {
            const double2 t = csub(u, v);
            u = cadd(u, v);
            v = cmul(t, w[0]);
        }
#pragma unroll
        for (int k = 1; k < 5; k++) {
            const int h = 16 >> k;
            const bool bit = (l & h) != 0;
            const double2 rcv = shfl_c<double>(bit ? u : v, h);
            if (bit) u = rcv;
            else v = rcv;
            const double2 t = csub(u, v);
            u = cadd(u, v);
            if (k < 3) v = cmul(t, w[k]);
            else if (k == 3) v = (l & 1) ? make_double2(t.y, -t.x) : t;
            else v = t;
        }
        if (live) {
            sub[swz(off + 2 * l, lg)] = u;
            sub[swz(off + 2 * l + 1, lg)] = v;
        }
    }
    __syncthreads();
}

// ----------------------------------------------------------------------------
// the kernel
// ----------------------------------------------------------------------------
// The eccentric anomaly at mean anomaly l (up to a multiple of 2 pi) by Newton's
// iteration from the FP32 solve at l itself, for the third-body pre-pass where
// its series does not apply (periods of days, eccentricities close to 1).  Two
// steps are enough up to e = 1 - 1e-6, at any l; from another spacecraft's anomaly
// the iteration can leave the root near periapsis (e = 0.99, anomalies 0.01 apart).
__device__ __noinline__ double kepler_newton(double l, double e, float ef, const double2 *__restrict__ sct)
{
    constexpr double kRound = 6755399441055744.0;
    const double k = fma(l, kInvTwoPi, kRound) - kRound;
    l = fma(-k, kTwoPiLo, fma(-k, kTwoPi, l));
    const float lf = d2f_scaled(l, 0), uf = kepler_solve_f(fminf(fabsf(lf), (float)kPi), ef);
    double u = f2d_bits(lf < 0.0f ? -uf : uf);
    for (int it = 0; it < 20; it++) {
        double s, c;
        sincos_tab(u, sct, s, c);
        const double f = fma(-e, s, u) - l, f1 = fma(-e, c, 1.0);
        const double d = f / (f1 - 0.5 * f * (e * s) / f1);
        u -= d;
        if (!(fabs(d) > 1e-7)) break;
    }
    return u;
}

// v_LOS of the three spacecraft at one sample (gbgpu/thirdbody.py:228-380), at
// the delayed times x0, x0 - del1, x0 - del2.  The eccentric anomaly u0 of
// spacecraft 1 comes from the FP32 solve; with g = (u0 - e sin u0 - l)/(1 - e cos u0)
// ~ 1e-6 for every spacecraft (their mean anomalies differ by n2 del, del < 9 s)
// the exact anomalies are u0 + d, d the reversion of the Taylor series at u0 to
// g^3 (the terms beyond the first in FP32), so one FP64 sincos and one
// reciprocal serve all three, and sin, cos and 1/(1 - e cos) at u0 + d follow
// from those at u0.  x0l is what the rounding of x0 left off; it and the rounding
// of n2 (x0 - T2) go into l.  A swap step of 1,024 pairs of N = 512 (1,971 FP64
// instructions per sample with a starter, a Newton step, two sincos, sin and
// atan2 per spacecraft, now 558): 3.64 -> 1.36 ms.
__device__ __forceinline__ void vlos3_fp64(const Bin &B, double x0, double x0l, double del1, double del2,
                                           const double2 *__restrict__ sct, double v[3])
{
    constexpr double kRound = 6755399441055744.0;
    const double e = B.kep.e2, eD = B.kep.eD;
    const double dx = x0 - B.T2, M = B.n2 * dx;
    const double k = fma(M, kInvTwoPi, kRound) - kRound;
    const double l = fma(-k, kTwoPi, M) + fma(-k, kTwoPiLo, fma(B.n2, x0l, fma(B.n2, dx, -M)));
    const float lf = d2f_scaled(l, 0);
    const float uf = kepler_solve_f(fminf(fabsf(lf), (float)kPi), B.e2f);
    const double u0 = f2d_bits(lf < 0.0f ? -uf : uf);
    double su, cu;
    sincos_tab(u0, sct, su, cu);
    const double f1 = fma(-e, cu, 1.0), i1 = recip_fp64(f1);
    const double f = fma(-e, su, u0) - l;
    const float suf = d2f_scaled(su, 0), cuf = d2f_scaled(cu, 0), i1f = d2f_scaled(i1, 0);
    const float a = 0.5f * B.e2f * suf * i1f, b = (1.0f / 6.0f) * B.e2f * cuf * i1f;
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const double dm = B.n2 * (s == 1 ? del1 : del2);
        const double g = (s == 0 ? f : f + dm) * i1;
        const float gf = d2f_scaled(g, 0);
        double sn, cs, i;
        if (fabsf(gf) * fmaxf(1.0f, fabsf(a)) < 1e-5f) {
            const double d = -(g + f2d_bits(gf * gf * fmaf(fmaf(2.0f * a, a, -b), gf, a)));
            const float df = d2f_scaled(d, 0);
            sn = fma(d, cu + f2d_bits(df * fmaf(df * (-1.0f / 6.0f), cuf, -0.5f * suf)), su);
            cs = fma(d, f2d_bits(df * fmaf(df * (1.0f / 6.0f), suf, -0.5f * cuf)) - su, cu);
            // 1/(1 - eD cos u) from 1/f1: x = 1 - (1 - eD cos u)/f1
            const double x = fma(-fma(-eD, cs, 1.0), i1, 1.0);
            const float xf = d2f_scaled(x, 0);
            i = fma(i1, x + f2d_bits(xf * fmaf(xf, xf, xf)), i1);
        } else {
            const double u = kepler_newton(s == 0 ? l : l - dm, e, B.e2f, sct);
            sincos_tab(u, sct, sn, cs);
            i = 1.0 / fma(-eD, cs, 1.0);
        }
        v[s] = fma(i, fma(B.kep.ka, sn, B.kep.kb * cs), B.kep.kc);
    }
}

// Third-body pre-passes (gbgpu/thirdbody.py:155-226) for a tile of cnt
// binaries with N = 2^lg samples:
//   A) k.P/c of every spacecraft -> kps, v_LOS -> vl, and g = v_LOS f_GW -> psi
//      (f_GW without fddot del^2/2, < 1e-21 of it);
//   B) trapezoid increments (xi_n - xi_{n-1}) (g_{n-1} + g_n) pi / c -> inc;
//   C) their inclusive prefix sum along n -> psi (the phase added to argS).
// FP64 throughout; inc and kps are scratch of 3 cnt N doubles each.
// Called by every thread of the block (contains barriers).
__device__ __forceinline__ void third_prepass(const Bin *bins, const double *__restrict__ tab,
                                              int cnt, int lg, double step, double Loc,
                                              const double2 *__restrict__ sct, double *psi,
                                              double *vl, double *inc, double *kps)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = 1 << lg, S = cnt << lg;
    for (int m = tid; m < S; m += kBlock) {
        const int p = m >> lg, n = m & (N - 1);
        const Bin &B = bins[p];
        double v[3] = {0.0, 0.0, 0.0}, kP[3] = {0.0, 0.0, 0.0}, fg[3] = {0.0, 0.0, 0.0};
        if (B.valid) {                        // else outputs unused: no Kepler solve
            double kr[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int c = 0; c < 3; c++) {
                kP[0] = fma(B.k[c], __ldg(tab + (size_t)c * N + n), kP[0]);
                kr[0] = fma(B.k[c], __ldg(tab + (size_t)(9 + c) * N + n), kr[0]);
                kr[1] = fma(B.k[c], __ldg(tab + (size_t)(12 + c) * N + n), kr[1]);
            }
            const double tm = f2d_bits((float)n) * step, xi = tm - kP[0];
            const double del1 = Loc * kr[0], del2 = Loc * (kr[0] + kr[1]);
            kP[1] = kP[0] + del1;
            kP[2] = kP[0] + del2;
            vlos3_fp64(B, xi, (tm - xi) - kP[0], del1, del2, sct, v);
            const double fd = fma(B.fddot, xi, B.fdot);
            fg[0] = fma(xi, 0.5 * (fd + B.fdot), B.f0);
            fg[1] = fma(-del1, fd, fg[0]);
            fg[2] = fma(-del2, fd, fg[0]);
        }
#pragma unroll
        for (int s = 0; s < 3; s++) {
            kps[(p * 3 + s) * N + n] = kP[s];
            vl[(p * 3 + s) * N + n] = v[s];
            psi[(p * 3 + s) * N + n] = v[s] * fg[s];
        }
    }
    __syncthreads();
    for (int m = tid; m < S; m += kBlock) {
        const int p = m >> lg, n = m & (N - 1);
#pragma unroll
        for (int s = 0; s < 3; s++) {
            const int o = (p * 3 + s) * N + n;
            double v = 0.0;
            // xi_n - xi_{n-1} = step - (kP_n - kP_{n-1})
            if (n > 0) v = (step - (kps[o] - kps[o - 1])) * (kPi / kCSI) * (psi[o - 1] + psi[o]);
            inc[o] = v;
        }
    }
    __syncthreads();
    // warp per (binary, spacecraft) row
    const int chunk = N >> 5;
    for (int row = warp; row < 3 * cnt; row += kBlock / 32) {
        const double *src = inc + (size_t)row * N + lane * chunk;
        double *dst = psi + (size_t)row * N + lane * chunk;
        double t = 0.0;
        for (int c = 0; c < chunk; c++) t += src[c];
        double incl = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            double y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        double run = incl - t;
        for (int c = 0; c < chunk; c++) {
            run += src[c];
            dst[c] = run;
        }
    }
    __syncthreads();
}

// the sum of conj(d) h / S times the output scale, which is real but for TDI-2: a
// real product keeps an infinite sum (a bin of zero PSD) from meeting 0 * inf
__device__ __forceinline__ double2 scaled_sum(double2 x, double2 scale)
{
    return scale.y == 0.0 ? make_double2(x.x * scale.x, x.y * scale.x) : cmul(x, scale);
}

// one bin's conj(d) h / S and |h|^2 / S added to the sums (gbgpu_utils.cu:172-178)
__device__ __forceinline__ void ll_add_fp64(double2 dA, double2 dE, double2 tA, double2 tE, double SA, double SE,
                                            bool same, double &sr, double &si, double &sh)
{
    const double wA = recip_fp64(SA);
    if (same) {
        // one PSD for both channels: their terms summed, then weighted once
        sr = fma(fma(dE.y, tE.y, fma(dE.x, tE.x, fma(dA.y, tA.y, dA.x * tA.x))), wA, sr);
        si = fma(fma(-dE.y, tE.x, fma(dE.x, tE.y, fma(-dA.y, tA.x, dA.x * tA.y))), wA, si);
        sh = fma(fma(tE.y, tE.y, fma(tE.x, tE.x, fma(tA.y, tA.y, tA.x * tA.x))), wA, sh);
        return;
    }
    const double wE = recip_fp64(SE);
    sr += (dA.x * tA.x + dA.y * tA.y) * wA + (dE.x * tE.x + dE.y * tE.y) * wE;
    si += (dA.x * tA.y - dA.y * tA.x) * wA + (dE.x * tE.y - dE.y * tE.x) * wE;
    sh += (tA.x * tA.x + tA.y * tA.y) * wA + (tE.x * tE.x + tE.y * tE.y) * wE;
}

// one bin of the output windows, from the transformed channels
__device__ __forceinline__ void wave_out_fp64(const KParams &K, const Bin &B, size_t o, int N, double2 X, double2 Y,
                                              double2 Z)
{
    const double is2 = 0.70710678118654752440, is6 = 0.40824829046386301637;
    const double2 Xd = cmul(X, B.scale), Yd = cmul(Y, B.scale), Zd = cmul(Z, B.scale);
    if (K.XYZ) {
        K.XYZ[o] = Xd;
        K.XYZ[o + N] = Yd;
        K.XYZ[o + 2 * N] = Zd;
    }
    if (K.AET) {
        // utility.py:24-38, with the divisions by sqrt 2, 6, 3 as
        // products with their reciprocals (<= 1 ulp apart)
        const double i3 = 0.57735026918962576451;
        K.AET[o] = make_double2((Zd.x - Xd.x) * is2, (Zd.y - Xd.y) * is2);
        K.AET[o + N] = make_double2((Xd.x - 2.0 * Yd.x + Zd.x) * is6, (Xd.y - 2.0 * Yd.y + Zd.y) * is6);
        K.AET[o + 2 * N] = make_double2((Xd.x + Yd.x + Zd.x) * i3, (Xd.y + Yd.y + Zd.y) * i3);
    }
}

// ----------------------------------------------------------------------------
// Few FP64 binaries: a cluster of 2^LC blocks, on as many SMs, per binary.
// One block per binary keeps its SM's FP64 units busy and leaves the other SMs
// idle.  Here block r builds the samples n = k N/2^LC + m of its N/4^LC values
// of m (all k), so that the transform's first stages (one DFT over k) need no
// exchange; their output k goes to the shared memory of block k, whose
// remaining N/2^LC points are a transform of their own.  Then each block writes
// its share of the window, or adds it to the sums or the template, in runs of 32 bins read from
// all blocks; block 0 adds up the sums.
// MODE_WAVE, MODE_LL and MODE_FILL, equal arms, 9 parameters, one N, with a
// workspace.
// Bound by the serial chain of one sample's FP64 instructions (a warp's cost 64
// cycles each) and its set-up in prep_kernel, no longer by one SM's FP64 units.
// One window of N = 1024: 133 -> 35 us, of N = 4096: 520 -> 80 us, both kernels.
// ----------------------------------------------------------------------------
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// address in block `rank` of the cluster of what is at p in this block
__device__ __forceinline__ unsigned cluster_addr(const void *p, int rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(unsigned a, double2 v)
{
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ double2 cluster_load(unsigned a)
{
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}

template <int MODE, int LC>
__global__ void __launch_bounds__(kBlock, 2) wave_cluster_kernel(const KParams K)
{
    constexpr int NCH = MODE == MODE_WAVE ? 3 : 2, ncl = 1 << LC;
    extern __shared__ __align__(16) unsigned char smem[];
    const gbx_wave_args &a = K.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slot = blockIdx.x >> LC, rank = blockIdx.x & (ncl - 1);
    const int lg = 31 - __clz(a.N), N = 1 << lg, lq = lg - LC, lr = lq - LC, Q = 1 << lq;
    Bin &B = *reinterpret_cast<Bin *>(smem);
    double2 *red = reinterpret_cast<double2 *>(smem + sizeof(Bin));       // block 0: [ncl][2]
    double2 *sct = red + 2 * ncl;
    double2 *own = sct + kScN;              // [NCH][Q] this block's samples
    double2 *buf = own + NCH * Q;           // [NCH][Q] this block's part of the transforms
    __shared__ double part[kBlock / 32][3];
    const double *tab = reinterpret_cast<const double *>(a.orbit[lg]);
    for (int k = tid; k < kScN; k += kBlock) sct[k] = g_sc_d[k];
    const int4 *src = reinterpret_cast<const int4 *>(static_cast<const Bin *>(a.workspace) + slot);
    for (int k = tid; k < (int)(sizeof(Bin) / 16); k += kBlock) reinterpret_cast<int4 *>(smem)[k] = src[k];
    __syncthreads();

    const double step = a.T * exp2_int(-lg);
    const bool chirp = fmaf(fabsf(B.fddotf), (float)a.T, fabsf(B.fdotf)) * K.T2f > 0.3f;
    for (int q = tid; q < Q; q += kBlock) {
        const int n = ((q >> lr) << lq) + (rank << lr) + (q & ((1 << lr) - 1));
        double2 o[3];
        if (B.valid) {
            slow_fp64<false, NCH == 2>(B, n, N, f2d_bits((float)n) * step, tab, K.Loc, sct, chirp, nullptr, nullptr, o);
        } else {
            o[0] = o[1] = o[2] = make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int c = 0; c < NCH; c++) own[(c << lq) + q] = o[c];
    }
    // (every block of the cluster runs before any writes into its memory)
    cluster_sync();
    for (int g = tid; g < (NCH << lr); g += kBlock) {
        const int c = g >> lr, ml = g & ((1 << lr) - 1), r = (rank << lr) + ml;
        double2 x[ncl];
#pragma unroll
        for (int k = 0; k < ncl; k++) x[k] = own[(c << lq) + (k << lr) + ml];
        dft_small_d<LC>(x);
        const double2 *dst = buf + (c << lq) + swz(r, lq);
        cluster_store(cluster_addr(dst, 0), x[0]);
#pragma unroll
        for (int m = 1; m < ncl; m++) cluster_store(cluster_addr(dst, m), cmul(x[m], twiddle_d<LC>(r, m, kTwN >> lg)));
    }
    cluster_sync();
    fft_dif_d(buf, NCH, lq);
    cluster_sync();

    double sr = 0.0, si = 0.0, sh = 0.0;
    bool out = false;
    for (int i = (warp * ncl + rank) * 32 + lane; i < N; i += ncl * kBlock) {
        const int pos = bitrev((i + (N >> 1)) & (N - 1), lg);    // fftshift
        const unsigned h = cluster_addr(buf + swz(pos & (Q - 1), lq), pos >> lq);
        if constexpr (MODE == MODE_WAVE) {
            if (B.b < 0) continue;
            wave_out_fp64(K, B, (size_t)B.b * 3 * N + i, N, cluster_load(h), cluster_load(h + (unsigned)(Q * 16)),
                          cluster_load(h + (unsigned)(Q * 32)));
            if (i == 0 && K.start_out) K.start_out[B.b] = B.start;
        } else if constexpr (MODE == MODE_FILL) {
            const int j = B.start + i;
            if (!B.valid || j < 0 || j >= K.L) continue;
            const double2 hA = cmul(cluster_load(h), B.scale), hE = cmul(cluster_load(h + (unsigned)(Q * 16)), B.scale);
            const size_t o = (size_t)B.gi * K.gstride + j;
            atomicAdd(&K.A_glob[o].x, hA.x);
            atomicAdd(&K.A_glob[o].y, hA.y);
            atomicAdd(&K.E_glob[o].x, hE.x);
            atomicAdd(&K.E_glob[o].y, hE.y);
        } else {
            const int j = B.start + i;
            if (!B.valid) continue;
            if (j < 0 || j >= K.L) {
                out = true;
                continue;
            }
            const size_t jd = (size_t)B.di * K.L + j, jn = (size_t)B.ni * K.L + j;
            const bool same = K.A_psd == K.E_psd;
            const double SA = __ldg(K.A_psd + jn), SE = same ? SA : __ldg(K.E_psd + jn);
            ll_add_fp64(__ldg(K.A_data + jd), __ldg(K.E_data + jd), cluster_load(h),
                        cluster_load(h + (unsigned)(Q * 16)), SA, SE, same, sr, si, sh);
        }
    }
    if constexpr (MODE == MODE_LL) {
        if (out) flag(a.status, GBX_FLAG_WINDOW);
        for (int o = 16; o > 0; o >>= 1) {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            si += __shfl_xor_sync(0xffffffffu, si, o);
            sh += __shfl_xor_sync(0xffffffffu, sh, o);
        }
        if (lane == 0) {
            part[warp][0] = sr;
            part[warp][1] = si;
            part[warp][2] = sh;
        }
        __syncthreads();
        if (tid == 0) {
            double t[3] = {0.0, 0.0, 0.0};
            for (int w = 0; w < kBlock / 32; w++)
                for (int k = 0; k < 3; k++) t[k] += part[w][k];
            cluster_store(cluster_addr(red + 2 * rank, 0), make_double2(t[0], t[1]));
            cluster_store(cluster_addr(red + 2 * rank + 1, 0), make_double2(t[2], 0.0));
        }
    }
    // (no block leaves while others read its memory)
    cluster_sync();
    if constexpr (MODE == MODE_LL) {
        if (rank == 0 && tid == 0 && B.b >= 0) {
            double2 d = make_double2(0.0, 0.0);
            double h = 0.0;
            for (int r = 0; r < ncl; r++) {
                d = cadd(d, red[2 * r]);
                h += red[2 * r + 1].x;
            }
            const double s4 = 4.0 * K.df;
            const double ch = s4 * (B.scale.x * B.scale.x + B.scale.y * B.scale.y);
            K.d_h[B.b] = B.valid ? scaled_sum(make_double2(s4 * d.x, s4 * d.y), B.scale) : make_double2(0.0, 0.0);
            K.h_h[B.b] = make_double2(B.valid ? ch * h : 0.0, 0.0);
        }
    }
}

// Third-body pre-passes of the mixed form for a tile of cnt binaries with
// N = 2^lg samples (the same model as third_prepass above, without FP64 work
// per spacecraft):
//   A) spacecraft 1: delayed time in FP64, one Kepler solve for v_LOS and
//      dv/dt (vlos_dt_mixed); spacecraft 2, 3: v_LOS linearised in their
//      k.P/c offsets (FP32, <= L/c = 8.3 s; the second-order error is below
//      3e-9 v for P2 >= 1 yr); g = v_LOS f_GW in FP32 -> gout;
//      k.P/c of every spacecraft in FP32 -> kps (scratch);
//   B) increments (xi_n - xi_{n-1}) (g_{n-1} + g_n) pi / c with
//      xi_n - xi_{n-1} = T/N - (kP_n - kP_{n-1}) (T/N as a float pair), and
//      their inclusive prefix sum along n as float pairs -> psi.
// Called by every thread of the block (contains barriers).
__device__ __forceinline__ void third_prepass_mixed(const Bin *bins, const double *__restrict__ tab,
                                                    int cnt, int lg, dfl stp, dfl *psi,
                                                    float *vl, float *kps, float *gout)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = 1 << lg, S = cnt << lg;
    const float *tabf = reinterpret_cast<const float *>(tab + (size_t)18 * N);
    for (int m = tid; m < S; m += kBlock) {
        const int p = m >> lg, n = m & (N - 1);
        const Bin &B = bins[p];
        if (!B.valid) {                       // outputs unused: no Kepler solve
#pragma unroll
            for (int s = 0; s < 3; s++) {
                vl[(p * 3 + s) * N + n] = 0.0f;
                kps[(p * 3 + s) * N + n] = 0.0f;
                gout[(p * 3 + s) * N + n] = 0.0f;
            }
            continue;
        }
        // spacecraft 1's delayed time n T/N - k.P_1/c as a float pair
        const dfl xi0 = df_add(df_mul_f(stp, (float)n), df_neg(kP1_pair(B, tabf, N, n)));
        float dv0;
        const float v0 = vlos_dt_mixed(xi0, B, dv0);
        float kPf[3];
#pragma unroll
        for (int s = 0; s < 3; s++)
            kPf[s] = fmaf(B.kf[0], __ldg(tabf + (size_t)(9 + 3 * s) * N + n),
                          fmaf(B.kf[1], __ldg(tabf + (size_t)(9 + 3 * s + 1) * N + n),
                               B.kf[2] * __ldg(tabf + (size_t)(9 + 3 * s + 2) * N + n)));
        const float x0 = xi0.h + xi0.l;
#pragma unroll
        for (int s = 0; s < 3; s++) {
            const float dk = s ? kPf[s] - kPf[0] : 0.0f;   // xi_s = xi_1 - dk
            const float v = fmaf(-dv0, dk, v0);
            const float xf = x0 - dk;
            const float fgw = fmaf(fmaf(0.5f * B.fddotf, xf, B.fdotf), xf, B.f0f);
            vl[(p * 3 + s) * N + n] = v;
            kps[(p * 3 + s) * N + n] = kPf[s];
            gout[(p * 3 + s) * N + n] = v * fgw;
        }
    }
    __syncthreads();
    // warp per (binary, spacecraft) row; lane owns a chunk of N/32 samples
    const float k = (float)(kPi / kCSI);
    const int chunk = N >> 5;
    for (int row = warp; row < 3 * cnt; row += kBlock / 32) {
        const float *kr = kps + (size_t)row * N, *gr = gout + (size_t)row * N;
        dfl *dst = psi + (size_t)row * N;
        const int c0 = lane * chunk;
        auto inc = [&](int n) -> float {
            if (n == 0) return 0.0f;
            const float d = (stp.h - (kr[n] - kr[n - 1])) + stp.l;
            return d * (gr[n - 1] + gr[n]) * k;
        };
        dfl t = {0.0f, 0.0f};
        for (int c = 0; c < chunk; c++) t = df_add(t, dfl{inc(c0 + c), 0.0f});
        dfl incl = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const dfl y = {__shfl_up_sync(0xffffffffu, incl.h, o), __shfl_up_sync(0xffffffffu, incl.l, o)};
            if (lane >= o) incl = df_add(incl, y);
        }
        dfl run = df_add(incl, df_neg(t));
        for (int c = 0; c < chunk; c++) {
            run = df_add(run, dfl{inc(c0 + c), 0.0f});
            dst[c0 + c] = run;
        }
    }
    __syncthreads();
}

// Runs of a fill tile (MODE_FILL, called by one thread): consecutive tile
// slots with one group and ascending starts less than N apart cover one
// contiguous span of output bins.  Run r holds slots run[r] .. run[r+1]-1,
// spans lo[r] .. lo[r] + off[r+1] - off[r] - 1; an invalid binary's run is
// empty; returns the number of runs.
__device__ __forceinline__ int fill_runs(const Bin *bins, int cnt, int N, int *run, int *lo, int *off)
{
    int nr = 0, acc = 0, hi = 0;
    for (int p = 0; p < cnt; p++) {
        const Bin &B = bins[p];
        const bool join = nr > 0 && B.valid && bins[p - 1].valid && B.gi == bins[p - 1].gi &&
                          B.start >= bins[p - 1].start && B.start - bins[p - 1].start < N;
        if (!join) {
            if (nr > 0) acc += hi - lo[nr - 1];
            off[nr] = acc;
            run[nr] = p;
            lo[nr] = B.start;
            nr++;
        }
        // a run's last member ends its span; an invalid binary's run is empty
        hi = B.valid ? B.start + N : lo[nr - 1];
    }
    acc += hi - lo[nr - 1];
    off[nr] = acc;
    run[nr] = cnt;
    return nr;
}

template <typename R, int MODE, bool THIRD, bool UNEQ>
__global__ void __launch_bounds__(kBlock, sizeof(R) == 4 ? 3 : 2) wave_kernel(const KParams K)
{
    using V = typename C2<R>::T;
    // transformed channels: X, Y, Z for the waveform outputs; A, E otherwise
    constexpr int NCH = MODE == MODE_WAVE ? 3 : 2;
    const R is2 = (R)0.70710678118654752440, is6 = (R)0.40824829046386301637;
    extern __shared__ __align__(16) unsigned char smem[];
    Bin *bins = reinterpret_cast<Bin *>(smem);
    double *red = reinterpret_cast<double *>(smem + sizeof(Bin) * K.maxP);
    // FP64 form: the sin/cos table lies between the reduction scratch and buf
    constexpr int kSc = sizeof(R) == 8 ? kScN : 0;
    double2 *sct = reinterpret_cast<double2 *>(smem + sizeof(Bin) * K.maxP +
                                               sizeof(double) * red_doubles(K.maxS));
    V *buf = reinterpret_cast<V *>(sct + kSc);
    __shared__ int s_tile;

    const gbx_wave_args &a = K.a;
    const int tid = threadIdx.x;
    for (int k = tid; k < kSc; k += kBlock) sct[k] = g_sc_d[k];
    const int ntiles = a.tiles ? a.ntiles : (a.num_bin + K.P - 1) / K.P;
    const double fstar = K.fstar;
    const float Loc = (float)(1.0 / (kTwoPi * fstar));         // L / c
    int iter = 0;

    for (;;) {
        if (tid == 0) {
            if (a.queue) s_tile = atomicAdd(a.queue, 1);
            else s_tile = blockIdx.x + iter * gridDim.x;
        }
        __syncthreads();
        const int tile = s_tile;
        iter++;
        if (tile >= ntiles) break;
        int lg, first, cnt;
        if (a.tiles) {
            lg = a.tiles[4 * tile];
            first = a.tiles[4 * tile + 1];
            cnt = a.tiles[4 * tile + 2];
        } else {
            lg = 31 - __clz(a.N);
            first = tile * K.P;
            cnt = min(K.P, a.num_bin - first);
        }
        const int N = 1 << lg;
        const double *tab = (lg >= 5 && lg <= GBX_MAX_LOG2N)
                                ? reinterpret_cast<const double *>(a.orbit[lg]) : nullptr;
        const int maxcnt = tile_pack(a.tile, lg, MODE == MODE_SWAP ? 2 : 1);
        if (tab == nullptr || cnt < 1 || cnt > maxcnt || first < 0 || first + cnt > a.num_bin ||
            (cnt << lg) > K.maxS || (sizeof(R) == 8 && lg > 12)) {
            flag(a.status, GBX_FLAG_TILE);
            __syncthreads();
            continue;
        }
        if (a.workspace) {
            // per-binary constants were prepared by prep_kernel: copy them in
            const int4 *src = reinterpret_cast<const int4 *>(
                static_cast<const Bin *>(a.workspace) + first);
            int4 *dst = reinterpret_cast<int4 *>(bins);
            const int n16 = cnt * (int)(sizeof(Bin) / 16);
            for (int k = tid; k < n16; k += kBlock) dst[k] = src[k];
        } else if (tid < cnt) {
            int slot = first + tid;
            int b = a.order ? a.order[slot] : slot;
            if (b < 0 || b >= a.num_bin) {
                flag(a.status, GBX_FLAG_TILE);
                memset(&bins[tid], 0, sizeof(Bin));
                bins[tid].b = -1;
            } else {
                setup_bin(bins[tid], K, b, N, MODE);
            }
        }
        __syncthreads();

        const int S = cnt << lg;                 // samples in this tile
        const double step = a.T * exp2_int(-lg);  // tm = n T/N (gbgpu.py:269), exact
        const dfl stepd = K.stepd[lg];

        double *psi = nullptr;          // FP64 form: cumulative Doppler phase
        dfl *psif = nullptr;            // mixed form: the same as float pairs
        R *vl = nullptr;
        if (THIRD) {
            if constexpr (sizeof(R) == 8) {
                psi = reinterpret_cast<double *>(buf + 3 * (size_t)maxcnt * N);
                vl = reinterpret_cast<R *>(psi + 3 * (size_t)maxcnt * N);
                double *scr = reinterpret_cast<double *>(buf);
                third_prepass(bins, tab, cnt, lg, step, K.Loc, sct, psi, vl, scr,
                              scr + 3 * (size_t)maxcnt * N);
            } else {
                // scratch: k.P/c and g in buf (6 floats per sample there)
                psif = reinterpret_cast<dfl *>(buf + 3 * (size_t)maxcnt * N);
                vl = reinterpret_cast<R *>(psif + 3 * (size_t)maxcnt * N);
                float *scr = reinterpret_cast<float *>(buf);
                third_prepass_mixed(bins, tab, cnt, lg, stepd, psif, reinterpret_cast<float *>(vl), scr,
                                    scr + 3 * (size_t)maxcnt * N);
            }
        }

        // slow part -> buf[(p*3 + channel)*N + n]
        for (int m = tid; m < S; m += kBlock) {
            const int p = m >> lg, n = m & (N - 1);
            const Bin &B = bins[p];
            const double tm = f2d_bits((float)n) * step;
            double ps[3] = {0.0, 0.0, 0.0};
            dfl psf[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
            R vv[3] = {0, 0, 0};
            if (THIRD) {
#pragma unroll
                for (int s = 0; s < 3; s++) {
                    if constexpr (sizeof(R) == 8) ps[s] = psi[(p * 3 + s) * N + n];
                    else psf[s] = psif[(p * 3 + s) * N + n];
                    vv[s] = vl[(p * 3 + s) * N + n];
                }
            }
            V o[3];
            if (!B.valid) {
                // nothing of this binary reaches the outputs (bad index, or a
                // zero-amplitude fill): skip the slow part
                o[0] = o[1] = o[2] = V{0, 0};
            } else if constexpr (sizeof(R) == 8 && !UNEQ) {
                const bool chirp = fmaf(fabsf(B.fddotf), (float)a.T, fabsf(B.fdotf)) * K.T2f > 0.3f;
                slow_fp64<THIRD, NCH == 2>(B, n, N, tm, tab, K.Loc, sct, chirp, ps, vv, o);
            } else if constexpr (sizeof(R) == 8) {
                slow_links_fp64(B, n, N, tm, a.tdi2, tab, fstar, o);
            } else {
                slow_mixed<THIRD>(B, n, N, stepd, Loc, tab, psf, vv, o);
            }
            if constexpr (NCH == 3 || (sizeof(R) == 8 && !UNEQ)) {
#pragma unroll
                for (int c = 0; c < NCH; c++) buf[(p * NCH + c) * N + swz(n, lg)] = o[c];
            } else {
                // A = (Z - X)/sqrt2, E = (X - 2Y + Z)/sqrt6 (utility.py:24-38) formed
                // before the transform: the FFT is linear, so two transforms suffice
                buf[(p * 2 + 0) * N + swz(n, lg)] = {(o[2].x - o[0].x) * is2, (o[2].y - o[0].y) * is2};
                buf[(p * 2 + 1) * N + swz(n, lg)] = {(o[0].x - 2 * o[1].x + o[2].x) * is6,
                                                     (o[0].y - 2 * o[1].y + o[2].y) * is6};
            }
        }
        __syncthreads();

        if constexpr (sizeof(R) == 8) fft_dif_d(buf, NCH * cnt, lg);
        else fft_dif<R>(buf, NCH * cnt, lg);

        // ------------------------------------------------------------ epilogue
        if (MODE == MODE_WAVE) {
            for (int m = tid; m < S; m += kBlock) {
                const int p = m >> lg, i = m & (N - 1);
                const Bin &B = bins[p];
                if (B.b < 0) continue;
                const int pos = bitrev((i + (N >> 1)) & (N - 1), lg);   // fftshift
                V X = buf[(p * 3 + 0) * N + swz(pos, lg)], Y = buf[(p * 3 + 1) * N + swz(pos, lg)],
                  Z = buf[(p * 3 + 2) * N + swz(pos, lg)];
                const size_t o = (size_t)B.b * 3 * N + i;
                if constexpr (sizeof(R) == 8) {
                    wave_out_fp64(K, B, o, N, X, Y, Z);
                } else {
                    // mixed form: the channels and the scale in FP32 (the values
                    // carry FP32 accuracy), widened to FP64 on the integer pipe
                    const float2 sc = make_float2(d2f_scaled(B.scale.x, 0), d2f_scaled(B.scale.y, 0));
                    if (K.XYZ) {
                        K.XYZ[o] = f2d(cmul(X, sc));
                        K.XYZ[o + N] = f2d(cmul(Y, sc));
                        K.XYZ[o + 2 * N] = f2d(cmul(Z, sc));
                    }
                    if (K.AET) {
                        const float i3 = 0.57735026918962576451f;
                        K.AET[o] = f2d(cmul(make_float2((Z.x - X.x) * is2, (Z.y - X.y) * is2), sc));
                        K.AET[o + N] = f2d(cmul(make_float2((X.x - 2.f * Y.x + Z.x) * is6,
                                                            (X.y - 2.f * Y.y + Z.y) * is6), sc));
                        K.AET[o + 2 * N] = f2d(cmul(make_float2((X.x + Y.x + Z.x) * i3,
                                                                (X.y + Y.y + Z.y) * i3), sc));
                    }
                }
                if (i == 0 && K.start_out) K.start_out[B.b] = B.start;
            }
        } else if (MODE == MODE_SWAP) {
            // binaries 2j (current source) and 2j+1 (proposal) of the tile form a
            // pair; threads [j*Tp2, (j+1)*Tp2) walk both windows.  With r the
            // residual row and Dh = h_new - h_old:
            //   dlogL = Re<r|Dh> - 1/2 <Dh|Dh>
            //         = Re<r|h_new> - Re<r|h_old> - (<h_new|h_new> + <h_old|h_old>)/2
            //           + Re<h_old|h_new>   (cross term on the windows' overlap)
            const int Tp2 = 2 * (kBlock / maxcnt);
            const int width = Tp2 < 32 ? Tp2 : 32;
            const int pr = tid / Tp2;
            const int i0 = tid - pr * Tp2;
            typedef typename std::conditional<sizeof(R) == 8, double, float>::type Acc;
            Acc acc8[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // Crn (2), Cro (2), Hn, Ho, Cx (2)
            const bool realsum = a.tdi2 != GBX_TDI2_BIT;
            // mixed form: FP32 sums over columns of the default tile's threads,
            // float pairs over the columns (as the likelihood)
            dfl tot8[8];
#pragma unroll
            for (int k = 0; k < 8; k++) tot8[k] = dfl{0.f, 0.f};
            const int Tv = sizeof(R) == 8 ? Tp2 : 2 * (kBlock / tile_pack(0, lg, 2));
            if (2 * pr + 1 < cnt) {
                const Bin &Bo = bins[2 * pr], &Bn = bins[2 * pr + 1];
                const int po = 2 * pr, pn = 2 * pr + 1;
                if (Bo.valid && Bn.valid) {
                    bool out = false;
                  for (int v = i0; v < Tv; v += Tp2) {
                    for (int e = v; e < 2 * N; e += Tv) {
                        const bool isnew = e < N;
                        const int i = isnew ? e : e - N;
                        const Bin &Bw = isnew ? Bn : Bo;
                        const int pw = isnew ? pn : po;
                        const int j = Bw.start + i;
                        if (j < 0 || j >= K.L) {
                            out = true;
                            continue;
                        }
                        const int pos = bitrev((i + (N >> 1)) & (N - 1), lg);
                        const V hA = buf[(pw * 2 + 0) * N + swz(pos, lg)], hE = buf[(pw * 2 + 1) * N + swz(pos, lg)];
                        const size_t jd = (size_t)Bn.di * K.L + j, jn = (size_t)Bn.ni * K.L + j;
                        const double2 dA = __ldg(K.A_data + jd), dE = __ldg(K.E_data + jd);
                        const double SA = __ldg(K.A_psd + jn), SE = __ldg(K.E_psd + jn);
                        Acc wA, wE, aR, aI, eR, eI;
                        if constexpr (sizeof(R) == 8) {
                            wA = recip_fp64(SA);
                            wE = K.A_psd == K.E_psd ? wA : recip_fp64(SE);
                            aR = dA.x; aI = dA.y; eR = dE.x; eI = dE.y;
                        } else {
                            wA = __frcp_rn(d2f_scaled(SA, Bn.eS));
                            wE = __frcp_rn(d2f_scaled(SE, Bn.eS));
                            aR = d2f_scaled(dA.x, Bn.eD); aI = d2f_scaled(dA.y, Bn.eD);
                            eR = d2f_scaled(dE.x, Bn.eD); eI = d2f_scaled(dE.y, Bn.eD);
                        }
                        const Acc hAr = hA.x, hAi = hA.y, hEr = hE.x, hEi = hE.y;
                        if constexpr (sizeof(R) == 8) {
                            if (realsum && K.A_psd == K.E_psd) {
                                // one weight per bin; the imaginary parts only
                                // meet complex (TDI-2) scales
                                const Acc cr = fma(eI, hEi, fma(eR, hEr, fma(aI, hAi, aR * hAr)));
                                const Acc hh2 = fma(hEi, hEi, fma(hEr, hEr, fma(hAi, hAi, hAr * hAr)));
                                acc8[isnew ? 0 : 2] = fma(cr, wA, acc8[isnew ? 0 : 2]);
                                acc8[isnew ? 4 : 5] = fma(hh2, wA, acc8[isnew ? 4 : 5]);
                                const int k = j - Bo.start;
                                if (isnew && k >= 0 && k < N) {
                                    const int pk = bitrev((k + (N >> 1)) & (N - 1), lg);
                                    const V oA = buf[(po * 2 + 0) * N + swz(pk, lg)],
                                            oE = buf[(po * 2 + 1) * N + swz(pk, lg)];
                                    acc8[6] = fma(fma(oE.y, hEi, fma(oE.x, hEr, fma(oA.y, hAi, oA.x * hAr))),
                                                  wA, acc8[6]);
                                }
                                continue;
                            }
                        }
                        // conj(r) h / S
                        const Acc cr = (aR * hAr + aI * hAi) * wA + (eR * hEr + eI * hEi) * wE;
                        const Acc ci = (aR * hAi - aI * hAr) * wA + (eR * hEi - eI * hEr) * wE;
                        const Acc hh2 = (hAr * hAr + hAi * hAi) * wA + (hEr * hEr + hEi * hEi) * wE;
                        if (isnew) {
                            acc8[0] += cr; acc8[1] += ci; acc8[4] += hh2;
                            const int k = j - Bo.start;
                            if (k >= 0 && k < N) {
                                const int pk = bitrev((k + (N >> 1)) & (N - 1), lg);
                                const V oA = buf[(po * 2 + 0) * N + swz(pk, lg)],
                                        oE = buf[(po * 2 + 1) * N + swz(pk, lg)];
                                const Acc oAr = oA.x, oAi = oA.y, oEr = oE.x, oEi = oE.y;
                                // conj(h_old) h_new / S
                                acc8[6] += (oAr * hAr + oAi * hAi) * wA + (oEr * hEr + oEi * hEi) * wE;
                                acc8[7] += (oAr * hAi - oAi * hAr) * wA + (oEr * hEi - oEi * hEr) * wE;
                            }
                        } else {
                            acc8[2] += cr; acc8[3] += ci; acc8[5] += hh2;
                        }
                    }
                    if constexpr (sizeof(R) == 4) {
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            tot8[k] = df_add(tot8[k], dfl{acc8[k], 0.f});
                            acc8[k] = 0;
                        }
                    }
                  }
                    if (out) flag(a.status, GBX_FLAG_WINDOW);
                }
            }
            {
                // group trees; only the group leaders convert to FP64
                const bool leader = (tid & (width - 1)) == 0;
                const int g = tid / width;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    if constexpr (sizeof(R) == 8) {
                        double x = acc8[k];
                        for (int o = width >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                        if (leader) red[8 * g + k] = x;
                    } else {
                        dfl x = tot8[k];
                        for (int o = width >> 1; o > 0; o >>= 1) {
                            dfl y = {__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o)};
                            x = df_add(x, y);
                        }
                        if (leader) red[8 * g + k] = (double)x.h + (double)x.l;
                    }
                }
            }
            __syncthreads();
            if (2 * tid + 1 < cnt) {
                const Bin &Bo = bins[2 * tid], &Bn = bins[2 * tid + 1];
                const int per = Tp2 / width;
                double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                for (int g = tid * per; g < (tid + 1) * per; g++)
#pragma unroll
                    for (int k = 0; k < 8; k++) t[k] += red[8 * g + k];
                double cdh = 4.0 * K.df, chh = 4.0 * K.df;
                if constexpr (sizeof(R) == 4) {
                    cdh *= exp2_int(Bn.eS - Bn.eD);
                    chh *= exp2_int(Bn.eS);
                }
                const double2 so = Bo.scale, sn = Bn.scale;
                const double rn = cmul(sn, make_double2(t[0], t[1])).x * cdh;
                const double ro = cmul(so, make_double2(t[2], t[3])).x * cdh;
                const double hn = (sn.x * sn.x + sn.y * sn.y) * t[4] * chh;
                const double ho = (so.x * so.x + so.y * so.y) * t[5] * chh;
                const double cx = cmul(make_double2(so.x, -so.y), cmul(sn, make_double2(t[6], t[7]))).x * chh;
                const bool ok = Bo.valid && Bn.valid && Bo.b >= 0 && Bn.b >= 0;
                if (Bn.b >= 0) K.dlogl[Bn.b >> 1] = ok ? (rn - ro - 0.5 * (hn + ho) + cx) : 0.0;
            }
        } else if (MODE == MODE_FILL) {
            // Pre-reduction: a run of consecutive tile slots with one group and
            // ascending starts less than N apart covers one contiguous span of
            // output bins; every bin of the span is summed over the run's
            // windows here and added with one atomic per component, instead of
            // one per window (a tile of binaries sorted by group and frequency
            // in a dense band needs a fraction of the atomics).  Unsorted
            // input gives runs of one binary: one atomic per window bin.
            __shared__ int s_run[kMaxPack + 1], s_lo[kMaxPack], s_off[kMaxPack + 1];
            __shared__ int s_nruns;
            // mixed form: the scale in FP32 (the values carry FP32 accuracy),
            // the product widened to FP64 on the integer pipe, as MODE_WAVE
            __shared__ float2 s_scf[kMaxPack];
            if (sizeof(R) == 4 && tid < cnt)
                s_scf[tid] = make_float2(d2f_scaled(bins[tid].scale.x, 0), d2f_scaled(bins[tid].scale.y, 0));
            if (tid == 0) s_nruns = fill_runs(bins, cnt, N, s_run, s_lo, s_off);
            __syncthreads();
            const int nr = s_nruns;
            const int U = s_off[nr];
            for (int m = tid; m < U; m += kBlock) {
                int r = 0;
                while (r + 1 < nr && s_off[r + 1] <= m) r++;
                const int j = s_lo[r] + (m - s_off[r]);
                if (j < 0 || j >= K.L) continue;
                double2 Ah = make_double2(0.0, 0.0), Eh = make_double2(0.0, 0.0);
                bool any = false;
                for (int p = s_run[r]; p < s_run[r + 1]; p++) {
                    const Bin &B = bins[p];
                    const int i = j - B.start;
                    if (i < 0 || i >= N) continue;
                    const int pos = bitrev((i + (N >> 1)) & (N - 1), lg);
                    const V hA = buf[(p * 2 + 0) * N + swz(pos, lg)], hE = buf[(p * 2 + 1) * N + swz(pos, lg)];
                    double2 a2, e2;
                    if constexpr (sizeof(R) == 4) {
                        a2 = f2d(cmul(hA, s_scf[p]));
                        e2 = f2d(cmul(hE, s_scf[p]));
                    } else {
                        a2 = cmul(make_double2(hA.x, hA.y), B.scale);
                        e2 = cmul(make_double2(hE.x, hE.y), B.scale);
                    }
                    // the first window adds nothing in FP64; later ones add in FP64
                    if (any) {
                        Ah = cadd(Ah, a2);
                        Eh = cadd(Eh, e2);
                    } else {
                        Ah = a2;
                        Eh = e2;
                        any = true;
                    }
                }
                const size_t o = (size_t)bins[s_run[r]].gi * K.gstride + j;
                atomicAdd(&K.A_glob[o].x, Ah.x);
                atomicAdd(&K.A_glob[o].y, Ah.y);
                atomicAdd(&K.E_glob[o].x, Eh.x);
                atomicAdd(&K.E_glob[o].y, Eh.y);
            }
        } else {  // MODE_LL
            // Threads [p*Tpb, (p+1)*Tpb) own binary p of the tile and walk its
            // window with stride Tpb, so each warp reads a contiguous run of the
            // data/PSD window.  Sums are FP64 (plain form) or, in the mixed form,
            // FP32 over the bins v, v + Tv, v + 2 Tv ... of a column v, Tv being
            // the threads a binary has in a tile of kTileMin samples, and in
            // float pairs over the columns: the FP32 sums (2 to 32 terms), and
            // so the result, do not depend on the tile.  Lanes are combined with
            // an FP64 or float-pair shuffle tree, and a binary's <= 16 group
            // partials are added by one thread per (binary, term).
            const int Tpb = kBlock / maxcnt;               // 256 / binaries per tile
            const int width = Tpb < 32 ? Tpb : 32;
            const int p = tid / Tpb;
            const int i0 = tid - p * Tpb;
            typedef typename std::conditional<sizeof(R) == 8, double, float>::type Acc;
            Acc sr = 0, si = 0, sh = 0;
            dfl xr = {0.f, 0.f}, xi = {0.f, 0.f}, xh = {0.f, 0.f};
            const int Tv = sizeof(R) == 8 ? Tpb : kBlock / tile_pack(0, lg, 1);
            // one PSD array for both channels (the usual call): the channels'
            // terms are summed, then weighted once
            const bool samepsd = K.A_psd == K.E_psd;
            if (p < cnt) {
                const Bin &B = bins[p];
                bool out = false;
                if (B.valid) {
                  for (int v = i0; v < Tv; v += Tpb) {
                    for (int i = v; i < N; i += Tv) {
                        const int j = B.start + i;
                        if (j < 0 || j >= K.L) {
                            out = true;
                            continue;
                        }
                        const int pos = bitrev((i + (N >> 1)) & (N - 1), lg);
                        const V tA = buf[(p * 2 + 0) * N + swz(pos, lg)], tE = buf[(p * 2 + 1) * N + swz(pos, lg)];
                        const size_t jd = (size_t)B.di * K.L + j, jn = (size_t)B.ni * K.L + j;
                        const double2 dA = __ldg(K.A_data + jd), dE = __ldg(K.E_data + jd);
                        if (samepsd) {
                            const double S = __ldg(K.A_psd + jn);
                            if constexpr (sizeof(R) == 8) {
                                ll_add_fp64(dA, dE, tA, tE, S, S, true, sr, si, sh);
                            } else {
                                const float w = __frcp_rn(d2f_scaled(S, B.eS));
                                const float aR = d2f_scaled(dA.x, B.eD), aI = d2f_scaled(dA.y, B.eD);
                                const float eR = d2f_scaled(dE.x, B.eD), eI = d2f_scaled(dE.y, B.eD);
                                sr = fmaf(fmaf(aR, tA.x, aI * tA.y) + fmaf(eR, tE.x, eI * tE.y), w, sr);
                                si = fmaf(fmaf(aR, tA.y, -aI * tA.x) + fmaf(eR, tE.y, -eI * tE.x), w, si);
                                sh = fmaf(fmaf(tA.x, tA.x, tA.y * tA.y) + fmaf(tE.x, tE.x, tE.y * tE.y), w, sh);
                            }
                            continue;
                        }
                        const double SA = __ldg(K.A_psd + jn), SE = __ldg(K.E_psd + jn);
                        if constexpr (sizeof(R) == 8) {
                            ll_add_fp64(dA, dE, tA, tE, SA, SE, false, sr, si, sh);
                        } else {
                            const float2 hA = tA, hE = tE;
                            const float wA = __frcp_rn(d2f_scaled(SA, B.eS));
                            const float wE = __frcp_rn(d2f_scaled(SE, B.eS));
                            const float aR = d2f_scaled(dA.x, B.eD), aI = d2f_scaled(dA.y, B.eD);
                            const float eR = d2f_scaled(dE.x, B.eD), eI = d2f_scaled(dE.y, B.eD);
                            sr += fmaf(aR, hA.x, aI * hA.y) * wA + fmaf(eR, hE.x, eI * hE.y) * wE;
                            si += fmaf(aR, hA.y, -aI * hA.x) * wA + fmaf(eR, hE.y, -eI * hE.x) * wE;
                            sh += fmaf(hA.x, hA.x, hA.y * hA.y) * wA + fmaf(hE.x, hE.x, hE.y * hE.y) * wE;
                        }
                    }
                    if constexpr (sizeof(R) == 4) {
                        xr = df_add(xr, dfl{sr, 0.f});
                        xi = df_add(xi, dfl{si, 0.f});
                        xh = df_add(xh, dfl{sh, 0.f});
                        sr = si = sh = 0;
                    }
                  }
                }
                if (out) flag(a.status, GBX_FLAG_WINDOW);
            }
            // lane tree within groups of `width` lanes (all lanes take part)
            double gr = 0.0, gi = 0.0, gh = 0.0;
            if constexpr (sizeof(R) == 8) {
                for (int o = width >> 1; o > 0; o >>= 1) {
                    sr += __shfl_xor_sync(0xffffffffu, sr, o);
                    si += __shfl_xor_sync(0xffffffffu, si, o);
                    sh += __shfl_xor_sync(0xffffffffu, sh, o);
                }
                gr = sr; gi = si; gh = sh;
            } else {
                for (int o = width >> 1; o > 0; o >>= 1) {
                    dfl yr = {__shfl_xor_sync(0xffffffffu, xr.h, o), __shfl_xor_sync(0xffffffffu, xr.l, o)};
                    dfl yi = {__shfl_xor_sync(0xffffffffu, xi.h, o), __shfl_xor_sync(0xffffffffu, xi.l, o)};
                    dfl yh = {__shfl_xor_sync(0xffffffffu, xh.h, o), __shfl_xor_sync(0xffffffffu, xh.l, o)};
                    xr = df_add(xr, yr);
                    xi = df_add(xi, yi);
                    xh = df_add(xh, yh);
                }
                // leaders keep the float pairs; the FP64 conversion happens
                // once per (binary, term) below, spread over lanes
                if ((tid & (width - 1)) == 0) {
                    float2 *red2 = reinterpret_cast<float2 *>(red);
                    const int g = tid / width;
                    red2[3 * g] = make_float2(xr.h, xr.l);
                    red2[3 * g + 1] = make_float2(xi.h, xi.l);
                    red2[3 * g + 2] = make_float2(xh.h, xh.l);
                }
            }
            if (sizeof(R) == 8 && (tid & (width - 1)) == 0) {
                const int g = tid / width;
                red[3 * g] = gr;
                red[3 * g + 1] = gi;
                red[3 * g + 2] = gh;
            }
            __syncthreads();
            // per (binary, term) sums over the binary's groups -> tsum (FP64)
            double *tsum = red + 3 * kMaxPack;
            {
                const int per = Tpb / width;
                for (int t = tid; t < 3 * cnt; t += kBlock) {
                    const int q = t / 3, c = t - 3 * q;
                    if constexpr (sizeof(R) == 8) {
                        double x = 0.0;
                        for (int g = q * per; g < (q + 1) * per; g++) x += red[3 * g + c];
                        tsum[t] = x;
                    } else {
                        const float2 *red2 = reinterpret_cast<const float2 *>(red);
                        dfl x = {0.f, 0.f};
                        for (int g = q * per; g < (q + 1) * per; g++) {
                            const float2 y = red2[3 * g + c];
                            x = df_add(x, dfl{y.x, y.y});
                        }
                        tsum[t] = (double)x.h + (double)x.l;
                    }
                }
            }
            __syncthreads();
            if (tid < cnt) {
                const Bin &B = bins[tid];
                const double tr = tsum[3 * tid], ti = tsum[3 * tid + 1], th = tsum[3 * tid + 2];
                const double s4 = 4.0 * K.df;
                double2 dh, hv;
                // undo the mixed form's power-of-two scalings and apply amp * 0.5T/N [* tdi2]
                const double cd = sizeof(R) == 8 ? s4 : s4 * exp2_int(B.eS - B.eD);
                const double ch = (sizeof(R) == 8 ? s4 : s4 * exp2_int(B.eS)) *
                                  (B.scale.x * B.scale.x + B.scale.y * B.scale.y);
                dh = scaled_sum(make_double2(cd * tr, cd * ti), B.scale);
                hv = make_double2(ch * th, 0.0);
                if (!B.valid) {
                    dh = make_double2(0.0, 0.0);
                    hv = make_double2(0.0, 0.0);
                }
                if (B.b >= 0) {
                    K.d_h[B.b] = dh;
                    K.h_h[B.b] = hv;
                }
            }
        }
        __syncthreads();
    }
}

// ----------------------------------------------------------------------------
// per-binary constants for every slot, computed once per launch by a fully
// occupied grid (one thread per binary) instead of by a few lanes of each tile
// ----------------------------------------------------------------------------
constexpr int kPrepBlock = 128;

template <int MODE>
__global__ void __launch_bounds__(kPrepBlock) prep_kernel(const KParams K)
{
    extern __shared__ __align__(16) unsigned char smem[];
    Bin *sb = reinterpret_cast<Bin *>(smem);
    const gbx_wave_args &a = K.a;
    const int s0 = blockIdx.x * kPrepBlock;
    const int slot = s0 + threadIdx.x;
    if (slot < a.num_bin) {
        int lg;
        if (a.tiles) {
            // tiles are sorted by first slot: binary search for the owning tile
            int lo = 0, hi = a.ntiles - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.tiles[4 * mid + 1] <= slot) lo = mid; else hi = mid - 1;
            }
            lg = a.tiles[4 * lo];
        } else {
            lg = 31 - __clz(a.N);
        }
        const int b = a.order ? a.order[slot] : slot;
        if (b < 0 || b >= a.num_bin || lg < 5 || lg > GBX_MAX_LOG2N) {
            flag(a.status, GBX_FLAG_TILE);
            memset(&sb[threadIdx.x], 0, sizeof(Bin));
            sb[threadIdx.x].b = -1;
        } else {
            setup_bin(sb[threadIdx.x], K, b, 1 << lg, MODE);
        }
    }
    __syncthreads();
    const int cnt = min(kPrepBlock, a.num_bin - s0);
    const int n16 = cnt * (int)(sizeof(Bin) / 16);
    const int4 *src = reinterpret_cast<const int4 *>(sb);
    int4 *dst = reinterpret_cast<int4 *>(static_cast<Bin *>(a.workspace) + s0);
    for (int k = threadIdx.x; k < n16; k += kPrepBlock) dst[k] = src[k];
}

constexpr int kPairMaxLog2N = 12;  // pair form: N <= 4096 (two 16-byte channels of 4096 fit)
#include "gbx_pair.cuh"
#include "gbx_grad.cuh"
#include "gbx_fisher.cuh"

// ----------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------
// nch transformed channels per binary (3 for the waveform outputs, 2 = A, E
// otherwise); the third-body pre-passes use three slots per sample of buf as
// FP64 scratch and keep psi and v_LOS after them
static size_t smem_bytes(int prec, bool third, int maxS, int nch, int maxP)
{
    size_t head = sizeof(Bin) * (size_t)maxP + sizeof(double) * (size_t)red_doubles(maxS) +
                  (prec == GBX_FP64 ? kScN * sizeof(double2) : 0);
    size_t rc = prec == GBX_FP64 ? sizeof(double2) : sizeof(float2);
    size_t r = prec == GBX_FP64 ? sizeof(double) : sizeof(float);
    size_t s = head + (third ? 3 : nch) * (size_t)maxS * rc;
    if (third) s += 3 * (size_t)maxS * (sizeof(double) + r);
    return s;
}

// the pair form's layout: constants, reduction scratch, sin/cos table, buffers
static size_t pair_smem_bytes(int maxS, int nch, int maxP)
{
    return sizeof(Bin) * (size_t)maxP + sizeof(double) * (size_t)red_doubles(maxS) +
           sizeof(float4) * (size_t)kScN + (size_t)nch * maxS * sizeof(cpx);
}

// per-binary constants into the workspace
template <int MODE>
static int launch_prep(const KParams &K, cudaStream_t st)
{
    const size_t psm = sizeof(Bin) * kPrepBlock;
    auto pk = prep_kernel<MODE>;
    int unused = 0;
    const int rc = kernel_fit((const void *)pk, kPrepBlock, psm, &unused);
    if (rc) return rc;
    pk<<<(K.a.num_bin + kPrepBlock - 1) / kPrepBlock, kPrepBlock, psm, st>>>(K);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? GBX_OK : cuda_error(e, "prep_kernel launch");
}

// persistent launch of one tile kernel (after the per-binary prep_kernel when
// the caller gave a workspace)
template <int MODE>
static int launch_tiles(void (*kern)(const KParams), size_t sm, const KParams &K, cudaStream_t st)
{
    int per_sm = 0;
    int rc = kernel_fit((const void *)kern, kBlock, sm, &per_sm);
    if (rc) return rc;
    cudaError_t e;
    if (K.a.blocks_per_sm > 0 && per_sm > K.a.blocks_per_sm) per_sm = K.a.blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    int nsm = num_sms();
    int ntiles = K.a.tiles ? K.a.ntiles : (K.a.num_bin + K.P - 1) / K.P;
    int grid = per_sm * nsm;
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) return GBX_OK;
    if (K.a.queue) {
        e = cudaMemsetAsync(K.a.queue, 0, sizeof(int), st);
        if (e != cudaSuccess) return cuda_error(e, "queue reset");
    }
    if (K.a.workspace) {
        rc = launch_prep<MODE>(K, st);
        if (rc) return rc;
    }
    kern<<<grid, kBlock, sm, st>>>(K);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "wave_kernel launch");
    return GBX_OK;
}

template <int MODE, int LC>
static size_t cluster_smem_bytes(int N)
{
    return sizeof(Bin) + sizeof(double2) * ((2 << LC) + kScN + (MODE == MODE_WAVE ? 6 : 4) * (size_t)(N >> LC));
}

// whether wave_cluster_kernel can be resident at all
template <int MODE, int LC>
static bool cluster_fits(const KParams &K)
{
    int n = 0;
    const void *kern = (const void *)wave_cluster_kernel<MODE, LC>;
    return kernel_fit(kern, kBlock, cluster_smem_bytes<MODE, LC>(K.a.N), &n, 1 << LC) == GBX_OK && n > 0;
}

template <int MODE, int LC>
static int launch_cluster(const KParams &K, cudaStream_t st)
{
    if (K.a.num_bin < 1) return GBX_OK;
    const int rc = launch_prep<MODE>(K, st);
    if (rc) return rc;
    cudaLaunchAttribute attr = {};
    cudaLaunchConfig_t cfg = cluster_config((unsigned)K.a.num_bin << LC, 1 << LC, kBlock,
                                            cluster_smem_bytes<MODE, LC>(K.a.N), &attr);
    cfg.stream = st;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, wave_cluster_kernel<MODE, LC>, K);
    return e == cudaSuccess ? GBX_OK : cuda_error(e, "wave_cluster_kernel launch");
}

template <typename R, int MODE, bool THIRD, bool UNEQ = false>
static int launch_one(const KParams &K, int maxS, cudaStream_t st)
{
    const size_t sm = smem_bytes(sizeof(R) == 8 ? GBX_FP64 : GBX_MIXED, THIRD, maxS,
                                 MODE == MODE_WAVE ? 3 : 2, K.maxP);
    return launch_tiles<MODE>(wave_kernel<R, MODE, THIRD, UNEQ>, sm, K, st);
}

// most binaries in one tile of this launch (the shared memory holds their constants)
static int max_pack(const gbx_wave_args *a, int minp)
{
    if (a->tiles == nullptr) return tile_pack(a->tile, 31 - __builtin_clz((unsigned)a->N), minp);
    int mp = 1;
    for (int k = 5; k <= GBX_MAX_LOG2N; k++)
        if (a->orbit[k]) mp = max(mp, tile_pack(a->tile, k, minp));
    return mp;
}

template <int MODE>
static int dispatch(KParams &K, int maxS, cudaStream_t st)
{
    K.maxS = maxS;
    K.maxP = max_pack(&K.a, MODE == MODE_SWAP ? 2 : 1);
    const bool third = K.a.nparams >= 14;
    // unequal arms are a separate instantiation: the equal-arm kernels carry none of it
    const bool uneq = (K.a.tdi2 & GBX_TDI_UNEQUAL) != 0;
    if (uneq && third) return set_error(GBX_ERR_UNSUPPORTED, "unequal arms cover the 9-parameter model");
    if (K.a.precision == GBX_PAIR) {
        if constexpr (MODE == MODE_WAVE || MODE == MODE_LL || MODE == MODE_FILL || MODE == MODE_SWAP) {
            if (third) return set_error(GBX_ERR_UNSUPPORTED, "the pair form covers the 9-parameter model");
            return launch_tiles<MODE>(uneq ? pair_kernel<MODE, true> : pair_kernel<MODE, false>,
                                      pair_smem_bytes(maxS, MODE == MODE_WAVE ? 3 : 2, K.maxP), K, st);
        } else {
            return set_error(GBX_ERR_UNSUPPORTED, "the pair form covers the waveform, likelihood, fill and swap entry points");
        }
    }
    if (K.a.precision == GBX_FP64) {
        if constexpr (MODE == MODE_WAVE || MODE == MODE_LL || MODE == MODE_FILL) {
            // Few binaries leave SMs idle under one block each: spread each over
            // a cluster.  Windows of N = 1024 (512, 4096), us, clusters of 8, of
            // 4, one block each: 1 binary 35 46 133 (32 32 72, 80 144 520); 30
            // binaries 49 48 138 (35 33 75, 155 146 524); 57 binaries 85 77 138
            // (57 47 76, 275 272 526); 76 binaries 116 106 137 (77 63 75, 340
            // 397 525).  N = 256 at 57 binaries: 52 32 44, at 76: 69 49 44.  Fills of
            // N = 1024, cluster and one block each: 1 binary 34 120, 57 69 122.  A
            // cluster needs a run of 32 samples per block: N >= 256.  The upper line is
            // where N = 256 crosses; longer windows would still gain at half as many
            // binaries as SMs.
            // Where no cluster can be resident (a partition of a GPU), one block each.
            if (!third && !uneq && K.a.tiles == nullptr && K.a.workspace && K.a.blocks_per_sm == 0) {
                const int lc = cluster_log2(K.a.num_bin, K.a.N, num_sms(), [&](int l) {
                    return l == 3 ? cluster_fits<MODE, 3>(K) : cluster_fits<MODE, 2>(K);
                });
                if (lc == 3) return launch_cluster<MODE, 3>(K, st);
                if (lc == 2) return launch_cluster<MODE, 2>(K, st);
            }
        }
        if (uneq) return launch_one<double, MODE, false, true>(K, maxS, st);
        return third ? launch_one<double, MODE, true>(K, maxS, st)
                     : launch_one<double, MODE, false>(K, maxS, st);
    }
    return third ? launch_one<float, MODE, true>(K, maxS, st)
                 : launch_one<float, MODE, false>(K, maxS, st);
}

// validates the shared arguments; returns max samples per tile in *maxS
static int check_wave(const gbx_wave_args *a, int *maxS)
{
    if (!a || !a->params) return set_error(GBX_ERR_ARG, "NULL wave args / params");
    if (a->num_bin < 0) return set_error(GBX_ERR_ARG, "num_bin < 0");
    if (a->nparams != 9 && a->nparams != 14) return set_error(GBX_ERR_ARG, "nparams must be 9 or 14");
    if (a->precision != GBX_FP64 && a->precision != GBX_MIXED && a->precision != GBX_PAIR)
        return set_error(GBX_ERR_ARG, "unknown precision %d", a->precision);
    if (!(a->T > 0.0) || !(a->armlength > 0.0)) return set_error(GBX_ERR_ARG, "T and armlength must be > 0");
    if (a->nparams == 14 && !(a->year > 0.0)) return set_error(GBX_ERR_ARG, "year must be > 0");
    if (a->tdi2 < 0 || a->tdi2 > (GBX_TDI2_BIT | GBX_TDI_UNEQUAL))
        return set_error(GBX_ERR_ARG, "tdi2=%d: bits GBX_TDI2_BIT and GBX_TDI_UNEQUAL only", a->tdi2);
    if ((a->tdi2 & GBX_TDI_UNEQUAL) && a->precision == GBX_MIXED)
        return set_error(GBX_ERR_UNSUPPORTED, "unequal arms are computed in the FP64 and pair forms only");
    if (a->workspace) {
        if (((uintptr_t)a->workspace & 15) != 0) return set_error(GBX_ERR_ARG, "workspace must be 16-byte aligned");
        if (a->workspace_bytes < gbx_wave_workspace_bytes(a->num_bin))
            return set_error(GBX_ERR_ARG, "workspace smaller than gbx_wave_workspace_bytes(num_bin)");
    }
    if (a->tile != 0 && (a->tile < 64 || a->tile > 4096 || (a->tile & (a->tile - 1)) != 0))
        return set_error(GBX_ERR_ARG, "tile=%d: need 0 or a power of two in [64, 4096]", a->tile);
    if (a->blocks_per_sm < 0) return set_error(GBX_ERR_ARG, "blocks_per_sm < 0");
    const int maxlg = a->precision == GBX_MIXED ? GBX_MAX_LOG2N : 12;
    if (a->tiles == nullptr) {
        int N = a->N;
        if (N < 32 || (N & (N - 1)) != 0) return set_error(GBX_ERR_UNSUPPORTED, "N=%d: need a power of two >= 32", N);
        int lg = 31 - __builtin_clz((unsigned)N);
        if (lg > maxlg) return set_error(GBX_ERR_UNSUPPORTED, "N=%d above the limit of this precision", N);
        if (!a->orbit[lg]) return set_error(GBX_ERR_ARG, "no orbit table for N=%d", N);
        *maxS = tile_pack(a->tile, lg, 1) * N;
    } else {
        if (a->ntiles < 0) return set_error(GBX_ERR_ARG, "ntiles < 0");
        // the N with a table bound the tile size
        int mx = 0;
        for (int k = 5; k <= maxlg; k++)
            if (a->orbit[k]) mx = max(mx, tile_pack(a->tile, k, 1) << k);
        if (mx == 0) return set_error(GBX_ERR_ARG, "no orbit tables");
        *maxS = mx;
    }
    return GBX_OK;
}

static KParams base_params(const gbx_wave_args *a)
{
    KParams K;
    memset(&K, 0, sizeof(K));
    K.a = *a;
    K.fstar = kCSI / (a->armlength * 2.0 * kPi);
    K.ifstar = 1.0 / K.fstar;
    for (int k = 0; k <= GBX_MAX_LOG2N; k++) K.stepd[k] = df_from(ldexp(a->T, -k));
    K.Locd = df_from(a->armlength / kCSI);
    K.Loc = a->armlength / kCSI;
    K.T2f = (float)(a->T * a->T);
    K.P = a->tiles == nullptr ? tile_pack(a->tile, 31 - __builtin_clz((unsigned)a->N), 1) : 1;
    return K;
}

}  // namespace gbx

using namespace gbx;

extern "C" size_t gbx_wave_workspace_bytes(int num_bin)
{
    if (num_bin <= 0) return 0;
    return ((size_t)num_bin * sizeof(Bin) + 255) & ~(size_t)255;
}

int gbx_twiddle_init(cudaStream_t st)
{
    tw_init_kernel<<<(kTwN / 2 + 255) / 256, 256, 0, st>>>();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "twiddle init");
    return GBX_OK;
}

extern "C" int gbx_waveform(const gbx_wave_args *a, void *XYZ_out, void *AET_out, int *start_out,
                            void *stream)
{
    int maxS = 0;
    int rc = check_wave(a, &maxS);
    if (rc) return rc;
    if (a->tiles) return set_error(GBX_ERR_ARG, "gbx_waveform takes a uniform N");
    rc = ensure_init((cudaStream_t)stream);
    if (rc) return rc;
    KParams K = base_params(a);
    K.XYZ = (double2 *)XYZ_out;
    K.AET = (double2 *)AET_out;
    K.start_out = start_out;
    return dispatch<MODE_WAVE>(K, maxS, (cudaStream_t)stream);
}

extern "C" int gbx_waveform_ll(const gbx_wave_args *a, const gbx_ll_args *l, void *d_h, void *h_h,
                               void *stream)
{
    int maxS = 0;
    int rc = check_wave(a, &maxS);
    if (rc) return rc;
    if (!l || !l->A_data || !l->E_data || !l->A_psd || !l->E_psd || !d_h || !h_h)
        return set_error(GBX_ERR_ARG, "NULL likelihood pointer");
    if (l->data_length <= 0 || l->num_data < 1 || l->num_psd < 1)
        return set_error(GBX_ERR_ARG, "data_length / num_data / num_psd must be positive");
    rc = ensure_init((cudaStream_t)stream);
    if (rc) return rc;
    KParams K = base_params(a);
    K.A_data = (const double2 *)l->A_data;
    K.E_data = (const double2 *)l->E_data;
    K.A_psd = l->A_psd;
    K.E_psd = l->E_psd;
    K.L = l->data_length;
    K.num_data = l->num_data;
    K.num_psd = l->num_psd;
    K.data_index = l->data_index;
    K.noise_index = l->noise_index;
    K.df = l->df;
    K.d_h = (double2 *)d_h;
    K.h_h = (double2 *)h_h;
    return dispatch<MODE_LL>(K, maxS, (cudaStream_t)stream);
}

extern "C" int gbx_waveform_fill(const gbx_wave_args *a, void *A_glob, void *E_glob,
                                 const int *group_index, int num_groups, int data_length,
                                 long long group_stride, void *stream)
{
    int maxS = 0;
    int rc = check_wave(a, &maxS);
    if (rc) return rc;
    if (!A_glob || !E_glob || !group_index) return set_error(GBX_ERR_ARG, "NULL fill pointer");
    if (data_length <= 0 || num_groups < 1) return set_error(GBX_ERR_ARG, "bad template shape");
    if (group_stride == 0) group_stride = data_length;
    if (group_stride < data_length) return set_error(GBX_ERR_ARG, "group_stride < data_length");
    rc = ensure_init((cudaStream_t)stream);
    if (rc) return rc;
    KParams K = base_params(a);
    K.A_glob = (double2 *)A_glob;
    K.E_glob = (double2 *)E_glob;
    K.group_index = group_index;
    K.num_groups = num_groups;
    K.gstride = group_stride;
    K.L = data_length;
    return dispatch<MODE_FILL>(K, maxS, (cudaStream_t)stream);
}

extern "C" int gbx_swap_ll(const gbx_wave_args *a, const gbx_ll_args *l, double *dlogl,
                           void *stream)
{
    int maxS = 0;
    int rc = check_wave(a, &maxS);
    if (rc) return rc;
    if (a->tiles || a->order) return set_error(GBX_ERR_ARG, "gbx_swap_ll takes a uniform N and no order");
    if (a->num_bin % 2) return set_error(GBX_ERR_ARG, "num_bin must be even: (old, new) pairs");
    if (!l || !l->A_data || !l->E_data || !l->A_psd || !l->E_psd || !dlogl)
        return set_error(GBX_ERR_ARG, "NULL likelihood pointer");
    if (l->data_length <= 0 || l->num_data < 1 || l->num_psd < 1)
        return set_error(GBX_ERR_ARG, "data_length / num_data / num_psd must be positive");
    rc = ensure_init((cudaStream_t)stream);
    if (rc) return rc;
    KParams K = base_params(a);
    K.P = tile_pack(a->tile, 31 - __builtin_clz((unsigned)a->N), 2);
    maxS = K.P * a->N;
    K.A_data = (const double2 *)l->A_data;
    K.E_data = (const double2 *)l->E_data;
    K.A_psd = l->A_psd;
    K.E_psd = l->E_psd;
    K.L = l->data_length;
    K.num_data = l->num_data;
    K.num_psd = l->num_psd;
    K.data_index = l->data_index;
    K.noise_index = l->noise_index;
    K.df = l->df;
    K.dlogl = dlogl;
    return dispatch<MODE_SWAP>(K, maxS, (cudaStream_t)stream);
}

extern "C" size_t gbx_grad_workspace_bytes(int num_bin)
{
    if (num_bin <= 0) return 0;
    return ((size_t)num_bin * (sizeof(Bin) + sizeof(GradExtra)) + 255) & ~(size_t)255;
}

// validates the gradient entry points' arguments (b: a copy of the caller's,
// workspace checked here, not by check_wave); *maxS as check_wave
static int check_grad(gbx_wave_args &b, const gbx_ll_args *l, int *maxS)
{
    const void *ws = b.workspace;
    const size_t wsb = b.workspace_bytes;
    b.workspace = nullptr;
    int rc = check_wave(&b, maxS);
    if (rc) return rc;
    if (b.precision != GBX_MIXED) return set_error(GBX_ERR_UNSUPPORTED, "gradients are computed in the mixed form only");
    if (b.nparams != 9 && b.nparams != 14)
        return set_error(GBX_ERR_UNSUPPORTED, "gradients cover the 9-parameter model and the 14-parameter third-body model");
    if (!ws || ((uintptr_t)ws & 15) != 0 || wsb < gbx_grad_workspace_bytes(b.num_bin))
        return set_error(GBX_ERR_ARG, "gradients need a 16-byte aligned workspace of gbx_grad_workspace_bytes(num_bin)");
    if (!l || !l->A_data || !l->E_data || !l->A_psd || !l->E_psd)
        return set_error(GBX_ERR_ARG, "NULL likelihood pointer");
    if (l->data_length <= 0 || l->num_data < 1 || l->num_psd < 1)
        return set_error(GBX_ERR_ARG, "data_length / num_data / num_psd must be positive");
    b.workspace = const_cast<void *>(ws);
    b.workspace_bytes = wsb;
    return GBX_OK;
}

static void set_ll(KParams &K, const gbx_ll_args *l)
{
    K.A_data = (const double2 *)l->A_data;
    K.E_data = (const double2 *)l->E_data;
    K.A_psd = l->A_psd;
    K.E_psd = l->E_psd;
    K.L = l->data_length;
    K.num_data = l->num_data;
    K.num_psd = l->num_psd;
    K.data_index = l->data_index;
    K.noise_index = l->noise_index;
    K.df = l->df;
}

// prep_grad_kernel + grad_kernel<third, SWAP> over the validated arguments
template <bool SWAP>
static int launch_grad(const gbx_wave_args &b, const gbx_ll_args *l, void *d_h, void *h_h,
                       double *grad, int maxS, cudaStream_t st)
{
    GradParams G;
    memset(&G, 0, sizeof(G));
    G.K = base_params(&b);
    KParams &K = G.K;
    set_ll(K, l);
    K.d_h = (double2 *)d_h;
    K.h_h = (double2 *)h_h;
    if (SWAP) {
        K.P = tile_pack(b.tile, 31 - __builtin_clz((unsigned)b.N), 2);
        maxS = K.P * b.N;
    }
    K.maxS = maxS;
    K.maxP = max_pack(&K.a, SWAP ? 2 : 1);
    G.grad = grad;
    const bool third = b.nparams == 14;
    auto kern = third ? grad_kernel<true, SWAP> : grad_kernel<false, SWAP>;
    const size_t sm = grad_smem_bytes(third, maxS, K.maxP);
    int per_sm = 0, unused = 0;
    int rc = kernel_fit((const void *)kern, kBlock, sm, &per_sm);
    if (rc) return rc;
    cudaError_t e;
    if (b.blocks_per_sm > 0 && per_sm > b.blocks_per_sm) per_sm = b.blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    const int ntiles = b.tiles ? b.ntiles : (b.num_bin + K.P - 1) / K.P;
    int grid = per_sm * num_sms();
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) return GBX_OK;
    if (b.queue) {
        e = cudaMemsetAsync(b.queue, 0, sizeof(int), st);
        if (e != cudaSuccess) return cuda_error(e, "queue reset");
    }
    const size_t psm = (sizeof(Bin) + sizeof(GradExtra)) * kPrepBlock;
    rc = kernel_fit((const void *)prep_grad_kernel, kPrepBlock, psm, &unused);
    if (rc) return rc;
    prep_grad_kernel<<<(b.num_bin + kPrepBlock - 1) / kPrepBlock, kPrepBlock, psm, st>>>(K);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "prep_grad_kernel launch");
    kern<<<grid, kBlock, sm, st>>>(G);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "grad_kernel launch");
    return GBX_OK;
}

extern "C" int gbx_waveform_ll_grad(const gbx_wave_args *a, const gbx_ll_args *l, void *d_h,
                                    void *h_h, double *grad, void *stream)
{
    if (!a) return set_error(GBX_ERR_ARG, "NULL wave args");
    int maxS = 0;
    gbx_wave_args b = *a;
    int rc = check_grad(b, l, &maxS);
    if (rc) return rc;
    if (!d_h || !h_h || !grad) return set_error(GBX_ERR_ARG, "NULL likelihood / gradient pointer");
    if (b.num_bin == 0) return GBX_OK;
    cudaStream_t st = (cudaStream_t)stream;
    rc = ensure_init(st);
    if (rc) return rc;
    return launch_grad<false>(b, l, d_h, h_h, grad, maxS, st);
}

extern "C" int gbx_swap_ll_grad(const gbx_wave_args *a, const gbx_ll_args *l, double *dlogl,
                                double *grad, void *stream)
{
    if (!a) return set_error(GBX_ERR_ARG, "NULL wave args");
    int maxS = 0;
    gbx_wave_args b = *a;
    int rc = check_grad(b, l, &maxS);
    if (rc) return rc;
    if (b.tiles || b.order) return set_error(GBX_ERR_ARG, "gbx_swap_ll_grad takes a uniform N and no order");
    if (b.num_bin % 2) return set_error(GBX_ERR_ARG, "num_bin must be even: (old, new) pairs");
    if (!grad) return set_error(GBX_ERR_ARG, "NULL gradient pointer");
    if (b.num_bin == 0) return GBX_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (dlogl) {
        // the change of log-likelihood itself: the swap kernel, as gbx_swap_ll
        rc = gbx_swap_ll(&b, l, dlogl, stream);
        if (rc) return rc;
    } else {
        rc = ensure_init(st);
        if (rc) return rc;
    }
    return launch_grad<true>(b, l, nullptr, nullptr, grad, maxS, st);
}

extern "C" int gbx_fisher(const gbx_wave_args *a, const double *A_psd, const double *E_psd,
                          int psd_length, int num_psd, const int *noise_index, double df,
                          double *fisher, void *stream)
{
    if (!a) return set_error(GBX_ERR_ARG, "NULL wave args");
    int maxS = 0;
    gbx_wave_args b = *a;
    gbx_ll_args l;
    memset(&l, 0, sizeof(l));
    // the likelihood arguments' checks, with the PSD rows standing in for the
    // data (never read)
    l.A_data = A_psd;
    l.E_data = E_psd;
    l.A_psd = A_psd;
    l.E_psd = E_psd;
    l.data_length = psd_length;
    l.num_data = 1;
    l.num_psd = num_psd;
    l.noise_index = noise_index;
    l.df = df;
    int rc = check_grad(b, &l, &maxS);
    if (rc) return rc;
    if (b.nparams != 9) return set_error(GBX_ERR_UNSUPPORTED, "Fisher matrices cover the 9-parameter model");
    if (b.tdi2 & GBX_TDI_UNEQUAL) return set_error(GBX_ERR_UNSUPPORTED, "Fisher matrices take equal arms");
    if (!fisher) return set_error(GBX_ERR_ARG, "NULL Fisher output");
    if (b.num_bin == 0) return GBX_OK;
    cudaStream_t st = (cudaStream_t)stream;
    rc = ensure_init(st);
    if (rc) return rc;
    FisherParams F;
    memset(&F, 0, sizeof(F));
    F.K = base_params(&b);
    KParams &K = F.K;
    set_ll(K, &l);
    K.A_data = nullptr;
    K.E_data = nullptr;
    K.data_index = nullptr;
    K.maxS = maxS;
    K.maxP = max_pack(&K.a, 1);
    F.fisher = fisher;
    const size_t sm = fisher_smem_bytes(maxS, K.maxP);
    if (sm > 227 * 1024) return set_error(GBX_ERR_UNSUPPORTED, "tile needs %zu B of shared memory (use a smaller tile)", sm);
    int per_sm = 0, unused = 0;
    rc = kernel_fit((const void *)fisher_kernel, kBlock, sm, &per_sm);
    if (rc) return rc;
    cudaError_t e;
    if (b.blocks_per_sm > 0 && per_sm > b.blocks_per_sm) per_sm = b.blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    const int ntiles = b.tiles ? b.ntiles : (b.num_bin + K.P - 1) / K.P;
    int grid = per_sm * num_sms();
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) return GBX_OK;
    if (b.queue) {
        e = cudaMemsetAsync(b.queue, 0, sizeof(int), st);
        if (e != cudaSuccess) return cuda_error(e, "queue reset");
    }
    const size_t psm = (sizeof(Bin) + sizeof(GradExtra)) * kPrepBlock;
    rc = kernel_fit((const void *)prep_grad_kernel, kPrepBlock, psm, &unused);
    if (rc) return rc;
    prep_grad_kernel<<<(b.num_bin + kPrepBlock - 1) / kPrepBlock, kPrepBlock, psm, st>>>(K);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "prep_grad_kernel launch");
    fisher_kernel<<<grid, kBlock, sm, st>>>(F);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "fisher_kernel launch");
    return GBX_OK;
}

// The end of a likelihood call on the device: logL from its terms and the
// status word as one more number, so that the caller reads everything back in
// one copy (instead of five elementwise launches and two copies).
namespace gbx {
__global__ void ll_finish_kernel(const double2 *d_h, const double2 *h_h, double d_d, int n,
                                 const int *status, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    // the reference's order, -1/2 (d_d + h_h - 2 d_h) (gbgpu.py:728)
    if (i < n) out[i] = -0.5 * __dsub_rn(__dadd_rn(d_d, h_h[i].x), 2.0 * d_h[i].x);
    else if (i == n) out[n] = status ? (double)*status : 0.0;
}
}  // namespace gbx

extern "C" int gbx_log_likelihood(const gbx_wave_args *a, const gbx_ll_args *l, void *d_h, void *h_h,
                                  double d_d, double *out, void *stream)
{
    if (!a || !out) return set_error(GBX_ERR_ARG, "NULL wave args / output");
    cudaStream_t st = (cudaStream_t)stream;
    if (a->status) {
        const cudaError_t e = cudaMemsetAsync(a->status, 0, sizeof(int), st);
        if (e != cudaSuccess) return cuda_error(e, "status reset");
    }
    const int rc = gbx_waveform_ll(a, l, d_h, h_h, stream);
    if (rc) return rc;
    const int n = a->num_bin;
    gbx::ll_finish_kernel<<<n / 256 + 1, 256, 0, st>>>((const double2 *)d_h, (const double2 *)h_h, d_d, n,
                                                       a->status, out);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? GBX_OK : cuda_error(e, "ll_finish_kernel launch");
}

// ----------------------------------------------------------------------------
// Diagnostic entry point for the FP32 math helpers
// ----------------------------------------------------------------------------
namespace gbx {
__global__ void math_selftest_kernel(const void *x, float *out, int n, int which, int e)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (which == 2) {
        out[i] = d2f_scaled(static_cast<const double *>(x)[i], e);
        return;
    }
    if (which == 3) {
        // (written as doubles)
        reinterpret_cast<double *>(out)[i] = sinc_fp64(static_cast<const double *>(x)[i], g_sc_d);
        return;
    }
    if (which == 4) {
        out[i] = d2f_rn(static_cast<const double *>(x)[i]);
        return;
    }
    const float xi = static_cast<const float *>(x)[i];
    float a, b;
    if (which == 0) sincos_mod(xi, a, b);
    else sinc_cos_f(xi, a, b);
    out[2 * i] = a;
    out[2 * i + 1] = b;
}
}  // namespace gbx

extern "C" int gbx_math_selftest(const void *x, float *out, int n, int which, int e, void *stream)
{
    if (n < 0 || (n > 0 && (!x || !out)) || which < 0 || which > 4)
        return set_error(GBX_ERR_ARG, "math selftest: bad arguments");
    if (n == 0) return GBX_OK;
    const int rc = ensure_init((cudaStream_t)stream);
    if (rc) return rc;
    gbx::math_selftest_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(x, out, n, which, e);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? GBX_OK : cuda_error(err, "math_selftest_kernel launch");
}

// ----------------------------------------------------------------------------
// Allocation-free variant of gbx_waveform_ll.
//
// Some callers cannot allocate device memory at all: a plug-in inside a host
// application that owns every device allocation and only lends it pointers,
// or an FFI caller that binds this C ABI but has no CUDA allocator of its own.
// They cannot provide the per-binary workspace or the work-queue counter, so
// this entry point keeps both in the file-scope array below.  Every GPU that
// loads the library holds the array (4 MiB + 256 B) until the process exits.
// ----------------------------------------------------------------------------
namespace gbx {
constexpr int kNoAllocMaxBin = GBX_NOALLOC_MAX_BINS;
// 512 bytes per binary: the published size (4 MiB + 256 B) stays fixed while Bin fits
static_assert(sizeof(Bin) <= 512, "the allocation-free scratch holds 512 bytes per binary");
constexpr size_t kNoAllocWsBytes = (size_t)kNoAllocMaxBin * 512;
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocWsBytes + 256];

static std::mutex g_noalloc_lock;
static void *g_noalloc_ptr[64] = {};

// The host-side name g_noalloc_scratch is only a stand-in for the device
// array; its device address comes from cudaGetSymbolAddress, once per device,
// with that device current.
static int noalloc_scratch(void **out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    if (dev < 0 || dev >= 64) return set_error(GBX_ERR_ARG, "device %d out of range", dev);
    std::lock_guard<std::mutex> g(g_noalloc_lock);
    if (g_noalloc_ptr[dev] == nullptr) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(scratch)");
        g_noalloc_ptr[dev] = ptr;
    }
    *out = g_noalloc_ptr[dev];
    return GBX_OK;
}
}  // namespace gbx

extern "C" int gbx_waveform_ll_noalloc(const gbx_wave_args *a, const gbx_ll_args *l, void *d_h,
                                       void *h_h, void *stream)
{
    if (!a) return set_error(GBX_ERR_ARG, "NULL wave args");
    if (a->num_bin > kNoAllocMaxBin)
        return set_error(GBX_ERR_ARG, "num_bin %d exceeds the %d binaries of the static scratch",
                         a->num_bin, kNoAllocMaxBin);
    void *scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    gbx_wave_args b = *a;
    b.workspace = scratch;
    b.workspace_bytes = kNoAllocWsBytes;
    // the queue counter lives after the workspace; it is reset on the stream
    // before every launch that uses it
    b.queue = b.tiles ? reinterpret_cast<int *>(static_cast<unsigned char *>(scratch) + kNoAllocWsBytes)
                      : nullptr;
    return gbx_waveform_ll(&b, l, d_h, h_h, stream);
}
