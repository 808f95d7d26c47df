// Per-cell arithmetic of the MHD step in two policies.
//
//   EX = true  ("exact"): the reference's own evaluation order and types.
//       The reference is C on float data, so each double literal (2.0, 4.0,
//       0.9 ...) promotes its sub-expression to double; those promotions are
//       kept (type W = double) and every abXYc "a*X + b*Y + c" keeps its
//       +0 and 0*Y terms.  The translation unit that instantiates EX = true is
//       compiled with --fmad=false, so results equal the reference built with
//       -ffp-contract=off bit for bit.
//   EX = false ("fast"): the same algorithm in the working precision R with
//       FMA contraction and one reciprocal per division by rho or c.
//
// Every function names the reference lines it restates.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>

namespace mhd {

template <typename R, bool EX>
using wide_t = typename std::conditional<EX, double, R>::type;

template <typename R>
__device__ __forceinline__ R rabs(R x)
{
    return fabs(x);
}
template <>
__device__ __forceinline__ float rabs<float>(float x)
{
    return fabsf(x);
}

// FAST-policy division, reciprocal and square root: CUDA's approximate forms (a few ulp)
// in FP32, subnormal operands included (a thin or cold gas has them), IEEE in FP64.
template <typename R>
__device__ __forceinline__ R fast_rcp(R x)
{
    return R(1) / x;
}
template <>
__device__ __forceinline__ float fast_rcp<float>(float x)
{
    return __fdividef(1.0f, x);
}
template <typename R>
__device__ __forceinline__ R fast_div(R x, R y)
{
    return x / y;
}
template <>
__device__ __forceinline__ float fast_div<float>(float x, float y)
{
    return __fdividef(x, y);
}
template <typename R>
__device__ __forceinline__ R fast_sqrt(R x)
{
    return sqrt(x);
}
template <>
__device__ __forceinline__ float fast_sqrt<float>(float x)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The approximations that flush subnormal operands and results to zero, which are
// cheaper, where neither can matter: the limiter's quotient is used only where the
// product of its two differences is positive, so their sum is at least 2^-75 (and above
// 2^126 both forms give 0); the EXACT forms below start from them inside range conditions.
// With the flushing quotient in the limiter, mul_if_pos and the kept field
// (mhd_fluidx2.cuh) four 256^3 steps take 10.12 ms plain and 8.79 ms fused, against 10.94 and
// 9.27 ms before, bit for bit; 9.93 and 8.62 ms with flushing forms for 1 / rho and the sound speed
// too, which lose densities below 2^-126 and sound speeds below 2^-63.
__device__ __forceinline__ float rcp_ftz(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_ftz(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x r where p > 0, else 0; and t - x where p > 0, else t: predicated, with no
// select.  (The two limited differences of a flux are rounded one by one, as
// they always were: a fused multiply-add is faster by 3% of a step, but the
// closure net amplifies a last-bit change of the state by 1e5.)
__device__ __forceinline__ float mul_if_pos(float p, float x, float r)
{
    float d = 0.f;
    asm("{\n\t.reg .pred q;\n\tsetp.gt.f32 q, %1, 0f00000000;\n\t@q mul.rn.f32 %0, %2, %3;\n\t}"
        : "+f"(d)
        : "f"(p), "f"(x), "f"(r));
    return d;
}
__device__ __forceinline__ float sub_if_pos(float p, float t, float x)
{
    asm("{\n\t.reg .pred q;\n\tsetp.gt.f32 q, %1, 0f00000000;\n\t@q sub.rn.f32 %0, %0, %2;\n\t}"
        : "+f"(t)
        : "f"(p), "f"(x));
    return t;
}

// ------------------------------------------- EXACT in FP32 without FP64
//
// The reference is C on float data whose double literals promote a few
// sub-expressions to double before they are rounded back to float.  This GPU
// runs FP64 at 1/60 of its FP32 rate (measured: 0.017 against 1.05 warp
// instructions per clock and scheduler), so those promotions were nearly all
// of the EXACT kernels' time.  Each is evaluated as an unevaluated sum of two
// floats instead (error-free sums and products: Dekker 1971, Knuth TAOCP 4.2.2)
// whose distance from the double expression is bounded, and rounded with
// Ziv's test (ACM TOMS 17, 1991): if both ends of the interval round to the
// same float, the double expression does too.  Where they do not (about one
// value in 2^16), or where a range condition of the bound fails (tiny or huge
// operands, infinities, NaN), the double expression itself is evaluated.
//
// Two EXACT 96^3 steps: 6.07 ms with the double sub-expressions (fluidx 340,
// advectbyzx 148 us per launch), 1.15 ms with these; same bits.

// sum + lo with |error| <= err around hi + lo: true if the rounding is certain
__device__ __forceinline__ bool ziv_round(float hi, float lo, float err, float& r)
{
    r = __fadd_rn(hi, __fsub_rn(lo, err));
    return r == __fadd_rn(hi, __fadd_rn(lo, err));
}

// s + e = a + b exactly (Knuth)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s = __fadd_rn(a, b);
    const float t = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
}

// float(2ab / (a + b)) with the product and the quotient in double, for a b > 0
static __device__ __noinline__ float vanleer_wide(float a, float b) { return float(2.0 * double(a) * double(b) / double(a + b)); }

__device__ __forceinline__ float vanleer_exact(float a, float b)
{
    float r = 0.f;
    if (__fmul_rn(a, b) > 0.f) {
        const float a2 = __fadd_rn(a, a), s = __fadd_rn(a, b);
        const float ph = __fmul_rn(a2, b), pl = __fmaf_rn(a2, b, -ph);  // 2ab = ph + pl
        const float y = rcp_ftz(s), q = __fmul_rn(ph, y);               // q within 2^-21.6 of the quotient
        const float e = __fmul_rn(__fadd_rn(__fmaf_rn(-q, s, ph), pl), y);
        // |q + e - quotient| <= 2^-42.6 |q| (the residual's, the product's and y's errors
        // on a correction of at most 2^-21.4 |q|), 2^-45 for lo -+ err, 2^-53 for the double
        const bool sure = ziv_round(q, e, fabsf(q) * 0x1p-41f, r);
        // the product's and the residual's low parts are exact above 2^-100
        if (!(sure && ph > 0x1p-100f && fabsf(q) > 0x1p-80f && fabsf(s) < 0x1p100f))
            r = vanleer_wide(a, b);
    }
    return r;
}

constexpr float kGammaF = float(5.0 / 3.0);
constexpr float kGm1F = float(double(kGammaF) - 1.0), kHalf2mgF = float((2.0 - double(kGammaF)) / 2.0);
static_assert(double(kGm1F) == double(kGammaF) - 1.0 && double(kHalf2mgF) == (2.0 - double(kGammaF)) / 2.0,
              "gamma - 1 and (2 - gamma) / 2 are floats");

// float((e - h/2)(gamma - 1) + (2 - gamma) bb / 2) in double
static __device__ __noinline__ float total_pressure_wide(float e, float h, float bb)
{
    return float((double(e) - double(h) / 2.0) * (double(kGammaF) - 1.0) + (2.0 - double(kGammaF)) * double(bb) / 2.0);
}

__device__ __forceinline__ float total_pressure_exact(float e, float h, float bb)
{
    float t, te, s, se, r;
    two_sum(e, __fmul_rn(-0.5f, h), t, te);
    const float p = __fmul_rn(t, kGm1F), pe = __fmaf_rn(te, kGm1F, __fmaf_rn(t, kGm1F, -p));
    const float c = __fmul_rn(kHalf2mgF, bb), ce = __fmaf_rn(kHalf2mgF, bb, -c);
    two_sum(p, c, s, se);
    // three roundings of terms of at most 2^-23 (|p| + |c|): within 2^-45.4 of it
    const float m = __fadd_rn(fabsf(p), fabsf(c));
    const bool sure = ziv_round(s, __fadd_rn(se, __fadd_rn(pe, ce)), m * 0x1p-44f, r);
    if (!(sure && m > 0x1p-90f && m < 0x1p100f))
        r = total_pressure_wide(e, h, bb);
    return r;
}

// float(a + sqrt(t)) in double, for a >= 0 and t >= 0
static __device__ __noinline__ float add_sqrt_wide(float a, float t) { return float(double(a) + sqrt(double(t))); }

__device__ __forceinline__ float add_sqrt_exact(float a, float t)
{
    float s, se, r;
    const float s0 = sqrt_ftz(t);  // within 2^-22: with the correction's own error 2^-42.5 of s0
    const float corr = __fmul_rn(__fmaf_rn(-s0, s0, t), __fmul_rn(0.5f, rcp_ftz(s0)));
    two_sum(a, s0, s, se);
    const bool sure = ziv_round(s, __fadd_rn(se, corr), s * 0x1p-41f, r);
    if (!(sure && s0 > 0x1p-40f && s < 0x1p60f))
        r = add_sqrt_wide(a, t);
    return r;
}

// float(v + sqrt(|2 bb + g| / rho)) in double, for v >= 0
static __device__ __noinline__ float cfl_wide(float v, float bb, float g, float rho)
{
    return float(double(v) + sqrt(fabs(double(bb) * 2.0 + double(g)) / double(rho)));
}

__device__ __forceinline__ float cfl_exact(float v, float bb, float g, float rho)
{
    float nh, nl, s, se, r;
    two_sum(__fadd_rn(bb, bb), g, nh, nl);
    if (nh < 0.f) {
        nh = -nh;
        nl = -nl;
    }
    const float y = rcp_ftz(rho), q = __fmul_rn(nh, y);
    const float e = __fmul_rn(__fadd_rn(__fmaf_rn(-q, rho, nh), nl), y);
    const float s0 = sqrt_ftz(q);
    const float corr = __fmul_rn(__fadd_rn(__fmaf_rn(-s0, s0, q), e), __fmul_rn(0.5f, rcp_ftz(s0)));
    two_sum(v, s0, s, se);
    // the quotient within 2^-42.6, the root within half of that and 2^-44 (corr up to 2^-21)
    const bool sure = ziv_round(s, __fadd_rn(se, corr), s * 0x1p-40f, r);
    if (!(sure && q > 0x1p-60f && q < 0x1p60f && rho > 0x1p-40f && rho < 0x1p40f && s < 0x1p60f))
        r = cfl_wide(v, bb, g, rho);
    return r;
}

// ------------------------------------------------ FP64 with fewer FP64 operations
//
// An FP64 warp instruction holds its scheduler's FP64 pipe for 60 cycles, so the
// FP64 kernels' time is their count.  The forms below give the reference's values
// with fewer: additions of +0 and products by 1 that only set the sign of a
// zero are left to the step's last sum, powers of two are moved to where they cost
// nothing, a product that is exact is fused with the sum after it, and signs, zeros,
// NaN and maxima of non-negative values are taken from the bits.
//
// They hold while the values they are applied to are zero or of 2^-480 .. 2^480
// (Range64; integer work beside the busy FP64 pipe): halves are exact, products of two
// neither overflow nor underflow, and differences are multiples of 2^-532.  A CTA that
// meets another value (tiny, huge, infinite, NaN) takes the reference's own expressions.
// Two FP64 steps of 64^3: 5.17 ms with the reference's expressions alone, 3.73 ms.

// Whether every value seen was zero or of 2^-480 .. 2^480.
struct Range64 {
    static constexpr unsigned kMin = (1023u - 480u) << 20, kMax = (1023u + 480u) << 20;  // high words
    unsigned lo = 0xffffffffu, hi = 0;

    __device__ __forceinline__ void see(double x)
    {
        const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
        hi = max(hi, h);
        lo = min(lo, (h | (__double2loint(x) != 0 ? 1u : 0u)) - 1u);  // zero: the largest unsigned
    }
    __device__ __forceinline__ bool ok() const { return lo >= kMin - 1u && hi < kMax; }
};

// x > 0 (false for NaN)
__device__ __forceinline__ bool positive64(double x)
{
    const long long b = __double_as_longlong(x);
    return b > 0 && b <= 0x7ff0000000000000LL;
}

// vanleer of a / 2 and b / 2
__device__ __forceinline__ double vanleer64(double a, double b)
{
    const double p = __dmul_rn(a, b);
    double r = 0.0;
    if (positive64(p))
        r = p / __dadd_rn(a, b);
    return r;
}

// cell_flux (below) in FP64 (R = double)
template <typename R>
__device__ __forceinline__ void cell_flux64(const R q[5], const R f[3], R v[5], R& ci)
{
    constexpr double gamma = 5.0 / 3.0, k2 = (2.0 - gamma) / 2.0;
    static_assert(k2 * 2.0 == 2.0 - gamma, "the half is exact");
    const double vx = q[1] / q[0];
    const double mm = __dadd_rn(__dadd_rn(__dmul_rn(q[1], q[1]), __dmul_rn(q[2], q[2])), __dmul_rn(q[3], q[3]));
    const double f00 = __dmul_rn(f[0], f[0]);
    const double bb = __dadd_rn(__dadd_rn(f00, __dmul_rn(f[1], f[1])), __dmul_rn(f[2], f[2]));
    // 2 - gamma and gamma - 1 times their operands, the half before the product
    const double ps = __dadd_rn(__dmul_rn(__fma_rn(-0.5, mm / q[0], q[4]), gamma - 1.0), __dmul_rn(k2, bb));
    v[0] = q[1];
    v[1] = __dsub_rn(__dadd_rn(__dmul_rn(q[1], vx), ps), f00);
    v[2] = __dsub_rn(__dmul_rn(q[2], vx), __dmul_rn(f[1], f[0]));
    v[3] = __dsub_rn(__dmul_rn(q[3], vx), __dmul_rn(f[2], f[0]));
    const double dot = __dadd_rn(__dadd_rn(__dmul_rn(f[0], q[1]), __dmul_rn(f[1], q[2])), __dmul_rn(f[2], q[3]));
    v[4] = __dsub_rn(__dmul_rn(__dadd_rn(q[4], ps), vx), __dmul_rn(f[0], dot) / q[0]);
    const double p = __fma_rn(-0.5, bb, ps);
    ci = __dadd_rn(fabs(vx), sqrt(fabs(__dadd_rn(bb, __dmul_rn(gamma, p)) / q[0])));
}

// abXYc_matrix2D with c = 0 (C/includefunc_spu.h:73-84): a*X + b*Y + 0.
template <typename R, bool EX>
__device__ __forceinline__ R lin(R a, R x, R b, R y)
{
    if constexpr (EX)
        return (a * x + b * y) + R(0);
    else
        return a * x + b * y;
}

// c*X + 0*X + 0 (the "fr = c*wr" form of C/tvd1.c:40,43,58,84).
template <typename R, bool EX>
__device__ __forceinline__ R scale0(R c, R x)
{
    if constexpr (EX)
        return (c * x + R(0) * x) + R(0);
    else
        return c * x;
}

// Limiter of C/tvd1.c:71-81,97-107 and C/tvdb.c:72-76:
// 0 unless a*b > 0, else 2ab/(a+b) (in double in the reference).
template <typename R, bool EX>
__device__ __forceinline__ R vanleer(R a, R b)
{
    using W = wide_t<R, EX>;
    if constexpr (EX && sizeof(R) == 4) {
        return vanleer_exact(a, b);
    } else if constexpr (EX) {
        R r = R(0);
        if (a * b > R(0))
            r = R(W(2.0) * W(a) * W(b) / W(a + b));
        return r;
    } else {  // branch-free: quotient for every cell, then the select
        const R ab = a * b;
        const R q = R(2) * ab * rcp_ftz(a + b);
        return (ab > R(0)) ? q : R(0);
    }
}

// mhdflux for one cell (C/mhdflux.c:21-46): flux v (before division by the
// pencil max c) and the cell's fast speed ci.  q = u record, f = cell-centred B.
template <typename R, bool EX>
__device__ __forceinline__ void cell_flux(const R q[5], const R f[3], R v[5], R& ci)
{
    using W = wide_t<R, EX>;
    const R gamma = R(5.0 / 3.0);
    if constexpr (EX) {
        R vx = q[1] / q[0];
        R mm = q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
        R bb = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
        R ps;
        if constexpr (sizeof(R) == 4)
            ps = total_pressure_exact(q[4], mm / q[0], bb);
        else
            ps = R((W(q[4]) - W(mm / q[0]) / W(2.0)) * (W(gamma) - W(1.0)) +
                   (W(2.0) - W(gamma)) * W(bb) / W(2.0));
        v[0] = q[1];
        v[1] = q[1] * vx + ps - f[0] * f[0];
        v[2] = q[2] * vx - f[1] * f[0];
        v[3] = q[3] * vx - f[2] * f[0];
        v[4] = (q[4] + ps) * vx - f[0] * (f[0] * q[1] + f[1] * q[2] + f[2] * q[3]) / q[0];
        if constexpr (sizeof(R) == 4) {
            // a difference of two floats rounds alike with and without the double between
            // (53 >= 2 * 24 + 2), so one fused step gives it
            const R p = __fmaf_rn(-0.5f, bb, ps);
            ci = add_sqrt_exact(fabsf(vx), fabsf((bb + gamma * p) / q[0]));
        } else {
            R p = R(W(ps) - W(bb) / W(2.0));
            ci = R(fabs(W(vx)) + sqrt(fabs(W((bb + gamma * p) / q[0]))));
        }
    } else {
        const R ri = fast_rcp(q[0]);
        const R vx = q[1] * ri;
        const R mm = q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
        const R bb = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
        const R ps = (q[4] - R(0.5) * mm * ri) * (gamma - R(1)) + R(0.5) * (R(2) - gamma) * bb;
        v[0] = q[1];
        v[1] = q[1] * vx + ps - f[0] * f[0];
        v[2] = q[2] * vx - f[1] * f[0];
        v[3] = q[3] * vx - f[2] * f[0];
        v[4] = (q[4] + ps) * vx - f[0] * (f[0] * q[1] + f[1] * q[2] + f[2] * q[3]) * ri;
        const R p = ps - R(0.5) * bb;
        ci = rabs(vx) + fast_sqrt(rabs((bb + gamma * p) * ri));
    }
}

// cell_flux in FAST for the two kernels that share pencil lengths (k_fluidx and k_fluidx_rag, by
// the size of the box): which products go into a multiply-add is written out where it was found to
// depend on the code around the call, so both give the same bits.  (Found by comparing the
// outputs of the 64 ways to write them with those of the kernel that took these lengths first;
// a run that feeds the state to the closure net needs it: the net amplifies a last-bit change by 1e5.)
__device__ __forceinline__ void cell_flux_pinned(const float q[5], const float f[3], float v[5], float& ci)
{
    constexpr float kG1 = kGammaF - 1.0f, kK = 0.5f * (2.0f - kGammaF);
    const float ri = fast_rcp(q[0]);
    const float vx = q[1] * ri;
    const float mm = q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
    const float p0 = __fmul_rn(f[0], f[0]);
    const float bb = __fmaf_rn(f[2], f[2], __fmaf_rn(f[1], f[1], p0));
    const float ps = __fmaf_rn(kK, bb, __fmul_rn(q[4] - 0.5f * mm * ri, kG1));
    v[0] = q[1];
    v[1] = __fsub_rn(__fmaf_rn(q[1], vx, ps), p0);
    v[2] = q[2] * vx - f[1] * f[0];
    v[3] = q[3] * vx - f[2] * f[0];
    const float dot = __fmaf_rn(f[2], q[3], __fmaf_rn(f[0], q[1], __fmul_rn(f[1], q[2])));
    v[4] = __fmaf_rn(__fadd_rn(q[4], ps), vx, -__fmul_rn(__fmul_rn(f[0], dot), ri));
    const float p = ps - 0.5f * bb;
    ci = fabsf(vx) + fast_sqrt(fabsf((bb + kGammaF * p) * ri));
}

// Divide the flux by the pencil max when it is positive (C/mhdflux.c:48-57).
template <typename R, bool EX>
__device__ __forceinline__ void scale_flux(R v[5], R c)
{
    if (c > R(0)) {
        if constexpr (EX) {
#pragma unroll
            for (int q = 0; q < 5; q++)
                v[q] = v[q] / c;
        } else {
            const R rc = fast_rcp(c);
#pragma unroll
            for (int q = 0; q < 5; q++)
                v[q] = v[q] * rc;
        }
    }
}

// max_3num (C/calcfl.c:65-89), strict '>' comparisons.
template <typename R>
__device__ __forceinline__ R max3(R a, R b, R c)
{
    if (a > b)
        return (a > c) ? a : c;
    return (b > c) ? b : c;
}

// Per-cell speed of calcfl (C/calcfl.c:44-54), from the face values f = b(:,i,j,k).
template <typename R, bool EX>
__device__ __forceinline__ R cfl_speed(const R q[5], const R f[3])
{
    using W = wide_t<R, EX>;
    const R gamma = R(5.0 / 3.0);
    if constexpr (EX) {
        R t1 = rabs(q[1] / q[0]);
        R t2 = rabs(q[2] / q[0]);
        R t3 = rabs(q[3] / q[0]);
        R v = max3(t1, t2, t3);
        R mm = q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
        R bb = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
        if constexpr (sizeof(R) == 4) {
            const R ps = total_pressure_exact(q[4], mm / q[0], bb);
            return cfl_exact(v, bb, gamma * __fmaf_rn(-0.5f, bb, ps), q[0]);
        }
        R ps = R((W(q[4]) - W(mm / q[0]) / W(2.0)) * (W(gamma) - W(1.0)) +
                 (W(2.0) - W(gamma)) * W(bb) / W(2.0));
        R p = R(W(ps) - W(bb) / W(2.0));
        return R(W(v) + sqrt(fabs(W(bb) * W(2.0) + W(gamma * p)) / W(q[0])));
    } else {
        const R ri = fast_rcp(q[0]);
        const R v = max3(rabs(q[1] * ri), rabs(q[2] * ri), rabs(q[3] * ri));
        const R mm = q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
        const R bb = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
        const R ps = (q[4] - R(0.5) * mm * ri) * (gamma - R(1)) + R(0.5) * (R(2) - gamma) * bb;
        const R p = ps - R(0.5) * bb;
        return v + fast_sqrt(rabs(bb * R(2) + gamma * p) * ri);
    }
}

// Per-cell steps of tvdb.  EXACT: the reference's values (compiled without contraction).
// FAST: every rounding is explicit (__fadd_rn, __fmul_rn and __fmaf_rn are never
// contracted), so k_advect2 to k_advect6 compute the same bits whatever the compiler
// does around the calls.  k_advect and k_advect_rag, which share the other lengths and the
// unaligned arrays, agree with each other: they divide for the face velocity and round the
// half step's product by itself, so there the last bits differ from the others'.
__device__ __forceinline__ float r_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double r_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float r_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double r_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float r_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double r_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float r_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double r_fma(double a, double b, double c) { return __fma_rn(a, b, c); }

// Raw face velocity (C/advectbyzxA1.c:34, C/advectbyzxB1.c:34) from m_x and
// rho of the pencil below (m) and the current one (c).
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_face(R mm, R mc, R rm, R rc)
{
    if constexpr (EX)
        return (mm + mc) / (rm + rc);
    else
        return fast_div(r_add(mm, mc), r_add(rm, rc));
}

// 1-2-1 smoothing of the face velocity (C/advectbyzxA1.c:36-41): vm, v, vp at i-1, i, i+1.
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_smooth(R vm, R v, R vp)
{
    using W = wide_t<R, EX>;
    if constexpr (EX && sizeof(R) == 4) {
        // the sum of two floats rounds alike with and without the double between, and the
        // quarter is exact unless it is subnormal; the sum may overflow where the quarter does not
        const R f = vm + vp, t = r_fma(R(2), v, f), m = fabsf(t);
        return (t == R(0) || (m > 0x1p-120f && m < 0x1p127f)) ? t * R(0.25)
                                                              : R((W(f) + W(2.0) * W(v)) / W(4.0));
    } else if constexpr (EX)
        return R((W(vm + vp) + W(2.0) * W(v)) / W(4.0));
    else
        return r_mul(r_fma(R(2), v, r_add(vm, vp)), R(0.25));
}

// b vg (C/tvdb.c:31-34), vg b1 (C/tvdb.c:55-60)
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_prod(R x, R y)
{
    if constexpr (EX)
        return x * y;
    else
        return r_mul(x, y);
}

// vh = (vg(i) + vg(i+1)) / 2 in the abXYc form (C/tvdb.c:25-29)
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_vh(R vg, R vgn)
{
    if constexpr (EX)
        return lin<R, EX>(R(0.5), vg, R(0.5), vgn);
    else
        return r_fma(R(0.5), vg, r_mul(R(0.5), vgn));
}

// Half step b1 = b - (f1(i) - f1(i-1)) dt / 2 (C/tvdb.c:41-47).
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_half(R bv, R f1, R fm, R dt)
{
    if constexpr (EX && sizeof(R) == 8)
        return bv - (f1 - fm) * dt / R(2);
    else if constexpr (EX)  // bv - x / 2 rounded once: the double between does not change a float
        return r_fma(R(-0.5), (f1 - fm) * dt, bv);
    else  // dt / 2 is loop-invariant: one fused multiply-add per cell
        return r_fma(r_sub(fm, f1), r_mul(dt, R(0.5)), bv);
}

// Limited upwind flux times dt at i+1/2 (C/tvdb.c:54-78) from vb = vg b1 at
// i-1, i, i+1, i+2 and the sign of vh(i).
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_flux(R vbm, R vb0, R vbp, R vbpp, R vh, R dt)
{
    if constexpr (EX) {
        // halves of differences: R(0.5) x rounds as the double quotient by 2.0 does
        R w, wp, wm;
        if (vh > R(0)) {
            w = vb0;
            wp = R(0.5) * (vbp - w);
            wm = R(0.5) * (w - vbm);
        } else {
            w = vbp;
            wp = R(0.5) * (w - vbpp);
            wm = R(0.5) * (vb0 - w);
        }
        const R dw = vanleer<R, EX>(wm, wp);
        return (w + dw) * dt;
    } else {
        // The same differences with the operands selected (no branch), and the
        // limiter on the undivided differences: with wm = dm/2, wp = dp/2,
        // 2 wm wp / (wm + wp) = dm dp / (dm + dp).
        const bool up = vh > R(0);
        const R w = up ? vb0 : vbp;
        const R dp = r_sub(vbp, up ? vb0 : vbpp);
        const R dm = r_sub(vb0, up ? vbm : vbp);
        const R p = r_mul(dm, dp);
        return r_mul(r_add(w, mul_if_pos(p, p, rcp_ftz(r_add(dm, dp)))), dt);
    }
}

// Advected field b - (flux(i) - flux(i-1)) (C/tvdb.c:79-88)
template <typename R, bool EX>
__device__ __forceinline__ R tvdb_new(R bv, R flux, R fm)
{
    if constexpr (EX)
        return bv - (flux - fm);
    else
        return r_sub(bv, r_sub(flux, fm));
}

}  // namespace mhd
