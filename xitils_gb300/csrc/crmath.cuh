// Correctly rounded float sin / cos / pow / exp / log for the sampling code.
//
// Why: a sampled direction decides which triangle the next ray hits and, inside
// microfacet normal mapping's random walk (Sandbox/MicrofacetBasedNormalMapping/
// Main.cpp:127-168), when the walk stops; a one-ulp difference in a sine or
// cosine there sends a path elsewhere. The reference calls the C library's float
// functions, which round correctly for all but about 1 % of the azimuths the
// samplers draw (counted against long double); CUDA's
// own sinf / cosf / powf are accurate to a few ulp but round differently far more
// often. An oracle whose float functions all round correctly renders the
// normal-mapping scenes within relMSE 3e-6 of the plain oracle, and the GPU
// renders within 1e-9 of that correctly rounded oracle; only on the longest
// diffuse paths (the occluded room, no depth limit) do the C library's own
// misroundings move an image by more (1.3e-4 at 128 x 128 x 4). So the samplers
// call the functions below, and the evaluation code (values, not decisions)
// keeps CUDA's faster ones.
//
// crSinCosf: double-float arithmetic (pairs of floats, Dekker 1971, "A
// floating-point technique for extending the available precision"; exact
// products with FMA), Cody-Waite argument reduction by pi/2 split into three
// floats, Taylor series of sin and cos on [-pi/4, pi/4] with the leading terms in
// double-float (relative error near 2^-43), and one final rounding of hi + lo to
// float. Results equal the correctly rounded float except when the exact value
// lies within about 2^-43 relative of a rounding boundary. Arguments beyond
// |x| = 8 (never passed by the samplers) take the double-precision path.
// crPowf / crExpf / crLogf: double-float evaluation with a rounding test, the
// double-precision function where the test cannot decide (see below). crAsinf: the
// double-precision function (error below 2 ulp of a double) rounded once to float --
// the correctly rounded float unless the exact value lies within a few double ulp of
// a float rounding boundary.
//
// Everything here is __host__ __device__ so that a host build can test it
// exhaustively against long double; device code uses explicitly rounded
// intrinsics so that no compiler contraction changes the error-free steps.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#if defined(__CUDA_ARCH__)
#define XGB_FADD(a, b) __fadd_rn(a, b)
#define XGB_FSUB(a, b) __fsub_rn(a, b)
#define XGB_FMUL(a, b) __fmul_rn(a, b)
#define XGB_FFMA(a, b, c) __fmaf_rn(a, b, c)
#define XGB_CR_TABLE static __device__ const
#define XGB_CR_NOINLINE __noinline__
#else
#define XGB_CR_TABLE static const
#define XGB_CR_NOINLINE
#define XGB_FADD(a, b) ((a) + (b))
#define XGB_FSUB(a, b) ((a) - (b))
#define XGB_FMUL(a, b) ((a) * (b))
#define XGB_FFMA(a, b, c) fmaf(a, b, c)
#endif

namespace xgb {
namespace cr {

struct Df {
    float hi, lo;
};

// a + b = s + e exactly (Knuth's TwoSum).
__host__ __device__ __forceinline__ Df twoSum(float a, float b) {
    const float s = XGB_FADD(a, b);
    const float bb = XGB_FSUB(s, a);
    const float e = XGB_FADD(XGB_FSUB(a, XGB_FSUB(s, bb)), XGB_FSUB(b, bb));
    return Df{s, e};
}
// a + b = s + e exactly when |a| >= |b| (Dekker's FastTwoSum).
__host__ __device__ __forceinline__ Df fastTwoSum(float a, float b) {
    const float s = XGB_FADD(a, b);
    return Df{s, XGB_FSUB(b, XGB_FSUB(s, a))};
}
// a * b = p + e exactly (FMA).
__host__ __device__ __forceinline__ Df twoProd(float a, float b) {
    const float p = XGB_FMUL(a, b);
    return Df{p, XGB_FFMA(a, b, -p)};
}
// Double-float sum, relatively accurate even under cancellation.
__host__ __device__ __forceinline__ Df add(Df a, Df b) {
    Df s = twoSum(a.hi, b.hi);
    const Df t = twoSum(a.lo, b.lo);
    s = fastTwoSum(s.hi, XGB_FADD(s.lo, t.hi));
    return fastTwoSum(s.hi, XGB_FADD(s.lo, t.lo));
}
// Double-float product.
__host__ __device__ __forceinline__ Df mul(Df a, Df b) {
    Df p = twoProd(a.hi, b.hi);
    p.lo = XGB_FFMA(a.hi, b.lo, p.lo);
    p.lo = XGB_FFMA(a.lo, b.hi, p.lo);
    return fastTwoSum(p.hi, p.lo);
}
// c + z * u for a constant c larger in magnitude than z * u (Horner step of a
// series whose terms decrease).
__host__ __device__ __forceinline__ Df horner(Df c, Df z, Df u) {
    const Df p = mul(z, u);
    Df s = fastTwoSum(c.hi, p.hi);
    s.lo = XGB_FADD(s.lo, XGB_FADD(c.lo, p.lo));
    return fastTwoSum(s.hi, s.lo);
}

// pi / 2 = kC1 + kC2 + kC3 - 9.5e-23, kC1 with 21 significant bits so that k kC1
// is exact for |k| <= 7.
constexpr float kC1 = 0x1.921fb0p+0f;
constexpr float kC2 = 0x1.5110b4p-22f;
constexpr float kC3 = 0x1.84698ap-48f;
constexpr float kTwoOverPi = 0x1.45f306p-1f;
// 1/n! as double-float (hi, lo) where the series needs it, float beyond
constexpr float kF3h = 0x1.555556p-3f, kF3l = -0x1.555556p-28f;
constexpr float kF4h = 0x1.555556p-5f, kF4l = -0x1.555556p-30f;
constexpr float kF5h = 0x1.111112p-7f, kF5l = -0x1.ddddde0p-32f;
constexpr float kF6h = 0x1.6c16c2p-10f, kF6l = -0x1.27d27ep-35f;
constexpr float kF7h = 0x1.a01a02p-13f, kF7l = -0x1.7f97fap-39f;
constexpr float kF8h = 0x1.a01a02p-16f, kF8l = -0x1.7f97fap-42f;
constexpr float kF9 = 0x1.71de3ap-19f, kF10 = 0x1.27e4fcp-22f, kF11 = 0x1.ae6456p-26f;
constexpr float kF12 = 0x1.1eed8ep-29f, kF13 = 0x1.612462p-33f, kF14 = 0x1.93974ap-37f;
constexpr float kF15 = 0x1.ae7f3ep-41f, kF16 = 0x1.ae7f3ep-45f;

// sin and cos of x, |x| <= 8, as unrounded double-floats; the quadrant in *q.
// Reduction: k = nearest integer to x 2/pi; t = x - k kC1 is exact (k kC1 is, and
// Sterbenz's lemma covers the subtraction); then k kC2 exactly as a double-float
// and k kC3 as a float. Series in z = r^2: the terms above 2^-40 of the leading
// one in double-float, the rest in float.
__host__ __device__ __forceinline__ void sinCosReduced(float x, Df* s, Df* c, int* q) {
    const float k = rintf(XGB_FMUL(x, kTwoOverPi));
    const float t = XGB_FFMA(-k, kC1, x);  // exact
    const Df p = twoProd(k, kC2);
    Df r = twoSum(t, -p.hi);
    r.lo = XGB_FSUB(XGB_FSUB(r.lo, p.lo), XGB_FMUL(k, kC3));
    r = fastTwoSum(r.hi, r.lo);
    *q = ((int)k) & 3;
    const Df z = mul(r, r);
    // sin r = r + r z (-1/3! + z (1/5! - z (1/7! - z (1/9! - z (1/11! - z (1/13! - z/15!))))))
    float ts = XGB_FFMA(z.hi, -kF15, kF13);
    ts = XGB_FFMA(z.hi, ts, -kF11);
    ts = XGB_FFMA(z.hi, ts, kF9);
    Df u = horner(Df{-kF7h, -kF7l}, z, Df{ts, 0.0f});
    u = horner(Df{kF5h, kF5l}, z, u);
    u = horner(Df{-kF3h, -kF3l}, z, u);
    const Df w = mul(mul(r, z), u);
    Df sr = fastTwoSum(r.hi, w.hi);
    sr.lo = XGB_FADD(sr.lo, XGB_FADD(r.lo, w.lo));
    *s = sr;
    // cos r = 1 + z (-1/2 + z (1/4! - z (1/6! - z (1/8! - z (1/10! - z (1/12! - z (1/14! - z/16!)))))))
    float tc = XGB_FFMA(z.hi, kF16, -kF14);
    tc = XGB_FFMA(z.hi, tc, kF12);
    tc = XGB_FFMA(z.hi, tc, -kF10);
    Df v = horner(Df{kF8h, kF8l}, z, Df{tc, 0.0f});
    v = horner(Df{-kF6h, -kF6l}, z, v);
    v = horner(Df{kF4h, kF4l}, z, v);
    v = horner(Df{-0.5f, 0.0f}, z, v);
    const Df y = mul(z, v);
    Df cr = fastTwoSum(1.0f, y.hi);
    cr.lo = XGB_FADD(cr.lo, y.lo);
    *c = cr;
}

}  // namespace cr

// Arguments the samplers never pass (a call, so that its code stays out of the kernels' way).
XGB_CR_NOINLINE static __host__ __device__ float2 sinCosDouble(float x) {
    return make_float2((float)sin((double)x), (float)cos((double)x));
}
// Correctly rounded (sinf(x), cosf(x)) (see the header of this file). Inlined:
// a call (measured) costs the terrain's shading more than the extra registers.
static __host__ __device__ __forceinline__ float2 crSinCos(float x) {
    const float ax = fabsf(x);
    if (!(ax <= 8.0f)) return sinCosDouble(x);  // or NaN / inf
    // |x^3 / 6| and x^2 / 2 below half an ulp: sin x rounds to x, cos x to 1
    if (ax < 0x1p-12f) return make_float2(x, 1.0f);
    cr::Df s, c;
    int q;
    cr::sinCosReduced(x, &s, &c, &q);
    const float sr = XGB_FADD(s.hi, s.lo), cr_ = XGB_FADD(c.hi, c.lo);  // one rounding of hi + lo
    return q == 0 ? make_float2(sr, cr_) : (q == 1 ? make_float2(cr_, -sr) : (q == 2 ? make_float2(-sr, -cr_)
                                                                                   : make_float2(-cr_, sr)));
}
__host__ __device__ __forceinline__ void crSinCosf(float x, float* sOut, float* cOut) {
    const float2 sc = crSinCos(x);
    *sOut = sc.x;
    *cOut = sc.y;
}

// ---- exp, log and pow in double-float, with a rounding test -----------------------
// GB300 runs FP64 at 1/64 of the FP32 rate: two FP64 pow calls per glossy vertex kept
// the FP64 pipe 68 % busy, and the EM fit's eight FP64 exp calls per sample and step
// 54 %. The functions below evaluate the value as hi + lo in float pairs to about 2^-41
// relative (table-driven: Tang, "Table-driven implementation of the exponential function
// in IEEE floating-point arithmetic", 1989, and of the logarithm, 1990), round it once,
// and keep the result only when hi + (lo - e) and hi + (lo + e) round to the same float
// for a bound e on the error (Ziv, "Fast evaluation of elementary mathematical functions
// with correctly rounded last bit", 1991); the one call in about 10^4 that is too close
// to a rounding boundary, and arguments outside the ranges below, take the
// double-precision function as before, so the results are the same floats.
namespace cr {

// 2^(j/16) = hi + lo
struct TabExp { float hi, lo; };
#define XGB_EXP_TABLE                                                                                                  \
    {{0x1.000000p+0f, 0.0f}, {0x1.0b5586p+0f, 0x1.9f3122p-25f}, {0x1.172b84p+0f, -0x1.c15742p-27f},                  \
     {0x1.2387a6p+0f, 0x1.ceac48p-25f}, {0x1.306fe0p+0f, 0x1.4636e2p-25f}, {0x1.3dea64p+0f, 0x1.824684p-25f},        \
     {0x1.4bfdaep+0f, -0x1.593abcp-25f}, {0x1.5ab07ep+0f, -0x1.5bd5ecp-27f}, {0x1.6a09e6p+0f, 0x1.9fcef4p-26f},      \
     {0x1.7a1148p+0f, -0x1.829fd0p-25f}, {0x1.8ace54p+0f, 0x1.15506ep-27f}, {0x1.9c4918p+0f, 0x1.51f848p-27f},       \
     {0x1.ae89fap+0f, -0x1.a94b14p-26f}, {0x1.c199bep+0f, -0x1.3d56b2p-27f}, {0x1.d5818ep+0f, -0x1.822dbcp-27f},     \
     {0x1.ea4afap+0f, 0x1.52486cp-27f}}
// for the 32 intervals [1 + j/32, 1 + (j+1)/32): c, a multiple of 2^-9 near the inverse of
// the interval's centre, and -log(c) = hi + lo
struct TabLog { float c, hi, lo; };
#define XGB_LOG_TABLE                                                                                                  \
    {{0x1.f8p-1f, 0x1.020566p-6f, -0x1.db29eep-32f}, {0x1.e9p-1f, 0x1.788596p-5f, -0x1.72a212p-31f},                  \
     {0x1.dbp-1f, 0x1.333d80p-4f, -0x1.f9f02ep-30f}, {0x1.cep-1f, 0x1.a4e764p-4f, 0x1.637870p-33f},                   \
     {0x1.c1p-1f, 0x1.0ce7ecp-3f, 0x1.b99852p-28f}, {0x1.b5p-1f, 0x1.4462bap-3f, -0x1.1b2612p-30f},                   \
     {0x1.aap-1f, 0x1.7898d8p-3f, 0x1.51131cp-29f}, {0x1.9fp-1f, 0x1.ae2ca6p-3f, 0x1.ece57ap-28f},                    \
     {0x1.95p-1f, 0x1.e020ccp-3f, 0x1.88d6aep-29f}, {0x1.8bp-1f, 0x1.09aa58p-2f, -0x1.a32726p-27f},                   \
     {0x1.82p-1f, 0x1.214456p-2f, 0x1.a1d71ap-27f}, {0x1.79p-1f, 0x1.396ce4p-2f, -0x1.4c8816p-27f},                   \
     {0x1.70p-1f, 0x1.522ae0p-2f, 0x1.ce28f6p-28f}, {0x1.68p-1f, 0x1.68ac84p-2f, -0x1.6395ecp-30f},                   \
     {0x1.60p-1f, 0x1.7fafa4p-2f, -0x1.09fabap-28f}, {0x1.59p-1f, 0x1.944144p-2f, -0x1.6bf9b4p-27f},                  \
     {0x1.52p-1f, 0x1.a93ed4p-2f, -0x1.ba930ep-29f}, {0x1.4bp-1f, 0x1.beacdap-2f, -0x1.d8e52ep-30f},                  \
     {0x1.44p-1f, 0x1.d49024p-2f, 0x1.b7be9ap-28f}, {0x1.3ep-1f, 0x1.e7b42cp-2f, 0x1.eed6bap-29f},                    \
     {0x1.38p-1f, 0x1.fb358ap-2f, 0x1.ef4910p-27f}, {0x1.32p-1f, 0x1.078bf0p-1f, 0x1.4cf15ap-27f},                    \
     {0x1.2dp-1f, 0x1.0ffb54p-1f, 0x1.09d23ap-28f}, {0x1.27p-1f, 0x1.1a4a74p-1f, -0x1.d21730p-27f},                   \
     {0x1.22p-1f, 0x1.230b0ep-1f, -0x1.d050dap-27f}, {0x1.1dp-1f, 0x1.2bf2a0p-1f, -0x1.9ef8f2p-27f},                  \
     {0x1.18p-1f, 0x1.35028ap-1f, 0x1.b3b190p-26f}, {0x1.13p-1f, 0x1.3e3c44p-1f, -0x1.b9c224p-27f},                   \
     {0x1.0fp-1f, 0x1.45bcc4p-1f, 0x1.93224ep-27f}, {0x1.0ap-1f, 0x1.4f45a8p-1f, 0x1.ad270cp-28f},                    \
     {0x1.06p-1f, 0x1.5707a2p-1f, 0x1.aee31ap-27f}, {0x1.02p-1f, 0x1.5ee82ap-1f, 0x1.448324p-26f}}
XGB_CR_TABLE TabExp kTabExp[16] = XGB_EXP_TABLE;
XGB_CR_TABLE TabLog kTabLog[32] = XGB_LOG_TABLE;

// log 2 = kL1 + kL2 + kL3 (15 significant bits in the first two, so that k kL1 and k kL2
// are exact), log(2) / 16 = kE1 + kE2 + kE3 (12 bits: exact times |n| < 2^12)
constexpr float kL1 = 0x1.62e400p-1f, kL2 = 0x1.7f7c00p-20f, kL3 = 0x1.1cf79ap-36f;
constexpr float kE1 = 0x1.62e000p-5f, kE2 = 0x1.0be000p-19f, kE3 = 0x1.be8e7cp-31f;
constexpr float kSixteenOverLog2 = 0x1.715476p+4f;

__host__ __device__ __forceinline__ int bitsOf(float x) {
#if defined(__CUDA_ARCH__)
    return __float_as_int(x);
#else
    int i; __builtin_memcpy(&i, &x, 4); return i;
#endif
}
__host__ __device__ __forceinline__ float floatOf(int i) {
#if defined(__CUDA_ARCH__)
    return __int_as_float(i);
#else
    float x; __builtin_memcpy(&x, &i, 4); return x;
#endif
}

// log x of a normal x in (0, 2) as a pair, to about 2^-43 absolute.
// x = 2^k m; r = m c - 1 (exact as a pair, |r| <= 2^-6); log x = k log 2 - log c + log(1 + r).
__host__ __device__ __forceinline__ Df logPair(float x) {
    const int b = bitsOf(x);
    const float k = (float)((b >> 23) - 127);
    const float m = floatOf((b & 0x7FFFFF) | 0x3F800000);
    const TabLog t = kTabLog[(b >> 18) & 31];
    const Df p = twoProd(m, t.c);
    const Df r = fastTwoSum(XGB_FSUB(p.hi, 1.0f), p.lo);
    const Df q = twoProd(r.hi, r.hi);
    float s = XGB_FFMA(r.hi, -0.125f, 0x1.249250p-3f);  // 1/3 - r/4 + r^2/5 - r^3/6 + r^4/7 - r^5/8
    s = XGB_FFMA(r.hi, s, -0x1.555556p-3f);
    s = XGB_FFMA(r.hi, s, 0x1.99999ap-3f);
    s = XGB_FFMA(r.hi, s, -0.25f);
    s = XGB_FFMA(r.hi, s, 0x1.555556p-2f);
    const Df a = twoSum(XGB_FMUL(k, kL1), t.hi);
    const Df c = twoSum(XGB_FMUL(k, kL2), r.hi);
    const Df d = twoSum(a.hi, c.hi);
    const Df e = twoSum(d.hi, XGB_FMUL(-0.5f, q.hi));
    float lo = XGB_FADD(XGB_FADD(a.lo, c.lo), XGB_FADD(d.lo, e.lo));
    lo = XGB_FADD(lo, XGB_FFMA(k, kL3, t.lo));
    // r.lo (1 - r.hi) - q.lo / 2 + r^3 s
    float w = XGB_FFMA(-r.hi, r.lo, r.lo);
    w = XGB_FFMA(-0.5f, q.lo, w);
    w = XGB_FFMA(XGB_FMUL(r.hi, q.hi), s, w);
    return fastTwoSum(e.hi, XGB_FADD(lo, w));
}

// exp(w.hi + w.lo) = 2^*e (hi + lo) with hi in [1, 2), |w| <= 150, to about 2^-41 relative.
__host__ __device__ __forceinline__ Df expPair(Df w, int* e) {
    const float n = rintf(XGB_FMUL(w.hi, kSixteenOverLog2));
    const Df r1 = twoSum(XGB_FFMA(-n, kE1, w.hi), XGB_FMUL(-n, kE2));
    const Df r = fastTwoSum(r1.hi, XGB_FADD(XGB_FFMA(-n, kE3, r1.lo), w.lo));
    const int ni = (int)n;
    *e = ni >> 4;
    const TabExp t = kTabExp[ni & 15];
    const Df q = twoProd(r.hi, r.hi);
    float s = XGB_FFMA(r.hi, 0x1.6c16c2p-10f, 0x1.111112p-7f);  // 1/6 + r/24 + r^2/120 + r^3/720
    s = XGB_FFMA(r.hi, s, 0x1.555556p-5f);
    s = XGB_FFMA(r.hi, s, 0x1.555556p-3f);
    float lo = XGB_FFMA(r.hi, r.lo, XGB_FMUL(0.5f, q.lo));
    lo = XGB_FADD(r.lo, XGB_FFMA(XGB_FMUL(r.hi, q.hi), s, lo));
    const Df u = fastTwoSum(r.hi, XGB_FMUL(0.5f, q.hi));  // expm1(r) = u.hi + (u.lo + lo)
    lo = XGB_FADD(lo, u.lo);
    const Df p = twoProd(t.hi, u.hi);
    const Df v = fastTwoSum(t.hi, p.hi);
    lo = XGB_FFMA(t.hi, lo, XGB_FFMA(t.lo, u.hi, t.lo));
    return fastTwoSum(v.hi, XGB_FADD(v.lo, XGB_FADD(p.lo, lo)));
}

constexpr float kExpError = 0x1p-39f;  // relative bound of expPair's error (and of pow's for |w| <= 64)

XGB_CR_NOINLINE static __host__ __device__ float powDouble(float x, float y) { return (float)pow((double)x, (double)y); }
XGB_CR_NOINLINE static __host__ __device__ float expDouble(float x) { return (float)exp((double)x); }
XGB_CR_NOINLINE static __host__ __device__ float logDouble(float x) { return (float)log((double)x); }

// a b - c d as the FP64 expression rounds it, (float)((double)a * b - (double)c * d): both
// products and their difference as exact sums of floats, then one rounding. That holds
// while the products neither overflow nor fall under 2^-102, where the low half of an
// exact product is lost: the callers pass unit vectors. Measured
// where it matters: the cross products of the samplers' frames, 31 FP64-pipe
// instructions per path of the terrain's shading at a sixteenth of an SM's issue
// rate each (61 % FP64 pipe; see k_shade in shade.cuh).
__host__ __device__ __forceinline__ float diffProd(float a, float b, float c, float d) {
    const Df p = twoProd(a, b), q = twoProd(c, d);
    const Df s = twoSum(p.hi, -q.hi);
    const Df t = twoSum(p.lo, -q.lo);
    const Df u = twoSum(s.lo, t.hi);
    const Df h = twoSum(s.hi, u.hi);
    return XGB_FADD(h.hi, XGB_FADD(h.lo, XGB_FADD(u.lo, t.lo)));
}

}  // namespace cr

// (float)(2 pi_d u) of the FP64 product, pi_d the double nearest pi.
__host__ __device__ __forceinline__ float crTwoPi(float u) {
    const float p = XGB_FMUL(u, 0x1.921fb6p+2f);
    const float e = XGB_FFMA(u, 0x1.921fb6p+2f, -p);
    return XGB_FADD(p, XGB_FFMA(u, -0x1.777a5cp-23f, e));
}
// (float)((double)x - pi_d)
__host__ __device__ __forceinline__ float crMinusPi(float x) {
    const cr::Df s = cr::twoSum(x, -0x1.921fb6p+1f);
    const cr::Df t = cr::twoSum(s.hi, 0x1.777a5cp-24f);
    return XGB_FADD(t.hi, XGB_FADD(t.lo, XGB_FADD(s.lo, 0x1p-48f)));
}
// (float)((double)x / pi_d)
__host__ __device__ __forceinline__ float crOverPi(float x) {
    const float p = XGB_FMUL(x, 0x1.45f306p-2f);
    const float e = XGB_FFMA(x, 0x1.45f306p-2f, -p);
    return XGB_FADD(p, XGB_FFMA(x, 0x1.b93910p-27f, e));
}

// exp(x): 0 below log(2^-150), double precision in the binades around the smallest normal
// floats, above 88 and for NaN.
__host__ __device__ __forceinline__ float crExpf(float x) {
    if (x < -104.0f) return 0.0f;
    if (!(x >= -87.0f && x <= 88.0f)) return cr::expDouble(x);
    int e;
    const cr::Df v = cr::expPair(cr::Df{x, 0.0f}, &e);
    const float err = XGB_FMUL(v.hi, cr::kExpError);
    const float a = XGB_FADD(v.hi, XGB_FSUB(v.lo, err)), b = XGB_FADD(v.hi, XGB_FADD(v.lo, err));
    if (a != b) return cr::expDouble(x);
    return XGB_FMUL(a, cr::floatOf((e + 127) << 23));
}
// log(x) for normal x in (0, 2) away from 1 (where hi + lo loses relative accuracy the test
// asks for the double-precision function).
__host__ __device__ __forceinline__ float crLogf(float x) {
    if (!(x >= 0x1p-100f && x < 2.0f)) return cr::logDouble(x);
    const cr::Df v = cr::logPair(x);
    const float err = 0x1p-41f + XGB_FMUL(fabsf(v.hi), 0x1p-41f);
    const float a = XGB_FADD(v.hi, XGB_FSUB(v.lo, err)), b = XGB_FADD(v.hi, XGB_FADD(v.lo, err));
    return a == b ? a : cr::logDouble(x);
}
// x^y for x in (0, 1] and exponents in (0, 2] (the glossy samplers), any other arguments
// in double precision.
__host__ __device__ __forceinline__ float crPowf(float x, float y) {
    if (!(x >= 0x1p-40f && x <= 1.0f && y > 0.0f && y <= 2.0f)) return x == 0.0f && y > 0.0f ? 0.0f : cr::powDouble(x, y);
    const cr::Df l = cr::logPair(x);
    cr::Df w = cr::twoProd(y, l.hi);
    w.lo = XGB_FFMA(y, l.lo, w.lo);
    int e;
    const cr::Df v = cr::expPair(w, &e);
    const float err = XGB_FMUL(v.hi, cr::kExpError);
    const float a = XGB_FADD(v.hi, XGB_FSUB(v.lo, err)), b = XGB_FADD(v.hi, XGB_FADD(v.lo, err));
    if (a != b) return cr::powDouble(x, y);
    return XGB_FMUL(a, cr::floatOf((e + 127) << 23));
}
// x^3 as pow(x, 3) rounds: the product of three floats as an exact sum, rounded once.
__host__ __device__ __forceinline__ float crCubef(float x) {
    const cr::Df q = cr::twoProd(x, x);
    const cr::Df p = cr::twoProd(q.hi, x), t = cr::twoProd(q.lo, x);
    const cr::Df l = cr::twoSum(p.lo, t.hi);
    const cr::Df h = cr::twoSum(p.hi, l.hi);
    return XGB_FADD(h.hi, XGB_FADD(h.lo, XGB_FADD(l.lo, t.lo)));
}
__host__ __device__ __forceinline__ float crAsinf(float x) { return (float)asin((double)x); }

}  // namespace xgb
