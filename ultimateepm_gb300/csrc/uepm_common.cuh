// uepm_common.cuh -- shared device types and helpers for the sm_103a band-structure kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cfloat>

namespace uepm {

// ------------------------------------------------------------------------------------------------
// Complex arithmetic on (re, im) pairs, written with explicit fused multiply-adds: on GB300 every
// FP64 instruction (add, mul or fma) costs one slot of the narrow FP64 pipe, so a complex
// multiply-accumulate is exactly 4 FMAs and nothing else.
template <typename T>
struct cx {
    T x, y;
};

template <typename T>
__host__ __device__ __forceinline__ cx<T> mk(T x, T y) {
    cx<T> r;
    r.x = x;
    r.y = y;
    return r;
}
template <typename T>
__device__ __forceinline__ cx<T> cadd(cx<T> a, cx<T> b) {
    return mk(a.x + b.x, a.y + b.y);
}
template <typename T>
__device__ __forceinline__ cx<T> csub(cx<T> a, cx<T> b) {
    return mk(a.x - b.x, a.y - b.y);
}
template <typename T>
__device__ __forceinline__ cx<T> cmul(cx<T> a, cx<T> b) {
    return mk(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// c + a * b
template <typename T>
__device__ __forceinline__ cx<T> cfma(cx<T> a, cx<T> b, cx<T> c) {
    return mk(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
// c + conj(a) * b
template <typename T>
__device__ __forceinline__ cx<T> cfmac(cx<T> a, cx<T> b, cx<T> c) {
    return mk(fma(a.x, b.x, fma(a.y, b.y, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
}
// c - a * conj(b)
template <typename T>
__device__ __forceinline__ cx<T> cfms_conjb(cx<T> a, cx<T> b, cx<T> c) {
    return mk(fma(-a.x, b.x, fma(-a.y, b.y, c.x)), fma(-a.y, b.x, fma(a.x, b.y, c.y)));
}
template <typename T>
__device__ __forceinline__ cx<T> cscale(cx<T> a, T s) {
    return mk(a.x * s, a.y * s);
}

// Quaternions w + x i + y j + z k, for Hermitian matrices that time reversal times inversion makes
// quaternionic (spin-orbit on an inversion-symmetric crystal): half the order of the complex spinor
// matrix, with a quarter of its elements. The products keep the operands' order.
template <typename T>
struct __align__(4 * sizeof(T) <= 16 ? 4 * sizeof(T) : 16) qt {
    T w, x, y, z;
};
template <typename T>
__host__ __device__ __forceinline__ qt<T> mkq(T w, T x, T y, T z) {
    qt<T> r;
    r.w = w;
    r.x = x;
    r.y = y;
    r.z = z;
    return r;
}
template <typename T>
__device__ __forceinline__ qt<T> cadd(qt<T> a, qt<T> b) {
    return mkq(a.w + b.w, a.x + b.x, a.y + b.y, a.z + b.z);
}
template <typename T>
__device__ __forceinline__ qt<T> csub(qt<T> a, qt<T> b) {
    return mkq(a.w - b.w, a.x - b.x, a.y - b.y, a.z - b.z);
}
template <typename T>
__device__ __forceinline__ qt<T> cscale(qt<T> a, T s) {
    return mkq(a.w * s, a.x * s, a.y * s, a.z * s);
}
// c + a * b
template <typename T>
__device__ __forceinline__ qt<T> cfma(qt<T> a, qt<T> b, qt<T> c) {
    return mkq(fma(a.w, b.w, fma(-a.x, b.x, fma(-a.y, b.y, fma(-a.z, b.z, c.w)))),
               fma(a.w, b.x, fma(a.x, b.w, fma(a.y, b.z, fma(-a.z, b.y, c.x)))),
               fma(a.w, b.y, fma(-a.x, b.z, fma(a.y, b.w, fma(a.z, b.x, c.y)))),
               fma(a.w, b.z, fma(a.x, b.y, fma(-a.y, b.x, fma(a.z, b.w, c.z)))));
}
template <typename T>
__device__ __forceinline__ qt<T> cmul(qt<T> a, qt<T> b) {
    return cfma(a, b, mkq<T>(0, 0, 0, 0));
}
// c + conj(a) * b
template <typename T>
__device__ __forceinline__ qt<T> cfmac(qt<T> a, qt<T> b, qt<T> c) {
    return cfma(mkq(a.w, -a.x, -a.y, -a.z), b, c);
}
// c - a * conj(b)
template <typename T>
__device__ __forceinline__ qt<T> cfms_conjb(qt<T> a, qt<T> b, qt<T> c) {
    return cfma(a, mkq(-b.w, b.x, b.y, b.z), c);
}
__device__ __forceinline__ qt<float> ldc(const qt<float>* p) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    return mkq(v.x, v.y, v.z, v.w);
}
__device__ __forceinline__ void stc(qt<float>* p, qt<float> a) {
    *reinterpret_cast<float4*>(p) = make_float4(a.w, a.x, a.y, a.z);
}
__device__ __forceinline__ qt<double> ldc(const qt<double>* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2  a = q[0], b = q[1];
    return mkq(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void stc(qt<double>* p, qt<double> a) {
    double2* q = reinterpret_cast<double2*>(p);
    q[0]       = make_double2(a.w, a.x);
    q[1]       = make_double2(a.y, a.z);
}

// 16-byte (double) / 8-byte (float) vector loads and stores of one complex element.
__device__ __forceinline__ cx<double> ldc(const cx<double>* p) {
    double2 v = *reinterpret_cast<const double2*>(p);
    return mk(v.x, v.y);
}
__device__ __forceinline__ cx<float> ldc(const cx<float>* p) {
    float2 v = *reinterpret_cast<const float2*>(p);
    return mk(v.x, v.y);
}
__device__ __forceinline__ void stc(cx<double>* p, cx<double> a) { *reinterpret_cast<double2*>(p) = make_double2(a.x, a.y); }
__device__ __forceinline__ void stc(cx<float>* p, cx<float> a) { *reinterpret_cast<float2*>(p) = make_float2(a.x, a.y); }

// Real-scalar counterparts of the complex helpers: the same kernel templates serve real symmetric
// matrices (H(k) is exactly real for diamond-structure local / symmetric-nonlocal EPM without SOC).
__device__ __forceinline__ double cadd(double a, double b) { return a + b; }
__device__ __forceinline__ float cadd(float a, float b) { return a + b; }
__device__ __forceinline__ double csub(double a, double b) { return a - b; }
__device__ __forceinline__ float csub(float a, float b) { return a - b; }
__device__ __forceinline__ double cmul(double a, double b) { return a * b; }
__device__ __forceinline__ float cmul(float a, float b) { return a * b; }
__device__ __forceinline__ double cfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float cfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double cfmac(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float cfmac(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double cfms_conjb(double a, double b, double c) { return fma(-a, b, c); }
__device__ __forceinline__ float cfms_conjb(float a, float b, float c) { return fmaf(-a, b, c); }
__device__ __forceinline__ double cscale(double a, double s) { return a * s; }
__device__ __forceinline__ float cscale(float a, float s) { return a * s; }
__device__ __forceinline__ double ldc(const double* p) { return *p; }
__device__ __forceinline__ float ldc(const float* p) { return *p; }
__device__ __forceinline__ void stc(double* p, double a) { *p = a; }
__device__ __forceinline__ void stc(float* p, float a) { *p = a; }

// Scalar traits: R = the real type, and the few operations that differ between real and complex.
template <typename S>
struct ST;
template <>
struct ST<double> {
    using R = double;
    static constexpr bool cplx = false;
    static __device__ __forceinline__ double zero() { return 0.0; }
    static __device__ __forceinline__ double one() { return 1.0; }
    static __device__ __forceinline__ double re(double a) { return a; }
    static __device__ __forceinline__ double im(double) { return 0.0; }
    static __device__ __forceinline__ double make(double r, double) { return r; }
    static __device__ __forceinline__ double conj(double a) { return a; }
    static __device__ __forceinline__ double norm(double a) { return a * a; }
    static __device__ __forceinline__ double neg(double a) { return -a; }
};
template <>
struct ST<float> {
    using R = float;
    static constexpr bool cplx = false;
    static __device__ __forceinline__ float zero() { return 0.f; }
    static __device__ __forceinline__ float one() { return 1.f; }
    static __device__ __forceinline__ float re(float a) { return a; }
    static __device__ __forceinline__ float im(float) { return 0.f; }
    static __device__ __forceinline__ float make(float r, float) { return r; }
    static __device__ __forceinline__ float conj(float a) { return a; }
    static __device__ __forceinline__ float norm(float a) { return a * a; }
    static __device__ __forceinline__ float neg(float a) { return -a; }
};
template <typename T>
struct ST<cx<T>> {
    using R = T;
    static constexpr bool cplx = true;
    static __device__ __forceinline__ cx<T> zero() { return mk<T>(0, 0); }
    static __device__ __forceinline__ cx<T> one() { return mk<T>(1, 0); }
    static __device__ __forceinline__ T re(cx<T> a) { return a.x; }
    static __device__ __forceinline__ T im(cx<T> a) { return a.y; }
    static __device__ __forceinline__ cx<T> make(T r, T i) { return mk<T>(r, i); }
    static __device__ __forceinline__ cx<T> conj(cx<T> a) { return mk<T>(a.x, -a.y); }
    static __device__ __forceinline__ T norm(cx<T> a) { return fma(a.x, a.x, a.y * a.y); }
    static __device__ __forceinline__ cx<T> neg(cx<T> a) { return mk<T>(-a.x, -a.y); }
};

template <typename T>
struct ST<qt<T>> {
    using R = T;
    static constexpr bool cplx = false;
    static __device__ __forceinline__ qt<T> zero() { return mkq<T>(0, 0, 0, 0); }
    static __device__ __forceinline__ qt<T> one() { return mkq<T>(1, 0, 0, 0); }
    static __device__ __forceinline__ T re(qt<T> a) { return a.w; }
    static __device__ __forceinline__ T im(qt<T>) { return 0; }  // of real values only
    static __device__ __forceinline__ qt<T> make(T r, T) { return mkq<T>(r, 0, 0, 0); }
    static __device__ __forceinline__ qt<T> conj(qt<T> a) { return mkq<T>(a.w, -a.x, -a.y, -a.z); }
    static __device__ __forceinline__ T norm(qt<T> a) { return fma(a.w, a.w, fma(a.x, a.x, fma(a.y, a.y, a.z * a.z))); }
    static __device__ __forceinline__ qt<T> neg(qt<T> a) { return mkq<T>(-a.w, -a.x, -a.y, -a.z); }
};
// The imaginary part's norm, and a scalar from a real number, for every scalar type.
__device__ __forceinline__ float  imag_norm(float) { return 0.f; }
__device__ __forceinline__ double imag_norm(double) { return 0.0; }
template <typename T>
__device__ __forceinline__ T imag_norm(cx<T> a) {
    return a.y * a.y;
}
template <typename T>
__device__ __forceinline__ T imag_norm(qt<T> a) {
    return fma(a.x, a.x, fma(a.y, a.y, a.z * a.z));
}

template <typename S>
struct is_quat {
    static constexpr bool value = false;
};
template <typename T>
struct is_quat<qt<T>> {
    static constexpr bool value = true;
};
// Re(conj(a) b)
template <typename T>
__device__ __forceinline__ T re_dot(qt<T> a, qt<T> b) {
    return fma(a.w, b.w, fma(a.x, b.x, fma(a.y, b.y, a.z * b.z)));
}
// sqrt(x) and its reciprocal, and 1 / x. FP64: PTX's approximations (relative error at most 2^-19.9 over 4 M
// values of all exponents) refined by one step of third order, with e = 1 - x y^2 and y (1 + e/2 + 3 e^2/8) (the binomial
// series of (1 - e)^-1/2), and e = 1 - x r and r (1 + e + e^2); the square root gets one correction by its
// residual. Errors of the third order are below 2^-58; what remains is the rounding of the last operations
// (relative errors at most 1.11e-16, 1.38e-16 and 1.11e-16 over those values). A dependent FP64 operation takes
// above 100 clocks on this pipe: the reflector's scalars took 4.9 k clocks per column with the library's square
// root and division and FP64 compares, 3.5 k so. Only where x and its approximation are normal numbers well
// inside the range (in_seed_range); elsewhere the library's.
__device__ __forceinline__ bool in_seed_range(double x) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;  // biased exponent
    return e > 200 && e < 1800;
}
__device__ __forceinline__ void sqrt_pair(double x, double& s, double& is) {  // x > 0
    if (!in_seed_range(x)) {
        s  = sqrt(x);
        is = 1.0 / s;
        return;
    }
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const double c = e * fma(0.375, e, 0.5);
    const double b = fma(t, c, t);
    is             = fma(y, c, y);
    s              = fma(0.5 * is, fma(-b, b, x), b);
}
__device__ __forceinline__ double recip(double x) {
    if (!in_seed_range(x)) return 1.0 / x;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ void sqrt_pair(float x, float& s, float& is) {
    s  = sqrtf(x);
    is = 1.f / s;
}
__device__ __forceinline__ float recip(float x) { return 1.f / x; }

// The reflector of a quaternion column (alpha; tail), |tail|^2 = tail2: H = I - v tau v^H with beta real,
// tau = (beta - alpha) / beta and v = (1; tail sc), sc = (alpha - beta)^-1 (zlarfg's, the operands in order).
template <typename T>
__device__ __forceinline__ void quat_reflector(qt<T> alpha, T tail2, T tiny, T& beta, qt<T>& tau, qt<T>& sc) {
    const T im = imag_norm(alpha);
    beta = alpha.w;
    tau = sc = mkq<T>(0, 0, 0, 0);
    if (tail2 <= tiny && im <= tiny) return;
    T ib;
    sqrt_pair(fma(alpha.w, alpha.w, tail2 + im), beta, ib);
    if (alpha.w >= 0) {
        beta = -beta;
        ib   = -ib;
    }
    const qt<T> df = mkq(alpha.w - beta, alpha.x, alpha.y, alpha.z);
    tau            = cscale(df, -ib);
    sc             = cscale(mkq(df.w, -df.x, -df.y, -df.z), recip(ST<qt<T>>::norm(df)));
}

// Lower-precision counterpart of a scalar type (FP64 -> FP32), for the mixed path.
template <typename S>
struct Lower;
template <>
struct Lower<double> {
    using type = float;
};
template <>
struct Lower<cx<double>> {
    using type = cx<float>;
};

// An FP64 matrix element carried as the unevaluated sum of two FP32 values, hi = fl32(v) and
// lo = fl32(v - hi) (about 48 significant bits, same size as the FP64 element): the mixed path's copy
// of H for the Rayleigh-Ritz products, which then run on the FP32 pipe.
struct __align__(8) ds2 {
    float hi, lo;
};
struct __align__(16) ds4 {
    float rhi, rlo, ihi, ilo;
};
template <typename S>
struct Split;
template <>
struct Split<double> {
    using type = ds2;
};
template <>
struct Split<cx<double>> {
    using type = ds4;
};
template <>
struct Lower<float> {
    using type = float;
};
template <>
struct Lower<cx<float>> {
    using type = cx<float>;
};
template <>
struct Lower<ds2> {
    using type = float;
};
template <>
struct Lower<ds4> {
    using type = cx<float>;
};

// Double-single accumulation (Dekker's exact product, Knuth's two-sum) with operations the compiler
// does not contract: acc += (xh + xl) * y with xh * y exact, carried as acc.h + acc.l.
struct dsacc {
    float h, l;
};
__device__ __forceinline__ void ds_add_prod(dsacc& a, float xh, float xl, float y) {
    const float p  = __fmul_rn(xh, y);
    const float pe = fmaf(xh, y, -p);
    const float s  = __fadd_rn(a.h, p);
    const float z  = __fsub_rn(s, a.h);
    const float er = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, z)), __fsub_rn(p, z));
    a.h            = s;
    a.l            = fmaf(xl, y, __fadd_rn(a.l, __fadd_rn(er, pe)));
}
// acc += x * y for FP32 x, y (the product exactly)
__device__ __forceinline__ void ds_add_prod(dsacc& a, float x, float y) {
    const float p  = __fmul_rn(x, y);
    const float pe = fmaf(x, y, -p);
    const float s  = __fadd_rn(a.h, p);
    const float z  = __fsub_rn(s, a.h);
    const float er = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, z)), __fsub_rn(p, z));
    a.h            = s;
    a.l            = __fadd_rn(a.l, __fadd_rn(er, pe));
}
__device__ __forceinline__ double ds_value(dsacc a) { return (double)a.h + (double)a.l; }

// Pairs of FP32 values in one 64-bit register pair (PTX's .f32x2 operations): two accumulations in the issue
// slots of one, each operation rounded as its scalar form, so the sums are the same bits.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
struct dsacc2 {
    f32x2 h, l;
};
// a += (xh + xl) y for both members; nxh = -xh
__device__ __forceinline__ void ds_add_prod(dsacc2& a, f32x2 xh, f32x2 nxh, f32x2 xl, f32x2 y) {
    const f32x2 p   = mul2(xh, y);
    const f32x2 npe = fma2(nxh, y, p);  // minus the product's rounding error
    const f32x2 s   = add2(a.h, p);
    const f32x2 z   = sub2(s, a.h);
    const f32x2 er  = add2(sub2(a.h, sub2(s, z)), sub2(p, z));
    a.h             = s;
    a.l             = fma2(xl, y, add2(a.l, sub2(er, npe)));
}

// Double-single numbers (an FP32 pair h + l, |l| <= ulp(h) / 2, about 48 significant bits) with the
// classical error-free transformations (Dekker, Knuth) on non-contracted FP32 operations: the mixed
// path evaluates the nonlocal matrix elements on the FP32 pipe with them instead of the FP64 pipe.
struct ds {
    float h, l;
};
__host__ __device__ inline ds ds_of_double(double v) {
    const float h = (float)v;
    return ds{h, (float)(v - (double)h)};
}
__device__ __forceinline__ ds ds_quick(float s, float e) {  // |s| >= |e|
    const float t = __fadd_rn(s, e);
    return ds{t, __fsub_rn(e, __fsub_rn(t, s))};
}
__device__ __forceinline__ ds ds_add(ds a, ds b) {
    const float s  = __fadd_rn(a.h, b.h);
    const float bb = __fsub_rn(s, a.h);
    const float e  = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, bb)), __fsub_rn(b.h, bb));
    return ds_quick(s, __fadd_rn(e, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ ds ds_neg(ds a) { return ds{-a.h, -a.l}; }
__device__ __forceinline__ ds ds_sub(ds a, ds b) { return ds_add(a, ds_neg(b)); }
__device__ __forceinline__ ds ds_mul(ds a, ds b) {
    const float p = __fmul_rn(a.h, b.h);
    const float e = fmaf(a.h, b.h, -p);
    return ds_quick(p, fmaf(a.h, b.l, fmaf(a.l, b.h, e)));
}
__device__ __forceinline__ ds ds_mulf(ds a, float b) {  // times an exact FP32 value
    const float p = __fmul_rn(a.h, b);
    const float e = fmaf(a.h, b, -p);
    return ds_quick(p, fmaf(a.l, b, e));
}
__device__ __forceinline__ ds ds_div(ds a, ds b) {  // long division, two quotient digits
    const float q1 = __fdiv_rn(a.h, b.h);
    const ds    r  = ds_sub(a, ds_mulf(b, q1));
    const float q2 = __fdiv_rn(r.h, b.h);
    return ds_quick(q1, q2);
}
__device__ __forceinline__ float ds_abs_hi(ds a) { return fabsf(a.h); }

// cp.async of one naturally aligned element of B = 4 or 8 bytes, global -> shared
template <int B>
__device__ __forceinline__ void cp_async_elem(void* dst, const void* src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <typename T>
__device__ __forceinline__ cx<T> warp_sum(cx<T> v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <typename T>
struct num;
template <>
struct num<double> {
    static __host__ __device__ constexpr double eps() { return DBL_EPSILON; }
    static __host__ __device__ constexpr double tiny() { return DBL_MIN; }
};
template <>
struct num<float> {
    static __host__ __device__ constexpr float eps() { return FLT_EPSILON; }
    static __host__ __device__ constexpr float tiny() { return FLT_MIN; }
};

// ------------------------------------------------------------------------------------------------
// Device-side material constants. Every derived constant is computed on the host in double with the
// reference's own expression (Material.h / Material.cpp / Hamiltonian.cpp / SpinOrbitFunctional.cpp),
// so the kernels start from bit-identical constants.
struct DevParams {
    int N;        // scalar basis size
    int n;        // matrix order (N or 2N)
    int nl;       // nonlocal correction on
    int soc;      // spin-orbit blocks on
    int square;   // nonlocal well: 1 square, 0 gaussian
    int has_R0a, has_R0c, has_A2a, has_A2c;
    int same_nl;  // anion and cation carry the same nonlocal parameters (their terms are equal)
    double kin_pref;      // two_pi_over_a * two_pi_over_a * diag_factor      (Hamiltonian.cpp:68-72)
    double grad_pref;     // 2 * diag_factor * (2pi/a)^2                      (Hamiltonian.cpp:167)
    double frac_to_phys;  // 1 / (2pi/a)                                      (Hamiltonian.cpp:190)
    // nonlocal (Material.cpp:139-208)
    double ff;            // fourier factor 2pi/a (1/m)
    double nl_df;         // pow(h_bar,2)/(2 m_e q_e)
    double Vpre;          // 4 pi / atomic volume
    double kF2;           // pow(fermi momentum, 2)
    double alpha0a, beta0a, A2a, alpha0c, beta0c, A2c;
    double R0a, R0c, R2a, R2c;
    double R0a2, R0c2, R2a2, R2c2;         // pow(R, 2.0)
    double R0a3h, R0c3h, R2a3h, R2c3h;     // pow(R, 3.0) / 2
    double R0a3t, R0c3t;                   // pow(R, 3.0) / 3
    double gpre_a, gpre_c;                 // 5 pi^1.5 (R2^3 / volume)
    // spin-orbit (SpinOrbitFunctional.cpp:20-138)
    unsigned pa, pc;
    double ra, rc, alpha_soc, mu_soc, kfac, bohr;
};

// The nonlocal constants of DevParams as double-single numbers, for the mixed path's square-well
// element on the FP32 pipe; products the FP64 element forms first are formed on the host in FP64
// (the same order of operations) and then split.
struct DevParamsDS {
    int  has_R0a, has_R0c, has_A2a, has_A2c, same_nl;
    ds   kF2;
    ds   alpha0a, nl_df_beta0a, alpha0c, beta0c_nl_df;  // A0 = alpha0 + (nl_df beta0) t
    ds   A2a_5, A2c_5;                                  // A2 5 (eV)
    // The F_l terms times Vpre = 4 pi / volume, so that every intermediate stays well inside FP32's
    // exponent range (R^2 / (n1^2 - n2^2) ~ 1e-41 in SI units is not): VR2s = Vpre R^2 / (2 pi / a)
    // for the far branch, whose norms are taken in units of 2 pi / a, VR3h = Vpre R^3 / 2 and
    // VR3t = Vpre R^3 / 3 for the near branch and its K = 0 limit.
    ds   VR0a2s, VR0c2s, VR2a2s, VR2c2s;
    ds   VR0a3h, VR0c3h, VR2a3h, VR2c3h, VR0a3t, VR0c3t;
    // gaussian d-wells: V2 = (gpre A2) P2 i2(x) e_i e_j with x = (R2^2 / 2) n1 n2
    int  square;
    ds   gA2a, gA2c, R2a2h, R2c2h;  // gpre A2, R2^2 / 2
    // spin-orbit: lambda_1 = mu B_c B_c', lambda_2 = (alpha mu) B_a B_a'
    ds   mu_soc, alpha_mu_soc;
};

// Per-(k, basis vector) quantities computed once per k in the row kernel and read by the
// element kernel. Layout: rows[(b * N + i) * ROW_STRIDE + field].
enum RowField {
    RF_KGX = 0, RF_KGY, RF_KGZ,   // k + G_i, reduced
    RF_KX, RF_KY, RF_KZ,          // (k + G_i) * 2pi/a, 1/m
    RF_NK,                        // |K_i|
    RF_KIN,                       // kinetic diagonal C |k+G_i|^2
    RF_J0A,                       // j_{-1}, j_0, j_1 at |K| R0_anion
    RF_J0C = RF_J0A + 3,          // j_{-1}, j_0, j_1 at |K| R0_cation
    RF_J2A = RF_J0C + 3,          // j_1, j_2, j_3 at |K| R2_anion (square well)
    RF_J2C = RF_J2A + 3,          // j_1, j_2, j_3 at |K| R2_cation (square well)
    RF_GEA = RF_J2C + 3,          // exp(-0.25 |K|^2 R2a^2) (gaussian well)
    RF_GEC,                       // exp(-0.25 |K|^2 R2c^2)
    RF_BC,                        // SOC radial factor B_period(|K|), cation
    RF_BA,                        // anion
    ROW_STRIDE = 24,
    // 1 / |K_i| (0 where K = 0), in a slot the well type leaves free: the gaussian exponentials'
    // slot for square wells, the l = 2 Bessel slot for gaussian wells
    RF_INVK_SQUARE = RF_GEA,
    RF_INVK_GAUSS  = RF_J2A,
    // in the mixed path's double-single copy of the rows only: |K_i| in units of 2 pi / a, in the
    // slot the well type leaves free
    RF_NKS32_SQUARE = RF_GEC,
    RF_NKS32_GAUSS  = RF_J2C
};

}  // namespace uepm
