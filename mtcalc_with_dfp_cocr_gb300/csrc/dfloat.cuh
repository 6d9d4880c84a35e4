// Double-float arithmetic: a value is the unevaluated sum hi + lo of two
// FP32 numbers (|lo| <= ulp(hi)/2), a 48-bit significand computed entirely on
// the FP32 pipes.  GB300 issues FP32 at 64x its FP64 rate, so a few FP32
// operations per double-float operation still run far ahead of FP64.
//
// Error-free transformations used (Knuth's two-sum, Dekker's fast two-sum,
// the FMA two-product; see Shewchuk 1997, Hida-Li-Bailey 2001):
//   two_sum(a, b)      = (s, e) with s + e = a + b exactly      (6 flops)
//   fast_two_sum(a, b) = (s, e), requires |a| >= |b|            (3 flops)
//   two_prod(a, b)     = (p, e) with p + e = a * b exactly      (2 flops)
// Sums of products are accumulated unnormalised (hi carries a two-sum chain,
// lo collects the error terms) and normalised once at the end.
#pragma once
#include <cuda_runtime.h>

namespace mtgpu {
namespace dfl {

struct df {
    float h, l;
};

__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

__device__ __forceinline__ void fast_two_sum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    e = __fsub_rn(b, __fsub_rn(s, a));
}

__device__ __forceinline__ df norm(float h, float l)
{
    df r;
    fast_two_sum(h, l, r.h, r.l);
    return r;
}

// unnormalised accumulator
struct acc {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(df x)
    {
        float s, e;
        two_sum(h, x.h, s, e);
        h = s;
        l = __fadd_rn(l, __fadd_rn(e, x.l));
    }
    // += x * y
    __device__ __forceinline__ void mac(df x, df y)
    {
        const float p = __fmul_rn(x.h, y.h);
        float pe = __fmaf_rn(x.h, y.h, -p);
        pe = __fmaf_rn(x.h, y.l, pe);
        pe = __fmaf_rn(x.l, y.h, pe);
        float s, e;
        two_sum(h, p, s, e);
        h = s;
        l = __fadd_rn(l, __fadd_rn(e, pe));
    }
    // += x * y with y a plain float
    __device__ __forceinline__ void macf(df x, float y)
    {
        const float p = __fmul_rn(x.h, y);
        float pe = __fmaf_rn(x.h, y, -p);
        pe = __fmaf_rn(x.l, y, pe);
        float s, e;
        two_sum(h, p, s, e);
        h = s;
        l = __fadd_rn(l, __fadd_rn(e, pe));
    }
    __device__ __forceinline__ df get() const { return norm(h, l); }
    __device__ __forceinline__ double to_double() const { return (double)h + (double)l; }
};

__device__ __forceinline__ df neg(df a) { return df{-a.h, -a.l}; }

__device__ __forceinline__ df add(df a, df b)
{
    acc t;
    t.h = a.h;
    t.l = a.l;
    t.add(b);
    return t.get();
}

// complex double-float; in memory a float4 (re.h, im.h, re.l, im.l), so that
// the high and the low parts of both components are register pairs for the
// packed operations below
struct dfc {
    df re, im;
};
__device__ __forceinline__ dfc from4(float4 v) { return dfc{df{v.x, v.z}, df{v.y, v.w}}; }
__host__ __device__ __forceinline__ float4 to4(df re, df im) { return make_float4(re.h, im.h, re.l, im.l); }
__device__ __forceinline__ float4 to4(dfc v) { return to4(v.re, v.im); }
__device__ __forceinline__ double2 to_d2(float4 v)
{
    return make_double2((double)v.x + (double)v.z, (double)v.y + (double)v.w);
}

// x + a * y  (complex)
__device__ __forceinline__ dfc caxpy(dfc x, dfc a, dfc y)
{
    acc r, i;
    r.h = x.re.h; r.l = x.re.l;
    i.h = x.im.h; i.l = x.im.l;
    r.mac(a.re, y.re);
    r.mac(neg(a.im), y.im);
    i.mac(a.re, y.im);
    i.mac(a.im, y.re);
    return dfc{r.get(), i.get()};
}

__device__ __forceinline__ dfc cmul(dfc a, dfc b)
{
    acc r, i;
    r.mac(a.re, b.re);
    r.mac(neg(a.im), b.im);
    i.mac(a.re, b.im);
    i.mac(a.im, b.re);
    return dfc{r.get(), i.get()};
}

// host/device conversion of an FP64 value (host side or rare device use)
__host__ __device__ __forceinline__ df from_double(double v)
{
    const float h = (float)v;
    return df{h, (float)(v - (double)h)};
}

// ---- packed pairs
// Blackwell's f32x2 instructions do one FP32 operation on two registers each:
// the same rate per value as the scalar ones (measured 125 against 120 values
// a clock and SM) in half the issue slots.  Both components of a complex
// value take the same operations wherever the other factor is real, and with
// one exchange of the components where it is complex, so the row kernels
// carry (re, im) pairs.  Every result equals the scalar operations' above.
using u64 = unsigned long long;
__device__ __forceinline__ u64 pk(float a, float b)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpk(u64 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a * b + 0: written as a plain product, an add of its result would be
// contracted to one multiply-add (ptxas does so for f32x2 in spite of .rn;
// a unit test of the accumulators below shows it)
__device__ __forceinline__ u64 mul2(u64 a, u64 b) { return fma2(a, b, 0ull); }
// a - b (b times -1 is exact)
__device__ __forceinline__ u64 sub2(u64 a, u64 b) { return fma2(b, 0xbf800000bf800000ull, a); }
__device__ __forceinline__ u64 swap2(u64 v)
{
    float a, b;
    unpk(v, a, b);
    return pk(b, a);
}

// a complex double-float (or two double-floats): high and low parts
struct cdf {
    u64 h, l;
};
__device__ __forceinline__ cdf cdf_of(float4 v) { return cdf{pk(v.x, v.y), pk(v.z, v.w)}; }
__device__ __forceinline__ float4 to4(cdf v)
{
    float4 r;
    unpk(v.h, r.x, r.y);
    unpk(v.l, r.z, r.w);
    return r;
}
// loads that stay where they are written, before the arithmetic: left to
// itself the compiler moves a load next to its use among the packed
// operations, and a row kernel's loads go out one latency after the other
__device__ __forceinline__ cdf ldn(const float4 *p)      // read-only during the kernel
{
    cdf v;
    asm volatile("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(v.h), "=l"(v.l) : "l"(p));
    return v;
}
__device__ __forceinline__ cdf ldg(const float4 *p)
{
    cdf v;
    asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.h), "=l"(v.l) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ cdf cswap(cdf v) { return cdf{swap2(v.h), swap2(v.l)}; }
__device__ __forceinline__ cdf czero() { return cdf{0ull, 0ull}; }
// a real double-float for both components
__device__ __forceinline__ cdf both(df v) { return cdf{pk(v.h, v.h), pk(v.l, v.l)}; }
__device__ __forceinline__ df lane0(cdf v)
{
    df r;
    float t;
    unpk(v.h, r.h, t);
    unpk(v.l, r.l, t);
    return r;
}
__device__ __forceinline__ df lane1(cdf v)
{
    df r;
    float t;
    unpk(v.h, t, r.h);
    unpk(v.l, t, r.l);
    return r;
}

// acc for both components
struct acc2 {
    u64 h = 0ull, l = 0ull;
    __device__ __forceinline__ void start(cdf x) { h = x.h; l = x.l; }
    __device__ __forceinline__ void add(cdf x)
    {
        const u64 s = add2(h, x.h), nb = sub2(h, s);
        const u64 e = add2(sub2(h, add2(s, nb)), add2(x.h, nb));
        h = s;
        l = add2(l, add2(e, x.l));
    }
    __device__ __forceinline__ void sub(cdf x)
    {
        const u64 s = sub2(h, x.h), nb = sub2(h, s);
        const u64 e = add2(sub2(h, add2(s, nb)), sub2(nb, x.h));
        h = s;
        l = add2(l, sub2(e, x.l));
    }
    // = x * y, component by component
    __device__ __forceinline__ void first(cdf x, cdf y)
    {
        h = mul2(x.h, y.h);
        l = err(x, y, sub2(0ull, h));
    }
    // += x * y
    __device__ __forceinline__ void mac(cdf x, cdf y)
    {
        const u64 p = mul2(x.h, y.h);
        const u64 pe = err(x, y, sub2(0ull, p));
        const u64 s = add2(h, p), b = sub2(s, h);
        const u64 e = add2(sub2(h, sub2(s, b)), sub2(p, b));
        h = s;
        l = add2(l, add2(e, pe));
    }
    // -= x * y
    __device__ __forceinline__ void msub(cdf x, cdf y)
    {
        const u64 np = sub2(0ull, mul2(x.h, y.h));
        const u64 pe = err(x, y, np);
        const u64 s = add2(h, np), b = sub2(s, h);
        const u64 e = add2(sub2(h, sub2(s, b)), sub2(np, b));
        h = s;
        l = add2(l, sub2(e, pe));
    }
    // x * y - p for np = -p, p = fl(x.h y.h)
    static __device__ __forceinline__ u64 err(cdf x, cdf y, u64 np)
    {
        u64 t = fma2(x.h, y.h, np);
        t = fma2(x.h, y.l, t);
        return fma2(x.l, y.h, t);
    }
    __device__ __forceinline__ cdf get() const
    {
        const u64 s = add2(h, l);
        return cdf{s, sub2(l, sub2(s, h))};
    }
};
__device__ __forceinline__ cdf csub(cdf a, cdf b)
{
    acc2 t;
    t.start(a);
    t.sub(b);
    return t.get();
}
// a complex factor of many products: (re, re) and (-im, im)
struct cfac {
    cdf r, i;
};
__device__ __forceinline__ cfac cfac_of(cdf v)
{
    const df r = lane0(v), i = lane1(v);
    return cfac{both(r), cdf{pk(-i.h, i.h), pk(-i.l, i.l)}};
}
__device__ __forceinline__ cfac cfac_of(dfc a)
{
    return cfac{both(a.re), cdf{pk(-a.im.h, a.im.h), pk(-a.im.l, a.im.l)}};
}
// x + a * y
__device__ __forceinline__ cdf caxpy(cdf x, const cfac &a, cdf y)
{
    acc2 t;
    t.start(x);
    t.mac(a.r, y);
    t.mac(a.i, cswap(y));
    return t.get();
}
__device__ __forceinline__ cdf cmul(const cfac &a, cdf y)
{
    acc2 t;
    t.first(a.r, y);
    t.mac(a.i, cswap(y));
    return t.get();
}

// ---- sums across threads
// A partial sum as three FP32 numbers a + b + c.  Adding two of them with
// two-sums on a and b keeps more than 60 bits (the error is that of c, about
// 2^-70 of the larger operand; below 2^-89 c leaves FP32's range and it is
// 2^-149), more than FP64's 53, in 21 FP32 operations:
// GB300 issues an FP64 add of a warp once in 16 cycles, so the FP64 trees
// over 256 threads that these sums replace took most of a small kernel.
// FP32's range is the limit of a and not FP64's: sums that could overflow are
// carried scaled by 2^-64 (float4 form, w = 1).
struct tf {
    float a, b, c;
};
__device__ __forceinline__ tf tf_add(tf x, tf y)
{
    float s, e, t, f, u, g;
    two_sum(x.a, y.a, s, e);
    two_sum(x.b, y.b, t, f);
    two_sum(e, t, u, g);
    return tf{s, u, __fadd_rn(__fadd_rn(x.c, y.c), __fadd_rn(f, g))};
}
__device__ __forceinline__ tf tf_scale(tf x, float s) { return tf{x.a * s, x.b * s, x.c * s}; }
__device__ __forceinline__ tf tf_of(df x) { return tf{x.h, x.l, 0.f}; }
__device__ __forceinline__ tf tf_neg(tf x) { return tf{-x.a, -x.b, -x.c}; }
// the sum of both components of an accumulator, and its first minus its second
__device__ __forceinline__ tf tf_sum(const acc2 &x)
{
    return tf_add(tf_of(lane0(cdf{x.h, x.l})), tf_of(lane1(cdf{x.h, x.l})));
}
__device__ __forceinline__ tf tf_diff(const acc2 &x)
{
    return tf_add(tf_of(lane0(cdf{x.h, x.l})), tf_neg(tf_of(lane1(cdf{x.h, x.l}))));
}
constexpr float kTfBig = 0x1p100f, kTfDown = 0x1p-64f;
// FP64 sums as three FP32 numbers each; true where they are scaled by 2^-64
// to stay in FP32's range (up to 2^192)
__device__ __forceinline__ bool tf_of(const double (&d)[2], tf (&v)[2])
{
    const bool down = fmax(fabs(d[0]), fabs(d[1])) >= kTfBig;
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const double s = down ? d[n] * kTfDown : d[n];
        const float a = (float)s;
        const double r = s - (double)a;
        const float b = (float)r;
        v[n] = tf{a, b, (float)(r - (double)b)};
    }
    return down;
}
__device__ __forceinline__ float4 tf_pack(tf x, float w) { return make_float4(x.a, x.b, x.c, w); }
__device__ __forceinline__ float4 tf4_add(float4 x, float4 y)
{
    tf u{x.x, x.y, x.z}, v{y.x, y.y, y.z};
    if (x.w != y.w) {
        if (x.w == 0.f) u = tf_scale(u, kTfDown);
        else v = tf_scale(v, kTfDown);
    }
    return tf_pack(tf_add(u, v), fmaxf(x.w, y.w));
}
__device__ __forceinline__ double tf4_double(float4 x)
{
    const double v = (double)x.x + ((double)x.y + (double)x.z);
    return x.w == 0.f ? v : v * 0x1p64;
}

}  // namespace dfl
}  // namespace mtgpu
