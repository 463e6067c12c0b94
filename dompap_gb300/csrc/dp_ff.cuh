// dp_ff.cuh — double-float ("float-float") arithmetic for the float64-parity
// pair kernels.
//
// GB300 executes float64 at 1/64 of the float32 rate, so the per-pair
// arithmetic of the parity mode runs on pairs (hi, lo) of floats carrying
// ~48 significant bits (relative error ~1e-14, far inside the 1e-10 parity
// bound), using the error-free transformations of Dekker (1971) and Knuth
// (TAOCP vol. 2): TwoSum, QuickTwoSum and an FMA-based TwoProduct. Functions
// without a double-float form (exp, cos, ...) are evaluated in float64 and
// split back.
#pragma once

struct dpff {
    float hi, lo;
    __device__ __forceinline__ dpff() : hi(0.0f), lo(0.0f) {}
    __device__ __forceinline__ constexpr dpff(float h, float l) : hi(h), lo(l) {}
    // from a double (exact split of its leading 48 bits)
    __device__ __forceinline__ dpff(double v) : hi((float)v), lo((float)(v - (double)(float)v)) {}
    __device__ __forceinline__ dpff(int v) : hi((float)v), lo(0.0f) {}
    __device__ __forceinline__ double to_double() const { return (double)hi + (double)lo; }
};

__device__ __forceinline__ dpff dpff_quick_two_sum(float a, float b) {
    const float s = a + b;
    return dpff(s, b - (s - a));
}

__device__ __forceinline__ dpff dpff_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return dpff(s, (a - (s - bb)) + (b - bb));
}

// Dekker's addition: absolute error below ~2^-47 (|x| + |y|), relative
// 2^-47 for operands of one sign; the pair sums need no more (their float64
// counterparts carry 2^-53 (|x| + |y|)), at about half the instructions of
// the sign-robust form.
__device__ __forceinline__ dpff operator+(dpff x, dpff y) {
    const dpff s = dpff_two_sum(x.hi, y.hi);
    return dpff_quick_two_sum(s.hi, s.lo + (x.lo + y.lo));
}

__device__ __forceinline__ dpff operator-(dpff x) { return dpff(-x.hi, -x.lo); }
__device__ __forceinline__ dpff operator-(dpff x, dpff y) { return x + (-y); }

__device__ __forceinline__ dpff operator*(dpff x, dpff y) {
    const float p = x.hi * y.hi;
    float e = fmaf(x.hi, y.hi, -p);
    e = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, e));
    return dpff_quick_two_sum(p, e);
}

__device__ __forceinline__ dpff dpff_mul_f(dpff x, float b) {
    const float p = x.hi * b;
    const float e = fmaf(x.lo, b, fmaf(x.hi, b, -p));
    return dpff_quick_two_sum(p, e);
}

__device__ __forceinline__ dpff operator/(dpff x, dpff y) {
    const float q1 = x.hi / y.hi;
    const dpff r = x - dpff_mul_f(y, q1);
    const float q2 = r.hi / y.hi;
    return dpff_quick_two_sum(q1, q2);
}

__device__ __forceinline__ dpff& operator+=(dpff& x, dpff y) {
    x = x + y;
    return x;
}

__device__ __forceinline__ bool operator<(dpff x, dpff y) { return x.hi < y.hi || (x.hi == y.hi && x.lo < y.lo); }
__device__ __forceinline__ bool operator>(dpff x, dpff y) { return y < x; }
__device__ __forceinline__ bool operator<=(dpff x, dpff y) { return !(y < x); }
__device__ __forceinline__ bool operator>=(dpff x, dpff y) { return !(x < y); }

// 1/sqrt(q): the float estimate y (rsqrtf, then one float Newton step, so
// y is within about an ulp and e below is ~2^-24) refined by one Newton step
// with its second-order term, y (1 + e/2 + 3e^2/8), e = 1 - q y^2. y^2 and
// q.hi y^2 are split exactly by FMA and 1 - p is exact (p is within a few
// ulp of 1); the result is good to ~1.2e-14 relative.
__device__ __forceinline__ dpff dpff_rsqrt(dpff q) {
    const float y0 = rsqrtf(q.hi);
    const float y = fmaf(0.5f * y0, fmaf(-(q.hi * y0), y0, 1.0f), y0);
    const float t = y * y;
    const float tl = fmaf(y, y, -t);   // y^2 = t + tl
    const float p = q.hi * t;
    const float pl = fmaf(q.hi, t, -p);  // q.hi t = p + pl
    const float e = ((1.0f - p) - pl) - fmaf(q.hi, tl, q.lo * t);
    return dpff_quick_two_sum(y, y * e * fmaf(0.375f, e, 0.5f));
}

// x^2 unnormalised: (p, e) with p + e = x^2 to ~2^-48 (for dpff_accumulate).
__device__ __forceinline__ dpff dpff_sqr_unnormalised(dpff x) {
    const float p = x.hi * x.hi;
    return dpff(p, fmaf(fmaf(2.0f, x.hi, x.lo), x.lo, fmaf(x.hi, x.hi, -p)));
}

__device__ __forceinline__ dpff dpff_add_f(dpff x, float b) {
    const dpff s = dpff_two_sum(x.hi, b);
    return dpff_quick_two_sum(s.hi, s.lo + x.lo);
}

// 1/q: the float estimate y (one ulp, so e = 1 - q y below is ~2^-23; its
// leading part 1 - q.hi y is exact by FMA), refined by y (1 + e + e^2):
// ~2^-47 relative.
__device__ __forceinline__ dpff dpff_rcp(dpff q) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(q.hi));
    const float e = fmaf(-q.lo, y, fmaf(-q.hi, y, 1.0f));
    return dpff_quick_two_sum(y, y * fmaf(e, e, e));
}

// The 64-bit fixed-point displacement v (units 2^-64 M) times M, U = M / 2^32 as
// a double-float, u24 = U.hi / 2^24. v = h 2^32 + l: what the nearest float of h
// leaves of it (at most 64) and the upper 24 bits of l make one 31-bit integer
// (a funnel shift), so three conversions carry ~48 leading bits of v; what is
// dropped lies below 2^-56 M, so M is not the box but at most eight times the
// cutoff (dp_sim::shift64): with M = 10,000 the force error was 30 times that of a
// short box. An h that rounds up to 2^31 saturates on the way
// back, one short of it. (An int64 split into 22 / 22 / 20 bits took the same
// three conversions and twice the instructions; rounding h towards zero, or
// leaving the product unnormalised, saves a few but costs a bit of accuracy.)
__device__ __forceinline__ dpff dpff_from_fixed(long long v, dpff U, float u24) {
    const int h = (int)(v >> 32);
    const float fh = __int2float_rn(h);
    int back = __float2int_rn(fh);
    if (back == 0x7FFFFFFF) back = (int)0x80000000u;
    const uint32_t rest = (uint32_t)h - (uint32_t)back;
    const float fl = __int2float_rn((int)__funnelshift_l((uint32_t)v, rest, 24));
    const float p = fh * U.hi;
    const float e = fmaf(fh, U.hi, -p);
    return dpff_quick_two_sum(p, fmaf(fl, u24, fmaf(fh, U.lo, e)));
}

// Compensated accumulation s += v (cascaded summation in the manner of
// Neumaier): s.hi carries the running float sum, s.lo collects the exact
// rounding errors of s.hi and the low parts of the addends, unnormalised;
// the value is s.hi + s.lo.
__device__ __forceinline__ void dpff_accumulate(dpff& s, dpff v) {
    const dpff t = dpff_two_sum(s.hi, v.hi);
    s.hi = t.hi;
    s.lo += t.lo + v.lo;
}

// s += x y without normalising the product first: its leading float p and
// the FMA-exact rounding error plus cross terms go to the two parts of s.
__device__ __forceinline__ void dpff_accumulate_prod(dpff& s, dpff x, dpff y) {
    const float p = x.hi * y.hi;
    const float pe = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, fmaf(x.hi, y.hi, -p)));
    const dpff t = dpff_two_sum(s.hi, p);
    s.hi = t.hi;
    s.lo += t.lo + pe;
}

// Exact float constants of generated expressions (dp_k<dpff>): x c and x + c
// with one float operand.
struct dpff_k {
    float v;
    __device__ __forceinline__ operator dpff() const { return dpff(v, 0.0f); }
};
template <>
struct dp_k_t<dpff> {
    typedef dpff_k type;
    static __device__ __forceinline__ dpff_k make(float v) { return dpff_k{v}; }
};
__device__ __forceinline__ dpff operator*(dpff x, dpff_k k) { return dpff_mul_f(x, k.v); }
__device__ __forceinline__ dpff operator*(dpff_k k, dpff x) { return dpff_mul_f(x, k.v); }
__device__ __forceinline__ dpff operator+(dpff x, dpff_k k) { return dpff_add_f(x, k.v); }
__device__ __forceinline__ dpff operator+(dpff_k k, dpff x) { return dpff_add_f(x, k.v); }
__device__ __forceinline__ dpff operator-(dpff x, dpff_k k) { return dpff_add_f(x, -k.v); }
__device__ __forceinline__ dpff operator-(dpff_k k, dpff x) { return dpff_add_f(-x, k.v); }
__device__ __forceinline__ dpff_k operator-(dpff_k k) { return dpff_k{-k.v}; }

// hi + lo in float64 with the two widenings done on bit patterns.
__device__ __forceinline__ double dpff_to_double(dpff x) { return dp_f2d(x.hi) + dp_f2d(x.lo); }

// Functions without a double-float form go through float64.
#define DPFF_VIA_DOUBLE(fn)                                                                    \
    __device__ __forceinline__ dpff fn(dpff x) { return dpff(fn(x.to_double())); }
DPFF_VIA_DOUBLE(exp)
DPFF_VIA_DOUBLE(log)
DPFF_VIA_DOUBLE(sin)
DPFF_VIA_DOUBLE(cos)
DPFF_VIA_DOUBLE(tan)
DPFF_VIA_DOUBLE(sinh)
DPFF_VIA_DOUBLE(cosh)
DPFF_VIA_DOUBLE(tanh)
DPFF_VIA_DOUBLE(erf)
DPFF_VIA_DOUBLE(erfc)
DPFF_VIA_DOUBLE(atan)
DPFF_VIA_DOUBLE(asin)
DPFF_VIA_DOUBLE(acos)
DPFF_VIA_DOUBLE(cbrt)
DPFF_VIA_DOUBLE(sqrt)
#undef DPFF_VIA_DOUBLE
__device__ __forceinline__ dpff fabs(dpff x) { return x.hi < 0.0f ? -x : x; }
__device__ __forceinline__ dpff pow(dpff x, dpff y) { return dpff(pow(x.to_double(), y.to_double())); }
