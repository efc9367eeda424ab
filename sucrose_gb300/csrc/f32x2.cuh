// Two FP32 values in one 64-bit register pair, and the packed instructions of
// sm_100 and later that add, multiply and fuse both at once (each result
// rounded as the scalar instruction rounds it). They halve the issue slots of
// a kernel that is bound by them. The helpers have the same names for float,
// so that a formula is written once for both widths.
#pragma once

#include "dfloat.cuh"

struct f2 {
    unsigned long long v;
};

SG_DEV f2 f2_of(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
SG_DEV void f2_split(f2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v)); }
SG_DEV f2 operator+(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
SG_DEV f2 operator-(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
SG_DEV f2 operator*(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
SG_DEV f2 fma_w(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
SG_DEV float fma_w(float a, float b, float c) { return fmaf(a, b, c); }

// A constant in both halves.
template <class T>
SG_DEV T all_w(float x);
template <>
SG_DEV float all_w<float>(float x) { return x; }
template <>
SG_DEV f2 all_w<f2>(float x) { return f2_of(x, x); }

// One comparison result per value.
struct mask2 {
    bool lo, hi;
};
template <class F>
SG_DEV f2 map_w(f2 a, F f) {
    float x, y;
    f2_split(a, x, y);
    return f2_of(f(x), f(y));
}
template <class F>
SG_DEV float map_w(float a, F f) { return f(a); }
SG_DEV mask2 less_w(f2 a, float b) {
    float x, y;
    f2_split(a, x, y);
    return {x < b, y < b};
}
SG_DEV bool less_w(float a, float b) { return a < b; }
SG_DEV mask2 not_above_w(f2 a, float b) {
    float x, y;
    f2_split(a, x, y);
    return {x <= b, y <= b};
}
SG_DEV bool not_above_w(float a, float b) { return a <= b; }
SG_DEV f2 select_w(mask2 m, f2 a, f2 b) {
    float ax, ay, bx, by;
    f2_split(a, ax, ay);
    f2_split(b, bx, by);
    return f2_of(m.lo ? ax : bx, m.hi ? ay : by);
}
SG_DEV float select_w(bool m, float a, float b) { return m ? a : b; }

// The type of a comparison's result.
template <class T>
struct MaskOf { using type = bool; };
template <>
struct MaskOf<f2> { using type = mask2; };
SG_DEV mask2 operator&&(mask2 a, mask2 b) { return {a.lo && b.lo, a.hi && b.hi}; }
SG_DEV mask2 less_w(f2 a, f2 b) {
    float ax, ay, bx, by;
    f2_split(a, ax, ay);
    f2_split(b, bx, by);
    return {ax < bx, ay < by};
}
SG_DEV mask2 not_above_w(f2 a, f2 b) {
    float ax, ay, bx, by;
    f2_split(a, ax, ay);
    f2_split(b, bx, by);
    return {ax <= bx, ay <= by};
}

// A sum of FP32 terms that loses no rounding error: two-sum's error of every
// addition goes into lo, so that sum and lo together hold about 48 bits whatever
// the terms' sizes and signs (Kahan's form, four instructions instead of seven,
// is exact only while the sum is the larger operand: 3e-9 of the terms'
// magnitudes on terms of both signs).
struct F2Sum {
    f2 hi, lo;
    SG_DEV void add(f2 v) {
        const f2 s = hi + v, b = s - hi;
        lo = lo + ((hi - (s - b)) + (v - b));
        hi = s;
    }
    // both halves, as hi + lo
    SG_DEV dfl total() const {
        float x, y, xl, yl;
        f2_split(hi, x, y);
        f2_split(lo, xl, yl);
        const dfl d = df_two_sum(x, y);
        return {d.hi, d.lo + (xl + yl)};
    }
};
