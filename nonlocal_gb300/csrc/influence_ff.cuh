// Influence functions in float-float (the pair assembly of mixed-precision solves) and in
// fixed point (the pair assembly and the flux post-processing).
#pragma once

#include <cmath>

#include "common.cuh"
#include "ff.cuh"

namespace nlgpu {

// shape<INF> in float-float (fast polynomial, polynomial and exponential with
// p divisible by n; the host sends the other kinds to the FP64 kernel)
// z0, z1: the coordinate differences in units of the radii
template<int INF>
__device__ __forceinline__ ff shape_ff(const Model& m, ff z0, ff z1, ff q, const ff* exp_table) {
    ff d;
    if (m.n == 2) d = ff_add(ff_mul(z0, z0), ff_mul(z1, z1));
    else if (m.n == 1) d = ff_add(ff_abs(z0), ff_abs(z1));
    else d = ff_add(ff_ipow(ff_abs(z0), m.n), ff_ipow(ff_abs(z1), m.n));
    if constexpr (INF == NLGPU_INFLUENCE_FAST_POLYNOMIAL) {
        return ff_lt(d, 1.0f) ? ff_sub(ff_make(1.0f), d) : ff_make(0.0f);
    } else {
        ff dp = d;
        if (m.p != m.n) {
            dp = ff_ipow(d, m.p / m.n);
            // beyond single precision the exponential is 0
            if (INF == NLGPU_INFLUENCE_EXPONENTIAL && !(dp.h <= 1e30f) && d.h <= 3.4e38f) dp = ff_make(1e30f);
        }
        if constexpr (INF == NLGPU_INFLUENCE_POLYNOMIAL)
            return ff_lt(d, 1.0f) ? ff_ipow(ff_sub(ff_make(1.0f), dp), int(m.q)) : ff_make(0.0f);
        else
            return ff_exp_nonpositive(ff_neg(ff_mul(q, dp)), exp_table);
    }
}

inline void fill_exp_table(FFExpTable& t) {
    for (int k = -FF_EXP_K; k <= FF_EXP_K; ++k) {
        const double x = std::exp(double(k) / double(FF_EXP_STEPS));
        const float hi = float(x);
        t.v[k + FF_EXP_K] = make_float2(hi, float(x - double(hi)));
    }
}

// float-float covers the continuous influence kinds with an integral power p / n; the
// rest runs the FP64 kernel
inline bool ff_supported(const Model& m) {
    if (m.n < 1) return false;
    if (m.influence == NLGPU_INFLUENCE_FAST_POLYNOMIAL) return true;
    if (m.influence == NLGPU_INFLUENCE_POLYNOMIAL || m.influence == NLGPU_INFLUENCE_EXPONENTIAL)
        return m.p >= 0 && m.p % m.n == 0;
    return false;
}

// ---------------------------------------------------------------- fixed point
// The influence functions of the usual exponents (n = 2) in 64-bit integers, for the
// pair assembly, whose contractions want fixed-point operands.  Coordinates in
// units of the radii are 59-bit integers with one exponent per mesh; 1 - d has an error of
// 2^-60 and its powers 60 bits, the exponential 54 (the units of q d log2(e), 2^-55, and of the two
// that fx_mulhi drops): as accurate as FP64, whose squared distance and exponential
// round to 53 bits each, on pipes that have 32 times the FP64 rate.

// floor-like a b 2^-64 of unsigned numbers, up to 2 below (the low halves' product is left out)
__device__ __forceinline__ unsigned long long fx_mulhi(unsigned long long a, unsigned long long b) {
    const unsigned ah = unsigned(a >> 32), al = unsigned(a), bh = unsigned(b >> 32), bl = unsigned(b);
    return (unsigned long long)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

constexpr int FX_SPLIT = 30;              // a number is hi 2^30 + lo
constexpr long long FX_ONE = 1ll << 60;   // influence values, and the polynomials' squared distance
constexpr int FX_EXP_UNIT = 54;           // the exponential's squared distance, in 2^-54
constexpr long long FX_FAR = 1ll << 62;   // any squared distance beyond 2^62 units

__device__ __forceinline__ int2 fx_split(long long z) {
    const long long hi = (z + (1 << (FX_SPLIT - 1))) >> FX_SPLIT;
    return make_int2(int(hi), int(z - (hi << FX_SPLIT)));
}

// x inv as an integer in 2^(ex - 58), ex >= 2 the exponent of the mesh's largest: the product to 106 bits
__device__ __forceinline__ int2 fx_coordinate(double x, double inv, int ex) {
    const double p = x * inv, r = fma(x, inv, -p);
    return fx_split(__double2ll_rn(scalbn(p, 58 - ex)) + __double2ll_rn(scalbn(r, 58 - ex)));
}

__device__ __forceinline__ long long fx_shift(long long v, int left) {
    return left >= 0 ? v << min(left, 63) : v >> min(-left, 63);
}

// the squared distance of two points (x hi, x lo, y hi, y lo) in 2^-UNIT
template<int UNIT>
__device__ __forceinline__ long long fx_distance(int4 a, int4 b, int ex) {
    const int xh = a.x - b.x, xl = a.y - b.y, yh = a.z - b.z, yl = a.w - b.w;
    const long long hh = (long long)xh * xh + (long long)yh * yh;
    const long long hl = (long long)xh * xl + (long long)yh * yl;
    const long long ll = (long long)xl * xl + (long long)yl * yl;
    const int s = 2 * ex + UNIT;   // hh 2^(s - 56) + hl 2^(s - 85) + ll 2^(s - 116)
    if ((hh >> max(118 - s, 0)) != 0) return FX_FAR;
    const long long d = fx_shift(hh, s - 56) + fx_shift(hl, s - 85) + fx_shift(ll, s - 116);
    return d & ~(d >> 63);   // the shifts round down
}

// the exponent of the coordinates' unit: of the largest one, given by its bits
constexpr int FX_MAX_EXPONENT = 20;   // below that the unit of the high words, 2^-8 radii, is far smaller than the radii
__device__ __forceinline__ int fx_exponent(const unsigned long long* extent) {
    const double x = __longlong_as_double((long long)*extent);
    return x >= 8.0 ? ilogb(x) : 2;
}

// x^n of 0 <= x <= 1
__device__ __forceinline__ long long fx_ipow(long long x, int n) {
    long long r = FX_ONE;
    for (int k = 0; k < n; ++k) r = k ? (long long)fx_mulhi((unsigned long long)r << 2, (unsigned long long)x << 2) : x;
    return r;
}

// exp(-q d) = 2^-(m + k / 256) e^-x from the mathematics of the exponential: q log2(e) d
// split into integer part m, k and a rest x / ln 2 below 1/256; 2^(-k / 256) from a
// table, 1 - e^-x by its series to x^5 (the sixth term is below 2^-60).
struct FXExp {
    unsigned long long rate;   // q log2(e) 2^(65 - shift), 2^62 to 2^63
    int shift;
    long long reach;           // where the value counts as zero (q d = 85, as in float-float)
};
constexpr int FX_EXP_K = 256;
struct FXExpTable {
    unsigned long long v[FX_EXP_K];   // 2^(63 - k / 256)
};

// value = v 2^-(63 + m); m = FX_EXP_ZERO: zero
constexpr int FX_EXP_ZERO = 1 << 20;
__device__ __forceinline__ unsigned long long fx_exp(long long d, const FXExp& f, const unsigned long long* table, int& m) {
    if (d > f.reach) {
        m = FX_EXP_ZERO;
        return 0;
    }
    const unsigned long long t = fx_mulhi((unsigned long long)d << f.shift, f.rate);   // in 2^-55
    m = int(t >> 55);
    const unsigned long long tab = table[unsigned(t >> 47) & 255u];
    const unsigned long long x = fx_mulhi(t << 17, 0xb17217f7d1cf79acull);   // ln 2 times the rest, in 2^-72
    const unsigned xh = unsigned(x >> 32), xl = unsigned(x);
    const unsigned long long x2 = ((unsigned long long)xh * xh >> 9) + (__umulhi(xh, xl) >> 8);   // x^2 / 2
    const unsigned x3 = __umulhi(__umulhi(unsigned(x2 >> 22), xh), 0x55555556u);                  // x^3 / 6, in 2^-58
    const unsigned x4 = __umulhi(x3, xh);                                                         // x^4 / 6, in 2^-66
    const unsigned x5 = __umulhi(__umulhi(x4, xh), 53687091u);                                    // x^5 / 120: 2^32 / 80
    const unsigned long long y = x - x2 + ((unsigned long long)x3 << 14) - ((unsigned long long)x4 << 4) + x5;
    return tab - (fx_mulhi(tab, y) >> 8);
}

// A value as v 2^-(63 + m) with v from 2^62 up to 2^63 (m = FX_EXP_ZERO: zero).  Kept so, an
// influence has as many bits near the horizon, where it is small, as elsewhere.
struct FXValue {
    unsigned long long v;
    int m;
};

// of x 2^-60, 0 <= x <= 2^60
__device__ __forceinline__ FXValue fx_normalised(long long x) {
    const int z = max(__clzll(x), 1);
    return x > 0 ? FXValue{(unsigned long long)x << (z - 1), z - 4} : FXValue{0, FX_EXP_ZERO};
}

__device__ __forceinline__ FXValue fx_power(FXValue x, int n) {
    if (n == 1 || (n > 0 && x.m == FX_EXP_ZERO)) return x;
    FXValue r{1ull << 63, 0};
    for (int k = 0; k < n; ++k) {   // 2^60 <= high product < 2^62
        const unsigned long long h = fx_mulhi(r.v, x.v);
        const int s = h >> 61 ? 1 : 2;
        r = FXValue{h << s, r.m + x.m + s - 1};
    }
    return r;
}

// shape<INF> of two points (n = 2 and the exponents that fx_supported names)
template<int INF>
__device__ __forceinline__ FXValue fx_shape(const Model& m, int4 a, int4 b, int ex, const FXExp& f,
                                            const unsigned long long* table) {
    if constexpr (INF == NLGPU_INFLUENCE_EXPONENTIAL) {
        FXValue r;
        r.v = fx_exp(fx_distance<FX_EXP_UNIT>(a, b, ex), f, table, r.m);
        return r;
    } else {
        const long long d = fx_distance<60>(a, b, ex);
        if constexpr (INF == NLGPU_INFLUENCE_FAST_POLYNOMIAL) return fx_normalised(FX_ONE - d);
        else return d < FX_ONE ? fx_power(fx_normalised(FX_ONE - fx_ipow(d, m.p / 2)), int(m.q)) : FXValue{0, FX_EXP_ZERO};
    }
}

// the double (its 53 bits rounded from 62 or 63)
__device__ __forceinline__ double fx_value(FXValue x) {
    const unsigned long long h = (x.v + 512) >> 10;   // 2^52 .. 2^53
    return x.m == FX_EXP_ZERO ? 0.0 : __longlong_as_double((long long)(((unsigned long long)(1021 - x.m) << 52) + h));
}

inline FXExp fx_exp_setup(double q) {
    const long double rate = (long double)q * 1.4426950408889634073599L;
    FXExp f{};
    f.shift = 3 + std::ilogb(rate);
    f.rate = static_cast<unsigned long long>(std::ldexp(rate, 65 - f.shift));
    f.reach = static_cast<long long>(std::ldexp(85.0 / q, FX_EXP_UNIT));
    return f;
}

// computed once: 0.2 ms where long double is a software type
inline const FXExpTable& fx_exp_table() {
    static const FXExpTable table = [] {
        FXExpTable t;
        for (int k = 0; k < FX_EXP_K; ++k)
            t.v[k] = static_cast<unsigned long long>(std::ldexp(std::exp2((long double)-k / FX_EXP_K), 63));
        return t;
    }();
    return table;
}

// the exponents the fixed-point forms cover.  q >= 0.333 keeps q d = 85 below FX_FAR.  Above 2 the
// unit of d, of which an error is q times as large, counts for more than FP64's rounding: matrix
// entries against the root of their diagonal entries' product, rms, 8-node mesh, fixed point and FP64:
// q = 1 4.6e-16 / 5.7e-16, 2 2.4e-16 / 2.4e-16, 3 1.8e-16 / 1.5e-16, 8 1.0e-16 / 5.7e-17
inline bool fx_supported(const Model& m) {
    if (m.n != 2) return false;
    if (m.influence == NLGPU_INFLUENCE_FAST_POLYNOMIAL) return true;
    if (m.influence == NLGPU_INFLUENCE_POLYNOMIAL) return m.p >= 0 && m.p % 2 == 0 && m.q >= 0.0 && m.q == std::floor(m.q) && m.q <= 16.0;
    return m.influence == NLGPU_INFLUENCE_EXPONENTIAL && m.p == 2 && m.q >= 0.333 && m.q <= 2.0;
}

}  // namespace nlgpu
