// Influence functions in float-float, shared by the pair assembly and the flux
// post-processing.
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
        const ff dp = ff_ipow(d, m.p / m.n);
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

// float-float covers the continuous influence kinds with an integral power
// p / n and constant conductivity; the rest runs the FP64 kernel
inline bool ff_supported(const Model& m) {
    if (m.n < 1) return false;
    if (m.influence == NLGPU_INFLUENCE_FAST_POLYNOMIAL) return true;
    if (m.influence == NLGPU_INFLUENCE_POLYNOMIAL || m.influence == NLGPU_INFLUENCE_EXPONENTIAL)
        return m.p >= 0 && m.p % m.n == 0;
    return false;
}

}  // namespace nlgpu
