// Values of the conductivity (and capacity) matrices.
//
// Reference: conductivity_matrix_2d::compute (conductivity_matrix_2d.hpp:166-193)
// runs integrator::operator() (integrator.hpp:62-91) for every
// (row node, eL containing it, eNL in neighbours(eL), jNL), recomputing
//   K_ij += (1 - p1) * sum_qL w_qL G_i(qL) . sum_qNL w_qNL phi(x_qL, x_qNL) Lambda(qNL) G_j(qNL)
//         + p1 * [eL == eNL] * sum_q w_q G_i(q) . Lambda(q) G_j(q) / |J(q)|
// (integrate_nonlocal :132-164, integrate_local :106-130) for each entry.
//
// Here the work is organised by element pair.  A CTA owns element eL: the CSR
// segments of its node rows (column numbers and value accumulators) sit in
// shared memory.  Each warp takes one neighbour eNL at a time, stages eNL's
// quadrature data in shared memory and evaluates the pair's whole block once,
// factorised as
//   Phi[qL][qNL] = c_qNL * shape(x_qL, x_qNL)       c_qNL = w_qNL norm (1 - p1) [lambda]
//   H[qL][j]     = sum_qNL Phi[qL][qNL] Lambda G_j(qNL)
//   K[i][j]      = sum_qL (w_qL G_i(qL)) . H[qL][j]
// and adds every entry the reference keeps (matrix_separator_base::part) to
// the shared accumulators; BOUND entries go to global memory.  When the
// problem is symmetric (constant conductivity) each unordered pair is
// evaluated once: the CTA of the element with the smaller (first node, number)
// key takes it, and the block's transposed entries -- which the reference
// computes from the swapped pair, the same value mathematically -- go to the
// other element's rows through global atomics (few with a banded numbering).
// When the CTA is done its accumulators are added to the global values.  Rows
// too long for shared memory fall back to global atomics with a binary search.
#include "common.cuh"
#include "ff.cuh"
#include "influence.cuh"
#include "influence_ff.cuh"

#include <cmath>

namespace nlgpu {

namespace {

constexpr int AS_THREADS = 256;
constexpr int AS_WARPS = AS_THREADS / 32;

// What the fixed-point form of the pair blocks (below) depends on over the whole mesh.  An
// element's x and y gradients share an exponent, so the smaller component has fewer bits;
// that matters where an element with |w_x| << |w_y| meets one with |g_x| >> |g_y|, whose
// products are then as large as the others'.  A power of two moved from one component's
// g to its w (ff_shift) leaves every product as it is and evens out what all elements
// have in common (a stretched mesh whose conductivity makes up for it); what remains is the
// loss.  FP64 solves allow 4 bits (58 - 4 against 53), mixed-precision ones 10 (48, as the
// influence values); meshes beyond that, and for fixed-point values coordinates of
// 2^(FX_MAX_EXPONENT + 1) radii, take the FP64 kernel: this form's returns at once and
// leaves a word that the host reads with the assembly's errors.
constexpr int FF_NONE = 1 << 12;   // the four below are the largest difference of exponents + FF_NONE; 0: no element
struct FFRange {
    unsigned long long extent;     // the bits of the largest finite |coordinate| in units of the radii
    int wx, wy, gx, gy;            // of w_x over w_y, w_y over w_x, g_x over g_y, g_y over g_x in an element
};
struct FFGate {
    const FFRange* range;          // null: no condition
    int max_loss;
    bool fixed;                    // fixed-point values
};

__device__ __forceinline__ void ff_losses(const FFRange* r, int& x, int& y) {   // before the shift
    x = r->wx == 0 || r->gy == 0 ? -FF_NONE : min(r->wx, r->gy) - FF_NONE;
    y = r->wy == 0 || r->gx == 0 ? -FF_NONE : min(r->wy, r->gx) - FF_NONE;
}
__device__ __forceinline__ int ff_shift(const FFRange* r) {   // w_x 2^shift, g_x 2^-shift
    int x, y;
    ff_losses(r, x, y);
    return min(256, max(-256, (y - x) >> 1));
}
__device__ __forceinline__ bool ff_in_range(const FFGate& g) {
    int x, y;
    ff_losses(g.range, x, y);
    const int s = ff_shift(g.range);
    return max(x + s, y - s) <= g.max_loss && (!g.fixed || int(g.range->extent >> 52) <= 1023 + FX_MAX_EXPONENT);
}

struct AssembleArgs {
    i64 E;
    i64 e0;                   // first element (the float-float kernel's tuning samples start later)
    const int32_t* elems;
    const double* qcoord;     // [e][q][2]
    const double* jac;        // [e][q]
    const double* deriv;      // [e][i][q][2]
    const i64* noff;
    const int32_t* nlist;
    const int32_t* minnode;
    const uint8_t* is_inner;
    const double* cond_field; // isotropic conductivity per quadrature point, or null
    const i64* in_rp; const int32_t* in_col; double* in_val;
    const i64* bd_rp; const int32_t* bd_col; double* bd_val;
    bool symmetric;
    int cap;                  // accumulator entries in shared memory
    int* error;               // set when an entry is missing from its pattern
    FFGate gate;              // the fixed-point form's range; beyond it error[1] is set and nothing done
};

__device__ __forceinline__ i64 find_col(const int32_t* col, i64 lo, i64 hi, int32_t c) {
    while (lo < hi) {
        const i64 mid = (lo + hi) >> 1;
        if (col[mid] < c) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void add_global(const i64* rp, const int32_t* col, double* val, int32_t r, int32_t c, double v,
                                           int* error) {
    const i64 pos = find_col(col, rp[r], rp[r + 1], c);
    if (pos < rp[r + 1] && col[pos] == c) atomicAdd(val + pos, v);
    else atomicExch(error, 1);
}

template<int NEN, int NQ>
struct PairSmem {
    double qx[NQ], qy[NQ];
    double gx[NEN * NQ], gy[NEN * NQ];
    double phi[NQ * NQ];
    double hx[NQ * NEN], hy[NQ * NEN];
    double c[NQ];             // c_qNL
    int32_t nodes[NEN];
};

template<int NEN, int NQ, int INF, bool SYM>
__global__ void __launch_bounds__(AS_THREADS) k_assemble_pairs(AssembleArgs a, Model m, Basis b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double eqx[NQ], eqy[NQ], egx[NEN * NQ], egy[NEN * NQ], ewx[NEN * NQ], ewy[NEN * NQ], ejac[NQ], elam[NQ];
    __shared__ int32_t enodes[NEN];
    __shared__ i64 row_start[NEN];
    __shared__ int row_len[NEN], row_off[NEN + 1];
    __shared__ int use_smem;

    auto* pairs = reinterpret_cast<PairSmem<NEN, NQ>*>(smem_raw);
    double* acc = reinterpret_cast<double*>(smem_raw + sizeof(PairSmem<NEN, NQ>) * AS_WARPS);
    int32_t* cols = reinterpret_cast<int32_t*>(acc + a.cap);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PairSmem<NEN, NQ>& ps = pairs[warp];
    const double cnl = m.norm * (1.0 - m.p1);
    const bool iso = m.cond_kind == NLGPU_CONDUCTIVITY_ISOTROPIC;

    for (i64 eL = blockIdx.x; eL < a.E; eL += gridDim.x) {
        // ---- element eL: quadrature data, weighted gradients and its node rows
        for (int t = threadIdx.x; t < NEN * NQ; t += AS_THREADS) {
            const double gx = a.deriv[2 * (eL * NEN * NQ + t)], gy = a.deriv[2 * (eL * NEN * NQ + t) + 1];
            egx[t] = gx; egy[t] = gy;
            ewx[t] = b.w[t % NQ] * gx; ewy[t] = b.w[t % NQ] * gy;
        }
        for (int t = threadIdx.x; t < NQ; t += AS_THREADS) {
            eqx[t] = a.qcoord[2 * (eL * NQ + t)];
            eqy[t] = a.qcoord[2 * (eL * NQ + t) + 1];
            ejac[t] = a.jac[eL * NQ + t];
            elam[t] = a.cond_field ? a.cond_field[eL * NQ + t] : m.cond[0];
        }
        if (threadIdx.x < NEN) {
            const int32_t r = a.elems[eL * NEN + threadIdx.x];
            enodes[threadIdx.x] = r;
            row_start[threadIdx.x] = a.in_rp[r];
            row_len[threadIdx.x] = a.is_inner[r] ? int(a.in_rp[r + 1] - a.in_rp[r]) : 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int off = 0;
            for (int i = 0; i < NEN; ++i) { row_off[i] = off; off += row_len[i]; }
            row_off[NEN] = off;
            use_smem = off <= a.cap;
        }
        __syncthreads();
        const bool smem_rows = use_smem;
        if (smem_rows) {
            for (int i = 0; i < NEN; ++i)
                for (int t = threadIdx.x; t < row_len[i]; t += AS_THREADS) {
                    cols[row_off[i] + t] = a.in_col[row_start[i] + t];
                    acc[row_off[i] + t] = 0.0;
                }
        }
        __syncthreads();
        const int32_t key_l = SYM ? a.minnode[eL] : 0;

        // ---- pairs (eL, eNL): one warp each
        const i64 kb = a.noff[eL], ke = a.noff[eL + 1];
        for (i64 k = kb + warp; k < ke; k += AS_WARPS) {
            const int32_t eNL = a.nlist[k];
            if constexpr (SYM) {   // the pair belongs to the element with the smaller key
                const int32_t key_n = a.minnode[eNL];
                if (key_n < key_l || (key_n == key_l && eNL < int32_t(eL))) continue;
            }
            for (int t = lane; t < NEN * NQ; t += 32) {
                ps.gx[t] = a.deriv[2 * (i64(eNL) * NEN * NQ + t)];
                ps.gy[t] = a.deriv[2 * (i64(eNL) * NEN * NQ + t) + 1];
            }
            if (lane < NQ) {
                ps.qx[lane] = a.qcoord[2 * (i64(eNL) * NQ + lane)];
                ps.qy[lane] = a.qcoord[2 * (i64(eNL) * NQ + lane) + 1];
                const double lam = a.cond_field ? a.cond_field[i64(eNL) * NQ + lane] : m.cond[0];
                ps.c[lane] = b.w[lane] * cnl * (iso ? lam : 1.0);
            }
            if (lane < NEN) ps.nodes[lane] = a.elems[i64(eNL) * NEN + lane];
            __syncwarp();
            for (int t = lane; t < NQ * NQ; t += 32) {
                const int qL = t / NQ, qNL = t % NQ;
                ps.phi[t] = ps.c[qNL] * shape<INF>(m, eqx[qL] - ps.qx[qNL], eqy[qL] - ps.qy[qNL]);
            }
            __syncwarp();
            for (int t = lane; t < NQ * NEN; t += 32) {
                const int qL = t / NEN, j = t % NEN;
                double h0 = 0.0, h1 = 0.0;
                #pragma unroll
                for (int qNL = 0; qNL < NQ; ++qNL) {
                    const double f = ps.phi[qL * NQ + qNL];
                    const double gx = ps.gx[j * NQ + qNL], gy = ps.gy[j * NQ + qNL];
                    if (m.cond_kind != NLGPU_CONDUCTIVITY_ANISOTROPIC) { h0 += f * gx; h1 += f * gy; }
                    else { h0 += f * (m.cond[0] * gx + m.cond[2] * gy); h1 += f * (m.cond[2] * gx + m.cond[1] * gy); }
                }
                if (m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC) { h0 *= m.cond[0]; h1 *= m.cond[1]; }
                ps.hx[t] = h0; ps.hy[t] = h1;
            }
            __syncwarp();
            const bool self = eNL == int32_t(eL);
            for (int t = lane; t < NEN * NEN; t += 32) {
                const int i = t / NEN, j = t % NEN;
                const int32_t r = enodes[i], c = ps.nodes[j];
                const bool r_in = a.is_inner[r], c_in = a.is_inner[c];
                // (r, c) from this pair; (c, r) from the swapped pair when it is folded into this one
                const bool fwd_inner = c_in && r_in && (!a.symmetric || r <= c);
                const bool fwd_bound = !c_in && r != c;
                const bool tr = SYM && !self;
                const bool bwd_inner = tr && c_in && r_in && c <= r;
                const bool bwd_bound = tr && !r_in && c != r;
                if (!fwd_inner && !fwd_bound && !bwd_inner && !bwd_bound) continue;
                double v = 0.0;
                #pragma unroll
                for (int qL = 0; qL < NQ; ++qL)
                    v = fma(ewy[i * NQ + qL], ps.hy[qL * NEN + j], fma(ewx[i * NQ + qL], ps.hx[qL * NEN + j], v));
                if (self) {
                    double loc = 0.0;
                    #pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const double ax = egx[i * NQ + q], ay = egy[i * NQ + q];
                        const double bx = egx[j * NQ + q], by = egy[j * NQ + q];
                        double val;
                        if (iso) val = elam[q] * (ax * bx + ay * by);
                        else if (m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC) val = m.cond[0] * ax * bx + m.cond[1] * ay * by;
                        else val = ax * (m.cond[0] * bx + m.cond[2] * by) + ay * (m.cond[2] * bx + m.cond[1] * by);
                        loc += b.w[q] * val / ejac[q];
                    }
                    v += m.p1 * loc;
                }
                if (fwd_inner) {
                    if (smem_rows) {
                        const i64 pos = find_col(cols, row_off[i], row_off[i + 1], c);
                        if (pos < row_off[i + 1] && cols[pos] == c) atomicAdd(acc + pos, v);
                        else atomicExch(a.error, 1);
                    } else {
                        add_global(a.in_rp, a.in_col, a.in_val, r, c, v, a.error);
                    }
                }
                if (fwd_bound) add_global(a.bd_rp, a.bd_col, a.bd_val, r, c, v, a.error);
                if (bwd_inner) add_global(a.in_rp, a.in_col, a.in_val, c, r, v, a.error);
                if (bwd_bound) add_global(a.bd_rp, a.bd_col, a.bd_val, c, r, v, a.error);
            }
            __syncwarp();
        }
        __syncthreads();
        if (smem_rows)
            for (int i = 0; i < NEN; ++i)
                for (int t = threadIdx.x; t < row_len[i]; t += AS_THREADS) {
                    const double v = acc[row_off[i] + t];
                    if (v != 0.0) atomicAdd(a.in_val + row_start[i] + t, v);
                }
        __syncthreads();
    }
}

// ---------------------------------------------------- float-float, fixed point
// The same pair blocks off the FP64 pipe: the influence values in fixed point
// (influence_ff.cuh, 60 bits) or float-float (ff.cuh, about 48 bits, for exponents that
// the former does not cover), both contractions in fixed point on the integer
// multipliers.  Both elements' gradients carry one exponent each (FFRange says where that
// is not enough) and the influence values one per pair, so that the entries at the
// horizon's edge, where they are small, keep their digits; a number is up to 61 bits in two signed
// words (hi 2^30 + lo), a multiply-add three 32 x 32 + 64-bit ones (hi hi, and
// hi lo + lo hi into a second accumulator; lo lo lies below the result's last bit),
// and the sums are exact.  Against the compensated float-float dot product (12
// FP32 instructions a term, errors of order 2^-48) that is a quarter of the
// instructions and half the pipe time (64 lanes a clock against 128); the gradients'
// 58 bits leave an error below FP64's (against extended precision and the root of the
// diagonal entries' product, rms, 12 x 14 bilinear and 6 x 8 8-node meshes: exponential
// 3.3e-16 and 9.7e-16 for the FP64 kernel's 5.2e-16 and 1.3e-15, 1 - d 1.2e-16 and 3.8e-16 for
// 1.8e-16 and 4.9e-16).
// Weights, Lambda and the constant factors are folded into the two staged copies
// of the gradients (k_ff_stage), the pairs this element owns are listed once per
// element, and a pair whose influence is zero everywhere ends there.
// 8-node 300 x 300 elements, exponential influence: 116.9 ms with the compensated
// dots, 76.5 with fixed point; 4-node 200 x 200: 7.4 and 4.2; 17.9 million listed
// 8-node pairs: 24.1 and 13.2 G instructions, 28.0 and 18.6 ms.  What bounds it
// now: issue, with no part that stands out (the scatter 15 %, the influence values
// 20, H 4, K 10, a CTA's rows 7); a column bitmap instead of the scatter's binary
// search costs as much as it saves.
// 16 or 32 warps per CTA (the FP64 kernel's 8 leave the pipes idle), chosen per
// problem by timing both on a sample of elements; a warp takes one 8-node pair or
// two 4-node pairs at a time (16 lanes cover a 4 x 4 block).

constexpr int FF_BAD = 1 << 20;   // exponent of an element with a non-finite value
constexpr int FF_LIST = 1024;     // candidates listed at a time

struct FFArgs {
    const int4* qcoord;     // [e][q]: coordinates in units of the radii, (x/r0 .h, .l, y/r1 .h, .l) or fixed point
    const FFRange* range;
    const int2* g;          // [e][q][x, y][j]: w_q norm (1 - p1) [lambda_q] Lambda G_j 2^(57 - exps.x) as hi 2^30 + lo
    const int4* w;          // [e][i][q]: w_q G_i 2^(57 - exps.y), (x hi, lo, y hi, lo)
    const int2* exps;       // [e]: the exponents of the largest |g| and |w|
    const int32_t* nodes;   // [e][j]: the node, its complement where it is not inner
    // the exponential's tables, copied to shared memory by each CTA
    FFExpTable ff_table;    // exp(k / 256)
    FXExpTable fx_table;    // 2^(-k / 256)
    FXExp fx_exp;
};

// the conductivity times a gradient, as the pair blocks use it
__device__ __forceinline__ double2 ff_flux(const Model& m, double gx, double gy) {
    if (m.cond_kind == NLGPU_CONDUCTIVITY_ISOTROPIC) return make_double2(gx, gy);
    if (m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC) return make_double2(m.cond[0] * gx, m.cond[1] * gy);
    return make_double2(m.cond[0] * gx + m.cond[2] * gy, m.cond[2] * gx + m.cond[1] * gy);
}

// One warp per element, on exponents: with an isotropic or orthotropic Lambda those of
// g are those of w moved by the two conductivities' (to one bit), so that the loops hold no
// FP64 operation.
__global__ void k_ff_range(i64 E, int nen, int nq, const double* __restrict__ deriv, const double* __restrict__ qcoord, Model m,
                           FFRange* __restrict__ range) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool aniso = m.cond_kind != NLGPU_CONDUCTIVITY_ISOTROPIC && m.cond_kind != NLGPU_CONDUCTIVITY_ORTHOTROPIC;
    auto high = [](double x) { return unsigned(__double2hiint(x)) & 0x7fffffffu; };
    auto exponent = [](unsigned high) { return high ? int(high >> 20) : -1500; };   // zero counts as far below
    const unsigned lx = m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC ? high(m.cond[0]) : 1u;
    const unsigned ly = m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC ? high(m.cond[1]) : 1u;
    const int lambda = exponent(lx) - exponent(ly);
    unsigned long long at = 0;   // the largest finite |coordinate| of the lane's axis, as bits
    int wx = 0, wy = 0, gx = 0, gy = 0;
    for (i64 e = (blockIdx.x * i64(blockDim.x) + threadIdx.x) / 32; e < E; e += i64(gridDim.x) * blockDim.x / 32) {
        for (int t = lane; t < 2 * nq; t += 32) {
            const unsigned long long x = (unsigned long long)__double_as_longlong(qcoord[2 * e * nq + t]) << 1 >> 1;
            if (x < 0x7ffull << 52) at = max(at, x);
        }
        unsigned top[4] = {0u, 0u, 0u, 0u};   // high words of the largest |w_x|, |w_y|, |g_x|, |g_y|
        for (int t = lane; t < nen * nq; t += 32) {
            const double2 d = reinterpret_cast<const double2*>(deriv)[e * nen * nq + t];
            top[0] = max(top[0], high(d.x)); top[1] = max(top[1], high(d.y));
            if (aniso) {
                const double2 g = ff_flux(m, d.x, d.y);
                top[2] = max(top[2], high(g.x)); top[3] = max(top[3], high(g.y));
            }
        }
        top[0] = __reduce_max_sync(full, top[0]);
        top[1] = __reduce_max_sync(full, top[1]);
        if (aniso) {
            top[2] = __reduce_max_sync(full, top[2]);
            top[3] = __reduce_max_sync(full, top[3]);
        }
        auto take = [](int d, int& ab, int& ba) {
            ab = max(ab, FF_NONE + d);
            ba = max(ba, FF_NONE - d);
        };
        const int d = exponent(top[0]) - exponent(top[1]);
        if (max(top[0], top[1]) >= 0x7ff00000u || (top[0] | top[1]) == 0u) continue;
        take(d, wx, wy);
        if (!aniso && lx && ly) take(d + lambda, gx, gy);
        else if (!aniso && (lx || ly)) take(lx && top[0] ? 3000 : ly && top[1] ? -3000 : 0, gx, gy);
        else if (aniso && max(top[2], top[3]) < 0x7ff00000u && (top[2] | top[3])) take(exponent(top[2]) - exponent(top[3]), gx, gy);
    }
    // the lanes of one axis, in units of its radius (2 nq and 32 are even: a lane keeps its axis)
    for (int o = 16; o > 1; o >>= 1) at = max(at, __shfl_xor_sync(full, at, o));
    unsigned long long extent =
        (unsigned long long)__double_as_longlong(fabs(__longlong_as_double((long long)at) * m.inv_r[lane & 1]));
    extent = max(extent, __shfl_xor_sync(full, extent, 1));
    // a CTA's first (200 x 200 elements, every warp's atomics on five words: 40 us)
    __shared__ FFRange cta;
    if (threadIdx.x == 0) cta = FFRange{0ull, 0, 0, 0, 0};
    __syncthreads();
    auto raise = [&](FFRange* r, unsigned long long x, int a, int b, int c, int d) {
        atomicMax(&r->extent, x);
        atomicMax(&r->wx, a); atomicMax(&r->wy, b); atomicMax(&r->gx, c); atomicMax(&r->gy, d);
    };
    if (lane == 0) raise(&cta, extent, wx, wy, gx, gy);
    __syncthreads();
    if (threadIdx.x == 0) raise(range, cta.extent, cta.wx, cta.wy, cta.gx, cta.gy);
}

// x 2^(57 - e), |x| < 2^(e + 1), by integer operations (the FP64 pipe's conversions made the staging 0.19 ms
// on 200 x 200 elements)
__device__ __forceinline__ int2 ff_fixed(double x, int e) {
    const long long b = __double_as_longlong(x);
    const int ex = int(b >> 52 & 0x7ff);
    const long long m = (b & 0xfffffffffffffll) | (1ll << 52);
    const int s = ex - 1018 - e;
    const long long z = ex == 0 || s < -53 ? 0 : s >= 0 ? m << min(s, 5) : (m + (1ll << (-s - 1))) >> -s;
    return fx_split(b < 0 ? -z : z);
}

// one warp per element
__global__ void k_ff_stage(i64 E, int nen, int nq, const int32_t* __restrict__ elems, const uint8_t* __restrict__ is_inner,
                           const double* __restrict__ deriv, const double* __restrict__ qcoord,
                           const double* __restrict__ cond_field, Model m, Basis b,
                           const FFRange* __restrict__ range, bool fixed, int4* __restrict__ qff,
                           int2* __restrict__ g, int4* __restrict__ w, int2* __restrict__ exps,
                           int32_t* __restrict__ nodes) {
    const double cnl = m.norm * (1.0 - m.p1);
    const bool iso = m.cond_kind == NLGPU_CONDUCTIVITY_ISOTROPIC;
    const int lane = threadIdx.x & 31;
    const int shift = ff_shift(range);
    const double up = scalbn(1.0, shift), down = scalbn(1.0, -shift);
    auto values = [&](i64 e, int t, double (&v)[4]) {   // (Lambda G scaled, w G) of (i, q) = (t / nq, t % nq)
        const double gx = deriv[2 * (e * nen * nq + t)], gy = deriv[2 * (e * nen * nq + t) + 1];
        const int q = t % nq;
        const double lam = cond_field ? cond_field[e * nq + q] : m.cond[0];
        const double c = b.w[q] * cnl * (iso ? lam : 1.0);
        const double2 g = ff_flux(m, gx, gy);
        v[0] = c * g.x * down; v[1] = c * g.y;
        v[2] = b.w[q] * gx * up; v[3] = b.w[q] * gy;
    };
    for (i64 e = (blockIdx.x * i64(blockDim.x) + threadIdx.x) / 32; e < E; e += i64(gridDim.x) * blockDim.x / 32) {
        // the high words of the largest magnitudes
        unsigned mg = 0u, mw = 0u;
        for (int t = lane; t < nen * nq; t += 32) {
            double v[4];
            values(e, t, v);
            auto high = [](double x) { return unsigned(__double2hiint(x)) & 0x7fffffffu; };
            mg = max(mg, max(high(v[0]), high(v[1])));
            mw = max(mw, max(high(v[2]), high(v[3])));
        }
        mg = __reduce_max_sync(0xffffffffu, mg);
        mw = __reduce_max_sync(0xffffffffu, mw);
        bool bad_g = mg >= 0x7ff00000u, bad_w = mw >= 0x7ff00000u;
        if (lane < nq) {
            const double x = qcoord[2 * (e * nq + lane)], y = qcoord[2 * (e * nq + lane) + 1];
            if (fixed) {   // fixed point has no NaN: the element's blocks become one
                const bool finite = isfinite(x * m.inv_r[0]) && isfinite(y * m.inv_r[1]);
                const int ex = fx_exponent(&range->extent);
                const int2 fx = fx_coordinate(finite ? x : 0.0, m.inv_r[0], ex);
                const int2 fy = fx_coordinate(finite ? y : 0.0, m.inv_r[1], ex);
                qff[e * nq + lane] = make_int4(fx.x, fx.y, fy.x, fy.y);
                bad_g = bad_g || !finite;
                bad_w = bad_w || !finite;
            } else {
                const ff fx = ff_from(x * m.inv_r[0]), fy = ff_from(y * m.inv_r[1]);
                qff[e * nq + lane] = make_int4(__float_as_int(fx.h), __float_as_int(fx.l), __float_as_int(fy.h),
                                               __float_as_int(fy.l));
            }
        }
        bad_g = __any_sync(0xffffffffu, bad_g);
        bad_w = __any_sync(0xffffffffu, bad_w);
        const int eg = bad_g ? FF_BAD : mg ? int(mg >> 20) - 1023 : 0, ew = bad_w ? FF_BAD : mw ? int(mw >> 20) - 1023 : 0;
        if (lane == 0) exps[e] = make_int2(eg, ew);
        for (int t = lane; t < nen * nq; t += 32) {
            double v[4];
            values(e, t, v);
            if (bad_g) v[0] = v[1] = 0.0;
            if (bad_w) v[2] = v[3] = 0.0;
            const int i = t / nq, q = t % nq;
            g[((e * nq + q) * 2 + 0) * nen + i] = ff_fixed(v[0], eg);
            g[((e * nq + q) * 2 + 1) * nen + i] = ff_fixed(v[1], eg);
            const int2 x = ff_fixed(v[2], ew), y = ff_fixed(v[3], ew);
            w[e * nen * nq + t] = make_int4(x.x, x.y, y.x, y.y);
        }
        if (lane < nen) {
            const int32_t r = elems[e * nen + lane];
            nodes[e * nen + lane] = is_inner[r] ? r : ~r;
        }
    }
}

// one pair's data
template<int NEN, int NQ>
struct PairFF {
    static constexpr int PS = (NQ + 1) / 2 * 2;   // influence values per row, padded to whole 16 bytes
    int4 q[NQ];           // eNL's points
    int2 phi[NQ * PS];    // shape(qL, qNL) 2^(60 - e_p), e_p an exponent of the pair's largest
    int4 h[NQ * NEN];     // H(qL, j): (x hi, lo, y hi, lo)
    int32_t nodes[NEN];
};

template<int NEN, int NQ, int INF, bool SYM, int WARPS, bool FIX>
__global__ void __launch_bounds__(WARPS * 32) k_assemble_pairs_ff(AssembleArgs a, FFArgs f, Model m, Basis b) {
    constexpr int THREADS = WARPS * 32;
    constexpr int LANES = NQ * NQ <= 16 ? 16 : 32, GROUPS = 32 / LANES;   // lanes per pair, pairs per warp
    constexpr int PR = (NQ * NQ + LANES - 1) / LANES;                     // influence values per lane
    constexpr int HL = 2 * NEN, HG = LANES / HL;                          // H: one lane per (direction, j), HG rows at a time
    constexpr int OUT = NEN * NEN / LANES;                                // block entries per lane
    constexpr int PS = PairFF<NEN, NQ>::PS;
    static_assert(NEN * NEN % LANES == 0 && LANES % HL == 0 && NEN % 4 == 0 && NEN * NEN / 4 / OUT * 4 == LANES, "lane layout");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr bool EXP = INF == NLGPU_INFLUENCE_EXPONENTIAL;
    __shared__ int4 eq[NQ];
    __shared__ int4 ew[NEN * NQ];
    __shared__ double egx[NEN * NQ], egy[NEN * NQ], ejac[NQ], elam[NQ];   // the self term stays FP64
    __shared__ int32_t enodes[NEN], einner[NEN];   // eL's nodes and whether each is inner
    __shared__ i64 row_start[NEN];
    __shared__ int row_len[NEN], row_off[NEN + 1];
    __shared__ int use_smem, listed;
    __shared__ int32_t list[FF_LIST];
    __shared__ ff etab[EXP && !FIX ? 2 * FF_EXP_K + 1 : 1];
    __shared__ unsigned long long xtab[EXP && FIX ? FX_EXP_K : 1];
    if constexpr (EXP && !FIX)
        for (int t = threadIdx.x; t < 2 * FF_EXP_K + 1; t += blockDim.x) etab[t] = ff{f.ff_table.v[t].x, f.ff_table.v[t].y};
    if constexpr (EXP && FIX)
        for (int t = threadIdx.x; t < FX_EXP_K; t += blockDim.x) xtab[t] = f.fx_table.v[t];
    if (!ff_in_range(a.gate)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) a.error[1] = 1;
        return;
    }
    const int ex = FIX ? fx_exponent(&f.range->extent) : 0;

    auto* pairs = reinterpret_cast<PairFF<NEN, NQ>*>(smem_raw);
    double* acc = reinterpret_cast<double*>(smem_raw + sizeof(PairFF<NEN, NQ>) * WARPS * GROUPS);
    int32_t* cols = reinterpret_cast<int32_t*>(acc + a.cap);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = lane / LANES, gl = lane % LANES;
    PairFF<NEN, NQ>& ps = pairs[warp * GROUPS + group];
    const bool iso = m.cond_kind == NLGPU_CONDUCTIVITY_ISOTROPIC;
    const ff qf = ff_from(m.q);

    for (i64 eL = a.e0 + blockIdx.x; eL < a.E; eL += gridDim.x) {
        // ---- element eL: quadrature data, weighted gradients and its node rows
        for (int t = threadIdx.x; t < NEN * NQ; t += THREADS) {
            egx[t] = a.deriv[2 * (eL * NEN * NQ + t)];
            egy[t] = a.deriv[2 * (eL * NEN * NQ + t) + 1];
            ew[t] = f.w[eL * NEN * NQ + t];
        }
        for (int t = threadIdx.x; t < NQ; t += THREADS) {
            eq[t] = f.qcoord[eL * NQ + t];
            ejac[t] = a.jac[eL * NQ + t];
            elam[t] = a.cond_field ? a.cond_field[eL * NQ + t] : m.cond[0];
        }
        if (threadIdx.x < NEN) {
            const int32_t r = a.elems[eL * NEN + threadIdx.x];
            const bool r_in = a.is_inner[r];
            enodes[threadIdx.x] = r;
            einner[threadIdx.x] = r_in;
            row_start[threadIdx.x] = a.in_rp[r];
            row_len[threadIdx.x] = r_in ? int(a.in_rp[r + 1] - a.in_rp[r]) : 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int off = 0;
            for (int i = 0; i < NEN; ++i) { row_off[i] = off; off += row_len[i]; }
            row_off[NEN] = off;
            use_smem = off <= a.cap;
            listed = 0;
        }
        __syncthreads();
        const bool smem_rows = use_smem;
        if (smem_rows) {
            for (int i = 0; i < NEN; ++i)
                for (int t = threadIdx.x; t < row_len[i]; t += THREADS) {
                    cols[row_off[i] + t] = a.in_col[row_start[i] + t];
                    acc[row_off[i] + t] = 0.0;
                }
        }
        const int32_t key_l = SYM ? a.minnode[eL] : 0;
        const int e_w = f.exps[eL].y;

        const i64 kb = a.noff[eL], ke = a.noff[eL + 1];
        for (i64 k0 = kb; k0 < ke; k0 += FF_LIST) {
            // ---- the pairs of this element: with unordered pairs, those whose key is not the smaller one's
            for (int t = warp * 32; t < FF_LIST && k0 + t < ke; t += THREADS) {
                const i64 k = k0 + t + lane;
                int32_t eNL = -1;
                bool own = k < ke;
                if (own) {
                    eNL = a.nlist[k];
                    if constexpr (SYM) {   // the pair belongs to the element with the smaller key
                        const int32_t key_n = a.minnode[eNL];
                        own = !(key_n < key_l || (key_n == key_l && eNL < int32_t(eL)));
                    }
                }
                const unsigned votes = __ballot_sync(0xffffffffu, own);
                int at = 0;
                if (lane == 0 && votes) at = atomicAdd(&listed, __popc(votes));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (own) list[at + __popc(votes & ((1u << lane) - 1u))] = eNL;
            }
            __syncthreads();
            const int count = listed;
            // ---- one group of lanes each
            for (int n0 = warp * GROUPS; n0 < count; n0 += WARPS * GROUPS) {
                bool active = n0 + group < count;
                const int32_t eNL = list[min(n0 + group, count - 1)];
                // eNL's gradients of this lane's (direction, j): used after the influence values
                int2 g[NQ];
#pragma unroll
                for (int q = 0; q < NQ; ++q) g[q] = f.g[(i64(eNL) * NQ + q) * HL + gl % HL];
                const int e_g = f.exps[eNL].x;
                if (gl < NQ) ps.q[gl] = f.qcoord[i64(eNL) * NQ + gl];
                if (gl < NEN) ps.nodes[gl] = f.nodes[i64(eNL) * NEN + gl];
                __syncwarp();
                const bool self = eNL == int32_t(eL);
                const bool bad = e_w + e_g >= FF_BAD / 2;
                int e_p = 0;
                bool finite = !bad;
                if constexpr (FIX) {
                    long long v[PR];
                    if constexpr (INF != NLGPU_INFLUENCE_FAST_POLYNOMIAL) {
                        int mv[PR], smallest = FX_EXP_ZERO;
#pragma unroll
                        for (int rnd = 0; rnd < PR; ++rnd) {
                            const int t = min(gl + LANES * rnd, NQ * NQ - 1);
                            const FXValue x = fx_shape<INF>(m, eq[t / NQ], ps.q[t % NQ], ex, f.fx_exp, xtab);
                            v[rnd] = (long long)(x.v >> 3);
                            mv[rnd] = x.m;
                            smallest = min(smallest, mv[rnd]);
                        }
#pragma unroll
                        for (int o = LANES / 2; o > 0; o >>= 1) smallest = min(smallest, __shfl_xor_sync(0xffffffffu, smallest, o));
                        active = active && (smallest != FX_EXP_ZERO || self || bad);
                        if (smallest != FX_EXP_ZERO) e_p = -smallest;
#pragma unroll
                        for (int rnd = 0; rnd < PR; ++rnd) v[rnd] >>= min(mv[rnd] - smallest, 63);
                    } else {
                        unsigned top = 0;   // the values' bits above 2^32, one more where there are none
#pragma unroll
                        for (int rnd = 0; rnd < PR; ++rnd) {
                            const int t = min(gl + LANES * rnd, NQ * NQ - 1);
                            const long long d = fx_distance<60>(eq[t / NQ], ps.q[t % NQ], ex);
                            v[rnd] = d < FX_ONE ? FX_ONE - d : 0;
                            top = max(top, unsigned(v[rnd] >> 32) | unsigned(v[rnd] != 0));
                        }
#pragma unroll
                        for (int o = LANES / 2; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
                        active = active && (top != 0 || self || bad);
                        // a pair at the horizon's edge: its small values moved up
                        const int s = max(__clz(int(top)) - 4, 0);
                        e_p = -s;
#pragma unroll
                        for (int rnd = 0; rnd < PR; ++rnd) v[rnd] <<= s;
                    }
                    if (!__any_sync(0xffffffffu, active)) continue;
#pragma unroll
                    for (int rnd = 0; rnd < PR; ++rnd) {
                        const int t = gl + LANES * rnd;
                        if (PR * LANES == NQ * NQ || t < NQ * NQ)
                            ps.phi[t / NQ * PS + t % NQ] = fx_split(v[rnd]);
                    }
                } else {
                    ff v[PR];
                    unsigned largest = 0;
#pragma unroll
                    for (int rnd = 0; rnd < PR; ++rnd) {
                        const int t = min(gl + LANES * rnd, NQ * NQ - 1);
                        const int4 xl = eq[t / NQ], xn = ps.q[t % NQ];
                        auto coord = [](int h, int l) { return ff{__int_as_float(h), __int_as_float(l)}; };
                        v[rnd] = shape_ff<INF>(m, ff_sub(coord(xl.x, xl.y), coord(xn.x, xn.y)),
                                               ff_sub(coord(xl.z, xl.w), coord(xn.z, xn.w)), qf, etab);
                        largest = max(largest, __float_as_uint(v[rnd].h) & 0x7fffffffu);
                    }
#pragma unroll
                    for (int o = LANES / 2; o > 0; o >>= 1) largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, o));
                    active = active && (largest != 0 || self || bad);
                    if (!__any_sync(0xffffffffu, active)) continue;
                    finite = finite && largest < 0x7f800000u;
                    const int e = max(int(largest >> 23) - 127, -100);
                    e_p = e + 7;
                    const float up = __int_as_float((127 + 23 - e) << 23);
#pragma unroll
                    for (int rnd = 0; rnd < PR; ++rnd) {
                        const int t = gl + LANES * rnd;
                        const float s = __fmul_rn(v[rnd].h, up);
                        const int hi = __float2int_rn(s);
                        const float rest = __fmaf_rn(v[rnd].l, up, __fsub_rn(s, __int2float_rn(hi)));
                        const int lo = __float2int_rn(__fmul_rn(rest, 1073741824.0f));   // 2^30
                        if (PR * LANES == NQ * NQ || t < NQ * NQ) ps.phi[t / NQ * PS + t % NQ] = make_int2(hi, lo);
                    }
                }
                __syncwarp();
                // H(qL, j) = sum_qNL shape G: unit 2^(e_p + e_g - 56)
#pragma unroll 1
                for (int qL = gl / HL; qL < NQ; qL += HG) {
                    long long s0 = 0, s1 = (1ll << 30) + (1 << 29);   // the two shifts below round
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const int2 p = ps.phi[qL * PS + q];
                        s0 += (long long)p.x * g[q].x;
                        s1 += (long long)p.x * g[q].y;
                        s1 += (long long)p.y * g[q].x;
                    }
                    const long long h = (s0 + (s1 >> 30)) >> 1;   // |h| < 2^60.4
                    const int lo = int(h), hi = int(h >> 32) + (lo < 0 ? 1 : 0);
                    // the low word to 30 bits, so that both cross products below have one unit
                    reinterpret_cast<int2*>(ps.h)[(qL * NEN + gl % NEN) * 2 + gl % HL / NEN] = make_int2(hi, ((lo >> 1) + 1) >> 1);
                }
                __syncwarp();
                // K(i, j) = sum_qL (w G_i) . H(qL, j): unit 2^(e_w + e_g + e_p - 51)
                const int i = gl >> 2, j0 = gl & 3;
                long long s0[OUT], s1[OUT];
#pragma unroll
                for (int o = 0; o < OUT; ++o) { s0[o] = 0; s1[o] = 1 << 29; }
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    const int4 w = ew[i * NQ + q];
#pragma unroll
                    for (int o = 0; o < OUT; ++o) {
                        const int4 h = ps.h[q * NEN + j0 + 4 * o];
                        s0[o] += (long long)w.x * h.x;
                        s0[o] += (long long)w.z * h.z;
                        s1[o] += (long long)w.x * h.y;
                        s1[o] += (long long)w.y * h.x;
                        s1[o] += (long long)w.z * h.w;
                        s1[o] += (long long)w.w * h.z;
                    }
                }
                const int e_k = e_w + e_g + e_p - 51;
                double unit = __hiloint2double((1023 + e_k) << 20, 0);
                if (!finite || abs(e_k) > 1000)   // a non-finite factor, or far out of range
                    unit = finite ? scalbn(1.0, e_k) : nan("");
                const int32_t r = enodes[i];
                const bool r_in = einner[i] != 0;
#pragma unroll
                for (int o = 0; o < OUT; ++o) {
                    const int j = j0 + 4 * o;
                    const int32_t cn = ps.nodes[j], c = cn < 0 ? ~cn : cn;
                    const bool c_in = cn >= 0;
                    const bool fwd_inner = active && c_in && r_in && (!a.symmetric || r <= c);
                    const bool fwd_bound = active && !c_in && r != c;
                    const bool tr = SYM && active && !self;
                    const bool bwd_inner = tr && c_in && r_in && c <= r;
                    const bool bwd_bound = tr && !r_in && c != r;
                    double val = __ll2double_rn(s0[o] + (s1[o] >> 30)) * unit;
                    if (self) {
                        double loc = 0.0;
#pragma unroll 1
                        for (int q = 0; q < NQ; ++q) {
                            const double ax = egx[i * NQ + q], ay = egy[i * NQ + q];
                            const double bx = egx[j * NQ + q], by = egy[j * NQ + q];
                            double u;
                            if (iso) u = elam[q] * (ax * bx + ay * by);
                            else if (m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC) u = m.cond[0] * ax * bx + m.cond[1] * ay * by;
                            else u = ax * (m.cond[0] * bx + m.cond[2] * by) + ay * (m.cond[2] * bx + m.cond[1] * by);
                            loc += b.w[q] * u / ejac[q];
                        }
                        val += m.p1 * loc;
                    }
                    if (fwd_inner) {
                        if (smem_rows) {
                            int lo = row_off[i], n = row_len[i];
                            while (n > 1) {   // the last column <= c
                                const int half = n >> 1;
                                if (cols[lo + half] <= c) lo += half;
                                n -= half;
                            }
                            if (n && cols[lo] == c) atomicAdd(acc + lo, val);
                            else atomicExch(a.error, 1);
                        } else {
                            add_global(a.in_rp, a.in_col, a.in_val, r, c, val, a.error);
                        }
                    }
                    if (fwd_bound) add_global(a.bd_rp, a.bd_col, a.bd_val, r, c, val, a.error);
                    if (bwd_inner) add_global(a.in_rp, a.in_col, a.in_val, c, r, val, a.error);
                    if (bwd_bound) add_global(a.bd_rp, a.bd_col, a.bd_val, c, r, val, a.error);
                }
                __syncwarp();
            }
            __syncthreads();
            if (threadIdx.x == 0) listed = 0;
            __syncthreads();
        }
        if (smem_rows)
            for (int i = 0; i < NEN; ++i)
                for (int t = threadIdx.x; t < row_len[i]; t += THREADS) {
                    const double v = acc[row_off[i] + t];
                    if (v != 0.0) atomicAdd(a.in_val + row_start[i] + t, v);
                }
        __syncthreads();
    }
}

// Local integrands, one thread per (e, i, j): conductivity
// (integrate_local, conductivity_matrix_2d.hpp:106-130) or capacity
// (integrate_basic_pair, heat_capacity_matrix_2d.hpp:30-37).
__global__ void k_assemble_local(i64 E, int nen, int nq, const int32_t* __restrict__ elems,
                                 const double* __restrict__ jac, const double* __restrict__ deriv,
                                 const uint8_t* __restrict__ is_inner, const double* __restrict__ cond_field,
                                 Model m, Basis b, int integrand, double weight, bool symmetric,
                                 const i64* __restrict__ rp, const int32_t* __restrict__ col, double* __restrict__ val,
                                 const i64* __restrict__ bd_rp, const int32_t* __restrict__ bd_col, double* __restrict__ bd_val) {
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < E * nen * nen; t += i64(gridDim.x) * blockDim.x) {
        const i64 e = t / (nen * nen);
        const int i = int((t / nen) % nen), j = int(t % nen);
        const int32_t r = elems[e * nen + i], c = elems[e * nen + j];
        const bool keep_inner = is_inner[c] && is_inner[r] && (!symmetric || r <= c);
        const bool keep_bound = !is_inner[c] && r != c && bd_rp != nullptr;
        if (!keep_inner && !keep_bound) continue;
        double integral = 0.0;
        for (int q = 0; q < nq; ++q) {
            if (integrand == 1) {
                integral += b.w[q] * b.qN[i * nq + q] * b.qN[j * nq + q] * jac[e * nq + q];
            } else {
                const double* di = deriv + 2 * ((e * nen + i) * nq + q);
                const double* dj = deriv + 2 * ((e * nen + j) * nq + q);
                double v;
                if (m.cond_kind == NLGPU_CONDUCTIVITY_ISOTROPIC)
                    v = (cond_field ? cond_field[e * nq + q] : m.cond[0]) * (di[0] * dj[0] + di[1] * dj[1]);
                else if (m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC) v = m.cond[0] * di[0] * dj[0] + m.cond[1] * di[1] * dj[1];
                else v = di[0] * (m.cond[0] * dj[0] + m.cond[2] * dj[1]) + di[1] * (m.cond[2] * dj[0] + m.cond[1] * dj[1]);
                integral += b.w[q] * v / jac[e * nq + q];
            }
        }
        integral *= weight;
        if (keep_inner) {
            const i64 pos = find_col(col, rp[r], rp[r + 1], c);
            if (pos < rp[r + 1] && col[pos] == c) atomicAdd(val + pos, integral);
        } else {
            const i64 pos = find_col(bd_col, bd_rp[r], bd_rp[r + 1], c);
            if (pos < bd_rp[r + 1] && bd_col[pos] == c) atomicAdd(bd_val + pos, integral);
        }
    }
}

__global__ void k_dirichlet_diagonal(i64 n, const uint8_t* __restrict__ is_inner, const i64* __restrict__ rp,
                                     double* __restrict__ val, double value) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x)
        if (!is_inner[r]) val[rp[r]] = value;
}

__global__ void k_gather_full(i64 nnz, const i64* __restrict__ map, const double* __restrict__ upper,
                              double* __restrict__ full, float* __restrict__ full32) {
    for (i64 k = blockIdx.x * i64(blockDim.x) + threadIdx.x; k < nnz; k += i64(gridDim.x) * blockDim.x) {
        const i64 s = map[k];
        const double v = s >= 0 ? upper[s] : 0.0;
        full[k] = v;
        if (full32) full32[k] = float(v);
    }
}

template<int NEN, int NQ, int INF>
void launch_pairs(Ctx& ctx, const AssembleArgs& a, bool sym) {
    const size_t fixed = sizeof(PairSmem<NEN, NQ>) * AS_WARPS;
    const size_t dyn = fixed + size_t(a.cap) * (sizeof(double) + sizeof(int32_t));
    const unsigned grid = unsigned(std::min<i64>(a.E, 152 * 16));
    if (sym) {
        auto kernel = k_assemble_pairs<NEN, NQ, INF, true>;
        NL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(dyn)));
        NL_LAUNCH(kernel, grid, AS_THREADS, dyn, ctx.stream, a, ctx.model, ctx.basis);
    } else {
        auto kernel = k_assemble_pairs<NEN, NQ, INF, false>;
        NL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(dyn)));
        NL_LAUNCH(kernel, grid, AS_THREADS, dyn, ctx.stream, a, ctx.model, ctx.basis);
    }
}

template<int NEN, int NQ>
void dispatch_influence(Ctx& ctx, const AssembleArgs& a, bool sym) {
    switch (ctx.model.influence) {
    case NLGPU_INFLUENCE_FAST_POLYNOMIAL: launch_pairs<NEN, NQ, NLGPU_INFLUENCE_FAST_POLYNOMIAL>(ctx, a, sym); break;
    case NLGPU_INFLUENCE_POLYNOMIAL: launch_pairs<NEN, NQ, NLGPU_INFLUENCE_POLYNOMIAL>(ctx, a, sym); break;
    case NLGPU_INFLUENCE_EXPONENTIAL: launch_pairs<NEN, NQ, NLGPU_INFLUENCE_EXPONENTIAL>(ctx, a, sym); break;
    default: launch_pairs<NEN, NQ, NLGPU_INFLUENCE_CONSTANT>(ctx, a, sym); break;
    }
}

template<int NEN, int NQ, int INF, int WARPS>
void launch_pairs_ff_w(Ctx& ctx, AssembleArgs a, const FFArgs& f, bool sym) {
    auto kernel = a.gate.fixed ? (sym ? k_assemble_pairs_ff<NEN, NQ, INF, true, WARPS, true>
                                      : k_assemble_pairs_ff<NEN, NQ, INF, false, WARPS, true>)
                               : (sym ? k_assemble_pairs_ff<NEN, NQ, INF, true, WARPS, false>
                                      : k_assemble_pairs_ff<NEN, NQ, INF, false, WARPS, false>);
    // the row accumulators take what shared memory the per-warp blocks leave
    int dev = 0, optin = 0;
    NL_CUDA(cudaGetDevice(&dev));
    NL_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa{};
    NL_CUDA(cudaFuncGetAttributes(&fa, kernel));
    const size_t fixed = sizeof(PairFF<NEN, NQ>) * WARPS * (NQ * NQ <= 16 ? 2 : 1);
    const size_t avail = size_t(optin) - fa.sharedSizeBytes;
    NL_REQUIRE(avail > fixed + 4096, NLGPU_ERR_UNSUPPORTED, "not enough shared memory for the pair assembly");
    a.cap = int((avail - fixed) / 12);
    const size_t dyn = fixed + size_t(a.cap) * (sizeof(double) + sizeof(int32_t));
    const unsigned grid = unsigned(std::max<i64>(1, std::min<i64>(a.E - a.e0, 152 * 16)));
    NL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(dyn)));
    NL_LAUNCH(kernel, grid, WARPS * 32, dyn, ctx.stream, a, f, ctx.model, ctx.basis);
}

// Warps per CTA: forced by NLGPU_OPTION_ASSEMBLY_WARPS, else tuned once per
// (element type, influence kind, pair mode) and context by timing both forms
// on the same sample of elements from the middle of the mesh, three per SM (their
// contributions are cleared afterwards: the matrices are zeroed again).
template<int NEN, int NQ, int INF>
void launch_pairs_ff(Ctx& ctx, AssembleArgs a, const FFArgs& f, bool sym) {
    int warps = ctx.ff_warps_option;
    // 32 was the choice on every workload measured; below this the four samples (12 elements an SM, a
    // fifth of the assembly at the limit) and the clearing of the matrices cost more than a choice gives
    if (warps == 0 && a.E < 152 * 64) warps = 32;
    if (warps == 0) {
        const int key = NEN * 1000 + INF * 10 + (sym ? 1 : 0) + (a.gate.fixed ? 2 : 0);
        auto it = ctx.ff_warps_tuned.find(key);
        if (it != ctx.ff_warps_tuned.end()) {
            warps = it->second;
        } else {
            const i64 sample = std::min<i64>(a.E, 152 * 3);
            AssembleArgs s = a;
            s.e0 = (a.E - sample) / 2;
            s.E = s.e0 + sample;
            double ms[2] = {0.0, 0.0};
            cudaEvent_t ev[2] = {};
            NL_CUDA(cudaEventCreate(&ev[0]));
            NL_CUDA(cudaEventCreate(&ev[1]));
            for (int rep = 0; rep < 2; ++rep)   // the first round warms up
                for (int v = 0; v < 2; ++v) {
                    NL_CUDA(cudaEventRecord(ev[0], ctx.stream));
                    if (v == 0) launch_pairs_ff_w<NEN, NQ, INF, 16>(ctx, s, f, sym);
                    else launch_pairs_ff_w<NEN, NQ, INF, 32>(ctx, s, f, sym);
                    NL_CUDA(cudaEventRecord(ev[1], ctx.stream));
                    NL_CUDA(cudaEventSynchronize(ev[1]));
                    float t = 0.0f;
                    NL_CUDA(cudaEventElapsedTime(&t, ev[0], ev[1]));
                    ms[v] = double(t);
                }
            cudaEventDestroy(ev[0]);
            cudaEventDestroy(ev[1]);
            ctx.inner.val.zero(ctx.stream);
            ctx.bound.val.zero(ctx.stream);
            warps = ms[1] < ms[0] ? 32 : 16;
            ctx.ff_warps_tuned[key] = warps;
            ctx.ff_tune_ms[0] = ms[0];
            ctx.ff_tune_ms[1] = ms[1];
        }
    }
    ctx.ff_warps_used = warps;
    if (warps == 32) launch_pairs_ff_w<NEN, NQ, INF, 32>(ctx, a, f, sym);
    else launch_pairs_ff_w<NEN, NQ, INF, 16>(ctx, a, f, sym);
}

template<int NEN, int NQ>
void dispatch_influence_ff(Ctx& ctx, const AssembleArgs& a, const FFArgs& f, bool sym) {
    // the polynomial 1 - d is the fast one
    const bool linear = a.gate.fixed && ctx.model.influence == NLGPU_INFLUENCE_POLYNOMIAL && ctx.model.p == 2 && ctx.model.q == 1.0;
    switch (linear ? NLGPU_INFLUENCE_FAST_POLYNOMIAL : ctx.model.influence) {
    case NLGPU_INFLUENCE_FAST_POLYNOMIAL: launch_pairs_ff<NEN, NQ, NLGPU_INFLUENCE_FAST_POLYNOMIAL>(ctx, a, f, sym); break;
    case NLGPU_INFLUENCE_POLYNOMIAL: launch_pairs_ff<NEN, NQ, NLGPU_INFLUENCE_POLYNOMIAL>(ctx, a, f, sym); break;
    default: launch_pairs_ff<NEN, NQ, NLGPU_INFLUENCE_EXPONENTIAL>(ctx, a, f, sym); break;
    }
}

}  // namespace

// Assembles p1*K_local + (1-p1)*K_nonlocal (or p1*K_local for a local model)
// into ctx.inner / ctx.bound, whose patterns are already built.
void assemble_full(Ctx& ctx) {
    ctx.inner.val.zero(ctx.stream);
    ctx.bound.val.zero(ctx.stream);
    const Model& m = ctx.model;
    if (!m.nonlocal()) {
        assemble_local(ctx, ctx.inner, m.p1, 0);
        return;
    }
    AssembleArgs a{};
    a.E = ctx.n_elems; a.elems = ctx.elems.p; a.qcoord = ctx.qcoord.p; a.jac = ctx.jac.p; a.deriv = ctx.deriv.p;
    a.noff = ctx.noff.p; a.nlist = ctx.nlist.p; a.minnode = ctx.elem_minnode.p; a.is_inner = ctx.is_inner.p;
    a.cond_field = ctx.cond_field.n ? ctx.cond_field.p : nullptr;
    a.in_rp = ctx.inner.rowptr.p; a.in_col = ctx.inner.col.p; a.in_val = ctx.inner.val.p;
    a.bd_rp = ctx.bound.rowptr.p; a.bd_col = ctx.bound.col.p; a.bd_val = ctx.bound.val.p;
    a.symmetric = ctx.symmetric;
    dbuf<int> err;
    err.resize(2);   // [an entry outside the pattern, beyond the fixed-point form's range]
    err.zero(ctx.stream);
    a.error = err.p;
    dbuf<FFRange> range;
    // unordered pairs need a symmetric influence and constant conductivity
    const bool sym = ctx.symmetric && !ctx.cond_field.n && !ctx.ordered_pairs;
    // The pair blocks in fixed point: the FP64 kernel's accuracy at a quarter of its
    // time (71 x 53 8-node elements, polynomial: 3.73 and 0.93 ms), so also for FP64 solves unless
    // that kernel is asked for.  The mixed-precision form takes the exponential in
    // float-float, 4 % faster (150 x 150 8-node: 18.6 against 19.3 ms) and accurate
    // enough for it; polynomials are as fast in fixed point (16.3 and 16.0).
    const bool fx = fx_supported(ctx.model);
    const bool fixed = fx && (ctx.ff_assembly ? ctx.model.influence != NLGPU_INFLUENCE_EXPONENTIAL : ctx.fx_assembly);
    const bool staged = fixed || (ctx.ff_assembly && ff_supported(ctx.model));
    if (staged) {
        const int nen = ctx.basis.nen, nq = ctx.basis.nq;
        ctx.ff_qcoord.reserve(size_t(ctx.n_elems * nq));
        ctx.ff_g.reserve(size_t(ctx.n_elems * nen * nq * 2));
        ctx.ff_w.reserve(size_t(ctx.n_elems * nen * nq));
        ctx.ff_exps.reserve(size_t(ctx.n_elems));
        ctx.ff_nodes.reserve(size_t(ctx.n_elems * nen));
        range.resize(1);
        range.zero(ctx.stream);
        a.gate = {range.p, ctx.ff_assembly ? 10 : 4, fixed};
        NL_LAUNCH(k_ff_range, grid_for(ctx.n_elems * 32, 256, 152 * 4), 256, 0, ctx.stream, ctx.n_elems, nen, nq, ctx.deriv.p,
                  ctx.qcoord.p, ctx.model, range.p);
        NL_LAUNCH(k_ff_stage, grid_for(ctx.n_elems * 32, 256), 256, 0, ctx.stream, ctx.n_elems, nen, nq, ctx.elems.p,
                  ctx.is_inner.p, ctx.deriv.p, ctx.qcoord.p, a.cond_field, ctx.model, ctx.basis, range.p, fixed,
                  ctx.ff_qcoord.p, ctx.ff_g.p, ctx.ff_w.p, ctx.ff_exps.p, ctx.ff_nodes.p);
        FFArgs f{ctx.ff_qcoord.p, range.p, ctx.ff_g.p, ctx.ff_w.p, ctx.ff_exps.p, ctx.ff_nodes.p, {}, {}, {}};
        if (ctx.model.influence == NLGPU_INFLUENCE_EXPONENTIAL && fixed) {
            f.fx_table = fx_exp_table();
            f.fx_exp = fx_exp_setup(ctx.model.q);
        } else if (ctx.model.influence == NLGPU_INFLUENCE_EXPONENTIAL) {
            fill_exp_table(f.ff_table);
        }
        if (nen == 4) dispatch_influence_ff<4, 4>(ctx, a, f, sym);
        else dispatch_influence_ff<8, 9>(ctx, a, f, sym);
    }
    auto in_fp64 = [&] {
        if (ctx.basis.nen == 4) {
            a.cap = int((200 * 1024 - sizeof(PairSmem<4, 4>) * AS_WARPS) / 12);
            dispatch_influence<4, 4>(ctx, a, sym);
        } else {
            a.cap = int((200 * 1024 - sizeof(PairSmem<8, 9>) * AS_WARPS) / 12);
            dispatch_influence<8, 9>(ctx, a, sym);
        }
    };
    int herr[2] = {0, 0};
    auto finish = [&] {
        set_dirichlet_diagonal(ctx, ctx.inner, 1.0);
        err.download(herr, 2, ctx.stream);
        NL_CUDA(cudaStreamSynchronize(ctx.stream));
    };
    if (!staged) in_fp64();
    finish();
    if (herr[1]) {
        in_fp64();
        finish();
    }
    NL_REQUIRE(herr[0] == 0, NLGPU_ERR_STATE, "assembly met an entry outside the sparsity pattern");
}

void assemble_local(Ctx& ctx, Csr& mtx, double weight, int integrand) {
    const int nen = ctx.basis.nen, nq = ctx.basis.nq;
    const i64 work = ctx.n_elems * nen * nen;
    const bool with_bound = &mtx == &ctx.inner;
    NL_LAUNCH(k_assemble_local, grid_for(work, 256), 256, 0, ctx.stream, ctx.n_elems, nen, nq, ctx.elems.p, ctx.jac.p,
              ctx.deriv.p, ctx.is_inner.p, ctx.cond_field.n ? ctx.cond_field.p : nullptr, ctx.model, ctx.basis,
              integrand, weight, ctx.symmetric || integrand == 1, mtx.rowptr.p, mtx.col.p, mtx.val.p,
              with_bound ? ctx.bound.rowptr.p : nullptr, with_bound ? ctx.bound.col.p : nullptr,
              with_bound ? ctx.bound.val.p : nullptr);
    set_dirichlet_diagonal(ctx, mtx, 1.0);
}

void set_dirichlet_diagonal(Ctx& ctx, Csr& mtx, double value) {
    NL_LAUNCH(k_dirichlet_diagonal, grid_for(mtx.rows, 256), 256, 0, ctx.stream, mtx.rows, ctx.is_inner.p,
              mtx.rowptr.p, mtx.val.p, value);
}

void gather_full(Ctx& ctx, Csr& full, const dbuf<i64>& map, const double* upper, float* full32) {
    NL_LAUNCH(k_gather_full, grid_for(full.nnz, 256), 256, 0, ctx.stream, full.nnz, map.p, upper, full.val.p, full32);
}

// ---------------------------------------------------------------- nonstationary
namespace {

// K <- dt K + C row by row (C's pattern is contained in K's), unit Dirichlet
// diagonal; bound <- dt bound (nonstationary_heat_equation_solver_2d.hpp:77-82).
__global__ void k_combine(i64 n, double dt, const uint8_t* __restrict__ is_inner, const i64* __restrict__ krp,
                          const int32_t* __restrict__ kcol, double* __restrict__ kval, const i64* __restrict__ crp,
                          const int32_t* __restrict__ ccol, const double* __restrict__ cval, const i64* __restrict__ brp,
                          double* __restrict__ bval) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
        for (i64 k = krp[r]; k < krp[r + 1]; ++k) kval[k] *= dt;
        for (i64 k = brp[r]; k < brp[r + 1]; ++k) bval[k] *= dt;
        i64 k = krp[r];
        for (i64 s = crp[r]; s < crp[r + 1]; ++s) {
            while (k < krp[r + 1] && kcol[k] != ccol[s]) ++k;
            if (k < krp[r + 1]) kval[k] += cval[s];
        }
        if (!is_inner[r]) kval[krp[r]] = 1.0;
    }
}

// Dirichlet vector of a step: value on every Dirichlet node (or the uploaded per-node values)
__global__ void k_step_dirichlet(i64 n, const uint8_t* __restrict__ is_inner, double value, bool per_node,
                                 double* __restrict__ xd) {
    for (i64 i = blockIdx.x * i64(blockDim.x) + threadIdx.x; i < n; i += i64(gridDim.x) * blockDim.x)
        xd[i] = is_inner[i] ? 0.0 : (per_node ? xd[i] : value);
}

__global__ void k_axpy_into(i64 n, double a, const double* __restrict__ x, double* __restrict__ y) {
    for (i64 i = blockIdx.x * i64(blockDim.x) + threadIdx.x; i < n; i += i64(gridDim.x) * blockDim.x) y[i] += a * x[i];
}

}  // namespace

void combine_nonstationary(Ctx& ctx, double dt) {
    NL_LAUNCH(k_combine, grid_for(ctx.n_nodes, 256), 256, 0, ctx.stream, ctx.n_nodes, dt, ctx.is_inner.p,
              ctx.inner.rowptr.p, ctx.inner.col.p, ctx.inner.val.p, ctx.capacity_m.rowptr.p, ctx.capacity_m.col.p,
              ctx.capacity_m.val.p, ctx.bound.rowptr.p, ctx.bound.val.p);
}

// rhs = dt * rhs_init + C T_prev, then the first-kind step with the step's Dirichlet values
void nonstationary_rhs(Ctx& ctx, double dirichlet_value, bool per_node_values, const double* radiation) {
    const i64 n = ctx.n_nodes;
    NL_LAUNCH(k_step_dirichlet, grid_for(n, 256), 256, 0, ctx.stream, n, ctx.is_inner.p, dirichlet_value,
              per_node_values, ctx.step_xd.p);
    spmv_full(ctx, ctx.capacity_full, ctx.temperature.p, ctx.step_tmp.p);
    NL_LAUNCH(k_axpy_into, grid_for(n, 256), 256, 0, ctx.stream, n, ctx.time_step, ctx.rhs_init.p, ctx.step_tmp.p);
    if (radiation)
        NL_LAUNCH(k_axpy_into, grid_for(n, 256), 256, 0, ctx.stream, n, ctx.time_step, radiation, ctx.step_tmp.p);
    apply_first_kind(ctx, ctx.bound, ctx.step_tmp.p, ctx.rhs.p, ctx.step_xd.p);
}

}  // namespace nlgpu
