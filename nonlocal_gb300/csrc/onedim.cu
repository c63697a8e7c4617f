// 1D stationary nonlocal heat conduction (stationary_heat_equation_solver_1d.hpp:43-122).
//
//   mesh: one segment [0, length], `elements` Lagrange elements of order 1 or 2,
//     neighbours e +- round(r / h) inside the segment (mesh_1d.hpp:119-122, 221-232);
//   assembly: p1 * local + (1 - p1) * nonlocal element blocks
//     (thermal_conductivity_assembler.hpp:64-125, assebmler_base.hpp:112-155),
//     upper band, node 0 Dirichlet: its row goes to the bound vector, entries
//     of column 0 in other rows are dropped, unit diagonal;
//   right-hand side: flux at the right end, source integral, first-kind step;
//   solve: LDL^T of the band matrix in natural order (the reference's
//     Eigen::SimplicialCholesky<..., Upper, NaturalOrdering>).
//
// Assembly: one thread per (element, neighbour element) pair computes the
// (order+1)^2 block.  Factorisation: blocks of 16 rows in one cluster of 16 CTAs
// (k_band_factor); the substitutions use the inverses of its diagonal blocks.
//
// 1D nonstationary (nonstationary_heat_equation_solver_1d.hpp:24-259):
// compute() assembles A = dt K + C (C the local capacity matrix c rho int N_i N_j,
// heat_capacity_assembler.hpp:30-58) with either end a temperature (its row and
// column routed out, unit diagonal, K's row kept as dt x bound) or a flux, and
// factors A once (LDL^T of the band).  calc_step() forms
// f = dt (flux + source) + C T_prev (inner entries of C only, as the
// reference's product), applies the first kind and solves with the factor: the
// solution the reference's ConjugateGradient reaches at machine tolerance.
#include "common.cuh"

#include <cmath>
#include <numbers>

namespace nlgpu {

namespace {

struct Line {
    int nen, nq;
    double qN[3 * 3], qNxi[3 * 3], w[3], x[3];
};

Line make_line(int order) {
    Line L{};
    L.nen = order + 1;
    L.nq = order == 1 ? 2 : 3;
    if (L.nq == 2) { L.x[0] = -1.0 / std::sqrt(3.0); L.x[1] = 1.0 / std::sqrt(3.0); L.w[0] = L.w[1] = 1.0; }
    else { L.x[0] = -std::sqrt(3.0 / 5.0); L.x[1] = 0.0; L.x[2] = std::sqrt(3.0 / 5.0); L.w[0] = 5.0 / 9.0; L.w[1] = 8.0 / 9.0; L.w[2] = 5.0 / 9.0; }
    for (int q = 0; q < L.nq; ++q) L.w[q] = L.w[q] * 1.0;
    for (int i = 0; i < L.nen; ++i)
        for (int q = 0; q < L.nq; ++q) {
            const double x = -1.0 + (L.x[q] - (-1.0)) * 1.0;
            double N, Nx;
            if (order == 1) { N = i == 0 ? (1 - x) / 2 : (1 + x) / 2; Nx = i == 0 ? -0.5 : 0.5; }
            else if (i == 0) { N = x * (x - 1) / 2; Nx = (2 * x - 1) / 2; }
            else if (i == 1) { N = (1 - x) * (1 + x); Nx = -2 * x; }
            else { N = x * (x + 1) / 2; Nx = (2 * x + 1) / 2; }
            L.qN[i * L.nq + q] = N; L.qNxi[i * L.nq + q] = Nx;
        }
    return L;
}

struct Problem1d {
    i64 E, n, nb, bw;          // elements, nodes, neighbour count, half bandwidth
    int order;
    double h, jac, r, p1, lambda, norm;
    int kind;                  // 0 bell, 1 triangle, 2 normal, 3 constant
    int fk0, fk1;              // temperature (first kind) at the left / right end
    int cv0, cv1;              // convection at the left / right end
    double h0, h1;             // their heat transfer coefficients
};

// influence_functions_1d.hpp:10-75
__device__ __forceinline__ double influence_1d(const Problem1d& P, double x, double y) {
    const double d = fabs(x - y);
    if (P.kind == 0) { const double t = d / P.r; return d < P.r ? P.norm * (1 - t * t) : 0.0; }
    if (P.kind == 1) { return d < P.r ? P.norm * (1 - d / P.r) : 0.0; }
    if (P.kind == 2) { return P.norm * exp((-0.5 / (P.r * P.r)) * ((x - y) * (x - y))); }
    return d < P.r ? P.norm : 0.0;
}

// assembler_base_1d::calc_matrix (assebmler_base.hpp:121-154): entries in the
// row or column of a first-kind end go to that end's bound vector (its row's
// entries; the diagonal becomes 1 later) or are dropped; the rest fill the
// upper band.  bound0 / boundN may be null (dropped).
__device__ __forceinline__ void band_add(const Problem1d& P, double* band, double* bound0, double* boundN, i64 row,
                                         i64 col, double v) {
    const i64 last = P.n - 1;
    if (P.fk0 && (row == 0 || col == 0)) {
        if (row == 0 && col != 0 && bound0) atomicAdd(bound0 + col, v);
        return;
    }
    if (P.fk1 && (row == last || col == last)) {
        if (row == last && col != last && boundN) atomicAdd(boundN + col, v);
        return;
    }
    if (row <= col) atomicAdd(band + row * (P.bw + 1) + (col - row), v);
}

__global__ void k_assemble_1d(Problem1d P, Line L, double* __restrict__ band, double* __restrict__ bound0,
                              double* __restrict__ boundN) {
    const i64 width = 2 * P.nb + 1;
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < P.E * width; t += i64(gridDim.x) * blockDim.x) {
        const i64 e = t / width, f = e - P.nb + t % width;
        if (f < 0 || f >= P.E) continue;
        const bool nonlocal = P.p1 < 0.999;
        // pairs below the diagonal keep only the node two neighbours share and the
        // right end's bound row
        if (f < e - 1 && !(P.fk1 && e == P.E - 1)) continue;
        double inner[3][3];   // [qL][j]: the influence once per pair of points, not per entry
        if (nonlocal) {
            double xl[3], xn[3];
            for (int q = 0; q < L.nq; ++q) {
                xl[q] = P.h * double(e) + (L.x[q] - (-1.0)) * P.jac;
                xn[q] = P.h * double(f) + (L.x[q] - (-1.0)) * P.jac;
            }
            for (int qL = 0; qL < L.nq; ++qL) {
                double g[3];
                for (int qNL = 0; qNL < L.nq; ++qNL) g[qNL] = influence_1d(P, xl[qL], xn[qNL]) * P.lambda * L.w[qNL];
                for (int j = 0; j < L.nen; ++j) {
                    double v = 0.0;
                    for (int qNL = 0; qNL < L.nq; ++qNL) v += g[qNL] * L.qNxi[j * L.nq + qNL];
                    inner[qL][j] = v;
                }
            }
        }
        for (int i = 0; i < L.nen; ++i) {
            const i64 row = e * P.order + i;
            for (int j = 0; j < L.nen; ++j) {
                const i64 col = f * P.order + j;
                if (nonlocal) {
                    double integral = 0.0;
                    for (int qL = 0; qL < L.nq; ++qL) integral += L.w[qL] * L.qNxi[i * L.nq + qL] * inner[qL][j];
                    band_add(P, band, bound0, boundN, row, col, (1.0 - P.p1) * integral);
                }
                if (f == e) {
                    double integral = 0.0;
                    for (int q = 0; q < L.nq; ++q) integral += P.lambda * L.w[q] * L.qNxi[i * L.nq + q] * L.qNxi[j * L.nq + q];
                    band_add(P, band, bound0, boundN, row, col, P.p1 * (integral / P.jac));
                }
            }
        }
    }
}

__global__ void k_rhs_1d(Problem1d P, Line L, double q_right, bool sin_source, double* __restrict__ f) {
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < P.E * L.nen; t += i64(gridDim.x) * blockDim.x) {
        const i64 e = t / L.nen;
        const int i = int(t % L.nen);
        if (!sin_source) continue;
        double integral = 0.0;
        for (int q = 0; q < L.nq; ++q)
            integral += L.w[q] * L.qN[i * L.nq + q] * sin(std::numbers::pi * (P.h * double(e) + (L.x[q] - (-1.0)) * P.jac));
        atomicAdd(f + e * P.order + i, integral * P.jac);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(f + P.n - 1, q_right);
}

__global__ void k_first_kind_1d(i64 n, const double* __restrict__ bound0, double t_left, double* __restrict__ f,
                                double* __restrict__ band) {
    for (i64 i = blockIdx.x * i64(blockDim.x) + threadIdx.x; i < n; i += i64(gridDim.x) * blockDim.x) {
        if (i == 0) { f[0] = t_left; band[0] = 1.0; }
        else f[i] -= bound0[i] * t_left;
    }
}

// Band LDL^T in blocks of BF_NB rows, one cluster of CTAS CTAs (upper band:
// band[i * (bw + 1) + (j - i)]).
//
// A row at a time, every pivot cost three CTA barriers and bw^2 / 2 updates with a
// division each on one SM's FP64 pipe (two lanes a clock): 33 us a pivot,
// 66.8 ms for 2 001 rows of half bandwidth 102.  Here a block of 16 pivots is the
// work of four warps in registers: they eliminate [A_kk | I], lane j < 16 holding
// column j of A_kk and lane 16 + j column j of I, which leaves D L^T and L^-1 at no
// extra instructions.  A warp's FP64 instruction holds its quarter of the SM's FP64
// pipe for 64 cycles, so the rows are dealt out over the four quarters: a pivot costs
// 5 to 8 of them instead of 6 to 21 in one warp.  That is the critical path, and
// everything else is spread over the cluster between two eliminations:
//   W = L^-1 A(block, columns after it)                 (the other 15 CTAs)
//   A(i, j) -= sum_k W(k, i) W(k, j) / d_k               (the other 15 CTAs)
//   next diagonal block: its own 16 columns of W, the update, the elimination   (first CTA)
// with a cluster barrier after each phase, of which the first CTA only
// passes the second one on its way.  The rows keep U = D^-1 W beyond
// their block; L^-1 and 1 / d are kept per block.  The right-hand side, when there
// is one, is one more column (its forward substitution comes for free).
// 2 001 rows of half bandwidth 102: 66.8 ms; 2.0 with the elimination in one warp (1.1
// of it) and W shared by all CTAs; 1.42 now.
constexpr int BF_NB = 16;
constexpr int BF_THREADS = 256;

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() {
    cluster_arrive();
    cluster_wait();
}

struct BandFactor {
    i64 n, bw;
    double* band;
    double* f;                // right-hand side, becomes L^-1 f (null: none)
    double* linv;             // [blocks][BF_NB][BF_NB]
    double* dinv;             // [blocks * BF_NB]
    double* w;                // [BF_NB][bw + 1] scratch
    int* failed;
    int in_shared;            // W is copied to shared memory
};

// 1 / d by two Newton steps from the hardware's approximation, without the
// division's special cases (the chain of pivots waits for it), where d and 1 / d are
// normal numbers.
__device__ __forceinline__ double reciprocal(double d) {
    if ((unsigned(__double2hiint(d)) >> 20 & 0x7ffu) - 2u >= 2042u) return 1.0 / d;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(fma(-d, r, 1.0), r, r);
    return fma(fma(-d, r, 1.0), r, r);
}

// Warps 0 .. 3 eliminate the diagonal block in `diag` (upper), a warp the rows i = part
// (mod 4) of [A | I]; writes L^-1 and 1 / d to global memory and to lk, dk.  A pivot's
// row goes round through shared memory.
constexpr int BF_PARTS = 4;
__device__ __forceinline__ void eliminate_block(const double (*diag)[BF_NB + 1], double (*row)[32], double* linv,
                                                double* dinv, double* lk, double* dk, int* failed, int part) {
    constexpr int OWN = BF_NB / BF_PARTS;
    const int lane = threadIdx.x & 31;
    double a[OWN];
#pragma unroll
    for (int q = 0; q < OWN; ++q) {
        const int i = BF_PARTS * q + part;
        a[q] = lane < BF_NB ? diag[min(i, lane)][max(i, lane)] : (i == lane - BF_NB ? 1.0 : 0.0);
    }
#pragma unroll
    for (int k = 0; k < BF_NB; ++k) {
        double* pivot = row[k & 1];
        if (part == k % BF_PARTS) pivot[lane] = a[k / BF_PARTS];
        asm volatile("bar.sync 1, %0;" ::"n"(BF_PARTS * 32) : "memory");
        // row k is final; by symmetry its entry i is the multiplier of row i
        const double t = pivot[lane], d = pivot[k], inv = reciprocal(d);
        if (part == 0 && lane == 0) {
            dinv[k] = dk[k] = inv;
            if (d == 0.0) *failed = 1;
        }
        const double s = -t * inv;
#pragma unroll
        for (int q = k / BF_PARTS; q < OWN; ++q)   // row k + 1, the next pivot's, is its warp's first
            if (BF_PARTS * q + part > k) a[q] = fma(pivot[BF_PARTS * q + part], s, a[q]);
    }
    if (lane >= BF_NB)
#pragma unroll
        for (int q = 0; q < OWN; ++q) {
            const int at = (BF_PARTS * q + part) * BF_NB + lane - BF_NB;
            linv[at] = lk[at] = a[q];
        }
}

// CTAS: 16, or 8 (the largest portable cluster) where no 16 fit
template<int CTAS>
__global__ void __launch_bounds__(BF_THREADS) k_band_factor(BandFactor p) {
    extern __shared__ double bf_w[];
    __shared__ double diag[BF_NB][BF_NB + 1], wn[BF_NB][BF_NB], scaled[BF_NB][BF_NB], dks[2][BF_NB], lk[BF_NB * BF_NB],
        pivots[2][32];
    const i64 w = p.bw + 1, blocks = (p.n + BF_NB - 1) / BF_NB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x;
    // entry (i, j >= i) of the matrix, rows past the end an identity
    auto entry = [&](i64 i, i64 j) {
        if (i >= p.n || j >= p.n) return i == j ? 1.0 : 0.0;
        return j - i <= p.bw ? p.band[i * w + (j - i)] : 0.0;
    };
    auto eliminate = [&](i64 kb) {   // the first CTA's warps 0 .. BF_PARTS - 1
        eliminate_block(diag, pivots, p.linv + kb * BF_NB * BF_NB, p.dinv + kb * BF_NB, lk, dks[kb & 1], p.failed, warp);
    };
    if (rank == 0) {
        diag[tid >> 4][tid & 15] = (tid >> 4) <= (tid & 15) ? entry(tid >> 4, tid & 15) : 0.0;
        __syncthreads();
        if (warp < BF_PARTS) eliminate(0);
    }
    for (i64 kb = 0; kb < blocks; ++kb) {
        cluster_barrier();
        const i64 k0 = kb * BF_NB, next = k0 + BF_NB;
        const int m = int(max(i64(0), min(p.bw, p.n - next)));   // columns after the block that it reaches
        const int cols = m + (p.f ? 1 : 0);
        double* dk = dks[kb & 1];
        if (rank == 0) {
            // the first CTA takes what the next elimination waits for: the 16 columns of W
            // over the next diagonal block, that block's update, the elimination
            if (kb + 1 < blocks) {
                const int r = tid >> 4, c = tid & 15;
                double v = 0.0, v2 = 0.0;
                if (c < m) {
#pragma unroll
                    for (int s = 0; s < BF_NB; s += 2) {
                        const double x = entry(k0 + s, next + c), y = entry(k0 + s + 1, next + c);
                        if (s <= r) v = fma(lk[r * BF_NB + s], x, v);
                        if (s + 1 <= r) v2 = fma(lk[r * BF_NB + s + 1], y, v2);
                    }
                }
                wn[r][c] = v + v2;
                scaled[r][c] = (v + v2) * dk[r];
            }
            cluster_arrive();
            if (kb + 1 < blocks) {
                __syncthreads();
                const int r = tid >> 4, c = tid & 15;
                double v = 0.0;
                if (r <= c) {
                    double u = 0.0, u2 = 0.0;
                    v = entry(next + r, next + c);
#pragma unroll
                    for (int k = 0; k < BF_NB; k += 2) {
                        u = fma(scaled[k][r], wn[k][c], u);
                        u2 = fma(scaled[k + 1][r], wn[k + 1][c], u2);
                    }
                    v -= u + u2;
                }
                diag[r][c] = v;
                __syncthreads();
                if (warp < BF_PARTS) eliminate(kb + 1);
            }
            cluster_wait();   // W is complete
            // the block's rows: U = D^-1 W, and L^-1 f
            if (warp >= BF_PARTS)
                for (int t = tid - 32 * BF_PARTS; t < BF_NB * cols; t += BF_THREADS - 32 * BF_PARTS) {
                    const int r = t / cols, c = t % cols;
                    if (k0 + r >= p.n) continue;
                    const double v = p.w[i64(r) * w + c];
                    if (c == m) p.f[k0 + r] = v;
                    else if (BF_NB + c - r <= p.bw) p.band[(k0 + r) * w + (BF_NB + c - r)] = v * dk[r];
                }
        } else {
            if (tid < BF_NB) dk[tid] = p.dinv[k0 + tid];
            lk[tid] = p.linv[kb * BF_NB * BF_NB + tid];
            __syncthreads();
            for (int t = tid * (CTAS - 1) + rank - 1; t < BF_NB * cols; t += (CTAS - 1) * BF_THREADS) {
                const int r = t / cols, c = t % cols;
                double v = 0.0, v2 = 0.0;
#pragma unroll
                for (int s = 0; s < BF_NB; s += 2) {
                    const double x = c < m ? entry(k0 + s, next + c) : (k0 + s < p.n ? p.f[k0 + s] : 0.0);
                    const double y = c < m ? entry(k0 + s + 1, next + c) : (k0 + s + 1 < p.n ? p.f[k0 + s + 1] : 0.0);
                    if (s <= r) v = fma(lk[r * BF_NB + s], x, v);
                    if (s + 1 <= r) v2 = fma(lk[r * BF_NB + s + 1], y, v2);
                }
                p.w[i64(r) * w + c] = v + v2;
            }
            cluster_barrier();
            const double* W = p.w;
            if (p.in_shared) {
                for (int t = tid; t < BF_NB * cols; t += BF_THREADS) bf_w[i64(t / cols) * w + t % cols] = p.w[i64(t / cols) * w + t % cols];
                W = bf_w;
                __syncthreads();
            }
            // a warp per row a, rows dealt out over the other CTAs
            for (int a = (rank - 1) + (CTAS - 1) * warp; a < m; a += (CTAS - 1) * (BF_THREADS / 32)) {
                double wa[BF_NB];
#pragma unroll
                for (int k = 0; k < BF_NB; ++k) wa[k] = W[k * w + a] * dk[k];
                // the next diagonal block is the first CTA's
                for (int b = (a < BF_NB ? BF_NB : a) + lane; b < cols; b += 32) {
                    double v = 0.0, v2 = 0.0;
#pragma unroll
                    for (int k = 0; k < BF_NB; k += 2) {
                        v = fma(wa[k], W[k * w + b], v);
                        v2 = fma(wa[k + 1], W[(k + 1) * w + b], v2);
                    }
                    if (b < m) p.band[(next + a) * w + (b - a)] -= v + v2;
                    else p.f[next + a] -= v + v2;
                }
                // the right-hand side's entry of a short window (m < 16)
                if (p.f && m < BF_NB && lane == 0) {
                    double v = 0.0;
#pragma unroll
                    for (int k = 0; k < BF_NB; ++k) v = fma(wa[k], W[k * w + m], v);
                    p.f[next + a] -= v;
                }
            }
        }
    }
}

// The substitutions with the factor of k_band_factor in one CTA, a block at a
// time: forward y = L^-1 f (skipped when the factorisation carried f along), then
// x = L^-T (D^-1 y - U x beyond the block).  The factor's entries of the next
// block are loaded while the current one is worked on, the vector stays in shared
// memory.  667 rows of half bandwidth 48: both substitutions 147 us a step, a row
// at a time in one warp about 460.
__global__ void __launch_bounds__(BF_THREADS) k_band_solve(i64 n, i64 bw, const double* __restrict__ band,
                                                           const double* __restrict__ linv,
                                                           const double* __restrict__ dinv, double* fg, bool forward,
                                                           bool in_shared) {
    extern __shared__ double bs_f[];
    __shared__ double blk[BF_NB];
    double* f = in_shared ? bs_f : fg;
    if (in_shared) {
        for (i64 i = threadIdx.x; i < n; i += BF_THREADS) f[i] = fg[i];
        __syncthreads();
    }
    const i64 w = bw + 1, blocks = (n + BF_NB - 1) / BF_NB;
    const int tid = threadIdx.x, r = tid >> 4, l = tid & 15;   // 16 lanes per row of a block
    auto sum16 = [](double v) {
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    if (forward) {
        double u[BF_NB], lv = 0.0;
        auto load = [&](i64 kb) {
            const i64 k0 = kb * BF_NB;
            lv = linv[kb * BF_NB * BF_NB + tid];
            const i64 j = k0 + BF_NB + tid;
#pragma unroll
            for (int s = 0; s < BF_NB; ++s) u[s] = j < n && BF_NB + tid - s <= bw ? band[(k0 + s) * w + (BF_NB + tid - s)] : 0.0;
        };
        load(0);
        for (i64 kb = 0; kb < blocks; ++kb) {
            const i64 k0 = kb * BF_NB;
            const double y = sum16(l <= r && k0 + l < n ? lv * f[k0 + l] : 0.0);
            if (l == 0) blk[r] = y;
            __syncthreads();
            if (tid < BF_NB && k0 + tid < n) f[k0 + tid] = blk[tid];
            const i64 j = k0 + BF_NB + tid;
            if (j < n && tid < bw) {
                double v = 0.0, v2 = 0.0;
#pragma unroll
                for (int s = 0; s < BF_NB; s += 2) { v = fma(u[s], blk[s], v); v2 = fma(u[s + 1], blk[s + 1], v2); }
                f[j] -= v + v2;
            }
            for (i64 c = tid + BF_THREADS; c < bw && k0 + BF_NB + c < n; c += BF_THREADS) {   // wide bands
                double v = 0.0;
                for (int s = 0; s < BF_NB; ++s)
                    if (BF_NB + c - s <= bw) v = fma(band[(k0 + s) * w + (BF_NB + c - s)], blk[s], v);
                f[k0 + BF_NB + c] -= v;
            }
            if (kb + 1 < blocks) load(kb + 1);
            __syncthreads();
        }
    }
    constexpr int PER = 8;   // entries of U per lane kept ahead: half bandwidths up to 128
    double u[PER], lv = 0.0, di = 0.0;
    auto load = [&](i64 kb) {
        const i64 i = kb * BF_NB + r;
        lv = linv[kb * BF_NB * BF_NB + l * BF_NB + r];
        di = dinv[i];
#pragma unroll
        for (int s = 0; s < PER; ++s) {
            const int c = l + 16 * s;
            u[s] = i < n && kb * BF_NB + BF_NB + c < n && BF_NB + c - r <= bw ? band[i * w + (BF_NB + c - r)] : 0.0;
        }
    };
    load(blocks - 1);
    for (i64 kb = blocks - 1; kb >= 0; --kb) {
        const i64 k0 = kb * BF_NB, i = k0 + r, j0 = k0 + BF_NB;
        double v = 0.0, v2 = 0.0;
#pragma unroll
        for (int s = 0; s < PER; ++s) {
            const i64 j = j0 + l + 16 * s;
            if (j < n && l + 16 * s < bw) (s & 1 ? v2 : v) = fma(u[s], f[j], s & 1 ? v2 : v);
        }
        v += v2;
        for (i64 c = l + 16 * PER; i < n && c < bw && j0 + c < n && BF_NB + c - r <= bw; c += 16)
            v = fma(band[i * w + (BF_NB + c - r)], f[j0 + c], v);
        v = sum16(v);
        if (l == 0) blk[r] = i < n ? fma(f[i], di, -v) : 0.0;
        __syncthreads();
        const double x = sum16(l >= r ? lv * blk[l] : 0.0);
        if (kb > 0) load(kb - 1);
        if (l == 0 && i < n) {
            f[i] = x;
            if (in_shared) fg[i] = x;
        }
        __syncthreads();
    }
}

// heat_capacity_assembler_1d::integrate: c rho sum_q w_q N_i N_j |J| per
// (element, i, j), routed as the conductivity (bound entries dropped)
__global__ void k_capacity_1d(Problem1d P, Line L, double factor, double* __restrict__ band) {
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < P.E * L.nen * L.nen; t += i64(gridDim.x) * blockDim.x) {
        const i64 e = t / (L.nen * L.nen);
        const int i = int(t / L.nen % L.nen), j = int(t % L.nen);
        double integral = 0.0;
        for (int q = 0; q < L.nq; ++q) integral += L.w[q] * L.qN[i * L.nq + q] * L.qN[j * L.nq + q];
        band_add(P, band, nullptr, nullptr, e * P.order + i, e * P.order + j, factor * (integral * P.jac));
    }
}

// A = dt K + C over the band, unit diagonal at first-kind ends (C too), bound
// vectors x dt; a convection end adds dt h to its diagonal (K gets h before the
// time step factor: convection_condition_1d.hpp:10-14,
// nonstationary_heat_equation_solver_1d.hpp:167-178).  The ends' diagonals are
// set by the thread of their band element.
__global__ void k_combine_1d(Problem1d P, double dt, double* __restrict__ a, double* __restrict__ c,
                             double* __restrict__ bound0, double* __restrict__ boundN) {
    const i64 w = P.bw + 1, last = P.n - 1;
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < P.n * w; t += i64(gridDim.x) * blockDim.x) {
        double v = dt * a[t] + c[t];
        if (t == 0) {
            if (P.fk0) { v = 1.0; c[0] = 1.0; }
            else if (P.cv0) v += dt * P.h0;
        }
        if (t == last * w) {
            if (P.fk1) { v = 1.0; c[t] = 1.0; }
            else if (P.cv1) v += dt * P.h1;
        }
        a[t] = v;
        if (t < P.n) { bound0[t] *= dt; boundN[t] *= dt; }
    }
}

// f = second-kind ends + source integral (before the time step factor)
__global__ void k_step_loads_1d(Problem1d P, Line L, double q_left, double q_right, bool sin_source,
                                double* __restrict__ f) {
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < P.E * L.nen; t += i64(gridDim.x) * blockDim.x) {
        const i64 e = t / L.nen;
        const int i = int(t % L.nen);
        if (!sin_source) continue;
        double integral = 0.0;
        for (int q = 0; q < L.nq; ++q)
            integral += L.w[q] * L.qN[i * L.nq + q] * sin(std::numbers::pi * (P.h * double(e) + (L.x[q] - (-1.0)) * P.jac));
        atomicAdd(f + e * P.order + i, integral * P.jac);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // a convection end's value is its ambient temperature
        if (!P.fk0) atomicAdd(f, P.cv0 ? P.h0 * q_left : q_left);
        if (!P.fk1) atomicAdd(f + P.n - 1, P.cv1 ? P.h1 * q_right : q_right);
    }
}

// f = dt f + C T_prev (symmetric band product), then the first kind of each
// temperature end: f -= bound T_end, f[end] = T_end (boundary_condition_first_kind_1d.hpp)
__global__ void k_step_rhs_1d(Problem1d P, double dt, const double* __restrict__ c, const double* __restrict__ t_prev,
                              const double* __restrict__ bound0, const double* __restrict__ boundN, double t_left,
                              double t_right, double* __restrict__ f) {
    const i64 w = P.bw + 1, last = P.n - 1;
    for (i64 i = blockIdx.x * i64(blockDim.x) + threadIdx.x; i < P.n; i += i64(gridDim.x) * blockDim.x) {
        double s = 0.0;
        for (i64 j = max(i64(0), i - P.bw); j < i; ++j) s += c[j * w + (i - j)] * t_prev[j];
        for (i64 j = i; j <= min(last, i + P.bw); ++j) s += c[i * w + (j - i)] * t_prev[j];
        double v = dt * f[i] + s;
        if (P.fk0) v -= bound0[i] * t_left;
        if (P.fk1) v -= boundN[i] * t_right;
        if (P.fk0 && i == 0) v = t_left;
        if (P.fk1 && i == last) v = t_right;
        f[i] = v;
    }
}

// L^-1 and 1 / d of the blocks, and the factorisation's scratch
struct BandWork {
    dbuf<double> linv, dinv, w;
    void resize(i64 n, i64 bw) {
        const size_t blocks = size_t((n + BF_NB - 1) / BF_NB);
        linv.resize(blocks * BF_NB * BF_NB);
        dinv.resize(blocks * BF_NB);
        w.resize(size_t(BF_NB) * size_t(bw + 1));
    }
};

template<int CTAS>
bool launch_band_factor(Ctx& ctx, const BandFactor& p, size_t smem) {
    auto kernel = k_band_factor<CTAS>;
    allow_shared(kernel);
    if (CTAS > 8) NL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CTAS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CTAS);
    cfg.blockDim = dim3(BF_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (CTAS > 8) {   // a part of a GPU may have no 16 SMs that one cluster can span
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            return false;
        }
    }
    NL_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    count_launch();
    return true;
}

// 2 001 rows of half bandwidth 102, the whole solve: 1.75 ms with 16 CTAs, 2.28 with 8
void band_factor(Ctx& ctx, i64 n, i64 bw, double* band, double* f, BandWork& work, int* failed) {
    work.resize(n, bw);
    BandFactor p{n, bw, band, f, work.linv.p, work.dinv.p, work.w.p, failed, 0};
    const size_t bytes = size_t(BF_NB) * size_t(bw + 1) * sizeof(double);
    p.in_shared = bytes <= 200 * 1024;
    const size_t smem = p.in_shared ? bytes : 0;
    if (ctx.band_ctas == 8 || !launch_band_factor<16>(ctx, p, smem)) launch_band_factor<8>(ctx, p, smem);
}

void band_solve(Ctx& ctx, i64 n, i64 bw, const double* band, const BandWork& work, double* f, bool forward) {
    const bool in_shared = n <= 24 * 1024;   // the vector in shared memory
    const size_t smem = in_shared ? size_t(n) * sizeof(double) : 0;
    allow_shared(k_band_solve);
    NL_LAUNCH(k_band_solve, 1, BF_THREADS, smem, ctx.stream, n, bw, band, work.linv.p, work.dinv.p, f, forward, in_shared);
}

// mesh, model and band geometry of one segment [0, length]
Problem1d make_problem_1d(i64 elements, int order, double length, double radius, double local_weight, int influence,
                          double conductivity) {
    NL_REQUIRE(influence >= 0 && influence <= 3, NLGPU_ERR_ARG, "unknown 1D influence kind");
    Problem1d P{};
    P.E = elements; P.order = order; P.n = elements * order + 1;
    P.h = length / double(elements);
    P.jac = P.h / (1.0 - (-1.0));
    P.r = radius; P.p1 = local_weight; P.lambda = conductivity; P.kind = influence;
    const bool nonlocal = local_weight < 0.999;
    NL_REQUIRE(!nonlocal || radius > 0.0, NLGPU_ERR_ARG, "nonlocal radius must be positive");
    P.nb = nonlocal ? i64(std::round(radius / P.h)) : 0;
    P.bw = nonlocal ? (P.nb + 1) * order : order;
    if (influence == 0) P.norm = 2.0 / (2 * radius * std::beta(0.5, 2.0));
    else if (influence == 1) P.norm = 1.0 / (2 * radius * std::beta(1.0, 2.0));
    else if (influence == 2) P.norm = 1.0 / (radius * std::sqrt(2 * std::numbers::pi));
    else P.norm = 0.5 / radius;
    NL_REQUIRE(double(P.n) * double(P.bw + 1) * 8.0 < 64e9, NLGPU_ERR_UNSUPPORTED, "1D band too large");
    return P;
}

}  // namespace

// Device state of nonstationary_heat_equation_solver_1d between compute and the steps.
struct OneDimState {
    Problem1d P{};
    Line L{};
    double dt = 0.0;
    dbuf<double> a, c, bound0, boundN, t, f;
    BandWork factor;
};

void nonstationary_1d_compute(Ctx& ctx, i64 elements, int order, double length, double radius, double local_weight,
                              int influence, double conductivity, double capacity, double density, double time_step,
                              int left_kind, int right_kind, const double* initial) {
    NL_REQUIRE(elements > 0 && (order == 1 || order == 2) && length > 0.0 && time_step > 0.0, NLGPU_ERR_ARG,
               "invalid 1D mesh or time step");
    for (const int k : {left_kind, right_kind})
        NL_REQUIRE(k == NLGPU_BC_TEMPERATURE || k == NLGPU_BC_FLUX || k == NLGPU_BC_CONVECTION, NLGPU_ERR_UNSUPPORTED,
                   "1D ends take a temperature, a flux or a convection");
    auto st = std::make_shared<OneDimState>();
    Problem1d& P = st->P;
    P = make_problem_1d(elements, order, length, radius, local_weight, influence, conductivity);
    P.fk0 = left_kind == NLGPU_BC_TEMPERATURE;
    P.fk1 = right_kind == NLGPU_BC_TEMPERATURE;
    P.cv0 = left_kind == NLGPU_BC_CONVECTION;
    P.cv1 = right_kind == NLGPU_BC_CONVECTION;
    P.h0 = P.cv0 ? ctx.od_heat_transfer[0] : 0.0;
    P.h1 = P.cv1 ? ctx.od_heat_transfer[1] : 0.0;
    st->L = make_line(order);
    st->dt = time_step;
    const size_t n = size_t(P.n), nb = size_t(P.n * (P.bw + 1));
    st->a.resize(nb); st->a.zero(ctx.stream);
    st->c.resize(nb); st->c.zero(ctx.stream);
    st->bound0.resize(n); st->bound0.zero(ctx.stream);
    st->boundN.resize(n); st->boundN.zero(ctx.stream);
    st->t.resize(n);
    st->f.resize(n);
    if (initial) st->t.upload(initial, n, ctx.stream);
    else st->t.zero(ctx.stream);
    dbuf<int> failed;
    failed.resize(1); failed.zero(ctx.stream);
    NL_LAUNCH(k_assemble_1d, grid_for(P.E * (2 * P.nb + 1), 128), 128, 0, ctx.stream, P, st->L, st->a.p, st->bound0.p,
              st->boundN.p);
    NL_LAUNCH(k_capacity_1d, grid_for(P.E * st->L.nen * st->L.nen, 256), 256, 0, ctx.stream, P, st->L,
              capacity * density, st->c.p);
    NL_LAUNCH(k_combine_1d, grid_for(i64(nb), 256), 256, 0, ctx.stream, P, time_step, st->a.p, st->c.p, st->bound0.p,
              st->boundN.p);
    band_factor(ctx, P.n, P.bw, st->a.p, nullptr, st->factor, failed.p);
    int hf = 0;
    NL_CUDA(cudaMemcpyAsync(&hf, failed.p, sizeof hf, cudaMemcpyDeviceToHost, ctx.stream));
    NL_CUDA(cudaStreamSynchronize(ctx.stream));
    NL_REQUIRE(!hf, NLGPU_ERR_NUMERICAL, "zero pivot in the 1D LDL^T factorisation");
    ctx.od = st;
}

void nonstationary_1d_step(Ctx& ctx, double left_value, double right_value, bool sin_source, double* temperature) {
    NL_REQUIRE(ctx.od, NLGPU_ERR_STATE, "call nlgpu_nonstationary_1d_compute first");
    OneDimState& st = *ctx.od;
    const Problem1d& P = st.P;
    const size_t n = size_t(P.n);
    st.f.zero(ctx.stream);
    NL_LAUNCH(k_step_loads_1d, grid_for(P.E * st.L.nen, 256), 256, 0, ctx.stream, P, st.L, left_value, right_value,
              sin_source, st.f.p);
    NL_LAUNCH(k_step_rhs_1d, grid_for(P.n, 256), 256, 0, ctx.stream, P, st.dt, st.c.p, st.t.p, st.bound0.p,
              st.boundN.p, left_value, right_value, st.f.p);
    band_solve(ctx, P.n, P.bw, st.a.p, st.factor, st.f.p, true);
    std::swap(st.t, st.f);
    if (temperature) st.t.download(temperature, n, ctx.stream);
    NL_CUDA(cudaStreamSynchronize(ctx.stream));
}

void nonstationary_1d_temperature(Ctx& ctx, double* temperature) {
    NL_REQUIRE(ctx.od, NLGPU_ERR_STATE, "call nlgpu_nonstationary_1d_compute first");
    ctx.od->t.download(temperature, size_t(ctx.od->P.n), ctx.stream);
    NL_CUDA(cudaStreamSynchronize(ctx.stream));
}

i64 nonstationary_1d_nodes(const Ctx& ctx) { return ctx.od ? ctx.od->P.n : 0; }

void stationary_1d(Ctx& ctx, i64 elements, int order, double length, double radius, double local_weight, int influence,
                   double conductivity, double t_left, double q_right, bool sin_source, double* temperature) {
    const Line L = make_line(order);
    Problem1d P = make_problem_1d(elements, order, length, radius, local_weight, influence, conductivity);
    P.fk0 = 1; P.fk1 = 0;   // temperature on the left, flux on the right
    dbuf<double> band, bound0, f;
    dbuf<int> failed;
    band.resize(size_t(P.n * (P.bw + 1))); band.zero(ctx.stream);
    bound0.resize(size_t(P.n)); bound0.zero(ctx.stream);
    f.resize(size_t(P.n)); f.zero(ctx.stream);
    failed.resize(1); failed.zero(ctx.stream);
    NL_LAUNCH(k_assemble_1d, grid_for(P.E * (2 * P.nb + 1), 128), 128, 0, ctx.stream, P, L, band.p, bound0.p,
              static_cast<double*>(nullptr));
    NL_LAUNCH(k_rhs_1d, grid_for(P.E * L.nen, 256), 256, 0, ctx.stream, P, L, q_right, sin_source, f.p);
    NL_LAUNCH(k_first_kind_1d, grid_for(P.n, 256), 256, 0, ctx.stream, P.n, bound0.p, t_left, f.p, band.p);
    BandWork factor;
    band_factor(ctx, P.n, P.bw, band.p, f.p, factor, failed.p);
    band_solve(ctx, P.n, P.bw, band.p, factor, f.p, false);
    int hf = 0;
    NL_CUDA(cudaMemcpyAsync(&hf, failed.p, sizeof hf, cudaMemcpyDeviceToHost, ctx.stream));
    f.download(temperature, size_t(P.n), ctx.stream);
    NL_CUDA(cudaStreamSynchronize(ctx.stream));
    NL_REQUIRE(!hf, NLGPU_ERR_NUMERICAL, "zero pivot in the 1D LDL^T factorisation");
}

}  // namespace nlgpu
