// ILLT applied by Jacobi sweeps on the triangles of the factor (FP32).
//
// The preconditioner is the same incomplete Cholesky factor U (S A S ~ U^T U,
// eigen_preconditioner.hpp:56-57 through the Lin-More restatement of
// solver.cu); only the way its two triangular systems are solved changes.
// Instead of the exact level-scheduled substitution -- one dependent step per
// level, a few hundred to a few thousand per sweep on these meshes -- each
// triangle is solved approximately by k Jacobi iterations (Anzt, Chow and
// Dongarra, "Iterative sparse triangular solves for preconditioning",
// Euro-Par 2015):
//
//   U^T y = S r:  y_0 = D^-1 S r,  y_t+1 = D^-1 S r - (D^-1 N) y_t
//   U z = y_k:    z_0 = D^-1 y_k,  z_t+1 = D^-1 y_k - (D^-1 N^T) z_t,  result S z_k
//
// with D the diagonal of U and N the strict lower part of U^T.  D^-1 N is
// nilpotent, so k sweeps give the first k + 1 terms of the Neumann series of
// each triangular inverse, and k >= the level count reproduces the exact
// solve.  The truncated operator is S F^T F S with F lower triangular and
// nonsingular: symmetric positive definite, so it is a valid CG
// preconditioner; FP32 rounding makes it slightly non-symmetric, which the
// flexible CG of mixed.cu absorbs.
//
// Two forms.  k_jacobi_all runs the whole application as one cooperative launch:
// a CTA owns consecutive rows, and a sweep's values are stored as 64-bit words of
// the float and the step's number, which a reader polls until the number is
// there: no barrier, no launch between sweeps, and a row waits only for the rows
// of its band.  k_jacobi32 is one sweep per launch (thread per row), for systems
// whose sweeps are bound by bandwidth (JA_MAX_NEAR, JA_MAX_FAR).
#include "common.cuh"

#include <algorithm>

namespace nlgpu {

namespace {

constexpr int JB_THREADS = 256;

// val = u[src] / u_ii of the entry's row (0 for padding); the sliced-ELL
// layouts themselves are built by iltbuild.cu
__global__ void k_jacobi_values(i64 n, const i64* __restrict__ slice, const i64* __restrict__ src,
                                const i64* __restrict__ u_rp, const double* __restrict__ u, float* __restrict__ val) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
        const i64 sl = r >> 5, lane = r & 31, beg = slice[sl], w = (slice[sl + 1] - beg) >> 5;
        const double inv = 1.0 / u[u_rp[r]];
        for (i64 k = 0; k < w; ++k) {
            const i64 e = beg + 32 * k + lane;
            val[e] = src[e] >= 0 ? float(u[src[e]] * inv) : 0.0f;
        }
    }
}

// c_i = s_i / u_ii, dinv_i = 1 / u_ii
__global__ void k_jacobi_diag(i64 n, const i64* __restrict__ u_rp, const double* __restrict__ u,
                              const double* __restrict__ scale, float* __restrict__ c, float* __restrict__ dinv) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
        const double inv = 1.0 / u[u_rp[r]];
        c[r] = float(scale[r] * inv);
        dinv[r] = float(inv);
    }
}

// One Jacobi sweep on a scaled triangle T (thread per row):
//   out_i = o_i (bs_i base_i - sum_j T_ij ys_j y_j)
// where bs, ys and o are optional per-row scales (nullptr: 1).  Skipped once
// the solver has stopped (flags[S_DONE]).
__global__ void __launch_bounds__(JB_THREADS) k_jacobi32(i64 n, const i64* __restrict__ slice,
                                                          const int32_t* __restrict__ col, const float* __restrict__ val,
                                                          const float* __restrict__ base, const float* __restrict__ bs,
                                                          const float* __restrict__ y, const float* __restrict__ ys,
                                                          const float* __restrict__ o, float* __restrict__ out,
                                                          const double* __restrict__ flags) {
    if (flags && flags[S_DONE] != 0.0) return;
    const i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x;
    if (r >= n) return;
    const i64 sl = r >> 5, beg = slice[sl] + (r & 31), w = (slice[sl + 1] - slice[sl]) >> 5;
    float acc = 0.0f;
    if (ys) {
        for (i64 k = 0; k < w; ++k) {
            const int32_t j = __ldg(col + beg + 32 * k);
            acc += __ldg(val + beg + 32 * k) * (y[j] * __ldg(ys + j));
        }
    } else {
        for (i64 k = 0; k < w; ++k) {
            const int32_t j = __ldg(col + beg + 32 * k);
            acc += __ldg(val + beg + 32 * k) * y[j];
        }
    }
    float b = base[r];
    if (bs) b *= bs[r];
    float v = b - acc;
    if (o) v *= o[r];
    out[r] = v;
}

// The application in one launch (see the top).  Bound by the 2 k dependent steps,
// each a store and a load through L2 (a message between SMs of different dies
// takes about 0.45 us) and the row's sum; a gather of a value from far away moves a
// 32-byte sector past L1 for its 8 bytes, where k_jacobi32 gathers floats through L1.
// Which form: by the entries of a triangle, and by the share of them whose columns lie more
// than two CTAs away: 0 for rows numbered along the mesh, 0 to 1.2 % after cuthill_mckee of
// the local graph, 4.8 to 8.1 % after that of the nonlocal graph, 97 % at random.  (The mean
// reach of the rows is below a CTA after the nonlocal cuthill_mckee, and says nothing.)  At
// 250x250 8-node, nonlocal cuthill_mckee, an application takes 72 million instructions and
// 10 million L2 requests, by rows 28 and 3.4.
// Microseconds an FCG iteration (twelve sweeps and everything else), one launch per sweep -> this:
// (a nonlocal matrix passes through L2 between two applications, a local one leaves the factor there):
//   short rows     bilinear 500x500, 1.0 million entries    109 -> 97, nonlocal 247 -> 240
//                  bilinear 600x600, 1.4                    139 -> 138, nonlocal 306 -> 293
//   longer ones    8-node 200x200, 0.88                     97 -> 79, nonlocal 300 -> 286
//                  8-node 225x225, 1.1                      nonlocal 389 -> 383
//                  8-node 250x250, 1.4                      114 -> 118, nonlocal 519 -> 556
//                  the same with a radius of 0.02           227 -> 262
//                  8-node 200x200, local cuthill_mckee, 0.88    100 -> 88
//                  8-node 300x300, 2.0                      140 -> 151
//                  8-node 300x300, local cuthill_mckee, 2.0 148 -> 276
//   far ones       8-node 170x170, nonlocal cuthill_mckee, 0.64    186 -> 173
//                  the same numbered at random              357 -> 349
//                  bilinear 400x400 at random, 0.64         125 -> 124
//                  8-node 200x200, nonlocal cuthill_mckee, 0.88    313 -> 391
//                  bilinear 500x500 at random, 1.0          157 -> 170
//                  8-node 250x250, nonlocal cuthill_mckee, 1.4     603 -> 919
constexpr int JA_THREADS = 1024;
constexpr int JA_MIN_ROWS = 64;
constexpr i64 JA_MAX_NEAR = 1700000, JA_MAX_LONG = 1200000, JA_MAX_FAR = 700000;   // entries of a triangle
constexpr i64 JA_LONG_ROW = 5;    // a row's mean entries: 4 on bilinear meshes, 7 on 8-node ones
constexpr double JA_FAR_SHARE = 0.03;
constexpr i64 JA_MAX_ROWS = 400000;    // 361 201 measured
constexpr int JA_MAX_SWEEPS = 32;
constexpr int JA_BATCH = 4;       // gathers in flight per lane
constexpr int JA_POLLS = 4096;

__device__ __forceinline__ unsigned long long ja_globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void ja_put(unsigned long long* p, float v, unsigned tag) {
    const unsigned long long w = (static_cast<unsigned long long>(tag) << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}

__device__ __forceinline__ unsigned long long ja_get(const unsigned long long* p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}

// a wait that runs out marks the CTA, which then waits no more; the host sees *error
__device__ __noinline__ unsigned long long ja_wait_long(const unsigned long long* p, unsigned tag, volatile int* gave_up,
                                                        int* error, unsigned long long limit_ns) {
    const unsigned long long t0 = ja_globaltimer();
    unsigned long long w = ja_get(p);
    while (unsigned(w >> 32) != tag && !*gave_up) {
        if (ja_globaltimer() - t0 > limit_ns) {
            atomicExch(error, 1);
            *gave_up = 1;
        }
        w = ja_get(p);
    }
    return w;
}

struct JacobiAll {
    i64 n;
    int rows;                 // per CTA, a multiple of 32
    int sweeps, lg;           // sweeps per triangle, log2 of the lanes per row
    const i64 *slo, *sup;     // slices, columns and values of both triangles
    const int32_t *clo, *cup;
    const float *vlo, *vup;
    const float *r, *c, *dinv, *scale;
    float* z;
    unsigned long long* steps;   // [sweeps + 1][n]
    unsigned* tags;              // [gridDim.x] last number each CTA used
    int* error;
    unsigned long long limit_ns;
};

// POLLS: of a value before the clock is read (a variant of its own for a wait limit of 0:
// with the number in a register a batch of 163 000 rows took 14 % longer)
template<int POLLS>
__global__ void __launch_bounds__(JA_THREADS) k_jacobi_all(JacobiAll a, const double* __restrict__ flags) {
    extern __shared__ float ja_base[];
    __shared__ int gave_up;
    if (flags && flags[S_DONE] != 0.0) return;
    const i64 r0 = i64(blockIdx.x) * a.rows;
    const int rows = int(min(a.n, r0 + a.rows) - r0);
    const int lane = threadIdx.x & 31, g = 1 << a.lg, sub = lane & (g - 1), per = 32 >> a.lg;
    unsigned tag = a.tags[blockIdx.x] + 1;
    if (threadIdx.x == 0) gave_up = 0;
    for (int i = threadIdx.x; i < rows; i += JA_THREADS) {
        const float y = a.c[r0 + i] * a.r[r0 + i];
        ja_base[i] = y;
        ja_put(a.steps + r0 + i, y, tag);
    }
    __syncthreads();
    // the rows a warp takes are the same in every sweep, and a row's own values pass
    // between them in its lanes' warp: no barrier
    for (int s = 1; s <= 2 * a.sweeps; ++s) {
        const bool upper = s > a.sweeps;
        const int t = upper ? s - a.sweeps : s;           // sweep of this triangle
        const bool last = t == a.sweeps;
        const i64* slice = upper ? a.sup : a.slo;
        const int32_t* cols = upper ? a.cup : a.clo;
        const float* vals = upper ? a.vup : a.vlo;
        // backward sweep t writes step t again: a row has read the forward results of every
        // row above it by then, and those are the rows that read its forward values
        const unsigned long long* in = a.steps + size_t(upper && t == 1 ? a.sweeps : t - 1) * size_t(a.n);
        unsigned long long* out = a.steps + size_t(t) * size_t(a.n);
        for (int i0 = int(threadIdx.x >> 5) * per; i0 < rows; i0 += (JA_THREADS / 32) * per) {
            const int i = i0 + (lane >> a.lg);
            const i64 row = r0 + i;
            float acc = 0.0f;
            if (i < rows) {
                const i64 b = __ldg(slice + (row >> 5));
                const int w = int((__ldg(slice + (row >> 5) + 1) - b) >> 5);
                const int32_t* col = cols + b + (row & 31);
                const float* val = vals + b + (row & 31);
                for (int k = sub; k < w; k += JA_BATCH * g) {
                    unsigned long long y[JA_BATCH];
                    int32_t j[JA_BATCH];
                    float v[JA_BATCH];
#pragma unroll
                    for (int u = 0; u < JA_BATCH; ++u)
                        if (k + u * g < w) {
                            j[u] = __ldg(col + 32 * (k + u * g));
                            v[u] = __ldg(val + 32 * (k + u * g));
                            y[u] = ja_get(in + j[u]);
                        }
#pragma unroll
                    for (int u = 0; u < JA_BATCH; ++u)
                        if (k + u * g < w) {
                            for (int tries = 0; unsigned(y[u] >> 32) != tag; ++tries) {
                                if (tries == POLLS) {
                                    y[u] = ja_wait_long(in + j[u], tag, &gave_up, a.error, a.limit_ns);
                                    break;
                                }
                                y[u] = ja_get(in + j[u]);
                            }
                            acc += v[u] * __uint_as_float(unsigned(y[u]));
                        }
                }
            }
            for (int o = g >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (i < rows && sub == 0) {
                float v = ja_base[i] - acc;
                if (!last) {
                    ja_put(out + row, v, tag + 1);
                } else if (!upper) {
                    v *= a.dinv[row];
                    ja_base[i] = v;   // the backward sweeps' base, read by this lane only
                    ja_put(out + row, v, tag + 1);
                } else {
                    a.z[row] = v * a.scale[row];
                }
            }
        }
        ++tag;
    }
    if (threadIdx.x == 0) a.tags[blockIdx.x] = tag;
}

void sweep(Ctx& ctx, i64 n, const JacobiSlab& s, const float* base, const float* bs, const float* y, const float* ys,
           const float* o, float* out, const double* flags) {
    NL_LAUNCH(k_jacobi32, unsigned((n + JB_THREADS - 1) / JB_THREADS), JB_THREADS, 0, ctx.stream, n, s.slice.p,
              s.col.p, s.val.p, base, bs, y, ys, o, out, flags);
}

}  // namespace

void jacobi_fill(Ctx& ctx, IncompleteCholesky& ic) {
    const i64 n = ic.n;
    for (JacobiSlab* s : {&ic.jlo, &ic.jup})
        NL_LAUNCH(k_jacobi_values, grid_for(n, 256), 256, 0, ctx.stream, n, s->slice.p, s->src.p, ic.rp.p, ic.u.p,
                  s->val.p);
    NL_LAUNCH(k_jacobi_diag, grid_for(n, 256), 256, 0, ctx.stream, n, ic.rp.p, ic.u.p, ic.scale.p, ic.jc.p, ic.jdinv.p);
}

i64 jacobi_cta_rows(i64 n) {
    int dev = 0, sms = 0;
    NL_CUDA(cudaGetDevice(&dev));
    NL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::max<i64>(JA_MIN_ROWS, ((n + sms - 1) / sms + 31) / 32 * 32);
}

void check_sweeps(Ctx& ctx) {
    if (!ctx.sweep_error.n) return;
    int err = 0;
    ctx.sweep_error.download(&err, 1, ctx.stream);
    NL_CUDA(cudaStreamSynchronize(ctx.stream));
    if (err == 0) return;
    ctx.sweep_error.zero(ctx.stream);
    throw error{NLGPU_ERR_TIMEOUT, "a triangular sweep gave up waiting for its data"};
}

void jacobi_apply32(Ctx& ctx, IncompleteCholesky& ic, int sweeps, const float* r, float* z, const double* flags) {
    NL_REQUIRE(sweeps >= 1, NLGPU_ERR_ARG, "at least one Jacobi sweep per triangle");
    const i64 n = ic.n;
    const i64 rows = jacobi_cta_rows(n);
    const i64 entries = ic.nnz - n;
    const i64 most = ic.far_share > JA_FAR_SHARE ? JA_MAX_FAR : entries > JA_LONG_ROW * n ? JA_MAX_LONG : JA_MAX_NEAR;
    if (n <= JA_MAX_ROWS && entries <= most && sweeps <= JA_MAX_SWEEPS) {
        const unsigned grid = unsigned((n + rows - 1) / rows);
        const size_t words = size_t(sweeps + 1) * size_t(n);
        // the CTAs' numbers go on from application to application; another split starts
        // afresh (outside any capture: a solve's first application is eager)
        if (ic.jsteps.n < words || ic.jsplit_n != n || ic.jsplit_rows != rows) {
            ic.jsteps.reserve(words);
            ic.jtags.reserve(grid);
            ic.jsteps.zero(ctx.stream);
            ic.jtags.zero(ctx.stream);
            ic.jsplit_n = n;
            ic.jsplit_rows = rows;
        }
        ctx.sweep_error.reserve(1);
        JacobiAll a{};
        a.n = n; a.rows = int(rows); a.sweeps = sweeps;
        while (a.lg < 2 && (rows << (a.lg + 1)) <= JA_THREADS && (2 << a.lg) <= ic.jlo.max_width) ++a.lg;
        a.slo = ic.jlo.slice.p; a.clo = ic.jlo.col.p; a.vlo = ic.jlo.val.p;
        a.sup = ic.jup.slice.p; a.cup = ic.jup.col.p; a.vup = ic.jup.val.p;
        a.r = r; a.c = ic.jc.p; a.dinv = ic.jdinv.p; a.scale = ic.scale32.p; a.z = z;
        a.steps = ic.jsteps.p; a.tags = ic.jtags.p; a.error = ctx.sweep_error.p;
        a.limit_ns = static_cast<unsigned long long>(ctx.wait_limit_us) * 1000ull;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(JA_THREADS);
        cfg.dynamicSmemBytes = size_t(rows) * sizeof(float);
        cfg.stream = ctx.stream;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        NL_CUDA(cudaLaunchKernelEx(&cfg, ctx.wait_limit_us > 0 ? k_jacobi_all<JA_POLLS> : k_jacobi_all<0>, a, flags));
        count_launch();
        return;
    }
    float* t[2] = {ic.jt0.p, ic.jt1.p};
    // forward: y_t+1 = c r - L y_t from y_0 = c r; the last sweep scales by 1 / u_ii
    const float* prev = r;
    const float* prev_scale = ic.jc.p;
    for (int s = 1; s <= sweeps; ++s) {
        float* out = s == sweeps ? ic.jy.p : t[s & 1];
        sweep(ctx, n, ic.jlo, r, ic.jc.p, prev, prev_scale, s == sweeps ? ic.jdinv.p : nullptr, out, flags);
        prev = out;
        prev_scale = nullptr;
    }
    // backward: z_t+1 = y~ - U z_t from z_0 = y~; the last sweep scales by s_i
    prev = ic.jy.p;
    for (int s = 1; s <= sweeps; ++s) {
        float* out = s == sweeps ? z : t[s & 1];
        sweep(ctx, n, ic.jup, ic.jy.p, nullptr, prev, nullptr, s == sweeps ? ic.scale32.p : nullptr, out, flags);
        prev = out;
    }
}

}  // namespace nlgpu
