// FP64 conjugate gradient as one persistent kernel: the whole solve (first
// residual, iterations, true residual, restarts) in one launch, with the ILLT
// applied by Jacobi sweeps on its triangles.
//
// Reference: slae::conjugate_gradient::solve (conjugate_gradient.hpp:48-79) with
// eigen_ILLT_preconditioner (eigen_preconditioner.hpp:57) or the identity.
//
// What bounds it.  One iteration reads the matrix once (FP64 SpMV) and each
// triangle of the factor once per sweep; on the sizes the FP64 path is used for
// (10^2 .. 10^5 rows, the matrix in L2) that is 1 to 30 us of work, so the
// dependent steps decide: about twenty sweeps, two reductions and the product.
//
// Triangular solves.  U^T y = S r and U z = y are solved by k Jacobi sweeps per
// triangle in FP64 (Anzt, Chow, Dongarra, "Iterative sparse triangular solves
// for preconditioning", Euro-Par 2015; jacobi.cu has the FP32 form): the first
// k + 1 terms of each triangular inverse's Neumann series, S F^T F S with F lower
// triangular and nonsingular, so symmetric positive definite and constant over
// the solve.  k comes from the factor itself: before the first iteration the
// forward sweeps run on a vector of +-1 until a sweep changes the iterate by at
// most PCG_SWEEP_TOL of its norm (3e-3: 9 to 14 sweeps on finite-element factors,
// at most one iteration in forty more than the exact solves; 4 fixed sweeps cost
// 10 to 35 % more iterations).  A factor that needs more than PCG_MAX_SWEEPS goes back to
// the exact level-scheduled solves (solver.cu).
//
// Dependent steps.  A CTA owns consecutive rows (all CTAs resident: cooperative
// launch).  The values that sweeps and reductions pass between CTAs carry
// their step's number: a double is stored as two 64-bit words, each half the
// bits and a 32-bit tag, and a reader polls the value it needs until the tag is
// there.  A step then costs one store and one load through L2 with no
// fence, no barrier and no wait for CTAs that it does not depend on (a sweep's
// rows need only the rows of their band).  Only the search direction p, which
// the product gathers from everywhere, goes through a fence and a barrier.
// Every wait is bounded and reports a timeout.
//   Measured (microseconds an iteration with the ILLT, GB300): 252 rows (17x13
// bilinear) 29, a counter barrier after every phase 54, the exact sweeps in one
// CTA and separate launches 100; 14 896 rows (151x97, local) 27 / 60 / 390;
// 11 538 rows of 570 (71x53 8-node) 62 / 127 / 800.  Identity, 5 499 rows of 330
// (48x37 8-node): 14.6 against 45.
// Reductions: one partial per CTA, re-added in a fixed order by one warp of every
// CTA, so all CTAs take the same decisions.
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace nlgpu {

namespace {

constexpr int PCG_THREADS = 512;
constexpr int PCG_WARPS = PCG_THREADS / 32;
constexpr int PCG_MAX_SWEEPS = 24;
constexpr double PCG_SWEEP_TOL = 3e-3;
constexpr int PCG_MIN_ROWS = 8;             // rows per CTA at least
constexpr int PCG_OWN_ROWS = 1024;          // a CTA's vectors stay in shared memory up to this many rows
constexpr i64 PCG_ITERS_PER_LAUNCH = 512;   // bounds a launch's duration
constexpr int PCG_RESTARTS = 4;
// every CTA polls every partial sum: each in a 128-byte line of its own, or the
// polls of 152 CTAs queue on a few lines (an all-CTA sum took 5 us side by side)
constexpr int SUM_STRIDE = 8;
constexpr int SUM_BATCH = 5;
constexpr unsigned long long PCG_WAIT_LIMIT_NS = 2000000000ull;
// scalars left for the host and the next launch
enum { PS_BB = 0, PS_RR, PS_RZ, PS_ITERS, PS_DONE, PS_SWEEPS, PS_EXACT, PS_RESTART, PS_TAG, PS_COUNT };
// a CTA's own vectors
enum { OV_X = 0, OV_R, OV_P, OV_Q, OV_Z, OV_BASE, OV_YF, OV_C, OV_DINV, OV_SCALE, OV_COUNT };

struct PcgTriangle {
    const i64* slice;
    const int32_t* col;
    const double* val;
};

struct PcgArgs {
    i64 n;
    int rows;                 // rows per CTA
    const i64* rp;
    const int32_t* col;
    const double* val;
    int lg;                   // log2 of the lanes per row of the product
    const double* b;
    double *x, *r, *p;
    double* own;              // [OV_COUNT][gridDim.x * rows] when the vectors do not fit shared memory
    PcgTriangle lo, up;       // ILLT: the scaled triangles, c = s / u_ii, 1 / u_ii, s
    const double *c, *dinv, *scale;
    ulonglong2* steps;        // [PCG_MAX_SWEEPS + 1][n] tagged sweep values
    int lgs;                  // log2 of the lanes per row of a sweep
    int staged, wlo, wup;     // the CTA's entries are copied to shared memory, wlo / wup per row
    ulonglong2* sums;         // [2][2][gridDim.x][SUM_STRIDE] tagged partial sums
    double* state;
    unsigned* counter;        // of the barriers
    int* error;
    double tol2;
    i64 max_iterations, iterations_here;
    int x_zero, resume;
};

__device__ __forceinline__ unsigned long long pcg_globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// tagged values: both 64-bit words are single accesses, so a reader that finds
// the tag in a word has that word's half of the value
__device__ __forceinline__ void put_tagged(ulonglong2* p, double v, unsigned tag) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
    const unsigned long long t = static_cast<unsigned long long>(tag) << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"((b & 0xffffffffull) | t), "l"((b >> 32) | t)
                 : "memory");
}

__device__ __forceinline__ ulonglong2 get_words(const ulonglong2* p) {
    ulonglong2 w;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
    return w;
}

__device__ __forceinline__ bool has_tag(ulonglong2 w, unsigned tag) {
    return unsigned(w.x >> 32) == tag && unsigned(w.y >> 32) == tag;
}

__device__ __forceinline__ double value_of(ulonglong2 w) {
    return __longlong_as_double(static_cast<long long>((w.y << 32) | (w.x & 0xffffffffull)));
}

// polls until the tag is there; a wait that runs out marks the CTA, which then
// waits no more and leaves the kernel at its next reduction.  The clock is read
// only after many polls (reading it costs as much as the value's way through L2).
__device__ __noinline__ ulonglong2 wait_long(const ulonglong2* p, unsigned tag, volatile int* gave_up, int* error) {
    const unsigned long long t0 = pcg_globaltimer();
    ulonglong2 w = get_words(p);
    while (!has_tag(w, tag) && !*gave_up) {
        if (pcg_globaltimer() - t0 > PCG_WAIT_LIMIT_NS) {
            atomicExch(error, 1);
            *gave_up = 1;
        }
        w = get_words(p);
    }
    return w;
}

__device__ __forceinline__ ulonglong2 wait_tagged(const ulonglong2* p, unsigned tag, volatile int* gave_up, int* error) {
    ulonglong2 w = get_words(p);
    for (int tries = 0; !has_tag(w, tag); ++tries) {
        if (tries == 4096) return wait_long(p, tag, gave_up, error);
        w = get_words(p);
    }
    return w;
}

struct Cta {
    int rows;                 // of this CTA
    i64 r0;
    double* own;              // own vectors, by local row
    size_t own_stride;
    __device__ __forceinline__ double* v(int k) const { return own + size_t(k) * own_stride; }
    const double *vlo, *vup;  // staged: entry k of local row i at k * stride + i
    const int32_t *clo, *cup;
    const int32_t *nlo, *nup; // staged: entries of each row
    int stride;
    const int* first;         // first entry of each own row, from the CTA's first (null: read rp)
    i64 entry0;
    double* sh;               // [2][2][PCG_WARPS]
    volatile int* gave_up;
    unsigned epoch, syncs;    // reductions and barriers so far
};

// Sums of N per-lane values over every CTA; thread 0 of each gets them and runs
// `post` on them (GB300's FP64 pipe takes 16 cycles for a warp's instruction, so the
// scalars are formed by one thread and read from shared memory), everybody sees
// what it wrote.  `any` (uniform in a warp): its lanes hold something; only the
// first `used` warps' may.  False when a wait ran out.
template<int N, class F>
__device__ __forceinline__ bool all_sum(const PcgArgs& a, Cta& c, double (&v)[N], bool any, int used, F&& post) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ++c.epoch;
    double* sh = c.sh + (c.epoch & 1) * 2 * PCG_WARPS;
    ulonglong2* out = a.sums + size_t(c.epoch & 1) * 2 * gridDim.x * SUM_STRIDE;
#pragma unroll
    for (int s = 0; s < N; ++s) {
        if (any) v[s] = warp_sum(v[s]);
        if (lane == 0) sh[s * PCG_WARPS + warp] = any ? v[s] : 0.0;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int s = 0; s < N; ++s) {
            double t = lane < PCG_WARPS ? sh[s * PCG_WARPS + lane] : 0.0;
            for (int o = 1; o < used; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) put_tagged(out + (size_t(s) * gridDim.x + blockIdx.x) * SUM_STRIDE, t, c.epoch);
        }
        double total[N];
#pragma unroll
        for (int s = 0; s < N; ++s) total[s] = 0.0;
        for (unsigned k0 = 0; k0 < gridDim.x; k0 += 32 * SUM_BATCH) {
            // a lane's words are polled together (one after another cost 0.9 us more)
            ulonglong2 w[SUM_BATCH][N];
            auto word = [&](int u, int s) {
                return out + (size_t(s) * gridDim.x + min(k0 + lane + 32 * u, gridDim.x - 1)) * SUM_STRIDE;
            };
#pragma unroll
            for (int u = 0; u < SUM_BATCH; ++u)
#pragma unroll
                for (int s = 0; s < N; ++s) w[u][s] = get_words(word(u, s));
            for (int tries = 0;; ++tries) {
                bool all = true;
#pragma unroll
                for (int u = 0; u < SUM_BATCH; ++u)
#pragma unroll
                    for (int s = 0; s < N; ++s)
                        if (!has_tag(w[u][s], c.epoch)) {
                            all = false;
                            w[u][s] = tries < 4096 ? get_words(word(u, s))
                                                   : wait_long(word(u, s), c.epoch, c.gave_up, a.error);
                        }
                if (__all_sync(0xffffffffu, all || *c.gave_up)) break;
            }
#pragma unroll
            for (int u = 0; u < SUM_BATCH; ++u)
#pragma unroll
                for (int s = 0; s < N; ++s)
                    if (k0 + lane + 32 * u < gridDim.x) total[s] += value_of(w[u][s]);
        }
#pragma unroll
        for (int s = 0; s < N; ++s) total[s] = warp_sum(total[s]);
        if (lane == 0) post(total);
    }
    __syncthreads();
    return *c.gave_up == 0;
}

// every CTA's global stores before it are visible to every CTA's loads after it
__device__ __forceinline__ bool all_sync(const PcgArgs& a, Cta& c) {
    ++c.syncs;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = c.syncs * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counter) : "memory");
        unsigned seen = 0;
        unsigned long long t0 = 0;
        for (int tries = 0;; ++tries) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.counter) : "memory");
            if (seen >= target || *c.gave_up) break;
            if (tries < 4096) continue;
            if (t0 == 0) t0 = pcg_globaltimer();
            else if (pcg_globaltimer() - t0 > PCG_WAIT_LIMIT_NS) {
                atomicExch(a.error, 1);
                *c.gave_up = 1;
            }
        }
    }
    __syncthreads();
    return *c.gave_up == 0;
}

// own q = (A v) on the CTA's rows, 2^lg lanes per row; neighbouring lanes take
// neighbouring entries, so a gather reads runs of columns.  DENSE: rows of LONG_ROW << lg
// entries and more (of a caller's matrix) take the whole warp; a variant of its own,
// since the test alone cost the others 2.5 % of an iteration.
template<bool DENSE>
__device__ __forceinline__ void pcg_spmv(const PcgArgs& a, const Cta& c, const double* v) {
    const int lane = threadIdx.x & 31, g = 1 << a.lg, sub = lane & (g - 1), per = 32 >> a.lg;
    for (int i0 = int(threadIdx.x >> 5) * per; i0 < c.rows; i0 += PCG_WARPS * per) {
        const int i = i0 + (lane >> a.lg);
        double s = 0.0, s2 = 0.0;
        bool dense = false;
        if (i < c.rows) {
            const i64 b = c.first ? c.entry0 + c.first[i] : a.rp[c.r0 + i];
            const int len = c.first ? c.first[i + 1] - c.first[i] : int(a.rp[c.r0 + i + 1] - b);
            if constexpr (DENSE) dense = len >= LONG_ROW << a.lg;
            const int32_t* col = a.col + b;
            const double* val = a.val + b;
            int k = dense ? len : sub;
            for (; k + 3 * g < len; k += 4 * g) {
                const int32_t j0 = __ldg(col + k), j1 = __ldg(col + k + g), j2 = __ldg(col + k + 2 * g),
                              j3 = __ldg(col + k + 3 * g);
                const double w0 = __ldg(val + k), w1 = __ldg(val + k + g), w2 = __ldg(val + k + 2 * g),
                             w3 = __ldg(val + k + 3 * g);
                s = fma(w0, v[j0], s);
                s2 = fma(w1, v[j1], s2);
                s = fma(w2, v[j2], s);
                s2 = fma(w3, v[j3], s2);
            }
            for (; k < len; k += g) s = fma(__ldg(val + k), v[__ldg(col + k)], s);
            s += s2;
        }
        for (int o = g >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (i < c.rows && sub == 0) c.v(OV_Q)[i] = s;
        if constexpr (DENSE)
            for (unsigned rows = __ballot_sync(0xffffffffu, dense && sub == 0); rows; rows &= rows - 1) {
                const int d = i0 + ((__ffs(rows) - 1) >> a.lg);
                const double t = dense_row(a.col, a.val, v, a.rp[c.r0 + d], a.rp[c.r0 + d + 1]);
                if (lane == 0) c.v(OV_Q)[d] = t;
            }
    }
    __syncthreads();
}

// One Jacobi sweep over the CTA's rows: base - T y, times o, where y are the values
// `in` with tag `tin`; the result goes to `out` with tag `tout` (out null: kept by
// the CTA only) and to the CTA's vector `keep` (may be null).  NORM: returns
// this lane's |result - y|^2 and |result|^2 over the rows that have entries.
constexpr int SWEEP_BATCH = 2;   // gathers in flight per lane (4 spills registers: 10 to 15 % slower)
template<bool NORM>
__device__ __forceinline__ double2 pcg_sweep(const PcgArgs& a, const Cta& c, bool upper, const double* base,
                                             const double* o, const ulonglong2* in, unsigned tin, ulonglong2* out,
                                             unsigned tout, double* keep) {
    const int lane = threadIdx.x & 31, g = 1 << a.lgs, sub = lane & (g - 1), per = 32 >> a.lgs;
    const PcgTriangle& t = upper ? a.up : a.lo;
    const double* sval = upper ? c.vup : c.vlo;
    const int32_t* scol = upper ? c.cup : c.clo;
    const int32_t* scount = upper ? c.nup : c.nlo;
    double2 acc = make_double2(0.0, 0.0);
    for (int i0 = int(threadIdx.x >> 5) * per; i0 < c.rows; i0 += PCG_WARPS * per) {
        const int i = i0 + (lane >> a.lgs);
        const i64 row = c.r0 + i;
        double s = 0.0;
        int width = 0;
        if (i < c.rows) {
            i64 first = 0;
            int step = c.stride;
            const double* val = sval + i;
            const int32_t* col = scol + i;
            if (a.staged) {
                width = scount[i];
            } else {
                first = t.slice[row >> 5];
                width = int((t.slice[(row >> 5) + 1] - first) >> 5);
                val = t.val + first + (row & 31);
                col = t.col + first + (row & 31);
                step = 32;
            }
            for (int k = sub; k < width; k += SWEEP_BATCH * g) {
                ulonglong2 w[SWEEP_BATCH];
                int32_t j[SWEEP_BATCH];
#pragma unroll
                for (int u = 0; u < SWEEP_BATCH; ++u)
                    if (k + u * g < width) {
                        j[u] = col[(k + u * g) * step];
                        w[u] = get_words(in + j[u]);
                    }
#pragma unroll
                for (int u = 0; u < SWEEP_BATCH; ++u)
                    if (k + u * g < width) {
                        if (!has_tag(w[u], tin)) w[u] = wait_tagged(in + j[u], tin, c.gave_up, a.error);
                        s = fma(val[(k + u * g) * step], value_of(w[u]), s);
                    }
            }
        }
        for (int h = g >> 1; h > 0; h >>= 1) s += __shfl_xor_sync(0xffffffffu, s, h);
        if (i < c.rows && sub == 0) {
            double v = base[i] - s;
            if constexpr (NORM) {
                if (width > 0) {
                    const double y = value_of(wait_tagged(in + row, tin, c.gave_up, a.error)), d = v - y;
                    acc.x = fma(d, d, acc.x);
                    acc.y = fma(v, v, acc.y);
                }
            }
            if (o) v *= o[i];
            if (out) put_tagged(out + row, v, tout);
            if (keep) keep[i] = v;
        }
    }
    return acc;
}

template<bool ILLT, bool DENSE>
__global__ void __launch_bounds__(PCG_THREADS, 1) k_pcg(PcgArgs a) {
    extern __shared__ __align__(16) unsigned char pcg_smem[];
    __shared__ double sh[4 * PCG_WARPS];
    __shared__ double bb, rz, rr, alpha, beta;   // written by thread 0
    __shared__ int gave_up, stop, done;
    const int tid = threadIdx.x;
    Cta c{};
    c.r0 = min(a.n, i64(blockIdx.x) * a.rows);
    c.rows = int(min(a.n, c.r0 + a.rows) - c.r0);
    c.stride = a.rows;
    c.sh = sh;
    c.gave_up = &gave_up;
    if (tid == 0) {
        gave_up = stop = done = 0;
        bb = rz = rr = 0.0;
    }
    unsigned char* free_smem = pcg_smem;
    c.own = a.own ? a.own + size_t(blockIdx.x) * a.rows : reinterpret_cast<double*>(pcg_smem);
    c.own_stride = a.own ? size_t(gridDim.x) * a.rows : size_t(a.rows);
    c.entry0 = a.rp[c.r0];
    if (!a.own) {
        free_smem += size_t(OV_COUNT) * a.rows * sizeof(double);
        int* first = reinterpret_cast<int*>(free_smem);
        for (int i = tid; i <= c.rows; i += PCG_THREADS) first[i] = int(a.rp[c.r0 + i] - c.entry0);
        c.first = first;
        free_smem += (size_t(a.rows) + 2) / 2 * 8;
    }

    auto each = [&](auto&& f) {
        for (int i = tid; i < c.rows; i += PCG_THREADS) f(i, c.r0 + i);
    };
    if constexpr (ILLT) {
        if (a.staged) {
            double* vlo = reinterpret_cast<double*>(free_smem);
            double* vup = vlo + size_t(a.wlo) * a.rows;
            int32_t* clo = reinterpret_cast<int32_t*>(vup + size_t(a.wup) * a.rows);
            int32_t* cup = clo + size_t(a.wlo) * a.rows;
            int32_t* nlo = cup + size_t(a.wup) * a.rows;
            int32_t* nup = nlo + a.rows;
            // a row's padding entries (its own column) come last
            auto copy = [&](const PcgTriangle& t, int i, i64 row, double* val, int32_t* col, int32_t* count) {
                const i64 first = t.slice[row >> 5];
                const int w = int((t.slice[(row >> 5) + 1] - first) >> 5);
                int real = 0;
                for (int k = 0; k < w; ++k) {
                    const int32_t j = t.col[first + 32 * k + (row & 31)];
                    if (j == int32_t(row)) break;
                    col[k * a.rows + i] = j;
                    val[k * a.rows + i] = t.val[first + 32 * k + (row & 31)];
                    ++real;
                }
                count[i] = real;
            };
            each([&](int i, i64 row) {
                copy(a.lo, i, row, vlo, clo, nlo);
                copy(a.up, i, row, vup, cup, nup);
            });
            c.vlo = vlo; c.clo = clo; c.nlo = nlo;
            c.vup = vup; c.cup = cup; c.nup = nup;
        }
        each([&](int i, i64 row) {
            c.v(OV_C)[i] = a.c[row];
            c.v(OV_DINV)[i] = a.dinv[row];
            c.v(OV_SCALE)[i] = a.scale[row];
        });
    }
    __syncthreads();

    const bool has_rows = (tid & ~31) < c.rows;
    const int row_warps = min(PCG_WARPS, (c.rows + 31) >> 5);   // `each` fills the first warps
    unsigned tag = a.resume ? unsigned(a.state[PS_TAG]) : 0u;
    int sweeps = a.resume ? int(a.state[PS_SWEEPS]) : 0;
    auto step = [&](int s) { return a.steps + size_t(s) * size_t(a.n); };

    if constexpr (ILLT) {
        if (!a.resume) {   // sweeps needed by this factor, from a vector of +-1
            each([&](int i, i64 row) {
                unsigned h = unsigned(row) * 2654435761u;
                h ^= h >> 15;
                const double v = (h & 1u) ? 1.0 : -1.0;
                c.v(OV_BASE)[i] = v;
                put_tagged(step(0) + row, v, tag + 1);
            });
            __syncthreads();
            ++tag;
            while (!stop && sweeps < PCG_MAX_SWEEPS) {
                const double2 nv = pcg_sweep<true>(a, c, false, c.v(OV_BASE), nullptr, step(sweeps), tag, step(sweeps + 1),
                                                   tag + 1, nullptr);
                ++tag;
                ++sweeps;
                double s[2] = {nv.x, nv.y};
                if (!all_sum<2>(a, c, s, true, PCG_WARPS, [&](const double* t) { stop = t[0] <= PCG_SWEEP_TOL * PCG_SWEEP_TOL * t[1]; })) return;
            }
            if (!stop) {
                if (blockIdx.x == 0 && tid == 0) { a.state[PS_EXACT] = 1.0; a.state[PS_DONE] = 1.0; }
                return;
            }
        }
    }

    // own z = M^-1 r from the own c r in BASE, already published as step 0 with
    // `tag`.  Forward sweep s writes step s, its last one the scaled y; backward sweep s
    // writes step s again: a row has read the y of every row above it by then, and
    // those are the rows that read its forward values.
    auto precondition = [&]() {
        if constexpr (ILLT) {
            for (int s = 1; s <= sweeps; ++s) {
                const bool last = s == sweeps;
                pcg_sweep<false>(a, c, false, c.v(OV_BASE), last ? c.v(OV_DINV) : nullptr, step(s - 1), tag, step(s), tag + 1,
                                 last ? c.v(OV_YF) : nullptr);
                ++tag;
            }
            const ulonglong2* in = step(sweeps);
            for (int s = 1; s <= sweeps; ++s) {
                const bool last = s == sweeps;
                pcg_sweep<false>(a, c, true, c.v(OV_YF), last ? c.v(OV_SCALE) : nullptr, in, tag, last ? nullptr : step(s),
                                 tag + 1, last ? c.v(OV_Z) : nullptr);
                in = step(s);
                ++tag;
            }
            __syncthreads();
        }
    };

    i64 it = 0, here = 0;
    int restart = 0;
    if (a.resume) {
        it = i64(a.state[PS_ITERS]);
        restart = int(a.state[PS_RESTART]);
        if (tid == 0) {
            bb = a.state[PS_BB];
            rz = a.state[PS_RZ];
        }
        each([&](int i, i64 row) {
            c.v(OV_X)[i] = a.x[row];
            c.v(OV_R)[i] = a.r[row];
            c.v(OV_P)[i] = a.p[row];
        });
        if (!all_sync(a, c)) return;   // every CTA has read the state before it is written again
    } else {
        each([&](int i, i64 row) { c.v(OV_X)[i] = a.x_zero ? 0.0 : a.x[row]; });
    }
    bool fresh = !a.resume;
    for (; restart < PCG_RESTARTS; ++restart) {
        if (fresh) {
            // r = b - A x, z = M^-1 r, p = z
            const bool zero = a.x_zero && restart == 0;
            if (!zero) pcg_spmv<DENSE>(a, c, a.x);
            double s[2] = {0.0, 0.0};
            each([&](int i, i64 row) {
                const double bi = a.b[row], ri = zero ? bi : bi - c.v(OV_Q)[i];
                c.v(OV_R)[i] = ri;
                if constexpr (ILLT) {
                    const double y = c.v(OV_C)[i] * ri;
                    c.v(OV_BASE)[i] = y;
                    put_tagged(step(0) + row, y, tag + 1);
                }
                s[0] = fma(ri, ri, s[0]);
                s[1] = fma(bi, bi, s[1]);
            });
            ++tag;
            if (!all_sum(a, c, s, has_rows, row_warps, [&](const double* t) {
                    rr = rz = t[0];
                    bb = t[1];
                    done = bb == 0.0 || rr <= a.tol2 * bb || !isfinite(rr);
                    stop = 0;
                })) return;
            if (done) break;
            if constexpr (ILLT) {
                precondition();
                double d[1] = {0.0};
                each([&](int i, i64) { d[0] = fma(c.v(OV_R)[i], c.v(OV_Z)[i], d[0]); });
                if (!all_sum(a, c, d, has_rows, row_warps, [&](const double* t) { rz = t[0]; })) return;
            }
            each([&](int i, i64 row) {
                const double v = c.v(ILLT ? OV_Z : OV_R)[i];
                c.v(OV_P)[i] = v;
                a.p[row] = v;
            });
            if (!all_sync(a, c)) return;
        }
        fresh = true;
        while (!stop && here < a.iterations_here) {
            pcg_spmv<DENSE>(a, c, a.p);
            double pq[1] = {0.0};
            each([&](int i, i64) { pq[0] = fma(c.v(OV_P)[i], c.v(OV_Q)[i], pq[0]); });
            if (!all_sum(a, c, pq, has_rows, row_warps, [&](const double* t) { alpha = rz / t[0]; })) return;
            double t[2] = {0.0, 0.0};
            each([&](int i, i64 row) {
                const double al = alpha;
                c.v(OV_X)[i] = fma(al, c.v(OV_P)[i], c.v(OV_X)[i]);
                const double v = fma(-al, c.v(OV_Q)[i], c.v(OV_R)[i]);
                c.v(OV_R)[i] = v;
                if constexpr (ILLT) {
                    const double y = c.v(OV_C)[i] * v;
                    put_tagged(step(0) + row, y, tag + 1);
                    c.v(OV_BASE)[i] = y;
                }
                t[0] = fma(v, v, t[0]);
            });
            ++tag;
            ++it;
            ++here;
            // the ILLT form checks the residual together with r.z: one reduction less an iteration
            if constexpr (ILLT) {
                __syncthreads();
                precondition();
                each([&](int i, i64) { t[1] = fma(c.v(OV_R)[i], c.v(OV_Z)[i], t[1]); });
            }
            if (!all_sum(a, c, t, has_rows, row_warps, [&](const double* u) {
                    rr = u[0];
                    const double rz_new = ILLT ? u[1] : u[0];
                    beta = rz_new / rz;
                    rz = rz_new;
                    stop = rr <= a.tol2 * bb || it >= a.max_iterations || !isfinite(rr);
                })) return;
            if (!stop) {
                each([&](int i, i64 row) {
                    const double v = fma(beta, c.v(OV_P)[i], c.v(ILLT ? OV_Z : OV_R)[i]);
                    c.v(OV_P)[i] = v;
                    a.p[row] = v;
                });
                if (!all_sync(a, c)) return;
            }
        }
        if (!stop) break;   // this launch's share of iterations: the next one goes on
        // the true residual decides
        each([&](int i, i64 row) { a.x[row] = c.v(OV_X)[i]; });
        if (!all_sync(a, c)) return;
        pcg_spmv<DENSE>(a, c, a.x);
        double s[1] = {0.0};
        each([&](int i, i64 row) {
            const double d = a.b[row] - c.v(OV_Q)[i];
            s[0] = fma(d, d, s[0]);
        });
        if (!all_sum(a, c, s, has_rows, row_warps, [&](const double* t) {
                rr = t[0];
                done = rr <= a.tol2 * bb || it >= a.max_iterations || !isfinite(rr) || restart + 1 == PCG_RESTARTS;
            })) return;
        if (done) break;
    }
    each([&](int i, i64 row) {
        a.x[row] = c.v(OV_X)[i];
        a.r[row] = c.v(OV_R)[i];
    });
    if (blockIdx.x == 0 && tid == 0) {
        a.state[PS_BB] = bb;
        a.state[PS_RR] = rr;
        a.state[PS_RZ] = rz;
        a.state[PS_ITERS] = double(it);
        a.state[PS_SWEEPS] = double(sweeps);
        a.state[PS_RESTART] = double(restart);
        a.state[PS_TAG] = double(tag);
        a.state[PS_DONE] = done ? 1.0 : 0.0;
    }
}

// FP64 values of a Jacobi slab, rows divided by their diagonal (0 for padding)
__global__ void k_jacobi_values64(i64 n, const i64* __restrict__ slice, const i64* __restrict__ src,
                                  const i64* __restrict__ u_rp, const double* __restrict__ u, double* __restrict__ val) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
        const i64 sl = r >> 5, beg = slice[sl] + (r & 31), w = (slice[sl + 1] - slice[sl]) >> 5;
        const double inv = 1.0 / u[u_rp[r]];
        for (i64 k = 0; k < w; ++k) {
            const i64 e = beg + 32 * k;
            val[e] = src[e] >= 0 ? u[src[e]] * inv : 0.0;
        }
    }
}

__global__ void k_jacobi_diag64(i64 n, const i64* __restrict__ u_rp, const double* __restrict__ u,
                                const double* __restrict__ scale, double* __restrict__ c, double* __restrict__ dinv) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
        const double inv = 1.0 / u[u_rp[r]];
        c[r] = scale[r] * inv;
        dinv[r] = inv;
    }
}

template<bool ILLT, bool DENSE>
void pcg_launch(Ctx& ctx, unsigned grid, size_t smem, PcgArgs& a) {
    auto kernel = k_pcg<ILLT, DENSE>;
    allow_shared(kernel);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(PCG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    NL_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    count_launch();
}

}  // namespace

// A x = b by CG with the ILLT (M, applied by FP64 Jacobi sweeps) or the identity
// (M null).  Returns false, x as the caller left it, when the factor needs the
// exact triangular solves or the sweeps' values do not fit the device's memory.
bool pcg_solve(Ctx& ctx, const Csr& A, const IncompleteCholesky* Mc, const double* b, double* x, double tolerance,
               i64 max_iterations, bool x_is_initial_guess, const CgChunkHook& on_chunk, CgResult& res) {
    const i64 n = A.rows;
    CgWork& w = ctx.cg;
    auto* M = const_cast<IncompleteCholesky*>(Mc);
    w.n = n;
    if (M) {   // 400 bytes a row, more than a classical matrix: where they do not fit, the exact solves
        try {
            w.steps.reserve(size_t(PCG_MAX_SWEEPS + 1) * size_t(n) * 2);
        } catch (const error& e) {
            if (e.code != NLGPU_ERR_OUT_OF_MEMORY) throw;
            return false;
        }
    }
    if (M && !M->j64_ready) {
        M->jlo.val64.resize(M->jlo.val.n);
        M->jup.val64.resize(M->jup.val.n);
        M->jc64.resize(size_t(n)); M->jdinv64.resize(size_t(n));
        for (JacobiSlab* s : {&M->jlo, &M->jup})
            NL_LAUNCH(k_jacobi_values64, grid_for(n, 256), 256, 0, ctx.stream, n, s->slice.p, s->src.p, M->rp.p, M->u.p,
                      s->val64.p);
        NL_LAUNCH(k_jacobi_diag64, grid_for(n, 256), 256, 0, ctx.stream, n, M->rp.p, M->u.p, M->scale.p, M->jc64.p,
                  M->jdinv64.p);
        M->j64_ready = true;
    }
    int dev = 0, sms = 0, optin = 0;
    NL_CUDA(cudaGetDevice(&dev));
    NL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    NL_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PcgArgs a{};
    a.n = n;
    // consecutive rows per CTA, at most one CTA per SM
    const i64 per_sm = (n + sms - 1) / sms;
    const i64 rows = std::max<i64>(PCG_MIN_ROWS, (per_sm + 3) / 4 * 4);
    NL_REQUIRE(rows < (i64(1) << 30), NLGPU_ERR_UNSUPPORTED, "system too large for the CG kernel");
    a.rows = int(rows);
    const unsigned grid = unsigned((n + rows - 1) / rows);
    const size_t room = size_t(optin) - 2048;
    size_t smem = 0;
    if (rows <= PCG_OWN_ROWS && A.nnz < (i64(1) << 31)) smem = size_t(OV_COUNT) * size_t(rows) * sizeof(double) + (size_t(rows) + 2) / 2 * 8;
    else w.q.reserve(size_t(OV_COUNT) * grid * size_t(rows));
    a.own = smem ? nullptr : w.q.p;
    if (M) {
        a.wlo = M->jlo.max_width; a.wup = M->jup.max_width;
        const size_t bytes = size_t(rows) * (size_t(a.wlo + a.wup) * (sizeof(double) + sizeof(int32_t)) + 2 * sizeof(int32_t));
        if (smem + bytes <= room) { a.staged = 1; smem += bytes; }
        NL_CUDA(cudaMemsetAsync(w.steps.p, 0, size_t(PCG_MAX_SWEEPS + 1) * size_t(n) * 16, ctx.stream));
        a.steps = reinterpret_cast<ulonglong2*>(w.steps.p);
        a.lo = {M->jlo.slice.p, M->jlo.col.p, M->jlo.val64.p};
        a.up = {M->jup.slice.p, M->jup.col.p, M->jup.val64.p};
        a.c = M->jc64.p; a.dinv = M->jdinv64.p; a.scale = M->scale.p;
        // lanes per row of a sweep: what one pass of the CTA's threads allows
        while (a.lgs < 3 && (rows << (a.lgs + 1)) <= PCG_THREADS && (2 << a.lgs) <= a.wlo) ++a.lgs;
    }
    // lanes per row of the product: FP64 pipe time of the CTA's warps (16 cycles an
    // instruction: a lane's entries and the reduction) plus the latency of a warp's rounds
    const double mean = double(A.nnz) / double(n);
    double best = 0.0;
    for (int lg = 0; lg <= 5; ++lg) {
        const double per_lane = std::ceil(mean / double(1 << lg));
        const double warps = std::ceil(double(rows) * double(1 << lg) / 32.0);
        const double cost = warps * (per_lane + lg + 1.0) * 16.0 +
                            std::ceil(warps / PCG_WARPS) * (40.0 * per_lane + 62.0 * lg + 600.0);
        if (lg == 0 || cost < best) { best = cost; a.lg = lg; }
    }
    const bool dense = A.longest >= i64(LONG_ROW) << a.lg;
    w.r.reserve(size_t(n));
    w.p.reserve(size_t(n));
    a.rp = A.rowptr.p;
    a.col = A.col.p;
    a.val = A.val.p;
    a.b = b; a.x = x; a.r = w.r.p; a.p = w.p.p;
    // [tagged sums | counter | state | error]
    const size_t sums = size_t(2) * 2 * 2 * SUM_STRIDE * grid + 16;   // the counter in a line of its own
    w.sync.reserve(sums + PS_COUNT + 1);
    a.sums = reinterpret_cast<ulonglong2*>(w.sync.p);
    a.counter = reinterpret_cast<unsigned*>(w.sync.p + sums - 16);
    a.state = w.sync.p + sums;
    a.error = reinterpret_cast<int*>(a.state + PS_COUNT);
    a.tol2 = tolerance * tolerance;
    a.max_iterations = std::min<i64>(max_iterations, i64(1) << 40);
    a.iterations_here = on_chunk ? 16 : PCG_ITERS_PER_LAUNCH;
    a.x_zero = x_is_initial_guess ? 0 : 1;
    NL_CUDA(cudaMemsetAsync(w.sync.p, 0, (sums + PS_COUNT + 1) * sizeof(double), ctx.stream));
    double h[PS_COUNT + 1];
    for (;;) {
        if (dense) M ? pcg_launch<true, true>(ctx, grid, smem, a) : pcg_launch<false, true>(ctx, grid, smem, a);
        else M ? pcg_launch<true, false>(ctx, grid, smem, a) : pcg_launch<false, false>(ctx, grid, smem, a);
        NL_CUDA(cudaMemcpyAsync(h, a.state, sizeof h, cudaMemcpyDeviceToHost, ctx.stream));
        NL_CUDA(cudaStreamSynchronize(ctx.stream));
        int error = 0;
        std::memcpy(&error, &h[PS_COUNT], sizeof error);
        NL_REQUIRE(error == 0, NLGPU_ERR_TIMEOUT, "a wait of the CG kernel gave up");
        if (h[PS_EXACT] != 0.0) return false;
        if (h[PS_DONE] != 0.0) break;
        if (on_chunk) on_chunk(i64(h[PS_ITERS]), x);
        a.resume = 1;
        NL_CUDA(cudaMemsetAsync(w.sync.p, 0, sums * sizeof(double), ctx.stream));
    }
    res = CgResult{};
    res.iterations = i64(h[PS_ITERS]);
    const double bb = h[PS_BB];
    if (bb == 0.0) {
        NL_CUDA(cudaMemsetAsync(x, 0, size_t(n) * sizeof(double), ctx.stream));
        res.converged = true;
        return true;
    }
    res.residual = std::sqrt(h[PS_RR] / bb);
    // sqrt(r.z) / |b| of the last preconditioned residual
    res.reference_residual = std::sqrt(std::fabs(h[PS_RZ]) / bb);
    res.converged = h[PS_RR] <= a.tol2 * bb;
    return true;
}

}  // namespace nlgpu
