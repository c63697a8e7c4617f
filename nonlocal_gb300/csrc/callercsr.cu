// The solver's full rows of a caller's symmetric matrix (slae::conjugate_gradient,
// conjugate_gradient.hpp:15-79: upper storage, int64 row pointers and columns).
//
// The caller's arrays go to the device as they are; the rows are counted, placed
// (each off-diagonal entry also into its column's row, in any order) and sorted
// there by column, equal columns in the caller's order.  On the host the same took
// 6 ms of vectors and sorts for 200 000 entries (61x45 nonlocal), here 0.1 ms and the
// copies.
#include "common.cuh"

#include <algorithm>

namespace nlgpu {

namespace {

constexpr int CC_THREADS = 256;

#define CC_ROWS(r)                                                                                            \
    for (i64 r = (blockIdx.x * i64(blockDim.x) + threadIdx.x) >> 5, warps_ = (i64(gridDim.x) * blockDim.x) >> 5; r < n; \
         r += warps_)

// entries per full row (warp per caller's row); a column below the diagonal or
// out of range raises *bad.  A row whose pointers decrease is empty.
__global__ void k_cc_count(i64 n, const i64* __restrict__ rp, const i64* __restrict__ col, i64 first,
                           unsigned long long* __restrict__ count, int* __restrict__ bad) {
    const int lane = threadIdx.x & 31;
    CC_ROWS(r) {
        int own = 0;
        for (i64 k = rp[r] + lane; k < rp[r + 1]; k += 32) {
            const i64 c = col[k - first];
            if (c < r || c >= n) { *bad = 1; continue; }
            ++own;
            if (c != r) atomicAdd(count + c, 1ull);
        }
        for (int o = 16; o > 0; o >>= 1) own += __shfl_xor_sync(0xffffffffu, own, o);
        if (lane == 0 && own) atomicAdd(count + r, (unsigned long long)own);
    }
}

// rows padded to multiples of 4 entries; the longest row
__global__ void k_cc_pad(i64 n, const i64* __restrict__ count, i64* __restrict__ padded, unsigned long long* longest) {
    unsigned long long m = 0;
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
        padded[r] = (count[r] + 3) & ~i64(3);
        m = max(m, static_cast<unsigned long long>(count[r]));
    }
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(longest, m);
}

// tsrc: the entry's place in the caller's arrays, its order among equal columns
__global__ void k_cc_place(i64 n, const i64* __restrict__ rp, const i64* __restrict__ col, i64 first,
                           const i64* __restrict__ full_rp, unsigned* __restrict__ cursor,
                           int32_t* __restrict__ tcol, i64* __restrict__ tsrc) {
    const int lane = threadIdx.x & 31;
    CC_ROWS(r) {
        for (i64 k = rp[r] + lane; k < rp[r + 1]; k += 32) {
            const i64 c = col[k - first];
            const i64 p = full_rp[r] + atomicAdd(cursor + r, 1u);
            tcol[p] = int32_t(c);
            tsrc[p] = k - first;
            if (c != r) {
                const i64 t = full_rp[c] + atomicAdd(cursor + c, 1u);
                tcol[t] = int32_t(r);
                tsrc[t] = k - first;
            }
        }
    }
}

// how many of the entries [b, b + len) come before (c, src), one of them; the sources
// decide only where a column stands twice
__device__ __forceinline__ i64 rank_among(const int32_t* __restrict__ tcol, const i64* __restrict__ tsrc, i64 b, i64 len,
                                          int32_t c, i64 src) {
    i64 rank = 0;
    int equal = 0;
    for (i64 j = b; j < b + len; ++j) {
        const int32_t o = __ldg(tcol + j);
        rank += o < c;
        equal += o == c;
    }
    if (equal > 1)
        for (i64 j = b; j < b + len; ++j) rank += __ldg(tcol + j) == c && __ldg(tsrc + j) < src;
    return rank;
}

// Longer rows are merged: a warp's ranking of a row costs its length squared / 32, 7.5 s
// for one of 100 000 entries, which the host sorted in 5 ms.  Such a row is cut into
// runs of CC_RUN entries, ranked by a CTA each, and pairs of runs are merged, an
// entry a thread: its place is its own in its run and the number of smaller ones in
// the other, by a binary search.  Below CC_RUN entries a row's ranking takes less than
// the launches of the passes.
constexpr int CC_RUN = 256;

// each row of up to CC_RUN entries by increasing column (an entry's place is the
// number of smaller ones), padding entries (row, 0) in every row
__global__ void k_cc_sort(i64 n, const i64* __restrict__ full_rp, const i64* __restrict__ count,
                          const int32_t* __restrict__ tcol, const i64* __restrict__ tsrc,
                          const double* __restrict__ values, int32_t* __restrict__ col, double* __restrict__ val) {
    const int lane = threadIdx.x & 31;
    CC_ROWS(r) {
        const i64 b = full_rp[r], len = count[r];
        if (len <= CC_RUN)
            for (i64 k = lane; k < len; k += 32) {
                const int32_t c = tcol[b + k];
                const i64 src = tsrc[b + k];
                const i64 to = b + rank_among(tcol, tsrc, b, len, c, src);
                col[to] = c;
                val[to] = values[src];
            }
        for (i64 k = b + len + lane; k < full_rp[r + 1]; k += 32) {
            col[k] = int32_t(r);
            val[k] = 0.0;
        }
    }
}

// runs of every row longer than CC_RUN (0 for the others)
__global__ void k_cc_runs(i64 n, const i64* __restrict__ count, i64* __restrict__ runs) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x)
        runs[r] = count[r] > CC_RUN ? (count[r] + CC_RUN - 1) / CC_RUN : 0;
}

// the row of each run (warp per row; runs: their exclusive sums)
__global__ void k_cc_run_rows(i64 n, const i64* __restrict__ runs, int32_t* __restrict__ row) {
    const int lane = threadIdx.x & 31;
    CC_ROWS(r)
        for (i64 k = runs[r] + lane; k < runs[r + 1]; k += 32) row[k] = int32_t(r);
}

// CTA per run, thread per entry.  width 0: sorts the run; else merges runs of `width`
// entries into runs of twice that.
__global__ void __launch_bounds__(CC_RUN) k_cc_merge(i64 total, const i64* __restrict__ runs, const int32_t* __restrict__ row,
                                                     const i64* __restrict__ full_rp, const i64* __restrict__ count,
                                                     i64 width, const int32_t* __restrict__ tcol,
                                                     const i64* __restrict__ tsrc, int32_t* __restrict__ ocol,
                                                     i64* __restrict__ osrc) {
    for (i64 q = blockIdx.x; q < total; q += gridDim.x) {
        const i64 r = row[q], b = full_rp[r], len = count[r];
        const i64 at = (q - runs[r]) * CC_RUN, k = at + threadIdx.x;   // of the row
        if (k >= len) continue;
        const int32_t c = tcol[b + k];
        const i64 src = tsrc[b + k];
        i64 to;
        if (width == 0) {
            to = at + rank_among(tcol, tsrc, b + at, min(i64(CC_RUN), len - at), c, src);
        } else {
            const i64 pair = k / (2 * width) * (2 * width);   // its two runs: [pair, pair + width), [pair + width, ...)
            const bool second = k - pair >= width;
            i64 lo = second ? pair : min(len, pair + width);
            const i64 other = lo;
            i64 hi = second ? pair + width : min(len, pair + 2 * width);
            while (lo < hi) {
                const i64 mid = (lo + hi) >> 1;
                const int32_t o = tcol[b + mid];
                if (o < c || (o == c && tsrc[b + mid] < src)) lo = mid + 1;
                else hi = mid;
            }
            to = (second ? k - width : k) + (lo - other);
        }
        ocol[b + to] = c;
        osrc[b + to] = src;
    }
}

__global__ void __launch_bounds__(CC_RUN) k_cc_finish(i64 total, const i64* __restrict__ runs, const int32_t* __restrict__ row,
                                                      const i64* __restrict__ full_rp, const i64* __restrict__ count,
                                                      const int32_t* __restrict__ tcol, const i64* __restrict__ tsrc,
                                                      const double* __restrict__ values, int32_t* __restrict__ col,
                                                      double* __restrict__ val) {
    for (i64 q = blockIdx.x; q < total; q += gridDim.x) {
        const i64 r = row[q], k = (q - runs[r]) * CC_RUN + threadIdx.x, e = full_rp[r] + k;
        if (k >= count[r]) continue;
        col[e] = tcol[e];
        val[e] = values[tsrc[e]];
    }
}

// the rows of more than CC_RUN entries
void sort_long_rows(Ctx& ctx, const Csr& A, const dbuf<i64>& count, dbuf<int32_t>& tcol, dbuf<i64>& tsrc,
                    const dbuf<double>& values) {
    const i64 n = A.rows;
    cudaStream_t s = ctx.stream;
    dbuf<i64> runs, osrc;
    dbuf<int32_t> row, ocol;
    runs.resize(size_t(n + 1));
    NL_CUDA(cudaMemsetAsync(runs.p + n, 0, sizeof(i64), s));
    NL_LAUNCH(k_cc_runs, grid_for(n, CC_THREADS), CC_THREADS, 0, s, n, count.p, runs.p);
    i64 total = 0;
    exclusive_scan(ctx, runs.p, runs.p, n + 1, &total);
    row.resize(size_t(total));
    ocol.resize(tcol.n);
    osrc.resize(tsrc.n);
    NL_LAUNCH(k_cc_run_rows, grid_for(n * 32, CC_THREADS, 152 * 64), CC_THREADS, 0, s, n, runs.p, row.p);
    const unsigned grid = unsigned(std::min<i64>(total, 152 * 64));
    auto pass = [&](i64 width) {
        NL_LAUNCH(k_cc_merge, grid, CC_RUN, 0, s, total, runs.p, row.p, A.rowptr.p, count.p, width, tcol.p, tsrc.p, ocol.p,
                  osrc.p);
        std::swap(tcol, ocol);
        std::swap(tsrc, osrc);
    };
    pass(0);
    for (i64 width = CC_RUN; width < A.longest; width *= 2) pass(width);
    NL_LAUNCH(k_cc_finish, grid, CC_RUN, 0, s, total, runs.p, row.p, A.rowptr.p, count.p, tcol.p, tsrc.p, values.p, A.col.p,
              A.val.p);
    NL_CUDA(cudaStreamSynchronize(s));   // the scratch buffers are freed on return
}

}  // namespace

void full_rows_from_caller(Ctx& ctx, i64 n, const int64_t* rowptr, const int64_t* col, const double* val, Csr& A) {
    const i64 first = *std::min_element(rowptr, rowptr + n + 1), last = *std::max_element(rowptr, rowptr + n + 1);
    NL_REQUIRE(first >= 0, NLGPU_ERR_ARG, "row pointers must not be negative");
    const size_t m = size_t(std::max<i64>(last - first, 1));
    cudaStream_t s = ctx.stream;
    dbuf<i64> rp, dcol, count;
    dbuf<double> dval;
    dbuf<int32_t> tcol;
    dbuf<i64> tsrc;
    dbuf<unsigned> cursor;
    dbuf<unsigned long long> found;   // [a bad column, the longest row]
    rp.upload(rowptr, size_t(n + 1), s);
    dcol.resize(m);
    dval.resize(m);
    if (last > first) {
        dcol.upload(col + first, m, s);
        dval.upload(val + first, m, s);
    }
    count.resize(size_t(n)); count.zero(s);
    cursor.resize(size_t(n)); cursor.zero(s);
    found.resize(2); found.zero(s);
    const unsigned grid = grid_for(n * 32, CC_THREADS, 152 * 64);
    NL_LAUNCH(k_cc_count, grid, CC_THREADS, 0, s, n, rp.p, dcol.p, first,
              reinterpret_cast<unsigned long long*>(count.p), reinterpret_cast<int*>(found.p));
    A.rows = n;
    A.rowptr.resize(size_t(n + 1));
    NL_CUDA(cudaMemsetAsync(A.rowptr.p + n, 0, sizeof(i64), s));
    NL_LAUNCH(k_cc_pad, grid_for(n, CC_THREADS), CC_THREADS, 0, s, n, count.p, A.rowptr.p, found.p + 1);
    unsigned long long h[2] = {0, 0};
    found.download(h, 2, s);
    i64 total = 0;
    exclusive_scan(ctx, A.rowptr.p, A.rowptr.p, n + 1, &total);   // synchronises
    NL_REQUIRE(h[0] == 0, NLGPU_ERR_ARG, "A must be the upper triangle with columns in range");
    A.nnz = total;
    A.longest = i64(h[1]);
    const size_t nnz = size_t(std::max<i64>(total, 1));
    A.col.resize(nnz); A.val.resize(nnz);
    tcol.resize(nnz); tsrc.resize(nnz);
    NL_LAUNCH(k_cc_place, grid, CC_THREADS, 0, s, n, rp.p, dcol.p, first, A.rowptr.p, cursor.p, tcol.p, tsrc.p);
    NL_LAUNCH(k_cc_sort, grid, CC_THREADS, 0, s, n, A.rowptr.p, count.p, tcol.p, tsrc.p, dval.p, A.col.p, A.val.p);
    if (A.longest > CC_RUN) sort_long_rows(ctx, A, count, tcol, tsrc, dval);
    NL_CUDA(cudaStreamSynchronize(s));   // the scratch buffers are freed on return
}

}  // namespace nlgpu
