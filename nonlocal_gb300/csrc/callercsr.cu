// The solver's full rows of a caller's symmetric matrix (slae::conjugate_gradient,
// conjugate_gradient.hpp:15-79: upper storage, int64 row pointers and columns).
//
// The caller's arrays go to the device as they are; the rows are counted, placed
// (each off-diagonal entry also into its column's row, in any order) and sorted
// there.  On the host the same took 6 ms of vectors and sorts for 200 000 entries
// (61x45 nonlocal), here 0.1 ms and the copies.
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

// rows padded to multiples of 4 entries
__global__ void k_cc_pad(i64 n, const i64* __restrict__ count, i64* __restrict__ padded) {
    for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x)
        padded[r] = (count[r] + 3) & ~i64(3);
}

__global__ void k_cc_place(i64 n, const i64* __restrict__ rp, const i64* __restrict__ col, const double* __restrict__ val,
                           i64 first, const i64* __restrict__ full_rp, unsigned* __restrict__ cursor,
                           int32_t* __restrict__ tcol, double* __restrict__ tval) {
    const int lane = threadIdx.x & 31;
    CC_ROWS(r) {
        for (i64 k = rp[r] + lane; k < rp[r + 1]; k += 32) {
            const i64 c = col[k - first];
            const double v = val[k - first];
            const i64 p = full_rp[r] + atomicAdd(cursor + r, 1u);
            tcol[p] = int32_t(c);
            tval[p] = v;
            if (c != r) {
                const i64 t = full_rp[c] + atomicAdd(cursor + c, 1u);
                tcol[t] = int32_t(r);
                tval[t] = v;
            }
        }
    }
}

// each row by increasing column (an entry's place is the number of smaller ones,
// equal columns by position), padding entries (row, 0)
__global__ void k_cc_sort(i64 n, const i64* __restrict__ full_rp, const i64* __restrict__ count,
                          const int32_t* __restrict__ tcol, const double* __restrict__ tval, int32_t* __restrict__ col,
                          double* __restrict__ val) {
    const int lane = threadIdx.x & 31;
    CC_ROWS(r) {
        const i64 b = full_rp[r], len = count[r];
        for (i64 k = lane; k < len; k += 32) {
            const int32_t c = tcol[b + k];
            i64 rank = 0;
            for (i64 j = 0; j < len; ++j) {
                const int32_t o = __ldg(tcol + b + j);
                rank += o < c || (o == c && j < k);
            }
            col[b + rank] = c;
            val[b + rank] = tval[b + k];
        }
        for (i64 k = b + len + lane; k < full_rp[r + 1]; k += 32) {
            col[k] = int32_t(r);
            val[k] = 0.0;
        }
    }
}

}  // namespace

void full_rows_from_caller(Ctx& ctx, i64 n, const int64_t* rowptr, const int64_t* col, const double* val, Csr& A) {
    const i64 first = *std::min_element(rowptr, rowptr + n + 1), last = *std::max_element(rowptr, rowptr + n + 1);
    NL_REQUIRE(first >= 0, NLGPU_ERR_ARG, "row pointers must not be negative");
    const size_t m = size_t(std::max<i64>(last - first, 1));
    cudaStream_t s = ctx.stream;
    dbuf<i64> rp, dcol, count;
    dbuf<double> dval, tval;
    dbuf<int32_t> tcol;
    dbuf<unsigned> cursor;
    dbuf<int> bad;
    rp.upload(rowptr, size_t(n + 1), s);
    dcol.resize(m);
    dval.resize(m);
    if (last > first) {
        dcol.upload(col + first, m, s);
        dval.upload(val + first, m, s);
    }
    count.resize(size_t(n)); count.zero(s);
    cursor.resize(size_t(n)); cursor.zero(s);
    bad.resize(1); bad.zero(s);
    const unsigned grid = grid_for(n * 32, CC_THREADS, 152 * 64);
    NL_LAUNCH(k_cc_count, grid, CC_THREADS, 0, s, n, rp.p, dcol.p, first,
              reinterpret_cast<unsigned long long*>(count.p), bad.p);
    A.rows = n;
    A.rowptr.resize(size_t(n + 1));
    NL_CUDA(cudaMemsetAsync(A.rowptr.p + n, 0, sizeof(i64), s));
    NL_LAUNCH(k_cc_pad, grid_for(n, CC_THREADS), CC_THREADS, 0, s, n, count.p, A.rowptr.p);
    int hbad = 0;
    bad.download(&hbad, 1, s);
    i64 total = 0;
    exclusive_scan(ctx, A.rowptr.p, A.rowptr.p, n + 1, &total);   // synchronises
    NL_REQUIRE(hbad == 0, NLGPU_ERR_ARG, "A must be the upper triangle with columns in range");
    A.nnz = total;
    const size_t nnz = size_t(std::max<i64>(total, 1));
    A.col.resize(nnz); A.val.resize(nnz);
    tcol.resize(nnz); tval.resize(nnz);
    NL_LAUNCH(k_cc_place, grid, CC_THREADS, 0, s, n, rp.p, dcol.p, dval.p, first, A.rowptr.p, cursor.p, tcol.p, tval.p);
    NL_LAUNCH(k_cc_sort, grid, CC_THREADS, 0, s, n, A.rowptr.p, count.p, tcol.p, tval.p, A.col.p, A.val.p);
    NL_CUDA(cudaStreamSynchronize(s));   // the scratch buffers are freed on return
}

}  // namespace nlgpu
