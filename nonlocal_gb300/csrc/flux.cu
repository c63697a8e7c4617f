// Heat flux of a solution: heat_equation_solution_2d::calc_flux
// (heat_equation_solution_2d.hpp:99-137).
//
//   1. local flux at every quadrature point, -Lambda grad T with
//      grad T = sum_i T_i (grad N_i . adj J) / |J| (gradient_in_qnodes,
//      mesh_2d_utils.hpp:40-60; local_flux_in_qnodes, heat_equation_solution_2d.hpp:72-96);
//   2. for a nonlocal model, at every quadrature point x of element eL the
//      influence-weighted average of the local flux over the neighbours'
//      quadrature points, flux = p1 local + (1 - p1) sum w |J| phi(x, x') local(x');
//   3. nodal values: the element-area-weighted mean, over the elements of a
//      node, of the flux at the Gauss point nearest to the node
//      (qnodes_to_nodes, mesh_2d_utils.hpp:82-101; mesh_2d::area, mesh_2d.hpp:225-234).
//
// Step 2 is the same pair loop as the assembly (every ordered neighbour pair,
// nq x nq influence evaluations): one warp per element eL, the lanes spread
// over the (eNL, qNL) points of its neighbour list, each accumulating the
// contributions to all of eL's quadrature points in registers, then a warp
// reduction; float-float for the influence kinds that have it unless
// NLGPU_ASSEMBLY_FP64 is set, FP64 otherwise.
#include "common.cuh"
#include "influence.cuh"
#include "influence_ff.cuh"

namespace nlgpu {

namespace {

constexpr int FX_THREADS = 256;

__global__ void k_flux_local(i64 E, int nen, int nq, const int32_t* __restrict__ elems, const double* __restrict__ deriv,
                             const double* __restrict__ jac, const double* __restrict__ cond_field, Model m,
                             const double* __restrict__ T, double* __restrict__ lx, double* __restrict__ ly) {
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < E * nq; t += i64(gridDim.x) * blockDim.x) {
        const i64 e = t / nq;
        const int q = int(t % nq);
        double gx = 0.0, gy = 0.0;
        for (int i = 0; i < nen; ++i) {
            const double v = T[elems[e * nen + i]];
            const double* d = deriv + 2 * ((e * nen + i) * nq + q);
            gx += v * d[0];
            gy += v * d[1];
        }
        gx /= jac[t];
        gy /= jac[t];
        double fx, fy;
        if (m.cond_kind == NLGPU_CONDUCTIVITY_ISOTROPIC) {
            const double c = cond_field ? cond_field[t] : m.cond[0];
            fx = gx * -c;
            fy = gy * -c;
        } else if (m.cond_kind == NLGPU_CONDUCTIVITY_ORTHOTROPIC) {
            fx = gx * -m.cond[0];
            fy = gy * -m.cond[1];
        } else {
            fx = -m.cond[0] * gx - m.cond[2] * gy;
            fy = -m.cond[2] * gx - m.cond[1] * gy;
        }
        lx[t] = fx;
        ly[t] = fy;
    }
}

// float-float covers sums whose terms are finite; the power of two that brings the
// largest to [1, 2)
__device__ __forceinline__ bool flux_in_range(const unsigned long long* largest) {
    return (*largest >> 52) < 0x7ff;
}
__device__ __forceinline__ double flux_power(const unsigned long long* largest, int sign) {
    const long long e = min(1022ll, max(-1022ll, static_cast<long long>(*largest >> 52) - 1023));
    return __longlong_as_double((1023 + sign * e) << 52);
}

template<int NQ, int INF>
__global__ void __launch_bounds__(FX_THREADS) k_flux_nonlocal(i64 E, const double* __restrict__ qcoord,
                                                              const double* __restrict__ jac, const i64* __restrict__ noff,
                                                              const int32_t* __restrict__ nlist, Model m, Basis b,
                                                              const double* __restrict__ lx,
                                                              const double* __restrict__ ly, double* __restrict__ fx,
                                                              double* __restrict__ fy,
                                                              const unsigned long long* __restrict__ largest) {
    if (largest && flux_in_range(largest)) return;   // done in float-float
    const int lane = threadIdx.x & 31;
    const i64 warps = i64(gridDim.x) * (blockDim.x >> 5);
    for (i64 eL = (blockIdx.x * i64(blockDim.x) + threadIdx.x) >> 5; eL < E; eL += warps) {
        double xq[NQ], yq[NQ], ax[NQ], ay[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            xq[q] = qcoord[2 * (eL * NQ + q)];
            yq[q] = qcoord[2 * (eL * NQ + q) + 1];
            ax[q] = 0.0;
            ay[q] = 0.0;
        }
        const i64 kb = noff[eL], items = (noff[eL + 1] - kb) * NQ;
        for (i64 it = lane; it < items; it += 32) {
            const int32_t eNL = nlist[kb + it / NQ];
            const int qn = int(it % NQ);
            const i64 s = i64(eNL) * NQ + qn;
            const double wj = b.w[qn] * jac[s];
            const double xs = qcoord[2 * s], ys = qcoord[2 * s + 1], vx = lx[s], vy = ly[s];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const double w = wj * (m.norm * shape<INF>(m, xq[q] - xs, yq[q] - ys));
                ax[q] += w * vx;
                ay[q] += w * vy;
            }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            ax[q] = warp_sum(ax[q]);
            ay[q] = warp_sum(ay[q]);
        }
        if (lane < NQ) {
            double sx = 0.0, sy = 0.0;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                if (q == lane) { sx = ax[q]; sy = ay[q]; }
            const i64 t = eL * NQ + lane;
            const double nw = 1.0 - m.p1;
            fx[t] = lx[t] * m.p1 + sx * nw;
            fy[t] = ly[t] * m.p1 + sy * nw;
        }
    }
}

// largest magnitude of w_q |J| norm times the local flux (as the bits of a double:
// non-negative doubles order like their bits, and NaN above infinity)
__global__ void k_flux_scale(i64 count, int nq, const double* __restrict__ jac, Model m, Basis b,
                             const double* __restrict__ lx, const double* __restrict__ ly,
                             unsigned long long* __restrict__ largest) {
    unsigned long long top = 0;
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < count; t += i64(gridDim.x) * blockDim.x) {
        const double w = b.w[t % nq] * jac[t] * m.norm;
        top = max(top, static_cast<unsigned long long>(__double_as_longlong(fabs(w * lx[t]))));
        top = max(top, static_cast<unsigned long long>(__double_as_longlong(fabs(w * ly[t]))));
    }
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((threadIdx.x & 31) == 0) atomicMax(largest, top);
}

// w_q |J| norm times the local flux in float-float, scaled
__global__ void k_flux_stage(i64 count, int nq, const double* __restrict__ jac, Model m, Basis b,
                             const double* __restrict__ lx, const double* __restrict__ ly,
                             const unsigned long long* __restrict__ largest, float4* __restrict__ load) {
    const double scale = flux_power(largest, -1);
    for (i64 t = blockIdx.x * i64(blockDim.x) + threadIdx.x; t < count; t += i64(gridDim.x) * blockDim.x) {
        const double w = b.w[t % nq] * jac[t] * m.norm;
        const ff vx = ff_from(w * lx[t] * scale), vy = ff_from(w * ly[t] * scale);
        load[t] = make_float4(vx.h, vx.l, vy.h, vy.l);
    }
}

// The nonlocal average as in k_flux_nonlocal with the influence values and the sums
// in float-float on the FP32 pipes: about 140 FP32 instructions per pair of points
// against 27 on the FP64 pipe, whose two lanes a clock bound that kernel (120x90
// 8-node, exponential: 8.38 ms, here 1.00; the error against 64-bit sums is no
// larger).  A source's coordinates are taken relative to the element's first point
// in FP64 (two subtractions and two products), so that float-float holds the
// distances, not the mesh coordinates; a lane's sums are compensated.
template<int NQ, int INF>
__global__ void __launch_bounds__(FX_THREADS, 2) k_flux_nonlocal_ff(i64 E, const double2* __restrict__ at,
                                                                 const float4* __restrict__ load,
                                                                 const i64* __restrict__ noff,
                                                                 const int32_t* __restrict__ nlist, Model m,
                                                                 FFExpTable table,
                                                                 const unsigned long long* __restrict__ largest,
                                                                 const double* __restrict__ lx,
                                                                 const double* __restrict__ ly, double* __restrict__ fx,
                                                                 double* __restrict__ fy) {
    __shared__ ff etab[2 * FF_EXP_K + 1];
    if (!flux_in_range(largest)) return;   // k_flux_nonlocal does it
    for (int t = threadIdx.x; t < 2 * FF_EXP_K + 1; t += FX_THREADS) etab[t] = ff{table.v[t].x, table.v[t].y};
    __syncthreads();
    const ff qf = ff_from(m.q);
    const double back = flux_power(largest, 1);
    const int lane = threadIdx.x & 31;
    const i64 warps = i64(gridDim.x) * (blockDim.x >> 5);
    for (i64 eL = (blockIdx.x * i64(blockDim.x) + threadIdx.x) >> 5; eL < E; eL += warps) {
        const double2 origin = at[eL * NQ];
        ff xq[NQ], yq[NQ];
        ffdot ax[NQ], ay[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double2 p = at[eL * NQ + q];
            xq[q] = ff_split((p.x - origin.x) * m.inv_r[0]);
            yq[q] = ff_split((p.y - origin.y) * m.inv_r[1]);
        }
        const i64 kb = noff[eL], items = (noff[eL + 1] - kb) * NQ;
        for (i64 it = lane; it < items; it += 32) {
            const i64 s = i64(nlist[kb + it / NQ]) * NQ + it % NQ;
            const double2 p = at[s];
            const float4 v = load[s];
            const ff xs = ff_split((p.x - origin.x) * m.inv_r[0]), ys = ff_split((p.y - origin.y) * m.inv_r[1]);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const ff w = shape_ff<INF>(m, ff_sub(xq[q], xs), ff_sub(yq[q], ys), qf, etab);
                ffdot_add(ax[q], w, ff{v.x, v.y});
                ffdot_add(ay[q], w, ff{v.z, v.w});
            }
        }
        double sx = 0.0, sy = 0.0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double tx = warp_sum(ff_to(ffdot_value(ax[q]))), ty = warp_sum(ff_to(ffdot_value(ay[q])));
            if (q == lane) { sx = tx; sy = ty; }
        }
        if (lane < NQ) {
            const i64 t = eL * NQ + lane;
            const double nw = 1.0 - m.p1;
            fx[t] = lx[t] * m.p1 + sx * back * nw;
            fy[t] = ly[t] * m.p1 + sy * back * nw;
        }
    }
}

__global__ void k_element_area(i64 E, int nen, int nq, const double* __restrict__ jac, Basis b, double* __restrict__ area) {
    for (i64 e = blockIdx.x * i64(blockDim.x) + threadIdx.x; e < E; e += i64(gridDim.x) * blockDim.x) {
        double a = 0.0;
        for (int q = 0; q < nq; ++q) {
            const double factor = b.w[q] * jac[e * nq + q];
            for (int i = 0; i < nen; ++i) a += factor * b.qN[i * nq + q];
        }
        area[e] = a;
    }
}

__global__ void k_flux_nodes(i64 n, const i64* __restrict__ ne_off, const int32_t* __restrict__ ne_elem,
                             const int8_t* __restrict__ ne_local, int nq, Basis b, const double* __restrict__ area,
                             const double* __restrict__ fx, const double* __restrict__ fy, double* __restrict__ ox,
                             double* __restrict__ oy) {
    for (i64 node = blockIdx.x * i64(blockDim.x) + threadIdx.x; node < n; node += i64(gridDim.x) * blockDim.x) {
        double sx = 0.0, sy = 0.0, s = 0.0;
        for (i64 k = ne_off[node]; k < ne_off[node + 1]; ++k) {
            const i64 e = ne_elem[k];
            const double a = area[e];
            const i64 q = e * nq + b.nearest[ne_local[k]];
            sx += a * fx[q];
            sy += a * fy[q];
            s += a;
        }
        ox[node] = sx / s;
        oy[node] = sy / s;
    }
}

template<int NQ>
void launch_nonlocal(Ctx& ctx, const double* lx, const double* ly, double* fx, double* fy,
                     const unsigned long long* largest) {
    const i64 E = ctx.n_elems;
    const unsigned grid = grid_for(E * 32, FX_THREADS, 152 * 64);
    switch (ctx.model.influence) {
    case NLGPU_INFLUENCE_FAST_POLYNOMIAL:
        NL_LAUNCH((k_flux_nonlocal<NQ, NLGPU_INFLUENCE_FAST_POLYNOMIAL>), grid, FX_THREADS, 0, ctx.stream, E,
                  ctx.qcoord.p, ctx.jac.p, ctx.noff.p, ctx.nlist.p, ctx.model, ctx.basis, lx, ly, fx, fy, largest);
        break;
    case NLGPU_INFLUENCE_POLYNOMIAL:
        NL_LAUNCH((k_flux_nonlocal<NQ, NLGPU_INFLUENCE_POLYNOMIAL>), grid, FX_THREADS, 0, ctx.stream, E,
                  ctx.qcoord.p, ctx.jac.p, ctx.noff.p, ctx.nlist.p, ctx.model, ctx.basis, lx, ly, fx, fy, largest);
        break;
    case NLGPU_INFLUENCE_EXPONENTIAL:
        NL_LAUNCH((k_flux_nonlocal<NQ, NLGPU_INFLUENCE_EXPONENTIAL>), grid, FX_THREADS, 0, ctx.stream, E,
                  ctx.qcoord.p, ctx.jac.p, ctx.noff.p, ctx.nlist.p, ctx.model, ctx.basis, lx, ly, fx, fy, largest);
        break;
    default:
        NL_LAUNCH((k_flux_nonlocal<NQ, NLGPU_INFLUENCE_CONSTANT>), grid, FX_THREADS, 0, ctx.stream, E,
                  ctx.qcoord.p, ctx.jac.p, ctx.noff.p, ctx.nlist.p, ctx.model, ctx.basis, lx, ly, fx, fy, largest);
        break;
    }
}

template<int NQ>
void launch_nonlocal_ff(Ctx& ctx, const float4* load, const unsigned long long* largest, const double* lx, const double* ly,
                        double* fx, double* fy) {
    const i64 E = ctx.n_elems;
    const unsigned grid = grid_for(E * 32, FX_THREADS, 152 * 64);
    FFExpTable table;
    fill_exp_table(table);
    auto launch = [&](auto kernel) {
        NL_LAUNCH(kernel, grid, FX_THREADS, 0, ctx.stream, E, reinterpret_cast<const double2*>(ctx.qcoord.p), load, ctx.noff.p,
                  ctx.nlist.p, ctx.model, table, largest, lx, ly, fx, fy);
    };
    switch (ctx.model.influence) {
    case NLGPU_INFLUENCE_FAST_POLYNOMIAL: launch(k_flux_nonlocal_ff<NQ, NLGPU_INFLUENCE_FAST_POLYNOMIAL>); break;
    case NLGPU_INFLUENCE_POLYNOMIAL: launch(k_flux_nonlocal_ff<NQ, NLGPU_INFLUENCE_POLYNOMIAL>); break;
    default: launch(k_flux_nonlocal_ff<NQ, NLGPU_INFLUENCE_EXPONENTIAL>); break;
    }
}

}  // namespace

void calc_flux(Ctx& ctx, const double* temperature, double* flux_x, double* flux_y) {
    const i64 E = ctx.n_elems, n = ctx.n_nodes;
    const int nen = ctx.basis.nen, nq = ctx.basis.nq;
    dbuf<double> lx, ly, fx, fy, area;
    dbuf<float4> load;
    dbuf<unsigned long long> largest;
    lx.resize(size_t(E * nq)); ly.resize(size_t(E * nq));
    area.resize(size_t(E));
    NL_LAUNCH(k_flux_local, grid_for(E * nq, FX_THREADS), FX_THREADS, 0, ctx.stream, E, nen, nq, ctx.elems.p,
              ctx.deriv.p, ctx.jac.p, ctx.cond_field.n ? ctx.cond_field.p : nullptr, ctx.model, temperature, lx.p, ly.p);
    const double* qx = lx.p;
    const double* qy = ly.p;
    if (ctx.model.nonlocal()) {
        fx.resize(size_t(E * nq)); fy.resize(size_t(E * nq));
        // float-float where the influence has a float-float form and every term is finite
        // (the FP64 kernel then returns at once), FP64 otherwise and where it is asked for
        const bool in_ff = ff_supported(ctx.model) && ctx.assembly_precision != NLGPU_ASSEMBLY_FP64;
        if (in_ff) {
            load.resize(size_t(E * nq));
            largest.resize(1);
            largest.zero(ctx.stream);
            NL_LAUNCH(k_flux_scale, grid_for(E * nq, FX_THREADS, 152 * 8), FX_THREADS, 0, ctx.stream, E * nq, nq, ctx.jac.p,
                      ctx.model, ctx.basis, lx.p, ly.p, largest.p);
            NL_LAUNCH(k_flux_stage, grid_for(E * nq, FX_THREADS), FX_THREADS, 0, ctx.stream, E * nq, nq, ctx.jac.p,
                      ctx.model, ctx.basis, lx.p, ly.p, largest.p, load.p);
            if (nq == 4) launch_nonlocal_ff<4>(ctx, load.p, largest.p, lx.p, ly.p, fx.p, fy.p);
            else launch_nonlocal_ff<9>(ctx, load.p, largest.p, lx.p, ly.p, fx.p, fy.p);
        }
        if (nq == 4) launch_nonlocal<4>(ctx, lx.p, ly.p, fx.p, fy.p, in_ff ? largest.p : nullptr);
        else launch_nonlocal<9>(ctx, lx.p, ly.p, fx.p, fy.p, in_ff ? largest.p : nullptr);
        qx = fx.p;
        qy = fy.p;
    }
    NL_LAUNCH(k_element_area, grid_for(E, FX_THREADS), FX_THREADS, 0, ctx.stream, E, nen, nq, ctx.jac.p, ctx.basis,
              area.p);
    NL_LAUNCH(k_flux_nodes, grid_for(n, FX_THREADS), FX_THREADS, 0, ctx.stream, n, ctx.ne_off.p, ctx.ne_elem.p,
              ctx.ne_local.p, nq, ctx.basis, area.p, qx, qy, flux_x, flux_y);
    NL_CUDA(cudaStreamSynchronize(ctx.stream));   // the scratch buffers are freed on return
}

}  // namespace nlgpu
