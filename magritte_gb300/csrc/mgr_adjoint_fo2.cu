// Differentiable formal solve on the GPU: the smooth FP64 J (forward) and its adjoint
// (backward) of Model::compute_radiation_field_feautrier_order_2 (model.cpp:353-390 ->
// Solver::solve_feautrier_order_2, solver.tpp:458-540), plus the device-pointer update
// of the model's frequencies that an autograd wrapper needs between calls.
//
// Both kernels run one warp per (origin, ray pair), over every origin or a list of them: a
// warp per origin left a 1k-point model on 8 warps an SM, each walking its ray pairs one
// after another.  The warp traces both halves into shared memory; for each line it runs the
// lanes over that line's quadrature points (so all lanes share the ray's elements, which the
// adjoint's warp sums need).  The forward stages u and a second kernel sums J(o, f) in the
// reference's ray-pair order.  The backward keeps each lane's per-pair elimination state in a
// scratch array of the warp's slot (recomputed, not saved by the forward) and adds its
// derivatives with one atomic per warp and entry; the frequencies' are staged per ray pair and
// summed in order, as u is.
//
// What bounds them: the FP64 pipe, with as many of 32 lanes live as a line has quadrature points,
// and instruction fetch (8 warps an SM on 335 KB of code; 553 KB with each half's sweep inlined).
// J and its gradients on a 13^3 sphere, 3 lines x 15: 23.1 -> 9.8 ms.
#include <algorithm>
#include <vector>

#include "mgr_adjoint_fo2.cuh"
#include "mgr_internal.h"

namespace mgr {

// u of the listed origins i0 .. i1 - 1 (every origin without a list) along every ray pair:
// U[((i - i0) * hnrays + rr) * F + f].
template <int AP>
__global__ void __launch_bounds__(256) fo2_s_kernel(DevModel m, uint32_t cap, const uint32_t* __restrict__ olist,
                                                    uint32_t i0, uint32_t i1, double* __restrict__ U, int* status) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t Lpad = (m.L + 1) & ~1u;
    double* sl = reinterpret_cast<double*>(smem);
    HalfSmem bk, fw;
    carve_halves(smem + (size_t)Lpad * 8 + (size_t)w * half_bytes_per_warp(cap), cap, bk, fw);
    for (uint32_t i = threadIdx.x; i < m.L; i += blockDim.x) sl[i] = m.sorted_line[i];
    __syncthreads();
    const uint64_t n = (uint64_t)(i1 - i0) * m.hnrays;
    for (uint64_t item = (uint64_t)blockIdx.x * nw + w; item < n; item += (uint64_t)gridDim.x * nw) {
        const uint32_t i = i0 + (uint32_t)(item / m.hnrays), rr = (uint32_t)(item % m.hnrays);
        const uint32_t o = olist ? olist[i] : i;
        int nb = 0, nf = 0;
        trace_pair<true, 0, 1>(m, o, rr, m.antipod[rr], cap, bk, fw, lane, status, nb, nf);
        if (nb < 0 || nf < 0) continue;  // status recorded by the trace
        for (uint32_t l = 0; l < m.L; l++)
            for (uint32_t q0 = 0; q0 < m.Q; q0 += 32) {
                const uint32_t q = q0 + lane;
                if (q < m.Q) {
                    const uint32_t f = m.lq2f[(size_t)l * m.Q + q];
                    const LaneS r = solve_lane_s<AP>(m, sl, o, m.nu[(size_t)o * m.F + f], l, bk, nb, fw, nf, nullptr);
                    U[(size_t)item * m.F + f] = r.u;
                }
            }
        __syncwarp();
    }
}

// J of the origins, summed over the ray pairs in order.
__global__ void __launch_bounds__(256) fo2_s_sum_kernel(DevModel m, const uint32_t* __restrict__ olist, uint32_t i0,
                                                        uint32_t i1, const double* __restrict__ U,
                                                        double* __restrict__ J, int* status) {
    const uint64_t n = (uint64_t)(i1 - i0) * m.F;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i = i0 + (uint32_t)(k / m.F), f = (uint32_t)(k % m.F);
        const uint32_t o = olist ? olist[i] : i;
        double v = 0.0;
        for (uint32_t rr = 0; rr < m.hnrays; rr++)
            v += U[((size_t)(i - i0) * m.hnrays + rr) * m.F + f] * (2.0 * ray_w(m, o, rr));
        J[(size_t)o * m.F + f] = v;
        if (!isfinite(v)) atomicOr(status, ST_NONFINITE);
    }
}

// The frequency derivatives of the origins, summed over the ray pairs in order (as the solve's
// results are, and the same from run to run; one thread a sum, atomic for origins listed twice).
__global__ void __launch_bounds__(256) fo2_nu_sum_kernel(DevModel m, const uint32_t* __restrict__ olist, uint32_t i0,
                                                         uint32_t i1, const double* __restrict__ gJ,
                                                         const double* __restrict__ GN, double* __restrict__ g_nu) {
    const uint64_t n = (uint64_t)(i1 - i0) * m.F;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i = i0 + (uint32_t)(k / m.F), f = (uint32_t)(k % m.F);
        const uint32_t o = olist ? olist[i] : i;
        if (gJ[(size_t)o * m.F + f] == 0.0) continue;
        double v = 0.0;
        for (uint32_t rr = 0; rr < m.hnrays; rr++) v += GN[((size_t)(i - i0) * m.hnrays + rr) * m.F + f];
        atomicAdd(g_nu + (size_t)o * m.F + f, v);
    }
}

// The adjoint of the listed origins i0 .. i1 - 1; frequency derivatives per ray pair in
// GN[((i - i0) * hnrays + rr) * F + f], for the frequencies with a derivative of the loss.
template <int AP>
__global__ void __launch_bounds__(256) fo2_adj_kernel(DevModel m, uint32_t cap, const uint32_t* __restrict__ olist,
                                                      uint32_t i0, uint32_t i1, const double* __restrict__ gJ,
                                                      AdjGrads g, double* __restrict__ GN, double* __restrict__ scratch,
                                                      uint32_t scratch_pairs, int* status) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t Lpad = (m.L + 1) & ~1u;
    double* sl = reinterpret_cast<double*>(smem);
    HalfSmem bk, fw;
    carve_halves(smem + (size_t)Lpad * 8 + (size_t)w * half_bytes_per_warp(cap), cap, bk, fw);
    for (uint32_t i = threadIdx.x; i < m.L; i += blockDim.x) sl[i] = m.sorted_line[i];
    __syncthreads();
    const size_t slot = (size_t)blockIdx.x * nw + w;
    const Fo2Scratch scr{scratch + slot * (size_t)scratch_pairs * 5 * 32 + lane, 32, scratch_pairs};
    const uint64_t n = (uint64_t)(i1 - i0) * m.hnrays;
    for (uint64_t item = (uint64_t)blockIdx.x * nw + w; item < n; item += (uint64_t)gridDim.x * nw) {
        const uint32_t i = i0 + (uint32_t)(item / m.hnrays), rr = (uint32_t)(item % m.hnrays);
        const uint32_t o = olist ? olist[i] : i;
        // origins without a derivative of the loss contribute nothing
        bool any = false;
        for (uint32_t f = lane; f < m.F; f += 32) any |= gJ[(size_t)o * m.F + f] != 0.0;
        if (!__any_sync(FULL_MASK, any)) continue;
        double vo[3] = {0.0, 0.0, 0.0};
        const uint32_t ar = m.antipod[rr];
        int nb = 0, nf = 0;
        trace_pair<true, 0, 1>(m, o, rr, ar, cap, bk, fw, lane, status, nb, nf);
        if (nb < 0 || nf < 0) continue;
        const double* db = ray_dir(m, o, rr);
        const double* df = ray_dir(m, o, ar);
        AdjGrads gb = g, gf = g;
        for (int k = 0; k < 3; k++) {
            gb.d[k] = db[k];
            gf.d[k] = df[k];
        }
        const AdjAcc acc_b{gb, m.L}, acc_f{gf, m.L};
        const double wt = 2.0 * ray_w(m, o, rr);
        for (uint32_t l = 0; l < m.L; l++)
            for (uint32_t q0 = 0; q0 < m.Q; q0 += 32) {
                const uint32_t q = q0 + lane;
                const uint32_t f = m.lq2f[(size_t)l * m.Q + (q < m.Q ? q : m.Q - 1)];
                const double gu = q < m.Q ? gJ[(size_t)o * m.F + f] * wt : 0.0;
                double gvb = 0.0, gvf = 0.0, gn = 0.0;
                if (__any_sync(FULL_MASK, gu != 0.0)) {
                    if (!solve_lane_s_adj<AP>(m, sl, o, m.nu[(size_t)o * m.F + f], l, bk, nb, fw, nf, gu, scr, acc_b,
                                              acc_f, gvb, gvf, gn)) {
                        if (lane == 0) atomicOr(status, ST_CAPACITY);
                        continue;
                    }
                    for (int k = 0; k < 3; k++) vo[k] += gvb * db[k] + gvf * df[k];
                }
                if (q < m.Q) GN[(size_t)item * m.F + f] = gn;
                __syncwarp();
            }
        for (int k = 0; k < 3; k++) {
            double v = vo[k];
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(FULL_MASK, v, off);
            if (lane == 0 && v != 0.0) atomicAdd(g.vel + 3 * (size_t)o + k, v);
        }
        __syncwarp();
    }
}

// Launch shape of the kernels: CTAs of up to 8 warps whose ray buffers fit in shared memory.
template <typename K>
static cudaError_t origin_launch_shape(MgrModel* model, K kern, uint32_t cap, uint64_t items, int* nw_out,
                                       size_t* smem_out, unsigned* grid_out) {
    const uint32_t Lpad = (model->dm.L + 1) & ~1u;
    int nw = 8;
    auto bytes = [&](int n) { return (size_t)Lpad * 8 + (size_t)n * half_bytes_per_warp(cap); };
    while (nw > 1 && bytes(nw) > 200 * 1024) nw /= 2;
    const size_t smem = bytes(nw);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nw * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    uint64_t grid = (uint64_t)model->sm_count * per_sm;
    const uint64_t need = (items + nw - 1) / nw;
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    *nw_out = nw;
    *smem_out = smem;
    *grid_out = (unsigned)grid;
    return cudaSuccess;
}

// Staged u of a pass of the smooth forward at most.
constexpr size_t kSmoothStageBytes = size_t(1) << 30;

static int check_smooth_model(MgrModel* model, const char* who) {
    if (!model->line_disc) {
        set_error(std::string(who) + ": the formal solve needs a line spectral discretisation");
        return MGR_ERR_UNSUPPORTED;
    }
    if (model->dm.sph) {
        set_error(std::string(who) + ": the differentiable formal solve does not support spherically symmetric models");
        return MGR_ERR_UNSUPPORTED;
    }
    if (model->dm.approx == APPROX_ONELINE) {
        set_error(std::string(who) + ": the differentiable formal solve supports the None and CloseLines "
                                     "approximations");
        return MGR_ERR_UNSUPPORTED;
    }
    return MGR_OK;
}

static int finish_stream(MgrModel* model, cudaError_t e, const char* who) {
    if (e == cudaSuccess) e = cudaStreamSynchronize(model->stream);
    if (e != cudaSuccess) return cuda_fail(e, who);
    int st = 0;
    e = cudaMemcpy(&st, model->status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemset(model->status, 0, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e, who);
    return decode_status(st);
}

}  // namespace mgr

using namespace mgr;

extern "C" {

int mgr_model_set_frequencies_device(MgrModel* model, const double* nu_dev) {
    MGR_MODEL_DEVICE(model);
    if (!model || !nu_dev) {
        set_error("mgr_model_set_frequencies_device: null argument");
        return MGR_ERR_ARGUMENT;
    }
    cudaError_t e = cudaMemcpyAsync(const_cast<double*>(model->dm.nu), nu_dev, (size_t)model->dm.P * model->dm.F * 8,
                                    cudaMemcpyDeviceToDevice, model->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(model->stream);
    if (e != cudaSuccess) return cuda_fail(e, "frequency update");
    model->inputs_replaced = true;
    return MGR_OK;
}

int mgr_formal_solve_fo2_smooth_device(MgrModel* model, const uint32_t* origins_dev, uint32_t n_origins,
                                       double* J_dev) {
    MGR_MODEL_DEVICE(model);
    if (!model || !J_dev) {
        set_error("mgr_formal_solve_fo2_smooth_device: null argument");
        return MGR_ERR_ARGUMENT;
    }
    int rc = check_smooth_model(model, "mgr_formal_solve_fo2_smooth_device");
    if (rc != MGR_OK) return rc;
    const uint32_t n_o = origins_dev ? n_origins : model->dm.P;
    if (n_o == 0) return MGR_OK;
    const uint32_t cap = model->half_cap;
    int nw;
    size_t smem;
    unsigned grid;
    // u staged, for as many origins at a time as a pass of kSmoothStageBytes (or the room there
    // is) holds
    const size_t per = (size_t)model->dm.hnrays * model->dm.F * sizeof(double);
    const size_t want = std::min<size_t>(n_o, std::max<size_t>(1, kSmoothStageBytes / per)) * per;
    if (!grow_pass(model, want, per))
        return cuda_fail(cudaErrorMemoryAllocation, "mgr_formal_solve_fo2_smooth_device: staging");
    const uint32_t pass = (uint32_t)std::min<size_t>(n_o, model->pass_bytes / per);
    auto run = [&](auto kern) -> cudaError_t {
        for (uint32_t i0 = 0; i0 < n_o; i0 += pass) {
            const uint32_t i1 = n_o - i0 > pass ? i0 + pass : n_o;
            cudaError_t r = origin_launch_shape(model, kern, cap, (uint64_t)(i1 - i0) * model->dm.hnrays, &nw, &smem,
                                                &grid);
            if (r != cudaSuccess) return r;
            count_launch();
            kern<<<grid, nw * 32, smem, model->stream>>>(model->dm, cap, origins_dev, i0, i1, model->pass, model->status);
            if ((r = cudaGetLastError()) != cudaSuccess) return r;
            const uint64_t threads = (uint64_t)(i1 - i0) * model->dm.F;
            const uint64_t blocks = std::min<uint64_t>((threads + 255) / 256, (uint64_t)model->sm_count * 16);
            count_launch();
            fo2_s_sum_kernel<<<(unsigned)blocks, 256, 0, model->stream>>>(model->dm, origins_dev, i0, i1, model->pass,
                                                                          J_dev, model->status);
            if ((r = cudaGetLastError()) != cudaSuccess) return r;
        }
        return cudaSuccess;
    };
    cudaError_t e = (model->dm.approx == APPROX_CLOSELINES) ? run(fo2_s_kernel<APPROX_CLOSELINES>)
                                                             : run(fo2_s_kernel<APPROX_NONE>);
    return finish_stream(model, e, "mgr_formal_solve_fo2_smooth_device");
}

int mgr_formal_solve_fo2_adjoint_device(MgrModel* model, const uint32_t* origins_dev, uint32_t n_origins,
                                        const double* gJ_dev, double* g_em_dev, double* g_op_dev, double* g_iw_dev,
                                        double* g_Sp_dev, double* g_vel_dev, double* g_nu_dev) {
    MGR_MODEL_DEVICE(model);
    if (!model || !gJ_dev || !g_em_dev || !g_op_dev || !g_iw_dev || !g_Sp_dev || !g_vel_dev || !g_nu_dev) {
        set_error("mgr_formal_solve_fo2_adjoint_device: null argument");
        return MGR_ERR_ARGUMENT;
    }
    int rc = check_smooth_model(model, "mgr_formal_solve_fo2_adjoint_device");
    if (rc != MGR_OK) return rc;
    const uint32_t n_o = origins_dev ? n_origins : model->dm.P;
    if (n_o == 0) return MGR_OK;
    const uint32_t cap = model->half_cap;
    // pairs of the longest ray pair: elements with the interpolation points of all
    // lines (Solver::get_ray_lengths_max), an upper bound of every line's count
    uint32_t* dmax = nullptr;
    uint32_t pairs = 0;
    cudaError_t e = cudaMalloc(&dmax, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemsetAsync(dmax, 0, sizeof(uint32_t), model->stream);
    if (e == cudaSuccess) e = launch_ray_lengths(model, dmax);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&pairs, dmax, sizeof(uint32_t), cudaMemcpyDeviceToHost, model->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(model->stream);
    cudaFree(dmax);
    if (e != cudaSuccess) return cuda_fail(e, "mgr_formal_solve_fo2_adjoint_device: ray lengths");
    if (pairs < 1) pairs = 1;
    AdjGrads g{g_em_dev, g_op_dev, g_iw_dev, g_Sp_dev, g_vel_dev, {0.0, 0.0, 0.0}};
    int nw;
    size_t smem;
    unsigned grid;
    // the frequency derivatives per ray pair, in passes as the forward's u
    const size_t per = (size_t)model->dm.hnrays * model->dm.F * sizeof(double);
    const size_t want = std::min<size_t>(n_o, std::max<size_t>(1, kSmoothStageBytes / per)) * per;
    if (!grow_pass(model, want, per))
        return cuda_fail(cudaErrorMemoryAllocation, "mgr_formal_solve_fo2_adjoint_device: staging");
    const uint32_t pass = (uint32_t)std::min<size_t>(n_o, model->pass_bytes / per);
    auto run = [&](auto kern) -> cudaError_t {
        cudaError_t r = origin_launch_shape(model, kern, cap, (uint64_t)pass * model->dm.hnrays, &nw, &smem, &grid);
        if (r != cudaSuccess) return r;
        r = grow_adj_scratch(model, (size_t)nw * pairs * 5 * 32 * sizeof(double), &grid);
        if (r != cudaSuccess) return r;
        for (uint32_t i0 = 0; i0 < n_o; i0 += pass) {
            const uint32_t i1 = n_o - i0 > pass ? i0 + pass : n_o;
            count_launch();
            kern<<<grid, nw * 32, smem, model->stream>>>(model->dm, cap, origins_dev, i0, i1, gJ_dev, g, model->pass,
                                                         model->adj_scratch, pairs, model->status);
            if ((r = cudaGetLastError()) != cudaSuccess) return r;
            const uint64_t threads = (uint64_t)(i1 - i0) * model->dm.F;
            const uint64_t blocks = std::min<uint64_t>((threads + 255) / 256, (uint64_t)model->sm_count * 16);
            count_launch();
            fo2_nu_sum_kernel<<<(unsigned)blocks, 256, 0, model->stream>>>(model->dm, origins_dev, i0, i1, gJ_dev,
                                                                           model->pass, g_nu_dev);
            if ((r = cudaGetLastError()) != cudaSuccess) return r;
        }
        return cudaSuccess;
    };
    e = (model->dm.approx == APPROX_CLOSELINES) ? run(fo2_adj_kernel<APPROX_CLOSELINES>)
                                                : run(fo2_adj_kernel<APPROX_NONE>);
    return finish_stream(model, e, "mgr_formal_solve_fo2_adjoint_device");
}

}  // extern "C"
