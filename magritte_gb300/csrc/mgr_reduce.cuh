// Per-origin reductions of the staged ray-pair results (the formal solve's second
// stage), shared by the single-model reduction kernel and the many-model batch so that
// both sum in the same order.
//   J(o, f)      = sum_rr u(rr, o, f) 2 w_rr, in ray-pair order       (solver.tpp:497-504)
//   Lambda(o, l) = sum_q sum_rr lambda_element(o, rr, f(l, q))         (update_Lambda,
//                  solver.tpp:1760-1800): lane q sums its quadrature point over the ray
//                  pairs in order, the warp then sums its lanes by a butterfly.
// U / LD hold u and L_diag at [(rr - rr0) * stride + (o - o0) * F + f].
#pragma once
#include "mgr_solve.cuh"

namespace mgr {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(FULL_MASK, v, off);
    return v;
}

// Both sums run over values that are already in L2 or stream from memory; what bound them was
// the FP64 pipe (one warp instruction per 16 cycles and SM), six multiplications and an
// addition per ALO element.  The factors that do not depend on the ray pair stand outside the
// sums over it: one multiplication-addition per element of either sum (formal solve of the 33^3
// sphere 19.0 -> 18.4 ms, short characteristics of the 20^3 sphere 1.60 -> 1.22 ms).

// ray_w(o, rr0 + k) as a pointer over k
__device__ __forceinline__ const double* ray_weights(const DevModel& m, uint32_t o, uint32_t rr0) {
    return m.rayw + (m.adaptive ? (size_t)o * m.nrays : (size_t)0) + rr0;
}

// Threads t = 0 .. nt-1 over the frequencies.  2 w u is summed as w u, doubled at the end: exact.
__device__ __forceinline__ void reduce_J_origin(const DevModel& m, uint32_t o, uint32_t rr0, uint32_t nR,
                                                const double* __restrict__ U, size_t u_stride, uint32_t u_o0,
                                                double* __restrict__ J, int t, int nt) {
    const double* wr = ray_weights(m, o, rr0);
    for (uint32_t f = (uint32_t)t; f < m.F; f += (uint32_t)nt) {
        const double* Uo = U + (size_t)(o - u_o0) * m.F + f;
        double s = 0.0;
#pragma unroll 8
        for (uint32_t k = 0; k < nR; k++) s = fma(Uo[(size_t)k * u_stride], wr[k], s);
        J[(size_t)o * m.F + f] = s * 2.0;
    }
}

// Warps w = 0 .. nw-1 over the lines, lanes over the quadrature points.  X: one array of
// L_diag, weighted 2 w (X2 null), or the two directions' factors of the short
// characteristics, each weighted w (lambda_element_sc0; 0 where no pair was solved).
__device__ __forceinline__ void reduce_lam_origin(const DevModel& m, uint32_t o, uint32_t rr0, uint32_t nR,
                                                  const double* __restrict__ X, const double* __restrict__ X2,
                                                  size_t x_stride, uint32_t x_o0, double* __restrict__ lam, int w,
                                                  int nw, int lane) {
    const double* wr = ray_weights(m, o, rr0);
    for (uint32_t l = (uint32_t)w; l < m.L; l += (uint32_t)nw) {
        // lane q: its elements over the ray pairs in order, then the ray-independent factors
        const uint32_t* l2f = m.lq2f + (size_t)l * m.Q;
        double s = 0.0;
        for (uint32_t q0 = 0; q0 < m.Q; q0 += 32) {
            const uint32_t q = q0 + lane;
            const uint32_t f = q < m.Q ? l2f[q] : 0xffffffffu;
            if (f == 0xffffffffu || !m.in_line[f]) continue;
            const double* Xo = X + (size_t)(o - x_o0) * m.F + f;
            double part = 0.0;
            if (X2) {
                const double* X2o = X2 + (size_t)(o - x_o0) * m.F + f;
#pragma unroll 4
                for (uint32_t k = 0; k < nR; k++)
                    part = fma(Xo[(size_t)k * x_stride] + X2o[(size_t)k * x_stride], wr[k], part);
            } else {
#pragma unroll 8
                for (uint32_t k = 0; k < nR; k++) part = fma(Xo[(size_t)k * x_stride], wr[k], part);
                part *= 2.0;
            }
            s += lambda_element_sc0(lambda_factors(m, m.sorted_line, o, f), part, 1.0);
        }
        s = warp_sum(s);
        if (lane == 0) lam[(size_t)o * m.L + l] = s;
    }
}

}  // namespace mgr
