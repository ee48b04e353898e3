// Helpers of the line-solve kernels (hh_tridiag.cu, hh_line_sym.cuh): the eigenvalue-shifted row
// coefficients, the steps of the factor recurrence, shuffles and asynchronous copies.
#ifndef HH_LINE_CUH
#define HH_LINE_CUH

#include "hh_internal.cuh"

namespace hh {

__device__ __forceinline__ double2 shifted(const double2 *__restrict__ tab, int rows, int r, double m0, double m1,
                                           double m2) {
    const double2 a = __ldg(tab + r), b = __ldg(tab + rows + r), c = __ldg(tab + 2 * rows + r),
                  d = __ldg(tab + 3 * rows + r);
    // ((a m0 + b m1) + c m2) + d, as the reference's LU.c:35 orders the 3D sum
    return make_double2(((a.x * m0 + b.x * m1) + c.x * m2) + d.x, ((a.y * m0 + b.y * m1) + c.y * m2) + d.y);
}

// ----------------------------------------------------------------- factors --------
constexpr int kSeg = 8;          // rows per thread in the solve

// One step of the factor recurrence, shared by the set-up and the solve so both produce the
// same values: L = sub / P_prev (as sub * (1/P_prev)), P = diag - L super_prev, returns 1/P.
__device__ __forceinline__ double2 factor_step(double2 sub, double2 dia, double2 sup_prev, double2 ui_prev,
                                               double2 &L) {
    L = make_double2(fma(sub.x, ui_prev.x, -(sub.y * ui_prev.y)), fma(sub.x, ui_prev.y, sub.y * ui_prev.x));
    const double2 P = make_double2(dia.x - fma(L.x, sup_prev.x, -(L.y * sup_prev.y)),
                                   dia.y - fma(L.x, sup_prev.y, L.y * sup_prev.x));
    const double  d = 1.0 / fma(P.x, P.x, P.y * P.y);
    return make_double2(P.x * d, -P.y * d);
}
__device__ __forceinline__ double2 first_pivot(double2 dia) {
    const double d = 1.0 / fma(dia.x, dia.x, dia.y * dia.y);
    return make_double2(dia.x * d, -dia.y * d);
}

__device__ __forceinline__ double2 shfl_up2(double2 v, int off) {
    return make_double2(__shfl_up_sync(0xffffffffu, v.x, off), __shfl_up_sync(0xffffffffu, v.y, off));
}
__device__ __forceinline__ double2 shfl_down2(double2 v, int off) {
    return make_double2(__shfl_down_sync(0xffffffffu, v.x, off), __shfl_down_sync(0xffffffffu, v.y, off));
}

// 16-byte asynchronous global -> shared copy; src_bytes = 0 writes zeros.
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

} // namespace hh

#endif
