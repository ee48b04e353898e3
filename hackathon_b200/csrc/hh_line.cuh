// Helpers of the line-solve kernels (hh_tridiag.cu, hh_line_sym.cuh): the eigenvalue-shifted row
// coefficients, the steps of the factor recurrence, shuffles and asynchronous copies.
#ifndef HH_LINE_CUH
#define HH_LINE_CUH

#include "hh_internal.cuh"

#include <type_traits>

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

// a + b c and a - b c with two fused multiply-adds per component
__device__ __forceinline__ double2 zfma(double2 a, double2 b, double2 c) {
    return make_double2(fma(b.x, c.x, fma(-b.y, c.y, a.x)), fma(b.x, c.y, fma(b.y, c.x, a.y)));
}
__device__ __forceinline__ double2 zfms(double2 a, double2 b, double2 c) {
    return make_double2(fma(-b.x, c.x, fma(b.y, c.y, a.x)), fma(-b.x, c.y, fma(-b.y, c.x, a.y)));
}
__device__ __forceinline__ double2 zaxpy(double2 a, double b, double2 c) { // a + b c, b real
    return make_double2(fma(b, c.x, a.x), fma(b, c.y, a.y));
}

// The line coefficients are complex (MT = double2) or, where k^2 is real, real (MT = double).  On
// real coefficients the real form does the arithmetic of the complex one without its exact zeros:
// every finite result has the same bits, with half the fused multiply-adds, half the latency of
// each recurrence step and half the registers and shared memory of the multipliers (tile input, line
// solve, complex -> real: 2D 1023^2 x 64 order 6 678 -> 597 us, order 4 528 -> 507 us; 2047^2 x 16 order 6
// 845 -> 726 us; 3D 255^3 x 4 order 6 709 -> 552 us).
__device__ __forceinline__ double2 zfma(double2 a, double b, double2 c) { return zaxpy(a, b, c); }
__device__ __forceinline__ double2 zfms(double2 a, double b, double2 c) { return zaxpy(a, -b, c); }
__device__ __forceinline__ double2 cmul(double a, double2 b) { return make_double2(a * b.x, a * b.y); }
__device__ __forceinline__ double  cmul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 mneg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ double  mneg(double a) { return -a; }
// crcp, factor_step and first_pivot on a zero imaginary part (the products rounded on their own, as there)
__device__ __forceinline__ double crcp(double x) { return x * (1.0 / __dmul_rn(x, x)); }
__device__ __forceinline__ double first_pivot(double dia) { return crcp(dia); }
__device__ __forceinline__ double factor_step(double sub, double dia, double sup_prev, double ui_prev, double &L) {
    L = sub * ui_prev;
    return crcp(dia - __dmul_rn(L, sup_prev));
}
template <typename MT> __device__ __forceinline__ MT coef_of(double2 v) {
    if constexpr (std::is_same_v<MT, double>) return v.x;
    else return v;
}
__device__ __forceinline__ double coef_re(double v) { return v; }
__device__ __forceinline__ double coef_re(double2 v) { return v.x; }
template <typename MT> constexpr bool is_real_v = std::is_same_v<MT, double>;

__device__ __forceinline__ double2 coef_full(double v) { return make_double2(v, 0.0); }
__device__ __forceinline__ double2 coef_full(double2 v) { return v; }

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
