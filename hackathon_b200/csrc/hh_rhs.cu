// The reference's right-hand-side assembly rhs() on the device, for plans of any stencil
// (variable k, Dirichlet data): 2D_Program/main_functions/rhs.c:4-150 and
// 3D_Program/main_functions/rhs.c:13-194 with the compact derivatives of
// 2D_Program/partial_derivatives/*.c and 3D_Program/partial_derivatives/*.c.
//
// The Helmholtz plans apply the constant-k operator in the mode basis inside the line solve
// (hh_tridiag.cu); this file is the general form, used where k varies along the line direction
// or the boundary data is not zero.  Its pieces:
//  * Pade derivatives (k_pade): T^-1 v along one axis, T = tridiag(1, d, 1), v the compact right-hand side
//    (12 (f_- - 2 f_0 + f_+) / h^2 for d = 10, 3 (f_+ - f_-) / h for d = 4) with the boundary values subtracted
//    at its two ends;
//  * the pointwise combination of rhs.c (2D :78-86, 3D :149-166) with the second-order
//    differences of 2nd_order*.c inline, and the Dirichlet corrections of the edges (2D rhs.c:126-148)
//    or z faces (3D rhs.c:167-174) at the points they reach.
//
// T^-1 without a sequential pass.  The Thomas recurrence of the reference runs a line from end to end;
// one thread per line left most of the chip idle (2D 511^2: 0.66 to 0.89 ms per derivative).  Here T
// is extended to the whole axis by odd reflection at both ends (v_{-1} = 0, v_{-1-k} = -v_{-1+k}), which
// leaves its solution unchanged, and on the whole axis
//     (T^-1 v)_i = (v_i - r (F_{i-1} + B_{i+1})) / sqrt(d^2 - 4),  F_i = v_i - r F_{i-1},  B_i = v_i - r B_{i+1},
// r = (d - sqrt(d^2 - 4)) / 2.  F and B forget their start by r per point (0.101 at d = 10, 0.268 at d = 4), so a
// thread forms them for its 8 points from W points outside (r^W < 1.3e-17), independently of every other.
// So the derivatives are the reference's to rounding, not its recurrence step by step, and what one point contributes
// beyond its W neighbours, under 1.3e-17 of its value, is left out.  The combination has the reference's terms in
// their order, with reciprocals of the spacings formed once in place of divisions, complex throughout (where
// the reference's 3D rhs.c:149 keeps its partial sums in real doubles; the two agree for real data, which is what
// the reference's own problems have).
#include "hh_internal.cuh"

#include <math.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

namespace hh {

namespace {

constexpr int kPadeThreads = 256, kSegP = 8;
constexpr int kReach10 = 17, kReach4 = 30; // points before r^w is below rounding: 1.2e-17 (d = 10), 7e-18 (d = 4)
constexpr int kSpanS = 64;           // outputs of a block along a strided axis: 8 segments x 32 columns
constexpr int kSpanX = 128, kRowsX = 16; // along x: 16 segments x 16 rows

// One derivative along one axis.  Line (c1, c2), 0 <= c1 < n1, 0 <= c2 < n2, has its interior point m
// (0 <= m < n) at f[f0 + c1 f1 + c2 f2 + m fa] (its neighbours at distance fa, the boundary points included)
// and its derivative at out[c1 o1 + c2 o2 + m oa]; its boundary values are bc[b0 + c1 + c2 b2] (near) and
// bface further on (far).  Strided axes have f1 = o1 = 1 (c1 runs along x), the x axis fa = oa = 1.
struct PadeJob {
    const double2 *f, *bc;
    double2       *out;
    int            n, n1, n2, w, xdir;
    long           f0, f1, f2, fa, o1, o2, oa, b0, b2, bface;
    double         scale, scale_lo; // 12 / h^2 (or 3 / h) over sqrt(d^2 - 4), as a sum of two doubles
    double         r, bscale;       // the decay of F and B; h^2 / 12 (or h / 3)
    unsigned       blocks, gx, gy;  // the job's blocks: gx by gy by (rest)
};
struct PadeJobs {
    PadeJob j[3];
    int     count;
};

__device__ __forceinline__ double2 zaxpy_r(double2 a, double b, double2 c) { // a + b c, b real
    return make_double2(fma(b, c.x, a.x), fma(b, c.y, a.y));
}

__device__ __forceinline__ void pade_async16(double2 *dst, const double2 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void pade_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The difference of f that point m takes, f_{m+1} - f_{m-1} (FIRST) or f_{m-1} - 2 f_m + f_{m+1}; p at m's
// extended position, `step` values between neighbours
template <bool FIRST> __device__ __forceinline__ double2 pade_diff(double2 lo, double2 mid, double2 hi) {
    if (FIRST) return make_double2(hi.x - lo.x, hi.y - lo.y);
    return make_double2(fma(-2.0, mid.x, lo.x + hi.x), fma(-2.0, mid.y, lo.y + hi.y));
}

// v_m of line (c1, c2) over 12 / h^2 (or 3 / h): odd reflection outside the line, the boundary value off the end
// points' v; F(e) is f at extended position e of the line (interior point m at m + 1)
template <int W, bool FIRST, typename Src>
__device__ __forceinline__ double2 pade_rhs(const PadeJob &J, int c1, int c2, int m, Src F) {
    bool neg = false;
    if (J.n > W) { // one reflection reaches the line (v = 0 at -1 and n)
        neg = (unsigned)m >= (unsigned)J.n;
        m = m < 0 ? -2 - m : (m >= J.n ? 2 * J.n - m : m);
        if ((unsigned)m >= (unsigned)J.n) return make_double2(0.0, 0.0);
    } else {
        const int per = 2 * (J.n + 1);
        int       q = (m + 1) % per;
        if (q < 0) q += per;
        if (q == 0 || q == J.n + 1) return make_double2(0.0, 0.0);
        neg = q > J.n + 1;
        m = (neg ? per - q : q) - 1;
    }
    double2 v = pade_diff<FIRST>(F(m), F(m + 1), F(m + 2));
    if (J.bc && (m == 0 || m == J.n - 1)) {
        const double2 b = J.bc[J.b0 + c1 + c2 * J.b2 + (m == 0 ? 0 : J.bface)];
        v = make_double2(fma(-J.bscale, b.x, v.x), fma(-J.bscale, b.y, v.y));
    }
    return neg ? make_double2(-v.x, -v.y) : v;
}

// The two sweeps of one segment of `top` <= 8 points; V(m) is v at the segment's point m, W points reached on
// either side, put(m, value) takes the results in order.
template <int W, bool FULL, typename Val, typename Put>
__device__ __forceinline__ void pade_sweeps(Val V, int top, const PadeJob &J, Put put) {
    const double r = J.r;
    double2 B = make_double2(0.0, 0.0), F = B, Bn[kSegP];
#pragma unroll
    for (int m = kSegP + W - 1; m >= 0; m--) {
        if (m < kSegP) Bn[m] = B;
        if (FULL || m < top + W) B = zaxpy_r(V(m), -r, B);
    }
#pragma unroll
    for (int m = -W; m < 0; m++) F = zaxpy_r(V(m), -r, F);
#pragma unroll
    for (int m = 0; m < kSegP; m++) {
        if (FULL || m < top) {
            const double2 vm = V(m);
            const double2 u = zaxpy_r(vm, -r, make_double2(F.x + Bn[m].x, F.y + Bn[m].y));
            put(m, make_double2(fma(u.x, J.scale, u.x * J.scale_lo), fma(u.y, J.scale, u.y * J.scale_lo)));
            F = zaxpy_r(vm, -r, F);
        }
    }
}

template <int W, typename Val, typename Put>
__device__ __forceinline__ void pade_segment(Val V, int top, const PadeJob &J, Put put) {
    if (top == kSegP) pade_sweeps<W, true>(V, top, J, put);
    else pade_sweeps<W, false>(V, top, J, put);
}

// One block: the values of f that its span reaches come in with asynchronous copies, v is formed from them
// and takes their place, then every thread sweeps one segment.
template <int W> __device__ __forceinline__ void pade_block(const PadeJob &J, unsigned blk, double2 *sm) {
    const int      t = threadIdx.x;
    const unsigned bx = blk % J.gx, by = blk / J.gx % J.gy, bz = blk / J.gx / J.gy;
    const double2  zero = make_double2(0.0, 0.0);
    constexpr bool FIRST = W == kReach4;
    if (!J.xdir) {
        // 32 neighbouring columns, kSpanS points: tiles [point][column]
        const int x0 = (int)bx * 32, m0 = (int)by * kSpanS, c2 = (int)bz, cc = t & 31, c = x0 + cc;
        const int span = min(kSpanS, J.n - m0), len = span + 2 * W;
        const int e0 = max(0, m0 - W), e1 = min(J.n + 1, m0 + span + W + 1); // extended positions needed
        const bool in = c < J.n1;
        {
            const double2 *f = J.f + J.f0 - J.fa + (in ? c : 0) * J.f1 + c2 * J.f2;
            const long     step = (kPadeThreads / 32) * J.fa;
            int            e = e0 + (t >> 5);
            f += e * J.fa;
            for (double2 *to = sm + t; e <= e1; e += kPadeThreads / 32, f += step, to += kPadeThreads) pade_async16(to, f);
        }
        pade_async_wait();
        __syncthreads();
        constexpr int  NV = (kSpanS + 2 * W + 7) / 8;
        double2        vv[NV];
        const double2 *at0 = sm + (m0 - W - e0) * 32 + t; // f left of point m0 - W + (t >> 5)
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int r = (t >> 5) + 8 * i, m = m0 - W + r;
            vv[i] = zero;
            if (in && r < len) {
                const double2 *l = at0 + 256 * i;
                if (m >= 1 && m <= J.n - 2) vv[i] = pade_diff<FIRST>(l[0], l[32], l[64]); // no end near: the same difference
                else vv[i] = pade_rhs<W, FIRST>(J, c, c2, m, [&](int e) { return sm[(e - e0) * 32 + cc]; });
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int r = (t >> 5) + 8 * i;
            if (r < len) sm[t + 256 * i] = vv[i];
        }
        __syncthreads();
        const int i0 = (t >> 5) * kSegP; // the thread's first point within the span
        if (i0 >= span || !in) return;
        const double2 *v = sm + (i0 + W) * 32 + cc;
        double2       *o = J.out + c + c2 * J.o2 + (long)(m0 + i0) * J.oa;
        pade_segment<W>([&](int m) { return v[m * 32]; }, min(kSegP, span - i0), J,
                        [&](int, double2 u) {
                            *o = u;
                            o += J.oa;
                        });
    } else {
        // kRowsX neighbouring rows, kSpanX points: tiles [row][point + point / 8] (the segments of 8 start on
        // different banks)
        constexpr int pitch = (kSpanX + 2 * W + 2) * 9 / 8 + 1;
        const int     m0 = (int)bx * kSpanX, span = min(kSpanX, J.n - m0), len = span + 2 * W;
        const int     e0 = max(0, m0 - W), e1 = min(J.n + 1, m0 + span + W + 1);
        const long    row0 = (long)by * kRowsX, rows = (long)J.n1 * J.n2;
        const int     nr = (int)min((long)kRowsX, rows - row0);
        // thread (r, k): row r, positions k + 16 i
        const int  r = t >> 4, k = t & 15;
        const bool in = r < nr;
        const int  c1 = in ? (int)((row0 + r) % J.n1) : 0, c2 = in ? (int)((row0 + r) / J.n1) : 0;
        double2   *row = sm + r * pitch;
        auto       at = [](int e) { return e + (e >> 3); };
        if (in) {
            const double2 *f = J.f + J.f0 - J.fa + c1 * J.f1 + c2 * J.f2;
            for (int e = e0 + k; e <= e1; e += 16) pade_async16(row + at(e - e0), f + e);
        }
        pade_async_wait();
        __syncthreads();
        constexpr int  NV = (kSpanX + 2 * W + 15) / 16;
        double2        vv[NV];
        const int      p0 = m0 - W - e0 + k; // f left of point m0 - W + k; at(p + 16 i) = at(p) + 18 i
        const double2 *lo = row + at(p0), *mi = row + at(p0 + 1), *hi = row + at(p0 + 2);
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int e = k + 16 * i, m = m0 - W + e;
            vv[i] = zero;
            if (in && e < len) {
                if (m >= 1 && m <= J.n - 2) vv[i] = pade_diff<FIRST>(lo[18 * i], mi[18 * i], hi[18 * i]);
                else vv[i] = pade_rhs<W, FIRST>(J, c1, c2, m, [&](int y) { return row[at(y - e0)]; });
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int e = k + 16 * i;
            if (e < len) row[at(k) + 18 * i] = vv[i];
        }
        __syncthreads();
        const int i0 = k * kSegP, top = in ? max(0, min(kSegP, span - i0)) : 0;
        double2   u[kSegP];
        if (top > 0) // at(8 k + W + m) = 9 k + at(W + m)
            pade_segment<W>([&](int m) { return row[9 * k + at(W + m)]; }, top, J, [&](int m, double2 x) { u[m] = x; });
        __syncthreads(); // the tile takes the results, for contiguous stores
#pragma unroll
        for (int m = 0; m < kSegP; m++)
            if (m < top) row[9 * k + m] = u[m];
        __syncthreads();
        if (in) {
            double2 *o = J.out + c1 * J.o1 + c2 * J.o2 + m0;
            for (int e = k; e < span; e += 16) o[e] = row[at(e)];
        }
    }
}

// Bound by shared memory (56 % of its wavefronts) and instruction issue: a point costs 1.5 to 2 values of v and a
// segment of 8 points 2 (W + 8) steps of one fused multiply-add per component.  Points with no end near take the
// plain difference at constant offsets: 33.7 -> 25.7 million warp instructions at 125^3, assembly and solve of 2D
// 511^2 51.1 -> 50.0 us, of 3D 125^3 255 -> 253.  All derivatives of an assembly share one launch.
__global__ void __launch_bounds__(kPadeThreads, 3) k_pade(const __grid_constant__ PadeJobs jobs) {
    extern __shared__ __align__(16) double2 pade_sm[];
    unsigned blk = blockIdx.x;
    int      ji = 0;
    while (ji + 1 < jobs.count && blk >= jobs.j[ji].blocks) blk -= jobs.j[ji++].blocks;
    pdl_wait();
    pdl_next();
    if (jobs.j[ji].w == kReach10) pade_block<kReach10>(jobs.j[ji], blk, pade_sm);
    else pade_block<kReach4>(jobs.j[ji], blk, pade_sm);
}

__device__ __forceinline__ double2 zmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 rmul(double a, double2 b) { return make_double2(a * b.x, a * b.y); }
// a - 2 b + c
__device__ __forceinline__ double2 d2(double2 a, double2 b, double2 c) {
    return make_double2(a.x - 2.0 * b.x + c.x, a.y - 2.0 * b.y + c.y);
}

// a field of derivatives at interior points, with its values on the boundary in two pairs of face arrays
// (null: zero)
struct Rhs2DArgs {
    const double2 *fe, *fxx, *fyy, *fy, *k2c, *k2y;
    const double2 *fxx_xb, *fxx_yb, *fyy_yb;
    const double2 *subt, *diagt, *supt; // plan rows [4][prow]: sub (bm at [1], am at [3]), diag (b at [1]), super (bp, ap)
    const double  *ux, *uy;
    double2       *rhs;
    int            nx, ny, order, prow;
    double         h2, h2_20, c_f, c_xxxx, c_yyyy, c_xxyy, c_y; // h^2, h^2/20, h^2/12, h^4/(360 hx^2), ..., h^4/60
};

// 2D combination, rhs.c:78-86 (order 6); orders 4 and 2, rhs.c:4-38; then the Dirichlet corrections of
// the points next to an edge, rhs.c:126-148 (the ring's corners belong to the edges y = const)
__global__ void __launch_bounds__(256) k_rhs2d_combine(const __grid_constant__ Rhs2DArgs A) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = blockIdx.y * 8 + (threadIdx.x >> 5);
    pdl_wait();
    pdl_next();
    if (i >= A.nx || j >= A.ny) return;
    const int  nx = A.nx, ny = A.ny;
    const long E = nx + 2, c = (i + 1) + (long)(j + 1) * E, q = i + (long)j * nx;
    double2    r;
    if (A.order == 6) {
        const double2 zero = make_double2(0.0, 0.0);
        auto face = [&](const double2 *b, long at) { return b ? b[at] : zero; };
        const double2 xx = A.fxx[q], yy = A.fyy[q];
        const double2 xl = i > 0 ? A.fxx[q - 1] : face(A.fxx_xb, j + 1);
        const double2 xr = i + 1 < nx ? A.fxx[q + 1] : face(A.fxx_xb, ny + 2 + j + 1);
        const double2 xd = j > 0 ? A.fxx[q - nx] : face(A.fxx_yb, i + 1);
        const double2 xu = j + 1 < ny ? A.fxx[q + nx] : face(A.fxx_yb, E + i + 1);
        const double2 yd = j > 0 ? A.fyy[q - nx] : face(A.fyy_yb, i + 1);
        const double2 yu = j + 1 < ny ? A.fyy[q + nx] : face(A.fyy_yb, E + i + 1);
        const double2 k2 = A.k2c[j];
        const double2 t1 = zmul(make_double2(1.0 - k2.x * A.h2_20, -(k2.y * A.h2_20)), A.fe[c]);
        const double2 t2 = rmul(A.c_f, zadd(xx, yy));
        const double2 t3 = zadd(rmul(A.c_xxxx, d2(xl, xx, xr)), rmul(A.c_yyyy, d2(yd, yy, yu)));
        const double2 t4 = rmul(A.c_xxyy, d2(xd, xx, xu));
        const double2 t5 = zmul(rmul(A.c_y, A.k2y[j]), A.fy[q]);
        r = rmul(A.h2, zadd(zadd(zadd(zadd(t1, t2), t3), t4), t5));
    } else if (A.order == 4) {
        const double  a = 2.0 / 3.0, b = 1.0 / 12.0;
        const double2 s = zadd(zadd(zadd(A.fe[c - E], A.fe[c + E]), A.fe[c - 1]), A.fe[c + 1]);
        r = rmul(A.h2, zadd(rmul(a, A.fe[c]), rmul(b, s)));
    } else {
        r = rmul(A.h2, A.fe[c]);
    }
    if ((A.ux || A.uy) && (i == 0 || j == 0 || i == nx - 1 || j == ny - 1)) {
        auto U = [&](const double *a, long at) { return a ? a[at] : 0.0; };
        auto ring = [&](int ie, int je) { // Dirichlet value at a point of the ring, zero inside
            if (je == 0) return U(A.uy, ie);
            if (je == ny + 1) return U(A.uy, E + ie);
            if (ie == 0) return U(A.ux, je);
            return ie == nx + 1 ? U(A.ux, ny + 2 + je) : 0.0;
        };
        auto sub = [&](double2 co, double u) { r = make_double2(r.x - co.x * u, r.y - co.y * u); };
        const int p = A.prow;
        sub(A.subt[p + j], ring(i, j));
        sub(A.subt[3 * p + j], ring(i + 1, j));
        sub(A.subt[p + j], ring(i + 2, j));
        sub(A.diagt[p + j], ring(i, j + 1));
        sub(A.diagt[p + j], ring(i + 2, j + 1));
        sub(A.supt[p + j], ring(i, j + 2));
        sub(A.supt[3 * p + j], ring(i + 1, j + 2));
        sub(A.supt[p + j], ring(i + 2, j + 2));
    }
    A.rhs[q] = r;
}

struct Rhs3DArgs {
    const double2 *f, *fxx, *fyy, *fzz, *k2_ext, *kp;
    const double2 *fxx_b, *fyy_b, *fzz_b; // face values, each near face then far face
    const double2 *subt, *supt, *ue;
    double2       *rhs;
    int            nx, ny, nz, order, prow;
    double h2_20, c_f, c_xxxx, c_yyyy, c_zzzz, c_xxyy, c_xxzz, c_yyzz, c_z; // hz^2/20, hz^2/12, hz^4/(360 hx^2), ..., hz^3/120
};

// 3D combination, rhs.c:149-166 (order 6); orders 4 and 2, rhs.c:13-62; then the z-face Dirichlet terms,
// rhs.c:24-29, 55-62, 167-174: layer 0 with the sub-diagonal layer's stencil (am, bm, cm, dm of layer
// 0), layer nz-1 with the super-diagonal one (ap..dp of nz-1).  fxx on the y and z faces, fyy on the x
// and z faces and fzz on the x and y faces are zero, as the reference leaves them.
//
// A thread marches through RUN layers of its (i, j) with the layers below, at and above in registers, the
// one after those on its way: each field crosses L2 once instead of three times.
// A block is 2^LW points wide in x, 256 / 2^LW in y.
template <int RUN, int LW> __global__ void __launch_bounds__(256) k_rhs3d_combine(const __grid_constant__ Rhs3DArgs A) {
    const int i = (blockIdx.x << LW) + (threadIdx.x & ((1 << LW) - 1)), j = (blockIdx.y << (8 - LW)) + (threadIdx.x >> LW);
    pdl_wait();
    pdl_next();
    if (i >= A.nx || j >= A.ny) return;
    const int     nx = A.nx, ny = A.ny, nz = A.nz, l0 = blockIdx.z * RUN, l1 = min(nz, l0 + RUN);
    const long    Ex = nx + 2, Ey = ny + 2, Exy = Ex * Ey, nxy = (long)nx * ny;
    const double2 zero = make_double2(0.0, 0.0);
    const bool    six = A.order == 6;
    const long    Cij = (i + 1) + (j + 1) * Ex, qij = i + (long)j * nx;
    auto face = [&](const double2 *b, long at) { return b ? b[at] : zero; };
    // the centre values of layer l (f at -1 .. nz, the derivatives zero outside, fzz its face values)
    auto F = [&](int l) { return A.f[Cij + (l + 1) * Exy]; };
    auto D = [&](const double2 *d, int l) { return l >= 0 && l < nz ? d[qij + l * nxy] : zero; };
    auto Z = [&](int l) {
        if (l < 0) return face(A.fzz_b, Cij);
        return l < nz ? A.fzz[qij + l * nxy] : face(A.fzz_b, Cij + Exy);
    };
    double2 fd = zero, f0 = zero, fu = zero, xd = zero, xx = zero, xu = zero, yd = zero, yy = zero, yu = zero, zd = zero,
            zz = zero, zu = zero;
    if (six) {
        fd = F(l0 - 1), f0 = F(l0), fu = F(l0 + 1);
        xd = D(A.fxx, l0 - 1), xx = D(A.fxx, l0), xu = D(A.fxx, l0 + 1);
        yd = D(A.fyy, l0 - 1), yy = D(A.fyy, l0), yu = D(A.fyy, l0 + 1);
        zd = Z(l0 - 1), zz = Z(l0), zu = Z(l0 + 1);
    }
    for (int l = l0; l < l1; l++) {
        const long C = Cij + (l + 1) * Exy, q = qij + l * nxy;
        double2    r;
        if (six) {
            double2 fn = zero, xn2 = zero, yn2 = zero, zn2 = zero; // layer l + 2, on its way
            if (l + 1 < l1) {
                fn = F(l + 2);
                xn2 = D(A.fxx, l + 2);
                yn2 = D(A.fyy, l + 2);
                zn2 = Z(l + 2);
            }
            const double2 xw = i > 0 ? A.fxx[q - 1] : face(A.fxx_b, (j + 1) + (l + 1) * Ey);
            const double2 xe = i + 1 < nx ? A.fxx[q + 1] : face(A.fxx_b, (j + 1) + (l + 1) * Ey + Ey * (nz + 2));
            const double2 xs = j > 0 ? A.fxx[q - nx] : zero, xn = j + 1 < ny ? A.fxx[q + nx] : zero;
            const double2 ys = j > 0 ? A.fyy[q - nx] : face(A.fyy_b, (i + 1) + (l + 1) * Ex);
            const double2 yn = j + 1 < ny ? A.fyy[q + nx] : face(A.fyy_b, (i + 1) + (l + 1) * Ex + Ex * (nz + 2));
            const double2 k2 = A.k2_ext[l + 1];
            const double2 first = zmul(make_double2(1.0 - k2.x * A.h2_20, -(k2.y * A.h2_20)), f0);
            const double2 second = rmul(A.c_f, zadd(zadd(xx, yy), zz));
            const double2 third = zadd(zadd(rmul(A.c_xxxx, d2(xw, xx, xe)), rmul(A.c_yyyy, d2(ys, yy, yn))),
                                       rmul(A.c_zzzz, d2(zd, zz, zu)));
            const double2 fourth = zadd(zadd(rmul(A.c_xxyy, d2(xs, xx, xn)), rmul(A.c_xxzz, d2(xd, xx, xu))),
                                        rmul(A.c_yyzz, d2(yd, yy, yu)));
            const double2 fifth = zmul(rmul(A.c_z, A.kp[l]), zsub(fu, fd));
            r = zadd(zadd(zadd(zadd(first, second), third), fourth), fifth);
            fd = f0, f0 = fu, fu = fn;
            xd = xx, xx = xu, xu = xn2;
            yd = yy, yy = yu, yu = yn2;
            zd = zz, zz = zu, zu = zn2;
        } else if (A.order == 4) {
            const double2 nb = zadd(zadd(zadd(zadd(zadd(A.f[C - 1], A.f[C + 1]), A.f[C - Ex]), A.f[C + Ex]), A.f[C - Exy]), A.f[C + Exy]);
            r = zadd(A.f[C], rmul(1.0 / 12.0, zsub(nb, rmul(6.0, A.f[C]))));
        } else {
            r = A.f[C];
        }
        if (A.ue) {
            for (int far = 0; far < 2; far++) {
                if (l != (far ? nz - 1 : 0)) continue;
                const double2 *e = A.ue + (far ? (nz + 1) * Exy : 0);
                auto           X = [&](int ie, int je) { return e[ie + je * Ex]; };
                if (A.order == 2) {
                    r = zsub(r, X(i + 1, j + 1));
                    continue;
                }
                const double2 *tab = far ? A.supt : A.subt;
                const double2  a = tab[l], bb = tab[A.prow + l], cc = tab[2 * A.prow + l], dd = tab[3 * A.prow + l];
                r = zsub(r, zmul(a, zadd(zadd(zadd(X(i, j), X(i + 2, j)), X(i, j + 2)), X(i + 2, j + 2))));
                r = zsub(r, zmul(bb, zadd(X(i, j + 1), X(i + 2, j + 1))));
                r = zsub(r, zmul(cc, zadd(X(i + 1, j), X(i + 1, j + 2))));
                r = zsub(r, zmul(dd, X(i + 1, j + 1)));
            }
        }
        A.rhs[q] = r;
    }
}

// Pade factors of tridiag(1, diag, 1) over n points, as the reference forms them
void pade_factors(int n, double diag, std::vector<double> &L, std::vector<double> &U) {
    L.assign((size_t)n, 0.0);
    U.assign((size_t)n, 0.0);
    U[0] = diag;
    for (int j = 1; j < n; j++) {
        L[(size_t)j] = 1.0 / U[(size_t)j - 1];
        U[(size_t)j] = diag - L[(size_t)j];
    }
}

// complex line of the reference's Pade recurrence on the host (the O(n) k profiles)
void pade_host(std::vector<double2> &v, double diag) {
    const int           n = (int)v.size();
    std::vector<double> L, U;
    pade_factors(n, diag, L, U);
    for (int j = 1; j < n; j++) v[j] = make_double2(v[j].x - L[j] * v[j - 1].x, v[j].y - L[j] * v[j - 1].y);
    v[n - 1] = make_double2(v[n - 1].x / U[n - 1], v[n - 1].y / U[n - 1]);
    for (int j = n - 2; j >= 0; j--) v[j] = make_double2((v[j].x - v[j + 1].x) / U[j], (v[j].y - v[j + 1].y) / U[j]);
}

double2 hmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

} // namespace

// Workspace of the assembly: `count` complex values, grown on demand (outside stream capture).
static int rhs_work(Ctx *c, long count, double2 **out) {
    if (c->rhs_elems < count) {
        HH_CUDA(cudaStreamSynchronize(c->stream));
        cudaFree(c->rhs_work);
        c->rhs_work = nullptr;
        c->rhs_elems = 0;
        HH_CUDA(cudaMalloc(&c->rhs_work, sizeof(double2) * (size_t)count));
        c->rhs_elems = count;
    }
    *out = c->rhs_work;
    return HH_OK;
}

// a small host table on the device, in the context's table area (stream-ordered upload)
struct TableArea {
    Ctx               *c;
    std::vector<char>  host;
    std::vector<size_t> offs;
    size_t add(const void *p, size_t bytes) {
        const size_t off = (host.size() + 255) / 256 * 256;
        host.resize(off + bytes);
        memcpy(host.data() + off, p, bytes);
        offs.push_back(off);
        return off;
    }
};

static int upload_tables(Ctx *c, TableArea &ta, char **dev) {
    if (c->rhs_tab_bytes < ta.host.size()) {
        HH_CUDA(cudaStreamSynchronize(c->stream));
        cudaFree(c->rhs_tab);
        c->rhs_tab = nullptr;
        c->rhs_tab_bytes = 0;
        HH_CUDA(cudaMalloc(&c->rhs_tab, ta.host.size()));
        c->rhs_tab_bytes = ta.host.size();
    }
    // a copy from pageable memory returns once the values are staged, so the caller may free them; a
    // capture would record their address instead
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    HH_CUDA(cudaStreamIsCapturing(c->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) {
        set_error("the order-6 right-hand side copies its k profile from the host: not during stream capture");
        return HH_ERR_CUDA;
    }
    HH_CUDA(cudaMemcpyAsync(c->rhs_tab, ta.host.data(), ta.host.size(), cudaMemcpyHostToDevice, c->stream));
    *dev = static_cast<char *>(c->rhs_tab);
    return HH_OK;
}

// a derivative job over tridiag(1, diag, 1) (10: second derivative, 4: first) with spacing h
static PadeJob pade_job(const double2 *f, double2 *out, const double *bc, int n, int n1, int n2, int diag, double h, bool xdir) {
    PadeJob J{};
    J.f = f;
    J.out = out;
    J.bc = (const double2 *)bc;
    J.n = n;
    J.n1 = n1;
    J.n2 = n2;
    J.xdir = xdir;
    J.w = diag == 4 ? kReach4 : kReach10;
    const long double hl = h, sc = diag == 4 ? 3.0L / hl : 12.0L / (hl * hl);
    J.bscale = (double)(1.0L / sc);
    const long double root = sqrtl((long double)diag * diag - 4.0L);
    J.r = (double)(2.0L / (diag + root));
    J.scale = (double)(sc / root);
    J.scale_lo = (double)(sc / root - (long double)J.scale);
    if (xdir) {
        J.gx = (unsigned)((n + kSpanX - 1) / kSpanX);
        J.gy = (unsigned)(((long)n1 * n2 + kRowsX - 1) / kRowsX);
        J.blocks = J.gx * J.gy;
    } else {
        J.gx = (unsigned)((n1 + 31) / 32);
        J.gy = (unsigned)((n + kSpanS - 1) / kSpanS);
        J.blocks = J.gx * J.gy * (unsigned)n2;
    }
    return J;
}

static size_t pade_smem(bool xdir, int w) {
    return sizeof(double2) * (xdir ? (size_t)kRowsX * ((kSpanX + 2 * w + 2) * 9 / 8 + 1) : (size_t)(kSpanS + 2 * w + 2) * 32);
}

static int launch_pade(Ctx *c, const PadeJobs &jobs) {
    long   blocks = 0;
    size_t shm = 0;
    for (int i = 0; i < jobs.count; i++) {
        const PadeJob &J = jobs.j[i];
        blocks += J.blocks;
        shm = std::max(shm, pade_smem(J.xdir, J.w));
    }
    if (blocks > 0x7fffffffL) {
        set_error("right-hand side: grid too large");
        return HH_ERR_UNSUPPORTED;
    }
    HH_TRY(allow_smem(k_pade, std::max(pade_smem(true, kReach4), pade_smem(false, kReach4))));
    return launch_kernel(c, k_pade, dim3((unsigned)blocks), kPadeThreads, shm, jobs);
}

int assemble_rhs2d(Plan *p, const hh_rhs2d_data *d, double2 *rhs) {
    Ctx       *c = p->ctx;
    const int  nx = p->nx, ny = p->ny, order = d->order;
    const long E = nx + 2, nxy = (long)nx * ny;
    Rhs2DArgs  A{};
    A.fe = (const double2 *)d->f_ext;
    if (order == 6) {
        // host: the k profiles (O(ny))
        std::vector<double2> k2c((size_t)ny), k2y((size_t)ny);
        const double2       *ke = (const double2 *)d->k_ext;
        for (int j = 0; j < ny; j++) {
            k2c[(size_t)j] = hmul(ke[j + 1], ke[j + 1]);
            const double2 kp2 = hmul(ke[j + 2], ke[j + 2]), km2 = hmul(ke[j], ke[j]);
            k2y[(size_t)j] = make_double2(3.0 * (kp2.x - km2.x) / d->hy, 3.0 * (kp2.y - km2.y) / d->hy);
        }
        if (d->k2y_bc) {
            const double2 *bc = (const double2 *)d->k2y_bc;
            k2y[0] = make_double2(k2y[0].x - bc[0].x, k2y[0].y - bc[0].y);
            k2y[(size_t)ny - 1] = make_double2(k2y[(size_t)ny - 1].x - bc[1].x, k2y[(size_t)ny - 1].y - bc[1].y);
        }
        pade_host(k2y, 4.0);
        TableArea    ta{c, {}, {}};
        const size_t o_k2c = ta.add(k2c.data(), 16 * k2c.size()), o_k2y = ta.add(k2y.data(), 16 * k2y.size());
        char        *tab;
        HH_TRY(upload_tables(c, ta, &tab));
        double2 *w = nullptr;
        HH_TRY(rhs_work(c, 3 * nxy, &w));
        double2 *fxx = w, *fyy = w + nxy, *fy = w + 2 * nxy;
        PadeJobs jobs;
        jobs.count = 3;
        // f_y: [1 4 1] along y (4th_order_first_derivative.c:60-98), boundary values fy_yb (interior x)
        PadeJob &Y1 = jobs.j[0] = pade_job(A.fe, fy, d->fy_yb, ny, nx, 1, 4, d->hy, false);
        Y1.f0 = 1 + E, Y1.f1 = 1, Y1.fa = E, Y1.o1 = 1, Y1.oa = nx, Y1.b0 = 0, Y1.bface = nx;
        // f_yy: [1 10 1] along y (4th_order_second_derivative.c:61-120)
        PadeJob &Y2 = jobs.j[1] = pade_job(A.fe, fyy, d->fyy_yb, ny, nx, 1, 10, d->hy, false);
        Y2.f0 = 1 + E, Y2.f1 = 1, Y2.fa = E, Y2.o1 = 1, Y2.oa = nx, Y2.b0 = 1, Y2.bface = E;
        // f_xx: [1 10 1] along x (4th_order_second_derivative.c:4-59)
        PadeJob &X2 = jobs.j[2] = pade_job(A.fe, fxx, d->fxx_xb, nx, ny, 1, 10, d->hx, true);
        X2.f0 = 1 + E, X2.f1 = E, X2.fa = 1, X2.o1 = nx, X2.oa = 1, X2.b0 = 1, X2.bface = ny + 2;
        HH_TRY(launch_pade(c, jobs));
        A.fxx = fxx, A.fyy = fyy, A.fy = fy;
        A.k2c = reinterpret_cast<const double2 *>(tab + o_k2c);
        A.k2y = reinterpret_cast<const double2 *>(tab + o_k2y);
        A.fxx_xb = (const double2 *)d->fxx_xb;
        A.fxx_yb = (const double2 *)d->fxx_yb;
        A.fyy_yb = (const double2 *)d->fyy_yb;
    }
    const double hx2 = d->hx * d->hx, hy2 = d->hy * d->hy, hy4 = hy2 * hy2;
    A.h2 = hy2;
    A.h2_20 = hy2 / 20.0;
    A.c_f = hy2 / 12.0;
    A.c_xxxx = hy4 / hx2 / 360.0;
    A.c_yyyy = hy2 / 360.0;
    A.c_xxyy = hy2 / 90.0;
    A.c_y = hy4 / 60.0;
    A.subt = p->subt, A.diagt = p->diagt, A.supt = p->rowc;
    A.ux = d->u_xb, A.uy = d->u_yb;
    A.rhs = rhs;
    A.nx = nx, A.ny = ny, A.order = order, A.prow = p->prow;
    dim3 grid((unsigned)((nx + 31) / 32), (unsigned)((ny + 7) / 8));
    return launch_kernel(c, k_rhs2d_combine, grid, 256, 0, A);
}

int assemble_rhs3d(Plan *p, const hh_rhs3d_data *d, double2 *rhs) {
    Ctx       *c = p->ctx;
    const int  nx = p->nx, ny = p->ny, nz = p->nz, order = d->order;
    const long Ex = nx + 2, Ey = ny + 2, Exy = Ex * Ey, nxy = (long)nx * ny, n3 = nxy * nz;
    Rhs3DArgs  A{};
    A.f = (const double2 *)d->f_ext;
    if (order == 6) {
        // host: d(k^2)/dz by the [1 4 1] scheme (4th_order_partials.c:296-340)
        const double2       *k2 = (const double2 *)d->k2_ext;
        std::vector<double2> kp((size_t)nz);
        for (int l = 0; l < nz; l++)
            kp[(size_t)l] = make_double2(3.0 * (k2[l + 2].x - k2[l].x) / d->hz, 3.0 * (k2[l + 2].y - k2[l].y) / d->hz);
        if (d->kz_bc) {
            const double2 *bc = (const double2 *)d->kz_bc;
            kp[0] = make_double2(kp[0].x + bc[0].x, kp[0].y + bc[0].y);
            kp[(size_t)nz - 1] = make_double2(kp[(size_t)nz - 1].x + bc[1].x, kp[(size_t)nz - 1].y + bc[1].y);
        }
        pade_host(kp, 4.0);
        TableArea    ta{c, {}, {}};
        const size_t o_kp = ta.add(kp.data(), 16 * kp.size()), o_k2 = ta.add(k2, 16 * (size_t)(nz + 2));
        char        *tab;
        HH_TRY(upload_tables(c, ta, &tab));
        double2 *w = nullptr;
        HH_TRY(rhs_work(c, 3 * n3, &w));
        double2 *fxx = w, *fyy = w + n3, *fzz = w + 2 * n3;
        PadeJobs jobs;
        jobs.count = 3;
        const long f0 = 1 + Ex + Exy;
        // f_xx along x (4th_order_partials.c:94-160): lines (j, l), boundary layout j + l (ny+2)
        PadeJob &X = jobs.j[0] = pade_job(A.f, fxx, d->fxx_b, nx, ny, nz, 10, d->hx, true);
        X.f0 = f0, X.f1 = Ex, X.f2 = Exy, X.fa = 1, X.o1 = nx, X.o2 = nxy, X.oa = 1;
        X.b0 = 1 + Ey, X.b2 = Ey, X.bface = Ey * (nz + 2);
        // f_yy along y (:162-227): lines (i, l), boundary layout i + l (nx+2)
        PadeJob &Y = jobs.j[1] = pade_job(A.f, fyy, d->fyy_b, ny, nx, nz, 10, d->hy, false);
        Y.f0 = f0, Y.f1 = 1, Y.f2 = Exy, Y.fa = Ex, Y.o1 = 1, Y.o2 = nxy, Y.oa = nx;
        Y.b0 = 1 + Ex, Y.b2 = Ex, Y.bface = Ex * (nz + 2);
        // f_zz along z (:229-294): lines (i, j), boundary layout i + j (nx+2)
        PadeJob &Z = jobs.j[2] = pade_job(A.f, fzz, d->fzz_b, nz, nx, ny, 10, d->hz, false);
        Z.f0 = f0, Z.f1 = 1, Z.f2 = Ex, Z.fa = Exy, Z.o1 = 1, Z.o2 = nx, Z.oa = nxy;
        Z.b0 = 1 + Ex, Z.b2 = Ex, Z.bface = Exy;
        HH_TRY(launch_pade(c, jobs));
        A.fxx = fxx, A.fyy = fyy, A.fzz = fzz;
        A.k2_ext = reinterpret_cast<const double2 *>(tab + o_k2);
        A.kp = reinterpret_cast<const double2 *>(tab + o_kp);
        A.fxx_b = (const double2 *)d->fxx_b;
        A.fyy_b = (const double2 *)d->fyy_b;
        A.fzz_b = (const double2 *)d->fzz_b;
    }
    const double hx2 = d->hx * d->hx, hy2 = d->hy * d->hy, hz2 = d->hz * d->hz, hz4 = hz2 * hz2;
    A.h2_20 = hz2 / 20.0;
    A.c_f = hz2 / 12.0;
    A.c_xxxx = hz4 / hx2 / 360.0;
    A.c_yyyy = hz4 / hy2 / 360.0;
    A.c_zzzz = hz2 / 360.0;
    A.c_xxyy = hz4 / hy2 / 90.0;
    A.c_xxzz = A.c_yyzz = hz2 / 90.0;
    A.c_z = hz2 * d->hz / 120.0;
    A.subt = p->subt, A.supt = p->rowc, A.ue = (const double2 *)d->ue_ext;
    A.rhs = rhs;
    A.nx = nx, A.ny = ny, A.nz = nz, A.order = order, A.prow = p->prow;
    if (nz > 65535 || (ny + 7) / 8 > 65535) {
        set_error("hh_rhs3d: %d x %d x %d is too large", nx, ny, nz);
        return HH_ERR_UNSUPPORTED;
    }
    // Layers per block: 16, or 8 or 4 where the blocks are then still all resident at once (two to an SM), so that a
    // small problem does not march through 16 layers on a part of the chip.  Assembly and solve against 16: 31^3
    // 47.0 -> 43.0 us, 48^3 54.2 -> 43.5, 63^3 65.5 -> 53.8.
    // As a kernel argument the run cost 2.5 % at 125^3; 32 layers in one wave were slower (127^3 238 -> 253 us).
    // Blocks 32 points wide, or 16 or 8 where nx is no more, whose lanes would idle: 8 x 300 x 300 at order 4 19.4 -> 8.2
    // us, 5 x 200 x 300 13.6 -> 6.3.
    auto width = [&](auto lw_c) {
        constexpr int LW = decltype(lw_c)::value;
        const long    bx = (nx + (1 << LW) - 1) >> LW, by = (ny + (256 >> LW) - 1) / (256 >> LW);
        auto          go = [&](auto kernel, int run) {
            return launch_kernel(c, kernel, dim3((unsigned)bx, (unsigned)by, (unsigned)((nz + run - 1) / run)), 256, 0, A);
        };
        if (bx * by * ((nz + 3) / 4) <= 2 * 148) return go(k_rhs3d_combine<4, LW>, 4);
        if (bx * by * ((nz + 7) / 8) <= 2 * 148) return go(k_rhs3d_combine<8, LW>, 8);
        return go(k_rhs3d_combine<16, LW>, 16);
    };
    if (nx <= 8) return width(std::integral_constant<int, 3>{});
    if (nx <= 16) return width(std::integral_constant<int, 4>{});
    return width(std::integral_constant<int, 5>{});
}

} // namespace hh
