// Shifted tridiagonal line solves for sm_100a (FP64 complex).
//
// Replaces the reference's per-mode Thomas solves: 2D_Program/solver_functions/solver.c:71-86
// (per x-mode i along y, factors from main_functions/LU.c:3-46) and
// 3D_Program/solver_functions/solver.c:483-496 / cuda_kernels.cu:208-249 (per (i,j) along z,
// factors from main_functions/LU.c:4-81).
//
// Geometry.  A right-hand side holds `lines` independent lines of `rows` points; point
// (row r, line q) sits at offset r*row_stride + q.  2D: line = x-mode i, row = y index j,
// row_stride = Nx (the DST output layout, no transpose).  3D: line = i + j*Nx, row = z
// layer l, row_stride = Nx*Ny.  Consecutive lines are contiguous, so a warp always reads
// whole row segments (the "interleaved" layout).
//
// Line matrix (row r, line q), with per-row coefficient tables and per-line multipliers mu:
//   sub(r,q)   = subc0[r] mu0[q] + subc1[r] mu1[q] + subc2[r] mu2[q] + subc3[r]
//   diag(r,q)  = same with diagc,   super(r,q) = same with supc
// 2D: mu = (0, lambda_i, 0):   sub = bm lambda + am, diag = b lambda + a, super = bp lambda + ap
// 3D: mu = (lx*ly, lx, ly):    sub = am lx ly + bm lx + cm ly + dm, etc.
// This is the reference's eigenvalue shift (2D LU.c:16-23, 3D LU.c:35-47) evaluated on the fly.
//
// Factorisation (set-up, once per plan): Thomas without pivoting, exactly the reference's
// recurrence  L_0 = 0, P_0 = diag_0,  L_r = sub_r / P_{r-1},  P_r = diag_r - L_r super_{r-1};
// the device keeps L_r and 1/P_r in [row][line] layout.
//
// Solve: each thread owns a segment of kSeg = 8 consecutive rows of one line.  Only the
// reciprocal pivot entering each segment is stored by the set-up; the thread re-runs the
// factor recurrence for its own rows into registers (the same arithmetic, so the factors are
// those of the sequential factorisation) and keeps them for every right-hand side of its
// chunk.  Forward substitution y_r = f_r - L_r y_{r-1} and back substitution
// x_r = (y_r - super_r x_{r+1}) / P_r are first-order linear recurrences: each segment applies
// its rows as an affine map y_out = A y_in + B of the value entering it.  A (product of the
// segment's multipliers) depends on the factors only; B comes from a local sweep.  The maps of
// a line are composed across its segments by a warp-shuffle scan plus one cross-warp level in
// shared memory, and every segment then re-runs its rows from the exact entering value.  The
// next right-hand side is prefetched into shared memory with cp.async while the current one
// is solved.  One HBM read and one HBM write per point; no per-point factor traffic.
//
// Fused right-hand-side operator (plans for the constant-k, homogeneous-Dirichlet class).  The
// compact RHS of 2D_Program/main_functions/rhs.c:4-97 and 3D_Program/main_functions/rhs.c:13-166
// is a polynomial in the 1D second-difference and Pade operators of each direction.  In the
// DST basis of the transformed direction(s) those operators are diagonal (second difference ->
// lambda - 2, Pade [1 10 1] -> 10 + lambda), so after the forward DST the RHS of line q is
//     order 6:  F = h^2 [ alpha g + beta D2 g + omega/12 + D2 omega/360 ],  omega = T^-1 (12 D2 g)
// where g is the transformed source along the line, D2 the second difference along the line
// (zero boundary values), T = tridiag(1, 10, 1) = D2 + 12 I the Pade matrix of the line
// direction, and alpha, beta depend on k and on the line's eigenvalues.  Because T = D2 + 12 I,
// omega = 12 g - 144 T^-1 g and D2 omega = 12 D2 g - 144 g + 1728 T^-1 g, so
//     order 6:  F = h^2 [ (alpha + 0.6) g + (beta + 1/30) D2 g - 7.2 T^-1 g ]
//     order 4:  F = h^2 [ alpha g + D2 g / 12 ],    order 2:  F = h^2 g
// It is applied in registers before the Helmholtz solve, so the RHS assembly costs no extra
// HBM traffic.
#include "hh_line.cuh"
#include "hh_line_sym.cuh"

#include <algorithm>

namespace hh {

struct LineCoef {
    const double2 *c[4]; // four per-row complex tables (rows each)
};

// One thread per line: runs the Thomas recurrence over the whole line (the reference's LU(),
// 2D LU.c:25-40 / 3D LU.c:51-72) and keeps 1/P of the row before each kSeg-row segment.
// CONST_ROWS: the stencil rows are the same along the line, so they are formed once (the same
// values the per-row evaluation gives) and the recurrence runs without memory traffic.
template <bool CONST_ROWS>
__global__ void k_factor(int lines, int rows, int prow, const double *__restrict__ mu,
                         const double2 *__restrict__ subt, const double2 *__restrict__ diagt,
                         const double2 *__restrict__ supt, double2 *__restrict__ Pv) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= lines) return;
    const double m0 = mu[q], m1 = mu[lines + q], m2 = mu[2 * lines + q];
    double2 ui = first_pivot(shifted(diagt, prow, 0, m0, m1, m2));
    double2 up_prev = shifted(supt, prow, 0, m0, m1, m2);
    const double2 sub_c = shifted(subt, prow, 0, m0, m1, m2), dia_c = shifted(diagt, prow, 0, m0, m1, m2);
    Pv[q] = make_double2(0.0, 0.0);
    for (int r = 1; r < rows; r++) {
        if (r % kSeg == 0) Pv[(long)(r / kSeg) * lines + q] = ui;
        double2 L;
        if constexpr (CONST_ROWS) {
            ui = factor_step(sub_c, dia_c, up_prev, ui, L);
        } else {
            ui = factor_step(shifted(subt, prow, r, m0, m1, m2), shifted(diagt, prow, r, m0, m1, m2), up_prev, ui,
                             L);
            up_prev = shifted(supt, prow, r, m0, m1, m2);
        }
    }
}

int launch_factor(Plan *p, const double2 *subt, const double2 *diagt, const double2 *supt) {
    const int nt = 64;
    if (p->const_rows)
        k_factor<true><<<(p->lines + nt - 1) / nt, nt, 0, p->ctx->stream>>>(p->lines, p->rows, p->prow, p->mu, subt,
                                                                             diagt, supt, p->Pv);
    else
        k_factor<false><<<(p->lines + nt - 1) / nt, nt, 0, p->ctx->stream>>>(p->lines, p->rows, p->prow, p->mu, subt,
                                                                              diagt, supt, p->Pv);
    HH_CUDA(cudaGetLastError());
    p->ctx->launches++;
    return HH_OK;
}

// ------------------------------------------------------------------- solve --------
// Thread (c, s): line c of the CTA (fastest), segment s.  A warp holds all CW lines and
// SPW = 32/CW consecutive segments of each, so a line's segments are spread over the warps.
struct Lane {
    int c, s, sl, w, lane, CW, SPW;
};

template <int NW> struct ScanSmem {
    double2 A[2][NW][32], B[2][NW][32]; // cross-warp totals / neighbour values (double buffered)
    double2 E[NW][32];                  // value entering each warp's first segment, per line
                                        // (rewritten only after the next scan's barrier)
    double  pl[9], pu[9];               // Pade factors of rows 0..8 (constant from row 9 on)
};

// shuffles within groups of NW lanes (the warps of one line in cross_warp_scan)
template <int NW> __device__ __forceinline__ double2 shfl_up_w(double2 v, int off) {
    return make_double2(__shfl_up_sync(0xffffffffu, v.x, off, NW), __shfl_up_sync(0xffffffffu, v.y, off, NW));
}
template <int NW> __device__ __forceinline__ double2 shfl_down_w(double2 v, int off) {
    return make_double2(__shfl_down_sync(0xffffffffu, v.x, off, NW), __shfl_down_sync(0xffffffffu, v.y, off, NW));
}

// Exclusive scan of the per-warp maps (sm.A, sm.B)[par][w][c] over w, for every line c of the CTA:
// sm.E[w][c] = value entering warp w.  Thread t < NW*CW handles (w = t % NW, c = t / NW); the NW
// warps of a line sit in consecutive lanes, so the scan is a width-NW shuffle scan.  FORWARD
// composes warps left to right, else right to left.
template <int NW, bool FORWARD>
__device__ __forceinline__ void cross_warp_scan(ScanSmem<NW> &sm, int par, int CW) {
    const int t = threadIdx.x;
    if ((t >> 5) < (NW * CW + 31) / 32) { // whole warps take part in the shuffles
        const bool in = t < NW * CW;
        const int  w = t % NW, c = t / NW;
        const int  pos = FORWARD ? w : NW - 1 - w;
        double2 A = make_double2(1.0, 0.0), B = make_double2(0.0, 0.0);
        if (in) {
            A = sm.A[par][w][c];
            B = sm.B[par][w][c];
        }
        for (int off = 1; off < NW; off <<= 1) {
            const double2 Ao = FORWARD ? shfl_up_w<NW>(A, off) : shfl_down_w<NW>(A, off);
            const double2 Bo = FORWARD ? shfl_up_w<NW>(B, off) : shfl_down_w<NW>(B, off);
            if (pos >= off) {
                B = cfma(B, A, Bo);
                A = cmul(A, Ao);
            }
        }
        double2 Ex = FORWARD ? shfl_up_w<NW>(B, 1) : shfl_down_w<NW>(B, 1);
        if (pos == 0) Ex = make_double2(0.0, 0.0);
        if (in) sm.E[w][c] = Ex;
    }
}

// Value entering segment s for the left-to-right composition of maps (A, B): y = A y_in + B.
template <int NW>
__device__ __forceinline__ double2 scan_forward(double2 A, double2 B, const Lane &L, ScanSmem<NW> &sm, int par) {
    for (int off = L.CW; off < 32; off <<= 1) {
        const double2 Al = shfl_up2(A, off), Bl = shfl_up2(B, off);
        if (L.lane >= off) {
            B = cfma(B, A, Bl);
            A = cmul(A, Al);
        }
    }
    double2 Ae = shfl_up2(A, L.CW), Be = shfl_up2(B, L.CW);
    if (L.sl == 0) { Ae = make_double2(1.0, 0.0); Be = make_double2(0.0, 0.0); }
    if (L.sl == L.SPW - 1) { sm.A[par][L.w][L.c] = A; sm.B[par][L.w][L.c] = B; }
    __syncthreads();
    cross_warp_scan<NW, true>(sm, par, L.CW);
    __syncthreads();
    return cfma(Be, Ae, sm.E[L.w][L.c]);
}

// Value entering segment s from the right (maps composed right-to-left).
template <int NW>
__device__ __forceinline__ double2 scan_backward(double2 A, double2 B, const Lane &L, ScanSmem<NW> &sm, int par) {
    for (int off = L.CW; off < 32; off <<= 1) {
        const double2 Ar = shfl_down2(A, off), Br = shfl_down2(B, off);
        if (L.lane + off < 32) {
            B = cfma(B, A, Br);
            A = cmul(A, Ar);
        }
    }
    double2 Ae = shfl_down2(A, L.CW), Be = shfl_down2(B, L.CW);
    if (L.sl == L.SPW - 1) { Ae = make_double2(1.0, 0.0); Be = make_double2(0.0, 0.0); }
    if (L.sl == 0) { sm.A[par][L.w][L.c] = A; sm.B[par][L.w][L.c] = B; }
    __syncthreads();
    cross_warp_scan<NW, false>(sm, par, L.CW);
    __syncthreads();
    return cfma(Be, Ae, sm.E[L.w][L.c]);
}

// Last value of segment s-1 and first value of segment s+1 (zero outside the line).
template <int NW>
__device__ __forceinline__ void neighbours(double2 lo, double2 hi, const Lane &L, ScanSmem<NW> &sm, int par,
                                           double2 &prev_hi, double2 &next_lo) {
    prev_hi = shfl_up2(hi, L.CW);
    next_lo = shfl_down2(lo, L.CW);
    if (L.sl == L.SPW - 1) sm.B[par][L.w][L.c] = hi;
    if (L.sl == 0) sm.A[par][L.w][L.c] = lo;
    __syncthreads();
    if (L.sl == 0) prev_hi = (L.w > 0) ? sm.B[par][L.w - 1][L.c] : make_double2(0.0, 0.0);
    if (L.sl == L.SPW - 1) next_lo = (L.w < NW - 1) ? sm.A[par][L.w + 1][L.c] : make_double2(0.0, 0.0);
}

struct SrcParams {
    int     dim;      // 2 or 3
    double  h2;       // h^2
    double2 k2h2_20;  // k^2 h^2 / 20
    const double *pl; // Pade [1 10 1] multipliers L_r = 1/U_{r-1} (L_0 = 0); zero past the line
    const double *pu; // Pade reciprocal pivots 1/U_r; zero past the line
    double linf, uinf;// both converge to 1/(5 + sqrt 24) exactly in double from row 9 on
};

// Pade factors of row r: rows 0..8 from shared memory, the fixed point up to the line end, zero
// past it (neutral padded rows).
template <int NW>
__device__ __forceinline__ double pade_l(const ScanSmem<NW> &sm, const SrcParams &sp, int r, int rows) {
    return r < 9 ? sm.pl[r] : (r < rows ? sp.linf : 0.0);
}
template <int NW>
__device__ __forceinline__ double pade_u(const ScanSmem<NW> &sm, const SrcParams &sp, int r, int rows) {
    return r < 9 ? sm.pu[r] : (r < rows ? sp.uinf : 0.0);
}

// SRC = 0: the input already is the transformed RHS.  SRC = 2/4/6: the input is the transformed
// source g and the compact operator of that order is applied first (see the file header).
// The stencil rows do not vary along the line (constant k); k_line_solve_rows below takes those that do.
// Rows past the end of a line are neutral: zero data, zero reciprocal pivots, zero Pade factors,
// so the sweeps run without per-row conditions.
template <int SRC, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_line_solve(const double2 *__restrict__ in, double2 *__restrict__ out, int lines, int rows, int prow,
                 long row_stride, long field, int batch, int rb, int CW, const double2 *__restrict__ Pv,
                 const double2 *__restrict__ subt, const double2 *__restrict__ diagt, const double2 *__restrict__ supt,
                 const double *__restrict__ mu, SrcParams sp) {
    constexpr int NW = NT / 32;
    __shared__ ScanSmem<NW> sm;
    extern __shared__ double2 pre[]; // [kSeg][NT] prefetch of the next right-hand side,
                                     // then (SRC == 6) [kSeg][NT] Pade scratch
    double2 *wsm = pre + kSeg * NT + threadIdx.x;
    Lane L;
    L.lane = threadIdx.x & 31;
    L.w = threadIdx.x >> 5;
    L.CW = CW;
    L.SPW = 32 / CW;
    L.c = threadIdx.x % CW;
    L.s = threadIdx.x / CW;
    L.sl = L.lane / CW;
    const int  q = blockIdx.x * CW + L.c;
    const bool live = q < lines;
    const int  qq = live ? q : 0;
    const int  r0 = L.s * kSeg;
    const double m0 = live ? mu[q] : 0.0, m1 = live ? mu[lines + q] : 0.0, m2 = live ? mu[2 * lines + q] : 0.0;
    const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);

    // ---- factors of this thread's rows, kept in registers for the whole chunk
    const double2 sub_c = shifted(subt, prow, 0, m0, m1, m2), sup_c = shifted(supt, prow, 0, m0, m1, m2);
    const double2 ui_in = (live && r0 > 0 && r0 < rows) ? Pv[(long)L.s * lines + q] : zero; // 1/P of row r0-1
    double2 ui[kSeg];
    double2 Af = one, Ab = one;
    {
        double2 uprev = ui_in;
        const double2 dia_c = shifted(diagt, prow, 0, m0, m1, m2);
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            const int r = r0 + u;
            double2   Lr = zero;
            ui[u] = zero;
            if (live && r < rows) {
                if (r == 0) ui[u] = first_pivot(dia_c);
                else ui[u] = factor_step(sub_c, dia_c, sup_c, uprev, Lr);
            } else if (live && r > 0 && u > 0) {
                Lr = cmul(sub_c, uprev); // first padded row: L is still formed from the last real pivot
            }
            uprev = ui[u];
            Af = cmul(Af, make_double2(-Lr.x, -Lr.y));
            const double2 tau = cmul(sup_c, ui[u]);
            Ab = cmul(Ab, make_double2(-tau.x, -tau.y));
        }
    }

    // per-line coefficients of the compact right-hand-side operator
    double2 alpha = one;
    double  beta = 0.0;
    if constexpr (SRC == 4) {
        alpha = make_double2(sp.dim == 2 ? (10.0 + m1) / 12.0 : (8.0 + m1 + m2) / 12.0, 0.0);
        beta = 1.0 / 12.0;
    } else if constexpr (SRC == 6) {
        if (sp.dim == 2) {
            const double muq = 12.0 * (m1 - 2.0) / (10.0 + m1);
            alpha = make_double2(1.6 + muq / 12.0 + (m1 - 2.0) * muq / 360.0 - sp.k2h2_20.x, -sp.k2h2_20.y);
            beta = muq / 90.0 + 1.0 / 30.0;
        } else {
            const double mx = 12.0 * (m1 - 2.0) / (10.0 + m1), my = 12.0 * (m2 - 2.0) / (10.0 + m2);
            alpha = make_double2(1.6 + (mx + my) / 12.0 + ((m1 - 2.0) * mx + (m2 - 2.0) * my) / 360.0 +
                                     (m2 - 2.0) * mx / 90.0 - sp.k2h2_20.x,
                                 -sp.k2h2_20.y);
            beta = (mx + my) / 90.0 + 1.0 / 30.0;
        }
    }
    double pa = 1.0, pb = 1.0; // Pade segment products
    if constexpr (SRC == 6) {
        if (threadIdx.x < 9) {
            sm.pl[threadIdx.x] = sp.pl[threadIdx.x];
            sm.pu[threadIdx.x] = sp.pu[threadIdx.x];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            pa *= -pade_l(sm, sp, r0 + u, rows);
            pb *= -pade_u(sm, sp, r0 + u, rows);
        }
    }

    const int  b_begin = blockIdx.y * rb;
    const int  b_end = min(batch, b_begin + rb);
    const long off0 = (long)r0 * row_stride + qq;
    auto prefetch = [&](int b) {
        const double2 *src = in + (long)b * field + off0;
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            const bool ok = live && r0 + u < rows;
            cp_async16(&pre[u * NT + threadIdx.x], ok ? src + (long)u * row_stride : in, ok ? 16 : 0);
        }
        cp_async_commit();
    };
    pdl_wait();
    pdl_next();
    prefetch(b_begin);
    int par = 0;
    for (int b = b_begin; b < b_end; b++) {
        double2 v[kSeg];
        cp_async_wait_all();
#pragma unroll
        for (int u = 0; u < kSeg; u++) v[u] = pre[u * NT + threadIdx.x];
        if (b + 1 < b_end) prefetch(b + 1);

        // ---- compact right-hand-side operator in the transformed basis
        if constexpr (SRC == 2) {
#pragma unroll
            for (int u = 0; u < kSeg; u++) v[u] = cscale(v[u], sp.h2);
        } else if constexpr (SRC == 4 || SRC == 6) {
            double2 before, after;
            neighbours(v[0], v[kSeg - 1], L, sm, par, before, after);
            par ^= 1;
            double2 zh = zero;
            if constexpr (SRC == 6) {
                // forward Pade sweep of g (local part): z_r = g_r - l_r z_{r-1}
#pragma unroll
                for (int u = 0; u < kSeg; u++) {
                    const double l = pade_l(sm, sp, r0 + u, rows);
                    zh = make_double2(v[u].x - l * zh.x, v[u].y - l * zh.y);
                    wsm[u * NT] = zh;
                }
            }
            double2 gprev = before;
#pragma unroll
            for (int u = 0; u < kSeg; u++) {
                const double2 g = v[u];
                const double2 hi = (u == kSeg - 1) ? after : v[u + 1];
                const double2 d2 = make_double2(gprev.x - 2.0 * g.x + hi.x, gprev.y - 2.0 * g.y + hi.y);
                gprev = g;
                v[u] = make_double2(fma(alpha.x, g.x, fma(-alpha.y, g.y, beta * d2.x)),
                                    fma(alpha.x, g.y, fma(alpha.y, g.x, beta * d2.y)));
            }
            if constexpr (SRC == 6) {
                // complete the forward sweep from the exact entering value, then the backward one:
                // w_r = (z_r - w_{r+1}) / U_r;  F += -7.2 w
                const double2 zin = scan_forward(make_double2(pa, 0.0), zh, L, sm, par);
                par ^= 1;
                double2 corr = zin;
#pragma unroll
                for (int u = 0; u < kSeg; u++) {
                    const double l = pade_l(sm, sp, r0 + u, rows);
                    corr = make_double2(-l * corr.x, -l * corr.y);
                    const double2 z = wsm[u * NT];
                    wsm[u * NT] = make_double2(z.x + corr.x, z.y + corr.y);
                }
                double2 wh = zero;
#pragma unroll
                for (int u = kSeg - 1; u >= 0; u--) {
                    const double  iu = pade_u(sm, sp, r0 + u, rows);
                    const double2 z = wsm[u * NT];
                    wh = make_double2((z.x - wh.x) * iu, (z.y - wh.y) * iu);
                }
                const double2 win = scan_backward(make_double2(pb, 0.0), wh, L, sm, par);
                par ^= 1;
                double2 wv = win;
#pragma unroll
                for (int u = kSeg - 1; u >= 0; u--) {
                    const double  iu = pade_u(sm, sp, r0 + u, rows);
                    const double2 z = wsm[u * NT];
                    wv = make_double2((z.x - wv.x) * iu, (z.y - wv.y) * iu);
                    v[u] = make_double2(fma(-7.2, wv.x, v[u].x), fma(-7.2, wv.y, v[u].y));
                }
            }
        }
        if constexpr (SRC == 4 || SRC == 6) {
#pragma unroll
            for (int u = 0; u < kSeg; u++) v[u] = cscale(v[u], sp.h2);
        }

        // ---- forward substitution y_r = f_r - L_r y_{r-1},  L_r = sub_r / P_{r-1}
        double2 yh = zero;
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            yh = cfms(v[u], cmul(sub_c, u == 0 ? ui_in : ui[u - 1]), yh);
        }
        double2 y = scan_forward(Af, yh, L, sm, par);
        par ^= 1;
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            y = cfms(v[u], cmul(sub_c, u == 0 ? ui_in : ui[u - 1]), y);
            v[u] = y;
        }

        // ---- back substitution x_r = (y_r - super_r x_{r+1}) / P_r
        double2 xh = zero;
#pragma unroll
        for (int u = kSeg - 1; u >= 0; u--) {
            xh = cmul(cfms(v[u], sup_c, xh), ui[u]);
        }
        double2 x = scan_backward(Ab, xh, L, sm, par);
        par ^= 1;
#pragma unroll
        for (int u = kSeg - 1; u >= 0; u--) {
            x = cmul(cfms(v[u], sup_c, x), ui[u]);
            v[u] = x;
        }

        double2 *dst = out + (long)b * field + off0;
#pragma unroll
        for (int u = 0; u < kSeg; u++)
            if (live && r0 + u < rows) dst[(long)u * row_stride] = v[u];
    }
}

// Per-row coefficients (variable k), assembled right-hand sides.  The same segments and scans, with the
// thread's multipliers kept: forming them from the four per-row tables at each use (two sweeps each
// way) read 4 complex values a row and sweep through L1 and bounded the solve.  MT = double: every table is
// real (real k), so the multipliers are, and the products lose their zero halves.
//   y_r = f_r - L_r y_{r-1},  x_r = (1/P_r) y_r - tau_r x_{r+1},  tau_r = super_r / P_r
// (line solve of 3D 125^3, real k: 60 -> 40 us; whole solves with complex k: 2D 511^2 32.8 -> 20.4 us, 2047^2 353
// -> 296.)
template <typename MT> __device__ __forceinline__ MT row_coef(const double2 *__restrict__ tab, int rows, int r, double m0,
                                                              double m1, double m2) {
    if constexpr (is_real_v<MT>) {
        const double *t = reinterpret_cast<const double *>(tab);
        return ((__ldg(t + 2 * r) * m0 + __ldg(t + 2 * (rows + r)) * m1) + __ldg(t + 2 * (2 * rows + r)) * m2) +
               __ldg(t + 2 * (3 * rows + r));
    } else {
        return shifted(tab, rows, r, m0, m1, m2);
    }
}

// SMT: the L_r and tau_r of a thread's rows but the first lie in shared memory, one column per thread, as complex
// ones of 512 threads do not fit their 128 registers.
template <int NT, int MINB, typename MT, bool SMT>
__global__ void __launch_bounds__(NT, MINB)
    k_line_solve_rows(const double2 *__restrict__ in, double2 *__restrict__ out, int lines, int rows, int prow,
                      long row_stride, long field, int batch, int rb, int CW, const double2 *__restrict__ Pv,
                      const double2 *__restrict__ subt, const double2 *__restrict__ diagt,
                      const double2 *__restrict__ supt, const double *__restrict__ mu) {
    constexpr int NW = NT / 32;
    __shared__ ScanSmem<NW> sm;
    extern __shared__ double2 pre[]; // [kSeg][NT] prefetch of the next right-hand side, then (SMT) [kSeg - 1][NT] of
                                     // the L_r and [kSeg - 1][NT] of the tau_r past the first
    [[maybe_unused]] MT *Ls = reinterpret_cast<MT *>(pre + kSeg * NT) + threadIdx.x, *ts = Ls + (kSeg - 1) * NT;
    Lane L;
    L.lane = threadIdx.x & 31;
    L.w = threadIdx.x >> 5;
    L.CW = CW;
    L.SPW = 32 / CW;
    L.c = threadIdx.x % CW;
    L.s = threadIdx.x / CW;
    L.sl = L.lane / CW;
    const int  q = blockIdx.x * CW + L.c;
    const bool live = q < lines;
    const int  qq = live ? q : 0;
    const int  r0 = L.s * kSeg;
    const double m0 = live ? mu[q] : 0.0, m1 = live ? mu[lines + q] : 0.0, m2 = live ? mu[2 * lines + q] : 0.0;
    const double2 zero = make_double2(0.0, 0.0);

    // ---- factors of this thread's rows, kept for the whole chunk.  Rows past the end of a line are neutral
    // (zero data, zero reciprocal pivots), so the sweeps run without per-row conditions.
    constexpr int NR = SMT ? 1 : kSeg; // of L_r and tau_r in registers
    MT Lr[NR], ui[kSeg], tau[NR];
    auto Lm = [&](int u) -> MT {
        if constexpr (SMT) return u == 0 ? Lr[0] : lds_keep(Ls + (u - 1) * NT);
        else return Lr[u];
    };
    auto tm = [&](int u) -> MT {
        if constexpr (SMT) return u == 0 ? tau[0] : lds_keep(ts + (u - 1) * NT);
        else return tau[u];
    };
    MT Af = coef_of<MT>(make_double2(1.0, 0.0)), Ab = Af;
    {
        MT uprev = (live && r0 > 0 && r0 < rows) ? coef_of<MT>(Pv[(long)L.s * lines + q]) : MT{}; // 1/P of row r0-1
        MT sp = r0 > 0 && r0 <= prow ? row_coef<MT>(supt, prow, r0 - 1, m0, m1, m2) : MT{};
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            const int r = r0 + u;
            MT        l{}, tu{};
            ui[u] = MT{};
            if (live && r < rows) {
                const MT dia = row_coef<MT>(diagt, prow, r, m0, m1, m2);
                if (r == 0) ui[u] = first_pivot(dia);
                else ui[u] = factor_step(row_coef<MT>(subt, prow, r, m0, m1, m2), dia, sp, uprev, l);
                sp = row_coef<MT>(supt, prow, r, m0, m1, m2);
                tu = cmul(sp, ui[u]);
            }
            uprev = ui[u];
            Af = cmul(Af, mneg(l));
            Ab = cmul(Ab, mneg(tu));
            if (u < NR) {
                Lr[u < NR ? u : 0] = l;
                tau[u < NR ? u : 0] = tu;
            } else {
                Ls[(u - 1) * NT] = l;
                ts[(u - 1) * NT] = tu;
            }
        }
    }
    const double2 Afc = coef_full(Af), Abc = coef_full(Ab); // (the scans compose complex maps)

    const int  b_begin = blockIdx.y * rb;
    const int  b_end = min(batch, b_begin + rb);
    const long off0 = (long)r0 * row_stride + qq;
    auto prefetch = [&](int b) {
        const double2 *src = in + (long)b * field + off0;
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            const bool ok = live && r0 + u < rows;
            cp_async16(&pre[u * NT + threadIdx.x], ok ? src + (long)u * row_stride : in, ok ? 16 : 0);
        }
        cp_async_commit();
    };
    pdl_wait();
    pdl_next();
    prefetch(b_begin);
    int par = 0;
    for (int b = b_begin; b < b_end; b++) {
        double2 v[kSeg];
        cp_async_wait_all();
#pragma unroll
        for (int u = 0; u < kSeg; u++) v[u] = pre[u * NT + threadIdx.x];
        if (b + 1 < b_end) prefetch(b + 1);
        double2 yh = zero;
#pragma unroll
        for (int u = 0; u < kSeg; u++) yh = zfms(v[u], Lm(u), yh);
        double2 y = scan_forward(Afc, yh, L, sm, par);
        par ^= 1;
#pragma unroll
        for (int u = 0; u < kSeg; u++) {
            y = zfms(v[u], Lm(u), y);
            v[u] = cmul(ui[u], y);
        }
        double2 xh = zero;
#pragma unroll
        for (int u = kSeg - 1; u >= 0; u--) xh = zfms(v[u], tm(u), xh);
        double2 x = scan_backward(Abc, xh, L, sm, par);
        par ^= 1;
#pragma unroll
        for (int u = kSeg - 1; u >= 0; u--) {
            x = zfms(v[u], tm(u), x);
            v[u] = x;
        }
        double2 *dst = out + (long)b * field + off0;
#pragma unroll
        for (int u = 0; u < kSeg; u++)
            if (live && r0 + u < rows) dst[(long)u * row_stride] = v[u];
    }
}

// Thread-count variants of the interleaved solve: NT threads per CTA, MINB CTAs per SM.
struct SolveVariant {
    int nt, minb;
};
static const SolveVariant kVariants[] = {{512, 1}, {256, 2}};
constexpr int kNumVariants = 2; // plus variants 2..6: k_line_solve_sym where the plan allows it

// segments per line: a power of two >= NT/32 (so at most 32 lines share a warp)
static int solve_geometry(int rows, int nt, int *CW, int *P) {
    int p = nt / 32;
    while (p * kSeg < rows) p <<= 1;
    if (p > nt) {
        set_error("line length %d exceeds %d", rows, nt * kSeg);
        return HH_ERR_UNSUPPORTED;
    }
    *P = p;
    *CW = nt / p;
    return HH_OK;
}

int padded_rows(int rows) {
    int best = rows;
    for (int v = 0; v < kNumVariants; v++) {
        int CW, P;
        if (solve_geometry(rows, kVariants[v].nt, &CW, &P) == HH_OK && P * kSeg > best) best = P * kSeg;
    }
    return best;
}

int solve_variant_count() { return kNumVariants + 5; }

// the chunk of right-hand sides per CTA: enough CTAs to fill the SMs twice, factors reused within a chunk
static int rows_chunk(long groups, int batch, int minb) {
    int rb = 1;
    while (rb < batch && groups * ((batch + 2 * rb - 1) / (2 * rb)) >= 2L * minb * 148) rb *= 2;
    return rb;
}

template <int NT, int MINB, typename MT, bool SMT = false>
static int launch_solve_rows(Plan *p, const double2 *in, double2 *out, int batch) {
    int CW, P;
    HH_TRY(solve_geometry(p->rows, NT, &CW, &P));
    const int shm = (int)(sizeof(double2) * kSeg * NT + (SMT ? sizeof(MT) * 2 * (kSeg - 1) * NT : 0));
    HH_CUDA(cudaFuncSetAttribute(k_line_solve_rows<NT, MINB, MT, SMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    const long groups = (p->lines + CW - 1) / CW;
    const int  rb = rows_chunk(groups, batch, MINB);
    dim3 grid((unsigned)groups, (unsigned)((batch + rb - 1) / rb));
    return launch_kernel(p->ctx, k_line_solve_rows<NT, MINB, MT, SMT>, grid, NT, (size_t)shm, in, out, p->lines, p->rows, p->prow,
                         p->row_stride, p->field, batch, rb, CW, p->Pv, p->subt, p->diagt, p->rowc, p->mu);
}

template <int SRC, int NT, int MINB>
static int launch_solve_t(Plan *p, const double2 *in, double2 *out, int batch) {
    int CW, P;
    HH_TRY(solve_geometry(p->rows, NT, &CW, &P));
    SrcParams sp;
    sp.dim = p->dim;
    sp.h2 = p->h * p->h;
    sp.k2h2_20 = make_double2(p->k2.x * sp.h2 / 20.0, p->k2.y * sp.h2 / 20.0);
    sp.pl = p->pade_l;
    sp.pu = p->pade_u;
    sp.linf = p->pade_linf;
    sp.uinf = p->pade_uinf;
    const int shm = (int)(sizeof(double2) * kSeg * NT) * (SRC == 6 ? 2 : 1);
    HH_CUDA(cudaFuncSetAttribute(k_line_solve<SRC, NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    const long groups = (p->lines + CW - 1) / CW;
    const int  rb = rows_chunk(groups, batch, MINB);
    const int chunks = (batch + rb - 1) / rb;
    dim3 grid((unsigned)groups, (unsigned)chunks);
    return launch_kernel(p->ctx, k_line_solve<SRC, NT, MINB>, grid, NT, (size_t)shm, in, out, p->lines, p->rows, p->prow,
                                                                       p->row_stride, p->field, batch, rb, CW, p->Pv,
                                                                       p->subt, p->diagt, p->rowc, p->mu, sp);
}

template <int NT, int MINB>
static int launch_solve_v(Plan *p, const double2 *in, double2 *out, int batch, int src) {
    switch (src) {
    case 0: return launch_solve_t<0, NT, MINB>(p, in, out, batch);
    case 2: return launch_solve_t<2, NT, MINB>(p, in, out, batch);
    case 4: return launch_solve_t<4, NT, MINB>(p, in, out, batch);
    case 6: return launch_solve_t<6, NT, MINB>(p, in, out, batch);
    default: set_error("source operator order %d", src); return HH_ERR_INVALID;
    }
}

static int launch_solve_const(Plan *p, const double2 *in, double2 *out, int batch, int src) {
    if (p->variant == 1) return launch_solve_v<256, 2>(p, in, out, batch, src);
    return launch_solve_v<512, 1>(p, in, out, batch, src);
}

// Per-row coefficients: variant 1 takes 256 threads, and variant 0 whichever of the two forms is the faster:
//  * 256 threads have less to set up and half the lines in a CTA (half as wide row pieces): real ones stand two on an
//    SM, complex ones keep their multipliers in 201 registers;
//  * 512 threads (complex ones with multipliers in shared memory) win where their CTAs fill half the SMs and the
//    row pieces of 256 would be narrow (real ones of up to 256 rows, about even, take them where they fill all SMs).
// Whole solves, 256 -> 512 threads, one right-hand side but where noted: real, 1023 lines of 127 rows 18.2 -> 21.0 us,
// of 511 32.4 -> 32.0, of 1023 77 -> 54.6, 255 of 2047 74 -> 44; complex, 1023 of 127 18.2 -> 21.1, 511 of 255
// 15.5 -> 17.5 (two right-hand sides 21.4 -> 20.2), 511 of 511 23.1 -> 20.3, 2047 of 2047 510 -> 294, 63 of 1023 16.4
// -> 21.2.  Lines past 2048 rows only fit 512; complex ones of few lines then keep their multipliers in (spilled)
// registers: 31 lines of 4095 64.9 us with shared memory, 50.8 so, 127 lines 74.1 and 76.7.
static bool rows_wide(const Plan *p, int batch) {
    int CW, P;
    if (p->rows > 256 * kSeg || solve_geometry(p->rows, 512, &CW, &P) != HH_OK) return true; // (past 4096 rows: refused)
    if (p->variant == 1) return false;
    const long groups = (p->lines + CW - 1) / CW, ctas = groups * batch;
    if (p->real_rows) return p->rows > 512 ? ctas >= 64 : p->rows > 256 ? ctas > 64 : groups >= 148;
    return p->rows > 128 && p->lines > 64 && ctas >= 64;
}

static int launch_solve_rows_any(Plan *p, const double2 *in, double2 *out, int batch) {
    const bool wide = rows_wide(p, batch);
    if (p->real_rows)
        return wide ? launch_solve_rows<512, 1, double>(p, in, out, batch) : launch_solve_rows<256, 2, double>(p, in, out, batch);
    if (!wide) return launch_solve_rows<256, 1, double2>(p, in, out, batch);
    return p->lines <= 64 && p->rows > 256 * kSeg ? launch_solve_rows<512, 1, double2>(p, in, out, batch)
                                                  : launch_solve_rows<512, 1, double2, true>(p, in, out, batch);
}

// The lines a CTA of the plan's line solve takes, the width of its row pieces in values
int line_group(const Plan *p, int batch, int src_order) {
    if (p->variant >= 2 && sym_solve_supported(p, src_order)) return 256 / sym_segments(p->rows, p->variant >= 5 ? 16 : kSeg);
    int       CW = 1, P;
    const int nt = p->const_rows ? (p->variant == 1 ? 256 : 512) : rows_wide(p, batch) ? 512 : 256;
    return solve_geometry(p->rows, nt, &CW, &P) == HH_OK ? CW : 1;
}

int launch_line_solve_sym(Plan *p, const double2 *in, double2 *out, int batch, int src_order);
bool sym_solve_supported(const Plan *p, int src_order);

int launch_line_solve(Plan *p, const double2 *in, double2 *out, int batch, int src_order) {
    if (p->variant >= 2 && sym_solve_supported(p, src_order)) return launch_line_solve_sym(p, in, out, batch, src_order);
    if (src_order == 6 && !p->pade_l) {
        set_error("order-6 source operator needs a Helmholtz plan");
        return HH_ERR_INVALID;
    }
    if (p->const_rows) return launch_solve_const(p, in, out, batch, src_order);
    if (src_order != 0) {
        set_error("the source operator needs a Helmholtz plan");
        return HH_ERR_INVALID;
    }
    return launch_solve_rows_any(p, in, out, batch);
}

int segment_count(int rows) { return (rows + kSeg - 1) / kSeg; }

// ------------------------------------------------------------- slab <-> lines ------
// The cut of transformed planes into the ranks' lines for a slab/pencil solve, and back: element
// (b, z, q) of a slab [batch][planes][nlines] is element (z, b, q - q0_s) of rank s's part
// [planes][batch][cnt_s] of the buffer, the parts in rank order, for the balanced contiguous
// split of [0, nlines) over `world` ranks (cnt_s = base + (s < extra), q0_s = s base +
// min(s, extra)).  One thread per element, consecutive threads on consecutive q.
__global__ void __launch_bounds__(256) k_lines_pack(const double2 *__restrict__ a, double2 *__restrict__ o,
                                                    int batch, int planes, int nlines, int world, int unpack) {
    const long row = blockIdx.y; // b * planes + z
    const long b = row / planes, z = row % planes;
    const int  base = nlines / world, extra = nlines % world, cut = (base + 1) * extra;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nlines; q += gridDim.x * blockDim.x) {
        const int  s = q < cut ? q / (base + 1) : extra + (q - cut) / base;
        const int  q0 = s * base + min(s, extra), cnt = base + (s < extra ? 1 : 0);
        const long si = row * nlines + q;
        const long di = (long)batch * planes * q0 + (z * batch + b) * cnt + (q - q0);
        if (unpack) o[si] = a[di];
        else o[di] = a[si];
    }
}

int launch_lines_pack(Ctx *c, const double2 *in, double2 *out, long batch, long planes, long nlines, int world,
                      bool unpack) {
    if (batch < 0 || planes < 1 || nlines < 1 || world < 1 || world > nlines || batch * planes > 65535 ||
        nlines > (1L << 30) || planes > (1L << 30)) {
        set_error("lines pack: batch %ld, planes %ld, lines %ld, ranks %d", batch, planes, nlines, world);
        return HH_ERR_INVALID;
    }
    if (batch == 0) return HH_OK;
    const long bx = std::min<long>((nlines + 255) / 256, 64);
    dim3 grid((unsigned)bx, (unsigned)(batch * planes));
    k_lines_pack<<<grid, 256, 0, c->stream>>>(in, out, (int)batch, (int)planes, (int)nlines, world, unpack ? 1 : 0);
    HH_CUDA(cudaGetLastError());
    c->launches++;
    return HH_OK;
}

// Default symmetric variant of a plan: 2, or 5 where the lines are longer than 8-row segments
// reach (more than 256 * 8 rows), so that such plans keep the symmetric kernel untuned.
int sym_default_variant(int rows) { return rows > 256 * kSeg ? 5 : 2; }

bool sym_solve_supported(const Plan *p, int src_order) {
    const int max_rows = 256 * (p->variant >= 5 ? 16 : kSeg);
    return p->sym && p->rows <= max_rows && (src_order != 6 || (p->pf_ok && p->pade_l));
}

int launch_line_solve_sym(Plan *p, const double2 *in, double2 *out, int batch, int src_order) {
    return p->real_coef ? launch_sym_real(p, in, out, batch, src_order, nullptr)
                        : launch_sym_cplx(p, in, out, batch, src_order, nullptr);
}

// The chunks of right-hand sides of a multi-plan launch: the single-plan choice for the whole batch, chunks never
// crossing a plan boundary.  HH_ERR_UNSUPPORTED when the plans do not all take one symmetric kernel.
static int multi_chunks(Plan *const *plans, const int *nrhs, int nplans, int src_order, std::vector<SymChunk> *chunks) {
    Plan *p0 = plans[0];
    int   total = 0;
    for (int i = 0; i < nplans; i++) {
        const Plan *pi = plans[i];
        if (pi->variant < 2 || pi->variant != p0->variant || !sym_solve_supported(pi, src_order)) {
            set_error("multi-plan line solve: plan %d does not take the symmetric kernel variant %d", i, p0->variant);
            return HH_ERR_UNSUPPORTED;
        }
        total += nrhs[i];
    }
    if (total == 0) return HH_OK;
    const int ks = (p0->variant >= 5) ? 16 : kSeg;
    const int P = sym_segments(p0->rows, ks), CW = 256 / P, nr = (p0->variant == 4 && P > 8) ? 2 : 1;
    const long groups = (p0->span() + CW - 1) / CW;
    int dev = 0, sms = 148;
    HH_CUDA(cudaGetDevice(&dev));
    HH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int rb = pick_rb(groups, total, (p0->variant == 2 ? 2 : 1) * sms, nr);
    for (int i = 0, b = 0; i < nplans; b += nrhs[i], i++)
        for (int b0 = b; b0 < b + nrhs[i]; b0 += rb) chunks->push_back(SymChunk{i, b0, std::min(b + nrhs[i], b0 + rb), 0});
    if (chunks->size() > 65535) {
        set_error("multi-plan line solve: %zu chunks", chunks->size());
        return HH_ERR_UNSUPPORTED;
    }
    return HH_OK;
}

static bool multi_in_arguments(int nplans, size_t chunks) { return nplans <= SymMulti::kPlans && chunks <= (size_t)SymMulti::kChunks; }

static size_t multi_table_bytes(int nplans, size_t chunks) { return sizeof(SymPlanRef) * (size_t)nplans + sizeof(SymChunk) * chunks; }

size_t line_solve_multi_table_bytes(Plan *const *plans, const int *nrhs, int nplans, int src_order) {
    long total = 0; // (a chunk holds at least one right-hand side: small batches need no look at the chunks)
    for (int i = 0; i < nplans; i++) total += nrhs[i];
    if (multi_in_arguments(nplans, (size_t)total)) return 0;
    std::vector<SymChunk> chunks;
    if (multi_chunks(plans, nrhs, nplans, src_order, &chunks) != HH_OK || multi_in_arguments(nplans, chunks.size())) return 0;
    return multi_table_bytes(nplans, chunks.size());
}

// One symmetric line-solve launch over the right-hand sides of several plans of one shape: plan i
// solves nrhs[i] consecutive fields of the batch (plans in order).  Every plan must take the
// symmetric kernel with the same variant; table_dev (line_solve_multi_table_bytes, nullptr where that is 0) receives
// the plan references and the chunk table in stream order, where they do not fit the kernel's arguments.  Returns
// HH_ERR_UNSUPPORTED when the plans do not qualify, before launching anything; so too for a device table inside a
// stream capture, which would record the address of the host tables freed on return instead of their contents.
int launch_line_solve_multi(Plan *const *plans, const int *nrhs, int nplans, const double2 *in, double2 *out,
                            int src_order, void *table_dev) {
    Plan *p0 = plans[0];
    int   total = 0;
    for (int i = 0; i < nplans; i++) total += nrhs[i];
    std::vector<SymChunk> chunks;
    HH_TRY(multi_chunks(plans, nrhs, nplans, src_order, &chunks));
    if (total == 0) return HH_OK;
    std::vector<SymPlanRef> refs((size_t)nplans);
    for (int i = 0; i < nplans; i++) {
        const Plan  *pi = plans[i];
        const double h2 = pi->h * pi->h;
        refs[(size_t)i] = SymPlanRef{pi->Pv, pi->subt, pi->diagt, make_double2(pi->k2.x * h2 / 20.0, pi->k2.y * h2 / 20.0)};
    }
    SymMulti m;
    m.nchunks = (int)chunks.size();
    if (multi_in_arguments(nplans, chunks.size())) {
        std::copy(refs.begin(), refs.end(), m.iref);
        std::copy(chunks.begin(), chunks.end(), m.ichunk);
    } else if (!table_dev || capturing(p0->ctx)) {
        set_error("multi-plan line solve: no table for %d plans in %zu chunks", nplans, chunks.size());
        return HH_ERR_UNSUPPORTED;
    } else {
        char *tab = static_cast<char *>(table_dev);
        HH_CUDA(cudaMemcpyAsync(tab, refs.data(), sizeof(SymPlanRef) * refs.size(), cudaMemcpyHostToDevice, p0->ctx->stream));
        HH_CUDA(cudaMemcpyAsync(tab + sizeof(SymPlanRef) * refs.size(), chunks.data(), sizeof(SymChunk) * chunks.size(),
                                cudaMemcpyHostToDevice, p0->ctx->stream));
        p0->ctx->fresh = true; // the kernel's set-up reads the table
        m.refs = reinterpret_cast<const SymPlanRef *>(tab);
        m.chunks = reinterpret_cast<const SymChunk *>(tab + sizeof(SymPlanRef) * refs.size());
    }
    // one kernel for all: the complex one (the same bits on a real plan) unless every plan is real
    bool real = true;
    for (int i = 0; i < nplans; i++) real = real && plans[i]->real_coef;
    return real ? launch_sym_real(p0, in, out, total, src_order, &m) : launch_sym_cplx(p0, in, out, total, src_order, &m);
}

} // namespace hh
