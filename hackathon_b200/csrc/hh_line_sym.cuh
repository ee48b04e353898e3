#ifndef HH_LINE_SYM_CUH
#define HH_LINE_SYM_CUH

#include "hh_line.cuh"
#include "hh_tma.cuh"

#include <algorithm>
#include <type_traits>

namespace hh {

// =====================================================================================
// Symmetric constant-row lines (the Helmholtz plans): k_line_solve_sym
//
// For constant k the line matrix is A = d I + s S with S = tridiag(1, 0, 1), the same s below
// and above the diagonal, and one (d, s) per line.  The kernel specialises the solve above for
// that case:
//  * CW (lines per CTA) is a compile-time constant, so every shuffle offset and loop unrolls;
//  * the segment multipliers of the affine maps depend on the factors only, so their scan
//    coefficients are formed once per chunk of right-hand sides (tables in shared memory) and
//    each right-hand side scans only its B values;
//  * every thread loads the two neighbouring rows of its segment with its own rows, so the
//    second differences of the compact operator need no exchange;
//  * order 6: A and the Pade matrix T = 10 I + S are both polynomials in S, so they commute and
//        A^-1 T^-1 = (s A^-1 - T^-1) / (10 s - d)
//    The order-6 right-hand side  F = h^2 [a6 g + b6 D2 g - 7.2 T^-1 g]  then gives
//        u = A^-1 F = A^-1 G + cT T^-1 g,   G = h^2 [(a6 - 7.2 s/(10s - d)) g + b6 D2 g],
//        cT = 7.2 h^2 / (10 s - d)
//    two independent solves that run side by side and share every scan and barrier.  The plan
//    checks |10 s - d| against |d|, |s| on every line before it selects this path.
// =====================================================================================

template <int NT> __host__ __device__ constexpr int ilog2_t() { return NT <= 1 ? 0 : 1 + ilog2_t<NT / 2>(); }

template <int NW, int CW, int NR, typename MT> struct SymSmem {
    uint64_t tbar[2];                 // completion of the tile copies (TMA-tile input)
    MT      AwF[NW][CW], AwB[NW][CW]; // warp totals of the segment multipliers (main solve)
    double  awF[NW][CW], awB[NW][CW]; // the same for the Pade solve (real multipliers)
    double2 BwF[NR][NW][CW], BwB[NR][NW][CW]; // warp totals of the B values, per right-hand side
    double2 EF[NR][NW][CW], EB[NR][NW][CW];   // value entering each warp (order 6)
    double2 bwF[NR][NW][CW], bwB[NR][NW][CW];
    double2 eF[NR][NW][CW], eB[NR][NW][CW];
    double  pl[11], pu[11];           // Pade factors: rows 0..8, the limit of rows 9 on, zero past the line
};

// Shared-memory reads of the scan tables that the compiler must not hoist out of the loop over
// right-hand sides (hoisting them would hold every stage multiplier in registers).
__device__ __forceinline__ double2 lds_keep(const double2 *p) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                 : "=d"(v.x), "=d"(v.y)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
    return v;
}
__device__ __forceinline__ double lds_keep(const double *p) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
    return v;
}

// Order 6 with 16-row segments and complex coefficients keeps its per-row multipliers
// tau_k = s ui_k in shared memory, one column per thread: in registers they would not fit beside the two
// solves' rows.
template <int SRC, int KS, typename MT> struct SymUIS {
    static constexpr bool value = SRC == 6 && KS >= 16 && !is_real_v<MT>;
};
// ... and its per-line constants (tau_0, 1/s, c1, cT, c2) in shared memory [5][NT], each read in
// the sweep that uses it, at the CTA widths where that measured faster with identical bits (line
// solve, TMA-tile input: 3D 127^3 x 16 0.352 -> 0.317 ms, 255^3 x 4 0.756 -> 0.714 ms, 2D
// 1023^2 x 64 0.690 -> 0.684 ms; slower at 2 and 8 lines per CTA: 2047^2 x 16 0.851 -> 0.878 ms,
// 511^2 x 32 0.100 -> 0.103 ms)
template <int SRC, int KS, int CW, typename MT> struct SymPCS {
    static constexpr bool value = SymUIS<SRC, KS, MT>::value && (CW == 4 || CW >= 16);
};

// Order 6 with 8-row segments scans its Pade sweeps: tables of the stage multipliers, [LOG + 1][NT] each way
// (16-row segments take their entering value from the neighbour and have none).
template <int SRC, int KS> struct SymTT {
    static constexpr int value = SRC == 6 && KS < 16 ? 1 : 0;
};

// Intra-warp inclusive scan of B over the segments of each line in the warp, with the stage
// multipliers tab[j * NT] (the thread's own map product at stage j).  FWD composes left to right.
template <int CW, bool FWD>
__device__ __forceinline__ double2 sym_warp_scan(double2 B, const double2 *tab, int NT_, int sl) {
    constexpr int SPW = 32 / CW;
#pragma unroll
    for (int j = 0; (1 << j) < SPW; j++) {
        const double2 Bo = FWD ? shfl_up2(B, CW << j) : shfl_down2(B, CW << j);
        const double2 m = lds_keep(tab + j * NT_);
        if (FWD ? (sl >= (1 << j)) : (sl + (1 << j) < SPW)) B = zfma(B, m, Bo);
    }
    return B;
}
template <int CW, bool FWD>
__device__ __forceinline__ double2 sym_warp_scan(double2 B, const double *tab, int NT_, int sl) {
    constexpr int SPW = 32 / CW;
#pragma unroll
    for (int j = 0; (1 << j) < SPW; j++) {
        const double2 Bo = FWD ? shfl_up2(B, CW << j) : shfl_down2(B, CW << j);
        const double  m = lds_keep(tab + j * NT_);
        if (FWD ? (sl >= (1 << j)) : (sl + (1 << j) < SPW)) B = zaxpy(B, m, Bo);
    }
    return B;
}

struct SymParams {
    double  h2;        // h^2
    double2 k2h2_20;   // k^2 h^2 / 20
    int     dim;
    double  linf, uinf;
    const double *pl, *pu; // Pade factors (rows >= 9 equal linf, uinf)
    double        cz[16];  // (-linf)^(k+1): how an entering value of the forward Pade sweep reaches row k
};

// TMA-tile input of the symmetric line solve: one right-hand side of the CTA's CW lines arrives
// as a tile [rows][CW] in shared memory, brought by tensor copies over a (double of a
// row, row, right-hand side) map in boxes of br rows, NBUF right-hand sides ahead.  Thread 0 issues the
// copies; the outputs are stored from registers as in the per-thread prefetch form.
template <int SRC, typename MT> struct SymTileBufs {
    static constexpr int value = SRC == 6 && !is_real_v<MT> ? 1 : 2; // complex order 6 spends the space on its pivots
};

struct SymTio {
    const CUtensorMap *in_map;
    double2           *tin;  // NBUF tiles of `tile` elements
    uint64_t          *bar;  // one per tile
    int               *err;
    int                x0, br, nbox, tile;
    unsigned           tile_bytes;
};

// One chunk of right-hand sides for the thread's segment, NR of them side by side (independent
// dependency chains, shared barriers).  TINT = the warp's rows all lie in [9, rows) (constant
// Pade factors).
template <int SRC, int NT, int CW, bool TINT, int NR, int KS, bool TIO, typename MT>
__device__ __forceinline__ void sym_chunk(const double2 *__restrict__ in, double2 *__restrict__ out, int rows,
                                          long row_stride, long field, int b_begin, int b_end, long off0,
                                          bool live, int r0, int sl, int w, int c, const MT (&Lr)[KS],
                                          const MT (&ui)[KS], const MT *uis, MT ui_in, MT s,
                                          MT c1, double c2, MT cT, SymSmem<NT / 32, CW, NR, MT> &sm,
                                          double2 *pre, const MT *tabF, const MT *tabB, const double *ttF,
                                          const double *ttB, const SymParams &sp, const SymTio &tio) {
    constexpr int NW = NT / 32, SPW = 32 / CW, LOG = ilog2_t<SPW>();
    constexpr int HALO = (SRC == 4 || SRC == 6) ? 1 : 0;
    constexpr int SLOTS = KS + 2;
    constexpr int  NBUF = SymTileBufs<SRC, MT>::value;
    static_assert(!TIO || NR == 1, "tile I/O moves one right-hand side at a time");
    // complex order 6: the warps' entering values are composed in sequence (threads [0, CW NR) for the
    // main solve, [128, 128 + CW NR) for the Pade solve)
    constexpr bool SEQ = SRC == 6 && !is_real_v<MT>;
    static_assert(!SEQ || (CW * NR <= 128 && NT >= 256), "cross-warp thread ranges");
    const int     t = threadIdx.x;
    const double2 zero = make_double2(0.0, 0.0);
    // Order 6 with 16-row segments: the Pade sweeps forget their entering value within a segment (its
    // factor shrinks by 0.101 a row, 1.2e-16 over 16 rows, less than the rounding of a row's own value), so a
    // segment takes its entering value from the neighbouring segment alone, without a scan, and the
    // forward sweep is completed as z_k + (-l)^(k+1) z_in, off the recurrence.  Segments past the first
    // start beyond row 9, where the factors are the limit; the first has no entering value.  (Line solve with
    // the scans -> without: 3D 255^3 x 4 506 -> 438 us, 127^3 x 16 207 -> 187 us, 2D 1023^2 x 64 552 -> 545 us,
    // 2047^2 x 16 699 -> 672 us; errors against 64-bit solutions unchanged.)
    constexpr bool WIN = SRC == 6 && KS >= 16;
    // Orders 0-4 keep the forward multipliers L_k and the reciprocal pivots ui_k in registers.
    // Order 6, where the two solves' rows fill the registers, keeps one value per row instead:
    // tau_k = s ui_k (= L_{k+1}), in the ui array or (16-row segments) in shared memory, one
    // column per thread.  The sweeps read their multipliers from it as they are, and the final
    // forward pass re-forms ui_k = (1/s) tau_k off the recurrence.
    constexpr bool UIS = SymUIS<SRC, KS, MT>::value;
    constexpr bool KEEP_L = SRC != 6;
    auto TV = [&](int k) -> MT {
        if constexpr (UIS) return lds_keep(uis + k * NT + t);
        else return ui[k];
    };
    constexpr bool PCS = SymPCS<SRC, KS, CW, MT>::value;
    const MT *pcs = reinterpret_cast<const MT *>(ttB + SymTT<SRC, KS>::value * (ilog2_t<32 / CW>() + 1) * NT);
    auto PC = [&](int j) -> MT { return lds_keep(pcs + j * NT + t); };
    const MT tau_in = PCS ? MT{} : cmul(s, ui_in); // L_0 = s / P of row r0 - 1
    const MT rs = PCS ? MT{} : (KEEP_L ? s : crcp(s));
    // forward multiplier of row r0 + k
    auto LF = [&](int k) -> MT {
        if constexpr (KEEP_L) return Lr[k];
        else if constexpr (PCS) return k == 0 ? PC(0) : TV(k - 1);
        else return k == 0 ? tau_in : TV(k - 1);
    };
    // backward multiplier of row r0 + k, tau_k = s ui_k (= L_{k+1} where that row exists)
    const MT tau_last = KEEP_L ? cmul(s, ui[KS - 1]) : s;
    auto TAU = [&](int k) -> MT {
        if constexpr (KEEP_L) return k + 1 < KS ? Lr[k + 1] : tau_last;
        else return TV(k);
    };
    // Pade factors of row r0 + k: the constants in warps whose rows all lie in [9, rows); elsewhere read
    // at each use (rp is r0, re-formed for every right-hand side: held, 2 KS factors would pin registers)
    int  rp = r0;
    auto PL = [&](int k) -> double {
        if constexpr (TINT) return sp.linf;
        const int r = rp + k;
        return lds_keep(sm.pl + (r < 9 ? r : (r < rows ? 9 : 10)));
    };
    auto PU = [&](int k) -> double {
        if constexpr (TINT) return sp.uinf;
        const int r = rp + k;
        return lds_keep(sm.pu + (r < 9 ? r : (r < rows ? 9 : 10)));
    };

    // the tile copies of right-hand side b into tile buffer u, issued by thread 0
    auto tile_load = [&](int b, int u) {
        double2 *dst = tio.tin + (long)u * tio.tile;
        mbar_expect_tx(tio.bar + u, tio.tile_bytes);
        for (int x = 0; x < tio.nbox; x++)
            tma_load_3d(dst + (long)x * tio.br * CW, tio.in_map, 2 * tio.x0, x * tio.br, b, tio.bar + u);
    };
    auto prefetch = [&](int b) {
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const bool     okb = live && b + r < b_end;
            const double2 *src = in + (long)(okb ? b + r : 0) * field + off0;
#pragma unroll
            for (int k = -HALO; k < KS + HALO; k++) {
                const bool ok = okb && r0 + k >= 0 && r0 + k < rows;
                cp_async16(&pre[(r * SLOTS + k + 1) * NT + t], ok ? src + (long)k * row_stride : in, ok ? 16 : 0);
            }
        }
        cp_async_commit();
    };
    if constexpr (!TIO) prefetch(b_begin); // with tile I/O the first tile was requested at kernel start
    int it = 0;
    for (int b = b_begin; b < b_end; b += NR, it++) {
        if constexpr (SRC == 6 && !TINT) asm volatile("" : "+r"(rp));
        double2 v[NR][KS], g[NR][KS], gm[NR], gp[NR];
        bool    landed = true;
        if constexpr (TIO) {
            const int u = NBUF == 2 ? (it & 1) : 0;
            landed = mbar_wait_parity(tio.bar + u, NBUF == 2 ? (it >> 1) & 1 : it & 1);
            const double2 *tl = tio.tin + (long)u * tio.tile + c;
#pragma unroll
            for (int k = 0; k < KS; k++) v[0][k] = (r0 + k < rows) ? tl[(r0 + k) * CW] : zero;
            // threads whose segment lies wholly past the end of the line (r0 > rows) read no halo:
            // row r0 - 1 is not in the tile
            gm[0] = (HALO && r0 > 0 && r0 <= rows) ? tl[(r0 - 1) * CW] : zero;
            gp[0] = (HALO && r0 + KS < rows) ? tl[(r0 + KS) * CW] : zero;
            fence_async_smem(); // these reads before the copy that refills the tile
        } else {
            cp_async_wait_all();
#pragma unroll
            for (int r = 0; r < NR; r++) {
#pragma unroll
                for (int k = 0; k < KS; k++) v[r][k] = pre[(r * SLOTS + k + 1) * NT + t];
                gm[r] = zero;
                gp[r] = zero;
                if constexpr (HALO) {
                    gm[r] = pre[(r * SLOTS) * NT + t];
                    gp[r] = pre[(r * SLOTS + KS + 1) * NT + t];
                }
            }
            if (b + NR < b_end) prefetch(b + NR);
        }

        // ---- compact right-hand side (order 6: the A^-1 part; g keeps the source for T^-1)
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if constexpr (SRC == 2) {
#pragma unroll
                for (int k = 0; k < KS; k++) v[r][k] = cscale(v[r][k], sp.h2);
            } else if constexpr (SRC == 4 || SRC == 6) {
                double2 prev = gm[r];
                const MT      c1v = PCS ? PC(2) : c1;
                const double  c2v = PCS ? coef_re(PC(4)) : c2;
#pragma unroll
                for (int k = 0; k < KS; k++) {
                    const double2 gk = v[r][k], nx = (k == KS - 1) ? gp[r] : v[r][k + 1];
                    const double2 d2 = make_double2(fma(-2.0, gk.x, prev.x + nx.x), fma(-2.0, gk.y, prev.y + nx.y));
                    prev = gk;
                    if constexpr (SRC == 6) g[r][k] = gk;
                    v[r][k] = zfma(make_double2(c2v * d2.x, c2v * d2.y), c1v, gk); // c2 D2 g + c1 g
                }
            }
        }

        // ---- forward elimination: local sweeps from a zero entering value
        double2 yh[NR], zh[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) { yh[r] = zero; zh[r] = zero; }
#pragma unroll
        for (int k = 0; k < KS; k++) {
            const MT l = LF(k);
#pragma unroll
            for (int r = 0; r < NR; r++) {
                yh[r] = zfms(v[r][k], l, yh[r]);
                if constexpr (SRC == 6) zh[r] = zaxpy(g[r][k], -PL(k), zh[r]);
                if constexpr (WIN) g[r][k] = zh[r];
            }
        }
        double2 Bfe[NR], bfe[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const double2 Bf = sym_warp_scan<CW, true>(yh[r], tabF + t, NT, sl);
            Bfe[r] = shfl_up2(Bf, CW);
            bfe[r] = zero;
            if (sl == SPW - 1) sm.BwF[r][w][c] = Bf;
            if constexpr (WIN) {
                bfe[r] = shfl_up2(zh[r], CW);
                if (sl == SPW - 1) sm.bwF[r][w][c] = zh[r];
            } else if constexpr (SRC == 6) {
                const double2 bf = sym_warp_scan<CW, true>(zh[r], ttF + t, NT, sl);
                bfe[r] = shfl_up2(bf, CW);
                if (sl == SPW - 1) sm.bwF[r][w][c] = bf;
            }
            if (sl == 0) { Bfe[r] = zero; bfe[r] = zero; }
        }
        if constexpr (TIO) {
            if (__syncthreads_or(!landed)) { // a tile copy did not land: report and leave together
                if (t == 0) {
                    atomicExch(tio.err, 1);
                    // copies still in flight get a bounded chance to land before the memory is released
                    for (int j = 0; j < NBUF && b + j < b_end; j++) {
                        const int jt = it + j;
                        mbar_wait_parity(tio.bar + (NBUF == 2 ? (jt & 1) : 0), NBUF == 2 ? (jt >> 1) & 1 : jt & 1);
                    }
                }
                return;
            }
            // every thread has read this tile: it takes the right-hand side NBUF ahead
            if (t == 0 && b + NBUF < b_end) tile_load(b + NBUF, NBUF == 2 ? (it & 1) : 0);
        } else {
            __syncthreads();
        }
        // The value entering each warp's segments of line c: the totals of the warps before it,
        // composed in order.  Orders 0-4: every warp forms its own (the totals stay until the next
        // barrier).  Order 6, whose two solves leave no registers for that: CW threads per solve
        // compose them in sequence into shared memory, behind one more barrier.
        if constexpr (SEQ) {
            if (t < CW * NR) {
                const int r = t / CW, cc = t % CW;
                double2   E = zero;
#pragma unroll
                for (int x = 0; x < NW; x++) {
                    sm.EF[r][x][cc] = E;
                    E = zfma(sm.BwF[r][x][cc], sm.AwF[x][cc], E);
                }
            } else if (!WIN && t >= 128 && t < 128 + CW * NR) {
                const int r = (t - 128) / CW, cc = (t - 128) % CW;
                double2   E = zero;
#pragma unroll
                for (int x = 0; x < NW; x++) {
                    sm.eF[r][x][cc] = E;
                    E = zaxpy(sm.bwF[r][x][cc], sm.awF[x][cc], E);
                }
            }
            __syncthreads();
        }
        {
            double2 EF[NR], eF[NR];
#pragma unroll
            for (int r = 0; r < NR; r++) { EF[r] = zero; eF[r] = zero; }
            if constexpr (!SEQ) {
#pragma unroll
                for (int x = 0; x < NW - 1; x++) {
                    if (x < w) {
                        const MT a = lds_keep(&sm.AwF[x][c]);
#pragma unroll
                        for (int r = 0; r < NR; r++) {
                            EF[r] = zfma(sm.BwF[r][x][c], a, EF[r]);
                            if constexpr (SRC == 6 && !WIN) eF[r] = zaxpy(sm.bwF[r][x][c], lds_keep(&sm.awF[x][c]), eF[r]);
                        }
                    }
                }
            }
            const MT      AeF = lds_keep(tabF + LOG * NT + t);
            double        aeF = 0.0;
            if constexpr (SRC == 6 && !WIN) aeF = lds_keep(ttF + LOG * NT + t);
            double2 y[NR], z[NR];
#pragma unroll
            for (int r = 0; r < NR; r++) {
                y[r] = zfma(Bfe[r], AeF, SEQ ? sm.EF[r][w][c] : EF[r]);
                z[r] = zero;
                if constexpr (WIN) z[r] = sl > 0 ? bfe[r] : (w > 0 ? sm.bwF[r][w > 0 ? w - 1 : 0][c] : zero);
                else if constexpr (SRC == 6) z[r] = zaxpy(bfe[r], aeF, SEQ ? sm.eF[r][w][c] : eF[r]);
            }
            // the rows keep ui_k y_k, so that the back substitution is x_k = ui_k y_k - tau_k x_{k+1}
            MT       tp = PCS ? PC(0) : tau_in;
            const MT rsv = PCS ? PC(1) : rs;
#pragma unroll
            for (int k = 0; k < KS; k++) {
                MT u, l;
                if constexpr (KEEP_L) {
                    u = ui[k];
                    l = Lr[k];
                } else {
                    const MT tk = TV(k);
                    u = cmul(rsv, tk);
                    l = tp;
                    tp = tk;
                }
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    y[r] = zfms(v[r][k], l, y[r]);
                    v[r][k] = cmul(u, y[r]);
                    if constexpr (WIN) {
                        g[r][k] = zaxpy(g[r][k], sp.cz[k], z[r]);
                    } else if constexpr (SRC == 6) {
                        z[r] = zaxpy(g[r][k], -PL(k), z[r]);
                        g[r][k] = z[r];
                    }
                }
            }
        }

        // ---- back substitution x_r = ui_r y_r - tau_r x_{r+1};  Pade: w_r = pu_r (z_r - w_{r+1})
        double2 xh[NR], wh[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) { xh[r] = zero; wh[r] = zero; }
#pragma unroll
        for (int k = KS - 1; k >= 0; k--) {
#pragma unroll
            for (int r = 0; r < NR; r++) {
                xh[r] = zfms(v[r][k], TAU(k), xh[r]);
                if constexpr (SRC == 6) wh[r] = cscale(csub(g[r][k], wh[r]), PU(k));
            }
        }
        double2 Bbe[NR], bbe[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const double2 Bb = sym_warp_scan<CW, false>(xh[r], tabB + t, NT, sl);
            Bbe[r] = shfl_down2(Bb, CW);
            bbe[r] = zero;
            if (sl == 0) sm.BwB[r][w][c] = Bb;
            if constexpr (WIN) {
                bbe[r] = shfl_down2(wh[r], CW);
                if (sl == 0) sm.bwB[r][w][c] = wh[r];
            } else if constexpr (SRC == 6) {
                const double2 bb = sym_warp_scan<CW, false>(wh[r], ttB + t, NT, sl);
                bbe[r] = shfl_down2(bb, CW);
                if (sl == 0) sm.bwB[r][w][c] = bb;
            }
            if (sl == SPW - 1) { Bbe[r] = zero; bbe[r] = zero; }
        }
        __syncthreads();
        // the value entering each warp from the warps after it, composed from the last one down
        // (as in the forward direction)
        if constexpr (SEQ) {
            if (t < CW * NR) {
                const int r = t / CW, cc = t % CW;
                double2   E = zero;
#pragma unroll
                for (int x = NW - 1; x >= 0; x--) {
                    sm.EB[r][x][cc] = E;
                    E = zfma(sm.BwB[r][x][cc], sm.AwB[x][cc], E);
                }
            } else if (!WIN && t >= 128 && t < 128 + CW * NR) {
                const int r = (t - 128) / CW, cc = (t - 128) % CW;
                double2   E = zero;
#pragma unroll
                for (int x = NW - 1; x >= 0; x--) {
                    sm.eB[r][x][cc] = E;
                    E = zaxpy(sm.bwB[r][x][cc], sm.awB[x][cc], E);
                }
            }
            __syncthreads();
        }
        {
            double2 EB[NR], eB[NR];
#pragma unroll
            for (int r = 0; r < NR; r++) { EB[r] = zero; eB[r] = zero; }
            if constexpr (!SEQ) {
#pragma unroll
                for (int xw = NW - 1; xw > 0; xw--) {
                    if (xw > w) {
                        const MT a = lds_keep(&sm.AwB[xw][c]);
#pragma unroll
                        for (int r = 0; r < NR; r++) {
                            EB[r] = zfma(sm.BwB[r][xw][c], a, EB[r]);
                            if constexpr (SRC == 6 && !WIN) eB[r] = zaxpy(sm.bwB[r][xw][c], lds_keep(&sm.awB[xw][c]), eB[r]);
                        }
                    }
                }
            }
            const MT      AeB = lds_keep(tabB + LOG * NT + t);
            double        aeB = 0.0;
            if constexpr (SRC == 6 && !WIN) aeB = lds_keep(ttB + LOG * NT + t);
            double2 x[NR], ww[NR];
            const MT cTv = PCS ? PC(3) : cT;
#pragma unroll
            for (int r = 0; r < NR; r++) {
                x[r] = zfma(Bbe[r], AeB, SEQ ? sm.EB[r][w][c] : EB[r]);
                ww[r] = zero;
                if constexpr (WIN) ww[r] = sl < SPW - 1 ? bbe[r] : (w < NW - 1 ? sm.bwB[r][w < NW - 1 ? w + 1 : w][c] : zero);
                else if constexpr (SRC == 6) ww[r] = zaxpy(bbe[r], aeB, SEQ ? sm.eB[r][w][c] : eB[r]);
            }
#pragma unroll
            for (int k = KS - 1; k >= 0; k--) {
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    x[r] = zfms(v[r][k], TAU(k), x[r]);
                    v[r][k] = x[r];
                    if constexpr (SRC == 6) {
                        ww[r] = cscale(csub(g[r][k], ww[r]), PU(k));
                        v[r][k] = zfma(v[r][k], cTv, ww[r]);
                    }
                }
            }
        }

#pragma unroll
        for (int r = 0; r < NR; r++) {
            if (b + r >= b_end) break;
            double2 *dst = out + (long)(b + r) * field + off0;
            if constexpr (PCS || is_real_v<MT>) {
                // one running address and a row count re-formed here: per-row offsets and
                // conditions hoisted out of the loop over right-hand sides would pin registers
                long rsd = row_stride;
                int  nk = live ? rows - r0 : 0;
                asm volatile("" : "+l"(rsd), "+r"(nk));
#pragma unroll
                for (int k = 0; k < KS; k++) {
                    if (k < nk) *dst = v[r][k];
                    dst += rsd;
                }
            } else {
#pragma unroll
                for (int k = 0; k < KS; k++)
                    if (live && r0 + k < rows) dst[(long)k * row_stride] = v[r][k];
            }
        }
    }
}

// Stage multipliers of the intra-warp scans for one per-segment multiplier a (complex, or real
// for the Pade solve): tab[j * NT] = the thread's map product before stage j, tab[LOG * NT] =
// the exclusive product.  Returns the inclusive product, which at the warp's last (forward) or
// first (backward) segment is the warp total.
__device__ __forceinline__ double shfl_up1(double v, int off) { return __shfl_up_sync(0xffffffffu, v, off); }
__device__ __forceinline__ double shfl_down1(double v, int off) { return __shfl_down_sync(0xffffffffu, v, off); }
__device__ __forceinline__ double2 shfl_up1(double2 v, int off) { return shfl_up2(v, off); }
__device__ __forceinline__ double2 shfl_down1(double2 v, int off) { return shfl_down2(v, off); }
__device__ __forceinline__ double  mul1(double a, double b) { return a * b; }
__device__ __forceinline__ double2 mul1(double2 a, double2 b) { return cmul(a, b); }

template <int CW, bool FWD, typename M>
__device__ __forceinline__ M sym_scan_table(M a, M *tab, int NT_, int sl, M one) {
    constexpr int SPW = 32 / CW;
    int           j = 0;
#pragma unroll
    for (; (1 << j) < SPW; j++) {
        tab[j * NT_] = a;
        const M o = FWD ? shfl_up1(a, CW << j) : shfl_down1(a, CW << j);
        if (FWD ? (sl >= (1 << j)) : (sl + (1 << j) < SPW)) a = mul1(a, o);
    }
    M e = FWD ? shfl_up1(a, CW) : shfl_down1(a, CW);
    if (FWD ? sl == 0 : sl == SPW - 1) e = one;
    tab[j * NT_] = e;
    return a;
}

// Elements of one TMA tile [rows][cw] (whole 128-byte units), and the rows per box.
__host__ __device__ inline int sym_tile_rows_per_box(int rows) { return rows < 256 ? rows : 256; }
__host__ __device__ inline int sym_tile_elems(int rows, int cw) {
    const int br = sym_tile_rows_per_box(rows), nbox = (rows + br - 1) / br;
    return (nbox * br * cw + 7) / 8 * 8;
}

// Several plans of one shape in one launch (hh_solve_source_multi): chunk j of the grid's y
// dimension solves right-hand sides [b0, b1) of the batch with the factors and wavenumber of plan
// `plan`; everything else (eigenvalues, Pade factors, h) is the same for plans of one shape.
struct SymPlanRef {
    const double2 *Pv, *subt, *diagt;
    double2        k2h2_20;
};
struct SymChunk {
    int plan, b0, b1, pad;
};
// The table of a multi-plan launch (none: nchunks 0): a small one travels in the kernel's arguments, because the
// two copies to device memory that larger ones take wait for the kernel before them and hold the line solve back
// (2D 255^2, 8 plans x 4: 55.7 us a solve with them, 48.4 without).
struct SymMulti {
    static constexpr int kPlans = 16, kChunks = 64;
    int               nchunks = 0;      // the grid's y extent
    const SymPlanRef *refs = nullptr;   // in device memory, or null: the arrays below
    const SymChunk   *chunks = nullptr;
    SymPlanRef        iref[kPlans];
    SymChunk          ichunk[kChunks];
};

template <int SRC, int NT, int CW, int MINB, int NR, int KS, bool TIO, typename MT>
__global__ void __launch_bounds__(NT, MINB)
    k_line_solve_sym(const double2 *__restrict__ in, double2 *__restrict__ out, int lines, int rows, long row_stride,
                     long field, int batch, int rb, const double2 *__restrict__ Pv_one, const double2 *__restrict__ subt_one,
                     const double2 *__restrict__ diagt_one, int prow, const double *__restrict__ mu, SymParams sp,
                     const __grid_constant__ CUtensorMap in_map, int *err, int pitch, int pitch_nx,
                     const __grid_constant__ SymMulti tab) {
    constexpr int NW = NT / 32, SPW = 32 / CW, LOG = ilog2_t<SPW>();
    constexpr int HALO = (SRC == 4 || SRC == 6) ? 1 : 0;
    __shared__ SymSmem<NW, CW, NR, MT> sm;
    extern __shared__ __align__(128) unsigned char dyn_raw[];
    // 128-byte aligned start (tensor copies need it; the allocation carries 128 bytes of slack)
    double2 *dyn = reinterpret_cast<double2 *>(dyn_raw + ((128u - (smem_u32(dyn_raw) & 127u)) & 127u));
    // per-thread prefetch slots [NR][KS + 2][NT], or the input tiles
    const int io_elems = TIO ? sym_tile_elems(rows, CW) * SymTileBufs<SRC, MT>::value : NR * (KS + 2) * NT;
    double2  *pre = dyn;
    MT *tabF = reinterpret_cast<MT *>(pre + io_elems);  // [LOG + 1][NT]
    MT *tabB = tabF + (LOG + 1) * NT;                   // [LOG + 1][NT]
    constexpr bool UIS = SymUIS<SRC, KS, MT>::value;
    MT *uis = tabB + (LOG + 1) * NT;               // [KS][NT] tau_k (UIS)
    double  *ttF = reinterpret_cast<double *>(uis + (UIS ? KS * NT : 0)); // [LOG + 1][NT] (SymTT)
    double  *ttB = ttF + SymTT<SRC, KS>::value * (LOG + 1) * NT;
    (void)HALO;

    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int c = t % CW, seg = t / CW, sl = lane / CW;
    // the line's position in a row of the field, and its number: with padded rows of `pitch` positions (3D),
    // position i + j pitch holds line i + j pitch_nx, and the positions from pitch_nx on none
    const int  at = blockIdx.x * CW + c;
    const bool gap = pitch && at % pitch >= pitch_nx;
    const int  q = pitch ? at / pitch * pitch_nx + at % pitch : at;
    // this CTA's right-hand sides and the plan they belong to
    int            b_begin, b_end;
    const double2 *Pv = Pv_one, *subt = subt_one, *diagt = diagt_one;
    if (tab.nchunks) {
        const SymChunk   ch = tab.chunks ? tab.chunks[blockIdx.y] : tab.ichunk[blockIdx.y];
        const SymPlanRef pr = tab.chunks ? tab.refs[ch.plan] : tab.iref[ch.plan];
        b_begin = ch.b0;
        b_end = ch.b1;
        Pv = pr.Pv;
        subt = pr.subt;
        diagt = pr.diagt;
        sp.k2h2_20 = pr.k2h2_20;
    } else {
        b_begin = blockIdx.y * rb;
        b_end = min(batch, b_begin + rb);
    }
    SymTio    tio{};
    if constexpr (TIO) {
        constexpr int NBUF = SymTileBufs<SRC, MT>::value;
        tio.in_map = &in_map;
        tio.tin = pre;
        tio.bar = sm.tbar;
        tio.err = err;
        tio.x0 = blockIdx.x * CW;
        tio.br = sym_tile_rows_per_box(rows);
        tio.nbox = (rows + tio.br - 1) / tio.br;
        tio.tile = sym_tile_elems(rows, CW);
        tio.tile_bytes = (unsigned)(tio.nbox * tio.br * CW * 16);
        if (t == 0) { // the first right-hand sides' tiles come in while the factors are set up
            const int b0 = b_begin, b1 = b_end;
            for (int u = 0; u < NBUF; u++) mbar_init(tio.bar + u, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            pdl_wait(); // (the fields are written after a tile has arrived: this thread's wait is enough)
            pdl_next();
            for (int u = 0; u < NBUF && b0 + u < b1; u++) {
                double2 *dst = tio.tin + (long)u * tio.tile;
                mbar_expect_tx(tio.bar + u, tio.tile_bytes);
                for (int x = 0; x < tio.nbox; x++)
                    tma_load_3d(dst + (long)x * tio.br * CW, tio.in_map, 2 * tio.x0, x * tio.br, b0 + u, tio.bar + u);
            }
        }
    }
    const bool live = q < lines && !gap;
    const int  qq = live ? q : 0;
    const int  r0 = seg * KS;
    const double m0 = mu[qq], m1 = mu[lines + qq], m2 = mu[2 * lines + qq];
    const MT one = coef_of<MT>(make_double2(1.0, 0.0)), zero = MT{};

    // ---- factors of the thread's rows (the set-up's recurrence, same arithmetic)
    const MT s = coef_of<MT>(shifted(subt, prow, 0, m0, m1, m2)), d = coef_of<MT>(shifted(diagt, prow, 0, m0, m1, m2));
    MT Lr[KS], ui[KS];
    MT Af = one, Ab = one;
    const MT ui_in = (live && r0 > 0 && r0 < rows) ? coef_of<MT>(Pv[(long)(r0 / 8) * lines + q]) : zero; // 1/P of row r0-1
    {
        MT uprev = ui_in;
#pragma unroll
        for (int k = 0; k < KS; k++) {
            const int r = r0 + k;
            Lr[k] = zero;
            ui[k] = zero;
            if (live && r < rows) {
                if (r == 0) ui[k] = first_pivot(d);
                else ui[k] = factor_step(s, d, s, uprev, Lr[k]);
            }
            uprev = ui[k];
            Af = cmul(Af, mneg(Lr[k]));
            const MT tau = cmul(s, ui[k]);
            Ab = cmul(Ab, mneg(tau));
            if constexpr (SRC == 6) { // order 6 keeps tau_k in place of ui_k
                if constexpr (UIS) uis[k * NT + t] = tau;
                else ui[k] = tau;
            }
        }
    }

    // ---- per-line coefficients of the compact right-hand side
    MT     c1 = one, cT = zero;
    double c2 = 0.0;
    if constexpr (SRC == 4) {
        c1 = coef_of<MT>(make_double2(sp.h2 * (sp.dim == 2 ? (10.0 + m1) / 12.0 : (8.0 + m1 + m2) / 12.0), 0.0));
        c2 = sp.h2 / 12.0;
    } else if constexpr (SRC == 6) {
        double2 a6;
        double  b6;
        if (sp.dim == 2) {
            const double muq = 12.0 * (m1 - 2.0) / (10.0 + m1);
            a6 = make_double2(1.6 + muq / 12.0 + (m1 - 2.0) * muq / 360.0 - sp.k2h2_20.x, -sp.k2h2_20.y);
            b6 = muq / 90.0 + 1.0 / 30.0;
        } else {
            const double mx = 12.0 * (m1 - 2.0) / (10.0 + m1), my = 12.0 * (m2 - 2.0) / (10.0 + m2);
            a6 = make_double2(1.6 + (mx + my) / 12.0 + ((m1 - 2.0) * mx + (m2 - 2.0) * my) / 360.0 +
                                  (m2 - 2.0) * mx / 90.0 - sp.k2h2_20.x,
                              -sp.k2h2_20.y);
            b6 = (mx + my) / 90.0 + 1.0 / 30.0;
        }
        // 1/(10 s - d)
        if constexpr (is_real_v<MT>) {
            const double den = crcp(10.0 * s - d), sr = s * den;
            c1 = sp.h2 * (a6.x - 7.2 * sr);
            cT = 7.2 * sp.h2 * den;
        } else {
            const double2 den = crcp(make_double2(10.0 * s.x - d.x, 10.0 * s.y - d.y));
            const double2 sr = cmul(s, den);
            c1 = make_double2(sp.h2 * (a6.x - 7.2 * sr.x), sp.h2 * (a6.y - 7.2 * sr.y));
            cT = make_double2(7.2 * sp.h2 * den.x, 7.2 * sp.h2 * den.y);
        }
        c2 = sp.h2 * b6;
        if constexpr (SymPCS<SRC, KS, CW, MT>::value) {
            double2 *pcs = reinterpret_cast<double2 *>(ttB + SymTT<SRC, KS>::value * (LOG + 1) * NT);
            pcs[t] = cmul(s, ui_in);
            pcs[NT + t] = crcp(s);
            pcs[2 * NT + t] = c1;
            pcs[3 * NT + t] = cT;
            pcs[4 * NT + t] = make_double2(c2, 0.0);
        }
    }

    // ---- scan tables (factor-only, shared by every right-hand side of the chunk)
    {
        const MT totF = sym_scan_table<CW, true>(Af, tabF + t, NT, sl, one);
        const MT totB = sym_scan_table<CW, false>(Ab, tabB + t, NT, sl, one);
        if (sl == SPW - 1) sm.AwF[w][c] = totF;
        if (sl == 0) sm.AwB[w][c] = totB;
    }
    if constexpr (SRC == 6) {
        if (t < 11) {
            sm.pl[t] = t < 9 ? sp.pl[t] : (t == 9 ? sp.linf : 0.0);
            sm.pu[t] = t < 9 ? sp.pu[t] : (t == 9 ? sp.uinf : 0.0);
        }
        if constexpr (SymTT<SRC, KS>::value) {
            __syncthreads();
            double af = 1.0, ab = 1.0;
#pragma unroll
            for (int k = 0; k < KS; k++) {
                const int r = r0 + k;
                af *= -(r < 9 ? sm.pl[r] : (r < rows ? sp.linf : 0.0));
                ab *= -(r < 9 ? sm.pu[r] : (r < rows ? sp.uinf : 0.0));
            }
            const double totF = sym_scan_table<CW, true>(af, ttF + t, NT, sl, 1.0);
            const double totB = sym_scan_table<CW, false>(ab, ttB + t, NT, sl, 1.0);
            if (sl == SPW - 1) sm.awF[w][c] = totF;
            if (sl == 0) sm.awB[w][c] = totB;
        }
    }
    __syncthreads();

    if constexpr (!TIO) {
        pdl_wait();
        pdl_next();
    }
    const long off0 = (long)r0 * row_stride + (live ? at : 0);
    // warps whose rows all lie in [9, rows) use the constant Pade factors
    const bool tint = (w * SPW * KS >= 9) && ((w + 1) * SPW * KS <= rows);
    if (SRC == 6 && tint)
        sym_chunk<SRC, NT, CW, true, NR, KS, TIO, MT>(in, out, rows, row_stride, field, b_begin, b_end, off0, live, r0, sl,
                                                  w, c, Lr, ui, uis, ui_in, s, c1, c2, cT, sm, pre, tabF, tabB, ttF,
                                                  ttB, sp, tio);
    else
        sym_chunk<SRC, NT, CW, false, NR, KS, TIO, MT>(in, out, rows, row_stride, field, b_begin, b_end, off0, live, r0,
                                                   sl, w, c, Lr, ui, uis, ui_in, s, c1, c2, cT, sm, pre, tabF, tabB,
                                                   ttF, ttB, sp, tio);
}

// Right-hand sides per CTA: the chunk whose grid has the smallest wave-quantised cost,
//   ceil(CTAs / resident CTAs) * (rb + 1),
// counting the per-chunk set-up (factors and scan tables) as about one right-hand side.
static int pick_rb(long groups, int batch, int resident, int nr) {
    int  best = nr, rb = nr;
    long best_cost = -1;
    for (; ; rb *= 2) {
        const int  r = rb < batch ? rb : batch;
        const long ctas = groups * ((batch + r - 1) / r);
        const long cost = ((ctas + resident - 1) / resident) * (long)(r + 1);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = r; }
        if (rb >= batch) break;
    }
    return best;
}

// (double, row, right-hand side) map of a batch of line-solve fields, boxes of cw lines by br rows.  A row
// of a box is one run of 16 cw bytes: with (re, im) as a dimension of its own the copy went out value
// by value and bounded the kernel (line solve, real coefficients: 2D 1023^2 x 64 order 6 597 -> 552 us, order 4
// 507 -> 467 us; 2D 511^2 x 32 order 4 62 -> 51 us; 3D 255^3 x 4 order 6 552 -> 506 us, order 4 497 -> 386 us)
static int encode_line_map(CUtensorMap *map, const double2 *base, const Plan *p, int batch, int cw, int br) {
    const unsigned long long dims[3] = {2ULL * (unsigned long long)p->span(), (unsigned long long)p->rows,
                                        (unsigned long long)batch};
    const unsigned long long strides[2] = {(unsigned long long)p->row_stride * 16, (unsigned long long)p->field * 16};
    const unsigned           box[3] = {2u * (unsigned)cw, (unsigned)br, 1};
    return encode_tensor_map(map, base, 3, dims, strides, box);
}

template <int SRC, int CW, int MINB, int NR, int KS, bool TIO, typename MT>
static int launch_sym_t(Plan *p, const double2 *in, double2 *out, int batch, const SymMulti *multi) {
    constexpr int NT = 256, SPW = 32 / CW, LOG = ilog2_t<SPW>();
    SymParams sp;
    sp.h2 = p->h * p->h;
    sp.k2h2_20 = make_double2(p->k2.x * sp.h2 / 20.0, p->k2.y * sp.h2 / 20.0);
    sp.dim = p->dim;
    sp.linf = p->pade_linf;
    sp.uinf = p->pade_uinf;
    sp.pl = p->pade_l;
    sp.pu = p->pade_u;
    double cz = 1.0;
    for (int k = 0; k < 16; k++) sp.cz[k] = cz *= -p->pade_linf;
    auto smem = [](int rows) {
        const int io_elems = TIO ? sym_tile_elems(rows, CW) * SymTileBufs<SRC, MT>::value : NR * (KS + 2) * NT;
        return 128 + (int)(sizeof(double2) * io_elems +
                           sizeof(MT) * (2 * (LOG + 1) * NT + (SymUIS<SRC, KS, MT>::value ? KS * NT : 0) +
                                         (SymPCS<SRC, KS, CW, MT>::value ? 5 * NT : 0)) +
                           sizeof(double) * 2 * SymTT<SRC, KS>::value * (LOG + 1) * NT);
    };
    const int shm = smem(p->rows);
    CUtensorMap in_map{};
    if constexpr (TIO) HH_TRY(encode_line_map(&in_map, in, p, batch, CW, sym_tile_rows_per_box(p->rows)));
    HH_TRY(allow_smem(k_line_solve_sym<SRC, NT, CW, MINB, NR, KS, TIO, MT>, smem(NT / CW * KS))); // (NT / CW segments a line)
    const long groups = (p->span() + CW - 1) / CW;
    int blocks_per_sm = 0, dev = 0, sms = 148;
    HH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, k_line_solve_sym<SRC, NT, CW, MINB, NR, KS, TIO, MT>, NT,
                                                          shm));
    HH_CUDA(cudaGetDevice(&dev));
    HH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int rb = pick_rb(groups, batch, std::max(1, blocks_per_sm) * sms, NR);
    const int chunks = multi ? multi->nchunks : (batch + rb - 1) / rb;
    dim3 grid((unsigned)groups, (unsigned)chunks);
    return launch_kernel(p->ctx, k_line_solve_sym<SRC, NT, CW, MINB, NR, KS, TIO, MT>, grid, NT, (size_t)shm,
        in, out, p->lines, p->rows, p->row_stride, p->field, batch, rb, p->Pv, p->subt, p->diagt, p->prow, p->mu, sp,
        in_map, p->ctx->err_word, p->pitch, p->nx, multi ? *multi : SymMulti{});
}

// The two builds of the kernel (hh_line_sym_real.cu, hh_line_sym_cplx.cu).
int launch_sym_real(Plan *p, const double2 *in, double2 *out, int batch, int src_order, const SymMulti *multi);
int launch_sym_cplx(Plan *p, const double2 *in, double2 *out, int batch, int src_order, const SymMulti *multi);

// TIO: tile I/O where a line group is at least two lines (32-byte row pieces or wider); one-line
// groups keep the per-thread prefetch.
// segments per line of the symmetric kernel: a power of two P >= rows / KS with 8 <= P <= 256
// (CW = 256 / P lines per CTA); P = 8 runs one right-hand side per pass
static int sym_segments(int rows, int ks) {
    int P = 8;
    while (P * ks < rows) P <<= 1;
    return P;
}

template <typename MT, int SRC, int MINB, int NR, int KS, bool TIO = false>
static int launch_sym_src(Plan *p, const double2 *in, double2 *out, int batch, const SymMulti *multi) {
    switch (sym_segments(p->rows, KS)) {
    case 8: return launch_sym_t<SRC, 32, MINB, 1, KS, TIO, MT>(p, in, out, batch, multi); // per-RHS scan arrays would not fit
    case 16: return launch_sym_t<SRC, 16, MINB, NR, KS, TIO, MT>(p, in, out, batch, multi);
    case 32: return launch_sym_t<SRC, 8, MINB, NR, KS, TIO, MT>(p, in, out, batch, multi);
    case 64: return launch_sym_t<SRC, 4, MINB, NR, KS, TIO, MT>(p, in, out, batch, multi);
    case 128: return launch_sym_t<SRC, 2, MINB, NR, KS, TIO, MT>(p, in, out, batch, multi); // 32-byte row pieces
    case 256: return launch_sym_t<SRC, 1, MINB, NR, KS, false, MT>(p, in, out, batch, multi);
    default: set_error("symmetric line solve: %d rows", p->rows); return HH_ERR_UNSUPPORTED;
    }
}

// Variants of the symmetric kernel: 2 = two CTAs per SM, 3 = one CTA per SM (no register cap),
// 4 = one CTA per SM with two right-hand sides per pass, 5 = one CTA per SM with 16-row segments
// (twice the lines per CTA: wider contiguous row pieces in global memory, half the scans; at
// order 6 the reciprocal pivots move to shared memory), 6 = variant 5 with each right-hand side
// brought in as a TMA tile where a CTA holds at least four lines.
template <typename MT, int SRC>
static int launch_sym_variant(Plan *p, const double2 *in, double2 *out, int batch, const SymMulti *multi) {
    switch (p->variant) {
    case 3: return launch_sym_src<MT, SRC, 1, 1, kSeg>(p, in, out, batch, multi);
    case 4: return launch_sym_src<MT, SRC, 1, 2, kSeg>(p, in, out, batch, multi);
    case 5: return launch_sym_src<MT, SRC, 1, 1, 16>(p, in, out, batch, multi);
    case 6: return launch_sym_src<MT, SRC, 1, 1, 16, true>(p, in, out, batch, multi);
    default: return launch_sym_src<MT, SRC, 2, 1, kSeg>(p, in, out, batch, multi);
    }
}

template <typename MT>
static int launch_sym_order(Plan *p, const double2 *in, double2 *out, int batch, int src_order, const SymMulti *multi) {
    switch (src_order) {
    case 0: return launch_sym_variant<MT, 0>(p, in, out, batch, multi);
    case 2: return launch_sym_variant<MT, 2>(p, in, out, batch, multi);
    case 4: return launch_sym_variant<MT, 4>(p, in, out, batch, multi);
    case 6: return launch_sym_variant<MT, 6>(p, in, out, batch, multi);
    default: set_error("source operator order %d", src_order); return HH_ERR_INVALID;
    }
}

} // namespace hh

#endif
