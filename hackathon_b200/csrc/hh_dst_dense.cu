// DST-I of any length as two half-size FP64 tensor-core products (sm_100a).
//
// Serves the lengths whose n + 1 is not a power of two in 64 .. 8192, which the FFT kernels of
// hh_dst.cu cannot take (the reference's own sizes among them: N = 100, 125, 500), in place of the
// reference's length-(2n+2) real FFTs (2D_Program/solver_functions/DST.c:6-44,
// 3D_Program/solver_functions/DST.c:148-204).
//
// With M = n + 1 the sine matrix splits by the mirror symmetry sin(pi (M-j) k / M) =
// -(-1)^k sin(pi j k / M):
//     S_k (k odd)  = sum_{j <= ceil(n/2)} sin(pi j k / M) a_j,   a_j = x_j + x_{M-j} (x_j alone at j = M/2)
//     S_k (k even) = sum_{j <= floor(n/2)} sin(pi j k / M) d_j,  d_j = x_j - x_{M-j}
// so a line of n complex values costs 2 n^2 real operations instead of 4 n^2, in sums half as long.
//
// A CTA takes NL lines, forms a and d of all of them in shared memory (so the transform may run in
// place), and its warps walk units (8 odd and 8 even outputs) x (NTW tiles of 4 complex lines =
// 8 real columns): mma.m8n8k4 in FP64 with the sine fragments as A and the lines as B.  The
// sines come from a table laid out fragment by fragment, the odd and the even matrix side by side,
// so that a lane reads both of its values with one 16-byte load, two steps ahead, and no shared
// memory is spent on them: every CTA reads the table once (4 n^2 bytes, from L1/L2).  The C
// fragment's two values are the real and imaginary part of one output, and the lane that holds output
// 2i of a line also holds output 2i + 1, so stores go out as 32-byte pairs.
//
// Bound by the FP64 tensor rate from n ~ 200 on (37 TF measured; 8000 rows of n = 500 take 139 us, 108 us
// of it at that rate), below that by the load and store phases.  Against one dot product per thread
// with uncoalesced sines before: 8000 rows of n = 500 5083 -> 139 us, 40000 rows of n = 100 585 -> 43.5
// us, columns 643 -> 42 us.
#include "hh_internal.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace hh {

namespace {

constexpr int kTabAhead = 2; // table steps in flight (a pair per pass of the product loop)
constexpr int kMmaSmemMax = 227 * 1024;
// the longest line that fits four to a CTA in both layouts (2 * 1200 * 6 * 16 bytes at n = 2400)
constexpr int kMmaMaxN = 2400;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// geometry shared by host and device: h1 odd outputs (and values a_j), k4 steps of four j
__host__ __device__ inline int half_up(int n) { return (n + 1) / 2; }
__host__ __device__ inline int k4_steps(int n) { return (half_up(n) + 3) / 4; }
__host__ __device__ inline int out_tiles(int n) { return (half_up(n) + 7) / 8; }
// threads of a CTA: four warps where there are at most four output tiles (n <= 64), whose blocks then are half as
// large and twice as many on an SM (61504 rows of n = 31 17.5 -> 14.9 us, 40000 of n = 50 18.7 -> 17.0), else eight
// (40000 of n = 100 43.9 us, 44.6 with four; 8000 of n = 500 139, 153 with four)
inline int mma_threads(int n) { return out_tiles(n) <= 4 ? 128 : 256; }
// Shared memory holds blocks of four a_j and then their four d_j, so that a lane reaches a step's both values of
// a line by constant offsets.  Pitches in complex values: a B fragment is 4 values of j by 8 real columns, read
// by half warps of 4 x 4; rows (line-major): pitch = 4 mod 8 puts the two lines of a half warp on
// different 64-byte halves of the banks; columns (j-major): pitch = 2 or 6 mod 8 puts its four j on
// four different 32-byte quarters
__host__ __device__ inline int rows_pitch(int n) { return 8 * k4_steps(n) + 4; }
__host__ __device__ inline int cols_pitch(int nl) { return nl + 2; } // nl is a multiple of 4

inline size_t mma_smem(bool cols, int n, int nl) {
    return sizeof(double2) * (cols ? (size_t)8 * k4_steps(n) * cols_pitch(nl) : (size_t)nl * rows_pitch(n));
}

// COLS: line c of a plane is column c (element j at c + j ld); otherwise row c (element j at c ld + j).
// What is not a product counts here: at n = 100 a warp's one unit is 208 of its instructions, and with plain
// indexing in the three phases it ran 1262, now 776 (40000 rows 49 -> 43.5 us, 8000 rows of n = 500 160 -> 139,
// 61504 of n = 31 23 -> 17.5, 100 columns x 400 planes 46 -> 42); so the addresses of a phase advance by
// constants, nothing is computed per thread that the launch can pass, and the first table steps of a unit are on
// their way before its lines are.
template <bool COLS, int NTW, int NT>
__global__ void __launch_bounds__(NT, 768 / NT)
    k_dst1_mma(const double2 *in, double2 *out, int n, long nlines, long in_ld, long out_ld, long in_plane,
               long out_plane, int groups, double coef, const double2 *__restrict__ tab) {
    extern __shared__ __align__(16) double2 mma_sm[];
    constexpr int NW = NT / 32;
    const int  h1 = half_up(n), ks = k4_steps(n), nl = 4 * NTW * groups;
    const int  pitch = COLS ? cols_pitch(nl) : rows_pitch(n);
    const int  lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int  units = out_tiles(n) * groups;
    const long l0 = (long)blockIdx.x * nl;
    const int  live = (int)min((long)nl, nlines - l0);
    const double2 zero = make_double2(0.0, 0.0);
    in += (long)blockIdx.y * in_plane + (COLS ? l0 : l0 * in_ld);
    out += (long)blockIdx.y * out_plane + (COLS ? l0 : l0 * out_ld);

    pdl_wait();
    pdl_next();
    auto tile_of = [&](int u) { return groups == 1 ? u : u / groups; };
    // (reads past a tile's last step stay in the table: it ends in kTabAhead spare steps)
    const double2 *q = tab + (long)tile_of(warp) * ks * 32 + lane;
    double2        cur[kTabAhead];
    if (warp < units)
#pragma unroll
        for (int i = 0; i < kTabAhead; i++) cur[i] = __ldg(q + i * 32);

    // ---- a_j and d_j of every line; zeros past the halves and for lines past the end
    const int mid = n & 1 ? n / 2 : -1; // x_mid stands alone
    double2   x[4], m[4];
    int       at[4], js[4];
    auto      put = [&]() {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (at[e] >= 0) {
                mma_sm[at[e]] = js[e] == mid ? x[e] : cadd(x[e], m[e]);
                mma_sm[at[e] + (COLS ? 4 * pitch : 4)] = js[e] == mid ? zero : csub(x[e], m[e]);
            }
    };
    if constexpr (COLS) {
        const int dj = NT / nl, dc = NT - dj * nl;
        int       j = threadIdx.x / nl, c = threadIdx.x - j * nl;
        while (j < 4 * ks) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                x[e] = m[e] = zero;
                if (j < h1 && c < live) {
                    x[e] = in[c + j * in_ld];
                    m[e] = in[c + (n - 1 - j) * in_ld];
                }
                at[e] = j < 4 * ks ? (2 * j - (j & 3)) * pitch + c : -1;
                js[e] = j;
                j += dj;
                c += dc;
                if (c >= nl) {
                    c -= nl;
                    j++;
                }
            }
            put();
        }
    } else {
        // a warp takes pieces of 32 j, `pieces` to a line
        const int pieces = (4 * ks + 31) / 32, dc = NW / pieces, dr = NW - dc * pieces;
        int       c = warp / pieces, r = warp - c * pieces;
        while (c < nl) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int j = 32 * r + lane;
                x[e] = m[e] = zero;
                if (j < h1 && c < live) {
                    const double2 *line = in + c * in_ld;
                    x[e] = line[j];
                    m[e] = line[n - 1 - j];
                }
                at[e] = j < 4 * ks && c < nl ? c * pitch + 2 * j - (j & 3) : -1;
                js[e] = j;
                c += dc;
                r += dr;
                if (r >= pieces) {
                    r -= pieces;
                    c++;
                }
            }
            put();
        }
    }
    __syncthreads();

    const int     kk = lane & 3, nn = lane >> 2; // the lane's j within a step and real column within a tile
    const double *lines = reinterpret_cast<const double *>(mma_sm) + (nn & 1);
    for (int u = warp; u < units; u += NW) {
        const int tile = tile_of(u), c0 = (u - tile * groups) * 4 * NTW;
        double    ao[NTW][2], ae[NTW][2];
#pragma unroll
        for (int t = 0; t < NTW; t++) ao[t][0] = ao[t][1] = ae[t][0] = ae[t][1] = 0.0;
        // rows: b[t] walks the line of tile t; columns: b[0] and b[1] walk the a_j and the d_j
        constexpr int NB = COLS ? 2 : NTW;
        const double *b[NB];
        if constexpr (COLS) {
            b[0] = lines + 2 * (kk * pitch + (nn >> 1) + c0);
            b[1] = b[0] + 8 * pitch;
        } else {
#pragma unroll
            for (int t = 0; t < NTW; t++) b[t] = lines + 2 * ((c0 + 4 * t + (nn >> 1)) * pitch + kk);
        }
        auto step = [&](double2 sine, int i) {
#pragma unroll
            for (int t = 0; t < NTW; t++) {
                dmma(ao[t], sine.x, COLS ? b[0][8 * t] : b[COLS ? 0 : t][16 * i]);
                dmma(ae[t], sine.y, COLS ? b[1][8 * t] : b[COLS ? 0 : t][16 * i + 8]);
            }
            if constexpr (COLS) {
                b[0] += 16 * pitch;
                b[1] += 16 * pitch;
            }
        };
        for (int k = kTabAhead; k <= ks; k += kTabAhead) {
            double2 nxt[kTabAhead];
            q += 32 * kTabAhead;
#pragma unroll
            for (int i = 0; i < kTabAhead; i++) nxt[i] = __ldg(q + i * 32);
#pragma unroll
            for (int i = 0; i < kTabAhead; i++) step(cur[i], i);
            if constexpr (!COLS)
#pragma unroll
                for (int t = 0; t < NTW; t++) b[t] += 16 * kTabAhead;
#pragma unroll
            for (int i = 0; i < kTabAhead; i++) cur[i] = nxt[i];
        }
        static_assert(kTabAhead == 2, "at most one step is left");
        if (ks & 1) step(cur[0], 0);
        if (u + NW < units) {
            q = tab + (long)tile_of(u + NW) * ks * 32 + lane;
#pragma unroll
            for (int i = 0; i < kTabAhead; i++) cur[i] = __ldg(q + i * 32);
        }
        // output 2i (S_{2i+1}) and 2i + 1 (S_{2i+2}) of line c0 + 4 t + kk
        const int  i2 = 16 * tile + 2 * nn;
        double2   *o = out + (COLS ? c0 + kk + i2 * out_ld : (c0 + kk) * out_ld + i2);
        const long next = COLS ? out_ld : 1;
#pragma unroll
        for (int t = 0; t < NTW; t++) {
            if (c0 + 4 * t + kk < live) {
                if (i2 < n) o[0] = make_double2(coef * ao[t][0], coef * ao[t][1]);
                if (i2 + 1 < n) o[next] = make_double2(coef * ae[t][0], coef * ae[t][1]);
            }
            o += COLS ? 4 : 4 * out_ld;
        }
    }
}

// the fragment table: (odd, even) sines of output row 8 tile + lane / 4 and value 4 k + lane % 4
__global__ void k_make_mma(int n, double2 *tab) {
    const int  h1 = half_up(n), p = n / 2, ks = k4_steps(n);
    const long tot = (long)out_tiles(n) * ks * 32;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < tot; e += (long)gridDim.x * blockDim.x) {
        const int  lane = (int)(e & 31);
        const long s = e >> 5;
        const long i = 8 * (s / ks) + (lane >> 2), j = 4 * (s % ks) + (lane & 3) + 1;
        const long m2 = 2L * (n + 1); // arguments reduced mod 2 (n + 1) keep sinpi's in [0, 2)
        double2    v = make_double2(0.0, 0.0);
        if (i < h1 && j <= h1) v.x = sinpi((double)((2 * i + 1) * j % m2) / (double)(n + 1));
        if (i < p && j <= p) v.y = sinpi((double)((2 * i + 2) * j % m2) / (double)(n + 1));
        tab[e] = v;
    }
}

// the full n x n sine matrix of the lengths past kMmaMaxN
__global__ void k_make_dense(int n, double *mat) {
    const long tot = (long)n * n;
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < tot; q += (long)gridDim.x * blockDim.x) {
        const long k = q / n, m = q % n;
        // (k+1)(m+1) reduced mod 2(n+1) keeps the argument of sinpi in [0, 2)
        const long num = ((k + 1) * (m + 1)) % (2L * (n + 1));
        mat[q] = sinpi((double)num / (double)(n + 1));
    }
}

// One line per CTA against the full matrix, for the lines too long for k_dst1_mma.  The matrix is
// symmetric: thread k walks column k, so that a warp reads neighbouring values.  Every CTA streams the whole matrix
// through L2, and what bounds it is the latency of those loads, so the CTA is as large as can be and each thread has
// 16 of them in flight (30 rows of n = 4000: one dot product per thread along a row, 128 threads 12.4 ms; along a column
// 15.4, so 2.4; 30 columns 11.4, 20.6 and 2.4).
constexpr int kDenseThreads = 1024;
constexpr int kDenseAhead = 16;  // matrix values a thread has in flight
constexpr int kDenseMaxN = 4096; // the longest line the transforms accept here
template <bool STRIDED>
__global__ void __launch_bounds__(kDenseThreads)
    k_dst1_dense(const double2 *__restrict__ in, double2 *__restrict__ out, int n, long in_ld, long out_ld,
                 long in_plane, long out_plane, const double *__restrict__ mat) {
    extern __shared__ __align__(128) unsigned char smem_dense[];
    double2   *x = reinterpret_cast<double2 *>(smem_dense);
    const long line = blockIdx.x;
    in += (long)blockIdx.y * in_plane;
    out += (long)blockIdx.y * out_plane;
    pdl_wait();
    pdl_next();
    for (int m = threadIdx.x; m < n; m += blockDim.x) x[m] = STRIDED ? in[line + (long)m * in_ld] : in[line * in_ld + m];
    __syncthreads();
    const double coef = sqrt(2.0 / (n + 1));
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double        sr = 0.0, si = 0.0;
        const double *col = mat + k;
        int           m = 0;
        for (; m + kDenseAhead <= n; m += kDenseAhead, col += (long)kDenseAhead * n) {
            double s[kDenseAhead];
#pragma unroll
            for (int i = 0; i < kDenseAhead; i++) s[i] = __ldg(col + (long)i * n);
#pragma unroll
            for (int i = 0; i < kDenseAhead; i++) {
                sr = fma(s[i], x[m + i].x, sr);
                si = fma(s[i], x[m + i].y, si);
            }
        }
        for (; m < n; m++, col += n) {
            const double s = __ldg(col);
            sr = fma(s, x[m].x, sr);
            si = fma(s, x[m].y, si);
        }
        const double2 r = make_double2(coef * sr, coef * si);
        if (STRIDED) out[line + (long)k * out_ld] = r;
        else out[line * out_ld + k] = r;
    }
}

// Lines per CTA: 4 ntw lines per warp unit, `groups` units side by side.
//  * groups: the least that gives all warps a unit (n <= 48 has fewer than four output tiles).
//  * ntw: the widest of 4, 3, 2 whose lines leave room for 24 warps on an SM (n = 100: 43.5 us at 4
//    against 44.5 at 3 and 48.1 at 2 for 40000 rows; n = 300: 38 us at 3 against 41 at 2; n = 500: 139 us
//    at 2 against 152 at 1, 146 at 3 with 16 warps), then 2 with 16 warps (n = 700), then 1 (n = 1000: 161 us,
//    169 at 2).  Columns take the width (up to 5) that
//    leaves the fewest idle columns in a plane's last tile (100 columns: 42 us at 5, 46.5 at 4).
//  * fewer lines per CTA where the launch would not give every SM sixteen warps (7688 rows of n = 31: 4.8 us at 24
//    lines, 6.4 at 48; 2500 rows of n = 50: 3.6 us at 8, 4.5 at 16).
constexpr int kRowsMaxNtw = 4, kColsMaxNtw = 5;
void dense_shape(bool cols, int n, long nlines, long planes, int *ntw, int *groups) {
    const int units = out_tiles(n), nt = mma_threads(n), warps = nt / 32, full = 768 / nt;
    int       g = units >= warps ? 1 : std::min(4, warps / units), w = 0;
    auto per_sm = [&](int v) { return kMmaSmemMax / (long)(mma_smem(cols, n, 4 * v * g) + 1024); };
    auto padded = [&](int v) { return (nlines + 4L * v * g - 1) / (4L * v * g) * (4L * v * g); };
    for (int v = cols ? kColsMaxNtw : kRowsMaxNtw; v >= 2; v--)
        if (per_sm(v) >= full && (w == 0 || (cols && padded(v) < padded(w)))) w = v;
    if (w == 0) w = per_sm(2) * 3 >= full * 2 ? 2 : 1;
    auto ctas = [&]() { return padded(w) / (4L * w * g) * planes; };
    const long slots = 148L * full;
    while (w > 2 && ctas() * 3 < slots * 2) w--;
    while (g > 1 && ctas() * 3 < slots * 2) g--;
    while (w > 1 && ctas() * 3 < slots) w--;
    *ntw = w;
    *groups = g;
}

template <bool COLS, int NTW, int NT>
int launch_mma(Ctx *c, int n, long nlines, long planes, const double2 *in, long in_ld, long in_plane, double2 *out,
               long out_ld, long out_plane, int groups, const double2 *tab) {
    const int    nl = 4 * NTW * groups;
    const size_t shm = mma_smem(COLS, n, nl);
    HH_TRY(allow_smem(k_dst1_mma<COLS, NTW, NT>, kMmaSmemMax));
    dim3 grid((unsigned)((nlines + nl - 1) / nl), (unsigned)planes);
    return launch_kernel(c, k_dst1_mma<COLS, NTW, NT>, grid, NT, shm, in, out, n, nlines, in_ld, out_ld, in_plane, out_plane,
                                                                 groups, std::sqrt(2.0 / (n + 1)), tab);
}

} // namespace

int dense_for(Ctx *c, int n, const double **mat) {
    std::lock_guard<std::mutex> g(c->mu);
    auto it = c->dense.find(n);
    if (it == c->dense.end()) {
        double *d = nullptr;
        if (n <= kMmaMaxN) {
            HH_CUDA(cudaMalloc(&d, sizeof(double2) * 32 * ((size_t)out_tiles(n) * k4_steps(n) + kTabAhead)));
            k_make_mma<<<256, 256, 0, c->stream>>>(n, reinterpret_cast<double2 *>(d));
        } else {
            HH_CUDA(cudaMalloc(&d, sizeof(double) * (size_t)n * (size_t)n));
            k_make_dense<<<256, 256, 0, c->stream>>>(n, d);
        }
        HH_CUDA(cudaGetLastError());
        c->launches++;
        c->fresh = true;
        c->dense[n] = d;
        it = c->dense.find(n);
    }
    *mat = it->second;
    return HH_OK;
}

int launch_dst_dense(Ctx *c, int n, bool cols, long nlines, long planes, const double2 *in, long in_ld, long in_plane,
                     double2 *out, long out_ld, long out_plane) {
    const double *mat;
    HH_TRY(dense_for(c, n, &mat));
    if (n > kMmaMaxN) {
        const size_t shm = sizeof(double2) * (size_t)n;
        auto         kern = cols ? k_dst1_dense<true> : k_dst1_dense<false>;
        HH_TRY(allow_smem(kern, sizeof(double2) * kDenseMaxN));
        dim3 grid((unsigned)nlines, (unsigned)planes);
        return launch_kernel(c, kern, grid, kDenseThreads, shm, in, out, n, in_ld, out_ld, in_plane, out_plane, mat);
    }
    const double2 *tab = reinterpret_cast<const double2 *>(mat);
    int ntw = 1, groups = 1;
    dense_shape(cols, n, nlines, planes, &ntw, &groups);
    auto pick = [&](auto ntw_c) {
        constexpr int W = decltype(ntw_c)::value;
        auto go = [&](auto launch) {
            return launch(c, n, nlines, planes, in, in_ld, in_plane, out, out_ld, out_plane, groups, tab);
        };
        const bool    small = mma_threads(n) == 128;
        if (cols) return small ? go(launch_mma<true, W, 128>) : go(launch_mma<true, W, 256>);
        if constexpr (W <= kRowsMaxNtw) return small ? go(launch_mma<false, W, 128>) : go(launch_mma<false, W, 256>);
        set_error("DST length %d: no tile shape", n);
        return (int)HH_ERR_UNSUPPORTED;
    };
    switch (ntw) {
    case 1: return pick(std::integral_constant<int, 1>{});
    case 2: return pick(std::integral_constant<int, 2>{});
    case 3: return pick(std::integral_constant<int, 3>{});
    case 4: return pick(std::integral_constant<int, 4>{});
    case 5: return pick(std::integral_constant<int, 5>{});
    }
    set_error("DST length %d: no tile shape", n);
    return HH_ERR_UNSUPPORTED;
}

} // namespace hh
