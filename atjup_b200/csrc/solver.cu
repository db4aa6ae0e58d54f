// Residual-controlled solve of the reference's pressure operator (ATJUP_SOLVE_RESIDUAL).
//
// The reference relaxes  A p = src  with red-black Gauss-Seidel sweeps and never forms a residual
// (PressureSolver.h:318-491). A is the 7-point metric Laplacian over the interior fluid cells
// (i = 1..im-2, j = 1..jm-2, k on the ring of km-1 meridians), faces into the obstacle dropped,
// boundary neighbours read through the 2-point Neumann folds p0 = 4/3 p1 - 1/3 p2 the sweep
// applies after every pass (PressureSolver.h:718-746). Its fixed point is what this solver
// computes, to a stated relative residual ||src - A p|| / ||src||.
//
// A is not symmetric (the folds), but D A is, for D = diag(y), y(i,j,k) = a_i d_j with
// a, d = (3/2, 1, ..., 1, 3/2): y is A's left null vector, so the right-hand side is first made
// compatible by removing its y-component, b <- b - (y.b / y.1) 1. The solve is preconditioned CG
// on -D A with a two-level SPD preconditioner built for this operator's 1e5 anisotropy
// (1/dr^2 = 1600 against 1/(r^2 dtheta^2) ~ 0.013):
//   - radial lines: each (j, k) column's tridiagonal part of A (all horizontal faces on the
//     diagonal) solved exactly -- this removes the radial stiffness;
//   - column modes: the column-constant fields, whose operator V^T (-D A) V is the 2-D horizontal
//     Laplacian d_j (S2 L_theta + S3_j L_phi) of the obstacle-free column sums; solved exactly by a
//     discrete Fourier transform over the meridian ring and one tridiagonal system in theta per
//     wavenumber (the reference's PRESS_BAROTROPIC idea, PressureSolver.h:49-67, 573-708, used
//     here as a preconditioner, so the obstacle need not be obstacle-free).
// Mixed precision: the Krylov vectors, the residual b - A p, the update of p and the column modes
// stay FP64; the preconditioner's radial line solves run in FP32.
//
// An iteration is six launches: A d with alpha; r's update with the line solves; the forward
// transform, the theta systems, the inverse transform with beta; p's update with the next
// direction. The column modes' correction is constant along a column, so it is added where the
// direction reads z, and its share of rho comes from the column sums. Every reduction ends in the
// kernel that forms it.
#include "ctx.cuh"
#include "line_role.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <utility>
#include <vector>

namespace atjup {
namespace {

constexpr int RB = 256;          // threads per reduction block
constexpr int NRED = 592;        // blocks of the flat kernels (4 per SM)
constexpr double kC43 = 4.0 / 3.0, kC13 = 1.0 / 3.0;

// per-cell code: bit 6 a fluid interior cell (an unknown of the system), bits 0-5 the faces of it
// that are not dropped (i+1, i-1, j+1, j-1, k+1, k-1)
enum : uint8_t { F_IP = 1, F_IM = 2, F_JP = 4, F_JM = 8, F_KP = 16, F_KM = 32, F_ON = 64,
                 F_ALL = 127 };

// device scalars of a solve
enum { SC_RHO = 0, SC_ALPHA, SC_BETA, SC_RR, SC_YRZ, SC_YB, SC_BB = 9, SC_RES, SC_MEAN, SC_FLOOR,
       SC_COUNT = 16 };

// Line factors of the preconditioner (-lower / pivot, -upper / pivot, 1 / pivot) in storage T. A column
// without an obstacle cell in it or beside it has the factors of its row: [jm - 2][im - 2] tables.
// The others (the columns that touch the obstacle) have their own, [im - 2][n_irr].
template <typename T>
struct Lines {
    T *ra = nullptr, *rc = nullptr, *rm = nullptr;
    T *ia = nullptr, *ic = nullptr, *im_ = nullptr;
    T* z = nullptr;                                  // the line solves' result
};

struct Solver {
    int NM = 0, N = 0, J = 0, n_irr = 0;
    double *b = nullptr, *p = nullptr, *r = nullptr, *d = nullptr, *q = nullptr;   // Krylov vectors
    Lines<double> l64;
    Lines<float> l32;
    int32_t* slot = nullptr;      // [J * N] irregular columns' index, -1 for the others
    double *g = nullptr, *e = nullptr;               // [J * N] column sums, column corrections
    double* gh = nullptr;         // [J][2][NM + 1] spectra
    double2* cs = nullptr;        // [N] cos, sin of 2 pi n / N
    double* fold = nullptr;       // [(J + 1) * (N + 4)] folded rows (rings too long for shared memory)
    double *tal = nullptr, *tcp = nullptr, *tm = nullptr;   // theta factors [(NM + 1) * J]: -lower /
                                  // pivot, modified upper, 1 / (pivot d_j)
    uint8_t* code = nullptr;      // [NP]
    double* part = nullptr;       // reduction partials, up to three per block
    unsigned* ticket = nullptr;   // blocks done, of the kernel running
    double* scal = nullptr;       // device scalars
    double* hs = nullptr;         // pinned host mirror of scal
    double* yw = nullptr;         // y on fluid interior cells, 0 elsewhere
};

// ---------------------------------------------------------------------------------------------
struct OpC {
    int im, jm, km, KP;
    double n1;
};

__device__ __forceinline__ double y_of(int i, int j, const OpC& q) {
    const double a = (i == 1 || i == q.im - 2) ? 1.5 : 1.0;
    return (j == 1 || j == q.jm - 2) ? a * 1.5 : a;
}

// Sum NV values over the grid in a fixed order: every block writes its partials, the block that
// finishes last adds them (thread-strided, then a tree: the same order whichever block it is).
// True in thread 0 of that block, with the totals in v. One launch in place of a reduction and a
// one-thread kernel that summed 592 partials in sequence (26 us a time, 147 times a solve).
template <int NV>
__device__ bool grid_sum(double (&v)[NV], double* __restrict__ part, unsigned* ticket) {
    __shared__ double sh[NV][32];
    __shared__ bool last;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, nth = blockDim.x * blockDim.y;
    const int nw = nth >> 5, lane = tid & 31, w = tid >> 5;
    const unsigned nblk = gridDim.x * gridDim.y * gridDim.z;
    const unsigned bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    auto block_sum = [&]() {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
            if (lane == 0) sh[q][w] = v[q];
        }
        __syncthreads();
        if (w == 0)
#pragma unroll
            for (int q = 0; q < NV; q++) {
                v[q] = lane < nw ? sh[q][lane] : 0.0;
                for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
            }
    };
    block_sum();
    if (tid == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) part[q * nblk + bid] = v[q];
        __threadfence();
        last = atomicInc(ticket, nblk - 1) == nblk - 1;     // wraps to 0 for the next kernel
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
#pragma unroll
    for (int q = 0; q < NV; q++) {
        v[q] = 0.0;
        for (unsigned n = tid; n < nblk; n += nth) v[q] += __ldcg(part + q * nblk + n);
    }
    block_sum();
    return tid == 0;
}

// On small grids every kernel of an iteration overlaps the tail of the one before (launch_pdl: 2.34 ->
// 2.01 ms a solve on 41x61x97, with the kernels of that time). On large ones blocks started early
// settle on the SMs that happen to drain first, and the uneven spread costs more than the launches
// (5.53 -> 6.00 ms on 41x181x361).
constexpr long SMALL_CELLS = 500000;
// The row kernels work in tiles: a colatitude row's meridians, two neighbouring ones per thread (the
// ring is even, rows start on 128-byte boundaries: 16-byte accesses), marched up a chunk of the
// radial levels, so the radial neighbours stay in registers and no index is divided per cell. A block
// holds as many tiles side by side as fit 512 threads and takes group after group; two blocks per SM
// reduce, since a block's sum, fence and ticket cost more than a tile (592 to 2,685 blocks of one
// tile each: 36 us for A d on the 41x181x361 shell, 13 us on 41x61x97, where reading it takes 4).
constexpr int ROW_T = 512, ROW_BLOCKS = 148 * 2;
struct Rows {
    int per, kb, nt;              // levels per chunk, meridian blocks per row, tiles
    dim3 block;                   // threads of a tile, tiles side by side
    int blocks;                   // of the reducing kernels
    bool small;                   // the kernels overlap the tails of those before them
};
Rows rows_of(const AtjupParams& P) {
    Rows R;
    const int N = P.km - 1, n = P.im - 2, J = P.jm - 2, pairs = N / 2;
    const int th = std::min(ROW_T, (pairs + 31) / 32 * 32), G = ROW_T / th;
    R.block = dim3(th, G);
    R.kb = (pairs + th - 1) / th;
    // the chunk length of the least time: rounds of tiles over all groups x (levels + the two planes
    // beside them)
    long best = -1;
    R.per = 1;
    for (int per = 1; per <= 10; per++) {
        const long nt = (long)R.kb * J * ((n + per - 1) / per);
        const long cost = (nt + (long)ROW_BLOCKS * G - 1) / ((long)ROW_BLOCKS * G) * (per + 2);
        if (best < 0 || cost < best) { best = cost; R.per = per; }
    }
    R.nt = R.kb * J * ((n + R.per - 1) / R.per);
    R.blocks = std::min(ROW_BLOCKS, (R.nt + G - 1) / G);
    R.small = (long)n * J * N < SMALL_CELLS;
    return R;
}
// tile t's meridian block, row and levels
struct Tile { int kb, j, i0, i1; };
__device__ __forceinline__ Tile tile_of(int t, const OpC& q, int kb, int per) {
    const int J = q.jm - 2, u = t / kb, ch = u / J;
    Tile x;
    x.kb = t - u * kb;
    x.j = u - ch * J + 1;
    x.i0 = 1 + ch * per;
    x.i1 = min(q.im - 1, x.i0 + per);
    return x;
}

// q = A d on the unknowns and d . (y A d); the last block forms alpha = rho / that. A sum of weighted
// differences (no cancellation of a large smooth d): a face's weight is its num, 0 where the face is
// dropped; a folded boundary face, num (1/3) (d_c - d_inward), takes num / 3 off the inward face's
// weight. Reads d, writes q and a byte of code per cell (17 B): 21 us on the 41x181x361 shell, bound by
// the latency of the neighbour rows. The form with one flat index (three integer divisions and seven
// mask bytes a cell) took 54 us, one with the edge cells' rows in a function of their own 29 us (their
// calls 12 us, the geometry loads 5).
__device__ __forceinline__ double row_of_A(uint8_t f, double wip, double wim, double wjp, double wjm,
                                           double fi, double fj, bool top, bool bot, bool last,
                                           bool fst, double n3, double xc, double xp, double xm,
                                           double xn, double xs, double xe, double xw) {
    // the fold of a boundary face that is dropped (an obstacle at the wall) goes with it
    double a = (f & F_IP) ? wip : 0.0, b = (f & F_IM) ? wim : 0.0;
    double c = (f & F_JP) ? wjp : 0.0, d = (f & F_JM) ? wjm : 0.0;
    if (top && (f & F_IP)) b -= fi;
    if (bot && (f & F_IM)) a -= fi;
    if (last && (f & F_JP)) d -= fj;
    if (fst && (f & F_JM)) c -= fj;
    return a * (xp - xc) + b * (xm - xc) + c * (xn - xc) + d * (xs - xc) +
           ((f & F_KP) ? n3 : 0.0) * (xe - xc) + ((f & F_KM) ? n3 : 0.0) * (xw - xc);
}

__global__ void __launch_bounds__(ROW_T, 2)
apply_kernel(const double* __restrict__ x, double* __restrict__ y, const uint8_t* __restrict__ code,
             const GeoIJ* __restrict__ geo, OpC q, int kb, int per, int nt, double* __restrict__ part,
             unsigned* ticket, double* __restrict__ scal) {
    const unsigned row = q.KP, plane = (unsigned)q.jm * row;     // every index is below 2^32
    const int N = q.km - 1, lane = threadIdx.x & 31;
    const double n1 = q.n1;
    double acc_dot[1] = {0.0};
    pdl_next();
    pdl_wait();
    for (int t = blockIdx.x * blockDim.y + threadIdx.y; t < nt; t += gridDim.x * blockDim.y) {
        const Tile w_ = tile_of(t, q, kb, per);
        const int j = w_.j, i0 = w_.i0, i1 = w_.i1, kk = 2 * (w_.kb * blockDim.x + threadIdx.x);
        const bool act = kk < N;
        const int k = min(kk, N - 2);
        // the chunk's geometry, a level per lane
        const GeoIJ& g = geo[min(i0 + lane, q.im - 1) * q.jm + j];
        const double g2 = g.num2, g3 = g.num3;
        const bool fst = j == 1, last = j == q.jm - 2;
        unsigned c = (unsigned)i0 * plane + (unsigned)j * row + k;
        const unsigned cr = (unsigned)j * row;                   // the row's k = 0, less the level
        const unsigned kw = k == 0 ? N - 1 : k - 1, ke = k + 2 == N ? 0 : k + 2;
        auto two = [&](unsigned o) { return *reinterpret_cast<const double2*>(x + o); };
        double2 xm = two(c - plane), xc = two(c);
        double dot = 0.0;
#pragma unroll 2
        for (int i = i0; i < i1; i++, c += plane) {
            const double2 xp = two(c + plane), xn = two(c + row), xs = two(c - row);
            const unsigned lev = (unsigned)i * plane + cr;
            const double xw = x[lev + kw], xe = x[lev + ke];
            const uchar2 f = *reinterpret_cast<const uchar2*>(code + c);
            const double n2 = __shfl_sync(0xffffffffu, g2, i - i0), n3 = __shfl_sync(0xffffffffu, g3, i - i0);
            const bool top = i == q.im - 2, bot = i == 1;
            const double fi = kC13 * n1, fj = kC13 * n2;
            const double wip = top ? 0.0 : n1, wim = bot ? 0.0 : n1;
            const double wjp = last ? 0.0 : n2, wjm = fst ? 0.0 : n2;
            double2 a;
            if (f.x == F_ALL && f.y == F_ALL) {
                const double wp = bot ? wip - fi : wip, wm = top ? wim - fi : wim;
                const double wn = fst ? wjp - fj : wjp, ws = last ? wjm - fj : wjm;
                a.x = wp * (xp.x - xc.x) + wm * (xm.x - xc.x) + wn * (xn.x - xc.x) + ws * (xs.x - xc.x) +
                      n3 * (xc.y - xc.x) + n3 * (xw - xc.x);
                a.y = wp * (xp.y - xc.y) + wm * (xm.y - xc.y) + wn * (xn.y - xc.y) + ws * (xs.y - xc.y) +
                      n3 * (xe - xc.y) + n3 * (xc.x - xc.y);
            } else {
                a.x = !f.x ? 0.0 : row_of_A(f.x, wip, wim, wjp, wjm, fi, fj, top, bot, last, fst, n3,
                                            xc.x, xp.x, xm.x, xn.x, xs.x, xc.y, xw);
                a.y = !f.y ? 0.0 : row_of_A(f.y, wip, wim, wjp, wjm, fi, fj, top, bot, last, fst, n3,
                                            xc.y, xp.y, xm.y, xn.y, xs.y, xe, xc.x);
            }
            if (act) {
                *reinterpret_cast<double2*>(y + c) = a;
                const double d = xc.x * a.x + xc.y * a.y;
                dot += (top || bot) ? 1.5 * d : d;
            }
            xm = xc;
            xc = xp;
        }
        acc_dot[0] += (fst || last) ? 1.5 * dot : dot;
    }
    if (grid_sum(acc_dot, part, ticket))
        scal[SC_ALPHA] = (acc_dot[0] != 0.0) ? scal[SC_RHO] / acc_dot[0] : 0.0;
}

// p += alpha d (the direction just used), then the next direction d = z + e + beta d, z + e being
// the preconditioned residual: the line solves' z and the column correction e of its column
// (first: p = 0, d = z + e).
template <typename T>
__global__ void __launch_bounds__(ROW_T)
direction_kernel(double* __restrict__ d, double* __restrict__ p, const T* __restrict__ z,
                 const double* __restrict__ e, const uint8_t* __restrict__ code, OpC q, int kb,
                 int per, int nt, const double* __restrict__ scal, int first) {
    const int t = blockIdx.x * blockDim.y + threadIdx.y;
    const Tile w_ = tile_of(t, q, kb, per);
    const int N = q.km - 1, k = 2 * (w_.kb * blockDim.x + threadIdx.x);
    pdl_next();
    pdl_wait();
    if (t >= nt || k >= N) return;
    const double alpha = scal[SC_ALPHA], beta = scal[SC_BETA];
    const double ex = e[(size_t)(w_.j - 1) * N + k], ey = e[(size_t)(w_.j - 1) * N + k + 1];
    const unsigned plane = (unsigned)q.jm * q.KP;
    unsigned c = (unsigned)w_.i0 * plane + (unsigned)w_.j * q.KP + k;
#pragma unroll 4
    for (int i = w_.i0; i < w_.i1; i++, c += plane) {
        const uchar2 f = *reinterpret_cast<const uchar2*>(code + c);
        double2 *dp = reinterpret_cast<double2*>(d + c), *pp = reinterpret_cast<double2*>(p + c);
        // the line solves' z of cells that are no unknowns is 0, and so are d and p there
        const double zx = f.x ? (double)z[c] + ex : 0.0, zy = f.y ? (double)z[c + 1] + ey : 0.0;
        if (first) {
            *pp = make_double2(0.0, 0.0);
            *dp = make_double2(zx, zy);
        } else {
            const double2 dc = *dp, pc = *pp;
            *pp = make_double2(pc.x + alpha * dc.x, pc.y + alpha * dc.y);
            *dp = make_double2(zx + beta * dc.x, zy + beta * dc.y);
        }
    }
}

// r <- r - mean - alpha q (init: r = b), mean being the y-component dropped at the last check, then
// the radial line solve A_line z = r of each (j, k) column, the column sum g = sum_i y r, and r.r,
// sum y r z, y.r over the grid.
//
// A column's substitutions are first-order recurrences, x_i = al_i x_{i-1} + be_i, so it is split into
// segments of up to LSEG levels, one warp each: a warp loads its levels of 32 columns at once, composes
// its affine map, takes its start value from the maps of the segments before it (shared memory), and
// runs the segment from there; the backward substitution likewise. Everything between the loads of
// r and q and the stores of r and z stays in registers: 32 bytes per cell. On 41x181x361 38 us (76 us
// with one thread per column and the factors as 3-D fields; 29 us that way with row tables, which
// leaves a 41x61x97 shell 177 warps of 39 levels in sequence: 20 us there, 12 us with segments).
// The factors are read as m = 1 / pivot, al = -lower m, c = -upper m.
template <typename T>
struct LineMaps {
    T map[LWARPS][2][32];         // each segment's affine map, per column
    double seg[LWARPS][32];       // its sum of y r
};
// One warp's segment of 32 columns. REG: every column has its row's factors (f: m, al, c of the row
// in shared memory); otherwise the columns have their own, n_irr apart, m = 0 marking a cell that is
// no unknown (r and z stay 0 there, and al = c = 0 end the recurrences).
template <typename T, bool REG>
__device__ __forceinline__ void line_segment(double (&rn)[LSEG], const double (&qq)[LSEG],
                                             double* r, T* z, unsigned o, unsigned plane, int h,
                                             int len, int n, const T* __restrict__ fm,
                                             const T* __restrict__ fa, const T* __restrict__ fc,
                                             unsigned fs, bool act, bool init, double mean,
                                             double alpha, double dj, const LineRole& R, int w,
                                             LineMaps<T>& M, double* g, double (&v)[3]) {
    const int lane = threadIdx.x & 31, s = R.s, S = R.S, w0 = R.w0;
    T x[LSEG], A = 1, B = 0;
    double gs = 0.0, ends = 0.0, rr = 0.0;
    // (read-only loads for the columns' own factors: they may move above the stores to r and z)
    auto f = [&](const T* t, int u) -> T { return REG ? t[u] : __ldg(t + u * fs); };
#pragma unroll
    for (int u = 0; u < LSEG; u++) {
        if (u >= len) break;
        const T m = f(fm, u), al = f(fa, u);
        double rv = init ? rn[u] : (rn[u] - mean) - alpha * qq[u];
        if (!REG && m == (T)0) rv = 0.0;
        if (act && (REG || m != (T)0)) r[o + u * plane] = rv;
        rn[u] = rv;
        rr += rv * rv;
        gs += rv;
        x[u] = (T)rv * m;
        A *= al;
        B = al * B + x[u];
    }
    if (h == 0 && len > 0) ends = rn[0];
#pragma unroll
    for (int u = 0; u < LSEG; u++)
        if (h + u == n - 1 && u < len) ends += rn[u];
    gs = dj * (gs + 0.5 * ends);
    M.map[w][0][lane] = A;
    M.map[w][1][lane] = B;
    M.seg[w][lane] = gs;
    __syncthreads();
    T p = 0;
    for (int e = 0; e < s; e++) p = M.map[w0 + e][0][lane] * p + M.map[w0 + e][1][lane];
    if (s == 0) {
        for (int e = 1; e < S; e++) gs += M.seg[w0 + e][lane];
        if (act) { *g = gs; v[2] += gs; }
    }
    A = 1;
    B = 0;
#pragma unroll
    for (int u = 0; u < LSEG; u++) {
        if (u >= len) break;
        p = f(fa, u) * p + x[u];
        x[u] = p;
    }
#pragma unroll
    for (int u = LSEG - 1; u >= 0; u--) {
        if (u >= len) continue;
        const T c = f(fc, u);
        A *= c;
        B = c * B + x[u];
    }
    __syncthreads();
    M.map[w][0][lane] = A;
    M.map[w][1][lane] = B;
    __syncthreads();
    p = 0;
    for (int e = S - 1; e > s; e--) p = M.map[w0 + e][0][lane] * p + M.map[w0 + e][1][lane];
    double rz = 0.0, rze = 0.0;
#pragma unroll
    for (int u = LSEG - 1; u >= 0; u--) {
        if (u >= len) continue;
        p = x[u] + f(fc, u) * p;
        if (act && (REG || fm[u * fs] != (T)0)) z[o + u * plane] = p;
        const double t = rn[u] * (double)p;
        rz += t;
        if (h + u == 0 || h + u == n - 1) rze += t;
    }
    if (act) {
        v[0] += rr;
        v[1] += dj * (rz + 0.5 * rze);
    }
}

template <typename T, bool INIT>
__global__ void __launch_bounds__(32 * LWARPS, 2)
line_kernel(const double* b, double* r, const double* __restrict__ qv, T* z, Lines<T> L,
            const int32_t* __restrict__ slot, int n_irr, double* __restrict__ g, OpC q, int S,
            double* __restrict__ part, unsigned* ticket, double* __restrict__ scal, double ysum,
            int check) {
    extern __shared__ __align__(16) unsigned char line_smem[];
    __shared__ LineMaps<T> M;
    const int n = q.im - 2, N = q.km - 1, J = q.jm - 2;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, CW = LWARPS / S;
    const LineRole R = line_role(w, S);
    const int kb = (N + 32 * CW - 1) / (32 * CW), h = R.s * LSEG, len = R.on ? min(LSEG, n - h) : 0;
    T* sf = reinterpret_cast<T*>(line_smem);      // the row's factors: m, al, c
    const unsigned plane = (unsigned)q.jm * q.KP;                // every index is below 2^32
    double v[3] = {0.0, 0.0, 0.0};                // r.r, y.(r z), y.r
    pdl_next();
    pdl_wait();
    const double alpha = INIT ? 0.0 : scal[SC_ALPHA], mean = INIT ? 0.0 : scal[SC_MEAN];
    for (int t = blockIdx.x; t < kb * J; t += gridDim.x) {
        // N need not be a multiple of the block's columns: the lanes beyond work on the row's last column
        // and store nothing. A warp without a group (S does not divide LWARPS) has no levels.
        const int j = t / kb + 1, kk = ((t - (j - 1) * kb) * CW + R.group) * 32 + lane;
        const bool act = R.on && kk < N;
        const int k = min(kk, N - 1);
        const unsigned o = plane + (unsigned)j * q.KP + k + (unsigned)h * plane;
        double rn[LSEG], qq[LSEG];
#pragma unroll
        for (int u = 0; u < LSEG; u++)
            if (u < len) {
                rn[u] = INIT ? b[o + u * plane] : r[o + u * plane];
                qq[u] = INIT ? 0.0 : qv[o + u * plane];
            }
        const int sl = R.on ? slot[(size_t)(j - 1) * N + k] : -1;
        __syncthreads();                          // the last tile's factors and maps are read
        for (int i = threadIdx.x; i < 3 * n; i += blockDim.x) {
            const int f = i / n;
            sf[i] = (f == 0 ? L.rm : f == 1 ? L.ra : L.rc)[(size_t)(j - 1) * n + i - f * n];
        }
        // a block whose columns all have the row's factors reads them from shared memory
        const bool irregular = __syncthreads_or(sl >= 0);
        const double dj = (j == 1 || j == q.jm - 2) ? 1.5 : 1.0;
        double* gc = g + (size_t)(j - 1) * N + k;
        if (!irregular) {
            line_segment<T, true>(rn, qq, r, z, o, plane, h, len, n, sf + h, sf + n + h, sf + 2 * n + h,
                                  1, act, INIT, mean, alpha, dj, R, w, M, gc, v);
        } else {
            const size_t ro = (size_t)(j - 1) * n + h;
            const T *m = L.rm + ro, *al = L.ra + ro, *c = L.rc + ro;
            unsigned fs = 1;
            if (sl >= 0) {
                const size_t fo = (size_t)h * n_irr + sl;
                m = L.im_ + fo; al = L.ia + fo; c = L.ic + fo;
                fs = n_irr;
            }
            line_segment<T, false>(rn, qq, r, z, o, plane, h, len, n, m, al, c, fs, act, INIT, mean,
                                   alpha, dj, R, w, M, gc, v);
        }
    }
    if (grid_sum(v, part, ticket)) {
        scal[SC_RR] = v[0];
        scal[SC_YRZ] = v[1];
        // drop the rounding drift of r out of the range of A (its y-component) at the checks
        scal[SC_MEAN] = check ? v[2] / ysum : 0.0;
    }
}

// The same for columns of more than LSEG LWARPS levels: one thread per column, the forward
// substitution kept in z.
template <typename T, bool INIT>
__global__ void __launch_bounds__(128)
line_long_kernel(const double* b, double* r, const double* __restrict__ qv, T* z, Lines<T> L,
                 const int32_t* __restrict__ slot, int n_irr, double* __restrict__ g, OpC q,
                 double* __restrict__ part, unsigned* ticket, double* __restrict__ scal, double ysum,
                 int check) {
    const int n = q.im - 2, N = q.km - 1, j = blockIdx.y + 1;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t plane = (size_t)q.jm * q.KP, b0 = (size_t)j * q.KP + k + plane;
    double v[3] = {0.0, 0.0, 0.0};
    pdl_next();
    pdl_wait();
    if (k < N) {
        const double alpha = INIT ? 0.0 : scal[SC_ALPHA], mean = INIT ? 0.0 : scal[SC_MEAN];
        const int sl = slot[(size_t)(j - 1) * N + k];
        const size_t st = sl < 0 ? 1 : n_irr, fo = sl < 0 ? (size_t)(j - 1) * n : (size_t)sl;
        const T *pm = (sl < 0 ? L.rm : L.im_) + fo, *pa = (sl < 0 ? L.ra : L.ia) + fo;
        const T* pc = (sl < 0 ? L.rc : L.ic) + fo;
        const double dj = (j == 1 || j == q.jm - 2) ? 1.5 : 1.0;
        double gs = 0.0;
        T prev = 0;
        for (int i = 0; i < n; i++) {
            const size_t c = b0 + i * plane;
            const T m = pm[i * st];
            if (m == (T)0) { prev = 0; continue; }
            const double rn = INIT ? b[c] : (r[c] - mean) - alpha * qv[c];
            r[c] = rn;
            v[0] += rn * rn;
            gs += ((i == 0 || i == n - 1) ? 1.5 * dj : dj) * rn;
            prev = (T)rn * m + pa[i * st] * prev;
            z[c] = prev;
        }
        T next = 0;
        for (int i = n - 1; i >= 0; i--) {
            const size_t c = b0 + i * plane;
            if (pm[i * st] == (T)0) { next = 0; continue; }
            next = z[c] + pc[i * st] * next;
            z[c] = next;
            v[1] += ((i == 0 || i == n - 1) ? 1.5 * dj : dj) * r[c] * (double)next;
        }
        g[(size_t)(j - 1) * N + k] = gs;
        v[2] = gs;
    }
    if (grid_sum(v, part, ticket)) {
        scal[SC_RR] = v[0];
        scal[SC_YRZ] = v[1];
        scal[SC_MEAN] = check ? v[2] / ysum : 0.0;
    }
}

// Folded sums of a real ring row for the DFT: with h = N / 2 the cosine of m (N - k) and the sine's
// negative repeat those of m k, and those of m (h - k) are (-1)^m cos and -(-1)^m sin of m k, so a
// quarter of the ring (k = 0 .. h / 2) carries every product: f[par][0] the cosine's, f[par][1] the
// sine's values for wavenumbers m of parity par. K4 = h / 2 + 1 entries each.
__device__ __forceinline__ void fold_row(const double* __restrict__ g, int N, double* f, int K4) {
    const int h = N / 2;
    auto ge = [&](int k) { return (k == 0 || k == h) ? g[k] : g[k] + g[N - k]; };
    auto go = [&](int k) { return (k == 0 || k == h) ? 0.0 : g[k] - g[N - k]; };
    for (int k = threadIdx.x; k < K4; k += blockDim.x) {
        const bool mid = 2 * k == h;
        const double e1 = ge(k), o1 = go(k), e2 = mid ? 0.0 : ge(h - k), o2 = mid ? 0.0 : go(h - k);
        f[k] = e1 + e2;
        f[K4 + k] = mid ? 0.0 : o1 - o2;
        f[2 * K4 + k] = mid ? 0.0 : e1 - e2;
        f[3 * K4 + k] = o1 + o2;
    }
}

// The cosine and sine table, in shared memory while it fits, with one entry of padding after every
// eight (16 bytes each): the threads of a warp read it at a common stride, and a stride of 8
// entries would meet one bank group only.
__device__ __forceinline__ int tab_at(int n) { return n + (n >> 3); }
constexpr int DFT_ROWS = 2;      // rows per block: the table is read once for both

// A block's table and its rows' DFT_ROWS x (N + 4) values
__device__ __forceinline__ double2* dft_tables(const double2* cs, double* fold_g, int N, int use_sm,
                                               unsigned char* smem, double** fold) {
    if (!use_sm) {
        *fold = fold_g + (size_t)blockIdx.x * DFT_ROWS * (N + 4);
        return nullptr;
    }
    double2* t = reinterpret_cast<double2*>(smem);
    for (int k = threadIdx.x; k < N; k += blockDim.x) t[tab_at(k)] = cs[k];
    *fold = reinterpret_cast<double*>(t + tab_at(N));
    return t;
}

// Forward real DFT of the column sums over the ring, a block per two rows: gh[jj][0][m] = sum_k g
// cos, gh[jj][1][m] = sum_k g sin. Half the threads take the even wavenumbers, half the odd ones,
// each running over the quarter of the ring that the folds leave (a quarter of the products of the
// plain sums, which read 1 MB of tables uncoalesced: 91 us; inverse 125 us).
__global__ void dft_fwd_kernel(const double* __restrict__ g, const double2* __restrict__ cs,
                               double* __restrict__ fold_g, double* __restrict__ gh, int N, int NM,
                               int J, int use_sm) {
    extern __shared__ __align__(16) unsigned char dft_smem[];
    const int K4 = N / 4 + 1, j0 = blockIdx.x * DFT_ROWS, H = blockDim.x >> 1, nf = N + 4;
    const bool two = j0 + 1 < J;
    double* f;
    const double2* tab = dft_tables(cs, fold_g, N, use_sm, dft_smem, &f);
    pdl_next();
    pdl_wait();
    fold_row(g + (size_t)j0 * N, N, f, K4);
    fold_row(g + (size_t)(two ? j0 + 1 : j0) * N, N, f + nf, K4);
    __syncthreads();
    const int par = threadIdx.x >= H, t0 = threadIdx.x - par * H;
    const double *fe = f + 2 * par * K4, *fo = fe + K4;
    for (int m = 2 * t0 + par; m <= NM; m += 2 * H) {
        double a = 0.0, b = 0.0, a2 = 0.0, b2 = 0.0;
        int idx = 0;
#pragma unroll 4
        for (int k = 0; k < K4; k++) {
            const double2 w = tab ? tab[tab_at(idx)] : cs[idx];
            a += fe[k] * w.x;
            b += fo[k] * w.y;
            a2 += fe[nf + k] * w.x;
            b2 += fo[nf + k] * w.y;
            idx += m;
            if (idx >= N) idx -= N;
        }
        double* o = gh + (size_t)j0 * 2 * (NM + 1) + m;
        o[0] = a;
        o[NM + 1] = b;
        if (two) { o[2 * (NM + 1)] = a2; o[3 * (NM + 1)] = b2; }
    }
}

// Per wavenumber, one warp for the cosine and sine parts: d_j (S2 L_theta - S3_j lam_m) e = g_hat
// with folded ends, by its tridiagonal factors (mode 0: row 1 pinned, its incompatible part dropped
// first; its sine part and the last mode's are 0). Both substitutions are first-order recurrences
// x_j = al_j x_{j-1} + be_j, so each lane runs its own stretch of rows, the lanes' affine maps are
// composed by a warp scan, and the stretch is run again from its start value: 2 x 2 J / 32 steps and
// ten shuffles in place of 2 J dependent steps on one thread (211 us a solve on 179 rows). The rows
// and factors are staged in shared memory (in place when they do not fit: use_sm 0).
constexpr int TW = 4;            // warps (wavenumbers) per block: a 32-byte sector of a spectrum row
__global__ void __launch_bounds__(32 * TW)
theta_solve_kernel(double* __restrict__ gh, const double* __restrict__ tal,
                   const double* __restrict__ tcp, const double* __restrict__ tm, int NM, int J,
                   int N, int use_sm) {
    extern __shared__ __align__(16) unsigned char theta_smem[];
    const int m = blockIdx.x * TW + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    pdl_next();
    if (m > NM) return;
    const int M1 = NM + 1;
    double* const eg = gh + m;                    // row jj: cosine at 2 jj M1, sine at (2 jj + 1) M1
    const double *al = tal + (size_t)m * J, *cp = tcp + (size_t)m * J, *mm = tm + (size_t)m * J;
    double *e = eg, *e2 = eg + M1;
    int es = 2 * M1;
    if (use_sm) {
        double* s = reinterpret_cast<double*>(theta_smem) + (size_t)(threadIdx.x >> 5) * 5 * J;
#pragma unroll 4
        for (int jj = lane; jj < J; jj += 32) { s[2 * J + jj] = al[jj]; s[3 * J + jj] = cp[jj]; s[4 * J + jj] = mm[jj]; }
        e = s; e2 = s + J; al = s + 2 * J; cp = s + 3 * J; mm = s + 4 * J;
        es = 1;
    }
    pdl_wait();
    if (use_sm)
#pragma unroll 4
        for (int jj = lane; jj < J; jj += 32) {
            e[jj] = eg[(size_t)jj * 2 * M1];
            e2[jj] = eg[(size_t)(2 * jj + 1) * M1];
        }
    __syncwarp();
    double mean0 = 0.0;
    const bool zero2 = m == 0 || 2 * m == N;
    if (m == 0) {
        double sg = 0.0;
        for (int jj = lane; jj < J; jj += 32) sg += e[(size_t)jj * es];
        for (int o = 16; o > 0; o >>= 1) sg += __shfl_xor_sync(0xffffffffu, sg, o);
        mean0 = sg / J;
    }
    const int R = (J + 31) / 32, lo = min(J, lane * R), hi = min(J, lo + R);
    // mm carries the row's 1 / d_j, and 0 for the pinned gauge row
    auto beta = [&](const double* x, int jj, double mean) { return (x[(size_t)jj * es] - mean) * mm[jj]; };
    double A = 1.0, B = 0.0, C = 0.0;
    for (int jj = lo; jj < hi; jj++) {
        const double a = al[jj];
        A *= a;
        B = a * B + beta(e, jj, mean0);
        C = a * C + beta(e2, jj, 0.0);
    }
    for (int o = 1; o < 32; o <<= 1) {
        const double Ap = __shfl_up_sync(0xffffffffu, A, o), Bp = __shfl_up_sync(0xffffffffu, B, o);
        const double Cp = __shfl_up_sync(0xffffffffu, C, o);
        if (lane >= o) { B = A * Bp + B; C = A * Cp + C; A *= Ap; }
    }
    double x = __shfl_up_sync(0xffffffffu, B, 1), y = __shfl_up_sync(0xffffffffu, C, 1);
    if (lane == 0) x = y = 0.0;
    for (int jj = lo; jj < hi; jj++) {
        const double a = al[jj];
        x = a * x + beta(e, jj, mean0);
        y = a * y + beta(e2, jj, 0.0);
        e[(size_t)jj * es] = x;
        e2[(size_t)jj * es] = y;
    }
    A = 1.0;
    B = C = 0.0;
    for (int jj = hi - 1; jj >= lo; jj--) {
        const double a = -cp[jj];
        A *= a;
        B = a * B + e[(size_t)jj * es];
        C = a * C + e2[(size_t)jj * es];
    }
    for (int o = 1; o < 32; o <<= 1) {
        const double Ap = __shfl_down_sync(0xffffffffu, A, o), Bp = __shfl_down_sync(0xffffffffu, B, o);
        const double Cp = __shfl_down_sync(0xffffffffu, C, o);
        if (lane + o < 32) { B = A * Bp + B; C = A * Cp + C; A *= Ap; }
    }
    x = __shfl_down_sync(0xffffffffu, B, 1);
    y = __shfl_down_sync(0xffffffffu, C, 1);
    if (lane == 31) x = y = 0.0;
    for (int jj = hi - 1; jj >= lo; jj--) {
        x = e[(size_t)jj * es] - cp[jj] * x;
        y = e2[(size_t)jj * es] - cp[jj] * y;
        e[(size_t)jj * es] = x;
        e2[(size_t)jj * es] = zero2 ? 0.0 : y;
    }
    if (use_sm) {
        __syncwarp();
        for (int jj = lane; jj < J; jj += 32) {
            eg[(size_t)jj * 2 * M1] = e[jj];
            eg[(size_t)(2 * jj + 1) * M1] = e2[jj];
        }
    }
}

// Inverse DFT into the column corrections e, a block per two rows, and rho = sum y r (z + e): the
// correction is constant along a column, so its part is sum over the columns of e g, and the line
// kernel has summed y r z. The last block forms beta = rho / rho_old (first: rho alone). Thread k
// of each half runs over the wavenumbers of one parity for the quarter k = 0 .. h / 2; the four
// meridians k, N - k, h - k, h + k are sums and differences of the halves.
__global__ void dft_inv_kernel(const double* __restrict__ gh, const double2* __restrict__ cs,
                               double* __restrict__ fold_g, double* __restrict__ e,
                               const double* __restrict__ g, int N, int NM, int J, int use_sm,
                               double* __restrict__ part, unsigned* ticket,
                               double* __restrict__ scal, int first) {
    extern __shared__ __align__(16) unsigned char dft_smem[];
    const int K4 = N / 4 + 1, j0 = blockIdx.x * DFT_ROWS, H = blockDim.x >> 1, h = N / 2, nf = N + 4;
    const int rows = j0 + 1 < J ? 2 : 1;
    const double inv_N = 1.0 / N;
    double* co;                                  // the rows' coefficients, cosine and sine side by side
    const double2* tab = dft_tables(cs, fold_g, N, use_sm, dft_smem, &co);
    pdl_next();
    pdl_wait();
    for (int m = threadIdx.x; m <= NM; m += blockDim.x) {
        const bool end = m == 0 || 2 * m == N;
        const double* o = gh + (size_t)j0 * 2 * (NM + 1) + m;
        for (int r = 0; r < rows; r++, o += 2 * (NM + 1)) {
            co[r * nf + 2 * m] = (end ? 1.0 : 2.0) * inv_N * o[0];
            co[r * nf + 2 * m + 1] = end ? 0.0 : 2.0 * inv_N * o[NM + 1];
        }
        if (rows == 1) co[nf + 2 * m] = co[nf + 2 * m + 1] = 0.0;
    }
    __syncthreads();
    const int par = threadIdx.x >= H, t0 = threadIdx.x - par * H;
    __shared__ double4 odd[512];
    double v[1] = {0.0};
    for (int kb = 0; kb < K4; kb += H) {
        const int k = kb + t0;
        double a = 0.0, b = 0.0, a2 = 0.0, b2 = 0.0;
        if (k < K4) {
            int idx = par ? k : 0;
            const int step = 2 * k >= N ? 2 * k - N : 2 * k;
#pragma unroll 4
            for (int m = par; m <= NM; m += 2) {
                const double2 w = tab ? tab[tab_at(idx)] : cs[idx];
                a += co[2 * m] * w.x;
                b += co[2 * m + 1] * w.y;
                a2 += co[nf + 2 * m] * w.x;
                b2 += co[nf + 2 * m + 1] * w.y;
                idx += step;
                if (idx >= N) idx -= N;
            }
        }
        if (par) odd[t0] = make_double4(a, b, a2, b2);
        __syncthreads();
        if (!par && k < K4) {
            const double4 o = odd[t0];
            auto put4 = [&](int jj, double a, double b, double ox, double oy) {
                const double* gr = g + (size_t)jj * N;
                double* er = e + (size_t)jj * N;
                auto put = [&](int kk, double x) { er[kk] = x; v[0] += x * gr[kk]; };
                put(k, (a + ox) + (b + oy));
                if (k > 0) put(N - k, (a + ox) - (b + oy));
                if (2 * k != h) {
                    put(h - k, (a - ox) - (b - oy));
                    if (k > 0) put(h + k, (a - ox) + (b - oy));
                }
            };
            put4(j0, a, b, o.x, o.y);
            if (rows == 2) put4(j0 + 1, a2, b2, o.z, o.w);
        }
        __syncthreads();
    }
    if (grid_sum(v, part, ticket)) {
        const double rho = scal[SC_YRZ] + v[0], old = scal[SC_RHO];
        if (!first) scal[SC_BETA] = (old != 0.0) ? rho / old : 0.0;
        scal[SC_RHO] = rho;
    }
}

// p64 += e64
__global__ void add_kernel(double* __restrict__ p, const double* __restrict__ e, size_t n) {
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (size_t)gridDim.x * blockDim.x)
        p[c] += e[c];
}

// r = b - A p in FP64 on the unknowns, with the sums of r^2 and of v^2, v = |A| |p|: eps * ||v|| is
// the rounding floor of the residual of an FP64 p (one ulp of p moves it that much).
__global__ void __launch_bounds__(ROW_T, 2)
residual_kernel(const double* __restrict__ b, const double* __restrict__ x, double* __restrict__ r,
                const uint8_t* __restrict__ code, const GeoIJ* __restrict__ geo, OpC q, int kb,
                int per, int nt, double* __restrict__ part, unsigned* ticket,
                double* __restrict__ scal) {
    const size_t row = q.KP, plane = (size_t)q.jm * row;
    const int N = q.km - 1;
    double acc[2] = {0.0, 0.0};
    for (int tl = blockIdx.x * blockDim.y + threadIdx.y; tl < nt; tl += gridDim.x * blockDim.y) {
        const Tile w_ = tile_of(tl, q, kb, per);
        const int j = w_.j, i0 = w_.i0, i1 = w_.i1;
        for (int k = w_.kb * 2 * blockDim.x + threadIdx.x; k < min(N, (w_.kb + 1) * 2 * (int)blockDim.x); k += blockDim.x) {
        const int dw = (k == 0) ? N - 1 : -1, de = (k == N - 1) ? 1 - N : 1;
        size_t c = (size_t)i0 * plane + (size_t)j * row + k;
        double xm = x[c - plane], xc = x[c];
        for (int i = i0; i < i1; i++, c += plane) {
            const double xp = x[c + plane], xn = x[c + row], xs = x[c - row];
            const double xe = x[c + de], xw = x[c + dw], bc = b[c];
            const uint8_t f = code[c];
            if (f & F_ON) {
                const GeoIJ& g = geo[i * q.jm + j];
                const double n1 = q.n1, n2 = g.num2, n3 = g.num3;
                double t[6] = {0, 0, 0, 0, 0, 0};
                // (|A| |x|)_c: the terms whose rounding bounds the residual of an FP64 x
                double den = 0.0, nb = 0.0;
                auto face = [&](int s, bool on, bool folded, double w, double out, double in) {
                    if (!on) return;
                    t[s] = folded ? w * kC13 * (xc - in) : w * (out - xc);
                    const double ww = folded ? w * kC13 : w;
                    den += ww;
                    nb += ww * fabs(folded ? in : out);
                };
                face(0, f & F_IP, i + 1 == q.im - 1, n1, xp, xm);
                face(1, f & F_IM, i - 1 == 0, n1, xm, xp);
                face(2, f & F_JP, j + 1 == q.jm - 1, n2, xn, xs);
                face(3, f & F_JM, j - 1 == 0, n2, xs, xn);
                face(4, f & F_KP, false, n3, xe, 0.0);
                face(5, f & F_KM, false, n3, xw, 0.0);
                const double ax = ((t[0] + t[1]) + (t[2] + t[3])) + (t[4] + t[5]);
                const double v = den * fabs(xc) + nb, out = bc - ax;
                acc[0] += out * out;
                acc[1] += v * v;
                r[c] = out;
            }
            xm = xc;
            xc = xp;
        }
        }
    }
    if (grid_sum(acc, part, ticket)) {
        scal[SC_RES] = acc[0];
        scal[SC_FLOOR] = acc[1];
    }
}

// One colour of point red-black SOR on A x = b (the same folded operator as apply_kernel and
// residual_kernel): x_c <- x_c + omega ((b_c - sum_off a_cf x_f) / a_cc - x_c) for the fluid
// interior cells with (i + j + k) % 2 == colour. A folded boundary face contributes +w/3 to a_cc
// and -w/3 to the inward neighbour's coefficient; a plain face -w to a_cc and +w to the
// neighbour's. Within one colour every cell reads only cells of the other colour (the phi ring
// has an even number of meridians), so the parallel pass equals the sequential one.
__global__ void __launch_bounds__(RB)
sor_kernel(const double* __restrict__ b, double* __restrict__ x, const uint8_t* __restrict__ s,
           const GeoIJ* __restrict__ geo, const double* __restrict__ yw, OpC q, int colour,
           double omega) {
    const size_t plane = (size_t)q.jm * q.KP, row = q.KP;
    const size_t NP = (size_t)q.im * plane;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < NP;
         c += (size_t)gridDim.x * blockDim.x) {
        if (!(yw[c] > 0.0)) continue;
        const int k = (int)(c % row);
        const int j = (int)((c / row) % q.jm);
        const int i = (int)(c / plane);
        if (((i + j + k) & 1) != colour) continue;
        const GeoIJ& g = geo[i * q.jm + j];
        const double n1 = q.n1, n2 = g.num2, n3 = g.num3;
        const int kw = (k == 0) ? q.km - 2 : k - 1;
        const int ke = (k == q.km - 2) ? 0 : k + 1;
        double diag = 0.0, off = 0.0;
        if (!s[c + plane]) {
            if (i + 1 == q.im - 1) { diag += n1 * kC13; off -= n1 * kC13 * x[c - plane]; }
            else { diag -= n1; off += n1 * x[c + plane]; }
        }
        if (!s[c - plane]) {
            if (i - 1 == 0) { diag += n1 * kC13; off -= n1 * kC13 * x[c + plane]; }
            else { diag -= n1; off += n1 * x[c - plane]; }
        }
        if (!s[c + row]) {
            if (j + 1 == q.jm - 1) { diag += n2 * kC13; off -= n2 * kC13 * x[c - row]; }
            else { diag -= n2; off += n2 * x[c + row]; }
        }
        if (!s[c - row]) {
            if (j - 1 == 0) { diag += n2 * kC13; off -= n2 * kC13 * x[c + row]; }
            else { diag -= n2; off += n2 * x[c - row]; }
        }
        if (!s[c - k + ke]) { diag -= n3; off += n3 * x[c - k + ke]; }
        if (!s[c - k + kw]) { diag -= n3; off += n3 * x[c - k + kw]; }
        if (diag == 0.0) continue;
        const double xc = x[c];
        x[c] = xc + omega * ((b[c] - off) / diag - xc);
    }
}

// b (masked copy of the source or the external right-hand side), p (masked warm start), and y.b
__global__ void __launch_bounds__(RB)
gather_kernel(const double* __restrict__ src, const double* __restrict__ p_dyn,
              const double* __restrict__ yw, double* __restrict__ b, double* __restrict__ p,
              size_t n, int warm, double* __restrict__ part, unsigned* ticket,
              double* __restrict__ scal) {
    double v[1] = {0.0};
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (size_t)gridDim.x * blockDim.x) {
        const double w = yw[c];
        const bool f = w > 0.0;
        const double bc = f ? src[c] : 0.0;
        b[c] = bc;
        p[c] = (f && warm) ? p_dyn[c] : 0.0;
        v[0] += w * bc;
    }
    if (grid_sum(v, part, ticket)) scal[SC_YB] = v[0];
}

// b -= (y.b / y.1) on the unknowns, and b.b
__global__ void __launch_bounds__(RB)
project_kernel(double* __restrict__ b, const double* __restrict__ yw, double* scal, double ysum,
               size_t n, double* __restrict__ part, unsigned* ticket) {
    const double mean = scal[SC_YB] / ysum;
    double v[1] = {0.0};
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (size_t)gridDim.x * blockDim.x)
        if (yw[c] > 0.0) {
            const double bc = b[c] - mean;
            b[c] = bc;
            v[0] += bc * bc;
        }
    if (grid_sum(v, part, ticket)) scal[SC_BB] = v[0];
}

// y.p
__global__ void __launch_bounds__(RB)
gauge_kernel(const double* __restrict__ p, const double* __restrict__ yw, size_t n,
             double* __restrict__ part, unsigned* ticket, double* __restrict__ scal) {
    double v[1] = {0.0};
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (size_t)gridDim.x * blockDim.x)
        v[0] += yw[c] * p[c];
    if (grid_sum(v, part, ticket)) scal[SC_YB] = v[0];
}

// p_dyn = p on fluid interior cells, with the y-weighted mean removed when `gauge`
__global__ void scatter_kernel(const double* __restrict__ p, const double* __restrict__ yw,
                               double* __restrict__ p_dyn, const double* __restrict__ scal,
                               double ysum, size_t n, int gauge) {
    const double mean = gauge ? scal[SC_YB] / ysum : 0.0;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
         c += (size_t)gridDim.x * blockDim.x)
        if (yw[c] > 0.0) p_dyn[c] = p[c] - mean;
}

// the per-cell code and y from the mask
__global__ void code_kernel(const uint8_t* __restrict__ s, uint8_t* __restrict__ code,
                            double* __restrict__ yw, OpC q) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    if (k >= q.KP) return;
    const size_t row = q.KP, plane = (size_t)q.jm * row;
    const size_t c = (size_t)i * plane + (size_t)j * row + k;
    uint8_t f = 0;
    if (i >= 1 && i <= q.im - 2 && j >= 1 && j <= q.jm - 2 && k <= q.km - 2 && !s[c]) {
        const int kw = (k == 0) ? q.km - 2 : k - 1, ke = (k == q.km - 2) ? 0 : k + 1;
        f = F_ON;
        if (!s[c + plane]) f |= F_IP;
        if (!s[c - plane]) f |= F_IM;
        if (!s[c + row]) f |= F_JP;
        if (!s[c - row]) f |= F_JM;
        if (!s[c - k + ke]) f |= F_KP;
        if (!s[c - k + kw]) f |= F_KM;
    }
    code[c] = f;
    yw[c] = f ? y_of(i, j, q) : 0.0;
}

// ---------------------------------------------------------------------------------------------
template <typename T>
int alloc_zero(T** p, size_t n) {
    ATJUP_CUDA(cudaMalloc(p, sizeof(T) * std::max<size_t>(n, 1)));
    ATJUP_CUDA(cudaMemset(*p, 0, sizeof(T) * std::max<size_t>(n, 1)));
    return ATJUP_OK;
}

template <typename T>
int upload_as(T** dst, const std::vector<double>& src) {
    std::vector<T> h(src.begin(), src.end());
    ATJUP_CUDA(cudaMalloc(dst, sizeof(T) * std::max<size_t>(h.size(), 1)));
    if (!h.empty()) ATJUP_CUDA(cudaMemcpy(*dst, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
    return ATJUP_OK;
}

template <typename T>
void free_lines(Lines<T>& l) {
    T* all[] = {l.ra, l.rc, l.rm, l.ia, l.ic, l.im_, l.z};
    for (T* p : all) cudaFree(p);
    l = Lines<T>();
}

// Dynamic shared memory of the DFT kernels (tables and folds), 0 when the ring is too long for it. With the
// kernels' own (17 KB in the inverse) it exceeds a launch's default 48 KB from 954 meridians on, so both
// are allowed DFT_SMEM whatever the ring: a limit set to one ring's need would also be the one left for
// another context with a longer ring.
constexpr size_t DFT_SMEM = 200 * 1024;
size_t dft_bytes(int N) {
    const size_t b = sizeof(double2) * (size_t)(N + N / 8 + 1) + sizeof(double) * DFT_ROWS * ((size_t)N + 4);
    return b <= DFT_SMEM ? b : 0;
}

// Build y, the cell codes, the line factors and the coarse (column-mode) factors from the mask and
// geometry.
int setup(AtjupCtx* c, Solver* S) {
    const AtjupParams& P = c->P;
    const int im = P.im, jm = P.jm, km = P.km, KP = c->KP;
    const size_t NP = c->NP;
    S->N = km - 1;
    S->NM = S->N / 2;
    S->J = jm - 2;
    const int N = S->N, NM = S->NM, J = S->J, n = im - 2;
    std::vector<uint8_t> s(NP);
    ATJUP_CUDA(cudaMemcpy(s.data(), c->solid, NP, cudaMemcpyDeviceToHost));
    std::vector<GeoIJ> geo((size_t)im * jm);
    ATJUP_CUDA(cudaMemcpy(geo.data(), c->geo, sizeof(GeoIJ) * geo.size(), cudaMemcpyDeviceToHost));
    const double n1 = 1.0 / (P.dr * P.dr);
    auto at = [&](int i, int j, int k) { return ((size_t)i * jm + j) * KP + k; };
    // columns that hold a solid cell at any level, walls included
    std::vector<uint8_t> hit((size_t)jm * km, 0);
    for (int i = 0; i < im; i++)
        for (int j = 0; j < jm; j++) {
            const uint8_t* row = &s[at(i, j, 0)];
            uint8_t* h = &hit[(size_t)j * km];
            for (int k = 0; k < km; k++) h[k] |= row[k];
        }
    double ysum = 0.0;
    for (int j = 1; j <= jm - 2; j++)
        for (int k = 0; k < N; k++) {
            const double d = (j == 1 || j == jm - 2) ? 1.5 : 1.0;
            if (!hit[(size_t)j * km + k]) { ysum += d * (n - 2 + 3.0); continue; }
            for (int i = 1; i <= im - 2; i++)
                if (!s[at(i, j, k)]) ysum += ((i == 1 || i == im - 2) ? 1.5 : 1.0) * d;
        }
    // Radial tridiagonal of A of one column: rows = unknowns; diagonal = -(sum of kept faces) plus
    // the fold terms; off-diagonals num1 (fold-modified at i = 1, im-2). `solid(i, j, k)` is the
    // mask the column sees.
    auto column = [&](int j, auto solid, double* la, double* lc, double* lm, size_t st) {
        double cprev = 0.0;
        bool prev_fluid = false;
        for (int i = 1; i <= im - 2; i++) {
            const size_t o = (size_t)(i - 1) * st;
            la[o] = lc[o] = lm[o] = 0.0;
            if (solid(i, 0, 0)) { prev_fluid = false; continue; }
            const GeoIJ& g = geo[(size_t)i * jm + j];
            double den = 0.0, diag = 0.0, lower = 0.0, upper = 0.0;
            if (!solid(i + 1, 0, 0)) {
                den += n1;
                if (i + 1 == im - 1) { diag += n1 * kC43; lower += -n1 * kC13; }
                else upper += n1;
            }
            if (!solid(i - 1, 0, 0)) {
                den += n1;
                if (i - 1 == 0) { diag += n1 * kC43; upper += -n1 * kC13; }
                else lower += n1;
            }
            if (!solid(i, 1, 0)) { den += g.num2; if (j + 1 == jm - 1) diag += g.num2 * kC43; }
            if (!solid(i, -1, 0)) { den += g.num2; if (j - 1 == 0) diag += g.num2 * kC43; }
            if (!solid(i, 0, 1)) den += g.num3;
            if (!solid(i, 0, -1)) den += g.num3;
            diag -= den;
            // neighbours outside the run (solid) carry no coupling
            if (!prev_fluid) lower = 0.0;
            if (i + 1 > im - 2 || solid(i + 1, 0, 0)) upper = 0.0;
            const double m = 1.0 / (diag - lower * cprev);
            la[o] = -lower * m;
            lm[o] = m;
            cprev = upper * m;
            lc[o] = -cprev;
            prev_fluid = true;
        }
    };
    std::vector<double> ra((size_t)J * n), rc((size_t)J * n), rm((size_t)J * n);
    std::vector<int32_t> slot((size_t)J * N, -1);
    std::vector<std::pair<int, int>> irr;
    for (int j = 1; j <= jm - 2; j++) {
        const size_t o = (size_t)(j - 1) * n;
        column(j, [](int, int, int) { return false; }, &ra[o], &rc[o], &rm[o], 1);
        for (int k = 0; k < N; k++) {
            const int kw = (k == 0) ? km - 2 : k - 1, ke = (k == km - 2) ? 0 : k + 1;
            if (hit[(size_t)j * km + k] | hit[(size_t)(j + 1) * km + k] | hit[(size_t)(j - 1) * km + k] |
                hit[(size_t)j * km + ke] | hit[(size_t)j * km + kw]) {
                slot[(size_t)(j - 1) * N + k] = (int32_t)irr.size();
                irr.emplace_back(j, k);
            }
        }
    }
    S->n_irr = (int)irr.size();
    std::vector<double> ia(irr.size() * n), ic(irr.size() * n), imv(irr.size() * n);
    for (size_t q = 0; q < irr.size(); q++) {
        const int j = irr[q].first, k = irr[q].second;
        column(j, [&](int i, int dj, int dk) {
            const int kk = dk == 0 ? k : dk > 0 ? ((k == km - 2) ? 0 : k + 1) : ((k == 0) ? km - 2 : k - 1);
            return s[at(i, j + dj, kk)] != 0;
        }, &ia[q], &ic[q], &imv[q], irr.size());
    }
    // coarse: S2 = sum_i a_i num2_i, S3_j = sum_i a_i num3_ij (obstacle-free column sums)
    std::vector<double> S3d(jm, 0.0);
    double S2 = 0.0;
    for (int i = 1; i <= im - 2; i++) {
        const double a = (i == 1 || i == im - 2) ? 1.5 : 1.0;
        S2 += a * geo[(size_t)i * jm + 1].num2;
        for (int j = 1; j <= jm - 2; j++) S3d[j] += a * geo[(size_t)i * jm + j].num3;
    }
    std::vector<double2> cs(N);
    for (int k = 0; k < N; k++) cs[k] = make_double2(std::cos(2.0 * M_PI * k / N), std::sin(2.0 * M_PI * k / N));
    // per wavenumber: rows jj = 0..J-1 (j = jj+1): S2 (e[j+1] + e[j-1] - 2 e[j]) - S3_j lam e[j],
    // folded at both ends (e[0] = 4/3 e[1] - 1/3 e[2]); mode 0: row 0 replaced by e[0] = 0
    std::vector<double> tal((size_t)(NM + 1) * J), tcp((size_t)(NM + 1) * J), tm((size_t)(NM + 1) * J);
    for (int m = 0; m <= NM; m++) {
        const double sl = std::sin(M_PI * m / N);
        const double lam = 4.0 * sl * sl;       // S3_j already carries 1 / dphi^2
        double cprev = 0.0;
        for (int jj = 0; jj < J; jj++) {
            const int j = jj + 1;
            double a = S2, b = -2.0 * S2 - S3d[j] * lam, cu = S2;
            if (jj == 0) { b += kC43 * S2; cu -= kC13 * S2; a = 0.0; }
            if (jj == J - 1) { b += kC43 * S2; a -= kC13 * S2; cu = 0.0; }
            if (m == 0 && jj == 0) { a = 0.0; b = 1.0; cu = 0.0; }
            const double mm = 1.0 / (b - a * cprev);
            tal[(size_t)m * J + jj] = -a * mm;
            tm[(size_t)m * J + jj] = (m == 0 && jj == 0) ? 0.0 : (jj == 0 || jj == J - 1) ? mm / 1.5 : mm;
            tcp[(size_t)m * J + jj] = cprev = cu * mm;
        }
    }
    int rc_;
    for (double** v : {&S->b, &S->p, &S->r, &S->d, &S->q, &S->l64.z})
        if ((rc_ = alloc_zero(v, NP))) return rc_;
    if ((rc_ = alloc_zero(&S->l32.z, NP)) || (rc_ = alloc_zero(&S->g, (size_t)J * N)) ||
        (rc_ = alloc_zero(&S->e, (size_t)J * N)) ||
        (rc_ = alloc_zero(&S->gh, 2 * (size_t)(NM + 1) * J)) ||
        (rc_ = alloc_zero(&S->part, 3 * std::max<size_t>({(size_t)NRED, (size_t)J * ((N + 31) / 32),
                                                          (size_t)ROW_BLOCKS}))) || (rc_ = alloc_zero(&S->ticket, 1)) ||
        (rc_ = alloc_zero(&S->scal, SC_COUNT)) || (rc_ = alloc_zero(&S->yw, NP)) ||
        (rc_ = alloc_zero(&S->code, NP)))
        return rc_;
    ATJUP_CUDA(cudaFuncSetAttribute(dft_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DFT_SMEM));
    ATJUP_CUDA(cudaFuncSetAttribute(dft_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DFT_SMEM));
    if (!dft_bytes(N) && (rc_ = alloc_zero(&S->fold, (size_t)(J + 1) * (N + 4)))) return rc_;
    if ((rc_ = upload_as(&S->l64.ra, ra)) || (rc_ = upload_as(&S->l64.rc, rc)) ||
        (rc_ = upload_as(&S->l64.rm, rm)) || (rc_ = upload_as(&S->l64.ia, ia)) ||
        (rc_ = upload_as(&S->l64.ic, ic)) || (rc_ = upload_as(&S->l64.im_, imv)) ||
        (rc_ = upload_as(&S->l32.ra, ra)) || (rc_ = upload_as(&S->l32.rc, rc)) ||
        (rc_ = upload_as(&S->l32.rm, rm)) || (rc_ = upload_as(&S->l32.ia, ia)) ||
        (rc_ = upload_as(&S->l32.ic, ic)) || (rc_ = upload_as(&S->l32.im_, imv)) ||
        (rc_ = upload_as(&S->tal, tal)) || (rc_ = upload_as(&S->tcp, tcp)) ||
        (rc_ = upload_as(&S->tm, tm)))
        return rc_;
    ATJUP_CUDA(cudaMalloc(&S->slot, sizeof(int32_t) * slot.size()));
    ATJUP_CUDA(cudaMemcpy(S->slot, slot.data(), sizeof(int32_t) * slot.size(), cudaMemcpyHostToDevice));
    ATJUP_CUDA(cudaMalloc(&S->cs, sizeof(double2) * N));
    ATJUP_CUDA(cudaMemcpy(S->cs, cs.data(), sizeof(double2) * N, cudaMemcpyHostToDevice));
    ATJUP_CUDA(cudaMallocHost(&S->hs, sizeof(double) * SC_COUNT));
    const OpC q{im, jm, km, KP, n1};
    code_kernel<<<dim3((KP + 127) / 128, jm, im), 128, 0, c->stream>>>(c->solid, S->code, S->yw, q);
    c->launches++;
    ATJUP_CHECK_LAUNCH("pressure_solve setup");
    ATJUP_CUDA(cudaStreamSynchronize(c->stream));
    c->yw_sum = ysum;
    return ATJUP_OK;
}

Solver* get_solver(AtjupCtx* c) { return reinterpret_cast<Solver*>(c->solver); }

// The preconditioner applied to the residual: the line solves (with r's update), then the column
// modes; leaves z, e and rho, beta (first: rho). INIT starts r from b.
template <typename T, bool INIT>
int precond(AtjupCtx* c, Solver* S, Lines<T>& L, const OpC& q, const Rows& R, int check) {
    cudaStream_t st = c->stream;
    const int N = S->N, J = S->J, NM = S->NM;
    const int n = q.im - 2, segs = (n + LSEG - 1) / LSEG;
    if (segs <= LWARPS) {
        const int cols = 32 * (LWARPS / segs), tiles = (N + cols - 1) / cols * J;
        ATJUP_CUDA(launch_pdl(R.small, line_kernel<T, INIT>, std::min(tiles, ROW_BLOCKS), 32 * LWARPS,
                              sizeof(T) * 3 * n, st, S->b, S->r, S->q, L.z, L, S->slot, S->n_irr, S->g,
                              q, segs, S->part, S->ticket, S->scal, c->yw_sum, check));
    } else {
        const int th = std::min(128, (N + 31) / 32 * 32);
        ATJUP_CUDA(launch_pdl(R.small, line_long_kernel<T, INIT>, dim3((N + th - 1) / th, J), th, 0, st,
                              S->b, S->r, S->q, L.z, L, S->slot, S->n_irr, S->g, q, S->part, S->ticket,
                              S->scal, c->yw_sum, check));
    }
    const size_t sm = dft_bytes(N), tsm = sizeof(double) * 5 * (size_t)J * TW;
    const int H = std::min(512, ((N / 4 + 1) + 31) / 32 * 32), use_sm = sm > 0;
    const int tuse = tsm <= 48 * 1024, first = INIT;
    const dim3 dgrid((J + DFT_ROWS - 1) / DFT_ROWS);
    ATJUP_CUDA(launch_pdl(R.small, dft_fwd_kernel, dgrid, 2 * H, sm, st, S->g, S->cs, S->fold, S->gh, N, NM, J,
                          use_sm));
    ATJUP_CUDA(launch_pdl(R.small, theta_solve_kernel, (NM + 1 + TW - 1) / TW, 32 * TW, tuse ? tsm : 0, st,
                          S->gh, S->tal, S->tcp, S->tm, NM, J, N, tuse));
    ATJUP_CUDA(launch_pdl(R.small, dft_inv_kernel, dgrid, 2 * H, sm, st, S->gh, S->cs, S->fold, S->e, S->g, N, NM,
                          J, use_sm, S->part, S->ticket, S->scal, first));
    c->launches += 4;
    return ATJUP_OK;
}

// One preconditioned CG solve of A x = b (S->b, of norm bnorm), x from zero into S->p, to
// ||r|| <= tol ||b||. The Krylov vectors are FP64; the preconditioner's radial lines run in
// precision T. Returns iterations; *rel = final recursive ||r|| / ||b||.
template <typename T>
int pcg(AtjupCtx* c, Solver* S, Lines<T>& L, double bnorm, double tol, int max_iter, int* iters,
        double* rel) {
    const AtjupParams& P = c->P;
    const OpC q{P.im, P.jm, P.km, c->KP, 1.0 / (P.dr * P.dr)};
    const Rows R = rows_of(P);
    cudaStream_t st = c->stream;
    *iters = 0;
    *rel = 0.0;
    if (bnorm == 0.0) {
        ATJUP_CUDA(cudaMemsetAsync(S->p, 0, sizeof(double) * c->NP, st));
        return ATJUP_OK;
    }
    int rc;
    if ((rc = precond<T, true>(c, S, L, q, R, 0))) return rc;
    ATJUP_CUDA(launch_pdl(R.small, direction_kernel<T>, (R.nt + R.block.y - 1) / R.block.y, R.block, 0, st, S->d, S->p, L.z, S->e, S->code, q,
                          R.kb, R.per, R.nt, S->scal, 1));
    c->launches++;
    const int every = 4;
    double rr = bnorm * bnorm;
    int it = 0;
    for (it = 1; it <= max_iter; it++) {
        const bool check = it % every == 0 || it == max_iter;
        ATJUP_CUDA(launch_pdl(R.small, apply_kernel, R.blocks, R.block, 0, st, S->d, S->q,
                              S->code, c->geo, q, R.kb, R.per, R.nt, S->part, S->ticket, S->scal));
        if ((rc = precond<T, false>(c, S, L, q, R, check))) return rc;
        ATJUP_CUDA(launch_pdl(R.small, direction_kernel<T>, (R.nt + R.block.y - 1) / R.block.y, R.block, 0, st, S->d, S->p, L.z, S->e, S->code,
                              q, R.kb, R.per, R.nt, S->scal, 0));
        c->launches += 2;
        if (check) {
            ATJUP_CUDA(cudaMemcpyAsync(S->hs, S->scal, sizeof(double) * SC_COUNT, cudaMemcpyDeviceToHost, st));
            ATJUP_CUDA(cudaStreamSynchronize(st));
            rr = S->hs[SC_RR];
            if (!std::isfinite(rr)) { set_error("pressure_solve: non-finite residual"); return ATJUP_ERR_NONFINITE; }
            if (std::sqrt(rr) <= tol * bnorm) break;
        }
    }
    ATJUP_CUDA(cudaGetLastError());
    *iters = std::min(it, max_iter);
    *rel = std::sqrt(rr) / bnorm;
    return ATJUP_OK;
}

}  // namespace

void solver_free(AtjupCtx* c) {
    Solver* S = get_solver(c);
    if (!S) return;
    free_lines(S->l64);
    free_lines(S->l32);
    double* all[] = {S->b, S->p, S->r, S->d, S->q, S->g, S->e, S->gh, S->fold, S->tal, S->tcp, S->tm,
                     S->part, S->scal, S->yw};
    for (double* p : all) cudaFree(p);
    cudaFree(S->slot);
    cudaFree(S->cs);
    cudaFree(S->code);
    cudaFree(S->ticket);
    if (S->hs) cudaFreeHost(S->hs);
    delete S;
    c->solver = nullptr;
}

int pressure_residual_solve(AtjupCtx* c, const AtjupSolveOpts* o, AtjupSolveStats* st) {
    const AtjupParams& P = c->P;
    if (!(o->rel_tol > 0.0) || o->max_iter < 1) { set_error("pressure_solve: bad tolerance or cap"); return ATJUP_ERR_ARG; }
    if (o->external_rhs && !c->solve_b) { set_error("pressure_solve: no external right-hand side set"); return ATJUP_ERR_ARG; }
    Solver* S = get_solver(c);
    int rc;
    if (!S) {
        S = new Solver();
        c->solver = S;
        if ((rc = setup(c, S))) { solver_free(c); return rc; }
    }
    cudaStream_t stm = c->stream;
    const size_t NP = c->NP;
    const int nb = NRED;
    OpC q{P.im, P.jm, P.km, c->KP, 1.0 / (P.dr * P.dr)};
    // right-hand side: the reference's clamped divergence source, or the caller's b
    const double* src = c->src;
    if (o->external_rhs) src = c->solve_b;
    else {
        if ((rc = launch_prepare_projection(c))) return rc;
        if ((rc = launch_pressure_source(c))) return rc;
    }
    const Rows R = rows_of(P);
    const double ysum = c->yw_sum;
    double* b64 = c->tmp;    // the projected right-hand side (FP64), kept for the refinement
    double* p64 = c->tmp2;   // the FP64 solution
    const int warm = o->external_rhs ? 0 : 1;
    gather_kernel<<<nb, RB, 0, stm>>>(src, c->f[ATJUP_F_P_DYN], S->yw, b64, p64, NP, warm, S->part,
                                      S->ticket, S->scal);
    // compatibility: remove the y-component of b
    project_kernel<<<nb, RB, 0, stm>>>(b64, S->yw, S->scal, ysum, NP, S->part, S->ticket);
    c->launches += 2;
    // r = b - A p into S->b, its norm and the rounding floor to the host
    auto residual = [&]() -> int {
        residual_kernel<<<R.blocks, R.block, 0, stm>>>(
            b64, p64, S->b, S->code, c->geo, q, R.kb, R.per, R.nt, S->part, S->ticket, S->scal);
        c->launches++;
        ATJUP_CUDA(cudaMemcpyAsync(S->hs, S->scal, sizeof(double) * SC_COUNT, cudaMemcpyDeviceToHost, stm));
        ATJUP_CUDA(cudaStreamSynchronize(stm));
        return ATJUP_OK;
    };
    if ((rc = residual())) return rc;
    const double bnorm = std::sqrt(S->hs[SC_BB]);
    int total_it = 0, inner = 0;
    double rel = 0.0, floor_rel = 0.0, prev = 1e300;
    const bool mixed = (o->precision == ATJUP_PREC_MIXED);
    // Iterative refinement with the residual formed in FP64: r = b - A p; solve A e = r by PCG
    // with FP64 Krylov vectors (the preconditioner in FP32 for the mixed form: the operator's
    // condition number, ~1e9, is above 1/eps of FP32, so FP32 can carry the preconditioner -- whose
    // radial-line and column-mode systems have condition numbers ~1e5 -- but not the residual);
    // p += e. Stops at the tolerance, or when the residual no longer falls (it has reached the
    // rounding floor of an FP64 p, which is reported).
    if (o->mode == ATJUP_SOLVE_SOR) {
        // point red-black SOR with omega, the residual checked every `check` sweeps
        const double omega = (o->omega > 0.0 && o->omega < 2.0) ? o->omega : 1.0;
        const int check = 50;
        int sweeps = 0;
        for (;;) {
            if (sweeps > 0 && (rc = residual())) return rc;
            rel = (bnorm > 0.0) ? std::sqrt(S->hs[SC_RES]) / bnorm : 0.0;
            floor_rel = (bnorm > 0.0) ? 2.220446049250313e-16 * std::sqrt(S->hs[SC_FLOOR]) / bnorm : 0.0;
            if (!std::isfinite(rel)) { set_error("pressure_solve: non-finite residual"); return ATJUP_ERR_NONFINITE; }
            if (rel <= o->rel_tol || sweeps >= o->max_iter) break;
            const int n = std::min(check, o->max_iter - sweeps);
            for (int t = 0; t < n; t++) {
                sor_kernel<<<nb, RB, 0, stm>>>(b64, p64, c->solid, c->geo, S->yw, q, 0, omega);
                sor_kernel<<<nb, RB, 0, stm>>>(b64, p64, c->solid, c->geo, S->yw, q, 1, omega);
            }
            c->launches += 2 * n;
            sweeps += n;
        }
        total_it = sweeps;
    }
    const int max_outer = (o->mode == ATJUP_SOLVE_SOR) ? -1 : 8;
    for (int outer = 0; outer <= max_outer; outer++) {
        if (outer > 0 && (rc = residual())) return rc;
        rel = (bnorm > 0.0) ? std::sqrt(S->hs[SC_RES]) / bnorm : 0.0;
        floor_rel = (bnorm > 0.0) ? 2.220446049250313e-16 * std::sqrt(S->hs[SC_FLOOR]) / bnorm : 0.0;
        if (!std::isfinite(rel)) { set_error("pressure_solve: non-finite residual"); return ATJUP_ERR_NONFINITE; }
        if (rel <= o->rel_tol || total_it >= o->max_iter || outer == max_outer) break;
        if (outer > 0 && rel > 0.5 * prev) break;            // stalled at the FP64 floor
        prev = rel;
        int it = 0;
        double inner_rel = 0.0;
        const int budget = o->max_iter - total_it;
        const double rnorm = std::sqrt(S->hs[SC_RES]);
        const double tgt = o->rel_tol * bnorm / std::max(rnorm, 1e-300);
        const double itol = std::min(1e-3, std::max(0.5 * tgt, 1e-12));
        if (mixed) rc = pcg<float>(c, S, S->l32, rnorm, itol, budget, &it, &inner_rel);
        else rc = pcg<double>(c, S, S->l64, rnorm, itol, budget, &it, &inner_rel);
        if (rc) return rc;
        add_kernel<<<nb, RB, 0, stm>>>(p64, S->p, NP);
        c->launches++;
        total_it += it;
        inner++;
    }
    // write the solution into p_dyn (fluid interior cells), fix the gauge for a cold start, fold
    if (o->external_rhs) {
        gauge_kernel<<<nb, RB, 0, stm>>>(p64, S->yw, NP, S->part, S->ticket, S->scal);
        c->launches++;
    }
    scatter_kernel<<<nb, RB, 0, stm>>>(p64, S->yw, c->f[ATJUP_F_P_DYN], S->scal, ysum, NP,
                                       o->external_rhs ? 1 : 0);
    c->launches++;
    if ((rc = launch_pressure_fold(c, c->f[ATJUP_F_P_DYN]))) return rc;
    ATJUP_CUDA(cudaGetLastError());
    if (st) {
        st->iterations = total_it;
        st->inner_solves = inner;
        st->rel_residual = rel;
        st->b_norm = bnorm;
        st->rel_floor = floor_rel;
    }
    // converged: at the tolerance, or within a small factor of the FP64 floor above it
    if (rel > o->rel_tol && rel > 8.0 * floor_rel) {
        char msg[160];
        snprintf(msg, sizeof(msg), "pressure_solve: relative residual %.3e above tolerance %.1e "
                 "(FP64 floor %.2e) after %d iterations", rel, o->rel_tol, floor_rel, total_it);
        set_error(msg);
        return ATJUP_ERR_NOT_CONVERGED;
    }
    return ATJUP_OK;
}

}  // namespace atjup
