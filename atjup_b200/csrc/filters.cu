// Shapiro filters and the column balance of v.
//
// Reference: JupiterUtils::damp_wiggles (lib/Utils.cpp:227-323, order 2) and damp_wiggles_ho
// (lib/Utils.cpp:334-453, order 4): direction-split passes k (periodic ring of km-1 meridians,
// k = km-1 written as the copy of k = 0), then j (clamped at the poles), then i (clamped at the
// fluid floor i_topography), each pass reading a full copy of the field. Here the k and j passes are
// one out-of-place kernel and the i pass another (each writes every cell, filtered, or copied where the
// reference skips), field -> scratch -> field, for up to three fields at once.
//
// cJupiterModel::balanceColumnV (InitValues_Jup.cpp:1500-1538): trapezoid column mean of r v
// over columns off the obstacle, then (zonal form) the row mean of those removed from every
// off-obstacle column of the row.
#include "ctx.cuh"

#include <algorithm>
#include <vector>

namespace atjup {
namespace {

struct FiltConst {
    int im, jm, km, KP, use_topo;
    double c4, c2;
};

// Up to three fields filtered by one launch.
constexpr int NF = 3;
struct FiltFields {
    const double* src[NF];
    double* dst[NF];
};

__device__ __forceinline__ int floor_at(const int32_t* topo, int use_topo, int j, int k, int km) {
    if (!use_topo) return 0;
    const int t = topo[(size_t)j * km + k];
    return t > 0 ? t : 0;
}

struct D2 {
    double x, y;
};

// The k and j passes of one level. A thread takes two neighbouring meridians (the ring is even and
// rows start on 128-byte boundaries: 16-byte accesses) and marches over a chunk of rows: it forms the k
// pass of the row ORDER / 2 ahead and keeps the last ORDER + 1 of them in registers, which the j pass
// then reads, so the k-filtered field is never stored. One more thread writes the seam column, which
// takes k = 0's result of the k pass. Cells whose stencil lies wholly above the floor (i >= hi, the
// highest floor of the columns within two cells along k, or along j) take the plain formula; the
// others test each neighbour. Bound by the latency of the rows at 20 warps per SM (64 registers; 74 us at
// 48, 78 us with the row loop unrolled to 122). u, v, w of the 41x181x361 shell: 52 us, 115 us in separate
// k and j passes that tested the floor of every neighbour at every level.
template <int ORDER>
__global__ void __launch_bounds__(256, 4)
shapiro_kj_kernel(FiltFields F, const int32_t* __restrict__ topo, const int32_t* __restrict__ hi_k,
                  const int32_t* __restrict__ hi_j, FiltConst q, int rows) {
    constexpr int H = ORDER / 2, W = 2 * H + 1;
    const int n = q.km - 1, ko = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int f = blockIdx.z / q.im, i = blockIdx.z - f * q.im;
    if (ko > n) return;
    const bool seam = ko == n;
    const int k = seam ? 0 : ko, km = k == 0 ? n - 2 : k - 2, kp = k == n - 2 ? 0 : k + 2;
    const unsigned row = q.KP, lev = (unsigned)i * q.jm;
    const double* __restrict__ src = f == 0 ? F.src[0] : f == 1 ? F.src[1] : F.src[2];
    double* __restrict__ dst = f == 0 ? F.dst[0] : f == 1 ? F.dst[1] : F.dst[2];
    const int j0 = blockIdx.y * rows, j1 = min(q.jm, j0 + rows);
    pdl_next();
    pdl_wait();
    auto order4 = [&](double vp2, double vp1, double cc, double vm1, double vm2) {
        const double d4 = vp2 - 4.0 * vp1 + 6.0 * cc - 4.0 * vm1 + vm2;
        return cc - q.c4 * d4;
    };
    auto order2 = [&](double vm, double cc, double vp) { return cc + q.c2 * (vm - 2.0 * cc + vp); };
    // the k pass at one meridian kk of row j near the floor: c its value, its neighbours m2..p2
    auto kslow = [&](int j, int kk, double m2, double m1, double c, double p1, double p2) -> double {
        auto wrap = [&](int x) { return x < 0 ? x + n : (x >= n ? x - n : x); };
        auto inf = [&](int x) { return i >= floor_at(topo, q.use_topo, j, wrap(x), q.km); };
        if (!inf(kk)) return c;
        const bool fm = inf(kk - 1), fp = inf(kk + 1);
        if (ORDER == 2) return order2(fm ? m1 : c, c, fp ? p1 : c);
        if (!fm || !fp) return c;
        return (inf(kk - 2) && inf(kk + 2)) ? order4(p2, p1, c, m1, m2) : order2(m1, c, p1);
    };
    // a row's values about the pair and its floors, read a row before they are used
    struct Raw { double2 a, b, c; int2 h; } nx;
    auto fetch = [&](int j) {
        const double* r = src + (lev + j) * row;
        nx.a = *reinterpret_cast<const double2*>(r + km);
        nx.b = *reinterpret_cast<const double2*>(r + k);
        nx.c = *reinterpret_cast<const double2*>(r + kp);
        nx.h = q.use_topo ? *reinterpret_cast<const int2*>(hi_k + j * row + k) : make_int2(0, 0);
    };
    auto kpass = [&](int j, const Raw& v) -> D2 {
        const double2 a = v.a, b = v.b, c = v.c;
        if (i >= v.h.x && i >= v.h.y)
            return ORDER == 4 ? D2{order4(c.x, b.y, b.x, a.y, a.x), order4(c.y, c.x, b.y, b.x, a.y)}
                              : D2{order2(a.y, b.x, b.y), order2(b.x, b.y, c.x)};
        return D2{kslow(j, k, a.x, a.y, b.x, b.y, c.x), kslow(j, k + 1, a.y, b.x, b.y, c.x, c.y)};
    };
    auto jslow = [&](int j, int kk, double m2, double m1, double c, double p1, double p2) -> double {
        auto inf = [&](int r) { return r >= 0 && r < q.jm && i >= floor_at(topo, q.use_topo, r, kk, q.km); };
        if (!inf(j)) return c;
        const bool fm = inf(j - 1), fp = inf(j + 1);
        if (ORDER == 2) return order2(fm ? m1 : c, c, fp ? p1 : c);
        if (!fm || !fp) return c;
        return (inf(j - 2) && inf(j + 2)) ? order4(p2, p1, c, m1, m2) : order2(m1, c, p1);
    };
    D2 w[W];
#pragma unroll
    for (int u = 0; u < W; u++) w[u] = D2{0.0, 0.0};
#pragma unroll
    for (int u = 0; u < W - 1; u++) {
        const int j = j0 - H + u;
        if (j >= 0 && j < q.jm) { fetch(j); w[u + 1] = kpass(j, nx); }
    }
    fetch(min(j0 + H, q.jm - 1));
#pragma unroll 1
    for (int j = j0; j < j1; j++) {
#pragma unroll
        for (int u = 0; u < W - 1; u++) w[u] = w[u + 1];
        const Raw now = nx;
        fetch(min(j + H + 1, q.jm - 1));
        const int2 h = q.use_topo ? *reinterpret_cast<const int2*>(hi_j + j * row + ko) : make_int2(0, 0);
        if (j + H < q.jm) w[W - 1] = kpass(j + H, now);
        const D2 c = w[H];
        D2 o;
        if (j >= H && j < q.jm - H && i >= h.x && i >= h.y) {
            if (ORDER == 4) {
                o.x = order4(w[H + 2 < W ? H + 2 : 0].x, w[H + 1].x, c.x, w[H - 1].x, w[0].x);
                o.y = order4(w[H + 2 < W ? H + 2 : 0].y, w[H + 1].y, c.y, w[H - 1].y, w[0].y);
            } else {
                o.x = order2(w[H - 1].x, c.x, w[H + 1].x);
                o.y = order2(w[H - 1].y, c.y, w[H + 1].y);
            }
        } else {
            o.x = jslow(j, ko, w[0].x, w[H - 1].x, c.x, w[H + 1].x, w[W - 1].x);
            o.y = seam ? 0.0 : jslow(j, ko + 1, w[0].y, w[H - 1].y, c.y, w[H + 1].y, w[W - 1].y);
        }
        double* y = dst + (lev + j) * row + ko;
        if (seam) *y = o.x;
        else *reinterpret_cast<double2*>(y) = make_double2(o.x, o.y);
    }
}

// The i pass: two meridians of a row per thread, marching up a chunk of the levels with the last
// ORDER + 1 in registers and two more levels on the way. Bound by memory (16 B per cell): u, v, w of the
// 41x181x361 shell in 29 us (131 MB), 44 us with one thread per cell.
template <int ORDER>
__global__ void __launch_bounds__(256)
shapiro_i_kernel(FiltFields F, const int32_t* __restrict__ topo, FiltConst q, int per, int chunks) {
    constexpr int H = ORDER / 2, W = 2 * H + 1;
    const int n = q.km - 1, k = 2 * (blockIdx.x * blockDim.x + threadIdx.x), j = blockIdx.y;
    const int f = blockIdx.z / chunks, i0 = (blockIdx.z - f * chunks) * per, i1 = min(q.im, i0 + per);
    if (k > n) return;
    const unsigned plane = (unsigned)q.jm * q.KP;
    // the row's last pair is the seam column and a padding lane
    const size_t b = (size_t)j * q.KP + k;
    const double* __restrict__ x = (f == 0 ? F.src[0] : f == 1 ? F.src[1] : F.src[2]) + b;
    double* __restrict__ y = (f == 0 ? F.dst[0] : f == 1 ? F.dst[1] : F.dst[2]) + b;
    pdl_next();
    pdl_wait();
    const int sx = floor_at(topo, q.use_topo, j, k, q.km);
    const int sy = k == n ? sx : floor_at(topo, q.use_topo, j, k + 1, q.km);
    auto one = [&](int i, int is, double m2, double m1, double c, double p1, double p2) -> double {
        if (i < is) return c;
        const bool fm1 = i - 1 >= is, fp1 = i + 1 <= q.im - 1;
        if (ORDER == 2) return c + q.c2 * ((fm1 ? m1 : c) - 2.0 * c + (fp1 ? p1 : c));
        if (!fm1 || !fp1) return c;
        if (i - 2 >= is && i + 2 <= q.im - 1) {
            const double d4 = p2 - 4.0 * p1 + 6.0 * c - 4.0 * m1 + m2;
            return c - q.c4 * d4;
        }
        return c + q.c2 * (m1 - 2.0 * c + p1);
    };
    auto at = [&](int i) -> D2 {
        const double2 v = *reinterpret_cast<const double2*>(x + (size_t)((unsigned)i * plane));
        return D2{v.x, v.y};
    };
    D2 w[W];
#pragma unroll
    for (int u = 0; u < W; u++) w[u] = D2{0.0, 0.0};
#pragma unroll
    for (int u = 0; u < W - 1; u++) {
        const int i = i0 - H + u;
        if (i >= 0 && i < q.im) w[u + 1] = at(i);
    }
    D2 n1 = at(min(i0 + H, q.im - 1)), n2 = at(min(i0 + H + 1, q.im - 1));   // two levels ahead
#pragma unroll 5
    for (int i = i0; i < i1; i++) {
#pragma unroll
        for (int u = 0; u < W - 1; u++) w[u] = w[u + 1];
        w[W - 1] = n1;
        n1 = n2;
        n2 = at(min(i + H + 2, q.im - 1));
        const double2 o = make_double2(one(i, sx, w[0].x, w[H - 1].x, w[H].x, w[H + 1].x, w[W - 1].x),
                                       one(i, sy, w[0].y, w[H - 1].y, w[H].y, w[H + 1].y, w[W - 1].y));
        double* yi = y + (size_t)((unsigned)i * plane);
        if (k == n) *yi = o.x;
        else *reinterpret_cast<double2*>(yi) = o;
    }
}

// balanceColumnV: the trapezoid column means of r v over the columns off the obstacle (one thread per
// column, the reference's summation order; eight levels' loads at a time)
constexpr int BU = 8;
__global__ void __launch_bounds__(64)
vcol_kernel(const double* __restrict__ v, const int32_t* __restrict__ topo,
            const double* __restrict__ rad, double* __restrict__ dvc, int im, int jm, int km, int KP,
            double dr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y + 1;
    if (k >= km || topo[(size_t)j * km + k] > 0) return;
    const size_t plane = (size_t)jm * KP, b = (size_t)j * KP + k;
    const double* x = v + b;
    double I1 = 0.0, I0 = 0.0, rv = rad[0] * x[0];
    for (int h = 1; h < im; h += BU) {
        double xv[BU], rr[BU];
#pragma unroll
        for (int u = 0; u < BU; u++)
            if (h + u < im) { xv[u] = x[(h + u) * plane]; rr[u] = rad[h + u]; }
#pragma unroll
        for (int u = 0; u < BU; u++) {
            if (h + u >= im) break;
            const double rn = rr[u] * xv[u];
            I1 += 0.5 * (rv + rn) * dr;
            I0 += 0.5 * ((u ? rr[u - 1] : rad[h - 1]) + rr[u]) * dr;
            rv = rn;
        }
    }
    dvc[b] = I1 / I0;
}

// Their mean over the row's meridians k < km-1 (zonal; by the first warp of every block of the row, in
// a fixed order), or without zonal the column's own, off a chunk of the levels of those columns.
__global__ void __launch_bounds__(384)
vsub_kernel(double* __restrict__ v, const int32_t* __restrict__ topo, const double* __restrict__ dvc,
            double* __restrict__ dvrow, int im, int jm, int km, int KP, int zonal, int per) {
    const int j = blockIdx.x + 1, i0 = blockIdx.y * per, i1 = min(im, i0 + per);
    const size_t plane = (size_t)jm * KP;
    const int32_t* tr = topo + (size_t)j * km;
    const double* dc = dvc + (size_t)j * KP;
    __shared__ double mean;
    if (zonal && threadIdx.x < 32) {
        double s = 0.0;
        int n = 0;
#pragma unroll 4
        for (int k = threadIdx.x; k < km - 1; k += 32)
            if (tr[k] == 0) { s += dc[k]; n++; }
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_down_sync(0xffffffffu, s, o);
            n += __shfl_down_sync(0xffffffffu, n, o);
        }
        if (threadIdx.x == 0) {
            mean = (n > 0) ? s / n : 0.0;
            if (blockIdx.y == 0) dvrow[j] = mean;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < km; k += blockDim.x) {
        if (tr[k] > 0) continue;
        const double d = zonal ? mean : dc[k];
        double* x = v + (size_t)j * KP + k;
#pragma unroll 4
        for (int i = i0; i < i1; i++) x[i * plane] -= d;
    }
}

}  // namespace

// hi_k, hi_j of the mask, [jm][KP] each: per column the highest floor of the columns within two cells
// along the ring (km-1 meridians; the seam column unused) and along j
int filter_tables(AtjupCtx* c, const int32_t* topo) {
    const int jm = c->P.jm, km = c->P.km, KP = c->KP, n = km - 1;
    const size_t N = (size_t)jm * KP;
    std::vector<int32_t> h(2 * N, 0);
    for (int j = 0; j < jm; j++)
        for (int k = 0; k < km; k++) {
            int a = 0, b = 0;
            for (int d = -2; d <= 2; d++) {
                a = std::max(a, (int)topo[(size_t)j * km + (k + d + 2 * n) % n]);
                if (j + d >= 0 && j + d < jm) b = std::max(b, (int)topo[(size_t)(j + d) * km + k]);
            }
            h[(size_t)j * KP + k] = a;
            h[N + (size_t)j * KP + k] = b;
        }
    if (!c->floor_hi) ATJUP_CUDA(cudaMalloc(&c->floor_hi, sizeof(int32_t) * 2 * N));
    ATJUP_CUDA(cudaMemcpy(c->floor_hi, h.data(), sizeof(int32_t) * 2 * N, cudaMemcpyHostToDevice));
    return ATJUP_OK;
}

// n fields (1 to 3), each filtered in place: the k and j passes into scratch, the i pass back.
int launch_shapiro_n(AtjupCtx* c, double* const* f, int n, int order, double strength, int passes,
                     int use_topo) {
    const AtjupParams& P = c->P;
    if ((long)P.im * n > MAX_GRID_Z) {         // a level and field per blockIdx.z: the fields one by one
        for (int x = 0; x < n; x++)
            if (int rc = launch_shapiro_n(c, f + x, 1, order, strength, passes, use_topo)) return rc;
        return ATJUP_OK;
    }
    FiltConst q{};
    q.im = P.im; q.jm = P.jm; q.km = P.km; q.KP = c->KP;
    q.use_topo = use_topo;
    q.c4 = strength / 16.0;
    q.c2 = strength * 0.25;
    // scratch: the Poisson source is formed anew by each pressure pass
    double* scratch[NF] = {c->tmp, c->tmp2, c->src};
    FiltFields there{}, back{};
    for (int x = 0; x < n; x++) {
        there.src[x] = back.dst[x] = f[x];
        there.dst[x] = scratch[x];
        back.src[x] = scratch[x];
    }
    const int pairs = (P.km - 1) / 2 + 1, th = std::min(256, (pairs + 31) / 32 * 32);
    const int kb = (pairs + th - 1) / th;
    // Rows and levels per thread (ORDER / 2 more are read on each side). A thread's are a chain of memory round
    // trips, so few while the warps of one row each, which is what the SMs can hold about twice over at 12500,
    // leave them idle; more where the reads beside a chunk are what counts. By a sweep of both over nine shells: one
    // field of 9x21x33 23.3 us at 8 and 16.6 at 1 row, of 41x61x97 26.8 and 16.6, of 41x181x361 36.9 and 32.9 at 3 to 4
    // (43.3 at 1), three fields of it 86.1 at 8 and 88.3 at 4; levels: 9x21x33 13.5 us at 1 and 16.5 at 5, 41x61x97
    // 16.5 at both, 33x121x243 20.8 at 5, 23.8 at 1 and 24.8 at 15, three fields of 41x181x361 91.2 at 15, 92.1 at 5.
    const long warps = (long)kb * (th / 32) * P.jm * P.im * n;
    const int rows = (int)std::min(8L, (warps + 12499) / 12500);
    const int per = warps <= 4000 ? 1 : warps <= 100000 ? 5 : 15;
    // The launches overlap the tails of the kernels before them (launch_pdl) but for the largest: one field of 9x21x33
    // 13.3 and 9.6 us so, of 41x61x97 16.4 and 12.6, of 41x181x361 32.8 and 28.7; with three of it too the
    // iteration with physics, whose second stream then finds fewer free blocks, 7890 and 7975 us.
    const bool overlap = warps <= 50000;
    const int chunks = (P.im + per - 1) / per;
    const dim3 gkj(kb, (P.jm + rows - 1) / rows, P.im * n), gi(kb, P.jm, n * chunks);
    const int32_t *hk = c->floor_hi, *hj = c->floor_hi + (size_t)P.jm * c->KP;
    for (int p = 0; p < passes; p++) {
        c->launches += 2;
        auto kj = order == 4 ? shapiro_kj_kernel<4> : shapiro_kj_kernel<2>;
        auto ip = order == 4 ? shapiro_i_kernel<4> : shapiro_i_kernel<2>;
        ATJUP_CUDA(launch_pdl(overlap, kj, gkj, th, 0, c->stream, there, c->topo, hk, hj, q, rows));
        ATJUP_CUDA(launch_pdl(overlap, ip, gi, th, 0, c->stream, back, c->topo, q, per, chunks));
    }
    ATJUP_CHECK_LAUNCH("shapiro");
    return ATJUP_OK;
}

int launch_shapiro(AtjupCtx* c, double* f, int order, double strength, int passes, int use_topo) {
    return launch_shapiro_n(c, &f, 1, order, strength, passes, use_topo);
}

int launch_balance_v(AtjupCtx* c) {
    const AtjupParams& P = c->P;
    c->launches += 2;
    return launch_balance_v_buffers(c->f[ATJUP_F_V], c->topo, c->rad, c->dvc, c->dvrow, P.im, P.jm,
                                    P.km, c->KP, P.dr, P.v_massbal_zonal, c->stream);
}

// The column balance of v on given buffers (the no-allocation entry point in noalloc.cu supplies its
// file-scope scratch): v [im][jm][pitch], topo [jm * km], rad [im], dvc [jm * pitch], dvrow [jm].
int launch_balance_v_buffers(double* v, const int32_t* topo, const double* rad, double* dvc,
                             double* dvrow, int im, int jm, int km, int pitch, double dr,
                             int zonal, cudaStream_t st) {
    const int th = std::min(384, (km + 31) / 32 * 32);
    const int per = 8;
    vcol_kernel<<<dim3((km + 63) / 64, jm - 2), 64, 0, st>>>(v, topo, rad, dvc, im, jm, km, pitch, dr);
    vsub_kernel<<<dim3(jm - 2, (im + per - 1) / per), th, 0, st>>>(v, topo, dvc, dvrow, im, jm, km,
                                                                   pitch, zonal, per);
    ATJUP_CHECK_LAUNCH("balance_v");
    return ATJUP_OK;
}

}  // namespace atjup
