// Boundary passes after the RK step, over the dynamics fields and, with the physics on, the
// species, the chemistry mass fluxes and the closure fields.
//
// Reference: BC_Jup::bcRadius (BC_Jup.h:185-263) around BoundaryConditions<M>::bcRadius
// (BoundaryConditions.h:151-250), bcTheta (253-336), bcPhi (339-360, periodic seam), and
// BC_Jup::bcSolidGround (BC_Jup.h:460-658). Each pass is independent per boundary row or column,
// so each is one kernel over that 2-D face; the solid-cell pass walks a list of the obstacle's
// cells (with their extrapolation partners) built once from the static mask.
#include "ctx.cuh"

namespace atjup {
namespace {

constexpr double kC43 = 4.0 / 3.0, kC13 = 1.0 / 3.0;

// Zonal means of v and w at levels im-3 and im-2 over the km-1 distinct meridians, taken before
// the radial pass for the zonal-mean-preserving sponge (ATJUP_BC_TOP_TAPER = 3).
__global__ void zonal_mean_kernel(const double* __restrict__ v, const double* __restrict__ w,
                                  double* __restrict__ zm, int im, int jm, int km, int KP) {
    const int j = blockIdx.x, l = blockIdx.y;
    const int i = im - 3 + l;
    const size_t b = ((size_t)i * jm + j) * KP;
    double sv = 0.0, sw = 0.0;
#pragma unroll 6
    for (int k = threadIdx.x; k < km - 1; k += 32) { sv += v[b + k]; sw += w[b + k]; }
    for (int o = 16; o > 0; o >>= 1) {
        sv += __shfl_down_sync(0xffffffffu, sv, o);
        sw += __shfl_down_sync(0xffffffffu, sw, o);
    }
    if (threadIdx.x == 0) {
        zm[(size_t)(2 * l) * jm + j] = sv / (km - 1);
        zm[(size_t)(2 * l + 1) * jm + j] = sw / (km - 1);
    }
}

// The fields of a pass with how it treats each (the reference's bc_fields_* lists, BC_Jup.h:275-350).
// The fields are independent of one another in every pass, so the grid takes one of them per block
// (blockIdx.z): a thread that walked the list, up to 23 fields with the physics, spent a memory round
// trip on each (26 to 42 us a pass on the 41x181x361 shell, 21 to 33 us on 13x37x49).
enum { FK_PLAIN = 0, FK_U, FK_V, FK_W, FK_SPECIES, FK_ZERO };
struct FieldList {
    double* f[32];
    uint8_t kind[32];
    int n;
};

// One (j, k) column of one field: 2-point Neumann at both radial walls (BoundaryConditions.h:176-193),
// then for u the rigid lid u = 0, for v and w the top taper (taper 3: zonal-mean preserving,
// BC_Jup.h:186-229), for a species the wall copy at i = 0 and positivity at both walls
// (BC_Jup.h:231-262). Each step is column- and field-local, so doing them per column in the reference's
// order equals the reference's sequence of whole-grid passes.
__global__ void radius_kernel(const __grid_constant__ FieldList L, const double* __restrict__ zm, int im,
                              int jm, int km, int KP, int lid_u, int taper) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, kind = L.kind[blockIdx.z];
    if (k >= km) return;
    double* x = L.f[blockIdx.z];
    const size_t plane = (size_t)jm * KP, b = (size_t)j * KP + k;
    const size_t c1 = b + (im - 1) * plane, c2 = b + (im - 2) * plane, c3 = b + (im - 3) * plane;
    const double b1 = x[b + plane], x2 = x[c2], x3 = x[c3];
    double b0 = kC43 * b1 - kC13 * x[b + 2 * plane];
    double x1 = kC43 * x2 - kC13 * x3;
    if (kind == FK_U && lid_u) b0 = x1 = 0.0;
    if (kind == FK_SPECIES) {
        b0 = b1;                                   // wall copy
        if (b0 < 0.0) b0 = 0.0;                    // positivity
        if (x1 < 0.0) x1 = 0.0;
    }
    if ((kind == FK_V || kind == FK_W) && taper != 0) {
        double y2, y3;
        x1 = 0.0;
        if (taper == 2) {
            const double x4 = x[b + (im - 4) * plane];
            y2 = (1.0 / 3.0) * x4;
            y3 = (2.0 / 3.0) * x4;
        } else {
            y2 = x2 * (1.0 / 3.0);
            y3 = x3 * (2.0 / 3.0);
        }
        if (taper == 3) {
            const double m3 = zm[kind == FK_V ? j : jm + j], m2 = zm[kind == FK_V ? 2 * jm + j : 3 * jm + j];
            y3 += (1.0 / 3.0) * m3;
            y2 += (2.0 / 3.0) * m2;
            x1 = m2;
        }
        x[c2] = y2;
        x[c3] = y3;
    }
    x[b] = b0;
    x[c1] = x1;
}

// Pole rows of one field (BoundaryConditions.h:253-336): rows 1..nfill copy row nfill+1 for an
// extrapolated field and ramp r/(nfill+1) of it for a zero field; the pole row copies row 1
// (extrapolated) or is zero.
__global__ void theta_kernel(const __grid_constant__ FieldList L, int im, int jm, int km, int KP, int nfill) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (k >= km) return;
    double* x = L.f[blockIdx.z];
    const bool zero = L.kind[blockIdx.z] == FK_ZERO;
    const size_t b = (size_t)i * jm * KP + k;
    auto at = [&](int jj) { return b + (size_t)jj * KP; };
    if (nfill > 0) {
        const int jf = nfill + 1;
        for (int r = 1; r <= nfill; r++) {
            const double ramp = (double)r / (double)jf;
            const double lo = x[at(jf)];
            x[at(r)] = zero ? ramp * lo : lo;
            const double hi = x[at(jm - 1 - jf)];         // after the row above: it may be this one
            x[at(jm - 1 - r)] = zero ? ramp * hi : hi;
        }
    }
    x[at(0)] = zero ? 0.0 : x[at(1)];
    x[at(jm - 1)] = zero ? 0.0 : x[at(jm - 2)];
}

__global__ void phi_kernel(const __grid_constant__ FieldList L, int jm, int km, int KP) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= jm) return;
    double* x = L.f[blockIdx.z] + ((size_t)i * jm + j) * KP;
    x[km - 1] = x[0];
}

// Solid cells (BC_Jup.h:496-590): velocities (FK_U) 0; surface cells with an extrapolation pair take the
// 2-point extrapolation of every scalar; the others set the scalars to 0, but keep t and p_stat
// (FK_PLAIN).
__global__ void solid_kernel(const SolidCell* __restrict__ Ls, int n, const __grid_constant__ FieldList S) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const SolidCell s = Ls[q];
    double* x = S.f[blockIdx.z];
    const int kind = S.kind[blockIdx.z];
    if (kind == FK_U) x[s.c] = 0.0;
    else if (s.kind == 1) x[s.c] = kC43 * x[s.a] - kC13 * x[s.b];
    else if (kind != FK_PLAIN) x[s.c] = 0.0;
}

__device__ __forceinline__ double safe_clamp(double v, double lo, double hi) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if ((b & 0x7FF0000000000000ULL) == 0x7FF0000000000000ULL) return lo;
    return (v < lo) ? lo : ((v > hi) ? hi : v);
}

// The sanitising clamps of the closure fields over the whole grid (BC_Jup.h:627-655), with the
// fixed bounds of that routine: k* in [0, 1000 m2/s2], omega* in [1e-10, 1e6], nue* in
// [0, 1e5 m2/s], prod in [0, 1e4], sources in [-1e4, 1e4]; NaN and Inf go to the lower bound.
// A value is stored only where the clamp changes it: almost none, and the fields need not be written
// again (171 MB read in place of 343 MB moved on the 41x181x361 shell).
struct SanArgs {
    double* f[8];              // tke, tken, dis, disn, nue, prod, tke_source, dis_source
    double lo[8], hi[8];
    size_t n;
};
__global__ void __launch_bounds__(256) sanitise_kernel(const __grid_constant__ SanArgs a) {
    double* f = a.f[blockIdx.y];
    const double lo = a.lo[blockIdx.y], hi = a.hi[blockIdx.y];
    const size_t c = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);      // rows are multiples of 16
    if (c >= a.n) return;
    const double2 v0 = *reinterpret_cast<const double2*>(f + c);
    const double2 v1 = *reinterpret_cast<const double2*>(f + c + 2);
    const double v[4] = {v0.x, v0.y, v1.x, v1.y};
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const double x = safe_clamp(v[u], lo, hi);
        if (__double_as_longlong(x) != __double_as_longlong(v[u])) f[c + u] = x;
    }
}

// Ambient temperature of the solid cells of one (i, j) row: the mean of t over its fluid cells.
__global__ void ambient_kernel(const int32_t* __restrict__ rows, const uint8_t* __restrict__ s,
                               double* __restrict__ t, int jm, int km, int KP) {
    const int r = rows[blockIdx.x];
    const size_t b = (size_t)r * KP;
    double sum = 0.0;
    int n = 0;
#pragma unroll 6
    for (int k = threadIdx.x; k < km; k += 32) {
        const double tk = t[b + k];
        if (!s[b + k]) { sum += tk; n++; }
    }
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        n += __shfl_down_sync(0xffffffffu, n, o);
    }
    sum = __shfl_sync(0xffffffffu, sum, 0);
    n = __shfl_sync(0xffffffffu, n, 0);
    if (n == 0) return;
    const double t_amb = sum / n;
    for (int k = threadIdx.x; k < km; k += 32)
        if (s[b + k]) t[b + k] = t_amb;
}

}  // namespace

int launch_bc(AtjupCtx* c, int which) {
    return launch_bc_ptrs(c, which, c->f[ATJUP_F_T], c->f[ATJUP_F_U], c->f[ATJUP_F_V],
                          c->f[ATJUP_F_W], c->f[ATJUP_F_P_DYN], c->f[ATJUP_F_P_STAT], c->phys_on);
}

// The passes on the given t, u, v, w, p_dyn, p_stat (the dry lists unless phys, which takes the
// context's other fields as well): the tangent-linear of the dry passes is this on perturbations.
int launch_bc_ptrs(AtjupCtx* c, int which, double* t, double* u, double* v, double* w,
                   double* p_dyn, double* p_stat, bool phys) {
    const AtjupParams& P = c->P;
    const bool ph = phys;
    // the field lists of the passes (BC_Jup.h:275-350) over the fields the device holds
    auto add = [](FieldList& L, double* x, int kind = FK_PLAIN) { L.kind[L.n] = kind; L.f[L.n++] = x; };
    auto add_species = [&](FieldList& L, int kind) {
        for (int s = 0; s < ATJUP_S_COUNT; s++) add(L, c->f[kScalarField[s]], kind);
    };
    auto add_turb = [&](FieldList& L) {
        add(L, c->f[ATJUP_F_TKE]); add(L, c->f[ATJUP_F_DIS]); add(L, c->f[ATJUP_F_NUE]);
        add(L, c->f[ATJUP_F_PROD]); add(L, c->f[ATJUP_F_TKE_SOURCE]); add(L, c->f[ATJUP_F_DIS_SOURCE]);
    };
    auto add_massflux = [&](FieldList& L, bool fluxlim, int kind) {
        add(L, c->f[ATJUP_F_MASSFLUX_H2S], kind); add(L, c->f[ATJUP_F_MASSFLUX_NH3], kind);
        add(L, c->f[ATJUP_F_MASSFLUX_NH4SH], kind);
        if (fluxlim) add(L, c->f[ATJUP_F_FLUXLIM_NH4SH], kind);
        // the diffusive fluxes travel with the mass fluxes in every list that has them
        add(L, c->f[ATJUP_F_DIFFLUX_H2S], kind); add(L, c->f[ATJUP_F_DIFFLUX_NH3], kind);
        add(L, c->f[ATJUP_F_DIFFLUX_NH4SH], kind);
    };
    if (which & ATJUP_BC_RADIUS) {
        FieldList L{};
        add(L, t); add(L, u, FK_U); add(L, v, FK_V); add(L, w, FK_W);
        if (ph) { add_species(L, FK_SPECIES); add_massflux(L, false, FK_PLAIN); add_turb(L); }
        if (P.top_taper == 3) {
            c->launches++;
            zonal_mean_kernel<<<dim3(P.jm, 2), 32, 0, c->stream>>>(v, w, c->zm, P.im, P.jm, P.km, c->KP);
        }
        c->launches++;
        radius_kernel<<<dim3((P.km + 127) / 128, P.jm, L.n), 128, 0, c->stream>>>(
            L, c->zm, P.im, P.jm, P.km, c->KP, P.lid_u, P.top_taper);
        ATJUP_CHECK_LAUNCH("bc_radius");
    }
    if (which & ATJUP_BC_THETA) {
        FieldList L{};
        add(L, t); add(L, u);
        add(L, v, FK_ZERO); add(L, w, FK_ZERO);
        if (ph) { add_species(L, FK_PLAIN); add_turb(L); add_massflux(L, true, FK_ZERO); }
        c->launches++;
        theta_kernel<<<dim3((P.km + 127) / 128, P.im, L.n), 128, 0, c->stream>>>(
            L, P.im, P.jm, P.km, c->KP, P.pole_fill_rows);
        ATJUP_CHECK_LAUNCH("bc_theta");
    }
    if (which & ATJUP_BC_PHI) {
        FieldList L{};
        add(L, t); add(L, u); add(L, v); add(L, w);
        if (ph) { add_species(L, FK_PLAIN); add_massflux(L, true, FK_PLAIN); add_turb(L); }
        c->launches++;
        phi_kernel<<<dim3((P.jm + 127) / 128, P.im, L.n), 128, 0, c->stream>>>(L, P.jm, P.km, c->KP);
        ATJUP_CHECK_LAUNCH("bc_phi");
    }
    if (which & ATJUP_BC_SOLID) {
        if (c->n_solid > 0) {
            FieldList S{};
            add(S, t); add(S, p_stat); add(S, p_dyn, FK_ZERO);
            add(S, u, FK_U); add(S, v, FK_U); add(S, w, FK_U);
            if (ph) { add_species(S, FK_ZERO); add_massflux(S, true, FK_ZERO); }
            c->launches++;
            solid_kernel<<<dim3((c->n_solid + 127) / 128, 1, S.n), 128, 0, c->stream>>>(c->solid_list,
                                                                                       c->n_solid, S);
            if (P.mount_t_ambient && c->n_amb_rows > 0) {
                c->launches++;
                ambient_kernel<<<c->n_amb_rows, 32, 0, c->stream>>>(c->amb_rows, c->solid, t, P.jm,
                                                                   P.km, c->KP);
            }
        }
        if (ph) {
            const double prod_max = 1.0e4, dis_max = 1.0e6;
            const double tke_max = 1000.0 / (P.u_0 * P.u_0), nue_max = 1.0e5 / (P.u_0 * P.L_atm * 1.0e3);
            const SanArgs a{{c->f[ATJUP_F_TKE], c->fn[ATJUP_F_TKE], c->f[ATJUP_F_DIS], c->fn[ATJUP_F_DIS],
                             c->f[ATJUP_F_NUE], c->f[ATJUP_F_PROD], c->f[ATJUP_F_TKE_SOURCE],
                             c->f[ATJUP_F_DIS_SOURCE]},
                            {0.0, 0.0, 1.0e-10, 1.0e-10, 0.0, 0.0, -prod_max, -prod_max},
                            {tke_max, tke_max, dis_max, dis_max, nue_max, prod_max, prod_max, prod_max},
                            c->NP};
            c->launches++;
            sanitise_kernel<<<dim3((unsigned)((c->NP / 4 + 255) / 256), 8), 256, 0, c->stream>>>(a);
        }
        ATJUP_CHECK_LAUNCH("bc_solid");
    }
    return ATJUP_OK;
}

}  // namespace atjup
