// The in-loop projection of the horizontal wind around the obstacle (projectAroundObstacle with
// in_loop = true, InitValues_Jup.cpp:1595-1822; called every ATJUP_CONE_PROJ_STRIDE iterations
// after the column balance of v, cJupiterModel.cpp:1356-1363).
//
// Per level i in 1..im-2 that holds solid cells, a box M cells wider than the obstacle's
// cross-section (clipped to j 1..jm-2, k 1..km-2, phi = 0 on a one-cell halo) and up to two SOR
// solves on it: with ATJUP_CONE_PROJ_DIV = H > 0 first the divergence solve (the cells within H
// cells, Chebyshev in 3-D, of the body take the 3-D face divergence s r D of the flow before the
// correction as a source and close their wall faces), then the wall-flux solve (a wall face
// carries the prescribed flux -U.n). Each solve is warm-started from its own phi of the previous
// call, runs lexicographic SOR (omega 1.9) until the largest change of a sweep is at most 1e-10
// of the largest |phi| (at most 40000 sweeps), and increments v and w by the average of the two
// face corrections of each direction (a wall face's correction is minus the cell's velocity).
// Finally the seam column k = km-1 takes v and w of k = 0.
//
// B200 form. Lexicographic SOR is replayed exactly as a pipelined wavefront: cell (a, b) of the
// box lies on the anti-diagonal d = a + b, its sweep-t update needs sweep t of (a-1, b) and
// (a, b-1) and sweep t-1 of (a+1, b) and (a, b+1), so step tau of the wavefront can update
// diagonal d = tau - 2(t-1) for every sweep t in flight at once. The cells of one step are then
// exactly the cells of one colour of the checkerboard, (a + b) = tau mod 2, less those whose sweep
// has not begun or is past the last; a step reads only the other colour, so the cells of a step
// are independent and one barrier between steps orders them. phi is stored split by colour (each
// row's cells of one colour contiguous), so a warp's lanes take consecutive cells of one row and
// read the four neighbours from consecutive words of the other colour.
//
// Each level is one thread-block cluster of C blocks (C = 4, or fewer when the GPU cannot hold
// every level's cluster at once: 26 levels on 104 SMs for the 41 x 181 x 361 grid). Block r owns
// a band of the box's rows with its phi, cell flags and constants in shared memory, and copies of the
// rows next to its band: the block that updates an edge row stores the new values in the neighbour's
// copy too (distributed shared memory), so every load is a local one. Each sweep's largest change and
// largest |phi| are kept per block in a ring slot; sweep t is complete after step D + 2(t-1)
// (D = NJ + NK - 2). Every CHECK_STEPS steps the blocks take the stopping test of the sweeps completed
// since, reading the C slots of each. The sweeps after the converged one have by then already updated
// the first diagonals; each block restores its band from the newest snapshot that precedes them (one
// every SNAP_EVERY steps, in HBM) and the cluster replays up to the converged sweep. The arithmetic is
// the reference's, operation for operation (this file is compiled without FMA contraction but for the
// quotients, which equal the division), so the result is the reference's to the bit.
//
// What bounds it: the issue of a step's instructions and its chain of dependent FP64 operations, on few
// cells (1500 a block and step on the 41 x 181 x 361 grid); no memory traffic to speak of. One projection
// there takes 5.7 ms (12.7 ms with the cells over all warps, the compiler's division, every cell
// raising its sweep's slot and a cluster barrier each step), 61 x 97 2.5 ms (4.9), 33 x 41 1.0 ms (1.6).
#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include <cooperative_groups.h>

#include "cone_plan.cuh"
#include "ctx.cuh"
#include "quot.cuh"

namespace cg = cooperative_groups;

namespace atjup {

namespace {

constexpr double CONE_OMEGA = 1.9;       // InitValues_Jup.cpp:1726
constexpr int CONE_MAXIT = 40000;        // InitValues_Jup.cpp:1728
constexpr double CONE_TOL = 1.0e-10;     // InitValues_Jup.cpp:1761
constexpr int SNAP_EVERY = 64;           // wavefront steps between snapshots
constexpr int CHECK_STEPS = 16;          // wavefront steps between stopping tests
constexpr int DRAIN_POLLS = 1 << 20;     // of the rows still under way when a solve is given up
// per box row: aN, aS, aL, A of a plain cell, 1 / A, s, s dphi (and one unused: rows of 64 bytes, read
// two doubles at a time)
constexpr int NROW = CONE_NROW;
enum { RC_N, RC_S, RC_L, RC_A, RC_RA, RC_SJ, RC_SD };

// cell flags of the box (uint32 per cell: these bits, the special-cell index above bit 6)
enum : uint32_t { CF_SOLID = 1, CF_N = 2, CF_S = 4, CF_W = 8, CF_E = 16, CF_NEAR = 32 };
constexpr uint32_t CF_WALL = CF_N | CF_S | CF_W | CF_E;

}  // namespace

// One level's box. Colour-split storage: cell (a', b') of the box with its halo (a' = a + 1 in
// 0..NJ+1, b' = b + 1 in 0..NK+1) sits at ((c (NJ + 2) + a') PW + b' / 2), c = (a' + b') mod 2;
// the flags of interior cell (a, b) at ((c NJ + a) PW + (b + 1) / 2).
struct ConeLevel {
    int i, jlo, klo, NJ, NK, PW, D, n_spec, n_tab;
    int64_t info_off;   // uint32 [2 * NJ * PW]: flags | special index << 6
    int64_t spec_off;   // int32 [n_spec]: (c NJ + a) PW + m of each special cell
    int64_t phi_off;    // double [2 * (NJ + 2) * PW] per warm-start buffer (halo included)
    int64_t snap_off;   // double [n_snap * C * 2 * (nbmax + 2) * PW]: per block, its band and the rows beside it
    int64_t tab_off;    // double [n_tab] (global-memory mode)
    int64_t row_off;    // double [NROW * NJ] (global-memory mode)
    int n_snap, ring;
};

struct ConeState {
    std::vector<ConeLevel> lv;
    ConeLevel* d_lv = nullptr;
    uint32_t* info = nullptr;
    int32_t* spec = nullptr;
    double* prev[2] = {nullptr, nullptr};   // 0: divergence solve, 1: wall-flux solve
    double* snap = nullptr;
    double* tab = nullptr;
    double* rows = nullptr;
    double* s = nullptr;                    // [jm] max(sinthe_min, |sin(the_j)|)
    int* stats = nullptr;                   // [2 * levels] sweeps of the last call
    int H = 0, M = 0;
    ConePlan plan{};
    int ring_max = 1;                       // the largest ring of the levels
    const void* kernel = nullptr;           // the plan's form of cone_kernel
};

namespace {

struct ConeArgs {
    const ConeLevel* lv;
    const uint32_t* info;
    const int32_t* spec;
    double* prev0;
    double* prev1;
    double* snap;
    double* tab;
    double* rows;
    const double* s;
    int* stats;
    const double* u;
    double* v;
    double* w;
    const uint8_t* solid;
    const double* rad;
    int jm, km, KP, H, C, ring_max, polls;
    double dr, dthe, dphi;
};

// RowForm: a block's barriers for the rows of its neighbours, [2 side + colour], north's side first; and what
// is kept once a wait on one of them has given up.
struct RowWaits {
    unsigned long long bar[4];
    int owed[4];                // rows that came after it, which no wait has taken
    int gave[2];                // the colour whose wait gave up, per side
    int lost;                   // any warp of the block gave up
};

// A block's band of a level's box as the kernel sees it. Local row la = 1..nb is box row
// a = A0 + la - 1 (halo coordinate a' = A0 + la); the words of colour x, local row la start at
// phi + x cs + la PW, la = 0 and nb + 1 being the copies of the rows beside the band (or the box's halo).
struct Box {
    double* phi;
    int cs;                     // colour stride of phi
    const uint32_t* info;       // flags of local row la, colour x at info + x ics + (la - 1) PW
    int ics;
    const double* tab;
    const double* rows;         // [NJ][NROW], indexed by box row
    unsigned long long* ring;   // [2 R]: largest change, largest |phi| of sweep t at t mod R
    double *push_n, *push_s;    // the neighbours' copies of this band's first and last row (colour 0), or null
    unsigned bar_n, bar_s;      // RowForm: those copies' barriers there (shared addresses)
    RowWaits* waits;            // and this block's own
    int polls;                  // of a wait for a neighbour's row
    int NJ, NK, PW, D, R;       // R a power of two
    int nb, A0;
    bool div;
    bool recip;                 // every row's A has a reciprocal quot() takes
    double dthe, dphi;
};

// phi of the cell at local row la (0..nb+1), halo column b' (0..NK+1)
__device__ __forceinline__ double phi_at(const Box& B, int la, int bp) {
    return B.phi[((B.A0 + la + bp) & 1) * B.cs + la * B.PW + (bp >> 1)];
}

// std::max(cur, x) as the reference folds it (a NaN x leaves cur), on the ring's bit patterns
__device__ __forceinline__ void ring_raise(unsigned long long* slot, double cur, double x) {
    if (x > cur) atomicMax(slot, (unsigned long long)__double_as_longlong(x));
}

// The constants of a box row: aN, aS, aL, A of a plain cell, rcp_of(A).
struct RowCoef {
    double N, S, L, A, rA;
};
__device__ __forceinline__ RowCoef row_coef(const Box& B, int la) {
    const double2* rc = reinterpret_cast<const double2*>(B.rows + (size_t)(B.A0 + la - 1) * NROW);
    const double2 c0 = rc[0], c1 = rc[1];
    return RowCoef{c0.x, c0.y, c1.x, c1.y, rc[2].x};
}

// A special cell's entry in tab, at 2 (f >> 6): of a wall cell A, rcp_of(A), the four faces' prescribed terms (zero
// in the divergence solve) and the divergence's source; of a cell near the body without a wall the source.
constexpr int TAB_WALL = 8, TAB_NEAR = 2;

// B and A of a cell with flags f and neighbours pN, pS, pW, pE (InitValues_Jup.cpp:1739-1758), in the reference's
// order of operations; r = rcp_of(A). (What a wall face adds to B is a constant of the cell.)
__device__ __forceinline__ double cone_sum(const RowCoef& R, double pN, double pS, double pW, double pE) {
    double Bs = R.N * pN;
    Bs += R.S * pS;
    Bs += R.L * pW;
    Bs += R.L * pE;
    return Bs;
}
__device__ __forceinline__ double cone_special(const Box& B, const RowCoef& R, uint32_t f, double Bs, double pN, double pS,
                                               double pW, double pE, double& A, double& r) {
    const double2* t = reinterpret_cast<const double2*>(B.tab) + (f >> 6);
    if (!(f & CF_WALL)) return B.div ? Bs + t[0].x : Bs;
    const double2 a = t[0], k0 = t[1], k1 = t[2];
    Bs = f & CF_N ? k0.x : R.N * pN;
    Bs += f & CF_S ? k0.y : R.S * pS;
    Bs += f & CF_W ? k1.x : R.L * pW;
    Bs += f & CF_E ? k1.y : R.L * pE;
    A = a.x;
    r = a.y;
    return B.div ? Bs + t[3].x : Bs;
}
// quot() takes the sum (A's side is B.recip)
__device__ __forceinline__ bool sum_ok(double Bs) {
    return 2u * (unsigned)__double2hiint(Bs) - (623u << 21) < (801u << 21);
}

// raises the band's slot of the sweep a cell with this diff = tau - a - b is in, or opens it
__device__ __forceinline__ void raise(const Box& B, unsigned diff, bool opens, double dch, double pabs) {
    unsigned long long* slot = B.ring + 2 * ((int)((diff >> 1) + 1) & (B.R - 1));
    if (opens) {
        slot[0] = (unsigned long long)__double_as_longlong(dch > 0.0 ? dch : 0.0);
        slot[1] = (unsigned long long)__double_as_longlong(pabs > 0.0 ? pabs : 0.0);
    } else {
        const double2 cur = *reinterpret_cast<const double2*>(slot);   // at most as large as it is now
        ring_raise(slot, cur.x, dch);
        ring_raise(slot + 1, cur.y, pabs);
    }
}

// The block's and the cluster's barriers, for code that a block's warps take in different copies.
__device__ __forceinline__ void block_sync() { asm volatile("barrier.sync.aligned 0;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The two forms of a wavefront step tau on the block's band: the cells of colour tau mod 2 whose sweep
// t = (tau - a - b) / 2 + 1 lies in [1, t_stop]; t2 = 2 t_stop.

// Any band: the 2^lg chunks of 32 words of a row go to neighbouring warps; lane l updates word
// 32 chunk + l of its rows, and every cell raises the ring slot itself.
struct WordForm {
    static constexpr int THREADS = 1024;
    int m, la0, la_step;
    __device__ __forceinline__ void init(const Box& B) {
        const int warp = threadIdx.x >> 5;
        int lg = 0;
        while ((32 << lg) < B.PW) lg++;
        m = ((warp & ((1 << lg) - 1)) << 5) + (threadIdx.x & 31);
        la0 = 1 + (warp >> lg);
        la_step = (THREADS / 32) >> lg;
    }
    __device__ __forceinline__ void load(const Box&) {}
    __device__ __forceinline__ void settle(const Box&) {}
    __device__ __forceinline__ void drain(const Box&) {}
    __device__ __forceinline__ void end_step() { cluster_sync(); }
    static constexpr bool WAITS = false;
    __device__ static bool odd_row(const Box&) { return false; }
    template <bool PAR, int c, bool REDUCE>
    __device__ __forceinline__ void step(const Box& B, int tau, unsigned t2) {
        for (int la = la0; la <= B.nb; la += la_step) {
            const int off = (c ^ (B.A0 + la)) & 1;              // b' of word 0 of this colour in the row
            const int b = off + 2 * m - 1;
            const unsigned diff = (unsigned)(tau - (B.A0 + la - 1) - b);
            if ((unsigned)b >= (unsigned)B.NK || diff >= t2) continue;
            const uint32_t f = B.info[c * B.ics + (la - 1) * B.PW + m];
            double dch = 0.0, pabs = 0.0;
            if (!(f & CF_SOLID)) {
                const int own = c * B.cs + la * B.PW + m;
                const double* n = B.phi + (c ^ 1) * B.cs + la * B.PW + m;
                const RowCoef R = row_coef(B, la);
                const double p = B.phi[own], pN = n[-B.PW], pS = n[B.PW], pW = n[off - 1], pE = n[off];
                double Bs = cone_sum(R, pN, pS, pW, pE), A = R.A, r = R.rA;
                if (f) Bs = cone_special(B, R, f, Bs, pN, pS, pW, pE, A, r);
                if (A > 0.0) {
                    const double x = B.recip && sum_ok(Bs) ? quot(Bs, A, r) : Bs / A;
                    const double pn = p + CONE_OMEGA * (x - p);
                    B.phi[own] = pn;
                    if (la == 1 && B.push_n) B.push_n[c * B.cs + m] = pn;
                    if (la == B.nb && B.push_s) B.push_s[c * B.cs + m] = pn;
                    dch = fabs(pn - p);
                    pabs = fabs(pn);
                }
            }
            // the band's first cell of the sweep, alone in it here at this step, opens the slot
            if (REDUCE) raise(B, diff, la == 1 && m == 0, dch, pabs);
        }
    }
};

// Bands of 2 to 28 rows of at most 64 words a colour: a warp per row, a lane with four consecutive cells of it,
// b = 4 lane - 1 + {0, 1, 2, 3}, of which a step takes the two of its colour: those with even b' (phase 0)
// or odd b' (phase 1), in turn. The row's constants and the lane's four values stay in registers, so a cell's
// west and east neighbours are there or one lane away, and a step loads the rows to the north and south, two
// words each, and stores two.
//
// A sweep is in a word at phase 0, again at phase 1, then in the next word. So its largest change and |phi|
// over the row travel with it from word to word, and at the row's last word they raise the band's ring slot:
// row la one step after row la - 1, so plain loads and stores do (each cell raising the slot by atomics took more
// instructions than its update: on 64 bits of shared memory they are loops, and the changes grow along a
// sweep more often than not).
//
// The block's barrier ends a step. Only the warps of the band's edge rows wait for a neighbour: each stores its
// row there every step with st.async, which counts the bytes on the neighbour's barrier of that side and
// colour, and waits for the neighbour's row before its own next step (two barriers a side: a row of
// one colour is sent only after the neighbour's row of the other colour arrived, so a phase is over before the
// next one's bytes come). A cluster barrier for each step took 725 cycles, more than the step's work.
//
// A wait gives up after B.polls polls (the blocks of a cluster run together, so a row is at most a few polls
// away). The warp then goes on without waiting, so that no other waits for it, until the stopping test, where
// every block of the cluster learns of it and the level's solve ends.
struct RowForm {
    static constexpr bool WAITS = true;
    static constexpr int ROWS = CONE_ROWS, THREADS = 32 * ROWS, WORDS = CONE_WORDS;
    double val[2][2];                    // [phase][word]
    double md[2], mp[2];                 // largest change and |phi| of the sweep in each word
    RowCoef R;
    int start[2][2];                     // the step of a cell's first sweep (never, for a cell the sweeps skip)
    unsigned special;                    // bit 2 P + w: the cell is a special one
    int q[2];                            // the lane's two words of each phase, in phi
    unsigned push, bar_there, bar_here;  // edge rows: the neighbour's copy of them (colour 0), the barriers (colour 0)
    unsigned phases;                     // parity of each colour's barrier
    int e0, la, lane, waiting;           // waiting: colour of the neighbour's row not waited for yet, or -1
    bool row_ok, edge, dead;
    __device__ __forceinline__ void init(const Box& B) {
        lane = threadIdx.x & 31;
        la = 1 + (threadIdx.x >> 5);
        row_ok = la <= B.nb;
        if (!row_ok) la = 1;
        const int m = 2 * lane;
        const int par = (B.A0 + la) & 1;
        R = row_coef(B, la);
        const int m_end = B.NK >> 1;     // the row's last word, at b = 2 m (or past the last cell, b = NK)
        special = 0;
        e0 = lane == (m_end >> 1) ? B.A0 + la - 1 + 2 * m_end : INT_MAX;
#pragma unroll
        for (int P = 0; P < 2; P++) {
            const int c = P ^ par;
            q[P] = c * B.cs + la * WORDS + m;
#pragma unroll
            for (int w = 0; w < 2; w++) {
                const int b = 4 * lane + 2 * w + P - 1;
                uint32_t x = CF_SOLID;
                if (row_ok && b >= 0 && b < B.NK) x = B.info[c * B.ics + (la - 1) * WORDS + m + w];
                const double A = x & CF_WALL ? B.tab[2 * (x >> 6)] : R.A;
                const bool skip = (x & CF_SOLID) || !(A > 0.0);
                start[P][w] = skip ? INT_MIN : B.A0 + la - 1 + b;
                if (!skip && ((x & CF_WALL) || (B.div && (x & CF_NEAR)))) special |= 1u << (2 * P + w);
            }
        }
        md[0] = md[1] = mp[0] = mp[1] = 0.0;
        double* to = la == 1 ? B.push_n : la == B.nb ? B.push_s : nullptr;      // a band has two rows at least
        edge = row_ok && to;
        if (edge) {
            push = (unsigned)__cvta_generic_to_shared(to) + 8 * m;
            bar_there = la == 1 ? B.bar_n : B.bar_s;
            bar_here = (unsigned)__cvta_generic_to_shared(&B.waits->bar[2 * side()]);
        }
        waiting = -1;
        load(B);
    }
    __device__ __forceinline__ void load(const Box& B) {
#pragma unroll
        for (int P = 0; P < 2; P++) {
            const double2 x = *reinterpret_cast<const double2*>(B.phi + q[P]);
            val[P][0] = x.x;
            val[P][1] = x.y;
        }
    }
    __device__ __forceinline__ int side() const { return la == 1 ? 0 : 1; }
    __device__ static bool poll(unsigned bar, unsigned parity, int polls) {
        unsigned done = 0;
        for (int tries = 0; !done && tries < polls; tries++)
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                         " selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        return done;
    }
    __device__ __forceinline__ void expect(unsigned bar, int rows) {
        if (lane == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(8 * WORDS * rows) : "memory");
    }
    // waits for the neighbour's row of the last step, until a wait has given up
    __device__ __forceinline__ void settle(const Box& B) {
        if (waiting < 0) return;
        if (dead) {
            if (lane == 0) B.waits->owed[2 * side() + waiting]++;
        } else {
            expect(bar_here + 8 * waiting, 1);
            const bool came = poll(bar_here + 8 * waiting, (phases >> waiting) & 1, B.polls);
            dead = __any_sync(0xffffffffu, !came);
            if (!dead) phases ^= 1u << waiting;
            else if (lane == 0) {
                B.waits->gave[side()] = waiting;
                B.waits->lost = 1;
            }
        }
        waiting = -1;
    }
    // After a wait has given up and every block has taken its last step: takes the rows that are still
    // under way, which may land in this block's memory until then.
    __device__ __forceinline__ void drain(const Box& B) {
        if (!edge || !dead) return;
#pragma unroll 1
        for (int c = 0; c < 2; c++) {
            const unsigned b = bar_here + 8 * c;
            unsigned ph = (phases >> c) & 1;
            if (B.waits->gave[side()] == c) {
                poll(b, ph, DRAIN_POLLS);
                ph ^= 1;
            }
            const int rows = B.waits->owed[2 * side() + c];
            if (rows > 0) {
                expect(b, rows);
                poll(b, ph, DRAIN_POLLS);
            }
        }
    }
    template <int P, int c, bool REDUCE>
    __device__ __forceinline__ void phase(const Box& B, int tau, unsigned t2) {
        if (edge) settle(B);
        const double2 n = *reinterpret_cast<const double2*>(B.phi + q[1 - P] - WORDS);
        const double2 s = *reinterpret_cast<const double2*>(B.phi + q[1 - P] + WORDS);
        const double(&o)[2] = val[1 - P];
        double W[2], E[2];
        if (P == 0) {
            W[0] = __shfl_up_sync(0xffffffffu, o[1], 1); E[0] = o[0];
            W[1] = o[0]; E[1] = o[1];
            if (REDUCE) {
                const double d = __shfl_up_sync(0xffffffffu, md[1], 1), x = __shfl_up_sync(0xffffffffu, mp[1], 1);
                md[1] = md[0]; mp[1] = mp[0];
                md[0] = lane == 0 ? 0.0 : d;
                mp[0] = lane == 0 ? 0.0 : x;
            }
        } else {
            W[0] = o[0]; E[0] = o[1];
            W[1] = o[1]; E[1] = __shfl_down_sync(0xffffffffu, o[0], 1);
        }
        double Bs[2] = {cone_sum(R, n.x, s.x, W[0], E[0]), cone_sum(R, n.y, s.y, W[1], E[1])};
        double A[2] = {R.A, R.A}, r[2] = {R.rA, R.rA}, x[2];
        if (special & (3u << (2 * P))) {
            const uint32_t* f = B.info + c * B.ics + (la - 1) * WORDS + 2 * lane;
            if (special & (1u << (2 * P))) Bs[0] = cone_special(B, R, f[0], Bs[0], n.x, s.x, W[0], E[0], A[0], r[0]);
            if (special & (2u << (2 * P))) Bs[1] = cone_special(B, R, f[1], Bs[1], n.y, s.y, W[1], E[1], A[1], r[1]);
        }
        const bool act[2] = {(unsigned)tau - (unsigned)start[P][0] < t2, (unsigned)tau - (unsigned)start[P][1] < t2};
        x[0] = quot(Bs[0], A[0], r[0]);
        x[1] = quot(Bs[1], A[1], r[1]);
        if ((act[0] && !(B.recip && sum_ok(Bs[0]))) || (act[1] && !(B.recip && sum_ok(Bs[1])))) {
            x[0] = Bs[0] / A[0];
            x[1] = Bs[1] / A[1];
        }
#pragma unroll
        for (int w = 0; w < 2; w++) {
            const double p = val[P][w], pn = p + CONE_OMEGA * (x[w] - p);
            if (REDUCE) {
                const double dch = fabs(pn - p), pabs = fabs(pn);
                md[w] = act[w] && dch > md[w] ? dch : md[w];
                mp[w] = act[w] && pabs > mp[w] ? pabs : mp[w];
            }
            val[P][w] = act[w] ? pn : p;
        }
        *reinterpret_cast<double2*>(B.phi + q[P]) = make_double2(val[P][0], val[P][1]);
        if (edge) {
            asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];"
                         :: "r"(push + 8 * c * B.cs), "d"(val[P][0]), "d"(val[P][1]), "r"(bar_there + 8 * c) : "memory");
            waiting = c;
        }
        if (REDUCE && P == 1 && tau >= e0 && (unsigned)(tau - e0) < t2) {
            double2* slot = reinterpret_cast<double2*>(B.ring + 2 * ((((tau - e0) >> 1) + 1) & (B.R - 1)));
            double2 cur = la == 1 ? make_double2(0.0, 0.0) : *slot;
            const double d = (B.NK >> 1) & 1 ? md[1] : md[0], y = (B.NK >> 1) & 1 ? mp[1] : mp[0];
            if (d > cur.x) cur.x = d;
            if (y > cur.y) cur.y = y;
            *slot = cur;
        }
    }
    // the warp's row begins with phase 1: warps of such rows take their own copy of the solve
    __device__ static bool odd_row(const Box& B) { return (B.A0 + 1 + (threadIdx.x >> 5)) & 1; }
    template <bool PAR, int c, bool REDUCE>
    __device__ __forceinline__ void step(const Box& B, int tau, unsigned t2) {
        if (row_ok) phase<c ^ (int)PAR, c, REDUCE>(B, tau, t2);
    }
    __device__ __forceinline__ void end_step() { block_sync(); }
};

// s r D of a cell within H cells of the body: its 3-D face divergence with face values the
// average of the two cells and zero through a face to a solid cell (InitValues_Jup.cpp:1653-1664).
__device__ double cone_face_div(const ConeArgs& A, int i, int j, int k) {
    const size_t row = (size_t)A.jm * A.KP;
    const size_t c = ((size_t)i * A.jm + j) * A.KP + k;
    const double r = A.rad[i], rp = r + 0.5 * A.dr, rm = r - 0.5 * A.dr;
    const double sj = A.s[j], sp = 0.5 * (sj + A.s[j + 1]), sm = 0.5 * (sj + A.s[j - 1]);
    const double up = A.solid[c + row] ? 0.0 : 0.5 * (A.u[c] + A.u[c + row]);
    const double um = A.solid[c - row] ? 0.0 : 0.5 * (A.u[c] + A.u[c - row]);
    const double vp = A.solid[c + A.KP] ? 0.0 : 0.5 * (A.v[c] + A.v[c + A.KP]);
    const double vm = A.solid[c - A.KP] ? 0.0 : 0.5 * (A.v[c] + A.v[c - A.KP]);
    const double wp = A.solid[c + 1] ? 0.0 : 0.5 * (A.w[c] + A.w[c + 1]);
    const double wm = A.solid[c - 1] ? 0.0 : 0.5 * (A.w[c] + A.w[c - 1]);
    return sj * r * (rp * rp * up - rm * rm * um) / (r * r * A.dr) + (sp * vp - sm * vm) / A.dthe +
           (wp - wm) / A.dphi;
}

// the band and the rows beside it, 0..nb+1 of both colours, between phi (colour stride cs) and a packed
// copy [2][nb + 2][PW] (to_packed) or back
__device__ void band_copy(double* phi, int cs, double* packed, int nb, int PW, bool to_packed) {
    const int n = (nb + 2) * PW;
    for (int col = 0; col < 2; col++)
        for (int x = threadIdx.x; x < n; x += blockDim.x) {
            if (to_packed) packed[col * n + x] = phi[col * cs + x];
            else phi[col * cs + x] = packed[col * n + x];
        }
}

// a wait of some block of the cluster has given up (after a cluster barrier)
__device__ __forceinline__ bool cluster_lost(const Box& B, int C) {
    cg::cluster_group cl = cg::this_cluster();
    int any = 0;
    for (int r = 0; r < C; r++) any |= *cl.map_shared_rank(&B.waits->lost, r);
    return any;
}

// Lexicographic SOR of one level's solve as the pipelined wavefront on the cluster; returns the
// reference's sweep count `it` (the converged sweep, or CONE_MAXIT + 1 without convergence), or -1 in every
// block when a neighbour's row did not come.
// snap: this block's snapshot ring, n_snap slots of 2 (nbmax + 2) PW doubles.
template <class Form, bool PAR>
__device__ __forceinline__ int cone_sor(const Box& B, Form& T, double* snap, int slot_sz, int n_snap, int* snap_tag, int* t_found, int C) {
    cg::cluster_group cl = cg::this_cluster();
    const int lane = threadIdx.x & 31;
    cluster_sync();              // the cluster's blocks hold their start: a neighbour may store its edge row here
    band_copy(B.phi, B.cs, snap, B.nb, B.PW, true);
    if (threadIdx.x == 0) {
        snap_tag[0] = -1;
        for (int s = 1; s < n_snap; s++) snap_tag[s] = INT_MIN;
    }
    cluster_sync();
    T.init(B);
    int next = 1 % n_snap, t_conv = 0, t_next = 1, it = CONE_MAXIT + 1;
    for (int tau = 1;; tau += 2) {
        T.template step<PAR, 0, true>(B, tau - 1, 2u * CONE_MAXIT);
        T.end_step();
        T.template step<PAR, 1, true>(B, tau, 2u * CONE_MAXIT);
        T.end_step();
        // a sweep's last raise comes up to one step after its last cell
        if (tau > B.D && (tau & (CHECK_STEPS - 1)) == CHECK_STEPS - 1) {
            // the sweeps t_next..t_done are complete, at most CHECK_STEPS / 2 of them: lane 4 q + r of
            // the first warp reads block r's slot of sweep t_next + q
            const int t_done = min((tau - B.D - 1) / 2 + 1, CONE_MAXIT);
            cluster_sync();      // the blocks' ring slots are theirs to read
            if (threadIdx.x < 32) {
                const int t = t_next + (lane >> 2);
                double dmax = 0.0, pmax = 0.0;
                if (t <= t_done && (lane & 3) < C) {
                    const double2 sl = *reinterpret_cast<const double2*>(
                        cl.map_shared_rank(B.ring + 2 * (t & (B.R - 1)), lane & 3));
                    dmax = sl.x;
                    pmax = sl.y;
                }
                for (int o = 1; o < 4; o <<= 1) {
                    dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
                    pmax = fmax(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
                }
                const unsigned conv = __ballot_sync(0xffffffffu, t <= t_done && dmax <= CONE_TOL * fmax(pmax, 1.0e-30));
                bool lost = false;
                if constexpr (Form::WAITS)
                    lost = __any_sync(0xffffffffu, lane < C && *cl.map_shared_rank(&B.waits->lost, lane < C ? lane : 0));
                if (lane == 0) *t_found = lost ? -1 : conv ? t_next + ((__ffs(conv) - 1) >> 2) : 0;
            }
            block_sync();
            t_conv = *t_found;
            if (t_conv != 0) break;
            t_next = t_done + 1;
            if (t_done == CONE_MAXIT) break;
        }
        if (tau % SNAP_EVERY == SNAP_EVERY - 1) {
            T.settle(B);
            block_sync();
            band_copy(B.phi, B.cs, snap + (size_t)next * slot_sz, B.nb, B.PW, true);
            if (threadIdx.x == 0) snap_tag[next] = tau;
            next = (next + 1) % n_snap;
            cluster_sync();      // the copies of the neighbours' rows are saved before the next step's stores
        }
    }
    T.settle(B);
    block_sync();
    if (t_conv > 0) {
        // back to the newest snapshot in which no cell is past sweep t_conv (the same slot in
        // every block), then replay with the sweeps capped at t_conv up to the step that
        // completes it
        it = t_conv;
        const int target = 2 * (t_conv - 1), tau_c = B.D + 2 * (t_conv - 1);
        int best = 0, btag = INT_MIN;
        for (int s = 0; s < n_snap; s++)
            if (snap_tag[s] != INT_MIN && snap_tag[s] <= target && snap_tag[s] > btag) { best = s; btag = snap_tag[s]; }
        band_copy(B.phi, B.cs, snap + (size_t)best * slot_sz, B.nb, B.PW, false);
        cluster_sync();
        T.load(B);
        for (int tau = btag + 1; tau <= tau_c; tau += 2) {     // from an even step; one past tau_c changes nothing
            T.template step<PAR, 0, false>(B, tau, 2u * t_conv);
            T.end_step();
            T.template step<PAR, 1, false>(B, tau + 1, 2u * t_conv);
            T.end_step();
        }
        T.settle(B);
        block_sync();
    }
    if constexpr (Form::WAITS) {
        cluster_sync();          // the blocks' last waits are over
        if (cluster_lost(B, C)) it = -1;
    }
    return it;
}

// SMEM: phi, flags and constants of the band in shared memory; else one block per level on HBM
template <bool SMEM, class Form>
__global__ void __launch_bounds__(Form::THREADS, 1) cone_kernel(ConeArgs A) {
    extern __shared__ __align__(16) unsigned char cone_smem[];
    __shared__ int snap_tag[64], t_found;
    cg::cluster_group cl = cg::this_cluster();
    const int C = A.C;
    const int r = (int)cl.block_rank();
    const int lvl = blockIdx.x / C;
    const ConeLevel L = A.lv[lvl];
    const int NJ = L.NJ, NK = L.NK, PW = L.PW, i = L.i;
    const int A0 = (r * NJ) / C, nb = ((r + 1) * NJ) / C - A0, nbmax = (NJ + C - 1) / C;
    Box B;
    B.NJ = NJ; B.NK = NK; B.PW = PW; B.D = L.D; B.R = L.ring;
    B.nb = nb; B.A0 = A0;
    B.dthe = A.dthe; B.dphi = A.dphi;
    B.ring = reinterpret_cast<unsigned long long*>(cone_smem);
    double* phi_local = reinterpret_cast<double*>(B.ring + 2 * A.ring_max);
    double *rows, *tab;
    B.push_n = B.push_s = nullptr;
    __shared__ RowWaits waits;
    Form T;
    if constexpr (Form::WAITS) {
        B.waits = &waits;
        B.polls = A.polls;
        T.phases = 0;
        T.dead = false;
        if (threadIdx.x == 0) {
            for (int x = 0; x < 4; x++) {
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((unsigned)__cvta_generic_to_shared(&waits.bar[x])) : "memory");
                waits.owed[x] = 0;
            }
            waits.gave[0] = waits.gave[1] = -1;
            waits.lost = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        // a row stored in the neighbour to the north is that block's southern one
        if (r > 0) B.bar_n = (unsigned)__cvta_generic_to_shared(cl.map_shared_rank(waits.bar + 2, r - 1));
        if (r < C - 1) B.bar_s = (unsigned)__cvta_generic_to_shared(cl.map_shared_rank(waits.bar, r + 1));
    }
    if constexpr (SMEM) {
        B.cs = (nbmax + 2) * PW;
        rows = phi_local + 2 * B.cs;
        tab = rows + NROW * NJ;
        uint32_t* inf = reinterpret_cast<uint32_t*>(tab + L.n_tab);
        B.ics = nbmax * PW;
        for (int x = threadIdx.x; x < 2 * nb * PW; x += blockDim.x) {
            const int col = x / (nb * PW), rr = x - col * nb * PW;
            inf[col * B.ics + rr] = A.info[L.info_off + (size_t)col * NJ * PW + (size_t)A0 * PW + rr];
        }
        B.info = inf;
        if (r > 0) B.push_n = cl.map_shared_rank(phi_local + (A0 - ((r - 1) * NJ) / C + 1) * PW, r - 1);
        if (r < C - 1) B.push_s = cl.map_shared_rank(phi_local, r + 1);
    } else {
        // one block per level: phi in place in the warm-start buffer, the rest in HBM
        B.cs = (NJ + 2) * PW;
        rows = A.rows + L.row_off;
        tab = A.tab + L.tab_off;
        B.ics = NJ * PW;
        B.info = A.info + L.info_off;
    }
    B.tab = tab;
    B.rows = rows;
    // the row coefficients (InitValues_Jup.cpp:1733-1735) and A of a cell with four fluid faces
    bool recip = true;
    for (int a = threadIdx.x; a < NJ; a += blockDim.x) {
        const int j = L.jlo + a;
        const double sj = A.s[j];
        const double aN = 0.5 * (sj + A.s[j - 1]) / (A.dthe * A.dthe);
        const double aS = 0.5 * (sj + A.s[j + 1]) / (A.dthe * A.dthe);
        const double aL = 1.0 / (sj * A.dphi * A.dphi);
        double a4 = 0.0;
        a4 += aN;
        a4 += aS;
        a4 += aL;
        a4 += aL;
        double* rc = rows + (size_t)a * NROW;
        rc[RC_N] = aN;
        rc[RC_S] = aS;
        rc[RC_L] = aL;
        rc[RC_A] = a4;
        rc[RC_RA] = rcp_of(a4);
        rc[RC_SJ] = sj;
        rc[RC_SD] = sj * A.dphi;
        recip = recip && aN > 0.0 && aS > 0.0 && aL > 0.0 && quot_ok(1.0, aN) && quot_ok(1.0, aS) && quot_ok(1.0, aL) && quot_ok(1.0, a4);
    }
    B.recip = __syncthreads_and(recip) != 0;
    const int32_t* spec = A.spec + L.spec_off;
    const int slot_sz = 2 * (nbmax + 2) * PW;
    double* snap = A.snap + L.snap_off + (size_t)r * L.n_snap * slot_sz;
    if (A.H == 0 && r == 0 && threadIdx.x == 0) A.stats[2 * lvl] = 0;
    for (int pass = A.H > 0 ? 0 : 1; pass < 2; pass++) {
        B.div = pass == 0;
        double* prev = (B.div ? A.prev0 : A.prev1) + L.phi_off;
        if constexpr (SMEM) {
            // the band with the rows beside it (zero at the box's halo)
            B.phi = phi_local;
            for (int col = 0; col < 2; col++)
                for (int x = threadIdx.x; x < (nb + 2) * PW; x += blockDim.x)
                    phi_local[col * B.cs + x] = prev[(size_t)col * (NJ + 2) * PW + (size_t)A0 * PW + x];
        } else {
            B.phi = prev + (size_t)A0 * PW;
        }
        // the per-cell constants of the band: the source of the divergence solve from the flow
        // before it, the wall-face velocities of the wall-flux solve from the flow it starts from
        __syncthreads();
        for (int x = threadIdx.x; x < L.n_spec; x += blockDim.x) {
            const int e = spec[x], mm = e % PW, rw = e / PW, a = rw % NJ, cc = rw / NJ;
            if (a < A0 || a >= A0 + nb) continue;
            const int b = ((cc ^ (a + 1)) & 1) + 2 * mm - 1;
            const int j = L.jlo + a, k = L.klo + b;
            const uint32_t f = A.info[L.info_off + e];
            double* t = tab + 2 * (f >> 6);
            const double src = B.div && (f & CF_NEAR) ? cone_face_div(A, i, j, k) : 0.0;
            if (!(f & CF_WALL)) { t[0] = src; continue; }
            const double* rc = rows + (size_t)a * NROW;
            double sum = 0.0;
            if (!(f & CF_N)) sum += rc[RC_N];
            if (!(f & CF_S)) sum += rc[RC_S];
            if (!(f & CF_W)) sum += rc[RC_L];
            if (!(f & CF_E)) sum += rc[RC_L];
            t[0] = sum;
            t[1] = rcp_of(sum);
            const size_t cix = ((size_t)i * A.jm + j) * A.KP + k;
            const double vp = A.v[cix], wp = A.w[cix], sj = rc[RC_SJ];
            t[2] = B.div ? 0.0 : -(rc[RC_N] * A.dthe * (-vp));
            t[3] = B.div ? 0.0 : -(rc[RC_S] * A.dthe * (vp));
            t[4] = B.div ? 0.0 : -(rc[RC_L] * sj * A.dphi * (-wp));
            t[5] = B.div ? 0.0 : -(rc[RC_L] * sj * A.dphi * (wp));
            t[6] = src;
        }
        const int it = Form::odd_row(B) ? cone_sor<Form, true>(B, T, snap, slot_sz, L.n_snap, snap_tag, &t_found, C)
                                        : cone_sor<Form, false>(B, T, snap, slot_sz, L.n_snap, snap_tag, &t_found, C);
        __syncthreads();
        if (Form::WAITS && it < 0) {
            // The level has no result: its winds are NaN, as the Runge-Kutta stage marks cells whose inputs did
            // not come, and the warm start stays the last call's.
            T.drain(B);
            const double nan = __longlong_as_double(0x7ff8000000000000ll);
            for (int x = threadIdx.x; x < nb * NK; x += blockDim.x) {
                const int la = 1 + x / NK, a = A0 + la - 1, bp = x % NK + 1;
                const int cc = (a + 1 + bp) & 1;
                if (B.info[cc * B.ics + (la - 1) * PW + (bp >> 1)] & CF_SOLID) continue;
                const size_t cix = ((size_t)i * A.jm + (L.jlo + a)) * A.KP + (L.klo + bp - 1);
                A.v[cix] = A.w[cix] = nan;
            }
            if (r == 0 && threadIdx.x == 0)
                for (int q = pass; q < 2; q++) A.stats[2 * lvl + q] = -1;
            cl.sync();           // the flags of every block are read
            return;
        }
        // v and w of the band incremented by the average of the two face corrections
        // (InitValues_Jup.cpp:1785-1793), a wall face's correction being minus the cell's velocity
        for (int x = threadIdx.x; x < nb * NK; x += blockDim.x) {
            const int la = 1 + x / NK, b = x - (la - 1) * NK;
            const int a = A0 + la - 1, bp = b + 1;
            const uint32_t inf = B.info[((a + b) & 1) * B.ics + (la - 1) * PW + (bp >> 1)];
            if (inf & CF_SOLID) continue;
            const size_t cix = ((size_t)i * A.jm + (L.jlo + a)) * A.KP + (L.klo + b);
            const double vp = A.v[cix], wp = A.w[cix], pp = phi_at(B, la, bp);
            const double sd = rows[(size_t)a * NROW + RC_SD];
            const double dN = (inf & CF_N) ? -vp : (pp - phi_at(B, la - 1, bp)) / A.dthe;
            const double dS = (inf & CF_S) ? -vp : (phi_at(B, la + 1, bp) - pp) / A.dthe;
            const double dW = (inf & CF_W) ? -wp : (pp - phi_at(B, la, bp - 1)) / sd;
            const double dE = (inf & CF_E) ? -wp : (phi_at(B, la, bp + 1) - pp) / sd;
            A.v[cix] = vp + 0.5 * (dN + dS);
            A.w[cix] = wp + 0.5 * (dW + dE);
        }
        // the band's phi is the warm start of the next call
        if constexpr (SMEM)
            for (int x = threadIdx.x; x < 2 * nb * PW; x += blockDim.x) {
                const int col = x / (nb * PW), rr = x - col * nb * PW;
                prev[(size_t)col * (NJ + 2) * PW + (size_t)(A0 + 1) * PW + rr] = phi_local[col * B.cs + PW + rr];
            }
        if (r == 0 && threadIdx.x == 0) A.stats[2 * lvl + pass] = it;
        // every block is past its last store to a neighbour, and the warm start is read after it is whole
        cl.sync();
    }
}

// the seam copy: v and w of k = km-1 from k = 0 in every (i, j) row (InitValues_Jup.cpp:1806-1807)
__global__ void cone_seam_kernel(double* v, double* w, int rows, int km, int KP) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    v[(size_t)r * KP + km - 1] = v[(size_t)r * KP];
    w[(size_t)r * KP + km - 1] = w[(size_t)r * KP];
}

}  // namespace

void cone_free(AtjupCtx* c) {
    ConeState* cs = static_cast<ConeState*>(c->cone);
    if (!cs) return;
    cudaFree(cs->d_lv);
    cudaFree(cs->info);
    cudaFree(cs->spec);
    cudaFree(cs->prev[0]);
    cudaFree(cs->prev[1]);
    cudaFree(cs->snap);
    cudaFree(cs->tab);
    cudaFree(cs->rows);
    cudaFree(cs->s);
    cudaFree(cs->stats);
    delete cs;
    c->cone = nullptr;
}

// The static part, once per grid: the levels that cut the obstacle with their boxes, the cell
// flags (solid, solid neighbours along j and k, within H cells of the body), the list of cells
// that carry a constant (wall or near cells), and the buffers: the warm starts of both solves
// (zero until the first call, as the reference's per-level phi_prev), the snapshots, the stats.
// The solid mask and sin(the_j) are read back from the device copies set_grid made.
int cone_prepare(AtjupCtx* c) {
    if (c->cone) return ATJUP_OK;
    if (!c->grid_set) { set_error("cone projection: set_grid first"); return ATJUP_ERR_ARG; }
    const AtjupParams& P = c->P;
    if (P.cone_proj_margin < 0 || P.cone_proj_div < 0) {
        set_error("cone projection: margin and div must be >= 0");
        return ATJUP_ERR_ARG;
    }
    const int im = P.im, jm = P.jm, km = P.km, KP = c->KP;
    std::vector<uint8_t> sol(c->NP);
    std::vector<double> sinthe(jm);
    ATJUP_CUDA(cudaMemcpyAsync(sol.data(), c->solid, c->NP, cudaMemcpyDeviceToHost, c->stream));
    ATJUP_CUDA(cudaMemcpyAsync(sinthe.data(), c->sin_the, sizeof(double) * jm, cudaMemcpyDeviceToHost, c->stream));
    ATJUP_CUDA(cudaStreamSynchronize(c->stream));
    auto S = [&](int i, int j, int k) { return sol[((size_t)i * jm + j) * KP + k] != 0; };
    std::vector<double> s(jm);
    for (int j = 0; j < jm; j++) s[j] = std::max(P.sinthe_min, std::fabs(sinthe[j]));
    const int H = P.cone_proj_div, M = P.cone_proj_margin;
    // within H cells (Chebyshev, 3-D, clipped to the grid) of a solid cell: a separable dilation
    // of the solid mask along k, j and i (InitValues_Jup.cpp:1634-1646)
    const size_t N = (size_t)im * jm * km;
    std::vector<uint8_t> near;
    if (H > 0) {
        std::vector<uint8_t> a(N), b(N);
        for (int i = 0; i < im; i++)
            for (int j = 0; j < jm; j++)
                for (int k = 0; k < km; k++) a[((size_t)i * jm + j) * km + k] = S(i, j, k);
        auto dilate = [&](const std::vector<uint8_t>& in, std::vector<uint8_t>& out, int axis) {
            const int n[3] = {im, jm, km};
            const size_t stride[3] = {(size_t)jm * km, (size_t)km, 1};
            for (int i = 0; i < im; i++)
                for (int j = 0; j < jm; j++)
                    for (int k = 0; k < km; k++) {
                        const int x[3] = {i, j, k};
                        const size_t at = ((size_t)i * jm + j) * km + k;
                        uint8_t v = 0;
                        for (int d = -H; d <= H && !v; d++) {
                            const int y = x[axis] + d;
                            if (y >= 0 && y < n[axis]) v = in[at + (ptrdiff_t)d * (ptrdiff_t)stride[axis]];
                        }
                        out[at] = v;
                    }
        };
        dilate(a, b, 2);
        dilate(b, a, 1);
        dilate(a, b, 0);
        near.swap(b);
    }
    auto* cs = new ConeState();
    cs->H = H;
    cs->M = M;
    // the boxes, and the flags of their cells row by row
    std::vector<std::vector<uint32_t>> flags;
    std::vector<ConeBox> boxes;
    for (int i = 1; i < im - 1; i++) {
        int jmin = jm, jmax = -1, kmin = km, kmax = -1;
        for (int j = 0; j < jm; j++)
            for (int k = 0; k < km; k++)
                if (S(i, j, k)) {
                    jmin = std::min(jmin, j); jmax = std::max(jmax, j);
                    kmin = std::min(kmin, k); kmax = std::max(kmax, k);
                }
        if (jmax < 0) continue;                      // above the body
        const int jlo = std::max(1, jmin - M), jhi = std::min(jm - 2, jmax + M);
        const int klo = std::max(1, kmin - M), khi = std::min(km - 2, kmax + M);
        if (jhi < jlo || khi < klo) continue;        // no cell in the box
        ConeLevel L{};
        L.i = i; L.jlo = jlo; L.klo = klo;
        L.NJ = jhi - jlo + 1; L.NK = khi - klo + 1;
        L.PW = (L.NK + 3) / 2;                       // words per row and colour, halo included
        L.D = L.NJ + L.NK - 2;
        L.ring = 1;
        // a power of two above the sweeps in flight and those that wait for their stopping test
        while (L.ring < L.D / 2 + 4 + CHECK_STEPS / 2) L.ring <<= 1;
        L.n_snap = (L.D + SNAP_EVERY) / SNAP_EVERY + 2;
        if (L.n_snap > 64 || L.PW > 32 * 32) {
            delete cs;
            set_error("cone projection: box too large");
            return ATJUP_ERR_UNSUPPORTED;
        }
        std::vector<uint32_t> fl((size_t)L.NJ * L.NK);
        for (int a = 0; a < L.NJ; a++)
            for (int b = 0; b < L.NK; b++) {
                const int j = jlo + a, k = klo + b;
                uint32_t f = 0;
                if (S(i, j, k)) f = CF_SOLID;
                else {
                    if (S(i, j - 1, k)) f |= CF_N;
                    if (S(i, j + 1, k)) f |= CF_S;
                    if (S(i, j, k - 1)) f |= CF_W;
                    if (S(i, j, k + 1)) f |= CF_E;
                    if (H > 0 && near[((size_t)i * jm + j) * km + k]) f |= CF_NEAR;
                    if (f) {
                        const int entry = f & CF_WALL ? TAB_WALL : TAB_NEAR;
                        f |= (uint32_t)(L.n_tab / 2) << 6;
                        L.n_tab += entry;
                        L.n_spec++;
                    }
                }
                fl[(size_t)a * L.NK + b] = f;
            }
        flags.push_back(std::move(fl));
        boxes.push_back(ConeBox{L.NJ, L.NK, L.ring, L.n_tab});
        cs->ring_max = std::max(cs->ring_max, L.ring);
        cs->lv.push_back(L);
    }
    c->cone = cs;
    const size_t nl = cs->lv.size();
    auto kernel_of = [](const ConePlan& p) {
        return p.row ? reinterpret_cast<const void*>(&cone_kernel<true, RowForm>)
                     : p.smem ? reinterpret_cast<const void*>(&cone_kernel<true, WordForm>)
                              : reinterpret_cast<const void*>(&cone_kernel<false, WordForm>);
    };
    // the most any plan takes, not this one's need: the limit is the kernel's, and another context's plan may take more
    auto allow = [&](const ConePlan& p) {
        return cudaFuncSetAttribute(kernel_of(p), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CONE_SMEM_CAP);
    };
    const ConePlan plan = cone_plan(boxes, [&](const ConePlan& p) {
        int n_active = 0;
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = p.C; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(nl * p.C));
        cfg.blockDim = dim3(p.threads);
        cfg.dynamicSmemBytes = p.bytes;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const bool ok = allow(p) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n_active, kernel_of(p), &cfg) == cudaSuccess && n_active >= (int)nl;
        if (!ok) cudaGetLastError();
        return ok;
    });
    cs->plan = plan;
    cs->kernel = kernel_of(plan);
    ATJUP_CUDA(allow(plan));
    // the buffers' layout at the form's words per row
    std::vector<uint32_t> info;
    std::vector<int32_t> spec;
    int64_t n_phi = 0, n_snap = 0, n_tab = 0, n_row = 0;
    for (size_t l = 0; l < nl; l++) {
        ConeLevel& L = cs->lv[l];
        L.PW = cone_words(boxes[l], plan.row);
        L.info_off = (int64_t)info.size();
        L.spec_off = (int64_t)spec.size();
        info.resize(info.size() + 2 * (size_t)L.NJ * L.PW, CF_SOLID);   // unused words: skipped
        for (int a = 0; a < L.NJ; a++)
            for (int b = 0; b < L.NK; b++) {
                const uint32_t f = flags[l][(size_t)a * L.NK + b];
                const int e = (((a + b) & 1) * L.NJ + a) * L.PW + ((b + 1) >> 1);
                info[L.info_off + e] = f;
                if (f & ~(uint32_t)CF_SOLID) spec.push_back(e);
            }
        L.phi_off = n_phi;  n_phi += 2 * (int64_t)(L.NJ + 2) * L.PW;
        L.tab_off = n_tab;  n_tab += L.n_tab;
        L.row_off = n_row;  n_row += NROW * (int64_t)L.NJ;
        const int64_t nbmax = (L.NJ + plan.C - 1) / plan.C;
        L.snap_off = n_snap;
        n_snap += (int64_t)plan.C * L.n_snap * 2 * (nbmax + 2) * L.PW;
    }
    ATJUP_CUDA(cudaMalloc(&cs->s, sizeof(double) * jm));
    ATJUP_CUDA(cudaMemcpy(cs->s, s.data(), sizeof(double) * jm, cudaMemcpyHostToDevice));
    ATJUP_CUDA(cudaMalloc(&cs->stats, sizeof(int) * 2 * std::max<size_t>(nl, 1)));
    ATJUP_CUDA(cudaMemset(cs->stats, 0, sizeof(int) * 2 * std::max<size_t>(nl, 1)));
    if (nl == 0) return ATJUP_OK;
    ATJUP_CUDA(cudaMalloc(&cs->d_lv, sizeof(ConeLevel) * nl));
    ATJUP_CUDA(cudaMemcpy(cs->d_lv, cs->lv.data(), sizeof(ConeLevel) * nl, cudaMemcpyHostToDevice));
    ATJUP_CUDA(cudaMalloc(&cs->info, sizeof(uint32_t) * info.size()));
    ATJUP_CUDA(cudaMemcpy(cs->info, info.data(), sizeof(uint32_t) * info.size(), cudaMemcpyHostToDevice));
    ATJUP_CUDA(cudaMalloc(&cs->spec, sizeof(int32_t) * std::max<size_t>(spec.size(), 1)));
    if (!spec.empty())
        ATJUP_CUDA(cudaMemcpy(cs->spec, spec.data(), sizeof(int32_t) * spec.size(), cudaMemcpyHostToDevice));
    for (double*& p : cs->prev) {
        ATJUP_CUDA(cudaMalloc(&p, sizeof(double) * n_phi));
        ATJUP_CUDA(cudaMemset(p, 0, sizeof(double) * n_phi));
    }
    ATJUP_CUDA(cudaMalloc(&cs->snap, sizeof(double) * n_snap));
    if (!plan.smem) {
        ATJUP_CUDA(cudaMalloc(&cs->tab, sizeof(double) * std::max<int64_t>(n_tab, 1)));
        ATJUP_CUDA(cudaMalloc(&cs->rows, sizeof(double) * n_row));
    }
    return ATJUP_OK;
}

// One in-loop projection on the context's stream (v and w in place).
int launch_cone_projection(AtjupCtx* c) {
    if (int rc = cone_prepare(c)) return rc;
    const AtjupParams& P = c->P;
    ConeState* cs = static_cast<ConeState*>(c->cone);
    if (!cs->lv.empty()) {
        ConeArgs A{};
        A.lv = cs->d_lv; A.info = cs->info; A.spec = cs->spec;
        A.prev0 = cs->prev[0]; A.prev1 = cs->prev[1]; A.snap = cs->snap;
        A.tab = cs->tab; A.rows = cs->rows; A.s = cs->s; A.stats = cs->stats;
        A.u = c->f[ATJUP_F_U]; A.v = c->f[ATJUP_F_V]; A.w = c->f[ATJUP_F_W];
        A.solid = c->solid; A.rad = c->rad;
        A.jm = P.jm; A.km = P.km; A.KP = c->KP; A.H = cs->H;
        A.C = cs->plan.C;
        A.ring_max = cs->ring_max;
        A.polls = c->cone_polls;
        A.dr = P.dr; A.dthe = P.dthe; A.dphi = P.dphi;
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs->plan.C; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(cs->lv.size() * cs->plan.C));
        cfg.blockDim = dim3(cs->plan.threads);
        cfg.dynamicSmemBytes = cs->plan.bytes;
        cfg.stream = c->stream;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        c->launches++;
        void* args[] = {&A};
        ATJUP_CUDA(cudaLaunchKernelExC(&cfg, cs->kernel, args));
        ATJUP_CHECK_LAUNCH("cone projection");
    }
    const int rows = P.im * P.jm;
    c->launches++;
    cone_seam_kernel<<<(rows + 255) / 256, 256, 0, c->stream>>>(c->f[ATJUP_F_V], c->f[ATJUP_F_W], rows, P.km, c->KP);
    ATJUP_CHECK_LAUNCH("cone seam");
    return ATJUP_OK;
}

}  // namespace atjup

using namespace atjup;

extern "C" {

int atjup_gpu_cone_project(AtjupCtx* c) {
    if (!c) return ATJUP_ERR_ARG;
    if (!c->grid_set) { set_error("cone_project: set_grid first"); return ATJUP_ERR_ARG; }
    return launch_cone_projection(c);
}

int atjup_gpu_cone_stats(AtjupCtx* c, int32_t* level_i, int32_t* sweeps, int32_t cap, int32_t* n_levels) {
    if (!c || !n_levels) return ATJUP_ERR_ARG;
    if (int rc = cone_prepare(c)) return rc;
    ConeState* cs = static_cast<ConeState*>(c->cone);
    const int nl = (int)cs->lv.size();
    *n_levels = nl;
    const int n = std::min(nl, std::max(cap, 0));
    if (n == 0) return ATJUP_OK;
    std::vector<int> st(2 * (size_t)nl);
    ATJUP_CUDA(cudaMemcpyAsync(st.data(), cs->stats, sizeof(int) * st.size(), cudaMemcpyDeviceToHost, c->stream));
    ATJUP_CUDA(cudaStreamSynchronize(c->stream));
    for (int l = 0; l < n; l++) {
        if (level_i) level_i[l] = cs->lv[l].i;
        if (sweeps) { sweeps[2 * l] = st[2 * l]; sweeps[2 * l + 1] = st[2 * l + 1]; }
    }
    for (int l = 0; l < nl; l++)
        if (st[2 * l] < 0 || st[2 * l + 1] < 0) {
            set_error("cone projection: a wait for a neighbour's row gave up on level " +
                      std::to_string(cs->lv[l].i) + "; its winds are NaN");
            return ATJUP_ERR_NONFINITE;
        }
    return ATJUP_OK;
}

int atjup_gpu_cone_wait_limit(AtjupCtx* c, int32_t polls) {
    if (!c || polls < 0) { set_error("cone_wait_limit: bad argument"); return ATJUP_ERR_ARG; }
    c->cone_polls = polls;
    return ATJUP_OK;
}

}  // extern "C"
