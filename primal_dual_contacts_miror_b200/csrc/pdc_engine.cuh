// The primal-dual interior-point Newton solve of one contact scene, executed by
// one thread block (CTA) with __syncthreads between phases.  A batched launch
// hands scenes to CTAs from an atomic work counter, so thousands of small,
// ragged scenes run concurrently on the 148 SMs of a B200, each scene's
// working set staying L1/L2 resident while its CTA iterates.
//
// Algorithm: the reference's PrimalDualForceSolver::fillForcesIntl
// (src/Solver/PrimalDual/PrimalDualForceSolver.cpp:167-511) with
// NonSmoothContactForce (src/Solver/PrimalDual/NonSmoothForces/NonSmoothContactForce.cpp:8-319).
// Differences in mechanism, not in the solution:
//  * the LDL^T solve (:385-394, < 2000 local bodies) is a sparse Cholesky
//    factorisation of 6x6 body blocks, assembled from the contacts' W = R K^-1 R^T
//    (6 doubles), up to 256 active bodies (block and warp teams) or 2048 (large
//    teams, unless the factor would be too deep);
//  * above that, and in place of AMGCL (:395-427), the system is never assembled:
//    block-Jacobi preconditioned CG, the product applied per contact and gathered
//    per body, converged to cfg.rtol_direct (direct branch) or cfg.rtol_iter with
//    the reference's AMGCL cap and Hu rule (iterative branch);
//  * the contact->body scatter, which the reference does with omp atomics
//    (NonSmoothContactForce.cpp:144,228,243), is a gather over per-body
//    incidence lists sorted by contact index, so results are bitwise
//    reproducible run to run.
#pragma once
#include "pdc_device.cuh"
#include "../../include/pdc.h"

namespace pdc {

struct EngineCfg {
    int max_iter;
    double tol;
    double mu;
    double mu_pair_lo, mu_pair_hi;  // per-pair friction when hi > lo
    unsigned long long mu_pair_seed;
    double restitution;
    int spring_based;
    int only_normal;   // OnlyNormalForce (OnlyNormalForce.cpp:7-217): 1-D force, no friction
    double compliance_coef;  // m_compliance numerator inputs
    double spring_k, spring_damp;
    int direct_threshold;
    int dense_max;  // direct branch: sparse Cholesky up to this many active bodies (<= kSparseMax)
    int dense_max_large;  // the same on the large-scene teams (<= kSparseMaxLarge)
    int warp_max_contacts;  // scenes up to this size are solved by one warp
    int warp_max_bodies;
    int grid_min_bodies;   // scenes with at least this many bodies are large
    int cluster_max_contacts;  // large scenes up to this many contacts go to a cluster team
    int cluster_max_bodies;    // ... if they have at most this many bodies
    int pcg_lanes;             // lanes per body in the PCG product (0: the team's default)
    int mixed;             // FP32 inner PCG + FP64 iterative refinement
    double inner_rtol;     // FP32 inner solve relative residual
    int max_outer;         // refinement steps before giving up
    double rtol_direct;
    int max_direct;
    double rtol_iter;
    int max_cg;
    int ls_max;  // line-search trials of a Newton step (PrimalDualForceSolver.cpp:437-440)
    int gd_max;  // ... and of the gradient-descent fallback (:454-456)
};

struct BatchPtrs {
    int n_scenes;
    int smem_blocks; // factor blocks that fit each thread block's dynamic shared memory
    int grid_large;  // the host launches the grid kernel for scenes >= grid_min_bodies
    // single-scene launch (body_off == nullptr): sizes and step passed by value
    int single_nb, single_nc;
    double single_dt, single_g[3];
    const int* __restrict__ body_off;
    const int* __restrict__ contact_off;
    const int* __restrict__ contact_cnt;  // optional: contacts used in each slice (else the slice size)
    const int* __restrict__ body_cnt;     // optional: bodies of each scene (else the slice size)
    const double* __restrict__ dt;
    const double* __restrict__ grav;
    // bodies (inputs)
    const double* __restrict__ vel;
    const double* __restrict__ ang;
    const double* __restrict__ mass;
    const double* __restrict__ inertia;
    const double* __restrict__ inv_inertia;
    const uint8_t* __restrict__ is_static;
    // contacts (inputs)
    const int* __restrict__ cbody;
    const double* __restrict__ frame;
    const double* __restrict__ arm;
    const double* __restrict__ depth;
    const double* __restrict__ cmu;
    // outputs
    double* dvel;
    double* dang;
    double* lforce;
    pdc_stats* stats;
    // per-body workspace
    int* inc_start;
    int* inc_cnt;
    int* inc_cur;
    uint8_t* local;
    // per scene: device time of its previous solve (ns; 0 = none), the planner's
    // longest-first key.  Null unless the handle keeps a history.
    unsigned int* cost = nullptr;
    int* lbody;    // the scene's local bodies (global index), ascending, in its body slice
    double* u;     // 6
    double* uold;  // 6
    double* du;    // 6
    double* r;     // 6
    double* z;     // 6
    double* p;     // 6
    double* p2;    // 6: PCG direction of the other parity
    double* q;     // 6: PCG A p
    double* rhs;   // 6
    double* ru;    // 6
    double* pinv;  // 21
    double* dsc;   // 6  Jacobi scale 1/sqrt(diag A) of the iterative branch
    // incidences of active bodies, in contact order per body, 2 per contact
    int* inc;       // contact << 1 | side
    int* inc_o;     // the other body (global index), -1 if static; the block and
                    // warp teams' factor keeps the block it adds to here
    int* inc_g;     // the incidences (slots) of each factor block, block by block
    int* islot;     // incidence index of (contact, side), -1 for a static side
    double* it;     // tiles of 32 incidences, kIncFields runs of 32 values each
    double* ct;     // tiles of 32 contacts, kFields runs of 32 values each
    // 12 side by side per incidence, for the body phases that read all of them:
    // W = R K^-1 R^T of its contact, packed (xx,yy,zz,xy,xz,yz), the lever arm of
    // its side, the lever arm of the other side
    double* G;
    // mixed precision (FP32 inner PCG): per-contact W and X, per-body vectors
    float* Wf;     // 6 per contact
    float* Xf;     // 3 per contact
    float* rF;     // 6 per body
    float* zF;
    float* pF;
    float* eF;
    float* pinvf;  // 21 per body
    int* didx;   // dense row-block of each active body
    int* dbody;  // body of each dense row-block (scene-relative slots)
    // per-team sparse-factorisation scratch (see SceneSolver::sparse_ws)
    double* dense;             // one slot per thread-block team (slot = block index)
    long long dense_stride;
    double* dense_warp;        // one slot per warp team (null: warp teams off)
    long long dense_stride_warp;
    // one slot for the large-scene teams (nullptr: they use PCG throughout)
    double* sparse_big = nullptr;
    long long sparse_big_doubles = 0;
    int* order_cta;   // scene queues written by plan_scenes_kernel
    int* order_warp;
    int* counts;      // [4]
    unsigned long long* timers;  // [4] ns: total, build, solve, line search
};

#define PDC_STATUS_BAD_INPUT 16

// Mixed precision tests its stop on the true residual in FP64, which rounding keeps
// above ~1e-14 |b|; the FP64 PCG's recurrence residual goes on below that (and has
// to: where the matrix is soft, stopping it at 1e-13 |b| leaves velocities 1e-5 off).
constexpr double kMixedRtolMin = 1e-13;

// Per-contact workspace: tiles of 32 contacts, one run of 32 values per field, so
// that a warp's loads and stores are coalesced and every field of a contact is
// a constant offset from one address.  (With a contact's components side by
// side, each of the ~60 loads per contact and phase touched up to 32 lines per
// warp, and the load-store unit bound the contact phases: 39 us per residual
// pass over 1,536 contacts; with one plane per component over the whole batch
// the ~60 addresses cost 3,900 bytes of register spills.)
enum ContactField {
    F_frame = 0,          // 9: copy of the input
    F_arm = 9,            // 6: lever arms of both sides (copy of the input)
    F_f = 15,             // 3
    F_lam = 18,           // 2
    F_fT = 20,            // 3: line-search trial, then 2: its multipliers
    F_lT = 23,
    F_fT2 = 25,           // the second trial of a pair
    F_lT2 = 28,
    F_df = 30,            // 3
    F_dl = 33,            // 2
    F_rf = 35,            // 3
    F_rl = 38,            // 2
    F_kn = 40,            // 1 (m_nonSmoothK normal slot)
    F_cv = 41,            // 2 constraint values
    F_gr = 43,            // 2 gradients
    F_hs = 45,            // 3 hessian (packed)
    F_tq = 48,            // 3: tangential-weight form T_t^T M^-1 T_t of both bodies (packed 2x2)
    F_wu = 51,            // 3: relative velocity J u at the iterate (line-search base)
    F_wd = 54,            // 3: J du of the search direction
    F_invC = 57,          // 2
    F_knInv = 59,         // 1
    F_ktInv = 60,         // 3 (packed symmetric inverse of K_t)
    F_sf = 63,            // 3
    kFields = 66
};
// Per-incidence workspace, in tiles of 32 likewise: sigma X of its contact (sigma
// = -1 on side 0, +1 on side 1), the lever arm of its side, and the X of the
// second line-search trial of a pair.
enum IncField { I_X = 0, I_arm = 3, I_X2 = 6, kIncFields = 9 };

// sparse direct solve: nodes per scene (bitset width)
constexpr int kSparseMax = 256;
constexpr int kSparseWords = kSparseMax / 32;
// off-diagonal factor blocks per scene: every pair of the kSparseMax nodes, so
// the direct branch never leaves the factor for lack of room (a settled heap of
// 256 boxes fills in to several thousand blocks)
constexpr int kRowCap = kSparseMax * (kSparseMax - 1) / 2;
// the same for a warp team, which takes scenes of at most kWarpMaxBodies bodies
constexpr int kWarpMaxBodies = 64;
constexpr int kRowCapWarp = kWarpMaxBodies * (kWarpMaxBodies - 1) / 2;
// doubles of a slot before its off-diagonal blocks: bitsets, index arrays, block
// descriptors and the node vector (the layout of SceneSolver::direct_ws), then the
// diagonal blocks, one per node, and two spare ones (a zero block and room to read
// past the last)
__host__ __device__ constexpr long long sparse_header_doubles(int off_diagonal) {
    return (4LL * (3LL * kSparseMax * kSparseWords + 12LL * (kSparseMax + 8)) + 16LL * (off_diagonal + kSparseMax + 2) +
            8LL * (6 * (kSparseMax + 2) + 36 * (kSparseMax + 2)) + 255) / 256 * 32;
}
// Levels whose update lists (column patterns) have at most this many entries
// are updated by a thread per row (substituted backward entry by entry).
constexpr int kShortList = 4;
// Dynamic shared memory of a thread block of the batched kernel: the node vector,
// then factor blocks (the adjacency bitsets while ordering).
constexpr int kSmemVector = 6 * (kSparseMax + 2);

// The large-scene teams (whole GPU, one cluster) solve one scene per launch and
// factor up to kSparseMaxLarge active bodies: the whole direct branch, which
// ends at 2,000 local bodies.  Their scratch is one slot of B.sparse_big.
constexpr int kSparseMaxLarge = 2048;
constexpr int kSparseWordsLarge = kSparseMaxLarge / 32;
constexpr int kRowCapLarge = 1 << 16;
// ints of the large slot's index arrays, before its double arrays
constexpr long long kSparseLargeIntWords =
    2LL * kSparseMaxLarge * kSparseWordsLarge + 12LL * (kSparseMaxLarge + 8) + 2LL * kRowCapLarge + 8;
// doubles of the large slot before its off-diagonal blocks
constexpr long long kSparseLargeHeaderDoubles = (kSparseLargeIntWords + 1) / 2 + 2LL * 36 * kSparseMaxLarge +
                                                4LL * 6 * kSparseMaxLarge;
// A large-team factor whose sequential depth exceeds kDirectDepthMax goes to
// PCG instead.  Depth, in row updates (about 0.75 us each on one cluster): per
// elimination level kLevelCost for the level's barrier and its chain of
// dependent loads (about 10 us measured), plus the largest column's per-lane
// row updates.  Contact graphs with short elimination trees (the stacks and
// heaps of a filling pile) factor in well under a PCG solve's time (1.3-2 ms
// per Newton step on these scenes); long strips and grid-like ones (a packed
// crate, whose top separators are dense) do not.
constexpr int kLevelCost = 14;
constexpr int kDirectDepthMax = 2048;
// Multiple minimum degree: a round eliminates independent nodes of degree up to
// the minimum + kMmdDelta; past kMmdMaxRounds rounds the scene goes to PCG.
constexpr int kMmdDelta = 2;
constexpr int kMmdMaxRounds = 512;

// W = R diag(kn, Kt^-1) R^T (packed symmetric)
__device__ __forceinline__ void frame_sandwich(const Frame& R, double kni, double t00, double t01, double t11,
                                               double* W) {
    // columns of R: n = (m0,m3,m6), t1 = (m1,m4,m7), t2 = (m2,m5,m8)
    double K[3][3] = {{kni, 0, 0}, {0, t00, t01}, {0, t01, t11}};
    double RK[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) RK[i][j] = R.m[i * 3 + 0] * K[0][j] + R.m[i * 3 + 1] * K[1][j] + R.m[i * 3 + 2] * K[2][j];
    auto e = [&](int i, int j) { return RK[i][0] * R.m[j * 3 + 0] + RK[i][1] * R.m[j * 3 + 1] + RK[i][2] * R.m[j * 3 + 2]; };
    W[0] = e(0, 0);
    W[1] = e(1, 1);
    W[2] = e(2, 2);
    W[3] = e(0, 1);
    W[4] = e(0, 2);
    W[5] = e(1, 2);
}
__device__ __forceinline__ d3 sym_mul(const double* W, d3 v) {
    return d3{W[0] * v.x + W[3] * v.y + W[4] * v.z, W[3] * v.x + W[1] * v.y + W[5] * v.z,
              W[4] * v.x + W[5] * v.y + W[2] * v.z};
}

// Per-pair friction coefficient of scene-local bodies i, j: splitmix64 of the
// seed xor the ordered pair key, top 53 bits as u in [0, 1), mu = lo + (hi-lo) u.
__device__ __noinline__ double pair_mu(int i, int j, double lo, double hi, unsigned long long seed) {
    const unsigned long long a = (unsigned long long)(unsigned)min(i, j), b = (unsigned long long)(unsigned)max(i, j);
    unsigned long long z = (seed ^ ((a << 32) | b)) + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const double u = (double)(z >> 11) * 0x1.0p-53;
    return fma(hi - lo, u, lo);
}

// Velocity of the contact point on body j: v + w x c  (zero for static / non-active)
__device__ __forceinline__ d3 point_vel(const double* u6, d3 c) {
    d3 v = ld3(u6), w = ld3(u6 + 3);
    return add3(v, cross3(w, c));
}

template <class Team>
class SceneSolver {
   public:
    const BatchPtrs& B;
    const EngineCfg& C;
    Team& T;
    int s, b0, nb, c0, nc, tid, nt;
    double dt, g[3];
    double cm, cs;  // charMass, charSpeed
    double compliance, reduction, spring_term;
    int n_local, n_active;
    bool dense_mode;
    int sp_nw;  // bitset words in use (large teams)
    bool in_smem = false;  // the factor's blocks are in shared memory, not in the team's slot
    int status;
    // sparse-factor capacities: the large-scene teams run one scene per launch
    static constexpr bool kLargeTeam = Team::kind >= 2;
    static constexpr int kSpMax = kLargeTeam ? kSparseMaxLarge : kSparseMax;
    static constexpr int kSpWords = kSpMax / 32;  // bitset row stride
    __device__ __forceinline__ int spw() const {
        if constexpr (kLargeTeam) return sp_nw;
        else return kSparseWords;
    }
    unsigned long long t_build, t_solve, t_ls, t_mark;

    __device__ SceneSolver(const BatchPtrs& b, const EngineCfg& c, Team& t, int scene)
        : B(b), C(c), T(t), s(scene) {
        if (B.body_off) {
            b0 = B.body_off[s];
            nb = B.body_cnt ? B.body_cnt[s] : B.body_off[s + 1] - b0;
            c0 = B.contact_off[s];
            nc = B.contact_cnt ? B.contact_cnt[s] : B.contact_off[s + 1] - c0;
            dt = B.dt[s];
            g[0] = B.grav[3 * s];
            g[1] = B.grav[3 * s + 1];
            g[2] = B.grav[3 * s + 2];
        } else {
            b0 = 0;
            nb = B.single_nb;
            c0 = 0;
            nc = B.single_nc;
            dt = B.single_dt;
            g[0] = B.single_g[0];
            g[1] = B.single_g[1];
            g[2] = B.single_g[2];
        }
        tid = T.rank;
        nt = T.size;
        status = 0;
        t_build = t_solve = t_ls = 0;
    }

    __device__ __forceinline__ unsigned long long now() {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        return t;
    }
    __device__ __forceinline__ bool active(int gb) const { return B.local[gb] && !B.is_static[gb]; }
    __device__ __forceinline__ double cmu(int gc) const {
        if (B.cmu) return B.cmu[gc];
        if (C.mu_pair_hi > C.mu_pair_lo)
            return pair_mu(B.cbody[2 * gc], B.cbody[2 * gc + 1], C.mu_pair_lo, C.mu_pair_hi, C.mu_pair_seed);
        return C.mu;
    }

    // fields of contact gc / of an incidence slot (kFields and kIncFields runs of 32)
    __device__ __forceinline__ double* contact(int gc) const {
        return B.ct + (long long)(gc >> 5) * (32 * kFields) + (gc & 31);
    }
    __device__ __forceinline__ double* incidence(int slot) const {
        return B.it + (long long)(slot >> 5) * (32 * kIncFields) + (slot & 31);
    }
    __device__ __forceinline__ static d3 fld3(const double* P, int f) {
        return d3{P[32 * f], P[32 * f + 32], P[32 * f + 64]};
    }
    __device__ __forceinline__ static void fst3(double* P, int f, d3 v) {
        P[32 * f] = v.x;
        P[32 * f + 32] = v.y;
        P[32 * f + 64] = v.z;
    }
    __device__ __forceinline__ static Frame frame(const double* P) {
        Frame f;
#pragma unroll
        for (int i = 0; i < 9; ++i) f.m[i] = P[32 * (F_frame + i)];
        return f;
    }
    __device__ __forceinline__ static d3 arm(const double* P, int side) { return fld3(P, F_arm + 3 * side); }
    __device__ __forceinline__ static void ld6(const double* p, double* v) {  // 16-byte aligned
        const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1],
                      c = reinterpret_cast<const double2*>(p)[2];
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
    }
    __device__ __forceinline__ static void st6(double* p, const double* v) {
        reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
        reinterpret_cast<double2*>(p)[2] = make_double2(v[4], v[5]);
    }
    // W (packed), own and other lever arm of an incidence
    __device__ __forceinline__ void ldg12(int slot, double* v) const {
        ld6(B.G + 12LL * slot, v);
        ld6(B.G + 12LL * slot + 6, v + 6);
    }

    // Gather sum over the incidences of body gb of sigma * [X; c x X], in incidence
    // order: the contacts left sigma X in the body's own incidence slots (put_x),
    // so the loads are independent of each other.  (Lanes splitting a body's
    // incidences change the order of the sums, and with it the rounding that an
    // unloaded symmetric stack amplifies.)
    __device__ __forceinline__ void gather(int gb, double out[6], int xf = I_X) const {
        const int st = B.inc_start[gb], n = B.inc_cnt[gb];
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0;
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const double* Q = incidence(st + k);
            const d3 x = fld3(Q, xf);
            const d3 t = cross3(fld3(Q, I_arm), x);
            a0 += x.x; a1 += x.y; a2 += x.z;
            a3 += t.x; a4 += t.y; a5 += t.z;
        }
        out[0] = a0; out[1] = a1; out[2] = a2; out[3] = a3; out[4] = a4; out[5] = a5;
    }
    // Contact gc's world vector X into the incidence slots of its two sides, with
    // the side's sign (-X for side 0, X for side 1; static sides have no slot)
    // -- field xf of the slots
    __device__ __forceinline__ void put_x(int gc, d3 x, int xf = I_X) const {
        const int2 sl = reinterpret_cast<const int2*>(B.islot)[gc];
        if (sl.x >= 0) fst3(incidence(sl.x), xf, scl3(-1.0, x));
        if (sl.y >= 0) fst3(incidence(sl.y), xf, x);
    }
    // (M / charMass) v  for an active body
    __device__ __forceinline__ void mass_mul(int gb, const double* v, double* y) const {
        const double m = B.mass[gb] / cm;
        const double* I = B.inertia + 6 * gb;
        double Ixx = I[0] / cm, Iyy = I[1] / cm, Izz = I[2] / cm, Ixy = I[3] / cm, Ixz = I[4] / cm, Iyz = I[5] / cm;
        y[0] = m * v[0];
        y[1] = m * v[1];
        y[2] = m * v[2];
        y[3] = Ixx * v[3] + Ixy * v[4] + Ixz * v[5];
        y[4] = Ixy * v[3] + Iyy * v[4] + Iyz * v[5];
        y[5] = Ixz * v[3] + Iyz * v[4] + Izz * v[5];
    }

    // ------------------------------------------------------------ set-up
    // Returns false if the scene has no contacts (outputs already written).
    __device__ bool setup() {
        for (int b = tid; b < nb; b += nt) {
            const int gb = b0 + b;
            B.dvel[3 * gb] = g[0] * dt;  // fillForces :85-88
            B.dvel[3 * gb + 1] = g[1] * dt;
            B.dvel[3 * gb + 2] = g[2] * dt;
            B.dang[3 * gb] = 0;
            B.dang[3 * gb + 1] = 0;
            B.dang[3 * gb + 2] = 0;
            B.inc_cnt[gb] = 0;
            B.inc_cur[gb] = 0;
            B.local[gb] = 0;
        }
        if (nc == 0) return false;
        T.sync();
        // count incidences, mark local bodies (renumbering :95-118)
        int bad = 0;
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            for (int j = 0; j < 2; ++j) {
                const int b = B.cbody[2 * gc + j];
                if (b < 0 || b >= nb) { bad = 1; continue; }
                B.local[b0 + b] = 1;
                if (!B.is_static[b0 + b]) atomicAdd(&B.inc_cnt[b0 + b], 1);
            }
        }
        double v[1] = {(double)bad};
        T.max(v);
        if (v[0] > 0) { status |= PDC_STATUS_BAD_INPUT; return false; }
        // exclusive scan of counts -> absolute start in inc[]
        T.scan(nb, 2 * c0, [&](int b) { return B.inc_cnt[b0 + b]; },
                   [&](int b, int excl) { B.inc_start[b0 + b] = excl; });
        // compact list of the local bodies: every later body phase runs over it
        T.scan(nb, 0, [&](int b) { return (int)B.local[b0 + b]; },
               [&](int b, int excl) {
                   if (B.local[b0 + b]) B.lbody[b0 + excl] = b0 + b;
               });
        // fill incidence lists (slot order arbitrary, sorted below)
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            for (int j = 0; j < 2; ++j) {
                const int gb = b0 + B.cbody[2 * gc + j];
                if (B.is_static[gb]) {
                    B.islot[2 * gc + j] = -1;
                    continue;
                }
                const int slot = atomicAdd(&B.inc_cur[gb], 1);
                B.inc[B.inc_start[gb] + slot] = (gc << 1) | j;
            }
        }
        // per-contact speeds for nonDimensionalParams (:38-63): velExt = v (+ g dt if active)
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            double* const P = contact(gc);
            const Frame R = ld_frame(B.frame + 9 * gc);
#pragma unroll
            for (int k = 0; k < 9; ++k) P[32 * (F_frame + k)] = R.m[k];
#pragma unroll
            for (int k = 0; k < 6; ++k) P[32 * (F_arm + k)] = B.arm[6 * gc + k];
            d3 half[2];
            bool hasStatic = false;
            for (int j = 0; j < 2; ++j) {
                const int gb = b0 + B.cbody[2 * gc + j];
                double ve[6];
                for (int r = 0; r < 3; ++r) {
                    ve[r] = B.vel[3 * gb + r];
                    ve[3 + r] = B.ang[3 * gb + r];
                }
                if (!B.is_static[gb]) {
                    for (int r = 0; r < 3; ++r) ve[r] = fma(g[r], dt, ve[r]);
                } else {
                    hasStatic = true;
                }
                // toLocal(j, velExt) = -T_j^T velExt: j=0 -> -R^T(v + w x c0); j=1 -> +R^T(v + w x c1)
                d3 pv = point_vel(ve, ld3(B.arm + 6 * gc + 3 * j));
                d3 h = to_frame(R, pv);
                half[j] = j ? h : scl3(-1.0, h);
            }
            d3 rel = add3(half[0], half[1]);
            const double nrel = sqrt(dot3(rel, rel));
            for (int j = 0; j < 2; ++j) {
                double sp = sqrt(dot3(half[j], half[j]));
                if (hasStatic) sp = dmax(sp, nrel);
                P[32 * (F_wu + j)] = sp;
            }
        }
        T.sync();
        // sort incidence lists, per-body speed, mass sums
        double acc[5] = {0, 0, 0, 0, 0};  // n_local, n_active, traceSum, m*speed, m
        for (int b = tid; b < nb; b += nt) {
            const int gb = b0 + b;
            if (!B.local[gb]) continue;
            acc[0] += 1;
            if (B.is_static[gb]) continue;
            const int st = B.inc_start[gb], n = B.inc_cnt[gb];
            for (int i = 1; i < n; ++i) {  // insertion sort by (contact, side)
                const int key = B.inc[st + i];
                int j = i - 1;
                while (j >= 0 && B.inc[st + j] > key) {
                    B.inc[st + j + 1] = B.inc[st + j];
                    --j;
                }
                B.inc[st + j + 1] = key;
            }
            double spd = 0;
            for (int k = 0; k < n; ++k) {
                const int e = B.inc[st + k];
                spd = dmax(spd, contact(e >> 1)[32 * (F_wu + (e & 1))]);
                const int go = b0 + B.cbody[2 * (e >> 1) + 1 - (e & 1)];
                B.inc_o[st + k] = B.is_static[go] ? -1 : go;
                B.islot[e] = st + k;  // e = 2 gc + side
                const double* P = contact(e >> 1);
                const d3 own = arm(P, e & 1), oth = arm(P, 1 - (e & 1));
                fst3(incidence(st + k), I_arm, own);
                const double a[6] = {own.x, own.y, own.z, oth.x, oth.y, oth.z};
                st6(B.G + 12LL * (st + k) + 6, a);
            }
            const double m = B.mass[gb];
            const double* I = B.inertia + 6 * gb;
            acc[1] += 1;
            acc[2] += 3 * m + (I[0] + I[1] + I[2]);  // genMassMat().trace()
            acc[3] += spd * m;
            acc[4] += m;
        }
        T.sum(acc);
        n_local = (int)acc[0];
        n_active = (int)acc[1];
        cm = (n_active > 0) ? acc[2] / n_active / 6 : 1;  // :36
        double csv = acc[3] / acc[4];                    // :72
        double gn = sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
        csv = dmax(csv, gn * dt * 0.25);
        csv = dmax(csv, 1e-4);
        cs = csv;
        // sparse direct solve for scenes on the direct branch (the SimplicialLDLT
        // analogue, :385-394): compact node numbering + symbolic factorisation
        {
            const int dmax = kLargeTeam ? C.dense_max_large : C.dense_max;
            const bool ws = kLargeTeam ? B.sparse_big != nullptr
                                       : (Team::kind == 1 ? B.dense_warp != nullptr : B.dense != nullptr);
            dense_mode = ws && n_local < C.direct_threshold && dmax > 0 && n_active <= dmax &&
                         n_active > 0 && dmax <= kSpMax;
        }
        if (dense_mode) {
            T.scan(nb, 0, [&](int b) { return active(b0 + b) ? 1 : 0; },
                   [&](int b, int excl) {
                       if (active(b0 + b)) {
                           B.didx[b0 + b] = excl;
                           B.dbody[b0 + excl] = b0 + b;
                       }
                   });
            if constexpr (kLargeTeam) dense_mode = sparse_symbolic_large();
            else dense_mode = sparse_symbolic();
        }
        // velocities (non-dimensional) :203-217
        for (int i = tid; i < n_local; i += nt) {
            const int gb = B.lbody[b0 + i];
            if (!B.local[gb]) continue;
            for (int r = 0; r < 3; ++r) {
                double v = B.vel[3 * gb + r], w = B.ang[3 * gb + r];
                double vo = v;
                if (!B.is_static[gb]) vo += __dmul_rn(g[r], dt);
                B.u[6 * gb + r] = v / cs;
                B.u[6 * gb + 3 + r] = w / cs;
                B.uold[6 * gb + r] = vo / cs;
                B.uold[6 * gb + 3 + r] = w / cs;
                B.du[6 * gb + r] = 0;
                B.du[6 * gb + 3 + r] = 0;
                B.ru[6 * gb + r] = 0;  // static rows stay zero (calculateResiduals :151-163)
                B.ru[6 * gb + 3 + r] = 0;
            }
        }
        // preprocess (NonSmoothContactForce.cpp:8-48) + initForces (:49-52)
        const double damp = C.spring_damp * C.spring_k;
        const double tk = dt * C.spring_k;
        compliance = 1. / (dt * (tk + damp));
        reduction = tk / (tk + damp);
        spring_term = (C.spring_based ? 1.0 : 0.0) * compliance * cm;
        T.sync();
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            double* const P = contact(gc);
            double k = 0;
            if (C.spring_based) {
                k += -reduction * B.depth[gc] / dt / cs;
            } else {
                d3 w = rel_vel(gc, P, B.u);
                k += w.x * C.restitution;
            }
            P[32 * F_kn] = k;
            {  // calculateTangentialWeight's mass term as a 2x2 form in the tangent direction
                const Frame R = frame(P);
                const d3 t1 = from_frame(R, d3{0.0, 1.0, 0.0}), t2 = from_frame(R, d3{0.0, 0.0, 1.0});
                double q00 = 0, q01 = 0, q11 = 0;
                for (int j = 0; j < 2; ++j) {
                    const int gb = b0 + B.cbody[2 * gc + j];
                    if (B.is_static[gb]) continue;
                    const d3 c = arm(P, j);
                    const d3 a = cross3(c, t1), e = cross3(c, t2);
                    const double im = 1.0 / B.mass[gb];
                    const double* J = B.inv_inertia + 6 * gb;
                    const d3 Ja = d3{J[0] * a.x + J[3] * a.y + J[4] * a.z, J[3] * a.x + J[1] * a.y + J[5] * a.z,
                                     J[4] * a.x + J[5] * a.y + J[2] * a.z};
                    const d3 Je = d3{J[0] * e.x + J[3] * e.y + J[4] * e.z, J[3] * e.x + J[1] * e.y + J[5] * e.z,
                                     J[4] * e.x + J[5] * e.y + J[2] * e.z};
                    q00 += im * dot3(t1, t1) + dot3(a, Ja);
                    q01 += im * dot3(t1, t2) + dot3(a, Je);
                    q11 += im * dot3(t2, t2) + dot3(e, Je);
                }
                fst3(P, F_tq, d3{q00, q01, q11});
            }
            fst3(P, F_f, d3{1.0, 0.0, 0.0});
            P[32 * F_lam] = 1e-2;
            P[32 * (F_lam + 1)] = C.only_normal ? 0.0 : 1e-2;  // only_normal: lambda_t absent
        }
        T.sync();
        return true;
    }

    // toLocal(vels) = -T0^T u0 - T1^T u1 = R^T[(v1 + w1 x c1) - (v0 + w0 x c0)]
    // (ContactInfo.h:46-51); non-local/static bodies read their (fixed) u.
    __device__ __forceinline__ d3 rel_vel(int gc, const double* P, const double* uvec) const {
        const int gb0 = b0 + B.cbody[2 * gc], gb1 = b0 + B.cbody[2 * gc + 1];
        double u0[6], u1[6];
        ld6(uvec + 6LL * gb0, u0);
        ld6(uvec + 6LL * gb1, u1);
        return to_frame(frame(P), sub3(point_vel(u1, arm(P, 1)), point_vel(u0, arm(P, 0))));
    }

    // Tangential weight (calculateTangentialWeight, NonSmoothContactForce.cpp:74-104)
    // The direction d = R (0, th0, th1) enters as hh_j = s_j [d; c_j x d], so the
    // sum over the active bodies of hh_j^T M_j^-1 hh_j is th^T Q th with the
    // per-contact Q = sum_j T_j,t^T M_j^-1 T_j,t computed once per solve (tq).
    __device__ __forceinline__ double tangential_weight(const double* P, d3 w, double rad) const {
        const double tn = sqrt(w.y * w.y + w.z * w.z);
        double th0 = w.y, th1 = w.z;
        if (tn > 0) { th0 = w.y / tn; th1 = w.z / tn; }
        const d3 Q = fld3(P, F_tq);
        const double fw = (Q.x * th0 * th0 + 2.0 * Q.y * th0 * th1 + Q.z * th1 * th1) * cm;
        return dmin(rad / (tn + 1e-8) * fw, 1.0);
    }

    // OnlyNormalForce residuals (OnlyNormalForce.cpp:46-89) and AC term (:202-217):
    // rf = -w_n (- compliance f_n) + lambda - k, rl = lambda (-f_n) + mu_c, unit
    // weight, AC = max(f_n - (w_n + k + spring f_n), 0) - f_n; X = -R (f_n, 0, 0).
    __device__ __forceinline__ void normal_residual(int gc, const double* P, const Frame& R, d3 w, double fn,
                                                    double ln, double muc, d3& rfo, double& rl0, double& wrf2,
                                                    double& rl2, double& ac2, int xf) const {
        const double kn = P[32 * F_kn];
        double r0 = 0 - w.x;
        if (C.spring_based) r0 -= compliance * cm * fn;
        r0 += ln;
        r0 -= kn;
        rl0 = ln * (-fn) + muc;
        wrf2 += r0 * r0;
        rl2 += rl0 * rl0;
        const double tp = fn - (w.x + kn + spring_term * fn);
        const double a0 = dmax(tp, 0.0) - fn;
        ac2 += a0 * a0;
        rfo = d3{r0, 0.0, 0.0};
        put_x(gc, scl3(-1.0, from_frame(R, d3{fn, 0.0, 0.0})), xf);
    }

    // Residuals of one contact (nonSmoothResiduals :119-172, ACVector :53-73) at
    // force fv and multiplier l1 with relative velocity w and cone gradient (g0,
    // g1): rf, its weighted square and |AC|^2; X = -R f into the incidence slots.
    __device__ __forceinline__ d3 cone_residual(int gc, const double* P, const Frame& R, d3 w, d3 fv, double l0,
                                                double l1, double g0, double g1, double mu, double& wrf2, double& ac2,
                                                int xf) const {
        const double kn = P[32 * F_kn], fn = fv.x;
        double r0 = 0 - w.x, r1 = 0 - w.y, r2 = 0 - w.z;
        if (C.spring_based) r0 -= compliance * cm * fn;
        r0 += l0;
        r1 -= l1 * g0;
        r2 -= l1 * g1;
        r0 -= kn;
        const double rad = cone_radius(fn, mu);
        const double wt = tangential_weight(P, w, rad);
        const double w1 = r1 * wt, w2 = r2 * wt;
        wrf2 += r0 * r0 + w1 * w1 + w2 * w2;
        // Alart-Curnier (:60-70)
        const double tp = fn - (w.x + kn + spring_term * fn);
        const double q0 = dmax(tp, 0.0) - fn;
        const double td0 = fv.y - w.y, td1 = fv.z - w.z;
        const double tdn = sqrt(td0 * td0 + td1 * td1);
        double p0 = td0, p1 = td1;
        if (!(tdn < rad)) { p0 = td0 * rad / tdn; p1 = td1 * rad / tdn; }
        const double q1 = p0 - fv.y, q2 = p1 - fv.z;
        ac2 += q0 * q0 + q1 * q1 + q2 * q2;
        put_x(gc, scl3(-1.0, from_frame(R, fv)), xf);
        return d3{r0, r1, r2};
    }

    // Residuals of one contact at the current iterate with its constraint values
    // and gradient just computed, before the centering term is known: adds
    // |wrf|^2, (lambda . c)^2 per constraint and |AC|^2; writes rf and X = -R f.
    __device__ __forceinline__ void contact_residual_c(int gc, double* P, d3 fv, double l0, double l1, double cn, double cc1,
                                                       double g0, double g1, double mu, double& wrf2, double& a2,
                                                       double& ac2) const {
        const d3 w = rel_vel(gc, P, B.u);
        fst3(P, F_wu, w);  // the line search steps from here: J(u + a du) = J u + a J du
        const Frame R = frame(P);
        d3 r;
        if (C.only_normal) {
            double rl0;
            normal_residual(gc, P, R, w, fv.x, l0, 0.0, r, rl0, wrf2, a2, ac2, I_X);
        } else {
            const double a0 = l0 * cn, a1 = l1 * cc1;
            a2 += a0 * a0 + a1 * a1;
            r = cone_residual(gc, P, R, w, fv, l0, l1, g0, g1, mu, wrf2, ac2, I_X);
        }
        fst3(P, F_rf, r);
    }

    // ru = M(u - uold) (+ gather of T_j f) of one active body (calculateResiduals :151-163)
    __device__ __forceinline__ void body_residual(int gb, const double* ub, int xf, double* v) const {
        double gth[6], d[6], y[6];
        ld6(B.uold + 6LL * gb, d);
        for (int r = 0; r < 6; ++r) d[r] = ub[r] - d[r];
        mass_mul(gb, d, y);
        gather(gb, gth, xf);
        for (int r = 0; r < 6; ++r) v[r] = y[r] + gth[r];
    }

    // ------------------------------------------------------------ Newton
    __device__ void newton(pdc_stats& st) {
        const int n_rigid = 6 * n_local, n_force = (C.only_normal ? 1 : 3) * nc,
                  n_cons = (C.only_normal ? 1 : 2) * nc;
        const bool direct = n_local < C.direct_threshold;
        double Hu = 1e-4, exitErr = 0;
        const double power = 0.66667;
        int it = 0, pcg_total = 0, ls_total = 0, gd_total = 0, precision_fallbacks = 0;
        bool ls_fail = false, nonfinite = false;
        for (it = 0; it < C.max_iter; ++it) {
            t_mark = now();
            // calculateConstraints (:105-118), surrogateDualGap and the residuals
            // (:292-300) in one contact pass: the centering mu_c = 0.1 * gap is
            // only known after the pass, so the pass keeps a = lambda . c per
            // constraint and its sums, and |rl|^2 = sum (a + mu_c)^2 is expanded
            // as sum a^2 + 2 mu_c sum a + n_cons mu_c^2 after the reduction; rl
            // itself (= lambda c + mu_c) is formed where it is used
            double e[5] = {0, 0, 0, 0, 0};  // ru2, wrf2, sum a^2, ac2, sum a
            for (int c = tid; c < nc; c += nt) {
                const int gc = c0 + c;
                double* const P = contact(gc);
                const d3 fv = fld3(P, F_f);
                const double cn = -fv.x;
                double cc1 = 0, mu = 0;  // only_normal: c = -f_n alone
                d3 h = d3{0.0, 0.0, 0.0};
                double g0 = 0, g1 = 0;
                if (!C.only_normal) {
                    mu = cmu(gc);
                    cc1 = cone_c(fv.x, fv.y, fv.z, mu);
                    cone_grad(fv.y, fv.z, g0, g1);
                    cone_hess(fv.y, fv.z, h.x, h.y, h.z);
                }
                P[32 * F_cv] = cn;
                P[32 * (F_cv + 1)] = cc1;
                P[32 * F_gr] = g0;
                P[32 * (F_gr + 1)] = g1;
                fst3(P, F_hs, h);
                const double l0 = P[32 * F_lam], l1 = P[32 * (F_lam + 1)];
                e[4] += __fma_rn(l0, cn, __dmul_rn(l1, cc1));
                contact_residual_c(gc, P, fv, l0, l1, cn, cc1, g0, g1, mu, e[1], e[2], e[3]);
            }
            T.sync();
            for (int i = tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (!active(gb)) continue;
                double ub[6], v[6];
                ld6(B.u + 6LL * gb, ub);
                body_residual(gb, ub, I_X, v);
                st6(B.ru + 6LL * gb, v);
                for (int r = 0; r < 6; ++r) e[0] += v[r] * v[r];
            }
            T.sum(e);
            const double sDualGap = -(e[4] / n_cons);
            const double muc = sDualGap * 0.1;
            e[2] = e[2] + 2.0 * muc * e[4] + (double)n_cons * muc * muc;
            const double err = e[0] + e[1] + e[2];
            const double sErr = err, sacErr = e[0] + e[3] + e[2];
            const double eps = Hu * pow(err, power * 0.5);
            const double momenErr = sqrt(e[0]) / n_rigid;
            exitErr = dmax(momenErr, sqrt(e[1]) / n_force);
            exitErr = dmax(exitErr, sqrt(e[2]) / n_cons);
            exitErr = dmax(exitErr, sDualGap);
            exitErr = dmin(exitErr, dmax(momenErr, sqrt(e[3]) / nc));
            if (exitErr < C.tol) break;

            // linsysAddition (:173-253): per-contact K, K^-1, sf, W, rhs vector
            for (int c = tid; c < nc; c += nt) {
                const int gc = c0 + c;
                double* const P = contact(gc);
                const double ln = P[32 * F_lam], lt = P[32 * (F_lam + 1)];
                const double cv0 = P[32 * F_cv], cv1 = P[32 * (F_cv + 1)];
                // only_normal regularises c - eps (OnlyNormalForce.cpp:104), not c - eps lambda
                const double ic0 = 1. / (cv0 - eps * (C.only_normal ? 1.0 : ln));
                const double ic1 = C.only_normal ? 0.0 : 1. / (cv1 - eps * lt);
                P[32 * F_invC] = ic0;
                P[32 * (F_invC + 1)] = ic1;
                const double g0 = P[32 * F_gr], g1 = P[32 * (F_gr + 1)];
                double lNorm = -ln * ic0;
                if (C.spring_based) lNorm += compliance * cm;
                // rl = lambda c + mu_c (nonSmoothResiduals :150-170), kept for the
                // force recovery and the gradient-descent fallback
                const double rl0 = ln * cv0 + muc;
                const double rl1 = C.only_normal ? 0.0 : lt * cv1 + muc;
                P[32 * F_rl] = rl0;
                P[32 * (F_rl + 1)] = rl1;
                const double a = -lt * ic1;
                const d3 rf = fld3(P, F_rf);
                const d3 sf = d3{rf.x + (-rl0 * ic0), rf.y + g0 * rl1 * ic1, rf.z + g1 * rl1 * ic1};
                fst3(P, F_sf, sf);
                const double kni = 1. / (eps + lNorm);
                P[32 * F_knInv] = kni;
                const d3 h = fld3(P, F_hs);
                const double k00 = eps + a * g0 * g0 + lt * h.x;
                const double k01 = 0 + a * g0 * g1 + lt * h.y;
                const double k11 = eps + a * g1 * g1 + lt * h.z;
                const double det = k00 * k11 - k01 * k01;
                double t00 = k11 / det, t01 = -k01 / det, t11 = k00 / det;
                if (C.only_normal) t00 = t01 = t11 = 0;  // no tangential block
                fst3(P, F_ktInv, d3{t00, t01, t11});
                const Frame R = frame(P);
                double W[6];
                frame_sandwich(R, kni, t00, t01, t11, W);
                const int2 sl = reinterpret_cast<const int2*>(B.islot)[gc];
                if (sl.x >= 0) st6(B.G + 12LL * sl.x, W);
                if (sl.y >= 0) st6(B.G + 12LL * sl.y, W);
                if (C.mixed)
                    for (int q = 0; q < 6; ++q) B.Wf[6 * gc + q] = (float)W[q];
                const d3 ks = d3{sf.x * kni, t00 * sf.y + t01 * sf.z, t01 * sf.y + t11 * sf.z};
                put_x(gc, from_frame(R, ks));
            }
            T.sync();
            // rhs = sum getTrans(j) K^-1 sf - ru; block-Jacobi blocks; PCG start
            double rr[3] = {0, 0, 0};  // r.z, b.b, |D b|^2 (iterative branch)
            const bool rows_mode = !kLargeTeam && dense_mode;
            if constexpr (!kLargeTeam) {
                if (dense_mode) {
                    if (Team::kind == 0 && in_smem) assemble_rows<Team::kind == 0>(eps);
                    else assemble_rows<false>(eps);
                }
            }
            for (int i = rows_mode ? n_local : tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (!active(gb)) continue;
                double gth[6];
                gather(gb, gth);
                double* rb = B.rhs + 6 * gb;
                for (int r = 0; r < 6; ++r) rb[r] = gth[r] - B.ru[6 * gb + r];
                // diagonal block: M/cm + eps I + sum_j T_j K^-1 T_j^T
                double P[21];
                for (int q = 0; q < 21; ++q) P[q] = 0;
                {
                    const double m = B.mass[gb] / cm;
                    const double* I = B.inertia + 6 * gb;
                    P[pk(0, 0)] = m + eps;
                    P[pk(1, 1)] = m + eps;
                    P[pk(2, 2)] = m + eps;
                    P[pk(3, 3)] = I[0] / cm + eps;
                    P[pk(4, 4)] = I[1] / cm + eps;
                    P[pk(5, 5)] = I[2] / cm + eps;
                    P[pk(4, 3)] = I[3] / cm;
                    P[pk(5, 3)] = I[4] / cm;
                    P[pk(5, 4)] = I[5] / cm;
                }
                const int st0 = B.inc_start[gb], n = B.inc_cnt[gb];
                for (int k = 0; k < n; ++k) {
                    double W[12];
                    ldg12(st0 + k, W);
                    const d3 c = ld3(W + 6);
                    // Y = C W (C = [c]x): column k of Y = c x W_col_k
                    const d3 wc0 = d3{W[0], W[3], W[4]}, wc1 = d3{W[3], W[1], W[5]}, wc2 = d3{W[4], W[5], W[2]};
                    // (rounded as assemble_rows rounds the factor's diagonal blocks)
                    const d3 y0 = cross_rn(c, wc0), y2 = cross_rn(c, wc2);
                    d3 y1 = cross_rn(c, wc1);
                    y1.y = __fma_rn(-c.x, wc1.z, __dmul_rn(c.z, wc1.x));
                    // Z = C Y^T: column k of Z = c x (row k of Y)
                    const d3 z0 = cross_rn(c, d3{y0.x, y1.x, y2.x});
                    const d3 z1 = cross_rn(c, d3{y0.y, y1.y, y2.y});
                    const d3 z2 = cross_rn(c, d3{y0.z, y1.z, y2.z});
                    P[pk(0, 0)] += W[0]; P[pk(1, 0)] += W[3]; P[pk(1, 1)] += W[1];
                    P[pk(2, 0)] += W[4]; P[pk(2, 1)] += W[5]; P[pk(2, 2)] += W[2];
                    P[pk(3, 0)] += y0.x; P[pk(3, 1)] += y1.x; P[pk(3, 2)] += y2.x;
                    P[pk(4, 0)] += y0.y; P[pk(4, 1)] += y1.y; P[pk(4, 2)] += y2.y;
                    P[pk(5, 0)] += y0.z; P[pk(5, 1)] += y1.z; P[pk(5, 2)] += y2.z;
                    P[pk(3, 3)] += z0.x; P[pk(4, 3)] += z0.y; P[pk(4, 4)] += z1.y;
                    P[pk(5, 3)] += z0.z; P[pk(5, 4)] += z1.z; P[pk(5, 5)] += z2.z;
                }
                if (!direct)  // the reference solves the scaled system D A D (:359-376)
                    for (int r = 0; r < 6; ++r) {
                        const double d = 1 / sqrt(P[pk(r, r)]);
                        B.dsc[6 * gb + r] = d;
                        rr[2] += (d * rb[r]) * (d * rb[r]);
                    }
                if (kLargeTeam && dense_mode) {
                    if constexpr (kLargeTeam) assemble_dense_rows(gb, P);
                } else {
                    double* Pi = B.pinv + 21 * gb;
                    if (!spd6_inverse(P, Pi)) {
                        for (int q = 0; q < 21; ++q) Pi[q] = 0;
                        for (int r = 0; r < 6; ++r) Pi[pk(r, r)] = 1.0 / P[pk(r, r)];
                    }
                    if (C.mixed)
                        for (int q = 0; q < 21; ++q) B.pinvf[21 * gb + q] = (float)Pi[q];
                }
                for (int r = 0; r < 6; ++r) rr[1] += rb[r] * rb[r];
            }
            if (rows_mode) T.sync();
            else T.sum(rr);  // sync: rhs, pinv complete
            const double bnorm = sqrt(rr[1]);
            // AMGCL's relative residual is measured in the scaled system: |D r| / |D b|
            const double bn = direct ? bnorm : sqrt(rr[2]);
            unsigned long long t1 = now();
            t_build += t1 - t_mark;
            t_mark = t1;

            // ---- linear solve: block-Jacobi PCG (replaces LDLT / AMGCL, :385-427)
            const double rtol = direct ? C.rtol_direct : C.rtol_iter;
            // lanes per body in the PCG product: chosen for the large-scene teams only
            const int lanes = (Team::spmv_lanes > 1 && C.pcg_lanes > 0) ? C.pcg_lanes : Team::spmv_lanes;
            const int maxit = direct ? C.max_direct : C.max_cg;
            int iters = 0;
            bool lin_bad = false;
            if (dense_mode) {
                if constexpr (kLargeTeam) lin_bad = !dense_solve_warp();
                else lin_bad = Team::kind == 0 && in_smem ? !direct_solve<Team::kind == 0>() : !direct_solve<false>();
            }
            // mixed precision: FP32 PCG with FP64 refinement where PCG runs; an
            // inner breakdown or a refinement that stops converging falls back
            // to the FP64 PCG below, from zero
            bool fp64_pcg = !dense_mode;
            if (!dense_mode && C.mixed) {
                bool conv = true;
                const bool ok = mixed_solve(eps, bnorm, dmax(rtol, kMixedRtolMin), iters, conv);
                pcg_total += iters;
                iters = 0;
                fp64_pcg = !(ok && conv);
                if (fp64_pcg) {
                    ++precision_fallbacks;
                    for (int i = tid; i < n_local; i += nt) {
                        const int gb = B.lbody[b0 + i];
                        for (int r = 0; r < 6; ++r) B.du[6 * gb + r] = 0;
                    }
                    T.sync();
                }
            }
            if (fp64_pcg) {
            // attempt 0: the solve; attempt 1 (iterative branch only): the
            // reference's fallback when AMGCL ends non-finite, an Eigen CG from
            // zero to machine precision with at most 2 n iterations (:416-421)
            double rtol_a = rtol;
            int maxit_a = maxit;
            for (int attempt = 0; attempt < 2; ++attempt) {
            iters = 0;
            if (!direct) {
                // AMGCL starts from the previous du taken as the scaled unknown
                // (:406-415), i.e. from D du here (this PCG runs on the unscaled
                // system; with block-Jacobi preconditioning its iterates are the
                // scaled PCG's times D); a zero right-hand side gives du = 0
                for (int i = tid; i < n_local; i += nt) {
                    const int gb = B.lbody[b0 + i];
                    if (!active(gb)) continue;
                    for (int r = 0; r < 6; ++r)
                        B.du[6 * gb + r] = (bn > 0 && attempt == 0) ? B.dsc[6 * gb + r] * B.du[6 * gb + r] : 0.0;
                }
                T.sync();
                spmv_to_X(B.du);
                T.sync();
            }
            double s2[2] = {0, 0};
            for (int i = tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (!active(gb)) continue;
                double r6[6];
                if (direct) {
                    for (int r = 0; r < 6; ++r) { r6[r] = B.rhs[6 * gb + r]; B.du[6 * gb + r] = 0; }
                } else {
                    double q6[6];
                    spmv_body(gb, B.du + 6 * gb, eps, q6);
                    for (int r = 0; r < 6; ++r) r6[r] = B.rhs[6 * gb + r] - q6[r];
                }
                double z6[6];
                prec(gb, r6, z6);
                for (int r = 0; r < 6; ++r) {
                    B.r[6 * gb + r] = r6[r];
                    B.z[6 * gb + r] = z6[r];
                    B.p[6 * gb + r] = 0;
                    s2[0] += r6[r] * z6[r];
                    const double rs = direct ? r6[r] : B.dsc[6 * gb + r] * r6[r];
                    s2[1] += rs * rs;
                }
            }
            T.sum(s2);
            double rz = s2[0];
            double res = (bn > 0) ? sqrt(s2[1]) / bn : 0.0;
            double beta = 0;
            if (bn == 0) {
                // zero right-hand side: du = x0 (zero on the direct branch)
            } else if (!(res < rtol_a)) {
                for (iters = 0; iters < maxit_a;) {
                    // p_new = z + beta p (p double-buffered by parity so that the
                    // neighbours' previous directions stay readable) and q = A p_new
                    const double* pp = (iters & 1) ? B.p2 : B.p;
                    double* pc = (iters & 1) ? B.p : B.p2;
                    double s3[1] = {0};
                    if constexpr (Team::spmv_lanes > 1) {
                        switch (lanes) {
                            case 8: pcg_product<8>(pp, pc, beta, eps, s3[0]); break;
                            case 4: pcg_product<4>(pp, pc, beta, eps, s3[0]); break;
                            case 2: pcg_product<2>(pp, pc, beta, eps, s3[0]); break;
                            default: pcg_product<1>(pp, pc, beta, eps, s3[0]); break;
                        }
                    } else {
                        for (int i = tid; i < n_local; i += nt) {
                            const int gb = B.lbody[b0 + i];
                            if (!active(gb)) continue;
                            double pn[6], q6[6];
                            for (int r = 0; r < 6; ++r) {
                                pn[r] = __dadd_rn(B.z[6 * gb + r], __dmul_rn(beta, pp[6 * gb + r]));
                                pc[6 * gb + r] = pn[r];
                            }
                            spmv_body_fused1(gb, pn, pp, beta, eps, q6);
                            for (int r = 0; r < 6; ++r) {
                                s3[0] += pn[r] * q6[r];
                                B.q[6 * gb + r] = q6[r];
                            }
                        }
                    }
                    T.sum(s3);
                    const double alpha = rz / s3[0];
                    double s4[2] = {0, 0};
                    for (int i = tid; i < n_local; i += nt) {
                        const int gb = B.lbody[b0 + i];
                        if (!active(gb)) continue;
                        double r6[6], z6[6];
                        for (int r = 0; r < 6; ++r) {
                            B.du[6 * gb + r] += alpha * pc[6 * gb + r];
                            r6[r] = B.r[6 * gb + r] - alpha * B.q[6 * gb + r];
                            B.r[6 * gb + r] = r6[r];
                        }
                        prec(gb, r6, z6);
                        for (int r = 0; r < 6; ++r) {
                            B.z[6 * gb + r] = z6[r];
                            const double rs = direct ? r6[r] : B.dsc[6 * gb + r] * r6[r];
                            s4[0] += rs * rs;
                            s4[1] += r6[r] * z6[r];
                        }
                    }
                    T.sum(s4);
                    ++iters;
                    res = sqrt(s4[0]) / bn;
                    if (!(res >= rtol_a)) break;  // converged or non-finite
                    beta = s4[1] / rz;
                    rz = s4[1];
                }
            }
            if (direct || attempt == 1 || isfinite(res)) {
                pcg_total += iters;  // the rerun's count replaces the first attempt's, as in the reference
                if (!isfinite(res)) {
                    if (direct) lin_bad = true;  // the LDLT failure rule (:390-394)
                    else nonfinite = true;       // du is the CG fallback's, whatever it is
                }
                break;
            }
            nonfinite = true;
            rtol_a = 2.220446049250313e-16;  // Eigen's default tolerance: machine epsilon
            maxit_a = 2 * n_rigid;           // ... and iteration cap: twice the unknowns
            T.sync();
            }  // attempts
            }  // PCG branch
            if (lin_bad) {  // LDLT failure analogue (:390-394): du = 0
                nonfinite = true;
                for (int i = tid; i < n_local; i += nt) {
                    const int gb = B.lbody[b0 + i];
                    for (int r = 0; r < 6; ++r) B.du[6 * gb + r] = 0;
                }
            }
            T.sync();
            // retrieveNonSmoothForceInc (:254-280)
            for (int c = tid; c < nc; c += nt) {
                const int gc = c0 + c;
                double* const P = contact(gc);
                const d3 w = rel_vel(gc, P, B.du);
                fst3(P, F_wd, w);
                const d3 d = sub3(fld3(P, F_sf), w);
                const double d0 = P[32 * F_knInv] * d.x;
                const d3 t = fld3(P, F_ktInv);
                const double e1 = t.x * d.y + t.y * d.z, e2 = t.y * d.y + t.z * d.z;
                fst3(P, F_df, d3{d0, e1, e2});
                P[32 * F_dl] = -P[32 * F_invC] * (-P[32 * F_lam] * d0 + P[32 * F_rl]);
                P[32 * (F_dl + 1)] = -P[32 * (F_invC + 1)] * (P[32 * (F_lam + 1)] * (P[32 * F_gr] * e1 + P[32 * (F_gr + 1)] * e2) +
                                                        P[32 * (F_rl + 1)]);
            }
            T.sync();
            t1 = now();
            t_solve += t1 - t_mark;
            t_mark = t1;

            // line search (:437-440), gradient-descent fallback (:444-467)
            int trials = 0;
            double step = line_search(sErr, sacErr, muc, C.ls_max, trials);
            ls_total += trials;
            bool useGD = false;
            if (step == 0) {
                useGD = true;
                gd_total++;
                for (int i = tid; i < n_local; i += nt) {
                    const int gb = B.lbody[b0 + i];
                    if (!B.local[gb]) continue;
                    for (int r = 0; r < 6; ++r) B.du[6 * gb + r] = -B.ru[6 * gb + r];
                }
                for (int c = tid; c < nc; c += nt) {
                    const int gc = c0 + c;
                    double* const P = contact(gc);
                    fst3(P, F_wd, scl3(-1.0, rel_vel(gc, P, B.ru)));  // J du with du = -ru
                    fst3(P, F_df, fld3(P, F_rf));
                    P[32 * F_dl] = P[32 * F_rl];
                    P[32 * (F_dl + 1)] = P[32 * (F_rl + 1)];
                }
                T.sync();
                step = line_search(sErr, sacErr, muc, C.gd_max, trials);
                ls_total += trials;
                if (step == 0) ls_fail = true;
            }
            // Hu update (:474-483)
            if (!useGD && step == 1) {
                if (!direct && iters == maxit) Hu *= 1.3;
                else Hu /= 4;
            } else {
                Hu *= 4;
            }
            Hu = dmax(Hu, 1e-6);
            t1 = now();
            t_ls += t1 - t_mark;
        }
        st.newton_iters = it;
        st.exit_err = exitErr;
        st.pcg_iters = pcg_total;
        st.ls_trials = ls_total;
        st.gd_fallbacks = gd_total;
        st.precision_fallbacks = precision_fallbacks;
        int stt = status;
        if (it >= C.max_iter) stt |= PDC_SCENE_MAX_ITER;
        if (ls_fail) stt |= PDC_SCENE_LS_FAIL;
        if (nonfinite || !isfinite(exitErr)) stt |= PDC_SCENE_NONFINITE;
        status = stt;
    }

    // ------------------------------------------- sparse direct solve (direct branch)
    // Scratch of the large-scene teams (one slot, B.sparse_big): bitset adjacency
    // / column patterns, elimination order, block-column offsets, diagonal
    // blocks, their Cholesky factors, the L blocks and node vectors.  Node i is
    // the i-th active body of the scene.
    struct Sparse {
        uint32_t* adj;   // [kSpMax][kSpWords]
        uint32_t* radj;  // [kSpMax][kSpWords] row patterns, bit k = column eliminated k-th
        int* perm;       // elimination position -> node
        int* ipos;       // node -> elimination position
        int* cstart;     // [n + 1] first L block of each node's column
        int* lvl_nodes;  // nodes grouped by elimination-tree height
        int* height;     // elimination-tree height of each node
        int* lvl_start;  // [levels + 1]
        int* rowptr;     // [n + 1] row lists: columns d with L(v, d) != 0
        int* deg;        // current degree of each node; later the level cursors
        int* sel;        // nodes eliminated in the current round
        int* lvl_work;   // largest column work of each level
        int* rowidx;     // [kRowCapLarge]
        int* rowoff;     // [kRowCapLarge] block index of L(u, d) for each row-list entry
        int* meta;       // [0] number of levels
        double* Dg;      // [n][36] diagonal blocks
        double* Ld;      // [n][36] Cholesky factor of each diagonal block
        double* Ldi;     // [n][6] reciprocal of the factor's diagonal
        double* y;       // [n][6]
        double* z;       // [n][6]
        double* x;       // [n][6]
        double* L;       // [cap][36] off-diagonal blocks, column by column
        int cap;
    };
    __device__ __forceinline__ Sparse sparse_ws() const {
        constexpr int M = kSparseMaxLarge, M8 = kSparseMaxLarge + 8;
        int* q = reinterpret_cast<int*>(B.sparse_big);
        Sparse S;
        S.adj = reinterpret_cast<uint32_t*>(q);
        q += M * kSparseWordsLarge;
        S.radj = reinterpret_cast<uint32_t*>(q);
        q += M * kSparseWordsLarge;
        S.perm = q; q += M8;
        S.ipos = q; q += M8;
        S.cstart = q; q += M8;
        S.lvl_nodes = q; q += M8;
        S.height = q; q += M8;
        S.lvl_start = q; q += M8;
        S.rowptr = q; q += M8;
        S.deg = q; q += M8;
        S.sel = q; q += M8;
        S.lvl_work = q; q += M8;
        q += 2 * M8;  // spare
        S.rowidx = q; q += kRowCapLarge;
        S.rowoff = q; q += kRowCapLarge;
        S.meta = q;
        double* d = B.sparse_big + (kSparseLargeIntWords + 1) / 2;
        S.Dg = d; d += 36 * M;
        S.Ld = d; d += 36 * M;
        S.Ldi = d; d += 6 * M;
        S.y = d; d += 6 * M;
        S.z = d; d += 6 * M;
        S.x = d; d += 6 * M;
        S.L = d;
        const long long left = B.sparse_big_doubles - kSparseLargeHeaderDoubles;
        S.cap = left > 0 ? (int)min(left / 36, (long long)kRowCapLarge) : 0;
        return S;
    }

    // Scratch of the block and warp teams (one slot per team).  Everything is
    // numbered by elimination position k (column k of the factor); the 6x6
    // blocks of all columns lie in level order, column by column, each column's
    // diagonal block first, so a block's index says what level it belongs to.
    struct Direct {
        uint32_t* adj;   // [kSparseMax][kSparseWords] node adjacency (thread blocks keep it in shared memory)
        uint32_t* colb;  // [kSparseMax][kSparseWords] column k's pattern: positions u > k with L(u, k) != 0
        uint32_t* rowb;  // [kSparseMax][kSparseWords] row k's pattern: positions d < k with L(k, d) != 0
        int* perm;       // position -> node
        int* ipos;       // node -> position
        int* height;     // node -> elimination-tree height, then position -> height
        int* deg;        // degree of each remaining node while ordering
        int* body;       // position -> body
        int* base;       // position -> index of the column's diagonal block
        int* lvl_cols;   // positions by (height, position)
        int* lvl_start;  // [levels + 1] first entry of each level in lvl_cols
        int* lvl_blk;    // [levels + 1] first block of each level
        int* lvl_len;    // [levels] longest update list of the level
        int* lvl_pat;    // [levels] most off-diagonal blocks of a column of the level
        int* meta;       // [0] levels, [1] blocks, [2] update-list entries (0: no lists)
        int4* desc;      // [blocks] first list entry; list length | column << 16 | row << 24;
                         // first and one past the last contact (slot, or entry of inc_g)
        double* y;       // [n + 1][6] right-hand side, then L^-1 of it, then the solution; node n is 0
        double* L;       // [blocks + 1][36], each in the order of frag(); a diagonal block
                         // becomes its Cholesky factor; the last is 0
        const uint32_t* list;  // update lists, each padded to an even length
        double* slot;    // [cap][36] room of the team's slot, for the blocks (when they
        int cap;         // do not fit the shared memory) and then the lists
    };
    __device__ __forceinline__ Direct direct_ws() const {
        // thread-block teams use slot blockIdx.x of B.dense, warp teams slot
        // (T.slot - gridDim.x) of B.dense_warp
        const bool warp_slot = Team::kind == 1;
        double* const first = warp_slot ? B.dense_warp + (long long)(T.slot - (int)gridDim.x) * B.dense_stride_warp
                                        : B.dense + (long long)T.slot * B.dense_stride;
        const long long stride = warp_slot ? B.dense_stride_warp : B.dense_stride;
        constexpr int M8 = kSparseMax + 8;
        Direct S;
        int4* d = reinterpret_cast<int4*>(first);
        constexpr int cap = Team::kind == 1 ? kRowCapWarp : kRowCap;
        S.desc = d; d += cap + kSparseMax + 2;
        double* v = reinterpret_cast<double*>(d);
        S.y = v; v += 6 * (kSparseMax + 2);
        int* q = reinterpret_cast<int*>(v);
        S.colb = reinterpret_cast<uint32_t*>(q); q += kSparseMax * kSparseWords;
        S.rowb = reinterpret_cast<uint32_t*>(q); q += kSparseMax * kSparseWords;
        S.adj = reinterpret_cast<uint32_t*>(q); q += kSparseMax * kSparseWords;
        S.perm = q; q += M8;
        S.ipos = q; q += M8;
        S.height = q; q += M8;
        S.deg = q; q += M8;
        S.body = q; q += M8;
        S.base = q; q += M8;
        S.lvl_cols = q; q += M8;
        S.lvl_start = q; q += M8;
        S.lvl_blk = q; q += M8;
        S.lvl_len = q; q += M8;
        S.lvl_pat = q; q += M8;
        S.meta = q;
        S.slot = first + sparse_header_doubles(cap) - 36LL * (kSparseMax + 2);
        S.cap = (int)((stride - (S.slot - first)) / 36) - 2;
        S.L = S.slot;
        if constexpr (Team::kind == 0) S.y = block_smem();
        S.list = reinterpret_cast<const uint32_t*>(in_smem ? S.slot : S.slot + 36LL * (S.meta[1] + 2));
        return S;
    }
    // The thread block's dynamic shared memory (node vector, then blocks).
    __device__ __forceinline__ static double* block_smem() {
        extern __shared__ __align__(16) double s_direct[];
        return s_direct;
    }
    // The blocks' address: shared memory when the factor fits there.
    template <bool SM>
    __device__ __forceinline__ static double* block_base(const Direct& S) {
        if constexpr (SM) return block_smem() + kSmemVector;
        else return S.L;
    }
    // rank of node u among the set bits of a column pattern (= its block slot)
    __device__ __forceinline__ static int bit_rank(const uint32_t* w, int u) {
        int r = 0;
        for (int k = 0; k < (u >> 5); ++k) r += __popc(w[k]);
        return r + __popc(w[u >> 5] & ((1u << (u & 31)) - 1u));
    }
    // Symbolic factorisation of the block and warp teams, once per step, every
    // part spread over the team: node adjacency from the incidence lists, strict
    // minimum-degree elimination on bitsets (ties to the smallest node), then --
    // numbered by elimination position -- column and row patterns, levels of
    // equal elimination-tree height, block storage in level order, and for every
    // block its update list: the pairs of earlier blocks whose products it takes.
    // The lists are what the numeric phase would otherwise look up bit by bit in
    // every Newton iteration; they go behind the blocks, and a factor too dense
    // to leave room for them (meta[2] = 0) walks the row patterns instead.
    // Returns false (the scene then uses PCG) if the factor does not fit.
    __device__ bool sparse_symbolic() {
        const Direct S = direct_ws();
        constexpr int W = kSparseWords;
        const int n = n_active;
        uint32_t* adj = S.adj;
        if constexpr (Team::kind == 0) {  // where the blocks will be
            if (B.smem_blocks * 288 >= kSparseMax * kSparseWords * 4)
                adj = reinterpret_cast<uint32_t*>(block_smem() + kSmemVector);
        }
        for (int q = tid; q < n * W; q += nt) adj[q] = 0;
        T.sync();
        for (int l = tid; l < n_local; l += nt) {
            const int gb = B.lbody[b0 + l];
            if (!active(gb)) continue;
            const int i = B.didx[gb];
            const int st0 = B.inc_start[gb], cnt = B.inc_cnt[gb];
            for (int k = 0; k < cnt; ++k) {
                const int go = B.inc_o[st0 + k];  // -1: static
                if (go == gb || go < 0 || !B.local[go]) continue;
                const int j = B.didx[go];
                adj[i * W + (j >> 5)] |= 1u << (j & 31);
            }
            int d = 0;
            for (int w = 0; w < W; ++w) d += __popc(adj[i * W + w]);
            S.deg[i] = d;
            S.ipos[i] = -1;
            S.height[i] = 0;
        }
        T.sync();
        for (int k = 0; k < n; ++k) {
            // argmin (degree, node) over the remaining nodes
            unsigned best = 0xffffffffu;
            for (int i = tid; i < n; i += nt)
                if (S.ipos[i] < 0) best = min(best, ((unsigned)S.deg[i] << 16) | (unsigned)i);
            const int v = (int)(T.min_u32(best) & 0xffffu);
            const uint32_t* av = adj + v * W;
            const int hv = S.height[v] + 1;
            for (int u = tid; u < n; u += nt) {
                if (u == v) {
                    S.perm[k] = v;
                    S.ipos[v] = k;
                    S.body[k] = B.dbody[b0 + v];
                }
                if (!((av[u >> 5] >> (u & 31)) & 1u)) continue;
                uint32_t* au = adj + u * W;
                int d = 0;
                for (int w = 0; w < W; ++w) {
                    uint32_t x = au[w] | av[w];
                    if (w == (u >> 5)) x &= ~(1u << (u & 31));
                    if (w == (v >> 5)) x &= ~(1u << (v & 31));
                    au[w] = x;
                    d += __popc(x);
                }
                S.deg[u] = d;
                S.height[u] = max(S.height[u], hv);
            }  // the next minimum's barrier orders these rows before their readers
        }
        T.sync();
        // patterns by position: word w of column k's and row k's pattern per item
        for (int q = tid; q < n * W; q += nt) {
            const int k = q / W, w = q - k * W;
            const int v = S.perm[k];
            uint32_t cb = 0, rb = 0;
            const int end = min(n, 32 * w + 32);
            for (int p = 32 * w; p < end; ++p) {
                const int o = S.perm[p];
                const uint32_t hit = p > k ? adj[v * W + (o >> 5)] >> (o & 31) : adj[o * W + (v >> 5)] >> (v & 31);
                if (p > k) cb |= (hit & 1u) << (p & 31);
                else if (p < k) rb |= (hit & 1u) << (p & 31);
            }
            S.colb[q] = cb;
            S.rowb[q] = rb;
        }
        for (int k = tid; k < n; k += nt) S.deg[k] = S.height[S.perm[k]];  // height by position
        T.sync();
        // position k's rank in (height, position) order and its first block: the
        // sum over the columns before it of their block counts
        for (int k = tid; k < n; k += nt) {
            int m = 0;
            for (int w = 0; w < W; ++w) m += __popc(S.colb[k * W + w]);
            S.height[k] = m + 1;  // blocks of the column, from here on
        }
        T.sync();
        int top = 0;
        for (int k = tid; k < n; k += nt) {
            const int h = S.deg[k];
            int rank = 0, first = 0;
            for (int j = 0; j < n; ++j) {
                const int hj = S.deg[j];
                if (hj < h || (hj == h && j < k)) {
                    ++rank;
                    first += S.height[j];
                }
            }
            S.lvl_cols[rank] = k;
            S.base[k] = first;
            if (rank == n - 1) S.meta[1] = first + S.height[k];
            top = max(top, h);
        }
        const int nlev = 0x7fffffff - (int)T.min_u32(0x7fffffffu - (unsigned)top) + 1;
        for (int l = tid; l <= nlev; l += nt) {  // levels: columns and blocks of smaller height
            int c = 0, b = 0;
            for (int j = 0; j < n; ++j)
                if (S.deg[j] < l) {
                    ++c;
                    b += S.height[j];
                }
            S.lvl_start[l] = c;
            S.lvl_blk[l] = b;
            S.lvl_len[l] = 0;
            S.lvl_pat[l] = 0;
        }
        if (tid == 0) S.meta[0] = nlev;
        T.sync();
        const int nblk = S.meta[1];
        if (nblk > S.cap) return false;
        // (column, row) and list length of every block: block (u, k) takes L(u, d)
        // L(k, d)^T for every d in the rows of both
        for (int q = tid; q < n * W; q += nt) {
            const int k = q / W, w = q - k * W;
            int b = S.base[k] + 1;
            for (int x = 0; x < w; ++x) b += __popc(S.colb[k * W + x]);
            uint32_t bits = S.colb[q];
            if (w == 0) S.desc[S.base[k]].y = (k << 16) | (k << 24);
            while (bits) {
                S.desc[b++].y = (k << 16) | (((w << 5) + __ffs(bits) - 1) << 24);
                bits &= bits - 1;
            }
        }
        T.sync();
        for (int i = tid; i < nblk; i += nt) {
            const int y = S.desc[i].y, k = (y >> 16) & 255, u = (y >> 24) & 255;
            int c = 0;
            for (int w = 0; w < W; ++w) c += __popc(S.rowb[k * W + w] & S.rowb[u * W + w]);
            if (c) atomicMax(&S.lvl_len[S.deg[k]], c);
            if (k == u) atomicMax(&S.lvl_pat[S.deg[k]], S.height[k] - 1);
            S.desc[i].y = y | c;
        }
        T.sync();
        T.scan(nblk, 0, [&](int i) { return ((S.desc[i].y & 0xffff) + 1) & ~1; },
               [&](int i, int excl) {
                   S.desc[i].x = excl;
                   if (i == nblk - 1) S.meta[2] = excl + (((S.desc[i].y & 0xffff) + 1) & ~1);
               });
        T.sync();
        const int total = S.meta[2];
        in_smem = Team::kind == 0 && nblk + 2 <= B.smem_blocks;
        const int used = in_smem ? 0 : nblk + 2;
        const bool listed = (long long)total * 4 <= (long long)(S.cap - used) * 288;
        if (!listed) {
            T.sync();  // everyone has read the total
            if (tid == 0) S.meta[2] = 0;
        } else {
            uint32_t* const list = reinterpret_cast<uint32_t*>(S.slot + 36LL * used);
            for (int i = tid; i < nblk; i += nt) {
                const int4 d = S.desc[i];
                const int k = (d.y >> 16) & 255, u = (d.y >> 24) & 255;
                int o = d.x;
                for (int w = 0; w < W; ++w) {
                    uint32_t bits = S.rowb[k * W + w] & S.rowb[u * W + w];
                    while (bits) {
                        list[o++] = update_entry(S, k, u, (w << 5) + __ffs(bits) - 1);
                        bits &= bits - 1;
                    }
                }
                if (d.y & 1) list[o] = zero_entry(S, k, u);
            }
        }
        // the contacts of each off-diagonal block: of a body's incidences those
        // whose other body is eliminated later, grouped by block, in incidence
        // order (inc_o is the PCG's and holds the incidence's block meanwhile)
        for (int k = tid; k < n; k += nt) {
            const int gb = S.body[k];
            const int st0 = B.inc_start[gb], cnt = B.inc_cnt[gb];
            const int b0k = S.base[k] + 1, b1k = S.base[k] + S.height[k];
            S.desc[b0k - 1].z = st0;  // the diagonal block takes all of them
            S.desc[b0k - 1].w = st0 + cnt;
            for (int b = b0k; b < b1k; ++b) S.desc[b].z = 0;
            for (int q = 0; q < cnt; ++q) {
                const int go = B.inc_o[st0 + q];
                int blk = -1;
                if (go >= 0 && go != gb && B.local[go]) {
                    const int u = S.ipos[B.didx[go]];
                    if (u > k) {
                        blk = b0k + bit_rank(S.colb + k * W, u);
                        S.desc[blk].z += 1;
                    }
                }
                B.inc_o[st0 + q] = blk;
            }
            int o = st0;  // ends of the blocks' ranges, then each range filled from its end
            for (int b = b0k; b < b1k; ++b) S.desc[b].z = S.desc[b].w = o += S.desc[b].z;
            for (int q = cnt - 1; q >= 0; --q) {
                const int blk = B.inc_o[st0 + q];
                if (blk >= 0) B.inc_g[S.desc[blk].z -= 1] = st0 + q;
            }
        }
        T.sync();
        return true;
    }
    // Update-list entry of block (u, k) and column d: the block indices of L(u, d)
    // and L(k, d); for the diagonal block (u = k) those of L(k, d) and of d itself,
    // whose substitution vector the forward sweep takes.
    __device__ __forceinline__ static uint32_t update_entry(const Direct& S, int k, int u, int d) {
        const uint32_t* cd = S.colb + d * kSparseWords;
        const uint32_t a = (uint32_t)(S.base[d] + 1 + bit_rank(cd, u));
        return (a << 16) | (u == k ? (uint32_t)d : (uint32_t)(S.base[d] + 1 + bit_rank(cd, k)));
    }
    // The entry that pads a list to an even length: the zero block (and node).
    __device__ __forceinline__ uint32_t zero_entry(const Direct& S, int k, int u) const {
        const uint32_t z = (uint32_t)S.meta[1];
        return (z << 16) | (u == k ? (uint32_t)n_active : z);
    }

    // Symbolic factorisation on the large-scene teams (up to kSparseMaxLarge
    // nodes), every step spread over the team.  Ordering: multiple minimum
    // degree (Liu, ACM TOMS 11(2), 1985) -- each round eliminates the remaining
    // nodes of degree at most the minimum + kMmdDelta that have no neighbour of
    // that kind with a smaller key (mmd_key).  Those nodes are pairwise
    // non-adjacent, so the round equals eliminating them one at a time (in node
    // order); each remaining neighbour merges their patterns into its own and
    // takes its elimination-tree height from them.
    // Rows of the factor come from a transposed bitset indexed by elimination
    // position, so every row list is in elimination order.  Returns false (PCG)
    // if the factor does not fit the slot or its sequential depth is too large.
    // Ordering key: degree, then a fixed hash of the node, then the node.  With
    // the hash, independent equal-degree nodes along a chain or a strip leave in
    // the same round, as in cyclic reduction, so a stack of L bodies gives an
    // elimination tree of height ~log L instead of L / 2 (ends inward).
    __device__ __forceinline__ static unsigned long long mmd_key(int deg, int i) {
        unsigned long long z = (unsigned long long)i * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return ((unsigned long long)deg << 32) | ((z >> 48) << 16) | (unsigned long long)i;
    }
    // Sequential work of a column with m off-diagonal blocks and a row list of
    // `len` entries: row updates per lane, plus its level's fixed cost.
    __device__ __forceinline__ static int column_work(int m, int len) {
        return kLevelCost + ((6 * (m + 1) + 31) >> 5) * (1 + len);
    }
    __device__ bool sparse_symbolic_large() {
        Sparse S = sparse_ws();
        const int n = n_active, nw = (n + 31) >> 5;
        constexpr int W = kSpWords;
        sp_nw = nw;
        for (int q = tid; q < n * W; q += nt) {
            S.adj[q] = 0;
            S.radj[q] = 0;
        }
        for (int q = tid; q <= n; q += nt) {
            S.ipos[q] = -1;
            S.height[q] = 0;
            S.lvl_start[q] = 0;
            S.lvl_work[q] = 0;
            S.cstart[q] = 0;  // columns eliminated so far whose pattern holds the node
        }
        T.sync();
        for (int l = tid; l < n_local; l += nt) {  // node rows, each built by its owner
            const int gb = B.lbody[b0 + l];
            if (!active(gb)) continue;
            const int i = B.didx[gb];
            const int st0 = B.inc_start[gb], cnt = B.inc_cnt[gb];
            for (int k = 0; k < cnt; ++k) {
                const int e = B.inc[st0 + k];
                const int go = b0 + B.cbody[2 * (e >> 1) + (1 - (e & 1))];
                if (go == gb || !active(go)) continue;
                const int j = B.didx[go];
                S.adj[i * W + (j >> 5)] |= 1u << (j & 31);
            }
        }
        T.sync();
        for (int i = tid; i < n; i += nt) {
            int d = 0;
            for (int w = 0; w < nw; ++w) d += __popc(S.adj[i * W + w]);
            S.deg[i] = d;
        }
        T.sync();
        int done = 0;
        double fill = 0;
        for (int round = 0; round < kMmdMaxRounds; ++round) {
            double m[1] = {-1e300};  // minimum degree over the remaining nodes
            for (int i = tid; i < n; i += nt)
                if (S.ipos[i] < 0) m[0] = dmax(m[0], -(double)S.deg[i]);
            T.max(m);
            if (m[0] < -1e299) break;  // all eliminated
            const int dmin = (int)(-m[0]);
            // candidates: degree <= dmin + kMmdDelta; a candidate is taken unless a
            // neighbouring candidate has a smaller key
            const int dcap = dmin + kMmdDelta;
            for (int i = tid; i < n; i += nt) {
                int pick = 0;
                if (S.ipos[i] < 0 && S.deg[i] <= dcap) {
                    pick = 1;
                    const unsigned long long ki = mmd_key(S.deg[i], i);
                    const uint32_t* ai = S.adj + i * W;
                    for (int w = 0; w < nw && pick; ++w) {
                        uint32_t bits = ai[w];
                        while (bits) {
                            const int j = (w << 5) + __ffs(bits) - 1;
                            bits &= bits - 1;
                            if (S.deg[j] <= dcap && mmd_key(S.deg[j], j) < ki) {
                                pick = 0;
                                break;
                            }
                        }
                    }
                }
                S.sel[i] = pick;
            }
            T.sync();
            T.scan(n, done, [&](int i) { return S.sel[i]; },
                   [&](int i, int excl) {
                       if (S.sel[i]) {
                           S.perm[excl] = i;
                           S.ipos[i] = excl;
                       }
                   });
            {
                // Nodes eliminated this round, and what their columns add to the
                // factor's blocks and to its depth (their patterns, heights and
                // row lists are final).  Both only grow, so a factor that will
                // not fit or will be too deep is left as soon as it is: the last
                // rounds, one node of a dense separator each, cost the most.
                double c[2] = {0.0, 0.0};
                for (int i = tid; i < n; i += nt) {
                    if (!S.sel[i]) continue;
                    c[0] += 1;
                    c[1] += S.deg[i];
                    atomicMax(&S.lvl_work[S.height[i]], column_work(S.deg[i], S.cstart[i]));
                }
                T.sum(c);
                done += (int)c[0];
                fill += c[1];
                if (fill > S.cap || fill > kRowCapLarge) return false;
            }
            for (int u = tid; u < n; u += nt) {  // remaining neighbours merge the eliminated patterns
                if (S.ipos[u] >= 0) continue;
                uint32_t* au = S.adj + u * W;
                int h = S.height[u];
                bool touched = false;
                for (int w = 0; w < nw; ++w) {
                    uint32_t bits = au[w];
                    while (bits) {
                        const int v = (w << 5) + __ffs(bits) - 1;
                        bits &= bits - 1;
                        if (!S.sel[v]) continue;
                        touched = true;
                        S.cstart[u] += 1;
                        h = max(h, S.height[v] + 1);
                        const uint32_t* av = S.adj + v * W;
                        for (int x = 0; x < nw; ++x) au[x] |= av[x];
                        au[w] &= ~(1u << (v & 31));
                    }
                }
                if (touched) {
                    au[u >> 5] &= ~(1u << (u & 31));
                    int d = 0;
                    for (int w = 0; w < nw; ++w) d += __popc(au[w]);
                    S.deg[u] = d;
                    S.height[u] = h;
                }
            }
            double depth[1] = {0.0};
            for (int l = tid; l < n; l += nt) depth[0] += S.lvl_work[l];
            T.sum(depth);
            if (depth[0] > kDirectDepthMax) return false;
        }
        if (done != n) return false;  // round limit
        // block offsets in elimination order
        T.scan(n, 0,
               [&](int k) {
                   int c = 0;
                   for (int w = 0; w < nw; ++w) c += __popc(S.adj[S.perm[k] * W + w]);
                   return c;
               },
               [&](int k, int excl) {
                   S.cstart[S.perm[k]] = excl;
                   if (k == n - 1) {
                       int c = 0;
                       for (int w = 0; w < nw; ++w) c += __popc(S.adj[S.perm[k] * W + w]);
                       S.cstart[n] = excl + c;
                   }
               });
        if (S.cstart[n] > S.cap || S.cstart[n] > kRowCapLarge) return false;
        // row patterns: bit ipos(d) of row u for every u in pattern(d)
        for (int d = tid; d < n; d += nt) {
            const int kd = S.ipos[d];
            const uint32_t* ad = S.adj + d * W;
            for (int w = 0; w < nw; ++w) {
                uint32_t bits = ad[w];
                while (bits) {
                    const int u = (w << 5) + __ffs(bits) - 1;
                    bits &= bits - 1;
                    atomicOr(&S.radj[u * W + (kd >> 5)], 1u << (kd & 31));
                }
            }
        }
        T.sync();
        T.scan(n, 0,
               [&](int u) {
                   int c = 0;
                   for (int w = 0; w < nw; ++w) c += __popc(S.radj[u * W + w]);
                   return c;
               },
               [&](int u, int excl) {
                   S.rowptr[u] = excl;
                   if (u == n - 1) S.rowptr[n] = S.cstart[n];
               });
        // row lists in elimination order; levels by elimination-tree height
        double hw[1] = {0.0};
        for (int u = tid; u < n; u += nt) {
            int a = S.rowptr[u];
            for (int w = 0; w < nw; ++w) {
                uint32_t bits = S.radj[u * W + w];
                while (bits) {
                    const int k = (w << 5) + __ffs(bits) - 1;
                    bits &= bits - 1;
                    const int d = S.perm[k];
                    S.rowidx[a] = d;
                    S.rowoff[a++] = S.cstart[d] + bit_rank(S.adj + d * W, u);
                }
            }
            atomicAdd(&S.lvl_start[S.height[u] + 1], 1);
            hw[0] = dmax(hw[0], (double)S.height[u]);
        }
        T.max(hw);
        const int nlev = (int)hw[0] + 1;
        if (tid == 0) {
            for (int l = 0; l < nlev; ++l) S.lvl_start[l + 1] += S.lvl_start[l];
            S.meta[0] = nlev;
        }
        T.sync();
        for (int l = tid; l < nlev; l += nt) S.deg[l] = S.lvl_start[l];  // level cursors
        T.sync();
        // Columns of a level are independent, so their order within the level
        // changes no result.  Sequential work of column v as dense_solve_warp
        // does it (one warp, lanes over the 6 (m + 1) block rows): each lane
        // takes ceil(6 (m + 1) / 32) rows, each updated once per row-list entry;
        // plus the level's fixed cost.
        for (int v = tid; v < n; v += nt) {
            S.lvl_nodes[atomicAdd(&S.deg[S.height[v]], 1)] = v;
            int m = 0;
            for (int w = 0; w < nw; ++w) m += __popc(S.adj[v * W + w]);
            atomicMax(&S.lvl_work[S.height[v]], column_work(m, S.rowptr[v + 1] - S.rowptr[v]));
        }
        T.sync();
        double depth[1] = {0.0};
        for (int l = tid; l < nlev; l += nt) depth[0] += S.lvl_work[l];
        T.sum(depth);
        return depth[0] <= kDirectDepthMax;
    }

    // Column block of active body gb (large-scene teams): the diagonal block P and, per incidence
    // with a body eliminated later, the off-diagonal block T_o K^-1 T_b^T
    // (linsysAddition's four blocks, :232-247).  Each column is owned by its
    // body's thread, so accumulation is race free and in incidence order.
    __device__ void assemble_dense_rows(int gb, const double* P) const {
        Sparse S = sparse_ws();
        const int i = B.didx[gb];
        double* D = S.Dg + 36 * i;
        for (int r = 0; r < 6; ++r)
            for (int c = 0; c < 6; ++c) D[r * 6 + c] = P[pk(r, c)];
        const uint32_t* ai = S.adj + i * kSpWords;
        int m = 0;
        for (int w = 0; w < spw(); ++w) m += __popc(ai[w]);
        double* col = S.L + 36LL * S.cstart[i];
        for (int q = 0; q < 36 * m; ++q) col[q] = 0.0;
        const int st0 = B.inc_start[gb], n = B.inc_cnt[gb];
        for (int k = 0; k < n; ++k) {
            const int e2 = B.inc[st0 + k];
            const int gc = e2 >> 1, side = e2 & 1;
            const int go = b0 + B.cbody[2 * gc + (1 - side)];
            if (!active(go) || go == gb) continue;
            const int j = B.didx[go];
            if (S.ipos[j] < S.ipos[i]) continue;  // that block lives in j's column
            double* blk = col + 36 * bit_rank(ai, j);
            // block (rows o, cols b) = -[[W, C_b W]^T-form]: the transpose of
            // A_bo = -[[W, W C_o^T], [C_b W, C_b W C_o^T]]
            double W[12];
            ldg12(st0 + k, W);
            const d3 cb = ld3(W + 6), co = ld3(W + 9);
            const d3 wr[3] = {d3{W[0], W[3], W[4]}, d3{W[3], W[1], W[5]}, d3{W[4], W[5], W[2]}};
            const d3 y0 = cross3(cb, wr[0]), y1 = cross3(cb, wr[1]), y2 = cross3(cb, wr[2]);
            const d3 yr[3] = {d3{y0.x, y1.x, y2.x}, d3{y0.y, y1.y, y2.y}, d3{y0.z, y1.z, y2.z}};
            for (int r = 0; r < 3; ++r) {
                const d3 tr = cross3(co, wr[r]);  // row r of W C_o^T
                const d3 br = cross3(co, yr[r]);  // row r of C_b W C_o^T
                // A_bo(r, 0..2) = -wr[r], A_bo(r, 3..5) = -tr, A_bo(3+r, 0..2) = -yr[r], A_bo(3+r, 3..5) = -br
                // stored transposed: blk(c, r) = A_bo(r, c)
                blk[0 * 6 + r] -= wr[r].x; blk[1 * 6 + r] -= wr[r].y; blk[2 * 6 + r] -= wr[r].z;
                blk[3 * 6 + r] -= tr.x;    blk[4 * 6 + r] -= tr.y;    blk[5 * 6 + r] -= tr.z;
                blk[0 * 6 + 3 + r] -= yr[r].x; blk[1 * 6 + 3 + r] -= yr[r].y; blk[2 * 6 + 3 + r] -= yr[r].z;
                blk[3 * 6 + 3 + r] -= br.x;    blk[4 * 6 + 3 + r] -= br.y;    blk[5 * 6 + 3 + r] -= br.z;
            }
        }
    }

    // Lower Cholesky factor of a 6x6 SPD block (row-major) and the reciprocals
    // of its diagonal; false if not SPD.
    __device__ __forceinline__ static bool chol6(const double* A, double* L, double* Li) {
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            double d = A[j * 6 + j];
#pragma unroll
            for (int k = 0; k < j; ++k) d -= L[j * 6 + k] * L[j * 6 + k];
            if (!(d > 0.0)) return false;
            const double ljj = sqrt(d);
            const double inv = 1.0 / ljj;
            L[j * 6 + j] = ljj;
            Li[j] = inv;
#pragma unroll
            for (int i = j + 1; i < 6; ++i) {
                double t = A[i * 6 + j];
#pragma unroll
                for (int k = 0; k < j; ++k) t -= L[i * 6 + k] * L[j * 6 + k];
                L[i * 6 + j] = t * inv;
            }
#pragma unroll
            for (int c = j + 1; c < 6; ++c) L[j * 6 + c] = 0.0;
        }
        return true;
    }
    // y = L^-1 b
    __device__ __forceinline__ static void lsolve6(const double* L, const double* Li, const double* b, double* y) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            double t = b[i];
#pragma unroll
            for (int k = 0; k < i; ++k) t -= L[i * 6 + k] * y[k];
            y[i] = t * Li[i];
        }
    }
    // x = L^-T y
    __device__ __forceinline__ static void ltsolve6(const double* L, const double* Li, const double* y, double* x) {
#pragma unroll
        for (int i = 5; i >= 0; --i) {
            double t = y[i];
#pragma unroll
            for (int k = i + 1; k < 6; ++k) t -= L[k * 6 + i] * x[k];
            x[i] = t * Li[i];
        }
    }
    // Position of element (r, c) of a 6x6 block in memory: columns 0-3 by rows,
    // then columns 4-5 by rows.  Lanes 0-23 of a warp read the first 24 doubles
    // as the k = 0..3 operand of an m8n8k4 product in one run, the last 12 give
    // half of a second operand, and a row is three aligned pairs.
    __device__ __forceinline__ static constexpr int frag(int r, int c) { return c < 4 ? 4 * r + c : 24 + 2 * r + c - 4; }
    __device__ __forceinline__ static void st_row(double* p, int r, const double* v) {
        *reinterpret_cast<double2*>(p + 4 * r) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2*>(p + 4 * r + 2) = make_double2(v[2], v[3]);
        *reinterpret_cast<double2*>(p + 24 + 2 * r) = make_double2(v[4], v[5]);
    }
    // (c0, c1) += A B for the warp's 8x4 A (a = A[lane / 4][lane % 4]), 4x8 B (b =
    // B[lane % 4][lane / 4]); the lane holds C[lane / 4][2 (lane % 4) + {0, 1}]
    __device__ __forceinline__ static void mma884(double& c0, double& c1, double a, double b) {
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(c0), "+d"(c1)
                     : "d"(a), "d"(b));
    }

    __device__ __forceinline__ static void ld_row(const double* p, int r, double* v) {
        const double2 a = *reinterpret_cast<const double2*>(p + 4 * r), b = *reinterpret_cast<const double2*>(p + 4 * r + 2),
                      c = *reinterpret_cast<const double2*>(p + 24 + 2 * r);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
    }
    // In place: the strictly lower part of a 6x6 SPD block's Cholesky factor and
    // the reciprocals of its diagonal (all that the substitutions read), and
    // y = L^-1 y; false if not SPD.
    __device__ __forceinline__ static bool chol6_block(double* A, double* y) {
        double L[6][6], inv[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            double d = A[frag(j, j)];
#pragma unroll
            for (int k = 0; k < j; ++k) d -= L[j][k] * L[j][k];
            if (!(d > 0.0)) return false;
            inv[j] = 1.0 / sqrt(d);
#pragma unroll
            for (int i = j + 1; i < 6; ++i) {
                double t = A[frag(i, j)];
#pragma unroll
                for (int k = 0; k < j; ++k) t -= L[i][k] * L[j][k];
                L[i][j] = t * inv[j];
            }
        }
        double b[6];
        ld6(y, b);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            A[frag(i, i)] = inv[i];
            double t = b[i];
#pragma unroll
            for (int k = 0; k < i; ++k) {
                A[frag(i, k)] = L[i][k];
                t -= L[i][k] * b[k];
            }
            b[i] = t * inv[i];
        }
        st6(y, b);
        return true;
    }

    // The Newton matrix and right-hand side of the block and warp teams' factor
    // (linsysAddition's four blocks, :232-247), one thread per pair of rows i, 3 +
    // i of a block: block (u, k) = T_u W T_k^T summed over the contacts of the two
    // bodies in incidence order, T_j = s_j [I; C_j] with C_j = [c_j]x, with the
    // sign of s_u s_k, i.e. [W, (C_k W)^T; C_u W, C_u (C_k W)^T]; a diagonal block
    // starts from M / cm + eps I, takes every contact of the body, and its threads
    // also sum rhs = sum T_j K^-1 sf - ru; blocks that only fill in are zero.  The
    // three threads of a block run the same instructions (component i of a cross
    // product by selecting its two factors).  Roundings are spelled out (which of
    // a cross product's two terms is fused), so that a change elsewhere in the
    // kernel cannot move the results of scenes that amplify the last bit.
    template <bool SM>
    __device__ void assemble_rows(double eps) const {
        const Direct S = direct_ws();
        double* const L = block_base<SM>(S);
        const int nblk = S.meta[1], items = 3 * nblk;
        for (int t = tid; t < items; t += nt) {
            const int b = t / 3, i = t - 3 * b;
            const int4 de = S.desc[b];
            const int k = (de.y >> 16) & 255, u = (de.y >> 24) & 255, gb = S.body[k];
            const bool diag = k == u, is0 = i == 0, is1 = i == 1;
            auto pick = [&](double x, double y, double z) { return is0 ? x : (is1 ? y : z); };  // component i
            auto cross_i = [&](double cp, double cq, d3 v) {  // component i of c x v, c_(i+1), c_(i+2) given
                return __fma_rn(cp, pick(v.z, v.x, v.y), -__dmul_rn(cq, pick(v.y, v.z, v.x)));
            };
            double lo[6] = {0, 0, 0, 0, 0, 0}, hi[6] = {0, 0, 0, 0, 0, 0}, fl = 0, fh = 0;
            if (diag) {
                const double m = B.mass[gb] / cm + eps;
                const double* I = B.inertia + 6 * gb;
                const double xx = I[0] / cm + eps, yy = I[1] / cm + eps, zz = I[2] / cm + eps;
                const double xy = I[3] / cm, xz = I[4] / cm, yz = I[5] / cm;
                lo[0] = pick(m, 0.0, 0.0); lo[1] = pick(0.0, m, 0.0); lo[2] = pick(0.0, 0.0, m);
                hi[3] = pick(xx, xy, xz); hi[4] = pick(xy, yy, yz); hi[5] = pick(xz, yz, zz);
            }
            for (int q = de.z; q < de.w; ++q) {
                const int slot = diag ? q : B.inc_g[q];
                double g[12];
                ldg12(slot, g);
                const d3 ck = ld3(g + 6), cu = diag ? ck : ld3(g + 9);
                const d3 w0 = d3{g[0], g[3], g[4]}, w1 = d3{g[3], g[1], g[5]}, w2 = d3{g[4], g[5], g[2]};
                const d3 y0 = cross_rn(ck, w0), y2 = cross_rn(ck, w2);  // columns of C_k W
                d3 y1 = cross_rn(ck, w1);
                y1.y = __fma_rn(-ck.x, w1.z, __dmul_rn(ck.z, w1.x));
                const double s = diag ? 1.0 : -1.0;
                lo[0] += s * pick(w0.x, w1.x, w2.x); lo[1] += s * pick(w0.y, w1.y, w2.y); lo[2] += s * pick(w0.z, w1.z, w2.z);
                lo[3] += s * pick(y0.x, y1.x, y2.x); lo[4] += s * pick(y0.y, y1.y, y2.y); lo[5] += s * pick(y0.z, y1.z, y2.z);
                const double cp = pick(cu.y, cu.z, cu.x), cq = pick(cu.z, cu.x, cu.y);
                hi[0] += s * cross_i(cp, cq, w0);
                hi[1] += s * (is1 ? __fma_rn(-cq, w1.z, __dmul_rn(cp, w1.x)) : cross_i(cp, cq, w1));
                hi[2] += s * cross_i(cp, cq, w2);
                hi[3] += s * cross_i(cp, cq, d3{y0.x, y1.x, y2.x});
                hi[4] += s * cross_i(cp, cq, d3{y0.y, y1.y, y2.y});
                hi[5] += s * cross_i(cp, cq, d3{y0.z, y1.z, y2.z});
                if (diag) {
                    const d3 x = fld3(incidence(slot), I_X);
                    fl += pick(x.x, x.y, x.z);
                    fh += cross_i(cp, cq, x);
                }
            }
            if (diag) {
                S.y[6 * k + i] = fl - B.ru[6 * gb + i];
                S.y[6 * k + 3 + i] = fh - B.ru[6 * gb + 3 + i];
            }
            st_row(L + 36 * b, i, lo);
            st_row(L + 36 * b, 3 + i, hi);
        }
        for (int t = tid; t < 36; t += nt) {
            L[36 * nblk + t] = 0.0;
            if (t < 6) S.y[6 * n_active + t] = 0.0;
        }
    }

    // Entry `r` of block (u, k)'s update list without the list: the r-th column
    // in the rows of both
    __device__ __forceinline__ uint32_t find_entry(const Direct& S, int k, int u, int r) const {
        for (int w = 0; w < kSparseWords; ++w) {
            uint32_t x = S.rowb[k * kSparseWords + w] & S.rowb[u * kSparseWords + w];
            const int c = __popc(x);
            if (r < c) {
                for (; r > 0; --r) x &= x - 1;
                return update_entry(S, k, u, (w << 5) + __ffs(x) - 1);
            }
            r -= c;
        }
        return zero_entry(S, k, u);
    }
    // Block i = (u, k) -= the products of its update list, by one warp: two
    // entries per round, the first four columns of each (heads) as one product
    // and the last two of both in a third.  Rows 6 and 7 of the operands hold
    // what lies there: they only reach rows and columns of the product that are
    // not used, but for a diagonal block, which multiplies L(k, d) by its own
    // transpose with y_d as row 6 of the second factor, so that column 6 of the
    // product is the forward substitution's part.  One entry is 6 cycles of the
    // load-store unit; a thread per block row, loading its factor's 36 values
    // again for every row, took 29.
    __device__ __forceinline__ void update_block(const Direct& S, double* L, int i, int4 de, bool listed,
                                                 int lane) const {
        const int row = lane >> 2, kk = lane & 3, n = de.y & 0xffff;
        const int k = (de.y >> 16) & 255, u = (de.y >> 24) & 255;
        const bool diag = k == u, ycol = diag && row == 6;
        const int tail = 24 + 2 * row + (kk & 1);
        const uint2* const list = reinterpret_cast<const uint2*>(S.list + de.x);
        double s0 = 0, s1 = 0, t0 = 0, t1 = 0;
        uint2 e = make_uint2(0, 0);
        if (listed) e = list[0];
        for (int q = 0; q < n; q += 2) {
            uint2 now = e;
            if (listed) {
                if (q + 2 < n) e = list[(q >> 1) + 1];
            } else {
                now = make_uint2(find_entry(S, k, u, q), find_entry(S, k, u, q + 1));
            }
            const double* const A0 = L + 36 * (now.x >> 16);
            const double* const A1 = L + 36 * (now.y >> 16);
            const double a0 = A0[lane], a1 = A1[lane], at = (kk < 2 ? A0 : A1)[tail];
            double b0, b1, bt;
            if (diag) {
                b0 = a0, b1 = a1, bt = at;
                if (ycol) {
                    const double *y0 = S.y + 6 * (now.x & 0xffffu), *y1 = S.y + 6 * (now.y & 0xffffu);
                    b0 = y0[kk];
                    b1 = y1[kk];
                    bt = (kk < 2 ? y0 : y1)[4 + (kk & 1)];
                }
            } else {
                const double* const B0 = L + 36 * (now.x & 0xffffu);
                const double* const B1 = L + 36 * (now.y & 0xffffu);
                b0 = B0[lane];
                b1 = B1[lane];
                bt = (kk < 2 ? B0 : B1)[tail];
            }
            mma884(s0, s1, a0, b0);
            mma884(t0, t1, a1, b1);
            mma884(s0, s1, at, bt);
        }
        s0 += t0;
        s1 += t1;
        if (row < 6) {
            if (kk < 3) {
                double2* c = reinterpret_cast<double2*>(L + 36 * i + (kk < 2 ? 4 * row + 2 * kk : 24 + 2 * row));
                const double2 v = *c;
                *c = make_double2(v.x - s0, v.y - s1);
            } else if (diag) {
                S.y[6 * k + row] -= s0;  // column 6
            }
        }
    }

    // The same for a level of short lists (at most kShortList entries): a thread
    // per block row, entry by entry.
    __device__ __forceinline__ void update_rows(const Direct& S, double* L, int i0, int i1, bool listed) const {
        for (int t = tid; t < 6 * (i1 - i0); t += nt) {
            const int i = i0 + t / 6, r = t - 6 * (i - i0);
            const int4 de = S.desc[i];
            const int n = de.y & 0xffff;
            if (n == 0) continue;
            const int k = (de.y >> 16) & 255, u = (de.y >> 24) & 255;
            const bool diag = k == u;
            double acc[6], yr = 0;
            ld_row(L + 36 * i, r, acc);
            if (diag) yr = S.y[6 * k + r];
            for (int q = 0; q < n; ++q) {
                const uint32_t e = listed ? S.list[de.x + q] : find_entry(S, k, u, q);
                const double* const A = L + 36 * (e >> 16);
                const double* const Bm = diag ? A : L + 36 * (e & 0xffffu);
                double x[6], b[6];
                ld_row(A, r, x);
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    ld_row(Bm, c, b);
                    double s = 0.0;
#pragma unroll
                    for (int p = 0; p < 6; ++p) s += x[p] * b[p];
                    acc[c] -= s;
                }
                if (diag) {
                    ld6(S.y + 6 * (e & 0xffffu), b);
                    double s = 0.0;
#pragma unroll
                    for (int p = 0; p < 6; ++p) s += x[p] * b[p];
                    yr -= s;
                }
            }
            st_row(L + 36 * i, r, acc);
            if (diag) S.y[6 * k + r] = yr;
        }
    }

    // Block Cholesky factorisation and both substitutions of the Newton system
    // (block and warp teams; left-looking), one elimination-tree level at a time,
    // the forward substitution riding along as one more column of each diagonal
    // block.  Per level: (1) the blocks take their updates, a warp per block or,
    // where the lists are short, a thread per row; (2) a thread per column
    // factors its diagonal block and finishes its part of the forward
    // substitution; (3) a thread per row scales the other blocks, A(u, k) L_kk^-T.
    // The backward substitution gives a column 8, 16 or 32 lanes (component x
    // blocks) and no barrier but the level's.  Levels of short lists and patterns
    // (stacks, columns, loose piles) sum entry by entry in elimination order.
    // Long lists run on the FP64 matrix instruction: it has the rate of the FP64
    // pipe, but feeds 256 multiply-adds from two loads per lane, wherever the blocks
    // are (in global memory, a thread per row instead: crate of 144 cubes 5.85 ->
    // 7.51 ms, 1,024 crates of up to 216 12.8 -> 16.9 ms).  Stands in for the
    // direct branch's SimplicialLDLT (:385-394).  Writes du; false on a
    // non-SPD pivot, which only marks the scene: later columns then compute
    // garbage in bounded loops.
    template <bool SM>
    __device__ bool direct_solve() {
        const Direct S = direct_ws();
        double* const L = block_base<SM>(S);
        const int nlev = S.meta[0];
        const bool listed = S.meta[2] > 0;
        const int lane = tid & 31, warp = tid >> 5, nwarp = nt >> 5;
        bool bad = false;
        int q1 = 0, i1 = 0;
        for (int l = 0; l < nlev; ++l) {
            const int q0 = q1, i0 = i1;
            q1 = S.lvl_start[l + 1];
            i1 = S.lvl_blk[l + 1];
            const int len = S.lvl_len[l];
            if (len > 0) {
                if (len <= kShortList) {
                    update_rows(S, L, i0, i1, listed);
                } else {
                    for (int i = i0 + warp; i < i1; i += nwarp) {
                        const int4 de = S.desc[i];
                        if ((de.y & 0xffff) != 0) update_block(S, L, i, de, listed, lane);
                    }
                }
                T.sync();
            }
            for (int q = q0 + tid; q < q1; q += nt) {
                const int k = S.lvl_cols[q];
                if (!chol6_block(L + 36 * S.base[k], S.y + 6 * k)) bad = true;
            }
            T.sync();
            if (i1 - i0 == q1 - q0) continue;  // no off-diagonal block in this level
            for (int t = tid; t < 6 * (i1 - i0); t += nt) {
                const int i = i0 + t / 6, r = t - 6 * (i - i0);
                const int y = S.desc[i].y, k = (y >> 16) & 255;
                if (((y >> 24) & 255) == k) continue;
                const double* const D = L + 36 * S.base[k];
                double a[6];
                ld_row(L + 36 * i, r, a);
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    double s = a[c];
#pragma unroll
                    for (int q = 0; q < c; ++q) s -= D[frag(c, q)] * a[q];
                    a[c] = s * D[frag(c, c)];
                }
                st_row(L + 36 * i, r, a);
            }
            T.sync();
        }
        if (T.any(bad)) return false;
        const int c8 = tid & 7, c = min(c8, 5);
        const int e0 = c < 4 ? c : 20 + c, es = c < 4 ? 4 : 2;  // column c of a block: e0 + r es
        int p1 = S.lvl_start[nlev];
        for (int l = nlev - 1; l >= 0; --l) {
            const int p0 = S.lvl_start[l], ncol = p1 - p0;
            p1 = p0;
            // 1, 2 or 4 groups of 8 lanes per column
            const int lg = S.lvl_pat[l] <= kShortList ? 0 : (ncol * 32 <= nt ? 2 : (ncol * 16 <= nt ? 1 : 0));
            const int sub = 1 << lg;
            const int ng = nt >> (3 + lg), grp = tid >> (3 + lg), j = (tid >> 3) & (sub - 1);
            for (int g0 = 0; g0 < ncol; g0 += ng) {
                const bool on = g0 + grp < ncol;
                const int k = S.lvl_cols[p0 + (on ? g0 + grp : 0)];
                const int blk = S.base[k];
                const int m = on ? S.height[k] - 1 : 0;
                double r = j == 0 ? S.y[6 * k + c] : 0.0;
#pragma unroll 2
                for (int a = 1 + j; a <= m; a += sub) {
                    const double* Lb = L + 36 * (blk + a) + e0;
                    const double* x = S.y + 6 * ((S.desc[blk + a].y >> 24) & 255);
                    double s = 0.0;
#pragma unroll
                    for (int p = 0; p < 6; ++p) s += Lb[es * p] * x[p];
                    r -= s;
                }
                for (int o = 8; o < 8 * sub; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
                const double* D = L + 36 * blk;
                double xs[6], x = 0.0;  // every lane: x = L_kk^-T r
#pragma unroll
                for (int p = 0; p < 6; ++p) xs[p] = __shfl_sync(0xffffffffu, r, p, 8);
#pragma unroll
                for (int p = 5; p >= 0; --p) {
                    double t = xs[p];
#pragma unroll
                    for (int q = p + 1; q < 6; ++q) t -= D[frag(q, p)] * xs[q];
                    xs[p] = t * D[frag(p, p)];
                    if (p == c) x = xs[p];
                }
                __syncwarp();
                if (on && j == 0 && c8 < 6) {
                    S.y[6 * k + c8] = x;
                    B.du[6 * S.body[k] + c8] = x;
                }
            }
            T.sync();
        }
        return true;
    }

    // node of the a-th set bit among the first nw words of a pattern
    __device__ __forceinline__ static int bit_select_n(const uint32_t* w, int a, int nw) {
        for (int k = 0; k < nw; ++k) {
            const int c = __popc(w[k]);
            if (a < c) {
                uint32_t x = w[k];
                for (int q = 0; q < a; ++q) x &= x - 1;
                return (k << 5) + __ffs(x) - 1;
            }
            a -= c;
        }
        return -1;
    }
    __device__ __forceinline__ static void warp_sum6(double* s) {
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[i] += __shfl_down_sync(0xffffffffu, s[i], o);
    }

    // The same factorisation and sweeps on the large-scene teams, which run one
    // scene, so a level's time is its slowest column's chain of dependent loads:
    // one warp per column (the level's columns strided over the team's warps).
    // Lanes take the rows of the column's blocks -- row r of each L(u, v), u in
    // pattern(v), and of the diagonal block -- and subtract their updates over
    // the column's row list in elimination order, in place; lane 0 factors the
    // diagonal block; then the lanes scale their rows by L_vv^-T, and the same
    // warp does the column's forward substitution (its row list's columns are
    // all in earlier levels), so one sweep over the levels factors and
    // substitutes forward.  In the substitutions the lanes split a column's sum
    // and combine it by a fixed shuffle tree.
    __device__ bool dense_solve_warp() {
        Sparse S = sparse_ws();
        const int nlev = S.meta[0];
        const int nw = spw();
        const int lane = tid & 31, gwarp = tid >> 5, nwarp = nt >> 5;
        int bad = 0;
        for (int l = 0; l < nlev; ++l) {
            for (int q = S.lvl_start[l] + gwarp; q < S.lvl_start[l + 1]; q += nwarp) {
                const int v = S.lvl_nodes[q];
                const uint32_t* av = S.adj + v * kSpWords;
                double* colv = S.L + 36LL * S.cstart[v];
                int m = 0;
                for (int w = 0; w < nw; ++w) m += __popc(av[w]);
                const int r0 = S.rowptr[v], r1 = S.rowptr[v + 1];
                for (int t = lane; t < 6 * (m + 1); t += 32) {
                    const int a = t / 6, r = t - 6 * a;
                    const bool diag = a == m;
                    const int u = diag ? v : bit_select_n(av, a, nw);
                    double* dst = diag ? S.Dg + 36 * v + 6 * r : colv + 36 * a + 6 * r;
                    double acc[6];
                    for (int c = 0; c < 6; ++c) acc[c] = dst[c];
                    for (int k = r0; k < r1; ++k) {
                        const double* Lvd = S.L + 36LL * S.rowoff[k];
                        const double* Lud = Lvd;
                        if (!diag) {
                            const int d = S.rowidx[k];
                            const uint32_t* ad = S.adj + d * kSpWords;
                            if (!((ad[u >> 5] >> (u & 31)) & 1u)) continue;
                            Lud = S.L + 36LL * (S.cstart[d] + bit_rank(ad, u));
                        }
                        double x[6];
                        for (int p = 0; p < 6; ++p) x[p] = Lud[6 * r + p];
                        for (int c = 0; c < 6; ++c) {
                            double s = 0.0;
                            for (int p = 0; p < 6; ++p) s += x[p] * Lvd[6 * c + p];
                            acc[c] -= s;
                        }
                    }
                    for (int c = 0; c < 6; ++c) dst[c] = acc[c];
                }
                __syncwarp();
                int ok = 0;
                if (lane == 0) {
                    double D[36], Lvv[36], Li[6];
                    for (int e = 0; e < 36; ++e) D[e] = S.Dg[36 * v + e];
                    if (chol6(D, Lvv, Li)) {
                        ok = 1;
                        for (int e = 0; e < 36; ++e) S.Ld[36 * v + e] = Lvv[e];
                        for (int e = 0; e < 6; ++e) S.Ldi[6 * v + e] = Li[e];
                    } else {
                        bad = 1;
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                __syncwarp();
                if (ok) {
                    for (int t = lane; t < 6 * m; t += 32) {  // L(u,v) = A(u,v) L_vv^-T, row by row
                        double* row = colv + 6 * t;
                        double out[6];
                        lsolve6(S.Ld + 36 * v, S.Ldi + 6 * v, row, out);
                        for (int c = 0; c < 6; ++c) row[c] = out[c];
                    }
                    // forward substitution of this column (every d of its row list
                    // is in an earlier level): y_v = L_vv^-1 (b_v - sum L(v,d) y_d)
                    double s6[6] = {0, 0, 0, 0, 0, 0};
                    for (int k = r0 + lane; k < r1; k += 32) {
                        const double* Lvd = S.L + 36LL * S.rowoff[k];
                        const double* yd = S.y + 6 * S.rowidx[k];
                        for (int i = 0; i < 6; ++i) {
                            double t = 0.0;
                            for (int c = 0; c < 6; ++c) t += Lvd[6 * i + c] * yd[c];
                            s6[i] += t;
                        }
                    }
                    warp_sum6(s6);
                    if (lane == 0) {
                        const int gb = B.dbody[b0 + v];
                        double b6[6], yv[6];
                        for (int r = 0; r < 6; ++r) b6[r] = B.rhs[6 * gb + r] - s6[r];
                        lsolve6(S.Ld + 36 * v, S.Ldi + 6 * v, b6, yv);
                        for (int r = 0; r < 6; ++r) S.y[6 * v + r] = yv[r];
                    }
                }
            }
            T.sync();  // level barrier; a failed pivot is checked once after the factorisation
        }
        {
            double fl[1] = {(double)bad};
            T.max(fl);
            bad = fl[0] > 0;
        }
        if (!bad) {
            for (int l = nlev - 1; l >= 0; --l) {  // backward: x_v = L_vv^-T (y_v - sum L(u,v)^T x_u)
                for (int q = S.lvl_start[l] + gwarp; q < S.lvl_start[l + 1]; q += nwarp) {
                    const int v = S.lvl_nodes[q];
                    const uint32_t* av = S.adj + v * kSpWords;
                    const double* colv = S.L + 36LL * S.cstart[v];
                    double s6[6] = {0, 0, 0, 0, 0, 0};
                    int a = 0;
                    for (int w = 0; w < nw; ++w) {
                        uint32_t bits = av[w];
                        while (bits) {
                            const int u = (w << 5) + __ffs(bits) - 1;
                            bits &= bits - 1;
                            if ((a & 31) == lane) {
                                const double* blk = colv + 36 * a;
                                const double* xu = S.x + 6 * u;
                                for (int c = 0; c < 6; ++c) {
                                    double t = 0.0;
                                    for (int r = 0; r < 6; ++r) t += blk[6 * r + c] * xu[r];
                                    s6[c] += t;
                                }
                            }
                            ++a;
                        }
                    }
                    warp_sum6(s6);
                    if (lane == 0) {
                        double r6[6], xv[6];
                        for (int r = 0; r < 6; ++r) r6[r] = S.y[6 * v + r] - s6[r];
                        ltsolve6(S.Ld + 36 * v, S.Ldi + 6 * v, r6, xv);
                        for (int r = 0; r < 6; ++r) S.x[6 * v + r] = xv[r];
                        const int gb = B.dbody[b0 + v];
                        for (int r = 0; r < 6; ++r) B.du[6 * gb + r] = xv[r];
                    }
                }
                T.sync();
            }
        }
        T.sync();
        return !bad;
    }

    // ------------------------------------------------ mixed precision solve
    // FP64 iterative refinement of A du = rhs around an FP32 block-Jacobi PCG:
    // r = rhs - A du in FP64 (matrix-free, FP64 W), e = A^-1 r approximately in
    // FP32 (FP32 W, X, vectors, preconditioner, FP32 accumulation), du += e.
    // Returns false on a non-finite residual; conv = refinement reached rtol.
    __device__ bool mixed_solve(double eps, double bnorm, double rtol, int& inner_total, bool& conv) {
        inner_total = 0;
        conv = true;
        for (int i = tid; i < n_local; i += nt) {
            const int gb = B.lbody[b0 + i];
            if (!active(gb)) continue;
            for (int r = 0; r < 6; ++r) {
                B.du[6 * gb + r] = 0;
                B.r[6 * gb + r] = B.rhs[6 * gb + r];
            }
        }
        T.sync();
        if (bnorm == 0) return true;
        double res = 1.0;
        const float epsf = (float)eps;
        for (int outer = 0;; ++outer) {
            if (!(res >= rtol)) break;
            if (outer >= C.max_outer) {
                conv = false;
                break;
            }
            // inner FP32 PCG on A e = r, e0 = 0
            double s2[2] = {0, 0};
            for (int i = tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (!active(gb)) continue;
                float r6[6], z6[6];
                for (int q = 0; q < 6; ++q) r6[q] = (float)B.r[6 * gb + q];
                prec_f(gb, r6, z6);
                for (int q = 0; q < 6; ++q) {
                    B.rF[6 * gb + q] = r6[q];
                    B.zF[6 * gb + q] = z6[q];
                    B.pF[6 * gb + q] = 0.f;
                    B.eF[6 * gb + q] = 0.f;
                    s2[0] += (double)(r6[q] * z6[q]);
                    s2[1] += (double)(r6[q] * r6[q]);
                }
            }
            T.sum(s2);
            float rz = (float)s2[0];
            const double r0 = sqrt(s2[1]);
            float beta = 0.f;
            for (int it = 0; it < C.max_direct && r0 > 0; ++it) {
                spmv_to_Xf(beta);
                T.sync();
                double s3[1] = {0};
                for (int i = tid; i < n_local; i += nt) {
                    const int gb = B.lbody[b0 + i];
                    if (!active(gb)) continue;
                    float pn[6], q6[6];
                    for (int q = 0; q < 6; ++q) {
                        pn[q] = __fadd_rn(B.zF[6 * gb + q], __fmul_rn(beta, B.pF[6 * gb + q]));
                        B.pF[6 * gb + q] = pn[q];
                    }
                    spmv_body_f(gb, pn, epsf, q6);
                    float acc = 0.f;
                    for (int q = 0; q < 6; ++q) {
                        acc += pn[q] * q6[q];
                        B.zF[6 * gb + q] = q6[q];
                    }
                    s3[0] += (double)acc;
                }
                T.sum(s3);
                // breakdown (p^T A p not positive in FP32, or a non-finite step):
                // keep the correction so far, the FP64 residual decides
                const float alpha = rz / (float)s3[0];
                if (!(s3[0] > 0.0) || !isfinite(alpha)) break;
                double s4[2] = {0, 0};
                for (int i = tid; i < n_local; i += nt) {
                    const int gb = B.lbody[b0 + i];
                    if (!active(gb)) continue;
                    float r6[6], z6[6];
                    for (int q = 0; q < 6; ++q) {
                        B.eF[6 * gb + q] += alpha * B.pF[6 * gb + q];
                        r6[q] = B.rF[6 * gb + q] - alpha * B.zF[6 * gb + q];
                        B.rF[6 * gb + q] = r6[q];
                    }
                    prec_f(gb, r6, z6);
                    float a0 = 0.f, a1 = 0.f;
                    for (int q = 0; q < 6; ++q) {
                        B.zF[6 * gb + q] = z6[q];
                        a0 += r6[q] * r6[q];
                        a1 += r6[q] * z6[q];
                    }
                    s4[0] += (double)a0;
                    s4[1] += (double)a1;
                }
                T.sum(s4);
                ++inner_total;
                if (!(sqrt(s4[0]) >= C.inner_rtol * r0)) break;
                beta = (float)s4[1] / rz;
                rz = (float)s4[1];
            }
            // du += e; FP64 residual r = rhs - A du
            for (int i = tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (!active(gb)) continue;
                for (int q = 0; q < 6; ++q) B.du[6 * gb + q] += (double)B.eF[6 * gb + q];
            }
            T.sync();
            spmv_to_X(B.du);
            T.sync();
            double s5[1] = {0};
            for (int i = tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (!active(gb)) continue;
                double q6[6];
                spmv_body(gb, B.du + 6 * gb, eps, q6);
                for (int q = 0; q < 6; ++q) {
                    const double rv = B.rhs[6 * gb + q] - q6[q];
                    B.r[6 * gb + q] = rv;
                    s5[0] += rv * rv;
                }
            }
            T.sum(s5);
            const double prev = res;
            res = sqrt(s5[0]) / bnorm;
            if (!isfinite(res)) return false;
            // a refinement step that does not halve the residual means the FP32
            // solve cannot resolve this system: let the FP64 solve take it
            if (outer > 0 && !(res < 0.5 * prev) && !(res < rtol)) {
                conv = false;
                break;
            }
        }
        return true;
    }
    // FP32 versions of the matrix-free product and the preconditioner
    __device__ __forceinline__ void spmv_to_Xf(float beta) const {
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            float pv[2][3];
            for (int j = 0; j < 2; ++j) {
                const int gb = b0 + B.cbody[2 * gc + j];
                if (B.is_static[gb]) {
                    pv[j][0] = pv[j][1] = pv[j][2] = 0.f;
                    continue;
                }
                float pn[6];
                for (int q = 0; q < 6; ++q) pn[q] = __fadd_rn(B.zF[6 * gb + q], __fmul_rn(beta, B.pF[6 * gb + q]));
                const d3 ca = arm(contact(gc), j);
                const float cx = (float)ca.x, cy = (float)ca.y, cz = (float)ca.z;
                pv[j][0] = pn[0] + (pn[4] * cz - pn[5] * cy);
                pv[j][1] = pn[1] + (pn[5] * cx - pn[3] * cz);
                pv[j][2] = pn[2] + (pn[3] * cy - pn[4] * cx);
            }
            const float* W = B.Wf + 6 * gc;
            const float d0 = pv[1][0] - pv[0][0], d1 = pv[1][1] - pv[0][1], d2 = pv[1][2] - pv[0][2];
            B.Xf[3 * gc] = W[0] * d0 + W[3] * d1 + W[4] * d2;
            B.Xf[3 * gc + 1] = W[3] * d0 + W[1] * d1 + W[5] * d2;
            B.Xf[3 * gc + 2] = W[4] * d0 + W[5] * d1 + W[2] * d2;
        }
    }
    __device__ __forceinline__ void spmv_body_f(int gb, const float* x6, float epsf, float* q6) const {
        const float icm = (float)(1.0 / cm);
        const float m = (float)B.mass[gb] * icm;
        const double* I = B.inertia + 6 * gb;
        const float Ixx = (float)I[0] * icm, Iyy = (float)I[1] * icm, Izz = (float)I[2] * icm;
        const float Ixy = (float)I[3] * icm, Ixz = (float)I[4] * icm, Iyz = (float)I[5] * icm;
        float a[6] = {m * x6[0], m * x6[1], m * x6[2], Ixx * x6[3] + Ixy * x6[4] + Ixz * x6[5],
                      Ixy * x6[3] + Iyy * x6[4] + Iyz * x6[5], Ixz * x6[3] + Iyz * x6[4] + Izz * x6[5]};
        const int st = B.inc_start[gb], n = B.inc_cnt[gb];
        for (int k = 0; k < n; ++k) {
            const int e = B.inc[st + k];
            const int gc = e >> 1, side = e & 1;
            const float sg = side ? 1.f : -1.f;
            const float x = sg * B.Xf[3 * gc], y = sg * B.Xf[3 * gc + 1], z = sg * B.Xf[3 * gc + 2];
            const d3 ca = fld3(incidence(st + k), I_arm);
            const float cx = (float)ca.x, cy = (float)ca.y, cz = (float)ca.z;
            a[0] += x; a[1] += y; a[2] += z;
            a[3] += cy * z - cz * y; a[4] += cz * x - cx * z; a[5] += cx * y - cy * x;
        }
        for (int q = 0; q < 6; ++q) q6[q] = a[q] + epsf * x6[q];
    }
    __device__ __forceinline__ void prec_f(int gb, const float* r6, float* z6) const {
        const float* Pi = B.pinvf + 21 * gb;
        for (int a = 0; a < 6; ++a) {
            float s = 0.f;
            for (int c = 0; c < 6; ++c) s += Pi[pk(a, c)] * r6[c];
            z6[a] = s;
        }
    }

    // X = W (v1p - v0p) of direction vec, with the direction of static /
    // non-active bodies taken as zero.
    __device__ __forceinline__ void spmv_to_X(const double* vec) const {
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            const double* P = contact(gc);
            const int2 sl = reinterpret_cast<const int2*>(B.islot)[gc];
            if (sl.x < 0 && sl.y < 0) continue;  // two static bodies
            double W[6];
            ld6(B.G + 12LL * max(sl.x, sl.y), W);  // both sides hold the contact's W
            d3 pv[2];
            for (int j = 0; j < 2; ++j) {
                const int gb = b0 + B.cbody[2 * gc + j];
                if (B.is_static[gb]) { pv[j] = d3{0, 0, 0}; continue; }
                double pn[6];
                ld6(vec + 6LL * gb, pn);
                pv[j] = point_vel(pn, arm(P, j));
            }
            put_x(gc, sym_mul(W, sub3(pv[1], pv[0])));
        }
    }
    // (M/cm + eps I) x + gather(X)  for one active body
    __device__ __forceinline__ void spmv_body(int gb, const double* x6, double eps, double* q6) const {
        double y[6], gth[6];
        mass_mul(gb, x6, y);
        gather(gb, gth);
        for (int r = 0; r < 6; ++r) q6[r] = y[r] + eps * x6[r] + gth[r];
    }
    // spmv_body of the direction pn = z + beta pp of body gb with each incident
    // contact's X = W (v1p - v0p) recomputed here (the other body's direction
    // from z + beta pp) instead of read from a contact phase: the same operations
    // as spmv_to_X + spmv_body, so the same bits, with no barrier between them.
    // One lane per body (block and warp teams): the same sums as the L = 1 case
    // of spmv_body_fused below, kept as its own loop for the block kernel's code.
    __device__ __forceinline__ void spmv_body_fused1(int gb, const double* pn, const double* pp, double beta,
                                                     double eps, double* q6) const {
        double y[6];
        mass_mul(gb, pn, y);
        const int st = B.inc_start[gb], n = B.inc_cnt[gb];
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0;
#pragma unroll 2
        for (int k = 0; k < n; ++k) {
            const int go = B.inc_o[st + k];
            double W[12];
            ldg12(st + k, W);
            const d3 arm = ld3(W + 6);
            const d3 pv_own = point_vel(pn, arm);
            d3 pv_oth = d3{0, 0, 0};
            if (go >= 0) {
                double po[6], zo[6];
                ld6(pp + 6LL * go, po);
                ld6(B.z + 6LL * go, zo);
                for (int r = 0; r < 6; ++r) po[r] = __dadd_rn(zo[r], __dmul_rn(beta, po[r]));
                pv_oth = point_vel(po, ld3(W + 9));
            }
            const d3 x = sym_mul(W, sub3(pv_own, pv_oth));  // sigma W (v1p - v0p)
            const d3 t = cross3(arm, x);
            a0 += x.x; a1 += x.y; a2 += x.z;
            a3 += t.x; a4 += t.y; a5 += t.z;
        }
        q6[0] = y[0] + eps * pn[0] + a0;
        q6[1] = y[1] + eps * pn[1] + a1;
        q6[2] = y[2] + eps * pn[2] + a2;
        q6[3] = y[3] + eps * pn[3] + a3;
        q6[4] = y[4] + eps * pn[4] + a4;
        q6[5] = y[5] + eps * pn[5] + a5;
    }
    // PCG product of every active body: p_new = z + beta pp into pc, q = A p_new,
    // and this thread's share of p_new . q.  L lanes per body split its
    // incidences; the loop runs in rounds so every lane of a warp takes the same
    // trips (the shuffles need the whole warp).
    template <int L>
    __device__ __forceinline__ void pcg_product(const double* pp, double* pc, double beta, double eps,
                                                double& pq) const {
        const int grp = tid / L, lg = tid - grp * L, ngrp = nt / L;
        for (int base = 0; base < n_local; base += ngrp) {
            const int i = base + grp;
            int gb = -1;
            if (i < n_local) {
                gb = B.lbody[b0 + i];
                if (!active(gb)) gb = -1;
            }
            double pn[6], q6[6];
            if (gb >= 0)
                for (int r = 0; r < 6; ++r) pn[r] = __dadd_rn(B.z[6 * gb + r], __dmul_rn(beta, pp[6 * gb + r]));
            spmv_body_fused<L>(gb, pn, pp, beta, eps, q6, lg);
            if (gb >= 0 && lg == 0) {
                for (int r = 0; r < 6; ++r) {
                    pc[6 * gb + r] = pn[r];
                    pq += pn[r] * q6[r];
                    B.q[6 * gb + r] = q6[r];
                }
            }
        }
    }
    // With L > 1, lane lg of the body's group takes incidences lg, lg + L, ...
    // and a butterfly of shuffles sums the groups' partials (each level adds the
    // same two values on both lanes, so every lane gets the same bits); gb < 0
    // (no body for this group) still takes part in the shuffles.
    template <int L>
    __device__ __forceinline__ void spmv_body_fused(int gb, const double* pn, const double* pp, double beta,
                                                    double eps, double* q6, int lg) const {
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0;
        const int st = (gb >= 0) ? B.inc_start[gb] : 0, n = (gb >= 0) ? B.inc_cnt[gb] : 0;
#pragma unroll 2
        for (int k = lg; k < n; k += L) {
            const int go = B.inc_o[st + k];
            double W[12];
            ldg12(st + k, W);
            const d3 arm = ld3(W + 6);
            const d3 pv_own = point_vel(pn, arm);
            d3 pv_oth = d3{0, 0, 0};
            if (go >= 0) {
                double po[6], zo[6];
                ld6(pp + 6LL * go, po);
                ld6(B.z + 6LL * go, zo);
                for (int r = 0; r < 6; ++r) po[r] = __dadd_rn(zo[r], __dmul_rn(beta, po[r]));
                pv_oth = point_vel(po, ld3(W + 9));
            }
            const d3 x = sym_mul(W, sub3(pv_own, pv_oth));  // sigma W (v1p - v0p)
            const d3 t = cross3(arm, x);
            a0 += x.x; a1 += x.y; a2 += x.z;
            a3 += t.x; a4 += t.y; a5 += t.z;
        }
        if constexpr (L > 1) {
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) {
                a0 += __shfl_xor_sync(0xffffffffu, a0, o, L);
                a1 += __shfl_xor_sync(0xffffffffu, a1, o, L);
                a2 += __shfl_xor_sync(0xffffffffu, a2, o, L);
                a3 += __shfl_xor_sync(0xffffffffu, a3, o, L);
                a4 += __shfl_xor_sync(0xffffffffu, a4, o, L);
                a5 += __shfl_xor_sync(0xffffffffu, a5, o, L);
            }
        }
        if (gb < 0) return;
        double y[6];
        mass_mul(gb, pn, y);
        q6[0] = y[0] + eps * pn[0] + a0;
        q6[1] = y[1] + eps * pn[1] + a1;
        q6[2] = y[2] + eps * pn[2] + a2;
        q6[3] = y[3] + eps * pn[3] + a3;
        q6[4] = y[4] + eps * pn[4] + a4;
        q6[5] = y[5] + eps * pn[5] + a5;
    }
    __device__ __forceinline__ void prec(int gb, const double* r6, double* z6) const {
        const double* Pi = B.pinv + 21 * gb;
        for (int a = 0; a < 6; ++a) {
            double s = 0;
            for (int c = 0; c < 6; ++c) s += Pi[pk(a, c)] * r6[c];
            z6[a] = s;
        }
    }

    // filterLineSearch (NonSmoothContactForce.cpp:281-319) applied to step*d at
    // force cf and multipliers l
    __device__ __forceinline__ void filter(const double* P, double step, double mu, d3 cf, const double* l, double* dfin,
                                           double* dlin) const {
        const d3 d = fld3(P, F_df);
        dfin[0] = step * d.x;
        dfin[1] = step * d.y;
        dfin[2] = step * d.z;
        double t0 = cf.x + dfin[0], t1 = cf.y + dfin[1], t2 = cf.z + dfin[2];
        if (t0 < 0) {
            t0 = 0;
            dfin[0] = t0 - cf.x;
            dfin[1] = t1 - cf.y;
            dfin[2] = t2 - cf.z;
        }
        if (cone_c(t0, t1, t2, mu) > 0) {
            // project(tf, tf) (LorentzCircleConstraint.cpp:36-49)
            const double rad = dmax(cone_radius(t0, mu) + 0, 0.0);
            const double s = rad / sqrt(__fma_rn(t2, t2, __dmul_rn(t1, t1)));
            dfin[0] = t0 - cf.x;
            dfin[1] = __dmul_rn(t1, s) - cf.y;
            dfin[2] = __dmul_rn(t2, s) - cf.z;
        }
        for (int k = 0; k < 2; ++k) {
            double e = step * P[32 * (F_dl + k)];
            if (e < 0 && l[k] + e < 0) e = -l[k];
            dlin[k] = e;
        }
    }

    // One contact of a line-search trial at `step` (filterLineSearch, the trial
    // point f + 0.99 df, lambda + 0.99 dl, and its residuals): trial values into
    // fo / lo, the world impulse into field xf of the incidence slots; adds |wrf|^2,
    // |rl|^2, |AC|^2 to q[1..3] and the directional terms to q[5], q[6].
    __device__ __forceinline__ void trial_contact(int gc, double step, double muc, int fo, int lo,
                                                  int xf, double* q) const {
        double* const P = contact(gc);
        double dfin[3], dlin[2], lI[2];
        const double l[2] = {P[32 * F_lam], P[32 * (F_lam + 1)]};
        const d3 cf = fld3(P, F_f);
        const double mu = cmu(gc);
        filter(P, step, mu, cf, l, dfin, dlin);
        for (int k = 0; k < 2; ++k) lI[k] = __dadd_rn(l[k], __dmul_rn(0.99, dlin[k]));
        const d3 fI = d3{__dadd_rn(cf.x, __dmul_rn(0.99, dfin[0])), __dadd_rn(cf.y, __dmul_rn(0.99, dfin[1])),
                         __dadd_rn(cf.z, __dmul_rn(0.99, dfin[2]))};
        fst3(P, fo, fI);
        for (int k = 0; k < 2; ++k) P[32 * (lo + k)] = lI[k];
        // residual at the trial point u + 0.99 step du: J is linear, so its
        // relative velocity is J u + 0.99 step J du (both stored per contact)
        const double a = __dmul_rn(0.99, step);
        const d3 wu = fld3(P, F_wu), wd = fld3(P, F_wd);
        const d3 w = d3{fma(a, wd.x, wu.x), fma(a, wd.y, wu.y), fma(a, wd.z, wu.z)};
        d3 rf;
        double rlv[2];
        contact_residual_w(gc, P, w, fI, lI, mu, muc, rf, rlv, q[1], q[2], q[3], xf);
        q[5] += dfin[0] * rf.x + dfin[1] * rf.y + dfin[2] * rf.z;
        q[6] += (dlin[0] / lI[0]) * rlv[0];
        if (!C.only_normal) q[6] += (dlin[1] / lI[1]) * rlv[1];
    }
    // One active body of a line-search trial: |ru|^2 at u + 0.99 step du into
    // q[0], du . ru into q[4]
    __device__ __forceinline__ void trial_body(int gb, double step, int xf, double* q) const {
        double ui[6], d[6], v[6], r2 = 0;
        trial_u(gb, step, ui, d);
        body_residual(gb, ui, xf, v);
        for (int r = 0; r < 6; ++r) r2 += v[r] * v[r];
        q[0] += r2;
        for (int r = 0; r < 6; ++r) q[4] += (step * d[r]) * v[r];
    }
    // Acceptance of trial t (lineSearch :606-630): 1 = accept, 2 = stop without
    // a step (the last trial failed), 0 = halve the step and go on.
    __device__ __forceinline__ static int ls_verdict(const double* e, double sErr, double sacErr, int t, int maxLS) {
        const double inErr = e[0] + e[1] + e[2];
        const double sacIn = e[0] + e[3] + e[2];
        const double gErr = -e[4] + e[5] + e[6];
        const bool acpt = (inErr < sErr) | (sacIn < sacErr);
        if ((acpt && gErr > 0) || (t == maxLS - 1)) return acpt ? 1 : 2;
        return 0;
    }
    // Commit of an accepted trial at `step` with trial values fo / lo
    __device__ __forceinline__ void ls_commit(double step, int fo, int lo) {
        for (int i = tid; i < n_local; i += nt) {
            const int gb = B.lbody[b0 + i];
            double ui[6], d[6];
            trial_u(gb, step, ui, d);
            st6(B.u + 6LL * gb, ui);
        }
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            double* const P = contact(gc);
            for (int k = 0; k < 3; ++k) P[32 * (F_f + k)] = P[32 * (fo + k)];
            for (int k = 0; k < 2; ++k) P[32 * (F_lam + k)] = P[32 * (lo + k)];
        }
        T.sync();
    }

    // lineSearch (PrimalDualForceSolver.cpp:562-635).  Commits the accepted
    // trial into (u, f, lam) and returns the step (0 = nothing accepted).
    // Thread-block teams with at most half a block of contacts and of local
    // bodies evaluate trials in pairs (step and step / 2, one on each half of
    // the block, the second with its own trial buffers): a contact or body sits
    // at the same lane of the same warp position within its half as in a
    // single trial, so every sum of the pair has the bits of the single
    // trial's, and the trials and their verdicts are the sequential ones.
    __device__ double line_search(double sErr, double sacErr, double muc, int maxLS, int& trials) {
        double step = 1.0;
        trials = 0;
        const int half = nt >> 1;
        if constexpr (Team::kind == 0) {
          if (nc <= half && n_local <= half) {
            const int j = tid >= half ? 1 : 0, k = tid - j * half;
            const int fo = j ? F_fT2 : F_fT, lo = j ? F_lT2 : F_lT, xo = j ? I_X2 : I_X;
            for (int t = 0; t < maxLS; t += 2) {
                const double sj = j ? step * 0.5 : step;
                double q[7] = {0, 0, 0, 0, 0, 0, 0};
                if (k < nc) trial_contact(c0 + k, sj, muc, fo, lo, xo, q);
                T.sync();
                if (k < n_local) {
                    const int gb = B.lbody[b0 + k];
                    if (active(gb)) trial_body(gb, sj, xo, q);
                }
                double e[14];
#pragma unroll
                for (int r = 0; r < 7; ++r) {
                    e[r] = j ? 0.0 : q[r];
                    e[7 + r] = j ? q[r] : 0.0;
                }
                T.sum(e);
                ++trials;
                int v = ls_verdict(e, sErr, sacErr, t, maxLS);
                if (v == 1) { ls_commit(step, F_fT, F_lT); return step; }
                if (v == 2) break;
                if (t + 1 >= maxLS) break;
                ++trials;
                v = ls_verdict(e + 7, sErr, sacErr, t + 1, maxLS);
                if (v == 1) { ls_commit(step * 0.5, F_fT2, F_lT2); return step * 0.5; }
                if (v == 2) break;
                step *= 0.25;
            }
            return 0.0;
          }
        }
        for (int t = 0; t < maxLS; ++t) {
            ++trials;
            double e[7] = {0, 0, 0, 0, 0, 0, 0};  // ru2, wrf2, rl2, ac2, du.ru, df.rf, (dl/l).rl
            for (int c = tid; c < nc; c += nt) trial_contact(c0 + c, step, muc, F_fT, F_lT, I_X, e);
            T.sync();
            for (int i = tid; i < n_local; i += nt) {
                const int gb = B.lbody[b0 + i];
                if (active(gb)) trial_body(gb, step, I_X, e);
            }
            T.sum(e);
            const int v = ls_verdict(e, sErr, sacErr, t, maxLS);
            if (v == 1) { ls_commit(step, F_fT, F_lT); return step; }
            if (v == 2) break;
            step *= 0.5;
        }
        return 0.0;
    }
    __device__ __forceinline__ void trial_u(int gb, double step, double* ui, double* d) const {
        ld6(B.u + 6LL * gb, ui);
        ld6(B.du + 6LL * gb, d);
        for (int r = 0; r < 6; ++r) ui[r] = __dadd_rn(ui[r], __dmul_rn(0.99, __dmul_rn(step, d[r])));
    }
    // contact residual with fresh constraints, given the relative velocity w
    __device__ __forceinline__ void contact_residual_w(int gc, const double* P, d3 w, d3 fv, const double* lv, double mu, double muc,
                                                       d3& rfo, double* rlo, double& wrf2, double& rl2, double& ac2,
                                                       int xf) const {
        const Frame R = frame(P);
        if (C.only_normal) {
            rlo[1] = 0;
            normal_residual(gc, P, R, w, fv.x, lv[0], muc, rfo, rlo[0], wrf2, rl2, ac2, xf);
            return;
        }
        double g0, g1;
        cone_grad(fv.y, fv.z, g0, g1);
        const double rl0 = lv[0] * (-fv.x) + muc, rl1 = lv[1] * cone_c(fv.x, fv.y, fv.z, mu) + muc;
        rl2 += rl0 * rl0 + rl1 * rl1;
        rfo = cone_residual(gc, P, R, w, fv, lv[0], lv[1], g0, g1, mu, wrf2, ac2, xf);
        rlo[0] = rl0; rlo[1] = rl1;
    }

    // KKT report at the final iterate (mu_c = 0) and write-back (:491-510).
    __device__ void finish(pdc_stats& st) {
        double e[2] = {0, 0};
        double mx[2] = {0, 0};
        for (int c = tid; c < nc; c += nt) {
            const int gc = c0 + c;
            double* const P = contact(gc);
            const d3 w = rel_vel(gc, P, B.u), fv = fld3(P, F_f);
            const double l[2] = {P[32 * F_lam], P[32 * (F_lam + 1)]};
            const double mu = cmu(gc);
            d3 rf;
            double rlv[2], d1 = 0, d2 = 0, d3v = 0;
            contact_residual_w(gc, P, w, fv, l, mu, 0.0, rf, rlv, d1, d2, d3v, I_X);
            e[1] += dot3(rf, rf);
            mx[0] = dmax(mx[0], dmax(fabs(rlv[0]), fabs(rlv[1])));
            mx[1] = dmax(mx[1], C.only_normal ? -fv.x : dmax(-fv.x, cone_c(fv.x, fv.y, fv.z, mu)));
            B.lforce[3 * gc] = fv.x * cs * cm;
            B.lforce[3 * gc + 1] = fv.y * cs * cm;
            B.lforce[3 * gc + 2] = fv.z * cs * cm;
        }
        T.sync();
        for (int i = tid; i < n_local; i += nt) {
            const int gb = B.lbody[b0 + i];
            double ub[6], v[6];
            ld6(B.u + 6LL * gb, ub);
            if (!B.is_static[gb]) {
                body_residual(gb, ub, I_X, v);
                for (int r = 0; r < 6; ++r) e[0] += v[r] * v[r];
            }
            for (int r = 0; r < 3; ++r) {
                B.dvel[3 * gb + r] = ub[r] * cs - B.vel[3 * gb + r];
                B.dang[3 * gb + r] = ub[3 + r] * cs - B.ang[3 * gb + r];
            }
        }
        T.sum(e);
        T.max(mx);
        st.kkt_stationarity = dmax(sqrt(e[0]) / (6.0 * n_local), sqrt(e[1]) / ((C.only_normal ? 1.0 : 3.0) * nc));
        st.kkt_complementarity = mx[0];
        st.kkt_cone = mx[1];
        st.char_mass = cm;
        st.char_speed = cs;
        st.n_local_bodies = n_local;
        if constexpr (kLargeTeam) st.factor_blocks = dense_mode ? sparse_ws().cstart[n_active] : 0;
        else st.factor_blocks = dense_mode ? direct_ws().meta[1] - n_active : 0;
        st.team = Team::kind;
        st.status = status;
    }
};

// Scene queues: a single-block kernel buckets the scenes by contact count
// (largest first, for load balance) into a CTA queue (large scenes) and a warp
// queue (small scenes), and resets the two work counters.
// counts[0] = #CTA scenes, [1] = #warp scenes, [2] = CTA counter, [3] = warp counter.
__global__ void __launch_bounds__(1024) plan_scenes_kernel(const __grid_constant__ BatchPtrs B,
                                                           const __grid_constant__ EngineCfg C) {
    __shared__ int hist[2][64];
    __shared__ int start[2][64];
    const int ns = B.n_scenes;
    if (threadIdx.x < 128) (&hist[0][0])[threadIdx.x] = 0;
    __syncthreads();
    auto size_of = [&](int s, int& nb, int& nc) {
        if (B.body_off) {
            nb = B.body_cnt ? B.body_cnt[s] : B.body_off[s + 1] - B.body_off[s];
            nc = B.contact_cnt ? B.contact_cnt[s] : B.contact_off[s + 1] - B.contact_off[s];
        } else {
            nb = B.single_nb;
            nc = B.single_nc;
        }
    };
    auto queue_of = [&](int nb, int nc) {
        if (B.grid_large && C.grid_min_bodies > 0 && nb >= C.grid_min_bodies) return 2;  // host launches it
        return (nc <= C.warp_max_contacts && nb <= C.warp_max_bodies) ? 1 : 0;
    };
    // longest first: the scene's previous solve time when known, else its
    // contact count (the scenes of a stepped simulation change slowly); buckets
    // of half an octave of the key, largest bucket first
    auto key_of = [&](int s, int nc) {
        const unsigned int c = B.cost ? B.cost[s] : 0u;
        return (int)min(c ? c : (unsigned int)nc * 2048u, 0x7fffffffu);
    };
    auto bucket_of = [&](int key) {
        const unsigned int k = (unsigned int)key + 1u;
        const int p = 31 - __clz(k);                          // floor(log2 k), 0..31
        const int half = (p > 0) ? (int)((k >> (p - 1)) & 1u) : 0;
        return 63 - (2 * p + half);
    };
    for (int s = threadIdx.x; s < ns; s += blockDim.x) {
        int nb, nc;
        size_of(s, nb, nc);
        const int q = queue_of(nb, nc);
        if (q < 2) atomicAdd(&hist[q][bucket_of(key_of(s, nc))], 1);
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        const int q = threadIdx.x;
        int acc = 0;
        for (int b = 0; b < 64; ++b) {
            start[q][b] = acc;
            acc += hist[q][b];
        }
        B.counts[q] = acc;
        B.counts[2 + q] = 0;
    }
    __syncthreads();
    for (int s = threadIdx.x; s < ns; s += blockDim.x) {
        int nb, nc;
        size_of(s, nb, nc);
        const int q = queue_of(nb, nc);
        if (q == 2) continue;  // large scene: solved by solve_scene_grid_kernel
        const int pos = atomicAdd(&start[q][bucket_of(key_of(s, nc))], 1);
        (q ? B.order_warp : B.order_cta)[pos] = s;
    }
}

template <class Team>
__device__ __forceinline__ void run_scene(const BatchPtrs& B, const EngineCfg& C, Team& T, int s) {
    SceneSolver<Team> S(B, C, T, s);
    pdc_stats st;
    st.status = 0;
    st.newton_iters = 0;
    st.pcg_iters = 0;
    st.ls_trials = 0;
    st.gd_fallbacks = 0;
    st.n_local_bodies = 0;
    st.factor_blocks = 0;
    st.team = Team::kind;
    st.n_contacts = S.nc;
    st.precision_fallbacks = 0;
    st.exit_err = 0;
    st.kkt_stationarity = 0;
    st.kkt_complementarity = 0;
    st.kkt_cone = 0;
    st.char_mass = 0;
    st.char_speed = 0;
    const unsigned long long t0 = S.now();
    if (S.setup()) {
        S.newton(st);
        S.finish(st);
    } else {
        st.status = S.status;
    }
    if (T.rank == 0 && B.cost) {
        const unsigned long long dtn = S.now() - t0;
        B.cost[s] = (unsigned int)(dtn < 0xffffffffull ? (dtn ? dtn : 1ull) : 0xffffffffull);
    }
    if (T.rank == 0) {
        if (B.stats) B.stats[s] = st;
        if (B.timers) {
            atomicAdd(&B.timers[0], S.now() - t0);
            atomicAdd(&B.timers[1], S.t_build);
            atomicAdd(&B.timers[2], S.t_solve);
            atomicAdd(&B.timers[3], S.t_ls);
        }
    }
    T.sync();
}

// Persistent solve: every CTA first drains the CTA queue (one scene per CTA),
// then each of its warps drains the warp queue (one scene per warp).
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) solve_scenes_kernel(const __grid_constant__ BatchPtrs B,
                                                           const __grid_constant__ EngineCfg C) {
    __shared__ double s_red[2 * 16 * 32];
    __shared__ int s_int[33];
    __shared__ int s_q;
    {
        CtaTeam T(s_red, s_int);
        const int n_cta = B.counts[0];
        for (;;) {
            if (threadIdx.x == 0) s_q = atomicAdd(&B.counts[2], 1);
            __syncthreads();
            const int q = s_q;
            __syncthreads();
            if (q >= n_cta) break;
            run_scene(B, C, T, B.order_cta[q]);
        }
    }
    const int warps = blockDim.x >> 5;
    WarpTeam W(gridDim.x + blockIdx.x * warps + (threadIdx.x >> 5));
    const int n_warp = B.counts[1];
    for (;;) {
        int q = 0;
        if (W.rank == 0) q = atomicAdd(&B.counts[3], 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= n_warp) break;
        run_scene(B, C, W, B.order_warp[q]);
    }
}

// Team of a large scene, decided on the device from its current contact count
// (the world's counts are only known there): a cluster team up to
// C.cluster_max_contacts contacts and C.cluster_max_bodies bodies, else the
// whole GPU.
__device__ __forceinline__ bool large_on_cluster(const BatchPtrs& B, const EngineCfg& C, int s) {
    int nb, nc;
    if (B.body_off) {
        nb = B.body_cnt ? B.body_cnt[s] : B.body_off[s + 1] - B.body_off[s];
        nc = B.contact_cnt ? B.contact_cnt[s] : B.contact_off[s + 1] - B.contact_off[s];
    } else {
        nb = B.single_nb;
        nc = B.single_nc;
    }
    return nc <= C.cluster_max_contacts && nb <= C.cluster_max_bodies;
}

// One large scene solved by the whole GPU (cooperative launch, grid team).
template <int THREADS>
__global__ void __launch_bounds__(THREADS) solve_scene_grid_kernel(const __grid_constant__ BatchPtrs B,
                                                                   const __grid_constant__ EngineCfg C, int scene,
                                                                   GridSync G) {
    if (large_on_cluster(B, C, scene)) return;  // same decision in every block
    __shared__ double s_red[8 * 32];
    __shared__ int s_int[33];
    GridTeam T(G, s_red, s_int);
    run_scene(B, C, T, scene);
}

// One large scene of moderate contact count solved by one thread-block cluster.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) solve_scene_cluster_kernel(const __grid_constant__ BatchPtrs B,
                                                                      const __grid_constant__ EngineCfg C,
                                                                      int scene) {
    if (!large_on_cluster(B, C, scene)) return;  // same decision in every block
    __shared__ double s_red[8 * 32];
    __shared__ double s_part[2 * 8];
    __shared__ int s_int[33];
    __shared__ int s_ipart[1];
    ClusterTeam T(s_red, s_part, s_int, s_ipart);
    run_scene(B, C, T, scene);
}

}  // namespace pdc
