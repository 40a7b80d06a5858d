// gx_adjoint.cu -- reverse-mode derivatives of short NVE horizons.
//
// The reference has no derivatives.  This file differentiates its tick
// (src/universe/mod.rs:356-369: kick, drift, wrap, forces, kick) with respect
// to the per-element LJ parameters sigma[10] and epsilon_k[10], for two
// smoothed observables: the potential energy after each tick and a
// Gaussian-kernel pair distribution averaged over sampled ticks.
//
// Forward.  The trajectory is recomputed in slot order (atoms never move
// between arrays) in FP64 with the reference's per-pair arithmetic
// (pair_f64_e24).  On a handle of mixed precision the forward is the mixed method
// instead: the FP32 pair law of the list passes (pair_f32) on the FP64
// minimum-image displacement rounded to FP32, the per-atom force summed in
// 2^-32 fixed point, and FP64 positions, velocities and observables; the
// backward below stays FP64, linearised on that trajectory.  A checkpoint of
// (x, v, a) is kept every K ticks.
//
// Backward.  Per segment: restore the checkpoint, recompute the segment's
// positions, then walk the ticks backwards.  With adjoints (Lx, Lv, La) of
// the state after tick t, tick t's adjoint is
//     Lx += dO_t/dx                           (observables at tick t)
//     W   = La + (dt/2) Lv                    (cotangent of a_t)
//     Lx += (da/dx)^T W,  Ltheta += (da/dtheta)^T W
//     Lv += dt Lx,  La = (dt/2) Lv            (drift and first kick)
// and (da/dx)^T W is the pairwise Hessian-vector product: with
// a_i = sum_j f(d_ij) n_ij / m_i, u = W_i/m_i - W_j/m_j and rho = n.u, the
// pair adds  f'(d) rho n + (f/d) (u - rho n)  to Lx_i (and the opposite to
// Lx_j).  Parameter partials are accumulated per atom (the own end of each
// visit takes half of the pair's derivative) and reduced per element once at
// the end.
//
// Launches.  A horizon is hundreds of ticks of a few thousand atoms, each a
// few microseconds of work: one cooperative launch runs the ticks of a chunk
// (k_adj_ticks), one the reverse sweep of a segment (k_adj_reverse), with one
// grid barrier per tick.  Eight lanes own one atom: partner j belongs to lane
// lane_of(j), and a lane visits its partners in ascending slot order, so each
// sum's order depends on the pairs in range alone, not on when the list was
// built: recomputed ticks reproduce the forward pass for any checkpoint
// spacing.  The lists hold the pairs within rc + skin and are rebuilt, inside
// the launch, on the ticks on which an atom may have moved skin/2 since.
// Where lists do not pay or do not fit, every tick sorts the atoms and walks
// their cells: the order then follows from the tick's positions.
// What bounds a tick is latency: 13 warps per SM walk lists of ten to twenty
// partners, each a chain of dependent FP64 operations.  8,000 atoms, 200
// ticks, mixed forward, both losses: 36.2 ms, where a sort, a staging and a
// pair pass over 27 cells per tick, one kernel each, took 143 ms; per tick,
// rebuilds included, 22 us for the recomputed ticks, 43 with the observables,
// 28 / 68 for the reverse sweep without / with g(r).  Lists of rc + 0.2 rc, as
// they were built: 31.4 ms where 0.1 takes 33.8, 0.15 32.3 and 0.25 33.5;
// sixteen lanes per atom 36.3 where eight take 34.7.
//
// The cutoffs are multiples of max sigma; their derivative goes to the
// lowest-index element attaining the max.  The hard-core clamp
// r = max(d, sigma/2) and the Coulomb/gravity clamp r = max(d, 0.5) are
// differentiated on the side the value takes; the periodic wrap and the
// minimum image have derivative one.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gx_gridsync.cuh"
#include "gx_law64.cuh"
#include "gx_pair_f32.cuh"

namespace gx {
namespace {

constexpr int kAdjThreads = 256;
constexpr int kAdjLanes = 8;              // lanes per atom
constexpr double kAdjSkin = 0.2;          // list skin in units of the cutoff
constexpr int kAdjTicksPerLaunch = 256;
constexpr int kAdjMaxBins = 512;
constexpr double kRonFrac = 0.9;  // r_on = 0.9 rc for every switched term (forces.rs:237, systems/forces.rs:118-124)
constexpr double kHistScale = 4294967296.0;
constexpr double kHistInv = 1.0 / 4294967296.0;
constexpr int kNOut = 2 * kNElem + 3;  // per-element sigma, epsilon sums + three cutoff sums

inline unsigned nblk(size_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Component k of a 3-vector field stored as three rows of `cap` doubles.
struct Vec3Field {
    double* p;
    size_t cap;
    __device__ __forceinline__ double& c(int k, uint32_t i) const { return p[(size_t)k * cap + i]; }
};

struct GrSpec {
    int bins;
    double dr, width, reach, c2;  // bin width, kernel width, truncation radius, -1/(2 w^2)
};

// Switch S(r) of smooth_cutoff (forces.rs:302-318) with its first two
// r-derivatives and the derivatives of S and dS/dr with respect to rc
// (r_on = 0.9 rc moves with it).
struct SwD {
    double S, S1, S2, Src, S1rc;
};
__device__ __forceinline__ SwD switch_d(double r, double ron, double rc) {
    SwD o{0.0, 0.0, 0.0, 0.0, 0.0};
    if (r <= ron) {
        o.S = 1.0;
        return o;
    }
    if (r >= rc) return o;
    double iw = 1.0 / (rc - ron);
    double u = (r - ron) * iw, omu = 1.0 - u;
    double Su = -30.0 * u * u * omu * omu;
    double Suu = -60.0 * u * omu * (1.0 - 2.0 * u);
    o.S = 1.0 + u * u * u * (-10.0 + u * (15.0 - 6.0 * u));
    o.S1 = Su * iw;
    o.S2 = Suu * iw * iw;
    double urc = -(kRonFrac + (1.0 - kRonFrac) * u) * iw;
    o.Src = Su * urc;
    o.S1rc = Suu * urc * iw - Su * (1.0 - kRonFrac) * iw * iw;
    return o;
}

// One pair's force magnitude f (repulsive > 0) and energy U with the
// derivatives the adjoint needs.
struct PairG {
    double f, fd, Ud;         // f, df/dd, dU/dd
    double fs, Us, fe, Ue;    // d/dsigma_ab, d/deps_ab of the LJ term
    double frc[3], Urc[3];    // d/drc of the LJ, Coulomb and gravity terms
};

__device__ __forceinline__ void central_term(double q, double d, double inv_d, double ron, double rc, PairG& o,
                                             int slot) {
    bool clamped = d < 0.5;  // r = max(d, 0.5), systems/forces.rs:283,293
    double rd = clamped ? 0.0 : 1.0;
    double ir = clamped ? 2.0 : inv_d;
    double v = q * ir, m = v * ir;
    double mr = -2.0 * m * ir, vr = -m;
    SwD w = switch_d(d, ron, rc);  // the switch is evaluated at d, not r
    o.f += m * w.S - v * w.S1;
    o.fd += mr * rd * w.S + m * w.S1 - vr * rd * w.S1 - v * w.S2;
    o.Ud += vr * rd * w.S + v * w.S1;
    o.frc[slot] = m * w.Src - v * w.S1rc;
    o.Urc[slot] = v * w.Src;
}

// inv_d = 1 / d; is = 1 / sg (a table of the element pairs).
__device__ __forceinline__ PairG pair_grad(const LawF64& L, double d, double inv_d, double sg, double is, double ep,
                                           double qa, double qb, double ma, double mb) {
    PairG o;
    o.f = o.fd = o.Ud = o.fs = o.Us = o.fe = o.Ue = 0.0;
    for (int k = 0; k < 3; ++k) o.frc[k] = o.Urc[k] = 0.0;
    if (d < L.lj_rc) {
        // force_switched_scalar (forces.rs:270-275): r = max(d, sigma/2)
        double half = 0.5 * sg;
        bool clamped = d < half;
        double r = clamped ? half : d, rd = clamped ? 0.0 : 1.0, rs = clamped ? 0.5 : 0.0;
        double s = clamped ? 2.0 : sg * inv_d, s2 = s * s, s6 = s2 * s2 * s2, s12 = s6 * s6;
        double v1 = 4.0 * (s12 - s6);                            // V / eps
        double m1 = 24.0 * is * s * (2.0 * s12 - s6);            // -dV/dr / eps
        double m1r = 24.0 * is * is * (7.0 * s6 * s2 - 26.0 * s12 * s2);
        double m1s = 144.0 * is * is * (4.0 * s12 * s - s6 * s);
        double v1s = 24.0 * is * (2.0 * s12 - s6);
        SwD w = switch_d(r, L.lj_ron, L.lj_rc);
        double F1 = m1 * w.S - v1 * w.S1;
        double fr = ep * (m1r * w.S + 2.0 * m1 * w.S1 - v1 * w.S2);
        double Ur = ep * (-m1 * w.S + v1 * w.S1);
        o.f = ep * F1;
        o.fd = fr * rd;
        o.Ud = Ur * rd;
        o.fs = ep * (m1s * w.S - v1s * w.S1) + fr * rs;
        o.Us = ep * v1s * w.S + Ur * rs;
        o.fe = F1;
        o.Ue = v1 * w.S;
        o.frc[0] = ep * (m1 * w.Src - v1 * w.S1rc);
        o.Urc[0] = ep * v1 * w.Src;
    }
    if (L.coul && d < L.coul_rc) central_term(L.k_e * qa * qb, d, inv_d, L.coul_ron, L.coul_rc, o, 1);
    if (L.grav && d < L.grav_rc) central_term(-L.G * ma * mb, d, inv_d, L.grav_ron, L.grav_rc, o, 2);
    return o;
}

template <int BS>
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = (threadIdx.x < BS / 32) ? sh[threadIdx.x] : 0.0;
    if (wid == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;
}

// Sum over the kAdjLanes lanes of one atom (a butterfly: every lane ends
// with the same bits, and the association is fixed, so recomputed ticks
// reproduce the forward pass exactly).
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
    for (int o = kAdjLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, kAdjLanes);
    return v;
}
// Integer partials: any order gives the same sum.
__device__ __forceinline__ long long lane_sum_ll(long long v) {
#pragma unroll
    for (int o = kAdjLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, kAdjLanes);
    return v;
}

// ---------------------------------------------------------------------------
// Kernels (slot order unless noted).

// Handle state (cell-sorted) -> slot order.
__global__ void k_adj_import(StateBuf b, uint32_t n, Vec3Field x, Vec3Field v, Vec3Field a, uint8_t* elem,
                             double* charge, double* mass, double* inv_mass, uint8_t* kind) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    uint32_t s = b.slot[p];
    x.c(0, s) = b.x[p];
    x.c(1, s) = b.y[p];
    x.c(2, s) = b.z[p];
    v.c(0, s) = b.vx[p];
    v.c(1, s) = b.vy[p];
    v.c(2, s) = b.vz[p];
    a.c(0, s) = b.ax[p];
    a.c(1, s) = b.ay[p];
    a.c(2, s) = b.az[p];
    elem[s] = b.elem[p];
    charge[s] = b.charge[p];
    mass[s] = b.mass[p];
    inv_mass[s] = b.inv_mass[p];
    kind[s] = b.kind[p];
}

// The lane that visits partner j: a multiplicative hash, so that no pattern of
// slots puts a neighbourhood on one lane.  With j % 8 the longest lane of an
// atom of a lattice whose side is a multiple of 8 holds 21 of 65 partners, and
// of slots a multiple of 8 apart all of them; with this multiplier, searched
// for lattices of side 8 to 80 and strides up to 65, 12 on average and at most
// 16.  Gradients of 262,144 atoms (side 64) take 62 ms instead of 81, those of
// 8,000 (side 20, which j % 8 deals out well) 36.2 instead of 35.5.
static_assert(kAdjLanes == 8, "three bits of the hash");
__device__ __forceinline__ uint32_t lane_of(uint32_t j) { return (j * 3192787907u) >> 29; }
constexpr uint32_t kAdjFound = 512;  // partners of one atom that a rebuild sorts at a time
constexpr uint32_t kAdjQueue = 128;  // distances that a warp collects for the histogram

// A rebuild's words of one warp: the partners found by a pass, as (lane, slot)
// keys padded to whole vectors; by lane, how many they are, how many earlier
// passes wrote, and where in the pool the lane's entries beyond its row go.
struct __align__(16) AdjFound {
    uint32_t key[kAdjFound + 4];
    uint32_t count[kAdjLanes], have[kAdjLanes], pool[kAdjLanes];
};

struct AdjArgs {
    GridGeom lg;  // list grid: cells >= rc + skin (with `walk` >= rc)
    GridGeom fg;  // force grid: its axes of two cells repeat pairs
    int two;      // the force grid has such an axis
    int plain;    // at least three force cells per axis, positions wrapped
    double half_box[3], inv_box[3];
    uint32_t n;
    size_t cap;
    LawF64 L;
    LawF32 L32;
    const PairF* tabf;
    const double *psig, *peps, *epsk;  // pair tables, epsilon_k
    const uint8_t *elem, *kind;
    const double *charge, *mass, *inv_mass;
    double* S;            // x, v, a: nine rows of cap
    double* ck;           // checkpoints of S, or null
    double* slabs;        // positions of a tick: (x, y, z, packed) per atom, 4 cap doubles each
    int first, last;      // ticks of this launch
    int K;
    int keep;             // tick t's positions stay in slab t - first; else two slabs take turns
    int obs;              // record the observables
    uint32_t* list;       // entry k of lane e = i * kAdjLanes + l at [k * kAdjLanes * cap + e], ascending slots
    uint32_t* cnt;
    uint32_t cap_l;
    uint32_t *pool, *off; // entry k >= cap_l of lane e at pool[off[e] + k - cap_l]
    unsigned long long* pool_used;  // words of the pool that the last rebuild asked for
    unsigned long long pool_cap;
    int walk;             // no lists: a sort and a walk over the cells every tick
    double* ref;          // positions at the last rebuild, three rows
    double* sorted;       // a rebuild's cell-sorted (x, y, z, slot); with `walk` slots in the scatter's order
    uint32_t* order;      // with `walk`: slots by cell, ascending in each
    uint32_t *key, *count, *start, *fill;
    uint32_t tile_log2;   // cells of one of the scan's tiles
    GridSync* sync;
    uint32_t* err;
    uint32_t polls;       // of a barrier before it gives up
    double *vpart, *pot;  // block partials (two turns), V_t
    unsigned long long* ghist;  // two turns of bins
    double* hacc;
    GrSpec gs;
    int every;
    double half_dt, dt, rl2, lim2;
    int wrap;
    // reverse sweep
    double *Ladj, *P;     // adjoints of x, v, a (nine rows); parameter partials (five rows)
    double* W;            // two turns of (W/m, -) per atom, 4 cap doubles each
    const double *alpha, *bw;
    int gr;
};

__device__ __forceinline__ double4 load_slab(const double* X, uint32_t j) {
    const double2* p = reinterpret_cast<const double2*>(X) + 2 * (size_t)j;
    const double2 u = p[0], w = p[1];
    return make_double4(u.x, u.y, w.x, w.y);
}
// The packed word of a slab: element, kind << 8, force cell << 32 (with `two`).
__device__ __forceinline__ uint32_t packed_elem(double w) { return (uint32_t)__double_as_longlong(w) & 255u; }
__device__ __forceinline__ uint32_t packed_kind(double w) { return ((uint32_t)__double_as_longlong(w) >> 8) & 255u; }
__device__ __forceinline__ uint32_t packed_cell(double w) { return (uint32_t)((unsigned long long)__double_as_longlong(w) >> 32); }

// Whether an atom may have left its list: the squared displacement of
// component l (of lanes 0 .. 2 of its group) since the rebuild, summed over
// the group.  `odd`: half-box translations of the wrap since then (mod 2).
__device__ __forceinline__ double moved2(const AdjArgs& a, uint32_t i, uint32_t l, bool live, double x, bool odd) {
    double d = 0.0;
    if (live && l < 3) {
        const double L = a.L.box[l];
        d = x - a.ref[l * a.cap + i] - (odd ? 0.5 * L : 0.0);
        d -= L * rint(d * a.inv_box[l]);
        d *= d;
    }
    return lane_sum(d);
}

// A minimum image to rounding, for the lists' tests, which have the skin's
// room: no division and no branch.
__device__ __forceinline__ double list_image(const AdjArgs& a, double d, int k) {
    return d - a.L.box[k] * rint(d * a.inv_box[k]);
}

// Neighbour cell k < 27 of cell (cx, cy, cz), every distinct one once (both
// sides of an axis only from three cells on); false for a repeated one.
__device__ __forceinline__ bool adj_cell(const GridGeom& g, uint32_t cx, uint32_t cy, uint32_t cz, uint32_t k,
                                         uint32_t& B) {
    const int ox = (int)(k % 3u) - 1, oy = (int)((k / 3u) % 3u) - 1, oz = (int)(k / 9u) - 1;
    if (!((ox == 0 || g.n[0] >= 3 || (ox > 0 && g.n[0] == 2)) && (oy == 0 || g.n[1] >= 3 || (oy > 0 && g.n[1] == 2)) &&
          (oz == 0 || g.n[2] >= 3 || (oz > 0 && g.n[2] == 2))))
        return false;
    B = encode(g, wrap_add(cx, ox, g.n[0]), wrap_add(cy, oy, g.n[1]), wrap_add(cz, oz, g.n[2]));
    return true;
}

// One pass over the candidates of atom i (position pi) for its list: 32 at a
// time out of the run that the scan `end` of the cells' counts makes of them
// (`base`: first candidate less the counts before it).  The partners with
// slots in [from, to) are counted by lane, the first kAdjFound of them kept.
__device__ __forceinline__ uint32_t adj_collect(const AdjArgs& a, const double4& pi, uint32_t i, uint32_t end,
                                                uint32_t base, uint32_t total, uint32_t from, uint32_t to,
                                                AdjFound& found) {
    constexpr int kAhead = 4;  // candidates of a lane in flight
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    if (lane < kAdjLanes) found.count[lane] = 0u;
    __syncwarp();
    uint32_t m2 = 0;
    for (uint32_t t0 = 0; t0 < total; t0 += 32 * kAhead) {  // every load before the tests
        double4 pj[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t t = t0 + 32u * u + lane;
            uint32_t k = 0;  // the first cell whose scan exceeds t
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1)
                if (__shfl_sync(0xffffffffu, end, k + step - 1) <= t) k += step;
            const uint32_t q = __shfl_sync(0xffffffffu, base, k) + t;
            pj[u] = make_double4(0.0, 0.0, 0.0, __longlong_as_double((long long)i));
            if (t < total) pj[u] = load_slab(a.sorted, q);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t j = (uint32_t)__double_as_longlong(pj[u].w);
            const double dx = list_image(a, pi.x - pj[u].x, 0), dy = list_image(a, pi.y - pj[u].y, 1),
                         dz = list_image(a, pi.z - pj[u].z, 2);
            const bool hit = j != i && j - from < to - from && dx * dx + dy * dy + dz * dz < a.rl2;
            const uint32_t mask = __ballot_sync(0xffffffffu, hit);
            const uint32_t at = m2 + __popc(mask & ((1u << lane) - 1u));
            if (hit) {
                if (at < kAdjFound) found.key[at] = lane_of(j) << 28 | j;
                atomicAdd(&found.count[lane_of(j)], 1u);
            }
            m2 += __popc(mask);
        }
    }
    __syncwarp();
    return m2;
}

// The pass's m2 <= kAdjFound partners into their lanes' lists, after those of
// earlier passes: a partner's place is the number of its lane's partners with
// smaller slots.
__device__ __forceinline__ void adj_emit(const AdjArgs& a, uint32_t i, uint32_t m2, AdjFound& found) {
    const uint32_t lane = threadIdx.x & 31u;
    const size_t stride = (size_t)kAdjLanes * a.cap;
    if (lane < 4) found.key[m2 + lane] = 0xffffffffu;
    __syncwarp();
    for (uint32_t k = lane; k < m2; k += 32) {  // the keys below this one, those of lower lanes aside
        const uint32_t key = found.key[k], l = key >> 28;
        uint32_t place = found.have[l];
        for (uint32_t q = 0; q < m2; q += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(&found.key[q]);
            place += (v.x < key) + (v.y < key) + (v.z < key) + (v.w < key);
        }
        for (uint32_t q = 0; q < l; ++q) place -= found.count[q];
        if (place < a.cap_l) a.list[place * stride + i * kAdjLanes + l] = key & 0x0fffffffu;
        else a.pool[found.pool[l] + (place - a.cap_l)] = key & 0x0fffffffu;
    }
    __syncwarp();
}

// Lists of the pairs within rc + skin of the positions X, by lane; their
// reference positions.  With `walk` the cells' slots in ascending order
// instead.  False when the launch is over: a barrier gave up, or the lists
// need more room than the pool has (kErrCapacity; the host repeats the call).
__device__ bool adj_rebuild(const AdjArgs& a, const double* X, uint32_t& target, int* s_ok, uint32_t* s_warp,
                            uint32_t* s_off, AdjFound* s_found) {
    const uint32_t tid = threadIdx.x, gt = blockIdx.x * kAdjThreads + tid, gs = gridDim.x * kAdjThreads;
    const uint32_t n = a.n, m = a.lg.ncell + 1, log2 = a.tile_log2, per = (1u << log2) / kScanTileCells;
    const uint32_t ntiles = (m - 1) / (1u << log2) + 1;  // of 1 << log2 cells, `per` scans in a row
    for (uint32_t i = gt; i < n; i += gs) {
        const double4 p = load_slab(X, i);
        const uint32_t c = cell_of(a.lg, p.x, p.y, p.z);
        a.key[i] = c;
        atomicAdd(&a.count[c], 1u);
    }
    if (!grid_barrier(a.sync, a.err, a.polls, target, s_ok)) return false;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        uint32_t total = 0;
        for (uint32_t u = 0; u < per; ++u) total = scan_tile<kAdjThreads>(a.count, t * per + u, m, total, s_warp);
        if (tid == 0) a.sync->tile[t] = total;
    }
    if (gt == 0 && !a.walk) *a.pool_used = 0ull;  // last read before this rebuild began
    if (!grid_barrier(a.sync, a.err, a.polls, target, s_ok)) return false;
    if (tid < ntiles) {
        uint32_t run = 0;
        for (uint32_t t = 0; t < tid; ++t) run += a.sync->tile[t];
        s_off[tid] = run;
    }
    __syncthreads();
    for (uint32_t c = gt; c < m; c += gs) a.start[c] = a.count[c] + s_off[c >> log2];
    for (uint32_t i = gt; i < n; i += gs) {
        const uint32_t c = a.key[i];
        const uint32_t at = a.count[c] + s_off[c >> log2] + atomicAdd(&a.fill[c], 1u);
        if (a.walk) {
            reinterpret_cast<uint32_t*>(a.sorted)[at] = i;
            continue;
        }
        const double4 p = load_slab(X, i);
        double2* to = reinterpret_cast<double2*>(a.sorted) + 2 * (size_t)at;
        to[0] = make_double2(p.x, p.y);
        to[1] = make_double2(p.z, __longlong_as_double((long long)i));
    }
    if (!grid_barrier(a.sync, a.err, a.polls, target, s_ok)) return false;
    for (uint32_t c = gt; c < m; c += gs) a.count[c] = a.fill[c] = 0u;  // for the next rebuild
    if (a.walk) {
        const uint32_t* tmp = reinterpret_cast<const uint32_t*>(a.sorted);
        for (uint32_t i = gt; i < n; i += gs) {
            const uint32_t lo = a.start[a.key[i]], hi = a.start[a.key[i] + 1];
            uint32_t p = lo;
            for (uint32_t q = lo; q < hi; ++q) p += tmp[q] < i ? 1u : 0u;
            a.order[p] = i;
        }
        return grid_barrier(a.sync, a.err, a.polls, target, s_ok);
    }
    // A warp per atom: lane k < 27 looks up neighbour cell k, and a scan of the
    // counts turns the candidates into one run.  Atoms of more partners than a
    // pass can sort take them by ranges of slots.
    const uint32_t lane = tid & 31u;
    AdjFound& found = s_found[tid / 32];
    for (uint32_t i = gt / 32u; i < n; i += gs / 32u) {
        const double4 pi = load_slab(X, i);
        if (lane < 3) a.ref[lane * a.cap + i] = lane == 0 ? pi.x : (lane == 1 ? pi.y : pi.z);
        uint32_t lo = 0, len = 0;
        if (lane < 27) {
            uint32_t cx, cy, cz, B;
            decode(a.lg, a.key[i], cx, cy, cz);
            if (adj_cell(a.lg, cx, cy, cz, lane, B)) {
                lo = a.start[B];
                len = a.start[B + 1] - lo;
            }
        }
        uint32_t end = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= (uint32_t)o) end += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31), base = lo - (end - len);
        uint32_t m2 = adj_collect(a, pi, i, end, base, total, 0u, n, found);
        const uint32_t mine = lane < kAdjLanes ? found.count[lane] : 0u;
        const uint32_t beyond = mine > a.cap_l ? mine - a.cap_l : 0u;
        if (lane < kAdjLanes) {
            a.cnt[i * kAdjLanes + lane] = mine;
            found.have[lane] = 0u;
        }
        bool room = true;
        if (__any_sync(0xffffffffu, beyond != 0u)) {
            uint32_t run = beyond;  // inclusive scan of the lanes' needs
#pragma unroll
            for (int o = 1; o < kAdjLanes; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= (uint32_t)o) run += v;
            }
            const uint32_t need = __shfl_sync(0xffffffffu, run, kAdjLanes - 1);
            unsigned long long at = lane == 0 ? atomicAdd(a.pool_used, (unsigned long long)need) : 0ull;
            at = __shfl_sync(0xffffffffu, at, 0);
            room = at + need <= a.pool_cap;
            if (room && lane < kAdjLanes) a.off[i * kAdjLanes + lane] = found.pool[lane] = (uint32_t)at + run - beyond;
        }
        if (!room) continue;  // the lists will not be read
        if (m2 <= kAdjFound) {
            adj_emit(a, i, m2, found);
            continue;
        }
        uint32_t width = n / (2 * m2 / kAdjFound + 1) + 1;
        for (uint32_t from = 0; from < n;) {
            const uint32_t to = min(from + width, n);
            m2 = adj_collect(a, pi, i, end, base, total, from, to, found);
            if (m2 > kAdjFound) {  // kAdjFound slots and fewer always fit
                width = (width + 1) / 2;
                continue;
            }
            adj_emit(a, i, m2, found);
            if (lane < kAdjLanes) found.have[lane] += found.count[lane];
            from = to;
            if (m2 < kAdjFound / 4) width = min(2 * width, n);
        }
    }
    if (!grid_barrier(a.sync, a.err, a.polls, target, s_ok)) return false;  // the lists are read by other threads
    if (*(volatile unsigned long long*)a.pool_used <= a.pool_cap) return true;
    if (gt == 0) atomicOr(a.err, kErrCapacity);
    grid_leave(a.sync);
    return false;
}

// Every partner of lane l of atom i, in an order that depends on the pairs in
// range alone: its list's ascending slots, with the slab entry loaded one
// partner ahead, or this tick's cells.
template <class V>
__device__ __forceinline__ void adj_partners(const AdjArgs& a, const double* X, uint32_t i, uint32_t l, V&& visit) {
    if (!a.walk) {
        const uint32_t e = i * kAdjLanes + l, m = a.cnt[e];
        if (m == 0) return;
        const size_t stride = (size_t)kAdjLanes * a.cap;
        const uint32_t* row = a.list + e;
        const uint32_t in_row = min(m, a.cap_l);
        uint32_t j = row[0], j1 = m > 1 ? row[stride] : j;
        double4 p = load_slab(X, j);
        for (uint32_t k = 0; k < m; ++k) {
            const double4 p1 = load_slab(X, j1);
            uint32_t j2 = j1;
            if (k + 2 < in_row) j2 = row[(k + 2) * stride];
            else if (k + 2 < m) j2 = a.pool[a.off[e] + (k + 2 - a.cap_l)];
            visit(j, p);
            j = j1;
            p = p1;
            j1 = j2;
        }
    } else {
        uint32_t cx, cy, cz, B;
        decode(a.lg, a.key[i], cx, cy, cz);
        for (uint32_t k = 0; k < 27; ++k) {
            if (!adj_cell(a.lg, cx, cy, cz, k, B)) continue;
            for (uint32_t q = a.start[B] + l, hi = a.start[B + 1]; q < hi; q += kAdjLanes) {
                const uint32_t j = a.order[q];
                if (j != i) visit(j, load_slab(X, j));
            }
        }
    }
}

// The minimum image of a difference of two positions: where both are wrapped
// and every pair within the cutoff is seen once, without the division.
__device__ __forceinline__ double adj_image(const AdjArgs& a, double d, int k) {
    return a.plain ? min_image_near(d, a.L.box[k], a.half_box[k]) : near_image(d, a.L.box[k]);
}

// The bins within the kernel's reach of distance d: f(bin, z, G) with
// z = d - centre and G = exp(c2 z^2).  An exponential per bin: a recurrence
// over the bins loses all of them where the one it starts from underflows
// (supports of some 38 widths), and its rounding grows with the square of
// their number (8,000 atoms, 200 ticks, both losses: 29.5 ms so, 34.6 with the
// exponentials).
template <class F>
__device__ __forceinline__ void gr_bins(const GrSpec& gs, double d, F&& f) {
    int k0 = (int)ceil((d - gs.reach) / gs.dr - 0.5), k1 = (int)floor((d + gs.reach) / gs.dr - 0.5);
    k0 = k0 < 0 ? 0 : k0;
    k1 = k1 > gs.bins - 1 ? gs.bins - 1 : k1;
    double at = k0 + 0.5;
    for (int b = k0; b <= k1; ++b, at += 1.0) {
        const double z = d - at * gs.dr;
        if (fabs(z) < gs.reach) f(b, z, exp(z * z * gs.c2));
    }
}

// Ticks first .. last.  With `obs` V_t and the smoothed histogram; with
// `keep` the last tick stops after the drift (the reverse sweep needs its
// positions only).  F32: the mixed method's pair law with the force summed
// in 2^-32 fixed point and a = F 2^-32 / m as the list path's finish takes
// it; the potential sums the FP32 pair energies in FP64.
template <bool F32>
__global__ void __launch_bounds__(kAdjThreads, 2) k_adj_ticks(const __grid_constant__ AdjArgs a) {
    // with obs a histogram per warp: low 16 bits' sums, then the rest's; with `walk`, whose terms nobody counted, 64-bit sums
    extern __shared__ __align__(16) uint32_t s_hist[];
    __shared__ double s_sig[kNElem * kNElem], s_eps[kNElem * kNElem], s_e24[kNElem * kNElem];
    __shared__ PairTab s_tab;
    __shared__ double sh[kAdjThreads / 32], s_queue[kAdjThreads / 32][kAdjQueue];
    __shared__ uint32_t s_queued[kAdjThreads / 32];
    __shared__ uint32_t s_warp[kAdjThreads / 32], s_off[kScanMaxTiles];
    __shared__ AdjFound s_found[kAdjThreads / 32];
    __shared__ int s_ok;
    const uint32_t tid = threadIdx.x, n = a.n, lanes = n * kAdjLanes;
    const uint32_t gt = blockIdx.x * kAdjThreads + tid, gs = gridDim.x * kAdjThreads;
    const uint32_t pad = (lanes + 31u) & ~31u;  // whole warps
    const size_t cap = a.cap;
    const int bins = a.obs ? a.gs.bins : 0;
    const double h3[3] = {xmul(0.5, a.L.box[0]), xmul(0.5, a.L.box[1]), xmul(0.5, a.L.box[2])};
    const bool recorder = blockIdx.x == gridDim.x - 1;
    uint32_t target = 0;
    if (*a.err & (kErrCapacity | kErrBarrier)) return;  // an earlier launch of the call ended early
    for (int k = tid; k < kNElem * kNElem; k += kAdjThreads) {
        s_sig[k] = a.psig[k];
        s_eps[k] = a.peps[k];
        s_e24[k] = xdiv(xmul(24.0, a.peps[k]), a.psig[k]);
    }
    if (F32)
        for (int k = tid; k < a.L32.nkinds * a.L32.nkinds; k += kAdjThreads) s_tab.put(k, a.tabf[k]);
    for (int k = tid; k < (kAdjThreads / 32) * 2 * bins; k += kAdjThreads) s_hist[k] = 0u;
    uint32_t* wh = s_hist + (tid / 32) * 2 * bins;
    uint32_t held = 0;  // terms that a bin of this warp's histogram may hold
    if (tid < kAdjThreads / 32) s_queued[tid] = 0u;
    auto into_warp = [&](int b, unsigned long long v) {
        if (a.walk) {
            atomicAdd(reinterpret_cast<unsigned long long*>(wh) + b, v);
            return;
        }
        atomicAdd(&wh[b], (uint32_t)v & 0xffffu);
        atomicAdd(&wh[bins + b], (uint32_t)(v >> 16));
    };
    for (uint32_t c = gt; c < a.lg.ncell + 1; c += gs) a.count[c] = a.fill[c] = 0u;
    // V_t and the histogram of a finished tick, by one block
    auto record = [&](int t) {
        const int turn = t & 1;
        double s = 0.0;
        for (uint32_t k = tid; k < gridDim.x; k += kAdjThreads) s = xadd(s, a.vpart[turn * gridDim.x + k]);
        s = block_sum<kAdjThreads>(s, sh);
        if (tid == 0) a.pot[t - 1] = s;
        if (bins && t % a.every == 0)
            for (int k = tid; k < bins; k += kAdjThreads) {
                unsigned long long* g = a.ghist + turn * bins + k;
                a.hacc[k] += (double)*g * kHistInv;
                *g = 0ull;
            }
    };
    int built = 0;  // the tick of the last rebuild
    for (int t = a.first; t <= a.last; ++t) {
        const int turn = t & 1, ask = t % 3;
        double* X = a.slabs + (size_t)(a.keep ? t - a.first : turn) * 4 * cap;
        const bool odd = a.wrap && ((t - built) & 1);
        const bool ckpt = a.ck && (t - 1) % a.K == 0;
        bool over = false;
        for (uint32_t e = gt; e < pad; e += gs) {  // kick, drift, wrap (integrate.rs:39-43, 62-66; boundary.rs:28-34)
            const uint32_t i = e / kAdjLanes, l = e % kAdjLanes;
            const bool live = i < n;
            double x = 0.0;
            if (live && l < 3) {
                double *sx = a.S + l * cap + i, *sv = sx + 3 * cap, *sa = sx + 6 * cap;
                x = *sx;
                double v = *sv;
                const double acc = *sa;
                if (ckpt) {
                    double* c = a.ck + (size_t)((t - 1) / a.K) * 9 * cap + l * cap + i;
                    c[0] = x;
                    c[3 * cap] = v;
                    c[6 * cap] = acc;
                }
                const double hb = l == 0 ? h3[0] : (l == 1 ? h3[1] : h3[2]);
                v = xadd(v, xmul(acc, a.half_dt));
                x = xadd(x, xmul(v, a.dt));
                if (a.wrap) x = xsub(rem_euclid(x, xmul(2.0, hb)), hb);
                *sv = v;
                *sx = x;
                X[4 * (size_t)i + l] = x;
                if (!isfinite(x)) atomicOr(a.err, kErrNonFinite);
            }
            uint32_t cell = 0;
            if (a.two) {
                const double px = __shfl_sync(0xffffffffu, x, 0, kAdjLanes), py = __shfl_sync(0xffffffffu, x, 1, kAdjLanes),
                             pz = __shfl_sync(0xffffffffu, x, 2, kAdjLanes);
                cell = cell_of(a.fg, px, py, pz);
            }
            if (live && l == 3)
                X[4 * (size_t)i + 3] = __longlong_as_double(
                    (long long)((unsigned long long)cell << 32 | (uint32_t)a.kind[i] << 8 | a.elem[i]));
            if (built && !a.walk) over |= !(moved2(a, i, l, live, x, odd) <= a.lim2);
        }
        if (t == a.last && a.keep) break;
        if (__syncthreads_or(over) && tid == 0) a.sync->request[ask] = 1u;
        if (!grid_barrier(a.sync, a.err, a.polls, target, &s_ok)) return;
        const bool rebuild = !built || a.walk || *(volatile uint32_t*)&a.sync->request[ask] != 0u;
        if (recorder) {
            if (a.obs && t > a.first) record(t - 1);
            if (tid == 0) a.sync->request[(ask + 2) % 3] = 0u;  // every block has read it before this barrier
        }
        if (rebuild) {
            if (!adj_rebuild(a, X, target, &s_ok, s_warp, s_off, s_found)) return;
            built = t;
        }
        const bool gr = bins > 0 && t % a.every == 0;
        double V = 0.0;
        auto flush = [&](uint32_t* hist, int warps, int from, int by) {  // adds histograms to the tick's and clears them
            for (int k = from; k < bins; k += by) {
                unsigned long long s = 0ull;
                for (int w = 0; w < warps; ++w) {
                    uint32_t* hw = hist + w * 2 * bins + k;
                    if (a.walk) {
                        unsigned long long* h64 = reinterpret_cast<unsigned long long*>(hist + w * 2 * bins) + k;
                        s += *h64;
                        *h64 = 0ull;
                        continue;
                    }
                    s += hw[0] + ((unsigned long long)hw[bins] << 16);
                    hw[0] = hw[bins] = 0u;
                }
                if (s) atomicAdd(&a.ghist[turn * bins + k], s);
            }
        };
        for (uint32_t e = gt; e < pad; e += gs) {  // pair pass and second kick
            const uint32_t i = e / kAdjLanes, l = e % kAdjLanes;
            bool direct = false;  // terms that may overflow the warp's histogram go to the tick's one by one
            if (gr && !a.walk) {  // 65,535 terms (of at most `two`'s eight visits of a pair) cannot overflow 32 bits
                const uint32_t most = a.two ? 65535u / 8u : 65535u;
                uint32_t terms = __reduce_add_sync(0xffffffffu, i < n ? min(a.cnt[e], 65536u) : 0u);
                direct = terms > most;
                if (direct) terms = 0u;
                if (held + terms > most) {
                    __syncwarp();
                    flush(wh, 1, (int)(tid & 31u), 32);
                    __syncwarp();
                    held = 0;
                }
                held += terms;
            }
            double ax = 0.0, ay = 0.0, az = 0.0;
            long long fx = 0, fy = 0, fz = 0;
            if (i < n) {
                const double4 pi = load_slab(X, i);
                const uint32_t ti = packed_elem(pi.w) * kNElem;
                const uint32_t kti = F32 ? packed_kind(pi.w) * a.L32.nkinds : 0u;
                const double qi = a.charge[i], mi = a.mass[i], inv_mi = a.inv_mass[i];
                adj_partners(a, X, i, l, [&](uint32_t j, const double4& pj) {
                    const double dx = adj_image(a, xsub(pi.x, pj.x), 0);
                    const double dy = adj_image(a, xsub(pi.y, pj.y), 1);
                    const double dz = adj_image(a, xsub(pi.z, pj.z), 2);
                    const double d2 = xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz));
                    if (d2 >= a.L.rc2) return;
                    const double d = xsqrt(d2);
                    if (d <= kEpsF64) return;
                    const int mult = a.two ? pair_multiplicity(a.fg, packed_cell(pi.w), packed_cell(pj.w)) : 1;
                    const bool count = j > i;
                    double Vij = 0.0;
                    if (F32) {
                        const float gx = (float)dx, gy = (float)dy, gz = (float)dz;
                        float fs, vf;
                        pair_f32(a.L32, s_tab[kti + packed_kind(pj.w)], dist2(gx, gy, gz), fs, vf);
                        long long qx, qy, qz;
                        quant3(fmul(gx, fs), fmul(gy, fs), fmul(gz, fs), qx, qy, qz, a.err);
                        fx += mult * qx;
                        fy += mult * qy;
                        fz += mult * qz;
                        Vij = (double)vf;
                    } else {
                        const uint32_t tt = ti + packed_elem(pj.w);
                        const bool far = a.L.coul || a.L.grav;
                        const double inv = __drcp_rn(d);
                        double fmag = 0.0;
                        pair_f64_e24(a.L, d, inv, s_sig[tt], s_eps[tt], s_e24[tt], qi, far ? a.charge[j] : 0.0, mi,
                                     far ? a.mass[j] : 0.0, fmag, Vij);
                        if (fmag != 0.0) {
                            for (int r = 0; r < mult; ++r) {
                                ax = xadd(ax, xmul(xmul(xmul(dx, inv), fmag), inv_mi));
                                ay = xadd(ay, xmul(xmul(xmul(dy, inv), fmag), inv_mi));
                                az = xadd(az, xmul(xmul(xmul(dz, inv), fmag), inv_mi));
                            }
                        }
                    }
                    if (!a.obs || !count) return;
                    for (int r = 0; r < mult; ++r) V = xadd(V, Vij);
                    if (!gr) return;
                    // half of the partners count: the warp takes their distances together below
                    if (!a.two && !direct) {
                        const uint32_t at = atomicAdd(&s_queued[tid / 32], 1u);
                        if (at < kAdjQueue) {
                            s_queue[tid / 32][at] = d;
                            return;
                        }
                    }
                    gr_bins(a.gs, d, [&](int b, double, double G) {
                        const unsigned long long v = (unsigned long long)(mult * llrint(G * kHistScale));
                        if (direct) atomicAdd(&a.ghist[turn * bins + b], v);
                        else into_warp(b, v);
                    });
                });
            }
            if (gr) {
                __syncwarp();
                const uint32_t queued = min(s_queued[tid / 32], kAdjQueue);
                for (uint32_t k = tid & 31u; k < queued; k += 32)
                    gr_bins(a.gs, s_queue[tid / 32][k],
                            [&](int b, double, double G) { into_warp(b, (unsigned long long)llrint(G * kHistScale)); });
                __syncwarp();
                if ((tid & 31u) == 0) s_queued[tid / 32] = 0u;
                __syncwarp();
            }
            // every lane of an atom is in the same warp and takes part
            if (F32) {
                fx = lane_sum_ll(fx);
                fy = lane_sum_ll(fy);
                fz = lane_sum_ll(fz);
            } else {
                ax = lane_sum(ax);
                ay = lane_sum(ay);
                az = lane_sum(az);
            }
            if (i < n && l < 3) {
                double acc = l == 0 ? ax : (l == 1 ? ay : az);
                if (F32) acc = xmul(xmul(__ll2double_rn(l == 0 ? fx : (l == 1 ? fy : fz)), kFixInv), a.inv_mass[i]);
                double* sv = a.S + (3 + l) * cap + i;
                sv[3 * cap] = acc;
                *sv = xadd(*sv, xmul(acc, a.half_dt));
            }
        }
        if (a.obs) {
            V = block_sum<kAdjThreads>(V, sh);
            if (tid == 0) a.vpart[turn * gridDim.x + blockIdx.x] = V;
            if (gr) {
                __syncthreads();
                flush(s_hist, kAdjThreads / 32, (int)tid, kAdjThreads);
                held = 0;
            }
        }
    }
    if (a.obs) {
        if (!grid_barrier(a.sync, a.err, a.polls, target, &s_ok)) return;
        if (recorder) record(a.last);
    }
    grid_leave(a.sync);
}

// The reverse sweep of ticks last .. first (see the file comment), from the
// positions that k_adj_ticks kept.  P rows: sigma, epsilon, rc_lj,
// rc_coulomb, rc_gravity partials per atom.
__global__ void __launch_bounds__(kAdjThreads, 2) k_adj_reverse(const __grid_constant__ AdjArgs a) {
    __shared__ double s_sig[kNElem * kNElem], s_eps[kNElem * kNElem], s_is[kNElem * kNElem];
    __shared__ double s_bw[kAdjMaxBins];
    __shared__ uint32_t s_warp[kAdjThreads / 32], s_off[kScanMaxTiles];
    __shared__ AdjFound s_found[kAdjThreads / 32];
    __shared__ int s_ok;
    const uint32_t tid = threadIdx.x, n = a.n, lanes = n * kAdjLanes;
    const uint32_t gt = blockIdx.x * kAdjThreads + tid, gs = gridDim.x * kAdjThreads;
    const uint32_t pad = (lanes + 31u) & ~31u;
    const size_t cap = a.cap;
    uint32_t target = 0;
    if (*a.err & (kErrCapacity | kErrBarrier)) return;  // an earlier launch of the call ended early
    for (int k = tid; k < kNElem * kNElem; k += kAdjThreads) {
        s_sig[k] = a.psig[k];
        s_eps[k] = a.peps[k];
        s_is[k] = 1.0 / a.psig[k];
    }
    if (a.gr)
        for (int k = tid; k < a.gs.bins; k += kAdjThreads) s_bw[k] = a.bw[k];
    for (uint32_t c = gt; c < a.lg.ncell + 1; c += gs) a.count[c] = a.fill[c] = 0u;
    for (uint32_t e = gt; e < lanes; e += gs) {  // W/m of the last tick
        const uint32_t i = e / kAdjLanes, l = e % kAdjLanes;
        if (l >= 3) continue;
        const double *lv = a.Ladj + (3 + l) * cap + i, *la = lv + 3 * cap;
        a.W[(size_t)(a.last & 1) * 4 * cap + 4 * (size_t)i + l] = (*la + a.half_dt * *lv) * a.inv_mass[i];
    }
    int built = 0;
    for (int t = a.last; t >= a.first; --t) {
        const double* X = a.slabs + (size_t)(t - a.first) * 4 * cap;
        const double* W = a.W + (size_t)(t & 1) * 4 * cap;
        const int ask = t % 3;
        if (!grid_barrier(a.sync, a.err, a.polls, target, &s_ok)) return;
        const bool rebuild = !built || a.walk || *(volatile uint32_t*)&a.sync->request[ask] != 0u;
        if (blockIdx.x == 0 && tid == 0) a.sync->request[(ask + 1) % 3] = 0u;  // tick t + 1's, read before this barrier
        if (rebuild) {
            if (!adj_rebuild(a, X, target, &s_ok, s_warp, s_off, s_found)) return;
            built = t;
        }
        const bool gr = a.gr && t % a.every == 0;
        const double alpha = a.alpha[t - 1];
        const double* Xp = t > a.first ? X - 4 * cap : nullptr;  // the next tick of the sweep
        const bool odd = a.wrap && ((built - (t - 1)) & 1);
        bool over = false;
        for (uint32_t e = gt; e < pad; e += gs) {
            const uint32_t i = e / kAdjLanes, l = e % kAdjLanes;
            double gx = 0.0, gy = 0.0, gz = 0.0;
            double Ps = 0.0, Pe = 0.0, Pr0 = 0.0, Pr1 = 0.0, Pr2 = 0.0;
            if (i < n) {
                const double4 pi = load_slab(X, i), wi = load_slab(W, i);
                const uint32_t ti = packed_elem(pi.w);
                const double qi = a.charge[i], mi = a.mass[i];
                const double ehalf = 0.5 / a.epsk[ti];
                adj_partners(a, X, i, l, [&](uint32_t j, const double4& pj) {
                    const double dx = adj_image(a, pi.x - pj.x, 0);
                    const double dy = adj_image(a, pi.y - pj.y, 1);
                    const double dz = adj_image(a, pi.z - pj.z, 2);
                    const double d2 = dx * dx + dy * dy + dz * dz;
                    if (d2 >= a.L.rc2) return;
                    const double d = sqrt(d2);
                    if (d <= kEpsF64) return;
                    const double inv = 1.0 / d;
                    const double nx = dx * inv, ny = dy * inv, nz = dz * inv;
                    const double4 wj = load_slab(W, j);
                    const double ux = wi.x - wj.x, uy = wi.y - wj.y, uz = wi.z - wj.z;
                    const double rho = nx * ux + ny * uy + nz * uz;
                    const uint32_t tt = ti * kNElem + packed_elem(pj.w);
                    const bool far = a.L.coul || a.L.grav;
                    const double ep = s_eps[tt];
                    const PairG G = pair_grad(a.L, d, inv, s_sig[tt], s_is[tt], ep, qi, far ? a.charge[j] : 0.0, mi,
                                              far ? a.mass[j] : 0.0);
                    double psi = 0.0;
                    if (gr)
                        gr_bins(a.gs, d, [&](int b, double z, double Gb) { psi += s_bw[b] * (2.0 * a.gs.c2 * z) * Gb; });
                    const double mult =
                        a.two ? (double)pair_multiplicity(a.fg, packed_cell(pi.w), packed_cell(pj.w)) : 1.0;
                    const double c1 = mult * (rho * G.fd + alpha * G.Ud + psi), c2 = mult * (G.f * inv);
                    gx += c1 * nx + c2 * (ux - rho * nx);
                    gy += c1 * ny + c2 * (uy - rho * ny);
                    gz += c1 * nz + c2 * (uz - rho * nz);
                    Ps += mult * (0.5 * (rho * G.fs + alpha * G.Us));
                    Pe += mult * (ep * ehalf * (rho * G.fe + alpha * G.Ue));
                    Pr0 += mult * (0.5 * (rho * G.frc[0] + alpha * G.Urc[0]));
                    if (a.L.coul) Pr1 += mult * (0.5 * (rho * G.frc[1] + alpha * G.Urc[1]));
                    if (a.L.grav) Pr2 += mult * (0.5 * (rho * G.frc[2] + alpha * G.Urc[2]));
                });
            }
            // every lane of an atom is in the same warp and takes part
            gx = lane_sum(gx);
            gy = lane_sum(gy);
            gz = lane_sum(gz);
            Ps = lane_sum(Ps);
            Pe = lane_sum(Pe);
            Pr0 = lane_sum(Pr0);
            if (a.L.coul) Pr1 = lane_sum(Pr1);
            if (a.L.grav) Pr2 = lane_sum(Pr2);
            double xp = 0.0;
            if (i < n && l < 3) {
                double* Lx = a.Ladj + l * cap + i;
                const double lx = Lx[0] + (l == 0 ? gx : (l == 1 ? gy : gz));
                const double lv = Lx[3 * cap] + a.dt * lx, la = a.half_dt * lv;
                Lx[0] = lx;
                Lx[3 * cap] = lv;
                Lx[6 * cap] = la;
                if (Xp) {
                    a.W[(size_t)((t - 1) & 1) * 4 * cap + 4 * (size_t)i + l] = (la + a.half_dt * lv) * a.inv_mass[i];
                    xp = Xp[4 * (size_t)i + l];
                }
            }
            if (i < n && l < 5)
                a.P[l * cap + i] += l == 0 ? Ps : (l == 1 ? Pe : (l == 2 ? Pr0 : (l == 3 ? Pr1 : Pr2)));
            if (Xp && !a.walk) over |= !(moved2(a, i, l, i < n, xp, odd) <= a.lim2);
        }
        if (Xp && __syncthreads_or(over) && tid == 0) a.sync->request[(ask + 2) % 3] = 1u;  // tick t - 1's
    }
    grid_leave(a.sync);
}

// out[e] = sum of sigma partials of element e, out[10 + e] epsilon partials,
// out[20..22] the cutoff partials; one block per output, fixed order.
__global__ void __launch_bounds__(256) k_adj_reduce(uint32_t n, const uint8_t* __restrict__ elem,
                                                    const double* __restrict__ P, size_t cap, double* out) {
    __shared__ double sh[256 / 32];
    int o = blockIdx.x;
    int row = o < kNElem ? 0 : (o < 2 * kNElem ? 1 : 2 + (o - 2 * kNElem));
    int e = o < 2 * kNElem ? o % kNElem : -1;
    double s = 0.0;
    for (uint32_t i = threadIdx.x; i < n; i += 256)
        if (e < 0 || elem[i] == e) s += P[(size_t)row * cap + i];
    s = block_sum<256>(s, sh);
    if (threadIdx.x == 0) out[o] = s;
}

__global__ void k_adj_export(uint32_t n, Vec3Field f, double* aos) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < 3; ++k) aos[3 * (size_t)i + k] = f.c(k, i);
}

}  // namespace

// Buffers of the adjoint, owned by one handle.
struct AdjBuffers {
    size_t cap = 0, n = 0;
    int T = 0, K = 0, nck = 0, bins = 0, every = 1, samples = 0;
    int cap_T = 0, cap_ck = 0, cap_K = 0, cap_bins = 0;
    double gr_rmax = 0, gr_width = 0, gr_support = 0;
    bool ready = false;
    bool f32 = false;  // the forward in the mixed method (a handle of mixed precision)
    uint8_t *kind = nullptr, *elem = nullptr;
    double *S = nullptr, *Ladj = nullptr, *P = nullptr, *ck = nullptr, *slabs = nullptr, *W = nullptr, *ref = nullptr;
    double *charge = nullptr, *mass = nullptr, *inv_mass = nullptr;
    double* sorted = nullptr;
    uint32_t *key = nullptr, *count = nullptr, *start = nullptr, *fill = nullptr;
    uint32_t *order = nullptr;
    uint32_t *list = nullptr, *cnt = nullptr, *off = nullptr, *pool = nullptr;  // one block, not in `owned`
    uint32_t* large_pool = nullptr;  // in place of the block's, once that was too small
    unsigned long long* pool_used = nullptr;
    size_t pool_cap = 0;  // words
    bool walk = false;    // this forward's ticks go without lists
    GridGeom lg{}, wg{};  // of the lists, and without them
    uint32_t cap_l = 0;
    size_t cap_cells = 0;
    int resident[3] = {0, 0, 0};  // blocks that fit: FP64 ticks, mixed ticks, the reverse sweep
    size_t resident_smem = 0;
    double *vpart = nullptr, *dV = nullptr, *alpha = nullptr, *bw = nullptr, *hacc = nullptr;
    unsigned long long* ghist = nullptr;
    GridSync* sync = nullptr;
    double *tab = nullptr;  // psig[100], peps[100], epsk[10], out[kNOut]
    std::vector<void*> owned;
};

static void adj_free_lists(AdjBuffers* A) {
    cudaFree(A->list);
    cudaFree(A->large_pool);
    A->list = A->cnt = A->off = A->pool = A->large_pool = nullptr;
    A->pool_cap = 0;
    A->cap_l = 0;
}

static void adj_release(AdjBuffers* A) {
    for (void* p : A->owned) cudaFree(p);
    A->owned.clear();
    adj_free_lists(A);
}

void adjoint_free(gx_handle* h) {
    if (!h || !h->adj) return;
    AdjBuffers* A = static_cast<AdjBuffers*>(h->adj);
    adj_release(A);
    delete A;
    h->adj = nullptr;
}

namespace {

// Lists hold up to this many partners an atom on average; above, and where
// their rows would take more than half of what memory is free, every tick
// sorts the atoms and walks their cells.  Twenty ticks and their gradient, ms,
// with lists / without: 27,000 atoms of 900 partners 66 / 76, of 2,130 260 /
// 245; 8,000 of 266 6.6 / 14.3, of 65 2.6 / 6.8.
constexpr double kAdjMostPartners = 1024.0;
constexpr size_t kAdjPoolMost = (size_t)1 << 28;  // words

// Cells >= min_cell, no more of them than atoms or one scan's tiles of 1,024
// cells.  (A limit of 65,536 cells whatever the atoms: 8,000,000 atoms, 122 in
// a cell, took 3.6 s for twenty ticks and their gradient, 2.0 so.)
bool adj_grid(const gx_handle* h, double min_cell, GridGeom* g) {
    const size_t most = std::max((size_t)kScanTileCells * kScanMaxTiles - 1, (size_t)h->n);
    int ok = 0;
    for (int k = 0; k < 64; ++k, min_cell *= 1.3) {
        *g = make_grid(h->p.box, min_cell, &ok);
        if (ok && g->ncell <= most) return true;
    }
    return false;
}

// The mean neighbourhood of a list.
double adj_mean(const gx_handle* h) {
    const double rl = h->fs.rc * (1.0 + kAdjSkin), vol = h->p.box[0] * h->p.box[1] * h->p.box[2];
    return std::min((double)h->n / vol * (4.0 / 3.0) * 3.14159265358979 * rl * rl * rl, (double)h->n);
}

// Rows of twice a lane's share of the mean neighbourhood, and a pool for what
// is denser (64,000 atoms, a cube at four times the mean density: 43 ms for
// twenty ticks and their gradient, 117 with a walk of 27 cells every tick, 427
// with a look at all atoms for the denser lanes).  Without lists when they
// cannot be had.
int adj_alloc_lists(gx_handle* h, AdjBuffers* A, double mean) {
    A->walk = mean > kAdjMostPartners;
    const uint32_t cap_l = (uint32_t)std::ceil(2.0 * mean / kAdjLanes) + 8u;
    if (A->walk || (A->list && cap_l <= A->cap_l)) return GX_OK;
    adj_free_lists(A);
    const size_t lanes = kAdjLanes * A->cap, rows = cap_l * lanes, pool = 16 * A->cap;
    const size_t bytes = (rows + 2 * lanes + pool) * sizeof(uint32_t);
    size_t free_bytes = ~(size_t)0, all = 0;
    if (bytes >> 30) GX_CUDA(h, cudaMemGetInfo(&free_bytes, &all));
    if (bytes > free_bytes / 2 || cudaMalloc((void**)&A->list, bytes) != cudaSuccess) {
        cudaGetLastError();
        A->list = nullptr;
        A->walk = true;
        return GX_OK;
    }
    A->cnt = A->list + rows;
    A->off = A->cnt + lanes;
    A->pool = A->off + lanes;
    A->cap_l = cap_l;
    A->pool_cap = pool;
    return GX_OK;
}

// The pool as large as the lists asked for, and as much again; without lists
// where that is too much.
int adj_more_pool(gx_handle* h, AdjBuffers* A) {
    unsigned long long need = 0;
    GX_CUDA(h, cudaMemcpy(&need, A->pool_used, sizeof need, cudaMemcpyDeviceToHost));
    cudaFree(A->large_pool);
    A->pool = A->large_pool = nullptr;
    A->pool_cap = 0;
    const size_t words = (size_t)std::min<unsigned long long>(2 * need, kAdjPoolMost);
    if (words < need || cudaMalloc((void**)&A->large_pool, words * sizeof(uint32_t)) != cudaSuccess) {
        cudaGetLastError();
        A->large_pool = nullptr;
        adj_free_lists(A);
        A->walk = true;
    } else {
        A->pool = A->large_pool;
        A->pool_cap = words;
    }
    return GX_OK;
}

int adj_alloc(gx_handle* h, AdjBuffers* A, size_t n, int T, int K, int bins) {
    int nck = (T + K - 1) / K;
    if (!adj_grid(h, h->fs.rc * (1.0 + kAdjSkin), &A->lg) || !adj_grid(h, h->fs.rc, &A->wg))
        return set_err(h, GX_ERR_ARG, "adjoint list grid is empty or too large");
    const double mean = adj_mean(h);
    const size_t cells = (size_t)std::max(A->lg.ncell, A->wg.ncell) + 1;
    if (n <= A->cap && T <= A->cap_T && nck <= A->cap_ck && K <= A->cap_K && bins <= A->cap_bins &&
        cells <= A->cap_cells && A->tab)
        return adj_alloc_lists(h, A, mean);
    adj_release(A);
    A->tab = nullptr;
    A->cap = 0;
    size_t cap = n < 1 ? 1 : n;
    cap = (cap + 31) & ~(size_t)31;
    int binc = bins < 1 ? 1 : bins;
    auto get = [&](void** p, size_t bytes) -> int {
        cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
        if (e != cudaSuccess) return cuda_err(h, e, "adjoint buffers");
        A->owned.push_back(*p);
        return GX_OK;
    };
    const size_t slabs = (size_t)std::max(std::min(K, T), 2);
    int rc = 0;
    rc |= get((void**)&A->S, 9 * cap * sizeof(double));
    rc |= get((void**)&A->Ladj, 9 * cap * sizeof(double));
    rc |= get((void**)&A->P, 5 * cap * sizeof(double));
    rc |= get((void**)&A->ck, (size_t)nck * 9 * cap * sizeof(double));
    rc |= get((void**)&A->slabs, slabs * 4 * cap * sizeof(double));
    rc |= get((void**)&A->W, 2 * 4 * cap * sizeof(double));
    rc |= get((void**)&A->ref, 3 * cap * sizeof(double));
    rc |= get((void**)&A->charge, cap * sizeof(double));
    rc |= get((void**)&A->mass, cap * sizeof(double));
    rc |= get((void**)&A->inv_mass, cap * sizeof(double));
    rc |= get((void**)&A->elem, cap);
    rc |= get((void**)&A->kind, cap);
    rc |= get((void**)&A->key, 2 * cap * sizeof(uint32_t));
    A->order = A->key + cap;
    rc |= get((void**)&A->sorted, 4 * cap * sizeof(double));
    rc |= get((void**)&A->count, cells * sizeof(uint32_t));
    rc |= get((void**)&A->start, cells * sizeof(uint32_t));
    rc |= get((void**)&A->fill, cells * sizeof(uint32_t));
    rc |= get((void**)&A->vpart, 2 * (nblk(cap * kAdjLanes, kAdjThreads) + 1) * sizeof(double));
    rc |= get((void**)&A->dV, (size_t)T * sizeof(double));
    rc |= get((void**)&A->alpha, (size_t)T * sizeof(double));
    rc |= get((void**)&A->bw, (size_t)binc * sizeof(double));
    rc |= get((void**)&A->ghist, 2 * (size_t)binc * sizeof(unsigned long long));
    rc |= get((void**)&A->hacc, (size_t)binc * sizeof(double));
    rc |= get((void**)&A->pool_used, sizeof(unsigned long long) + sizeof(GridSync));
    A->sync = reinterpret_cast<GridSync*>(A->pool_used + 1);
    rc |= get((void**)&A->tab, (2 * kNElem * kNElem + kNElem + kNOut) * sizeof(double));
    if (rc) {
        adj_release(A);
        A->tab = nullptr;
        return rc;
    }
    A->cap = cap;
    A->cap_T = T;
    A->cap_ck = nck;
    A->cap_K = K;
    A->cap_bins = binc;
    A->cap_cells = cells;
    return adj_alloc_lists(h, A, mean);
}

Vec3Field field(double* base, size_t cap) { return Vec3Field{base, cap}; }

GrSpec gr_spec(const AdjBuffers* A) {
    GrSpec g;
    g.bins = A->bins;
    g.dr = A->bins > 0 ? A->gr_rmax / A->bins : 1.0;
    g.width = A->gr_width;
    g.reach = A->gr_support * A->gr_width;
    g.c2 = A->gr_width > 0 ? -0.5 / (A->gr_width * A->gr_width) : 0.0;
    return g;
}

AdjArgs adj_args(gx_handle* h, AdjBuffers* A) {
    AdjArgs a{};
    a.lg = A->walk ? A->wg : A->lg;
    a.tile_log2 = 10;
    static_assert(kScanTileCells == 1u << 10, "");
    a.fg = h->fgrid;
    a.two = a.fg.n[0] == 2 || a.fg.n[1] == 2 || a.fg.n[2] == 2;
    a.plain = a.fg.n[0] >= 3 && a.fg.n[1] >= 3 && a.fg.n[2] >= 3 && h->p.enable_boundaries;
    for (int k = 0; k < 3; ++k) {
        a.half_box[k] = 0.5 * h->p.box[k];
        a.inv_box[k] = 1.0 / h->p.box[k];
    }
    a.n = (uint32_t)A->n;
    a.cap = A->cap;
    a.L = make_law64(h);
    if (A->f32) a.L32 = make_law32(h);
    a.tabf = h->d_pairf;
    a.psig = A->tab;
    a.peps = A->tab + kNElem * kNElem;
    a.epsk = A->tab + 2 * kNElem * kNElem;
    a.elem = A->elem;
    a.kind = A->kind;
    a.charge = A->charge;
    a.mass = A->mass;
    a.inv_mass = A->inv_mass;
    a.S = A->S;
    a.slabs = A->slabs;
    a.K = A->K;
    a.list = A->list;
    a.cnt = A->cnt;
    a.cap_l = A->cap_l;
    a.pool = A->pool;
    a.off = A->off;
    a.pool_used = A->pool_used;
    a.pool_cap = A->pool_cap;
    a.walk = A->walk ? 1 : 0;
    a.order = A->order;
    a.ref = A->ref;
    a.key = A->key;
    a.sorted = A->sorted;
    a.count = A->count;
    a.start = A->start;
    a.fill = A->fill;
    while (a.tile_log2 < 32 && (a.lg.ncell >> a.tile_log2) >= kScanMaxTiles) ++a.tile_log2;
    a.sync = A->sync;
    a.err = h->derr;
    a.polls = h->wait_polls;
    a.vpart = A->vpart;
    a.pot = A->dV;
    a.ghist = A->ghist;
    a.hacc = A->hacc;
    a.gs = gr_spec(A);
    a.every = A->every;
    a.half_dt = 0.5 * h->p.dt;
    a.dt = h->p.dt;
    const double rl = h->fs.rc * (1.0 + kAdjSkin), lim = 0.5 * kAdjSkin * h->fs.rc * (1.0 - 1e-6);
    a.rl2 = rl * rl;
    a.lim2 = lim * lim;
    a.wrap = h->p.enable_boundaries ? 1 : 0;
    a.Ladj = A->Ladj;
    a.P = A->P;
    a.W = A->W;
    a.alpha = A->alpha;
    a.bw = A->bw;
    return a;
}

// k_adj_ticks' histograms: one per warp, two words a bin.
constexpr size_t hist_bytes(int bins) { return (size_t)(kAdjThreads / 32) * 2 * bins * sizeof(uint32_t); }

// One cooperative launch of kernel `which` (AdjBuffers::resident).
int adj_launch(gx_handle* h, AdjBuffers* A, int which, AdjArgs& a) {
    const void* kern = which == 2 ? (const void*)k_adj_reverse
                                  : (which == 1 ? (const void*)k_adj_ticks<true> : (const void*)k_adj_ticks<false>);
    const size_t smem = which < 2 ? hist_bytes(A->bins) : 0;
    if (smem != A->resident_smem && which < 2) {
        A->resident[0] = A->resident[1] = 0;
        A->resident_smem = smem;
    }
    int& resident = A->resident[which];
    if (!resident) {
        int per = 0, sms = 0;
        // the limit belongs to the kernel, not to this handle: the most that any handle asks for
        if (which < 2)
            GX_CUDA(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_bytes(kAdjMaxBins)));
        GX_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kAdjThreads, smem));
        GX_CUDA(h, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->p.device));
        resident = std::max(per * sms, 1);
    }
    const unsigned grid = std::min(nblk((size_t)a.n * kAdjLanes, kAdjThreads), (unsigned)resident);
    void* args[] = {&a};
    GX_CUDA(h, cudaLaunchCooperativeKernel(kern, grid, kAdjThreads, args, smem, h->stream));
    ++h->launches;
    return GX_OK;
}

double gr_norm(const gx_handle* h, const AdjBuffers* A, int k) {
    const double pi = 3.14159265358979323846;
    double vol = h->p.box[0] * h->p.box[1] * h->p.box[2];
    double npair = 0.5 * (double)A->n * ((double)A->n - 1.0);
    double dr = A->gr_rmax / A->bins, r = (k + 0.5) * dr;
    return vol / (npair * 4.0 * pi * r * r * std::sqrt(2.0 * pi) * A->gr_width);
}

// The outcome of a call's launches; *again: the lists needed more room and
// have it now, or do without.
int check_err(gx_handle* h, AdjBuffers* A, bool* again) {
    uint32_t e = 0;
    *again = false;
    GX_CUDA(h, cudaMemcpyAsync(&e, h->derr, sizeof e, cudaMemcpyDeviceToHost, h->stream));
    GX_CUDA(h, cudaStreamSynchronize(h->stream));
    if (!e) return GX_OK;
    cudaMemsetAsync(h->derr, 0, sizeof(uint32_t), h->stream);
    if (e & kErrBarrier) {  // a block gave up at a barrier: the words are no longer zero
        cudaMemsetAsync(A->sync, 0, sizeof(GridSync), h->stream);
        return set_err(h, GX_ERR_TIMEOUT, "a bounded device wait timed out in the adjoint");
    }
    if (e & kErrNonFinite) return set_err(h, GX_ERR_NONFINITE, "non-finite position in the adjoint trajectory");
    if (e & kErrSaturation)  // the fixed-point force of the mixed forward
        return set_err(h, GX_ERR_SATURATION, "fixed-point force saturated in the adjoint trajectory");
    if (e & kErrCapacity) {
        *again = true;
        return adj_more_pool(h, A);
    }
    return GX_OK;
}

}  // namespace
}  // namespace gx

using namespace gx;

int gx_adjoint_forward(gx_handle* h, const gx_adjoint_spec* spec, double* potential, double* gr) {
    if (!h || !spec || !potential) return GX_ERR_ARG;
    int rc = GX_OK;
    if ((rc = check_state(h))) return rc;
    if (h->n == 0) return set_err(h, GX_ERR_ARG, "the adjoint needs at least one atom");
    if ((rc = settle_step_errors(h))) return rc;  // a queued step's error first: the word is cleared below
    h->nl_fresh = false;  // conservative: the passes below may reorder or move the resident state
    if (spec->nsteps < 1 || spec->checkpoint_every < 1) return set_err(h, GX_ERR_ARG, "nsteps and checkpoint_every must be >= 1");
    if (spec->gr_bins < 0 || spec->gr_bins > kAdjMaxBins) return set_err(h, GX_ERR_ARG, "gr_bins must be in [0, 512]");
    if (spec->gr_bins > 0) {
        if (spec->gr_every < 1 || !(spec->gr_rmax > 0.0) || !(spec->gr_width > 0.0) || !(spec->gr_support > 0.0))
            return set_err(h, GX_ERR_ARG, "g(r) spec needs gr_every >= 1 and positive rmax, width, support");
        if (spec->gr_rmax + spec->gr_support * spec->gr_width > h->fs.rc)
            return set_err(h, GX_ERR_ARG, "gr_rmax + gr_support * gr_width exceeds the force cutoff");
    }
    if (h->p.enable_thermostat || h->p.enable_bond_interaction)
        return set_err(h, GX_ERR_UNSUPPORTED, "the adjoint covers NVE ticks without the bond spring");
    for (int e = 0; e < kNElem; ++e)
        if (!(h->p.epsilon_k[e] > 0.0)) return set_err(h, GX_ERR_UNSUPPORTED, "the adjoint needs every epsilon_k > 0");
    if (h->n >= (1u << 28)) return set_err(h, GX_ERR_CAPACITY, "too many atoms");
    if (h->precision == GX_MIXED && h->nkinds > kMaxKinds)
        return set_err(h, GX_ERR_UNSUPPORTED, "the mixed forward supports at most 16 distinct (element, charge) kinds");
    // NVE only, so no Berendsen scale can be pending on the handle's velocities.
    if (!h->adj) h->adj = new AdjBuffers();
    AdjBuffers* A = static_cast<AdjBuffers*>(h->adj);
    A->ready = false;
    const int T = spec->nsteps, K = spec->checkpoint_every;
    if ((rc = adj_alloc(h, A, h->n, T, K, spec->gr_bins))) return rc;
    A->T = T;
    A->K = K;
    A->nck = (T + K - 1) / K;
    A->bins = spec->gr_bins;
    A->every = spec->gr_bins > 0 ? spec->gr_every : 1;
    A->gr_rmax = spec->gr_rmax;
    A->gr_width = spec->gr_width;
    A->gr_support = spec->gr_support;
    A->samples = 0;
    A->n = h->n;
    A->f32 = h->precision == GX_MIXED;
    const uint32_t n = (uint32_t)h->n;
    const size_t cap = A->cap;
    // pair table, epsilon_k
    std::vector<double> tab(2 * kNElem * kNElem + kNElem, 0.0);
    std::memcpy(tab.data(), h->fs.pair_sigma, sizeof h->fs.pair_sigma);
    std::memcpy(tab.data() + kNElem * kNElem, h->fs.pair_eps, sizeof h->fs.pair_eps);
    for (int e = 0; e < kNElem; ++e) tab[2 * kNElem * kNElem + e] = h->p.epsilon_k[e];
    GX_CUDA(h, cudaMemcpyAsync(A->tab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    StateBuf& b = h->buf[h->cur];
    GX_CUDA(h, cudaMemsetAsync(A->sync, 0, sizeof(GridSync), h->stream));
    if (A->bins > 0) A->samples = T / A->every;
    std::vector<double> hacc(A->bins > 0 ? A->bins : 0);
    for (bool again = true; again;) {
        GX_LAUNCH(h, k_adj_import, nblk(n, 256), 256, b, n, field(A->S, cap), field(A->S + 3 * cap, cap),
                  field(A->S + 6 * cap, cap), A->elem, A->charge, A->mass, A->inv_mass, A->kind);
        if (A->bins > 0) {
            GX_CUDA(h, cudaMemsetAsync(A->hacc, 0, A->bins * sizeof(double), h->stream));
            GX_CUDA(h, cudaMemsetAsync(A->ghist, 0, 2 * A->bins * sizeof(unsigned long long), h->stream));
        }
        AdjArgs args = adj_args(h, A);
        args.ck = A->ck;
        args.obs = 1;
        for (int t0 = 0; t0 < T; t0 += kAdjTicksPerLaunch) {
            args.first = t0 + 1;
            args.last = std::min(t0 + kAdjTicksPerLaunch, T);
            if ((rc = adj_launch(h, A, A->f32 ? 1 : 0, args))) return rc;
        }
        GX_CUDA(h, cudaMemcpyAsync(potential, A->dV, T * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
        if (A->bins > 0)
            GX_CUDA(h, cudaMemcpyAsync(hacc.data(), A->hacc, A->bins * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
        GX_CUDA(h, cudaStreamSynchronize(h->stream));
        GX_CUDA(h, cudaGetLastError());
        if ((rc = check_err(h, A, &again))) return rc;
    }
    if (gr)
        for (int k = 0; k < A->bins; ++k) gr[k] = A->samples ? hacc[k] * gr_norm(h, A, k) / A->samples : 0.0;
    A->ready = true;
    return GX_OK;
}

int gx_adjoint_backward(gx_handle* h, const double* dl_dpotential, const double* dl_dgr, double* grad_sigma,
                        double* grad_epsilon_k, double* grad_pos0, double* grad_vel0, double* grad_acc0) {
    if (!h || !grad_sigma || !grad_epsilon_k) return GX_ERR_ARG;
    AdjBuffers* A = static_cast<AdjBuffers*>(h->adj);
    if (!A || !A->ready) return set_err(h, GX_ERR_STATE, "call gx_adjoint_forward first");
    if (h->n != A->n) return set_err(h, GX_ERR_STATE, "atom count changed since gx_adjoint_forward");
    int rc = settle_step_errors(h);
    if (rc) return rc;
    const uint32_t n = (uint32_t)A->n;
    const size_t cap = A->cap;
    const int T = A->T, K = A->K;
    // cotangents
    std::vector<double> alpha(T, 0.0), bw(A->bins > 0 ? A->bins : 1, 0.0);
    if (dl_dpotential)
        for (int t = 0; t < T; ++t) alpha[t] = dl_dpotential[t];
    if (dl_dgr && A->bins > 0 && A->samples > 0)
        for (int k = 0; k < A->bins; ++k) bw[k] = dl_dgr[k] * gr_norm(h, A, k) / A->samples;
    GX_CUDA(h, cudaMemcpyAsync(A->alpha, alpha.data(), T * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    GX_CUDA(h, cudaMemcpyAsync(A->bw, bw.data(), bw.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    double* out = A->tab + 2 * kNElem * kNElem + kNElem;
    double sums[kNOut];
    for (bool again = true; again;) {
        GX_CUDA(h, cudaMemsetAsync(A->Ladj, 0, 9 * cap * sizeof(double), h->stream));
        GX_CUDA(h, cudaMemsetAsync(A->P, 0, 5 * cap * sizeof(double), h->stream));
        AdjArgs args = adj_args(h, A);
        args.gr = dl_dgr && A->bins > 0;
        args.keep = 1;
        for (int s = A->nck - 1; s >= 0; --s) {
            args.first = s * K + 1;
            args.last = std::min((s + 1) * K, T);
            GX_CUDA(h, cudaMemcpyAsync(A->S, A->ck + (size_t)s * 9 * cap, 9 * cap * sizeof(double),
                                       cudaMemcpyDeviceToDevice, h->stream));
            if ((rc = adj_launch(h, A, A->f32 ? 1 : 0, args))) return rc;
            if ((rc = adj_launch(h, A, 2, args))) return rc;
        }
        GX_LAUNCH(h, k_adj_reduce, kNOut, 256, n, A->elem, A->P, cap, out);
        GX_CUDA(h, cudaMemcpyAsync(sums, out, sizeof sums, cudaMemcpyDeviceToHost, h->stream));
        double* dsts[3] = {grad_pos0, grad_vel0, grad_acc0};
        double* stage = A->W;  // 8 * cap, free once the sweep is done
        for (int q = 0; q < 3; ++q) {
            if (!dsts[q] || !n) continue;
            GX_LAUNCH(h, k_adj_export, nblk(n, 256), 256, n, field(A->Ladj + (size_t)q * 3 * cap, cap), stage);
            GX_CUDA(h, cudaMemcpyAsync(dsts[q], stage, 3 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
            GX_CUDA(h, cudaStreamSynchronize(h->stream));
        }
        GX_CUDA(h, cudaStreamSynchronize(h->stream));
        GX_CUDA(h, cudaGetLastError());
        if ((rc = check_err(h, A, &again))) return rc;
    }
    // The cutoffs: lj_rc = max(lj_cutoff_factor, 1) * max pair sigma (LjTable::new,
    // forces.rs:223-237), coulomb/gravity rc = max(factor, 1) * max sigma
    // (systems/forces.rs:108-116); the derivative goes to the first element
    // attaining the largest sigma.
    int mstar = 0;
    for (int e = 1; e < kNElem; ++e)
        if (h->p.sigma[e] > h->p.sigma[mstar]) mstar = e;
    double drc = std::fmax(h->p.lj_cutoff_factor, 1.0) * sums[2 * kNElem + 0];
    if (h->p.enable_electrostatics) drc += std::fmax(h->p.coulomb_cutoff, 1.0) * sums[2 * kNElem + 1];
    if (h->p.enable_gravity) drc += std::fmax(h->p.gravity_cutoff, 1.0) * sums[2 * kNElem + 2];
    for (int e = 0; e < kNElem; ++e) {
        grad_sigma[e] = sums[e] + (e == mstar ? drc : 0.0);
        grad_epsilon_k[e] = sums[kNElem + e];
    }
    return GX_OK;
}
