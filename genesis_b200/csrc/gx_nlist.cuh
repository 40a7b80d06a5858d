// gx_nlist.cuh -- the persistent neighbour list's state and the device
// functions that the per-kernel tick (gx_nlist.cu) and the one-launch tick of
// small universes (gx_nltick.cu) share.
#pragma once

#include "gx_gridsync.cuh"
#include "gx_law64.cuh"
#include "gx_pair_f32.cuh"

namespace gx {

// Device words of the one-launch ticks (gx_nltick.cu).
struct TickSync {
    GridSync grid;                 // rebuilds requested by tick parity
    unsigned long long acc[2][4];  // by tick parity: potential, pair count, bond energy
};

struct NlState {
    GridGeom lg{};            // list grid: cells >= r_c + skin
    double skin = -1.0;       // < 0: default (0.1 r_c)
    double skin_used = 0.0;
    int half = -1;            // list kind built: 0 full, 1 half (variant 6)
    int tpp = 0;              // threads per atom in the list pass (1, 2, 4, 8; 0: nl_auto_lanes);
                              // with it or `block` set, the work shape is the per-kernel tick's
    int slots = 16;           // variant 7: stash slots per thread (8 or 16)
    int brick = 1;            // variant 8: 0 = bricks of 4 cells (1024 staged atoms), 1 = 8 cells (2048)
    int block = 0;            // variant 6, one lane per atom: 0 = far ends always global, 128 or 256 = far
                              // ends inside a block of that many atoms summed in shared memory
    int cap_nb = 0;           // list entries per atom
    double expect = 0.0;      // neighbours within r_c + skin at the mean density
    size_t cap = 0;           // atoms the buffers hold
    uint32_t* list = nullptr; // entry e of atom p at list[e * cap + p]
    uint32_t* cnt = nullptr;  // entries per atom (> cap_nb: overflowed)
    float4* ref = nullptr;    // home-frame positions at the last rebuild
    uint32_t* flag = nullptr; // [0] rebuild requested, [1] rebuilds done, [2] half-box translations since (mod 2),
                              // [3] runs of a captured rebuild body
    CellList cl;
    // A captured tick puts the rebuild in the body of a conditional (IF)
    // graph node, set from flag[0], so that a tick without a rebuild does
    // not launch it at all.  The body is captured from a second stream.
    cudaStream_t side = nullptr;
    uint64_t body_kernels = 0;  // kernels in the body (counted when it runs)
    uint32_t body_runs_seen = 0;
    TickSync* tick_sync = nullptr;
    bool tick_sync_dirty = false;  // a launch gave up: clear the words before the next one
    int tick_blocks[4] = {0, 0, 0, 0};  // resident blocks of the one-launch tick: without / with records, mixed then FP64
};

// Universes up to this many atoms and expected half-list entries run their
// ticks in one launch (gx_nltick.cu, where both sides' times stand).
constexpr size_t kTickMaxAtoms = 65536;
constexpr double kTickMaxEntries = 1.7e6;
constexpr size_t kTickMaxAtoms64 = 24576;  // FP64 ticks
// Ticks of one launch at most, so that a long call stays a queue of launches.
constexpr int kTicksPerLaunch = 256;

// Lanes per atom of the list pass where none were set: enough to fill
// the chip and to share the long lists of a condensed state, one where the
// gathers of a homogeneous one set the time.  Microseconds per half-list pass
// with 1 / 2 / 4 / 8 lanes on the lattice: 31 / 21 / 15 / 10 at 4,096 atoms,
// 31 / 23 / 17 / 19 at 32,768, 34 / 25 / 27 / 27 at 59,319, 44 / 42 / 41 / 45
// at 125,000, 76 / 71 / 76 / 90 at 262,144, 124 / 129 / 146 / 177 at 512,000,
// 221 / 236 / 274 / 357 at 1,000,000, 435 / 477 / 563 / 709 at 2,097,152; per
// tick after 1,000 ticks of condensation with charges and gravity:
// 96 / 73 / 60 / 59 at 32,768, 107 / 89 / 82 / 77 at 59,319,
// 263 / 234 / 223 / 232 at 262,144.  The full list (variant 5) has the same
// lines: per captured tick, 1 / 2 / 4 / 8 lanes, 43 / 35 / 29 / 26 at 4,096,
// 49 / 41 / 36 / 38 at 32,768, 56 / 49 / 50 / 48 at 59,319, 79 / 80 / 77 / 78
// at 125,000, 133 / 129 / 133 / 141 at 262,144, 218 / 217 / 225 / 240 at
// 512,000, 382 / 387 / 404 / 437 at 1,000,000, 819 / 829 / 875 / 947 at
// 2,097,152.
inline int nl_auto_lanes(uint32_t n) {
    if (n <= 98304) return 8;
    if (n <= 327680) return 4;
    return n <= (1u << 20) ? 2 : 1;
}

constexpr uint32_t kIdxMask = (1u << 27) - 1u;  // a list word: 27-bit neighbour position, 5-bit neighbour-cell code

// Offset of a coordinate from its home cell's origin in the frame of the
// last rebuild (`shift` = the translation to undo, 0 or L/2), unwrapped
// across the periodic boundary (the atom may have left its home cell).
__device__ __forceinline__ double home_local(double v, double L, double c, uint32_t i, double shift) {
    double u = xsub(rem_euclid(xadd(xadd(v, xmul(0.5, L)), shift), L), xmul((double)i, c));
    if (u > 0.5 * L) u = xsub(u, L);
    else if (u < -0.5 * L) u = xadd(u, L);
    return u;
}

__device__ __forceinline__ float4 stage_one(const GridGeom& g, const StateBuf& b, uint32_t home, uint32_t i,
                                            double x, double y, double z, bool half) {
    uint32_t ix, iy, iz;
    decode(g, home, ix, iy, iz);
    return make_float4((float)home_local(x, g.L[0], g.cell[0], ix, half ? xmul(0.5, g.L[0]) : 0.0),
                       (float)home_local(y, g.L[1], g.cell[1], iy, half ? xmul(0.5, g.L[1]) : 0.0),
                       (float)home_local(z, g.L[2], g.cell[2], iz, half ? xmul(0.5, g.L[2]) : 0.0),
                       __int_as_float((int)b.kind[i]));
}

// The Berendsen scale (thermostat.rs:58-71) of n atoms with kinetic energy K.
__device__ __forceinline__ double berendsen_scale(double K, uint32_t n, double k, double target, double tau) {
    if (n == 0) return 1.0;
    const double t = xdiv(xmul(2.0 / 3.0, xdiv(K, (double)n)), k);
    if (!(isfinite(t) && t > 0.0)) return 1.0;
    return xsqrt(fmax(xadd(1.0, xmul(xdiv(1.0, tau), xsub(xdiv(target, t), 1.0))), 0.0));
}

// Neighbour-cell code: (ox+1) + 3(oy+1) + 9(oz+1); 13 is the home cell.
__device__ __forceinline__ void code_shift(const GridGeom& g, uint32_t code, float& sx, float& sy, float& sz) {
    int ox = (int)(code % 3u) - 1, oy = (int)((code / 3u) % 3u) - 1, oz = (int)(code / 9u) - 1;
    sx = -(float)ox * g.cellf[0];
    sy = -(float)oy * g.cellf[1];
    sz = -(float)oz * g.cellf[2];
}

__device__ __forceinline__ uint32_t cell_at(const GridGeom& g, uint32_t cx, uint32_t cy, uint32_t cz, uint32_t code) {
    int ox = (int)(code % 3u) - 1, oy = (int)((code / 3u) % 3u) - 1, oz = (int)(code / 9u) - 1;
    return encode(g, wrap_add(cx, ox, g.n[0]), wrap_add(cy, oy, g.n[1]), wrap_add(cz, oz, g.n[2]));
}

// Kick (integrate.rs:38-45, with the pending scale of thermostat.rs:68-70),
// drift (integrate.rs:62-66), wrap (boundary.rs:28-34) of one atom with the
// same exact FP64 operations as k_kick/k_drift/k_wrap; then the home-frame
// staging.  True when the atom moved too far since the last rebuild.
__device__ __forceinline__ bool nl_advance_one(const StateBuf& b, uint32_t i, const double* lambda, double half_dt,
                                               double dt, double hx, double hy, double hz, int wrap,
                                               const GridGeom& g, const uint32_t* home, float4* pos4,
                                               const float4* ref, float lim2, bool half, uint32_t* err) {
    double vx = b.vx[i], vy = b.vy[i], vz = b.vz[i];
    if (lambda) {
        double l = *lambda;
        vx = xmul(vx, l);
        vy = xmul(vy, l);
        vz = xmul(vz, l);
    }
    vx = xadd(vx, xmul(b.ax[i], half_dt));
    vy = xadd(vy, xmul(b.ay[i], half_dt));
    vz = xadd(vz, xmul(b.az[i], half_dt));
    double x = xadd(b.x[i], xmul(vx, dt)), y = xadd(b.y[i], xmul(vy, dt)), z = xadd(b.z[i], xmul(vz, dt));
    if (wrap) {
        x = xsub(rem_euclid(x, xmul(2.0, hx)), hx);
        y = xsub(rem_euclid(y, xmul(2.0, hy)), hy);
        z = xsub(rem_euclid(z, xmul(2.0, hz)), hz);
    }
    b.vx[i] = vx;
    b.vy[i] = vy;
    b.vz[i] = vz;
    b.x[i] = x;
    b.y[i] = y;
    b.z[i] = z;
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) {
        atomicOr(err, kErrNonFinite);
        return true;
    }
    const float4 p = stage_one(g, b, home[i], i, x, y, z, half);
    pos4[i] = p;
    const float4 r = ref[i];
    const float dx = p.x - r.x, dy = p.y - r.y, dz = p.z - r.z;
    return !(dx * dx + dy * dy + dz * dz <= lim2);
}

// The same lists from one warp per atom.  Lane k < 27 looks up neighbour
// cell k (skipped or out of reach: no candidates), a warp scan of the 27
// counts turns the candidates into one run t = 0 .. total - 1, and the lanes
// take it 32 at a time, each finding its candidate's cell by a binary search
// over the scan and its place in the list from the ballot: the candidates,
// the test and the order are k_nl_build's, so the lists are the same words.
// A small build is bound by the serial walk of one atom's ~150 candidates
// (one thread per atom leaves most of the chip idle), a large one by
// instructions, of which the searches and shuffles here take twice as many.
// Microseconds per build, half list, warp / thread per atom: 11 / 78 at
// 4,096 atoms, 25 / 78 at 32,768, 37 / 73 at 59,319, 72 / 83 at 125,000,
// 142 / 100 at 262,144; full list (FP64): 13 / 99, 37 / 94, 54 / 86,
// 107 / 104, 217 / 171.
template <bool HALF>
__device__ __forceinline__ void nl_build_warp_one(const GridGeom& g, const float4* pos4, const uint32_t* home,
                                                  const uint32_t* start, uint32_t p, float rl2, uint32_t* list,
                                                  size_t stride, int cap_nb, uint32_t* cnt) {
    const uint32_t lane = threadIdx.x & 31u;
    const float4 pi = pos4[p];
    const uint32_t c = home[p];
    uint32_t cx, cy, cz;
    decode(g, c, cx, cy, cz);
    float qx = pi.x, qy = pi.y, qz = pi.z;  // the atom in this lane's cell frame
    uint32_t lo = 0, len = 0;
    if (lane < 27) {
        const int ox = (int)(lane % 3u) - 1, oy = (int)((lane / 3u) % 3u) - 1, oz = (int)(lane / 9u) - 1;
        const uint32_t B = cell_at(g, cx, cy, cz, lane);
        const float slack = 1e-3f;  // as k_nl_build
        const float mx = fmaxf((ox > 0 ? g.cellf[0] - pi.x : (ox < 0 ? pi.x : 0.f)) - slack, 0.f);
        const float my = fmaxf((oy > 0 ? g.cellf[1] - pi.y : (oy < 0 ? pi.y : 0.f)) - slack, 0.f);
        const float mz = fmaxf((oz > 0 ? g.cellf[2] - pi.z : (oz < 0 ? pi.z : 0.f)) - slack, 0.f);
        if (!(HALF && B < c) && dist2(mx, my, mz) < rl2) {
            lo = HALF && B == c ? p + 1 : start[B];
            len = start[B + 1] - lo;
        }
        float sx, sy, sz;
        code_shift(g, lane, sx, sy, sz);
        qx = fadd(pi.x, sx);
        qy = fadd(pi.y, sy);
        qz = fadd(pi.z, sz);
    }
    uint32_t end = len;  // inclusive scan: the candidates of cells 0 .. lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= (uint32_t)o) end += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
    const uint32_t base = lo - (end - len);  // candidate t of this cell is atom base + t
    uint32_t m = 0;
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const uint32_t t = t0 + lane;
        uint32_t k = 0;  // the first cell whose scan exceeds t
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1)
            if (__shfl_sync(0xffffffffu, end, k + step - 1) <= t) k += step;
        const uint32_t q = __shfl_sync(0xffffffffu, base, k) + t;
        const float x = __shfl_sync(0xffffffffu, qx, k), y = __shfl_sync(0xffffffffu, qy, k),
                    z = __shfl_sync(0xffffffffu, qz, k);
        bool hit = false;
        if (t < total && (HALF || q != p)) {
            const float4 pj = pos4[q];
            hit = dist2(fsub(x, pj.x), fsub(y, pj.y), fsub(z, pj.z)) < rl2;
        }
        const uint32_t found = __ballot_sync(0xffffffffu, hit);
        const uint32_t e = m + __popc(found & ((1u << lane) - 1u));
        if (hit && e < (uint32_t)cap_nb) list[(size_t)e * stride + p] = q | (k << 27);
        m += __popc(found);
    }
    if (lane == 0) cnt[p] = m;
}

template <int BS>
__device__ __forceinline__ unsigned long long block_sum_u(unsigned long long v, unsigned long long* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = (threadIdx.x < BS / 32) ? sh[threadIdx.x] : 0ull;
    if (wid == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;
}

template <int BS>
__device__ __forceinline__ double block_sum_d(double v, double* sh) {
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

// a = F 2^-32 (1/m) (as k_fix_to_acc) and v += a dt/2 (as k_kick) of one
// atom; returns |v|^2.
__device__ __forceinline__ double nl_finish_one(const StateBuf& b, const long long* F, size_t fstride, uint32_t i,
                                                double half_dt) {
    const double im = b.inv_mass[i];
    const double ax = xmul(xmul(__ll2double_rn(F[i]), kFixInv), im);
    const double ay = xmul(xmul(__ll2double_rn(F[fstride + i]), kFixInv), im);
    const double az = xmul(xmul(__ll2double_rn(F[2 * fstride + i]), kFixInv), im);
    b.ax[i] = ax;
    b.ay[i] = ay;
    b.az[i] = az;
    const double vx = xadd(b.vx[i], xmul(ax, half_dt));
    const double vy = xadd(b.vy[i], xmul(ay, half_dt));
    const double vz = xadd(b.vz[i], xmul(az, half_dt));
    b.vx[i] = vx;
    b.vy[i] = vy;
    b.vz[i] = vz;
    return xadd(xadd(xmul(vx, vx), xmul(vy, vy)), xmul(vz, vz));
}

// The FP64 pass over one atom's full list, the reference's exact per-pair
// arithmetic: lane `sub` of `lanes` takes entries sub, sub + lanes, ... in the
// build's order, positions loaded one entry ahead.  V and the pair count take
// each unordered pair once (the later sorted position's visit).
struct Acc64 {
    double ax = 0.0, ay = 0.0, az = 0.0, V = 0.0;
    unsigned int np = 0;
};

__device__ __forceinline__ void nl_atom64(const GridGeom& g, const StateBuf& b, const uint32_t* home,
                                          const uint32_t* start, const LawF64& L, const double* psig,
                                          const double* peps, const uint32_t* list, size_t stride, int cap_nb,
                                          const uint32_t* cnt, uint32_t i, uint32_t sub, uint32_t lanes, Acc64& a) {
    const double xi = b.x[i], yi = b.y[i], zi = b.z[i];
    const int ti = b.elem[i] * kNElem;
    const double qi = b.charge[i], mi = b.mass[i], inv_mi = b.inv_mass[i];
    // the list grid has >= 3 cells per axis (min_image_near)
    const double hx = xmul(0.5, L.box[0]), hy = xmul(0.5, L.box[1]), hz = xmul(0.5, L.box[2]);
    const auto visit = [&](uint32_t j, double xj, double yj, double zj) {
        const double dx = min_image_near(xsub(xi, xj), L.box[0], hx);
        const double dy = min_image_near(xsub(yi, yj), L.box[1], hy);
        const double dz = min_image_near(xsub(zi, zj), L.box[2], hz);
        const double d2 = xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz));
        if (d2 >= L.rc2) return;
        const int tt = ti + b.elem[j];  // psig, then peps, then (24 eps) / sigma, each kNElem^2
        const double qj = b.charge[j], mj = L.grav ? b.mass[j] : 0.0;
        const double d = xsqrt(d2);
        if (d <= kEpsF64) return;
        const double inv = __drcp_rn(d);
        double fmag, Vij = 0.0;
        pair_f64_e24(L, d, inv, psig[tt], peps[tt], peps[kNElem * kNElem + tt], qi, qj, mi, mj, fmag, Vij);
        if (j > i) {
            a.V = xadd(a.V, Vij);
            ++a.np;
        }
        if (fmag != 0.0) {
            a.ax = xadd(a.ax, xmul(xmul(xmul(dx, inv), fmag), inv_mi));
            a.ay = xadd(a.ay, xmul(xmul(xmul(dy, inv), fmag), inv_mi));
            a.az = xadd(a.az, xmul(xmul(xmul(dz, inv), fmag), inv_mi));
        }
    };
    const uint32_t m = cnt[i];
    if (m <= (uint32_t)cap_nb) {
        if (sub >= m) return;
        const uint32_t* lp = list + i;
        uint32_t j = lp[(size_t)sub * stride] & kIdxMask;
        double xj = b.x[j], yj = b.y[j], zj = b.z[j];
        for (uint32_t e = sub; e < m; e += lanes) {
            const uint32_t next = e + lanes < m ? lp[(size_t)(e + lanes) * stride] & kIdxMask : j;
            const double xn = b.x[next], yn = b.y[next], zn = b.z[next];
            visit(j, xj, yj, zj);
            j = next;
            xj = xn;
            yj = yn;
            zj = zn;
        }
    } else {  // overflowed list: the lanes split each of the 27 home-grid cells
        uint32_t cx, cy, cz;
        decode(g, home[i], cx, cy, cz);
        for (uint32_t code = 0; code < 27; ++code) {
            const uint32_t B = cell_at(g, cx, cy, cz, code);
            for (uint32_t q = start[B] + sub, hi = start[B + 1]; q < hi; q += lanes)
                if (q != i) visit(q, b.x[q], b.y[q], b.z[q]);
        }
    }
}

// The lanes' sums of one atom, in a fixed association (every lane ends with
// them).
__device__ __forceinline__ void nl_sum64(Acc64& a, uint32_t lanes) {
    for (uint32_t o = lanes >> 1; o > 0; o >>= 1) {
        a.ax += __shfl_xor_sync(0xffffffffu, a.ax, o);
        a.ay += __shfl_xor_sync(0xffffffffu, a.ay, o);
        a.az += __shfl_xor_sync(0xffffffffu, a.az, o);
        a.V += __shfl_xor_sync(0xffffffffu, a.V, o);
    }
}

// Lanes per atom of the FP64 pass: enough that no lane's chain of dependent
// operations sets the pass.  Microseconds per pass with 1 / 2 / 4 / 8 / 16 / 32
// lanes: 64 / 37 / 23 / 14 / 12 / 10 at 512 atoms, 68 / 39 / 25 / 16 / 12 / 14
// at 4,096, 70 / 39 / 25 / 27 / 27 / 31 at 13,824; with 1 / 2 / 4:
// 86 / 53 / 39 at 32,768, 248 / 225 / 217 at 250,047, 876 / 805 / 811 at
// 1,000,000.
inline uint32_t nl_auto_lanes64(uint32_t n) {
    if (n <= 8192) return n <= 2048 ? 32 : 16;
    return n <= 400000 ? 4 : 2;
}

// FP64 second kick of one atom (as k_kick); returns |v|^2.
__device__ __forceinline__ double nl_finish64_one(const StateBuf& b, uint32_t i, double half_dt) {
    const double vx = xadd(b.vx[i], xmul(b.ax[i], half_dt));
    const double vy = xadd(b.vy[i], xmul(b.ay[i], half_dt));
    const double vz = xadd(b.vz[i], xmul(b.az[i], half_dt));
    b.vx[i] = vx;
    b.vy[i] = vy;
    b.vz[i] = vz;
    return xadd(xadd(xmul(vx, vx), xmul(vy, vy)), xmul(vz, vz));
}

}  // namespace gx
