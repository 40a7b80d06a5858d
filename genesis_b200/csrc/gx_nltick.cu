// gx_nltick.cu -- the neighbour-list ticks of a small universe in one launch.
//
// A tick of gx_nlist.cu is ten launches and a conditional node.  Up to tens
// of thousands of atoms each of them lasts one to ten microseconds, most of it
// launch and drain, so the gaps set the tick.  Here one cooperative launch
// runs every tick of a step call: the blocks of the grid are all resident
// (cudaLaunchCooperativeKernel), each phase strides over the atoms with the
// device functions of gx_nlist.cuh, and a grid barrier separates the phases:
//
//   advance          kick, drift, wrap, staging, displacement test
//   -- barrier --    the rebuild request is final
//   [rebuild]        keys and counts, scan, scatter, rank and gather, copy
//                    back and staging, lists by one warp per atom (six
//                    barriers), only on the ticks that ask for it
//   pair pass        8 .. 32 lanes per atom over its half list (FP64: 4 .. 32
//                    over its full list), and the observed-bond spring
//   -- barrier --    the force sums are final
//   finish           a = F 2^-32 / m, kick, kinetic-energy partials
//   -- barrier --    with the thermostat: every block sums the partials and
//                    takes the same scale
//
// The sums are the per-kernel tick's: integers for the forces, and for K and
// the speed sum 256-atom blocks combined in k_thermostat_lambda's order, so
// the trajectory is the same bits (tested).  An atom is advanced and finished
// by the same thread, so no barrier is needed between a tick's end and the
// next one's start.  A record is taken by one block while the next tick runs,
// from partials and counters kept per tick parity.
//
// A phase is bound by the latency of its few dependent accesses and the
// barrier, not by bytes or operations.  Microseconds per recorded NVE tick,
// rebuilds included, here / as a graph of kernels: 16 / 32 at 512 atoms,
// 19 / 33 at 4,096, 25 / 40 at 13,824, 41 / 48 at 32,768, 54 / 63 at 59,319;
// from about 1.7 M list entries the kernels win (73 / 73 at 2.6 M, 98 / 93 at
// 3.4 M, 202 / 143 at 7.1 M): their pair pass keeps more warps resident than
// the one kernel that holds every phase.  Four blocks per SM (64 registers):
// 54 us at 59,319 atoms, against 55 with three and 57 with five.  FP64, here /
// as kernels: 21 / 36 at 512 atoms, 26 / 43 at 4,096, 46 / 62 at 13,824, 78 /
// 74 at 32,768.
#include <algorithm>

#include "gx_gridsync.cuh"
#include "gx_law64.cuh"
#include "gx_nlist.cuh"

namespace gx {
namespace {

constexpr int kTickThreads = 256;           // as k_nl_finish's blocks: one partial per 256 atoms
constexpr uint32_t kPartRow = 2048;         // partials per parity (reduction rows hold at least 4,096)

struct TickArgs {
    StateBuf b, o;  // the live state, and the buffer a rebuild sorts into
    GridGeom g;
    uint32_t n, lanes_log2;
    LawF32 L;
    LawF64 L64;
    const PairF* tab;
    const double *psig, *peps;
    uint32_t *key, *home, *pos_of_slot;
    float4 *pos4, *ref;
    uint32_t *count, *start, *fill, *tmp;
    uint32_t* list;
    size_t stride;
    int cap_nb;
    uint32_t* cnt;
    long long* F;
    size_t fstride;
    double *kpart, *spart, *vpart, *dscal;
    uint32_t* flag;
    uint32_t* err;
    TickSync* sync;
    gx_tick_stats* rec;
    const uint32_t* bonds;
    const unsigned long long* nbonds;
    size_t bonds_cap;
    double k_bind, r_eq_factor, curv_factor;
    double half_dt, dt, hx, hy, hz;
    double k_thermal, target, tau;
    float lim2, rl2;
    int wrap, thermo, nticks;
    uint32_t polls;  // of a barrier before it gives up
};

// Sum of part[0 .. nb) in k_thermostat_lambda's order (valid in thread 0).
__device__ __forceinline__ double part_sum(const double* part, int nb, double* sh) {
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += kTickThreads) s = xadd(s, part[i]);
    return block_sum_d<kTickThreads>(s, sh);
}

// The record of one finished tick, by one block: K and the speed sum from its
// partials, the potential, bond energy and pair count from its counters.
template <bool F64>
__device__ __forceinline__ void take_record(const TickArgs& a, int tick, double lam, int nb, double* sh) {
    const int par = tick & 1;
    const double K = part_sum(a.kpart + par * kPartRow, nb, sh);
    const double S = part_sum(a.spart + par * kPartRow, nb, sh);
    const double V64 = F64 ? part_sum(a.vpart + par * kPartRow, nb, sh) : 0.0;
    if (threadIdx.x != 0) return;
    const unsigned long long* c = a.sync->acc[par];
    const double V = F64 ? V64 : xmul(__ll2double_rn((long long)c[0]), kFixInv);
    const double Vb = xmul(__ll2double_rn((long long)c[2]), kFixInv);
    gx_tick_stats& r = a.rec[tick];
    r.kinetic = a.thermo ? xmul(xmul(K, lam), lam) : K;
    r.speed_sum = a.thermo ? xmul(S, lam) : S;
    r.potential = V;
    r.bond_energy = Vb;
    r.lambda = a.thermo ? lam : 1.0;
    r.pairs = c[1];
    a.dscal[1] = K;
    a.dscal[2] = V;
    a.dscal[3] = Vb;
    a.dscal[4] = S;
}

// F64: the plain FP64 tick over the full list (nl_atom64); the atoms'
// potentials lie in the room of the fixed-point sums until the finish.
template <bool REC, bool F64>
__global__ void __launch_bounds__(kTickThreads, F64 ? 3 : 4) k_nl_ticks(const __grid_constant__ TickArgs a) {
    __shared__ PairTab st;
    __shared__ ShiftTab s_shift;
    __shared__ double sh[kTickThreads / 32];
    __shared__ unsigned long long shu[kTickThreads / 32];
    __shared__ uint32_t s_warp[kTickThreads / 32], s_off[kScanMaxTiles];
    __shared__ double s_lam;
    __shared__ int s_ok;
    const uint32_t tid = threadIdx.x, n = a.n;
    const uint32_t gt = blockIdx.x * kTickThreads + tid, gs = gridDim.x * kTickThreads;
    const uint32_t m = a.g.ncell + 1, ntiles = (m + kScanTileCells - 1) / kScanTileCells;
    const int nb = (int)((n + kTickThreads - 1) / kTickThreads);
    const bool recorder = blockIdx.x == gridDim.x - 1;
    uint32_t target = 0;  // thread 0's count of barrier arrivals
    if (*a.err & kErrBarrier) return;  // the launch before this one gave up
    const int nk2 = F64 ? 0 : a.L.nkinds * a.L.nkinds;
    double* vat = reinterpret_cast<double*>(a.F);
    for (int t = tid; t < nk2; t += kTickThreads) st.put(t, a.tab[t]);
    if (tid < 27) {
        float sx, sy, sz;
        code_shift(a.g, tid, sx, sy, sz);
        s_shift.put(tid, sx, sy, sz);
    }
    for (uint32_t c = gt; c < m; c += gs) a.count[c] = a.fill[c] = 0u;  // counted into before the next use
    if (recorder && tid < 4) a.sync->acc[0][tid] = 0ull;
    if (tid == 0) s_lam = a.dscal[0];  // 1 unless a scale is pending
    uint32_t parity = a.flag[2], rebuilds = 0;
    const bool asked = a.flag[0] != 0u;
    __syncthreads();
    for (int tick = 0; tick < a.nticks; ++tick) {
        const int par = tick & 1;
        const bool half = ((parity + (a.wrap ? 1u : 0u)) & 1u) != 0u;
        bool over = false;
        for (uint32_t i = gt; i < n; i += gs) {
            if (!F64) {
                a.F[i] = 0;
                a.F[a.fstride + i] = 0;
                a.F[2 * a.fstride + i] = 0;
            }
            over |= nl_advance_one(a.b, i, &s_lam, a.half_dt, a.dt, a.hx, a.hy, a.hz, a.wrap, a.g, a.home, a.pos4,
                                   a.ref, a.lim2, half, a.err);
        }
        if (__syncthreads_or(over) && tid == 0) a.sync->grid.request[par] = 1u;
        if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
        const bool rebuild = (tick == 0 && asked) || *(volatile uint32_t*)&a.sync->grid.request[par] != 0u;
        if (recorder) {  // the other parity's words: every block has left that tick's pair pass
            if (REC && tick > 0) take_record<F64>(a, tick - 1, s_lam, nb, sh);
            __syncthreads();
            if (tid < 4) a.sync->acc[par ^ 1][tid] = 0ull;
            if (tid == 4) a.sync->grid.request[par ^ 1] = 0u;
        }
        if (!a.thermo && tid == 0) s_lam = 1.0;
        if (rebuild) {
            for (uint32_t i = gt; i < n; i += gs) {
                const uint32_t c = cell_of(a.g, a.b.x[i], a.b.y[i], a.b.z[i]);
                a.key[i] = c;
                atomicAdd(&a.count[c], 1u);
            }
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
                const uint32_t total = scan_tile<kTickThreads>(a.count, t, m, 0u, s_warp);
                if (tid == 0) a.sync->grid.tile[t] = total;
            }
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            if (tid < ntiles) {  // tile offsets, in every block
                uint32_t run = 0;
                for (uint32_t t = 0; t < tid; ++t) run += a.sync->grid.tile[t];
                s_off[tid] = run;
            }
            __syncthreads();
            for (uint32_t c = gt; c < m; c += gs) a.start[c] = a.count[c] + s_off[c / kScanTileCells];
            for (uint32_t i = gt; i < n; i += gs) {
                const uint32_t c = a.key[i];
                a.tmp[a.count[c] + s_off[c / kScanTileCells] + atomicAdd(&a.fill[c], 1u)] = i;
            }
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            for (uint32_t i = gt; i < n; i += gs) {  // as k_rank_gather: ascending source order within a cell
                const uint32_t c = a.key[i], lo = a.start[c], hi = a.start[c + 1];
                uint32_t p = lo;
                for (uint32_t q = lo; q < hi; ++q) p += a.tmp[q] < i ? 1u : 0u;
                a.o.x[p] = a.b.x[i];
                a.o.y[p] = a.b.y[i];
                a.o.z[p] = a.b.z[i];
                a.o.vx[p] = a.b.vx[i];
                a.o.vy[p] = a.b.vy[i];
                a.o.vz[p] = a.b.vz[i];
                a.o.ax[p] = a.b.ax[i];
                a.o.ay[p] = a.b.ay[i];
                a.o.az[p] = a.b.az[i];
                a.o.charge[p] = a.b.charge[i];
                a.o.mass[p] = a.b.mass[i];
                a.o.inv_mass[p] = a.b.inv_mass[i];
                a.o.elem[p] = a.b.elem[i];
                a.o.kind[p] = a.b.kind[i];
                const uint32_t s = a.b.slot[i];
                a.o.slot[p] = s;
                a.home[p] = c;
                a.pos_of_slot[s] = p;
            }
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            for (uint32_t p = gt; p < n; p += gs) {
                const double x = a.o.x[p], y = a.o.y[p], z = a.o.z[p];
                a.b.x[p] = x;
                a.b.y[p] = y;
                a.b.z[p] = z;
                a.b.vx[p] = a.o.vx[p];
                a.b.vy[p] = a.o.vy[p];
                a.b.vz[p] = a.o.vz[p];
                a.b.ax[p] = a.o.ax[p];
                a.b.ay[p] = a.o.ay[p];
                a.b.az[p] = a.o.az[p];
                a.b.charge[p] = a.o.charge[p];
                a.b.mass[p] = a.o.mass[p];
                a.b.inv_mass[p] = a.o.inv_mass[p];
                a.b.elem[p] = a.o.elem[p];
                a.b.kind[p] = a.o.kind[p];
                a.b.slot[p] = a.o.slot[p];
                const float4 f = stage_one(a.g, a.o, a.home[p], p, x, y, z, false);
                a.pos4[p] = f;
                a.ref[p] = f;
            }
            for (uint32_t c = gt; c < m; c += gs) a.count[c] = a.fill[c] = 0u;
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            for (uint32_t p = gt / 32u; p < n; p += gs / 32u)
                nl_build_warp_one<!F64>(a.g, a.pos4, a.home, a.start, p, a.rl2, a.list, a.stride, a.cap_nb, a.cnt);
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            parity = 0u;
            ++rebuilds;
        } else if (a.wrap) {
            parity ^= 1u;
        }
        if (F64) {  // pair pass: k_nl_force64
            const uint32_t lanes = 1u << a.lanes_log2, sub = tid & (lanes - 1u);
            const uint32_t end = ((n << a.lanes_log2) + 31u) & ~31u;  // whole warps
            unsigned int np = 0;
            for (uint32_t t = gt; t < end; t += gs) {
                const uint32_t i = t >> a.lanes_log2;
                Acc64 f;
                if (i < n)
                    nl_atom64(a.g, a.b, a.home, a.start, a.L64, a.psig, a.peps, a.list, a.stride, a.cap_nb, a.cnt, i,
                              sub, lanes, f);
                nl_sum64(f, lanes);
                if (i < n && sub == 0) {
                    a.b.ax[i] = f.ax;
                    a.b.ay[i] = f.ay;
                    a.b.az[i] = f.az;
                    vat[i] = f.V;
                }
                np += f.np;
            }
            if (REC) {
                const unsigned long long c = block_sum_u<kTickThreads>(np, shu);
                if (tid == 0 && c) atomicAdd(&a.sync->acc[par][1], c);
            }
        } else {  // pair pass: k_nl_force_tpp's loop
            const uint32_t lanes = 1u << a.lanes_log2, sub = tid & (lanes - 1u);
            const uint32_t end = ((n << a.lanes_log2) + 31u) & ~31u;  // whole warps
            long long vq = 0;
            unsigned int np = 0;
            for (uint32_t t = gt; t < end; t += gs) {
                const uint32_t p = t >> a.lanes_log2;
                PairAcc f;
                if (p < n) {
                    const float4 pi = a.pos4[p];
                    const int ki = __float_as_int(pi.w);
                    const uint32_t mc = a.cnt[p];
                    if (mc <= (uint32_t)a.cap_nb) {
                        const uint32_t* lp = a.list + p;
                        uint32_t e = sub;
                        for (; e + lanes < mc; e += 2u * lanes) {  // two entries per round, loads first
                            const uint32_t w0 = lp[(size_t)e * a.stride], w1 = lp[(size_t)(e + lanes) * a.stride];
                            const uint32_t q0 = w0 & kIdxMask, q1 = w1 & kIdxMask;
                            const float4 p0 = a.pos4[q0], p1 = a.pos4[q1];
                            const float4 s0 = s_shift[w0 >> 27], s1 = s_shift[w1 >> 27];
                            nl_pair(a.L, st, ki, pi, p0, s0.x, s0.y, s0.z, REC, f, a.err, a.F, q0, a.fstride);
                            nl_pair(a.L, st, ki, pi, p1, s1.x, s1.y, s1.z, REC, f, a.err, a.F, q1, a.fstride);
                        }
                        if (e < mc) {
                            const uint32_t w = lp[(size_t)e * a.stride], q = w & kIdxMask;
                            const float4 s0 = s_shift[w >> 27];
                            nl_pair(a.L, st, ki, pi, a.pos4[q], s0.x, s0.y, s0.z, REC, f, a.err, a.F, q, a.fstride);
                        }
                    } else {  // overflowed list: the group splits each of the 27 home-grid cells
                        const uint32_t c = a.home[p];
                        uint32_t cx, cy, cz;
                        decode(a.g, c, cx, cy, cz);
                        for (uint32_t code = 0; code < 27; ++code) {
                            const uint32_t B = cell_at(a.g, cx, cy, cz, code);
                            if (B < c) continue;
                            const float4 s0 = s_shift[code];
                            for (uint32_t q = a.start[B] + sub, hi = a.start[B + 1]; q < hi; q += lanes)
                                if (q > p)
                                    nl_pair(a.L, st, ki, pi, a.pos4[q], s0.x, s0.y, s0.z, REC, f, a.err, a.F, q,
                                            a.fstride);
                        }
                    }
                }
                for (uint32_t o = lanes >> 1; o > 0; o >>= 1) {  // stays within the atom's lanes
                    f.fx += __shfl_xor_sync(0xffffffffu, f.fx, o);
                    f.fy += __shfl_xor_sync(0xffffffffu, f.fy, o);
                    f.fz += __shfl_xor_sync(0xffffffffu, f.fz, o);
                }
                if (p < n && sub == 0) {
                    atomicAdd((unsigned long long*)&a.F[p], (unsigned long long)f.fx);
                    atomicAdd((unsigned long long*)&a.F[a.fstride + p], (unsigned long long)f.fy);
                    atomicAdd((unsigned long long*)&a.F[2 * a.fstride + p], (unsigned long long)f.fz);
                }
                vq += f.vq;
                np += f.np;
            }
            if (a.bonds) {  // the observed-bond spring (k_bonds), every pair within the cutoff once
                const size_t bonds = min((size_t)*a.nbonds, a.bonds_cap);
                long long vb = 0;
                for (size_t t = gt; t < bonds; t += gs) {
                    const uint32_t ia = a.pos_of_slot[a.bonds[2 * t]], ib = a.pos_of_slot[a.bonds[2 * t + 1]];
                    double nx, ny, nz, fm, vv;
                    if (!bond_f64(a.L64, a.b, ia, ib, a.psig, a.peps, a.k_bind, a.r_eq_factor, a.curv_factor, nx, ny,
                                  nz, fm, vv))
                        continue;
                    vb += __double2ll_rn(xmul(vv, kFixScale));
                    if (fm != 0.0) bond_to_fixed(a.F, a.fstride, ia, ib, nx, ny, nz, fm);
                }
                if (REC && vb) atomicAdd(&a.sync->acc[par][2], (unsigned long long)vb);
            }
            if (REC) {
                const unsigned long long s = block_sum_u<kTickThreads>((unsigned long long)vq, shu);
                const unsigned long long c = block_sum_u<kTickThreads>(np, shu);
                if (tid == 0) {
                    if (s) atomicAdd(&a.sync->acc[par][0], s);
                    if (c) atomicAdd(&a.sync->acc[par][1], c);
                }
            }
        }
        if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
        for (uint32_t v = blockIdx.x; v < (uint32_t)nb; v += gridDim.x) {
            const uint32_t i = v * kTickThreads + tid;  // the thread that advances atom i
            double ks = 0.0, ss = 0.0, vs = 0.0;
            if (i < n) {
                const double l2 = F64 ? nl_finish64_one(a.b, i, a.half_dt)
                                      : nl_finish_one(a.b, a.F, a.fstride, i, a.half_dt);
                ks = xadd(0.0, xmul(xmul(0.5, a.b.mass[i]), l2));
                if (REC) ss = xadd(0.0, xsqrt(l2));
                if (REC && F64) vs = xadd(0.0, vat[i]);
            }
            if (REC || a.thermo) {
                ks = block_sum_d<kTickThreads>(ks, sh);
                if (tid == 0) a.kpart[par * kPartRow + v] = ks;
            }
            if (REC) {
                ss = block_sum_d<kTickThreads>(ss, sh);
                if (tid == 0) a.spart[par * kPartRow + v] = ss;
            }
            if (REC && F64) {
                vs = block_sum_d<kTickThreads>(vs, sh);
                if (tid == 0) a.vpart[par * kPartRow + v] = vs;
            }
        }
        if (a.thermo) {
            if (!grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;
            const double K = part_sum(a.kpart + par * kPartRow, nb, sh);
            if (tid == 0) s_lam = berendsen_scale(K, n, a.k_thermal, a.target, a.tau);
            __syncthreads();
        }
    }
    if (REC && !a.thermo && !grid_barrier(&a.sync->grid, a.err, a.polls, target, &s_ok)) return;  // the last partials
    if (recorder) {
        if (REC) take_record<F64>(a, a.nticks - 1, s_lam, nb, sh);
        if (tid == 0) {
            a.dscal[0] = a.thermo ? s_lam : 1.0;
            a.flag[0] = 0u;
            a.flag[1] += rebuilds;
            a.flag[2] = parity;
        }
    }
    grid_leave(&a.sync->grid);
}

// Lanes per atom of the pair pass: as many as keep the chip filled, since a
// phase is bound by one atom's chain of gathers.  Microseconds per recorded
// NVE tick at 32 / 16 / 8 / 4 lanes: 16.3 / 17.9 / 20.9 / 30.4 at 512 atoms,
// 22.0 / 20.1 / 22.1 / 31.7 at 4,096, 30.3 / 26.1 / 25.5 / 33.4 at 13,824,
// 49.7 / 42.0 / 42.9 / 52.4 at 32,768 and - / 59.5 / 56.1 / 63.0 at 59,319.
inline uint32_t tick_lanes(uint32_t n) { return n <= 2048 ? 32 : (n <= 8192 ? 16 : 8); }
// The FP64 pass keeps the per-kernel tick's lanes: its sums depend on them.
inline uint32_t tick_lanes64(uint32_t n) { return nl_auto_lanes64(n); }

}  // namespace

// One launch covers the plain half-list tick (variant 6, which the automatic
// one is here): no work shape set, no collision pass, no per-launch timing,
// and a size at which the launches and not the work set the tick.
bool nl_ticks_eligible(gx_handle* h) {
    const bool mixed = h->precision == GX_MIXED;
    if (h->n == 0 || h->n > (mixed ? kTickMaxAtoms : kTickMaxAtoms64)) return false;
    if (mixed ? h->kernel_variant != 0 && h->kernel_variant != 6 : bonds_on(h)) return false;  // the FP64 spring adds to finished accelerations
    if (h->p.enable_collisions || h->prof_on || h->pass_timing) return false;
    const NlState* s = static_cast<const NlState*>(h->nl);
    if (!s || (mixed && 0.5 * s->expect * (double)h->n > kTickMaxEntries)) return false;
    return s->tpp == 0 && s->block == 0 && s->half == (mixed ? 1 : 0) && s->lg.ncell < kScanTileCells * kScanMaxTiles;
}

// nticks ticks with the records (may be null) at rec[0 .. nticks).
int nl_ticks(gx_handle* h, int nticks, gx_tick_stats* rec, bool thermo, double tau, double* kpart, double* spart) {
    NlState* s = static_cast<NlState*>(h->nl);
    const uint32_t n = (uint32_t)h->n;
    if (!s->tick_sync) {
        GX_CUDA(h, cudaMalloc(&s->tick_sync, sizeof(TickSync)));
        s->tick_sync_dirty = true;
    }
    if (s->tick_sync_dirty) {
        GX_CUDA(h, cudaMemsetAsync(s->tick_sync, 0, sizeof(TickSync), h->stream));
        s->tick_sync_dirty = false;
    }
    const bool f64 = h->precision != GX_MIXED;
    auto kern = f64 ? (rec ? k_nl_ticks<true, true> : k_nl_ticks<false, true>)
                    : (rec ? k_nl_ticks<true, false> : k_nl_ticks<false, false>);
    int& resident = s->tick_blocks[(f64 ? 2 : 0) + (rec ? 1 : 0)];
    if (!resident) {
        int per = 0, sms = 0;
        GX_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kTickThreads, 0));
        GX_CUDA(h, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->p.device));
        resident = std::max(per * sms, 1);
    }
    TickArgs a{};
    a.b = h->buf[h->cur];
    a.o = h->buf[h->cur ^ 1];
    a.g = s->lg;
    a.n = n;
    const uint32_t lanes = f64 ? tick_lanes64(n) : tick_lanes(n);
    uint32_t log2 = 0;
    while ((1u << log2) < lanes) ++log2;
    a.lanes_log2 = log2;
    if (!f64) a.L = make_law32(h);
    a.L64 = make_law64(h);
    a.tab = h->d_pairf;
    a.psig = d_psig(h);
    a.peps = a.psig + kNElem * kNElem;
    a.key = h->key;
    a.home = h->key_sorted;
    a.pos_of_slot = h->pos_of_slot;
    a.pos4 = h->pos4;
    a.ref = s->ref;
    a.count = s->cl.count;
    a.start = s->cl.start;
    a.fill = s->cl.fill;
    a.tmp = s->cl.tmp;
    a.list = s->list;
    a.stride = s->cap;
    a.cap_nb = s->cap_nb;
    a.cnt = s->cnt;
    a.F = h->F;
    a.fstride = h->cap;
    a.kpart = kpart;
    a.spart = spart;
    a.vpart = h->red;  // row 0 of the block partials
    a.dscal = h->dscal;
    a.flag = s->flag;
    a.err = h->derr;
    a.sync = s->tick_sync;
    if (bonds_on(h)) {
        a.bonds = h->bonds;
        a.nbonds = dnbonds(h);
        a.bonds_cap = h->bonds_cap;
        a.k_bind = h->fs.bond_k_bind;
        a.r_eq_factor = h->fs.r_eq_factor;
        a.curv_factor = h->fs.curv_factor;
    }
    a.half_dt = 0.5 * h->p.dt;
    a.dt = h->p.dt;
    a.hx = 0.5 * h->p.box[0];
    a.hy = 0.5 * h->p.box[1];
    a.hz = 0.5 * h->p.box[2];
    a.k_thermal = h->p.thermal_constant;
    a.target = h->p.thermostat_temperature;
    a.tau = tau;
    const float lim = (float)(0.5 * s->skin_used * (1.0 - 1e-4));
    const float rl = (float)((h->fs.rc + s->skin_used) * (1.0 + 1e-6));
    a.lim2 = lim * lim;
    a.rl2 = rl * rl;
    a.wrap = h->p.enable_boundaries ? 1 : 0;
    a.thermo = thermo ? 1 : 0;
    a.polls = h->wait_polls;
    const size_t blocks = ((size_t)n * lanes + kTickThreads - 1) / kTickThreads;
    const unsigned grid = (unsigned)std::min<size_t>(blocks, (size_t)resident);
    for (int done = 0; done < nticks; done += kTicksPerLaunch) {
        a.nticks = std::min(nticks - done, kTicksPerLaunch);
        a.rec = rec ? rec + done : nullptr;
        void* args[] = {&a};
        GX_CUDA(h, cudaLaunchCooperativeKernel((const void*)kern, grid, kTickThreads, args, 0, h->stream));
        ++h->launches;
    }
    h->lambda_pending = thermo;
    return GX_OK;
}

}  // namespace gx
