// gx_pair_f32.cuh -- the mixed path's FP32 pair law, shared by its kernels.
//
// One in-cutoff pair: Lennard-Jones with the hardened core r = max(d, σ/2)
// and the quintic switch on [r_on, r_c] (force_switched_scalar, lj_raw,
// smooth_cutoff, switched: src/physics/forces.rs:270-353), plus Coulomb with
// the absolute core max(d, 0.5) and its own switch on d
// (src/systems/forces.rs:282-289), plus gravity -G m_i m_j / r^2 with the
// same core and its own switch (forces.rs:291-299, gravity_raw
// src/physics/forces.rs:338-341).  Returns the force magnitude divided by d
// (so F_vec = delta * fs) and the switched potential.
//
// Every operation is an explicit round-to-nearest intrinsic or fmaf, so the
// compiler has no contraction choices left: all pair kernels produce the same
// bits for the same pair, which keeps the fixed-point sums identical across
// kernel variants and launch shapes.
#pragma once

#include "gx_internal.cuh"

namespace gx {

struct LawF32 {
    float rc2, lj_rc, lj_ron, inv_lj_w, coul_rc, coul_ron, inv_coul_w;
    int coul, nkinds;
    int grav = 0;
    float grav_rc = 0.f, grav_ron = 0.f, inv_grav_w = 0.f;
    int one_switch = 0;   // Coulomb has LJ's cutoff and switch, the cores lie below them
    float fq_max = 0.f;  // below it, 2^32 |F| / d times any displacement within the cutoff fits a fixed-point sum
};

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }

// (pi - pj) + shift: exactly antisymmetric under swapping the pair's ends.
__device__ __forceinline__ float delta1(float a, float b, float s) { return fadd(fsub(a, b), s); }
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
    return fmaf(dz, dz, fmaf(dy, dy, fmul(dx, dx)));
}

// min(max(a * b, 0), 1) in one instruction (0 for a NaN, as fmaxf gives).
__device__ __forceinline__ float fmul_sat(float a, float b) {
    float r;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The PTX instruction flushes subnormal arguments to zero (its manual's .ftz),
// so those take rsqrtf; normal ones kept the bits of every mixed trajectory.
__device__ __forceinline__ float rsqrt_normal(float d2) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d2));
    return r;
}
__device__ __forceinline__ float rsqrt_any(float d2) {
    return d2 < 1.17549435e-38f ? rsqrtf(d2) : rsqrt_normal(d2);
}

// quintic switch 1 - 10u^3 + 15u^4 - 6u^5 and its derivative (per unit u)
__device__ __forceinline__ void switch5(float u, float& sw, float& dsw_du) {
    float u2 = fmul(u, u);
    float p = fmaf(-6.f, u, 15.f);       // 15 - 6u
    p = fmaf(p, u, -10.f);               // -10 + u(15 - 6u)
    sw = fmaf(fmul(u2, u), p, 1.f);
    float omu = fsub(1.f, u);
    dsw_du = fmul(fmul(fmul(-30.f, u2), omu), omu);
}

// The pair table in shared memory.  The list passes are bound by L1's data
// passes (80 % busy at 512,000 atoms): a scattered 16-byte gather, three
// 64-bit reductions and the table reads of each pair.  So what every pair
// takes (sigma, 4 eps, 24 eps, the charges' product) is one 16-byte word, and
// the core's 2 / sigma and the masses' product are read where a pair needs
// them (sigma / 2 is exact).  With the shifts below one bank per axis, the
// half-list pass of 2,097,152 atoms took 465 us (527 with 32-byte rows and
// 16-byte shifts), 131 at 512,000 (145), and the 256-replica batch's 290
// (300).  What bounds it since is the number of instructions (79 % issue), so
// the law below spends none twice: one switch for two terms of the same
// cutoff, one range check for a force's three components, clamps folded into
// products (436 us, 123 at 512,000).
struct PairTab {
    float4 main[kMaxKinds * kMaxKinds];
    float2 rest[kMaxKinds * kMaxKinds];
    struct Ref {
        const PairTab* t;
        int i;
    };
    __device__ __forceinline__ Ref operator[](int i) const { return Ref{this, i}; }
    __device__ __forceinline__ void put(int i, const PairF& p) {
        main[i] = make_float4(p.sigma, p.eps4, p.eps24, p.qq);
        rest[i] = make_float2(p.inv_half_sigma, p.gm);
    }
};

// Periodic shifts by neighbour-cell code, one bank per code and axis: a read
// is one pass whatever codes the lanes hold.
struct ShiftTab {
    float x[32], y[32], z[32];
    __device__ __forceinline__ float4 operator[](uint32_t c) const { return make_float4(x[c], y[c], z[c], 0.f); }
    __device__ __forceinline__ void put(uint32_t c, float sx, float sy, float sz) {
        x[c] = sx;
        y[c] = sy;
        z[c] = sz;
    }
};

__device__ __forceinline__ void pair_f32(const LawF32& L, PairTab::Ref ref, float d2, float inv_d, float& fs,
                                         float& v) {
    float d = fmul(d2, inv_d);
    float f = 0.f;
    v = 0.f;
    const float4 row = ref.t->main[ref.i];
    const float sigma = row.x, eps4 = row.y, eps24 = row.z, qq = row.w;
    if (d < L.lj_rc) {
        float r = d, inv_r = inv_d;
        if (d < fmul(0.5f, sigma)) {  // the hardened core
            r = fmul(0.5f, sigma);
            inv_r = ref.t->rest[ref.i].x;
        }
        float s = fmul(sigma, inv_r);
        float s2 = fmul(s, s);
        float s6 = fmul(fmul(s2, s2), s2);
        float s12 = fmul(s6, s6);
        float vl = fmul(eps4, fsub(s12, s6));
        float ml = fmul(fmul(eps24, inv_r), fmaf(2.f, s12, -s6));
        // u clamped to [0, 1] instead of branching: S(0) = 1 and S'(0) = -0
        // give f = fmaf(ml, 1, +-0) = ml and v = vl exactly, S(1) = 0 gives
        // zeros, so the result is bit-identical to skipping the switch
        // outside (r_on, r_c) -- and no lane of a warp diverges on it.
        float u = fmul_sat(fsub(r, L.lj_ron), L.inv_lj_w);
        float sw, dsdu;
        switch5(u, sw, dsdu);
        float dsw = fmul(dsdu, L.inv_lj_w);
        f = fmaf(ml, sw, -fmul(vl, dsw));
        v = fmul(vl, sw);
        if (L.one_switch) {  // in the core too: S(0) and S'(0) for r = sigma / 2 and for d
            float inv_c = d < 0.5f ? 2.f : inv_d;
            float vc = fmul(qq, inv_c);
            float mc = fmul(vc, inv_c);
            f = fadd(f, fmaf(mc, sw, -fmul(vc, dsw)));
            v = fadd(v, fmul(vc, sw));
        }
    }
    if (L.coul && !L.one_switch && d < L.coul_rc) {
        float inv_r = d < 0.5f ? 2.f : inv_d;
        float vc = fmul(qq, inv_r);
        float mc = fmul(vc, inv_r);
        float u = fmul_sat(fsub(d, L.coul_ron), L.inv_coul_w);  // as above
        float sw, dsdu;
        switch5(u, sw, dsdu);
        float dsw = fmul(dsdu, L.inv_coul_w);
        f = fadd(f, fmaf(mc, sw, -fmul(vc, dsw)));
        v = fadd(v, fmul(vc, sw));
    }
    if (L.grav && d < L.grav_rc) {
        float inv_r = d < 0.5f ? 2.f : inv_d;
        float vg = -fmul(ref.t->rest[ref.i].y, inv_r);  // attractive
        float mg = fmul(vg, inv_r);
        float u = fmul_sat(fsub(d, L.grav_ron), L.inv_grav_w);  // as above
        float sw, dsdu;
        switch5(u, sw, dsdu);
        float dsw = fmul(dsdu, L.inv_grav_w);
        f = fadd(f, fmaf(mg, sw, -fmul(vg, dsw)));
        v = fadd(v, fmul(vg, sw));
    }
    fs = fmul(f, inv_d);
}

__device__ __forceinline__ void pair_f32(const LawF32& L, PairTab::Ref ref, float d2, float& fs, float& v) {
    pair_f32(L, ref, d2, rsqrt_any(d2), fs, v);
}

// One FP32 value to 2^-32 fixed point; flags saturation / non-finite.
__device__ __forceinline__ long long quant(float v, uint32_t* err) {
    float s = fmul(v, kFixScaleF);
    if (!(fabsf(s) < 9.0e18f)) {
        atomicOr(err, isfinite(v) ? kErrSaturation : kErrNonFinite);
        return 0;
    }
    return __float2ll_rn(s);
}

// The three components of one pair force: quant of each, with one range
// check on the fast path (the same integers and flags as three quant calls;
// a NaN fails the check and takes the per-component path, which flags it).
__device__ __forceinline__ void quant3(float fx, float fy, float fz, long long& qx, long long& qy, long long& qz,
                                       uint32_t* err) {
    const float ux = fmul(fx, kFixScaleF), uy = fmul(fy, kFixScaleF), uz = fmul(fz, kFixScaleF);
    if (fabsf(ux) < 9.0e18f && fabsf(uy) < 9.0e18f && fabsf(uz) < 9.0e18f) {
        qx = __float2ll_rn(ux);
        qy = __float2ll_rn(uy);
        qz = __float2ll_rn(uz);
    } else {
        qx = quant(fx, err);
        qy = quant(fy, err);
        qz = quant(fz, err);
    }
}

LawF32 make_law32(const gx_handle* h);

// Thread-per-atom pair pass with per-thread candidate lists (gx_force_tiled.cu);
// any grid, atom indices below 2^27.
void launch_force_mixed_lists(gx_handle* h, const GridGeom& g, const float4* pos4, const uint32_t* key,
                              const uint32_t* start, uint32_t n, const LawF32& L, const PairF* tab, long long* F,
                              size_t fstride, unsigned long long* vacc, unsigned long long* npairs, uint32_t* err);

// Tiled mixed pair pass (gx_force_tiled.cu); needs >= 3 cells on every axis.
void launch_force_mixed_tiled(gx_handle* h, const GridGeom& g, const float4* pos4, const uint32_t* start,
                              const LawF32& L, const PairF* tab, long long* F, size_t fstride,
                              unsigned long long* vacc, unsigned long long* npairs, uint32_t* err);

// One list entry's pair for the list passes: the law only inside r_c, the
// quantised force summed into `a`, with `far` also subtracted from the far
// end q (half lists), and with `once` the potential and pair count.
struct PairAcc {
    long long fx = 0, fy = 0, fz = 0, vq = 0;
    unsigned int np = 0;  // in-cutoff pairs of one thread (widened when summed)
};

// far != null: also subtract the pair force from the far end q (HALF lists).
__device__ __forceinline__ void nl_pair(const LawF32& L, const PairTab& st, int ki, float4 pi, float4 pj, float sx,
                                        float sy, float sz, bool once, PairAcc& a, uint32_t* err,
                                        long long* far = nullptr, uint32_t q = 0, size_t fstride = 0) {
    float dx = delta1(pi.x, pj.x, sx), dy = delta1(pi.y, pj.y, sy), dz = delta1(pi.z, pj.z, sz);
    float d2 = dist2(dx, dy, dz);
    if (!(d2 < L.rc2)) return;
    float inv_d;
    if (d2 >= 1.17549435e-38f) {
        inv_d = rsqrt_normal(d2);
    } else {
        if (d2 == 0.f) return;
        inv_d = rsqrtf(d2);
    }
    float fs, v;
    pair_f32(L, st[ki * L.nkinds + __float_as_int(pj.w)], d2, inv_d, fs, v);
    // The force quantised with 2^32 folded into its magnitude (a power of two:
    // the same integers) and one range check for the three components; what
    // fails it takes quant3's checks of each.  The far end's share is
    // quantised: the conversion rounds to nearest even, symmetric in sign, so
    // this end's is exactly its negative.
    const float fq = fmul(fs, -kFixScaleF);
    long long qx, qy, qz;
    if (fabsf(fq) < L.fq_max) {
        qx = __float2ll_rn(fmul(dx, fq));
        qy = __float2ll_rn(fmul(dy, fq));
        qz = __float2ll_rn(fmul(dz, fq));
    } else {
        quant3(-fmul(dx, fs), -fmul(dy, fs), -fmul(dz, fs), qx, qy, qz, err);
    }
    a.fx -= qx;
    a.fy -= qy;
    a.fz -= qz;
    if (far) {
        atomicAdd((unsigned long long*)&far[q], (unsigned long long)qx);
        atomicAdd((unsigned long long*)&far[fstride + q], (unsigned long long)qy);
        atomicAdd((unsigned long long*)&far[2 * fstride + q], (unsigned long long)qz);
    }
    if (once) {
        a.vq += quant(v, err);
        ++a.np;
    }
}

}  // namespace gx
