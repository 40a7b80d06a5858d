// gx_law64.cuh -- the FP64 pair law shared by the plain force pass and the
// adjoint's forward recomputation (src/physics/forces.rs:270-353,
// src/systems/forces.rs:270-299), evaluated with the reference's operation
// order so every pair's force and energy are bit-identical to it.
#pragma once

#include "gx_internal.cuh"

namespace gx {

struct LawF64 {
    double lj_rc, lj_ron, coul_rc, coul_ron, grav_rc, grav_ron;
    double rc2;
    double k_e, G;
    double box[3];
    int coul, grav;
    double lj_iw, coul_iw, grav_iw;  // 1 / (rc - r_on), correctly rounded
    int one_switch;                  // LJ and Coulomb have the same switch
};

// a / b, correctly rounded, from y = 1 / b correctly rounded (Markstein, IBM
// J. Res. Dev. 34 (1990) 111): a y lies within two units of the last place,
// one remainder step makes it faithful and a second one exact.  Quotients
// near the ends of the range, zeros and non-finite ones take the division.
// Five operations where a division takes over twenty; the reciprocal of a
// distance or of a switch's width serves several quotients.
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q0 = xmul(a, y);
    if (!(fabs(q0) > 0x1p-900 && fabs(q0) < 0x1p900)) return xdiv(a, b);
    const double q1 = fma(fma(-b, q0, a), y, q0);
    return fma(fma(-b, q1, a), y, q1);
}

// smooth_cutoff, src/physics/forces.rs:302-318 (exact FP64).
// iw = 1 / (rc - ron), correctly rounded.
__device__ __forceinline__ void smooth_f64(double r, double ron, double rc, double iw, double& sw, double& dsw) {
    if (r <= ron) { sw = 1.0; dsw = 0.0; return; }
    if (r >= rc) { sw = 0.0; dsw = 0.0; return; }
    double w = xsub(rc, ron);
    double u = div_by(xsub(r, ron), w, iw);
    double u2 = xmul(u, u);
    double u3 = xmul(u2, u);
    double u4 = xmul(u3, u);
    double u5 = xmul(u4, u);
    sw = xsub(xadd(xsub(1.0, xmul(10.0, u3)), xmul(15.0, u4)), xmul(6.0, u5));
    double omu = xsub(1.0, u);
    dsw = div_by(xmul(xmul(xmul(-30.0, u2), omu), omu), w, iw);
}

// One pair's LJ + Coulomb + gravity scalar (systems/forces.rs:270-299), exact.
// inv = 1 / d correctly rounded.  e24s = (24 ep) / sg, which depends on the
// element pair only: it comes from a table computed with the same two IEEE
// operations.  A term of no strength adds a zero and is left out.
__device__ __forceinline__ void pair_f64_e24(const LawF64& L, double d, double inv, double sg, double ep, double e24s,
                                             double qa, double qb, double ma, double mb, double& fmag, double& V) {
    fmag = 0.0;
    double sw = 0.0, dsw = 0.0;
    const double half = xmul(0.5, sg);
    if (d < L.lj_rc) {  // force_switched_scalar, forces.rs:270-275; lj_raw :346-353
        const double r = fmax(d, half);
        const double s = d >= half ? div_by(sg, d, inv) : xdiv(sg, r);
        const double s6 = xmul(xmul(xmul(xmul(xmul(s, s), s), s), s), s);
        const double s12 = xmul(s6, s6);
        const double v = xmul(xmul(4.0, ep), xsub(s12, s6));
        const double m = xmul(xmul(e24s, s), xsub(xmul(2.0, s12), s6));
        smooth_f64(r, L.lj_ron, L.lj_rc, L.lj_iw, sw, dsw);
        fmag = xadd(fmag, xsub(xmul(m, sw), xmul(v, dsw)));
        V = xadd(V, xmul(v, sw));
    }
    const auto central = [&](double q) {  // coulomb_raw :330-333, gravity_raw :338-341
        const double r = fmax(d, 0.5);
        const double m = xdiv(q, xmul(r, r));
        const double v = d >= 0.5 ? div_by(q, d, inv) : xdiv(q, r);
        fmag = xadd(fmag, xsub(xmul(m, sw), xmul(v, dsw)));
        V = xadd(V, xmul(v, sw));
    };
    if (L.coul && d < L.coul_rc) {  // :282-289
        const double q = xmul(xmul(L.k_e, qa), qb);
        if (q != 0.0) {
            if (!(L.one_switch && d >= half)) smooth_f64(d, L.coul_ron, L.coul_rc, L.coul_iw, sw, dsw);
            central(q);
        }
    }
    if (L.grav && d < L.grav_rc) {  // :292-299
        const double mm = xmul(xmul(L.G, ma), mb);
        if (mm != 0.0) {
            smooth_f64(d, L.grav_ron, L.grav_rc, L.grav_iw, sw, dsw);
            central(-mm);
        }
    }
}

// One observed bond's spring (src/systems/forces.rs:305-317,
// bond_harmonic_raw forces.rs:290-293), exact: the unit normal, the force
// magnitude and the energy.  False when the pair is out of the spring's reach.
__device__ __forceinline__ bool bond_f64(const LawF64& L, const StateBuf& b, uint32_t ia, uint32_t ib,
                                         const double* psig, const double* peps, double k_bind, double r_eq_factor,
                                         double curv_factor, double& nx, double& ny, double& nz, double& fm,
                                         double& vv) {
    const double dx = min_image1(xsub(b.x[ia], b.x[ib]), L.box[0]);
    const double dy = min_image1(xsub(b.y[ia], b.y[ib]), L.box[1]);
    const double dz = min_image1(xsub(b.z[ia], b.z[ib]), L.box[2]);
    const double d2 = xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz));
    const double d = xsqrt(d2);
    if (!(d2 < L.rc2 && d > kEpsF64)) return false;
    const int ta = b.elem[ia], tb = b.elem[ib];
    const double sg = psig[ta * kNElem + tb], ep = peps[ta * kNElem + tb];
    const double r_eq = xmul(sg, r_eq_factor);
    const double rc_bond = xmul(k_bind, sg);
    if (!(d < rc_bond)) return false;
    const double kk = xdiv(xmul(curv_factor, ep), xmul(sg, sg));
    const double dr = xsub(d, r_eq);
    const double m = xmul(-kk, dr);
    const double v = xmul(xmul(xmul(0.5, kk), dr), dr);
    double sw, dsw;
    smooth_f64(d, r_eq, rc_bond, __drcp_rn(xsub(rc_bond, r_eq)), sw, dsw);
    fm = xsub(xmul(m, sw), xmul(v, dsw));
    vv = xmul(v, sw);
    const double inv = xdiv(1.0, d);
    nx = xmul(dx, inv);
    ny = xmul(dy, inv);
    nz = xmul(dz, inv);
    return true;
}

// The spring's force quantised into the mixed path's fixed-point sums.
__device__ __forceinline__ void bond_to_fixed(long long* F, size_t fstride, uint32_t ia, uint32_t ib, double nx,
                                              double ny, double nz, double fm) {
    const long long q[3] = {__double2ll_rn(xmul(xmul(nx, fm), kFixScale)),
                            __double2ll_rn(xmul(xmul(ny, fm), kFixScale)),
                            __double2ll_rn(xmul(xmul(nz, fm), kFixScale))};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        atomicAdd((unsigned long long*)&F[c * fstride + ia], (unsigned long long)q[c]);
        atomicAdd((unsigned long long*)&F[c * fstride + ib], (unsigned long long)(-q[c]));
    }
}

inline LawF64 make_law64(const gx_handle* h) {
    LawF64 L;
    L.lj_rc = h->fs.lj_rc;
    L.lj_ron = h->fs.lj_ron;
    L.coul_rc = h->fs.coul_rc;
    L.coul_ron = h->fs.coul_ron;
    L.grav_rc = h->fs.grav_rc;
    L.grav_ron = h->fs.grav_ron;
    L.rc2 = h->fs.rc * h->fs.rc;
    L.k_e = h->p.coulomb_constant;
    L.G = h->p.gravity_constant;
    for (int k = 0; k < 3; ++k) L.box[k] = h->p.box[k];
    L.lj_iw = 1.0 / (L.lj_rc - L.lj_ron);
    L.coul_iw = 1.0 / (L.coul_rc - L.coul_ron);
    L.grav_iw = 1.0 / (L.grav_rc - L.grav_ron);
    L.one_switch = L.lj_rc == L.coul_rc && L.lj_ron == L.coul_ron;
    L.coul = h->p.enable_electrostatics ? 1 : 0;
    L.grav = h->p.enable_gravity ? 1 : 0;
    return L;
}

}  // namespace gx
