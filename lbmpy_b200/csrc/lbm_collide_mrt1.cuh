// MRT collision when every moment of order >= 3 relaxes with rate 1 and the shear moments share one rate
// (lbmpy's [shear, bulk, 1, ...], and its single-rate default, where the bulk rate is 1 too;
// methods/creationfunctions.py:600-706).
#pragma once
#include "lbm_collide.cuh"

namespace lbm {

// Weight 3 w of the odd part of a direction of squared length c2.  The axis value takes what the rounded
// values of the other directions leave of the momentum: 2 axis + 8 edge (+ 8 corner) = 1.
template <int Q, class R> constexpr double mrt1_odd(int c2) {
    auto rounded = [](double v) { return std::is_same<R, double>::value ? v : double(float(v)); };
    const double edge = rounded(1.0 / (Q == 19 ? 12.0 : 18.0)), corner = Q == 19 ? 0.0 : rounded(1.0 / 72.0);
    return c2 == 1 ? 0.5 - 4.0 * edge - 4.0 * corner : c2 == 2 ? edge : corner;
}

// A moment that relaxes with rate 1 ends at its equilibrium, so the state after the collision is the
// equilibrium plus what is left of the second-order non-equilibrium Pi.  The weighted-orthogonal
// second-order moments span the second-order Hermite polynomials, on which the projection is
//   w_i [ 9/2 (c_a c_b - delta_ab / 3) Q_ab + 3/2 (|c|^2 - 1) B ],
// Q = (1 - shear) dev(Pi), B = (1 - bulk) tr(Pi).  The force populations (Luo and Guo:
// w_i (9 (c.F)(c.u) + 3 c.F - 3 u.F); Simple: 3 w_i c.F) have an odd part of first order, which stays
// whole, and an even part on the same polynomials, scaled per rate by Guo.
//
// The state is rebuilt from its moments, so that rounded weights would scale mass and momentum by the
// same factor in every step: the rest population closes the mass, and the axis weights close the momentum
// (mrt1_odd), which leaves rounding noise alone, as a collision that adds small changes does.
//
// Ten sums of the populations are all that is kept of them: about half the arithmetic of the
// transforms of collide_mrt and fewer registers (D3Q19 FP32 pull: 48 registers with 12 bytes spilled, collide_mrt 64 with
// 20).
template <int Q, class R, class P>
__device__ __forceinline__ R collide_mrt1(R (&f)[Q], const P& p) {
    using L = Lat<Q>;
    const bool shift = p.force_model == FM_GUO;
    const Macro<Q, R> m = conserved<Q, R>(f, p, shift);
    R sxx = 0, syy = 0, szz = 0, sxy = 0, sxz = 0, syz = 0;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        if (L::cx(i) != 0) sxx += f[i];
        if (L::cy(i) != 0) syy += f[i];
        if (L::cz(i) != 0) szz += f[i];
        if (L::cx(i) * L::cy(i) == 1) sxy += f[i]; else if (L::cx(i) * L::cy(i) == -1) sxy -= f[i];
        if (L::cx(i) * L::cz(i) == 1) sxz += f[i]; else if (L::cx(i) * L::cz(i) == -1) sxz -= f[i];
        if (L::cy(i) * L::cz(i) == 1) syz += f[i]; else if (L::cy(i) * L::cz(i) == -1) syz -= f[i];
    }
    const R rf = p.compressible ? m.rho : R(1);
    const R third = m.drho * R(1.0 / 3.0);
    // rf u_a u_b, then the non-equilibrium moments
    const R eu[6] = {rf * m.ux * m.ux, rf * m.uy * m.uy, rf * m.uz * m.uz,
                     rf * m.ux * m.uy, rf * m.ux * m.uz, rf * m.uy * m.uz};
    R q[6] = {sxx - eu[0] - third, syy - eu[1] - third, szz - eu[2] - third, sxy - eu[3], sxz - eu[4], syz - eu[5]};
    R ws = p_rate<R>(p, 4), wb = p_rate<R>(p, 9), om = R(0);
    if (p.sgs == 1) {
        const R s2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + R(2) * (q[3] * q[3] + q[4] * q[4] + q[5] * q[5]);
        using ::sqrt;          // and, by its argument type, the packed pairs' own
        const R pi = sqrt(R(2) * s2) / m.rho_ref;
        const R tau0 = p_tau0<R>(p);
        om = R(2) / (tau0 + sqrt(p_c18<R>(p) * pi + tau0 * tau0));
        if ((p.sgs_mask >> 4) & 1u) ws = om;
        if ((p.sgs_mask >> 9) & 1u) wb = om;
    }
    const R tr = q[0] + q[1] + q[2], t3 = tr * R(1.0 / 3.0), ks = R(1) - ws;
    R b = (R(1) - wb) * tr;
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] = ks * (q[a] - t3);
#pragma unroll
    for (int a = 3; a < 6; ++a) q[a] = ks * q[a];
    R Fx = R(0), Fy = R(0), Fz = R(0);
    if (p.force_model != FM_NONE) {
        Fx = p_force<R>(p, 0); Fy = p_force<R>(p, 1); Fz = p_force<R>(p, 2);
        if (p.force_model != FM_SIMPLE) {
            const R gs = p.force_model == FM_GUO ? R(1) - R(0.5) * ws : R(1);
            const R gb = p.force_model == FM_GUO ? R(1) - R(0.5) * wb : R(1);
            const R x2 = R(2) * m.ux * Fx, y2 = R(2) * m.uy * Fy, z2 = R(2) * m.uz * Fz;
            const R tf = x2 + y2 + z2, tf3 = tf * R(1.0 / 3.0);
            q[0] += gs * (x2 - tf3); q[1] += gs * (y2 - tf3); q[2] += gs * (z2 - tf3);
            q[3] += gs * (m.ux * Fy + m.uy * Fx);
            q[4] += gs * (m.ux * Fz + m.uz * Fx);
            q[5] += gs * (m.uy * Fz + m.uz * Fy);
            b += gb * tf;
        }
    }
    // momentum after the collision (Guo's velocity holds half the force already)
    const R hf = R(shift ? 0.5 : 1.0);
    const R jx = rf * m.ux + hf * Fx, jy = rf * m.uy + hf * Fy, jz = rf * m.uz + hf * Fz;
    R sum = R(0);              // of the even parts of the pairs
#pragma unroll
    for (int q2 = 0; q2 < (Q - 1) / 2; ++q2) {
        const int i = L::pair(q2), j = L::inv(i);   // (i, inverse) share the even part, the odd part changes sign
        const double w = L::w(i);
        const int c2 = L::cx(i) * L::cx(i) + L::cy(i) * L::cy(i) + L::cz(i) * L::cz(i);
        R e = R(w) * m.drho;
#pragma unroll
        for (int a = 0; a < 6; ++a) e = cmad(e, L::eqquad(true, i, a), eu[a]);
        if (c2 != 1) e = cmad(e, 1.5 * w * (c2 - 1), b);
        e = cmad(e, L::cx(i) != 0 ? 4.5 * w : 0.0, q[0]);
        e = cmad(e, L::cy(i) != 0 ? 4.5 * w : 0.0, q[1]);
        e = cmad(e, L::cz(i) != 0 ? 4.5 * w : 0.0, q[2]);
        e = cmad(e, 9.0 * w * L::cx(i) * L::cy(i), q[3]);
        e = cmad(e, 9.0 * w * L::cx(i) * L::cz(i), q[4]);
        e = cmad(e, 9.0 * w * L::cy(i) * L::cz(i), q[5]);
        R o = R(0);
        o = cmad(o, mrt1_odd<Q, R>(c2) * L::cx(i), jx);
        o = cmad(o, mrt1_odd<Q, R>(c2) * L::cy(i), jy);
        o = cmad(o, mrt1_odd<Q, R>(c2) * L::cz(i), jz);
        sum += e;
        f[i] = e + o;
        f[j] = e - o;
    }
    f[0] = m.drho - R(2) * sum;
    return om;
}

}  // namespace lbm
