// gdem_adjoint_vjp.cuh -- the reverse-mode derivative of one contact of the
// adjoint step: the adjoints of a contact's inputs from those of its outputs
// (force, torques, tangential spring, normal), by the chain rule through the
// expressions of contactLaw (gdem_adjoint_law.cuh), in reverse order.
// A derivative is that of the branch taken by the value, and the derivative of
// a norm at zero is zero, as on the dual numbers of gdem_dual.cuh.
//
// Why: one sweep yields all inputs' adjoints for about four evaluations of
// the law, where a dual-number column yields one input's (18 per side of a
// contact).
#pragma once
#include "gdem_adjoint_law.cuh"

namespace gdem {

using W3 = V3<double>;

__host__ __device__ __forceinline__ W3 w3zero() { return v3(0., 0., 0.); }
__host__ __device__ __forceinline__ void acc(W3& a, W3 b) { a = a + b; }
// 1 / a, or 0 at a = 0 (the derivative of a norm there)
__host__ __device__ __forceinline__ double invOrZero(double a) { return a > 0. ? 1. / a : 0.; }
// adjoint of a in |a| = na
__host__ __device__ __forceinline__ W3 normBar(W3 a, double na, double bar) {
  return (bar * invOrZero(na)) * a;
}
// adjoint of a in a / |a| (na > 0)
__host__ __device__ __forceinline__ W3 unitBar(W3 a, double na, W3 bar) {
  const double i = 1. / na;
  return i * (bar - (vdot(a, bar) * i * i) * a);
}

// Adjoints of u, v, x in rotateFromTo(u, v, x) from that of its result.
__host__ __device__ __forceinline__ void rotateBar(W3 u, W3 v, W3 x, W3 bar, W3& ub, W3& vb,
                                                   W3& xb) {
  const double uu = vdot(u, u), vv = vdot(v, v);
  const double nn = sqrt(uu * vv);
  double real = nn + vdot(u, v);
  const bool opposite = real < 1.e-6 * nn;
  const bool first = fabs(u.x) > fabs(u.z);
  W3 vect;
  if (opposite) {
    real = 0.;
    vect = first ? v3(-u.y, u.x, 0.) : v3(0., -u.z, u.y);
  } else {
    vect = vcross(u, v);
  }
  const double nq = sqrt(vdot(vect, vect) + real * real);
  const double s = 1. / nq;
  const W3 qv = s * vect;
  const double qw = real * s;
  const double xq = vdot(x, qv), rq = vdot(bar, qv), ab = vdot(bar, x);
  acc(xb, (qw * qw - vdot(qv, qv)) * bar + (2. * rq) * qv + (2. * qw) * vcross(bar, qv));
  const double qwb = 2. * qw * ab + 2. * vdot(vcross(qv, x), bar);
  const W3 qvb = (-2. * ab) * qv + (2. * xq) * bar + (2. * rq) * x + (2. * qw) * vcross(x, bar);
  const double sb = vdot(qvb, vect) + qwb * real;
  const double nqb = -sb * s * s;
  const W3 vectb = s * qvb + (nqb * s) * vect;
  if (opposite) {
    if (first) acc(ub, v3(vectb.y, -vectb.x, 0.));
    else acc(ub, v3(0., vectb.z, -vectb.y));
    return;
  }
  const double realb = s * qwb + nqb * s * real;
  const double nnb = realb * invOrZero(nn);
  acc(ub, vcross(v, vectb) + realb * v + (nnb * vv) * u);
  acc(vb, vcross(vectb, u) + realb * u + (nnb * uu) * v);
}

// Inputs of the law and the levers' ends; the adjoints of a law call.
struct LawArgs {
  W3 pc, pen, x0, v0, w0, x1, v1, w1, kd, pn;
  double kn, en, muc;
};

// Adjoints g of the inputs of a contact with outputs f = contactLaw().f on
// body 0 (-f on body 1), the torques (pc - x0) x f and (pc - x1) x (-f), the
// new spring kd and the new normal pn, from the adjoints F0, T0, F1, T1, kdb,
// pnb of those outputs.
__host__ __device__ inline void contactBar(ModelDesc const& m, double dt, LawArgs const& in,
                                           double m0, double m1, bool existed, W3 F0, W3 T0, W3 F1,
                                           W3 T1, W3 kdb, W3 pnb, LawArgs& g) {
  const double PI = 3.14159265358979323846;
  // ---- values, as contactLaw computes them
  const double npen = vnorm(in.pen);
  const W3 unit = in.pen / npen;
  const W3 n = roundSmall(unit);
  const W3 l0 = in.pc - in.x0, l1 = in.pc - in.x1;
  const W3 U = (in.v0 + vcross(in.w0, l0)) - (in.v1 + vcross(in.w1, l1));
  const double c = vdot(U, n);
  const W3 vn = c * n, vt = U - vn;
  const double len = log(in.en);
  const double root = sqrt(PI * PI + len * len);
  const double beta = len / root;
  const double mass = 1. / (1. / m0 + 1. / m1);
  const double gn = -2. * beta * sqrt(in.kn * mass);
  const bool etat_of_beta = m.etat == -1.;
  const double etat = etat_of_beta ? -beta * sqrt(in.kn / mass) : m.etat;
  const double gt = 2. * etat * mass;
  const W3 FN = in.kn * in.pen - gn * vn;
  const double nFN = vnorm(FN);
  const W3 visc = (-gt) * vt;
  W3 f, vtb = w3zero(), viscb = w3zero(), nb = pnb, kd1b = w3zero();
  double nFNb = 0., gtb = 0., mucb = 0.;
  // ---- force adjoint (the torques' lever arms follow below)
  const W3 fb = F0 - F1 + vcross(T0, l0) - vcross(T1, l1);
  g.kd = g.pn = w3zero();
  if (!m.memory) {
    // Hooke: the viscous force, capped at muc |FN|
    const double fcap = in.muc * nFN;
    if (fcap < vnorm(visc)) {
      const double nvt = vnorm(vt);
      W3 t = w3zero();
      if (nvt > 1.0e-10) {
        t = (-1. / nvt) * vt;
        acc(vtb, unitBar(vt, nvt, (-fcap) * fb));
      }
      f = FN + fcap * t;
      const double cb = vdot(fb, t);
      mucb += cb * nFN;
      nFNb += cb * in.muc;
    } else {
      f = FN + visc;
      acc(viscb, fb);
    }
  } else {
    W3 kd = w3zero();
    if (existed) kd = rotateFromTo(in.pn, n, in.kd);
    kd = kd + (dt * m.kt) * vt;
    W3 t = w3zero(), s = w3zero();
    const double nut = vnorm(vt);
    double ns = 0.;
    const bool sliding = nut > 0.001;
    bool resting = false;
    if (sliding) {
      t = (-1. / nut) * vt;
    } else {
      s = kd + gt * vt;
      ns = vnorm(s);
      resting = (vnorm(kd) > m.epst || vnorm(gt * vt) > m.epst) && ns > m.epst;
      if (resting) t = (-1. / ns) * s;
    }
    const W3 trial = visc - kd;
    const double nFT = vnorm(trial);
    W3 tb, kd2b = w3zero();
    if (nFT <= in.muc * nFN) {
      f = FN + nFT * t;
      tb = nFT * fb;
      const W3 trialb = normBar(trial, nFT, vdot(fb, t));
      kd2b = kdb - trialb;
      acc(viscb, trialb);
    } else {
      const double cap = in.muc * nFN;
      f = FN + cap * t;
      tb = cap * fb;
      double capb = vdot(fb, t);
      if (m.kt != 0.) {
        const double ikt = 1. / m.kt;
        acc(tb, (-cap * ikt) * kdb);
        capb -= ikt * vdot(kdb, t);
        acc(viscb, ikt * kdb);
      } else {
        kd2b = kdb;
      }
      mucb += capb * nFN;
      nFNb += capb * in.muc;
    }
    if (sliding) {
      acc(vtb, unitBar(vt, nut, -tb));
    } else if (resting) {
      const W3 sb = unitBar(s, ns, -tb);
      acc(kd2b, sb);
      acc(vtb, gt * sb);
      gtb += vdot(sb, vt);
    }
    acc(vtb, (dt * m.kt) * kd2b);
    if (existed) rotateBar(in.pn, n, in.kd, kd2b, g.pn, nb, g.kd);
  }
  // ---- lever arms of the torques
  W3 l0b = vcross(f, T0), l1b = -vcross(f, T1);
  // ---- viscous and normal forces
  acc(vtb, (-gt) * viscb);
  gtb -= vdot(viscb, vt);
  const W3 FNb = fb + normBar(FN, nFN, nFNb);
  g.pen = in.kn * FNb;
  g.kn = vdot(FNb, in.pen);
  const double gnb = -vdot(FNb, vn);
  // ---- the damping coefficients
  double betab = gnb * (-2. * sqrt(in.kn * mass));
  g.kn += gnb * (-beta * sqrt(mass / in.kn));
  if (etat_of_beta) {
    betab += gtb * (-2. * mass * sqrt(in.kn / mass));
    g.kn += gtb * (-beta * sqrt(mass / in.kn));
  }
  g.en = betab * (PI * PI / (root * root * root)) / in.en;
  g.muc = mucb;
  // ---- the split of the relative velocity
  const W3 vnb = (-gn) * FNb - vtb;
  const double cb = vdot(n, vnb);
  acc(nb, c * vnb + cb * U);
  const W3 Ub = vtb + cb * n;
  g.v0 = Ub;
  g.v1 = -Ub;
  g.w0 = vcross(l0, Ub);
  g.w1 = -vcross(l1, Ub);
  acc(l0b, vcross(Ub, in.w0));
  acc(l1b, -vcross(Ub, in.w1));
  g.pc = l0b + l1b;
  g.x0 = -l0b;
  g.x1 = -l1b;
  // ---- the normal (components rounded to zero carry nothing)
  if (n.x == 0.) nb.x = 0.;
  if (n.y == 0.) nb.y = 0.;
  if (n.z == 0.) nb.z = 0.;
  acc(g.pen, unitBar(in.pen, npen, nb));
}

// Adjoints of the two centres in sphereSphereG's contact point and overlap
// vector, added to xab, xbb.
__host__ __device__ inline void sphereSphereBar(W3 xa, double ra, W3 xb, double rb, W3 pcb,
                                                W3 penb, W3& xab, W3& xbb) {
  const W3 AB = xb - xa;
  const double nAB = vnorm(AB), dist = nAB - (ra + rb), q = (dist * 0.5 + ra) / nAB;
  const W3 e = AB / nAB;
  const double qb = vdot(pcb, AB);
  // pc = xa + q AB, pen = dist e, dist = nAB - (ra + rb)
  const double nb = vdot(penb, e) + qb * (0.5 - q) / nAB;
  const W3 ABb = q * pcb + unitBar(AB, nAB, dist * penb) + nb * e;
  acc(xab, pcb - ABb);
  acc(xbb, ABb);
}

// Adjoint of the centre in sphereWallG, added to xb: one dual-number column
// per axis (the geometry alone is cheap and has a dozen cases).
__host__ __device__ inline void sphereWallBar(W3 x, double r, WallDesc const& w, W3 pcb, W3 penb,
                                              W3& xb) {
  double g[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    V3<Dual<1>> xd = v3(dconst<1>(x.x), dconst<1>(x.y), dconst<1>(x.z)), pc, pen;
    if (d == 0) xd.x.d[0] = 1.;
    else if (d == 1) xd.y.d[0] = 1.;
    else xd.z.d[0] = 1.;
    g[d] = 0.;
    if (sphereWallG(xd, r, w, pc, pen))
      g[d] = pcb.x * pc.x.d[0] + pcb.y * pc.y.d[0] + pcb.z * pc.z.d[0] + penb.x * pen.x.d[0] +
             penb.y * pen.y.d[0] + penb.z * pen.z.d[0];
  }
  acc(xb, v3(g[0], g[1], g[2]));
}

}  // namespace gdem
