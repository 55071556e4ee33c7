"""The reverse-mode derivative of one contact (gdem_adjoint_vjp.cuh) against
its dual-number columns, on the host: every branch of the law (Hooke and
HookeMemory, sliding and resting, stick and slip, first contact and carried
history, opposite normals, kt = 0, a given etat), random outputs' adjoints.

Both are exact derivatives of the same expressions, so an input vector's
adjoint agrees to the rounding of a few hundred operations, amplified by the
cancellation between its terms: 1e-9 of the vector's largest column."""
import os
import subprocess
import textwrap
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "pacific_b200" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

PROGRAM = textwrap.dedent(r"""
    #include <algorithm>
    #include <cmath>
    #include <cstdio>
    #include <random>
    using std::fabs; using std::log; using std::sqrt;
    #include "gdem_adjoint_vjp.cuh"
    using namespace gdem;
    typedef Dual<1> D;
    static V3<D> lift(W3 a) { return v3(dconst<1>(a.x), dconst<1>(a.y), dconst<1>(a.z)); }
    static double dy(W3 l, V3<D> y) { return l.x * y.x.d[0] + l.y * y.y.d[0] + l.z * y.z.d[0]; }
    static double& comp(W3& a, int d) { return d == 0 ? a.x : (d == 1 ? a.y : a.z); }
    static D& comp(V3<D>& a, int d) { return d == 0 ? a.x : (d == 1 ? a.y : a.z); }
    int main() {
      std::mt19937 gen(3);
      std::uniform_real_distribution<double> U(-1, 1);
      auto rv = [&](double s) { return v3(s * U(gen), s * U(gen), s * U(gen)); };
      double worst = 0.;
      int cases = 0;
      for (int it = 0; it < 20000; ++it) {
        ModelDesc m{};
        m.memory = it % 3 != 0;
        m.kt = it % 7 == 0 ? 0. : 2857.;
        m.etat = it % 5 == 0 ? 0.3 : -1.;
        const double dt = 1e-5, ra = 1e-3, rb = 1.1e-3, m0 = 1e-5, m1 = it % 2 ? 1.3e-5 : 1e20;
        const double kn = 1e4, en = 0.7, muc = it % 4 == 0 ? 0.02 : 0.5;
        const bool existed = (it / 2) % 2;
        const W3 xa = rv(0.01);
        W3 dir = rv(1.);
        if (it % 9 == 0) dir.x = 0.;
        dir = dir / vnorm(dir);
        const W3 xb = xa + (ra + rb - std::pow(10., -8. + 3. * fabs(U(gen)))) * dir;
        const double vs = it % 6 < 3 ? 5e-5 : 0.1;
        const W3 va = rv(vs), vb = rv(vs), wa = rv(1e3 * vs), wb = rv(1e3 * vs);
        const W3 kd = rv(std::pow(10., -6. + 4. * fabs(U(gen))));
        W3 pn = it % 13 == 0 ? dir : -dir + (it % 11 ? rv(1e-3) : rv(1.));
        pn = pn / vnorm(pn);
        const W3 F0 = rv(1.), T0 = rv(1e3), F1 = rv(1.), T1 = rv(1e3), kb = rv(1.), nb = rv(1e-2);
        W3 pc, pen;
        if (!sphereSphereG(xa, ra, xb, rb, pc, pen)) continue;
        ++cases;
        LawArgs in{pc, pen, xa, va, wa, xb, vb, wb, kd, pn, kn, en, muc}, g;
        contactBar(m, dt, in, m0, m1, existed, F0, T0, F1, T1, kb, nb, g);
        sphereSphereBar(xa, ra, xb, rb, g.pc, g.pen, g.x0, g.x1);
        W3 got[8] = {g.x0, g.x1, g.v0, g.v1, g.w0, g.w1, g.kd, g.pn};
        const double gp[3] = {g.kn, g.en, g.muc};
        const int vectors = existed && m.memory ? 8 : 6;
        for (int q = 0; q < vectors + 3; ++q) {
          double size = 0., err = 0.;
          for (int d = 0; d < (q < vectors ? 3 : 1); ++d) {
            V3<D> i[8] = {lift(xa), lift(xb), lift(va), lift(vb), lift(wa), lift(wb), lift(kd), lift(pn)};
            D p[3] = {dconst<1>(kn), dconst<1>(en), dconst<1>(muc)};
            if (q < vectors) comp(i[q], d).d[0] = 1.;
            else p[q - vectors].d[0] = 1.;
            V3<D> pcd, pend;
            sphereSphereG(i[0], ra, i[1], rb, pcd, pend);
            const LawOut<D> o = contactLaw(m, dt, p[0], p[1], p[2], pcd, pend, i[0], i[2], i[4], m0,
                                           i[1], i[3], i[5], m1, existed, i[6], i[7]);
            const double ref = dy(F0, o.f) + dy(T0, vcross(pcd - i[0], o.f)) - dy(F1, o.f) +
                               dy(T1, vcross(pcd - i[1], -o.f)) + dy(kb, o.kd) + dy(nb, o.pn);
            const double val = q < vectors ? comp(got[q], d) : gp[q - vectors];
            size = std::max(size, fabs(ref));
            err = std::max(err, fabs(val - ref));
          }
          // (adjoints far below the outputs' own, O(1), are left to the absolute bound)
          if (!(err <= 1e-9 * size + 1e-12)) std::printf("case %d input %d: %g of %g\n", it, q, err, size);
          worst = std::max(worst, err / (size + 1e-3));
        }
      }
      std::printf("%d cases, worst %g\n", cases, worst);
      return cases > 15000 && worst < 1e-9 ? 0 : 1;
    }
""")


def test_contact_adjoint_matches_dual_columns(tmp_path):
    if not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("no CUDA headers")
    src = tmp_path / "vjp.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "vjp"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CUDA}", f"-I{CSRC}",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "case " not in r.stdout, r.stdout[-2000:]
