"""The Rys-quadrature arithmetic (csrc/hfgpu_rys_math.cuh) compiled with g++ and run on the host.

The kernel's phases are walked with one thread per group on buffers of exactly the sizes the
kernel lays out.  For classes from (ss|ss) to (dd|dd) and random primitive quartets (small and
large T, contracted, A = B) the 45 second-derivative entries equal the one-thread op tables of the
same class (gen_eri.gen_hess_table, themselves pinned to the reference by the GPU tests).  Both
sums are of a few thousand products of values up to ~10 times their result, so 1e-11 of the largest
entry bounds their rounding.  The gradient is checked against the Hessian by central differences
(h = 1e-4: truncation and rounding both near 1e-8 of the largest entry; 1e-6 is asked).  The form with
one thread per direction (csrc/hfgpu_rys3.cuh) equals the group form to 1e-11 in both orders.
"""
import importlib.util
import os
import shutil
import subprocess

import pytest

from test_hess_line_host import EXEC, ROOT, STUB, _gen_eri

CSRC = os.path.join(ROOT, "hfscf_b200", "csrc")

DRIVER = r"""
struct double2 { double x, y; };
struct int3 { int x, y, z; };
inline int3 make_int3(int x, int y, int z) { return {x, y, z}; }
#define __host__
inline double2 __ldg(const double2* p) { return *p; }
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
constexpr int ncart_of(int L) { return (L + 1) * (L + 2) / 2; }
#include "rys_math.h"
#include "rys_data.h"

struct Shells { double A[3], B[3], C[3], D[3], a[2], b[2], c[2], d[2]; };

static void make(PrimPair<double>& P, double a, double b, const double* X, const double* Y) {
  P.p = a + b; P.ip = 1.0 / P.p;
  const double Pc[3] = {(a * X[0] + b * Y[0]) / P.p, (a * X[1] + b * Y[1]) / P.p, (a * X[2] + b * Y[2]) / P.p};
  P.Px = Pc[0]; P.Py = Pc[1]; P.Pz = Pc[2];
  P.PAx = Pc[0] - X[0]; P.PAy = Pc[1] - X[1]; P.PAz = Pc[2] - X[2];
  double r2 = 0;
  for (int i = 0; i < 3; ++i) r2 += (X[i] - Y[i]) * (X[i] - Y[i]);
  P.Kp = std::exp(-a * b / P.p * r2) * std::sqrt(2 * std::pow(M_PI, 2.5)) / P.p;
}

template <int LA, int LB, int LC, int LD, int ORD>
void rys_run(const Shells& s, const double* W, double* out) {
  using D = RysDims<LA, LB, LC, LD, ORD>;
  std::vector<double> rw(D::kRW), g2(D::kG2), bv(D::kBV), vt(D::kVT);
  double acc[D::NOUT] = {0.0};
  for (int ib = 0; ib < 2; ++ib)
    for (int ik = 0; ik < 2; ++ik) {
      PrimPair<double> P, Q;
      make(P, s.a[ib], s.b[ib], s.A, s.B);
      make(Q, s.c[ik], s.d[ik], s.C, s.D);
      const double p = P.p, q = Q.p, ipq = 1.0 / (p + q);
      const double PQ[3] = {P.Px - Q.Px, P.Py - Q.Py, P.Pz - Q.Pz};
      const double PA[3] = {P.PAx, P.PAy, P.PAz}, QC[3] = {Q.PAx, Q.PAy, Q.PAz};
      const double T = p * q * ipq * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
      const double pre = P.Kp * Q.Kp * std::sqrt(ipq);
      for (int v = 0; v < D::kRW; ++v)
        rw[v] = rys_value<D::NR>(rys_data, T, v) * (v < D::NR ? 1.0 : pre);
      for (int it = 0; it < 3 * D::NR; ++it) {
        const int r = it / 3, d = it % 3;
        const double B00 = 0.5 * rw[r] * ipq, u = 2 * B00 * PQ[d];
        rys_vrr<D::E, D::F, D::FS>(d == 2 ? rw[D::NR + r] : 1.0, PA[d] - q * u, QC[d] + p * u, B00, P.ip * (0.5 - B00 * q),
                            Q.ip * (0.5 - B00 * p), g2.data() + it * D::GS);
      }
      for (int r = 0; r < D::NR; ++r) {
        for (int it = 0; it < 3 * (D::F + 1); ++it) {
          const int d = it / (D::F + 1), f = it % (D::F + 1);
          rys_bra<LA, LB, ORD, D::FS>(g2.data() + (r * 3 + d) * D::GS + f, s.A[d] - s.B[d], 2 * s.a[ib], 2 * s.b[ib],
                                      bv.data() + d * D::BS + f);
        }
        for (int it = 0; it < 3 * D::NB; ++it) {
          const int d = it / D::NB, ij = it % D::NB;
          rys_ket<LC, LD, ORD, D::NB, D::FS, 3 * D::NX>(bv.data() + d * D::BS + ij * D::FS, s.C[d] - s.D[d], 2 * s.c[ik],
                                                        vt.data() + d * D::NX + ij);
        }
        for (int e = 0; e < D::NCART; ++e) {
          const int t = rys_index<LA, LB, LC, LD>(e);
          double X[D::NV], Y[D::NV], Z[D::NV];
          for (int v = 0; v < D::NV; ++v) {
            X[v] = vt.at((t & 255) + v * 3 * D::NX);
            Y[v] = vt.at(D::NX + (t >> 8 & 255) + v * 3 * D::NX);
            Z[v] = vt.at(2 * D::NX + (t >> 16) + v * 3 * D::NX);
          }
          rys_accumulate<ORD>(W[e], X, Y, Z, acc);
        }
      }
    }
  for (int x = 0; x < D::NOUT; ++x) out[x] = acc[x];
}

// the same by the three threads, one per direction, of hfgpu_rys3.cuh
template <int LA, int LB, int LC, int LD, int ORD>
void rys3_run(const Shells& s, const double* W, double* out) {
  using D = Rys3Dims<LA, LB, LC, LD, ORD>;
  std::vector<double> rw(2 * D::NR);
  double acc[3][D::NACC] = {{0.0}};
  auto renamed = [&](int d, int e) {  // weight of the integral whose exponents along d, d+1, d+2 are e's
    auto back = [&](int l, int c) {
      const int3 v = rys_comp(l, c);
      return d == 0 ? c : (d == 1 ? rys_cart(l, v.z, v.x) : rys_cart(l, v.y, v.z));
    };
    return W[((back(LA, e / (D::CB * D::CC * D::CD)) * D::CB + back(LB, e / (D::CC * D::CD) % D::CB)) * D::CC +
              back(LC, e / D::CD % D::CC)) * D::CD + back(LD, e % D::CD)];
  };
  std::vector<double> Wd[3];
  for (int d = 0; d < 3; ++d)
    for (int e = 0; e < D::NCART; ++e) Wd[d].push_back(renamed(d, e));
  for (int ib = 0; ib < 2; ++ib)
    for (int ik = 0; ik < 2; ++ik) {
      PrimPair<double> P, Q;
      make(P, s.a[ib], s.b[ib], s.A, s.B);
      make(Q, s.c[ik], s.d[ik], s.C, s.D);
      const double p = P.p, q = Q.p, ipq = 1.0 / (p + q);
      const double PQ[3] = {P.Px - Q.Px, P.Py - Q.Py, P.Pz - Q.Pz};
      const double PA[3] = {P.PAx, P.PAy, P.PAz}, QC[3] = {Q.PAx, Q.PAy, Q.PAz};
      const double T = p * q * ipq * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
      const double pre = P.Kp * Q.Kp * std::sqrt(ipq), wa = 2 * s.a[ib], wb = 2 * s.b[ib], wc = 2 * s.c[ik];
      for (int v = 0; v < 2 * D::NR; ++v) rw[v] = rys_value<D::NR>(rys_data, T, v) * (v < D::NR ? 1.0 : pre);
      for (int r = 0; r < D::NR; ++r) {
        std::vector<double> V(3 * D::DV);
        double g[3][D::E + 1][D::F + 1];
        for (int d = 0; d < 3; ++d) {
          const double B00 = 0.5 * rw[r] * ipq, u = 2 * B00 * PQ[d];
          rys3_vrr<D::E, D::F>(d == 2 ? rw[D::NR + r] : 1.0, PA[d] - q * u, QC[d] + p * u, B00,
                               P.ip * (0.5 - B00 * q), Q.ip * (0.5 - B00 * p), g[d]);
          for (int i = 0; i <= LA; ++i)
            for (int j = 0; j <= LB; ++j) {
              double w[4][D::NK];
              rys3_variants<LA, LB, LC, LD, ORD, false>(g[d], s.A[d] - s.B[d], s.C[d] - s.D[d], wa, wb, wc, i, j, w);
              for (int v = 0; v < D::NSH; ++v)
                for (int kl = 0; kl < D::NK; ++kl) V.at(d * D::DV + v * D::NX + (i * (LB + 1) + j) * D::NK + kl) = w[v][kl];
            }
        }
        for (int d = 0; d < 3; ++d)
          for (int i = 0; i <= LA; ++i)
            for (int j = 0; j <= LB; ++j) {
              double w[ORD == 2 ? 10 : 4][D::NK];
              rys3_variants<LA, LB, LC, LD, ORD, ORD == 2>(g[d], s.A[d] - s.B[d], s.C[d] - s.D[d], wa, wb, wc, i, j, w);
              rys3_accumulate<LA, LB, LC, LD, ORD>(w, i, j, V.data() + (d + 1) % 3 * D::DV, V.data() + (d + 2) % 3 * D::DV,
                                                   Wd[d].data(), acc[d]);
            }
      }
    }
  for (int d = 0; d < 3; ++d)
    for (int A = 0; A < 3; ++A)
      for (int B = 0; B < 3; ++B)
        if (ORD == 1) {
          out[3 * A + d] = acc[d][A];
        } else {
          const int r = 3 * A + d, c = 3 * B + (d + 1) % 3;
          if (A <= B) out[rys_tri(r, 3 * B + d)] = acc[d][rys_second(A, B) - 4];
          out[r < c ? rys_tri(r, c) : rys_tri(c, r)] = acc[d][6 + 3 * A + B];
        }
}

// largest difference of the Hessian from the op tables, and of the gradient's central differences
// from the Hessian, relative to the largest entry
template <int LA, int LB, int LC, int LD, typename Tab>
void rys_check(unsigned seed, double far, bool same, double* worst) {
  std::srand(seed);
  auto u = [](double lo, double hi) { return lo + (hi - lo) * (std::rand() / (double)RAND_MAX); };
  Shells s;
  for (int i = 0; i < 3; ++i) {
    s.A[i] = u(-1, 1);
    s.B[i] = same ? s.A[i] : u(-1, 1);
    s.C[i] = u(-1, 1) + far;
    s.D[i] = u(-1, 1) + far;
  }
  for (int i = 0; i < 2; ++i) {
    s.a[i] = u(0.2, 3.0); s.b[i] = u(0.2, 3.0); s.c[i] = u(0.2, 3.0); s.d[i] = u(0.2, 3.0);
  }
  constexpr int NC = RysDims<LA, LB, LC, LD, 2>::NCART;
  std::vector<double> W(NC);
  for (auto& w : W) w = u(-1, 1);
  PrimPair<double> bp[2], kp[2];
  for (int i = 0; i < 2; ++i) {
    make(bp[i], s.a[i], s.b[i], s.A, s.B);
    make(kp[i], s.c[i], s.d[i], s.C, s.D);
  }
  double AB[3], CD[3], ht[45], hr[45], gp[9], gm[9], mx = 0;
  for (int i = 0; i < 3; ++i) { AB[i] = s.A[i] - s.B[i]; CD[i] = s.C[i] - s.D[i]; }
  run_table<Tab>(bp, s.a, s.b, 2, kp, s.c, 2, AB, CD, W.data(), ht);
  rys_run<LA, LB, LC, LD, 2>(s, W.data(), hr);
  for (int x = 0; x < 45; ++x) mx = std::max(mx, std::fabs(ht[x]));
  for (int x = 0; x < 45; ++x) worst[0] = std::max(worst[0], std::fabs(ht[x] - hr[x]) / mx);
  if constexpr (NC <= 81) {
    rys3_run<LA, LB, LC, LD, 2>(s, W.data(), ht);
    for (int x = 0; x < 45; ++x) worst[2] = std::max(worst[2], std::fabs(ht[x] - hr[x]) / mx);
    rys_run<LA, LB, LC, LD, 1>(s, W.data(), gp);
    rys3_run<LA, LB, LC, LD, 1>(s, W.data(), gm);
    double gx = 0;
    for (int x = 0; x < 9; ++x) gx = std::max(gx, std::fabs(gp[x]));
    for (int x = 0; x < 9; ++x) worst[2] = std::max(worst[2], std::fabs(gp[x] - gm[x]) / gx);
  }
  const double h = 1e-4;
  for (int r = 0; r < 9; ++r) {
    double* X[3] = {s.A, s.B, s.C};
    double& x = X[r / 3][r % 3];
    const double x0 = x;
    x = x0 + h;
    rys_run<LA, LB, LC, LD, 1>(s, W.data(), gp);
    x = x0 - h;
    rys_run<LA, LB, LC, LD, 1>(s, W.data(), gm);
    x = x0;
    for (int c = 0; c < 9; ++c) {
      const double want = hr[r <= c ? rys_tri(r, c) : rys_tri(c, r)];
      worst[1] = std::max(worst[1], std::fabs((gp[c] - gm[c]) / (2 * h) - want) / mx);
    }
  }
}
"""


@pytest.mark.parametrize("cls", [(0, 0, 0, 0), (1, 0, 0, 0), (1, 1, 1, 0), (1, 1, 1, 1), (2, 0, 1, 1), (2, 1, 0, 0), (2, 1, 2, 0),
                                 (2, 2, 1, 0), (2, 2, 2, 2)], ids=lambda c: "".join("spd"[x] for x in c))
def test_rys_derivatives_match_the_op_tables(tmp_path, cls):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    spec = importlib.util.spec_from_file_location("gen_rys_for_test", os.path.join(CSRC, "gen_rys.py"))
    rys = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(rys)
    rys.emit(str(tmp_path))
    data = (tmp_path / "rys_table.cu").read_text()
    data = data[data.index("= {") + 2:data.index("};") + 2]
    (tmp_path / "rys_data.h").write_text("static const double rys_data[] = " + data + "\n")
    (tmp_path / "rys_math.h").write_text(
        open(os.path.join(CSRC, "hfgpu_rys_math.cuh")).read().replace("generated/rys_layout.cuh", "rys_layout.cuh"))
    table, _ = _gen_eri().gen_hess_table(*cls)
    t = "".join(map(str, cls))
    args = ", ".join(map(str, cls))
    main = ["int main() {", "  double w[3] = {0, 0, 0};"]
    for seed, far, same in ((1, 0.0, "false"), (2, 1.0, "true"), (3, 3.0, "false")):
        main.append(f"  rys_check<{args}, HessTable{t}>({seed}, {far}, {same}, w);")
    main += ['  std::printf("%.3e %.3e %.3e\\n", w[0], w[1], w[2]);', "}"]
    src = tmp_path / "rys.cpp"
    src.write_text("\n".join([STUB, "#include <vector>", table, EXEC, DRIVER] + main))
    exe = tmp_path / "rys"
    subprocess.run([gxx, "-std=c++17", "-O1", "-fsanitize=address", "-I", str(tmp_path), str(src), "-o", str(exe)],
                   check=True)
    hess, grad, three = map(float, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert hess < 1e-11, hess
    assert grad < 1e-6, grad
    assert three < 1e-11, three
