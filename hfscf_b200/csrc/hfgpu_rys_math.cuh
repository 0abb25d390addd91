// Arithmetic of the Rys-quadrature kernels (hfgpu_rys.cuh): quadrature values, the recurrences of
// the two-dimensional integrals, their derivative variants and the contraction of one integral.
// No CUDA headers, so that a host test can compile it with stand-ins for the qualifiers.
#pragma once
#include <type_traits>

#include "generated/rys_layout.cuh"

// Walk of a launch's quartets, in 64 bits: without a block limit the stride covers the whole list, so that
// a 32-bit index would pass 2^31 in its first step from 2^30 quartets on, turn negative and read in front
// of the list.  Each of the `walkers` of a block (its warps, or one) takes `per` quartets at a time.
__host__ __device__ constexpr long long rys_first(unsigned block, int walkers, int walker, int per) {
  return ((long long)block * walkers + walker) * per;
}
__host__ __device__ constexpr long long rys_stride(unsigned blocks, int walkers, int per) {
  return (long long)blocks * walkers * per;
}
// Blocks of a launch over nq quartets, at most `most` (0: no limit).
__host__ __device__ constexpr unsigned rys_blocks(long long nq, int walkers, int per, int most) {
  const long long n = (nq + (long long)walkers * per - 1) / ((long long)walkers * per);
  return (unsigned)(most > 0 && n > most ? most : n);
}

// Value v of the n-point rule at T: squared root v (v < n) or weight v - n.
template <int N>
__device__ __forceinline__ double rys_value(const double* __restrict__ tab, double T, int v) {
  if (T < rys_tmax(N)) {
    const int k = (int)(T * kRysInvH);
    const double d = T - (k + 0.5) * kRysH;
    const double2* c = reinterpret_cast<const double2*>(tab + rys_offset(N) + (size_t)(k * 2 * N + v) * kRysCoef);
    double2 q[kRysCoef / 2];
#pragma unroll
    for (int j = 0; j < kRysCoef / 2; ++j) q[j] = __ldg(c + j);
    double f = q[kRysCoef / 2 - 1].y;
#pragma unroll
    for (int j = kRysCoef / 2 - 1; j >= 0; --j) {
      if (j < kRysCoef / 2 - 1) f = q[j].y + f * d;
      f = q[j].x + f * d;
    }
    return f;
  }
  const double s = rsqrt(T);
  return v < N ? c_rys_herm[N - 1][0][v] * s * s : c_rys_herm[N - 1][1][v - N] * s;
}

// Exponents of x, y, z in component c of a shell of momentum l (order of gen_eri.py cart()).
__device__ __forceinline__ int3 rys_comp(int l, int c) {
  const int i = c >= 3 ? 2 : (c >= 1 ? 1 : 0);
  const int j = c - i * (i + 1) / 2;
  return make_int3(l - i, i - j, j);
}

// Sizes of class (LA LB|LC LD) at derivative order ORD, and the layout of one group's shared memory
// (values of type R): [roots and weights | 2-D integrals of every root | bra variants of one root |
// variant tables of one root | W]; the first part doubles as the scratch of the weights' pure ->
// Cartesian transform.
template <int LA, int LB, int LC, int LD, int ORD>
struct RysDims {
  static constexpr int NR = (LA + LB + LC + LD + ORD) / 2 + 1;
  static constexpr int E = LA + LB + ORD, F = LC + LD + ORD;  // highest bra and ket orders
  static constexpr int NB = (LA + 1) * (LB + 1), NK = (LC + 1) * (LD + 1), NX = NB * NK;
  static constexpr int NBV = ORD == 2 ? 6 : 3;   // bra variants: 1, A, B, (AA, BB, AB)
  static constexpr int NV = ORD == 2 ? 10 : 4;   // all variants, see rys_ket
  static constexpr int NOUT = ORD == 2 ? 45 : 9;
  static constexpr int CB = ncart_of(LB), CC = ncart_of(LC), CD = ncart_of(LD);
  static constexpr int NCART = ncart_of(LA) * CB * CC * CD;
  // Strides are odd, so that threads on consecutive columns (f) or rows (ij) use different banks.
  static constexpr int FS = (F + 1) | 1;              // column stride of the 2-D tables
  static constexpr int GS = ((E + 1) * FS) | 1;       // 2-D integrals of one root and direction
  static constexpr int BS = (NBV * NB * FS) | 1;      // bra variants of one direction
  static constexpr int kRW = 2 * NR;
  static constexpr int kG2 = NR * 3 * GS;
  static constexpr int kBV = 3 * BS;
  static constexpr int kVT = NV * 3 * NX;
  static constexpr int kMain = kRW + kG2 + kBV + kVT;
  static constexpr int kWork = kMain > 2 * NCART ? kMain : 2 * NCART;
  static constexpr int kUsed = kWork + NCART + (ORD == 2 ? 46 : 0);
  // values per group of G threads: G above a multiple of 32, so that the groups of a warp working on
  // the same place of their tables use different banks (4-byte and 8-byte values alike)
  static constexpr int group(int G) { return kUsed + ((G - kUsed) % 32 + 32) % 32; }
};

// The packed 2-D table positions (x | y << 8 | z << 16) of Cartesian integral e of a class: ket tuple
// times NB plus bra tuple.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ int rys_index(int e) {
  constexpr int CB = ncart_of(LB), CC = ncart_of(LC), CD = ncart_of(LD), NB = (LA + 1) * (LB + 1);
  const int3 a = rys_comp(LA, e / (CB * CC * CD)), b = rys_comp(LB, e / (CC * CD) % CB);
  const int3 c = rys_comp(LC, e / CD % CC), d = rys_comp(LD, e % CD);
  auto at = [](int i, int j, int k, int l) { return (k * (LD + 1) + l) * NB + i * (LB + 1) + j; };
  return at(a.x, b.x, c.x, d.x) | at(a.y, b.y, c.y, d.y) << 8 | at(a.z, b.z, c.z, d.z) << 16;
}

// Vertical recurrence of the 2-D integrals of one root and direction: g[e FS + f].
template <int E, int F, int FS, typename R>
__device__ __forceinline__ void rys_vrr(R i00, R C, R Cp, R B00, R B10, R B01, R* __restrict__ g) {
  R prev2[E + 1], prev[E + 1], cur[E + 1];
  cur[0] = i00;
#pragma unroll
  for (int e = 1; e <= E; ++e) cur[e] = C * cur[e - 1] + (e > 1 ? R(e - 1) * B10 * cur[e - 2] : R(0));
#pragma unroll
  for (int e = 0; e <= E; ++e) g[e * FS] = cur[e];
#pragma unroll
  for (int f = 1; f <= F; ++f) {
#pragma unroll
    for (int e = 0; e <= E; ++e) {
      prev2[e] = f > 1 ? prev[e] : R(0);
      prev[e] = cur[e];
    }
#pragma unroll
    for (int e = 0; e <= E; ++e) {
      R v = Cp * prev[e];
      if (f > 1) v += R(f - 1) * B01 * prev2[e];
      if (e > 0) v += R(e) * B00 * prev[e - 1];
      cur[e] = v;
      g[e * FS + f] = v;
    }
  }
}

// Horizontal transfer of one index pair: h[i][j], i <= I, j <= J, i + j <= N, from h[i][0] = s[i].
template <int N, int I, int J, typename R>
__device__ __forceinline__ void rys_hrr(const R (&s)[N + 1], R d, R (&h)[N + 1][J + 1]) {
#pragma unroll
  for (int i = 0; i <= N; ++i) h[i][0] = s[i];
#pragma unroll
  for (int j = 1; j <= J; ++j)
#pragma unroll
    for (int i = 0; i <= N; ++i)
      if (i + j <= N) h[i][j] = h[i + 1][j - 1] + d * h[i][j - 1];
}

// Bra variants of one (direction, f): bv[(v NB + ij) FS], from the column g[e FS].
template <int LA, int LB, int ORD, int FS, typename R>
__device__ __forceinline__ void rys_bra(const R* __restrict__ g, R AB, R wa, R wb, R* __restrict__ bv) {
  constexpr int E = LA + LB + ORD, J = LB + ORD, NB = (LA + 1) * (LB + 1);
  R s[E + 1], h[E + 1][J + 1];
#pragma unroll
  for (int e = 0; e <= E; ++e) s[e] = g[e * FS];
  rys_hrr<E, E, J>(s, AB, h);
#pragma unroll
  for (int i = 0; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) {
      const int at = (i * (LB + 1) + j) * FS;
      auto put = [&](int v, R x) { bv[v * NB * FS + at] = x; };
      put(0, h[i][j]);
      R A = wa * h[i + 1][j], B = wb * h[i][j + 1];
      if (i > 0) A -= R(i) * h[i - 1][j];
      if (j > 0) B -= R(j) * h[i][j - 1];
      put(1, A);
      put(2, B);
      if constexpr (ORD == 2) {
        R AA = wa * (wa * h[i + 2][j] - R(2 * i + 1) * h[i][j]);
        if (i > 1) AA += R(i * (i - 1)) * h[i - 2][j];
        R BB = wb * (wb * h[i][j + 2] - R(2 * j + 1) * h[i][j]);
        if (j > 1) BB += R(j * (j - 1)) * h[i][j - 2];
        R x = wb * h[i + 1][j + 1];  // B of (i+1, j), then of (i-1, j)
        if (j > 0) x -= R(j) * h[i + 1][j - 1];
        R AB2 = wa * x;
        if (i > 0) {
          R y = wb * h[i - 1][j + 1];
          if (j > 0) y -= R(j) * h[i - 1][j - 1];
          AB2 -= R(i) * y;
        }
        put(3, AA);
        put(4, BB);
        put(5, AB2);
      }
    }
}

// Ket transfer and C derivatives of one (direction, bra tuple): variant v of ket tuple kl into
// vt[v VS + kl NB].  Variants: 0 1, 1 A, 2 B, 3 C; second order 4 AA, 5 BB, 6 CC, 7 AB, 8 AC, 9 BC.
template <int LC, int LD, int ORD, int NB, int FS, int VS, typename R>
__device__ __forceinline__ void rys_ket(const R* __restrict__ bv, R CD, R wc, R* __restrict__ vt) {
  auto transfer = [&](auto cord, int v, auto out) {
    constexpr int CO = decltype(cord)::value;  // C derivatives this bra variant still takes
    constexpr int N = LC + LD + CO;
    R s[N + 1], h[N + 1][LD + 1];
#pragma unroll
    for (int f = 0; f <= N; ++f) s[f] = bv[v * NB * FS + f];
    rys_hrr<N, N, LD>(s, CD, h);
#pragma unroll
    for (int k = 0; k <= LC; ++k)
#pragma unroll
      for (int l = 0; l <= LD; ++l) {
        R* o = vt + (k * (LD + 1) + l) * NB;
        o[out[0] * VS] = h[k][l];
        if constexpr (CO >= 1) {
          R c = wc * h[k + 1][l];
          if (k > 0) c -= R(k) * h[k - 1][l];
          o[out[1] * VS] = c;
        }
        if constexpr (CO >= 2) {
          R c = wc * (wc * h[k + 2][l] - R(2 * k + 1) * h[k][l]);
          if (k > 1) c += R(k * (k - 1)) * h[k - 2][l];
          o[out[2] * VS] = c;
        }
      }
  };
  struct Out {
    int i[3];
    __device__ constexpr int operator[](int k) const { return i[k]; }
  };
  if constexpr (ORD == 2) {
    transfer(std::integral_constant<int, 2>{}, 0, Out{{0, 3, 6}});
    transfer(std::integral_constant<int, 1>{}, 1, Out{{1, 8, 0}});
    transfer(std::integral_constant<int, 1>{}, 2, Out{{2, 9, 0}});
    transfer(std::integral_constant<int, 0>{}, 3, Out{{4, 0, 0}});
    transfer(std::integral_constant<int, 0>{}, 4, Out{{5, 0, 0}});
    transfer(std::integral_constant<int, 0>{}, 5, Out{{7, 0, 0}});
  } else {
    transfer(std::integral_constant<int, 1>{}, 0, Out{{0, 3, 0}});
    transfer(std::integral_constant<int, 0>{}, 1, Out{{1, 0, 0}});
    transfer(std::integral_constant<int, 0>{}, 2, Out{{2, 0, 0}});
  }
}

// Position of second derivative (P, Q) of one direction among the variants, P <= Q in A, B, C.
__host__ __device__ constexpr int rys_second(int P, int Q) {
  return P == Q ? 4 + P : 6 + P + Q;  // AB 7, AC 8, BC 9
}
// Position of (r, s), r <= s, in the 45-entry upper triangle of the 9 x 9 block (as hess_tri).
__host__ __device__ constexpr int rys_tri(int r, int s) { return r * 9 - r * (r - 1) / 2 + (s - r); }

// One integral's contribution to the sums: X, Y, Z its variants in the three directions.
template <int ORD, typename R, int NV, int NOUT>
__device__ __forceinline__ void rys_accumulate(R w, const R (&X)[NV], const R (&Y)[NV], const R (&Z)[NV],
                                               R (&acc)[NOUT]) {
  const R wx = w * X[0], wz = w * Z[0];
  const R yz = Y[0] * wz, xz = X[0] * wz, xy = wx * Y[0];
  if constexpr (ORD == 1) {
#pragma unroll
    for (int P = 0; P < 3; ++P) {
      acc[3 * P + 0] += X[1 + P] * yz;
      acc[3 * P + 1] += Y[1 + P] * xz;
      acc[3 * P + 2] += Z[1 + P] * xy;
    }
  } else {
    const R wy = w * Y[0];
#pragma unroll
    for (int P = 0; P < 3; ++P)
#pragma unroll
      for (int Q = P; Q < 3; ++Q) {
        const int v = rys_second(P, Q);
        acc[rys_tri(3 * P + 0, 3 * Q + 0)] += X[v] * yz;
        acc[rys_tri(3 * P + 1, 3 * Q + 1)] += Y[v] * xz;
        acc[rys_tri(3 * P + 2, 3 * Q + 2)] += Z[v] * xy;
      }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
      const R xp = X[1 + P] * wz, xq = X[1 + P] * wy, yp = Y[1 + P] * wx;
#pragma unroll
      for (int Q = 0; Q < 3; ++Q) {
        // (P, x) with (Q, y); (P, x) with (Q, z); (P, y) with (Q, z)
        const int rx = 3 * P, sy = 3 * Q + 1, sz = 3 * Q + 2, ry = 3 * P + 1;
        acc[rx < sy ? rys_tri(rx, sy) : rys_tri(sy, rx)] += xp * Y[1 + Q];
        acc[rx < sz ? rys_tri(rx, sz) : rys_tri(sz, rx)] += xq * Z[1 + Q];
        acc[ry < sz ? rys_tri(ry, sz) : rys_tri(sz, ry)] += yp * Z[1 + Q];
      }
    }
  }
}


// ---------------------------------------------------------------------------
// One thread per direction (hfgpu_rys3.cuh): thread d of a quartet's three owns direction d, calls it
// x, the next one y and the previous one z.  By cyclic symmetry every thread runs the same code on
// the Cartesian integrals with their components renamed.
// ---------------------------------------------------------------------------
// Index of component (lx, ly, lz = l - lx - ly) of a shell (order of gen_eri.py cart()).
__host__ __device__ constexpr int rys_cart(int l, int lx, int ly) {
  return (l - lx) * (l - lx + 1) / 2 + (l - lx - ly);
}

template <int LA, int LB, int LC, int LD, int ORD>
struct Rys3Dims {
  static constexpr int NR = (LA + LB + LC + LD + ORD) / 2 + 1;
  static constexpr int E = LA + LB + ORD, F = LC + LD + ORD;
  static constexpr int NB = (LA + 1) * (LB + 1), NK = (LC + 1) * (LD + 1), NX = NB * NK;
  static constexpr int CB = ncart_of(LB), CC = ncart_of(LC), CD = ncart_of(LD);
  static constexpr int NCART = ncart_of(LA) * CB * CC * CD;
  static constexpr int NSH = ORD == 2 ? 4 : 1;    // variants the other two directions read: 1 (A, B, C)
  static constexpr int NACC = ORD == 2 ? 15 : 3;  // sums of one thread
  static constexpr int at(int i, int j, int k, int l) { return ((i * (LB + 1) + j) * (LC + 1) + k) * (LD + 1) + l; }
  // shared memory of a warp's quartet: [roots and weights | the three directions' shared variants |
  // three renamed copies of W]; direction strides are 1 and the quartet's stride 3 above a
  // multiple of 16, so that consecutive threads (quartet, direction) use consecutive banks
  static constexpr int up(int n, int r) { return n + ((r - n) % 16 + 16) % 16; }
  static constexpr int DV = up(NSH * NX, 1), DW = up(NCART, 1);
  static constexpr int kV = 2 * NR, kW = kV + 3 * DV;
  static constexpr int kQuartet = up(kW + 3 * DW, 3);
};

// h[i][j] of the horizontal transfer from the column s[e] = h[e][0], j <= 4 (binomial form).
template <typename S, typename R>
__device__ __forceinline__ R rys_h(const S& s, R d, int i, int j) {
  R v = s(i);
  R c = R(1);
#pragma unroll
  for (int m = 1; m <= 4; ++m)
    if (m <= j) {
      c = c * R(j - m + 1) / R(m);
      v = c * s(i + m) + d * v;
    }
  return v;
}

// Variants (numbered as in rys_ket) of one direction for bra tuple (i, j) and every ket tuple:
// o[v][k (LD+1) + l], from the 2-D integrals g[e][f].  SECOND: all ten, else the first four.
template <int LA, int LB, int LC, int LD, int ORD, bool SECOND, typename R>
__device__ __forceinline__ void rys3_variants(const R (&g)[LA + LB + ORD + 1][LC + LD + ORD + 1], R AB, R CD, R wa, R wb,
                                              R wc, int i, int j,
                                              R (&o)[SECOND ? 10 : 4][(LC + 1) * (LD + 1)]) {
  constexpr int F = LC + LD + ORD;
  R u[SECOND ? 6 : 3][F + 1];
#pragma unroll
  for (int f = 0; f <= F; ++f) {
    auto s = [&](int e) { return g[e][f]; };
    auto h = [&](int a, int b) { return rys_h(s, AB, a, b); };
    u[0][f] = h(i, j);
    if (f <= F - 1) {
      R A = wa * h(i + 1, j), B = wb * h(i, j + 1);
      if (i > 0) A -= R(i) * h(i - 1, j);
      if (j > 0) B -= R(j) * h(i, j - 1);
      u[1][f] = A;
      u[2][f] = B;
    }
    if constexpr (SECOND) {
      if (f <= F - 2) {
        R AA = wa * (wa * h(i + 2, j) - R(2 * i + 1) * h(i, j)), BB = wb * (wb * h(i, j + 2) - R(2 * j + 1) * h(i, j));
        if (i > 1) AA += R(i * (i - 1)) * h(i - 2, j);
        if (j > 1) BB += R(j * (j - 1)) * h(i, j - 2);
        R x = wb * h(i + 1, j + 1);
        if (j > 0) x -= R(j) * h(i + 1, j - 1);
        R ab = wa * x;
        if (i > 0) {
          R y = wb * h(i - 1, j + 1);
          if (j > 0) y -= R(j) * h(i - 1, j - 1);
          ab -= R(i) * y;
        }
        u[3][f] = AA;
        u[4][f] = BB;
        u[5][f] = ab;
      }
    }
  }
#pragma unroll
  for (int k = 0; k <= LC; ++k)
#pragma unroll
    for (int l = 0; l <= LD; ++l) {
      const int x = k * (LD + 1) + l;
      auto h = [&](int v, int c, int d) {
        auto s = [&](int f) { return u[v][f]; };
        return rys_h(s, CD, c, d);
      };
      auto C = [&](int v) {
        R c = wc * h(v, k + 1, l);
        if (k > 0) c -= R(k) * h(v, k - 1, l);
        return c;
      };
      o[0][x] = h(0, k, l);
      o[1][x] = h(1, k, l);
      o[2][x] = h(2, k, l);
      o[3][x] = C(0);
      if constexpr (SECOND) {
        o[4][x] = h(3, k, l);
        o[5][x] = h(4, k, l);
        R cc = wc * (wc * h(0, k + 2, l) - R(2 * k + 1) * h(0, k, l));
        if (k > 1) cc += R(k * (k - 1)) * h(0, k - 2, l);
        o[6][x] = cc;
        o[7][x] = h(5, k, l);
        o[8][x] = C(1);
        o[9][x] = C(2);
      }
    }
}

// Adds the integrals whose own-direction exponents are (i, j) on the bra: o their own variants, n and
// m the next and previous direction's shared variants by tuple, W the renamed weights.  acc: order 1
// dA, dB, dC of the own direction; order 2 AA BB CC AB AC BC of the own direction, then (P own, Q next).
template <int LA, int LB, int LC, int LD, int ORD, typename R>
__device__ __forceinline__ void rys3_accumulate(const R (&o)[ORD == 2 ? 10 : 4][(LC + 1) * (LD + 1)], int i, int j,
                                                const R* n, const R* m, const R* W, R* acc) {
  using D = Rys3Dims<LA, LB, LC, LD, ORD>;
#pragma unroll
  for (int k = 0; k <= LC; ++k)
#pragma unroll
    for (int l = 0; l <= LD; ++l) {
      R S0 = R(0), S1[3] = {R(0), R(0), R(0)};
#pragma unroll
      for (int i2 = 0; i2 <= LA; ++i2)
#pragma unroll
        for (int j2 = 0; j2 <= LB; ++j2)
#pragma unroll
          for (int k2 = 0; k2 <= LC; ++k2)
#pragma unroll
            for (int l2 = 0; l2 <= LD; ++l2)
              if (i2 <= LA - i && j2 <= LB - j && k2 <= LC - k && l2 <= LD - l) {
                const int e = ((rys_cart(LA, i, i2) * D::CB + rys_cart(LB, j, j2)) * D::CC + rys_cart(LC, k, k2)) * D::CD +
                              rys_cart(LD, l, l2);
                const R wm = W[e] * m[D::at(LA - i - i2, LB - j - j2, LC - k - k2, LD - l - l2)];
                const int t = D::at(i2, j2, k2, l2);
                S0 += n[t] * wm;
                if constexpr (ORD == 2)
#pragma unroll
                  for (int Q = 0; Q < 3; ++Q) S1[Q] += n[(1 + Q) * D::NX + t] * wm;
              }
      const int x = k * (LD + 1) + l;
      if constexpr (ORD == 1) {
#pragma unroll
        for (int P = 0; P < 3; ++P) acc[P] += o[1 + P][x] * S0;
      } else {
#pragma unroll
        for (int v = 0; v < 6; ++v) acc[v] += o[4 + v][x] * S0;
#pragma unroll
        for (int P = 0; P < 3; ++P)
#pragma unroll
          for (int Q = 0; Q < 3; ++Q) acc[6 + 3 * P + Q] += o[1 + P][x] * S1[Q];
      }
    }
}

// Vertical recurrence of one root and direction into registers, g[e][f].
template <int E, int F, typename R>
__device__ __forceinline__ void rys3_vrr(R i00, R C, R Cp, R B00, R B10, R B01, R (&g)[E + 1][F + 1]) {
  g[0][0] = i00;
#pragma unroll
  for (int e = 1; e <= E; ++e) g[e][0] = C * g[e - 1][0] + (e > 1 ? R(e - 1) * B10 * g[e > 1 ? e - 2 : 0][0] : R(0));
#pragma unroll
  for (int f = 1; f <= F; ++f)
#pragma unroll
    for (int e = 0; e <= E; ++e) {
      R v = Cp * g[e][f - 1];
      if (f > 1) v += R(f - 1) * B01 * g[e][f > 1 ? f - 2 : 0];
      if (e > 0) v += R(e) * B00 * g[e > 0 ? e - 1 : 0][f - 1];
      g[e][f] = v;
    }
}

// ---------------------------------------------------------------------------
// Undifferentiated integrals (rys_quartet_kernel): a thread takes (a, c, d) component triples and all
// components of b, whose 2-D integrals lie next to each other in the tables.
// ---------------------------------------------------------------------------
template <int LA, int LB, int LC, int LD>
struct RysJKDims {
  static constexpr int NR = (LA + LB + LC + LD) / 2 + 1, E = LA + LB, F = LC + LD;
  static constexpr int NB = (LA + 1) * (LB + 1), NK = (LC + 1) * (LD + 1), NX = NB * NK;
  static constexpr int CA = ncart_of(LA), CB = ncart_of(LB), CC = ncart_of(LC), CD = ncart_of(LD);
  static constexpr int NCART = CA * CB * CC * CD, NT = CA * CC * CD;  // integrals, triples
  static constexpr int FS = (F + 1) | 1, GS = ((E + 1) * FS) | 1, BS = (NB * FS) | 1;
  // shared memory of a group: [roots and weights | 2-D integrals | bra-transferred | transferred], all
  // roots at once; afterwards the Cartesian block and its transform's scratch
  static constexpr int kRW = 2 * NR, kG2 = NR * 3 * GS, kBV = NR * 3 * BS, kVT = NR * 3 * NX;
  static constexpr int kUsed = kRW + kG2 + kBV + kVT > 2 * NCART ? kRW + kG2 + kBV + kVT : 2 * NCART;
  static constexpr int kGroup = kUsed | 1;
};

// Table positions (x | y << 10 | z << 20) of triple t = (a CC + c) CD + d, for b = s.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ int rys_triple(int t) {
  constexpr int CC = ncart_of(LC), CD = ncart_of(LD), NB = (LA + 1) * (LB + 1);
  const int3 a = rys_comp(LA, t / (CC * CD)), c = rys_comp(LC, t / CD % CC), d = rys_comp(LD, t % CD);
  auto at = [](int i, int k, int l) { return (k * (LD + 1) + l) * NB + i * (LB + 1); };
  return at(a.x, c.x, d.x) | at(a.y, c.y, d.y) << 10 | at(a.z, c.z, d.z) << 20;
}

// Bra transfer of one column: bv[(i (LB+1) + j) FS] = h[i][j] from g[e FS].
template <int LA, int LB, int FS, typename R>
__device__ __forceinline__ void rys_jk_bra(const R* __restrict__ g, R AB, R* __restrict__ bv) {
  constexpr int E = LA + LB;
  R s[E + 1], h[E + 1][LB + 1];
#pragma unroll
  for (int e = 0; e <= E; ++e) s[e] = g[e * FS];
  rys_hrr<E, E, LB>(s, AB, h);
#pragma unroll
  for (int i = 0; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) bv[(i * (LB + 1) + j) * FS] = h[i][j];
}

// Ket transfer of one bra tuple: vt[(k (LD+1) + l) NB] from the row bv[f].
template <int LC, int LD, int NB, typename R>
__device__ __forceinline__ void rys_jk_ket(const R* __restrict__ bv, R CD, R* __restrict__ vt) {
  constexpr int F = LC + LD;
  R s[F + 1], h[F + 1][LD + 1];
#pragma unroll
  for (int f = 0; f <= F; ++f) s[f] = bv[f];
  rys_hrr<F, F, LD>(s, CD, h);
#pragma unroll
  for (int k = 0; k <= LC; ++k)
#pragma unroll
    for (int l = 0; l <= LD; ++l) vt[(k * (LD + 1) + l) * NB] = h[k][l];
}

// Adds one root's contribution to the CB integrals of a triple: x, y, z its rows of the tables.
template <int LB, typename R, int CB>
__device__ __forceinline__ void rys_jk_triple(const R* __restrict__ x, const R* __restrict__ y,
                                              const R* __restrict__ z, R (&acc)[CB]) {
  R X[LB + 1], Y[LB + 1], Z[LB + 1];
#pragma unroll
  for (int j = 0; j <= LB; ++j) {
    X[j] = x[j];
    Y[j] = y[j];
    Z[j] = z[j];
  }
#pragma unroll
  for (int i = 0; i <= LB; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) acc[i * (i + 1) / 2 + j] += X[LB - i] * Y[i - j] * Z[j];
}
