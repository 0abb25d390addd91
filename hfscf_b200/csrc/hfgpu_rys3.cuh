// The Rys-quadrature derivatives of hfgpu_rys.cuh for the small classes: three threads per quartet,
// one per direction, with the 2-D integrals and their derivative variants in registers.
//
// A group of threads over shared-memory tables moves about 30 table values per 60 arithmetic
// instructions through the shared-memory pipe, which ran 80-97% busy at 17-25% of the FP64 pipe.  Here
// a thread builds the tables of its own direction in registers and shares only the value and first
// derivatives of its 2-D integrals (4 of 10 variants; the value alone for a gradient) with the other
// two.  It sums the derivatives of its own direction and the mixed ones with the next direction, as
// sums over the other two directions first: 5 operations per integral and 15 per own tuple.
// Ten quartets per warp; two lanes repeat the work of another pair.
#pragma once
#include "hfgpu_rys.cuh"

// SPLIT = 10: a warp takes one quartet, its ten thread triples every tenth primitive quartet, for launches
// of few quartets, which would otherwise wait for the longest quartet's primitive loop.
template <int LA, int LB, int LC, int LD, int ORD, typename R, int BLOCK, int SPLIT>
__global__ void __launch_bounds__(BLOCK) rys3_kernel(GradArgs<R> a, RysOut o, int pure,
                                                     const int2* __restrict__ quartets, int nq) {
  using D = Rys3Dims<LA, LB, LC, LD, ORD>;
  extern __shared__ __align__(16) unsigned char rys_sm[];
  static_assert(SPLIT == 1 || SPLIT == 10, "triples per quartet");
  constexpr int WARPS = BLOCK / 32, SLOTS = 10, QW = SLOTS / SPLIT;  // thread triples and quartets per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = lane < 30 ? lane / 3 : 9, d = lane % 3, nd = (d + 1) % 3, pd = (d + 2) % 3;
  double* gsum = reinterpret_cast<double*>(rys_sm);
  R* base = reinterpret_cast<R*>(gsum + (ORD == 1 ? 3 * o.smem_atoms : 0)) + (size_t)warp * SLOTS * D::kQuartet;
  R* rw = base + (size_t)slot * D::kQuartet;
  R* V = rw + D::kV;
  R* W0 = rw + D::kW + 2 * D::DW;                       // d = 0: the weights as they are
  R* W = d == 0 ? W0 : rw + D::kW + (d - 1) * D::DW;    // renamed for this thread's direction
  // source of the renamed weights: integral e in own, next, previous order
  int* rot = reinterpret_cast<int*>(reinterpret_cast<R*>(gsum + (ORD == 1 ? 3 * o.smem_atoms : 0)) +
                                    (size_t)WARPS * SLOTS * D::kQuartet);
  for (int x = threadIdx.x; x < 2 * D::NCART; x += BLOCK) {
    const int e = x % D::NCART, r = x < D::NCART ? 1 : 2;
    auto back = [&](int l, int c) {  // component with own, next, previous exponents at r, r + 1, r + 2
      const int3 v = rys_comp(l, c);
      return r == 1 ? rys_cart(l, v.z, v.x) : rys_cart(l, v.y, v.z);
    };
    rot[x] = ((back(LA, e / (D::CB * D::CC * D::CD)) * D::CB + back(LB, e / (D::CC * D::CD) % D::CB)) * D::CC +
              back(LC, e / D::CD % D::CC)) * D::CD + back(LD, e % D::CD);
  }
  if (ORD == 1)
    for (int i = threadIdx.x; i < 3 * o.smem_atoms; i += BLOCK) gsum[i] = 0.0;
  __syncthreads();
  const int np = a.nparts > 1 ? a.nparts : 1, p0 = np > 1 ? a.part : 0;
  for (long long q0 = rys_first(blockIdx.x, WARPS, warp, QW); q0 < nq; q0 += rys_stride(gridDim.x, WARPS, QW)) {
    const long long qi = q0 + slot / SPLIT;
    const bool live = qi < nq;
    const int2 pq = quartets[(size_t)(live ? qi : nq - 1) * np + p0];
    const PairInfo P = a.pairs[pq.x];
    const PairInfo Q = a.pairs[pq.y];
    double s8 = 8.0;
    if (P.sa == P.sb) s8 *= 0.5;
    if (Q.sa == Q.sb) s8 *= 0.5;
    if (pq.x == pq.y) s8 *= 0.5;
    rys_weights<LA, LB, LC, LD, 3, R>(a, pure, P, Q, s8, d, W0, rw);
    if (d > 0)
      for (int e = 0; e < D::NCART; ++e) W[e] = W0[rot[(d - 1) * D::NCART + e]];
    // this triple's primitive quartets: first, first + SPLIT, ...
    const int all = live ? P.nprim * Q.nprim : 0, first = SPLIT > 1 ? slot : 0;
    const int mine = SPLIT > 1 ? (all > first ? (all - first + SPLIT - 1) / SPLIT : 0) : all;
    const int bo = mine > 0 ? P.prim_off : 0, ko = mine > 0 ? Q.prim_off : 0;
    const PrimPair<R>* bp = a.prims + bo;
    const PrimPair<R>* kp = a.prims + ko;
    const R AB = R(d == 0 ? P.ABx : (d == 1 ? P.ABy : P.ABz)), CD = R(d == 0 ? Q.ABx : (d == 1 ? Q.ABy : Q.ABz));
    R acc[D::NACC];
#pragma unroll
    for (int x = 0; x < D::NACC; ++x) acc[x] = R(0);
    int most = mine;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, off));
    int ib = 0, ik = 0;
    if (SPLIT > 1 && mine > 0) {
      ib = first / Q.nprim;
      ik = first - ib * Q.nprim;
    }
    for (int x = 0; x < most; ++x) {
      const bool on = x < mine;  // quartets with fewer primitive quartets add zeros
      const R p = bp[ib].p, ip = bp[ib].ip, q = kp[ik].p, iq = kp[ik].ip;
      const R wa = R(2) * a.alpha_a[bo + ib], wb = R(2) * a.alpha_b[bo + ib], wc = R(2) * a.alpha_a[ko + ik];
      const R rs = rsqrt_t(p + q);
      const R ipq = rs * rs;
      const R PQx = bp[ib].Px - kp[ik].Px, PQy = bp[ib].Py - kp[ik].Py, PQz = bp[ib].Pz - kp[ik].Pz;
      const R T = p * q * ipq * (PQx * PQx + PQy * PQy + PQz * PQz);
      const R pre = on ? bp[ib].Kp * kp[ik].Kp * rs : R(0);
      const R PQd = d == 0 ? PQx : (d == 1 ? PQy : PQz);
      const R PA = (&bp[ib].PAx)[d], QC = (&kp[ik].PAx)[d];
#pragma unroll
      for (int v = 0; v < (2 * D::NR + 2) / 3; ++v)
        if (3 * v + d < 2 * D::NR) {
          const R f = R(rys_value<D::NR>(o.tab, double(T), 3 * v + d));
          rw[3 * v + d] = 3 * v + d < D::NR ? f : f * pre;
        }
      __syncwarp();
#pragma unroll 1
      for (int r = 0; r < D::NR; ++r) {
        R g[D::E + 1][D::F + 1];
        {
          const R B00 = R(0.5) * rw[r] * ipq, u = R(2) * B00 * PQd;
          rys3_vrr<D::E, D::F>(d == 2 ? rw[D::NR + r] : R(1), PA - q * u, QC + p * u, B00, ip * (R(0.5) - B00 * q),
                               iq * (R(0.5) - B00 * p), g);
        }
        // this direction's shared variants
#pragma unroll
        for (int i = 0; i <= LA; ++i)
#pragma unroll
          for (int j = 0; j <= LB; ++j) {
            R w[4][D::NK];
            rys3_variants<LA, LB, LC, LD, ORD, false>(g, AB, CD, wa, wb, wc, i, j, w);
#pragma unroll
            for (int v = 0; v < D::NSH; ++v)
#pragma unroll
              for (int kl = 0; kl < D::NK; ++kl) V[d * D::DV + v * D::NX + (i * (LB + 1) + j) * D::NK + kl] = w[v][kl];
          }
        __syncwarp();
        R n[D::NSH * D::NX], m[D::NX];
#pragma unroll
        for (int t = 0; t < D::NSH * D::NX; ++t) n[t] = V[nd * D::DV + t];
#pragma unroll
        for (int t = 0; t < D::NX; ++t) m[t] = V[pd * D::DV + t];
        __syncwarp();
#pragma unroll
        for (int i = 0; i <= LA; ++i)
#pragma unroll
          for (int j = 0; j <= LB; ++j) {
            R w[ORD == 2 ? 10 : 4][D::NK];
            rys3_variants<LA, LB, LC, LD, ORD, ORD == 2>(g, AB, CD, wa, wb, wc, i, j, w);
            rys3_accumulate<LA, LB, LC, LD, ORD>(w, i, j, n, m, W, acc);
          }
      }
      __syncwarp();  // the roots are read no more
      if (x + 1 < mine) {
        ik += SPLIT;
        while (ik >= Q.nprim) {
          ik -= Q.nprim;
          ++ib;
        }
      }
    }
    if constexpr (SPLIT > 1) {  // sum over the triples into lanes 0-2 (lanes 30 and 31 repeat others)
#pragma unroll
      for (int x = 0; x < D::NACC; ++x) {
        R v = acc[x];
        v += __shfl_down_sync(0xffffffffu, v, 15);
        const R v1 = __shfl_down_sync(0xffffffffu, v, 3), v2 = __shfl_down_sync(0xffffffffu, v, 6);
        const R v3 = __shfl_down_sync(0xffffffffu, v, 9), v4 = __shfl_down_sync(0xffffffffu, v, 12);
        acc[x] = v + v1 + v2 + v3 + v4;
      }
    }
    const bool lead = lane < 30 && slot % SPLIT == 0;  // holds its quartet's sums
    if constexpr (ORD == 1) {
      if (lead && live) {
        double* gout = (o.smem_atoms > 0 ? gsum : a.grad) + d;
        const double gA = double(acc[0]), gB = double(acc[1]), gC = double(acc[2]);
        atomicAdd(gout + 3 * P.atom_a, gA);
        atomicAdd(gout + 3 * P.atom_b, gB);
        atomicAdd(gout + 3 * Q.atom_a, gC);
        atomicAdd(gout + 3 * Q.atom_b, -(gA + gB + gC));
      }
    } else {
      // the 45 entries of each quartet to shared memory, then into the output warp-wide
      R* h45 = base + (size_t)slot * 45;
      if (SPLIT == 1 || lead)
#pragma unroll
      for (int A = 0; A < 3; ++A)
#pragma unroll
        for (int B = 0; B < 3; ++B) {
          if (A <= B) h45[rys_tri(3 * A + d, 3 * B + d)] = acc[rys_second(A, B) - 4];
          const int r = 3 * A + d, c = 3 * B + nd;
          h45[r < c ? rys_tri(r, c) : rys_tri(c, r)] = acc[6 + 3 * A + B];
        }
      const int at[4] = {P.atom_a, P.atom_b, Q.atom_a, Q.atom_b};
      hess_add_warp(lead && d == 0 && live, base, 1, 15, at, hess_copy(o.hess, o.natoms, o.copies), 3 * o.natoms);
    }
    __syncwarp();
  }
  if (ORD == 1 && o.smem_atoms > 0) {
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * o.smem_atoms; i += BLOCK)
      if (gsum[i] != 0.0) atomicAdd(a.grad + i, gsum[i]);
  }
}

template <int LA, int LB, int LC, int LD, int ORD, typename R, int SPLIT>
static bool launch_rys3(const GradArgs<R>& a, const RysOut& o, int pure, const int2* q, int nq, int max_blocks,
                        cudaStream_t s) {
  if (nq <= 0) return true;
  using D = Rys3Dims<LA, LB, LC, LD, ORD>;
  constexpr int BLOCK = 64, SLOTS = BLOCK / 32 * 10, QB = SLOTS / SPLIT;
  constexpr size_t kTables = (size_t)SLOTS * D::kQuartet * sizeof(R) + 2 * (size_t)D::NCART * sizeof(int);
  const size_t bytes = kTables + (ORD == 1 ? 3 * sizeof(double) * (size_t)o.smem_atoms : 0);
  auto k = rys3_kernel<LA, LB, LC, LD, ORD, R, BLOCK, SPLIT>;
  if (!allow_shared<kTables + (ORD == 1 ? kGradSmemBytes : 0)>(k, bytes)) return false;
  k<<<rys_blocks(nq, 1, QB, max_blocks), BLOCK, bytes, s>>>(a, o, pure, q, nq);
  return true;
}
