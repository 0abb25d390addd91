// J/K (and packed, Schwarz) kernel of the large classes by Rys quadrature: one warp per quartet.
//
// The recurrences on contracted classes hold 324-1296 Cartesian integrals and as many intermediates
// per quartet; one thread per quartet spills them and one warp per quartet over op tables waits for
// table rows.  Here a warp keeps the transferred 2-D integrals of all roots in shared memory (0.5-10 KB)
// and every lane sums its integrals over roots and primitive quartets in registers, in triples
// (a, c, d) with all components of b: LB + 1 neighbouring loads per direction serve 3 or 6 integrals.
#pragma once
#include "hfgpu_kernels.cuh"
#include "hfgpu_rys_math.cuh"

template <int LA, int LB, int LC, int LD, int BLOCK>
__global__ void __launch_bounds__(BLOCK) rys_quartet_kernel(QuartetArgs<double> qa, const double* __restrict__ rys_tab,
                                                            const int2* __restrict__ quartets, int nq) {
  using D = RysJKDims<LA, LB, LC, LD>;
  using R = double;
  extern __shared__ __align__(16) unsigned char rys_sm[];
  constexpr int WARPS = BLOCK / 32, KT = (D::NT + 31) / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  R* rw = reinterpret_cast<R*>(rys_sm) + (size_t)warp * D::kGroup;
  R* g2 = rw + D::kRW;
  R* bv = g2 + D::kG2;
  R* vt = bv + D::kBV;
  int* tab = reinterpret_cast<int*>(reinterpret_cast<R*>(rys_sm) + (size_t)WARPS * D::kGroup);
  for (int t = threadIdx.x; t < D::NT; t += BLOCK) tab[t] = rys_triple<LA, LB, LC, LD>(t);
  __syncthreads();
  const JKArgs<R>& a = qa.jk;
  nq = launch_count(qa, nq);
  for (long long qi = rys_first(blockIdx.x, WARPS, warp, 1); qi < nq; qi += rys_stride(gridDim.x, WARPS, 1)) {
    const int2 pq = quartets[quartet_slot(qa, (int)qi)];
    const PairInfo P = a.pairs[pq.x];
    const PairInfo Q = a.pairs[pq.y];
    bool skip = false;
    if (qa.mode == QMODE_JK && a.dmax != nullptr) {
      const float* dm = a.dmax;
      const int ns = a.nshell;
      float m = 4.f * fmaxf(dm[P.sa * ns + P.sb], dm[Q.sa * ns + Q.sb]);
      m = fmaxf(m, fmaxf(fmaxf(dm[P.sa * ns + Q.sa], dm[P.sa * ns + Q.sb]), fmaxf(dm[P.sb * ns + Q.sa], dm[P.sb * ns + Q.sb])));
      skip = P.schwarz * Q.schwarz * double(m) < a.dtol;
    }
    if (a.counters != nullptr && lane == 0) {
      atomicAdd(a.counters + (skip ? 1 : 0), 1ull);
      if (!skip) atomicAdd(a.counters + 2, (unsigned long long)(P.nprim * Q.nprim));
    }
    if (skip) continue;
    R acc[KT][D::CB];
#pragma unroll
    for (int k = 0; k < KT; ++k)
#pragma unroll
      for (int b = 0; b < D::CB; ++b) acc[k][b] = R(0);
    const PrimPair<R>* bp = a.prims + P.prim_off;
    const PrimPair<R>* kp = a.prims + Q.prim_off;
    for (int ib = 0; ib < P.nprim; ++ib)
      for (int ik = 0; ik < Q.nprim; ++ik) {
        const R p = bp[ib].p, ip = bp[ib].ip, q = kp[ik].p, iq = kp[ik].ip;
        const R rs = rsqrt_t(p + q);
        const R ipq = rs * rs;
        const R PQx = bp[ib].Px - kp[ik].Px, PQy = bp[ib].Py - kp[ik].Py, PQz = bp[ib].Pz - kp[ik].Pz;
        const R T = p * q * ipq * (PQx * PQx + PQy * PQy + PQz * PQz);
        const R pre = bp[ib].Kp * kp[ik].Kp * rs;
        if (lane < D::kRW) {
          const R f = rys_value<D::NR>(rys_tab, T, lane);
          rw[lane] = lane < D::NR ? f : f * pre;
        }
        __syncwarp();
        if (lane < 3 * D::NR) {
          const int r = lane / 3, d = lane - 3 * r;
          const R B00 = R(0.5) * rw[r] * ipq, u = R(2) * B00 * (d == 0 ? PQx : (d == 1 ? PQy : PQz));
          rys_vrr<D::E, D::F, D::FS>(d == 2 ? rw[D::NR + r] : R(1), (&bp[ib].PAx)[d] - q * u, (&kp[ik].PAx)[d] + p * u,
                                     B00, ip * (R(0.5) - B00 * q), iq * (R(0.5) - B00 * p), g2 + lane * D::GS);
        }
        __syncwarp();
        for (int it = lane; it < 3 * D::NR * (D::F + 1); it += 32) {
          const int rd = it / (D::F + 1), f = it - rd * (D::F + 1), d = rd % 3;
          rys_jk_bra<LA, LB, D::FS>(g2 + rd * D::GS + f, d == 0 ? P.ABx : (d == 1 ? P.ABy : P.ABz), bv + rd * D::BS + f);
        }
        __syncwarp();
        for (int it = lane; it < 3 * D::NR * D::NB; it += 32) {
          const int rd = it / D::NB, ij = it - rd * D::NB, d = rd % 3;
          rys_jk_ket<LC, LD, D::NB>(bv + rd * D::BS + ij * D::FS, d == 0 ? Q.ABx : (d == 1 ? Q.ABy : Q.ABz),
                                    vt + rd * D::NX + ij);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < KT; ++k)
          if ((k + 1) * 32 <= D::NT || k * 32 + lane < D::NT) {
            const int t = tab[k * 32 + lane];
            const R* x = vt + (t & 1023);
            const R* y = vt + D::NX + (t >> 10 & 1023);
            const R* z = vt + 2 * D::NX + (t >> 20);
#pragma unroll
            for (int r = 0; r < D::NR; ++r)
              rys_jk_triple<LB>(x + r * 3 * D::NX, y + r * 3 * D::NX, z + r * 3 * D::NX, acc[k]);
          }
        __syncwarp();  // the tables are read no more
      }
    R* A = rw;
#pragma unroll
    for (int k = 0; k < KT; ++k)
      if ((k + 1) * 32 <= D::NT || k * 32 + lane < D::NT) {
        const int t = k * 32 + lane, ca = t / (D::CC * D::CD), cd = t - ca * D::CC * D::CD;
#pragma unroll
        for (int b = 0; b < D::CB; ++b) A[(ca * D::CB + b) * D::CC * D::CD + cd] = acc[k][b];
      }
    __syncwarp();
    group_finish<LA, LB, LC, LD, R, 32>(qa, pq, P, Q, A, A + D::NCART, nullptr, lane);
    __syncwarp();
  }
}

template <int LA, int LB, int LC, int LD>
static bool launch_rys_quartet(const QuartetArgs<double>& a, const double* tab, const int2* q, int nq, cudaStream_t s) {
  if (nq <= 0) return true;
  using D = RysJKDims<LA, LB, LC, LD>;
  constexpr int BLOCK = 64;
  const size_t bytes = (size_t)(BLOCK / 32) * D::kGroup * sizeof(double) + (size_t)D::NT * sizeof(int);
  auto k = rys_quartet_kernel<LA, LB, LC, LD, BLOCK>;
  if (bytes > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return false;
  k<<<rys_blocks(nq, BLOCK / 32, 1, 0), BLOCK, bytes, s>>>(a, tab, q, nq);
  return true;
}
