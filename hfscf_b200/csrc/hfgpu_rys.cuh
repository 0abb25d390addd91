// Derivative integrals by Rys quadrature, contracted with the density weights on the fly.
//
// (ab|cd) = pre sum_i w_i Ix(t_i) Iy(t_i) Iz(t_i) (Dupuis, Rys & King, J. Chem. Phys. 65, 111
// (1976)): every Cartesian integral of a primitive quartet is a sum over a few roots of products
// of two-dimensional integrals, and a derivative acts on one factor only.  A group of G threads
// shares one quartet.  Per primitive quartet it evaluates the roots, runs the vertical recurrence
// of the 2-D integrals (one thread per root and direction), and per root builds the tables of the
// transferred 2-D integrals in every derivative variant (1, A, B, C, and for second derivatives
// AA, BB, CC, AB, AC, BC) in shared memory; then each thread takes integrals (a b c d) and adds
// W_abcd times the products of variants into its own 9 (gradient) or 45 (Hessian) sums, which are
// reduced over the group once per quartet.  The centre D follows from translational invariance.
//
// Why this form: the recurrences on contracted Cartesian classes hold hundreds to thousands of
// intermediates per quartet (24 k table rows for a (dp|pp) Hessian), which spill or run from
// op tables; here the state of a root is a few hundred table entries whatever the class, the code
// is compact, and the inner loop is register arithmetic on broadcast-friendly shared-memory loads.
#pragma once
#include "hfgpu_hess_kernels.cuh"
#include "hfgpu_rys_math.cuh"

// Synchronises the threads of a group: G <= 32 the whole warp (its groups run in step), else the
// block, which is one group.
template <int G>
__device__ __forceinline__ void rys_sync() {
  if constexpr (G <= 32)
    __syncwarp();
  else
    __syncthreads();
}

// Weight block of a quartet, Cartesian, into W (see grad_weights for its definition); t: scratch of
// 2 NCART values for a pure basis.
template <int LA, int LB, int LC, int LD, int G, typename R>
__device__ __forceinline__ void rys_weights(const GradArgs<R>& a, int pure, const PairInfo& P, const PairInfo& Q,
                                            double s8, int lane, R* W, R* t) {
  constexpr int Ls[4] = {LA, LB, LC, LD};
  constexpr int NCART = ncart_of(LA) * ncart_of(LB) * ncart_of(LC) * ncart_of(LD);
  int dims[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) dims[q] = pure ? npure_of(Ls[q]) : ncart_of(Ls[q]);
  long long blk;
  int nm;
  mol_block(a.mol_off, a.mol_n, P.mol, a.n, blk, nm);
  const double* DJ = off_ptr(a.DJ, blk);
  const double* DK = off_ptr(a.DK, blk);
  const int tot = dims[0] * dims[1] * dims[2] * dims[3];
  R* dst = pure ? t : W;
  for (int e = lane; e < tot; e += G) {
    const int l = e % dims[3], k = (e / dims[3]) % dims[2], j = (e / (dims[3] * dims[2])) % dims[1];
    const int i = e / (dims[3] * dims[2] * dims[1]);
    const int ia = P.fa + i, jb = P.fb + j, kc = Q.fa + k, ld = Q.fb + l;
    double w = DJ ? a.cJ * __ldg(DJ + (size_t)ia * nm + jb) * __ldg(DJ + (size_t)kc * nm + ld) : 0.0;
    for (int m = 0; m < a.nK; ++m) {
      const double* D = DK + (size_t)m * nm * nm;
      w -= 0.5 * a.cK *
           (__ldg(D + (size_t)ia * nm + kc) * __ldg(D + (size_t)jb * nm + ld) +
            __ldg(D + (size_t)ia * nm + ld) * __ldg(D + (size_t)jb * nm + kc));
    }
    dst[e] = R(s8 * w);
  }
  rys_sync<G>();
  if (!pure) return;
  const R* in = t;
#pragma unroll
  for (int st = 0; st < 4; ++st) {
    const int nc = ncart_of(Ls[st]), np = npure_of(Ls[st]);
    R* o = st == 3 ? W : (st & 1 ? t : t + NCART);
    int nd[4] = {dims[0], dims[1], dims[2], dims[3]};
    nd[st] = nc;
    const int n = nd[0] * nd[1] * nd[2] * nd[3];
    for (int e = lane; e < n; e += G) {
      int id[4];
      int r = e;
#pragma unroll
      for (int q = 3; q >= 0; --q) {
        id[q] = r % nd[q];
        r /= nd[q];
      }
      R v = R(0);
      for (int c = 0; c < np; ++c) {
        const double y = c_ylm[Ls[st]][id[st] * np + c];
        if (y == 0.0) continue;
        int jd[4] = {id[0], id[1], id[2], id[3]};
        jd[st] = c;
        v += R(y) * in[((jd[0] * dims[1] + jd[1]) * dims[2] + jd[2]) * dims[3] + jd[3]];
      }
      o[e] = v;
    }
    rys_sync<G>();
#pragma unroll
    for (int q = 0; q < 4; ++q) dims[q] = nd[q];
    in = o;
  }
}

// Output of a launch: order 1 GradArgs::grad; order 2 hess and copies as in HessOut.
struct RysOut {
  const double* __restrict__ tab;  // quadrature tables
  double* __restrict__ hess;
  int natoms;
  int smem_atoms;  // order 1: > 0 = the block sums its 3 x smem_atoms entries in shared memory first
  int copies;
};

// G threads per quartet, BLOCK threads per block (BLOCK = G when G > 32), grid-stride over quartets.
// Dynamic shared memory: [BLOCK / G groups of RysDims::group(G) values | NCART packed 2-D indexes of
// the integrals | order 1: 3 smem_atoms doubles].
template <int LA, int LB, int LC, int LD, int ORD, typename R, int G, int BLOCK>
__global__ void __launch_bounds__(BLOCK) rys_deriv_kernel(GradArgs<R> a, RysOut o, int pure,
                                                          const int2* __restrict__ quartets, int nq) {
  using D = RysDims<LA, LB, LC, LD, ORD>;
  static_assert(G <= 32 ? (BLOCK % 32 == 0 && 32 % G == 0) : BLOCK == G, "group size");
  extern __shared__ __align__(16) unsigned char rys_sm[];
  constexpr int GROUPS = BLOCK / G;
  const int lane = threadIdx.x % G, grp = threadIdx.x / G;
  double* gsum = reinterpret_cast<double*>(rys_sm);
  R* rw = reinterpret_cast<R*>(gsum + (ORD == 1 ? 3 * o.smem_atoms : 0)) + (size_t)grp * D::group(G);
  R* g2 = rw + D::kRW;
  R* bv = g2 + D::kG2;
  R* vt = bv + D::kBV;
  R* W = rw + D::kWork;
  int* tab = reinterpret_cast<int*>(rw + (size_t)(GROUPS - grp) * D::group(G));
  for (int e = threadIdx.x; e < D::NCART; e += BLOCK) tab[e] = rys_index<LA, LB, LC, LD>(e);
  if (ORD == 1)
    for (int i = threadIdx.x; i < 3 * o.smem_atoms; i += BLOCK) gsum[i] = 0.0;
  __syncthreads();
  const int np = a.nparts > 1 ? a.nparts : 1, p0 = np > 1 ? a.part : 0;
  for (long long q0 = rys_first(blockIdx.x, 1, 0, GROUPS); q0 < nq; q0 += rys_stride(gridDim.x, 1, GROUPS)) {
    // groups of a warp run in step: one past the end works on quartet nq - 1 with no primitives
    const bool live = q0 + grp < nq;
    const int2 pq = quartets[(size_t)(live ? q0 + grp : nq - 1) * np + p0];
    const PairInfo P = a.pairs[pq.x];
    const PairInfo Q = a.pairs[pq.y];
    double s8 = 8.0;
    if (P.sa == P.sb) s8 *= 0.5;
    if (Q.sa == Q.sb) s8 *= 0.5;
    if (pq.x == pq.y) s8 *= 0.5;
    rys_weights<LA, LB, LC, LD, G, R>(a, pure, P, Q, s8, lane, W, rw);
    const int mine = live ? P.nprim * Q.nprim : 0;
    // (a group without primitive quartets reads pair 0 and adds zeros)
    const int bo = mine > 0 ? P.prim_off : 0, ko = mine > 0 ? Q.prim_off : 0;
    const PrimPair<R>* bp = a.prims + bo;
    const PrimPair<R>* kp = a.prims + ko;
    const R ABx = R(P.ABx), ABy = R(P.ABy), ABz = R(P.ABz), CDx = R(Q.ABx), CDy = R(Q.ABy), CDz = R(Q.ABz);
    R acc[D::NOUT];
#pragma unroll
    for (int x = 0; x < D::NOUT; ++x) acc[x] = R(0);
    int most = mine;
    if constexpr (G < 32) {
#pragma unroll
      for (int off = 16; off >= G; off >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, off));
    }
    int ib = 0, ik = 0;
    for (int x = 0; x < most; ++x) {
      const bool on = G >= 32 || x < mine;  // groups with fewer primitive quartets add zeros
      const R p = bp[ib].p, ip = bp[ib].ip, q = kp[ik].p, iq = kp[ik].ip;
      const R wa = R(2) * a.alpha_a[bo + ib], wb = R(2) * a.alpha_b[bo + ib];
      const R wc = R(2) * a.alpha_a[ko + ik];
      const R rs = rsqrt_t(p + q);
      const R ipq = rs * rs;
      const R PQx = bp[ib].Px - kp[ik].Px, PQy = bp[ib].Py - kp[ik].Py, PQz = bp[ib].Pz - kp[ik].Pz;
      const R T = p * q * ipq * (PQx * PQx + PQy * PQy + PQz * PQz);
      const R pre = on ? bp[ib].Kp * kp[ik].Kp * rs : R(0);
      for (int v = lane; v < D::kRW; v += G) {
        const R f = R(rys_value<D::NR>(o.tab, double(T), v));
        rw[v] = v < D::NR ? f : f * pre;
      }
      rys_sync<G>();
      for (int it = lane; it < 3 * D::NR; it += G) {
        const int r = it / 3, d = it - 3 * r;
        const R t2 = rw[r];
        const R B00 = R(0.5) * t2 * ipq;
        const R B10 = ip * (R(0.5) - B00 * q), B01 = iq * (R(0.5) - B00 * p);
        const R PQd = d == 0 ? PQx : (d == 1 ? PQy : PQz);
        const R PA = d == 0 ? bp[ib].PAx : (d == 1 ? bp[ib].PAy : bp[ib].PAz);
        const R QC = d == 0 ? kp[ik].PAx : (d == 1 ? kp[ik].PAy : kp[ik].PAz);
        const R u = R(2) * B00 * PQd;
        rys_vrr<D::E, D::F, D::FS>(d == 2 ? rw[D::NR + r] : R(1), PA - q * u, QC + p * u, B00, B10, B01,
                                   g2 + it * D::GS);
      }
      rys_sync<G>();
      for (int r = 0; r < D::NR; ++r) {
        for (int it = lane; it < 3 * (D::F + 1); it += G) {
          const int d = it / (D::F + 1), f = it - d * (D::F + 1);
          rys_bra<LA, LB, ORD, D::FS>(g2 + (r * 3 + d) * D::GS + f, d == 0 ? ABx : (d == 1 ? ABy : ABz), wa, wb,
                                      bv + d * D::BS + f);
        }
        rys_sync<G>();  // also: every thread is done with the previous root's variant tables
        for (int it = lane; it < 3 * D::NB; it += G) {
          const int d = it / D::NB, ij = it - d * D::NB;
          rys_ket<LC, LD, ORD, D::NB, D::FS, 3 * D::NX>(bv + d * D::BS + ij * D::FS,
                                                        d == 0 ? CDx : (d == 1 ? CDy : CDz), wc, vt + d * D::NX + ij);
        }
        rys_sync<G>();
        for (int e = lane; e < D::NCART; e += G) {
          const int t = tab[e];
          const R* vx = vt + (t & 255);
          const R* vy = vt + D::NX + (t >> 8 & 255);
          const R* vz = vt + 2 * D::NX + (t >> 16);
          R X[D::NV], Y[D::NV], Z[D::NV];
#pragma unroll
          for (int v = 0; v < D::NV; ++v) {
            X[v] = vx[v * 3 * D::NX];
            Y[v] = vy[v * 3 * D::NX];
            Z[v] = vz[v * 3 * D::NX];
          }
          rys_accumulate<ORD>(W[e], X, Y, Z, acc);
        }
      }
      if (x + 1 < mine && ++ik == Q.nprim) {
        ik = 0;
        ++ib;
      }
    }
    // sums over the group, then (order 2) through shared memory into the output
#pragma unroll
    for (int x = 0; x < D::NOUT; ++x)
#pragma unroll
      for (int off = (G < 32 ? G : 32) / 2; off > 0; off >>= 1) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
    if constexpr (G > 32) {
      rys_sync<G>();  // the tables are read no more
      if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int x = 0; x < D::NOUT; ++x) rw[(threadIdx.x >> 5) * D::NOUT + x] = acc[x];
      rys_sync<G>();
      if (threadIdx.x == 0)
        for (int w = 1; w < G / 32; ++w)
#pragma unroll
          for (int x = 0; x < D::NOUT; ++x) acc[x] += rw[w * D::NOUT + x];
    }
    if constexpr (ORD == 1) {
      if (lane == 0 && live) {
        double* gout = o.smem_atoms > 0 ? gsum : a.grad;
        const int at[3] = {P.atom_a, P.atom_b, Q.atom_a};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double gA = double(acc[d]), gB = double(acc[3 + d]), gC = double(acc[6 + d]);
          atomicAdd(gout + 3 * at[0] + d, gA);
          atomicAdd(gout + 3 * at[1] + d, gB);
          atomicAdd(gout + 3 * at[2] + d, gC);
          atomicAdd(gout + 3 * Q.atom_b + d, -(gA + gB + gC));
        }
      }
    } else {
      R* h45 = W + D::NCART;
      if (lane == 0)
#pragma unroll
        for (int x = 0; x < 45; ++x) h45[x] = acc[x];
      rys_sync<G>();
      const int at[4] = {P.atom_a, P.atom_b, Q.atom_a, Q.atom_b};
      if (live) hess_add_block(h45, at, hess_copy(o.hess, o.natoms, o.copies), 3 * o.natoms, lane, G);
    }
    rys_sync<G>();
  }
  if (ORD == 1 && o.smem_atoms > 0) {
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * o.smem_atoms; i += BLOCK)
      if (gsum[i] != 0.0) atomicAdd(a.grad + i, gsum[i]);
  }
}

// Threads per block of group size G: blocks of several warps while their groups' shared memory
// stays small enough for several blocks on an SM.
template <typename D, typename R, int G>
constexpr int rys_block() {
  return G > 32 ? G
                : (128 / G * D::group(G) * (int)sizeof(R) <= 72 * 1024
                       ? 128
                       : (64 / G * D::group(G) * (int)sizeof(R) <= 72 * 1024 ? 64 : 32));
}

// Lets kernel k take `bytes` of dynamic shared memory where that is above the 48 KB of any kernel.  MOST, the
// most that any launch of k can ask for, is what is set: the limit is the kernel's, not the launch's, and
// a handle on another thread may be about to launch k with more sums of its own.
template <size_t MOST, typename K>
inline bool allow_shared(K* k, size_t bytes) {
  static_assert(MOST <= 227 * 1024, "shared memory of a block");
  return bytes <= 48 * 1024 ||
         cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST) == cudaSuccess;
}

// Launches class (LA LB|LC LD) at derivative order ORD with G threads per quartet over quartets
// q[0, nq), at most max_blocks blocks (0: one group of quartets per block).
template <int LA, int LB, int LC, int LD, int ORD, typename R, int G>
static bool launch_rys(const GradArgs<R>& a, const RysOut& o, int pure, const int2* q, int nq, int max_blocks,
                       cudaStream_t s) {
  if (nq <= 0) return true;
  using D = RysDims<LA, LB, LC, LD, ORD>;
  constexpr int BLOCK = rys_block<D, R, G>(), GROUPS = BLOCK / G;
  constexpr size_t kTables = (size_t)GROUPS * D::group(G) * sizeof(R) + (size_t)D::NCART * sizeof(int);
  const size_t bytes = kTables + (ORD == 1 ? 3 * sizeof(double) * (size_t)o.smem_atoms : 0);
  auto k = rys_deriv_kernel<LA, LB, LC, LD, ORD, R, G, BLOCK>;
  if (!allow_shared<kTables + (ORD == 1 ? kGradSmemBytes : 0)>(k, bytes)) return false;
  k<<<rys_blocks(nq, 1, GROUPS, max_blocks), BLOCK, bytes, s>>>(a, o, pure, q, nq);
  return true;
}
