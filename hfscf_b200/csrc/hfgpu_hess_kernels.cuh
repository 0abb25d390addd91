// Adjoint second derivatives of the two-electron energy at a fixed density: the two-electron
// part of the analytic Hessian, sum_abcd W_abcd d2(ab|cd)/dX dY, with the same weight block
// W as the adjoint gradient (RHF: W = 8 s [2 D_ab D_cd - (D_ac D_bd + D_ad D_bc)/2]).
//
// Replaces the reference's second-derivative ERI tensors and their contraction:
// Erios::compute_contracted_shell_quartet_deriv2_qq / _pq (src/integrals/hfscf_oserideriv2qq.cpp:28-853,
// hfscf_oserideriv2pq.cpp:23-891) and Mol::scf_hessian::calc_scf_hessian_tei
// (src/hessian/hfscf_hessian_ints.cpp:20-303), which store six packed derivative tensors per
// direction pair and then contract them once per atom pair.  Here nothing is stored: per unique
// shell quartet the class's generated op tables run the VRR two orders higher, the HRR of ten
// exponent-weighted sets and the contraction of every shifted integral with W, and the quartet's
// 12 x 12 block (centres A, B, C, D by x, y, z; D from translational invariance) is added into
// the 3 natoms x 3 natoms Hessian.  Two forms: hess_kernel, one thread per quartet on
// thread-interleaved global scratch (gen_eri.py gen_hess_table), and hess_line_kernel, one thread
// per quartet on straight-line register code (gen_hess_line, the classes whose terms fit at most 24
// passes of 64 accumulators).  The default of most classes is the Rys-quadrature form of
// hfgpu_rys.cuh.
#pragma once
#include "hfgpu_kernels.cuh"

// Hessian output of a launch: 3 natoms x 3 natoms, row-major, half of it (HessEntry), in `copies` (a power
// of two) partial sums one after another, of which a block adds into one: the rounding of a sum grows
// with its size, and each copy's is a share of the whole.  What a Hessian leaves of translational
// invariance shows it (the entries largely cancel over the atoms): (H2O)4 and n-octane at their core-guess
// densities 6e-13 to 2e-12 with one copy, 4e-13 to 1.3e-12 with 32, and no less with 128 or 512 (what is left
// comes from the quartets); random densities 5 to 7 times less than with one.  Times as with one copy.
struct HessOut {
  double* __restrict__ hess;
  int natoms;
  int copies;
};

__device__ __forceinline__ double* hess_copy(double* hess, int natoms, int copies) {
  return hess + (size_t)(blockIdx.x & (copies - 1)) * 9 * natoms * natoms;
}

// Executor of a table-mode Hessian class.  Weight sets, in the generator's order:
// 1, 2a_a, 2a_b, 2a_c, (2a_a)^2, (2a_b)^2, (2a_c)^2, 2a_a 2a_b, 2a_a 2a_c, 2a_b 2a_c.
// h45: the 45 upper-triangle entries of the 9 x 9 block over (A, B, C) x (x, y, z).
template <typename Tab>
__device__ void hess_table(const PrimPair<double>* __restrict__ bp, const double* __restrict__ ea,
                           const double* __restrict__ eb, int nbp, const PrimPair<double>* __restrict__ kp,
                           const double* __restrict__ ec, int nkp, double ABx, double ABy, double ABz, double CDx,
                           double CDy, double CDz, const BoysTable<double>& boys, Strided<double> W,
                           Strided<double> vs, Strided<double> hs, Strided<double> h45) {
  using R = double;
  vs[0] = R(0);
  hs[0] = R(0);
  for (int x = 1; x <= Tab::NACC; ++x) hs[x] = R(0);
  const int4* vo = Tab::vrr();  // packed rows: gen_eri.py pack_grad_vrr / pack_hess_hrr
  const int2* ho = Tab::hrr();
  for (int ib = 0; ib < nbp; ++ib) {
    const R p = bp[ib].p, ip = bp[ib].ip, Px = bp[ib].Px, Py = bp[ib].Py, Pz = bp[ib].Pz;
    const R PAx = bp[ib].PAx, PAy = bp[ib].PAy, PAz = bp[ib].PAz, Kab = bp[ib].Kp;
    const R wa = R(2) * ea[ib], wb = R(2) * eb[ib];
    for (int ik = 0; ik < nkp; ++ik) {
      const R q = kp[ik].p, iq = kp[ik].ip, Qx = kp[ik].Px, Qy = kp[ik].Py, Qz = kp[ik].Pz;
      const R QCx = kp[ik].PAx, QCy = kp[ik].PAy, QCz = kp[ik].PAz, Kcd = kp[ik].Kp;
      const R wc = R(2) * ec[ik];
      const R pq = p + q;
      const R rsq = rsqrt_t(pq);
      const R ipq = rsq * rsq;
      const R rho = p * q * ipq;
      const R rp = q * ipq, rq = p * ipq;
      const R inv2p = R(0.5) * ip, inv2q = R(0.5) * iq, inv2pq = R(0.5) * ipq;
      const R PQx = Px - Qx, PQy = Py - Qy, PQz = Pz - Qz;
      const R T = rho * (PQx * PQx + PQy * PQy + PQz * PQz);
      const R pre = Kab * Kcd * rsq;
      R F[Tab::L + 1];
      boys.template eval<Tab::L>(T, pre, F);
#pragma unroll
      for (int m = 0; m <= Tab::L; ++m) vs[1 + m] = F[m];
      for (int o = 0; o < Tab::NVOPS; ++o) {
        const int4 op = __ldg(vo + o);
        const int kind = op.w & 15, dir = (op.w >> 4) & 15, dst = op.x & 0xffff;
        const int sa = (unsigned)op.x >> 16, sb = op.y & 0xffff, sc = (unsigned)op.y >> 16, sd = op.z & 0xffff;
        if (kind == 2) {
          R w;
          switch (dir) {
            case 0: w = R(1); break;
            case 1: w = wa; break;
            case 2: w = wb; break;
            case 3: w = wc; break;
            case 4: w = wa * wa; break;
            case 5: w = wb * wb; break;
            case 6: w = wc * wc; break;
            case 7: w = wa * wb; break;
            case 8: w = wa * wc; break;
            default: w = wb * wc; break;
          }
          hs[1 + dst] += w * vs[sa];
          continue;
        }
        const R PQd = dir == 0 ? PQx : (dir == 1 ? PQy : PQz);
        const int k1 = (op.w >> 8) & 255;
        if (kind == 0) {
          const R PA = dir == 0 ? PAx : (dir == 1 ? PAy : PAz);
          vs[dst] = PA * vs[sa] - rp * PQd * vs[sb] + small_int<R>(k1) * inv2p * (vs[sc] - rp * vs[sd]);
        } else {
          const R QC = dir == 0 ? QCx : (dir == 1 ? QCy : QCz);
          const int sg = (unsigned)op.z >> 16, k2 = (unsigned)op.w >> 16;
          vs[dst] = QC * vs[sa] + rq * PQd * vs[sb] + small_int<R>(k1) * inv2q * (vs[sc] - rq * vs[sd]) +
                    small_int<R>(k2) * inv2pq * vs[sg];
        }
      }
    }
  }
  for (int x = 0; x < 45; ++x) h45[x] = R(0);
  for (int o = 0; o < Tab::NHOPS; ++o) {
    const int2 op = __ldg(ho + o);
    const int kind = (op.y >> 16) & 15;
    const int sx = (unsigned)op.x >> 16;
    if (kind == 2) {
      const int wi = op.x & 0xffff, k = (op.y & 0xffff) - 128, hi = (op.y >> 20) & 63;
      h45[hi] += R(k) * W[wi] * hs[sx];
    } else {
      const int dst = op.x & 0xffff, sy = op.y & 0xffff, dir = (op.y >> 20) & 15;
      const R d = kind == 0 ? (dir == 0 ? ABx : (dir == 1 ? ABy : ABz)) : (dir == 0 ? CDx : (dir == 1 ? CDy : CDz));
      hs[dst] = hs[sx] + d * hs[sy];
    }
  }
}

// Position of coordinate pair (r, s), r <= s, of the 9 x 9 block in the 45-entry upper triangle.
__device__ __forceinline__ int hess_tri(int r, int s) { return r * 9 - r * (r - 1) / 2 + (s - r); }

// The 3 natoms x 3 natoms output collects, per pair of coordinates, one of its two symmetric
// entries: U with H = U + U^T (hess_finish_kernel), so that a quartet adds 78 values, not 144.  Of
// centre blocks X < Y every entry is added, of X = Y those with i < j and half of those with i = j.
// (Two centres on one atom need no special case.)
//
// Entry t of the 78: centres X <= Y of A, B, C, D and directions i, j.  Six centre pairs of nine
// entries, then four symmetric blocks of six.
struct HessEntry {
  int X, i, Y, j;
  __device__ __forceinline__ explicit HessEntry(int t) {
    if (t < 54) {
      const int k = t / 9;
      X = k < 3 ? 0 : (k < 5 ? 1 : 2);
      Y = k < 3 ? k + 1 : (k < 5 ? k - 1 : 3);
      i = t % 9 / 3;
      j = t % 3;
    } else {
      const int n = (t - 54) % 6;
      X = Y = (t - 54) / 6;
      i = n < 3 ? 0 : (n < 5 ? 1 : 2);
      j = n < 3 ? n : (n < 5 ? n - 2 : 2);
    }
  }
  // Its value from the quartet's 45 entries over A, B, C: a D row or column is minus the sum of the
  // others (translational invariance).
  template <typename H>
  __device__ __forceinline__ double value(const H& h45) const {
    double v = 0.0;
#pragma unroll 1
    for (int u = X < 3 ? X : 0; u < (X < 3 ? X + 1 : 3); ++u)
#pragma unroll 1
      for (int w = Y < 3 ? Y : 0; w < (Y < 3 ? Y + 1 : 3); ++w) {
        const int m = 3 * u + i, n = 3 * w + j;
        v += double(h45[m < n ? hess_tri(m, n) : hess_tri(n, m)]);
      }
    if ((X == 3) != (Y == 3)) v = -v;
    return X == Y && i == j ? 0.5 * v : v;
  }
  __device__ __forceinline__ long long offset(const int (&at)[4], int n3) const {
    const int r = X == 0 ? at[0] : (X == 1 ? at[1] : (X == 2 ? at[2] : at[3]));
    const int c = Y == 0 ? at[0] : (Y == 1 ? at[1] : (Y == 2 ? at[2] : at[3]));
    return (long long)(3 * r + i) * n3 + 3 * c + j;
  }
};

// Adds entries first, first + step, ... of one quartet (atoms at[0..3]) into U.
template <typename H>
__device__ __forceinline__ void hess_add_block(const H& h45, const int (&at)[4], double* U, int n3, int first,
                                               int step) {
#pragma unroll 1
  for (int t = first; t < 78; t += step) {
    const HessEntry e(t);
    atomicAdd(U + e.offset(at, n3), e.value(h45));
  }
}

// Adds the blocks of a warp's quartets (one per valid lane, atoms at, 45 entries in shared memory at
// h45[x stride + lane qstride]) into U: the warp walks its quartets, each lane owning up to three of the 78
// entries, and adds to memory only when the entry's place changes.  The lists are bra-major, so the
// bra atoms hold for most of a warp and a ket atom for runs of it: few atomics, none against each
// other.  (One lane per quartet adding its own 78 entries retried 32 compare-and-swap loops per
// value, and as unrolled code it missed the instruction cache.)  Called by all lanes.
__device__ __forceinline__ void hess_add_warp(bool valid, const double* h45, int stride, int qstride,
                                              const int (&at)[4], double* U, int n3) {
  struct Column {
    const double* p;
    int stride;
    __device__ __forceinline__ double operator[](int x) const { return p[x * stride]; }
  };
  __syncwarp();
  const int lane = threadIdx.x & 31;
  const HessEntry e[3] = {HessEntry(lane), HessEntry(lane + 32), HessEntry(lane + 64 < 78 ? lane + 64 : 77)};
  double sum[3] = {0.0, 0.0, 0.0};
  long long cur[3] = {-1, -1, -1};
#pragma unroll 1
  for (unsigned m = __ballot_sync(0xffffffffu, valid); m; m &= m - 1) {
    const int q = __ffs(m) - 1;
    int aq[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) aq[c] = __shfl_sync(0xffffffffu, at[c], q);
    const Column h{h45 + q * qstride, stride};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (k == 2 && lane + 64 >= 78) continue;
      const long long off = e[k].offset(aq, n3);
      if (off != cur[k]) {
        if (cur[k] >= 0) atomicAdd(U + cur[k], sum[k]);
        cur[k] = off;
        sum[k] = 0.0;
      }
      sum[k] += e[k].value(h);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (cur[k] >= 0) atomicAdd(U + cur[k], sum[k]);
  __syncwarp();
}

// hess += U + U^T, U the sum of the copies.
static __global__ void hess_finish_kernel(const double* __restrict__ U, double* __restrict__ hess, int n3, int copies) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nn = (size_t)n3 * n3;
  if (e >= nn) return;
  const size_t r = e / n3, t = e % n3 * n3 + r;
  double v = 0.0;
  for (int k = 0; k < copies; ++k) v += U[k * nn + e] + U[k * nn + t];
  hess[e] += v;
}

template <int LA, int LB, int LC, int LD, bool PURE, typename Tab>
__device__ __forceinline__ void hess_quartet(const GradArgs<double>& a, int tid, const int2 pq, const PairInfo& P,
                                             const PairInfo& Q) {
  using Dm = BlockDims<LA, LB, LC, LD, PURE>;
  double s = 8.0;
  if (P.sa == P.sb) s *= 0.5;
  if (Q.sa == Q.sb) s *= 0.5;
  if (pq.x == pq.y) s *= 0.5;
  // scratch per thread: [VRR slots | HRR slots | 45 outputs | W cart | 2 transform buffers]
  double* base = a.scratch + tid;
  const int st = a.scratch_threads;
  Strided<double> vs{base, st};
  Strided<double> hs{base + (size_t)Tab::NVSLOT * st, st};
  Strided<double> h45{base + (size_t)(Tab::NVSLOT + Tab::NHSLOT) * st, st};
  Strided<double> Wc{base + (size_t)(Tab::NVSLOT + Tab::NHSLOT + 45) * st, st};
  Strided<double> t0{base + (size_t)(Tab::NVSLOT + Tab::NHSLOT + 45 + Dm::NCART) * st, st};
  Strided<double> t1{base + (size_t)(Tab::NVSLOT + Tab::NHSLOT + 45 + 2 * Dm::NCART) * st, st};
  if constexpr (PURE) {
    grad_weights<Dm::NA, Dm::NB, Dm::NC, Dm::ND>(a.DJ, a.cJ, a.nK, a.DK, a.cK, a.n, P.fa, P.fb, Q.fa, Q.fb, s, t0);
    // pure -> Cartesian weights, one index at a time: t0 -> t1 -> t0 -> t1 -> Wc
    const int Ls[4] = {LA, LB, LC, LD};
    int dims[4] = {Dm::NA, Dm::NB, Dm::NC, Dm::ND};
    Strided<double> src = t0, dst = t1;
    for (int stp = 0; stp < 4; ++stp) {
      const int nc = ncart_of(Ls[stp]), np = npure_of(Ls[stp]);
      int nd[4] = {dims[0], dims[1], dims[2], dims[3]};
      nd[stp] = nc;
      Strided<double> out = (stp == 3) ? Wc : dst;
      const int tot = nd[0] * nd[1] * nd[2] * nd[3];
      for (int e = 0; e < tot; ++e) {
        int id[4];
        int r = e;
        for (int qq = 3; qq >= 0; --qq) {
          id[qq] = r % nd[qq];
          r /= nd[qq];
        }
        double v = 0.0;
        for (int c = 0; c < np; ++c) {
          const double y = c_ylm[Ls[stp]][id[stp] * np + c];
          if (y == 0.0) continue;
          int jd[4] = {id[0], id[1], id[2], id[3]};
          jd[stp] = c;
          v += y * src[((jd[0] * dims[1] + jd[1]) * dims[2] + jd[2]) * dims[3] + jd[3]];
        }
        out[e] = v;
      }
      for (int qq = 0; qq < 4; ++qq) dims[qq] = nd[qq];
      Strided<double> tmp = src;
      src = dst;
      dst = tmp;
    }
  } else {
    grad_weights<Dm::NA, Dm::NB, Dm::NC, Dm::ND>(a.DJ, a.cJ, a.nK, a.DK, a.cK, a.n, P.fa, P.fb, Q.fa, Q.fb, s, Wc);
  }
  hess_table<Tab>(a.prims + P.prim_off, a.alpha_a + P.prim_off, a.alpha_b + P.prim_off, P.nprim,
                  a.prims + Q.prim_off, a.alpha_a + Q.prim_off, Q.nprim, P.ABx, P.ABy, P.ABz, Q.ABx, Q.ABy, Q.ABz,
                  a.boys, Wc, vs, hs, h45);
}

template <int LA, int LB, int LC, int LD, typename Tab>
__global__ void __launch_bounds__(128) hess_kernel(GradArgs<double> a, HessOut o, int pure,
                                                   const int2* __restrict__ quartets, int nq) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nthr = gridDim.x * blockDim.x;
  const Strided<double> h45{a.scratch + tid + (size_t)(Tab::NVSLOT + Tab::NHSLOT) * a.scratch_threads,
                            a.scratch_threads};
  const int np = a.nparts > 1 ? a.nparts : 1, p0 = np > 1 ? a.part : 0;
  for (long long t = tid; t < nq; t += nthr) {
    const int2 pq = quartets[(size_t)t * np + p0];
    const PairInfo P = a.pairs[pq.x];
    const PairInfo Q = a.pairs[pq.y];
    if (pure)
      hess_quartet<LA, LB, LC, LD, true, Tab>(a, tid, pq, P, Q);
    else
      hess_quartet<LA, LB, LC, LD, false, Tab>(a, tid, pq, P, Q);
    const int at[4] = {P.atom_a, P.atom_b, Q.atom_a, Q.atom_b};
    hess_add_block(h45, at, hess_copy(o.hess, o.natoms, o.copies), 3 * o.natoms, 0, 1);
  }
}

// ---------------------------------------------------------------------------
// Straight-line form: one thread per quartet, the class's generated code (gen_eri.py
// gen_hess_line) with every value in registers, in passes of at most 64 accumulators.  Each pass
// adds its terms into the thread's 45 entries of the 9 x 9 block, kept in shared memory (45 x 128
// doubles per block, behind the block's Hessian when that is in shared memory too) so that they
// hold no registers through the primitive loops; the 12 x 12 block goes into the output once per
// quartet.  For the many-quartet classes, whose table forms spend their time on level barriers
// or on global scratch round trips rather than on the few dozen ops of a level.
// ---------------------------------------------------------------------------
constexpr int kHessLineThreads = 128;
constexpr int kHessLineStride = kHessLineThreads + 1;  // odd: the lanes of hess_add_warp read one column
constexpr int kHessLineH45Bytes = 45 * kHessLineStride * (int)sizeof(double);

// grad_weights with every loop over the block unrolled, so that W stays in registers
template <int NA, int NB, int NC, int ND>
__device__ __forceinline__ void hess_line_weights(const double* __restrict__ DJ, double cJ, int nK,
                                                  const double* __restrict__ DK, double cK, int n, int fa, int fb,
                                                  int fc, int fd, double s8, double* W) {
#pragma unroll
  for (int i = 0; i < NA; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const double dab = DJ ? __ldg(DJ + (size_t)(fa + i) * n + fb + j) : 0.0;
#pragma unroll
      for (int k = 0; k < NC; ++k)
#pragma unroll
        for (int l = 0; l < ND; ++l) {
          double w = DJ ? cJ * dab * __ldg(DJ + (size_t)(fc + k) * n + fd + l) : 0.0;
          for (int m = 0; m < nK; ++m) {
            const double* D = DK + (size_t)m * n * n;
            w -= 0.5 * cK *
                 (__ldg(D + (size_t)(fa + i) * n + fc + k) * __ldg(D + (size_t)(fb + j) * n + fd + l) +
                  __ldg(D + (size_t)(fa + i) * n + fd + l) * __ldg(D + (size_t)(fb + j) * n + fc + k));
          }
          W[((i * NB + j) * NC + k) * ND + l] = s8 * w;
        }
    }
}

template <int LA, int LB, int LC, int LD, bool PURE, typename Line>
__device__ __forceinline__ void hess_line_quartet(const GradArgs<double>& a, const int2 pq, const PairInfo& P,
                                                  const PairInfo& Q, Strided<double> h45) {
  using Dm = BlockDims<LA, LB, LC, LD, PURE>;
  double s = 8.0;
  if (P.sa == P.sb) s *= 0.5;
  if (Q.sa == Q.sb) s *= 0.5;
  if (pq.x == pq.y) s *= 0.5;
  // the weight block, Cartesian, fetched by each pass after its primitive loops
  auto weights = [&](double* Wc) {
    if constexpr (PURE) {
      double Wp[Dm::NOUT];
      hess_line_weights<Dm::NA, Dm::NB, Dm::NC, Dm::ND>(a.DJ, a.cJ, a.nK, a.DK, a.cK, a.n, P.fa, P.fb, Q.fa, Q.fb, s,
                                                        Wp);
      ClassCode<LA, LB, LC, LD>::template from_pure<double>(Wp, Wc);
    } else {
      hess_line_weights<Dm::NA, Dm::NB, Dm::NC, Dm::ND>(a.DJ, a.cJ, a.nK, a.DK, a.cK, a.n, P.fa, P.fb, Q.fa, Q.fb, s,
                                                        Wc);
    }
  };
#pragma unroll
  for (int x = 0; x < 45; ++x) h45[x] = 0.0;
  Line::template run<double>(a.prims + P.prim_off, a.alpha_a + P.prim_off, a.alpha_b + P.prim_off, P.nprim,
                             a.prims + Q.prim_off, a.alpha_a + Q.prim_off, Q.nprim, P.ABx, P.ABy, P.ABz, Q.ABx,
                             Q.ABy, Q.ABz, a.boys, weights, h45);
}

// dynamic shared memory: the h45 slices
template <int LA, int LB, int LC, int LD, typename Line>
__global__ void __launch_bounds__(kHessLineThreads) hess_line_kernel(GradArgs<double> a, HessOut o, int pure,
                                                                     const int2* __restrict__ quartets, int nq) {
  extern __shared__ double hess_sh[];
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nthr = gridDim.x * blockDim.x;
  const Strided<double> h45{hess_sh + threadIdx.x, kHessLineStride};
  const int np = a.nparts > 1 ? a.nparts : 1, p0 = np > 1 ? a.part : 0;
  // whole warps stay in the loop together (lanes past the end add nothing), for hess_add_warp
  const int lane = threadIdx.x & 31;
  for (int t0 = tid - lane; t0 < nq;) {  // t0, the warp's first quartet, never passes nq (t0 + nthr can pass 2^31)
    const bool valid = lane < nq - t0;
    int at[4] = {0, 0, 0, 0};
    if (valid) {
      const int2 pq = quartets[(size_t)(t0 + lane) * np + p0];
      const PairInfo P = a.pairs[pq.x];
      const PairInfo Q = a.pairs[pq.y];
      at[0] = P.atom_a;
      at[1] = P.atom_b;
      at[2] = Q.atom_a;
      at[3] = Q.atom_b;
      if (pure)
        hess_line_quartet<LA, LB, LC, LD, true, Line>(a, pq, P, Q, h45);
      else
        hess_line_quartet<LA, LB, LC, LD, false, Line>(a, pq, P, Q, h45);
    }
    hess_add_warp(valid, hess_sh + (threadIdx.x & ~31), kHessLineStride, 1, at,
                  hess_copy(o.hess, o.natoms, o.copies), 3 * o.natoms);
    if (nthr >= nq - t0) break;
    t0 += nthr;
  }
}
