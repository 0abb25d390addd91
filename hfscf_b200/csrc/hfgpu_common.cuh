// Device-side data layout and helpers shared by the two-electron kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define PI_2_5 34.986836655249725  // 2 pi^(5/2), hfscfmath::PI_25 (src/math/hfscf_math.hpp:25)

// ---------------------------------------------------------------------------
// Primitive pair of a shell pair (a b): p = alpha_a + alpha_b, ip = 1/p, P,
// PA = P - A and Kp = K sqrt(2 pi^2.5) / p with K = exp(-alpha_a alpha_b / p |AB|^2) c_a c_b
// (BASIS::ShellPair::set_params, src/integrals/hfscf_shellpair.cpp:33-61).  Kp is
// scaled so that the [00|00] prefactor K_ab K_cd 2 pi^2.5 / (p q sqrt(p+q)) is
// Kp_ab Kp_cd / sqrt(p+q).  eb2 is the square of the ket exponent, used only by the
// kinetic-energy integrals (for a folded self pair, the mean over (i, j) and (j, i)).
// 80 bytes in FP64 (five 16-byte loads).
// ---------------------------------------------------------------------------
template <typename R>
struct __align__(sizeof(R) * 2) PrimPair {
  R p, ip, Px, Py, Pz, PAx, PAy, PAz, Kp, eb2;
};

// One canonical shell pair (La >= Lb after an optional swap of the two shells).
struct PairInfo {
  int sa, sb;        // shell indices
  int fa, fb;        // first function of each shell in the final (pure or Cartesian) basis
  int prim_off;      // first primitive pair
  int nprim;         // primitive pairs kept
  int cls;           // pair class: 0 ss, 1 ps, 2 pp, 3 ds, 4 dp, 5 dd
  int atom_a, atom_b;
  int mol;           // molecule of a batched handle (0 otherwise); fa, fb are local to it
  double ABx, ABy, ABz;  // A - B
  double schwarz;        // sqrt(max |(ab|ab)|) over the pair's functions
};

// Status word written by kernels that detect a problem (bad input seen on device).
enum : int { HFGPU_DEV_OK = 0, HFGPU_DEV_NONFINITE = 1 };

template <typename R>
__device__ __forceinline__ R sqrt_t(R x);
template <>
__device__ __forceinline__ double sqrt_t<double>(double x) { return sqrt(x); }
template <>
__device__ __forceinline__ float sqrt_t<float>(float x) { return sqrtf(x); }
// Exact value of a small non-negative int (0 <= k < 2^22) without an int -> float
// conversion instruction (those issue on the narrow XU pipe): k is written into the low
// mantissa bits of 1.5 * 2^52 (1.5 * 2^23 in FP32) and the offset subtracted.
template <typename R>
__device__ __forceinline__ R small_int(int k);
template <>
__device__ __forceinline__ double small_int<double>(int k) {
  return __hiloint2double(0x43380000, k) - 6755399441055744.0;
}
template <>
__device__ __forceinline__ float small_int<float>(int k) {
  return __int_as_float(0x4B400000 | k) - 12582912.0f;
}

template <typename R>
__device__ __forceinline__ R exp_t(R x);
template <>
__device__ __forceinline__ double exp_t<double>(double x) { return exp(x); }
template <>
__device__ __forceinline__ float exp_t<float>(float x) { return expf(x); }
template <typename R>
__device__ __forceinline__ R rsqrt_t(R x);
template <>
__device__ __forceinline__ double rsqrt_t<double>(double x) { return rsqrt(x); }
template <>
__device__ __forceinline__ float rsqrt_t<float>(float x) { return rsqrtf(x); }

// ---------------------------------------------------------------------------
// Boys function F_m(T), m = 0..M, scaled by `pre`.
//
// Method (Gill, Johnson & Pople, Int. J. Quantum Chem. 40, 745 (1991); Helgaker,
// Jorgensen & Olsen, "Molecular Electronic-Structure Theory", sec. 9.8.2):
//   T <  tmax: F_M from a polynomial in d = T_k - T about the nearest grid point T_k = k h, then the
//              stable downward recursion F_{m-1} = (2T F_m + e^-T) / (2m - 1).  FP64: h = 1/32 (so
//              that T_k and d are exact), the degree-5 interpolation polynomial of the interval, and
//              e^-T = e^-T_k e^d with e^-T_k tabulated and e^d, |d| <= h/2, from its degree-6 Taylor
//              polynomial (remainder below (h/2)^7 / 7! = 5e-17).  FP32: h = 0.1, the Taylor
//              expansion sum_j F_{M+j}(T_k) d^j / j!, j = 0..3, and the library's exponential;
//   T >= tmax: F_0 = sqrt(pi/T)/2 (erf(sqrt T) = 1 to double precision there) and the upward
//              recursion F_{m+1} = ((2m+1) F_m - e^-T) / (2T), in FP64 without e^-T (a library
//              exponential on the far side made the anthracene J/K classes up to (pp|ps) 6-10% slower).
//              Upward from F_0, not down from F_M: F_10 underflows from T = 1e29 on, F_0 nowhere.
//
// FP64 row of (order M, grid point k), rows of one order contiguous: 48 bytes, three 16-byte loads,
// since the low classes wait for the L1 wavefronts of these rows (one per lane and load).  Values
// c0, c1, c2, c3 in full; the fifth 8 bytes hold the upper halves of c4 (in the low word) and of
// c5 (in the high word): read as one double they are c5, and c4 is the low word over a zero one;
// then e^-T_k.  c0..c3 are fitted to what c4 and c5 leave as rounded, so that the rounding of c4
// and c5 costs only its share beyond degree 3, 2^-21 (h/2)^4 / 8 of c4: 2e-17 of F_0, 1e-16 of F_10.
// Against 80-bit values over T in [0, 70] the relative error of F_M is 3e-16 at most and 6e-17 on average
// (M = 0) to 4e-15 and 2e-16 (M = 10).  The 64-byte row of seven Taylor terms at h = 0.1 before it had
// 6e-15 and 9e-17 to 9e-14 and 2e-15, and this row at h = 1/16 6e-15 and 1.2e-16 to 5e-14 and 3.6e-15 (a
// larger mean, because the interpolation error fills the interval and the Taylor error only its ends).
// The four loads of the 64-byte row cost anthracene's J/K build 3% (19.0 ms against 18.4 at the time); the
// twice as long table of h = 1/32 costs it 2% of that again (15.5 -> 15.8 ms, octane 2.22 -> 2.25).
// FP32 row: F_{M+j}(T_k) / j!, j = 0..3, then e^-T_k and padding (32 bytes).
// ---------------------------------------------------------------------------
#define BOYS_H_D 0.03125
#define BOYS_H_F 0.1
// Grid points (T_k = 0 .. 63 in FP64, 36 in FP32) and the end of the table's use.  FP64, order M: the
// first whole T at which F_M without e^-T and with erf = 1 is within 1e-16 of F_M, so that the asymptotic
// side needs no exponential.
#define BOYS_NGRID_D 2017
#define BOYS_NGRID_F 361
#define BOYS_TMAX_F 36.0
__host__ __device__ constexpr double boys_tmax_d(int M) {
  constexpr double t[11] = {36.0, 39.0, 43.0, 46.0, 49.0, 51.0, 54.0, 56.0, 58.0, 61.0, 63.0};
  return t[M];
}
// Grid points of order M that an FP64 evaluation can reach, and the rows of the orders below M.
__host__ __device__ constexpr int boys_points_d(int M) { return (int)(boys_tmax_d(M) * 32.0) + 1; }
__host__ __device__ constexpr int boys_rows_below_d(int M) {
  int n = 0;
  for (int m = 0; m < M; ++m) n += boys_points_d(m);
  return n;
}
#define BOYS_MMAX 10             // orders M = 0 .. 10 have rows
#define BOYS_ROW_D 6             // values per FP64 row
#define BOYS_ROW_F 8             // values per FP32 row

// The FP64 evaluation on the grid of 1/INVH: row(k, c, ek) reads the NC coefficients and e^-T_k of grid
// point k of order M; e^d from its Taylor polynomial of degree NE.
template <int M, int INVH, int NC, int NE, class Row>
__device__ __forceinline__ void boys_eval_d(double T, double pre, const Row& row, double* F) {
  constexpr double tmax = boys_tmax_d(M);
  if (T < tmax) {
    // nearest grid index without int/float conversions (they go through the narrow XU
    // pipe): adding 1.5 * 2^52 leaves round(T / h) in the low mantissa bits
    const double sh = T * INVH + 6755399441055744.0;
    const double d = (sh - 6755399441055744.0) * (1.0 / INVH) - T;  // T_k - T, exact
    double c[NC], ek;
    row(__double2loint(sh), c, ek);
    double f = c[NC - 1];
#pragma unroll
    for (int j = NC - 2; j >= 0; --j) f = c[j] + f * d;
    F[M] = f;
    if constexpr (M > 0) {
      constexpr double inv_fact[9] = {1.0,         1.0,         0.5,          1.0 / 6.0,    1.0 / 24.0,
                                      1.0 / 120.0, 1.0 / 720.0, 1.0 / 5040.0, 1.0 / 40320.0};
      double x = inv_fact[NE];
#pragma unroll
      for (int j = NE - 1; j >= 0; --j) x = inv_fact[j] + d * x;
      const double e = ek * x, t2 = T + T;
#pragma unroll
      for (int m = M; m > 0; --m) F[m - 1] = (t2 * F[m] + e) * (1.0 / (2 * m - 1));
    }
  } else {
    const double rt = rsqrt(T), it = rt * rt;
    F[0] = 0.88622692545275801365 * rt;  // sqrt(pi)/2 / sqrt(T)
#pragma unroll
    for (int m = 0; m < M; ++m) F[m + 1] = F[m] * ((m + 0.5) * it);
  }
#pragma unroll
  for (int m = 0; m <= M; ++m) F[m] *= pre;
}

// The FP32 evaluation; row(k) returns the four Taylor terms of grid point k of order M.
template <int M, class Row>
__device__ __forceinline__ void boys_eval_f(float T, float pre, const Row& row, float* F) {
  if (T < float(BOYS_TMAX_F)) {
    const int k = __float2int_rn(T * 10.0f);
    const float d = float(k) * float(BOYS_H_F) - T;
    const float4 r0 = row(k);
    float f = r0.w;
    f = r0.z + f * d;
    f = r0.y + f * d;
    f = r0.x + f * d;
    F[M] = f;
    if constexpr (M > 0) {
      const float e = exp_t<float>(-T), t2 = T + T;
#pragma unroll
      for (int m = M; m > 0; --m) F[m - 1] = (t2 * F[m] + e) * float(1.0 / (2 * m - 1));
    }
  } else {
    const float rt = rsqrt_t<float>(T);
    const float it = rt * rt;
    F[0] = 0.88622692545275801365f * rt;
    if constexpr (M > 0) {
      const float e = exp_t<float>(-T);
      const float h = 0.5f * it;
#pragma unroll
      for (int m = 0; m < M; ++m) F[m + 1] = (float(2 * m + 1) * F[m] - e) * h;
    }
  }
#pragma unroll
  for (int m = 0; m <= M; ++m) F[m] *= pre;
}

template <typename R>
struct BoysTable {
  const R* __restrict__ tab;  // per order boys_points_d(M) rows of BOYS_ROW_D, or BOYS_NGRID_F of BOYS_ROW_F

  template <int M>
  __device__ __forceinline__ void eval(R T, R pre, R* F) const {
    static_assert(M <= BOYS_MMAX, "Boys order beyond the table");
    if constexpr (sizeof(R) == 8) {
      boys_eval_d<M, 32, 6, 6>(T, pre, [&](int k, double* c, double& ek) {
        constexpr int first = boys_rows_below_d(M);
        const double2* r = reinterpret_cast<const double2*>(tab) + 3 * (first + k);
        const double2 r0 = r[0], r1 = r[1], r2 = r[2];
        c[0] = r0.x, c[1] = r0.y, c[2] = r1.x, c[3] = r1.y;
        c[4] = __hiloint2double(__double2loint(r2.x), 0);
        c[5] = r2.x;
        ek = r2.y;
      }, F);
    } else {
      boys_eval_f<M>(T, pre, [&](int k) {
        return *reinterpret_cast<const float4*>(tab + ((size_t)M * BOYS_NGRID_F + k) * BOYS_ROW_F);
      }, F);
    }
  }
};

__host__ __device__ constexpr int ncart_of(int L) { return (L + 1) * (L + 2) / 2; }
__host__ __device__ constexpr int npure_of(int L) { return 2 * L + 1; }

// ---------------------------------------------------------------------------
// Boys table of one order staged in shared memory.
//
// A block puts the table of the kernel's single order MS there once with one bulk copy
// (stage_to_shared).  FP64: the grid of 1/8 with the eight full coefficients of the degree-7 interpolation
// polynomial (its error, (h/2)^8 / (8! 2^7) F_{M+8}, is below 5e-17 of F_M) and e^d to degree 8, because a
// block's residency hangs on the bytes: 20.8 kB (M = 0) to 28.3 kB (M = 4) against 55 to 75 kB of the rows
// above, with which J/K builds in this form took 3.25 ms on n-octane and 28.1 on
// anthracene, 2.33 and 18.2 with these (2.37 and 19.8 with rows of 48 bytes on the grid of 1/16).
// Values are stored as planes: planes j = 0..3 of (c_2j, c_2j+1) over the grid points and one plane of
// e^-T_k, so that the lanes of a warp, holding different T, spread over the banks by grid point; FP32 has
// one plane of float4 (the Taylor terms 0..3 of its rows).  Global layout: per order, boys_plane_stride<R>()
// bytes from the last, its planes back to back: boys_plane_bytes<R>(M) bytes.
// ---------------------------------------------------------------------------
#define BOYS_STAGED_INVH 8
#define BOYS_STAGED_COEF 8
#define BOYS_STAGED_MMAX 4       // orders that are staged (classes of la + lb + lc + ld up to it)

__host__ __device__ constexpr int boys_staged_points_d(int M) { return (int)(boys_tmax_d(M) * BOYS_STAGED_INVH) + 1; }

template <typename R>
__host__ __device__ constexpr int boys_plane_bytes(int M) {  // a multiple of 16; 5.8 kB in FP32
  return (sizeof(R) == 8 ? (8 * (BOYS_STAGED_COEF + 1) * boys_staged_points_d(M) + 15) / 16 : BOYS_NGRID_F) * 16;
}
template <typename R>
__host__ __device__ constexpr int boys_plane_stride() {
  return boys_plane_bytes<R>(BOYS_STAGED_MMAX);
}

template <typename R, int MS>
struct BoysShared {
  const R* tab;  // shared memory: the planes of order MS

  template <int M>
  __device__ __forceinline__ void eval(R T, R pre, R* F) const {
    static_assert(M == MS && M <= BOYS_STAGED_MMAX, "the staged table holds one order");
    if constexpr (sizeof(R) == 8) {
      boys_eval_d<M, BOYS_STAGED_INVH, BOYS_STAGED_COEF, 8>(T, pre, [&](int k, double* c, double& ek) {
        constexpr int n = boys_staged_points_d(M);
        const double2* P = reinterpret_cast<const double2*>(tab) + k;
#pragma unroll
        for (int j = 0; j < BOYS_STAGED_COEF / 2; ++j) {
          const double2 v = P[j * n];
          c[2 * j] = v.x;
          c[2 * j + 1] = v.y;
        }
        ek = M > 0 ? tab[BOYS_STAGED_COEF * n + k] : 0.0;
      }, F);
    } else {
      boys_eval_f<M>(T, pre, [&](int k) { return reinterpret_cast<const float4*>(tab)[k]; }, F);
    }
  }
};

// Status codes a kernel leaves in its status word (device int, 0 = fine).
enum : int { HFGPU_DEV_STAGE_TIMEOUT = 2, HFGPU_DEV_ABORTED = 3 };
// Polls of a bounded mbarrier wait (each followed by a short sleep): about 0.1 s in all.
#define HFGPU_STAGE_MAX_POLLS (1 << 20)

// Copies `bytes` (a multiple of 16; both addresses 16-byte aligned) from global memory into
// this block's shared memory with one bulk copy of the TMA unit (cp.async.bulk, completing on
// the mbarrier `mbar` in shared memory), called by every thread of the block.  The wait for the
// copy is bounded: after HFGPU_STAGE_MAX_POLLS polls the block records
// HFGPU_DEV_STAGE_TIMEOUT in *status and the function returns false (every thread gets the same
// answer).  issue = false arms the barrier for `bytes` without issuing any copy, so that the
// wait runs out: the bounded-wait test, never used by a build.
__device__ __forceinline__ bool stage_to_shared(void* smem_dst, const void* gmem_src, unsigned bytes,
                                                unsigned long long* mbar, int* status, bool issue = true) {
  const unsigned mb = (unsigned)__cvta_generic_to_shared(mbar);
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
    if (issue)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                   "l"(gmem_src), "r"(bytes), "r"(mb)
                   : "memory");
  }
  unsigned done = 0;
  for (int i = 0; i < HFGPU_STAGE_MAX_POLLS; ++i) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mb)
        : "memory");
    if (done) break;
    __nanosleep(64);
  }
  const int ok = __syncthreads_and(done != 0);
  if (!ok) {
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, HFGPU_DEV_STAGE_TIMEOUT);
    // a copy that was issued may still be in flight: give it one more bounded wait before the
    // block leaves (and its shared memory goes to another block)
    if (issue) {
      for (int i = 0; i < HFGPU_STAGE_MAX_POLLS && !done; ++i) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mb)
            : "memory");
        if (!done) __nanosleep(64);
      }
    }
    __syncthreads();
  }
  return ok != 0;
}
