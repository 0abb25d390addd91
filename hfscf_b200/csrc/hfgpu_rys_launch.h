// Host-visible launchers of the Rys-quadrature derivative kernels (one translation unit per class,
// generated by gen_eri.py).
#pragma once
#include <cuda_runtime.h>

template <typename R>
struct GradArgs;
template <typename R>
struct QuartetArgs;
struct RysOut;

namespace hfgpu {

// Variants: groups of threads over shared-memory tables, fewest, middle and most threads per quartet (null
// where no form or default reaches them), and (null for the larger classes) three threads per quartet, one per direction (kRysThree), or ten such
// triples per quartet (kRysSplit).
constexpr int kRysVariants = 5, kRysThree = 3, kRysSplit = 4;

struct RysLaunchers {
  int la, lb, lc, ld;
  // defaults, -1: straight-line code instead.  A gradient class of at most three_prims primitive quartets
  // per quartet on average runs three threads per quartet in FP64.
  int grad_variant, three_prims, hess_variant;
  // quartets q[0, nq) on at most max_blocks blocks (0: no limit); false when the launch's shared
  // memory could not be had
  bool (*grad_d[kRysVariants])(const GradArgs<double>&, const RysOut&, int pure, const int2* q, int nq, int max_blocks,
                               cudaStream_t);
  bool (*grad_f[kRysVariants])(const GradArgs<float>&, const RysOut&, int pure, const int2* q, int nq, int max_blocks,
                               cudaStream_t);
  bool (*hess[kRysVariants])(const GradArgs<double>&, const RysOut&, int pure, const int2* q, int nq, int max_blocks,
                             cudaStream_t);
  // undifferentiated integrals, one warp per quartet (the large classes; null otherwise)
  bool (*quartet)(const QuartetArgs<double>&, const double* tab, const int2* q, int nq, cudaStream_t);
};

extern const RysLaunchers* const kRysLaunchers[];

}  // namespace hfgpu

// Device address of the quadrature tables on the current device (nullptr on failure).
const double* hfgpu_rys_table();
