// Host-visible launchers of the per-class adjoint Hessian kernels (one translation unit per class,
// generated by gen_eri.py next to the J/K and gradient units).
#pragma once
#include <cuda_runtime.h>

template <typename R>
struct GradArgs;
struct HessOut;

namespace hfgpu {

struct HessLaunchers {
  int la, lb, lc, ld;
  // hess_kernel over quartets q[0, nq) with grid blocks of 128 threads
  void (*launch)(const GradArgs<double>&, const HessOut&, int pure, const int2* q, int nq, int grid, cudaStream_t);
  int (*scratch_slots)(int pure);  // doubles of scratch per thread
  // straight-line form (hess_line_kernel, one thread per quartet on register code, grid blocks of
  // 128 threads); false when the class has none
  bool has_line;
  bool (*launch_line)(const GradArgs<double>&, const HessOut&, int pure, const int2* q, int nq, int grid,
                      cudaStream_t);
};

extern const HessLaunchers* const kHessLaunchers[];
extern const int kNumHessClasses;

}  // namespace hfgpu
