// Preconditioner solve of one-dimensional stiff problems in a single kernel.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "internal.h"

namespace rdcu {

class LinePrecond {
 public:
  // The lines of n fields of N points (two fields per complex line): false when they do
  // not fit a cluster of up to eight CTAs (N / C complex values each, at most 4096 over
  // all lines), N has a prime factor above 13, or memory runs out.
  bool init(int n, int N, double L, const std::vector<LinEntry>& lin);
  void release();
  ~LinePrecond() { release(); }
  // z = N (I + alpha J_lin)^-1 r, alpha read from device memory; r and z may not overlap
  cudaError_t apply(const double* r, double* z, const double* alpha_dev, cudaStream_t st) const;

  size_t device_bytes = 0;

 private:
  int n_ = 0, N_ = 0, C_ = 1, block_ = 0;
  double dx_ = 1.0;
  LinePlan plan_{};
  double2* tw_ = nullptr;
  LinTable lin_{};
  double* sinv_ = nullptr;
  double* cosv_ = nullptr;
};

}  // namespace rdcu
