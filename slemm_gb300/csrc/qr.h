// qr.h — column-pivoted Householder QR of the fixed-effects design on the GPU (qr.cu).
#pragma once

#include "internal.h"

#include <vector>

namespace slemm {

// QR of rr∘X (host arrays: n×c with leading dimension ldx, rr of n) on a stream.  The constructor only queues
// the work, so host work can run until finish(); the arrays have to live until then.
class DesignQr {
 public:
  DesignQr(const float* X, int64_t ldx, const float* rr, int64_t n, int c, cudaStream_t st);
  ~DesignQr()   // left early: the copies may still read the inputs
  {
    if (!waited_) cudaStreamSynchronize(st_);
  }
  DesignQr(const DesignQr&) = delete;
  DesignQr& operator=(const DesignQr&) = delete;
  // Waits.  rank by Eigen's rule |R_ii| > eps_f32·min(n, c)·|R_00|, R·Pᵀ (rank×c, column-major), and whether
  // every entry of X is finite; Q is that of all c columns if rank == c.
  void finish();
  int rank = 0;
  bool finite = true;
  std::vector<double> RPt;
  // Q's columns as FP32, ld apart, rows n … rows − 1 zero (device memory)
  void store(float* out, int64_t ld, int64_t rows) const;
  // (I − QQᵀ)(rr∘y) as FP32, times rr once more if `scale` (device memory)
  void project(const float* d_y, float* out, bool scale) const;

 private:
  int64_t n_;
  int c_;
  cudaStream_t st_;
  bool waited_ = false;
  DevBuf work_, basis_, rr_;
  double *Q_ = nullptr, *v_ = nullptr;
  float* d_rr_ = nullptr;
  std::vector<double> head_;
};

// The handle's projection (slemm_gpu_set_projection) from Q of all c columns.
void set_projection_qr(slemm_geno* g, const DesignQr& qr, int c);

}  // namespace slemm
