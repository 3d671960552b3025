// gram.h — projected Gram blocks of SNP rows and their batched systems (gram.cu).
#pragma once

#include "internal.h"

#include <memory>
#include <vector>

namespace slemm {

// Per-SNP statistics (device) with z = x − a: h = Σ rr²·z, p = Σ x and t = Qᵀ(rr∘z) (cq × ld) as hi+lo FP32
// pairs, xx = ‖(I − QQᵀ)(rr∘z)‖², and xy = (x − gm)ᵀy (0 without y).  a is the mean weighted by rr² where the
// projection takes the intercept out, else gm.  As a column of a Gram block a SNP is stored as (rr²∘z − f)·sc.x with
// residual weights, f = h/n where gm is far from the weighted mean and has to stay, else 0, and sc = {2^e, 2^−e} of
// its range; and as its counts x = z − f, f = −a, without.
struct GramStats {
  float* a;
  float* f;
  float2* sc;
  float2* h;
  float2* p;
  float2* t;
  double* xy;
  double* xx;
  int64_t ld;
};
struct GramStatsBuf {
  DevBuf buf;
  GramStats s{};
  GramStats make(int64_t m, int cq, cudaStream_t st)
  {
    buf.stream = st;
    buf.ordered = true;
    s.ld = m;
    s.xy = (double*)buf.ensure((size_t)m * (2 * sizeof(double) + ((size_t)cq + 3) * sizeof(float2) + 2 * sizeof(float)));
    s.xx = s.xy + m;
    s.h = reinterpret_cast<float2*>(s.xx + m);
    s.p = s.h + m;
    s.sc = s.p + m;
    s.t = s.sc + m;
    s.a = reinterpret_cast<float*>(s.t + (size_t)cq * m);
    s.f = s.a + m;
    return s;
  }
};

// Statistics of every SNP of a handle at the centring values gm (m): y (n, may be nullptr), rr (n_pad,
// nullptr: all 1), Q (n_pad × cq), all on the device; cols = {y, rr, Q, n_pad, cq}, guess as for exact_dots.
void gram_stats(slemm_geno* g, const float* gm, const ExactCols& cols, int guess, GramStatsBuf& out);
void gram_stats_gather(const GramStats& src, const int64_t* d_idx, int64_t cnt, int cq, GramStatsBuf& out, cudaStream_t st);

// A packed SNP-major copy of m rows (all with the same individuals) and its rows' statistics.
struct GramSide {
  const uint8_t* G;
  int64_t m;
  GramStats stats;
};
// One block: out[c·ldo + i] = (P(rr∘z_{r0+i}))ᵀ(P(rr∘z_{c0+c})) for product rows r0 … r0 + rows − 1 of R (r0 a
// multiple of 128, rows of 256; rows past R.m are not written) and columns c0 … c0 + ncols − 1 of C.
struct GramJob {
  int64_t r0, rows, c0, ncols;
  float* out;
};
// The rows of a block that has to hold SNPs s0 … s0 + cnt − 1 of R: at most round_up(cnt, 256) + 256.
void gram_rows(const GramSide& R, int64_t s0, int64_t cnt, GramJob& job);
// The blocks of one pair of sides.  g gives the stream, the work buffers and the individuals; rr (n_pad) ==
// nullptr: all 1.  With R and C the same side and a block's columns among its rows: `lower`
// wants the rows up to each column's own SNP alone (out's others are left alone), `mirrored` has the columns'
// SNPs from the other half as well.  The host tables of the copies it queues go into `keep`.
enum class GramHalf { all, lower, mirrored };
// Host memory that queued copies read: a copy from pageable memory need not be staged on a machine whose GPU reads
// pageable memory.  Waits for the stream before it lets go, unless the caller has and says so.
struct HostKeep {
  cudaStream_t stream;
  std::vector<std::shared_ptr<void>> held;
  explicit HostKeep(cudaStream_t st) : stream(st) {}
  HostKeep(const HostKeep&) = delete;
  HostKeep& operator=(const HostKeep&) = delete;
  ~HostKeep()
  {
    if (!held.empty()) cudaStreamSynchronize(stream);
  }
  template <class T>
  T& make()
  {
    const auto p = std::make_shared<T>();
    held.push_back(p);
    return *p;
  }
  void waited() { held.clear(); }
};
void gram_blocks(slemm_geno* g, const GramSide& R, const GramSide& C, const std::vector<GramJob>& jobs, int cq, const float* rr,
                 int64_t ldo, GramHalf half, HostKeep& keep);

// A batch of nb systems of s unknowns (layout in gram.cu); offA, offZ and t are device arrays.
struct SpdBatch {
  float* A;
  int64_t strideA;
  float* Z;
  const int64_t* offA;
  const int64_t* offZ;
  const int* t;
  int64_t ld;
  int s, nb, t_max;
};
// q[offZ[b] + r] = z_rᵀ(A_b + diag(ridge_b))⁻¹z_r for every row z_r of Z_b; A and Z are overwritten.
void spd_row_norms(const SpdBatch& B, const float* ridge, double* q, int* status, cudaStream_t st);
// part[b·blocks …] sums to zᵀ(A_b + diag(ridge_b))⁻¹z with z the row which[b] of A_b (t = 1, Z has room for
// one row per system).  With x an FP32 solution of M x = z, 2zᵀx − xᵀMx differs from zᵀM⁻¹z by
// rᵀM⁻¹r only, r = z − Mx: accurate to the square of the solution's own error.
int spd_quadform_blocks(int s);
void spd_quadforms(const SpdBatch& B, const float* ridge, const int64_t* which, double* part, int* status, cudaStream_t st);

}  // namespace slemm
