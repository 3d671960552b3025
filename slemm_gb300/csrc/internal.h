// internal.h — handle layout and internal entry points shared by the translation units.
#pragma once

#include "common.h"

struct slemm_geno {
  int device = 0;
  int64_t n = 0, m = 0;           // kept individuals, SNPs
  int64_t n_pad = 0, m_pad = 0;   // padded to kTileM
  // Two tiled 2-bit copies of the count matrix (layout in geno.cu):
  //   G : M = SNPs (m_pad rows),        K = individuals (n_pad)  → Z_cᵀU direction
  //   GT: M = individuals (n_pad rows), K = SNPs (m_pad)         → Z_c V direction
  slemm::DevBuf G, GT;
  slemm::DevBuf gm, w, rr;        // FP32, padded with zeros (rr padded with 0)
  slemm::DevBuf Q;                // n_pad × c column-major, zero padded rows
  int c = 0;
  bool weights_set = false;
  bool rr_one = false;            // every rr of set_weights is 1
  int prec = SLEMM_PREC_FP16X2;
  int per_vector = 0;
  int lanczos_mode = 0;           // SLEMM_LANCZOS_* bits of the seeds run on this handle
  int autotune = 0;               // tensor-core plans: 0 the fixed rule, 1 the tuner's, 2 the fixed rule
                                  // with two CTAs per SM wherever N ≤ 64
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  // work buffers
  slemm::DevBuf ws_B, ws_D, ws_red, ws_small, ws_T, ws_in, ws_out;
  slemm::DevBuf err;              // int error word of the kernels' bounded waits (zeroed at create)
  slemm::HostScal scal;           // mapped host scalars of the Lanczos steps
  // per-SNP class counts n1, n2 in device memory ([2][m_pad] int32), summed by the pack kernel
  // while it builds the tiles (every handle genotype_create packs; a copy derived from another
  // handle's tiles, like slemm_gwa's model-SNP copy, has none and counts its tiles instead —
  // `dcounts_valid` says which)
  slemm::DevBuf dcounts;
  bool dcounts_valid = false;
  // Z_cᵀ1 per SNP, pc_j − n·gm_j (FP64, stored FP32): the exact product of the centred matrix
  // with a constant vector, set with the weights; the operators remove each input column's mean
  // and add it back through this term (see ops.cu)
  slemm::DevBuf gcorr;
  // A trait view (slemm_gpu_genotype_view) aliases its parent's packed copies (G, GT, n_pad, m_pad
  // are the parent's) and analyses a subset of the parent's individuals: ind_map[r] is the packed
  // individual position of view row r (n entries), ind_inv[i] the view row of position i or −1
  // (n_pad entries), kmask the field masks of the kept positions per K-tile (4 words each, the low
  // bit of each kept 2-bit field) for its own integer counts.
  bool is_view = false;
  slemm::DevBuf ind_map, ind_inv, kmask;
  // per-SNP popcount and class counts of the packed copy (immutable): host copies on first request
  std::vector<int64_t> counts_pc;
  std::vector<int32_t> counts_c1, counts_c2;
  // optional per-launch timing of the packed products (CUDA events on `stream`)
  struct GemmRecord {
    cudaEvent_t start, stop;
    int tc, N, k, pieces, splits, dir;   // dir 1: Zᵀ pass (M = SNPs), 2: Z pass (M = individuals)
    int plan;                            // tensor-core ring plan (GemmArgs::plan)
  };
  bool profiling = false;
  std::vector<GemmRecord> prof_pending;
  std::vector<cudaEvent_t> event_pool;
  struct GemmStat {
    int tc, N, k, pieces, dir, splits, plan;
    int64_t launches;
    double ms;
  };
  std::vector<GemmStat> prof_stats;
  // Every device buffer of the handle: all are stream-ordered on `stream` (the pool keeps freed
  // blocks cached, so building and dropping handles costs no device-wide synchronisation).
  template <class F>
  void for_each_buf(F&& f)
  {
    for (slemm::DevBuf* b : {&G, &GT, &gm, &w, &rr, &Q, &ws_B, &ws_D, &ws_red, &ws_small, &ws_T, &ws_in, &ws_out, &err,
                             &dcounts, &gcorr, &ind_map, &ind_inv, &kmask})
      f(*b);
  }
  void bind_stream()
  {
    for_each_buf([&](slemm::DevBuf& b) {
      b.stream = stream;
      b.ordered = true;
    });
  }
};

namespace slemm {

// ops.cu — one operator application on device buffers (column-major, ld given).
void op_device(slemm_geno* g, int kind, float tau0, const float* in, int64_t ld_in, int k,
               float* out, int64_t ld_out);
// H0 operator on a mixed block: columns 0 … nq−1 as H0_quadform_mv, the rest as H0_ldet_mv
// (kind LDET; QUADFORM means nq = k).
void op_device_mixed(slemm_geno* g, int kind, float tau0, const float* in, int64_t ld_in, int k,
                     float* out, int64_t ld_out, int nq);

// The same operator on U (n×k, ld = n) with the rest of a Lanczos step on its result (lanczos.cu): FP16X2
// handles only, false (and nothing done) otherwise.  tmp: n×k scratch.  Uprev (nullptr at the first step)
// and Unext: n×k.  beta[k] (device, hi+lo): β of the step before, replaced by this step's.  scal[c],
// scal[stride + c], scal[2·stride + c] (host-mapped): δ, ‖·‖², ‖U_next‖²; scal_err: the error word.
bool op_lanczos_step(slemm_geno* g, int kind, float tau0, const float* U, int k, float* tmp, int nq, const float* Uprev,
                     float* Unext, float2* beta, double* scal, int stride, double* scal_err);

// Centred Z_cᵀU over SNP rows [r0, r0 + rows) (multiples of 256) on the tensor cores at precision
// prec (SLEMM_PREC_FP16X2, BF16X2 or BF16X3; ops.cu).
void rows_product(slemm_geno* g, int64_t r0, int64_t rows, const float* U, int64_t ldu, int k, float* out,
                  int64_t ldo, int prec);

// exact.cu — exact products of the packed counts with dense columns.
// d_tgv[i] = shift + Σ_j count_ij·d_alpha[j] (FP64 effects, largest magnitude amax, smallest nonzero one amin: ∞
// if there is none).
void exact_gebv(slemm_geno* g, const double* d_alpha, double amax, double amin, double shift, double* d_tgv);
// The columns of exact_dots over individuals i < n, FP32 values in this order: y (when given), rr·Q_l
// for l < cq, rr² (when rr is given; rr == nullptr means every rr is 1).
struct ExactCols {
  const float* y;
  const float* rr;
  const float* Q;
  int64_t ldq;
  int cq;
  int count() const { return (y ? 1 : 0) + cq + (rr ? 1 : 0); }
};
// dots[c·m + j] = Σ_i count_ij·column_c(i) for every SNP j, tot[c] = Σ_i column_c(i) (NaN for a column
// with a non-finite value, and so its dots), and with rr given and twos != nullptr
// twos[j] = 2·Σ_i rr_i²·[count_ij = 2].  Device pointers; at least one column.  The host waits for the columns'
// numbers of digits, or with a guess > 0 queues passes of that many for each: once the caller has waited for the
// stream, exact_dots_done says whether they were enough, and if not all of it is to be run again without a guess.
void exact_dots(slemm_geno* g, const ExactCols& a, double* dots, double* tot, double* twos, int guess = 0);
// The guess of short calls (0: none).  Score terms at n = 3,000, m = 900 take 112 µs with the wait and 101 without;
// 12 digits (36 bits between the largest and the smallest value) of every column cost nothing while the product's N
// is at most 96, where an MMA takes its least time, and past 2^31 counts (0.12 ms a product) the wait is under 3 %.
int exact_dots_guess(const slemm_geno* g, const ExactCols& a);
bool exact_dots_done(const slemm_geno* g, const ExactCols& a, int guess);

// MC-REML's criterion terms (ops.cu), device memory: Py = rr∘e and norms[c] = ‖e_c‖², e_0 = P·PV_0 and
// e_c = P(PV_c + st·PV_{q+c}), c = 1 … q; and X ← √w∘X (m×k), norms[c] = ‖X_c‖².
void first_order_terms(slemm_geno* g, const float* PV, int q, float st, float* Py, double* norms);
void weighted_norms(slemm_geno* g, float* X, int k, double* norms);

// Column reductions with FP64 accumulation, deterministic two-stage (ops.cu).
// dots[c] = Σ_i a[i,c]·b[i,c] over i < n for c < k (b == nullptr → Σ a²).  Result on device.
void col_dots(slemm_geno* g, const float* a, int64_t lda, const float* b, int64_t ldb,
              int64_t n, int k, double* d_out);
// QtX[l,c] = Σ_i Q[i,l]·X[i,c], double c×k on device.
void proj_coeffs(slemm_geno* g, const float* X, int64_t ldx, int k, double* d_QtX);
// X[:,c] -= Σ_l Q[:,l] QtX[l,c].
void proj_apply(slemm_geno* g, float* X, int64_t ldx, int k, const double* d_QtX);

// lanczos.cu — seed on a device RHS block (n×t, ld = n); `groups` splits the columns into
// groups with their own stopping rule (empty = one group).
slemm_lseed* lanczos_seed_device(slemm_geno* g, int kind, float tau0, const float* dB, int t,
                                 float tol, int maxit, bool verbose, std::vector<int> groups,
                                 int p_freq, int nq = 0);
// Solve for the columns of group `grp`; X has that group's columns (ld = ldx) on device.
int lanczos_solve_device(slemm_lseed* S, double sigma, double tol, float* dX, int64_t ldx, int grp);
// Batched tridiagonal eigensolve on the host (FP64 implicit QL per probe over host threads): delta
// nld×t and beta (nld+1)×t in, D and W2 nld×t out, eigenvalues ascending per probe.
void tridiag_eig_host(const double* delta, const double* beta, int t, int nld, double* D, double* W2);
// L_Solve coefficients of group grp at shift σ (X = Σ_i coef[i·tc+c]·V_i[:,c], V_0 = B, V_i = U_i).
int solve_coeffs(const slemm_lseed* S, double sigma, double tol, int grp, std::vector<double>& coef);
// Inner products B[:,a]ᵀV_i[:,b] for i = 0 … J and each (a, b) pair (V_0 = B), host result
// mom[i·npairs + p].
void lanczos_moments(slemm_lseed* S, const std::vector<std::pair<int, int>>& pairs, int J, std::vector<double>& mom);
// Accessors of the seed object (defined in lanczos.cu).
int lseed_iters(const slemm_lseed* S, int grp);
const double* lseed_delta(const slemm_lseed* S);   // iters × t (row j = step j)
const double* lseed_beta(const slemm_lseed* S);    // (iters+1) × t
int lseed_t(const slemm_lseed* S);
void lseed_free(slemm_lseed* S);

// probes.cu — the reference's normalised Rademacher block (n×n_V, ld) on the device.
void rademacher_device(int seed, int64_t n, int n_V, float* dV, int64_t ld, cudaStream_t st);

// The first nA + nB samples of std::normal_distribution<float>(0, 1) over std::mt19937(seed + 54321), the
// first nA into dA, the others into dB (device).  The constructor queues them; finish() waits and checks
// that enough draws were made (and makes more if not): the samples may be used after it.
class NormalDraws {
 public:
  NormalDraws(int seed, int64_t nA, float* dA, int64_t nB, float* dB, cudaStream_t st);
  void finish();

 private:
  void launch();
  uint32_t seed_;
  int64_t nA_, total_, pairs_ = 0;
  float *dA_, *dB_;
  cudaStream_t st_;
  int blocks_ = 0;
  DevBuf words_, offs_;
};

// geno.cu — per-SNP popcounts (missing = 1) and class counts n1 (fields 01), n2 (fields 10).
void row_counts_device(slemm_geno* g, int64_t* pc, int32_t* c1, int32_t* c2);

int64_t workspace_bytes(const slemm_geno* g);
// Reads (and clears) the device error word; throws if a kernel gave up a bounded wait.
void check_device_error(slemm_geno* g);
void profile_collect(slemm_geno* g);

}  // namespace slemm
