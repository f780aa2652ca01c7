// hm_ara.h -- what the stages of the batched ARA build share: the problems of
// a batch, their state, and the launchers of the per-block stages.
//
// Workspace of a problem (working precision W): Q (m x k), Y (m x s) and B
// (n x k), column-major with the row count rounded up to 4 (ara_ld), so that
// every column starts on a 16-byte boundary; the padding rows are zero.
#pragma once
#include <vector>

#include "hm_internal.h"

namespace hm {

constexpr int kMaxCols = 256;  // max basis columns of one block (rank cap)
constexpr int kMaxBs = 32;     // max sample columns of a round

__host__ __device__ __forceinline__ int ara_ld(int rows) { return (rows + 3) & ~3; }

struct Prob {
  int r0, m, c0, n;
  int kmax;
  int level;
  int u, v;
  int gid;                     // its number among the problems that were listed with it (the sample's stream)
  int qcap;                    // columns Q has room for now (<= kmax)
  void *q, *y, *b;             // Q, Y, B in the working precision
  double tscale2;              // (this block's tolerance / the build's)^2: 1, or the level schedule's
};

struct ProbState {
  double normA2;
  double est;
  int k;
  int active;
  int converged;
  int rounds;
  int r;      // rank after truncation (<= k)
  int rhi;    // mixed precision: columns [0, rhi) keep a BF16 low part
};

// ---- orthogonalisation of one round's samples (hm_orth.cu) -------------------
// The problems of a batch by the kernel shape that handles them: the height m
// decides (one CTA with the sample resident in shared memory, or a cluster of
// CTAs that split the rows).
struct OrthPlan {
  struct Class {
    int rows = 0;     // rows of a CTA's slice that stay in shared memory
    int cluster = 1;  // CTAs per problem
    int first = 0, count = 0;  // problems: ids[first .. first + count)
    int kcap = 0;     // widest basis of the class
  };
  std::vector<Class> classes;
  DevBuf<int> ids;
};

// W: float or double.  Fills the plan (ids copied on `s`).
template <typename W>
hm_status orth_plan(const std::vector<Prob>& probs, OrthPlan* plan, cudaStream_t s);

// One ARA round of every active problem: Y's bs sample columns are projected
// against Q, tested (est = ||Y'||^2 / bs <= thresh2 tscale2 ||A||^2), and
// otherwise orthonormalised and appended to Q.
template <typename W>
hm_status orth_round(const OrthPlan& plan, const Prob* probs, ProbState* st, int bs, double thresh2, cudaStream_t s);

// ---- truncation (hm_trunc.cu) --------------------------------------------------
constexpr int kTruncMax = 128;  // widest basis the SVD truncation handles (wider: kept as sampled)

// Eigenvectors of the truncated blocks of a batch: problem p's W_r (k x r,
// FP32, column-major) starts at w + woff[p].
struct TruncWork {
  DevBuf<long long> woff;
  DevBuf<float> w;
};

// From B = A^T Q and the states (k set; hst: their host copies): the rank r
// and low-part columns rhi of every problem, and W_r.  tol2, rbudget: the
// truncation and BF16 rounding budgets relative to ||A||_F^2.
template <typename W>
hm_status trunc_rank(const std::vector<Prob>& bp, const std::vector<ProbState>& hst, const Prob* probs, ProbState* st,
                     double tol2, double rbudget, TruncWork* tw, cudaStream_t s);

// U = Q W_r and V = B W_r of the problems with dst_u >= 0, FP32, column-major
// without padding.  rows, cols: the batch's 64-row tiles (problem, tile) over
// the blocks' rows and columns.
template <typename W>
hm_status trunc_pack(const Prob* probs, const ProbState* st, const TruncWork& tw, const int2* rows, size_t nrows,
                     const int2* cols, size_t ncols, const long long* dst_u, const long long* dst_v,
                     float* dst, cudaStream_t s);

}  // namespace hm
