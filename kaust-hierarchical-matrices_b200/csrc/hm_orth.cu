// hm_orth.cu -- one ARA round per block: projection, stopping test,
// orthonormalisation of the sample.
//
// Per block and round (k basis columns Q, bs <= 32 sample columns Y, m rows):
//   C = Q^T Y, Y -= Q C       twice (classical Gram-Schmidt)
//   est = ||Y||_F^2 / bs      below the threshold: done
//   Y <- orthonormal(Y)       pivoted Cholesky-QR, then two refinements, with
//                             one more projection against Q before the second
//   Q <- [Q Y]
// Gram matrices, their Cholesky factors and the triangular transforms are
// FP64; samples and bases are in the working precision.
//
// What bounds it: the arithmetic is small (4 m k bs + 3 m bs^2 multiply-adds)
// and most blocks are leaf-sized, so a round is a chain of short steps.  Hence
//  - the sample stays in shared memory for the whole round, Q is staged there
//    32 columns at a time and every stage reads both as 16-byte vectors;
//  - the FP64 Gram matrix and the triangular transform run on the FP64 tensor
//    instruction (mma.sync m8n8k4), whose two operands are the same fragment
//    for a Gram tile, so each sample value is loaded and converted once per
//    tile row instead of once per product;
//  - the Cholesky factor is one warp's work (lane = row, left-looking), which
//    forms the inverse factor in the same sweep from the same broadcast reads,
//    so applying it is a matrix product and not a substitution per row;
//  - a block taller than one CTA's shared memory is split over a cluster of up
//    to eight CTAs; C and the Gram matrix are summed through distributed
//    shared memory, each entry by one thread in rank order (deterministic),
//    and every CTA factors its own copy.  Slices beyond the resident rows are
//    streamed from L2, with neighbouring stages fused per chunk.
// Measured against one CTA per block of any height, thread 0 factoring and
// per-thread column arrays in local memory (all rounds of a build, device
// time): 2^17-point Matern (61891 blocks) 114 -> 19.8 ms, 60001-point mixture
// with ranks to 256 (7380 blocks) 230 -> 18.1 ms, 8192-point 2-D exponential
// in FP64 7.0 -> 1.9 ms.  What is left is latency: barriers around the
// single-warp factorisations, and in the tall classes two CTAs per SM.
#include <cooperative_groups.h>

#include <algorithm>

#include "hm_ara.h"
#include "hm_mma.cuh"

namespace hm {
namespace {

namespace cg = cooperative_groups;

constexpr int kGld = 33;  // leading dimension of the 32 x 32 FP64 matrices

template <typename W>
struct Vec;
template <>
struct Vec<float> {
  using T = float4;
  static constexpr int N = 4;
  static __device__ __forceinline__ void get(const T& v, float (&x)[4]) { x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w; }
  static __device__ __forceinline__ T put(const float (&x)[4]) { return make_float4(x[0], x[1], x[2], x[3]); }
};
template <>
struct Vec<double> {
  using T = double2;
  static constexpr int N = 2;
  static __device__ __forceinline__ void get(const T& v, double (&x)[2]) { x[0] = v.x, x[1] = v.y; }
  static __device__ __forceinline__ T put(const double (&x)[2]) { return make_double2(x[0], x[1]); }
};

// The ten 8 x 8 tiles of the upper triangle of a 32 x 32 Gram matrix, dealt to
// four warps (three, three, two, two).
__device__ __forceinline__ void gram_tile(int group, int i, int& a, int& b) {
  // group 0: (0,0) (0,1) (0,2); 1: (0,3) (1,1) (1,2); 2: (1,3) (2,2); 3: (2,3) (3,3)
  const unsigned codes = group == 0 ? 0x020100u : group == 1 ? 0x121103u : group == 2 ? 0xff2213u : 0xff3323u;
  const unsigned c = (codes >> (8 * i)) & 0xffu;
  a = c == 0xffu ? -1 : (int)(c >> 4);
  b = (int)(c & 15u);
}

struct OrthArgs {
  const Prob* probs;
  ProbState* st;
  const int* ids;
  int bs;
  int kcap;
  double thresh2;
};

// Cholesky G[p][p] = L L^T of the first `cols` rows and columns of G with the
// order p chosen by the largest remaining diagonal (pivot) or as it is, and
// Z = P^T L^{-T} in the same sweep: Y Z has orthonormal columns.  Stops at the
// first pivot <= tau; returns the rank r (columns r.. of Z are zero).  Column
// j of L overwrites column p_j of G, which later steps do not read otherwise.
// One warp; lane = row of G and row of Z.
__device__ int chol_inverse(double* G, double* Z, int* perm, int cols, bool pivot, double tau) {
  const int lane = threadIdx.x & 31;
#pragma unroll 8
  for (int j = 0; j < 32; ++j) Z[lane * kGld + j] = 0.0;
  bool open = lane < cols;
  double diag = open ? G[lane * kGld + lane] : 0.0;
  double* grow = G + lane * kGld;
  double* zrow = Z + lane * kGld;
  int r = 0;
  __syncwarp();
  for (int j = 0; j < cols; ++j) {
    int p = j;
    if (pivot) {
      // the largest remaining diagonal by its leading 32 bits (the order of
      // pivots within 1e-6 of each other does not matter), the lowest row first
      const unsigned key = open && diag > 0.0 ? (unsigned)__double2hiint(diag) : 0u;
      const unsigned top = __reduce_max_sync(0xffffffffu, key);
      if (top == 0u) break;
      p = __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
    }
    const double dp = __shfl_sync(0xffffffffu, diag, p);
    if (!(dp > tau)) break;
    const double* prow = G + p * kGld;
    double s0 = grow[p], s1 = 0.0, z0 = lane == p ? 1.0 : 0.0, z1 = 0.0;
    int b = 0;
    for (; b + 1 < j; b += 2) {
      const int c0 = perm[b], c1 = perm[b + 1];
      const double l0 = prow[c0], l1 = prow[c1];
      s0 = fma(-grow[c0], l0, s0);
      s1 = fma(-grow[c1], l1, s1);
      z0 = fma(-l0, zrow[b], z0);
      z1 = fma(-l1, zrow[b + 1], z1);
    }
    if (b < j) {
      const int c0 = perm[b];
      const double l0 = prow[c0];
      s0 = fma(-grow[c0], l0, s0);
      z0 = fma(-l0, zrow[b], z0);
    }
    const double rd = rsqrt(dp);
    double l = open ? (s0 + s1) * rd : 0.0;
    if (lane == p) {
      l = dp * rd;
      open = false;
    }
    diag = fma(-l, l, diag);
    grow[p] = l;  // column p: read by this lane alone so far
    zrow[j] = (z0 + z1) * rd;
    if (lane == 0) perm[j] = p;
    r = j + 1;
    __syncwarp();
  }
  return r;
}

// NT threads, up to RW rows of Y resident per CTA.  CL: a cluster of CTAs
// splits the rows of a block (else one CTA per block).
template <typename W, int NT, int RW, bool CL>
__global__ void __launch_bounds__(NT) k_orth(OrthArgs a) {
  using V = Vec<W>;
  constexpr int N = V::N;
  constexpr int LD = RW + N;         // 16-byte vectors of eight neighbouring columns fall into eight bank groups
  constexpr int NW = NT / 32, H = NW / 4;  // warps; row halves of a Gram matrix
  constexpr int RV = RW / N;
  constexpr int TJ = 32 * 8 / NT;    // rows of C per thread and 32-column group of Q
  constexpr bool kPart = CL || H > 1;  // Gram partials are summed over halves and CTAs
  static_assert(sizeof(double) * H * 32 * kGld <= sizeof(W) * 32 * LD, "Gram partials fit in Q's stage");
  extern __shared__ __align__(16) unsigned char osm[];
  double* Gl = reinterpret_cast<double*>(osm);                 // [32][33]
  double* Zs = Gl + 32 * kGld;                                 // [32][33]
  W* Ys = reinterpret_cast<W*>(Zs + 32 * kGld);                // [32][LD]
  W* Qs = Ys + 32 * LD;                                        // [32][LD]
  double* Gp = reinterpret_cast<double*>(Qs);                  // [H][32][33] Gram partials (kPart) between uses of Qs
  W* Cs = Qs + 32 * LD;                                        // [kcap][32], column c at 4 (c % 8) + c / 8
  __shared__ int perm[32];
  __shared__ int rank_sh;

  const int nrank = CL ? (int)cg::this_cluster().num_blocks() : 1;
  const int rank = CL ? (int)cg::this_cluster().block_rank() : 0;
  const int pid = a.ids[blockIdx.x / nrank];
  ProbState S = a.st[pid];
  if (!S.active) return;  // the whole cluster
  const Prob P = a.probs[pid];
  const int ld = ara_ld(P.m), bs = a.bs;
  const int slice = CL ? ((ld + 4 * nrank - 1) / (4 * nrank)) * 4 : ld;
  const int row0 = min(ld, rank * slice), rows = min(ld, row0 + slice) - row0;
  const int nch = max(1, (rows + RW - 1) / RW);
  const bool resident = nch == 1;
  W* Q = reinterpret_cast<W*>(P.q) + row0;
  W* Y = reinterpret_cast<W*>(P.y) + row0;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int cgi = t & 7;
  int k = S.k;
  int qtag = -1;

  auto sync_all = [&]() {
    if (CL)
      cg::this_cluster().sync();
    else
      __syncthreads();
  };
  // rows [ch RW, ch RW + RW) of `cols` columns of a column-major array (zero beyond) -> dst
  auto load_cols = [&](const W* src, W* dst, int ch, int cols) {
    const int left = rows - ch * RW;
    for (int e = t; e < 32 * RV; e += NT) {
      const int c = e / RV, v = e % RV;
      typename V::T x;
      if (c < cols && v * N < left)
        x = *reinterpret_cast<const typename V::T*>(src + (size_t)c * ld + (size_t)ch * RW + v * N);
      else
        x = typename V::T{};
      *reinterpret_cast<typename V::T*>(dst + c * LD + v * N) = x;
    }
  };
  auto store_cols = [&](W* dst, int ch, int cols) {
    const int left = rows - ch * RW;
    for (int e = t; e < cols * RV; e += NT) {
      const int c = e / RV, v = e % RV;
      if (v * N < left)
        *reinterpret_cast<typename V::T*>(dst + (size_t)c * ld + (size_t)ch * RW + v * N) =
            *reinterpret_cast<const typename V::T*>(Ys + c * LD + v * N);
    }
  };
  auto stage_q = [&](int ch, int g) {
    const int tag = ch * 16 + g;
    if (qtag == tag) return;
    qtag = tag;
    __syncthreads();
    load_cols(Q + (size_t)(32 * g) * ld, Qs, ch, k - 32 * g);
    __syncthreads();
  };
  const int ngroups = (k + 31) >> 5;
  // C (+)= Q^T Y over chunk ch
  auto project = [&](int ch) {
    for (int g = 0; g < ngroups; ++g) {
      stage_q(ch, g);
      W acc[TJ][4];
#pragma unroll
      for (int q = 0; q < TJ; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = W(0);
      const int j0 = t >> 3;
      const int rv = min(RV, (rows - ch * RW + N - 1) / N);
#pragma unroll 2
      for (int v = 0; v < rv; ++v) {
        W q[TJ][N], y[4][N];
#pragma unroll
        for (int i = 0; i < TJ; ++i)
          V::get(*reinterpret_cast<const typename V::T*>(Qs + (j0 + i * (NT / 8)) * LD + v * N), q[i]);
#pragma unroll
        for (int b = 0; b < 4; ++b)
          V::get(*reinterpret_cast<const typename V::T*>(Ys + (cgi + 8 * b) * LD + v * N), y[b]);
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
          for (int i = 0; i < TJ; ++i)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[i][b] = fma(q[i][n], y[b][n], acc[i][b]);
      }
#pragma unroll
      for (int i = 0; i < TJ; ++i) {
        W* c = Cs + (32 * g + j0 + i * (NT / 8)) * 32 + 4 * cgi;
#pragma unroll
        for (int b = 0; b < 4; ++b) c[b] = ch == 0 ? acc[i][b] : c[b] + acc[i][b];
      }
    }
    __syncthreads();
  };
  // the whole C in every CTA of the cluster
  auto sum_c = [&]() {
    if (!CL) return;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    for (int e = rank * NT + t; e < ngroups * 32 * 32; e += nrank * NT) {
      W s = W(0);
      for (int q = 0; q < nrank; ++q) s += *cl.map_shared_rank(Cs + e, q);
      for (int q = 0; q < nrank; ++q) *cl.map_shared_rank(Cs + e, q) = s;
    }
    cl.sync();
  };
  // Y -= Q C over chunk ch
  auto subtract = [&](int ch) {
    for (int g = 0; g < ngroups; ++g) {
      stage_q(ch, g);
      const int nj = min(32, k - 32 * g);
      for (int w = t; w < RV * 8; w += NT) {
        const int v = w >> 3;  // w & 7 == cgi
        W y[4][N];
#pragma unroll
        for (int b = 0; b < 4; ++b)
          V::get(*reinterpret_cast<const typename V::T*>(Ys + (cgi + 8 * b) * LD + v * N), y[b]);
#pragma unroll 4
        for (int j = 0; j < nj; ++j) {
          W q[N];
          V::get(*reinterpret_cast<const typename V::T*>(Qs + j * LD + v * N), q);
          const W* c = Cs + (32 * g + j) * 32 + 4 * cgi;
          W cv[4];
#pragma unroll
          for (int b = 0; b < 4; ++b) cv[b] = c[b];
#pragma unroll
          for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int n = 0; n < N; ++n) y[b][n] = fma(-q[n], cv[b], y[b][n]);
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
          *reinterpret_cast<typename V::T*>(Ys + (cgi + 8 * b) * LD + v * N) = V::put(y[b]);
      }
      __syncthreads();
    }
  };
  // Gram accumulators of this warp's tiles, kept over the chunks
  double ga[3][2];
  const int gg = warp & 3, gh = warp >> 2;
  auto gram_clear = [&]() {
#pragma unroll
    for (int i = 0; i < 3; ++i) ga[i][0] = ga[i][1] = 0.0;
  };
  auto gram_add = [&](int ch) {
    const int nq = (min(RW, rows - ch * RW) + 3) >> 2;  // row quads
    int ta[3], tb[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) gram_tile(gg, i, ta[i], tb[i]);
    const W* y = Ys + (lane >> 2) * LD + (lane & 3);
    for (int q = gh; q < nq; q += H) {
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (ta[i] >= 0)
          mma_f64(ga[i], (double)y[8 * ta[i] * LD + 4 * q], (double)y[8 * tb[i] * LD + 4 * q]);
    }
  };
  // -> Gl in every CTA (both triangles)
  auto gram_done = [&]() {
    double* dst = kPart ? Gp + gh * 32 * kGld : Gl;
    const int g = lane >> 2, c = 2 * (lane & 3);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      int x, y;
      gram_tile(gg, i, x, y);
      if (x < 0) continue;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = 8 * x + g, s = 8 * y + c + u;
        if (r <= s) {
          dst[r * kGld + s] = ga[i][u];
          if (!kPart) dst[s * kGld + r] = ga[i][u];
        }
      }
    }
    if (!kPart) {
      __syncthreads();
      return;
    }
    qtag = -1;
    sync_all();
    for (int e = rank * NT + t; e < 32 * 32; e += nrank * NT) {
      const int r = e >> 5, s = e & 31;
      if (r > s) continue;
      double v = 0.0;
      for (int q = 0; q < nrank; ++q)
        for (int h = 0; h < H; ++h) {
          double* part = Gp + (h * 32 + r) * kGld + s;
          v += CL ? *cg::this_cluster().map_shared_rank(part, q) : *part;
        }
      for (int q = 0; q < nrank; ++q) {
        double* up = Gl + r * kGld + s;
        double* lo = Gl + s * kGld + r;
        if (CL) {
          *cg::this_cluster().map_shared_rank(up, q) = v;
          *cg::this_cluster().map_shared_rank(lo, q) = v;
        } else {
          *up = v;
          *lo = v;
        }
      }
    }
    sync_all();
  };
  // Y <- Y Z over chunk ch (columns beyond the rank become zero)
  auto transform = [&](int ch, int cols) {
    const int nr8 = (min(RW, rows - ch * RW) + 7) >> 3;
    const int nq = (cols + 3) >> 2;
    const int g = lane >> 2, c = lane & 3;
    for (int i = warp; i < nr8; i += NW) {
      double d[4][2];
#pragma unroll
      for (int n = 0; n < 4; ++n) d[n][0] = d[n][1] = 0.0;
      for (int q = 0; q < nq; ++q) {
        const double y = (double)Ys[(4 * q + c) * LD + 8 * i + g];
        const double* z = Zs + (4 * q + c) * kGld + g;
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_f64(d[n], y, z[8 * n]);
      }
      __syncwarp();  // the warp's rows have been read
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        Ys[(8 * n + 2 * c) * LD + 8 * i + g] = (W)d[n][0];
        Ys[(8 * n + 2 * c + 1) * LD + 8 * i + g] = (W)d[n][1];
      }
    }
    __syncthreads();
  };
  // every chunk of Y in turn through shared memory; keep: write it back
  auto chunks = [&](bool keep, auto&& body) {
    for (int ch = 0; ch < nch; ++ch) {
      if (!resident) {
        __syncthreads();
        load_cols(Y, Ys, ch, bs);
        __syncthreads();
      }
      body(ch);
      if (!resident && keep) {
        __syncthreads();
        store_cols(Y, ch, bs);
      }
    }
  };
  auto factor = [&](int cols, bool pivot, double tau) {
    if (warp == 0) {
      const int r = chol_inverse(Gl, Zs, perm, cols, pivot, tau);
      if (lane == 0) rank_sh = r;
    }
    __syncthreads();
    return rank_sh;
  };

  if (resident) {
    load_cols(Y, Ys, 0, bs);
    __syncthreads();
  }
  // ---- projection against the basis, twice ----
  gram_clear();
  if (k > 0) {
    chunks(false, [&](int ch) { project(ch); });
    sum_c();
    // the second pass writes C while no CTA reads it: each CTA sums its own
    // chunks only after its last use of the first C
    if (resident) {
      subtract(0);
      project(0);
    } else {
      chunks(true, [&](int ch) { subtract(ch); });
      chunks(false, [&](int ch) { project(ch); });
    }
    sum_c();
    chunks(true, [&](int ch) {
      subtract(ch);
      gram_add(ch);
    });
  } else {
    chunks(false, [&](int ch) { gram_add(ch); });
  }
  gram_done();
  // ---- stopping test ----
  double tr = 0.0;
  for (int c = 0; c < bs; ++c) tr += Gl[c * kGld + c];
  const double est = tr / bs;
  const bool conv = est <= a.thresh2 * P.tscale2 * S.normA2 || S.normA2 == 0.0;
  const bool capped = !conv && k + bs > P.kmax;
  __syncthreads();  // the diagonal has been read
  int r = 0;
  if (!conv && !capped) {
    // ---- orthonormalisation; columns below 1e-5 of the sample's norm are noise ----
    r = factor(bs, true, 1e-10 * tr);
    if (r > 0) {
      gram_clear();
      chunks(true, [&](int ch) {
        transform(ch, bs);
        gram_add(ch);
      });
      gram_done();
      int cols = r;
      r = factor(cols, false, 0.0);
      if (r > 0) {
        gram_clear();
        if (k > 0) {
          // R^{-1} of an ill-conditioned sample magnifies whatever the
          // Gram-Schmidt passes left along the basis: project once more
          chunks(true, [&](int ch) {
            transform(ch, cols);
            project(ch);
          });
          sum_c();
          chunks(true, [&](int ch) {
            subtract(ch);
            gram_add(ch);
          });
        } else {
          chunks(true, [&](int ch) {
            transform(ch, cols);
            gram_add(ch);
          });
        }
        gram_done();
        cols = r;
        r = factor(cols, true, 1e-12 * cols);  // a refinement that loses rank keeps the leading columns
        if (r > 0)
          chunks(false, [&](int ch) {
            transform(ch, cols);
            store_cols(Q + (size_t)k * ld, ch, r);
          });
      }
    }
  }
  if (CL) cg::this_cluster().sync();  // no CTA leaves while another may still read its shared memory
  if (rank == 0 && t == 0) {
    S.est = est;
    S.rounds += 1;
    S.k = k + r;
    if (conv || capped || r == 0) {
      S.active = 0;
      S.converged = !capped;
    }
    a.st[pid] = S;
  }
}

// Rows a CTA keeps resident: as many as leave room for Q's stage and C at the
// widest basis (256 columns) in either precision.
template <typename W>
constexpr int tall_rows() {
  return sizeof(W) == 4 ? 256 : 128;
}

template <typename W, int RW>
size_t orth_smem(int kcap) {
  return sizeof(double) * 32 * kGld * 2 + sizeof(W) * 2 * 32 * (RW + Vec<W>::N) + sizeof(W) * (size_t)kcap * 32;
}

template <typename W, int NT, int RW, bool CL>
hm_status launch(const OrthPlan::Class& c, OrthArgs a, cudaStream_t s) {
  const size_t smem = orth_smem<W, RW>(c.kcap);
  // the limit is the function's, not this launch's: always that of the widest
  // basis, so that threads that build at once do not lower one another's
  HM_CUDA(cudaFuncSetAttribute(k_orth<W, NT, RW, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)orth_smem<W, RW>(kMaxCols)));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)c.count * c.cluster);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)c.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  if (CL) {
    cfg.attrs = &at;
    cfg.numAttrs = 1;
  }
  HM_CUDA(cudaLaunchKernelEx(&cfg, k_orth<W, NT, RW, CL>, a));
  return HM_OK;
}

}  // namespace

// Heights: up to 64 and up to 128 rows on 128 threads (several CTAs per SM),
// up to tall_rows on 256 threads, above that clusters of 2, 4 and 8 CTAs so
// that a slice stays resident up to 8 tall_rows rows.
template <typename W>
hm_status orth_plan(const std::vector<Prob>& probs, OrthPlan* plan, cudaStream_t s) {
  constexpr int kTall = tall_rows<W>();
  const int top[6] = {64, 128, kTall, 2 * kTall, 4 * kTall, 1 << 30};
  std::vector<int> of[6];
  int kcap[6] = {};
  for (size_t i = 0; i < probs.size(); ++i) {
    int c = 0;
    while (probs[i].m > top[c]) ++c;
    of[c].push_back((int)i);
    kcap[c] = std::max(kcap[c], probs[i].kmax);
  }
  std::vector<int> ids;
  plan->classes.clear();
  for (int c = 5; c >= 0; --c) {  // the tall blocks first: their rounds are the longest
    if (of[c].empty()) continue;
    OrthPlan::Class k;
    k.rows = std::min(top[c], kTall);
    k.cluster = c < 3 ? 1 : 1 << (c - 2);
    k.first = (int)ids.size();
    k.count = (int)of[c].size();
    k.kcap = (kcap[c] + 31) & ~31;
    plan->classes.push_back(k);
    ids.insert(ids.end(), of[c].begin(), of[c].end());
  }
  HM_TRY(plan->ids.alloc_async(std::max<size_t>(ids.size(), 1), s));
  HM_CUDA(cudaMemcpyAsync(plan->ids.p, ids.data(), sizeof(int) * ids.size(), cudaMemcpyHostToDevice, s));
  return HM_OK;
}

template <typename W>
hm_status orth_round(const OrthPlan& plan, const Prob* probs, ProbState* st, int bs, double thresh2,
                     cudaStream_t s) {
  constexpr int kTall = tall_rows<W>();
  for (const OrthPlan::Class& c : plan.classes) {
    OrthArgs a{probs, st, plan.ids.p + c.first, bs, c.kcap, thresh2};
    if (c.cluster > 1)
      HM_TRY((launch<W, 256, kTall, true>(c, a, s)));
    else if (c.rows <= 64)
      HM_TRY((launch<W, 128, 64, false>(c, a, s)));
    else if (c.rows <= 128)
      HM_TRY((launch<W, 128, 128, false>(c, a, s)));
    else if constexpr (kTall > 128)
      HM_TRY((launch<W, 256, kTall, false>(c, a, s)));
  }
  return HM_OK;
}

template hm_status orth_plan<float>(const std::vector<Prob>&, OrthPlan*, cudaStream_t);
template hm_status orth_plan<double>(const std::vector<Prob>&, OrthPlan*, cudaStream_t);
template hm_status orth_round<float>(const OrthPlan&, const Prob*, ProbState*, int, double, cudaStream_t);
template hm_status orth_round<double>(const OrthPlan&, const Prob*, ProbState*, int, double, cudaStream_t);

}  // namespace hm
