// hm_hmatrix.cu -- H-matrix construction by batched adaptive randomized
// approximation (ARA) on kernel entries generated from the points.
//
// Reference: createColumnMajorLRMatrix (src/constructTLRMatrix.cu:13-151)
// compresses leaf tiles with kblas_ara_batch and generateHMatrixFromStruct
// (src/constructHMatrixFromStruct.cu:13-103) recompresses coarser blocks from
// the leaf factors with lr_kblas_ara_batch, both from the un-vendored KBLAS
// fork.  The ARA they call is the blocked adaptive range finder of Halko,
// Martinsson & Tropp (2011, Alg. 4.2) as batched by Boukaram, Turkiyyah &
// Keyes (2019): draw a Gaussian sample block, project out the basis found so
// far, stop when the sample's norm says the residual is below the tolerance,
// otherwise orthonormalise it and append it; finally B = A^T Q, A ~ Q B^T.
//
// B200 design.  Every block of every level is compressed directly from the
// kernel function (no dense tiles in HBM, no leaf-TLR stage): each ARA pass is
// one batched "kernel block x tall-skinny" launch (k_kmm_fast and its FP64 and
// general forms) whose tiles are generated on the fly from the tree-ordered
// FP32 coordinates, so the O(N^2) part never touches memory.  Orthogonalisation
// runs per block in one CTA, tall blocks in a cluster of up to eight
// (hm_orth.cu): block classical Gram-Schmidt applied twice against the basis,
// then a pivoted Cholesky-QR of the sample with two Cholesky-QR refinements,
// Gram matrices in FP64.  The kernel matrix
// is symmetric, so of each block pair (u, v) / (v, u) only the one with v > u is
// compressed; the mirror block uses the same factors exchanged.  Leaf blocks
// that do not reach the tolerance within the leaf rank cap (bucket/2 as in
// src/constructTLRMatrix.cu:14) are stored dense, as are the diagonal leaves.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <array>
#include <numeric>
#include <type_traits>

#include "hm_ara.h"
#include "hm_hmatrix.h"
#include "hm_mma.cuh"
#include "hm_structure.h"

namespace hm {

hm_status matvec_plan_build(hm_hmatrix h, int nrhs_cap, cudaStream_t stream);

namespace {

constexpr int kTR = 64;        // rows of a KMM tile
constexpr int kTC = 64;        // columns per KMM chunk
constexpr int kKmmThreads = 256;
constexpr int kColGroup = 128; // projection columns per sketch launch
constexpr int kQCols = 64;     // basis columns a problem starts with room for
template <typename W>
struct KmmArgs {
  const Prob* probs;
  ProbState* st;
  const int2* items;  // (problem, tile)
  const float* pts;   // tree-ordered FP32 coordinates [d][npts]
  int npts, d;
  KernelParams kp;
  int mode;           // 0: Y = A Omega (bs columns); 1: B = A^T Q (k columns)
  int col0;           // projection: first basis column of this launch (128 per launch)
  int bs;
  uint32_t seed;
  int round;
};

// ---------------------------------------------------------------------------
// k_kmm: out(rows x s) = K(rows, cols) W(cols x s) for one 64-row tile.
// Thread t: row r = t % 64, q = t / 64 splits the s output columns into
// `nslab` slabs of 32 and the chunk columns into 4/nslab groups.  FP32 working
// precision in more than three dimensions (the others: k_kmm_fast, k_kmm64).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kKmmThreads) k_kmm(KmmArgs<float> a) {
  using W = float;
  extern __shared__ __align__(16) unsigned char kmm_raw[];
  W* Wsm = reinterpret_cast<W*>(kmm_raw);          // [kTC][kColGroup]
  float* Asm = reinterpret_cast<float*>(Wsm + kTC * kColGroup);  // [kTC][kTR]
  float* colc = Asm + kTC * kTR;                   // [d][kTC]
  double* red = reinterpret_cast<double*>(colc + kMaxDim * kTC);  // [kKmmThreads/32]

  const int2 it = a.items[blockIdx.x];
  const Prob P = a.probs[it.x];
  const ProbState S = a.st[it.x];
  if (a.mode == 0 && !S.active) return;
  const int col0 = a.mode ? a.col0 : 0;
  const int s = min(kColGroup, (a.mode == 0 ? a.bs : S.k) - col0);
  if (s <= 0) return;
  const int mr = a.mode ? P.n : P.m;        // rows of the operator
  const int nc = a.mode ? P.m : P.n;        // columns of the operator
  const int rbase = a.mode ? P.c0 : P.r0;
  const int cbase = a.mode ? P.r0 : P.c0;
  const int ldo = ara_ld(mr), ldq = ara_ld(P.m);
  W* out = reinterpret_cast<W*>(a.mode ? P.b : P.y) + (size_t)col0 * ldo;
  const W* Q = reinterpret_cast<const W*>(P.q) + (size_t)col0 * ldq;  // mode 1: W = Q (m x k)
  const int nslab = s <= 32 ? 1 : (s <= 64 ? 2 : 4);
  const int ncg = 4 / nslab;
  const int t = threadIdx.x, r = t & 63, q = t >> 6;
  const int slab = q % nslab, cg = q / nslab;
  const int row = it.y * kTR + r;
  const bool row_ok = row < mr;
  float rc[kMaxDim];
#pragma unroll
  for (int k = 0; k < kMaxDim; ++k)
    rc[k] = (k < a.d && row_ok) ? a.pts[(size_t)k * a.npts + rbase + row] : 0.f;
  W acc[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) acc[c] = W(0);
  double nrm = 0.0;
  const bool want_norm = a.mode == 0 && a.round == 0;
  const int wcols = nslab * 32;

  for (int c0 = 0; c0 < nc; c0 += kTC) {
    // column coordinates and the W chunk
    if (t < kTC) {
      int j = c0 + t;
      for (int k = 0; k < a.d; ++k) colc[k * kTC + t] = j < nc ? a.pts[(size_t)k * a.npts + cbase + j] : 0.f;
    }
    for (int e = t; e < kTC * wcols; e += kKmmThreads) {
      int jj = e % kTC, cc = e / kTC;
      int j = c0 + jj;
      W w = W(0);
      if (j < nc && cc < s) {
        if (a.mode == 0)
          w = (W)gauss_at(a.seed, (uint32_t)P.gid, (uint32_t)j, (uint32_t)(a.round * kMaxBs + cc));
        else
          w = Q[(size_t)cc * ldq + j];
      }
      Wsm[jj * kColGroup + cc] = w;
    }
    __syncthreads();
    // kernel entries of this thread's row, columns q, q+4, ...
    for (int jj = q; jj < kTC; jj += 4) {
      float v = 0.f;
      if (row_ok && c0 + jj < nc) {
        float r2 = 0.f;
        for (int k = 0; k < a.d; ++k) {
          float df = rc[k] - colc[k * kTC + jj];
          r2 = fmaf(df, df, r2);
        }
        v = kernel_r2(a.kp, r2);
        if (want_norm) nrm += (double)v * (double)v;
      }
      Asm[jj * kTR + r] = v;
    }
    __syncthreads();
    for (int jj = cg; jj < kTC; jj += ncg) {
      W av = (W)Asm[jj * kTR + r];
      const W* w = Wsm + jj * kColGroup + slab * 32;
#pragma unroll
      for (int c = 0; c < 32; ++c) acc[c] = fma(av, w[c], acc[c]);
    }
    __syncthreads();
  }
  // reduce over column groups through shared memory (reuses Asm/Wsm)
  if (ncg > 1) {
    W* part = Wsm;  // [4][32][64] (reuses the W chunk)
    for (int c = 0; c < 32; ++c) part[(q * 32 + c) * kTR + r] = acc[c];
    __syncthreads();
    if (cg == 0) {
      for (int g = 1; g < ncg; ++g) {
        int qq = g * nslab + slab;
        for (int c = 0; c < 32; ++c) acc[c] += part[(qq * 32 + c) * kTR + r];
      }
    }
  }
  if (cg == 0 && row < ldo) {  // the padding rows get their zeros
    for (int c = 0; c < 32; ++c) {
      int col = slab * 32 + c;
      if (col < s) out[(size_t)col * ldo + row] = acc[c];
    }
  }
  if (want_norm) {
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    __syncthreads();
    if ((t & 31) == 0) red[t >> 5] = nrm;
    __syncthreads();
    if (t == 0) {
      double tot = 0;
      for (int w = 0; w < kKmmThreads / 32; ++w) tot += red[w];
      atomicAdd(&a.st[it.x].normA2, tot);
    }
  }
}

// ---------------------------------------------------------------------------
// k_kmm64: the same product in FP64 (tolerances below what FP32 sums resolve)
// on the FP64 tensor instruction (mma.sync m8n8k4).  CTA = 4 warps = 64
// operator rows, warp = 16 rows: a lane evaluates two FP32 kernel entries per
// four columns, which are its A fragments; the right-hand operand (Gaussian
// numbers, or the basis) is staged as FP64, 64 rows at a time.  A warp whose
// rows lie past the block only helps to stage.
// Bound by the FP64 pipe (8 NT multiply-adds per entry) and the entries' 25
// instructions alike.  Measured against one row per thread with FP64 FMAs on 32
// columns whatever the sample's width: a 120000-point 2-D build's sketches and
// projections 482 -> 155 ms.
// D: dimension compiled for (0: any); NT: column tiles of 8.
// ---------------------------------------------------------------------------
template <int D, int NT>
__global__ void __launch_bounds__(128) k_kmm64(KmmArgs<double> a) {
  constexpr int LDC = 8 * NT + 4;  // a half-warp's 4 rows x 4 columns fall into 16 banks
  constexpr int DD = D ? D : kMaxDim;
  __shared__ double Wsm[kTC * LDC];
  __shared__ float colc[DD][kTC];
  __shared__ double red[4];
  const int2 it = a.items[blockIdx.x];
  const Prob P = a.probs[it.x];
  const ProbState S = a.st[it.x];
  if (a.mode == 0 && !S.active) return;
  const int col0 = a.mode ? a.col0 : 0;
  const int s = min(8 * NT, (a.mode == 0 ? a.bs : S.k) - col0);
  if (s <= 0) return;
  const int d = D ? D : a.d;
  const int mr = a.mode ? P.n : P.m;        // rows of the operator
  const int nc = a.mode ? P.m : P.n;        // columns of the operator
  const int rbase = a.mode ? P.c0 : P.r0;
  const int cbase = a.mode ? P.r0 : P.c0;
  const int ldo = ara_ld(mr), ldq = ara_ld(P.m);
  double* out = reinterpret_cast<double*>(a.mode ? P.b : P.y) + (size_t)col0 * ldo;
  const double* Q = reinterpret_cast<const double*>(P.q) + (size_t)col0 * ldq;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int row0 = it.y * kTR + warp * 16;
  const bool busy = row0 < mr;  // the whole warp
  const int ra = row0 + g, rb = ra + 8;
  const bool ra_ok = ra < mr, rb_ok = rb < mr;
  float rca[DD], rcb[DD];
#pragma unroll
  for (int k = 0; k < DD; ++k) {
    rca[k] = k < d && ra_ok ? a.pts[(size_t)k * a.npts + rbase + ra] : 0.f;
    rcb[k] = k < d && rb_ok ? a.pts[(size_t)k * a.npts + rbase + rb] : 0.f;
  }
  const int ntiles = (s + 7) >> 3;
  double acc[2][NT][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[i][n][0] = acc[i][n][1] = 0.0;
  double nrm = 0.0;
  const bool want_norm = a.mode == 0 && a.round == 0;
  for (int c0 = 0; c0 < nc; c0 += kTC) {
    __syncthreads();
    for (int e = tid; e < d * kTC; e += 128) {
      const int k = e / kTC, j = c0 + e % kTC;
      colc[k][e % kTC] = j < nc ? a.pts[(size_t)k * a.npts + cbase + j] : 0.f;
    }
    for (int e = tid; e < kTC * 8 * ntiles; e += 128) {
      const int jj = e % kTC, cc = e / kTC, j = c0 + jj;
      double w = 0.0;
      if (j < nc && cc < s)
        w = a.mode == 0 ? (double)gauss_at(a.seed, (uint32_t)P.gid, (uint32_t)j, (uint32_t)(a.round * kMaxBs + cc))
                        : Q[(size_t)cc * ldq + j];
      Wsm[jj * LDC + cc] = w;
    }
    __syncthreads();
    if (!busy) continue;
    const int nq = (min(kTC, nc - c0) + 3) >> 2;
    for (int q = 0; q < nq; ++q) {
      const int jj = 4 * q + t;
      float r2a = 0.f, r2b = 0.f;
#pragma unroll
      for (int k = 0; k < DD; ++k) {
        if (D || k < d) {
          const float c = colc[k][jj], da = rca[k] - c, db = rcb[k] - c;
          r2a = fmaf(da, da, r2a);
          r2b = fmaf(db, db, r2b);
        }
      }
      const bool in = c0 + jj < nc;
      const double va = in && ra_ok ? (double)kernel_r2(a.kp, r2a) : 0.0;
      const double vb = in && rb_ok ? (double)kernel_r2(a.kp, r2b) : 0.0;
      if (want_norm) nrm = fma(va, va, fma(vb, vb, nrm));
      const double* w = Wsm + jj * LDC + g;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        if (n < ntiles) {
          const double b = w[8 * n];
          mma_f64(acc[0][n], va, b);
          mma_f64(acc[1][n], vb, b);
        }
      }
    }
  }
  if (busy) {  // rows mr .. ldo - 1 (padding) get their zeros
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      if (n >= ntiles) continue;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = 8 * n + 2 * t + u;
        if (c < s) {
          if (ra < ldo) out[(size_t)c * ldo + ra] = acc[0][n][u];
          if (rb < ldo) out[(size_t)c * ldo + rb] = acc[1][n][u];
        }
      }
    }
  }
  if (want_norm) {
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) red[warp] = nrm;
    __syncthreads();
    if (tid == 0) atomicAdd(&a.st[it.x].normA2, red[0] + red[1] + red[2] + red[3]);
  }
}

template <int NT>
void launch_kmm64(unsigned grid, cudaStream_t s, const KmmArgs<double>& a) {
  if (a.d == 1)
    k_kmm64<1, NT><<<grid, 128, 0, s>>>(a);
  else if (a.d == 2)
    k_kmm64<2, NT><<<grid, 128, 0, s>>>(a);
  else if (a.d == 3)
    k_kmm64<3, NT><<<grid, 128, 0, s>>>(a);
  else
    k_kmm64<0, NT><<<grid, 128, 0, s>>>(a);
}
// cols: right-hand columns the launch must cover, at most kGroup64
constexpr int kGroup64 = 64;
void launch_kmm64(int cols, unsigned grid, cudaStream_t s, const KmmArgs<double>& a) {
  if (cols <= 16)
    launch_kmm64<2>(grid, s, a);
  else if (cols <= 32)
    launch_kmm64<4>(grid, s, a);
  else
    launch_kmm64<8>(grid, s, a);
}

// ---------------------------------------------------------------------------
// k_kmm_fast: the same product on the tensor cores (FP32 working precision),
// specialised on the dimension (1-3), the kernel and its derivative.  CTA = 4
// warps = 64 operator rows, warp = 16 rows; each lane evaluates the eight
// kernel entries of its m16n8k16 A fragment in registers and splits them into
// BF16 hi + lo (relative error ~2^-17 of an entry).  Sample pass: W = a Gaussian
// table whose entries are BF16 numbers, 2 MMAs per tile.  Projection pass: W = Q
// split hi + lo, 3 MMAs per tile (hi*hi, lo*hi, hi*lo).  Coordinates are
// pre-scaled so that each entry costs one hardware square root and one hardware
// exp2 (PTX sqrt.approx / ex2.approx, both within a few ulp of FP32), the row
// coordinates stay in registers, and the right-hand operand (the Gaussian table
// in sampling mode, the basis Q in projection mode) is read as prepacked BF16
// pairs straight from L1/L2 instead of being restaged per chunk.
// Instruction issue bounds it, then the special-function unit (two of its
// operations per entry; 75 % busy with 16 sampled columns): distances, kernel
// values, the norm and the splits are done two entries per instruction
// (FP32 pairs), only a block's ragged last step masks columns, and the MMAs of
// a k-step stand in one straight run (the tables are padded to the tiles the
// variant takes, so there is no test per tile).  First sampling round of a
// 2^17-point 3-D Matern build, one batch: 32 columns 8.0 -> 5.7 ms, 16 columns
// 6.4 -> 4.4 ms.
// ---------------------------------------------------------------------------
constexpr int kCC = 128;  // columns per coordinate chunk
// column tiles of 8 of the right-hand tables: the Gaussian table has as many
// as the sampling kernel's variant multiplies (its padding tiles are zeros),
// the basis table an even number
__host__ __device__ constexpr int sample_tiles(int bs) { return bs <= 16 ? 2 : bs <= 32 ? 4 : 8; }
__host__ __device__ constexpr int q_tiles(int k) { return (k + 15) >> 4 << 1; }

struct KmmFastArgs {
  const Prob* probs;
  ProbState* st;
  const int2* items;
  const float* pts;
  int npts;
  float scale;   // coordinate scale (see kval)
  float dscale;  // derivative factor
  int deriv;     // entries of dK/dl instead of K
  int bs, round;
  // right-hand operand tables in fragment order: word (k-step, column tile,
  // lane (g,t)) holds the m16n8k16 B fragment {b0, b1} with
  // b0 = {W[16 ks + 2t][8 nt + g], W[16 ks + 2t + 1][..]}, b1 = rows + 8
  const uint2* om;          // sampling: the Gaussian table, NT column tiles (see sample_tiles)
  const uint4* qt;          // projection: {hi b0, hi b1, lo b0, lo b1} of Q, per problem, tiles in pairs
  const long long* qpoff;   // per problem (batch index), 16-byte words
  int col0;                 // projection: first basis column of this launch
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr float kLn2f = 0.6931471805599453f;

// r2: squared distances of the scaled coordinates, two entries.
//   KIND 0 (exp):    scale = log2(e)/l,         a = r log2(e)/l,  K = 2^-a
//   KIND 1 (Matern): scale = sqrt(3) log2(e)/l,  K = (1 + a ln2) 2^-a
//   KIND 2 (Gauss):  scale = sqrt(log2(e)/2)/l,  K = 2^-r2
// derivatives dK/dl: exp a ln2 K / l, Matern (a ln2)^2 2^-a / l,
// Gauss K q / l with q = r^2/l^2 = 2 ln2 r2.
template <int KIND, bool DERIV>
__device__ __forceinline__ f32x2 kval2(f32x2 r2, f32x2 dscale) {
  float x, y;
  unpack2(r2, x, y);
  if (KIND == 2) {
    const f32x2 v = pack2(ex2_approx(-x), ex2_approx(-y));
    return DERIV ? mul2(mul2(v, r2), dscale) : v;
  }
  x = sqrt_approx(x);
  y = sqrt_approx(y);
  const f32x2 a = pack2(x, y), e = pack2(ex2_approx(-x), ex2_approx(-y));
  if (KIND == 1) {
    const f32x2 ln2 = pack2(kLn2f, kLn2f);
    const f32x2 al = mul2(a, ln2);
    return DERIV ? mul2(mul2(mul2(al, al), e), dscale) : mul2(fma2(a, ln2, pack2(1.f, 1.f)), e);
  }
  return DERIV ? mul2(mul2(a, e), dscale) : e;
}

// CTAs an SM shall hold.  Projection of up to 64 columns: 3 (151 registers) 11.1
// ms, 4 9.1, 5 8.5; two sampled tiles: 8 or 9 4.8 ms, left to the compiler (0) 4.4.
constexpr int kmm_ctas(int nt) { return nt == 2 ? 0 : nt == 4 ? 8 : nt == 8 ? 5 : 3; }

template <int D, int KIND, int MODE, int NT>
__global__ void __launch_bounds__(128, kmm_ctas(NT)) k_kmm_fast(KmmFastArgs a) {
  __shared__ __align__(8) float colc[D][kCC];  // negated: a difference is one packed add
  __shared__ double red[4];
  const int2 it = a.items[blockIdx.x];
  const Prob P = a.probs[it.x];
  const ProbState S = a.st[it.x];
  if (MODE == 0 && !S.active) return;
  const int col0 = MODE ? a.col0 : 0;
  const int s = (MODE == 0 ? a.bs : S.k) - col0;  // output columns of this launch
  if (s <= 0) return;
  const int mr = MODE ? P.n : P.m;
  const int nc = MODE ? P.m : P.n;
  const int rbase = MODE ? P.c0 : P.r0;
  const int cbase = MODE ? P.r0 : P.c0;
  const int ld = ara_ld(mr);
  float* out = reinterpret_cast<float*>(MODE ? P.b : P.y) + (size_t)col0 * ld;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ra = it.y * kTR + warp * 16 + g, rb = ra + 8;
  const bool ra_ok = ra < mr, rb_ok = rb < mr;
  const bool deriv = a.deriv != 0;
  f32x2 rca[D], rcb[D];
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const float xa = ra_ok ? a.pts[(size_t)k * a.npts + rbase + ra] * a.scale : 0.f;
    const float xb = rb_ok ? a.pts[(size_t)k * a.npts + rbase + rb] * a.scale : 0.f;
    rca[k] = pack2(xa, xa);
    rcb[k] = pack2(xb, xb);
  }
  const f32x2 dscale = pack2(a.dscale, a.dscale);
  static_assert(NT % 2 == 0, "column tiles are taken in pairs");
  const int tnt = MODE ? q_tiles(S.k) : NT;  // column tiles of the table
  const int ntiles = MODE ? min(NT, tnt - (col0 >> 3)) : NT;
  const uint4* qt = MODE ? a.qt + a.qpoff[it.x] + (col0 >> 3) * 32 + lane : nullptr;
  const uint2* om = MODE ? nullptr : a.om + lane;
  f32x2 acc[NT][2];  // rows ra, rb; columns 8 nt + 2t, + 1
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = pack2(0.f, 0.f);
  f32x2 nrma = pack2(0.f, 0.f), nrmb = nrma;
  const bool want_norm = MODE == 0 && a.round == 0;
  const int nks = (nc + 15) >> 4;
  for (int kg = 0; kg < nks; ++kg) {
    const int c0 = (kg * 16) / kCC * kCC;
    if (kg * 16 == c0) {  // first k-step of a coordinate chunk
      __syncthreads();
      for (int e = threadIdx.x; e < D * kCC; e += blockDim.x) {
        const int k = e / kCC, jj = e % kCC;
        colc[k][jj] = c0 + jj < nc ? -(a.pts[(size_t)k * a.npts + cbase + c0 + jj] * a.scale) : 0.f;
      }
      __syncthreads();
    }
    // B fragments of the k-step (16 columns of the block), one word per lane
    // and column tile: issued before the entries are generated, used after
    uint32_t bh[NT][2], bl[NT][2];
#pragma unroll
    for (int n2 = 0; n2 < NT; n2 += 2)
      if (MODE == 0 || n2 < ntiles) {
#pragma unroll
        for (int nt = n2; nt < n2 + 2; ++nt) {
          if (MODE == 1) {
            const uint4 v = __ldg(qt + nt * 32);
            bh[nt][0] = v.x;
            bh[nt][1] = v.y;
            bl[nt][0] = v.z;
            bl[nt][1] = v.w;
          } else {
            const uint2 v = __ldg(om + nt * 32);
            bh[nt][0] = v.x;
            bh[nt][1] = v.y;
          }
        }
      }
    if (MODE == 1)
      qt += tnt * 32;
    else
      om += NT * 32;
    const int cb = kg * 16 - c0 + 2 * t;  // chunk columns cb, cb+1, cb+8, cb+9
    f32x2 e[4];                           // row ra: pairs cb, cb+8; row rb: pairs cb, cb+8
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      f32x2 ra2, rb2;
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const f32x2 cc = *reinterpret_cast<const f32x2*>(&colc[k][cb + 8 * h]);
        const f32x2 da = add2(rca[k], cc), db = add2(rcb[k], cc);
        ra2 = k ? fma2(da, da, ra2) : mul2(da, da);
        rb2 = k ? fma2(db, db, rb2) : mul2(db, db);
      }
      e[h] = ra2;
      e[2 + h] = rb2;
    }
    if (deriv) {
#pragma unroll
      for (int q = 0; q < 4; ++q) e[q] = kval2<KIND, true>(e[q], dscale);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) e[q] = kval2<KIND, false>(e[q], dscale);
    }
    if (kg * 16 + 16 > nc) {  // the last k-step of a ragged block: columns past it are zeros
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = kg * 16 + 2 * t + 8 * (q & 1);
        float x, y;
        unpack2(e[q], x, y);
        e[q] = pack2(c < nc ? x : 0.f, c + 1 < nc ? y : 0.f);
      }
    }
    if (want_norm) {
      nrma = fma2(e[1], e[1], fma2(e[0], e[0], nrma));
      nrmb = fma2(e[3], e[3], fma2(e[2], e[2], nrmb));
    }
    uint32_t ah[4], al[4];
    split2(e[0], ah[0], al[0]);  // row g, cols cb, cb+1
    split2(e[2], ah[1], al[1]);  // row g+8
    split2(e[1], ah[2], al[2]);  // row g, cols cb+8, cb+9
    split2(e[3], ah[3], al[3]);  // row g+8
#pragma unroll
    for (int n2 = 0; n2 < NT; n2 += 2)
      if (MODE == 0 || n2 < ntiles) {
        float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (MODE == 1) mma_bf16(d[j], ah[0], ah[1], ah[2], ah[3], bl[n2 + j][0], bl[n2 + j][1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_bf16(d[j], al[0], al[1], al[2], al[3], bh[n2 + j][0], bh[n2 + j][1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_bf16(d[j], ah[0], ah[1], ah[2], ah[3], bh[n2 + j][0], bh[n2 + j][1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[n2 + j][0] = add2(acc[n2 + j][0], pack2(d[j][0], d[j][1]));
          acc[n2 + j][1] = add2(acc[n2 + j][1], pack2(d[j][2], d[j][3]));
        }
      }
  }
  // rows mr .. ld - 1 (padding) get their zeros
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    if (nt < ntiles) {
      const int c = nt * 8 + 2 * t;
      float x, y;
      unpack2(acc[nt][0], x, y);
      if (ra < ld) {
        if (c < s) out[(size_t)c * ld + ra] = ra_ok ? x : 0.f;
        if (c + 1 < s) out[(size_t)(c + 1) * ld + ra] = ra_ok ? y : 0.f;
      }
      unpack2(acc[nt][1], x, y);
      if (rb < ld) {
        if (c < s) out[(size_t)c * ld + rb] = rb_ok ? x : 0.f;
        if (c + 1 < s) out[(size_t)(c + 1) * ld + rb] = rb_ok ? y : 0.f;
      }
    }
  }
  if (want_norm) {
    float na, na1, nb, nb1;
    unpack2(nrma, na, na1);
    unpack2(nrmb, nb, nb1);
    double dn = (ra_ok ? (double)na + na1 : 0.0) + (rb_ok ? (double)nb + nb1 : 0.0);
    for (int o = 16; o > 0; o >>= 1) dn += __shfl_xor_sync(0xffffffffu, dn, o);
    if (lane == 0) red[warp] = dn;
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&a.st[it.x].normA2, red[0] + red[1] + red[2] + red[3]);
  }
}

// Gaussian table of one sampling round in fragment order (see KmmFastArgs):
// W[j][c] is the BF16-rounded N(0,1) value for (round, j, c), zero for c >= bs.
__global__ void k_omega_pack(uint2* om, int ksteps, int bs, int nt_tot, uint32_t seed, int round) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)ksteps * nt_tot * 32;
       e += (long long)gridDim.x * blockDim.x) {
    const int lane = (int)(e & 31), g = lane >> 2, t = lane & 3;
    const long long w = e >> 5;
    const int nt = (int)(w % nt_tot), ks = (int)(w / nt_tot);
    const int c = nt * 8 + g, j = ks * 16 + 2 * t;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    if (c < bs) {
      const uint32_t st = 0x51ed270bu + round;
      x[0] = gauss_at(seed, st, (uint32_t)j, (uint32_t)c);
      x[1] = gauss_at(seed, st, (uint32_t)(j + 1), (uint32_t)c);
      x[2] = gauss_at(seed, st, (uint32_t)(j + 8), (uint32_t)c);
      x[3] = gauss_at(seed, st, (uint32_t)(j + 9), (uint32_t)c);
    }
    om[e] = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
  }
}

// Q (m x k, column-major, ld m) of each problem in fragment order, hi and lo
// (see KmmFastArgs): k-steps over the rows padded to whole coordinate chunks,
// column tiles over k padded to 16.
__global__ void k_pack_q(const Prob* probs, const ProbState* st, const long long* qpoff, uint4* qt) {
  const Prob P = probs[blockIdx.x];
  const int k = st[blockIdx.x].k;
  if (k <= 0) return;
  const int ntq = q_tiles(k);
  const int ksteps = (P.m + kCC - 1) / kCC * (kCC / 16);
  const float* Q = reinterpret_cast<const float*>(P.q);
  uint4* q = qt + qpoff[blockIdx.x];
  for (int e = threadIdx.x; e < ksteps * ntq * 32; e += blockDim.x) {
    const int lane = e & 31, g = lane >> 2, t = lane & 3;
    const int w = e >> 5;
    const int nt = w % ntq, ks = w / ntq;
    const int c = nt * 8 + g, i = ks * 16 + 2 * t;
    float x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = i + (r & 1) + 8 * (r >> 1);
      x[r] = (c < k && row < P.m) ? Q[(size_t)c * ara_ld(P.m) + row] : 0.f;
    }
    uint4 o;
    split_bf16x2(x[0], x[1], o.x, o.z);
    split_bf16x2(x[2], x[3], o.y, o.w);
    q[e] = o;
  }
}

// nt: right-hand column tiles the launch must cover (sample block / 8, or
// the largest basis of the batch / 8)
template <int D, int KIND>
void launch_kmm_fast3(int mode, int nt, unsigned grid, cudaStream_t s, const KmmFastArgs& a) {
  if (mode == 0) {
    if (nt <= 2)
      k_kmm_fast<D, KIND, 0, 2><<<grid, 128, 0, s>>>(a);
    else if (nt <= 4)
      k_kmm_fast<D, KIND, 0, 4><<<grid, 128, 0, s>>>(a);
    else
      k_kmm_fast<D, KIND, 0, 8><<<grid, 128, 0, s>>>(a);
  } else {
    if (nt <= 4)
      k_kmm_fast<D, KIND, 1, 4><<<grid, 128, 0, s>>>(a);
    else if (nt <= 8)
      k_kmm_fast<D, KIND, 1, 8><<<grid, 128, 0, s>>>(a);
    else
      k_kmm_fast<D, KIND, 1, kColGroup / 8><<<grid, 128, 0, s>>>(a);
  }
}
template <int D>
void launch_kmm_fast2(int kind, int mode, int nt, unsigned grid, cudaStream_t s, const KmmFastArgs& a) {
  if (kind == HM_KERNEL_GAUSS)
    launch_kmm_fast3<D, 2>(mode, nt, grid, s, a);
  else if (kind == HM_KERNEL_MATERN32)
    launch_kmm_fast3<D, 1>(mode, nt, grid, s, a);
  else
    launch_kmm_fast3<D, 0>(mode, nt, grid, s, a);
}
void launch_kmm_fast(int d, int kind, int mode, int nt, unsigned grid, cudaStream_t s, const KmmFastArgs& a) {
  if (d == 1)
    launch_kmm_fast2<1>(kind, mode, nt, grid, s, a);
  else if (d == 2)
    launch_kmm_fast2<2>(kind, mode, nt, grid, s, a);
  else
    launch_kmm_fast2<3>(kind, mode, nt, grid, s, a);
}

// ---------------------------------------------------------------------------
// dense blocks
// ---------------------------------------------------------------------------
struct QMove {  // a basis that moves to wider storage
  const void* from;
  long long to, count;  // elements
};

template <typename W>
__global__ void k_move_q(const QMove* __restrict__ moves, W* __restrict__ base) {
  const QMove m = moves[blockIdx.x];
  const W* from = reinterpret_cast<const W*>(m.from);
  for (long long e = blockIdx.y * blockDim.x + threadIdx.x; e < m.count; e += (long long)gridDim.y * blockDim.x)
    base[m.to + e] = from[e];
}

struct DenseItem {
  int r0, m, c0, n;
  long long off;
};

__global__ void k_dense_gen(const DenseItem* items, const float* pts, int npts, int d,
                            KernelParams kp, float* dst) {
  const DenseItem it = items[blockIdx.x];
  size_t tot = (size_t)it.m * it.n;
  for (size_t e = threadIdx.x; e < tot; e += blockDim.x) {
    int i = (int)(e % it.m), j = (int)(e / it.m);
    int gi = it.r0 + i, gj = it.c0 + j;
    float r2 = 0.f;
    for (int k = 0; k < d; ++k) {
      float df = pts[(size_t)k * npts + gi] - pts[(size_t)k * npts + gj];
      r2 = fmaf(df, df, r2);
    }
    float v = kernel_r2(kp, r2);
    if (gi == gj && !kp.deriv) v += kp.nugget;
    dst[it.off + e] = v;
  }
}

size_t kmm_smem() {
  using W = float;
  return sizeof(W) * (kTC * kColGroup) + sizeof(float) * (kTC * kTR + kMaxDim * kTC) +
         sizeof(double) * (kKmmThreads / 32);
}

}  // namespace

// leaf_lo, leaf_hi: the block-row shard, leaves [leaf_lo, leaf_hi) (all
// leaves for a whole matrix).  A shard compresses only the pairs whose row or
// column cluster overlaps its rows, and only its own diagonal leaves.
hm_status hmatrix_build(hm_kdtree t, hm_structure s, const double* d_points, const hm_build_opts* o,
                        cudaStream_t stream, hm_hmatrix* out, int leaf_lo, int leaf_hi) {
  if (!out) return fail(HM_ERR_INVALID, "hm_hmatrix_build: out is NULL");
  *out = nullptr;
  if (!t || !s || !o) return fail(HM_ERR_INVALID, "hm_hmatrix_build: null argument");
  if (s->tree != t) return fail(HM_ERR_INVALID, "hm_hmatrix_build: structure was built on another tree");
  if (leaf_hi < 0) leaf_hi = 1 << t->depth;
  if (leaf_lo < 0 || leaf_lo >= leaf_hi || leaf_hi > (1 << t->depth))
    return fail(HM_ERR_INVALID, "hm_hmatrix_build_rows: need 0 <= leaf_begin < leaf_end <= 2^depth");
  (void)d_points;  // the tree keeps its own tree-ordered copy of the points
  hm_build_opts opt = *o;
  if (opt.kernel < 0 || opt.kernel > 2) return fail(HM_ERR_INVALID, "hm_hmatrix_build: unknown kernel");
  if (!(opt.ell > 0) || !(opt.tol > 0) || opt.tol >= 1)
    return fail(HM_ERR_INVALID, "hm_hmatrix_build: need ell > 0 and 0 < tol < 1");
  if (opt.sample_block <= 0) opt.sample_block = 16;
  if (opt.sample_block > kMaxBs) return fail(HM_ERR_UNSUPPORTED, "hm_hmatrix_build: sample_block > 32");
  if (opt.leaf_max_rank <= 0) opt.leaf_max_rank = std::max(1, t->bucket / 2);
  if (opt.max_rank <= 0) opt.max_rank = 64;
  const int bs = opt.sample_block;
  if (opt.max_rank > kMaxCols || opt.leaf_max_rank > kMaxCols)
    return fail(HM_ERR_UNSUPPORTED, "hm_hmatrix_build: rank caps must be <= 256");
  if (opt.level_schedule != 0 && opt.level_schedule != 1)
    return fail(HM_ERR_INVALID, "hm_hmatrix_build: level_schedule must be 0 or 1");

  cudaEvent_t ev0, ev1;
  HM_CUDA(cudaEventCreate(&ev0));
  HM_CUDA(cudaEventCreate(&ev1));
  HM_CUDA(cudaEventRecord(ev0, stream));

  auto* h = new hm_hmatrix_s();
  auto cleanup = [&](hm_status st) {
    delete h;
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    return st;
  };
  h->tree = t;
  h->structure = s;
  h->n = t->n;
  h->d = t->d;
  h->depth = t->depth;
  h->opts = opt;
  h->leaf_lo = leaf_lo;
  h->leaf_hi = leaf_hi;
  h->kp.kind = opt.kernel;
  h->kp.deriv = opt.derivative ? 1 : 0;
  h->kp.ell = (float)opt.ell;
  h->kp.inv_ell = (float)(1.0 / opt.ell);
  h->kp.nugget = (float)opt.nugget;
  const int depth = t->depth;
  const std::vector<int>& lo = t->h_offsets;
  auto coff = [&](int level, int c) { return lo[(size_t)c << (depth - level)]; };
  // Rank cap and tolerance of a level-l block.  Uniform: the leaf cap at the
  // leaf level, max_rank above it, tol everywhere.  The reference's schedule
  // (level_schedule = 1): the tolerance doubles at each level above the
  // leaves (src/constructHMatrixFromStruct.cu:31,54: tol 2^(depth - l) at
  // level l) and the cap is bucket 2^i, divided by 4 beyond i = 5, with
  // i = depth - 1 - l (generateMaxRanks, src/helperFunctions.cu:67-74),
  // within this build's largest basis.
  auto level_cap = [&](int l) {
    if (l == depth) return opt.leaf_max_rank;
    if (opt.level_schedule != 1) return opt.max_rank;
    const int i = depth - 1 - l;
    long long c = (long long)t->bucket << std::min(i, 20);
    if (i > 5) c /= 4;
    return (int)std::min<long long>(c, kMaxCols);
  };
  auto level_tscale2 = [&](int l) {
    if (opt.level_schedule != 1 || l >= depth) return 1.0;
    const double f = std::ldexp(1.0, depth - l);
    return f * f;
  };
  // rows of the shard; a pair is needed when its rows or its columns overlap them
  const int row_lo = lo[leaf_lo], row_hi = lo[leaf_hi];
  auto needed = [&](int r0, int m, int c0, int n) {
    return (r0 < row_hi && r0 + m > row_lo) || (c0 < row_hi && c0 + n > row_lo);
  };

  PhaseTrace tr("build");
  // ---- the problems: stored pairs (row cluster v > column cluster u) ------
  std::vector<uint32_t> tiles(std::max<long long>(s->start[depth], 1));
  if (s->start[depth] > 0)
    HM_CUDA(cudaMemcpy(tiles.data(), s->tiles.p, 4 * (size_t)s->start[depth], cudaMemcpyDeviceToHost));
  std::vector<Prob> probs;
  for (int l = 1; l <= depth; ++l) {
    for (long long i = s->start[l - 1]; i < s->start[l]; ++i) {
      uint32_t z = tiles[i];
      int u = (int)compact16(z), v = (int)compact16(z >> 1);
      if (v <= u) continue;
      Prob P{};
      P.level = l;
      P.u = u;
      P.v = v;
      P.r0 = coff(l, v);
      P.m = coff(l, v + 1) - P.r0;
      P.c0 = coff(l, u);
      P.n = coff(l, u + 1) - P.c0;
      P.kmax = std::min(level_cap(l), std::min(P.m, P.n));
      P.tscale2 = level_tscale2(l);
      if (!needed(P.r0, P.m, P.c0, P.n)) continue;
      probs.push_back(P);
    }
  }
  const long long nprob0 = (long long)probs.size();

  tr.mark("problems", stream, -1, 0);
  // ---- batches bounded by the workspace budget -----------------------------
  const size_t freeb = dev_available();
  // per-problem results that survive the batch: rank (-1: stored dense, -2:
  // split into its child blocks), low-part columns, and the factor location.
  // A problem that misses the tolerance at its rank cap above the leaf level
  // appends its four child pairs to `probs`, so these grow with it.
  std::vector<int> rank(nprob0, 0), conv(nprob0, 0), rhis(nprob0, 0);
  std::vector<double> nrm(nprob0, 0.0);
  long long pstart = 0;
  const double thresh2 = 0.09 * opt.tol * opt.tol;  // (0.3 tol)^2
  long long lr_count = 0, dense_count = 0, rank_sum = 0, split_count = 0;
  int max_rank_seen = 0;
  long long factor_bytes = 0, dense_bytes = 0, unconverged = 0;

  std::vector<const float*> fu(nprob0, nullptr), fv(nprob0, nullptr);
  std::vector<const float*> fd(nprob0, nullptr), fdt(nprob0, nullptr);
  auto grow = [&](size_t np) {
    rank.resize(np, 0);
    conv.resize(np, 0);
    rhis.resize(np, 0);
    nrm.resize(np, 0.0);
    fu.resize(np, nullptr);
    fv.resize(np, nullptr);
    fd.resize(np, nullptr);
    fdt.resize(np, nullptr);
  };

  // Sketches, bases and projections run in FP64 when the tolerance is below
  // what FP32 sums over a block can resolve (~u*sqrt(m) relative), else FP32.
  const bool fp64 = opt.tol < 5e-6;
  auto batch_loop = [&](auto tag) -> hm_status {
    using W = decltype(tag);
    if (std::is_same<W, float>::value)
      HM_CUDA(cudaFuncSetAttribute(k_kmm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kmm_smem()));
    // The specialised sketch kernels draw a double-width first sample (the
    // generation of the kernel block, not its product with the sample, is
    // the cost of a pass, so blocks of rank bs..2 bs finish a pass earlier).
    // The residual is estimated from the sample itself, as in the reference's
    // ARA (separate test columns measured slower on the 2^20-point Matern
    // build: wider first passes, wider bases).
    constexpr bool kTensorW = std::is_same<W, float>::value;
    const bool fastW = kTensorW && t->d <= 3;
    const int bs_first = fastW ? std::min(2 * bs, kMaxBs) : bs;  // round 0 columns
    const int wmax = std::max(bs_first, bs);                      // widest sample
    // Greedy batches.  A problem starts with room for kQCols basis columns and
    // its sample; the few that need more move to wider storage when they do
    // (below), and B is allocated at its exact width after the rounds.  The
    // budget, an eighth of all problems' need between kBatchMin and kBatchMax,
    // gives every launch enough blocks and keeps what is mapped and unmapped
    // per build small (mapping a GB takes 0.2 to 100 ms on a shared host).
    // Problems listed together share one first-round width, whatever the batch.
    constexpr size_t kBatchMin = size_t(1) << 30, kBatchMax = size_t(12) << 30;
    auto need_of = [&](const Prob& P) {
      return ((size_t)ara_ld(P.m) * (std::min(P.kmax, kQCols) + wmax) + (size_t)ara_ld(P.n) * kMaxBs) * sizeof(W);
    };
    // The most a problem can come to if its basis reaches the cap: every width
    // its basis had (superseded ones stay until the end of the batch), B, the
    // packed basis, the Gram partials and its factors or dense blocks.  A batch
    // whose blocks all did would need up to 12 times the budget, so the sum over
    // a batch stays within three quarters of the memory there is.
    auto most_of = [&](const Prob& P) {
      const size_t m = ara_ld(P.m), n = ara_ld(P.n), k = P.kmax;
      size_t q = std::min(P.kmax, kQCols), w = q + wmax;
      while (q < k) w += q = std::min(2 * q, k);
      size_t bytes = (m * w + n * k) * sizeof(W);
      if (fastW) bytes += (size_t)(P.m + kCC - 1) / kCC * (kCC / 16) * q_tiles(P.kmax) * 32 * sizeof(uint4);
      const size_t kt = std::min<size_t>(k, kTruncMax);
      bytes += kt * kt * ((n + 2047) / 2048 * sizeof(double) + sizeof(float));
      const size_t factors = (size_t)(P.m + P.n) * k, blocks = P.level == depth ? 2 * (size_t)P.m * P.n : 0;
      return bytes + std::max(factors, blocks) * sizeof(float);
    };
    DevBuf<W> ws, wb;  // Q and Y; B (kept from batch to batch)
    size_t room = freeb / 4 * 3;  // memory for the next batch
    size_t budget = 0;
    int gen_bs0 = 0;  // first-round columns of the problems listed last
    long long gen_end = 0;
    auto next_batch = [&](long long ps) {
      if (ps >= gen_end) {
        gen_end = (long long)probs.size();
        size_t all = 0;
        gen_bs0 = bs_first;  // as wide as every block's rank cap allows
        for (long long i = ps; i < gen_end; ++i) {
          probs[i].gid = (int)(i - ps);
          all += need_of(probs[i]);
          if (probs[i].kmax < gen_bs0) gen_bs0 = std::max(bs, probs[i].kmax / 8 * 8);
        }
        budget = std::min(std::max(all / 8, kBatchMin), std::min<size_t>(freeb / 8, kBatchMax));
      }
      long long pe = ps;
      size_t sz = 0, most = 0;
      bool asked = ps == 0;  // (70 us: only a batch of some size asks again)
      while (pe < gen_end) {
        const size_t need = need_of(probs[pe]);
        most += most_of(probs[pe]);
        if (!asked && most > freeb / 16) {
          asked = true;
          room = (dev_available() + (ws.n + wb.n) * sizeof(W)) / 4 * 3;
        }
        if (pe > ps && (sz + need > budget || most > room)) break;
        sz += need;
        ++pe;
      }
      return pe;
    };
    while (pstart < (long long)probs.size()) {
      const long long pend = next_batch(pstart);
      const int nb = (int)(pend - pstart);
      tr.mark("batch begin", stream, nb, 0);
      std::vector<Prob> bp(probs.begin() + pstart, probs.begin() + pend);
      size_t off = 0;
      std::vector<int2> items_rows, items_cols;
      for (int i = 0; i < nb; ++i) {
        Prob& P = bp[i];
        P.qcap = std::min(P.kmax, kQCols);
        off += (size_t)ara_ld(P.m) * (P.qcap + wmax);
        for (int tt = 0; tt * kTR < P.m; ++tt) items_rows.push_back(make_int2(i, tt));
        for (int tt = 0; tt * kTR < P.n; ++tt) items_cols.push_back(make_int2(i, tt));
      }
      if (off > ws.n) {
        hm_status st0 = ws.alloc_async(off, stream);
        if (st0) return st0;
      }
      off = 0;
      for (int i = 0; i < nb; ++i) {
        Prob& P = bp[i];
        P.q = ws.p + off;
        off += (size_t)ara_ld(P.m) * P.qcap;
        P.y = ws.p + off;
        off += (size_t)ara_ld(P.m) * wmax;
      }
      DevBuf<Prob> dprobs;
      DevBuf<ProbState> dst;
      DevBuf<int2> drows, dcols;
      hm_status st;
      if ((st = dprobs.alloc_async(nb, stream)) || (st = dst.alloc_async(nb, stream)) ||
          (st = drows.alloc_async(items_rows.size(), stream)) || (st = dcols.alloc_async(items_cols.size(), stream)))
        return st;
      std::vector<ProbState> hst(nb);
      for (auto& x : hst) {
        x = ProbState{};
        x.active = 1;
      }
      HM_CUDA(cudaMemcpyAsync(dprobs.p, bp.data(), sizeof(Prob) * nb, cudaMemcpyHostToDevice, stream));
      HM_CUDA(cudaMemcpyAsync(dst.p, hst.data(), sizeof(ProbState) * nb, cudaMemcpyHostToDevice, stream));
      HM_CUDA(cudaMemcpyAsync(drows.p, items_rows.data(), sizeof(int2) * items_rows.size(),
                              cudaMemcpyHostToDevice, stream));
      HM_CUDA(cudaMemcpyAsync(dcols.p, items_cols.data(), sizeof(int2) * items_cols.size(),
                              cudaMemcpyHostToDevice, stream));

      KmmArgs<W> ka;
      ka.probs = dprobs.p;
      ka.st = dst.p;
      ka.pts = t->pts_tree_f.p;
      ka.npts = t->n;
      ka.d = t->d;
      ka.kp = h->kp;
      ka.bs = bs;
      ka.seed = (uint32_t)(opt.seed ^ (opt.seed >> 32)) ^ 0x5bd1e995u;
      OrthPlan orth;
      if ((st = orth_plan<W>(bp, &orth, stream))) return st;
      // FP32 working precision and d <= 3: specialised tensor-core sketch
      // kernels; d > 3: the SIMT kernel; FP64: the FP64 tensor instruction
      constexpr bool kTensor = std::is_same<W, float>::value;
      const bool fast = kTensor && t->d <= 3;
      KmmFastArgs kf{};
      DevBuf<uint2> om2;
      const int bs0 = gen_bs0;
      const int om_nt = sample_tiles(std::max(bs0, bs));
      int om_rows2 = 0;
      if (fast) {
        int max_n = 1;
        for (const Prob& P : bp) max_n = std::max(max_n, P.n);
        om_rows2 = (max_n + kCC - 1) / kCC * (kCC / 2);  // column pairs; k-steps = om_rows2 / 8
        if ((st = om2.alloc_async((size_t)(om_rows2 / 8) * om_nt * 32, stream))) return st;
        const double il = 1.0 / opt.ell, log2e = 1.4426950408889634, ln2 = 0.6931471805599453;
        double sc = log2e * il, dsc = ln2 * il;
        if (opt.kernel == HM_KERNEL_MATERN32) {
          sc = std::sqrt(3.0) * log2e * il;
          dsc = il;
        } else if (opt.kernel == HM_KERNEL_GAUSS) {
          sc = std::sqrt(0.5 * log2e) * il;
          dsc = 2.0 * ln2 * il;
        }
        kf.probs = dprobs.p;
        kf.st = dst.p;
        kf.pts = t->pts_tree_f.p;
        kf.npts = t->n;
        kf.scale = (float)sc;
        kf.dscale = (float)dsc;
        kf.deriv = opt.derivative != 0;
        kf.bs = bs;
        kf.om = om2.p;
      }
      tr.mark("batch setup", stream, nb, 0);
      const int max_rounds = kMaxCols / bs + 2;
      std::vector<DevBuf<W>> grown;  // wider bases, until the end of the batch
      for (int round = 0; round < max_rounds; ++round) {
        // sample columns: double width in the first round and again from the
        // fourth on (the blocks still active by then are the high-rank ones;
        // entry generation, not the sample width, is the cost of a round, so
        // wider rounds mean fewer of them; earlier, a wider basis would cost
        // more in the projection than it saves)
        const int rbs = fast && round != 1 && round != 2 ? bs0 : bs;
        // active bases without room for this round's columns move to storage
        // of twice the width (at most their cap)
        {
          std::vector<QMove> moves;
          size_t more = 0;
          for (int i = 0; i < nb; ++i) {
            Prob& P = bp[i];
            const int k = hst[i].k;
            if (!hst[i].active || k + rbs <= P.qcap || P.qcap >= P.kmax) continue;
            P.qcap = std::min(P.kmax, std::max(2 * P.qcap, k + rbs));
            moves.push_back(QMove{P.q, (long long)more, (long long)ara_ld(P.m) * k});
            more += (size_t)ara_ld(P.m) * P.qcap;
          }
          if (!moves.empty()) {
            grown.emplace_back();
            if ((st = grown.back().alloc_async(more, stream))) return st;
            W* base = grown.back().p;
            size_t j = 0;
            for (int i = 0; i < nb && j < moves.size(); ++i)
              if (bp[i].q == moves[j].from) bp[i].q = base + moves[j++].to;
            DevBuf<QMove> dm;
            if ((st = dm.alloc_async(moves.size(), stream))) return st;
            HM_CUDA(cudaMemcpyAsync(dm.p, moves.data(), sizeof(QMove) * moves.size(), cudaMemcpyHostToDevice, stream));
            k_move_q<W><<<dim3((unsigned)moves.size(), 8), 256, 0, stream>>>(dm.p, base);
            HM_LAUNCH_CHECK();
            HM_CUDA(cudaMemcpyAsync(dprobs.p, bp.data(), sizeof(Prob) * nb, cudaMemcpyHostToDevice, stream));
          }
        }
        if (fast) {
          k_omega_pack<<<592, 256, 0, stream>>>(om2.p, om_rows2 / 8, rbs, sample_tiles(rbs), ka.seed, round);
          HM_LAUNCH_CHECK();
          kf.round = round;
          kf.bs = rbs;
          kf.items = drows.p;
          launch_kmm_fast(t->d, opt.kernel, 0, sample_tiles(rbs), (unsigned)items_rows.size(), stream, kf);
        } else {
          ka.mode = 0;
          ka.col0 = 0;
          ka.round = round;
          ka.items = drows.p;
          if constexpr (kTensor)
            k_kmm<<<(unsigned)items_rows.size(), kKmmThreads, kmm_smem(), stream>>>(ka);
          else
            launch_kmm64(rbs, (unsigned)items_rows.size(), stream, ka);
        }
        HM_LAUNCH_CHECK();
        tr.mark("  round sketch", stream, round, 1);
        if ((st = orth_round<W>(orth, dprobs.p, dst.p, rbs, thresh2, stream))) return st;
        tr.mark("  round orth", stream, round, 2);
        HM_CUDA(cudaMemcpyAsync(hst.data(), dst.p, sizeof(ProbState) * nb, cudaMemcpyDeviceToHost, stream));
        HM_CUDA(cudaStreamSynchronize(stream));
        bool any = false;
        for (auto& x : hst) any |= x.active != 0;
        if (!any) break;
      }
      tr.mark("sample rounds", stream, nb, 2);
      // B = A^T Q
      {
        size_t bsz = 0;
        for (int i = 0; i < nb; ++i) bsz += (size_t)ara_ld(bp[i].n) * hst[i].k;
        if (bsz > wb.n && (st = wb.alloc_async(bsz, stream))) return st;
        bsz = 0;
        for (int i = 0; i < nb; ++i) {
          bp[i].b = wb.p + bsz;
          bsz += (size_t)ara_ld(bp[i].n) * hst[i].k;
        }
        HM_CUDA(cudaMemcpyAsync(dprobs.p, bp.data(), sizeof(Prob) * nb, cudaMemcpyHostToDevice, stream));
      }
      DevBuf<uint4> qt;
      DevBuf<long long> dqpoff;
      DevBuf<int2> dcls;
      if (fast) {
        std::vector<long long> qpoff(nb);
        size_t qw = 0;
        for (int i = 0; i < nb; ++i) {
          qpoff[i] = (long long)qw;
          if (hst[i].k > 0)
            qw += (size_t)(bp[i].m + kCC - 1) / kCC * (kCC / 16) * (size_t)q_tiles(hst[i].k) * 32;
        }
        if ((st = qt.alloc_async(std::max<size_t>(qw, 1), stream)) || (st = dqpoff.alloc_async(nb, stream)))
          return st;
        tr.mark("  q table alloc (MB)", stream, (long long)(qw * 16 >> 20), 3);
        HM_CUDA(cudaMemcpyAsync(dqpoff.p, qpoff.data(), sizeof(long long) * nb, cudaMemcpyHostToDevice, stream));
        k_pack_q<<<nb, 256, 0, stream>>>(dprobs.p, dst.p, dqpoff.p, qt.p);
        HM_LAUNCH_CHECK();
        tr.mark("  q pack", stream, nb, 3);
        kf.qt = qt.p;
        kf.qpoff = dqpoff.p;
        // one launch per basis-width class, so the narrow (most) blocks run
        // with few accumulator registers
        // (bases wider than 128 columns take a second launch for columns
        // 128.. of the same items)
        std::vector<int2> cls[4];
        for (const int2& ic : items_cols) {
          const int kk = hst[ic.x].k;
          if (kk <= 0) continue;
          cls[kk <= 32 ? 0 : (kk <= 64 ? 1 : (kk <= kColGroup ? 2 : 3))].push_back(ic);
        }
        const int cls_nt[4] = {4, 8, kColGroup / 8, kColGroup / 8};
        size_t ncls = 0;
        for (auto& c : cls) ncls += c.size();
        if ((st = dcls.alloc_async(std::max<size_t>(ncls, 1), stream))) return st;
        size_t o = 0;
        for (int c = 0; c < 4; ++c) {
          if (cls[c].empty()) continue;
          HM_CUDA(cudaMemcpyAsync(dcls.p + o, cls[c].data(), sizeof(int2) * cls[c].size(), cudaMemcpyHostToDevice,
                                  stream));
          kf.items = dcls.p + o;
          for (int c0 = 0; c0 < (c == 3 ? kMaxCols : kColGroup); c0 += kColGroup) {
            kf.col0 = c0;
            launch_kmm_fast(t->d, opt.kernel, 1, cls_nt[c], (unsigned)cls[c].size(), stream, kf);
            HM_LAUNCH_CHECK();
          }
          o += cls[c].size();
        }
        kf.col0 = 0;
      } else {
        ka.mode = 1;
        ka.items = dcols.p;
        int kmx = 0;
        for (int i = 0; i < nb; ++i) kmx = std::max(kmx, hst[i].k);
        constexpr int kGroup = kTensor ? kColGroup : kGroup64;
        for (int c0 = 0; c0 < kmx; c0 += kGroup) {
          ka.col0 = c0;
          if constexpr (kTensor)
            k_kmm<<<(unsigned)items_cols.size(), kKmmThreads, kmm_smem(), stream>>>(ka);
          else
            launch_kmm64(std::min(kGroup, kmx - c0), (unsigned)items_cols.size(), stream, ka);
          HM_LAUNCH_CHECK();
        }
        ka.col0 = 0;
      }
      HM_LAUNCH_CHECK();

      tr.mark("projection", stream, nb, 3);
      // ---- truncation: Gram of B, its eigenpairs, truncated rank ------------
      HM_CUDA(cudaMemcpyAsync(hst.data(), dst.p, sizeof(ProbState) * nb, cudaMemcpyDeviceToHost, stream));
      HM_CUDA(cudaStreamSynchronize(stream));
      // error budget (relative, squared): sampling residual <= 0.09 tol^2 (the
      // stopping test), truncation 0.45 tol^2 (FP32 form) or 0.35 tol^2 plus
      // 0.15 tol^2 of BF16 rounding (mixed form)
      const bool mixed = opt.precision == HM_PREC_MIXED;
      TruncWork tw;
      if ((st = trunc_rank<W>(bp, hst, dprobs.p, dst.p, (mixed ? 0.35 : 0.45) * opt.tol * opt.tol,
                              mixed ? 0.15 * opt.tol * opt.tol : 0.0, &tw, stream)))
        return st;
      HM_CUDA(cudaMemcpyAsync(hst.data(), dst.p, sizeof(ProbState) * nb, cudaMemcpyDeviceToHost, stream));
      HM_CUDA(cudaStreamSynchronize(stream));

      tr.mark("truncation", stream, nb, 4);
      // ---- results: low rank where converged; otherwise the four child
      // blocks (above the leaf level) or dense (leaf blocks) -----------------
      std::vector<long long> du(nb, -1), dv(nb, -1);
      std::vector<DenseItem> dens;
      std::vector<Prob> children;
      size_t chunk_floats = 0;
      for (int i = 0; i < nb; ++i) {
        const Prob& P = bp[i];
        const ProbState& S = hst[i];
        long long gi = pstart + i;
        nrm[gi] = S.normA2;
        const bool capped = !(S.converged || S.active);
        if (capped && P.level < depth) {
          // the pair as the reference's recursion would have recorded it had
          // it been inadmissible (src/HMatrixStructure.cu:27-89): its four
          // child pairs (2v + b, 2u + a), compressed in a later batch; every
          // child keeps row cluster > column cluster
          rank[gi] = -2;
          ++split_count;
          const int cl = P.level + 1;
          for (int b2 = 0; b2 < 2; ++b2)
            for (int a2 = 0; a2 < 2; ++a2) {
              Prob C{};
              C.level = cl;
              C.u = 2 * P.u + a2;
              C.v = 2 * P.v + b2;
              C.r0 = coff(cl, C.v);
              C.m = coff(cl, C.v + 1) - C.r0;
              C.c0 = coff(cl, C.u);
              C.n = coff(cl, C.u + 1) - C.c0;
              if (C.m <= 0 || C.n <= 0 || !needed(C.r0, C.m, C.c0, C.n)) continue;
              C.kmax = std::min(level_cap(cl), std::min(C.m, C.n));
              C.tscale2 = level_tscale2(cl);
              children.push_back(C);
            }
          continue;
        }
        if (!capped) {
          du[i] = (long long)chunk_floats;
          chunk_floats += (size_t)P.m * S.r;
          dv[i] = (long long)chunk_floats;
          chunk_floats += (size_t)P.n * S.r;
          rank[gi] = S.r;
          rhis[gi] = std::min(S.rhi, S.r);
          conv[gi] = 1;
        } else {
          // the block and its mirror, each column-major, so every dense read in
          // the matvec is coalesced
          DenseItem di;
          di.r0 = P.r0;
          di.m = P.m;
          di.c0 = P.c0;
          di.n = P.n;
          di.off = (long long)chunk_floats;
          chunk_floats += (size_t)P.m * P.n;
          dens.push_back(di);
          DenseItem dt;
          dt.r0 = P.c0;
          dt.m = P.n;
          dt.c0 = P.r0;
          dt.n = P.m;
          dt.off = (long long)chunk_floats;
          chunk_floats += (size_t)P.m * P.n;
          dens.push_back(dt);
          rank[gi] = -1;
        }
      }
      DevBuf<float> chunk;
      if ((st = chunk.alloc(std::max<size_t>(chunk_floats, 1)))) return st;
      DevBuf<long long> ddu, ddv;
      DevBuf<DenseItem> ddi;
      if ((st = ddu.alloc_async(nb, stream)) || (st = ddv.alloc_async(nb, stream))) return st;
      HM_CUDA(cudaMemcpyAsync(ddu.p, du.data(), sizeof(long long) * nb, cudaMemcpyHostToDevice, stream));
      HM_CUDA(cudaMemcpyAsync(ddv.p, dv.data(), sizeof(long long) * nb, cudaMemcpyHostToDevice, stream));
      static_assert(kTR == 64, "trunc_pack's tiles are the sketch's row tiles");
      if ((st = trunc_pack<W>(dprobs.p, dst.p, tw, drows.p, items_rows.size(), dcols.p, items_cols.size(), ddu.p, ddv.p,
                              chunk.p, stream)))
        return st;
      if (!dens.empty()) {
        if ((st = ddi.alloc_async(dens.size(), stream))) return st;
        HM_CUDA(cudaMemcpyAsync(ddi.p, dens.data(), sizeof(DenseItem) * dens.size(), cudaMemcpyHostToDevice,
                                stream));
        k_dense_gen<<<(unsigned)dens.size(), 256, 0, stream>>>(ddi.p, t->pts_tree_f.p, t->n, t->d, h->kp,
                                                               chunk.p);
        HM_LAUNCH_CHECK();
      }
      HM_CUDA(cudaStreamSynchronize(stream));
      size_t pk = 0, dk = 0;
      for (int i = 0; i < nb; ++i) {
        long long gi = pstart + i;
        if (rank[gi] == -2) continue;  // split
        if (rank[gi] >= 0) {
          fu[gi] = chunk.p + du[i];
          fv[gi] = chunk.p + dv[i];
          ++pk;
          lr_count += 2;
          rank_sum += 2 * (long long)rank[gi];
          max_rank_seen = std::max(max_rank_seen, rank[gi]);
          factor_bytes += 4ll * (bp[i].m + bp[i].n) * rank[gi];
        } else {
          fd[gi] = chunk.p + dens[dk].off;
          fdt[gi] = chunk.p + dens[dk + 1].off;
          dk += 2;
          dense_count += 2;
          dense_bytes += 8ll * bp[i].m * bp[i].n;
        }
      }
      tr.mark("factors", stream, nb, 4);
      h->storage.push_back(std::move(chunk));
      pstart = pend;
      if (!children.empty()) {
        probs.insert(probs.end(), children.begin(), children.end());
        grow(probs.size());
        tr.mark("split into children", stream, (long long)children.size(), 0);
      }
    }
    return HM_OK;
  };
  {
    hm_status bst = fp64 ? batch_loop(double(0)) : batch_loop(float(0));
    if (bst) return cleanup(bst);
  }

  // ---- diagonal leaves ------------------------------------------------------
  h->diag_fly = opt.diag_from_coords > 0 || (opt.diag_from_coords < 0 && opt.derivative != 0);
  if (!h->diag_fly) {
    const int nown = leaf_hi - leaf_lo;  // the shard's leaves (all of them for a whole matrix)
    std::vector<DenseItem> dens(nown);
    size_t tot = 0;
    for (int q = 0; q < nown; ++q) {
      const int l = leaf_lo + q;
      dens[q].r0 = lo[l];
      dens[q].m = lo[l + 1] - lo[l];
      dens[q].c0 = lo[l];
      dens[q].n = dens[q].m;
      dens[q].off = (long long)tot;
      tot += (size_t)dens[q].m * dens[q].m;
    }
    DevBuf<float> chunk;
    DevBuf<DenseItem> ddi;
    hm_status st;
    if ((st = chunk.alloc(std::max<size_t>(tot, 1))) || (st = ddi.alloc_async(nown, stream))) return cleanup(st);
    HM_CUDA(cudaMemcpyAsync(ddi.p, dens.data(), sizeof(DenseItem) * nown, cudaMemcpyHostToDevice, stream));
    k_dense_gen<<<nown, 256, 0, stream>>>(ddi.p, t->pts_tree_f.p, t->n, t->d, h->kp, chunk.p);
    HM_LAUNCH_CHECK();
    HM_CUDA(cudaStreamSynchronize(stream));
    for (int l = 0; l < nown; ++l) {
      DenseBlock db;
      db.r0 = dens[l].r0;
      db.m = dens[l].m;
      db.c0 = dens[l].c0;
      db.n = dens[l].n;
      db.trans = 0;
      db.D = chunk.p + dens[l].off;
      if (db.m > 0) h->h_dense.push_back(db);
    }
    dense_count += nown;
    dense_bytes += 4ll * (long long)tot;
    h->storage.push_back(std::move(chunk));
  }

  tr.mark("diagonal leaves", stream, -1, 5);
  // ---- block lists (both orientations) --------------------------------------
  const long long nprob = (long long)probs.size();
  for (long long i = 0; i < nprob; ++i) {
    const Prob& P = probs[i];
    if (rank[i] == -2) continue;  // split: its children are in the list
    if (rank[i] >= 0) {
      LRBlock b{};
      b.level = P.level;
      b.k = rank[i];
      b.r0 = P.r0;
      b.m = P.m;
      b.c0 = P.c0;
      b.n = P.n;
      b.U = fu[i];
      b.V = fv[i];
      b.khi = std::min(rhis[i], rank[i]);
      h->h_lr.push_back(b);
      LRBlock bt = b;
      bt.r0 = P.c0;
      bt.m = P.n;
      bt.c0 = P.r0;
      bt.n = P.m;
      bt.U = fv[i];
      bt.V = fu[i];
      h->h_lr.push_back(bt);
    } else {
      DenseBlock db{P.r0, P.m, P.c0, P.n, 0, fd[i]};
      h->h_dense.push_back(db);
      DenseBlock dt{P.c0, P.n, P.r0, P.m, 0, fdt[i]};
      h->h_dense.push_back(dt);
    }
  }
  tr.mark("block lists", stream, -1, 6);
  // ---- factor panels: the mixed form's BF16 hi + lo tiles, or the FP32
  // form's FP32 tiles (both forms multiply on panels) ---------------------------
  {
    std::vector<MxPair> mp;
    for (long long i = 0; i < nprob; ++i) {
      if (rank[i] <= 0) continue;
      const Prob& P = probs[i];
      mp.push_back(
          MxPair{P.level, P.r0, P.m, P.c0, P.n, rank[i], std::min(rhis[i], rank[i]), fu[i], fv[i], P.v, P.u});
    }
    std::vector<MxDenseIn> md;
    for (const DenseBlock& db : h->h_dense) md.push_back(MxDenseIn{db.r0, db.m, db.c0, db.n, db.D});
    h->mx.fmt = opt.precision == HM_PREC_MIXED ? 0 : 1;
    hm_status mst = mixed_build(h, mp, md, stream);
    if (mst) return cleanup(mst);
    if (opt.precision == HM_PREC_MIXED) {
      h->stats.mixed_bytes = h->mx.store_tiles * 512;
      release_fp32(h);
    }
  }
  h->stats.num_lowrank = lr_count;
  h->stats.num_dense = dense_count;
  h->stats.rank_sum = rank_sum;
  h->stats.max_rank_seen = max_rank_seen;
  h->stats.factor_bytes = factor_bytes;
  h->stats.dense_bytes = dense_bytes;
  h->stats.num_unconverged = unconverged;
  h->stats.num_split = split_count;
  tr.mark("mixed panels", stream, -1, 6);
  hm_status st = matvec_plan_build(h, 16, stream);
  if (st) return cleanup(st);
  tr.mark("matvec plan", stream, -1, 7);
  for (int i = 0; i < PhaseTrace::kSlots; ++i) h->stats.phase_seconds[i] = tr.sec[i];
  HM_CUDA(cudaEventRecord(ev1, stream));
  HM_CUDA(cudaEventSynchronize(ev1));
  float ms = 0;
  HM_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
  h->stats.build_seconds = ms * 1e-3;
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  *out = h;
  return HM_OK;
}

void release_fp32(hm_hmatrix_s* h) {
  h->chunk_meta.clear();
  for (const auto& c : h->storage) h->chunk_meta.push_back({c.p, c.n});
  {
    FreeTogether together;
    h->storage.clear();
  }
  h->fp32_released = true;
}

// Device memory held by the matrix: factor and dense storage, the mixed
// form's panels and tables, the product's plan and workspaces.
long long device_bytes(const hm_hmatrix_s* h) {
  long long b = 0;
  auto add = [&b](const auto& buf) { b += (long long)(buf.n * sizeof(*buf.p)); };
  for (const auto& c : h->storage) add(c);
  const MatvecPlan& P = h->plan;
  add(P.lr), add(P.p1), add(P.multi), add(P.groups), add(P.leaf_ptr), add(P.leaf_blk), add(P.dense);
  add(P.leaf_dptr), add(P.leaf_dblk), add(P.T), add(P.Xp), add(P.Yp);
  const MxPlan& M = h->mx;
  add(M.store), add(M.panels), add(M.pan_of), add(M.units), add(M.tile_leaf), add(M.leaf_tile0), add(M.tslot);
  add(M.mtiles), add(M.dense), add(M.leaf_dptr), add(M.leaf_dblk);
  return b;
}

}  // namespace hm

extern "C" {

void hm_build_opts_default(int d, hm_build_opts* o) {
  if (!o) return;
  o->kernel = HM_KERNEL_EXP;
  o->ell = d == 3 ? 0.2 : 0.1;  // src/TLRMatrixHelpers.cu:40-42
  o->nugget = 0.0;
  o->tol = 1e-5;                // src/config.h:127
  o->max_rank = 64;
  o->leaf_max_rank = 0;
  o->sample_block = 16;         // src/constructTLRMatrix.cu:73
  o->precision = HM_PREC_FP32;
  o->derivative = 0;
  o->seed = 0;
  o->diag_from_coords = -1;
  o->level_schedule = 0;
}

hm_status hm_hmatrix_build(hm_kdtree t, hm_structure s, const double* d_points, const hm_build_opts* opts,
                           void* stream, hm_hmatrix* out) {
  const hm_status st = hm::hmatrix_build(t, s, d_points, opts, hm::as_stream(stream), out, 0, -1);
  hm::dev_settle();
  return st;
}

hm_status hm_hmatrix_build_rows(hm_kdtree t, hm_structure s, const double* d_points, const hm_build_opts* opts,
                                int leaf_begin, int leaf_end, void* stream, hm_hmatrix* out) {
  if (out) *out = nullptr;
  if (!t) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_build_rows: null tree");
  if (leaf_begin < 0 || leaf_begin >= leaf_end || leaf_end > (1 << t->depth))
    return hm::fail(HM_ERR_INVALID, "hm_hmatrix_build_rows: need 0 <= leaf_begin < leaf_end <= 2^depth");
  const hm_status st = hm::hmatrix_build(t, s, d_points, opts, hm::as_stream(stream), out, leaf_begin, leaf_end);
  hm::dev_settle();
  return st;
}

hm_status hm_hmatrix_stats_get(hm_hmatrix h, hm_hmatrix_stats* st) {
  if (!h || !st) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_stats_get: null argument");
  *st = h->stats;
  st->device_bytes = hm::device_bytes(h);
  return HM_OK;
}

hm_status hm_hmatrix_blocks(hm_hmatrix h, long long* num_lowrank, long long* num_dense, int* lowrank,
                            int* dense) {
  if (!h) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_blocks: null matrix");
  if (num_lowrank) *num_lowrank = (long long)h->h_lr.size();
  if (num_dense) *num_dense = (long long)h->h_dense.size();
  if (lowrank)
    for (size_t i = 0; i < h->h_lr.size(); ++i) {
      const hm::LRBlock& b = h->h_lr[i];
      int* r = lowrank + 6 * i;
      r[0] = b.r0;
      r[1] = b.m;
      r[2] = b.c0;
      r[3] = b.n;
      r[4] = b.k;
      r[5] = b.level;
    }
  if (dense)
    for (size_t i = 0; i < h->h_dense.size(); ++i) {
      const hm::DenseBlock& b = h->h_dense[i];
      int* r = dense + 5 * i;
      r[0] = b.r0;
      r[1] = b.m;
      r[2] = b.c0;
      r[3] = b.n;
      r[4] = b.trans;
    }
  return HM_OK;
}

// Host copy of an FP32 array of the matrix (a factor or a dense block, count
// floats): from its storage, or rebuilt from the panels once released.
static hm_status fetch_fp32(hm_hmatrix h, const float* src, size_t count, float* dst) {
  if (!count) return HM_OK;
  if (!h->fp32_released) {
    HM_CUDA(cudaMemcpy(dst, src, sizeof(float) * count, cudaMemcpyDeviceToHost));
    return HM_OK;
  }
  const int loc = hm::mixed_find_loc(h, src);
  if (loc < 0) return hm::fail(HM_ERR_INVALID, "no panel holds this block");
  hm::DevBuf<float> tmp;
  HM_TRY(tmp.alloc(count));
  HM_TRY(hm::mixed_unpack(h, {{loc, tmp.p}}, nullptr));
  HM_CUDA(cudaMemcpy(dst, tmp.p, sizeof(float) * count, cudaMemcpyDeviceToHost));
  return HM_OK;
}

hm_status hm_hmatrix_block_factors(hm_hmatrix h, int i, float* U, float* V) {
  if (!h) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_block_factors: null matrix");
  if (i < 0 || (size_t)i >= h->h_lr.size()) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_block_factors: bad index");
  const hm::LRBlock& b = h->h_lr[i];
  if (U && b.k) HM_TRY(fetch_fp32(h, b.U, (size_t)b.m * b.k, U));
  if (V && b.k) HM_TRY(fetch_fp32(h, b.V, (size_t)b.n * b.k, V));
  return HM_OK;
}

hm_status hm_hmatrix_dense_block(hm_hmatrix h, int i, float* D) {
  if (!h) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_dense_block: null matrix");
  if (i < 0 || (size_t)i >= h->h_dense.size()) return hm::fail(HM_ERR_INVALID, "hm_hmatrix_dense_block: bad index");
  const hm::DenseBlock& b = h->h_dense[i];
  if (D && b.m && b.n) HM_TRY(fetch_fp32(h, b.D, (size_t)b.m * b.n, D));
  return HM_OK;
}

void hm_hmatrix_free(hm_hmatrix h) {
  {
    hm::FreeTogether together;
    delete h;
  }
  hm::dev_settle();
}

}  // extern "C"
