// hm_trunc.cu -- truncation of the sampled blocks.
//
// A ~ Q B^T with B = A^T Q (n x k).  The eigenpairs (lambda_j, w_j) of
// G = B^T B give the singular values sqrt(lambda_j) of that approximation and
// A ~ (Q W_r)(B W_r)^T with the smallest r whose discarded sum of lambda fits
// the tolerance left after the sampling residual.  Columns come out in
// decreasing singular value; U = Q W_r is orthonormal, |V_j| = sqrt(lambda_j).
//
// Three kernels, each launched per width class (k <= 32, 64, 128), so that a
// narrow block neither pays for the widest block's shared memory nor waits in
// a large CTA:
//   k_gram   G on the FP64 tensor instruction (mma.sync m8n8k4: a Gram tile's
//            two operands are the same fragment), the values converted to
//            FP64 once while staged; blocks of more than kGramRows rows in
//            chunks, whose partial sums the next kernel adds in order.
//   k_eig    pivoted Cholesky G = L L^T (one warp, lane = row; or one thread
//            per row), then one-sided Jacobi on L's columns: after the pivoted
//            factor they are graded and close to orthogonal, so few sweeps
//            remain, a rotation touches two columns instead of two rows, two
//            columns and an accumulated W, and the normalised columns are the
//            eigenvectors.  Rotation angles are taken in FP32 (an angle only
//            has to reduce the inner product; the next visit sees what is
//            left), cosine and sine are completed to FP64, so the columns stay
//            orthogonally equivalent to L in FP64.  One barrier per step.
//   k_pack   64-row tiles of U and V, 4 x 4 sums per thread.
// Bound by instruction issue and barriers (k_eig) and L2 latency (k_gram).
// Measured against two-sided Jacobi with shared memory sized by the batch's
// widest block, one CTA per block and per-thread column arrays (device time of
// a build, Gram / eigenpairs / factors):
//   2^17-point Matern, k mostly <= 32    22.3 / 37.0 / 18.4 -> 0.86 / 5.6 / 1.8 ms
//   60001-point mixture, k to 256        10.5 / 154 / 58.6  -> 2.8 / 9.7 / 0.7 ms
//   20000-point Gauss, K and dK/dl       7.3 / 246 / 18.8   -> 2.4 / 16.8 / 1.2 ms
#include <algorithm>

#include "hm_ara.h"
#include "hm_mma.cuh"

namespace hm {
namespace {

constexpr int kGramRows = 2048;  // rows of B per CTA
constexpr int kTile = 64;        // rows of U or V per CTA of k_pack

template <typename W>
struct Row4 {  // four consecutive rows of one column
  W x[4];
  __device__ __forceinline__ void load(const W* p) {
    if (sizeof(W) == 4) {
      const float4 v = *reinterpret_cast<const float4*>(p);
      x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
    } else {
      const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
      x[0] = a.x, x[1] = a.y, x[2] = b.x, x[3] = b.y;
    }
  }
};

// Items (problem, row chunk); G's partial of chunk c at goff[problem] + c k^2
// (upper triangle).
template <typename W, int KT, int NW>
__global__ void __launch_bounds__(32 * NW) k_gram(const int2* __restrict__ items, const Prob* __restrict__ probs,
                                                  const ProbState* __restrict__ st, const long long* __restrict__ goff,
                                                  double* __restrict__ G) {
  constexpr int RS = KT == 128 ? 32 : 64;  // rows staged at a time
  constexpr int LD = RS + 4;               // a half-warp's 4 columns x 4 rows fall into 16 banks
  constexpr int NT = 32 * NW;
  constexpr int T = KT / 8, MAXT = (T * (T + 1) / 2 + NW - 1) / NW;
  extern __shared__ __align__(16) unsigned char gsm[];
  double* Bs = reinterpret_cast<double*>(gsm);  // [KT][LD]
  const int2 it = items[blockIdx.x];
  const Prob P = probs[it.x];
  const int k = st[it.x].k, ld = ara_ld(P.n);
  const int row0 = it.y * kGramRows, row1 = min(ld, row0 + kGramRows);
  const W* B = reinterpret_cast<const W*>(P.b);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int nt = (k + 7) >> 3, ntiles = nt * (nt + 1) / 2;
  // this warp's tiles (a <= b), numbered row by row of the upper triangle
  int ta[MAXT], tb[MAXT];
#pragma unroll
  for (int i = 0; i < MAXT; ++i) {
    int w = warp + i * NW, a = 0;
    if (w < ntiles) {
      while (w >= nt - a) w -= nt - a, ++a;
      ta[i] = a;
      tb[i] = a + w;
    } else {
      ta[i] = -1;
      tb[i] = 0;
    }
  }
  double acc[MAXT][2];
#pragma unroll
  for (int i = 0; i < MAXT; ++i) acc[i][0] = acc[i][1] = 0.0;
  const double* mine = Bs + (lane >> 2) * LD + (lane & 3);
  for (int i0 = row0; i0 < row1; i0 += RS) {
    __syncthreads();
    for (int e = t; e < nt * 8 * (RS / 4); e += NT) {
      const int c = e / (RS / 4), v = e % (RS / 4);
      Row4<W> x;
      if (c < k && i0 + 4 * v < row1)
        x.load(B + (size_t)c * ld + i0 + 4 * v);
      else
        x.x[0] = x.x[1] = x.x[2] = x.x[3] = W(0);
      double2* d = reinterpret_cast<double2*>(Bs + c * LD + 4 * v);
      d[0] = make_double2((double)x.x[0], (double)x.x[1]);
      d[1] = make_double2((double)x.x[2], (double)x.x[3]);
    }
    __syncthreads();
    const int nq = min(RS, row1 - i0) >> 2;
    for (int q = 0; q < nq; ++q) {
#pragma unroll
      for (int i = 0; i < MAXT; ++i)
        if (ta[i] >= 0) mma_f64(acc[i], mine[8 * ta[i] * LD + 4 * q], mine[8 * tb[i] * LD + 4 * q]);
    }
  }
  double* g = G + goff[it.x] + (size_t)it.y * k * k;
#pragma unroll
  for (int i = 0; i < MAXT; ++i) {
    if (ta[i] < 0) continue;
    const int r = 8 * ta[i] + (lane >> 2), c = 8 * tb[i] + 2 * (lane & 3);
    if (r < k && c < k && r <= c) g[r * k + c] = acc[i][0];
    if (r < k && c + 1 < k && r <= c + 1) g[r * k + c + 1] = acc[i][1];
  }
}

// Pivoted Cholesky G = L L^T in place, thread i = row i (KT threads take
// part): step j writes L's column to the storage of G's column p_j, the pivot.
// A is column-major, A[c * LD + row]; untouched columns (below tau) are zeroed.
template <int KT, int LD>
__device__ void chol_columns(double* A, int k, double tau, int* perm, unsigned* red, int* piv) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool mine = t < k;
  bool open = mine;
  double diag = mine ? A[t * LD + t] : 0.0;
  for (int j = 0; j < k; ++j) {
    // the largest remaining diagonal by its leading 32 bits, the lowest row first
    const unsigned key = open && diag > tau ? (unsigned)__double2hiint(diag) : 0u;
    unsigned top = __reduce_max_sync(0xffffffffu, key);
    int p;
    if (KT == 32) {
      if (top == 0u) break;
      p = __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
    } else {
      if (lane == 0 && warp < KT / 32) red[warp] = top;
      if (t == 0) *piv = KT;
      __syncthreads();
      top = 0u;
#pragma unroll
      for (int w = 0; w < KT / 32; ++w) top = max(top, red[w]);
      if (top == 0u) break;  // every thread alike
      if (key == top) atomicMin(piv, t);
      __syncthreads();
      p = *piv;
    }
    double s0 = mine ? A[p * LD + t] : 0.0, s1 = 0.0;
    if (open) {
      int b = 0;
      for (; b + 1 < j; b += 2) {
        const double* c0 = A + perm[b] * LD;
        const double* c1 = A + perm[b + 1] * LD;
        s0 = fma(-c0[t], c0[p], s0);
        s1 = fma(-c1[t], c1[p], s1);
      }
      if (b < j) {
        const double* c0 = A + perm[b] * LD;
        s0 = fma(-c0[t], c0[p], s0);
      }
    }
    double dp;
    if (KT == 32) {
      dp = __shfl_sync(0xffffffffu, diag, p);
    } else {
      __shared__ double dsh;
      if (t == p) dsh = diag;
      __syncthreads();
      dp = dsh;
    }
    const double rd = rsqrt(dp);
    double l = open ? (s0 + s1) * rd : 0.0;
    if (t == p) {
      l = dp * rd;
      open = false;
    }
    diag = fma(-l, l, diag);
    if (mine) A[p * LD + t] = l;
    if (t == 0) perm[j] = p;
    if (KT == 32)
      __syncwarp();
    else
      __syncthreads();
  }
  // rows still open never became pivots: their columns hold no part of L
  if (open)
    for (int i = 0; i < k; ++i) A[t * LD + i] = 0.0;
}

// One CTA of 4 KT threads per problem: eight lanes per column pair, KT / 2
// pairs per step.
template <int KT>
__global__ void __launch_bounds__(4 * KT) k_eig(const int* __restrict__ ids, const Prob* __restrict__ probs,
                                                ProbState* __restrict__ st, const long long* __restrict__ goff,
                                                const double* __restrict__ G, const long long* __restrict__ woff,
                                                float* __restrict__ Wr, double tol2, double rbudget) {
  constexpr int NT = 4 * KT, LD = KT + 2, RL = KT / 8;  // rows per lane
  extern __shared__ __align__(16) unsigned char esm[];
  double* A = reinterpret_cast<double*>(esm);  // [KT][LD], column-major
  double* nrm = A + KT * LD;                   // [KT] squared column norms
  int* order = reinterpret_cast<int*>(nrm + KT);  // [KT]; the Cholesky order before
  __shared__ double off_sh[NT / 32];
  __shared__ unsigned red[4];
  __shared__ int piv, r_sh;
  const int p = ids[blockIdx.x];
  const ProbState S = st[p];
  const int k = S.k, t = threadIdx.x;
  if (k > KT || k <= 1) {  // kept as sampled: every column keeps its low part
    if (t == 0) {
      st[p].r = k;
      st[p].rhi = k;
      if (k == 1) Wr[woff[p]] = 1.f;
    }
    return;
  }
  const Prob P = probs[p];
  const int nch = (ara_ld(P.n) + kGramRows - 1) / kGramRows;
  const double* g = G + goff[p];
  for (int e = t; e < k * k; e += NT) {
    const int r = e / k, c = e % k;
    if (r > c) continue;
    double v = 0.0;
    for (int q = 0; q < nch; ++q) v += g[(size_t)q * k * k + e];
    A[c * LD + r] = v;
    A[r * LD + c] = v;
  }
  __syncthreads();
  // to a trace in [1, 2) (an exact power of two), so that FP32 angles neither
  // overflow nor vanish
  double trace = 0.0;
  for (int i = 0; i < k; ++i) trace += A[i * LD + i];
  const int ex = trace > 0.0 ? ilogb(trace) : 0;
  const double unit = scalbn(1.0, -ex), back = scalbn(1.0, ex);
  __syncthreads();
  for (int e = t; e < k * k; e += NT) {
    double* a = A + (e / k) * LD + e % k;
    *a *= unit;
  }
  trace *= unit;
  __syncthreads();
  if (KT > 32)  // pivots below the rounding of G's diagonal carry nothing
    chol_columns<KT, LD>(A, k, 2e-16 * trace, order, red, &piv);
  else if (t < 32)
    chol_columns<KT, LD>(A, k, 2e-16 * trace, order, red, &piv);
  __syncthreads();
  // ---- one-sided Jacobi: pairs of a round-robin tournament over kp columns ----
  const int kp = (k + 1) & ~1, rounds = kp - 1;
  const int pr = t >> 3, l8 = t & 7;
  const unsigned lanes = 0xffu << (t & 24);  // this pair's lanes
  for (int sweep = 0; sweep < 12; ++sweep) {
    for (int c = pr; c < k; c += NT / 8) {  // norms afresh once a sweep
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < RL; ++i) {
        const int r = l8 + 8 * i;
        const double x = r < k ? A[c * LD + r] : 0.0;
        s = fma(x, x, s);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(lanes, s, o);
      if (l8 == 0) nrm[c] = s;
    }
    __syncthreads();
    double off = 0.0;
    for (int step = 0; step < rounds; ++step) {
      if (pr < kp / 2) {
        int a, b;
        if (pr == 0) {
          a = step;
          b = rounds;
        } else {
          a = step + pr;
          if (a >= rounds) a -= rounds;
          b = step - pr;
          if (b < 0) b += rounds;
        }
        if (a < k && b < k) {  // an odd k's dummy column rests
          double* ca = A + a * LD + l8;
          double* cb = A + b * LD + l8;
          double x[RL], y[RL], d = 0.0;
#pragma unroll
          for (int i = 0; i < RL; ++i) {
            const bool in = l8 + 8 * i < k;
            x[i] = in ? ca[8 * i] : 0.0;
            y[i] = in ? cb[8 * i] : 0.0;
            d = fma(x[i], y[i], d);
          }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) d += __shfl_xor_sync(lanes, d, o);
          const double na = nrm[a], nb = nrm[b];
          off = fma(d, d, off);
          if (fabs(d) > 1e-18 * trace && d * d > 1e-30 * (na * nb)) {
            // tan of the angle that makes the columns orthogonal: 2d / (D + sign(D) sqrt(D^2 + 4 d^2)), D = nb - na
            const float fx = (float)(2.0 * d), fy = (float)(nb - na);
            const float h = 1.0f / fmaxf(fmaxf(fabsf(fx), fabsf(fy)), 1e-37f);
            const float ux = fx * h, uy = fy * h;
            const float tf = ux / (uy + copysignf(sqrtf(fmaf(ux, ux, uy * uy)), uy));
            const double tt = (double)tf, q = fma(tt, tt, 1.0);
            double c = (double)rsqrtf((float)q);
            c = c * fma(-0.5 * q * c, c, 1.5);
            c = c * fma(-0.5 * q * c, c, 1.5);
            const double s = tt * c;
#pragma unroll
            for (int i = 0; i < RL; ++i) {
              if (l8 + 8 * i < k) {
                ca[8 * i] = fma(c, x[i], -s * y[i]);
                cb[8 * i] = fma(c, y[i], s * x[i]);
              }
            }
            __syncwarp(lanes);  // every lane of the pair has read the norms
            if (l8 == 0) {
              // |c a - s b|^2 and |s a + c b|^2 for whatever angle was taken
              const double cc = c * c, ss = s * s, cs2 = 2.0 * c * s * d;
              nrm[a] = fma(cc, na, fma(ss, nb, -cs2));
              nrm[b] = fma(ss, na, fma(cc, nb, cs2));
            }
          }
        }
      }
      __syncthreads();
    }
    // sum of d^2 over the pairs of the sweep (one lane per pair counts)
    if (l8 != 0) off = 0.0;
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
    if ((t & 31) == 0) off_sh[t >> 5] = off;
    __syncthreads();
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) sum += off_sh[w];
    if (sum <= 1e-26 * trace * trace) break;
    __syncthreads();
  }
  // ---- eigenvalues, their order, the ranks ----
  for (int c = pr; c < k; c += NT / 8) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < RL; ++i) {
      const int r = l8 + 8 * i;
      const double x = r < k ? A[c * LD + r] : 0.0;
      s = fma(x, x, s);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(lanes, s, o);
    if (l8 == 0) nrm[c] = s;
  }
  __syncthreads();
  for (int i = t; i < k; i += NT) {
    const double li = nrm[i];
    int rk = 0;
    for (int j = 0; j < k; ++j) {
      const double lj = nrm[j];
      rk += (lj > li) || (lj == li && j < i);
    }
    order[rk] = i;
  }
  __syncthreads();
  if (t == 0) {
    // discard the smallest eigenvalues while their sum fits the budget
    const double ts2 = P.tscale2;
    const double budget = tol2 * ts2 * S.normA2 - S.est;
    double tail = 0.0;
    int r = k;
    if (S.converged && budget > 0) {
      while (r > 1) {
        const double l = nrm[order[r - 1]] * back;
        if (tail + l > budget) break;
        tail += l;
        --r;
      }
    }
    // Mixed precision: column j of U V^T carries |u_j||v_j| = sigma_j; rounding
    // both to BF16 perturbs it by at most ~2 * 2^-9 sigma_j.  The trailing
    // columns whose rounding error fits rbudget keep only their BF16 high part.
    int rhi = r;
    if (rbudget > 0) {
      double rt = 0.0;
      const double c = 2.0 * 0x1p-18;  // (2^-9)^2 for each of u_j and v_j
      while (rhi > 0) {
        const double l = nrm[order[rhi - 1]] * back;
        if (rt + c * l > rbudget * ts2 * S.normA2) break;
        rt += c * l;
        --rhi;
      }
    }
    r_sh = r;
    st[p].r = r;
    st[p].rhi = rhi;
  }
  __syncthreads();
  float* w = Wr + woff[p];
  for (int e = t; e < k * r_sh; e += NT) {
    const int a = e % k, c = order[e / k];
    const double n2 = nrm[c];
    w[e] = n2 > 0.0 ? (float)(A[c * LD + a] * rsqrt(n2)) : 0.f;
  }
}

// Rows [64 tile, 64 tile + 64) of U = Q W_r (SIDE 0) or V = B W_r (SIDE 1).
// Thread: 4 rows x 4 columns of up to 32 columns at a time; a half-warp's rows
// are one 256-byte run of a basis column.
template <typename W, int SIDE>
__global__ void __launch_bounds__(128) k_pack(const int2* __restrict__ items, const Prob* __restrict__ probs,
                                              const ProbState* __restrict__ st, const long long* __restrict__ woff,
                                              const float* __restrict__ Wr, const long long* __restrict__ at,
                                              float* __restrict__ dst) {
  __shared__ __align__(16) float wsh[kTruncMax * 32];  // [k][32]
  const int2 it = items[blockIdx.x];
  const int p = it.x, k = st[p].k, r = st[p].r;
  if (at[p] < 0 || r <= 0) return;
  const Prob P = probs[p];
  const int rows = SIDE ? P.n : P.m, ld = ara_ld(rows);
  const W* src = reinterpret_cast<const W*>(SIDE ? P.b : P.q);
  float* out = dst + at[p];
  const int t = threadIdx.x;
  if (k > kTruncMax) {  // kept as sampled (W_r = I)
    for (int e = t; e < kTile * r; e += 128) {
      const int i = it.y * kTile + e % kTile;
      if (i < rows) out[(size_t)(e / kTile) * rows + i] = (float)src[(size_t)(e / kTile) * ld + i];
    }
    return;
  }
  const int i0 = it.y * kTile + 4 * (t & 15), c0 = 4 * (t >> 4);
  const float* w = Wr + woff[p];
  for (int cb = 0; cb < r; cb += 32) {
    const int nc = min(32, r - cb);
    __syncthreads();
    for (int e = t; e < 32 * k; e += 128) {
      const int c = e / k, a = e % k;
      wsh[a * 32 + c] = c < nc ? w[(size_t)(cb + c) * k + a] : 0.f;
    }
    __syncthreads();
    if (i0 >= ld || c0 >= nc) continue;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const W* q = src + i0;
#pragma unroll 4
    for (int a = 0; a < k; ++a) {
      Row4<W> x;
      x.load(q + (size_t)a * ld);
      const float4 v = *reinterpret_cast<const float4*>(wsh + a * 32 + c0);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float xi = (float)x.x[i];
        acc[i][0] = fmaf(xi, v.x, acc[i][0]);
        acc[i][1] = fmaf(xi, v.y, acc[i][1]);
        acc[i][2] = fmaf(xi, v.z, acc[i][2]);
        acc[i][3] = fmaf(xi, v.w, acc[i][3]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c0 + c >= nc) break;
      float* o = out + (size_t)(cb + c0 + c) * rows + i0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i0 + i < rows) o[i] = acc[i][c];
    }
  }
}

template <int KT>
constexpr size_t gram_smem() {
  return sizeof(double) * KT * ((KT == 128 ? 32 : 64) + 4);
}
template <int KT>
constexpr size_t eig_smem() {
  return sizeof(double) * (KT * (KT + 2) + KT) + sizeof(int) * KT;
}

template <typename W, int KT, int NW>
hm_status launch_gram(const int2* items, size_t count, const Prob* probs, const ProbState* st,
                      const long long* goff, double* G, cudaStream_t s) {
  if (!count) return HM_OK;
  HM_CUDA(cudaFuncSetAttribute(k_gram<W, KT, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gram_smem<KT>()));
  k_gram<W, KT, NW><<<(unsigned)count, 32 * NW, gram_smem<KT>(), s>>>(items, probs, st, goff, G);
  HM_LAUNCH_CHECK();
  return HM_OK;
}
template <int KT>
hm_status launch_eig(const int* ids, size_t count, const Prob* probs, ProbState* st, const long long* goff,
                     const double* G, const TruncWork& tw, double tol2, double rbudget, cudaStream_t s) {
  if (!count) return HM_OK;
  HM_CUDA(cudaFuncSetAttribute(k_eig<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)eig_smem<KT>()));
  k_eig<KT><<<(unsigned)count, 4 * KT, eig_smem<KT>(), s>>>(ids, probs, st, goff, G, tw.woff.p, tw.w.p, tol2, rbudget);
  HM_LAUNCH_CHECK();
  return HM_OK;
}

template <typename T>
hm_status upload(DevBuf<T>& d, const std::vector<T>& v, cudaStream_t s) {
  HM_TRY(d.alloc_async(std::max<size_t>(v.size(), 1), s));
  HM_CUDA(cudaMemcpyAsync(d.p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, s));
  return HM_OK;
}

}  // namespace

template <typename W>
hm_status trunc_rank(const std::vector<Prob>& bp, const std::vector<ProbState>& hst, const Prob* probs, ProbState* st,
                     double tol2, double rbudget, TruncWork* tw, cudaStream_t s) {
  const size_t nb = bp.size();
  std::vector<long long> goff(nb, 0), woff(nb, 0);
  std::vector<int2> items[3];
  std::vector<int> ids[3];
  size_t gtot = 0, wtot = 0;
  for (size_t i = 0; i < nb; ++i) {
    const int k = hst[i].k;
    if (k <= 0) continue;  // r = rhi = 0 as initialised
    const int c = k <= 32 || k > kTruncMax ? 0 : (k <= 64 ? 1 : 2);
    ids[c].push_back((int)i);
    if (k > kTruncMax) continue;
    woff[i] = (long long)wtot;
    wtot += (size_t)k * k;
    if (k <= 1) continue;
    const int nch = (ara_ld(bp[i].n) + kGramRows - 1) / kGramRows;
    goff[i] = (long long)gtot;
    gtot += (size_t)nch * k * k;
    for (int q = 0; q < nch; ++q) items[c].push_back(make_int2((int)i, q));
  }
  std::vector<int2> all_items;
  std::vector<int> all_ids;
  for (int c = 0; c < 3; ++c) {
    all_items.insert(all_items.end(), items[c].begin(), items[c].end());
    all_ids.insert(all_ids.end(), ids[c].begin(), ids[c].end());
  }
  DevBuf<long long> dgoff;
  DevBuf<double> G;
  DevBuf<int2> ditems;
  DevBuf<int> dids;
  HM_TRY(upload(dgoff, goff, s));
  HM_TRY(upload(tw->woff, woff, s));
  HM_TRY(upload(ditems, all_items, s));
  HM_TRY(upload(dids, all_ids, s));
  HM_TRY(G.alloc_async(std::max<size_t>(gtot, 1), s));
  HM_TRY(tw->w.alloc_async(std::max<size_t>(wtot, 1), s));
  const int2* it = ditems.p;
  HM_TRY((launch_gram<W, 32, 4>(it, items[0].size(), probs, st, dgoff.p, G.p, s)));
  it += items[0].size();
  HM_TRY((launch_gram<W, 64, 4>(it, items[1].size(), probs, st, dgoff.p, G.p, s)));
  it += items[1].size();
  HM_TRY((launch_gram<W, 128, 8>(it, items[2].size(), probs, st, dgoff.p, G.p, s)));
  const int* id = dids.p;
  // the widest first: their CTAs run the longest
  HM_TRY(launch_eig<128>(id + ids[0].size() + ids[1].size(), ids[2].size(), probs, st, dgoff.p, G.p, *tw, tol2, rbudget, s));
  HM_TRY(launch_eig<64>(id + ids[0].size(), ids[1].size(), probs, st, dgoff.p, G.p, *tw, tol2, rbudget, s));
  HM_TRY(launch_eig<32>(id, ids[0].size(), probs, st, dgoff.p, G.p, *tw, tol2, rbudget, s));
  return HM_OK;
}

template <typename W>
hm_status trunc_pack(const Prob* probs, const ProbState* st, const TruncWork& tw, const int2* rows, size_t nrows,
                     const int2* cols, size_t ncols, const long long* dst_u, const long long* dst_v,
                     float* dst, cudaStream_t s) {
  if (nrows) k_pack<W, 0><<<(unsigned)nrows, 128, 0, s>>>(rows, probs, st, tw.woff.p, tw.w.p, dst_u, dst);
  HM_LAUNCH_CHECK();
  if (ncols) k_pack<W, 1><<<(unsigned)ncols, 128, 0, s>>>(cols, probs, st, tw.woff.p, tw.w.p, dst_v, dst);
  HM_LAUNCH_CHECK();
  return HM_OK;
}

template hm_status trunc_rank<float>(const std::vector<Prob>&, const std::vector<ProbState>&, const Prob*, ProbState*,
                                     double, double, TruncWork*, cudaStream_t);
template hm_status trunc_rank<double>(const std::vector<Prob>&, const std::vector<ProbState>&, const Prob*, ProbState*,
                                      double, double, TruncWork*, cudaStream_t);
template hm_status trunc_pack<float>(const Prob*, const ProbState*, const TruncWork&, const int2*, size_t, const int2*,
                                     size_t, const long long*, const long long*, float*, cudaStream_t);
template hm_status trunc_pack<double>(const Prob*, const ProbState*, const TruncWork&, const int2*, size_t, const int2*,
                                      size_t, const long long*, const long long*, float*, cudaStream_t);

}  // namespace hm
