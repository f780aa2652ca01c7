// hm_mixed_tc.cu -- the mixed form's 128-column passes on the Blackwell
// tensor cores (tcgen05.mma, accumulator in tensor memory).
//
// A pass of 128 right-hand sides multiplies every factor element 128 times
// (hi and lo: up to 3 BF16 products each), more than the warp-level MMA
// keeps up with at HBM speed.
//
// Phase 1 (k_mx_p1_tc): one CTA per SM walks its units -- up to 16 column
// tiles of a panel, all with low parts or none, over a chunk of row tiles --
// and per 32-row tile issues D (128 columns x 128 right-hand sides, FP32 in
// TMEM) += V^T X as tcgen05.mma of M = 128, N = 128, K = 16:
//   A = V^T: the unit's P1 tiles of one row tile, one bulk copy (TMA
//     engine): the tiles are stored in the K-major core-matrix layout with the
//     64-byte swizzle (column 8 j + g's 64-byte row at 512 j + 64 g; SBO 512).
//     A K block t holds rows rho(t, e) = 8 (e / 2) + 2 t + e % 2, a
//     permutation of the tile's rows, harmless in a sum as B uses the same.
//   B = X: the pass's image per 32-row tile written by k_mx_split_x (hi 8 KB,
//     then lo; right-hand side n at 16 (n % 8) + 128 (n / 8), K block c at
//     2048 c: SBO 128, LBO 2048), one bulk copy each.
// Columns with low parts take three products per tile (V_hi X_hi, V_hi X_lo,
// V_lo X_hi), one row tile per step; the others one, two row tiles per step.
//
// Warp roles, no CTA-wide barrier in the loop: two copy warps take the steps in
// turn, each lane one bulk copy into one of six 32 KB stages (counted in bytes
// on the stage's "full" mbarrier); one lane of the MMA warp waits for it, issues
// the step's MMAs and commits them to the stage's "empty" mbarrier; chains of
// four steps go into one of four TMEM accumulators (128 columns each), committed
// to its "ready" mbarrier; four drain warps (TMEM lanes 32 (w % 4) ..) read a
// ready accumulator out (tcgen05.ld), add it to their FP32 sums with
// round-to-nearest adds, and release it.  Units and blocks are dealt to the CTAs
// in row order, each to the least loaded, and every role holds 32 descriptors at
// a time, one per lane.
// What bounds it: instructions.  A step's MMAs take about 400 clocks, but with
// one copy warp laying out and issuing a phase-2 step's 10-20 copies took 1600
// clocks, and issuing its MMAs from a loop over K 730; copying 16 bytes per
// step, three stages or chains of 16 steps changed nothing.  Two copy warps
// (four, or 8 and 16 drain warps, take issue slots from the MMA warp: 8-20 %
// slower), straight-line MMA code and 32 descriptors per load give, at 131072
// mixture points, 0.31 ms for phase 1 (0.38 before) and 0.36 ms for phase 2
// (1.15 with A rearranged word by word, 0.60 with one copy warp).
// The tensor core's own sums do not round to nearest, so the chains are kept
// short: 24 MMAs for columns with low parts, a drift far below the BF16 hi + lo
// rounding of T.  At a unit's end each drain thread
// stores its column (its TMEM lane): as T (into the mirror column's slots,
// split hi + lo or hi only) when the panel is projected in one row chunk,
// else as the chunk's partial S (per column its 128 FP32 sums, contiguous).
// Every wait is bounded; a wait that gives up raises an abort flag that the
// other roles see, sets the error word, and the kernel ends after every
// issued copy and MMA has completed.
//
// T of such a pass is kept in 2 KB blocks, one per 8 columns and part (hi,
// lo): the MN-major core-matrix image of B = T for phase 2 (right-hand sides
// n, columns c: 2 (n % 8) + 128 (n / 8) + 16 c bytes; SBO 128, LBO 2048),
// in which a column's 8 consecutive right-hand sides are 16 contiguous bytes:
// a drain thread writes its column with 16-byte stores.
//
// Phase 2 (k_mx_p2_tc): one CTA per SM walks blocks of 4 row tiles (128
// rows), D (128 rows x 128 right-hand sides) += U T per ancestor panel and
// D X per dense block, M = 128, N = 128.  A = the P1 tiles of phase 1 again,
// read as an M-major operand: a tile's column is 32 rows in 64 contiguous
// bytes, so the K-major image of V^T is the M-major image of U and the copy
// engine moves it as it is; the rows of D come out in the tiles' order rho and
// go to their place at the store.  (Rearranging the other tile order by 4-byte
// cp.async with 27 copy warps took 1.15 ms at 131072 mixture points.)  Dense
// blocks' 32 x 32 tiles are K-major images as stored (dense_word): their rows
// are in the same order rho, their columns in X's, so that B is X's image of
// the column cluster's tile.  Panels' columns with low parts
// take three products per 16 columns, 32 columns per step; the others one per
// 16 columns, 64 per step; dense blocks three per 16 columns, 32 per step.
#include <atomic>

#include "hm_hmatrix.h"
#include "hm_mixed.h"
#include "hm_mma.cuh"
#include "hm_tc.cuh"

namespace hm {
namespace {

constexpr int kTcStage = 32768;          // bytes per stage
constexpr uint32_t kIdesc = tc_idesc_bf16(128, 128);
constexpr uint32_t kIdescBmn = tc_idesc_bf16(128, 128) | (1u << 16);  // B MN-major

// ---- phase 1 ------------------------------------------------------------------
constexpr int kP1Stages = 6;
constexpr int kP1Bufs = 4;       // TMEM accumulators of 128 columns (all 512)
constexpr int kP1Chain = 4;      // steps per MMA chain
constexpr int kDrainWarps = 4;  // drain warps of either phase (a multiple of 4: one per 32 TMEM lanes)
constexpr int kDrainCols = 512 / kDrainWarps;        // right-hand sides per drain warp
constexpr int kCopyWarps = 2;  // copy warp w takes every kCopyWarps-th step from w on
constexpr int kMmaWarp = kCopyWarps, kDrainWarp0 = kCopyWarps + 1;
constexpr int kTcThreads = 32 * (kDrainWarp0 + kDrainWarps);
// shared memory: stages, then mbarriers full[S], empty[S], ready[B], free[B],
// done; then the TMEM address and the abort flag
constexpr int kP1BarBytes = 8 * (2 * kP1Stages + 2 * kP1Bufs + 1);
constexpr size_t kP1Smem = (size_t)kP1Stages * kTcStage + kP1BarBytes + 16;

// Stage layout (bytes): columns with low parts: A_hi 0, A_lo 8192, B_hi
// 16384, B_lo 24576 (one row tile); without: A_hi of row tile k at 8192 k,
// B_hi at 16384 + 8192 k (two row tiles).  A: 64-byte swizzle, SBO 512, K
// chunk q (16 rows) at +32 q bytes; B: no swizzle, SBO 128, LBO 2048, K chunk
// q at +4096 q.

// 16-byte word (right-hand sides 8 q .. 8 q + 7, column pos % 8) of T's block pos / 8
__device__ __forceinline__ long long tb_word(long long pos, int q) { return (pos >> 3) * 128 + q * 8 + (pos & 7); }
// 8 values as BF16 hi, and their BF16 lo (value - hi)
__device__ __forceinline__ void split8(const float* v, uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split_bf16x2(v[2 * i], v[2 * i + 1], h[i], l[i]);
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Drain thread m (the unit's column m, its TMEM lane) of a finished unit: T
// or the chunk's partial S (column c of S tile i at floats 128 (8 i + c)),
// right-hand sides R0 .. R0 + 8 NQ - 1.
template <int NQ>
__device__ __forceinline__ void p1_store(long long out_tile, int nct, int flags, const float (&acc)[8 * NQ], int q0,
                                         int2 e, float* __restrict__ S, uint4* __restrict__ Tb, int m) {
  const int jt = m >> 3, c = m & 7;
  if (jt >= nct) return;
  if (flags & 2) {
    const bool pad = e.x < 0;  // a padding column: zeros into its own slots
    const long long hp = pad ? -1 - (long long)e.x : e.x;
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      uint4 hi, lo;
      split8(acc + 8 * q, hi, lo);
      Tb[tb_word(hp, q0 + q)] = pad ? z : hi;
      if (e.y >= 0) Tb[tb_word(e.y, q0 + q)] = pad ? z : lo;
    }
  } else {
    float4* out = reinterpret_cast<float4*>(S + ((out_tile + jt) * 8 + c) * 128) + 2 * q0;
#pragma unroll
    for (int q = 0; q < 2 * NQ; ++q) out[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
  }
}

__device__ __forceinline__ int p1_step_tiles(int flags, int left) { return (flags & 1) ? 1 : min(2, left); }

// CTA c's units are [cta_ptr[c], cta_ptr[c + 1]).  Every role holds 32 units'
// descriptors at a time, one per lane.
__global__ void __launch_bounds__(kTcThreads, 1)
    k_mx_p1_tc(const TcUnit* __restrict__ units, const int* __restrict__ cta_ptr, const uint4* __restrict__ store,
               const uint4* __restrict__ Xtc, const int2* __restrict__ tslot_tc, float* __restrict__ S,
               uint4* __restrict__ Tb, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t full = sbase + (uint32_t)(kP1Stages * kTcStage), empty = full + 8u * kP1Stages;
  const uint32_t ready = empty + 8u * kP1Stages, freeb = ready + 8u * kP1Bufs, done = freeb + 8u * kP1Bufs;
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + kP1Stages * kTcStage + kP1BarBytes);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  if (tid == 0) {
    for (int i = 0; i < kP1Stages; ++i) {
      mbar_init(full + 8u * i, 1);  // thread 0's expect_tx (bulk copies)
      mbar_init(empty + 8u * i, 1);
    }
    for (int i = 0; i < kP1Bufs; ++i) {
      mbar_init(ready + 8u * i, 1);
      mbar_init(freeb + 8u * i, kDrainWarps);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(slot), 128 * kP1Bufs);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(slot);
  const int u0 = cta_ptr[blockIdx.x], u1 = cta_ptr[blockIdx.x + 1];
  bool failed = false;
  auto give_up = [&]() {
    failed = true;
    *abort_flag = 1;
  };

  if (warp < kCopyWarps) {  // ---- producers: one copy per lane
    // lanes 0, 1: A_hi of row tile r + lane; 2, 3: X_hi; 4: A_lo; 5: X_lo
    long long j = 0, last = -1;
    for (int ub = u0; ub < u1 && !failed; ub += 32) {
      TcUnit W{};
      if (ub + lane < u1) W = units[ub + lane];
      const int nu = min(32, u1 - ub);
      for (int i = 0; i < nu && !failed; ++i) {
        const int nrt = __shfl_sync(0xffffffffu, W.nrt, i), flags = __shfl_sync(0xffffffffu, W.flags, i);
        const bool lo = flags & 1;
        const int per = lo ? 1 : 2, nsteps = (nrt + per - 1) / per;
        const int first = (int)((warp - j) & (kCopyWarps - 1));  // this warp's first step of the unit
        if (first < nsteps) {
          const long long vhi = __shfl_sync(0xffffffffu, W.vhi, i), vlo = __shfl_sync(0xffffffffu, W.vlo, i);
          const int shi = __shfl_sync(0xffffffffu, W.shi, i), slo = __shfl_sync(0xffffffffu, W.slo, i);
          const int nct = __shfl_sync(0xffffffffu, W.nct, i), xtile = __shfl_sync(0xffffffffu, W.xtile, i);
          const uint32_t abytes = (uint32_t)nct * 512u;
          // this lane's copy: of the step's row tile k, from src0 + tile * step
          const int k = lo ? 0 : lane & 1;
          const bool is_x = lane == 2 || lane == 3 || lane == 5;
          const uint4* src0 = is_x ? Xtc + (size_t)xtile * 1024 + (lane == 5 ? 512 : 0)
                                   : store + (lane < 2 ? vhi : vlo) * 32;
          const long long adv = is_x ? 1024 : (long long)(lane < 2 ? shi : slo) * 32;
          const uint32_t dst = (is_x ? 16384u : 0u) + (uint32_t)((lane < 4 ? lane & 1 : 1) * 8192);
          const uint32_t size = is_x ? 8192u : abytes;
          const bool mine = lo ? (lane == 0 || lane == 2 || lane == 4 || lane == 5) : lane < 4;
          for (int st = first; st < nsteps; st += kCopyWarps) {
            const long long js = j + st;
            const int s = (int)(js % kP1Stages), r = st * per, nt = min(per, nrt - r);
            const uint32_t base = sbase + (uint32_t)(s * kTcStage), bar = full + 8u * s;
            int ok = 1;
            if (lane == 0) {
              if (js >= kP1Stages &&
                  !mbar_wait_or(empty + 8u * s, (uint32_t)(((js - kP1Stages) / kP1Stages) & 1), abort_flag)) {
                give_up();
                ok = 0;
              } else {
                mbar_arrive_expect_tx(bar, (uint32_t)(lo ? 2 : nt) * (abytes + 8192u));
              }
            }
            if (!__shfl_sync(0xffffffffu, ok, 0)) {
              failed = true;
              break;
            }
            if (mine && k < nt) bulk_g2s(base + dst, src0 + (r + k) * adv, size, bar);
            last = js;
          }
        }
        j += nsteps;
      }
    }
    // The kernel may not end with copies in flight.  The MMAs wait for every
    // step's, but not once any role has given up, which this warp need not have
    // seen: its last copies are waited for here (bounded), whatever happened.
    if (lane == 0)
      for (long long js = last; js >= 0 && js > last - kP1Stages; js -= kCopyWarps)
        mbar_wait(full + 8u * (uint32_t)(js % kP1Stages), (uint32_t)((js / kP1Stages) & 1), kWaitClocks / 8);
    __syncwarp();
  } else if (warp == kMmaWarp) {  // ---- MMA issuer (lane 0; the others hold descriptors)
    const uint64_t adesc0 = tc_sdesc_sw64(sbase, 512), bdesc0 = tc_sdesc(sbase, 2048, 128);
    long long j = 0;
    int chain = -1;
    for (int ub = u0; ub < u1 && !failed; ub += 32) {
      int w_nrt = 0, w_flags = 0;
      if (ub + lane < u1) w_nrt = units[ub + lane].nrt, w_flags = units[ub + lane].flags;
      const int nu = min(32, u1 - ub);
      for (int i = 0; i < nu && !failed; ++i) {
        const int nrt = __shfl_sync(0xffffffffu, w_nrt, i), flags = __shfl_sync(0xffffffffu, w_flags, i);
        const bool lo = flags & 1;
        int in_chain = 0;
        for (int r = 0; r < nrt && !failed;) {
          const int nt = p1_step_tiles(flags, nrt - r), s = (int)(j % kP1Stages);
          if (in_chain == 0) ++chain;
          if (lane == 0) {
            if (in_chain == 0 && chain >= kP1Bufs &&
                !mbar_wait_or(freeb + 8u * (uint32_t)(chain % kP1Bufs), (uint32_t)((chain / kP1Bufs - 1) & 1),
                              abort_flag))
              give_up();
            if (!failed && !mbar_wait_or(full + 8u * s, (uint32_t)((j / kP1Stages) & 1), abort_flag)) give_up();
            if (!failed) {
              tc_fence_after();
              // descriptors of this stage; an offset of o bytes adds o >> 4 to the start address field
              const uint64_t da = adesc0 + (uint64_t)((s * kTcStage) >> 4),
                             db = bdesc0 + (uint64_t)((s * kTcStage) >> 4);
              const uint32_t d = tmem + (uint32_t)((chain % kP1Bufs) * 128);
              uint32_t acc = in_chain == 0 ? 0u : 1u;
              if (lo) {
#pragma unroll
                for (int p = 0; p < 3; ++p) {  // V_hi X_hi, V_hi X_lo, V_lo X_hi
                  const uint32_t pa = p == 2 ? 8192u : 0u, pb = p == 1 ? 24576u : 16384u;
#pragma unroll
                  for (int q = 0; q < 2; ++q) {
                    tc_mma_bf16(d, da + ((pa + (uint32_t)(q * 32)) >> 4), db + ((pb + (uint32_t)(q * 4096)) >> 4),
                                kIdesc, acc);
                    acc = 1u;
                  }
                }
              } else {
                for (int k = 0; k < nt; ++k)
#pragma unroll
                  for (int q = 0; q < 2; ++q) {
                    tc_mma_bf16(d, da + ((uint32_t)(k * 8192 + q * 32) >> 4),
                                db + ((16384u + (uint32_t)(k * 8192 + q * 4096)) >> 4), kIdesc, acc);
                    acc = 1u;
                  }
              }
              tc_commit(empty + 8u * s);
            }
          }
          failed = __shfl_sync(0xffffffffu, failed, 0);
          r += nt;
          ++j;
          if (r >= nrt || ++in_chain == kP1Chain) {
            if (lane == 0 && !failed) tc_commit(ready + 8u * (uint32_t)(chain % kP1Bufs));
            in_chain = 0;
          }
        }
      }
    }
    if (lane == 0) tc_commit(done);  // arrives once every MMA issued above is done
  } else {  // ---- drain warps: TMEM lanes 32 (warp % 4) .., kDrainCols right-hand sides each
    const int m = (warp & 3) * 32 + lane, h = (warp - kDrainWarp0) >> 2;
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(h * kDrainCols);
    float acc[kDrainCols];
#pragma unroll
    for (int i = 0; i < kDrainCols; ++i) acc[i] = 0.f;
    int chain = -1;
    for (int ub = u0; ub < u1 && !failed; ub += 32) {
      long long w_out = 0;
      int w_nct = 0, w_nrt = 0, w_flags = 0;
      if (ub + lane < u1) {
        const TcUnit& W = units[ub + lane];
        w_out = W.out, w_nct = W.nct, w_nrt = W.nrt, w_flags = W.flags;
      }
      const int nu = min(32, u1 - ub);
      for (int i = 0; i < nu && !failed; ++i) {
        const long long out = __shfl_sync(0xffffffffu, w_out, i);
        const int nct = __shfl_sync(0xffffffffu, w_nct, i), nrt = __shfl_sync(0xffffffffu, w_nrt, i);
        const int flags = __shfl_sync(0xffffffffu, w_flags, i);
        // the column's slots, fetched while the unit's steps run
        int2 e = make_int2(-1, -1);
        if ((flags & 2) && (m >> 3) < nct) e = __ldg(tslot_tc + (out + (m >> 3)) * 8 + (m & 7));
        const int nsteps = (flags & 1) ? nrt : (nrt + 1) / 2;
        const int nchains = (nsteps + kP1Chain - 1) / kP1Chain;
        for (int c = 0; c < nchains; ++c) {
          ++chain;
          const uint32_t b = (uint32_t)(chain % kP1Bufs);
          if (!warp_wait_or(ready + 8u * b, (uint32_t)((chain / kP1Bufs) & 1), abort_flag)) {
            give_up();
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < kDrainCols / 32; ++q) {
            uint32_t v[32];
            tc_ld32(mine + b * 128u + (uint32_t)(q * 32), v);
            tc_wait_ld();
#pragma unroll
            for (int k = 0; k < 32; ++k) acc[q * 32 + k] += __uint_as_float(v[k]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(freeb + 8u * b);
        }
        if (failed) break;
        p1_store<kDrainCols / 8>(out, nct, flags, acc, h * (kDrainCols / 8), e, S, Tb, m);
#pragma unroll
        for (int k = 0; k < kDrainCols; ++k) acc[k] = 0.f;
      }
    }
  }
  if (failed) atomicOr(err, 1);
  // the tensor memory is released once every MMA is done (thread 0 waits,
  // bounded; the others wait at the barrier)
  if (tid == 0 && !mbar_wait(done, 0, 5 * kWaitClocks)) atomicOr(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128 * kP1Bufs);
  }
}

// ---- chunk reduction (panels projected in several row chunks) -----------------
// The chunk partials of each column summed in chunk order, as T blocks: one
// thread per column tile, column c and 8 right-hand sides q.
__global__ void k_mx_reduce_tc(const int2* __restrict__ mtiles, long long nmt, const MxPanel* __restrict__ panels,
                               const float* __restrict__ S, const int2* __restrict__ tslot_tc,
                               uint4* __restrict__ Tb) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nmt * 128) return;
  const int2 mt = mtiles[i >> 7];
  const int c = (int)((i >> 4) & 7), q = (int)(i & 15);
  const MxPanel P = panels[mt.x];
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int ch = 0; ch < P.nchunkt; ++ch) {
    const float4* a = reinterpret_cast<const float4*>(S + ((P.s0t + (long long)ch * P.nct + mt.y) * 8 + c) * 128 + 8 * q);
    const float4 a0 = a[0], a1 = a[1];
    v[0] += a0.x;
    v[1] += a0.y;
    v[2] += a0.z;
    v[3] += a0.w;
    v[4] += a1.x;
    v[5] += a1.y;
    v[6] += a1.z;
    v[7] += a1.w;
  }
  const int2 e = __ldg(tslot_tc + (P.t0 + mt.y) * 8 + c);
  const bool pad = e.x < 0;
  const long long hp = pad ? -1 - (long long)e.x : e.x;
  uint4 hi, lo;
  split8(v, hi, lo);
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  Tb[tb_word(hp, q)] = pad ? z : hi;
  if (e.y >= 0) Tb[tb_word(e.y, q)] = pad ? z : lo;
}

// ---- phase 2 ------------------------------------------------------------------
// Warp roles as in phase 1.  Stage layout (bytes): kinds 0, 2, 3: A_hi 0 (row
// tile k at 2048 k), A_lo 8192, B_hi 16384, B_lo 24576; kind 1: A_hi 0 (row
// tile k at 4096 k), B_hi 16384 (8 K blocks).  A: column tiles as stored (P1
// order), 512 bytes each, M-major with the 64-byte swizzle: 32 rows of a
// column are 64 contiguous bytes, the row tiles (LBO) and the groups of 8
// columns (512 = SBO) apart; kind 2: dense tiles as stored, K-major with the
// 64-byte swizzle, groups of 8 rows 512 (SBO) apart.  Row i of a tile is
// rho(i / 8, i % 8).  B: T blocks
// MN-major (right-hand side n at 2 (n % 8) + 128 (n / 8), column c at 16 c;
// SBO 128, LBO 2048), X's image K-major (n at 16 (n % 8) + 128 (n / 8); SBO
// 128, LBO 2048).  Row tiles outside a step's mask, the odd last column tile
// of a step and kind 3's operands are copied from the store's zero tiles.
constexpr int kP2Stages = 6;
constexpr int kP2Bufs = 4;       // TMEM accumulators of 128 columns (all 512)
constexpr int kP2Chain = 4;      // steps per MMA chain
constexpr int kP2BarBytes = 8 * (2 * kP2Stages + 2 * kP2Bufs + 1);
constexpr size_t kP2Smem = (size_t)kP2Stages * kTcStage + kP2BarBytes + 16;
constexpr uint32_t kIdescABmn = kIdescBmn | (1u << 15);  // A and B MN-major

__global__ void __launch_bounds__(kTcThreads, 1)
    k_mx_p2_tc(const int* __restrict__ cta_ptr, const int* __restrict__ cta_blocks, int tile0, int tile_end,
               const int* __restrict__ step_ptr, const P2Step* __restrict__ steps, const uint4* __restrict__ store, long long zero_tile,
               const uint4* __restrict__ Tb, const uint4* __restrict__ Xtc, const int* __restrict__ tile_leaf,
               const int* __restrict__ leaf_tile0, const int* __restrict__ leaf_off,
               float* __restrict__ Y, int ldy, int nr, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t full = sbase + (uint32_t)(kP2Stages * kTcStage), empty = full + 8u * kP2Stages;
  const uint32_t ready = empty + 8u * kP2Stages, freeb = ready + 8u * kP2Bufs, done = freeb + 8u * kP2Bufs;
  uint32_t* slot = reinterpret_cast<uint32_t*>(smem + kP2Stages * kTcStage + kP2BarBytes);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  if (tid == 0) {
    for (int i = 0; i < kP2Stages; ++i) {
      mbar_init(full + 8u * i, 1);  // thread 0's expect_tx (bulk copies)
      mbar_init(empty + 8u * i, 1);
    }
    for (int i = 0; i < kP2Bufs; ++i) {
      mbar_init(ready + 8u * i, 1);
      mbar_init(freeb + 8u * i, kDrainWarps);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(slot), 128 * kP2Bufs);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(slot);
  const int b0 = cta_ptr[blockIdx.x], b1 = cta_ptr[blockIdx.x + 1];
  bool failed = false;
  auto give_up = [&]() {
    failed = true;
    *abort_flag = 1;
  };

  if (warp < kCopyWarps) {  // ---- producers: one copy per lane
    // lanes 0-3: A_hi of row tile k; 4-7: A_lo; 8-11, 12-15: their odd last
    // column tiles (zeros); 16, 17: B_hi, B_lo; 18, 19: their odd last blocks
    const uint4* zero = store + zero_tile * 32;
    const int k = lane & 3;
    const bool is_b = lane >= 16, is_pad = is_b ? lane >= 18 : lane >= 8;
    const bool is_lo = is_b ? lane & 1 : (lane >> 2) & 1;
    const uint32_t dst0 = (is_b ? 16384u : 0u) + (is_lo ? 8192u : 0u);
    long long j = 0, last = -1;
    for (int bi = b0; bi < b1 && !failed; ++bi) {
      const int b = cta_blocks[bi], i0 = step_ptr[b], ns = step_ptr[b + 1] - i0;
      P2Step W{};  // this warp's next 32 steps, one per lane
      const int first = (int)((warp - j) & (kCopyWarps - 1));
      for (int q = 0, st = first; st < ns; ++q, st += kCopyWarps) {
        const int at = q & 31;
        if (at == 0 && st + kCopyWarps * lane < ns) W = steps[i0 + st + kCopyWarps * lane];
        const long long a_hi = __shfl_sync(0xffffffffu, W.a_hi, at), a_lo = __shfl_sync(0xffffffffu, W.a_lo, at);
        const long long b_hi = __shfl_sync(0xffffffffu, W.b_hi, at), b_lo = __shfl_sync(0xffffffffu, W.b_lo, at);
        const int s_hi = __shfl_sync(0xffffffffu, W.a_stride, at), s_lo = __shfl_sync(0xffffffffu, W.a_stride_lo, at);
        const int info = __shfl_sync(0xffffffffu, W.info, at);
        const long long js = j + st;
        const int s = (int)(js % kP2Stages);
        const int kind = info & 3, mask = info >> 8;
        const int cnt = kind == 3 ? 2 : (info >> 2) & 15, odd = cnt & 1;
        const bool lo = kind == 0 || kind == 2;
        const uint32_t base = sbase + (uint32_t)(s * kTcStage), bar = full + 8u * s;
        const uint32_t rs = kind == 1 ? 4096u : 2048u;
        const uint32_t ahi = (uint32_t)(512 * cnt), bhi = kind == 2 ? 8192u : (uint32_t)(2048 * cnt);
        const uint32_t whole = is_b ? bhi : ahi;
        const uint32_t dst = dst0 + (is_b ? 0u : (uint32_t)k * rs) + (is_pad ? whole : 0u);
        const uint32_t size = is_pad ? (is_b ? 2048u : 512u) : whole;
        const bool mine = lane < 20 && (lo || !is_lo) && (odd || !is_pad);
        const uint4* src = is_b ? (kind == 2 ? Xtc : Tb) + (is_lo ? b_lo : b_hi)
                                : store + (is_lo ? a_lo + (long long)k * s_lo : a_hi + (long long)k * s_hi) * 32;
        if (is_pad || kind == 3 || (!is_b && !((mask >> k) & 1))) src = zero;
        int ok = 1;
        if (lane == 0) {
          if (js >= kP2Stages &&
              !mbar_wait_or(empty + 8u * s, (uint32_t)(((js - kP2Stages) / kP2Stages) & 1), abort_flag)) {
            give_up();
            ok = 0;
          } else {
            const uint32_t part = 4u * ahi + bhi + (odd ? 4096u : 0u);  // 4 row tiles and B, and the odd zeros
            mbar_arrive_expect_tx(bar, lo ? 2u * part : part);
          }
        }
        if (!__shfl_sync(0xffffffffu, ok, 0)) {
          failed = true;
          break;
        }
        if (mine) bulk_g2s(base + dst, src, size, bar);
        last = js;
      }
      j += ns;
    }
    // The kernel may not end with copies in flight.  The MMAs wait for every
    // step's, but not once any role has given up, which this warp need not have
    // seen: its last copies are waited for here (bounded), whatever happened.
    if (lane == 0)
      for (long long js = last; js >= 0 && js > last - kP2Stages; js -= kCopyWarps)
        mbar_wait(full + 8u * (uint32_t)(js % kP2Stages), (uint32_t)((js / kP2Stages) & 1), kWaitClocks / 8);
    __syncwarp();
  } else if (warp == kMmaWarp) {  // ---- MMA issuer (lane 0; the others hold descriptors)
    const uint64_t adesc0 = tc_sdesc_sw64_mn(sbase, 2048, 512), adesc1 = tc_sdesc_sw64_mn(sbase, 4096, 512);
    const uint64_t adesc2 = tc_sdesc_sw64(sbase, 512);   // dense tiles: groups of 8 rows, row tiles end to end
    const uint64_t bdesc0 = tc_sdesc(sbase, 2048, 128);  // T blocks and X's image: SBO 128, LBO 2048
    long long j = 0;
    int chain = -1;
    for (int bi = b0; bi < b1 && !failed; ++bi) {
      const int b = cta_blocks[bi], e = step_ptr[b + 1];
      int in_chain = 0, w_info = 0;
      for (int i0 = step_ptr[b], i = i0; i < e && !failed; ++i) {
        const int at = (i - i0) & 31;
        if (at == 0 && i + lane < e) w_info = steps[i + lane].info;
        const int info = __shfl_sync(0xffffffffu, w_info, at);
        const int s = (int)(j % kP2Stages);
        if (in_chain == 0) ++chain;
        if (lane == 0) {
          if (in_chain == 0 && chain >= kP2Bufs &&
              !mbar_wait_or(freeb + 8u * (uint32_t)(chain % kP2Bufs), (uint32_t)((chain / kP2Bufs - 1) & 1),
                            abort_flag))
            give_up();
          if (!failed && !mbar_wait_or(full + 8u * s, (uint32_t)((j / kP2Stages) & 1), abort_flag)) give_up();
          if (!failed) {
            tc_fence_after();
            const int kind = info & 3, cnt = (info >> 2) & 15, nq = kind == 3 ? 1 : (cnt + 1) >> 1;
            // this stage's start; an offset of o bytes adds o >> 4 to the start address field
            const uint64_t off = (uint64_t)((s * kTcStage) >> 4);
            const uint64_t da = (kind == 1 ? adesc1 : kind == 2 ? adesc2 : adesc0) + off, db = bdesc0 + off;
            const uint32_t d = tmem + (uint32_t)((chain % kP2Bufs) * 128);
            uint32_t acc = in_chain == 0 ? 0u : 1u;
            // 16 columns at a time: two column tiles (1024 bytes of A) or half a dense tile's rows (32 bytes),
            // two K blocks (4096 bytes of B at 16384).  Dense tiles and X's image are K-major, panels' tiles and T
            // blocks MN-major.
            if (kind == 1) {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (q < nq) tc_mma_bf16(d, da + q * 64, db + (1024 + q * 256), kIdescABmn, q ? 1u : acc);
            } else if (kind == 2) {
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                tc_mma_bf16(d, da + q * 2, db + (1024 + q * 256), kIdesc, q ? 1u : acc);  // D_hi X_hi
                tc_mma_bf16(d, da + q * 2, db + (1536 + q * 256), kIdesc, 1u);          // D_hi X_lo
                tc_mma_bf16(d, da + (512 + q * 2), db + (1024 + q * 256), kIdesc, 1u);  // D_lo X_hi
              }
            } else {
#pragma unroll
              for (int q = 0; q < 2; ++q)
                if (q < nq) {
                  tc_mma_bf16(d, da + q * 64, db + (1024 + q * 256), kIdescABmn, q ? 1u : acc);  // U_hi T_hi
                  if (kind != 3) {
                    tc_mma_bf16(d, da + q * 64, db + (1536 + q * 256), kIdescABmn, 1u);        // U_hi T_lo
                    tc_mma_bf16(d, da + (512 + q * 64), db + (1024 + q * 256), kIdescABmn, 1u);  // U_lo T_hi
                  }
                }
            }
            tc_commit(empty + 8u * s);
          }
        }
        failed = __shfl_sync(0xffffffffu, failed, 0);
        ++j;
        if (i + 1 == e || ++in_chain == kP2Chain) {
          if (lane == 0 && !failed) tc_commit(ready + 8u * (uint32_t)(chain % kP2Bufs));
          in_chain = 0;
        }
      }
    }
    if (lane == 0) tc_commit(done);  // arrives once every MMA issued above is done
  } else {  // ---- drain warps: TMEM lanes 32 (warp % 4) .., a row of the block and kDrainCols columns each
    const int m = (warp & 3) * 32 + lane, h = (warp - kDrainWarp0) >> 2;
    const int in_tile = 8 * ((lane & 7) >> 1) + 2 * (lane >> 3) + (lane & 1);  // rho(lane / 8, lane % 8)
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(h * kDrainCols);
    float acc[kDrainCols];
#pragma unroll
    for (int i = 0; i < kDrainCols; ++i) acc[i] = 0.f;
    int chain = -1;
    for (int bi = b0; bi < b1 && !failed; ++bi) {
      const int b = cta_blocks[bi];
      const int nsteps = step_ptr[b + 1] - step_ptr[b];
      const int nchains = (nsteps + kP2Chain - 1) / kP2Chain;
      const int G = tile0 + 4 * b + (m >> 5);
      int row = -1;
      if (G < tile_end) {
        const int x = tile_leaf[G];
        const int r = leaf_off[x] + 32 * (G - leaf_tile0[x]) + in_tile;
        if (r < leaf_off[x + 1]) row = r;
      }
      for (int c = 0; c < nchains; ++c) {
        ++chain;
        const uint32_t bb = (uint32_t)(chain % kP2Bufs);
        if (!warp_wait_or(ready + 8u * bb, (uint32_t)((chain / kP2Bufs) & 1), abort_flag)) {
          give_up();
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < kDrainCols / 32; ++q) {
          uint32_t v[32];
          tc_ld32(mine + bb * 128u + (uint32_t)(q * 32), v);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[q * 32 + i] += __uint_as_float(v[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(freeb + 8u * bb);
      }
      if (failed) break;
      if (row >= 0) {
        float* y = Y + (size_t)(h * kDrainCols) * ldy + row;
#pragma unroll
        for (int i = 0; i < kDrainCols; ++i, y += ldy)
          if (h * kDrainCols + i < nr) *y = acc[i];
      }
#pragma unroll
      for (int i = 0; i < kDrainCols; ++i) acc[i] = 0.f;
    }
  }
  if (failed) atomicOr(err, 2);
  if (tid == 0 && !mbar_wait(done, 0, 5 * kWaitClocks)) atomicOr(err, 2);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128 * kP2Bufs);
  }
}

}  // namespace

hm_status mixed_tc_pass(hm_hmatrix_s* h, int nr, const uint4* Xtc, float* S, uint4* Tb, float* Y, int ldy,
                        cudaStream_t s, KernelMarks* km) {
  MxPlan& M = h->mx;
  // the kernels' shared-memory limit, once per device of this process
  static std::atomic<unsigned long long> attr_done{0};
  int dev = 0;
  HM_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !((attr_done.load() >> dev) & 1ull)) {
    HM_CUDA(cudaFuncSetAttribute(k_mx_p1_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP1Smem));
    HM_CUDA(cudaFuncSetAttribute(k_mx_p2_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP2Smem));
    if (dev < 64) attr_done |= 1ull << dev;
  }
  const long long xbytes = 4ll * h->n * 128;  // X's image: hi + lo of 128 right-hand sides
  if (M.num_tc_units > 0) {
    k_mx_p1_tc<<<M.tc_ctas, kTcThreads, kP1Smem, s>>>(M.tc_units.p, M.tc_ptr.p, M.store.p, Xtc, M.tslot_tc.p, S, Tb,
                                                M.tc_err.p);
    HM_LAUNCH_CHECK();
    if (km) km->mark("k_mx_p1_tc", M.bytes_p1 + xbytes, s);
  }
  if (M.nmt_tc > 0) {
    k_mx_reduce_tc<<<(unsigned)((M.nmt_tc * 128 + 255) / 256), 256, 0, s>>>(M.mtiles_tc.p, M.nmt_tc, M.panels.p, S,
                                                                            M.tslot_tc.p, Tb);
    HM_LAUNCH_CHECK();
    if (km) km->mark("k_mx_reduce_tc", 4096ll * M.s_tiles_tc + 4096ll * M.nmt_tc, s);
  }
  if (M.p2_blocks > 0) {
    k_mx_p2_tc<<<M.p2_ctas, kTcThreads, kP2Smem, s>>>(M.p2_cta_ptr.p, M.p2_cta_blocks.p, M.p2_tile0,
                                                M.p2_tile0 + M.p2_tiles, M.p2_step_ptr.p, M.p2_steps.p, M.store.p, M.zero_tile, Tb, Xtc, M.tile_leaf.p, M.leaf_tile0.p,
                                                h->tree->offsets.p, Y, ldy, nr, M.tc_err.p);
    HM_LAUNCH_CHECK();
    if (km) km->mark("k_mx_p2_tc", M.bytes_p2 + xbytes + 4ll * h->n * nr, s);
  }
  return HM_OK;
}

}  // namespace hm

extern "C" hm_status hm_hmatrix_check(hm_hmatrix h, void* stream) {
  using namespace hm;
  if (!h) return fail(HM_ERR_INVALID, "hm_hmatrix_check: null matrix");
  HM_CUDA(cudaStreamSynchronize(as_stream(stream)));
  if (!h->mx.tc_err.p) return HM_OK;
  int v = 0;
  HM_CUDA(cudaMemcpy(&v, h->mx.tc_err.p, sizeof v, cudaMemcpyDeviceToHost));
  if (v == 0) return HM_OK;
  HM_CUDA(cudaMemset(h->mx.tc_err.p, 0, sizeof v));
  return fail(HM_ERR_TIMEOUT, std::string("a bounded wait of the tcgen05 ") +
                                  (v == 1 ? "phase-1 kernel" : v == 2 ? "phase-2 kernel" : "kernels of both phases") +
                                  " gave up: products since the last check are wrong");
}
