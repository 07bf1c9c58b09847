// Cascade of direct-form-II biquads of the batched filter bank, forward and
// adjoint, split along time into 1024-sample units that warps filter
// independently, with no wait between CTAs and no CTA barrier.
//
// A unit is one warp; each lane owns 32 consecutive samples as two chunks of 16, A and B, held
// as packed pairs (A_i, B_i): every FP32 operation on samples is a packed one (fma.rn.f32x2,
// each half rounded as fmaf).  The FMA pipe's rate is the same, but a packed instruction takes
// half the issue slots, and one warp scan serves 1024 samples instead of 512.  These passes wait
// on latency: issue slots 30 to 55 % used, the FMA pipe 22 to 52 %, 10 to 43 % of the warps resident.  Per
// stage the chunks are run from a zero state for their end states, a lane's two
// end states combine, the lanes' end states are combined by a warp scan of the affine maps
// s -> M s + e (M = A^16 and its powers, A the stage's 2x2 companion matrix,
// formed in FP64 and rounded once; the unit's entry state joins the first
// lane's end state before the scan), and the chunks run again from their true initial states:
// w[i] = u[i] - a1 w[i-1] - a2 w[i-2], y[i] = b0 w[i] + b1 w[i-1] + b2 w[i-2].  (Correcting the
// first run's sequence by the free response instead, w[i] += alpha_i w1 + beta_i w2, has no
// second serial chain but keeps the sequence in 32 registers a lane and reads 16 more
// table vectors a stage: slower, with 250 registers in the adjoint.)
//
// Units are chained through the whole cascade at once.  With the state of
// all S stages at a unit's start as one 2S-vector z, the state at its end is
// Phi z + e, where e is the end state when every stage starts the unit from
// zero and Phi = A_c^1024, A_c the cascade's 2S x 2S one-step transition (block
// lower-triangular: stage p's output drives stage p + 1).  So:
//   pass 1 (bank_agg_kernel): e of every unit but the channel's last, by filtering it from a
//           zero state.  (As dot products with the impulse responses from the cascade's
//           input to each stage's internal sequence, two multiply-adds a sample and stage
//           instead of seven: 1603 us a step against 1587 on 2048 channels of up to 262144
//           samples, the adjoint 4 % faster on a thousand channels of 20000 samples and 12 to 24
//           stages, the forward up to 17 % slower on channels of 1100 to 6000 samples; and the
//           responses take 8 KB of work buffer a channel and stage, 138 MB instead of 70 for
//           work and scratch of 4096 channels of 1100 samples and 8 stages.)
//   pass 2 (bank_chain_fast_kernel up to 16 stages, bank_chain_kernel beyond):
//           per channel, z_0 = 0, z_{j+1} = Phi z_j + e_j, j over the
//           channel's units (in two levels through Phi^32 over groups of 32
//           units in FP32, or one unit after another in FP64); z_j is stored
//           (2 floats per unit and stage): the checkpoints;
//   pass 3 (bank_unit_kernel): every unit from its checkpoint: y.
// The adjoint is the same cascade run backwards in time with the stages in
// reverse order (v[t] = g[t] - a1 v[t+1] - a2 v[t+2], lambda[t] = b0 v[t] +
// b1 v[t+1] + b2 v[t+2]: g the stage's output gradient, lambda its input
// gradient), chained the same way from the channel's end; its last pass
// (bank_adjoint_kernel) recomputes each unit's forward from the forward
// checkpoints, keeping every stage's internal sequence w_s in shared memory,
// and accumulates the coefficient gradients
//     dL/db_i = sum_t g[t] w[t-i],   dL/da_i = -sum_t lambda[t] w[t-i]
// in FP32 per unit, then in FP64 per channel in a fixed order (bank_sums_kernel):
// bitwise repeatable.
#include <algorithm>

#include <cuda_runtime.h>

#include "dsplib_internal.h"
#include "scan_common.cuh"

namespace dsplib {
namespace {

using scan::M2;
using scan::M2f;
using scan::P2;
using scan::dup;
using scan::fma2;
using scan::mul2;
using scan::pk;
using scan::up;

constexpr int kL = 16;          // samples per chunk
constexpr int kLane = 2 * kL;   // samples per lane: chunks A and B
constexpr int kUnit = 32 * kLane; // samples per unit (warp): 1024
constexpr int kWarps = 4;       // units per CTA
constexpr int kThreads = 32 * kWarps;
constexpr int kRow = kLane + 2; // staging row of a lane's samples, pairs (A_i, B_i) adjacent (conflict-free)
constexpr int kStage = 32 * kRow;
constexpr int kUnitLog2 = 10;   // Phi = A_c^(2^10)
constexpr int kChainFastStages = 16; // cascades the FP32 register chain takes
constexpr int kChainGroup = 32;      // units of one of its groups

static_assert(kUnit == kBankSpan, "unit size");

// Stage table (floats): [0, 5) b0 b1 b2 a1 a2; [8 + 4k, 12 + 4k) P[k] = M^(2^k), M = A^16,
// row-major: a lane's second chunk, its 32 samples, and 2, 4, 8 and 16 lanes.
constexpr int kTabP = 8, kPowers = 6;
static_assert(kTabP + 4 * kPowers <= kBankTabFloats && kBankTabFloats % 4 == 0, "stage table layout");

__device__ __forceinline__ M2f tabP(const float *tb, int k)
{
   const float4 q = *(const float4 *) (tb + kTabP + 4 * k);
   return {q.x, q.y, q.z, q.w};
}

__device__ __forceinline__ float2 shflDown(float2 v, int d)
{
   v.x = __shfl_down_sync(0xffffffffu, v.x, d);
   v.y = __shfl_down_sync(0xffffffffu, v.y, d);
   return v;
}

// ------------------------------------------------------------------ stage tables

__global__ void __launch_bounds__(128) bank_tables_kernel(const float *coefs, int totalStages, float *tables)
{
   const int g = blockIdx.x * blockDim.x + threadIdx.x;
   if (g >= totalStages) return;
   const float *cf = coefs + 5LL * g;
   float *tb = tables + (long long) g * kBankTabFloats;
   for (int k = 0; k < 5; k++) tb[k] = cf[k];
   for (int k = 5; k < kTabP; k++) tb[k] = 0.0f;
   const double a1 = cf[3], a2 = cf[4];
   M2 M = {-a1, -a2, 1.0, 0.0};
   for (int r = 1; r < kL; r <<= 1) M = scan::mmul(M, M);
   for (int k = 0; k < kPowers; k++) {
      const M2f f = scan::toF(M);
      *(float4 *) (tb + kTabP + 4 * k) = make_float4(f.a, f.b, f.c, f.d);
      M = scan::mmul(M, M);
   }
}

// ------------------------------------------------------------------ cascade transitions

// Lower block-triangular 2S x 2S matrix in 2x2 blocks (p, q), q <= p, block index
// p (p + 1) / 2 + q, each block 4 doubles row-major.
__host__ __device__ inline int blk(int p, int q) { return p * (p + 1) / 2 + q; }

// Processing position p -> stage: forward p, adjoint S - 1 - p.
__device__ __forceinline__ int stageAt(int p, int S, bool adj) { return adj ? S - 1 - p : p; }

// Phi = A_c^1024 for one channel and direction, one CTA: A_c in shared memory, ten
// squarings C(p,q) = sum_{m=q..p} B(p,m) B(m,q) between two shared buffers; then, where it is
// used, Phi^32.  Per channel: Phi forward, Phi adjoint, Phi^32 forward, Phi^32 adjoint.
__global__ void __launch_bounds__(128) bank_transition_kernel(const RaggedChan *chans, const float *coefs,
                                                              double *phi)
{
   extern __shared__ double dynT[];
   const RaggedChan c = chans[blockIdx.x];
   const bool adj = blockIdx.y != 0;
   const int S = c.S;
   if (S == 0) return;
   const int nb = S * (S + 1) / 2;
   double *B = dynT, *C = dynT + 4 * nb;
   const float *cf = coefs + c.cOff;
   for (int b = threadIdx.x; b < nb; b += blockDim.x) {
      int p = 0;
      while (blk(p + 1, 0) <= b) p++;
      const int q = b - blk(p, 0);
      const int sp = stageAt(p, S, adj);
      double *o = B + 4 * b;
      if (q == p) {
         o[0] = -(double) cf[5 * sp + 3];
         o[1] = -(double) cf[5 * sp + 4];
         o[2] = 1.0;
         o[3] = 0.0;
      }
      else {
         // stage q's state reaches stage p's input through the direct terms b0 of the stages between
         const int sq = stageAt(q, S, adj);
         const double b0 = cf[5 * sq], b1 = cf[5 * sq + 1], b2 = cf[5 * sq + 2];
         double d0 = b1 - b0 * (double) cf[5 * sq + 3], d1 = b2 - b0 * (double) cf[5 * sq + 4];
         for (int m = q + 1; m < p; m++) {
            const double g = cf[5 * stageAt(m, S, adj)];
            d0 *= g;
            d1 *= g;
         }
         o[0] = d0;
         o[1] = d1;
         o[2] = 0.0;
         o[3] = 0.0;
      }
   }
   __syncthreads();
   for (int it = 0; it < kUnitLog2; it++) {
      for (int b = threadIdx.x; b < nb; b += blockDim.x) {
         int p = 0;
         while (blk(p + 1, 0) <= b) p++;
         const int q = b - blk(p, 0);
         double r0 = 0.0, r1 = 0.0, r2 = 0.0, r3 = 0.0;
         for (int m = q; m <= p; m++) {
            const double *x = B + 4 * blk(p, m), *y = B + 4 * blk(m, q);
            r0 = fma(x[0], y[0], fma(x[1], y[2], r0));
            r1 = fma(x[0], y[1], fma(x[1], y[3], r1));
            r2 = fma(x[2], y[0], fma(x[3], y[2], r2));
            r3 = fma(x[2], y[1], fma(x[3], y[3], r3));
         }
         double *o = C + 4 * b;
         o[0] = r0;
         o[1] = r1;
         o[2] = r2;
         o[3] = r3;
      }
      __syncthreads();
      double *t = B;
      B = C;
      C = t;
   }
   double *dst = phi + c.phiOff + (adj ? 4LL * nb : 0);
   for (int i = threadIdx.x; i < 4 * nb; i += blockDim.x) dst[i] = B[i];
   // five more squarings: Phi^32, the transition over a group of 32 units, where there are two
   // groups and the chain takes them (bank_chain_fast_kernel)
   if (S > kChainFastStages || c.Lu <= kChainGroup * kUnit) return;
   for (int it = 0; it < 5; it++) {
      for (int b = threadIdx.x; b < nb; b += blockDim.x) {
         int p = 0;
         while (blk(p + 1, 0) <= b) p++;
         const int q = b - blk(p, 0);
         double r0 = 0.0, r1 = 0.0, r2 = 0.0, r3 = 0.0;
         for (int m = q; m <= p; m++) {
            const double *x = B + 4 * blk(p, m), *y = B + 4 * blk(m, q);
            r0 = fma(x[0], y[0], fma(x[1], y[2], r0));
            r1 = fma(x[0], y[1], fma(x[1], y[3], r1));
            r2 = fma(x[2], y[0], fma(x[3], y[2], r2));
            r3 = fma(x[2], y[1], fma(x[3], y[3], r3));
         }
         double *o = C + 4 * b;
         o[0] = r0;
         o[1] = r1;
         o[2] = r2;
         o[3] = r3;
      }
      __syncthreads();
      double *t = B;
      B = C;
      C = t;
   }
   dst = phi + c.phiOff + 8LL * nb + (adj ? 4LL * nb : 0);
   for (int i = threadIdx.x; i < 4 * nb; i += blockDim.x) dst[i] = B[i];
}

// Per channel (one warp): z_0 = 0, checkpoint z_j, z_{j+1} = Phi z_j + e_j over the
// channel's units (adjoint: from the last unit back).  z in FP64; cascades of more than
// 16 stages (those of up to 16 take bank_chain_fast_kernel).
__global__ void __launch_bounds__(32) bank_chain_kernel(const RaggedChan *chans, const int *order, const double *phi,
                                                        const float2 *agg, float2 *ckpt, int adj)
{
   extern __shared__ double dynC[];
   const RaggedChan c = chans[order[blockIdx.x]];
   const int S = c.S, lane = threadIdx.x;
   if (S <= kChainFastStages) return; // bank_chain_fast_kernel
   const int nb = S * (S + 1) / 2, n2 = 2 * S;
   double *P = dynC, *z = dynC + 4 * nb;
   const double *src = phi + c.phiOff + (adj ? 4LL * nb : 0);
   for (int i = lane; i < 4 * nb; i += 32) P[i] = src[i];
   for (int r = lane; r < n2; r += 32) z[r] = 0.0;
   __syncwarp();
   const int units = (c.Lu + kUnit - 1) / kUnit;
   for (int k = 0; k < units; k++) {
      const int j = adj ? units - 1 - k : k;
      const long long base = c.ckOff + (long long) j * S;
      for (int p = lane; p < S; p += 32) ckpt[base + p] = make_float2((float) z[2 * p], (float) z[2 * p + 1]);
      if (k + 1 == units) break;
      double nz[4];
      for (int i = 0; i < 4; i++) {
         const int r = lane + 32 * i;
         if (r >= n2) break;
         const int p = r >> 1, row = r & 1;
         const float2 e = agg[base + p];
         double acc0 = row ? e.y : e.x, acc1 = 0.0;
         for (int q = 0; q <= p; q++) {
            const double *x = P + 4 * blk(p, q) + 2 * row;
            acc0 = fma(x[0], z[2 * q], acc0);
            acc1 = fma(x[1], z[2 * q + 1], acc1);
         }
         nz[i] = acc0 + acc1;
      }
      __syncwarp();
      for (int i = 0; i < 4; i++) {
         const int r = lane + 32 * i;
         if (r < n2) z[r] = nz[i];
      }
      __syncwarp();
   }
}

// The same chain for cascades of up to 16 stages (2S <= 32), in FP32 (the transitions
// rounded once from their FP64 products), in two levels so that its depth is about
// 2 x 32 + units / 32 steps instead of one step per unit: each warp of the CTA runs
// groups of 32 units from a zero state (group aggregates), warp 0 chains the groups
// with Phi^32, then every group runs again from its true start and writes the
// checkpoints.  In a step, lane r holds state component r and row r of the
// transition in registers; z is broadcast by shuffles.  Group states sit in shared
// memory for channels of up to 48 groups, in the caller's buffer beyond.
constexpr int kChainWarps = 8;
constexpr int kChainSharedGroups = 48;

// Row r of a transition (lane r's) at rows[r * kRowPad + k], zero beyond n2 and above the
// block diagonal: in shared memory rather than registers, which keeps the kernel's register
// count low enough for four CTAs per SM (the rows are read conflict-free: lane r, column q
// sits in bank (r + q) mod 32).
constexpr int kRowPad = 2 * kChainFastStages + 1;
__device__ __forceinline__ void loadRows(float *rows, const double *P, int n2, int tid, int nthreads)
{
   constexpr int n = 2 * kChainFastStages * kRowPad;
   for (int i0 = tid; i0 < n; i0 += 4 * nthreads) { // four loads in flight per thread
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
         const int i = i0 + u * nthreads, r = i / kRowPad, k = i % kRowPad;
         const int p = r >> 1, q = k >> 1;
         v[u] = (i < n && r < n2 && k < n2 && q <= p) ? (float) P[4 * blk(p, q) + 2 * (r & 1) + (k & 1)] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
         if (i0 + u * nthreads < n) rows[i0 + u * nthreads] = v[u];
   }
}

// z' = row . z + e (lane r: component r), z broadcast from lanes 0 .. n2 - 1.  A zero state stays out of
// the products: the transition of an unstable cascade may exceed FP32 (1024 samples of a pole at 1.09, or
// 32 units of one at 1.003), which is nothing to a signal that has not begun.
__device__ __forceinline__ float chainStep(const float *row, float z, float e, int n2)
{
   if (!__any_sync(0xffffffffu, z != 0.0f)) return e;
   float a0 = e, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
#pragma unroll
   for (int q = 0; q < 2 * kChainFastStages; q += 4) {
      if (q >= n2) break;
      a0 = fmaf(row[q], __shfl_sync(0xffffffffu, z, q), a0);
      a1 = fmaf(row[q + 1], __shfl_sync(0xffffffffu, z, q + 1), a1);
      a2 = fmaf(row[q + 2], __shfl_sync(0xffffffffu, z, q + 2), a2);
      a3 = fmaf(row[q + 3], __shfl_sync(0xffffffffu, z, q + 3), a3);
   }
   return (a0 + a1) + (a2 + a3);
}

__global__ void __launch_bounds__(kChainWarps * 32) bank_chain_fast_kernel(const RaggedChan *chans, const int *order,
                                                                           const double *phi, const float2 *agg,
                                                                           float2 *ckpt, float *groupBuf, int adj)
{
   __shared__ float sE[kChainWarps][kChainGroup * 2 * kChainFastStages]; // a group's aggregates, per warp
   __shared__ float sG[kChainSharedGroups * 2 * kChainFastStages];       // group states
   __shared__ float sRow[2][2 * kChainFastStages * kRowPad];             // Phi and Phi^32
   const RaggedChan c = chans[order[blockIdx.x]];
   const int S = c.S, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   if (S == 0 || S > kChainFastStages) return;
   const int n2 = 2 * S, nb = S * (S + 1) / 2;
   const int units = (c.Lu + kUnit - 1) / kUnit, groups = (units + kChainGroup - 1) / kChainGroup;
   float *G = groups <= kChainSharedGroups ? sG : groupBuf + c.grpOff;
   const float *ag = (const float *) (agg + c.ckOff);
   float *ck = (float *) (ckpt + c.ckOff);
   // unit of step k of group g (processing order), and that group's units in memory order
   auto unitOf = [&](int g, int k) { return adj ? units - 1 - (g * kChainGroup + k) : g * kChainGroup + k; };
   auto stageGroup = [&](int g, int gn) {
      const int j0 = adj ? units - g * kChainGroup - gn : g * kChainGroup;
      const float *src = ag + (long long) j0 * n2;
      const int n = gn * n2;
      __syncwarp();
      for (int q0 = lane; q0 < n; q0 += 4 * 32) { // four loads in flight per lane
         float r[4];
#pragma unroll
         for (int u = 0; u < 4; u++)
            if (q0 + 32 * u < n) r[u] = src[q0 + 32 * u];
#pragma unroll
         for (int u = 0; u < 4; u++)
            if (q0 + 32 * u < n) sE[warp][q0 + 32 * u] = r[u];
      }
      __syncwarp();
      return j0;
   };
   loadRows(sRow[0], phi + c.phiOff + (adj ? 4LL * nb : 0), n2, threadIdx.x, blockDim.x);
   if (groups > 1) loadRows(sRow[1], phi + c.phiOff + 8LL * nb + (adj ? 4LL * nb : 0), n2, threadIdx.x, blockDim.x);
   __syncthreads();
   const float *row = sRow[0] + lane * kRowPad;
   // 1. group aggregates from a zero state (the last group's is not needed)
   for (int g = warp; g + 1 < groups; g += kChainWarps) {
      const int j0 = stageGroup(g, kChainGroup);
      float z = 0.0f;
      for (int k = 0; k < kChainGroup; k++)
         z = chainStep(row, z, lane < n2 ? sE[warp][(unitOf(g, k) - j0) * n2 + lane] : 0.0f, n2);
      if (lane < n2) G[g * n2 + lane] = z;
   }
   __syncthreads();
   // 2. true group starts: Z_0 = 0, Z_{g+1} = Phi^32 Z_g + E_g
   if (warp == 0) {
      const float *rowQ = sRow[1] + lane * kRowPad;
      float Z = 0.0f;
      for (int g = 0; g < groups; g++) {
         const float E = (lane < n2 && g + 1 < groups) ? G[g * n2 + lane] : 0.0f;
         __syncwarp();
         if (lane < n2) G[g * n2 + lane] = Z;
         if (g + 1 < groups) Z = chainStep(rowQ, Z, E, n2);
      }
   }
   __syncthreads();
   // 3. every group from its true start: the checkpoints
   for (int g = warp; g < groups; g += kChainWarps) {
      const int gn = min(kChainGroup, units - g * kChainGroup);
      const int j0 = stageGroup(g, gn);
      float z = lane < n2 ? G[g * n2 + lane] : 0.0f;
      for (int k = 0; k < gn; k++) {
         const int j = unitOf(g, k);
         if (lane < n2) ck[(long long) j * n2 + lane] = z;
         if (k + 1 < gn) z = chainStep(row, z, lane < n2 ? sE[warp][(j - j0) * n2 + lane] : 0.0f, n2);
      }
   }
}

// ------------------------------------------------------------------ unit passes

// A warp's staging area: row l holds lane l's 32 samples, sample i at column
// 2 (i % 16) + i / 16, so that a lane's pair i is one 8-byte access and 32 consecutive
// samples are 32 distinct banks.
__device__ __forceinline__ int stageCol(int i) { return 2 * (i & 15) + (i >> 4); }

__device__ __forceinline__ void stageRead(P2 (&v)[kL], const float *stage, int lane)
{
   __syncwarp();
#pragma unroll
   for (int i = 0; i < kL; i++) v[i].v = *(const unsigned long long *) (stage + lane * kRow + 2 * i);
   __syncwarp();
}

// The unit's samples of a row, zero at t >= n.  fetchUnit issues the coalesced loads (sample
// t0 + lane + 32 j in r[j]); stageUnit turns them into the lane's pairs, so that a kernel can
// put other work between the two.
__device__ __forceinline__ void fetchUnit(float (&r)[kLane], const float *row, int t0, int n, int lane)
{
   const float *p = row + t0 + lane;
   if (t0 + kUnit <= n) {
#pragma unroll
      for (int j = 0; j < kLane; j++) r[j] = p[32 * j];
   }
   else {
#pragma unroll
      for (int j = 0; j < kLane; j++) r[j] = t0 + lane + 32 * j < n ? p[32 * j] : 0.0f;
   }
}
__device__ __forceinline__ void stageUnit(P2 (&v)[kL], const float (&r)[kLane], float *stage, int lane)
{
   const int col = stageCol(lane);
#pragma unroll
   for (int j = 0; j < kLane; j++) stage[j * kRow + col] = r[j];
   stageRead(v, stage, lane);
}
// The same of a 16-byte-aligned row allocated to a multiple of 16 floats (the FIR output
// plane): 16-byte loads, samples 4 (lane + 32 j) .. + 3 in r[j].
__device__ __forceinline__ void fetchPlane(float4 (&r)[kL / 2], const float *row, int t0, int n, int lane)
{
   const int np = (n + 15) & ~15;
#pragma unroll
   for (int j = 0; j < kL / 2; j++) {
      const int t = t0 + 4 * (lane + 32 * j);
      r[j] = t < np ? *(const float4 *) (row + t) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (t0 + kUnit > n) {
         if (t + 0 >= n) r[j].x = 0.0f;
         if (t + 1 >= n) r[j].y = 0.0f;
         if (t + 2 >= n) r[j].z = 0.0f;
         if (t + 3 >= n) r[j].w = 0.0f;
      }
   }
}
__device__ __forceinline__ void stagePlane(P2 (&v)[kL], const float4 (&r)[kL / 2], float *stage, int lane)
{
   const int i = 4 * (lane & 7); // sample within its lane's row lane / 8 + 4 j
   float *d = stage + (lane >> 3) * kRow + stageCol(i);
#pragma unroll
   for (int j = 0; j < kL / 2; j++) {
      d[4 * j * kRow + 0] = r[j].x;
      d[4 * j * kRow + 2] = r[j].y;
      d[4 * j * kRow + 4] = r[j].z;
      d[4 * j * kRow + 6] = r[j].w;
   }
   stageRead(v, stage, lane);
}

__device__ __forceinline__ void storeUnit(const P2 (&v)[kL], float *row, int t0, int n, float *stage, int lane)
{
#pragma unroll
   for (int i = 0; i < kL; i++) *(unsigned long long *) (stage + lane * kRow + 2 * i) = v[i].v;
   __syncwarp();
   const float *s = stage + stageCol(lane);
   float *p = row + t0 + lane;
   if (t0 + kUnit <= n) {
#pragma unroll
      for (int j = 0; j < kLane; j++) p[32 * j] = s[j * kRow];
   }
   else {
#pragma unroll
      for (int j = 0; j < kLane; j++)
         if (t0 + lane + 32 * j < n) p[32 * j] = s[j * kRow];
   }
   __syncwarp();
}

// Coefficients of a stage as packed operands.
struct StageCoef {
   P2 b0, b1, b2, na1, na2;
};
__device__ __forceinline__ StageCoef stageCoef(const float *tb)
{
   const float4 q = *(const float4 *) tb;
   return {dup(q.x), dup(q.y), dup(q.z), dup(-q.w), dup(-tb[4])};
}

// End states of both chunks from a zero state: (w[15], w[14]).
__device__ __forceinline__ void zeroStateEnd(const P2 (&v)[kL], const StageCoef &c, P2 &w15, P2 &w14)
{
   P2 p1 = dup(0.0f), p2 = p1;
#pragma unroll
   for (int i = 0; i < kL; i++) {
      const P2 w = fma2(c.na1, p1, fma2(c.na2, p2, v[i]));
      p2 = p1;
      p1 = w;
   }
   w15 = p1;
   w14 = p2;
}

// The same in reverse time, v[i] = g[i] - a1 v[i+1] - a2 v[i+2]: (v[0], v[1]).
__device__ __forceinline__ void zeroStateEndRev(const P2 (&g)[kL], const StageCoef &c, P2 &v0, P2 &v1)
{
   P2 p1 = dup(0.0f), p2 = p1;
#pragma unroll
   for (int i = kL - 1; i >= 0; i--) {
      const P2 v = fma2(c.na1, p1, fma2(c.na2, p2, g[i]));
      p2 = p1;
      p1 = v;
   }
   v0 = p1;
   v1 = p2;
}

// Initial states (w1, w2) of this lane's chunks, packed, from the zero-state end states.  Forward
// time: the lane's end state is M e_A + e_B; the first lane's takes the unit's entry before
// the scan over the lanes (maps of 32 samples: powers of M^2 = P[1]), which then carries it on.
// Returns the state at the lane's end.
__device__ __forceinline__ float2 chunkStateUp(P2 e1, P2 e2, float2 entry, const float *tb, int lane, P2 &w1, P2 &w2)
{
   const float2 x = up(e1), y = up(e2);
   const float2 eA = make_float2(x.x, y.x), eB = make_float2(x.y, y.y);
   const M2f M = tabP(tb, 0);
   float2 val = scan::affine(M, eA, eB);
   if (lane == 0) val = scan::affine(tabP(tb, 1), entry, val);
#pragma unroll
   for (int k = 0; k < 5; k++) {
      const float2 o = scan::shflUp(val, 1 << k, 32);
      if (lane >= (1 << k)) val = scan::affine(tabP(tb, k + 1), o, val);
   }
   float2 a = scan::shflUp(val, 1, 32);
   if (lane == 0) a = entry;
   const float2 b = scan::affine(M, a, eA);
   w1 = pk(a.x, b.x);
   w2 = pk(a.y, b.y);
   return val;
}

// Reverse time: chunk B comes before A, lane 31 first.
__device__ __forceinline__ float2 chunkStateDown(P2 e1, P2 e2, float2 entry, const float *tb, int lane, P2 &v1, P2 &v2)
{
   const float2 x = up(e1), y = up(e2);
   const float2 eA = make_float2(x.x, y.x), eB = make_float2(x.y, y.y);
   const M2f M = tabP(tb, 0);
   float2 val = scan::affine(M, eB, eA);
   if (lane == 31) val = scan::affine(tabP(tb, 1), entry, val);
#pragma unroll
   for (int k = 0; k < 5; k++) {
      const float2 o = shflDown(val, 1 << k);
      if (lane + (1 << k) < 32) val = scan::affine(tabP(tb, k + 1), o, val);
   }
   float2 b = shflDown(val, 1);
   if (lane == 31) b = entry;
   const float2 a = scan::affine(M, b, eB);
   v1 = pk(a.x, b.x);
   v2 = pk(a.y, b.y);
   return val;
}

// One stage of the forward cascade over a unit, in place; keep(i, w) takes its internal sequence.
template <typename Keep>
__device__ __forceinline__ void forwardStage(P2 (&v)[kL], float2 entry, const float *tb, int lane, Keep keep)
{
   const StageCoef c = stageCoef(tb);
   P2 q1, q2;
   zeroStateEnd(v, c, q1, q2);
   chunkStateUp(q1, q2, entry, tb, lane, q1, q2);
#pragma unroll
   for (int i = 0; i < kL; i++) {
      const P2 w = fma2(c.na1, q1, fma2(c.na2, q2, v[i]));
      v[i] = fma2(c.b0, w, fma2(c.b1, q1, mul2(c.b2, q2)));
      keep(i, w);
      q2 = q1;
      q1 = w;
   }
}

// A unit's per-stage states, read once: lane l holds stage l in lo and stage l + 32 in hi
// (up to 64 stages); entryAt broadcasts stage p.
struct UnitStates {
   float2 lo, hi;
};
__device__ __forceinline__ UnitStates loadStates(const float2 *src, int S, int lane)
{
   UnitStates u;
   u.lo = lane < S ? src[lane] : make_float2(0.0f, 0.0f);
   u.hi = lane + 32 < S ? src[lane + 32] : make_float2(0.0f, 0.0f);
   return u;
}
__device__ __forceinline__ float2 entryAt(const UnitStates &u, int p)
{
   return scan::shflIdx(p < 32 ? u.lo : u.hi, p & 31);
}

struct UnitArgs {
   const RaggedChan *chans;
   const int2 *units; // (channel, unit index within the channel)
   int nUnits;
   int Smax;
   const float *tables;
   const float *in;   // forward: FIR output plane; adjoint aggregates: output gradient (packed)
   float *out;        // y (packed, tail zeros)
   float2 *agg;       // unit aggregates, 2 floats per stage (processing order)
   const float2 *ckpt;
   // with the loss: gradient gy = scale (y - target) on the valid samples, the unit's
   // sum of (y - target)^2 in lossPart[unit], and the adjoint's unit aggregates in aggA
   const float *target;
   float *gy;
   double *lossPart;
   float2 *aggA;
   float scale;
};

// Copy the channel's stage tables into the warp's slice of shared memory, four loads
// per lane in flight before their stores.
__device__ __forceinline__ void loadTables(float *dst, const float *tables, const RaggedChan &c, int lane)
{
   const float4 *src = (const float4 *) (tables + (c.cOff / 5) * kBankTabFloats);
   const int n4 = c.S * (kBankTabFloats / 4);
   for (int i0 = lane; i0 < n4; i0 += 4 * 32) {
      float4 r[4];
#pragma unroll
      for (int j = 0; j < 4; j++)
         if (i0 + 32 * j < n4) r[j] = src[i0 + 32 * j];
#pragma unroll
      for (int j = 0; j < 4; j++)
         if (i0 + 32 * j < n4) ((float4 *) dst)[i0 + 32 * j] = r[j];
   }
   __syncwarp();
}

// Aggregates of a unit (held by the warp, overwritten): its stages' end states from a zero state,
// as the scans over the lanes give them; the last stage is not run again for its output.
template <bool ADJ>
__device__ __forceinline__ void unitAggregates(P2 (&v)[kL], const float *sTab, int S, float2 *agg, int lane)
{
   const float2 zero = make_float2(0.0f, 0.0f);
   for (int p = 0; p < S; p++) {
      const float *tb = sTab + stageAt(p, S, ADJ) * kBankTabFloats;
      const StageCoef c = stageCoef(tb);
      P2 q1, q2;
      if (ADJ) zeroStateEndRev(v, c, q1, q2);
      else zeroStateEnd(v, c, q1, q2);
      const float2 end = ADJ ? chunkStateDown(q1, q2, zero, tb, lane, q1, q2) : chunkStateUp(q1, q2, zero, tb, lane, q1, q2);
      if (lane == (ADJ ? 0 : 31)) agg[p] = end;
      if (p + 1 == S) break;
#pragma unroll
      for (int k = 0; k < kL; k++) {
         const int i = ADJ ? kL - 1 - k : k;
         const P2 w = fma2(c.na1, q1, fma2(c.na2, q2, v[i]));
         v[i] = fma2(c.b0, w, fma2(c.b1, q1, mul2(c.b2, q2)));
         q2 = q1;
         q1 = w;
      }
   }
}

// Pass 1.  ADJ = false: every unit of the FIR output plane but its channel's last (whose end
// no unit starts from); ADJ = true: every unit of the packed output gradient but the first.
template <bool ADJ> __global__ void __launch_bounds__(kThreads) bank_agg_kernel(UnitArgs a)
{
   extern __shared__ float4 dynG[];
   __shared__ __align__(16) float sStage[kWarps][kStage];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int ui = blockIdx.x * kWarps + warp;
   if (ui >= a.nUnits) return;
   float *sTab = (float *) dynG + (size_t) warp * a.Smax * kBankTabFloats;
   const int2 U = a.units[ui];
   const RaggedChan c = a.chans[U.x];
   const int t0 = U.y * kUnit;
   if (c.S == 0 || (ADJ ? U.y == 0 : t0 + kUnit >= c.Lu)) return;
   P2 v[kL];
   if (ADJ) {
      float r[kLane];
      fetchUnit(r, a.in + c.xOff, t0, c.Lu, lane);
      loadTables(sTab, a.tables, c, lane);
      stageUnit(v, r, sStage[warp], lane);
   }
   else {
      float4 r[kL / 2];
      fetchPlane(r, a.in + c.pOff, t0, c.Lu, lane);
      loadTables(sTab, a.tables, c, lane);
      stagePlane(v, r, sStage[warp], lane);
   }
   unitAggregates<ADJ>(v, sTab, c.S, a.agg + c.ckOff + (long long) U.y * c.S, lane);
}

// Pass 3: y from the checkpoints; with MSE also the loss gradient, the unit's sum of squares
// and the adjoint's aggregates.
template <bool MSE>
__global__ void __launch_bounds__(kThreads) bank_unit_kernel(UnitArgs a)
{
   extern __shared__ float4 dynU[];
   __shared__ __align__(16) float sStage[kWarps][kStage];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int ui = blockIdx.x * kWarps + warp;
   if (ui >= a.nUnits) return;
   float *sTab = (float *) dynU + (size_t) warp * a.Smax * kBankTabFloats;
   const int2 U = a.units[ui];
   const RaggedChan c = a.chans[U.x];
   const int S = c.S, Lu = c.Lu, t0 = U.y * kUnit;
   const long long base = c.ckOff + (long long) U.y * S;
   // the unit's entry states and input are requested before the tables' copy waits on its own loads
   const UnitStates ent = loadStates(a.ckpt + base, S, lane);
   P2 v[kL];
   {
      float4 r[kL / 2];
      fetchPlane(r, a.in + c.pOff, t0, Lu, lane);
      loadTables(sTab, a.tables, c, lane);
      stagePlane(v, r, sStage[warp], lane);
   }
   for (int p = 0; p < S; p++) forwardStage(v, entryAt(ent, p), sTab + p * kBankTabFloats, lane, [](int, P2) {});
   storeUnit(v, a.out + c.xOff, t0, Lu, sStage[warp], lane);
   if (t0 + kUnit >= Lu)
      for (int t = Lu + lane; t < c.L; t += 32) a.out[c.xOff + t] = 0.0f;
   if (MSE) {
      // the target is read here, not with the unit's other loads: held across the stages it
      // costs 32 registers a thread and the occupancy they buy, and copied to a second staging
      // area meanwhile (cp.async) the step took 1820 us instead of 1804
      P2 tg[kL];
      {
         float r[kLane];
         fetchUnit(r, a.target + c.xOff, t0, Lu, lane);
         stageUnit(tg, r, sStage[warp], lane);
      }
      double sq = 0.0;
#pragma unroll
      for (int i = 0; i < kL; i++) {
         const float2 y = up(v[i]), t = up(tg[i]);
         const int ta = t0 + lane * kLane + i;
         const float da = y.x - t.x, db = y.y - t.y;
         const bool va = ta < Lu, vb = ta + kL < Lu;
         v[i] = pk(va ? a.scale * da : 0.0f, vb ? a.scale * db : 0.0f);
         if (va) sq += (double) da * da;
         if (vb) sq += (double) db * db;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (lane == 0) a.lossPart[ui] = sq;
      storeUnit(v, a.gy + c.xOff, t0, Lu, sStage[warp], lane);
      if (t0 + kUnit >= Lu)
         for (int t = Lu + lane; t < c.L; t += 32) a.gy[c.xOff + t] = 0.0f;
      if (U.y > 0) unitAggregates<true>(v, sTab, S, a.aggA + base, lane);
   }
}

struct AdjArgs {
   const RaggedChan *chans;
   const int2 *units;
   int nUnits;
   int Smax;
   const float *tables;
   const float *u;       // FIR output plane
   const float *gy;      // output gradient (packed)
   const float2 *ckptF;  // forward checkpoints
   const float2 *ckptA;  // adjoint checkpoints (processing order)
   float *g;             // gradient w.r.t. the FIR output (the scratch's plane)
   float *part;          // 5 coefficient-gradient sums per unit and stage
   int first;            // this launch's first unit (a bucket of one stage count)
   int group;            // stages kept at once (adjointGroup)
};

// Stages whose sequences a unit keeps in shared memory at once; deeper cascades are taken in
// groups of stages, last group first, the forward run again up to each: a unit of eight
// stages runs twelve forward stages instead of eight but takes 17 KB instead of 34, and the
// SM holds twelve warps instead of six (2048-channel bank step 1856 -> 1804 us; groups of
// three 1803, five 1817, six 1844).  Deeper ones (us of the backward by group): 1000 channels of
// 20000, 16 stages 4: 786, 8: 812, 16: 1070; 24 stages 4: 1295, 8: 1243, 24: 2060.  Where all units of the
// plan are resident at once anyway, they keep as many stages as leaves them so: nothing is gained from
// more warps there (64 channels of 1100, 64 stages 4: 264, 11: 167, 48: 125).
constexpr int kAdjStages = 4;
constexpr int kAdjWarps = 16;                    // a warp takes 128 registers a thread
constexpr size_t kSmemSm = 228 * 1024, kSmemCta = 227 * 1024; // shared memory of an SM, and of one CTA

// Dynamic shared memory by the deepest cascade of a plan.  The kernels' limits are set for the deepest
// that any plan has, always the same: calls on several threads do not lower each other's.
static size_t transitionShared(int S) { return (size_t) 8 * S * (S + 1) / 2 * sizeof(double); }
static size_t chainShared(int S) { return (size_t) (4 * S * (S + 1) / 2 + 2 * S) * sizeof(double); }
static size_t unitShared(int S) { return (size_t) kWarps * S * kBankTabFloats * sizeof(float); }
static size_t adjointShared(int S, int group)
{
   const size_t seq = (size_t) group * kL * 32 * 2, stage = kStage;
   return ((size_t) S * kBankTabFloats + (seq > stage ? seq : stage)) * sizeof(float);
}
static int adjointGroup(int S, int nUnits)
{
   const int sms = deviceSms() > 0 ? deviceSms() : 148, each = (nUnits + sms - 1) / sms; // units an SM
   int group = S < kAdjStages ? S : kAdjStages;
   while (each <= kAdjWarps && group < S && adjointShared(S, group + 1) <= kSmemCta &&
          each * (adjointShared(S, group + 1) + 1024) <= kSmemSm)
      group++;
   return group;
}

// Stage sequences of one unit in shared memory: per stage of a group 16 rows of 32 pairs, so that
// the lanes of the warp touch distinct banks.  One warp per CTA: the sequences are the bulk of the CTA's
// shared memory, and single-warp CTAs pack the SM most tightly.
__global__ void __launch_bounds__(32) bank_adjoint_kernel(AdjArgs a)
{
   extern __shared__ float4 dynA[];
   const int lane = threadIdx.x;
   float *sTab = (float *) dynA;
   const int2 U = a.units[a.first + blockIdx.x];
   const RaggedChan c = a.chans[U.x];
   unsigned long long *W = (unsigned long long *) (sTab + (size_t) c.S * kBankTabFloats); // sized for c.S stages
   // The staging rows of the loads and stores share the stage sequences' space: the inputs are
   // read before the sequences are written, the input gradient stored after the last of them
   // was read (at least 32 x 34 floats: adjointShared).
   float *sStage = (float *) W;
   const int S = c.S, Lu = c.Lu, t0 = U.y * kUnit;
   const long long base = c.ckOff + (long long) U.y * S;
   const UnitStates entF = loadStates(a.ckptF + base, S, lane), entA = loadStates(a.ckptA + base, S, lane);
   P2 v[kL], g[kL];
   {
      float4 r[kL / 2];
      float q[kLane];
      fetchPlane(r, a.u + c.pOff, t0, Lu, lane);
      fetchUnit(q, a.gy + c.xOff, t0, Lu, lane);
      loadTables(sTab, a.tables, c, lane);
      stageUnit(g, q, sStage, lane);
      stagePlane(v, r, sStage, lane);
   }
   for (int s1 = S; s1 > 0;) {
      const int s0 = max(0, s1 - a.group);
      if (s1 < S) { // a further group: the unit's input again
         float4 r[kL / 2];
         __syncwarp();
         fetchPlane(r, a.u + c.pOff, t0, Lu, lane);
         stagePlane(v, r, sStage, lane);
      }
      // 1. the forward of this unit from its checkpoints; the group's sequences kept
      for (int s = 0; s < s1; s++) {
         const float *tb = sTab + s * kBankTabFloats;
         if (s >= s0) {
            unsigned long long *Ws = W + (s - s0) * kL * 32 + lane;
            forwardStage(v, entryAt(entF, s), tb, lane, [&](int i, P2 q) { Ws[i * 32] = q.v; });
         }
         else forwardStage(v, entryAt(entF, s), tb, lane, [](int, P2) {});
      }
      // 2. the stages' adjoints, last stage first, in reverse time
      for (int s = s1 - 1; s >= s0; s--) {
         const float *tb = sTab + s * kBankTabFloats;
         const StageCoef cf = stageCoef(tb);
         const unsigned long long *Ws = W + (s - s0) * kL * 32 + lane;
         P2 n1, n2;
         zeroStateEndRev(g, cf, n1, n2);
         chunkStateDown(n1, n2, entryAt(entA, S - 1 - s), tb, lane, n1, n2);
         // forward sequence of this stage: before chunk A the previous lane's chunk B (lane 0:
         // the unit's checkpoint state), before chunk B chunk A
         P2 w0 = P2{Ws[(kL - 1) * 32]}, w1 = P2{Ws[(kL - 2) * 32]}, m1, m2; // w[i], w[i-1]; w[-1], w[-2]
         {
            const float2 l1 = up(w0), l2 = up(w1), e = entryAt(entF, s);
            const float p1 = __shfl_up_sync(0xffffffffu, l1.y, 1), p2 = __shfl_up_sync(0xffffffffu, l2.y, 1);
            m1 = pk(lane == 0 ? e.x : p1, l1.x);
            m2 = pk(lane == 0 ? e.y : p2, l2.x);
         }
         P2 pp[5];
#pragma unroll
         for (int k = 0; k < 5; k++) pp[k] = dup(0.0f);
#pragma unroll
         for (int i = kL - 1; i >= 0; i--) {
            const P2 w2 = i >= 2 ? P2{Ws[(i - 2) * 32]} : (i == 1 ? m1 : m2);
            const P2 vt = fma2(cf.na1, n1, fma2(cf.na2, n2, g[i]));
            const P2 lam = fma2(cf.b0, vt, fma2(cf.b1, n1, mul2(cf.b2, n2)));
            pp[0] = fma2(g[i], w0, pp[0]);
            pp[1] = fma2(g[i], w1, pp[1]);
            pp[2] = fma2(g[i], w2, pp[2]);
            pp[3] = fma2(lam, w1, pp[3]);
            pp[4] = fma2(lam, w2, pp[4]);
            g[i] = lam;
            n2 = n1;
            n1 = vt;
            w0 = w1;
            w1 = w2;
         }
         float pr[5];
#pragma unroll
         for (int k = 0; k < 5; k++) {
            const float2 h = up(pp[k]);
            pr[k] = k < 3 ? h.x + h.y : -(h.x + h.y);
         }
         // the five sums over the warp by halving: at each step a lane keeps half of its
         // values and adds the partner's copy of them; lane 4 k ends with sum k (9 shuffles)
         const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
         float q[4], q2[2];
#pragma unroll
         for (int j = 0; j < 4; j++) {
            const float lo = pr[j], hi = j == 0 ? pr[4] : 0.0f;
            q[j] = (b4 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b4 ? lo : hi, 16);
         }
#pragma unroll
         for (int j = 0; j < 2; j++)
            q2[j] = (b3 ? q[j + 2] : q[j]) + __shfl_xor_sync(0xffffffffu, b3 ? q[j] : q[j + 2], 8);
         float r = (b2 ? q2[1] : q2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? q2[0] : q2[1], 4);
         r += __shfl_xor_sync(0xffffffffu, r, 2);
         r += __shfl_xor_sync(0xffffffffu, r, 1);
         const int k = lane >> 2;
         if ((lane & 3) == 0 && k < 5) a.part[(base + s) * 5 + k] = r;
      }
      s1 = s0;
   }
   __syncwarp(); // every lane's last read of the stage sequences precedes the staging writes
   storeUnit(g, a.g + c.gOff, t0, Lu, sStage, lane);
}

// Coefficient gradients of one channel (one CTA): its threads in groups of one thread a coefficient,
// group g adds the partial sums of units g, g + G, ... in FP64, four loads in flight, so that the CTA
// reads consecutive rows whole; then the groups' sums are added in order (bitwise repeatable).  Bound by
// the latency of the longest channel's loads (lanes along the units, 160 bytes apart for 8 stages, took
// 23 us on 16 channels of up to 900 thousand samples, now 12.7; 256 of up to 262144 13.0, now 8.0).
constexpr int kSumThreads = 512;
__device__ __forceinline__ void coefSums(const RaggedChan &c, const float *part, float *gcoefs)
{
   __shared__ double sums[kSumThreads];
   const int n = 5 * c.S, units = (c.Lu + kUnit - 1) / kUnit;
   if (n == 0) return;
   const int G = blockDim.x / n, g = threadIdx.x / n; // launchBankSums: a thread a coefficient at least
   const float *p = part + c.ckOff * 5 + threadIdx.x; // unit g's row
   const long long st = (long long) G * n;
   if (g < G) {
      double acc = 0.0;
      int j = g;
      for (; j + 3 * G < units; j += 4 * G, p += 4 * st) {
         const float v0 = p[0], v1 = p[st], v2 = p[2 * st], v3 = p[3 * st];
         acc += (double) v0;
         acc += (double) v1;
         acc += (double) v2;
         acc += (double) v3;
      }
      for (; j < units; j += G, p += st) acc += (double) *p;
      sums[threadIdx.x] = acc;
   }
   __syncthreads();
   if (threadIdx.x < n) {
      double acc = 0.0;
      for (int k = 0; k < G; k++) acc += sums[k * n + threadIdx.x];
      gcoefs[c.cOff + threadIdx.x] = (float) acc;
   }
}

// Taps gradients of one channel: its runs' sums (512 a run, runs in time order) added in that order in
// FP64, gtaps[T - 1 - c] = sum_run part[run][c].
__device__ __forceinline__ void tapSums(const RaggedChan &c, int run0, int run1, const float *part, float *gtaps)
{
   for (int k = threadIdx.x; k < c.T; k += blockDim.x) {
      double s = 0.0;
      for (int i = run0; i < run1; i++) s += part[(long long) i * kFirBfMaxTaps + k];
      gtaps[c.hOff + c.T - 1 - k] = (float) s;
   }
}

// Both, the last of the adjoint, in one launch.
__global__ void __launch_bounds__(kSumThreads) bank_sums_kernel(const RaggedChan *chans, const float *part, float *gcoefs,
                                                                const int *dhStart, const float *dhPart, float *gtaps)
{
   const RaggedChan c = chans[blockIdx.x];
   if (blockIdx.y == 0) coefSums(c, part, gcoefs);
   else tapSums(c, dhStart[blockIdx.x], dhStart[blockIdx.x + 1], dhPart, gtaps);
}

} // namespace

long long bankTransitionDoubles(int S) { return 8LL * S * (S + 1); } // Phi and Phi^32, both directions

cudaError_t launchBankTables(const BankLaunch &b, const float *coefs, int totalStages, float *tables, double *phi,
                             cudaStream_t s)
{
   if (totalStages <= 0) return cudaSuccess;
   bank_tables_kernel<<<(totalStages + 127) / 128, 128, 0, s>>>(coefs, totalStages, tables);
   cudaError_t e = cudaFuncSetAttribute(bank_transition_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int) transitionShared(kRaggedMaxStages));
   if (e != cudaSuccess) return e;
   // one warp per (channel, direction) while the block count is small (up to 36 blocks of
   // 2 x 2 for 8 stages): the squarings' barriers then cost a warp, not four
   bank_transition_kernel<<<dim3(b.C, 2), b.Smax <= 8 ? 32 : 128, transitionShared(b.Smax), s>>>(b.chans, coefs, phi);
   countLaunch(2);
   return cudaGetLastError();
}

template <bool MSE> static cudaError_t launchUnits(const UnitArgs &a, cudaStream_t s)
{
   cudaError_t e = cudaFuncSetAttribute(bank_unit_kernel<MSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int) unitShared(kRaggedMaxStages));
   if (e != cudaSuccess) return e;
   bank_unit_kernel<MSE><<<(a.nUnits + kWarps - 1) / kWarps, kThreads, unitShared(a.Smax), s>>>(a);
   countLaunch();
   return cudaGetLastError();
}

// Aggregates of every unit that another starts from; none where every channel is one unit.
template <bool ADJ> static cudaError_t launchAggregates(const BankLaunch &b, const UnitArgs &a, cudaStream_t s)
{
   if (b.nUnits == b.C) return cudaSuccess;
   cudaError_t e = cudaFuncSetAttribute(bank_agg_kernel<ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int) unitShared(kRaggedMaxStages));
   if (e != cudaSuccess) return e;
   bank_agg_kernel<ADJ><<<(a.nUnits + kWarps - 1) / kWarps, kThreads, unitShared(a.Smax), s>>>(a);
   countLaunch();
   return cudaGetLastError();
}

cudaError_t launchBankForward(const BankLaunch &b, cudaStream_t s)
{
   if (b.nUnits <= 0) return cudaSuccess;
   UnitArgs a{b.chans, b.units, b.nUnits, b.Smax, b.tables, b.u, nullptr, b.aggF, nullptr};
   cudaError_t e = launchAggregates<false>(b, a, s);
   if (e != cudaSuccess) return e;
   bank_chain_fast_kernel<<<b.C, kChainWarps * 32, 0, s>>>(b.chans, b.chainOrder, b.phi, b.aggF, b.ckptF, b.groupF, 0);
   countLaunch();
   if (b.Smax > kChainFastStages) {
      if ((e = cudaFuncSetAttribute(bank_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int) chainShared(kRaggedMaxStages))) != cudaSuccess)
         return e;
      bank_chain_kernel<<<b.C, 32, chainShared(b.Smax), s>>>(b.chans, b.chainOrder, b.phi, b.aggF, b.ckptF, 0);
      countLaunch();
   }
   a.out = b.y;
   a.ckpt = b.ckptF;
   if (b.target) {
      a.target = b.target;
      a.gy = b.gyOut;
      a.lossPart = b.lossPart;
      a.aggA = b.aggA;
      a.scale = b.scale;
      return launchUnits<true>(a, s);
   }
   return launchUnits<false>(a, s);
}

cudaError_t launchBankBackward(const BankLaunch &b, cudaStream_t s)
{
   if (b.nUnits <= 0) return cudaSuccess;
   cudaError_t e = cudaSuccess;
   if (!b.aggReady) {
      UnitArgs a{b.chans, b.units, b.nUnits, b.Smax, b.tables, b.gy, nullptr, b.aggA, nullptr};
      if ((e = launchAggregates<true>(b, a, s)) != cudaSuccess) return e;
   }
   bank_chain_fast_kernel<<<b.C, kChainWarps * 32, 0, s>>>(b.chans, b.chainOrder, b.phi, b.aggA, b.ckptA, b.groupA, 1);
   countLaunch();
   if (b.Smax > kChainFastStages) {
      if ((e = cudaFuncSetAttribute(bank_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int) chainShared(kRaggedMaxStages))) != cudaSuccess)
         return e;
      bank_chain_kernel<<<b.C, 32, chainShared(b.Smax), s>>>(b.chans, b.chainOrder, b.phi, b.aggA, b.ckptA, 1);
      countLaunch();
   }
   if ((e = cudaFuncSetAttribute(bank_adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kSmemCta)) !=
       cudaSuccess)
      return e;
   AdjArgs d{b.chans, b.units, b.nUnits, b.Smax, b.tables, b.u, b.gy, b.ckptF, b.ckptA, b.g, b.part, 0, 0};
   // One launch per stage count, each with the shared memory its cascades need, spread over
   // the caller's stream and the auxiliary ones so that CTAs of different buckets share the
   // SMs (and no launch waits for another's tail).
   const int lanes = 1 + b.nAux;
   if (b.nAux > 0) {
      if ((e = cudaEventRecord(b.fork, s)) != cudaSuccess) return e;
      for (int i = 0; i < b.nAux; i++)
         if ((e = cudaStreamWaitEvent(b.aux[i], b.fork, 0)) != cudaSuccess) return e;
   }
   for (int k = 0; k < b.nBuckets; k++) {
      d.first = b.bucketStart[k];
      const int n = b.bucketStart[k + 1] - b.bucketStart[k];
      if (n <= 0) continue;
      const cudaStream_t st = (k % lanes) == 0 ? s : b.aux[(k % lanes) - 1];
      d.group = adjointGroup(b.bucketS[k], b.nUnits);
      bank_adjoint_kernel<<<n, 32, adjointShared(b.bucketS[k], d.group), st>>>(d);
      countLaunch();
   }
   for (int i = 0; i < b.nAux; i++) {
      if ((e = cudaEventRecord(b.join[i], b.aux[i])) != cudaSuccess) return e;
      if ((e = cudaStreamWaitEvent(s, b.join[i], 0)) != cudaSuccess) return e;
   }
   return cudaGetLastError();
}

cudaError_t launchBankSums(const BankLaunch &b, const int *dhStart, const float *dhPart, float *gtaps, cudaStream_t s)
{
   static_assert(5 * kRaggedMaxStages <= kSumThreads, "a thread a coefficient");
   // small CTAs where the channels are short (backward of 4096 channels of 1100 samples, 8 stages: 275 us with
   // large ones, 250 with small ones)
   const int least = std::max(128, (5 * b.Smax + 31) / 32 * 32);
   bank_sums_kernel<<<dim3(b.C, 2), b.nUnits > 16 * b.C ? kSumThreads : least, 0, s>>>(b.chans, b.part, b.gcoefs, dhStart, dhPart, gtaps);
   countLaunch();
   return cudaGetLastError();
}

} // namespace dsplib
