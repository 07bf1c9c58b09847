// Tensor-core (tcgen05) FIR kernels for sm_100a.
//
// FIR as a Toeplitz contraction.  A tile of consecutive outputs of one channel
// is computed by an M = 128 (rows) x N (phases) accumulator in TMEM:
//     D[a][b] = sum_m A[a][m] * B[m][b] = y[j0 + P*a + b]
//     A[a][m] = x[j0 + P*a + m]            (data, Hankel: row a starts P samples after row a-1)
//     B[m][b] = g[m - b], g[c] = h[T-1-c]  (taps band, zero outside 0 <= m-b < T)
// The Hankel matrix A is never expanded: the shared-memory descriptors make
// consecutive rows overlap inside the raw signal segment.
//
// int8/int16 (kind::i8, P = N = 16 or 32, tile 2048 or 4096): an 8-bit core-matrix row
//   is 16 bytes = 16 samples, so with P = 16 the no-swizzle K-major descriptor with
//   LBO = 16 B and SBO = 128 B reads row a at byte 16a of the segment; with P = 32 the
//   segment's even and odd 16-byte chunks lie in two parts, LBO apart.
//   int8: one s8 x s8 product.  int16: x = 256*xh + xl, g = 256*gh + gl (xh, gh
//   signed bytes, xl, gl unsigned); y = 65536*hh + 256*(hl + lh) + ll, each an
//   exact int32 kind::i8 accumulation recombined exactly in 64 bits; modulo
//   2^16 the hh term vanishes, so the wrap mode issues three products.
//   Output stage: wrap (natural-C) or Q mode (round half up, shift, saturate).
//
// float (split-BF16x3, kind::f16, P = 64, N = 128, tile 8192): each operand is
//   split into BF16 hi + lo (lo = bf16(v - hi)); the signal planes are stored
//   as consecutive 128-byte blocks of 64 samples in the 128-byte-swizzle
//   K-major layout, whose 8-row atoms have a 128-byte row pitch, so with the
//   descriptor starting at block kb row a reads block a + kb.  B's 128 rows hold
//   g_hi and g_lo by phase in alternate groups of eight (bfBand):
//     MMA 1: D += A_hi x B        (x_hi*g_hi | x_hi*g_lo)
//     MMA 2: D += A_lo x B        (x_lo*g_hi | x_lo*g_lo)
//     y[j0 + 64a + b] = D[a][column of g_hi, b] + D[a][column of g_lo, b]
//   The three products hi*hi, hi*lo, lo*hi leave the lo*lo term (2^-16 of each
//   product) out, 1.25e-5 of the peak output on the 256-tap FIR workload; the
//   fourth rides in the same MMA (N = 128 instead of 64 for the lo plane) at no
//   measurable cost here (the tile loop is not MMA-bound) and brings it to 8.7e-6.
//
// All kernels are persistent: one wave of CTAs strides over runs of consecutive tiles.  The
// integer kernel keeps a band of shared taps for all of a CTA's tiles and fetches each tile's
// segment during the one before.
// All waits on the tensor core are bounded; on expiry the kernel sets the error word it
// was given (the calling handle's or plan's), frees its TMEM and exits.
#include <algorithm>
#include <climits>
#include <cstdio>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "dsplib_internal.h"
#include "tc_common.cuh"

namespace dsplib {

// Set the error word of the call (mapped page-locked host memory; a plain store, since
// atomics on host memory are not available on every system).
__device__ __forceinline__ void raiseError(int *err)
{
   if (err) *(volatile int *) err = 1;
}

namespace {

constexpr int kRows = 128;

// ------------------------------------------------------------------ integer

constexpr int kThreads = 128;
constexpr int kMaxTapsTc = 2048;
constexpr int kIntTuneTile = 2048; // outputs a tile counts as in the autotuner's keys

// Sizes of a form with P outputs a row (16 or 32), for T taps and the longest lead.
template <typename T, int P> struct IntShape {
   static constexpr int tile = kRows * P;
   static constexpr int planes = sizeof(T);              // byte planes of a sample
   static constexpr int per = 16 / (int) sizeof(T);      // samples a 16-byte vector
   static constexpr int align = P * sizeof(T) >= 32 ? 32 / (int) sizeof(T) : 16; // outputs a row starts at a multiple of
   static constexpr int cols(bool q) { return planes == 1 ? P : (q ? 3 : 2) * P; } // accumulator columns
   static constexpr uint32_t tmemCols(bool q) { return cols(q) <= 32 ? 32 : cols(q) <= 64 ? 64 : 128; }
   static constexpr int perSm(bool q) { return planes == 1 ? 8 : tmemCols(q) == 128 ? 4 : 6; } // CTAs an SM
   static constexpr int pre = (tile + kMaxTapsTc + 64) * (int) sizeof(T) / 16 / kThreads + 1; // vectors a thread
   __host__ __device__ static int K(int taps) { return ((P - 1 + taps + per - 1 + 31) / 32) * 32; }
   __host__ __device__ static int seg(int taps) { return tile - P + K(taps); }
   // Chunk c (16 samples) of the segment is chunk c / (P / 16) of part c % (P / 16): with P = 16
   // bytes a row the rows of a core matrix follow one another; a longer row is read as P / 16
   // such parts.  The padding spreads the parts over the banks.
   __host__ __device__ static int part(int taps)
   {
      const int n = P / 16, chunks = (seg(taps) / 16 + n - 1) / n;
      return n == 1 ? chunks * 16 : ((chunks * 16 + 63) / 128) * 128 + 64;
   }
   __host__ __device__ static int plane(int taps) { return P / 16 * part(taps); }
   static constexpr int lead = per - 1; // longest
   __host__ __device__ static int taps(int t) { return (K(t) + P + lead + 4 + 15) / 16 * 16; } // bytes of gb, one plane
   __host__ __device__ static int band(int t) { return (K(t) - 16 + P + lead) * 16; }          // bytes, one plane
   __host__ __device__ static size_t smem(int t) { return 16 + (size_t) planes * (taps(t) + band(t) + 2 * plane(t)); }
};

// Four int8 Q-mode outputs (round half up, shift, saturate) packed into one word, byte k =
// output k: two saturating pack conversions instead of a clamp per output and byte moves.
__device__ __forceinline__ uint32_t outStage8x4(int v0, int v1, int v2, int v3, int shift)
{
   if (shift > 0) {
      const int r = 1 << (shift - 1);
      v0 = (v0 + r) >> shift, v1 = (v1 + r) >> shift, v2 = (v2 + r) >> shift, v3 = (v3 + r) >> shift;
   }
   uint32_t hi, d;
   asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(v3), "r"(v2));
   asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(v1), "r"(v0), "r"(hi));
   return d;
}

// Two int16 Q-mode outputs packed into one word (low half = v0): round half up and shift in
// 64 bits, narrow to 32 bits with saturation, then one saturating pack conversion.
__device__ __forceinline__ uint32_t outStage16x2(long long v0, long long v1, int shift)
{
   if (shift > 0) {
      const long long r = 1LL << (shift - 1);
      v0 = (v0 + r) >> shift, v1 = (v1 + r) >> shift;
   }
   int w0, w1;
   uint32_t d;
   asm("cvt.sat.s32.s64 %0, %1;" : "=r"(w0) : "l"(v0));
   asm("cvt.sat.s32.s64 %0, %1;" : "=r"(w1) : "l"(v1));
   asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(d) : "r"(w1), "r"(w0));
   return d;
}

__device__ __forceinline__ void cpAsync16(void *dst, const void *src)
{
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smemAddr(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cpAsyncWaitAll() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Store 32 bytes to a 32-byte aligned address as one access.
__device__ __forceinline__ void store32(void *p, const uint32_t *w)
{
   asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                : "memory");
}

// Integer FIR.  Integer sums do not depend on how they are grouped, so a channel's tile grid is
// laid to suit its rows: a row of P outputs starts on a 16- or 32-byte boundary of y (`shift`
// outputs before the channel's first one, never stored), and the input window of a tile starts
// `lead` samples before its first output's, on a 16-byte boundary, with as many zero taps in
// front.  Every load and store is then a whole aligned vector but those at a channel's ends, and
// a row goes from its TMEM lane to memory through one thread's registers.
//
// Runs are equal shares of all tiles of all channels in turn, one for each resident CTA, so
// no SM waits for another's last channel (runs of whole or half channels: 3.4 waves of 888
// CTAs on 1000 channels).  A tile is a chain of fetch, barrier, MMAs, drain of some 4000 clk,
// hidden by the 4 to 8 CTAs of an SM; the MMAs take a third of the shared memory's rate and
// instructions 60 % of the issue slots (4096 x 16384 int8, 128 taps).  An earlier form with
// tiles of 2048 from each channel's first sample on read rows off the 16-byte boundary sample by
// sample, and assembled the output vectors through shared memory with funnel shifts: 4096
// channels x 16384 int8 samples x 128 taps 63.5 us, now 41.8 (20.5 at the copy rate); 1000
// channels x 10007 int16 samples x 201 taps 85.4, now 25.8; 4096 x 16384 int16 111, now 91,
// in Q mode 171, now 118.
template <typename T> struct IntRow {
   const T *x;
   T *y;
   int l, shift, lead;
};

// Tiles of a channel, with the largest shift any channel needs.
template <typename T, int P> __host__ __device__ inline int intTiles(const FirLaunch &a)
{
   constexpr int al = IntShape<T, P>::align;
   const bool aligned = ((uintptr_t) a.y & (al * sizeof(T) - 1)) == 0 && a.outPitch % al == 0;
   return (int) (((long long) a.outSize + (aligned ? 0 : al - 1) + kRows * P - 1) / (kRows * P));
}

// ONE: shared taps and channels of one tile each.
template <typename T, int QMODE, int P, bool ONE>
__global__ void __launch_bounds__(kThreads, IntShape<T, P>::perSm(QMODE)) fir_int_tc_kernel(FirLaunch a, uint32_t tilesPerRun)
{
   using Sh = IntShape<T, P>;
   constexpr bool SPLIT = sizeof(T) == 2;
   constexpr int per = Sh::per, kTile = Sh::tile, kParts = P / 16;
   const int T_ = a.T;
   const int Kt = Sh::K(T_), seg = Sh::seg(T_), part = Sh::part(T_), planeBytes = Sh::plane(T_);
   extern __shared__ __align__(128) unsigned char sm[];
   uint64_t *mbar = (uint64_t *) sm;
   uint32_t *tslot = (uint32_t *) (sm + 8);
   // Reversed taps g[c] = h[T-1-c] as bytes (int16: high and low byte planes) at byte
   // P - 1 + bandLead + c of gb0 / gb1, zero elsewhere: one 32-bit word per thread to build.
   uint32_t *gb0 = (uint32_t *) (sm + 16);
   uint32_t *gb1 = (uint32_t *) (sm + 16 + Sh::taps(T_));
   unsigned char *B0 = sm + 16 + Sh::planes * Sh::taps(T_);
   unsigned char *B1 = B0 + Sh::band(T_);
   unsigned char *Abase = B0 + (size_t) Sh::planes * Sh::band(T_);
   auto A = [&](int buf, int plane) { return Abase + (buf * Sh::planes + plane) * planeBytes; };

   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   if (warp == 0) tc::tmemAlloc(tslot, Sh::tmemCols(QMODE));
   if (tid == 0) tc::mbarInit(mbar, 1);
   tc::fenceBeforeSync();
   __syncthreads();
   tc::fenceAfterSync();
   const uint32_t tmem = *tslot;

   const int inExtent = a.outSize + T_ - 1;
   // Runs of tilesPerRun consecutive tiles (of all channels in turn); CTAs stride over the runs.
   // The band is built anew when the channel's taps or its lead are others than the last tile's; shared
   // taps of channels of one tile each are built for the longest lead, and the shorter ones read the
   // band from a later start (anew for each lead, 3000 channels x 3347 int16 samples x 2048 taps took 131 us
   // instead of 109; but a start off the 128-byte boundary slows the MMAs' reads: 4096 channels x 16384 int8
   // samples x 128 taps, five tiles a channel, 43.3 us so, 41.7 built anew).
   const uint32_t nt = (uint32_t) intTiles<T, P>(a);
   const uint32_t nTiles = (uint32_t) a.batch * nt; // with the grid below 2^32: memory bounds it
   auto rowOf = [&](int l) {
      IntRow<T> r;
      r.l = l;
      r.x = (const T *) a.x + (long long) l * a.inPitch;
      r.y = (T *) a.y + (long long) l * a.outPitch;
      r.shift = (int) ((uintptr_t) r.y / sizeof(T)) & (Sh::align - 1);
      r.lead = (int) (((uintptr_t) r.x / sizeof(T)) - r.shift) & (per - 1);
      return r;
   };
   // The segment of tile t as 16-byte vectors, samples outside the row zero: int8 straight into
   // shared memory, int16 into registers (its byte planes are parted when the tile's turn comes).
   constexpr int kPre = SPLIT ? Sh::pre : 1;
   const int nvec = (seg + per - 1) / per;
   int4 pre[kPre];
   auto slot8 = [&](int buf, int k) { return (int4 *) (A(buf, 0) + (k % kParts) * part + (k / kParts) * 16); };
   auto fetch = [&](const IntRow<T> &r, uint32_t t, int buf) {
      const long long s0 = (long long) t * kTile - r.shift - r.lead;
      const T *p = r.x + s0;
      auto edge = [&](int k) {
         const long long q = s0 + (long long) k * per;
         if (q <= -per || q >= inExtent) return make_int4(0, 0, 0, 0);
         __align__(16) T tmp[per];
#pragma unroll
         for (int e = 0; e < per; e++) tmp[e] = (q + e >= 0 && q + e < inExtent) ? p[k * per + e] : (T) 0;
         return *(const int4 *) tmp;
      };
      // vectors [v0, v1) lie inside the row
      const int v0 = s0 < 0 ? (int) ((-s0 + per - 1) / per) : 0;
      const int v1 = (int) min((long long) nvec, (inExtent - s0) / per);
      if (SPLIT) {
#pragma unroll
         for (int i = 0; i < kPre; i++) {
            const int k = tid + i * kThreads;
            if (k >= v0 && k < v1) pre[i] = ((const int4 *) p)[k];
            else if (k < nvec) pre[i] = edge(k);
         }
      }
      else {
         for (int k = tid; k < nvec; k += kThreads) {
            if (k >= v0 && k < v1) cpAsync16(slot8(buf, k), (const int4 *) p + k);
            else *slot8(buf, k) = edge(k);
         }
      }
   };
   uint32_t iter = 0;
   int bandOf = -1, bandLead = -1; // channel and lead of the taps the band holds
   int buf = 0;
   bool bad = false; // this thread's wait gave up
   const uint32_t nRuns = (nTiles + tilesPerRun - 1) / tilesPerRun;
   uint32_t run = blockIdx.x, tile = run * tilesPerRun;
   bool more = run < nRuns;
   IntRow<T> r = rowOf(more ? (int) (tile / nt) : 0);
   uint32_t t = tile % nt, end = min(nTiles, tile + tilesPerRun);
   if (more) fetch(r, t, 0);
   while (more) {
      if (SPLIT) {
#pragma unroll
         for (int i = 0; i < kPre; i++) {
            const int k = tid + i * kThreads, c = k >> 1; // vector k = half of chunk c
            const int o = (c % kParts) * part + (c / kParts) * 16 + (k & 1) * 8;
            const int4 &v = pre[i];
            if (k < nvec) {
               *(uint2 *) (A(buf, 0) + o) = make_uint2(__byte_perm(v.x, v.y, 0x7531), __byte_perm(v.z, v.w, 0x7531));
               *(uint2 *) (A(buf, 1) + o) = make_uint2(__byte_perm(v.x, v.y, 0x6420), __byte_perm(v.z, v.w, 0x6420));
            }
         }
      }
      if (ONE ? bandOf < 0 : bandOf < 0 || (a.filtPitch != 0 && bandOf != r.l) || bandLead != r.lead) {
         const T *h = (const T *) a.h + (long long) r.l * a.filtPitch;
         // the previous band's last MMAs are complete (waited); its words were read before that
         for (int wd = tid; wd < Sh::taps(T_) / 4; wd += kThreads) {
            uint32_t w0 = 0, w1 = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
               const int c = 4 * wd + j - (P - 1) - (ONE ? Sh::lead : r.lead);
               const int g = (c >= 0 && c < T_) ? (int) h[T_ - 1 - c] : 0;
               if (SPLIT) {
                  w0 |= (uint32_t) ((g >> 8) & 0xFF) << (8 * j);
                  w1 |= (uint32_t) (g & 0xFF) << (8 * j);
               }
               else {
                  w0 |= (uint32_t) (g & 0xFF) << (8 * j);
               }
            }
            gb0[wd] = w0;
            if (SPLIT) gb1[wd] = w1;
         }
         __syncthreads();
         // Taps band, K-major no-swizzle, phases in reverse (column n = phase P-1-n): element
         // (m, n) = g[m + n - (P-1) - lead] = byte m + n + bandLead - lead of gb, so the 16-byte chunk of
         // m = 16q, column n depends on 16q + n alone and is held once, at 16 (16q + n + bandLead - lead);
         // gathered from five words with funnel shifts.
         for (int ch = tid; ch < Kt - 16 + P + (ONE ? Sh::lead : 0); ch += kThreads) {
            const int w = ch >> 2, sh = (ch & 3) * 8;
#pragma unroll
            for (int pl = 0; pl < Sh::planes; pl++) {
               const uint32_t *gb = pl ? gb1 : gb0;
               const uint32_t v0 = gb[w], v1 = gb[w + 1], v2 = gb[w + 2], v3 = gb[w + 3], v4 = gb[w + 4];
               uint4 o;
               o.x = __funnelshift_r(v0, v1, sh);
               o.y = __funnelshift_r(v1, v2, sh);
               o.z = __funnelshift_r(v2, v3, sh);
               o.w = __funnelshift_r(v3, v4, sh);
               *(uint4 *) ((pl ? B1 : B0) + 16 * ch) = o;
            }
         }
         bandOf = r.l;
         bandLead = ONE ? Sh::lead : r.lead;
      }
      if (!SPLIT) cpAsyncWaitAll();
      tc::fenceProxyAsync();
      tc::fenceBeforeSync();
      // segment[buf] and band written, previous accumulators drained by every warp; a wait that gave
      // up ends all together
      if (__syncthreads_or(bad)) break;
      if (warp == 0 && tc::electOne()) {
         tc::fenceAfterSync();
         constexpr uint32_t al = kParts == 1 ? 16 : 0;
         const uint32_t lbo = al ? al : (uint32_t) part;
         const uint64_t dA0 = tc::descNoSwizzle(tc::smemAddr(A(buf, 0)), lbo, 128);
         const uint64_t dA1 = tc::descNoSwizzle(tc::smemAddr(A(buf, 1)), lbo, 128);
         const uint32_t skip = ONE ? 16 * (Sh::lead - r.lead) : 0;
         uint64_t dB0 = tc::descNoSwizzle(tc::smemAddr(B0) + skip, 256, 128);
         uint64_t dB1 = tc::descNoSwizzle(tc::smemAddr(B1) + skip, 256, 128);
         // 32 taps a step: two chunks of the segment, 512 bytes of the band (descriptor addresses count 16)
         for (int kk = 0; kk < Kt / 32; kk++, dB0 += 32, dB1 += 32) {
            const uint32_t off = (2 * kk % kParts) * (part / 16) + 2 * kk / kParts;
            if (!SPLIT) tc::mmaI8(tmem, dA0 + off, dB0, tc::idesc(2, 1, 1, kRows, P), kk > 0);
            else {
               tc::mmaI8(tmem, dA0 + off, dB1, tc::idesc(2, 1, 0, kRows, P), kk > 0);     // hi*lo
               tc::mmaI8(tmem, dA1 + off, dB0, tc::idesc(2, 0, 1, kRows, P), true);       // lo*hi
               tc::mmaI8(tmem + P, dA1 + off, dB1, tc::idesc(2, 0, 0, kRows, P), kk > 0); // lo*lo
               if (QMODE) tc::mmaI8(tmem + 2 * P, dA0 + off, dB0, tc::idesc(2, 1, 1, kRows, P), kk > 0); // hi*hi
            }
         }
         tc::commit(mbar);
      }
      __syncwarp();
      // fetch the next tile's segment now; int16 samples are written to shared memory after this
      // tile's drain
      const IntRow<T> cur = r;
      const uint32_t tNow = t;
      if (++tile == end) {
         run += gridDim.x;
         more = run < nRuns;
         if (more) {
            tile = run * tilesPerRun;
            end = min(nTiles, tile + tilesPerRun);
            r = rowOf((int) (tile / nt));
            t = tile % nt;
         }
      }
      else if (++t == nt) {
         r = rowOf(r.l + 1);
         t = 0;
      }
      if (more) fetch(r, t, buf ^ 1);
      if (!tc::mbarWait(mbar, iter & 1)) {
         bad = true;
         raiseError(a.err);
      }
      iter++;
      buf ^= 1;
      tc::fenceAfterSync();
      if (!bad) {
         // Drain: warp w owns TMEM lanes 32w..32w+31 = rows; P consecutive outputs a row, columns reversed.
         const uint32_t lanes = tmem + ((uint32_t) (warp * 32) << 16);
         const long long j0 = (long long) tNow * kTile - cur.shift + (warp * 32 + lane) * P;
         constexpr int kPiece = Sh::align; // outputs a store
         constexpr int kGroups = kPiece / 16;
         constexpr int kWords = kPiece * (int) sizeof(T) / 4;
#pragma unroll
         for (int h = 0; h < P / kPiece; h++) {
            __align__(16) uint32_t w[kWords];
#pragma unroll
            for (int g = 0; g < kGroups; g++) {
               const int col = P - 16 - kPiece * h - 16 * g;
               uint32_t acc[3][16];
               tc::tmemLoad16(lanes + col, acc[0]);
               if (SPLIT) tc::tmemLoad16(lanes + P + col, acc[1]);
               if (SPLIT && QMODE) tc::tmemLoad16(lanes + 2 * P + col, acc[2]);
               tc::tmemWaitLoad();
#pragma unroll
               for (int b = 0; b < 16; b += 4) { // outputs b..b+3 = columns 15-b..12-b
                  const int c = 15 - b;
                  uint32_t *d = w + (16 * g + b) * (int) sizeof(T) / 4;
                  if (SPLIT && QMODE) {
#pragma unroll
                     for (int e = 0; e < 4; e += 2) {
                        auto sum = [&](int k) {
                           return ((long long) (int) acc[2][k] << 16) + ((long long) (int) acc[0][k] << 8) +
                                  (long long) (int) acc[1][k];
                        };
                        d[e / 2] = outStage16x2(sum(c - e), sum(c - e - 1), a.shift);
                     }
                  }
                  else if (SPLIT) { // modulo 2^16 the hi*hi term vanishes
#pragma unroll
                     for (int e = 0; e < 4; e += 2)
                        d[e / 2] = __byte_perm((acc[0][c - e] << 8) + acc[1][c - e],
                                               (acc[0][c - e - 1] << 8) + acc[1][c - e - 1], 0x5410);
                  }
                  else if (QMODE)
                     d[0] = outStage8x4((int) acc[0][c], (int) acc[0][c - 1], (int) acc[0][c - 2], (int) acc[0][c - 3],
                                        a.shift);
                  else // modulo 2^8
                     d[0] = __byte_perm(__byte_perm(acc[0][c], acc[0][c - 1], 0x0040),
                                        __byte_perm(acc[0][c - 2], acc[0][c - 3], 0x0040), 0x5410);
               }
            }
            const long long j = j0 + kPiece * h;
            if (j >= 0 && j + kPiece <= a.outSize) {
               if (kWords == 8) store32(cur.y + j, w);
               else *(uint4 *) (cur.y + j) = *(const uint4 *) w;
            }
            else if (j > -kPiece && j < a.outSize) {
               const int b0 = j < 0 ? (int) -j : 0, b1 = (int) min((long long) kPiece, a.outSize - j);
#pragma unroll
               for (int b = 0; b < kPiece; b++)
                  if (b >= b0 && b < b1)
                     cur.y[j + b] = SPLIT ? (T) (w[b / (SPLIT ? 2 : 4)] >> (16 * (b & 1))) : (T) (w[b / 4] >> (8 * (b & 3)));
            }
         }
      }
   }
   if (!SPLIT) cpAsyncWaitAll();
   tc::fenceBeforeSync();
   __syncthreads();
   if (warp == 0) tc::tmemFree(tmem, Sh::tmemCols(QMODE));
}

// CTAs per SM of the longest wave the autotuner may ask for.
template <typename T> constexpr int intLaunchBound() { return sizeof(T) == 2 ? 6 : 8; }

template <typename T, int QMODE, int P> static cudaError_t launchIntTcP(const FirLaunch &a, cudaStream_t s)
{
   using Sh = IntShape<T, P>;
   const size_t smem = Sh::smem(a.T);
   const auto fn = a.filtPitch == 0 && intTiles<T, P>(a) == 1 ? fir_int_tc_kernel<T, QMODE, P, true>
                                                              : fir_int_tc_kernel<T, QMODE, P, false>;
   // the same limit for every call: calls on several threads do not lower each other's
   cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) Sh::smem(kMaxTapsTc));
   if (e != cudaSuccess) return e;
   const uint32_t nt = (uint32_t) intTiles<T, P>(a);
   // persistent: one wave of resident CTAs striding over the runs (CTAs per SM: the autotuner's
   // choice or the launch bound, fewer when shared memory runs out first)
   const int bySmem = (int) ((228u * 1024u) / (smem + 1024u));
   int perSm = a.tunePerSm > 0 ? a.tunePerSm : Sh::perSm(QMODE);
   perSm = std::max(1, std::min({perSm, bySmem, Sh::perSm(QMODE)}));
   const long long wave = (long long) perSm * (deviceSms() > 0 ? deviceSms() : 148);
   const long long total = (long long) a.batch * nt;
   const long long tpr = a.tuneTpc > 0 ? std::min<long long>(a.tuneTpc, nt) : (total + wave - 1) / wave;
   const long long runs = (total + tpr - 1) / tpr;
   FirLaunch k = a;
   // int8: |acc| <= 2048 * 2^14 = 2^25, so every shift from 27 up rounds to zero, as 31
   // (the largest the 32-bit output stage can take) does.
   if (sizeof(T) == 1 && k.shift > 31) k.shift = 31;
   fn<<<(unsigned) std::min(runs, wave), kThreads, smem, s>>>(k, (uint32_t) tpr);
   countLaunch();
   return cudaGetLastError();
}

// Rows of 32 outputs read each byte of the segment half as often in the MMAs (40 clk of shared
// memory a step of 32 taps for 4096 outputs instead of 36 for 2048); rows of 16 do where half the
// larger tile would be empty (a channel within 2048 outputs) and where every tile has an SM of
// its own, for the shorter way through it.  In us, 32 against 16: int8 4096 channels x 16384
// samples x 128 taps 39.3 / 55.5, int16 1000 x 10007 x 201 25.8 / 27.4; int16 4096 x 1100 x 33
// 22.8 / 18.7, int8 4096 x 2048 x 16 18.6 / 16.5, int8 16 x 4096 x 64 6.05 / 5.0.
template <typename T, int QMODE> static cudaError_t launchIntTc(const FirLaunch &a, cudaStream_t s)
{
   const int nt = intTiles<T, 16>(a);
   if (nt == 1 || (long long) nt * a.batch <= (deviceSms() > 0 ? deviceSms() : 148)) return launchIntTcP<T, QMODE, 16>(a, s);
   return launchIntTcP<T, QMODE, 32>(a, s);
}

// ------------------------------------------------------------------ split-BF16x3

constexpr int kBfPhases = 64;
constexpr int kBfTile = kRows * kBfPhases;
constexpr int kBfMaxTaps = kFirBfMaxTaps;
static_assert(kBfTile == kFirBfTile, "ragged run tiles and kernel tiles must agree");

__host__ __device__ constexpr int bfK(int T) { return ((63 + T + 15) / 16) * 16; }
__host__ __device__ constexpr int bfBlocks(int T) { return kRows + (bfK(T) + 63) / 64; }

// Two values as BF16 hi + lo (lo = bf16(v - hi)), packed (a in the low half): one paired
// conversion per plane.
__device__ __forceinline__ void splitBf16x2(float a, float b, uint32_t &hi, uint32_t &lo)
{
   const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
   const __nv_bfloat162 l = __floats2bfloat162_rn(a - __low2float(h), b - __high2float(h));
   hi = *(const uint32_t *) &h;
   lo = *(const uint32_t *) &l;
}

// A run of consecutive output tiles [t0, t1) of one channel:
//     y[j] = sum_{c<T} x[inShift + j + c] * g(c),  x zero outside [0, inLen),
//     g(c) = h[T-1-c] (reverse = 1: DSPLIB_fir correlation order) or h[c] (reverse = 0).
// A tile's window starts `lead` samples before its first output's, on a 16-byte boundary, and
// the taps have as many zeros in front: every raw copy and every read of it is then aligned
// (the same for all tiles of a channel: a tile is 8192 samples).
struct BfRun {
   const float *x;
   const float *h;
   float *y;
   long long inShift, inLen;
   int outLen, T, reverse, t0, t1;
   int lead, K; // K: taps contracted, leading zeros and phases included
   __device__ void align()
   {
      lead = (int) ((((long long) ((uintptr_t) x >> 2)) + inShift) & 3);
      K = bfK(T + lead);
   }
};

// Pipeline of the split-BF16x3 FIR.  One persistent CTA per SM; the warps of a role
// walk the CTA's tiles in the same order and meet only on mbarriers, so the fetch of a tile,
// the split of the one before, its predecessor's MMAs and the drain of the one before that
// run at the same time:
//   warp 17      (fetch) bulk-copies raw FP32 tiles into a ring of two slots;
//   warps 0-7    (split) write raw tile n as hi/lo planes into set b = n % 2 once tile n - 2's
//                MMAs have read it, and with a run's first tile its taps band;
//   warp 16      (MMA)   one thread issues tile n's MMAs into accumulator b once the planes
//                are full and the accumulator is drained;
//   warps 8-15   (drain) read accumulator b, free it, add the hi and lo taps' columns
//                and store them by whole lines through shared memory.
// What bounds it: the SM's shared-memory data path.  The MMAs read 8 KB each (two N = 128
// MMAs per 16 taps, 64 clocks each at 128 bytes a clock: 2560 clocks a tile of 8192 outputs
// with 256 taps), and raw tile, planes, staged outputs and stores pass the same path, about
// 1800 clocks more.  Measured on 1024 channels x 65536 samples x 256 taps: 143 us in a short
// run (175 us in a long one, under the power cap) against 240 us for the earlier form, where
// 16 warps split and drained in lock step behind five barriers a tile, an expanded band
// (256 bytes a tap) was built for every run and the issuing thread gave an MMA every 100 clocks.
constexpr int kBfSplitWarps = 8, kBfSplitThreads = 32 * kBfSplitWarps;
constexpr int kBfDrainWarps = 8;
constexpr int kBfMmaWarp = kBfSplitWarps + kBfDrainWarps;
constexpr int kBfFetchWarp = kBfMmaWarp + 1;
constexpr int kBfCta = 32 * (kBfFetchWarp + 1);
constexpr uint32_t kBfTmemCols = 256; // two accumulators of 128 columns
constexpr int kBfMaxBlocks = bfBlocks(kBfMaxTaps + 3);
constexpr int kBfQuads = (kBfMaxBlocks * 16 + kBfSplitThreads - 1) / kBfSplitThreads; // 4-sample groups per split thread

// Shared memory: barriers and the TMEM slot (1024 bytes), two sets of hi/lo planes, an
// output tile, two raw tiles, two taps bands (runs alternate, so the next run's band is built while this one's is read).
constexpr size_t kBfRawFloats = (size_t) kBfMaxBlocks * 64;
constexpr size_t kBfPlane = (size_t) ((kBfMaxBlocks * 128 + 1023) & ~1023);
__host__ __device__ constexpr size_t bfBandBytes(int T) { return (size_t) (bfK(T + 3) / 8 + 8) * 256; }
__host__ __device__ constexpr size_t bfSmemBytes(int Tmax) { return 2048 + 4 * kBfPlane + kBfTile * 4 + 8 * kBfRawFloats + 2 * bfBandBytes(Tmax); }
static_assert(kBfSplitWarps == 8, "a tile's flags are one 64-bit word");
static_assert(bfSmemBytes(kBfMaxTaps) <= 227 * 1024, "two plane sets and two of the longest bands fit");

struct BfSmem {
   uint64_t *mmaDone, *planesFull, *accFree; // one per plane set / accumulator
   uint64_t *rawFull, *rawFree;              // one per raw slot
   uint64_t *edges;                          // the split warps have written a raw tile's edges
   uint32_t *tslot;
   unsigned char *notFinite; // per tile (eight in turn) and split warp: it met a sample that is not finite
   unsigned char *sets, *bands;
   float *stage; // one output tile, 1024 floats per drain warp
   float *raw;
   size_t bandBytes;
   __device__ float *slot(int k) const { return raw + (size_t) k * kBfRawFloats; }
   __device__ unsigned char *hi(int b) const { return sets + (size_t) (2 * b) * kBfPlane; }
   __device__ unsigned char *lo(int b) const { return sets + (size_t) (2 * b + 1) * kBfPlane; }
   __device__ unsigned char *band(int k) const { return bands + (size_t) (k & 1) * bandBytes; }
};

__device__ __forceinline__ BfSmem bfSmemLayout(unsigned char *smraw, int Tmax)
{
   BfSmem L;
   unsigned char *sm = (unsigned char *) (((uintptr_t) smraw + 1023) & ~(uintptr_t) 1023);
   L.mmaDone = (uint64_t *) sm;
   L.planesFull = L.mmaDone + 2;
   L.accFree = L.planesFull + 2;
   L.rawFull = L.accFree + 2;
   L.rawFree = L.rawFull + 2;
   L.edges = L.rawFree + 2;
   L.tslot = (uint32_t *) (L.edges + 1);
   L.notFinite = sm + 512;
   L.sets = sm + 1024;
   L.stage = (float *) (L.sets + 4 * kBfPlane);
   L.raw = L.stage + kBfTile;
   L.bands = (unsigned char *) (L.raw + 2 * kBfRawFloats);
   L.bandBytes = bfBandBytes(Tmax);
   return L;
}

// Blocks of tile t that its valid output rows read (a short last tile needs fewer; the rows
// beyond are computed from stale planes and never stored).
__device__ __forceinline__ int bfTileBlocks(const BfRun &r, int t)
{
   const int outs = (int) min((long long) kBfTile, (long long) r.outLen - (long long) t * kBfTile);
   return (outs + kBfPhases - 1) / kBfPhases + (r.K + 63) / 64;
}

// A raw window: `len` samples from input index w0 on, w0 on a 16-byte boundary of the row x of
// inLen samples.  The bulk copy takes its part inside the input, [lo, hi), both ends on
// 16-byte boundaries; the split threads write the rest (up to 3 samples at each end, and the
// zeros outside the input).
struct BfWindow {
   const float *x;
   long long inLen, w0, lo, hi;
   int len;
   __device__ uint32_t bytes() const { return (uint32_t) (hi - lo) * 4u; }
};
__device__ __forceinline__ BfWindow bfWindow(const float *x, long long inLen, long long w0, int len)
{
   BfWindow w{x, inLen, w0, w0, w0, len};
   if (w0 < 0) w.lo = w0 + ((-w0 + 3) & ~3LL);
   w.hi = w0 + ((min(w0 + len, inLen) - w0) & ~3LL);
   if (w.hi < w.lo) w.hi = w.lo;
   return w;
}
__device__ __forceinline__ void bfFixEdges(const BfWindow &w, float *raw, int tid)
{
   for (int i = tid; i < (int) (w.lo - w.w0); i += kBfSplitThreads) {
      const long long q = w.w0 + i;
      raw[i] = (q >= 0 && q < w.inLen) ? w.x[q] : 0.0f;
   }
   for (int i = (int) (w.hi - w.w0) + tid; i < w.len; i += kBfSplitThreads) {
      const long long q = w.w0 + i;
      raw[i] = (q >= 0 && q < w.inLen) ? w.x[q] : 0.0f;
   }
}
// All split warps have written the edges: a bounded wait like the others (a warp that gave up
// elsewhere would leave a named barrier waiting for good).
__device__ __forceinline__ bool bfEdgesWritten(uint64_t *bar, uint32_t &phase, int lane)
{
   __syncwarp();
   if (lane == 0) tc::mbarArrive(bar);
   return tc::mbarWait(bar, phase++ & 1);
}
// The window of tile t of a run.
__device__ __forceinline__ BfWindow bfTileWindow(const BfRun &r, int t, int blocks)
{
   return bfWindow(r.x, r.inLen, r.inShift - r.lead + (long long) t * kBfTile, blocks * kBfPhases);
}

// Split a raw tile into the planes: sample i (64 per 128-byte block k = i / 64) goes to
// block k, 16-byte chunk c = (i % 64) / 8 stored at k * 128 + ((c ^ (k & 7)) * 16), as hi and lo
// BF16.  A thread takes 4 samples (consecutive lanes, consecutive addresses) and writes half a
// chunk of each plane; its groups are 16 blocks apart, so they share c and k & 7.  The first
// FULL of its up to GROUPS groups need no test.  Returns bits of its samples that BF16 holds no
// finite value for.
template <int FULL, int GROUPS>
__device__ __forceinline__ uint32_t bfSplit(const float *raw, int nQuad, unsigned char *hi, unsigned char *lo, int tid)
{
   const int k = tid >> 4, off = k * 128 + ((((tid >> 1) & 7) ^ (k & 7)) << 4) + (tid & 1) * 8;
   const float4 *src = (const float4 *) raw + tid;
   uint32_t bad = 0;
   hi += off;
   lo += off;
#pragma unroll
   for (int u0 = 0; u0 < GROUPS; u0 += 4) {
      float4 f[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
         if (u0 + u < GROUPS && (u0 + u < FULL || tid + (u0 + u) * kBfSplitThreads < nQuad))
            f[u] = src[(u0 + u) * kBfSplitThreads];
#pragma unroll
      for (int u = 0; u < 4; u++)
         if (u0 + u < GROUPS && (u0 + u < FULL || tid + (u0 + u) * kBfSplitThreads < nQuad)) {
            uint2 hv, lv;
            splitBf16x2(f[u].x, f[u].y, hv.x, lv.x);
            splitBf16x2(f[u].z, f[u].w, hv.y, lv.y);
            *(uint2 *) (hi + (u0 + u) * (kBfSplitThreads * 8)) = hv;
            *(uint2 *) (lo + (u0 + u) * (kBfSplitThreads * 8)) = lv;
            // an exponent of all ones carries into the sign
            bad |= (((hv.x & 0x7f807f80u) + 0x00800080u) | ((hv.y & 0x7f807f80u) + 0x00800080u)) & 0x80008000u;
         }
   }
   return bad;
}

// Taps band of a run.  Column n = 16 u + 8 v + i of the accumulator (u < 8, v = 0: hi taps,
// 1: lo taps, i < 8) is phase b = 63 - (8 u + i); its operand row holds g[m - b], so the
// 16-byte chunk q (taps m = 8 q .. 8 q + 7) of that row is G[8 (q + u) + i ..], G[k] = g[k - 63 - lead]:
// it depends on q + u only.  With the phases in this order the K-major descriptor of the
// band therefore reads one copy of each chunk, at (q + u) * 256 + v * 128 + i * 16 (256 bytes
// between K chunks, 128 between groups of 8 columns), K / 8 + 8 rows of 256 bytes in all
// instead of 256 bytes a tap.
__device__ __forceinline__ void bfBand(const BfRun &r, unsigned char *band, int tid)
{
   const int T = r.T, n = r.K + 64;
   for (int c = tid; c < n; c += kBfSplitThreads) { // c = 8 (q + u) + i
      uint32_t hv[4], lv[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
         const int k0 = c + 2 * e - 63 - r.lead, k1 = k0 + 1;
         const float g0 = (k0 >= 0 && k0 < T) ? r.h[r.reverse ? T - 1 - k0 : k0] : 0.0f;
         const float g1 = (k1 >= 0 && k1 < T) ? r.h[r.reverse ? T - 1 - k1 : k1] : 0.0f;
         splitBf16x2(g0, g1, hv[e], lv[e]);
      }
      unsigned char *d = band + (c >> 3) * 256 + (c & 7) * 16;
      *(uint4 *) d = make_uint4(hv[0], hv[1], hv[2], hv[3]);
      *(uint4 *) (d + 128) = make_uint4(lv[0], lv[1], lv[2], lv[3]);
   }
}

// A sample that is not finite makes the 64 outputs of every row NaN whose window holds it: row a
// contracts the samples [64 a, 64 a + bfK(T)), most of them with zeros of the band.  The lead
// makes the contracted window begin up to 3 samples earlier and end up to 15 later.  Outputs that
// only such a sample spoiled are computed anew, in FP32 as the plain kernel does: rows of 32
// outputs y[64 i + lane], row i's window at input index q0 + 64 i, `first` outputs into the row's 64.
__device__ __noinline__ void bfRestoreRows(const float *x, long long inLen, long long q0, const float *h, int T, int reverse,
                                           int lead, float *y, long long left, int first)
{
   const int lane = threadIdx.x & 31, K0 = bfK(T), K = bfK(T + lead);
   auto spoils = [](float v) { return (__float_as_uint(__bfloat162float(__float2bfloat16_rn(v))) & 0x7f800000u) == 0x7f800000u; };
   auto bad = [&](long long q) { return q >= 0 && q < inLen && spoils(x[q]); };
   // lane = row: spoiled from outside its window, and not by its first samples
   bool mine = false;
   if (lane * kBfPhases < left) {
      const long long q = q0 + lane * kBfPhases;
      for (int k = 1; k <= lead; k++) mine = mine || bad(q - k);
      for (int k = K0; k < K - lead; k++) mine = mine || bad(q + k);
      for (int k = 0; k < 2; k++) mine = mine && !bad(q + k);
   }
   uint32_t rows = __ballot_sync(0xffffffffu, mine);
   if (!rows) return;
   bool tap = false;
   for (int c = lane; c < T; c += 32) tap = tap || spoils(h[c]);
   if (__any_sync(0xffffffffu, tap)) return;
   for (; rows; rows &= rows - 1) {
      const int row = __ffs(rows) - 1;
      const long long q = q0 + row * kBfPhases;
      bool inside = false;
      for (int k = lane; k < K0; k += 32) inside = inside || bad(q + k);
      if (__any_sync(0xffffffffu, inside)) continue;
      float sum = 0.0f;
      for (int c = 0; c < T; c++) {
         const long long i = q + first + lane + c;
         if (i >= 0 && i < inLen) sum = fmaf(x[i], h[reverse ? T - 1 - c : c], sum);
      }
      if (row * kBfPhases + lane < left) y[row * kBfPhases + lane] = sum;
   }
}

// Drain one accumulator: warp (quad, half) takes 32 rows of 32 phases each, outputs
// 64 (32 quad + lane) + 32 (1 - half) .. + 32 of tile t, one row a lane.  The sums go to the
// warp's own 4 KB of shared memory, the 16-byte units of a row permuted by the row (eight
// rows store to distinct banks), and leave as whole coalesced lines.  (Stored from
// registers, a warp's store covers 32 rows, and the kernel is bound by its partial lines:
// 207 us on 1024 x 65536 x 256 taps; with four drain warps instead of eight 195 us, their
// chain of loads, sums and stores then being the longest of the pipeline.)
__device__ __forceinline__ void bfDrain(const BfRun &r, const BfSmem &L, uint32_t acc, int b, int t, int dw, int lane)
{
   const int quad = dw & 3, half = dw >> 2;
   const int o0 = quad * (32 * kBfPhases) + 32 * (1 - half); // first output of the warp's first row
   const long long j0 = (long long) t * kBfTile + o0;
   float *stage = L.stage + dw * (32 * 32);
   __syncwarp(); // the previous tile has left the staging rows
#pragma unroll
   for (int p = 0; p < 2; p++) {
      uint32_t d[32];
      tc::tmemLoad32(acc + ((uint32_t) (quad * 32) << 16) + half * 64 + p * 32, d);
      tc::tmemWaitLoad();
      if (p == 1) { // the warp's part is in registers
         tc::fenceBeforeSync();
         __syncwarp();
         if (lane == 0) tc::mbarArrive(L.accFree + b);
      }
      // columns 16 u + i (hi taps) and 16 u + 8 + i: phase 63 - 8 (4 half + 2 p + u) - i
#pragma unroll
      for (int u = 0; u < 2; u++)
#pragma unroll
         for (int v = 0; v < 2; v++) {
            auto sum = [&](int i) { return __uint_as_float(d[16 * u + i]) + __uint_as_float(d[16 * u + 8 + i]); };
            const int unit = 7 - 2 * (2 * p + u) - v;
            *(float4 *) (stage + lane * 32 + ((unit ^ (lane & 7)) << 2)) =
                make_float4(sum(4 * v + 3), sum(4 * v + 2), sum(4 * v + 1), sum(4 * v));
         }
   }
   __syncwarp();
   float *y = r.y + j0;
   const long long left = (long long) r.outLen - j0; // valid outputs from the warp's first one on
   if (((uintptr_t) y & 15) == 0 && left >= 31 * kBfPhases + 32) {
#pragma unroll
      for (int i = 0; i < 8; i++) { // unit lane % 8 of row 4 i + lane / 8
         const int row = 4 * i + (lane >> 3);
         *(float4 *) (y + row * kBfPhases + (lane & 7) * 4) =
             *(const float4 *) (stage + row * 32 + (((lane & 7) ^ (row & 7)) << 2));
      }
   }
   else {
#pragma unroll
      for (int row = 0; row < 32; row++) {
         const float v = stage[row * 32 + (((lane >> 2) ^ (row & 7)) << 2) + (lane & 3)];
         if (row * kBfPhases + lane < left) y[row * kBfPhases + lane] = v;
      }
   }
}

// MMA thread: the Toeplitz contraction of one tile into accumulator d, committed to done.
__device__ __forceinline__ void bfIssue(int K, uint32_t ahi, uint32_t alo, uint32_t bt, uint32_t d, uint64_t *done)
{
   const uint32_t id128 = tc::idesc(1, 1, 1, kRows, 128);
   // The swizzle is applied on absolute shared-memory address bits, so a start
   // that is not atom-aligned (block k16 / 4 of the plane) keeps base offset 0.
   uint64_t dHi = tc::descSw128(ahi, 1024, 0), dLo = tc::descSw128(alo, 1024, 0), dB = tc::descNoSwizzle(bt, 256, 128);
   int k16 = 0;
   // descriptor addresses count 16 bytes: 16 taps are 32 bytes of a plane, two rows (512 bytes) of the band
   for (; k16 + 4 <= K / 16; k16 += 4, dHi += 8, dLo += 8, dB += 128) {
#pragma unroll
      for (int sub = 0; sub < 4; sub++) {
         tc::mmaF16(d, dHi + 2 * sub, dB + 32 * sub, id128, k16 + sub > 0);
         tc::mmaF16(d, dLo + 2 * sub, dB + 32 * sub, id128, true);
      }
   }
   for (; k16 < K / 16; k16++, dHi += 2, dLo += 2, dB += 32) {
      tc::mmaF16(d, dHi, dB, id128, k16 > 0);
      tc::mmaF16(d, dLo, dB, id128, true);
   }
   tc::commit(done);
}

// The kernel body: `get(i)` describes run i (i < nRuns); runs are taken in turn by the
// CTAs of the grid.  Every wait is bounded: a role whose wait gives up raises the error word
// and leaves, and the others follow as theirs give up.  LEAD = false: every run's lead is zero (the test
// for samples that are not finite takes 2 % of the time).
template <bool LEAD, typename Get>
__device__ __forceinline__ void bfPipeline(const BfSmem &L, int nRuns, int *err, Get get)
{
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   if (warp == 0) tc::tmemAlloc(L.tslot, kBfTmemCols);
   if (tid == 0) {
      for (int k = 0; k < 2; k++) {
         tc::mbarInit(L.mmaDone + k, 1);
         tc::mbarInit(L.planesFull + k, kBfSplitWarps);
         tc::mbarInit(L.accFree + k, kBfDrainWarps);
         tc::mbarInit(L.rawFull + k, 1);
         tc::mbarInit(L.rawFree + k, kBfSplitWarps);
      }
      tc::mbarInit(L.edges, kBfSplitWarps);
      tc::fenceMbarInit();
   }
   tc::fenceBeforeSync();
   __syncthreads();
   tc::fenceAfterSync();
   const uint32_t tmem = *L.tslot;
   uint32_t n = 0; // tile n of this CTA uses plane set and accumulator n % 2, phase (n / 2) % 2
   if (warp < kBfSplitWarps) {
      bool ok = true;
      int runs = 0, before = 0; // runs so far, tiles of the previous one
      uint32_t edge = 0;
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x, runs++) {
         const BfRun r = get(i);
         // The band's buffer was last read by the run before the previous one: its MMAs are
         // known to be complete (tile n - 3 or earlier) if the previous run had two tiles or
         // more, else once tile n - 2's are.
         if (before >= 2 || n < 2) bfBand(r, L.band(runs), tid);
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1), blocks = bfTileBlocks(r, t);
            // the MMAs of tile n - 2 have read set b, and the raw tile has landed
            ok = n < 2 || tc::mbarWait(L.mmaDone + b, ((n >> 1) - 1) & 1);
            if (t == r.t0 && before < 2 && n >= 2) bfBand(r, L.band(runs), tid);
            ok = ok && tc::mbarWait(L.rawFull + b, (n >> 1) & 1);
            const long long w0 = r.inShift - r.lead + (long long) t * kBfTile;
            if (w0 < 0 || w0 + blocks * kBfPhases > r.inLen) { // the same for every split thread
               if (ok) bfFixEdges(bfTileWindow(r, t, blocks), L.slot(b), tid);
               ok = ok && bfEdgesWritten(L.edges, edge, lane);
            }
            if (!ok) {
               raiseError(err);
               break;
            }
            const uint32_t bad =
                blocks >= kRows ? bfSplit<kRows * 16 / kBfSplitThreads, kBfQuads>(L.slot(b), blocks * 16, L.hi(b), L.lo(b), tid)
                                : bfSplit<0, kBfQuads>(L.slot(b), blocks * 16, L.hi(b), L.lo(b), tid);
            if (LEAD) {
               const bool any = __any_sync(0xffffffffu, bad);
               if (lane == 0) L.notFinite[(n & 7) * kBfSplitWarps + warp] = any;
            }
            tc::fenceProxyAsync();
            __syncwarp();
            if (lane == 0) {
               tc::mbarArrive(L.planesFull + b);
               tc::mbarArrive(L.rawFree + b);
            }
         }
         before = r.t1 - r.t0;
      }
   }
   else if (warp < kBfMmaWarp) {
      bool ok = true;
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x) {
         const BfRun r = get(i);
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1);
            if (!tc::mbarWait(L.mmaDone + b, (n >> 1) & 1)) {
               raiseError(err);
               ok = false;
               break;
            }
            tc::fenceAfterSync();
            bfDrain(r, L, tmem + (uint32_t) b * 128, b, t, warp - kBfSplitWarps, lane);
            // tile n + 8 is split after accumulator n + 4 was freed by every drain warp
            if (LEAD && *(const volatile uint64_t *) (L.notFinite + (n & 7) * kBfSplitWarps)) {
               const BfRun q = get(i); // not held across the tiles
               const int first = 32 * (1 - ((warp - kBfSplitWarps) >> 2));
               const long long j0 = (long long) t * kBfTile + (warp & 3) * (32 * kBfPhases);
               __syncwarp(); // the warp's outputs are stored
               if (q.lead)
                  bfRestoreRows(q.x, q.inLen, q.inShift + j0, q.h, q.T, q.reverse, q.lead, q.y + j0 + first,
                                (long long) q.outLen - j0 - first, first);
            }
         }
      }
   }
   else if (warp == kBfMmaWarp && tc::electOne()) {
      bool ok = true;
      int runs = 0;
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x, runs++) {
         const BfRun r = get(i);
         const int K = r.K;
         const uint32_t bt = tc::smemAddr(L.band(runs));
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1);
            if (!tc::mbarWait(L.planesFull + b, (n >> 1) & 1) ||
                (n >= 2 && !tc::mbarWait(L.accFree + b, ((n >> 1) - 1) & 1))) {
               raiseError(err);
               ok = false;
               break;
            }
            tc::fenceAfterSync();
            bfIssue(K, tc::smemAddr(L.hi(b)), tc::smemAddr(L.lo(b)), bt, tmem + (uint32_t) b * 128, L.mmaDone + b);
         }
      }
      // n MMA groups were committed: wait (bounded) for the last two before TMEM is released
      for (uint32_t k = n >= 2 ? n - 2 : 0; k < n; k++) (void) tc::mbarWait(L.mmaDone + (k & 1), (k >> 1) & 1);
   }
   else if (warp == kBfFetchWarp && tc::electOne()) {
      bool ok = true;
      uint32_t issued = 0;
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x) {
         const BfRun r = get(i);
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1);
            if (n >= 2 && !tc::mbarWait(L.rawFree + b, ((n >> 1) - 1) & 1)) {
               raiseError(err);
               ok = false;
               break;
            }
            const BfWindow w = bfTileWindow(r, t, bfTileBlocks(r, t));
            if (w.bytes()) {
               tc::mbarExpectTx(L.rawFull + b, w.bytes());
               tc::bulkLoad(L.slot(b) + (w.lo - w.w0), r.x + w.lo, w.bytes(), L.rawFull + b);
            }
            else tc::mbarArrive(L.rawFull + b);
            issued = n + 1;
         }
      }
      // copies still in flight land (bounded) before shared memory is given up
      for (uint32_t k = issued >= 2 ? issued - 2 : 0; k < issued; k++)
         (void) tc::mbarWait(L.rawFull + (k & 1), (k >> 1) & 1);
   }
   tc::fenceBeforeSync();
   __syncthreads();
   tc::fenceAfterSync();
   if (warp == 0) tc::tmemFree(tmem, kBfTmemCols);
}

// Dense batch: run i = tiles [part * tilesPerRun, ...) of channel i / parts.
template <bool LEAD> __global__ void __launch_bounds__(kBfCta, 1) fir_bf16x3_tc_kernel(FirLaunch a, int tilesPerRun)
{
   extern __shared__ __align__(16) unsigned char smraw[];
   const int nt = (a.outSize + kBfTile - 1) / kBfTile;
   const int parts = (nt + tilesPerRun - 1) / tilesPerRun;
   bfPipeline<LEAD>(bfSmemLayout(smraw, a.T), a.batch * parts, a.err, [&](int i) {
      const int l = i / parts, part = i - l * parts;
      BfRun r;
      r.x = (const float *) a.x + (long long) l * a.inPitch;
      r.h = (const float *) a.h + (long long) l * a.filtPitch;
      r.y = (float *) a.y + (long long) l * a.outPitch;
      r.inShift = 0;
      r.inLen = (long long) a.outSize + a.T - 1;
      r.outLen = a.outSize;
      r.T = a.T;
      r.reverse = 1;
      r.t0 = part * tilesPerRun;
      r.t1 = min(nt, r.t0 + tilesPerRun);
      r.align();
      return r;
   });
}

// Work lists of the batched filter bank: runs of consecutive tiles of one channel, longest
// first.  dx = 0: forward, y = valid correlation of x with the taps (DSPLIB_fir order);
// dx = 1: input gradient, the full convolution of the output gradient with the taps.
__global__ void __launch_bounds__(kBfCta, 1)
    fir_bf16x3_ragged_kernel(const RaggedChan *chans, const int4 *runs, int nRuns, const float *in,
                             const float *taps, float *out, int dx, int Tmax, int *err)
{
   extern __shared__ __align__(16) unsigned char smraw[];
   bfPipeline<true>(bfSmemLayout(smraw, Tmax), nRuns, err, [&](int i) {
      const int4 it = runs[i];
      const RaggedChan c = chans[it.x];
      BfRun r;
      r.x = in + (dx ? c.gOff : c.xOff);  // input gradient: the gradient plane of the scratch
      r.h = taps + c.hOff;
      r.y = out + (dx ? c.xOff : c.pOff); // forward: the FIR output plane of the work buffer
      r.T = c.T;
      r.inShift = dx ? -(long long) (c.T - 1) : 0;
      r.inLen = dx ? c.L - c.T + 1 : c.L;
      r.outLen = dx ? c.L : c.L - c.T + 1;
      r.reverse = dx ? 0 : 1;
      r.t0 = it.y;
      r.t1 = it.y + it.z;
      r.align();
      return r;
   });
}

// ------------------------------------------------------------------ taps gradient (split-BF16x3)

// Taps gradient of the filter bank, dh_lag[c] = sum_j gu[j] x[j + c] (c < T), on the
// tensor cores.  With j = 64 r + s (row r, phase s) and t' = c + s:
//     D[t'][s] = sum_r x[64 r + t'] gu[64 r + s],      dh_lag[c] = sum_s D[c + s][s],
// a GEMM whose contraction runs over the rows r (time) and whose operands are both
// the signal planes as staged for the forward kernels, read MN-major: A = X^T
// (M = 128 positions t', 64 per 128-byte block, block r + t'/64 of the x plane, so the
// second 64-wide atom of a tile starts one block (128 bytes) after the first), B = G
// (N = 64 phases, block r of the gradient plane).  One accumulator tile per 128
// positions (Mt = ceil((T + 63) / 128) <= 5 tiles of 64 TMEM columns) collects the three
// split products x_hi g_hi + x_lo g_hi + x_hi g_lo over every row of a run; the diagonal
// sums are taken once per run, in a fixed order.
//
// The roles are those of the forward kernel: fetch (raw x and gradient tiles of 64 rows, a
// ring of two), split (8 warps), MMA, and 8 warps that take the diagonal sums of run j
// while the tensor core works on run j + 1 (accumulators of alternate runs 256 columns
// apart; a run of five tiles takes 320 columns and waits for its neighbours).  Bound by the
// shared-memory data path, as the forward kernel: per 64 rows 36 MMAs of 6 KB and 48 clocks
// each (256 taps), and raw tiles, planes and their reads, about 900 clocks.  On the
// 2048-channel bank 319 us against 404 us for one CTA a run that staged a tile of both signals
// in lock step (100 clocks an MMA, set-up and diagonal sums of every run exposed).
constexpr int kDhRows = 64;                       // rows (of 64 samples) per staged tile
constexpr int kDhTile = kDhRows * kBfPhases;
constexpr int kDhMaxMt = (kBfMaxTaps + 6 + 63 + 127) / 128;
constexpr int kDhXBlocks = kDhRows - 1 + 2 * kDhMaxMt; // x blocks a tile's A operands reach
constexpr size_t kDhXPlane = ((kDhXBlocks * 128 + 1023) / 1024) * 1024;
constexpr size_t kDhGPlane = kDhRows * 128;
constexpr size_t kDhSet = 2 * kDhXPlane + 2 * kDhGPlane; // x hi, x lo, g hi, g lo
constexpr int kDhRawX = kDhXBlocks * 64, kDhRawG = kDhTile; // floats
constexpr int kDhXQuads = (kDhXBlocks * 16 + kBfSplitThreads - 1) / kBfSplitThreads;
constexpr int kDhGQuads = kDhRows * 16 / kBfSplitThreads;
constexpr int kDhPitch = 65;                      // floats per staged accumulator row
constexpr size_t kDhSmem = 2048 + 2 * kDhSet + 8 * (size_t) (kDhRawX + kDhRawG) + 4 * (size_t) kRows * kDhPitch;
constexpr int kDhDrainThreads = 32 * kBfDrainWarps;
constexpr uint32_t kDhDrainBar = 2;
static_assert(kDhSmem <= 227 * 1024, "plane sets, raw ring and accumulator staging fit");
static_assert(kDhMaxMt * 64 <= 512 && 4 * 64 <= 256, "accumulator tiles fit the TMEM columns");

// MN-major operand with 128-byte swizzle: 64-element atoms (128-byte rows, 8 rows per
// 1024-byte swizzle atom along K), lbo = byte distance between atoms along M/N,
// sbo = byte distance between 8-row groups along K.
__device__ __forceinline__ uint64_t descSw128Mn(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
   uint64_t d = 0;
   d |= (uint64_t) ((saddr >> 4) & 0x3FFF);
   d |= (uint64_t) ((lbo >> 4) & 0x3FFF) << 16;
   d |= (uint64_t) ((sbo >> 4) & 0x3FFF) << 32;
   d |= (uint64_t) 1 << 46;
   d |= (uint64_t) 2 << 61;
   return d;
}

struct DhRun {
   const float *x, *g;
   int L, Lu, T, Mt, t0, t1, slot; // tiles [t0, t1) of kDhTile samples; slot: its partial sums
   int leadX, leadG;               // samples before a tile that its windows start at, on 16-byte boundaries
};

// 16-row steps of tile t that hold gradient samples (the rows beyond are not contracted), and
// its windows.
__device__ __forceinline__ int dhSteps(const DhRun &r, int t)
{
   return min(kDhRows / 16, (r.Lu + r.leadG - t * kDhTile + 1023) / 1024);
}
__device__ __forceinline__ BfWindow dhWindowX(const DhRun &r, int t, int steps)
{
   return bfWindow(r.x, r.L, (long long) t * kDhTile - r.leadX, (16 * steps - 1 + 2 * r.Mt) * kBfPhases);
}
__device__ __forceinline__ BfWindow dhWindowG(const DhRun &r, int t, int steps)
{
   return bfWindow(r.g, r.Lu, (long long) t * kDhTile - r.leadG, 16 * steps * kBfPhases);
}

__global__ void __launch_bounds__(kBfCta, 1)
    fir_dh_bf16x3_kernel(const RaggedChan *chans, const int4 *runs, int nRuns, const float *x, const float *gu,
                         float *part, int *err)
{
   extern __shared__ __align__(16) unsigned char smraw[];
   unsigned char *sm = (unsigned char *) (((uintptr_t) smraw + 1023) & ~(uintptr_t) 1023);
   uint64_t *mmaDone = (uint64_t *) sm, *planesFull = mmaDone + 2; // per plane set
   uint64_t *rawFull = mmaDone + 4, *rawFree = mmaDone + 6;        // per raw slot
   uint64_t *accFull = mmaDone + 8, *accFree = mmaDone + 10;       // per parity of the run
   uint64_t *edges = mmaDone + 12;
   uint32_t *tslot = (uint32_t *) (mmaDone + 13);
   unsigned char *sets = sm + 1024;
   float *raw = (float *) (sets + 2 * kDhSet);
   float *Ds = raw + 2 * (kDhRawX + kDhRawG);
   auto set = [&](int b) { return sets + (size_t) b * kDhSet; };
   auto slotX = [&](int b) { return raw + b * (kDhRawX + kDhRawG); };
   auto slotG = [&](int b) { return raw + b * (kDhRawX + kDhRawG) + kDhRawX; };
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   auto get = [&](int i) {
      const int4 it = runs[i]; // {channel, first tile, tiles, partial slot}, tiles of 8192 samples
      const RaggedChan c = chans[it.x];
      DhRun r;
      r.x = x + c.xOff;
      r.g = gu + c.gOff;
      r.L = c.L;
      r.Lu = c.Lu;
      r.T = c.T;
      // windows on 16-byte boundaries, the input's at least as far ahead as the gradient's:
      // position t' = c + s + leadX - leadG
      r.leadG = (int) (((uintptr_t) r.g >> 2) & 3);
      r.leadX = (int) (((uintptr_t) r.x >> 2) & 3);
      if (r.leadX < r.leadG) r.leadX += 4;
      r.Mt = (c.T + r.leadX - r.leadG + 63 + 127) / 128;
      r.t0 = it.y * (kBfTile / kDhTile);
      r.t1 = min((it.y + it.z) * (kBfTile / kDhTile), (c.Lu + r.leadG + kDhTile - 1) / kDhTile);
      // the channel's last run takes a tile more where the lead pushes the last samples into it
      if (it.y + it.z == (c.Lu + kBfTile - 1) / kBfTile) r.t1 = (c.Lu + r.leadG + kDhTile - 1) / kDhTile;
      r.slot = it.w;
      return r;
   };
   if (warp == 0) tc::tmemAlloc(tslot, 512);
   if (tid == 0) {
      for (int k = 0; k < 2; k++) {
         tc::mbarInit(mmaDone + k, 1);
         tc::mbarInit(planesFull + k, kBfSplitWarps);
         tc::mbarInit(rawFull + k, 1);
         tc::mbarInit(rawFree + k, kBfSplitWarps);
         tc::mbarInit(accFull + k, 1);
         tc::mbarInit(accFree + k, kBfDrainWarps);
      }
      tc::mbarInit(edges, kBfSplitWarps);
      tc::fenceMbarInit();
   }
   tc::fenceBeforeSync();
   __syncthreads();
   tc::fenceAfterSync();
   const uint32_t tmem = *tslot;
   uint32_t n = 0; // tile n of this CTA uses plane set and raw slot n % 2, phase (n / 2) % 2
   uint32_t j = 0; // run j likewise the accumulators
   bool ok = true;
   if (warp < kBfSplitWarps) {
      uint32_t edge = 0;
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x) {
         const DhRun r = get(i);
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1), steps = dhSteps(r, t);
            ok = (n < 2 || tc::mbarWait(mmaDone + b, ((n >> 1) - 1) & 1)) && tc::mbarWait(rawFull + b, (n >> 1) & 1);
            const long long e = (long long) t * kDhTile;
            const int xb = 16 * steps - 1 + 2 * r.Mt, gb = 16 * steps;
            // the same for every split thread
            if ((t == 0 && r.leadX + r.leadG > 0) || e - r.leadX + xb * kBfPhases > r.L ||
                e - r.leadG + gb * kBfPhases > r.Lu) {
               if (ok) {
                  bfFixEdges(dhWindowX(r, t, steps), slotX(b), tid);
                  bfFixEdges(dhWindowG(r, t, steps), slotG(b), tid);
                  ok = bfEdgesWritten(edges, edge, lane);
               }
            }
            if (!ok) {
               raiseError(err);
               break;
            }
            unsigned char *B = set(b);
            bfSplit<0, kDhXQuads>(slotX(b), xb * 16, B, B + kDhXPlane, tid);
            bfSplit<0, kDhGQuads>(slotG(b), gb * 16, B + 2 * kDhXPlane, B + 2 * kDhXPlane + kDhGPlane, tid);
            tc::fenceProxyAsync();
            __syncwarp();
            if (lane == 0) {
               tc::mbarArrive(planesFull + b);
               tc::mbarArrive(rawFree + b);
            }
         }
      }
   }
   else if (warp < kBfMmaWarp) {
      const int dt = tid - kBfSplitThreads, quad = warp & 3, half = (warp - kBfSplitWarps) >> 2;
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x, j++) {
         const DhRun r = get(i);
         const uint32_t base = tmem + (r.Mt > 4 ? 0 : (j & 1) * 256) + ((uint32_t) (quad * 32) << 16) + half * 32;
         ok = tc::mbarWait(accFull + (j & 1), (j >> 1) & 1);
         if (tc::namedSyncOr(kDhDrainBar, kDhDrainThreads, !ok)) {
            raiseError(err);
            ok = false;
            break;
         }
         tc::fenceAfterSync();
         // lag c adds D[c + shift + s][s] over s, accumulator tile by tile; a thread takes two lags
         float acc[2] = {0.0f, 0.0f};
         const int shift = r.leadX - r.leadG;
         for (int m = 0; m < r.Mt; m++) {
            uint32_t d[32];
            tc::tmemLoad32(base + 64 * m, d);
            tc::tmemWaitLoad();
            if (m + 1 == r.Mt) {
               tc::fenceBeforeSync();
               __syncwarp();
               if (lane == 0) tc::mbarArrive(accFree + (j & 1));
            }
            float *row = Ds + (quad * 32 + lane) * kDhPitch + half * 32;
#pragma unroll
            for (int k = 0; k < 32; k++) row[k] = __uint_as_float(d[k]);
            tc::namedSync(kDhDrainBar, kDhDrainThreads);
#pragma unroll
            for (int u = 0; u < 2; u++) {
               const int c = dt + u * kDhDrainThreads, first = c + shift - 128 * m; // row of s = 0 in this tile
               if (c < r.T && first > -64 && first < 128) {
                  const float *diag = Ds + first * kDhPitch; // row first + sp, column sp
                  for (int s0 = 0; s0 < 64; s0 += 16) { // 16 loads in flight
                     float v[16];
#pragma unroll
                     for (int k = 0; k < 16; k++) {
                        const int row = first + s0 + k;
                        v[k] = (row >= 0 && row < 128) ? diag[(s0 + k) * (kDhPitch + 1)] : 0.0f;
                     }
#pragma unroll
                     for (int k = 0; k < 16; k++) acc[u] += v[k];
                  }
               }
            }
            tc::namedSync(kDhDrainBar, kDhDrainThreads);
         }
#pragma unroll
         for (int u = 0; u < 2; u++) {
            const int c = dt + u * kDhDrainThreads;
            if (c < r.T) part[(long long) r.slot * kBfMaxTaps + c] = acc[u];
         }
      }
   }
   else if (warp == kBfMmaWarp && tc::electOne()) {
      const uint32_t id = tc::idesc(1, 1, 1, kRows, 64) | (1u << 15) | (1u << 16); // both operands MN-major
      bool wide = false; // the run before took five tiles
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x, j++) {
         const DhRun r = get(i);
         const uint32_t base = tmem + (r.Mt > 4 ? 0 : (j & 1) * 256);
         // the run before the previous one has been read, and the previous one too where its columns overlap
         if ((j >= 2 && !tc::mbarWait(accFree + (j & 1), ((j >> 1) - 1) & 1)) ||
             (j >= 1 && (wide || r.Mt > 4) && !tc::mbarWait(accFree + ((j - 1) & 1), ((j - 1) >> 1) & 1))) {
            raiseError(err);
            ok = false;
            break;
         }
         wide = r.Mt > 4;
         const int Mt = r.Mt;
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1), steps = dhSteps(r, t);
            if (!tc::mbarWait(planesFull + b, (n >> 1) & 1)) {
               raiseError(err);
               ok = false;
               break;
            }
            tc::fenceAfterSync();
            unsigned char *B = set(b);
            // descriptor addresses count 16 bytes: a block is 8, the lo planes follow the hi ones
            uint64_t dX = descSw128Mn(tc::smemAddr(B), 128, 1024);
            uint64_t dG = descSw128Mn(tc::smemAddr(B + 2 * kDhXPlane), 128, 1024);
            for (int ks = 0; ks < steps; ks++, dX += 128, dG += 128) {
#pragma unroll
               for (int m = 0; m < kDhMaxMt; m++)
                  if (m < Mt) {
                     tc::mmaF16(base + 64 * m, dX + 16 * m, dG, id, t > r.t0 || ks > 0);
                     tc::mmaF16(base + 64 * m, dX + (16 * m + kDhXPlane / 16), dG, id, true);
                     tc::mmaF16(base + 64 * m, dX + 16 * m, dG + kDhGPlane / 16, id, true);
                  }
            }
            tc::commit(mmaDone + b);
         }
         if (ok) tc::commit(accFull + (j & 1));
      }
      // wait (bounded) for the last two tiles' MMAs before TMEM is released
      for (uint32_t k = n >= 2 ? n - 2 : 0; k < n; k++) (void) tc::mbarWait(mmaDone + (k & 1), (k >> 1) & 1);
   }
   else if (warp == kBfFetchWarp && tc::electOne()) {
      for (int i = blockIdx.x; ok && i < nRuns; i += gridDim.x) {
         const DhRun r = get(i);
         for (int t = r.t0; t < r.t1; t++, n++) {
            const int b = (int) (n & 1), steps = dhSteps(r, t);
            if (n >= 2 && !tc::mbarWait(rawFree + b, ((n >> 1) - 1) & 1)) {
               raiseError(err);
               ok = false;
               break;
            }
            const BfWindow wx = dhWindowX(r, t, steps), wg = dhWindowG(r, t, steps);
            const uint32_t bytes = wx.bytes() + wg.bytes();
            if (bytes) tc::mbarExpectTx(rawFull + b, bytes);
            else tc::mbarArrive(rawFull + b);
            if (wx.bytes()) tc::bulkLoad(slotX(b) + (wx.lo - wx.w0), r.x + wx.lo, wx.bytes(), rawFull + b);
            if (wg.bytes()) tc::bulkLoad(slotG(b) + (wg.lo - wg.w0), r.g + wg.lo, wg.bytes(), rawFull + b);
         }
      }
      // copies still in flight land (bounded) before shared memory is given up
      for (uint32_t k = n >= 2 ? n - 2 : 0; k < n; k++) (void) tc::mbarWait(rawFull + (k & 1), (k >> 1) & 1);
   }
   tc::fenceBeforeSync();
   __syncthreads();
   tc::fenceAfterSync();
   if (warp == 0) tc::tmemFree(tmem, 512);
}
} // namespace

bool firIntTcSupported(const FirLaunch &a)
{
   return (a.dtype == DSPLIB_INT8 || a.dtype == DSPLIB_INT16) && a.T >= 1 && a.T <= kMaxTapsTc && a.outSize > 0;
}

cudaError_t launchFirIntTc(const FirLaunch &a, bool qmode, cudaStream_t s)
{
   if (a.dtype == DSPLIB_INT8) return qmode ? launchIntTc<int8_t, 1>(a, s) : launchIntTc<int8_t, 0>(a, s);
   if (a.dtype == DSPLIB_INT16) return qmode ? launchIntTc<int16_t, 1>(a, s) : launchIntTc<int16_t, 0>(a, s);
   return cudaErrorInvalidValue;
}

bool firBf16x3Supported(const FirLaunch &a) { return a.dtype == DSPLIB_FLOAT32 && a.T >= 1 && a.T <= kBfMaxTaps; }

// Tiles per run (the built-in rule, when the autotuner has no entry): long runs build
// fewer bands, short ones spread evenly over the SMs; at least 8 runs an SM keep the last
// wave's idle share below an eighth.
static int bfTilesPerRun(int nt, int batch)
{
   const long long sms = deviceSms() > 0 ? deviceSms() : 148;
   int tpr = nt;
   while (tpr > 1 && (long long) ((nt + tpr - 1) / tpr) * batch < sms * 8) tpr = (tpr + 1) / 2;
   return tpr;
}

cudaError_t launchFirBf16x3(const FirLaunch &a, cudaStream_t s)
{
   if (!firBf16x3Supported(a)) return cudaErrorNotSupported;
   const size_t smem = bfSmemBytes(a.T);
   const bool aligned = ((uintptr_t) a.x & 15) == 0 && (a.batch == 1 || a.inPitch % 4 == 0); // no row has a lead
   const auto fn = aligned ? fir_bf16x3_tc_kernel<false> : fir_bf16x3_tc_kernel<true>;
   cudaError_t e =
       cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bfSmemBytes(kBfMaxTaps));
   if (e != cudaSuccess) return e;
   const int nt = (a.outSize + kBfTile - 1) / kBfTile;
   const int tpr = a.tuneTpc > 0 ? (a.tuneTpc < nt ? a.tuneTpc : nt) : bfTilesPerRun(nt, a.batch);
   const long long runs = (long long) a.batch * ((nt + tpr - 1) / tpr);
   if (runs > INT_MAX) return cudaErrorInvalidValue;
   const int sms = deviceSms() > 0 ? deviceSms() : 148;
   fn<<<(int) std::min<long long>(runs, sms), kBfCta, smem, s>>>(a, tpr);
   countLaunch();
   return cudaGetLastError();
}

cudaError_t launchFirBf16x3Ragged(const RaggedChan *chans, const int4 *runs, int nRuns, const float *in,
                                  const float *taps, float *out, bool dx, int Tmax, int *err, cudaStream_t s)
{
   if (Tmax < 1 || Tmax > kBfMaxTaps) return cudaErrorNotSupported;
   if (nRuns <= 0) return cudaSuccess;
   const size_t smem = bfSmemBytes(Tmax);
   cudaError_t e =
       cudaFuncSetAttribute(fir_bf16x3_ragged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bfSmemBytes(kBfMaxTaps));
   if (e != cudaSuccess) return e;
   int sms = 148, dev = 0;
   if (cudaGetDevice(&dev) == cudaSuccess) (void) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
   const int grid = nRuns < sms ? nRuns : sms;
   fir_bf16x3_ragged_kernel<<<grid, kBfCta, smem, s>>>(chans, runs, nRuns, in, taps, out, dx ? 1 : 0, Tmax, err);
   countLaunch();
   return cudaGetLastError();
}

std::string firTuneKey(const FirLaunch &a, FirKernelKind kind)
{
   char buf[160];
   if (kind == FIR_F32_BF16X3 && firBf16x3Supported(a)) {
      const int nt = (a.outSize + kBfTile - 1) / kBfTile;
      snprintf(buf, sizeof(buf), "fir_bf16x3|T=%d|tiles=2^%d|batch=2^%d|nch=%d|sms=%d", a.T, tuneClass(nt),
               tuneClass(a.batch), a.filtPitch ? 1 : 0, deviceSms());
      return buf;
   }
   if ((kind == FIR_INT_WRAP_TC || kind == FIR_INT_Q_TC) && firIntTcSupported(a)) {
      const int nt = (a.outSize + kIntTuneTile - 1) / kIntTuneTile;
      snprintf(buf, sizeof(buf), "fir_int|dtype=%d|q=%d|T=%d|tiles=2^%d|batch=2^%d|sms=%d", a.dtype,
               kind == FIR_INT_Q_TC ? 1 : 0, a.T, tuneClass(nt), tuneClass(a.batch), deviceSms());
      return buf;
   }
   return std::string();
}

// bf16x3: the choice is the tiles per CTA; int: tiles per run (0: the built-in even split) * 16 +
// CTAs per SM.
std::vector<int> firTuneCandidates(const FirLaunch &a, FirKernelKind kind)
{
   std::vector<int> c;
   if (firTuneKey(a, kind).empty()) return c;
   // tiles per CTA: powers of two up to a whole channel, and the built-in rule's value
   auto tileCounts = [](int nt, int rule) {
      std::vector<int> t;
      for (int v = 1; v < nt && v <= 64; v *= 2) t.push_back(v);
      t.push_back(nt < 64 ? nt : 64);
      t.push_back(rule);
      return t;
   };
   if (kind == FIR_F32_BF16X3) {
      const int nt = (a.outSize + kBfTile - 1) / kBfTile;
      c = tileCounts(nt, bfTilesPerRun(nt, a.batch));
   }
   else {
      const int nt = (a.outSize + kIntTuneTile - 1) / kIntTuneTile;
      const int bound = a.dtype == DSPLIB_INT16 ? intLaunchBound<int16_t>() : intLaunchBound<int8_t>();
      for (int t : tileCounts(nt, 0))
         for (int per = 4; per <= bound; per += 2) c.push_back(t * 16 + per);
   }
   std::sort(c.begin(), c.end());
   c.erase(std::unique(c.begin(), c.end()), c.end());
   return c;
}

void firApplyChoice(FirLaunch &a, FirKernelKind kind, int choice)
{
   if (choice <= 0) return;
   if (kind == FIR_F32_BF16X3) a.tuneTpc = choice;
   else if (kind == FIR_INT_WRAP_TC || kind == FIR_INT_Q_TC) {
      a.tuneTpc = choice / 16;
      a.tunePerSm = choice % 16;
   }
}

cudaError_t launchFirDhBf16x3Ragged(const RaggedChan *chans, const int4 *runs, int nRuns, const float *x,
                                    const float *gu, float *part, int *err, cudaStream_t s)
{
   if (nRuns <= 0) return cudaSuccess;
   cudaError_t e =
       cudaFuncSetAttribute(fir_dh_bf16x3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kDhSmem);
   if (e != cudaSuccess) return e;
   const int sms = deviceSms() > 0 ? deviceSms() : 148;
   fir_dh_bf16x3_kernel<<<nRuns < sms ? nRuns : sms, kBfCta, kDhSmem, s>>>(chans, runs, nRuns, x, gu, part, err);
   countLaunch();
   return cudaGetLastError();
}


} // namespace dsplib
