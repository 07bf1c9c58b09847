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
// int8/int16 (kind::i8, P = 16, N = 16, tile 2048): an 8-bit core-matrix row
//   is 16 bytes = 16 samples, so the no-swizzle K-major descriptor with
//   LBO = 16 B and SBO = 128 B reads row a at byte 16a of the segment.
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
// All kernels are persistent: one wave of CTAs strides over runs of consecutive tiles of one
// channel.  The integer kernel keeps a band of shared taps for all of a CTA's runs
// and fetches each run's first segment during the previous run's last tile.
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

constexpr int kPhases = 16;
constexpr int kTile = kRows * kPhases;
constexpr int kThreads = 128;
constexpr int kMaxTapsTc = 2048;

__host__ __device__ inline int bandK(int T) { return ((T + 15 + 31) / 32) * 32; }

template <typename T> struct IntLimits;
template <> struct IntLimits<int8_t> { static constexpr long long lo = -128, hi = 127; };
template <> struct IntLimits<int16_t> { static constexpr long long lo = -32768, hi = 32767; };

// int8: |acc| <= 2048 * 2^14 fits 32 bits, so the output stage stays in 32-bit arithmetic.
template <int QMODE> __device__ __forceinline__ int8_t outStage8(int acc, int shift)
{
   if (!QMODE) return (int8_t) acc; // modulo 2^8
   if (shift > 0) acc = (acc + (1 << (shift - 1))) >> shift;
   return (int8_t) max(-128, min(127, acc));
}

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

template <typename T, int QMODE>
__device__ __forceinline__ T outStage(long long acc, int shift)
{
   if (!QMODE) return (T) acc; // modulo 2^bits
   if (shift > 0) acc = (acc + (1LL << (shift - 1))) >> shift;
   if (acc < IntLimits<T>::lo) acc = IntLimits<T>::lo;
   if (acc > IntLimits<T>::hi) acc = IntLimits<T>::hi;
   return (T) acc;
}

// One 16-byte vector (16 / sizeof(T) samples) of the segment starting at xs, the
// samples at or beyond `avail` read as zero: whole vectors load as one access, the one
// vector that straddles the row end element by element.
template <typename T> __device__ __forceinline__ int4 loadSegVec(const T *xs, long long k, long long avail)
{
   constexpr int per = 16 / sizeof(T);
   const long long s0 = k * per;
   if (s0 + per <= avail) return ((const int4 *) xs)[k];
   __align__(16) T tmp[per];
#pragma unroll
   for (int e = 0; e < per; e++) tmp[e] = (s0 + e < avail) ? xs[s0 + e] : (T) 0;
   return *(const int4 *) tmp;
}

// Write one 16-byte vector of samples into the byte plane(s): int8 -> A0; int16 ->
// A0 = high (signed) bytes, A1 = low (unsigned) bytes.
template <typename T>
__device__ __forceinline__ void putSegVec(const int4 &v, int k, unsigned char *A0, unsigned char *A1)
{
   if (sizeof(T) == 1) {
      ((int4 *) A0)[k] = v;
   }
   else {
      const int16_t *e = (const int16_t *) &v;
      __align__(8) unsigned char hb[8], lb[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
         hb[i] = (unsigned char) (e[i] >> 8);
         lb[i] = (unsigned char) (e[i] & 0xFF);
      }
      ((uint2 *) A0)[k] = *(uint2 *) hb;
      ((uint2 *) A1)[k] = *(uint2 *) lb;
   }
}

// Stage seg samples of xs (row positions j0 .. j0 + seg - 1, zero from inExtent on) into
// the byte plane(s).  16-byte vectors when xs is aligned, samples otherwise.
template <typename T>
__device__ __forceinline__ void intStage(const T *xs, long long j0, long long inExtent, int seg, unsigned char *A0,
                                         unsigned char *A1, int tid)
{
   constexpr bool SPLIT = sizeof(T) == 2;
   constexpr int per = 16 / sizeof(T); // samples per 16-byte vector
   const long long avail = inExtent - j0;
   if ((((uintptr_t) xs) & 15) == 0) {
      for (int k = tid; k < seg / per; k += kThreads) putSegVec<T>(loadSegVec<T>(xs, k, avail), k, A0, A1);
   }
   else {
      for (int k = tid; k < seg; k += kThreads) {
         const int v = (k < avail) ? (int) xs[k] : 0;
         if (SPLIT) {
            A0[k] = (unsigned char) (v >> 8);
            A1[k] = (unsigned char) (v & 0xFF);
         }
         else {
            A0[k] = (unsigned char) v;
         }
      }
   }
}

// Write n consecutive outputs dst[0..n) of one tile from shared memory, where
// the tile's 16-byte chunk ci (bytes 16ci .. 16ci+15 of the output run) sits at
// byte offset cpos(ci) of stage.  The accumulator drain leaves one output row
// per lane, so storing straight from registers would make every lane of a warp
// hit a different row (one memory transaction per lane and instruction); from
// shared memory a warp writes contiguous 16-byte vectors instead.  The vectors
// are aligned to the destination: when dst is not 16-byte aligned (row pitches
// such as N - T + 1 elements), each vector is assembled from two stage chunks
// with a funnel shift, and a head and tail of scalar stores cover the ends.
template <typename T, typename ChunkPos>
__device__ __forceinline__ void storeTile(T *dst, int n, const unsigned char *stage, ChunkPos cpos, int tid,
                                          int nthreads)
{
   auto elem = [&](int k) {
      const int byte = k * (int) sizeof(T);
      return *(const T *) (stage + cpos(byte >> 4) + (byte & 15));
   };
   const int hb = (16 - (int) ((uintptr_t) dst & 15)) & 15; // bytes before the first 16-byte boundary
   const int head = min(n, hb / (int) sizeof(T));
   const int nvec = (n - head) * (int) sizeof(T) / 16;
   if (tid < head) dst[tid] = elem(tid);
   const int q = hb >> 2, r = (hb & 3) * 8;
   unsigned char *dv = (unsigned char *) dst + hb;
   for (int v = tid; v < nvec; v += nthreads) {
      const uint4 a = *(const uint4 *) (stage + cpos(v));
      uint4 o = a;
      if (hb) {
         const uint4 b = *(const uint4 *) (stage + cpos(v + 1));
         uint32_t w0, w1, w2, w3, w4;
         switch (q) { // uniform across the CTA
         case 0: w0 = a.x, w1 = a.y, w2 = a.z, w3 = a.w, w4 = b.x; break;
         case 1: w0 = a.y, w1 = a.z, w2 = a.w, w3 = b.x, w4 = b.y; break;
         case 2: w0 = a.z, w1 = a.w, w2 = b.x, w3 = b.y, w4 = b.z; break;
         default: w0 = a.w, w1 = b.x, w2 = b.y, w3 = b.z, w4 = b.w; break;
         }
         o.x = __funnelshift_r(w0, w1, r);
         o.y = __funnelshift_r(w1, w2, r);
         o.z = __funnelshift_r(w2, w3, r);
         o.w = __funnelshift_r(w3, w4, r);
      }
      *(uint4 *) (dv + 16 * v) = o;
   }
   for (int k = head + nvec * (16 / (int) sizeof(T)) + tid; k < n; k += nthreads) dst[k] = elem(k);
}

template <typename T, int QMODE>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 2 ? 6 : 8) fir_int_tc_kernel(FirLaunch a, int tilesPerCta)
{
   constexpr bool SPLIT = sizeof(T) == 2;
   constexpr uint32_t kCols = SPLIT ? 64 : 32; // TMEM columns (accumulators of 16 columns each)
   const int T_ = a.T;
   const int Kt = bandK(T_);
   const int seg = kTile + Kt;            // samples one tile reads (multiple of 32)
   const int nplane = SPLIT ? 2 : 1;
   extern __shared__ __align__(128) unsigned char sm[];
   uint64_t *mbar = (uint64_t *) sm;
   uint32_t *tslot = (uint32_t *) (sm + 8);
   // Reversed taps g[c] = h[T-1-c] as bytes (int16: high and low byte planes) at
   // byte 16 + c of gb0 / gb1, zero elsewhere: one 32-bit word per thread to build.
   const int gbWords = (Kt + 20) / 4;
   uint32_t *gb0 = (uint32_t *) (sm + 16);
   uint32_t *gb1 = gb0 + gbWords;
   unsigned char *B0 = sm + 16 + ((gbWords * 4 * nplane + 15) & ~15);
   unsigned char *B1 = B0 + (size_t) Kt * 16;
   unsigned char *Abase = B0 + (size_t) Kt * 16 * nplane;
   // A[buf][plane]: seg bytes each
   auto A = [&](int buf, int plane) { return Abase + (size_t) (buf * nplane + plane) * seg; };
   T *ostage = (T *) (Abase + (size_t) 2 * nplane * seg); // one tile of outputs, row-major

   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   if (warp == 0) tc::tmemAlloc(tslot, kCols);
   if (tid == 0) tc::mbarInit(mbar, 1);
   tc::fenceBeforeSync();
   __syncthreads();
   tc::fenceAfterSync();
   const uint32_t tmem = *tslot;

   const int nt = (a.outSize + kTile - 1) / kTile;
   const long long inExtent = (long long) a.outSize + T_ - 1;
   // Work item = tiles [part * tilesPerCta, ...) of one channel; CTAs stride over the items
   // (persistent: the taps band of shared taps is built once per CTA, and each item's first
   // segment is fetched during the previous item's last tile).
   const int nParts = (nt + tilesPerCta - 1) / tilesPerCta;
   const long long nItems = (long long) a.batch * nParts;
   uint32_t iter = 0;
   bool failed = false;
   int bandOf = -1; // channel whose taps the band holds
   int buf = 0;
   long long item = blockIdx.x;
   if (item < nItems) {
      const int l = (int) (item / nParts), t0 = (int) (item % nParts) * tilesPerCta;
      intStage<T>((const T *) a.x + (long long) l * a.inPitch + (long long) t0 * kTile, (long long) t0 * kTile,
                  inExtent, seg, A(0, 0), A(0, 1), tid);
   }
   for (; item < nItems && !failed; item += gridDim.x) {
      const int l = (int) (item / nParts);
      const int t0 = (int) (item % nParts) * tilesPerCta;
      const int t1 = min(nt, t0 + tilesPerCta);
      const T *x = (const T *) a.x + (long long) l * a.inPitch;
      T *y = (T *) a.y + (long long) l * a.outPitch;
      if (bandOf < 0 || (a.filtPitch != 0 && bandOf != l)) {
         const T *h = (const T *) a.h + (long long) l * a.filtPitch;
         __syncthreads(); // the previous band's last MMAs are complete (waited) before it changes
         for (int wd = tid; wd < gbWords; wd += kThreads) {
            uint32_t w0 = 0, w1 = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
               const int c = 4 * wd + j - 16;
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
         // Taps band, K-major no-swizzle: 16-byte chunk ch = 16q + 8i + r (byte 16 ch) holds
         // B[m = 16q + e][b = 8i + r] = g[16q + e - 8i - r], e < 16: bytes gb[16 + 16q - 8i - r + e],
         // gathered from five words with funnel shifts.
         for (int ch = tid; ch < Kt; ch += kThreads) {
            const int base = 16 + 16 * (ch >> 4) - 8 * ((ch >> 3) & 1) - (ch & 7);
            const int w = base >> 2, sh = (base & 3) * 8;
#pragma unroll
            for (int pl = 0; pl < (SPLIT ? 2 : 1); pl++) {
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
         bandOf = l;
      }
      for (int t = t0; t < t1; t++) {
         const long long j0 = (long long) t * kTile;
         tc::fenceProxyAsync();
         __syncthreads(); // segment[buf] and band written; previous accumulators drained
         if (tid == 0) {
            tc::fenceAfterSync();
            const uint32_t a0 = tc::smemAddr(A(buf, 0)), a1 = tc::smemAddr(A(buf, 1));
            const uint32_t b0 = tc::smemAddr(B0), b1 = tc::smemAddr(B1);
            for (int kk = 0; kk < Kt / 32; kk++) {
               const uint64_t dA0 = tc::descNoSwizzle(a0 + 32 * kk, 16, 128);
               const uint64_t dB0 = tc::descNoSwizzle(b0 + 512 * kk, 256, 128);
               if (!SPLIT) {
                  tc::mmaI8(tmem, dA0, dB0, tc::idesc(2, 1, 1, kRows, kPhases), kk > 0);
               }
               else {
                  const uint64_t dA1 = tc::descNoSwizzle(a1 + 32 * kk, 16, 128);
                  const uint64_t dB1 = tc::descNoSwizzle(b1 + 512 * kk, 256, 128);
                  if (QMODE) tc::mmaI8(tmem, dA0, dB0, tc::idesc(2, 1, 1, kRows, kPhases), kk > 0); // hi*hi
                  tc::mmaI8(tmem + 16, dA0, dB1, tc::idesc(2, 1, 0, kRows, kPhases), kk > 0);       // hi*lo
                  tc::mmaI8(tmem + 16, dA1, dB0, tc::idesc(2, 0, 1, kRows, kPhases), true);         // lo*hi
                  tc::mmaI8(tmem + 32, dA1, dB1, tc::idesc(2, 0, 0, kRows, kPhases), kk > 0);       // lo*lo
               }
            }
            tc::commit(mbar);
         }
         // Fetch the next segment (this item's next tile, or the next item's first) into
         // registers now; it is written to shared memory after this tile's drain, so the
         // load latency hides behind the MMAs and the drain.
         constexpr int kPre = SPLIT ? 5 : 3; // 16-byte vectors per thread: (2048 + 2080) * sizeof(T) / 16 / 128
         int4 pre[kPre];
         const T *xn = nullptr;
         long long jn = 0;
         if (t + 1 < t1) {
            xn = x;
            jn = j0 + kTile;
         }
         else if (item + gridDim.x < nItems) {
            const long long ni = item + gridDim.x;
            xn = (const T *) a.x + (long long) (ni / nParts) * a.inPitch;
            jn = (long long) (ni % nParts) * tilesPerCta * kTile;
         }
         const bool preVec = xn != nullptr && ((((uintptr_t) (xn + jn)) & 15) == 0);
         const int nvec = seg * (int) sizeof(T) / 16;
         if (preVec) {
#pragma unroll
            for (int i = 0; i < kPre; i++) {
               const int k = tid + i * kThreads;
               if (k < nvec) pre[i] = loadSegVec<T>(xn + jn, k, inExtent - jn);
            }
         }
         const bool done = tc::mbarWait(mbar, iter & 1);
         if (!done && tid == 0) raiseError(a.err);
         failed = __syncthreads_or(!done) != 0;
         iter++;
         tc::fenceAfterSync();
         if (!failed) {
            // Drain: warp w owns TMEM lanes 32w..32w+31 = rows a; 16 consecutive outputs per row.
            const uint32_t lanes = (uint32_t) (warp * 32) << 16;
            uint32_t acc[3][16];
            tc::tmemLoad16(tmem + lanes, acc[0]);
            if (SPLIT) {
               tc::tmemLoad16(tmem + lanes + 16, acc[1]);
               tc::tmemLoad16(tmem + lanes + 32, acc[2]);
            }
            tc::tmemWaitLoad();
            const int row = warp * 32 + lane;
            __align__(16) T out[16];
            if (SPLIT && QMODE) {
               uint32_t w[8];
#pragma unroll
               for (int b = 0; b < 16; b += 2) {
                  const long long v0 = ((long long) (int) acc[0][b] << 16) + ((long long) (int) acc[1][b] << 8) +
                                       (long long) (int) acc[2][b];
                  const long long v1 = ((long long) (int) acc[0][b + 1] << 16) +
                                       ((long long) (int) acc[1][b + 1] << 8) + (long long) (int) acc[2][b + 1];
                  w[b / 2] = outStage16x2(v0, v1, a.shift);
               }
               *(uint4 *) &out[0] = make_uint4(w[0], w[1], w[2], w[3]);
               *(uint4 *) &out[8] = make_uint4(w[4], w[5], w[6], w[7]);
            }
            if (!SPLIT && QMODE) {
               uint4 w;
               w.x = outStage8x4((int) acc[0][0], (int) acc[0][1], (int) acc[0][2], (int) acc[0][3], a.shift);
               w.y = outStage8x4((int) acc[0][4], (int) acc[0][5], (int) acc[0][6], (int) acc[0][7], a.shift);
               w.z = outStage8x4((int) acc[0][8], (int) acc[0][9], (int) acc[0][10], (int) acc[0][11], a.shift);
               w.w = outStage8x4((int) acc[0][12], (int) acc[0][13], (int) acc[0][14], (int) acc[0][15], a.shift);
               *(uint4 *) &out[0] = w;
            }
#pragma unroll
            for (int b = 0; b < 16; b++) {
               long long v;
               if (!SPLIT) {
                  if (!QMODE) out[b] = (T) outStage8<QMODE>((int) acc[0][b], a.shift);
                  continue;
               }
               if (QMODE) continue; // packed above
               v = (long long) (int) (((uint32_t) acc[1][b] << 8) + (uint32_t) acc[2][b]);
               out[b] = outStage<T, QMODE>(v, a.shift);
            }
            int4 *os = (int4 *) (ostage + row * kPhases);
            os[0] = *(int4 *) &out[0];
            if (SPLIT) os[1] = *(int4 *) &out[8];
         }
         tc::fenceBeforeSync();
         if (failed) break;
         __syncthreads(); // the output tile is complete in shared memory
         storeTile<T>(y + j0, (int) min((long long) kTile, (long long) a.outSize - j0),
                      (const unsigned char *) ostage, [](int ci) { return ci * 16; }, tid, kThreads);
         if (preVec) {
            unsigned char *N0 = A(buf ^ 1, 0), *N1 = A(buf ^ 1, 1);
#pragma unroll
            for (int i = 0; i < kPre; i++) {
               const int k = tid + i * kThreads;
               if (k < nvec) putSegVec<T>(pre[i], k, N0, N1);
            }
         }
         else if (xn != nullptr) {
            intStage<T>(xn + jn, jn, inExtent, seg, A(buf ^ 1, 0), A(buf ^ 1, 1), tid); // unaligned row
         }
         buf ^= 1;
      }
   }
   __syncthreads();
   if (warp == 0) tc::tmemFree(tmem, kCols);
}

// Tiles per CTA (the built-in rule, when the autotuner has no entry): a whole channel
// when there are enough channels to fill the GPU several times over, else split so that
// at least ~2 waves of CTAs exist.
inline int tilesPerCtaFor(int nt, int batch, int ctasPerSm)
{
   const long long sms = deviceSms() > 0 ? deviceSms() : 148;
   int tpc = nt;
   while (tpc > 1 && (long long) ((nt + tpc - 1) / tpc) * batch < sms * ctasPerSm * 2) tpc = (tpc + 1) / 2;
   return tpc;
}

template <typename T> constexpr int intLaunchBound() { return sizeof(T) == 2 ? 6 : 8; }

template <typename T, int QMODE> cudaError_t launchIntTc(const FirLaunch &a, cudaStream_t s)
{
   constexpr bool SPLIT = sizeof(T) == 2;
   const int Kt = bandK(a.T);
   const int nplane = SPLIT ? 2 : 1;
   const size_t gbBytes = (size_t) ((Kt + 20) / 4) * 4 * nplane;
   const size_t smem = 16 + ((gbBytes + 15) & ~(size_t) 15) + (size_t) Kt * 16 * nplane +
                       2 * (size_t) nplane * (kTile + Kt) + (size_t) kTile * sizeof(T);
   auto fn = fir_int_tc_kernel<T, QMODE>;
   cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
   if (e != cudaSuccess) return e;
   const int nt = (a.outSize + kTile - 1) / kTile;
   const int tpc = a.tuneTpc > 0 ? (a.tuneTpc < nt ? a.tuneTpc : nt) : tilesPerCtaFor(nt, a.batch, 8);
   const long long items = (long long) a.batch * ((nt + tpc - 1) / tpc);
   // persistent: one wave of resident CTAs striding over the work items (CTAs per SM: the
   // autotuner's choice or the launch bound, fewer when shared memory runs out first)
   const int bySmem = (int) ((228u * 1024u) / (smem + 1024u));
   const int want = a.tunePerSm > 0 ? a.tunePerSm : intLaunchBound<T>();
   const int perSm = want < bySmem ? want : bySmem;
   const int sms = deviceSms() > 0 ? deviceSms() : 148;
   const long long wave = (long long) (perSm > 0 ? perSm : 1) * sms;
   const int grid = (int) (items < wave ? items : wave);
   FirLaunch k = a;
   // int8: |acc| <= 2048 * 2^14 = 2^25, so every shift from 27 up rounds to zero, as 31
   // (the largest the 32-bit output stage can take) does.
   if (!SPLIT && k.shift > 31) k.shift = 31;
   fn<<<grid, kThreads, smem, s>>>(k, tpc);
   countLaunch();
   return cudaGetLastError();
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
static_assert(bfSmemBytes(kBfMaxTaps) <= 227 * 1024, "two plane sets and two of the longest bands fit");

struct BfSmem {
   uint64_t *mmaDone, *planesFull, *accFree; // one per plane set / accumulator
   uint64_t *rawFull, *rawFree;              // one per raw slot
   uint64_t *edges;                          // the split warps have written a raw tile's edges
   uint32_t *tslot;
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
// FULL of its up to GROUPS groups need no test.
template <int FULL, int GROUPS>
__device__ __forceinline__ void bfSplit(const float *raw, int nQuad, unsigned char *hi, unsigned char *lo, int tid)
{
   const int k = tid >> 4, off = k * 128 + ((((tid >> 1) & 7) ^ (k & 7)) << 4) + (tid & 1) * 8;
   const float4 *src = (const float4 *) raw + tid;
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
         }
   }
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
// and leaves, and the others follow as theirs give up.
template <typename Get>
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
            if (blocks >= kRows) bfSplit<kRows * 16 / kBfSplitThreads, kBfQuads>(L.slot(b), blocks * 16, L.hi(b), L.lo(b), tid);
            else bfSplit<0, kBfQuads>(L.slot(b), blocks * 16, L.hi(b), L.lo(b), tid);
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
__global__ void __launch_bounds__(kBfCta, 1) fir_bf16x3_tc_kernel(FirLaunch a, int tilesPerRun)
{
   extern __shared__ __align__(16) unsigned char smraw[];
   const int nt = (a.outSize + kBfTile - 1) / kBfTile;
   const int parts = (nt + tilesPerRun - 1) / tilesPerRun;
   bfPipeline(bfSmemLayout(smraw, a.T), a.batch * parts, a.err, [&](int i) {
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
   bfPipeline(bfSmemLayout(smraw, Tmax), nRuns, err, [&](int i) {
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
   cudaError_t e =
       cudaFuncSetAttribute(fir_bf16x3_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
   if (e != cudaSuccess) return e;
   const int nt = (a.outSize + kBfTile - 1) / kBfTile;
   const int tpr = a.tuneTpc > 0 ? (a.tuneTpc < nt ? a.tuneTpc : nt) : bfTilesPerRun(nt, a.batch);
   const long long runs = (long long) a.batch * ((nt + tpr - 1) / tpr);
   if (runs > INT_MAX) return cudaErrorInvalidValue;
   const int sms = deviceSms() > 0 ? deviceSms() : 148;
   fir_bf16x3_tc_kernel<<<(int) std::min<long long>(runs, sms), kBfCta, smem, s>>>(a, tpr);
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
       cudaFuncSetAttribute(fir_bf16x3_ragged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
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
      const int nt = (a.outSize + kTile - 1) / kTile;
      snprintf(buf, sizeof(buf), "fir_int|dtype=%d|q=%d|T=%d|tiles=2^%d|batch=2^%d|sms=%d", a.dtype,
               kind == FIR_INT_Q_TC ? 1 : 0, a.T, tuneClass(nt), tuneClass(a.batch), deviceSms());
      return buf;
   }
   return std::string();
}

// bf16x3: the choice is the tiles per CTA; int: tiles per CTA * 16 + CTAs per SM.
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
      const int nt = (a.outSize + kTile - 1) / kTile;
      const int bound = a.dtype == DSPLIB_INT16 ? intLaunchBound<int16_t>() : intLaunchBound<int8_t>();
      for (int t : tileCounts(nt, tilesPerCtaFor(nt, a.batch, 8)))
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
