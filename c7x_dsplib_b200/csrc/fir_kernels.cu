// FIR CUDA kernels for sm_100a.
//
//   fir_direct_kernel  one output per thread per tile, taps in shared memory.
//                      MODE_NATC reproduces the reference natural-C kernel
//                      (src/DSPLIB_fir/DSPLIB_fir_cn.cpp:54-83) bit for bit:
//                      integers wrap modulo 2^32 before the truncating store
//                      (the reference sums modulo 2^bits; 2^bits divides 2^32),
//                      floats are summed in tap order with separately rounded
//                      multiply and add.  MODE_Q keeps the exact accumulator
//                      and applies round-half-up / shift / saturate.
//   fir_f32_simt_kernel the plain FP32 CUDA-core kernel: 8 consecutive outputs and
//                      the 8 half a tile further per thread as packed pairs in
//                      registers, taps unrolled by 8, packed fused multiply-add.
//   fir_f32_few_kernel  the same arithmetic for few outputs of many taps: the taps
//                      split over groups of threads and the CTAs of a cluster.
//
// Layout (channel-major, DSPLIB_fir_cn.cpp:57-58): x[l*inPitch + t],
// y[l*outPitch + j]; stored taps h[T-1-c] multiply x[j+c].
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "dsplib_internal.h"
#include "scan_common.cuh"

namespace cg = cooperative_groups;

namespace dsplib {

namespace {

constexpr int MODE_NATC = 0;
constexpr int MODE_Q = 1;

template <typename T> struct QLimits;
template <> struct QLimits<int8_t> { static constexpr long long lo = -128, hi = 127; };
template <> struct QLimits<int16_t> { static constexpr long long lo = -32768, hi = 32767; };
template <> struct QLimits<int32_t> { static constexpr long long lo = -2147483648LL, hi = 2147483647LL; };

template <typename T, int MODE> struct Acc;
template <> struct Acc<float, MODE_NATC> {
   float v = 0.0f;
   __device__ void add(float x, float h) { v = __fadd_rn(v, __fmul_rn(x, h)); }
   __device__ float out(int) const { return v; }
};
template <typename T> struct Acc<T, MODE_NATC> {
   uint32_t v = 0;
   __device__ void add(T x, T h) { v += (uint32_t) (int32_t) x * (uint32_t) (int32_t) h; }
   __device__ T out(int) const { return (T) v; }
};
template <typename T> struct Acc<T, MODE_Q> {
   // int8/int16 products fit 31 bits; 2^32 taps would still fit int64.  int32
   // products need 63 bits, so that case accumulates in 128 bits.
   using W = typename std::conditional<sizeof(T) == 4, __int128, long long>::type;
   W v = 0;
   __device__ void add(T x, T h) { v += (W) x * (W) h; }
   __device__ T out(int shift) const
   {
      W r = v;
      if (shift > 0) r = (r + ((W) 1 << (shift - 1))) >> shift;
      if (r < (W) QLimits<T>::lo) r = (W) QLimits<T>::lo;
      if (r > (W) QLimits<T>::hi) r = (W) QLimits<T>::hi;
      return (T) r;
   }
};

constexpr int kDirTile = 1024; // outputs per CTA
constexpr int kDirTaps = 1024; // taps per shared-memory block
constexpr int kDirThreads = 256;

template <typename T, int MODE>
__global__ void __launch_bounds__(kDirThreads) fir_direct_kernel(FirLaunch a)
{
   __shared__ T xs[kDirTile + kDirTaps];
   __shared__ T hs[kDirTaps];
   const int j0 = blockIdx.x * kDirTile;
   const long long inExtent = (long long) a.outSize + a.T - 1; // samples of a row that are read
   for (int l = blockIdx.y; l < a.batch; l += gridDim.y) {
      const T *x = (const T *) a.x + (long long) l * a.inPitch;
      const T *h = (const T *) a.h + (long long) l * a.filtPitch;
      T *y = (T *) a.y + (long long) l * a.outPitch;
      Acc<T, MODE> acc[kDirTile / kDirThreads];
      for (int cb = 0; cb < a.T; cb += kDirTaps) {
         const int tb = min(kDirTaps, a.T - cb);
         for (int k = threadIdx.x; k < kDirTile + tb - 1; k += kDirThreads) {
            long long idx = (long long) j0 + cb + k;
            xs[k] = idx < inExtent ? x[idx] : (T) 0;
         }
         for (int k = threadIdx.x; k < tb; k += kDirThreads) hs[k] = h[a.T - 1 - (cb + k)];
         __syncthreads();
#pragma unroll
         for (int r = 0; r < kDirTile / kDirThreads; r++) {
            const int j = threadIdx.x + r * kDirThreads;
            if (j0 + j < a.outSize) {
               for (int c = 0; c < tb; c++) acc[r].add(xs[j + c], hs[c]);
            }
         }
         __syncthreads();
      }
#pragma unroll
      for (int r = 0; r < kDirTile / kDirThreads; r++) {
         const int j = threadIdx.x + r * kDirThreads;
         if (j0 + j < a.outSize) y[j0 + j] = acc[r].out(a.shift);
      }
   }
}

// FLOAT32 filters in Q mode (InitArgs.enableQ): the C7x fixed-point MMA path of
// src/DSPLIB_fir/DSPLIB_fir_ci.cpp:1559-1625.  Signal and taps are scaled by 2^Q and
// converted to int32 (round to nearest even, saturating; NaN -> 0), the products are
// summed exactly (128 bits), the sum is shifted right by Q with half-LSB rounding and
// saturated to int32 (the MMA output stage, X_SHIFT = Q with rounding and saturation),
// then converted to float and scaled by 2^-Q.
__device__ __forceinline__ int quantQ(float v, float scale) { return __float2int_rn(v * scale); }

__global__ void __launch_bounds__(kDirThreads) fir_floatq_kernel(FirLaunch a)
{
   __shared__ int xs[kDirTile + kDirTaps];
   __shared__ int hs[kDirTaps];
   const int j0 = blockIdx.x * kDirTile;
   const long long inExtent = (long long) a.outSize + a.T - 1;
   const int Q = a.shift;
   const float scale = ldexpf(1.0f, Q), unscale = ldexpf(1.0f, -Q);
   for (int l = blockIdx.y; l < a.batch; l += gridDim.y) {
      const float *x = (const float *) a.x + (long long) l * a.inPitch;
      const float *h = (const float *) a.h + (long long) l * a.filtPitch;
      float *y = (float *) a.y + (long long) l * a.outPitch;
      __int128 acc[kDirTile / kDirThreads];
#pragma unroll
      for (int r = 0; r < kDirTile / kDirThreads; r++) acc[r] = 0;
      for (int cb = 0; cb < a.T; cb += kDirTaps) {
         const int tb = min(kDirTaps, a.T - cb);
         for (int k = threadIdx.x; k < kDirTile + tb - 1; k += kDirThreads) {
            long long idx = (long long) j0 + cb + k;
            xs[k] = idx < inExtent ? quantQ(x[idx], scale) : 0;
         }
         for (int k = threadIdx.x; k < tb; k += kDirThreads) hs[k] = quantQ(h[a.T - 1 - (cb + k)], scale);
         __syncthreads();
#pragma unroll
         for (int r = 0; r < kDirTile / kDirThreads; r++) {
            const int j = threadIdx.x + r * kDirThreads;
            if (j0 + j < a.outSize)
               for (int c = 0; c < tb; c++) acc[r] += (__int128) ((long long) xs[j + c] * (long long) hs[c]);
         }
         __syncthreads();
      }
#pragma unroll
      for (int r = 0; r < kDirTile / kDirThreads; r++) {
         const int j = threadIdx.x + r * kDirThreads;
         if (j0 + j < a.outSize) {
            __int128 v = acc[r];
            if (Q > 0) v = (v + ((__int128) 1 << (Q - 1))) >> Q;
            if (v < (__int128) INT32_MIN) v = INT32_MIN;
            if (v > (__int128) INT32_MAX) v = INT32_MAX;
            y[j0 + j] = (float) (int) v * unscale;
         }
      }
   }
}

using scan::P2;
using scan::dup;
using scan::fma2;
using scan::pk;
using scan::up;

// Plain FP32 FIR.  A thread keeps 8 pairs (y[j], y[j + H]) of outputs, H half the tile, so that
// every multiply-add is a packed one (each half rounded as fmaf) on pairs (x[k], x[k + H]) kept
// interleaved in shared memory and taps stored twice.  The taps are added in ascending order.
// Bound by the FMA pipe: per 8 taps 64 packed multiply-adds (128 cycles of the pipe) against
// 8 vector loads (20 shared-memory cycles); with scalar multiply-adds the issue slots and the
// shared-memory reads (two-way conflicts) held the pipe at 40 %.  256 channels x 32768 samples x
// 255 taps: 145 -> 91 us (47 of the 67 TFLOP/s that packed multiply-adds alone reach).
constexpr int kSimtTile = 2048; // outputs per CTA, 16 per thread
constexpr int kSimtTaps = 256;  // taps per shared-memory block
constexpr int kSimtThreads = kSimtTile / 16;

// Pair k of a window: 8 pairs (64 bytes) and 16 bytes of padding, so that the vector loads of
// eight threads, 8 pairs apart, touch distinct banks.
__device__ __forceinline__ int pairAt(int k) { return k + (k >> 3) * 2; }
constexpr int pairsPadded(int n) { return n / 8 * 10; } // n a multiple of 8

// acc[r] += sum_{c < n} w[8 t + r + c] g[c] for the thread at w = window + pairAt(8 t); n a multiple
// of 8 (taps beyond the filter are zero), the window 8 pairs longer.
__device__ __forceinline__ void simtTaps(P2 (&acc)[8], const P2 *w, const P2 *g, int n)
{
   P2 v[16];
   auto load8 = [](P2 *d, const P2 *src) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
         const ulonglong2 u = *(const ulonglong2 *) (src + 2 * q);
         d[2 * q].v = u.x;
         d[2 * q + 1].v = u.y;
      }
   };
   load8(v, w);
#pragma unroll 2
   for (int c = 0; c < n; c += 8) {
      w += 10;
      P2 h[8];
      load8(v + 8, w);
      load8(h, g + c);
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
         for (int r = 0; r < 8; r++) acc[r] = fma2(v[r + i], h[i], acc[r]);
#pragma unroll
      for (int r = 0; r < 8; r++) v[r] = v[r + 8];
   }
}

__global__ void __launch_bounds__(kSimtThreads) fir_f32_simt_kernel(FirLaunch a)
{
   __shared__ __align__(16) P2 xs[pairsPadded(kSimtTile / 2 + kSimtTaps + 8)];
   __shared__ __align__(16) P2 gs[kSimtTaps];
   const int tid = threadIdx.x;
   const int j0 = blockIdx.x * kSimtTile;
   const int outs = min(kSimtTile, a.outSize - j0);
   const int H = ((outs + 1) / 2 + 7) & ~7; // a short tile is halved too
   const long long inExtent = (long long) a.outSize + a.T - 1;
   for (int l = blockIdx.y; l < a.batch; l += gridDim.y) {
      const float *x = (const float *) a.x + (long long) l * a.inPitch;
      const float *h = (const float *) a.h + (long long) l * a.filtPitch;
      float *y = (float *) a.y + (long long) l * a.outPitch + j0;
      P2 acc[8];
#pragma unroll
      for (int r = 0; r < 8; r++) acc[r] = dup(0.0f);
      for (int cb = 0; cb < a.T; cb += kSimtTaps) {
         const int tb = min(kSimtTaps, a.T - cb);
         const int tbr = (tb + 7) & ~7;
         const long long q0 = (long long) j0 + cb;
         for (int k = tid; k < H + tbr + 8; k += kSimtThreads) {
            const long long q = q0 + k;
            xs[pairAt(k)] = pk(q < inExtent ? x[q] : 0.0f, q + H < inExtent ? x[q + H] : 0.0f);
         }
         for (int k = tid; k < tbr; k += kSimtThreads) gs[k] = dup(k < tb ? h[a.T - 1 - (cb + k)] : 0.0f);
         __syncthreads();
         if (8 * tid < H) simtTaps(acc, xs + 10 * tid, gs, tbr);
         __syncthreads();
      }
      // the outputs through shared memory, so that the global stores are coalesced (rows of 8
      // padded to 9: distinct banks)
      float *os = (float *) xs;
      if (8 * tid < H) {
#pragma unroll
         for (int r = 0; r < 8; r++) {
            const float2 v = up(acc[r]);
            os[9 * tid + r] = v.x;
            os[9 * (tid + H / 8) + r] = v.y;
         }
      }
      __syncthreads();
      for (int k = tid; k < outs; k += kSimtThreads) y[k] = os[k + (k >> 3)];
      __syncthreads();
   }
}

// Few outputs of many taps (the taps gradient of an FIR layer is such a filter): one cluster of
// kFewCluster CTAs per channel, each a range of the taps, and in it groups of GT threads that
// hold all outputs (8 pairs a thread, up to 16 GT outputs) and take 64 taps in turn; the
// groups' sums and then the CTAs' are added in order through (distributed) shared memory, so
// results repeat bit for bit.  With the kernel above one CTA a channel ran all taps, 16 of 256
// threads on 128 outputs: 434 -> 16 us for 64 channels, 128 outputs, 16257 taps.
constexpr int kFewThreads = 128, kFewTaps = 64, kFewCluster = 8;

template <int GT> __global__ void __launch_bounds__(kFewThreads) fir_f32_few_kernel(FirLaunch a)
{
   constexpr int H = 8 * GT, Q = kFewThreads / GT, TB = Q * kFewTaps; // half tile, groups, taps per block
   constexpr int kWindow = pairsPadded(H + TB + 8), kSums = Q * 9 * GT; // pairs; the groups' sums reuse the window
   __shared__ __align__(16) P2 xs[kWindow > kSums ? kWindow : kSums];
   __shared__ __align__(16) P2 gs[TB];
   __shared__ float part[2 * H];
   float *red = (float *) xs; // [Q][9 * 2 GT]
   const int tid = threadIdx.x, grp = tid / GT, t = tid % GT;
   cg::cluster_group cl = cg::this_cluster();
   const int rank = (int) cl.block_rank(), K = (int) cl.num_blocks();
   const int l = blockIdx.y;
   const float *x = (const float *) a.x + (long long) l * a.inPitch;
   const float *h = (const float *) a.h + (long long) l * a.filtPitch;
   float *y = (float *) a.y + (long long) l * a.outPitch;
   const long long inExtent = (long long) a.outSize + a.T - 1;
   // this CTA's taps: whole blocks
   const int blocks = (a.T + TB - 1) / TB, per = (blocks + K - 1) / K;
   const int c1 = (int) min((long long) a.T, (long long) (rank + 1) * per * TB);
   P2 acc[8];
#pragma unroll
   for (int r = 0; r < 8; r++) acc[r] = dup(0.0f);
   for (long long cb = (long long) rank * per * TB; cb < c1; cb += TB) {
      const int tb = (int) min((long long) TB, c1 - cb);
      for (int k = tid; k < H + TB + 8; k += kFewThreads) {
         const long long q = cb + k;
         xs[pairAt(k)] = pk(q < inExtent ? x[q] : 0.0f, q + H < inExtent ? x[q + H] : 0.0f);
      }
      for (int k = tid; k < TB; k += kFewThreads) gs[k] = dup(k < tb ? h[a.T - 1 - (cb + k)] : 0.0f);
      __syncthreads();
      const int left = tb - grp * kFewTaps; // in steps of 8 taps, as the other kernel: no sample further off meets a zero tap
      if (left > 0)
         simtTaps(acc, xs + pairsPadded(grp * kFewTaps) + 10 * t, gs + grp * kFewTaps, min(kFewTaps, (left + 7) & ~7));
      __syncthreads();
   }
#pragma unroll
   for (int r = 0; r < 8; r++) {
      const float2 v = up(acc[r]);
      red[grp * (18 * GT) + 9 * t + r] = v.x;
      red[grp * (18 * GT) + 9 * (t + GT) + r] = v.y;
   }
   __syncthreads();
   for (int o = tid; o < 2 * H; o += kFewThreads) {
      float v = 0.0f;
      for (int q = 0; q < Q; q++) v += red[q * (18 * GT) + o + (o >> 3)];
      part[o] = v;
   }
   cl.sync();
   for (int o = rank * kFewThreads + tid; o < a.outSize; o += K * kFewThreads) {
      float v = 0.0f;
      for (int d = 0; d < K; d++) v += cl.map_shared_rank(part, d)[o];
      y[o] = v;
   }
   cl.sync(); // no CTA leaves while others read its sums
}

template <int GT> cudaError_t launchFew(const FirLaunch &a, cudaStream_t s)
{
   for (int l0 = 0; l0 < a.batch; l0 += 65535) {
      FirLaunch b = a;
      b.x = (const float *) a.x + (long long) l0 * a.inPitch;
      b.h = (const float *) a.h + (long long) l0 * a.filtPitch;
      b.y = (float *) a.y + (long long) l0 * a.outPitch;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(kFewCluster, a.batch - l0 < 65535 ? a.batch - l0 : 65535);
      cfg.blockDim = dim3(kFewThreads);
      cfg.stream = s;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = kFewCluster;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      const cudaError_t e = cudaLaunchKernelEx(&cfg, fir_f32_few_kernel<GT>, b);
      if (e != cudaSuccess) return e;
      countLaunch();
   }
   return cudaGetLastError();
}

// Up to 512 outputs of at least 1024 taps: the taps are split where one CTA a channel leaves SMs idle,
// or keeps most of its threads idle for long enough.  A split channel costs 8 CTAs (50 us a thousand
// channels up to 2048 taps), an undivided one its taps in turn.  In us, undivided / split, 128 outputs: up
// to two channels an SM, 150 of 1024 taps 19 / 13, 296 of 1024 19 / 21, of 1280 23 / 21; up to five, 700 of
// 1024 31 / 39, of 1280 39 / 39, of 1536 45 / 39; more, 1184 of 1536 51 / 63, 8000 of 2304 479 / 478, of 2560
// 529 / 485; with 512 outputs a block holds fewer taps: 1184 of 3072 102 / 120, of 4096 133 / 125.
bool firFewOutputs(const FirLaunch &a)
{
   const int sms = deviceSms() > 0 ? deviceSms() : 148;
   if (a.outSize > 512 || a.T < 1024) return false;
   if (a.batch <= 2 * sms) return true;
   if (a.batch <= 5 * sms) return a.T >= 1536;
   return a.T >= (a.outSize <= 256 ? 2560 : 4096);
}

template <typename T, int MODE> cudaError_t launchDirect(const FirLaunch &a, cudaStream_t s)
{
   dim3 grid((a.outSize + kDirTile - 1) / kDirTile, a.batch < 65535 ? a.batch : 65535);
   fir_direct_kernel<T, MODE><<<grid, kDirThreads, 0, s>>>(a);
   countLaunch();
   return cudaGetLastError();
}

} // namespace

cudaError_t launchFirBf16x3(const FirLaunch &a, cudaStream_t s);

cudaError_t launchFir(const FirLaunch &a, FirKernelKind kind, cudaStream_t s)
{
   if (a.batch <= 0 || a.outSize <= 0) return cudaSuccess;
   switch (kind) {
   case FIR_NATC:
      switch (a.dtype) {
      case DSPLIB_INT8: return launchDirect<int8_t, MODE_NATC>(a, s);
      case DSPLIB_INT16: return launchDirect<int16_t, MODE_NATC>(a, s);
      case DSPLIB_INT32: return launchDirect<int32_t, MODE_NATC>(a, s);
      case DSPLIB_FLOAT32: return launchDirect<float, MODE_NATC>(a, s);
      default: return cudaErrorInvalidValue;
      }
   case FIR_QMODE:
      switch (a.dtype) {
      case DSPLIB_INT8: return launchDirect<int8_t, MODE_Q>(a, s);
      case DSPLIB_INT16: return launchDirect<int16_t, MODE_Q>(a, s);
      case DSPLIB_INT32: return launchDirect<int32_t, MODE_Q>(a, s);
      default: return cudaErrorInvalidValue;
      }
   case FIR_F32_SIMT: {
      if (a.dtype != DSPLIB_FLOAT32) return cudaErrorInvalidValue;
      if (firFewOutputs(a)) {
         if (a.outSize <= 128) return launchFew<8>(a, s);
         if (a.outSize <= 256) return launchFew<16>(a, s);
         return launchFew<32>(a, s);
      }
      dim3 grid((a.outSize + kSimtTile - 1) / kSimtTile, a.batch < 65535 ? a.batch : 65535);
      fir_f32_simt_kernel<<<grid, kSimtThreads, 0, s>>>(a);
      countLaunch();
      return cudaGetLastError();
   }
   case FIR_F32_Q: {
      if (a.dtype != DSPLIB_FLOAT32 || a.shift < 0 || a.shift > kFirMaxFloatQ) return cudaErrorInvalidValue;
      dim3 grid((a.outSize + kDirTile - 1) / kDirTile, a.batch < 65535 ? a.batch : 65535);
      fir_floatq_kernel<<<grid, kDirThreads, 0, s>>>(a);
      countLaunch();
      return cudaGetLastError();
   }
   case FIR_F32_BF16X3:
      if (a.dtype != DSPLIB_FLOAT32) return cudaErrorInvalidValue;
      return launchFirBf16x3(a, s);
   case FIR_INT_WRAP_TC:
   case FIR_INT_Q_TC:
      if (!firIntTcSupported(a)) return cudaErrorInvalidValue;
      return launchFirIntTc(a, kind == FIR_INT_Q_TC, s);
   }
   return cudaErrorInvalidValue;
}

// ------------------------------------------------------------------ streaming window

// Advance the windows of a streaming filter, [hist | block] elements a channel: the last `hist`
// elements move to the front and the new block takes the place behind them.  Element i of the
// history is read, and the element that replaces it written, by one thread, and no other
// touches its two places (block >= hist), so nothing has to wait.  V elements a copy where the
// rows of `in` allow (a window's block starts on a 16-byte boundary).  Bound by its launch.
template <typename E, int V>
__global__ void __launch_bounds__(256) stream_window_kernel(char *win, long long pitch, const char *in,
                                                            long long inPitch, int channels, int hist, int block)
{
   const int body = block - hist, nv = body / V, items = hist + nv + (body - nv * V);
   for (int c = blockIdx.y; c < channels; c += gridDim.y) {
      E *w = (E *) (win + c * pitch);
      const E *x = (const E *) (in + c * inPitch);
      for (long long k = (long long) blockIdx.x * blockDim.x + threadIdx.x; k < items; k += (long long) gridDim.x * blockDim.x) {
         if (k < hist) {
            w[k] = w[block + k];
            w[block + k] = x[body + k];
         }
         else if (k - hist < nv) {
            const long long q = (k - hist) * V;
            if (V > 1) *(int4 *) (w + hist + q) = *(const int4 *) (x + q);
            else w[hist + q] = x[q];
         }
         else {
            const long long q = k - hist - nv + (long long) nv * V;
            w[hist + q] = x[q];
         }
      }
   }
}

cudaError_t launchStreamWindow(char *win, long long pitch, const void *in, long long inPitch, int channels, int hist,
                               int block, int elt, cudaStream_t s)
{
   const int V = 16 / elt;
   const bool wide = ((((uintptr_t) win + (size_t) hist * elt) | (uintptr_t) pitch | (uintptr_t) in | (uintptr_t) inPitch) & 15) == 0;
   const long long items = wide ? hist + (long long) (block - hist) / V + V - 1 : block;
   const dim3 grid((unsigned) std::min<long long>((items + 255) / 256, 1024), (unsigned) std::min(channels, 65535));
   auto go = [&](auto e) {
      using E = decltype(e);
      if (wide) stream_window_kernel<E, 16 / (int) sizeof(E)><<<grid, 256, 0, s>>>(win, pitch, (const char *) in, inPitch, channels, hist, block);
      else stream_window_kernel<E, 1><<<grid, 256, 0, s>>>(win, pitch, (const char *) in, inPitch, channels, hist, block);
   };
   if (elt == 1) go((uint8_t) 0);
   else if (elt == 2) go((uint16_t) 0);
   else if (elt == 4) go((uint32_t) 0);
   else return cudaErrorInvalidValue;
   countLaunch();
   return cudaGetLastError();
}

// ------------------------------------------------------------------ adjoint

// The operands of the two filters of the adjoint, from rows gy [batch, M] and h [rows, T]
// (M = N - T + 1): gy with T - 1 zeros on both sides, the taps reversed, gy reversed.
__global__ void __launch_bounds__(256) fir_adjoint_operands_kernel(const float *gy, const float *h, float *wide, float *hrev,
                                                                   float *grev, int batch, int rows, int M, int T)
{
   const long long W = M + 2LL * (T - 1);
   const long long nw = wide ? batch * W : 0, nh = wide ? (long long) rows * T : 0, ng = grev ? (long long) batch * M : 0;
   for (long long k = (long long) blockIdx.x * blockDim.x + threadIdx.x; k < nw + nh + ng; k += (long long) gridDim.x * blockDim.x) {
      if (k < nw) {
         const long long l = k / W, j = k - l * W - (T - 1);
         wide[k] = j >= 0 && j < M ? gy[l * M + j] : 0.f;
      }
      else if (k < nw + nh) {
         const long long q = k - nw, l = q / T;
         hrev[q] = h[l * T + (T - 1 - (q - l * T))];
      }
      else {
         const long long q = k - nw - nh, l = q / M;
         grev[q] = gy[l * M + (M - 1 - (q - l * M))];
      }
   }
}

__global__ void __launch_bounds__(256) reverse_rows_kernel(const float *in, float *out, int rows, int n)
{
   for (long long k = (long long) blockIdx.x * blockDim.x + threadIdx.x; k < (long long) rows * n; k += (long long) gridDim.x * blockDim.x) {
      const long long l = k / n;
      out[k] = in[l * n + (n - 1 - (k - l * n))];
   }
}

size_t firAdjointScratch(int batch, int rows, int N, int T, bool wantX, bool wantH)
{
   const size_t M = (size_t) (N - T + 1);
   auto up = [](size_t n) { return (n + 31) & ~(size_t) 31; };
   return (wantX ? up(batch * (M + 2 * (size_t) (T - 1))) + up((size_t) rows * T) : 0) +
          (wantH ? up(batch * M) + up((size_t) batch * T) : 0);
}

// dx = FIR of the widened gy with the reversed taps, dh = the FIR of x with each channel's
// reversed gy as its taps, reversed.  One launch makes the operands (five of the framework's
// took 27 us of host time).
cudaError_t launchFirAdjoint(const float *gy, const float *x, const float *h, float *gx, float *gh, float *scratch,
                             int batch, int rows, int N, int T, cudaStream_t s)
{
   const int M = N - T + 1;
   auto up = [](size_t n) { return (n + 31) & ~(size_t) 31; };
   const size_t W = (size_t) M + 2 * (size_t) (T - 1);
   float *wide = nullptr, *hrev = nullptr, *grev = nullptr, *lag = nullptr;
   if (gx) {
      wide = scratch;
      hrev = wide + up(batch * W);
      scratch = hrev + up((size_t) rows * T);
   }
   if (gh) {
      grev = scratch;
      lag = grev + up((size_t) batch * M);
   }
   auto blocks = [](size_t n) { return (unsigned) std::min<size_t>((n + 255) / 256, 148 * 16); };
   const size_t items = (gx ? batch * W + (size_t) rows * T : 0) + (gh ? (size_t) batch * M : 0);
   if (items == 0) return cudaSuccess;
   fir_adjoint_operands_kernel<<<blocks(items), 256, 0, s>>>(gy, h, wide, hrev, grev, batch, rows, M, T);
   countLaunch();
   cudaError_t e = cudaGetLastError();
   FirLaunch a{};
   a.dtype = DSPLIB_FLOAT32;
   a.batch = batch;
   if (gx && e == cudaSuccess) {
      a.x = wide, a.h = hrev, a.y = gx;
      a.T = T, a.outSize = N;
      a.inPitch = (long long) W, a.outPitch = N, a.filtPitch = rows > 1 ? T : 0;
      e = launchFir(a, FIR_F32_SIMT, s);
   }
   if (gh && e == cudaSuccess) {
      a.x = x, a.h = grev, a.y = lag;
      a.T = M, a.outSize = T;
      a.inPitch = N, a.outPitch = T, a.filtPitch = M;
      e = launchFir(a, FIR_F32_SIMT, s);
      if (e != cudaSuccess) return e;
      reverse_rows_kernel<<<blocks((size_t) batch * T), 256, 0, s>>>(lag, gh, batch, T);
      countLaunch();
      e = cudaGetLastError();
   }
   return e;
}

} // namespace dsplib
