// Streaming (overlap-save) FIR over consecutive blocks.
//
// DSPLIB_fir is a "valid" filter: a call on N input samples per channel gives
// N - T + 1 outputs, and a caller that filters a continuous signal block by
// block has to carry the last T - 1 input samples of every channel into the
// next call itself (the reference leaves that to the caller).  A stream keeps
// that history on the device: each call takes N new samples per channel and
// returns N outputs per channel, the first T - 1 of them computed over the
// previous block's tail (zeros before the first block).
//
// Each channel has a device window [T - 1 history | N new]; between calls its last T - 1
// samples are the history.  Per call, on the handle's stream, one kernel moves the history to
// the window's head and the new block behind it, and DSPLIB_fir_exec runs over the windows;
// if it refuses, or a copy does, the history is moved back.  Blocks in host memory (or on another device), blocks
// shorter than the history, whose old and new place overlap, and blocks whose rows do not all
// start on a multiple of the sample size are moved by copies.
// (Three 2-D copies around the filter, with the history in a buffer of its own, took 18.4 us
// a call on 16 channels x 4096 int16 samples x 64 taps; now 10.2.)
#include <climits>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "dsplib_internal.h"

namespace dsplib {

struct FirStream {
   FirPriv *handle = nullptr; // internal DSPLIB_fir handle over the windows
   void *buf = nullptr;       // the windows
   void *hist = nullptr;      // channels x (T - 1) elements: the history on its way, where the copies are used
   char *win = nullptr;       // first window: rows of T - 1 + N elements
   size_t pitch = 0;          // bytes between windows; a window's new block starts on a 16-byte boundary
   int channels = 0, T = 0, N = 0, elt = 0;
   size_t inPitch = 0;        // bytes between the caller's input rows

   size_t histBytes() const { return (size_t) (T - 1) * elt; }
   size_t blockBytes() const { return (size_t) N * elt; }
   char *tail() const { return win + blockBytes(); }
};

// History between the window's tail and its head goes through the buffer: the two may overlap.
static cudaError_t takeHistory(const FirStream *s, const char *from, cudaStream_t cs)
{
   const size_t hb = s->histBytes();
   return hb ? cudaMemcpy2DAsync(s->hist, hb, from, s->pitch, hb, s->channels, cudaMemcpyDeviceToDevice, cs) : cudaSuccess;
}
static cudaError_t putHistory(const FirStream *s, char *to, cudaStream_t cs)
{
   const size_t hb = s->histBytes();
   return hb ? cudaMemcpy2DAsync(to, s->pitch, s->hist, hb, hb, s->channels, cudaMemcpyDeviceToDevice, cs) : cudaSuccess;
}

// Whether a kernel on the current device may read p.
static bool onThisDevice(const void *p)
{
   cudaPointerAttributes at;
   int dev = -1;
   if (cudaPointerGetAttributes(&at, p) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) {
      (void) cudaGetLastError();
      return false;
   }
   return at.type == cudaMemoryTypeDevice && at.device == dev;
}

static void destroyStream(FirStream *s)
{
   if (!s) return;
   cudaFree(s->buf);
   cudaFree(s->hist);
   std::free(s->handle);
   delete s;
}

} // namespace dsplib

using namespace dsplib;

extern "C" {

DSPLIB_STATUS DSPLIB_gpu_firStreamCreate(DSPLIB_gpu_firStream *stream, const DSPLIB_fir_InitArgs *args,
                                         const DSPLIB_bufParams2D_t *bufParamsIn,
                                         const DSPLIB_bufParams2D_t *bufParamsFilter,
                                         const DSPLIB_bufParams2D_t *bufParamsOut)
{
   if (!stream || !args || !bufParamsIn || !bufParamsFilter || !bufParamsOut) return DSPLIB_ERR_NULL_POINTER;
   *stream = nullptr;
   const int elt = DSPLIB_sizeof((uint32_t) bufParamsIn->data_type);
   const int T = args->filterSize, N = args->dataSize, C = args->batchSize;
   if (elt <= 0) return DSPLIB_ERR_INVALID_TYPE;
   if (T < 1 || N < 1 || C < 1 || (int) bufParamsOut->dim_x != N || bufParamsIn->stride_y < N * elt)
      return DSPLIB_ERR_INVALID_DIMENSION;
   FirStream *s = new FirStream();
   s->channels = C;
   s->T = T;
   s->N = N;
   s->elt = elt;
   s->inPitch = (size_t) bufParamsIn->stride_y;
   const int W = T - 1 + N;
   DSPLIB_fir_InitArgs a = *args;
   a.dataSize = W;
   DSPLIB_bufParams2D_t win = *bufParamsIn;
   win.dim_x = (uint32_t) W;
   win.dim_y = (uint32_t) C;
   // the new block on a 16-byte boundary: wide copies, and wide loads in the filter
   const bool padded = (long long) W * elt <= INT_MAX - 32;
   const int lead = padded ? (int) (-s->histBytes() & 15) : 0;
   s->pitch = padded ? ((size_t) lead + (size_t) W * elt + 15) & ~(size_t) 15 : (size_t) W * elt;
   win.stride_y = (int32_t) s->pitch;
   DSPLIB_bufParams2D_t filt = *bufParamsFilter, out = *bufParamsOut;
   s->handle = (FirPriv *) std::calloc(1, (size_t) DSPLIB_fir_getHandleSize(&a));
   DSPLIB_STATUS st = s->handle ? DSPLIB_fir_init(s->handle, &win, &filt, &out, &a) : DSPLIB_ERR_FAILURE;
   if (st == DSPLIB_SUCCESS &&
       (cudaMalloc(&s->buf, (size_t) C * s->pitch) != cudaSuccess ||
        (T > 1 && cudaMalloc(&s->hist, (size_t) C * s->histBytes()) != cudaSuccess)))
      st = DSPLIB_ERR_FAILURE;
   s->win = (char *) s->buf + lead;
   if (st == DSPLIB_SUCCESS && T > 1 && cudaMemset2D(s->tail(), s->pitch, 0, s->histBytes(), C) != cudaSuccess)
      st = DSPLIB_ERR_FAILURE;
   if (st != DSPLIB_SUCCESS) {
      (void) cudaGetLastError();
      destroyStream(s);
      return st;
   }
   *stream = (DSPLIB_gpu_firStream) s;
   return DSPLIB_SUCCESS;
}

DSPLIB_kernelHandle DSPLIB_gpu_firStreamHandle(DSPLIB_gpu_firStream stream)
{
   return stream ? (DSPLIB_kernelHandle) ((FirStream *) stream)->handle : nullptr;
}

DSPLIB_STATUS DSPLIB_gpu_firStreamExec(DSPLIB_gpu_firStream stream, const void *pIn, void *pFilter, void *pOut)
{
   FirStream *s = (FirStream *) stream;
   if (!s || !pIn || !pFilter || !pOut) return DSPLIB_ERR_NULL_POINTER;
   HandleCommon *hc = &s->handle->common;
   const cudaStream_t cs = hc->stream;
   cudaError_t e = cudaSuccess;
   const bool own = onThisDevice(pIn);
   const bool whole = (((uintptr_t) pIn | s->inPitch) & (size_t) (s->elt - 1)) == 0; // the kernel loads whole samples
   if (own && whole && s->N >= s->T - 1) {
      if ((e = launchStreamWindow(s->win, (long long) s->pitch, pIn, (long long) s->inPitch, s->channels, s->T - 1,
                                  s->N, s->elt, cs)))
         return cudaFail(hc, e, "stream: fill window");
   }
   else {
      const char *what = "stream: restore history";
      injectArm(hc);
      if ((e = injectCheck(takeHistory(s, s->tail(), cs))) != cudaSuccess) return cudaFail(hc, e, what);
      e = injectCheck(putHistory(s, s->win, cs));
      if (e == cudaSuccess) {
         what = "stream: copy block";
         e = injectCheck(cudaMemcpy2DAsync(s->win + s->histBytes(), s->pitch, pIn, s->inPitch, s->blockBytes(),
                                           s->channels, cudaMemcpyDefault, cs));
      }
      if (e != cudaSuccess) {
         (void) putHistory(s, s->tail(), cs); // the head or the block may have gone over it
         return cudaFail(hc, e, what);
      }
      injectPass(hc);
   }
   const DSPLIB_STATUS st = DSPLIB_fir_exec(s->handle, s->win, pFilter, pOut);
   if (st != DSPLIB_SUCCESS) { // a refused call leaves the history as it was
      if (takeHistory(s, s->win, cs) == cudaSuccess) (void) putHistory(s, s->tail(), cs);
      return st;
   }
   // a host block is copied in asynchronously: complete before returning unless async level 2
   if (mustSync(hc, false, !own && !isDevicePtr(pIn)) && (e = cudaStreamSynchronize(cs)))
      return cudaFail(hc, e, "stream: execution");
   return DSPLIB_SUCCESS;
}

DSPLIB_STATUS DSPLIB_gpu_firStreamReset(DSPLIB_gpu_firStream stream)
{
   FirStream *s = (FirStream *) stream;
   if (!s) return DSPLIB_ERR_NULL_POINTER;
   if (s->T > 1 && cudaMemset2DAsync(s->tail(), s->pitch, 0, s->histBytes(), s->channels,
                                     s->handle->common.stream) != cudaSuccess)
      return cudaFail(&s->handle->common, cudaGetLastError(), "stream: reset");
   return DSPLIB_SUCCESS;
}

DSPLIB_STATUS DSPLIB_gpu_firStreamDestroy(DSPLIB_gpu_firStream stream)
{
   FirStream *s = (FirStream *) stream;
   if (!s) return DSPLIB_ERR_NULL_POINTER;
   (void) cudaStreamSynchronize(s->handle->common.stream);
   destroyStream(s);
   return DSPLIB_SUCCESS;
}

} // extern "C"
