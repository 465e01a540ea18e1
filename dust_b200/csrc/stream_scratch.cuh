// stream_scratch.cuh -- device scratch of the entry points without a handle.
//
// Those calls are queued on the caller's stream and return, so a second call on
// another stream may run while the first still reads its scratch.  Each call
// takes one of a few slots (the buffers, and an event after their last use): its
// own stream's, an unused one, one whose last use has finished, or else the
// least recently used one, for which its stream waits.  The pool is locked while
// a call is queued, so host threads may call at the same time.  Buffers grow and
// are kept; there are never more than SLOTS sets of them.  A captured call holds
// its buffers' addresses without an event: the caller keeps the graph's launches
// apart from other calls.
#pragma once

#include <mutex>

#include "fmm_internal.h"

class StreamScratch {
 public:
  struct Slot {
    DevBuf raw, geo, work;
    cudaStream_t st = nullptr;
    cudaEvent_t done = nullptr;
    int dev = -1;
    unsigned long long turn = 0;
  };

  // One call's hold of a slot: ends with the call.
  class Use {
   public:
    Use(StreamScratch &p, cudaStream_t st) : lock_(p.mu_), st_(st) { status = p.take(st, *this); }
    ~Use() {
      if (s && !capturing_) cudaEventRecord(s->done, st_);
    }
    Use(const Use &) = delete;
    Use &operator=(const Use &) = delete;
    Slot *operator->() { return s; }
    int status = DUST_OK;

   private:
    friend class StreamScratch;
    std::lock_guard<std::mutex> lock_;
    cudaStream_t st_;
    Slot *s = nullptr;
    bool capturing_ = false;
  };

  static StreamScratch &get() {
    static StreamScratch *p = new StreamScratch();  // never destroyed: no teardown at exit
    return *p;
  }

 private:
  static constexpr int SLOTS = 4;

  int take(cudaStream_t st, Use &u) {
    int dev = 0;
    DUST_CUDA(cudaGetDevice(&dev));
    // (a stream being captured can neither wait for events from outside nor
    // record them for outside: there the caller keeps calls apart)
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) cudaGetLastError();
    u.capturing_ = cs != cudaStreamCaptureStatusNone;
    Slot *s = nullptr;
    for (Slot &c : slot_)
      if (!s && c.dev == dev && c.st == st) s = &c;
    for (Slot &c : slot_)
      if (!s && c.dev < 0) s = &c;
    // (a query is among the calls that spoil another stream's capture of this
    // thread, or of any in the global mode, unless this thread's mode is relaxed)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    DUST_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    for (Slot &c : slot_)
      if (!s && !u.capturing_ && c.dev == dev) {
        if (cudaEventQuery(c.done) == cudaSuccess)
          s = &c;
        else
          cudaGetLastError();  // not ready
      }
    DUST_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    for (int same = 1; same >= 0 && !s; --same)
      for (Slot &c : slot_)
        if ((!same || c.dev == dev) && (!s || c.turn < s->turn)) s = &c;
    if (s->dev >= 0 && s->dev != dev) {  // another device's: given back
      devbuf_free(s->raw);
      devbuf_free(s->geo);
      devbuf_free(s->work);
      cudaEventDestroy(s->done);
      s->done = nullptr;
      s->dev = -1;
    }
    if (s->dev < 0)
      DUST_CUDA(cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming));
    else if (!u.capturing_)
      DUST_CUDA(cudaStreamWaitEvent(st, s->done, 0));
    s->dev = dev;
    s->st = st;
    s->turn = ++turn_;
    u.s = s;
    return DUST_OK;
  }

  std::mutex mu_;
  Slot slot_[SLOTS];
  unsigned long long turn_ = 0;
};
