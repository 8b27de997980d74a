// How the copy-in of a call with host buffers is ordered behind the calls before it (w4a16_marlin_gemm_host).  Host code
// without CUDA, so that the rules can be checked on the CPU.
//
// Every kernel of this library waits for the completion of the one before it (griddepcontrol.wait) before it ends, so a kernel
// that has waited has waited for everything before it.  But a GEMM lets its successor start (griddepcontrol.launch_dependents)
// before it has waited itself, and the copy-in of COPY_EARLY and COPY_LATE does the same: what such a chain has in front of it
// when it starts goes back, kernel by kernel, to the last one that waited FIRST, and all calls since then may be unfinished.
// Those are the open calls.
//
// Other threads may launch meanwhile, on this stream or others, and only what is known to be in front of a copy-in can be taken
// for the open calls.  So the process counts its launches, once before and once after each, and the records of the chain: a
// call that finds the counter where the last record has left it, and that record's call itself saw nothing but its own two
// counts between its decision and its record, has nothing else between itself and that call.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <array>

namespace w4a16 {

enum CopyIn {
  COPY_FIRST = 0,   // waits, then lets the GEMM behind it start: everything before is over for all that follows
  COPY_LATE = 1,    // lets the GEMM start (it prefetches its weights), waits, copies: shares a buffer with the last call only
  COPY_EARLY = 2,   // copies beside the open calls' GEMMs and waits at its end: shares none
};

struct HostBuffers {
  const void *a_host, *a_stage, *c_stage, *c_host;
  size_t a_bytes, c_bytes;
};

// Where a call's work goes.  capture: 0, or the id of the capture that the stream is in: captured work is not in front of what
// the stream runs next, nor the other way round.  id: outside of a capture the stream's id, which no other stream of the process
// ever has (a handle may come back, and that of the per-thread default stream stands for one stream per thread).
struct Place {
  int dev;
  const void *stream;
  unsigned long long id, capture;
  bool operator==(const Place &o) const { return dev == o.dev && stream == o.stream && id == o.id && capture == o.capture; }
};

class HostChain {
 public:
  // The last call of this kind was on this stream.
  bool same_stream(const Place &p) const { return any_ && place_.dev == p.dev && place_.stream == p.stream; }

  // count: the process's counter now
  CopyIn order(const Place &p, uint64_t count, const HostBuffers &b) const {
    if (!any_ || !(place_ == p) || count_ == 0 || count_ != count || n_open_ >= MAX_OPEN) return COPY_FIRST;
    // What the copy-in reads and writes.  A buffer shared with the call right before is waited for anyway; one shared with an
    // older call (a buffer that comes back) closes the list instead of making every later call wait for its predecessor: four
    // layers with buffers of their own, called over and over, wait once a pass.
    for (size_t i = 0; i < n_open_; ++i) {
      const HostBuffers &o = open_[i];
      if (overlap(b.a_host, b.a_bytes, o.c_host, o.c_bytes) || overlap(b.a_stage, b.a_bytes, o.c_stage, o.c_bytes) ||
          overlap(b.a_stage, b.a_bytes, o.a_stage, o.a_bytes))
        return i + 1 < n_open_ ? COPY_FIRST : COPY_LATE;
    }
    return COPY_EARLY;
  }

  // After the call.  seen: the counter at its decision; now: the counter before this record's own count.
  void record(const Place &p, uint64_t seen, uint64_t now, CopyIn how, const HostBuffers &b) {
    any_ = true, place_ = p;
    count_ = now == seen + 2 ? now + 1 : 0;
    if (how == COPY_FIRST) n_open_ = 0;
    if (n_open_ < MAX_OPEN)
      open_[n_open_++] = b;
    else
      count_ = 0;   // (threads that decided at the same time)
  }

  // After a call that went through the copy engines, or failed half-way: the next copy-in waits first.
  void forget(const Place &p) { any_ = true, place_ = p, count_ = 0; }

 private:
  static bool overlap(const void *a, size_t na, const void *b, size_t nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + nb && y < x + na;
  }
  static constexpr size_t MAX_OPEN = 8;
  bool any_ = false;
  Place place_{};
  uint64_t count_ = 0;
  std::array<HostBuffers, MAX_OPEN> open_{};
  size_t n_open_ = 0;
};

}  // namespace w4a16
