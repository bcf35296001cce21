// thx_staging.h -- internal: pinned host staging ring for stream-ordered
// uploads (pure C++; the device calls come from the policy Dev).
//
// A copy is written into the ring on the host and sent with an asynchronous
// copy, so the call neither waits for the stream nor goes through the driver's
// pageable path.  Space is taken and retired in FIFO order; a span is retired
// once its copy's event has completed.  The lock covers that bookkeeping and
// the enqueueing, not the writing: callers on several threads write their
// spans at the same time.
//
// Dev: Stream, Event, kNoSpace (a status), and, with 0 for success,
//   alloc(void **, bytes), free(void *), copy(dst, src, bytes, stream),
//   create(Event *), destroy(Event), record(Event, Stream), wait(Event),
//   drain(Stream).
#pragma once
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <vector>

#include "thx_ring.h"

namespace thx {

template <class Dev>
class StagingRing {
 public:
  using Stream = typename Dev::Stream;
  using Event = typename Dev::Event;

  ~StagingRing() {
    for (Span &sp : spans_)
      if (sp.state == QUEUED) Dev::destroy(sp.done);
    for (Event ev : spare_) Dev::destroy(ev);
    if (buf_) Dev::free(buf_);
  }
  int init(size_t bytes) {
    void *p = nullptr;
    if (Dev::alloc(&p, bytes)) return Dev::kNoSpace;
    buf_ = static_cast<unsigned char *>(p);
    space_.reset(bytes);
    return 0;
  }
  // Host -> device copy of `bytes` on stream s through the ring (copies of
  // more than half the ring go directly).
  int copy(void *dst, const void *src, size_t bytes, Stream s) {
    if (!buf_ || round_up(bytes) > most()) return Dev::copy(dst, src, bytes, s);
    return piece(dst, bytes, s, [&](void *to) { std::memcpy(to, src, bytes); });
  }
  // The same of `count` items of `size` bytes that write(to, first, n) forms,
  // in pieces of at most half the ring.
  template <typename F>
  int fill(void *dst, size_t size, size_t count, Stream s, F &&write) {
    const size_t per = most() / size;
    if (!buf_ || per == 0) return Dev::kNoSpace;
    for (size_t first = 0; first < count; first += per) {
      const size_t n = std::min(per, count - first);
      const int st = piece(static_cast<unsigned char *>(dst) + first * size, n * size, s,
                           [&](void *to) { write(to, first, n); });
      if (st) return st;
    }
    return 0;
  }
  // host seconds spent waiting for space and writing into the ring
  void times(double *wait_s, double *copy_s) {
    std::lock_guard<std::mutex> lock(mu_);
    *wait_s = wait_s_;
    *copy_s = copy_s_;
  }

 private:
  using Clock = std::chrono::steady_clock;
  enum State { WRITING, QUEUED, UNUSED };
  struct Span {
    State state = WRITING;
    Event done{};  // of a queued span's copy
  };
  static size_t round_up(size_t n) { return (n + 255) & ~size_t(255); }
  size_t most() const { return space_.capacity() / 2 / 256 * 256; }
  static double since(Clock::time_point t) { return std::chrono::duration<double>(Clock::now() - t).count(); }

  template <typename F>
  int piece(void *dst, size_t bytes, Stream s, F &&write) {
    const size_t need = round_up(bytes);
    size_t off;
    int st;
    std::unique_lock<std::mutex> lock(mu_);
    const auto t0 = Clock::now();
    while (!space_.place(need, &off)) {  // wait for the oldest span
      if (spans_.front().state == WRITING) {
        changed_.wait(lock);  // another thread has yet to queue its copy
        continue;
      }
      if (spans_.front().state == QUEUED) {
        if ((st = Dev::wait(spans_.front().done))) return st;
        spare_.push_back(spans_.front().done);
      }
      spans_.pop_front();
      space_.pop();
    }
    wait_s_ += since(t0);
    Event ev;
    if (!spare_.empty()) {
      ev = spare_.back();
      spare_.pop_back();
    } else if ((st = Dev::create(&ev))) {
      return st;
    }
    space_.push(off, need);
    spans_.emplace_back();
    Span &sp = spans_.back();  // a deque's elements stay where they are
    lock.unlock();
    const auto t1 = Clock::now();
    write(buf_ + off);
    const double copy_s = since(t1);
    lock.lock();
    copy_s_ += copy_s;
    st = Dev::copy(dst, buf_ + off, bytes, s);
    if (st) {
      sp.state = UNUSED;
      spare_.push_back(ev);
    } else {
      sp.state = QUEUED;
      sp.done = ev;
      // unrecorded, the event would report complete at once: wait for the
      // stream before the span can be reused
      if ((st = Dev::record(ev, s))) Dev::drain(s);
    }
    changed_.notify_all();
    return st;
  }

  std::mutex mu_;
  std::condition_variable changed_;  // a span has been written
  double wait_s_ = 0.0, copy_s_ = 0.0;
  unsigned char *buf_ = nullptr;
  RingSpace space_;
  std::deque<Span> spans_;  // one per live span of space_, oldest first
  std::vector<Event> spare_;
};

}  // namespace thx
