// host_pipe.h -- host arrays in and out of device buffers, with conversion.
//
// The arrays that a program passes are ordinary pageable memory, often in
// another precision than the handle's.  A pipe owns slots, two per host thread,
// pinned where that pays; each thread converts its own share of the array slot by
// slot while its previous slot is being copied, so conversion, page faults of a fresh
// destination and the copy overlap and spread over the cores.  (Converting a
// 256^3 FP64 array on one thread into a temporary and copying that pageable
// temporary took most of 131 ms for set, 100 steps and get; with the pipe the
// same pass takes 33 ms, 18 of them in the steps.)
//
// An array that needs no conversion and is pinned already goes as one copy: the
// link alone bounds it (512^3 FP32: 10.7 ms in, 10.6 out; through the slots 15.1
// and 14.2).
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>
#include <type_traits>
#include <vector>

#include "user_buffer.h"

namespace opfc {

// Pages of ordinary memory, from the system and back to it: a large block freed to
// the C library would raise the size from which it maps blocks, for the program's
// own arrays too.
inline void *map_pages(size_t bytes) {
  void *p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED) return nullptr;
  madvise(p, bytes, MADV_HUGEPAGE);  // fewer faults; where it is refused, ordinary pages
  return p;
}

// running compensated (Neumaier) sum in four independent lanes, so that the
// additions of one element do not wait for those of the one before
struct LaneSum {
  double s[4] = {0, 0, 0, 0}, c[4] = {0, 0, 0, 0};
  void add(int l, double v) {
    const double t = s[l] + v;
    c[l] += (std::fabs(s[l]) >= std::fabs(v)) ? (s[l] - t) + v : (v - t) + s[l];
    s[l] = t;
  }
};

class HostPipe {
 public:
  static constexpr size_t kShareBytes = size_t(1) << 20;  // device bytes that are worth a thread
  static constexpr size_t kMinSlot = size_t(1) << 19, kMaxSlot = size_t(1) << 20;
  static constexpr size_t kNeverPin = size_t(1) << 17, kPinAtOnce = size_t(1) << 25;
  static constexpr size_t kOneCopyFrom = size_t(4) << 20, kOneCopyTo = size_t(20) << 20;
  static constexpr int kMaxThreads = 16;

  ~HostPipe() { release(); }

  // an ensemble's `arrays` of up to `bytes` device bytes: they come in any order, and
  // slots that grow with them are paid for each time (setting 64 members: 50 ms so, 36
  // with one set of slots).  A few are all read out once before the slots are pinned
  // (8 members 2.6 ms so, 21 with the pinning), many repay it in their first read-out (64
  // members 50 ms, 70 to 86 without).
  void expect(size_t bytes, int arrays) {
    expect_ = bytes;
    once_ = arrays < 16 ? arrays : 1;
  }

  // n values host (H) -> device (D) on stream s; with `parts`, the compensated
  // sums of the host values are appended to it.  Returns before the last copies
  // have run (the slots are not touched again before they have; a pinned array
  // that goes as one copy has to stay as it is until then).
  template <typename H, typename D>
  cudaError_t in(int device, const H *src, D *dst, size_t n, cudaStream_t s, std::vector<double> *parts) {
    if (std::is_same<H, D>::value && !parts && one_copy_in(src, n * sizeof(D)))
      return cudaMemcpyAsync(dst, src, n * sizeof(D), cudaMemcpyHostToDevice, s);
    return run<D>(device, n, s, false, parts, [=](size_t lo, size_t hi, D *const *slot, cudaEvent_t *ev, LaneSum *sum) {
      const size_t step = slot_ / sizeof(D);
      cudaError_t e = cudaSuccess;
      int k = 0;
      for (size_t i = lo; i < hi && e == cudaSuccess; i += step, k ^= 1) {
        const size_t len = std::min(step, hi - i);
        if ((e = cudaEventSynchronize(ev[k])) != cudaSuccess) break;
        convert(src + i, slot[k], len);
        if (sum)
          for (size_t q = 0; q < len; ++q) sum->add(q & 3, (double)src[i + q]);
        e = cudaMemcpyAsync(dst + i, slot[k], len * sizeof(D), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k], s);
      }
      return e;
    });
  }

  // n values device (D) -> host (H), complete on return
  template <typename D, typename H>
  cudaError_t out(int device, const D *src, H *dst, size_t n, cudaStream_t s) {
    const bool same = std::is_same<H, D>::value;
    const size_t bytes = std::max(n * sizeof(D), expect_);
    const bool first = !pinned_ && bytes <= kPinAtOnce && outs_++ < once_;
    if (same && (first || pinned_host_memory(pointer_attributes(dst)))) {
      const cudaError_t e = cudaMemcpyAsync(dst, src, n * sizeof(D), cudaMemcpyDeviceToHost, s);
      return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    }
    if (first) return out_once(src, dst, n, s);
    return run<D>(device, n, s, true, nullptr, [=](size_t lo, size_t hi, D *const *slot, cudaEvent_t *ev, LaneSum *) {
      const size_t step = slot_ / sizeof(D);
      cudaError_t e = cudaSuccess;
      auto issue = [&](size_t i, int k) {
        if (i >= hi || e != cudaSuccess) return;
        e = cudaMemcpyAsync(slot[k], src + i, std::min(step, hi - i) * sizeof(D), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k], s);
      };
      for (int k = 0; k < 2; ++k)  // an earlier call's copies out of the slots
        if (e == cudaSuccess) e = cudaEventSynchronize(ev[k]);
      issue(lo, 0);
      issue(lo + step, 1);
      int k = 0;
      for (size_t i = lo; i < hi && e == cudaSuccess; i += step, k ^= 1) {
        if ((e = cudaEventSynchronize(ev[k])) != cudaSuccess) break;
        convert(slot[k], dst + i, std::min(step, hi - i));
        issue(i + 2 * step, k);
      }
      return e;
    });
  }

  void release() {
    for (cudaEvent_t e : ev_)
      if (e) cudaEventDestroy(e);
    ev_.clear();
    if (pin_ && pinned_)
      cudaFreeHost(pin_);
    else if (pin_)
      munmap(pin_, pin_bytes_);
    pin_ = nullptr;
    pinned_ = tried_pin_ = false;
    threads_ = 0;
    slot_ = 0;
  }

 private:
  char *pin_ = nullptr;
  size_t pin_bytes_ = 0;
  bool tried_pin_ = false;  // the slots are pinned, or pinning was refused
  bool pinned_ = false;  // else pageable: the copies are then slower and synchronous, with the same result
  int threads_ = 0;  // threads with slots and events
  size_t slot_ = 0;  // bytes of a slot
  size_t expect_ = 0;
  int outs_ = 0, once_ = 1;  // arrays out while the slots were not pinned, and how many go so
  std::vector<cudaEvent_t> ev_;

  template <typename A, typename B> static void convert(const A *a, B *b, size_t n) {
    if (sizeof(A) == sizeof(B))
      std::memcpy(b, a, n * sizeof(A));
    else
      for (size_t i = 0; i < n; ++i) b[i] = (B)a[i];
  }

  // Whether an array without conversion goes in as one copy: pinned, or the slots
  // are not pinned, or of a size that staging does not speed up (128x64x64 FP64 0.32 ms
  // so, 0.43 through pinned slots; 128^3 1.1 and 1.4; but 256x256x128 5.4 and 4.0, and
  // at 64^3 0.21 either way with the next array out 0.35 and 0.23, its threads being
  // warm).
  bool one_copy_in(const void *host, size_t bytes) const {
    return !pinned_ || (bytes >= kOneCopyFrom && bytes < kOneCopyTo) || pinned_host_memory(pointer_attributes(host));
  }

  static int threads_for(size_t bytes) {
    const size_t cores = std::max(1u, std::thread::hardware_concurrency());
    return (int)std::min<size_t>({(size_t)kMaxThreads, cores, std::max<size_t>(1, (bytes + kShareBytes - 1) / kShareBytes)});
  }

  // Slots and events for arrays of `bytes`: a slot holds an eighth of a thread's share
  // (512 KiB to 1 MiB; through 256 KiB slots 64 MiB out took 3.3 ms, 2.0 so), or one
  // thread's array.  Pinning costs 2 to 3 ms and 0.3 to
  // 0.6 ms a MiB, once for a handle.  Arrays in go through ordinary slots at nearly
  // the same rate (128^3 FP32 from FP64 1.0 to 2.3 ms either way).  Arrays out are
  // much faster through pinned ones, most of all into fresh pages (FP64, one copy /
  // pinned slots: 64x16x24 78 / 42 us, 64^3 360 / 223, 128^3 2200 / 1450, 256x256x128
  // 14.8 / 2.7 ms), so the second array out pins (a small ensemble's second read-out): the
  // first goes as one copy, into a temporary where it needs conversion, as handles are
  // often read out once.  Arrays of more than 32 MiB repay the pinning at once.
  cudaError_t ensure(size_t bytes, bool pin) {
    bytes = std::max(bytes, expect_);
    pin = pin && bytes > kNeverPin;
    const int threads = threads_for(bytes);
    const size_t part = threads == 1 ? bytes : std::max(kMinSlot, bytes / threads / 8);
    const size_t slot = std::min(kMaxSlot, (part + 4095) / 4096 * 4096);
    if (threads <= threads_ && slot <= slot_ && (!pin || tried_pin_)) return cudaSuccess;
    for (cudaEvent_t e : ev_) cudaEventSynchronize(e);  // copies out of the old slots
    release();
    cudaError_t e = cudaSuccess;
    pin_bytes_ = 2 * slot * threads;
    if (pin) {
      e = cudaHostAlloc((void **)&pin_, pin_bytes_, cudaHostAllocDefault);
      if (e != cudaSuccess) cudaGetLastError();
      tried_pin_ = true;
    }
    pinned_ = pin && e == cudaSuccess;
    if (!pinned_ && !(pin_ = static_cast<char *>(map_pages(pin_bytes_)))) return cudaErrorMemoryAllocation;
    slot_ = slot;
    for (int i = 0; i < 2 * threads; ++i) {
      cudaEvent_t v = nullptr;
      if ((e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming)) != cudaSuccess) {
        release();
        return e;
      }
      ev_.push_back(v);
    }
    threads_ = threads;
    return cudaSuccess;
  }

  // f(t, lo, hi) on T threads, this one included, for their shares of n values
  template <typename F> static void share(int T, size_t n, const F &f) {
    const size_t each = ((n + T - 1) / T + 3) / 4 * 4;
    auto work = [&](int t) { f(t, std::min(n, each * t), std::min(n, each * t + each)); };
    std::vector<std::thread> th;
    th.reserve(T);
    int started = 1;  // share 0 runs here
    try {
      for (; started < T; ++started) th.emplace_back(work, started);
    } catch (...) {  // no more threads (or no memory for one): the rest runs here too
    }
    work(0);
    for (int t = started; t < T; ++t) work(t);
    for (auto &x : th) x.join();
  }

  template <typename D, typename H> static cudaError_t out_once(const D *src, H *dst, size_t n, cudaStream_t s) {
    D *tmp = static_cast<D *>(map_pages(n * sizeof(D)));
    if (!tmp) return cudaErrorMemoryAllocation;
    cudaError_t e = cudaMemcpyAsync(tmp, src, n * sizeof(D), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess)
      share(threads_for(n * sizeof(D)), n, [&](int, size_t lo, size_t hi) { convert(tmp + lo, dst + lo, hi - lo); });
    munmap(tmp, n * sizeof(D));
    return e;
  }

  // f(lo, hi, slots, events, sum) on each thread's share of n values of D.  The
  // per-thread default stream is another stream on every thread: the caller's own
  // thread then does it all.
  template <typename D, typename F>
  cudaError_t run(int device, size_t n, cudaStream_t s, bool pin, std::vector<double> *parts, const F &f) {
    const int T = s == cudaStreamPerThread ? 1 : threads_for(n * sizeof(D));
    cudaError_t e = ensure(n * sizeof(D), pin);
    if (e != cudaSuccess) return e;
    std::vector<cudaError_t> rc(T, cudaSuccess);
    std::vector<LaneSum> sums(parts ? T : 0);
    share(T, n, [&](int t, size_t lo, size_t hi) {
      D *slot[2] = {reinterpret_cast<D *>(pin_ + 2 * t * slot_), reinterpret_cast<D *>(pin_ + (2 * t + 1) * slot_)};
      rc[t] = cudaSetDevice(device);
      if (rc[t] == cudaSuccess) rc[t] = f(lo, hi, slot, &ev_[2 * t], parts ? &sums[t] : nullptr);
    });
    for (cudaError_t r : rc)
      if (r != cudaSuccess) return r;
    if (parts)
      for (const LaneSum &l : sums)
        for (int i = 0; i < 4; ++i) {
          parts->push_back(l.s[i]);
          parts->push_back(l.c[i]);
        }
    return cudaSuccess;
  }
};

}  // namespace opfc
