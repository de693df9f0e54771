// The pages of large result buffers, made present by host threads while the
// device computes (host code, no CUDA).
#pragma once

#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <memory>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace sparx {

// A fresh buffer's page faults otherwise fall into its download (125 MB of
// supports: 4.9 -> 3.1 ms).  Contents are left alone; a kernel without
// MADV_POPULATE_WRITE, or a host that gives no more threads, faults as before.
//
// The threads go on while the results come down.  The end waits only for the parts
// they are at, and for no thread that is not at one: where the device is done soon,
// the download's own sixteen threads fault the pages in as fast, and a thread the host
// has not run yet (the upload's threads still spin on every core) would be waited for
// until the next scheduler tick, 2 to 4 ms.  A thread left behind finds `stop` set
// before it touches anything (it says it is busy, then looks; the end stops, then
// looks who is busy).  ER n = 2 * 10^5, m = 2 * 10^6 (16 MB of results after 0.5 ms
// of kernels): the call 4.0 ms when the device's end joined the threads, 1.6 so.
class Prefault {
 public:
  static constexpr int kThreads = 4;
  // kPart: what one page table maps, so that no two threads want the same one's lock
  // (parts of 256 KB: the slowest tenth of R-MAT-20 triangle calls 19.4 ms, so 18.4)
  static constexpr size_t kPart = 2ull << 20, kLeast = 16ull << 20;  // kLeast: bytes worth starting threads for

  // the buffer's whole pages
  void add(void* p, size_t bytes) {
    const uintptr_t page = 4096, b = ((uintptr_t)p + page - 1) & ~(page - 1), e = ((uintptr_t)p + bytes) & ~(page - 1);
    if (e <= b) return;
    total += e - b;
    for (uintptr_t at = b; at < e;) {
      const uintptr_t to = std::min<uintptr_t>((at / kPart + 1) * kPart, e);
      work->parts.push_back({at, to - at});
      at = to;
    }
  }

  void start() {
    if (total < kLeast) return;
    try {
      for (; started_ < kThreads; ++started_) std::thread(run, work).detach();
    } catch (const std::system_error&) {
      // no (more) threads: those there are do what they can
    }
  }

  int started() const { return started_; }
  bool idle() const { return work->next >= work->parts.size() && !work->busy; }  // every part is done

  Prefault() = default;
  Prefault(const Prefault&) = delete;
  Prefault& operator=(const Prefault&) = delete;
  ~Prefault() {
    work->stop = true;
    while (work->busy) std::this_thread::yield();
  }

 private:
  struct Work {
    std::vector<std::pair<uintptr_t, size_t>> parts;
    std::atomic<size_t> next{0};
    std::atomic<int> busy{0};
    std::atomic<bool> stop{false};
  };
  static void run(std::shared_ptr<Work> w) {
    for (bool more = true; more;) {
      ++w->busy;
      size_t k;
      more = !w->stop && (k = w->next++) < w->parts.size() &&
             madvise((void*)w->parts[k].first, w->parts[k].second, MADV_POPULATE_WRITE) == 0;
      --w->busy;
    }
  }
  std::shared_ptr<Work> work = std::make_shared<Work>();
  size_t total = 0;
  int started_ = 0;
};

}  // namespace sparx
