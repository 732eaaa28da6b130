// cgfd_stager.h -- copies between the caller's (pageable) host arrays and the device through pinned
// chunks that host threads and the copy engine work on side by side.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "cgfd_b200.h"
#include "cgfd_setup.h"

#define CGFD_CK(call)                                                                            \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess)                                                                       \
      throw cgfd::Error(CGFD_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));      \
  } while (0)

namespace cgfd {

// Host -> device copies of the caller's model arrays (pageable memory) through two pinned
// chunks: host threads fill one chunk while the copy engine drains the other, so the upload
// runs at the slower of a parallel host memcpy and the host link instead of the driver's
// serial pageable path. One stager per device, allocated on first use and kept for the life
// of the process (2 x 64 MiB of pinned host memory): allocating and freeing pinned memory per
// problem would synchronise the device under the serving loop's concurrent problems. Users
// hold its lock for a whole upload; each chunk is refilled only after the copy out of it
// has completed (per-chunk events), so no device-wide synchronisation is involved. Where the host has
// no pinned memory to give, transfers take the plain pageable copy.
class PinnedStager {
 public:
  static constexpr size_t kChunk = size_t(64) << 20;
  // fields below this size go through the plain pageable copy
  static constexpr size_t kMinBytes = size_t(16) << 20;
  // read-backs below this size likewise (they are slower per byte on the pageable path: a fresh host
  // array's pages are touched there for the first time)
  static constexpr size_t kMinOut = size_t(1) << 20;

  static PinnedStager &for_device(int device) {
    static std::mutex mu;
    static std::vector<PinnedStager *> all;
    std::lock_guard<std::mutex> lk(mu);
    if ((int)all.size() <= device) all.resize(device + 1, nullptr);
    if (!all[device]) all[device] = new PinnedStager();
    return *all[device];
  }
  std::mutex &mutex() { return mu_; }

  // device -> caller's (pageable) host memory, the reverse pipeline, of `parts` parts of n bytes each:
  // produce(q) enqueues on st whatever leaves part q at src, the copy engine then fills one chunk while
  // host threads empty the other into dst + q n. The host threads also take the first-touch page
  // faults of a fresh host array side by side, which the driver's pageable path takes one after the
  // other: 9 fields of 480x480x240 came back in 507 ms that way, of 100x100x60 in 10.2 ms.
  template <typename Produce>
  void copy_out(void *dst, const void *src, size_t n, int parts, cudaStream_t st, Produce produce) {
    const size_t per = (n + kChunk - 1) / kChunk, nch = per * parts;
    auto issue = [&](size_t c) {
      const size_t o = c % per * kChunk, m = std::min(kChunk, n - o);
      if (o == 0) produce((int)(c / per));
      CGFD_CK(cudaEventSynchronize(done_[c & 1]));
      CGFD_CK(cudaMemcpyAsync(buf_[c & 1], static_cast<const char *>(src) + o, m, cudaMemcpyDeviceToHost, st));
      CGFD_CK(cudaEventRecord(done_[c & 1], st));
    };
    if (nch == 0) return;
    if (!ready()) {
      for (int q = 0; q < parts; q++) {
        produce(q);
        CGFD_CK(cudaMemcpyAsync(static_cast<char *>(dst) + q * n, src, n, cudaMemcpyDeviceToHost, st));
      }
      return;
    }
    issue(0);
    for (size_t c = 0; c < nch; c++) {
      if (c + 1 < nch) issue(c + 1);
      CGFD_CK(cudaEventSynchronize(done_[c & 1]));
      const size_t o = c % per * kChunk, m = std::min(kChunk, n - o);
      char *out = static_cast<char *>(dst) + c / per * n + o;
      const long long pieces = (long long)((m + kPiece - 1) / kPiece);
#pragma omp parallel for schedule(static)
      for (long long q = 0; q < pieces; q++) {
        const size_t a = (size_t)q * kPiece;
        std::memcpy(out + a, buf_[c & 1] + a, std::min(kPiece, m - a));
      }
    }
    next_ = (int)(nch & 1);
  }
  void copy_out(void *dst, const void *src, size_t n, cudaStream_t st) {
    copy_out(dst, src, n, 1, st, [](int) {});
  }

  void copy(void *dst, const void *src, size_t n, cudaStream_t st) {
    if (!ready()) {
      CGFD_CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st));
      return;
    }
    for (size_t o = 0; o < n; o += kChunk) {
      const size_t m = std::min(kChunk, n - o);
      const int b = next_;
      next_ ^= 1;
      CGFD_CK(cudaEventSynchronize(done_[b]));  // the previous copy out of this chunk has finished
      const char *in = static_cast<const char *>(src) + o;
      const long long pieces = (long long)((m + kPiece - 1) / kPiece);
#pragma omp parallel for schedule(static)
      for (long long q = 0; q < pieces; q++) {
        const size_t a = (size_t)q * kPiece;
        std::memcpy(buf_[b] + a, in + a, std::min(kPiece, m - a));
      }
      CGFD_CK(cudaMemcpyAsync(static_cast<char *>(dst) + o, buf_[b], m, cudaMemcpyHostToDevice, st));
      CGFD_CK(cudaEventRecord(done_[b], st));
    }
  }

 private:
  PinnedStager() = default;
  bool ready() {  // both chunks, allocated on first use (the device is current)
    for (int b = 0; b < 2; b++) {
      if (!done_[b]) CGFD_CK(cudaEventCreateWithFlags(&done_[b], cudaEventDisableTiming));
      if (!buf_[b] && cudaHostAlloc(reinterpret_cast<void **>(&buf_[b]), kChunk, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        buf_[b] = nullptr;
        return false;
      }
    }
    return true;
  }
  static constexpr size_t kPiece = size_t(1) << 18;
  std::mutex mu_;
  char *buf_[2] = {nullptr, nullptr};
  cudaEvent_t done_[2] = {nullptr, nullptr};
  int next_ = 0;
};

}  // namespace cgfd
