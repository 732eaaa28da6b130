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
// serial pageable path. One stager per device; its pinned memory (2 x 64 MiB at most) is kept for
// the life of the process: allocating and freeing it per problem would synchronise the device under
// the serving loop's concurrent problems. A chunk is made of 8 MiB pieces that are allocated when a
// transfer first needs them: pinned memory takes about 0.35 ms per MiB to allocate, which a short
// transfer does not win back (the first layer model of 192x176x96 in a process: 63 ms with whole chunks,
// 21 with pieces, 40 unstaged), and a long one is faster in long chunks (9 fields of 480x480x240 read
// back in 74 ms by chunks of 64 MiB, 115 by 8). So a read-back takes a sixth of its bytes per chunk, the
// upload of a field up to 32 MiB (9 fields of 320x320x160: 15 ms, 22 by 64 MiB; of 200x200x100: 3.9 ms
// whole, 4.8 in halves), and each is cut evenly. Users hold its lock
// for a whole upload; each chunk is refilled only after the copy out of it has completed (per-chunk
// events), so no device-wide synchronisation is involved. Where the host has no pinned memory to give,
// transfers take the plain pageable copy.
class PinnedStager {
 public:
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
    const size_t chunk = even(n, ready(n * parts / 6));
    if (chunk == 0) {
      for (int q = 0; q < parts; q++) {
        produce(q);
        CGFD_CK(cudaMemcpyAsync(static_cast<char *>(dst) + q * n, src, n, cudaMemcpyDeviceToHost, st));
      }
      return;
    }
    const size_t per = (n + chunk - 1) / chunk, nch = per * parts;
    auto issue = [&](size_t c) {
      const size_t o = c % per * chunk, m = std::min(chunk, n - o);
      if (o == 0) produce((int)(c / per));
      CGFD_CK(cudaEventSynchronize(done_[c & 1]));
      for (size_t a = 0; a < m; a += kPiece)
        CGFD_CK(cudaMemcpyAsync(buf_[c & 1][a / kPiece], static_cast<const char *>(src) + o + a, std::min(kPiece, m - a),
                                cudaMemcpyDeviceToHost, st));
      CGFD_CK(cudaEventRecord(done_[c & 1], st));
    };
    if (nch == 0) return;
    issue(0);
    for (size_t c = 0; c < nch; c++) {
      if (c + 1 < nch) issue(c + 1);
      CGFD_CK(cudaEventSynchronize(done_[c & 1]));
      const size_t o = c % per * chunk;
      char *out = static_cast<char *>(dst) + c / per * n + o;
      for_spans(std::min(chunk, n - o), buf_[c & 1], [&](size_t a, char *b, size_t m) { std::memcpy(out + a, b, m); });
    }
    next_ = (int)(nch & 1);
  }
  void copy_out(void *dst, const void *src, size_t n, cudaStream_t st) {
    copy_out(dst, src, n, 1, st, [](int) {});
  }

  void copy(void *dst, const void *src, size_t n, cudaStream_t st) {
    const size_t chunk = even(n, ready(std::min(n, kMaxIn)));
    if (chunk == 0) {
      CGFD_CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st));
      return;
    }
    for (size_t o = 0; o < n; o += chunk) {
      const size_t m = std::min(chunk, n - o);
      const int b = next_;
      next_ ^= 1;
      CGFD_CK(cudaEventSynchronize(done_[b]));  // the previous copy out of this chunk has finished
      const char *in = static_cast<const char *>(src) + o;
      for_spans(m, buf_[b], [&](size_t a, char *to, size_t len) { std::memcpy(to, in + a, len); });
      for (size_t a = 0; a < m; a += kPiece)
        CGFD_CK(cudaMemcpyAsync(static_cast<char *>(dst) + o + a, buf_[b][a / kPiece], std::min(kPiece, m - a),
                                cudaMemcpyHostToDevice, st));
      CGFD_CK(cudaEventRecord(done_[b], st));
    }
  }

 private:
  static constexpr size_t kPiece = size_t(8) << 20, kSpan = size_t(1) << 18;
  static constexpr size_t kPieces = 8;  // of a chunk, at most
  static constexpr size_t kMaxIn = 4 * kPiece;  // of a chunk of an upload

  PinnedStager() = default;
  // Bytes that both chunks hold once pieces for n are there (the device is current); 0: no pinned memory.
  size_t ready(size_t n) {
    const size_t want = std::min(kPieces, std::max<size_t>(1, (n + kPiece - 1) / kPiece));
    for (int b = 0; b < 2; b++)
      if (!done_[b]) CGFD_CK(cudaEventCreateWithFlags(&done_[b], cudaEventDisableTiming));
    for (size_t s = 0; s < want; s++)
      for (int b = 0; b < 2; b++)
        if (!buf_[b][s] && cudaHostAlloc(reinterpret_cast<void **>(&buf_[b][s]), kPiece, cudaHostAllocPortable) != cudaSuccess) {
          cudaGetLastError();
          buf_[b][s] = nullptr;
          return s * kPiece;
        }
    return want * kPiece;
  }
  // n bytes in equal chunks of at most `most`: the length of one
  static size_t even(size_t n, size_t most) {
    if (most == 0 || n <= most) return most;
    const size_t parts = (n + most - 1) / most;
    return std::min(most, ((n + parts - 1) / parts + 4095) / 4096 * 4096);
  }
  // fn(offset, pinned bytes there, length) over the first m bytes of a chunk, by the host threads
  template <typename Fn>
  static void for_spans(size_t m, char *const *piece, Fn fn) {
    const long long spans = (long long)((m + kSpan - 1) / kSpan);
#pragma omp parallel for schedule(static)
    for (long long q = 0; q < spans; q++) {
      const size_t a = (size_t)q * kSpan;
      fn(a, piece[a / kPiece] + a % kPiece, std::min(kSpan, m - a));
    }
  }
  std::mutex mu_;
  char *buf_[2][kPieces] = {};
  cudaEvent_t done_[2] = {nullptr, nullptr};
  int next_ = 0;
};

}  // namespace cgfd
