// Tables that a rebind rewrites, on their way to the device: staged in a ring
// of pinned, mapped host slots and put in place by a kernel on the caller's
// stream, which reads the slot over the host link.  A copy-engine transfer
// (cudaMemcpyAsync) would queue behind the caller's own bulk host-to-device
// copies on the same engine — the next pardo iteration's operands streaming
// in — and hold the stream for as long as they take; from pageable memory it
// would also hold the host until the stream's earlier work is done.
#pragma once

#include <algorithm>
#include <cstring>
#include <vector>

#include "a4g_internal.h"

namespace a4g {

struct TableCopy {
  const unsigned long long* src;
  unsigned long long* dst;
  int64_t words;  // 8-byte words
};
constexpr int kMaxTableCopies = 16;
struct TableCopies {
  TableCopy c[kMaxTableCopies];
  int n;
};

static __global__ void __launch_bounds__(256) copy_tables_kernel(TableCopies t) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int i = 0; i < t.n; ++i) {
    const TableCopy c = t.c[i];
    for (int64_t w = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; w < c.words; w += stride) c.dst[w] = c.src[w];
  }
}

// begin (takes the next slot, waiting for the copy that last read it), add per
// table, launch.
class TableStage {
 public:
  ~TableStage() {
    for (int i = 0; i < kRing; ++i)
      if (ev_[i]) cudaEventSynchronize(ev_[i]), cudaEventDestroy(ev_[i]);
    if (h_) cudaFreeHost(h_);
  }
  int begin(size_t bytes) {
    if (!h_ || bytes_ < bytes) {
      for (int i = 0; i < kRing; ++i)
        if (busy_[i]) {
          A4G_CUDA(cudaEventSynchronize(ev_[i]));
          busy_[i] = false;
        }
      if (h_) cudaFreeHost(h_), h_ = nullptr;
      bytes_ = std::max<size_t>(bytes, 8);
      void* h = nullptr;
      A4G_CUDA(cudaHostAlloc(&h, bytes_ * kRing, cudaHostAllocMapped));
      h_ = static_cast<char*>(h);
      void* d = nullptr;
      A4G_CUDA(cudaHostGetDevicePointer(&d, h, 0));
      d_ = static_cast<char*>(d);
      for (int i = 0; i < kRing; ++i)
        if (!ev_[i]) A4G_CUDA(cudaEventCreateWithFlags(&ev_[i], cudaEventDisableTiming));
    }
    slot_ = next_;
    next_ = (next_ + 1) % kRing;
    if (busy_[slot_]) A4G_CUDA(cudaEventSynchronize(ev_[slot_]));
    busy_[slot_] = false;
    used_ = 0;
    copies_.clear();
    return A4G_OK;
  }
  int add(void* dev, const void* host, size_t bytes) {
    if (!bytes) return A4G_OK;
    if (used_ + bytes > bytes_) return fail(A4G_ERR_RANGE, "rebind: staging slot overflow");
    const size_t at = size_t(slot_) * bytes_ + used_;
    std::memcpy(h_ + at, host, bytes);
    copies_.push_back({reinterpret_cast<const unsigned long long*>(d_ + at), static_cast<unsigned long long*>(dev),
                       int64_t(bytes / 8)});
    used_ += bytes;
    return A4G_OK;
  }
  int launch(cudaStream_t s) {
    int64_t words = 0;
    for (const TableCopy& c : copies_) words = std::max(words, c.words);
    const int grid = int(std::max<int64_t>(1, std::min<int64_t>(64, (words + 255) / 256)));
    for (size_t i = 0; i < copies_.size(); i += kMaxTableCopies) {
      TableCopies t{};
      t.n = int(std::min<size_t>(kMaxTableCopies, copies_.size() - i));
      for (int k = 0; k < t.n; ++k) t.c[k] = copies_[i + size_t(k)];
      copy_tables_kernel<<<grid, 256, 0, s>>>(t);
      A4G_CUDA(cudaGetLastError());
    }
    A4G_CUDA(cudaEventRecord(ev_[slot_], s));
    busy_[slot_] = true;
    return A4G_OK;
  }

 private:
  static constexpr int kRing = 4;
  char* h_ = nullptr;
  char* d_ = nullptr;  // the same memory as the device sees it
  size_t bytes_ = 0, used_ = 0;
  int next_ = 0, slot_ = 0;
  cudaEvent_t ev_[kRing] = {};
  bool busy_[kRing] = {};
  std::vector<TableCopy> copies_;
};

}  // namespace a4g
