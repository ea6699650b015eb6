// Small feeds on their way to the device. A request is some dozens of arrays of a few KB; a cudaMemcpyAsync for each costs
// the host more than the bytes do. So Feed copies a small array into pinned memory that the device can read (the caller's
// buffer is free as soon as Feed returns) and one kernel brings all of them over, enqueued before anything that could see
// the inputs. 36 arrays of a request: 7 us on the device instead of 63, and the call 110 us shorter.
//
// The pinned buffer is [descriptors][arrays]; `used_` is where the next array goes. Either arrays wait in it (`items_` is
// not empty) or a flushed batch is being read from it (`in_flight_`), never both. With neither, it is free from the start.
#pragma once

#include <algorithm>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "runtime.h"
#include "xdlb200.h"

namespace blaze {

// BlobT: `template <typename T> T* as()` gives the device address at the time of the flush
template <typename BlobT>
class FeedStage {
 public:
  static constexpr size_t kMaxFeed = 32 << 10;       // longer arrays: the copy engine is as cheap as the host's memcpy
  static constexpr size_t kMaxItems = 128, kBytes = 512 << 10;
  FeedStage() = default;
  FeedStage(const FeedStage&) = delete;
  ~FeedStage() {
    if (in_flight_) cudaStreamSynchronize(stream_);
    if (host_) cudaFreeHost(host_);
  }

  bool pending(const BlobT* b) const { return Find(b) < items_.size(); }
  // forgets the feed of this blob that waits: a later one that does not go through here replaces it
  void Drop(const BlobT* b) {
    const size_t i = Find(b);
    if (i < items_.size()) items_.erase(items_.begin() + (long)i);
  }
  void Add(BlobT* b, const void* data, size_t len, cudaStream_t stream) {
    if (!host_) {
      CUDA_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&host_), kBytes, cudaHostAllocMapped | cudaHostAllocPortable));
      CUDA_CHECK(cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev_), host_, 0));
    }
    const size_t i = Find(b);
    if (i < items_.size() && items_[i].len == len) {  // fed again before anything read it: the new data take its place
      memcpy(host_ + items_[i].at, data, len);
      return;
    }
    Drop(b);
    if (items_.size() == kMaxItems || used_ + len > kBytes) Flush(stream);
    if (in_flight_) {                                 // what the last kernel read may still be on its way
      CUDA_CHECK(cudaStreamSynchronize(stream_));
      Done();
    }
    if (items_.empty()) used_ = kArrays;              // (a dropped feed may have been the only one)
    BLAZE_CONDITION_THROW(used_ + len <= kBytes, "a feed of ", len, " bytes does not fit the staging buffer");
    memcpy(host_ + used_, data, len);
    items_.push_back(Item{b, used_, len});
    used_ = (used_ + len + 15) / 16 * 16;
  }
  // enqueues the copies that wait
  void Flush(cudaStream_t stream) {
    if (items_.empty()) return;
    xb_copy_item* d = reinterpret_cast<xb_copy_item*>(host_);
    size_t longest = 0;
    for (size_t i = 0; i < items_.size(); ++i) {
      d[i].src = dev_ + items_[i].at; d[i].dst = items_[i].blob->template as<void>(); d[i].bytes = (int64_t)items_[i].len;
      longest = std::max(longest, items_[i].len);
    }
    const int n = (int)items_.size();
    items_.clear();
    in_flight_ = true;
    stream_ = stream;
    XB_CHECK(xb_copy_segments(reinterpret_cast<const xb_copy_item*>(dev_), n, (int64_t)longest, stream));
  }
  // the stream of the last Flush has been synchronised since
  void Done() { in_flight_ = false; }

 private:
  struct Item { BlobT* blob; size_t at, len; };
  static constexpr size_t kArrays = kMaxItems * sizeof(xb_copy_item);
  static_assert(kArrays + kMaxFeed <= kBytes, "an empty buffer takes any array that comes here");
  size_t Find(const BlobT* b) const {
    size_t i = 0;
    while (i < items_.size() && items_[i].blob != b) ++i;
    return i;
  }
  char *host_ = nullptr, *dev_ = nullptr;
  size_t used_ = kArrays;
  std::vector<Item> items_;
  cudaStream_t stream_ = nullptr;
  bool in_flight_ = false;
};

}  // namespace blaze
