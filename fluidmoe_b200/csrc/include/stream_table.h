// What launches keep from one to the next on the same stream (counters that they use in rotation).
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace fm {

// One State per (device, stream).  A stream is known by its id, which no other stream of the process ever has: the handle
// of a destroyed stream may come back as another one while the old one's launches are still under way, and the two
// would share what only the order of one stream keeps apart.  For the same reason the handle that stands for a stream of
// each thread is a stream for each thread here.  Streams are not told apart once kMaxStreams are known, dead ones
// among them; later ones get no state and the caller does without.
template <class State>
class StreamTable {
 public:
  static constexpr size_t kMaxStreams = 64;
  std::mutex mu;      // held by the caller while it uses a state

  // False when nothing may be enqueued besides the launch itself (another stream's capture forbids it).  `*state` is
  // null on a stream that is being captured, whose launches will run again, and beyond kMaxStreams.
  bool find(cudaStream_t stream, State** state) {
    *state = nullptr;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    if (cap != cudaStreamCaptureStatusNone) return true;
    unsigned long long id = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaStreamGetId(stream, &id) != cudaSuccess) {
      (void)cudaGetLastError();
      return true;
    }
    const auto key = std::make_pair(dev, id);
    const auto it = table_.find(key);
    if (it != table_.end()) *state = &it->second;
    else if (table_.size() < kMaxStreams) *state = &table_[key];
    return true;
  }

 private:
  std::map<std::pair<int, unsigned long long>, State> table_;
};

}  // namespace fm
