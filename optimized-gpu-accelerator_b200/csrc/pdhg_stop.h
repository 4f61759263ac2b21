// Stop word of a running kernel: a device word that the host sets from beside
// the kernel's stream, by a copy on a stream of its own.
//
// Nothing orders that copy with the kernel, and it can be late (behind another
// thread's uploads, say): the kernel may have ended without it.  So the word
// lives and dies on the copy's stream: it goes back to the pool after every
// copy that was sent to it.  (Read from host-mapped memory instead, it cost
// the GPU a microsecond per block and check, one after the other over the bus:
// 65 ms of the 65 ms of 1,024 small members of 80 checks each.)
#pragma once

#include "pdhg_host_common.h"

namespace b2p {

class StopWord {
 public:
  StopWord() = default;
  StopWord(const StopWord&) = delete;
  StopWord& operator=(const StopWord&) = delete;

  // Zero on return, for kernels of any stream.
  void create(int device) {
    one_ = static_cast<int32_t*>(PinnedCache::get(sizeof(int32_t)));
    *one_ = 1;
    B2P_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    B2P_CUDA(cudaMallocFromPoolAsync(&word_, sizeof(int32_t), device_pool(device), stream_));
    B2P_CUDA(cudaMemsetAsync(word_, 0, sizeof(int32_t), stream_));
    B2P_CUDA(cudaStreamSynchronize(stream_));
  }

  // The kernels that read the word must have ended.
  ~StopWord() {
    if (word_) cudaFreeAsync(word_, stream_);
    if (stream_) {
      cudaStreamSynchronize(stream_);
      cudaStreamDestroy(stream_);
    }
    PinnedCache::put(one_, sizeof(int32_t));
  }

  const volatile int32_t* get() const { return static_cast<const volatile int32_t*>(word_); }

  // The next read of the word after the copy got through sees 1.
  void raise() { B2P_CUDA(cudaMemcpyAsync(word_, one_, sizeof(int32_t), cudaMemcpyHostToDevice, stream_)); }

 private:
  void* word_ = nullptr;
  int32_t* one_ = nullptr;
  cudaStream_t stream_ = nullptr;
};

}  // namespace b2p
