// Device memory and stream sets of the interpreters of one GPU.
//
// An interpreter owns a few hundred device buffers (every tensor of the module stays resident) and two streams. With
// cudaMalloc / cudaFree each of them costs a driver call that also waits for the whole device, and
// cudaGetDeviceProperties and the stream and event calls cost milliseconds more: the auto-tuner, which loads one small
// module per tuned op, spent 95% of its time there (102 ms for 17 modules of a few ops; 5 ms per module).
// Weights, tables and staging therefore come from a stream-ordered memory pool of this library's own
// (cudaMallocFromPoolAsync), and the streams and events of a destroyed interpreter are handed to the next one. Tensors,
// whose addresses callers ask for (tpucb_interp_tensor_device), are blocks of cudaMalloc, which other processes can open
// (cudaIpcGetMemHandle) and peers can read; the blocks of a destroyed module are kept for the next one.
//
// All are bounded and given back: when a module goes, free memory above kPoolKeepBytes (the pool) and kBlockKeepBytes (the
// blocks, a hundredth of the GPU's memory) returns to the driver, at most kPoolKeepStreams idle stream sets are kept, and when the last interpreter of a GPU goes, everything
// goes. Several threads may use it at once (one mutex around the lists; the pool calls are thread-safe themselves). A pool
// buffer is allocated and freed on its interpreter's stream, which is idle when the interpreter is destroyed; a block is
// given back only when nothing uses it any more, so the next owner need not wait for the former one's stream.
#pragma once
#include "host_common.h"

#include <algorithm>
#include <iterator>
#include <mutex>

namespace tpucb {

constexpr size_t kPoolKeepBytes = 256u << 20;
constexpr size_t kBlockKeepBytes = 2048ull << 20;
constexpr size_t kPoolKeepStreams = 8;

// The error word of an interpreter: kernels that give up write their code here and, through `host`, into pinned host
// memory (report_error), so that the host learns of it from its own memory after an ordinary stream synchronisation: the
// read-back of the device word cost every synchronous call a second driver round trip (14.5 us for a synchronisation with
// it, 4 us without).
struct ErrWord {
  int code;
  int pad_;
  int *host;
};

// A ring of pinned slots that pieces of an upload pass through, each allocated at its first use. Of a set's two, `small` serves
// uploads below kLargeUpload: the driver cuts requests below 1 MB from pinned chunks of 2 MB (1 to 3 ms each, then 3 us a
// request), and these slots, the download buffer and the error word fit the chunk that the error word was cut from (four
// slots of 1 MB made the first call of a module 2.5 to 5 ms longer). Larger uploads are 8 to 15% faster with more than
// 512 KB handed to the copying threads at once (154 MB: 5.2 ms against 6.1) and have the time to allocate for it.
constexpr size_t kLargeUpload = 64u << 20;
constexpr int kMaxUploadSlots = 4;
struct UploadRing {
  size_t slot_bytes;
  int slots;
  int next = 0;
  uint8_t *mem[kMaxUploadSlots] = {};
  cudaEvent_t read[kMaxUploadSlots] = {}; // the copies that read the slot are done
};
constexpr size_t kDownloadBytes = 32u << 10; // its pinned download buffer (256 KB written that way: 11 us more than by a copy)

struct StreamSet {
  cudaStream_t stream = nullptr, copy_stream = nullptr;
  cudaEvent_t upload_done[2] = {nullptr, nullptr}, staging_free[2] = {nullptr, nullptr};
  ErrWord *d_err = nullptr; // the interpreter's device error word
  int *h_err = nullptr;     // ... and its host part
  // pinned, device-visible buffers of set_tensor / get_tensor, allocated at first use
  float *download = nullptr;
  UploadRing small{512u << 10, 3}, large{1u << 20, 4};
};

class DevicePool {
public:
  // The pools live until the process ends (no CUDA call from a static destructor).
  static DevicePool &of(int device) {
    static std::mutex m;
    static std::map<int, DevicePool *> *pools = new std::map<int, DevicePool *>();
    std::lock_guard<std::mutex> lock(m);
    DevicePool *&p = (*pools)[device];
    if (!p) p = new DevicePool(device);
    return *p;
  }

  int sm_count = 148;

  // One interpreter more on this device (current on the calling thread): its streams, events and error word (zero).
  StreamSet acquire() {
    std::lock_guard<std::mutex> lock(m_);
    StreamSet s;
    if (!idle_.empty()) {
      s = idle_.back();
      idle_.pop_back();
    } else {
      TPUCB_CUDA(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
      TPUCB_CUDA(cudaStreamCreateWithFlags(&s.copy_stream, cudaStreamNonBlocking));
      for (int i = 0; i < 2; ++i) {
        TPUCB_CUDA(cudaEventCreateWithFlags(&s.upload_done[i], cudaEventDisableTiming));
        TPUCB_CUDA(cudaEventCreateWithFlags(&s.staging_free[i], cudaEventDisableTiming));
      }
      TPUCB_CUDA(cudaMallocFromPoolAsync((void **)&s.d_err, sizeof(ErrWord), mem_, s.stream));
      TPUCB_CUDA(cudaHostAlloc((void **)&s.h_err, 64, cudaHostAllocMapped));
      const ErrWord w{0, 0, s.h_err};
      TPUCB_CUDA(cudaMemcpyAsync(s.d_err, &w, sizeof(w), cudaMemcpyHostToDevice, s.stream));
    }
    ++live_;
    *s.h_err = 0;
    TPUCB_CUDA(cudaMemsetAsync(&s.d_err->code, 0, sizeof(int), s.stream));
    return s;
  }
  // ... and one less. Nothing may still run on its streams and all of its buffers are freed.
  void release(const StreamSet &s) {
    cudaStreamSynchronize(s.stream);
    trim();
    std::lock_guard<std::mutex> lock(m_);
    idle_.push_back(s);
    if (--live_ > 0 && idle_.size() <= kPoolKeepStreams) return;
    while (!idle_.empty() && (live_ == 0 || idle_.size() > kPoolKeepStreams)) {
      StreamSet &d = idle_.back();
      cudaFreeAsync(d.d_err, d.stream);
      cudaStreamSynchronize(d.stream);
      cudaFreeHost(d.h_err);
      if (d.download) cudaFreeHost(d.download);
      for (UploadRing *r : {&d.small, &d.large})
        for (int i = 0; i < kMaxUploadSlots; ++i) {
          if (r->mem[i]) cudaFreeHost(r->mem[i]);
          if (r->read[i]) cudaEventDestroy(r->read[i]);
        }
      for (int i = 0; i < 2; ++i) {
        cudaEventDestroy(d.upload_done[i]);
        cudaEventDestroy(d.staging_free[i]);
      }
      cudaStreamDestroy(d.copy_stream);
      cudaStreamDestroy(d.stream);
      idle_.pop_back();
    }
    if (live_ == 0) {
      drop_blocks(0);
      cudaMemPoolTrimTo(mem_, 0);
    }
  }

  void *alloc(size_t bytes, cudaStream_t stream) {
    void *p = nullptr;
    TPUCB_CUDA(cudaMallocFromPoolAsync(&p, bytes ? bytes : 16, mem_, stream));
    return p;
  }

  // A tensor's storage: a free block of at most a quarter more, or a new one (a block of 1 MB and more costs the driver 0.3 ms
  // to allocate and as much to free).
  void *alloc_block(size_t bytes) {
    const size_t need = (std::max<size_t>(bytes, 16) + 511) / 512 * 512;
    std::lock_guard<std::mutex> lock(m_);
    auto it = free_blocks_.lower_bound(need);
    if (it != free_blocks_.end() && it->first <= need + need / 4) {
      it = std::prev(free_blocks_.upper_bound(it->first)); // of its size the one freed last: L2 and TLB may still hold it
      void *p = it->second;
      free_bytes_ -= it->first;
      blocks_[p] = it->first;
      free_blocks_.erase(it);
      return p;
    }
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, need);
    if (e == cudaErrorMemoryAllocation) { // what lies free here may make room
      cudaGetLastError();
      drop_blocks(0);
      cudaMemPoolTrimTo(mem_, 0);
      e = cudaMalloc(&p, need);
    }
    TPUCB_CUDA(e);
    blocks_[p] = need;
    return p;
  }
  // Nothing on the device may still use the block.
  void free_block(void *p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(m_);
    auto it = blocks_.find(p);
    free_blocks_.insert({it->second, p});
    free_bytes_ += it->second;
    blocks_.erase(it);
    drop_blocks(kBlockKeepBytes);
  }

  // Gives the driver back what lies free above kPoolKeepBytes. Called where a module's buffers have been freed; in between
  // the pool holds on to what it has (its release threshold counts the memory in use too, so with any finite threshold
  // a process that holds a large module would unmap and map again at every synchronisation: 40 ms spikes).
  void trim() {
    uint64_t used = 0;
    if (cudaMemPoolGetAttribute(mem_, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess)
      cudaMemPoolTrimTo(mem_, used + kPoolKeepBytes);
  }

private:
  // Gives free blocks back to the driver, the largest first, until no more than `keep` bytes are left.
  void drop_blocks(size_t keep) {
    while (free_bytes_ > keep) {
      auto it = std::prev(free_blocks_.end());
      cudaFree(it->second);
      free_bytes_ -= it->first;
      free_blocks_.erase(it);
    }
  }

  explicit DevicePool(int device) {
    int major = 0, minor = 0;
    TPUCB_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    TPUCB_CUDA(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
    TPUCB_CHECK(major == 10, "this backend is written for sm_100a (B200); device %d is sm_%d%d", device, major, minor);
    TPUCB_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    TPUCB_CUDA(cudaMemPoolCreate(&mem_, &props));
    uint64_t keep = UINT64_MAX; // see trim()
    TPUCB_CUDA(cudaMemPoolSetAttribute(mem_, cudaMemPoolAttrReleaseThreshold, &keep));
  }

  std::mutex m_;
  cudaMemPool_t mem_ = nullptr;
  std::vector<StreamSet> idle_;
  std::multimap<size_t, void *> free_blocks_; // by size
  std::map<void *, size_t> blocks_;           // in use
  size_t free_bytes_ = 0;
  int live_ = 0;
};

} // namespace tpucb
