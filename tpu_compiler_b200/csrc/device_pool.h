// Device memory and stream sets of the interpreters of one GPU.
//
// An interpreter owns a few hundred device buffers (every tensor of the module stays resident) and two streams. With
// cudaMalloc / cudaFree each of them costs a driver call that also waits for the whole device, and
// cudaGetDeviceProperties and the stream and event calls cost milliseconds more: the auto-tuner, which loads one small
// module per tuned op, spent 95% of its time there (102 ms for 17 modules of a few ops; 5 ms per module).
// Buffers therefore come from a stream-ordered memory pool of this library's own (cudaMallocFromPoolAsync), and the
// streams and events of a destroyed interpreter are handed to the next one.
//
// Both are bounded and given back: when a module goes, free memory above kPoolKeepBytes returns to the driver, at most
// kPoolKeepStreams idle stream sets are kept, and when the last interpreter of a GPU goes, everything goes.
// Several threads may use it at once (one mutex around the lists; the pool calls are thread-safe themselves). A buffer is
// allocated and freed on its interpreter's stream, which is idle when the interpreter is destroyed.
#pragma once
#include "host_common.h"

#include <mutex>

namespace tpucb {

constexpr size_t kPoolKeepBytes = 256u << 20;
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

constexpr size_t kUploadSlot = 1u << 20; // bytes of one of the pinned upload slots of a stream set
constexpr int kUploadSlots = 4;
constexpr size_t kDownloadBytes = 32u << 10; // its pinned download buffer (256 KB written that way: 11 us more than by a copy)

struct StreamSet {
  cudaStream_t stream = nullptr, copy_stream = nullptr;
  cudaEvent_t upload_done[2] = {nullptr, nullptr}, staging_free[2] = {nullptr, nullptr};
  ErrWord *d_err = nullptr; // the interpreter's device error word
  int *h_err = nullptr;     // ... and its host part
  // pinned, device-visible buffers of set_tensor / get_tensor, allocated at first use
  float *download = nullptr;
  uint8_t *upload = nullptr;
  cudaEvent_t upload_read[kUploadSlots] = {}; // the kernels that read the slot are done
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
      if (d.upload) cudaFreeHost(d.upload);
      for (cudaEvent_t e : d.upload_read)
        if (e) cudaEventDestroy(e);
      for (int i = 0; i < 2; ++i) {
        cudaEventDestroy(d.upload_done[i]);
        cudaEventDestroy(d.staging_free[i]);
      }
      cudaStreamDestroy(d.copy_stream);
      cudaStreamDestroy(d.stream);
      idle_.pop_back();
    }
    if (live_ == 0) cudaMemPoolTrimTo(mem_, 0);
  }

  void *alloc(size_t bytes, cudaStream_t stream) {
    void *p = nullptr;
    TPUCB_CUDA(cudaMallocFromPoolAsync(&p, bytes ? bytes : 16, mem_, stream));
    return p;
  }

  cudaMemPool_t handle() const { return mem_; }

  // Gives the driver back what lies free above kPoolKeepBytes. Called where a module's buffers have been freed; in between
  // the pool holds on to what it has (its release threshold counts the memory in use too, so with any finite threshold
  // a process that holds a large module would unmap and map again at every synchronisation: 40 ms spikes).
  void trim() {
    uint64_t used = 0;
    if (cudaMemPoolGetAttribute(mem_, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess)
      cudaMemPoolTrimTo(mem_, used + kPoolKeepBytes);
  }

private:
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
  int live_ = 0;
};

} // namespace tpucb
