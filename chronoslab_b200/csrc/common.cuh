// Shared helpers of the chronos_b200 library: status handling, device buffers,
// warp/block reductions.  sm_100a only.
#pragma once

#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "errors.h"

namespace chronos {

#define CHRONOS_CUDA(call)                                                        \
  do {                                                                              \
    cudaError_t e_ = (call);                                                        \
    if (e_ != cudaSuccess) {                                                        \
      throw ::chronos::Error(CHRONOS_ECUDA, std::string(#call) + ": " +             \
                                                cudaGetErrorString(e_) + " at " +   \
                                                __FILE__ + ":" + std::to_string(__LINE__)); \
    }                                                                               \
  } while (0)

#define CHRONOS_CHECK_LAUNCH() CHRONOS_CUDA(cudaGetLastError())

// Bytes held by live DBuf allocations of this process, and the cap that
// CHRONOS_DEVICE_ALLOC_CAP (bytes; unset or 0: none) puts on them.  The cap
// turns an allocation beyond it into CHRONOS_ENOMEM exactly as a failing
// cudaMalloc would, so out-of-memory handling is testable without filling a
// GPU.
inline std::atomic<int64_t> &device_bytes_live() {
  static std::atomic<int64_t> live{0};
  return live;
}
inline int64_t device_alloc_cap() {
  static const int64_t cap = [] {
    const char *e = std::getenv("CHRONOS_DEVICE_ALLOC_CAP");
    return e ? (int64_t)std::atoll(e) : (int64_t)0;
  }();
  return cap;
}

// The streams that the library's work runs on (entry points that take a
// caller's stream join it by events).  A buffer is freed after waiting for
// them, and a stream is waited for before it is destroyed.  The lock also
// covers the library's stream captures, and the joining of a handle's stream to
// a caller's capture: a stream that is being captured must not be synchronised.
struct LibStreams {
  std::mutex mu;
  std::vector<std::pair<int, cudaStream_t>> list;       // device, stream
};
inline LibStreams &lib_streams() {
  static LibStreams *s = new LibStreams;                // outlives static objects
  return *s;
}
inline cudaStream_t stream_create() {
  int dev = 0;
  cudaStream_t st = nullptr;
  CHRONOS_CUDA(cudaGetDevice(&dev));
  CHRONOS_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  LibStreams &l = lib_streams();
  std::lock_guard<std::mutex> lk(l.mu);
  l.list.emplace_back(dev, st);
  return st;
}
inline void stream_destroy(cudaStream_t st) {
  if (!st) return;
  cudaStreamSynchronize(st);
  {
    LibStreams &l = lib_streams();
    std::lock_guard<std::mutex> lk(l.mu);
    for (size_t k = 0; k < l.list.size(); ++k)
      if (l.list[k].second == st) {
        l.list.erase(l.list.begin() + k);
        break;
      }
  }
  cudaStreamDestroy(st);
}
// Waits for the device's library streams; false where a caller's capture holds
// one of them (its earlier work may still be running).
inline bool wait_lib_streams(int device) {
  LibStreams &l = lib_streams();
  std::lock_guard<std::mutex> lk(l.mu);
  bool all = true;
  for (auto &e : l.list) {
    if (e.first != device) continue;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(e.second, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
      cudaStreamSynchronize(e.second);
    else
      all = false;
  }
  return all;
}

// Waits for everything queued on a device, the work of streams that are not the
// library's too, and beside a capture (where cudaDeviceSynchronize is not allowed):
// cudaFree of memory from cudaMalloc is that wait.  The word is taken when the
// need for the wait arises, so that a full device cannot prevent it.
class DeviceWait {
 public:
  DeviceWait() = default;
  ~DeviceWait() { wait(); }
  DeviceWait(const DeviceWait &) = delete;
  DeviceWait &operator=(const DeviceWait &) = delete;
  bool armed() const { return armed_; }
  void arm() {
    if (armed_) return;
    armed_ = true;
    Relaxed mode;
    if (cudaMalloc(&word_, sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      word_ = nullptr;
    }
  }
  void wait() {
    if (!armed_) return;
    Relaxed mode;
    const cudaError_t e = word_ ? cudaFree(word_) : cudaDeviceSynchronize();
    if (e != cudaSuccess) cudaGetLastError();
    word_ = nullptr;
    armed_ = false;
  }

 private:
  // cudaMalloc and cudaFree allowed on this thread whatever is being captured
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  };
  void *word_ = nullptr;
  bool armed_ = false;
};

// Device memory comes from one memory pool per device, owned by the library
// (the default pool's settings are the host program's).  A setup makes and
// drops hundreds of buffers, and mapping and unmapping their pages was most of
// the time of its small steps: the sixteen sparse products that fold the levels
// of Poisson 32^3 took 15.4 ms with cudaMalloc and cudaFree, 6.6 ms with the
// pool; a setup of diffusion 36^3 55 and 36 ms.  The pool keeps at most
// kPoolKeepBytes beyond what is in use; what exceeds it goes back to the driver
// at once, all of it before an allocation is given up (and at exit).
// Allocations and frees are ordered on a stream of the pool's own.  A free
// waits for the library's streams first (cudaFree waits for the device), so
// memory never returns to the pool while work that the library queued may still
// use it; a handle that a caller's capture took in waits for the device before
// it frees, since replays run on the caller's streams (Hier::replays).
constexpr int64_t kPoolKeepBytes = (int64_t)512 << 20;
struct DevicePool {
  int device = -1;
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;

  cudaError_t alloc(void **p, size_t bytes) {
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      cudaStreamSynchronize(st);                        // frees still in its queue
      cudaMemPoolTrimTo(pool, 0);
      e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    }
    // the memory is there for every stream once the pool's own has passed it
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
  }
  // p: nothing queued uses it any more
  void free_idle(void *p) {
    cudaFreeAsync(p, st);
  }
  void trim() {
    uint64_t held = 0, used = 0;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
        held > used + (uint64_t)kPoolKeepBytes) {
      cudaStreamSynchronize(st);
      cudaMemPoolTrimTo(pool, used + (uint64_t)kPoolKeepBytes);
    }
  }
};
// The current device's pool.
inline DevicePool &device_pool() {
  static std::mutex mu;
  static DevicePool *pools = new DevicePool[64];        // outlives static buffers
  int dev = 0;
  CHRONOS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) throw Error(CHRONOS_EINVAL, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(mu);
  DevicePool &d = pools[dev];
  if (!d.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    CHRONOS_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = UINT64_MAX;                       // trim() bounds it
    CHRONOS_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    CHRONOS_CUDA(cudaStreamCreateWithFlags(&d.st, cudaStreamNonBlocking));   // allocations only
    d.device = dev;
    d.pool = pool;
  }
  return d;
}
// Makes a pool's device current for the scope.
class OnDevice {
 public:
  explicit OnDevice(int dev) {
    if (cudaGetDevice(&was_) == cudaSuccess && was_ != dev) {
      cudaSetDevice(dev);
      changed_ = true;
    }
  }
  ~OnDevice() { if (changed_) cudaSetDevice(was_); }
  OnDevice(const OnDevice &) = delete;
  OnDevice &operator=(const OnDevice &) = delete;

 private:
  int was_ = 0;
  bool changed_ = false;
};

// Deferred frees.  A free waits for all work queued on the device, so
// while a batch setup builds hierarchies on several host threads, one
// thread's free of a setup temporary would wait for every other thread's
// queued kernels; and nothing can be waited for while a caller's capture holds a
// handle's stream: such a buffer is kept until a later free.  A free of many
// buffers also takes one wait this way: 64 problems with a stream each took 590 ms
// to free with a wait a buffer (335 with cudaFree), 36 ms with one.
// Inside a DeferFrees scope (any thread) the buffers a DBuf
// lets go of are kept -- never reused -- and freed, after one wait for the
// streams, when the outermost scope ends or an allocation would be refused.
// They stay counted in device_bytes_live() until then.
struct DeferredFrees {
  struct Entry { void *p; int64_t bytes; DevicePool *pool; };
  std::mutex mu;
  std::vector<Entry> list;
  std::atomic<int> depth{0};
};
inline DeferredFrees &deferred_frees() {
  static DeferredFrees d;
  return d;
}
inline void flush_deferred_frees() {
  DeferredFrees &d = deferred_frees();
  std::vector<DeferredFrees::Entry> list;
  {
    std::lock_guard<std::mutex> lk(d.mu);
    list.swap(d.list);
  }
  DevicePool *synced = nullptr;
  for (auto &e : list) {
    OnDevice on(e.pool->device);
    if (e.pool != synced) {
      if (!wait_lib_streams(e.pool->device)) {
        std::lock_guard<std::mutex> lk(d.mu);
        d.list.push_back(e);
        continue;
      }
      synced = e.pool;
    }
    e.pool->free_idle(e.p);
    device_bytes_live() -= e.bytes;
  }
  if (synced) {
    OnDevice on(synced->device);
    synced->trim();
  }
}
// State that an owner keeps between its calls only to spare the next one making it
// again.  A call takes it, and parks it again, idle, when it is done; parked states
// of every owner are given up before an allocation is refused.
struct IdleStates {
  std::mutex mu;
  std::vector<std::pair<const void *, std::shared_ptr<void>>> list;
  std::shared_ptr<void> take(const void *owner) {
    std::shared_ptr<void> s;
    std::lock_guard<std::mutex> lk(mu);
    for (size_t k = 0; k < list.size() && !s; ++k)
      if (list[k].first == owner) {
        s = std::move(list[k].second);
        list.erase(list.begin() + k);
      }
    return s;
  }
  void park(const void *owner, std::shared_ptr<void> s) {
    std::lock_guard<std::mutex> lk(mu);
    list.emplace_back(owner, std::move(s));
  }
  void give_up() {
    decltype(list) all;
    std::lock_guard<std::mutex> lk(mu);
    all.swap(list);
    for (auto &e : all) e.second.reset();
  }
};
inline IdleStates &idle_states() {
  static IdleStates *s = new IdleStates;                // outlives static handles
  return *s;
}
// Gives back what the library holds without need.
inline void give_back() {
  idle_states().give_up();
  flush_deferred_frees();
}

// Whether the device (and CHRONOS_DEVICE_ALLOC_CAP) has room for so many bytes more.
inline bool device_room_now(int64_t bytes) {
  const int64_t cap = device_alloc_cap();
  if (cap > 0 && device_bytes_live().load() + bytes > cap) return false;
  uint64_t held = 0, used = 0;
  DevicePool &pool = device_pool();
  CHRONOS_CUDA(cudaMemPoolGetAttribute(pool.pool, cudaMemPoolAttrReservedMemCurrent, &held));
  CHRONOS_CUDA(cudaMemPoolGetAttribute(pool.pool, cudaMemPoolAttrUsedMemCurrent, &used));
  const int64_t idle = (int64_t)(held - std::min(used, held));
  if (idle >= bytes) return true;
  size_t avail = 0, total = 0;
  CHRONOS_CUDA(cudaMemGetInfo(&avail, &total));
  return (int64_t)avail + idle >= bytes;
}
inline bool device_room(int64_t bytes) {
  if (device_room_now(bytes)) return true;
  give_back();
  return device_room_now(bytes);
}
class DeferFrees {
 public:
  explicit DeferFrees(bool from_here = true) { if (from_here) start(); }
  // (a function that lets go of several buffers at its end makes one such object in
  // front of them and starts it there: one wait for them all)
  void start() {
    if (!on_) deferred_frees().depth++;
    on_ = true;
  }
  ~DeferFrees() {
    if (on_ && --deferred_frees().depth == 0) flush_deferred_frees();
  }
  DeferFrees(const DeferFrees &) = delete;
  DeferFrees &operator=(const DeferFrees &) = delete;

 private:
  bool on_ = false;
};

// Owning device allocation (from the device's pool), movable, typed.
template <typename T>
class DBuf {
 public:
  DBuf() = default;
  explicit DBuf(size_t n) { alloc(n); }
  ~DBuf() { release(); }
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
  DBuf(DBuf &&o) noexcept : p_(o.p_), n_(o.n_), pool_(o.pool_) { o.p_ = nullptr; o.n_ = 0; }
  DBuf &operator=(DBuf &&o) noexcept {
    if (this != &o) {
      release();
      p_ = o.p_; n_ = o.n_; pool_ = o.pool_;
      o.p_ = nullptr; o.n_ = 0;
    }
    return *this;
  }
  void alloc(size_t n) {
    release();
    if (n == 0) return;
    const int64_t bytes = (int64_t)(n * sizeof(T)), cap = device_alloc_cap();
    auto beyond_cap = [&] { return cap > 0 && device_bytes_live().load() + bytes > cap; };
    // what is kept without need is given back before a refusal
    if (beyond_cap()) give_back();
    if (beyond_cap())
      throw Error(CHRONOS_ENOMEM, "allocation of " + std::to_string(bytes) +
                                      " bytes beyond CHRONOS_DEVICE_ALLOC_CAP");
    DevicePool &pool = device_pool();
    void *p = nullptr;
    cudaError_t e = pool.alloc(&p, n * sizeof(T));
    if (e == cudaErrorMemoryAllocation) {
      give_back();
      e = pool.alloc(&p, n * sizeof(T));
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      throw Error(CHRONOS_ENOMEM, "device allocation of " + std::to_string(n * sizeof(T)) +
                                      " bytes failed: " + cudaGetErrorString(e));
    }
    p_ = static_cast<T *>(p);
    pool_ = &pool;
    n_ = n;
    device_bytes_live() += bytes;
  }
  void release() {
    if (p_) {
      DeferredFrees &d = deferred_frees();
      bool kept = false;
      {
        std::lock_guard<std::mutex> lk(d.mu);
        d.list.push_back({p_, (int64_t)(n_ * sizeof(T)), pool_});
        kept = d.depth.load() > 0;
      }
      if (!kept) flush_deferred_frees();
    }
    p_ = nullptr;
    n_ = 0;
  }
  void upload(const T *h, size_t n, cudaStream_t s = 0) {
    if (n_ < n) alloc(n);
    if (n) CHRONOS_CUDA(cudaMemcpyAsync(p_, h, n * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void upload(const std::vector<T> &h, cudaStream_t s = 0) { upload(h.data(), h.size(), s); }
  void download(T *h, size_t n, cudaStream_t s = 0) const {
    if (n) CHRONOS_CUDA(cudaMemcpyAsync(h, p_, n * sizeof(T), cudaMemcpyDeviceToHost, s));
  }
  std::vector<T> to_host(cudaStream_t s = 0) const {
    std::vector<T> h(n_);
    download(h.data(), n_, s);
    CHRONOS_CUDA(cudaStreamSynchronize(s));
    return h;
  }
  void zero(cudaStream_t s = 0) {
    if (n_) CHRONOS_CUDA(cudaMemsetAsync(p_, 0, n_ * sizeof(T), s));
  }
  T *get() const { return p_; }
  size_t size() const { return n_; }
  operator T *() const { return p_; }

 private:
  T *p_ = nullptr;
  size_t n_ = 0;
  DevicePool *pool_ = nullptr;
};

// ---- device helpers ------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over groups of L consecutive lanes (L a power of two <= 32); every lane
// of the group ends with the group sum.
template <int L, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic block reduction of one double per thread; result valid in
// thread 0.  blockDim.x must be a multiple of 32 and <= 1024.
__device__ __forceinline__ double block_sum(double v, double *smem32) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) smem32[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    r = lane < nw ? smem32[lane] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  return r;
}

// Orders this thread's earlier accesses before its later ones for the whole
// GPU (release before, acquire after a ticket).
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Lets a kernel's blocks have as much dynamic shared memory as the device gives a
// block.  The limit belongs to the process: set to each call's own size,
// concurrent setups lowered it under one another's launches.
template <typename Kernel> inline void allow_dynamic_smem(Kernel kern) {
  int dev = 0, most = 0;
  cudaFuncAttributes fa{};
  CHRONOS_CUDA(cudaGetDevice(&dev));
  CHRONOS_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  CHRONOS_CUDA(cudaFuncGetAttributes(&fa, kern));
  CHRONOS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    most - (int)fa.sharedSizeBytes));
}

// ---- programmatic dependent launch ------------------------------------------
// Kernels of the solve loop begin with pdl_begin(): griddepcontrol.wait
// returns once the preceding kernel of the stream has completed and its
// writes are visible (a no-op for a kernel launched without the attribute),
// then griddepcontrol.launch_dependents lets the next kernel's blocks be
// scheduled while this one drains.  Nothing is read or written before the
// wait, so the order of memory effects is the plain stream order.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
}

// Programmatic dependent launch is on unless CHRONOS_PDL=0 in the environment.
inline bool pdl_enabled() {
  static const int on = [] {
    const char *e = std::getenv("CHRONOS_PDL");
    return (e && e[0] == '0') ? 0 : 1;
  }();
  return on != 0;
}

// Launch of a kernel that begins with pdl_begin(), with the programmatic
// stream serialization attribute when enabled.
template <typename... KArgs, typename... Args>
void launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  CHRONOS_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
}

inline int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    CHRONOS_CUDA(cudaGetDevice(&dev));
    CHRONOS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  return sms;
}

inline unsigned ceil_div(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

}  // namespace chronos
