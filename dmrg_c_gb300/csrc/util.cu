// util.cu -- error state, device / stream management, small host helpers.
#include <atomic>
#include <chrono>
#include <cstdarg>
#include <exception>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace dg {

namespace {
thread_local char g_err[1024] = {0};
std::atomic<long> g_launches{0};
}

void count_launch(long k) { g_launches.fetch_add(k, std::memory_order_relaxed); }

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

const char *last_error() { return g_err; }

void require_device() {
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0) {
    set_error("no CUDA device available (%s)", e == cudaSuccess ? "0 devices" : cudaGetErrorString(e));
    throw Error{DG_ERR_NODEVICE};
  }
}

// ---- streams ----------------------------------------------------------------------------
// A thread's stream goes back to its device's list when the thread ends, and the next thread
// takes it from there.  The worker threads of the batched and served forms live for one call or
// one engine; with a stream created for each of them and never given back, every stream a
// process had ever used stayed in the driver's list that a stream-ordered allocation walks:
// after ~100 batched calls of 9 threads each a resident expectation value took 10.5 ms instead
// of 0.25 ms and a batched solve of 24 chains 76 ms instead of 27.
// A call that gave up (a wait that ran out, an allocation that failed) leaves work queued on its
// stream: such a stream stays in the list, and is passed over until the work has finished, so that
// no other thread waits behind it.
namespace {
// Queries of streams and events that another thread's stream capture must not see.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() {
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaPeekAtLastError() == cudaErrorNotReady) cudaGetLastError();   // a query's, no error of the caller's
  }
};
constexpr int kMaxPoolDevices = 64;
constexpr size_t kKeptStreams = 64;   // idle streams kept per device; more are destroyed
struct IdleStreams {
  std::mutex mu;
  std::vector<cudaStream_t> idle[kMaxPoolDevices];
};
// never destroyed: threads may end after static destruction has begun
IdleStreams &idle_streams() {
  static IdleStreams *s = new IdleStreams();
  return *s;
}
struct ThreadStream {
  cudaStream_t s = nullptr;
  int dev = -1;
  void give_back() {
    if (!s) return;
    bool kept = false;
    if (dev >= 0 && dev < kMaxPoolDevices) {
      IdleStreams &is = idle_streams();
      std::lock_guard<std::mutex> lk(is.mu);
      if (is.idle[dev].size() < kKeptStreams) {
        is.idle[dev].push_back(s);
        kept = true;
      }
    }
    if (!kept) cudaStreamDestroy(s);
    s = nullptr;
  }
  void take(int device) {
    if (device >= 0 && device < kMaxPoolDevices) {
      IdleStreams &is = idle_streams();
      std::lock_guard<std::mutex> lk(is.mu);
      std::vector<cudaStream_t> &idle = is.idle[device];
      if (!idle.empty()) {
        RelaxedCapture relaxed;
        for (size_t i = idle.size(); i-- > 0 && !s;)
          if (cudaStreamQuery(idle[i]) == cudaSuccess) {
            s = idle[i];
            idle.erase(idle.begin() + (long)i);
          }
      }
    }
    if (!s) DG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    dev = device;
  }
  ~ThreadStream() { give_back(); }
};
}  // namespace

cudaStream_t stream() {
  thread_local ThreadStream t;
  int cur = 0;
  DG_CUDA(cudaGetDevice(&cur));
  if (!t.s || t.dev != cur) {
    t.give_back();
    t.take(cur);
  }
  return t.s;
}

// ---- device memory pool ---------------------------------------------------------------
namespace {
std::mutex g_pool_mutex;
cudaMemPool_t g_pools[kMaxPoolDevices] = {nullptr};

uint64_t pool_keep_bytes() {
  const char *s = getenv("DG_POOL_KEEP_MB");
  if (s && *s) return (uint64_t)strtoull(s, nullptr, 10) << 20;
  return 8ull << 30;
}
}  // namespace

cudaMemPool_t device_pool() {
  int dev = 0;
  DG_CUDA(cudaGetDevice(&dev));
  DG_REQUIRE(dev >= 0 && dev < kMaxPoolDevices, DG_ERR_ARG, "device %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (!g_pools[dev]) {
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    DG_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = pool_keep_bytes();
    DG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pools[dev] = pool;
  }
  return g_pools[dev];
}

// Pool holds: while any is active on a device, its pool keeps all the memory it has mapped
// across synchronisations (release threshold unbounded), so that allocations of a batch or an
// engine whose working set exceeds the default keep do not unmap and map physical memory each
// time another thread synchronises.  The last hold restores the keep and trims to it.
namespace {
int g_pool_holds[kMaxPoolDevices] = {0};
}
void pool_hold(int device, bool acquire) {
  if (device < 0 || device >= kMaxPoolDevices) return;
  int prev = 0;
  DG_CUDA(cudaGetDevice(&prev));
  DG_CUDA(cudaSetDevice(device));
  cudaMemPool_t pool = device_pool();
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  int &h = g_pool_holds[device];
  if (acquire) {
    if (h++ == 0) {
      uint64_t all = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &all);
    }
  } else if (h > 0 && --h == 0) {
    uint64_t keep = pool_keep_bytes();
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolTrimTo(pool, keep);
  }
  cudaSetDevice(prev);
}

void *pool_alloc(size_t bytes, cudaStream_t st) {
  void *p = nullptr;
  DG_CUDA(cudaMallocFromPoolAsync(&p, bytes ? bytes : 1, device_pool(), st));
  return p;
}

void pool_free(void *p, cudaStream_t st) {
  if (p) cudaFreeAsync(p, st);
}

// ---- mapped host blocks ------------------------------------------------------------------
// One list for the process: a block returned by one thread serves the next solve of any thread
// (a worker thread of the batched form lives for one call; with a list per thread it allocated
// its blocks anew and freed them at its end, and freeing pinned memory waits for the device).
// A solve returns its blocks after its stream has drained, except when an error unwinds it: kernels
// it has queued may then still write them.  Such a block waits behind an event recorded on the
// stream and is handed out again only after that.
namespace {
struct MappedBlock {
  void *h;
  size_t bytes;
  cudaEvent_t written = nullptr;   // the block's last writers (blocks in `busy`)
};
constexpr size_t kKeptBlocks = 256, kKeptBlockBytes = size_t(64) << 20;   // more are freed
struct MappedList {
  std::mutex mu;
  std::vector<MappedBlock> idle, busy;
  size_t bytes = 0;   // of both
  bool room(size_t more) const { return idle.size() + busy.size() < kKeptBlocks && bytes + more <= kKeptBlockBytes; }
  // Blocks whose writers have finished become idle.
  void collect() {
    if (busy.empty()) return;
    RelaxedCapture relaxed;
    for (size_t i = busy.size(); i-- > 0;)
      if (cudaEventQuery(busy[i].written) == cudaSuccess) {
        cudaEventDestroy(busy[i].written);
        idle.push_back(MappedBlock{busy[i].h, busy[i].bytes});
        busy[i] = busy.back();
        busy.pop_back();
      }
  }
};
MappedList &mapped_list() {   // never destroyed, as idle_streams()
  static MappedList *l = new MappedList();
  return *l;
}
}  // namespace

void *mapped_acquire(size_t bytes, size_t *got) {
  size_t want = 4096;
  while (want < bytes) want <<= 1;
  {
    MappedList &l = mapped_list();
    std::lock_guard<std::mutex> lk(l.mu);
    l.collect();
    size_t best = l.idle.size();   // the smallest block that fits
    for (size_t i = 0; i < l.idle.size(); ++i)
      if (l.idle[i].bytes >= want && (best == l.idle.size() || l.idle[i].bytes < l.idle[best].bytes)) best = i;
    if (best < l.idle.size()) {
      const MappedBlock b = l.idle[best];
      l.idle[best] = l.idle.back();
      l.idle.pop_back();
      l.bytes -= b.bytes;
      *got = b.bytes;
      return b.h;
    }
  }
  void *h = nullptr;
  DG_CUDA(cudaHostAlloc(&h, want, cudaHostAllocMapped | cudaHostAllocPortable));
  *got = want;
  return h;
}

namespace {
// An event behind everything this thread has queued; null if it cannot be had.
cudaEvent_t event_behind_stream() {
  cudaEvent_t ev = nullptr;
  try {
    cudaStream_t st = stream();
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return nullptr;
    if (cudaEventRecord(ev, st) == cudaSuccess) return ev;
    cudaEventDestroy(ev);
  } catch (const Error &) {
  }
  return nullptr;
}
}  // namespace

void mapped_return(void *h, size_t bytes) {
  if (!h) return;
  const bool unwinding = std::uncaught_exceptions() > 0;
  const cudaEvent_t written = unwinding ? event_behind_stream() : nullptr;
  if (unwinding && !written) return;   // nothing says when its writers end: given up
  MappedList &l = mapped_list();
  {
    std::lock_guard<std::mutex> lk(l.mu);
    if (l.room(bytes)) {
      (unwinding ? l.busy : l.idle).push_back(MappedBlock{h, bytes, written});
      l.bytes += bytes;
      return;
    }
  }
  if (written) cudaEventDestroy(written);
  cudaFreeHost(h);   // (waits for the device)
}

// What the lists hold idle goes back: the pinned blocks and the current device's streams.
static void release_idle() {
  std::vector<MappedBlock> blocks;
  {
    MappedList &l = mapped_list();
    std::lock_guard<std::mutex> lk(l.mu);
    l.collect();
    blocks.swap(l.idle);
    for (const MappedBlock &b : blocks) l.bytes -= b.bytes;
  }
  for (const MappedBlock &b : blocks) cudaFreeHost(b.h);
  int dev = 0;
  DG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxPoolDevices) return;
  std::vector<cudaStream_t> streams;
  {
    IdleStreams &is = idle_streams();
    std::lock_guard<std::mutex> lk(is.mu);
    streams.swap(is.idle[dev]);
  }
  for (cudaStream_t s : streams) cudaStreamDestroy(s);   // (work still queued on one runs to its end)
}

int sm_count() {
  thread_local int cached = -1, dev = -1;
  int cur = 0;
  DG_CUDA(cudaGetDevice(&cur));
  if (cached < 0 || dev != cur) {
    DG_CUDA(cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, cur));
    dev = cur;
  }
  return cached;
}

int vector_grid(long n) {
  long need = (n + kThreads - 1) / kThreads;
  long cap = (long)sm_count() * 4;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}

bool runs_cluster16(const void *kernel, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, bool> known;
  int dev = 0;
  DG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  const auto it = known.find({dev, kernel});
  if (it != known.end()) return it->second;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 16;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters >= 1;
  if (!ok) cudaGetLastError();   // refused, not an error
  return known[{dev, kernel}] = ok;
}

bool is_device_ptr(const void *p) {
  if (!p) return false;
  cudaPointerAttributes a;
  cudaError_t e = cudaPointerGetAttributes(&a, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

bool is_device_only_ptr(const void *p) {
  if (!p) return false;
  cudaPointerAttributes a;
  cudaError_t e = cudaPointerGetAttributes(&a, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice;
}

double now_ms() {
  using namespace std::chrono;
  return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

}  // namespace dg

extern "C" {

const char *dg_last_error(void) { return dg::last_error(); }

int dg_device_count(void) {
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return count;
}

const char *dg_version(void) { return "dmrg_gb300 0.1 (sm_103a)"; }

long dg_kernel_launches(void) { return dg::g_launches.load(); }

int dg_release_pool(void) {
  return dg::guarded([&] {
    dg::require_device();
    DG_CUDA(cudaStreamSynchronize(dg::stream()));
    DG_CUDA(cudaMemPoolTrimTo(dg::device_pool(), 0));
    dg::release_idle();
  });
}

}  // extern "C"
