// Support counting that allocates no memory, for callers that may not call
// cudaMalloc: code that runs inside another framework's memory arena or
// allocator (which owns every device allocation and accounts for it), hosts
// with a fixed device-memory budget handed out up front, and code paths that
// must not trigger the implicit device synchronisation cudaMalloc/cudaFree can
// cause.  The caller passes device buffers it already owns for the inputs and
// the output; the only scratch, the support bitmaps, lives in the file-scope
// device array below, which every GPU that loads this library holds until the
// process exits.
//
// Same result as gs_support_count (support[k] = number of distinct graph ids
// among the records whose key is k), computed by the same three steps:
// clear the bitmap, set bit [key][graph] per record, popcount per key.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "../../include/gspan_gb300.h"
#include "gs_stamp.cuh"

namespace {

constexpr unsigned kScratchWords = GS_NOALLOC_MAX_BITMAP_WORDS;  // 4 MiB
constexpr int kMaxDevices = 64;
constexpr int kBlock = 256;

// The scratch shared by every call on a device.
static __device__ __align__(256) uint32_t g_noalloc_bitmap[kScratchWords];

std::mutex g_mu;

}  // namespace

namespace gsgb {
// the library's thread-local error text (gs_last_error), kept in gs_capi.cpp
void capi_set_error(const char *msg);
}  // namespace gsgb

namespace {

struct ErrText {
  void operator=(const char *m) { gsgb::capi_set_error(m); }
} t_msg;

using gsgb::after_previous;

// The scratch is 16-byte aligned and a multiple of 16 bytes.
__global__ void k_clear(uint32_t *bm, long long words)
{
  const long long stride = (long long)gridDim.x * blockDim.x, n = (words + 3) / 4;
  for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    reinterpret_cast<uint4 *>(bm)[i] = make_uint4(0, 0, 0, 0);
}

__device__ __forceinline__ void mark(uint32_t *bm, int k, int g, int n_keys, int n_graphs, int words)
{
  if((unsigned)k >= (unsigned)n_keys || (unsigned)g >= (unsigned)n_graphs) return;
  atomicOr(&bm[(long long)k * words + (g >> 5)], 1u << (g & 31));
}

// Records outside [0, n_keys) x [0, n_graphs) are skipped.  vec: both arrays are
// 16-byte aligned, four records a step and the next four's loads in flight; the
// first are loaded before the clear is waited for.  Bound by the bitmap ORs:
// 4 M records into 1,000 keys x 30,011 graphs take 31 us, 126 ORs per ns to
// words that few share; the loads alone would take 5.  The call: 43.0 -> 34.8 us
// with one record a step and three launches apart before.
__global__ void k_mark(uint32_t *bm, const int32_t *__restrict__ keys, const int32_t *__restrict__ gids, long long n,
                       int n_keys, int n_graphs, int words, int vec)
{
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n4 = vec ? n >> 2 : 0;
  const int4 *const k4 = reinterpret_cast<const int4 *>(keys), *const g4 = reinterpret_cast<const int4 *>(gids);
  int4 k_n = make_int4(0, 0, 0, 0), g_n = k_n;
  if(i0 < n4) {
    k_n = __ldg(&k4[i0]);
    g_n = __ldg(&g4[i0]);
  }
  after_previous();
  for(long long i = i0; i < n4; i += stride) {
    const int4 k = k_n, g = g_n;
    if(i + stride < n4) {
      k_n = __ldg(&k4[i + stride]);
      g_n = __ldg(&g4[i + stride]);
    }
    mark(bm, k.x, g.x, n_keys, n_graphs, words);
    mark(bm, k.y, g.y, n_keys, n_graphs, words);
    mark(bm, k.z, g.z, n_keys, n_graphs, words);
    mark(bm, k.w, g.w, n_keys, n_graphs, words);
  }
  for(long long i = 4 * n4 + i0; i < n; i += stride) mark(bm, __ldg(&keys[i]), __ldg(&gids[i]), n_keys, n_graphs, words);
}

// kSupWarps warps per key (1, or the block).
template <int kSupWarps> __global__ void k_count(const uint32_t *bm, int n_keys, int words, int32_t *support)
{
  after_previous();
  constexpr int kPer = kSupWarps * 32;
  const int t = threadIdx.x % kPer;
  __shared__ int sums[kBlock / 32];
  for(int key = (blockIdx.x * kBlock + threadIdx.x) / kPer; key < n_keys; key += gridDim.x * (kBlock / kPer)) {
    int c = 0;
    for(int w = t; w < words; w += kPer) c += __popc(bm[(long long)key * words + w]);
    for(int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if(kSupWarps > 1) {
      if((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = c;
      __syncthreads();
      for(int q = 1; q < kSupWarps; q++) c += t == 0 ? sums[q] : 0;
      __syncthreads();
    }
    if(t == 0) support[key] = c;
  }
}

// Per device: the scratch's device address and the SM count, looked up once.
struct DevInfo {
  uint32_t *addr = nullptr;
  int sms = 0;
};
DevInfo g_dev[kMaxDevices];

// Launch that may begin while the kernel ahead of it in the stream ends (its
// griddepcontrol.wait holds it until that one's writes are there).
template <class... P, class... A> cudaError_t launch_early(void (*f)(P...), int grid, cudaStream_t s, A... args)
{
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3(kBlock);
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, f, P(args)...);
}

int grid_for(long long n, int sms)
{
  long long b = (n + kBlock - 1) / kBlock;
  if(b < 1) b = 1;
  const long long cap = 8LL * sms;  // 8 blocks of 256 threads per SM, grid-stride beyond
  return (int)(b < cap ? b : cap);
}

// Restores the calling thread's current device on every return path.
struct CurrentDevice {
  int prev = -1;
  bool changed = false;
  bool set(int dev)
  {
    if(cudaGetDevice(&prev) != cudaSuccess) {
      cudaGetLastError();
      prev = -1;
    }
    if(prev == dev) return true;
    if(cudaSetDevice(dev) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    changed = prev >= 0;
    return true;
  }
  ~CurrentDevice()
  {
    if(changed) cudaSetDevice(prev);
  }
};

// The device that owns `p` (device or managed memory), or -1.
int device_of(const void *p)
{
  cudaPointerAttributes a;
  if(cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  if(a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged) return -1;
  return a.device;
}

// Scratch address and SM count of device `dev`, which must be current.  The
// first call per device resolves the address with cudaGetSymbolAddress
// (which may load the module) and caches it for the life of the process.
gs_status device_info(int dev, DevInfo *out)
{
  if(dev < 0 || dev >= kMaxDevices) {
    t_msg = "gs_support_count_noalloc: device index out of range";
    return GS_ERR_LIMIT;
  }
  std::lock_guard<std::mutex> g(g_mu);
  DevInfo &d = g_dev[dev];
  if(!d.addr) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_bitmap);
    int sms = 0;
    if(e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if(e != cudaSuccess || !p || sms <= 0) {
      cudaGetLastError();
      t_msg = "gs_support_count_noalloc: cudaGetSymbolAddress of the scratch failed";
      return GS_ERR_CUDA;
    }
    d.sms = sms;
    d.addr = (uint32_t *)p;
  }
  *out = d;
  return GS_OK;
}

}  // namespace

extern "C" gs_status gs_support_count_noalloc(const int32_t *d_keys, const int32_t *d_graph_ids, int64_t n_records,
                                              int32_t n_keys, int32_t n_graphs, int32_t *d_support, void *stream)
{
  t_msg = "";
  if(n_records < 0 || n_keys < 0 || n_graphs < 0 || (n_records > 0 && (!d_keys || !d_graph_ids)) ||
     (n_keys > 0 && !d_support)) {
    t_msg = "gs_support_count_noalloc: invalid arguments";
    return GS_ERR_USAGE;
  }
  if(n_keys == 0) return GS_OK;
  const long long words = n_graphs > 0 ? ((long long)n_graphs + 31) / 32 : 1;
  if((long long)n_keys * words > (long long)kScratchWords) {
    t_msg = "gs_support_count_noalloc: n_keys * ceil(n_graphs/32) exceeds the 1048576-word (4 MiB) scratch";
    return GS_ERR_LIMIT;
  }
  // The work runs on the device that holds d_support; the stream must belong to it.
  const int dev = device_of(d_support);
  if(dev < 0) {
    t_msg = "gs_support_count_noalloc: d_support is not device memory";
    return GS_ERR_USAGE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  CurrentDevice cur;
  if(!cur.set(dev)) {
    t_msg = "gs_support_count_noalloc: cannot make the device of d_support current";
    return GS_ERR_CUDA;
  }
  if(s) {
    int sdev = -1;
    if(cudaStreamGetDevice(s, &sdev) != cudaSuccess) {
      cudaGetLastError();
      t_msg = "gs_support_count_noalloc: invalid stream";
      return GS_ERR_USAGE;
    }
    if(sdev != dev) {
      t_msg = "gs_support_count_noalloc: the stream belongs to another device than d_support";
      return GS_ERR_USAGE;
    }
  }
  // An error left pending by the caller's earlier work is reported as such
  // and left in place (peek, not get), so a launch error below is this call's.
  const cudaError_t pending = cudaPeekAtLastError();
  if(pending != cudaSuccess) {
    t_msg = "gs_support_count_noalloc: an earlier CUDA error is pending; nothing was launched";
    return GS_ERR_CUDA;
  }
  DevInfo di;
  gs_status st = device_info(dev, &di);
  if(st != GS_OK) return st;
  uint32_t *bm = di.addr;
  const long long nw = (long long)n_keys * words;
  k_clear<<<grid_for((nw + 3) / 4, di.sms), kBlock, 0, s>>>(bm, nw);
  if(cudaGetLastError() != cudaSuccess) {
    t_msg = "gs_support_count_noalloc: launch of the scratch clear failed";
    return GS_ERR_CUDA;
  }
  if(n_records > 0) {
    const int vec = ((uintptr_t)d_keys | (uintptr_t)d_graph_ids) % 16 == 0 ? 1 : 0;
    launch_early(k_mark, grid_for(vec ? (n_records + 3) / 4 : n_records, di.sms), s, bm, d_keys, d_graph_ids, n_records,
                 n_keys, n_graphs, (int)words, vec);
    if(cudaGetLastError() != cudaSuccess) {
      t_msg = "gs_support_count_noalloc: launch of the record marking failed";
      return GS_ERR_CUDA;
    }
  }
  // a block per key where a warp would take more than 8 rounds
  if(words > kBlock)
    launch_early(k_count<kBlock / 32>, grid_for((long long)n_keys * kBlock, di.sms), s, (const uint32_t *)bm, n_keys,
                 (int)words, d_support);
  else
    launch_early(k_count<1>, grid_for((long long)n_keys * 32, di.sms), s, (const uint32_t *)bm, n_keys, (int)words,
                 d_support);
  if(cudaGetLastError() != cudaSuccess) {
    t_msg = "gs_support_count_noalloc: launch of the popcount failed";
    return GS_ERR_CUDA;
  }
  return GS_OK;
}
