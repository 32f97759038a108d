// Device ordering of scan results.
//
// The public calls return matches sorted by (start, pattern_id, end)
// (GpuMatcher::scan, core/src/gpu/mod.rs:380-386) and tagged matches by
// (source_id, start, pattern_id, end) (core/src/batch.rs:157-163).  The order
// is made on the device by a least-significant-key-first sequence of stable
// radix sorts over an index permutation (CUB's DeviceRadixSort, with its
// temporary storage taken from the scratch so that no call allocates):
//   pass 1  end
//   pass 2  start << 32 | pattern_id
//   pass 3  source_id                  (tagged matches only)
// Stability makes the result the lexicographic order of the full key, ties
// included.  Records are gathered once, through the final permutation.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include "ws_launch.h"
#include "ws_matcher.h"

namespace ws {
namespace {

template <class R>
__global__ void k_keys_end(const R* rec, uint32_t n, uint64_t* key, uint32_t* idx) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    key[i] = rec[i].end;
    idx[i] = i;
  }
}

template <class R>
__global__ void k_keys_start_pid(const R* rec, const uint32_t* idx, uint32_t n, uint64_t* key) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const R& r = rec[idx[i]];
    key[i] = ((uint64_t)r.start << 32) | r.pattern_id;
  }
}

__global__ void k_keys_source(const ws_tagged_match* rec, const uint32_t* idx, uint32_t n, uint64_t* key) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    key[i] = rec[idx[i]].source_id;
}

template <class R>
__global__ void k_gather(const R* rec, const uint32_t* idx, uint32_t n, R* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = rec[idx[i]];
}

__global__ void k_narrow(const ws_match64* in, uint32_t n, ws_match* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const ws_match64 w = in[i];
    out[i] = ws_match{w.pattern_id, (uint32_t)w.start, (uint32_t)w.end};
  }
}

// Key and index double buffers plus CUB's temporary storage, in the scratch.
struct Bufs {
  uint64_t* key[2];
  uint32_t* idx[2];
  void* temp;
  size_t temp_bytes;
  int cur = 0;  // which of the double buffers holds the current keys / indices
};

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

Bufs bufs(Scratch& s, uint32_t n) {
  Bufs b{};
  cub::DoubleBuffer<uint64_t> k(nullptr, nullptr);
  cub::DoubleBuffer<uint32_t> v(nullptr, nullptr);
  check_cuda(cub::DeviceRadixSort::SortPairs(nullptr, b.temp_bytes, k, v, (int)n, 0, 64), "radix sort size");
  const size_t kb = align256((size_t)n * 8), vb = align256((size_t)n * 4);
  ensure(s.sortbuf, 2 * kb + 2 * vb + align256(b.temp_bytes));
  uint8_t* p = s.sortbuf.as<uint8_t>();
  b.key[0] = reinterpret_cast<uint64_t*>(p);
  b.key[1] = reinterpret_cast<uint64_t*>(p + kb);
  b.idx[0] = reinterpret_cast<uint32_t*>(p + 2 * kb);
  b.idx[1] = reinterpret_cast<uint32_t*>(p + 2 * kb + vb);
  b.temp = p + 2 * kb + 2 * vb;
  return b;
}

// One stable pass over key bits [0, bits): the indices follow their keys.
void pass(Bufs& b, uint32_t n, int bits, cudaStream_t st) {
  cub::DoubleBuffer<uint64_t> k(b.key[b.cur], b.key[b.cur ^ 1]);
  cub::DoubleBuffer<uint32_t> v(b.idx[b.cur], b.idx[b.cur ^ 1]);
  check_cuda(cub::DeviceRadixSort::SortPairs(b.temp, b.temp_bytes, k, v, (int)n, 0, bits, st), "radix sort");
  if (k.selector) b.cur ^= 1;
}

unsigned grid(uint32_t n) { return (unsigned)std::min<uint32_t>((n + 255) / 256, 148u * 8); }

template <class R>
void sort_records(Scratch& s, const R* d_in, R* d_out, uint64_t n, cudaStream_t st, bool tagged) {
  if (n > kMaxDeviceSorted)
    raise(WS_ERR_OVERFLOW, "too many matches to order on the device", 0, n, kMaxDeviceSorted);
  if (n == 0) return;
  const uint32_t m = (uint32_t)n;
  Bufs b = bufs(s, m);
  k_keys_end<R><<<grid(m), 256, 0, st>>>(d_in, m, b.key[0], b.idx[0]);
  check_cuda(cudaGetLastError(), "k_keys_end");
  pass(b, m, 32, st);
  k_keys_start_pid<R><<<grid(m), 256, 0, st>>>(d_in, b.idx[b.cur], m, b.key[b.cur]);
  check_cuda(cudaGetLastError(), "k_keys_start_pid");
  pass(b, m, 64, st);
  if (tagged) {
    k_keys_source<<<grid(m), 256, 0, st>>>(reinterpret_cast<const ws_tagged_match*>(d_in), b.idx[b.cur], m,
                                           b.key[b.cur]);
    check_cuda(cudaGetLastError(), "k_keys_source");
    pass(b, m, 64, st);
  }
  k_gather<R><<<grid(m), 256, 0, st>>>(d_in, b.idx[b.cur], m, d_out);
  check_cuda(cudaGetLastError(), "k_gather");
}

// Orders up to kSmallResults matches (kSmallTagged tagged ones) of a finished
// scan in the shared memory of one block and writes them, after the true count,
// into host-mapped memory: small results cost the host one wait, and no copies.
// For more than that or `cap` (or a failed scan's count) only the count is
// written.  The five
// launches and two copies this replaces took 45 us of a 4 KiB scan.
struct SmallKey {
  uint64_t source, start_pid;
  uint32_t end;
};
__device__ __forceinline__ SmallKey small_key(const ws_match& r) {
  return {0, ((uint64_t)r.start << 32) | r.pattern_id, r.end};
}
__device__ __forceinline__ SmallKey small_key(const ws_tagged_match& r) {
  return {r.source_id, ((uint64_t)r.start << 32) | r.pattern_id, r.end};
}
__device__ __forceinline__ void from_key(const SmallKey& k, ws_match& r) {
  r = ws_match{(uint32_t)k.start_pid, (uint32_t)(k.start_pid >> 32), k.end};
}
__device__ __forceinline__ void from_key(const SmallKey& k, ws_tagged_match& r) {
  r = ws_tagged_match{k.source, (uint32_t)k.start_pid, (uint32_t)(k.start_pid >> 32), k.end, 0};
}

template <class R, uint32_t kMost>
__global__ void __launch_bounds__(1024) small_results_kernel(const R* rec, const unsigned long long* count, uint64_t cap,
                                                             unsigned long long* host_count, R* host_rows) {
  pdl_begin();
  constexpr bool kTagged = sizeof(R) == sizeof(ws_tagged_match);
  __shared__ uint64_t src[kTagged ? kMost : 1], key[kMost];
  __shared__ uint32_t end[kMost];
  const unsigned long long n64 = *count;
  if (threadIdx.x == 0) *host_count = n64;
  if (n64 > kMost || n64 > cap) return;
  const uint32_t n = (uint32_t)n64;
  uint32_t m = 1;
  while (m < n) m <<= 1;
  for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
    SmallKey k{~0ull, ~0ull, ~0u};
    if (i < n) k = small_key(rec[i]);
    if (kTagged) src[i] = k.source;
    key[i] = k.start_pid;
    end[i] = k.end;
  }
  __syncthreads();
  for (uint32_t size = 2; size <= m; size <<= 1)
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
        const uint32_t j = i ^ stride;
        if (j <= i) continue;
        const SmallKey x{kTagged ? src[i] : 0, key[i], end[i]}, y{kTagged ? src[j] : 0, key[j], end[j]};
        const bool more = x.source != y.source         ? x.source > y.source
                          : x.start_pid != y.start_pid ? x.start_pid > y.start_pid
                                                       : x.end > y.end;
        if (more == ((i & size) == 0)) {
          if (kTagged) { src[i] = y.source; src[j] = x.source; }
          key[i] = y.start_pid;
          key[j] = x.start_pid;
          end[i] = y.end;
          end[j] = x.end;
        }
      }
      __syncthreads();
    }
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
    from_key(SmallKey{kTagged ? src[i] : 0, key[i], end[i]}, host_rows[i]);
}

// The scratch's host-mapped result: the count, then rows from byte 64 on.
uint8_t* result_buffer(Scratch& s) {
  if (!s.result)
    check_cuda(cudaHostAlloc(reinterpret_cast<void**>(&s.result),
                             64 + std::max(kSmallResults * sizeof(ws_match), kSmallTagged * sizeof(ws_tagged_match)),
                             cudaHostAllocMapped), "cudaHostAlloc(result)");
  void* d = nullptr;
  check_cuda(cudaHostGetDevicePointer(&d, s.result, 0), "cudaHostGetDevicePointer");
  return static_cast<uint8_t*>(d);
}

}  // namespace

void enqueue_results(Scratch& s, const ws_match* d_res, const unsigned long long* d_count, uint64_t cap,
                     cudaStream_t st) {
  uint8_t* d = result_buffer(s);
  launch_pdl(small_results_kernel<ws_match, kSmallResults>, 1, 1024, 0, st, 
      d_res, d_count, cap, reinterpret_cast<unsigned long long*>(d), reinterpret_cast<ws_match*>(d + 64));
  check_cuda(cudaGetLastError(), "small_results_kernel");
}

void enqueue_results(Scratch& s, const ws_tagged_match* d_res, const unsigned long long* d_count, uint64_t cap,
                     cudaStream_t st) {
  uint8_t* d = result_buffer(s);
  launch_pdl(small_results_kernel<ws_tagged_match, kSmallTagged>, 1, 1024, 0, st, 
      d_res, d_count, cap, reinterpret_cast<unsigned long long*>(d), reinterpret_cast<ws_tagged_match*>(d + 64));
  check_cuda(cudaGetLastError(), "small_results_kernel");
}

void sort_matches_device(Scratch& s, const ws_match* d_in, ws_match* d_out, uint64_t n, cudaStream_t st) {
  sort_records(s, d_in, d_out, n, st, false);
}

void sort_tagged_device(Scratch& s, const ws_tagged_match* d_in, ws_tagged_match* d_out, uint64_t n,
                        cudaStream_t st) {
  sort_records(s, d_in, d_out, n, st, true);
}

void narrow_matches_device(const ws_match64* d_in, ws_match* d_out, uint64_t n, cudaStream_t st) {
  if (n > kMaxDeviceSorted)
    raise(WS_ERR_OVERFLOW, "too many matches to order on the device", 0, n, kMaxDeviceSorted);
  if (n == 0) return;
  k_narrow<<<grid((uint32_t)n), 256, 0, st>>>(d_in, (uint32_t)n, d_out);
  check_cuda(cudaGetLastError(), "k_narrow");
}

}  // namespace ws
