// Device memory helpers and a deterministic exclusive scan.
#pragma once
#include "common.cuh"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <vector>

namespace irsb {

// Owning device array with amortised growth (contents preserved on growth).
template <typename T>
struct DevVec {
  T* p = nullptr;
  size_t n = 0;    // logical size
  size_t cap = 0;  // allocated elements
  DevVec() = default;
  DevVec(const DevVec&) = delete;
  DevVec& operator=(const DevVec&) = delete;
  ~DevVec() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = cap = 0;
  }
  bool reserve(size_t want, cudaStream_t s) {
    if (want <= cap) return true;
    size_t nc = cap ? cap : 1;
    while (nc < want) nc *= 2;
    T* q = nullptr;
    if (!IRSB_CK(cudaMalloc(&q, nc * sizeof(T)))) return false;
    if (p && n) {
      if (!IRSB_CK(cudaMemcpyAsync(q, p, n * sizeof(T), cudaMemcpyDeviceToDevice, s))) {
        cudaFree(q);
        return false;
      }
      if (!IRSB_CK(cudaStreamSynchronize(s))) return false;
    }
    if (p) cudaFree(p);
    p = q;
    cap = nc;
    return true;
  }
  bool resize(size_t want, cudaStream_t s) {
    if (!reserve(want, s)) return false;
    n = want;
    return true;
  }
  // exact-size allocation without preserving contents
  bool alloc_exact(size_t want) {
    if (want <= cap) {
      n = want;
      return true;
    }
    release();
    if (want == 0) return true;
    if (!IRSB_CK(cudaMalloc(&p, want * sizeof(T)))) return false;
    cap = want;
    n = want;
    return true;
  }
  size_t bytes() const { return n * sizeof(T); }
};

// Bytes of page-locked host memory that the library's objects hold (its value
// "pinned_bytes"). Getting such memory takes 0.5 - 1 ms for a few bytes and
// milliseconds for a large map, in the first run of a new object.
inline std::atomic<long long>& pinned_bytes() {
  static std::atomic<long long> bytes{0};
  return bytes;
}

// Pinned host buffer.
template <typename T>
struct HostVec {
  T* p = nullptr;
  size_t n = 0;
  HostVec() = default;
  HostVec(const HostVec&) = delete;
  HostVec& operator=(const HostVec&) = delete;
  ~HostVec() { release(); }
  void release() {
    if (p) {
      cudaFreeHost(p);
      pinned_bytes() -= (long long)(n * sizeof(T));
    }
    p = nullptr;
    n = 0;
  }
  bool alloc(size_t want) {
    if (want == n && p) return true;
    release();
    if (want == 0) return true;
    if (!IRSB_CK(cudaMallocHost(&p, want * sizeof(T)))) return false;
    n = want;
    pinned_bytes() += (long long)(n * sizeof(T));
    return true;
  }
};

// Host memory that transfers fill, on pages of its own so that it can be pinned
// in place. Pinned memory makes a transfer faster but takes long to get
// (pinned_bytes), so this one starts pageable and is pinned when it has been used
// pin_after times: the owner sets that to about what getting it costs over what a
// use gains, so that an object that runs once never pays for it and one that runs
// often pays about twice at most.
template <typename T>
struct HostBuf {
  T* p = nullptr;
  HostBuf() = default;
  HostBuf(const HostBuf&) = delete;
  HostBuf& operator=(const HostBuf&) = delete;
  ~HostBuf() { release(); }
  void release() {
    if (pinned_) {
      cudaHostUnregister(p);
      pinned_bytes() -= (long long)bytes_;
    }
    std::free(p);
    p = nullptr;
    bytes_ = 0;
    uses_ = 0;
    pinned_ = false;
  }
  // Room for want values, to be filled once; contents kept only where it suffices.
  bool prepare(size_t want, long long pin_after) {
    constexpr size_t kPage = 4096;
    if (want * sizeof(T) > bytes_) {
      release();
      const size_t room = (want * sizeof(T) + kPage - 1) / kPage * kPage;
      p = static_cast<T*>(std::aligned_alloc(kPage, room));
      if (!p) {
        std::fprintf(stderr, "Error. No host memory for %zu bytes.\n", room);
        return false;
      }
      bytes_ = room;
    } else if (uses_ == pin_after) {
      pinned_ = cudaHostRegister(p, bytes_, cudaHostRegisterDefault) == cudaSuccess;
      if (pinned_) pinned_bytes() += (long long)bytes_;
      else cudaGetLastError();  // stays pageable
    }
    uses_++;
    return true;
  }

 private:
  size_t bytes_ = 0;
  long long uses_ = 0;
  bool pinned_ = false;
};

// ---------------------------------------------------------------- grid barrier
// Barrier of a cooperative grid, one 64-bit word per barrier (zeroed before
// the launch): every CTA adds 1 + 2^32 * value, value the sum of its threads'
// `value` given on the first lane of each warp (>= 0, below 2^31 in all), and
// leaves with the sum over the grid once all have arrived. Writes before the
// barrier are visible after it to plain loads (not to the read-only path). The
// wait is bounded: after `spins` reads of the word (about a microsecond each;
// a cooperative grid is resident as a whole, so it is never reached) or when
// another CTA gave up, *err is set and the sum returned is -1.
__device__ __forceinline__ int grid_barrier_sum(unsigned long long* word, int value, int* err, long long spins) {
  __shared__ int s_value, s_sum;
  if (threadIdx.x == 0) s_value = 0;
  __syncthreads();
  if ((threadIdx.x & 31) == 0 && value) atomicAdd(&s_value, value);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // this CTA's writes before its arrival
    atomicAdd(word, 1ull + ((unsigned long long)s_value << 32));
    int sum = -1;
    for (long long n = 0; n < spins; n++) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
      if ((v & 0xffffffffull) == gridDim.x) {
        sum = int(v >> 32);
        break;
      }
      if ((n & 1023) == 1023 && *(volatile int*)err) break;
    }
    if (sum < 0) atomicExch(err, 1);
    __threadfence();
    s_sum = sum;
  }
  __syncthreads();
  return s_sum;
}

// CTAs of a cooperative grid: `want`, at most what is resident at once.
template <typename K>
bool cooperative_grid(K kernel, int threads, long long want, int* grid, size_t smem = 0) {
  int dev = 0, sms = 0, per_sm = 0;
  IRSB_CKR(cudaGetDevice(&dev));
  IRSB_CKR(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  IRSB_CKR(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  const long long most = (long long)sms * per_sm;
  *grid = int(want < 1 ? 1 : (want > most ? most : want));
  return true;
}

// ---------------------------------------------------------------- scan
// Exclusive prefix sum of n values (int or long long input), written as long
// long. Three passes: per-block totals, a single-block scan of the totals, and
// a per-block local scan plus offset. Deterministic (integer arithmetic).
constexpr int kScanBlock = 512;
constexpr int kScanItems = 4;  // per thread
constexpr int kScanTile = kScanBlock * kScanItems;

template <typename In>
__global__ void scan_block_totals(const In* __restrict__ in, long long n, const int* __restrict__ dn,
                                  long long* __restrict__ totals) {
  __shared__ long long red[kScanBlock / 32];
  if (dn) n = *dn;
  long long base = (long long)blockIdx.x * kScanTile;
  long long s = 0;
  for (int k = 0; k < kScanItems; k++) {
    long long i = base + (long long)k * kScanBlock + threadIdx.x;
    if (i < n) s += (long long)in[i];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    long long v = threadIdx.x < kScanBlock / 32 ? red[threadIdx.x] : 0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) totals[blockIdx.x] = v;
  }
}

// Single block: in-place exclusive scan of `totals` (m entries), grand total to *sum.
__global__ void scan_totals_single(long long* __restrict__ totals, long long m, long long* __restrict__ sum) {
  __shared__ long long warp_sums[kScanBlock / 32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (long long start = 0; start < m; start += kScanBlock) {
    long long i = start + threadIdx.x;
    long long v = i < m ? totals[i] : 0;
    long long x = v;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
      long long ws = lane < kScanBlock / 32 ? warp_sums[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, ws, o);
        if (lane >= o) ws += y;
      }
      if (lane < kScanBlock / 32) warp_sums[lane] = ws;
    }
    __syncthreads();
    long long incl = x + (w > 0 ? warp_sums[w - 1] : 0) + carry;
    if (i < m) totals[i] = incl - v;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) carry = incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *sum = carry;
}

template <typename In>
__global__ void scan_block_apply(const In* __restrict__ in, long long n, const int* __restrict__ dn,
                                 const long long* __restrict__ offsets, long long* __restrict__ out) {
  __shared__ long long warp_sums[kScanBlock / 32];
  if (dn) n = *dn;
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = offsets[blockIdx.x];
  __syncthreads();
  long long base = (long long)blockIdx.x * kScanTile;
  for (int k = 0; k < kScanItems; k++) {
    long long i = base + (long long)k * kScanBlock + threadIdx.x;
    long long v = i < n ? (long long)in[i] : 0;
    long long x = v;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
      long long ws = lane < kScanBlock / 32 ? warp_sums[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, ws, o);
        if (lane >= o) ws += y;
      }
      if (lane < kScanBlock / 32) warp_sums[lane] = ws;
    }
    __syncthreads();
    long long incl = x + (w > 0 ? warp_sums[w - 1] : 0) + carry;
    if (i < n) out[i] = incl - v;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) carry = incl;
    __syncthreads();
  }
}

struct ScanScratch {
  DevVec<long long> totals;
  DevVec<long long> sum;
};

// out[i] = sum_{j<i} in[j] over the *dn (read on the device, at most n_cap)
// values of `in`; *sum (device; sc.sum when not given) receives the grand
// total. The scratch must already hold the blocks for n_cap (scan_reserve).
template <typename In>
bool exclusive_scan_dev(const In* in, const int* dn, long long n_cap, long long* out, ScanScratch& sc, cudaStream_t s,
                        long long* sum = nullptr) {
  long long nb = (n_cap + kScanTile - 1) / kScanTile;
  if (nb < 1) nb = 1;
  scan_block_totals<In><<<unsigned(nb), kScanBlock, 0, s>>>(in, n_cap, dn, sc.totals.p);
  scan_totals_single<<<1, kScanBlock, 0, s>>>(sc.totals.p, nb, sum ? sum : sc.sum.p);
  scan_block_apply<In><<<unsigned(nb), kScanBlock, 0, s>>>(in, n_cap, dn, sc.totals.p, out);
  return IRSB_CK(cudaGetLastError());
}

inline bool scan_reserve(ScanScratch& sc, long long n_cap, cudaStream_t s) {
  long long nb = (n_cap + kScanTile - 1) / kScanTile;
  return sc.totals.reserve(size_t(nb < 1 ? 1 : nb), s) && sc.sum.reserve(1, s);
}

}  // namespace irsb
