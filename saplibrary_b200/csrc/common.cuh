// Shared utilities of the sap_b200 library: error plumbing, device buffers,
// launch accounting and the asynchronous-copy PTX wrappers.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <unordered_map>
#include <utility>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/sap_b200.h"

namespace sapb {

// Library failure carrying a C-ABI status code.  Reference failures use the
// sap::system_error::Reason values (sap/exception.h:16-23).
#ifndef SAPB_ERROR_DEFINED
#define SAPB_ERROR_DEFINED
struct Error : public std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};
#endif

inline void cuda_check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    int code = (e == cudaErrorMemoryAllocation) ? SAP_ERR_OUT_OF_MEMORY : SAP_ERR_CUDA;
    throw Error(code, std::string(what) + ": " + cudaGetErrorString(e));
  }
}
#define SAPB_CUDA(x) ::sapb::cuda_check((x), #x)

// Message returned by sap_last_error() on the calling thread.
void set_last_error(const std::string& msg);

// Number of kernels enqueued by this library (reported by the bench).
extern std::atomic<int64_t> g_launches;
extern std::atomic<int64_t> g_lib_calls;
inline void count_launch(int k = 1) { g_launches.fetch_add(k, std::memory_order_relaxed); }
inline void count_lib_call() { g_lib_calls.fetch_add(1, std::memory_order_relaxed); }
#define SAPB_LAUNCHED() do { ::sapb::count_launch(); SAPB_CUDA(cudaGetLastError()); } while (0)

// Event bracketing of the launches of one selected kernel (sap_profile_*).
struct ProfScope {
  bool on = false;
  cudaStream_t s = nullptr;
  cudaEvent_t a = nullptr, b = nullptr;
  ProfScope(const char* name, cudaStream_t st);
  ~ProfScope();
};
#define SAPB_PROF(name, stream) ::sapb::ProfScope _sapb_prof_scope(name, stream)

// The streams that ever touch a group of device buffers (a solver's own ones).
// The buffers a thread allocates inside a HomeScope belong to its home, those
// allocated outside of one have none.
struct StreamHome {
  std::vector<cudaStream_t> streams;
  void add(cudaStream_t s) { streams.push_back(s); }
  void remove(cudaStream_t s) { streams.erase(std::remove(streams.begin(), streams.end(), s), streams.end()); }
  // all work on the streams is done; false when that cannot be told
  bool wait() const {
    bool ok = true;
    for (cudaStream_t s : streams) ok = cudaStreamSynchronize(s) == cudaSuccess && ok;
    if (!ok) (void)cudaGetLastError();  // nobody's next launch failed
    return ok;
  }
};
// A home without streams: for buffers that only calls touch which wait for their
// work before they return.
inline const std::shared_ptr<StreamHome>& idle_home() {
  static const auto* h = new std::shared_ptr<StreamHome>(std::make_shared<StreamHome>());
  return *h;
}
class HomeScope {
 public:
  explicit HomeScope(std::shared_ptr<StreamHome> h) : old_(std::move(h)) { std::swap(old_, current()); }
  ~HomeScope() { std::swap(old_, current()); }
  HomeScope(const HomeScope&) = delete;
  HomeScope& operator=(const HomeScope&) = delete;
  static std::shared_ptr<StreamHome>& current() {
    static thread_local std::shared_ptr<StreamHome> h;
    return h;
  }

 private:
  std::shared_ptr<StreamHome> old_;
};

// Device blocks kept for reuse (DBuf): cudaMalloc and cudaFree cost some 0.2 ms
// each whatever the size, and a setup, or a solver made for one batch of
// systems, makes dozens of them (24 systems in four stacks: 568 of each, 0.2 s
// of a 0.21 s call).  A block is taken by the next request on its device that
// fills at least half of it.  Only blocks with a home are kept: give() waits for
// the home's streams, so that a kept block has no work left on it, and never for
// the device, which would break a graph capture open in another thread.  The
// pool holds at most kMaxFreeBytes (1 % of the memory), larger blocks go
// straight back, an allocation that fails empties it and tries again, and
// sap_trim_memory() empties it on request.
class DevicePool {
 public:
  static DevicePool& instance() {
    static DevicePool* pool = new DevicePool();  // no driver call during static teardown
    return *pool;
  }
  // an allocation that is not kept
  void* take_plain(size_t bytes) {
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();  // not sticky
      trim();
      e = cudaMalloc(&p, bytes);
      if (e != cudaSuccess) (void)cudaGetLastError();
    }
    SAPB_CUDA(e);
    return p;
  }
  static void give_plain(void* p) {
    if (p && cudaFree(p) != cudaSuccess) (void)cudaGetLastError();
  }
  void* take(size_t bytes) {
    bytes = rounded(bytes);
    int dev = 0;
    SAPB_CUDA(cudaGetDevice(&dev));
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto it = free_.lower_bound({dev, bytes});
      if (it != free_.end() && it->first.first == dev && it->first.second / 2 <= bytes) {
        void* p = it->second.p;
        used_[p] = it->first;
        free_bytes_ -= it->first.second;
        free_.erase(it);
        return p;
      }
    }
    void* p = take_plain(bytes);
    std::lock_guard<std::mutex> lk(mu_);
    used_[p] = {dev, bytes};
    return p;
  }
  void give(void* p, const StreamHome& home) {
    if (!p) return;
    Key k;
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto it = used_.find(p);
      k = it->second;
      used_.erase(it);
    }
    bool kept = false;
    if (k.second <= kMaxFreeBytes / 2 && home.wait()) try {
        std::lock_guard<std::mutex> lk(mu_);
        free_.emplace(k, Block{p, given_++});
        free_bytes_ += k.second;
        kept = true;
      } catch (const std::bad_alloc&) {  // (give() runs in destructors)
      }
    if (kept) shrink(kMaxFreeBytes);
    else give_plain(p);
  }
  // every kept block back to the driver
  void trim() { shrink(0); }

 private:
  using Key = std::pair<int, size_t>;  // device, bytes
  static constexpr size_t kMaxFreeBytes = size_t(1) << 31;
  struct Block {
    void* p;
    unsigned long long age;  // position in the order of give()
  };
  // kept blocks beyond `bytes` back to the driver, the longest unused first (they
  // are left from other sizes; what a program uses again and again stays)
  void shrink(size_t bytes) {
    while (true) {
      void* p;
      {
        std::lock_guard<std::mutex> lk(mu_);
        if (free_bytes_ <= bytes || free_.empty()) return;
        auto old = std::min_element(free_.begin(), free_.end(),
                                    [](const auto& a, const auto& b) { return a.second.age < b.second.age; });
        p = old->second.p;
        free_bytes_ -= old->first.second;
        free_.erase(old);
      }
      give_plain(p);
    }
  }
  // small blocks in powers of two, others in steps of 1 MB
  static size_t rounded(size_t b) {
    if (b > (size_t(1) << 20)) return (b + (size_t(1) << 20) - 1) >> 20 << 20;
    size_t r = 512;
    while (r < b) r *= 2;
    return r;
  }
  std::mutex mu_;
  std::multimap<Key, Block> free_;
  unsigned long long given_ = 0;
  std::unordered_map<void*, Key> used_;
  size_t free_bytes_ = 0;
};

// Lets a kernel take `bytes` of dynamic shared memory on the current device.
// The limit belongs to the kernel, not to a solver: one kernel serves several
// widths and lengths, from any thread, so it is only ever raised.
inline void allow_smem_of(const void* kernel, size_t bytes) {
  if (bytes <= 40 * 1024) return;  // allowed by default, beside a kernel's static arrays
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> limit;
  int dev = 0;
  SAPB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  size_t& l = limit[{dev, kernel}];
  if (bytes <= l) return;
  SAPB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  l = bytes;
}
template <class... A>
inline void allow_smem(void (*kernel)(A...), size_t bytes) {
  allow_smem_of(reinterpret_cast<const void*>(kernel), bytes);
}

// Owning device buffer; its memory from the pool when it is allocated inside a
// HomeScope.
template <typename T>
class DBuf {
 public:
  DBuf() = default;
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept { swap(o); }
  DBuf& operator=(DBuf&& o) noexcept { release(); swap(o); return *this; }
  ~DBuf() { release(); }

  void alloc(size_t n) {
    if (n == n_ && p_) return;
    release();
    n_ = n;
    if (!n) return;
    DevicePool& pool = DevicePool::instance();
    home_ = HomeScope::current();
    p_ = static_cast<T*>(home_ ? pool.take(n * sizeof(T)) : pool.take_plain(n * sizeof(T)));
  }
  // grow-only: at least n elements (a smaller request keeps the buffer)
  void ensure(size_t n) {
    if (n > n_ || !p_) alloc(n);
  }
  // ensure(n) and copy n host elements to the front
  void put(const T* h, size_t n, cudaStream_t s) {
    ensure(n);
    if (n) SAPB_CUDA(cudaMemcpyAsync(p_, h, n * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void put(const std::vector<T>& h, cudaStream_t s) { put(h.data(), h.size(), s); }
  void zero(cudaStream_t s) {
    if (n_) SAPB_CUDA(cudaMemsetAsync(p_, 0, n_ * sizeof(T), s));
  }
  void upload(const T* h, size_t n, cudaStream_t s) {
    alloc(n);
    if (n) SAPB_CUDA(cudaMemcpyAsync(p_, h, n * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void upload(const std::vector<T>& h, cudaStream_t s) { upload(h.data(), h.size(), s); }
  void download(std::vector<T>& h, cudaStream_t s) const {
    h.resize(n_);
    if (n_) SAPB_CUDA(cudaMemcpyAsync(h.data(), p_, n_ * sizeof(T), cudaMemcpyDeviceToHost, s));
  }
  void release() {
    if (home_) DevicePool::instance().give(p_, *home_);
    else DevicePool::give_plain(p_);
    home_.reset();
    p_ = nullptr;
    n_ = 0;
  }
  T* get() const { return p_; }
  size_t size() const { return n_; }

 private:
  void swap(DBuf& o) { std::swap(p_, o.p_); std::swap(n_, o.n_); std::swap(home_, o.home_); }
  T* p_ = nullptr;
  size_t n_ = 0;
  std::shared_ptr<StreamHome> home_;
};

// Allocator whose value construction leaves trivially constructible elements
// uninitialised: a HostVec resized to hold a copy is first touched by the
// (parallel) copy itself instead of being zero-filled by one thread.
template <typename T>
struct DefaultInitAllocator : std::allocator<T> {
  template <typename U>
  struct rebind {
    using other = DefaultInitAllocator<U>;
  };
  DefaultInitAllocator() = default;
  template <typename U>
  DefaultInitAllocator(const DefaultInitAllocator<U>&) noexcept {}
  template <typename U>
  void construct(U* p) noexcept {
    ::new (static_cast<void*>(p)) U;
  }
  template <typename U, typename... A>
  void construct(U* p, A&&... a) {
    ::new (static_cast<void*>(p)) U(std::forward<A>(a)...);
  }
};
template <typename T>
using HostVec = std::vector<T, DefaultInitAllocator<T>>;

// Page-locked host blocks kept for reuse (PinnedPoolAllocator): a block
// released by one host copy of a matrix is taken by the next copy that fits
// in it (at most twice its size), so repeated copies neither fault in fresh
// pages nor go through the driver's pageable staging when they are
// uploaded.  Free blocks beyond kMaxFreeBytes go back to the driver, largest
// first.  Where page-locked memory cannot be had, blocks come from malloc.
// The pool is never destroyed (no driver call during static teardown).
class PinnedPool {
 public:
  static PinnedPool& instance() {
    static PinnedPool* pool = new PinnedPool();
    return *pool;
  }
  void* take(size_t bytes) {
    if (bytes == 0) bytes = 1;
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto it = free_.lower_bound(bytes);
      if (it != free_.end() && it->first / 2 <= bytes) {
        void* p = it->second;
        used_[p] = it->first;
        free_bytes_ -= it->first;
        free_.erase(it);
        return p;
      }
    }
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocDefault) == cudaSuccess && p) {
      std::lock_guard<std::mutex> lk(mu_);
      used_[p] = bytes;
      return p;
    }
    (void)cudaGetLastError();  // a failed allocation is not sticky: clear it
    p = std::malloc(bytes);
    if (!p) throw std::bad_alloc();
    std::lock_guard<std::mutex> lk(mu_);
    plain_[p] = bytes;
    return p;
  }
  void give(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(mu_);
    auto pl = plain_.find(p);
    if (pl != plain_.end()) {
      plain_.erase(pl);
      std::free(p);
      return;
    }
    auto it = used_.find(p);
    if (it == used_.end()) return;
    free_.emplace(it->second, p);
    free_bytes_ += it->second;
    used_.erase(it);
    shrink(kMaxFreeBytes);
  }
  // every free block back to the driver
  void trim() {
    std::lock_guard<std::mutex> lk(mu_);
    shrink(0);
  }

 private:
  void shrink(size_t bytes) {
    while (free_bytes_ > bytes && !free_.empty()) {
      auto big = std::prev(free_.end());
      free_bytes_ -= big->first;
      if (cudaFreeHost(big->second) != cudaSuccess) (void)cudaGetLastError();
      free_.erase(big);
    }
  }
  static constexpr size_t kMaxFreeBytes = size_t(1) << 31;
  std::mutex mu_;
  std::multimap<size_t, void*> free_;
  std::unordered_map<void*, size_t> used_, plain_;
  size_t free_bytes_ = 0;
};

// Allocator over PinnedPool with the construction of DefaultInitAllocator
// (elements left uninitialised until the copy writes them).
template <typename T>
struct PinnedPoolAllocator {
  using value_type = T;
  PinnedPoolAllocator() = default;
  template <typename U>
  PinnedPoolAllocator(const PinnedPoolAllocator<U>&) noexcept {}
  T* allocate(size_t n) { return static_cast<T*>(PinnedPool::instance().take(n * sizeof(T))); }
  void deallocate(T* p, size_t) noexcept { PinnedPool::instance().give(p); }
  template <typename U>
  void construct(U* p) noexcept {
    ::new (static_cast<void*>(p)) U;
  }
  template <typename U, typename... A>
  void construct(U* p, A&&... a) {
    ::new (static_cast<void*>(p)) U(std::forward<A>(a)...);
  }
  template <typename U>
  bool operator==(const PinnedPoolAllocator<U>&) const noexcept { return true; }
  template <typename U>
  bool operator!=(const PinnedPoolAllocator<U>&) const noexcept { return false; }
};
template <typename T>
using PinnedHostVec = std::vector<T, PinnedPoolAllocator<T>>;

// Page-locked host buffer (grow-only) for device->host copies at full speed.
template <typename T>
class PinnedBuf {
 public:
  PinnedBuf() = default;
  PinnedBuf(const PinnedBuf&) = delete;
  PinnedBuf& operator=(const PinnedBuf&) = delete;
  ~PinnedBuf() {
    if (p_) cudaFreeHost(p_);
  }
  T* reserve(size_t n) {
    if (n > cap_ || !p_) {
      if (p_) cudaFreeHost(p_);
      p_ = nullptr;
      cap_ = 0;
      SAPB_CUDA(cudaMallocHost(reinterpret_cast<void**>(&p_), (n ? n : 1) * sizeof(T)));
      cap_ = n;
    }
    return p_;
  }
  T* get() const { return p_; }

 private:
  T* p_ = nullptr;
  size_t cap_ = 0;
};

// --- asynchronous global->shared copies (sm_80+ cp.async) ---------------------
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
// 16 bytes, both addresses 16-byte aligned, past L1
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
template <typename T>
__device__ __forceinline__ void cp_async_val(T* smem, const T* gmem) {
  if constexpr (sizeof(T) == 8) cp_async8(smem, gmem);
  else cp_async4(smem, gmem);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// a / b from y = 1 / b (itself correctly rounded) with one multiply and two
// FMAs: Markstein's quotient correction (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990; Muller et al., Handbook of Floating-Point Arithmetic,
// Markstein's theorem): q0 = RN(a y) is within one ulp of a / b, the
// remainder r = a - b q0 is exact through the FMA, and RN(q0 + r y) =
// RN(a / b) as long as nothing underflows or overflows; for a = 0, q0 = +-0
// is the quotient.  `ok` is false outside exponent ranges that guarantee
// this (non-finite, subnormal, very large or very small operands), where the
// caller must use the division; with ok true the result equals a / b.
// The ranges are tested on the magnitudes' leading bits (integers, beside the
// chain of multiply-adds).
template <typename T>
struct DivRange;
template <>
struct DivRange<double> {  // 2^-960, 2^-1000, 2^1000
  static constexpr unsigned lo_a = 63u << 20, lo = 23u << 20, hi = 2023u << 20;
  static __device__ __forceinline__ unsigned mag(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
};
template <>
struct DivRange<float> {  // 2^-96, 2^-120, 2^120
  static constexpr unsigned lo_a = 31u << 23, lo = 7u << 23, hi = 247u << 23;
  static __device__ __forceinline__ unsigned mag(float v) { return (unsigned)__float_as_int(v) & 0x7fffffffu; }
};
template <typename T>
__device__ __forceinline__ T div_rcp_fast(T a, T b, T y, bool& ok) {
  using L = DivRange<T>;
  const T q0 = a * y;
  const T r = fma(-q0, b, a);
  const T q = fma(r, y, q0);
  constexpr unsigned span = L::hi - L::lo;
  ok = L::mag(y) - L::lo < span && (a == T(0) || (L::mag(a) >= L::lo_a && L::mag(q0) - L::lo < span));
  return a == T(0) ? q0 : q;
}

// 1 / b without a branch: Newton's iteration on the hardware's approximation,
// y <- y + y (1 - b y) with fused multiply-adds.  Once y is within one unit in
// the last place, one more step gives the correctly rounded reciprocal unless
// b's significand is all ones (Markstein, IBM J. Res. Dev. 34(1), 1990).  `ok`
// is false for that significand and outside DivRange, where the caller must
// use the division; with ok true the result equals T(1) / b.
__device__ __forceinline__ float rcp_fast(float b, bool& ok) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
#pragma unroll
  for (int i = 0; i < 2; i++) y = fmaf(y, fmaf(-b, y, 1.f), y);
  ok = DivRange<float>::mag(b) - DivRange<float>::lo < DivRange<float>::hi - DivRange<float>::lo &&
       (__float_as_uint(b) & 0x7fffffu) != 0x7fffffu;
  return y;
}
__device__ __forceinline__ double rcp_fast(double b, bool& ok) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));  // about 20 bits
#pragma unroll
  for (int i = 0; i < 3; i++) y = fma(y, fma(-b, y, 1.0), y);
  ok = DivRange<double>::mag(b) - DivRange<double>::lo < DivRange<double>::hi - DivRange<double>::lo &&
       (__double_as_longlong(b) & 0xfffffffffffffll) != 0xfffffffffffffll;
  return y;
}

// boostValue (sap/device/factor_band_const.cuh:29-40): pivots with
// |p| <= BURST_VALUE are replaced by +-BURST_NEW_VALUE.
template <typename T>
__device__ __forceinline__ T boost_pivot(T v) {
  const T thr = (T)1e-7, nv = (T)1e-4;
  if (v > thr || v < -thr) return v;
  return v < (T)0 ? -nv : nv;
}

}  // namespace sapb
