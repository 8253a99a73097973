// Host engine: planning, device buffers, the band pipeline and the
// stream-ordered device entry.  Replaces the reference's CudaBlockPipeline /
// PcfBlockOp / CudaOffsetDataManager stack
// (include/sbear/cuda/cuda_block_executor.cuh:108-341, pcf_block_op.cuh:32-123,
// cuda_offset_data_manager.cuh:24-44) with a GB300-first design:
//   * the whole CSR is uploaded once (no per-tile re-uploads);
//   * the kernel writes the condensed (or dense) result directly, so a band
//     of rows [rb, re) is one contiguous output range that is copied with a
//     single cudaMemcpyAsync straight into the caller's matrix — there is no
//     dense tile, no memset, no host scatter;
//   * bands alternate between two device buffers so the copy of band b
//     overlaps the kernel of band b + 1.
#include "sbg_internal.hpp"
#include "host_copy.hpp"
#include "fixed_point.cuh"

#include <cuda.h>  // CUcontext / CUresult types; the two driver calls are looked up through the runtime

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>

namespace sbg
{
  // ---- errors & settings ----------------------------------------------------

  static thread_local std::string t_last_error;

  void set_last_error(const std::string& msg) { t_last_error = msg; }
  const char* last_error() { return t_last_error.c_str(); }

  void throw_cuda(cudaError_t e, const char* file, int line)
  {
    const char* base = file;
    for (const char* p = file; *p; ++p)
      if (*p == '/') base = p + 1;
    std::string msg = std::string(base) + ":" + std::to_string(line) + ": " + cudaGetErrorString(e);
    int st = (e == cudaErrorMemoryAllocation) ? ST_OUT_OF_MEMORY
           : (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? ST_NO_DEVICE : ST_CUDA;
    cudaGetLastError();  // clear a sticky-free error so later calls start clean
    throw Error(st, msg);
  }

  static std::atomic<uint64_t> g_kernel_launches{0};

  cudaError_t launched()
  {
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
  }

  void count_launches(uint64_t n) { g_kernel_launches.fetch_add(n, std::memory_order_relaxed); }
  void uncount_launches(uint64_t n) { g_kernel_launches.fetch_sub(n, std::memory_order_relaxed); }

  uint64_t kernel_launches() { return g_kernel_launches.load(std::memory_order_relaxed); }

  Settings& settings()
  {
    static Settings s;
    return s;
  }

  // ---- device allocations ----------------------------------------------------

  static std::atomic<uint64_t> g_alloc_limit{~0ull};
  static std::atomic<uint64_t> g_alloc_held{0};
  static std::atomic<uint64_t> g_alloc_count{0};

  static void reserve_bytes(size_t bytes)
  {
    const uint64_t held = g_alloc_held.fetch_add(bytes, std::memory_order_relaxed) + bytes;
    const uint64_t limit = g_alloc_limit.load(std::memory_order_relaxed);
    if (held > limit || held < bytes)
    {
      g_alloc_held.fetch_sub(bytes, std::memory_order_relaxed);
      throw Error(ST_OUT_OF_MEMORY, "device allocation of " + std::to_string(bytes) + " bytes refused: " +
                                        std::to_string(held - bytes) + " bytes held, limit " +
                                        std::to_string(limit) + " (sbg_set_alloc_limit)");
    }
  }

  unsigned long long current_context_id()
  {
    using CtxGetCurrentFn = CUresult (*)(CUcontext*);
    using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
      cudaDriverEntryPointQueryResult q;
      void* fn = nullptr;
      if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
        get_current = reinterpret_cast<CtxGetCurrentFn>(fn);
      fn = nullptr;
      if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
        get_id = reinterpret_cast<CtxGetIdFn>(fn);
      cudaGetLastError();
    });
    if (!get_current || !get_id) throw Error(ST_CUDA, "cuCtxGetCurrent / cuCtxGetId not available from the driver");
    CUcontext ctx = nullptr;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
    unsigned long long id = 0;
    if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
  }

  // Stream-ordered allocations come from one memory pool per device that
  // keeps up to POOL_KEEP bytes between calls; what is free above that goes
  // back to the device at the next synchronisation, and all of it when an
  // allocation of the library fails.  (The device's default pool keeps
  // nothing: after a synchronisation the next call's first allocation maps
  // memory again, 88 to 150 us against 2; a cudaFree is 55.)  The pool and
  // its ordering between streams and threads are CUDA's own.  It goes with the
  // context it was made in: after a device reset the next call makes another.
  static constexpr uint64_t POOL_KEEP = 256ull << 20;

  static cudaMemPool_t device_pool()
  {
    static std::mutex mu;
    static std::map<std::pair<int, unsigned long long>, cudaMemPool_t> pools;  // by device and context
    int dev = 0;
    SBG_CUDA(cudaGetDevice(&dev));
    unsigned long long ctx = current_context_id();
    if (ctx == 0)  // none yet in this thread
    {
      SBG_CUDA(cudaSetDevice(dev));  // makes the device's own current
      ctx = current_context_id();
    }
    std::lock_guard<std::mutex> lock(mu);
    cudaMemPool_t& kept = pools[{dev, ctx}];
    if (!kept)
    {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      cudaMemPool_t pool = nullptr;
      if (cudaMemPoolCreate(&pool, &props) != cudaSuccess)
      {
        cudaGetLastError();
        return nullptr;  // the default pool then serves
      }
      uint64_t keep = POOL_KEEP;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
      kept = pool;
    }
    return kept;
  }

  static cudaError_t pool_malloc(void** p, size_t bytes, cudaStream_t st)
  {
    const cudaMemPool_t pool = device_pool();
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st);
  }

  // After a failed allocation: what the pool keeps goes back.
  static void pool_give_back()
  {
    cudaGetLastError();
    if (const cudaMemPool_t pool = device_pool()) cudaMemPoolTrimTo(pool, 0);
  }

  void* device_malloc(size_t bytes)
  {
    reserve_bytes(bytes);
    void* p = nullptr;
    cudaError_t e = cudaSuccess;
    for (int attempt = 0; attempt < 2; ++attempt)
    {
      e = cudaMalloc(&p, bytes);
      if (e != cudaErrorMemoryAllocation) break;
      if (attempt == 0) pool_give_back();
    }
    if (e != cudaSuccess)
    {
      g_alloc_held.fetch_sub(bytes, std::memory_order_relaxed);
      throw_cuda(e, __FILE__, __LINE__);
    }
    g_alloc_count.fetch_add(1, std::memory_order_relaxed);
    return p;
  }

  void device_free(void* p, size_t bytes) noexcept
  {
    if (!p) return;
    cudaFree(p);
    g_alloc_held.fetch_sub(bytes, std::memory_order_relaxed);
  }

  void* device_malloc_async(size_t bytes, cudaStream_t st)
  {
    reserve_bytes(bytes);
    void* p = nullptr;
    cudaError_t e = pool_malloc(&p, bytes, st);
    if (e == cudaErrorMemoryAllocation)
    {
      pool_give_back();
      e = pool_malloc(&p, bytes, st);
    }
    if (e != cudaSuccess)
    {
      g_alloc_held.fetch_sub(bytes, std::memory_order_relaxed);
      throw_cuda(e, __FILE__, __LINE__);
    }
    g_alloc_count.fetch_add(1, std::memory_order_relaxed);
    return p;
  }

  void device_free_async(void* p, size_t bytes, cudaStream_t st) noexcept
  {
    if (!p) return;
    cudaFreeAsync(p, st);
    g_alloc_held.fetch_sub(bytes, std::memory_order_relaxed);
  }

  void set_alloc_limit(uint64_t bytes) { g_alloc_limit.store(bytes, std::memory_order_relaxed); }
  uint64_t device_allocations() { return g_alloc_count.load(std::memory_order_relaxed); }
  uint64_t device_bytes_held() { return g_alloc_held.load(std::memory_order_relaxed); }

  void DeviceBuffer::reset(size_t bytes)
  {
    release();
    if (bytes)
    {
      m_ptr = device_malloc(bytes);
      m_bytes = bytes;
    }
  }

  void DeviceBuffer::release()
  {
    if (m_ptr)
    {
      device_free(m_ptr, m_bytes);
      m_ptr = nullptr;
      m_bytes = 0;
    }
  }

  DeviceInfo device_info()
  {
    static std::mutex mu;
    static std::map<int, DeviceInfo> cache;
    int dev = 0;
    SBG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(dev);
    if (it != cache.end()) return it->second;
    DeviceInfo d;
    d.device = dev;
    SBG_CUDA(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
    int optin = 0;
    SBG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    d.smem_optin = (size_t)optin;
    int per_sm = 0, threads = 0;
    SBG_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    SBG_CUDA(cudaDeviceGetAttribute(&threads, cudaDevAttrMaxThreadsPerMultiProcessor, dev));
    d.smem_per_sm = (size_t)per_sm;
    d.threads_per_sm = threads;
    cache[dev] = d;
    return d;
  }

  int ctas_per_sm(const DeviceInfo& dev, int warps, size_t smem_bytes)
  {
    const int threads = std::max(1, warps) * 32;
    int n = std::max(1, dev.threads_per_sm / threads);
    n = std::min(n, std::max(1, 65536 / (threads * 64)));  // the register file at 64 per thread
    const size_t per = smem_bytes + 1024;
    if (smem_bytes > 0 && dev.smem_per_sm > 0) n = std::min<int>(n, std::max<size_t>(1, dev.smem_per_sm / per));
    return n;
  }

  // ---- input contract ------------------------------------------------------

  template <typename T>
  void validate_pcfs(const PcfSet<T>& s, const char* what)
  {
    if (s.n == 0) return;
    if (!s.off || !s.pts) throw Error(ST_INVALID_ARGUMENT, std::string(what) + ": null points/offsets");
    if (s.off[0] != 0) throw Error(ST_INVALID_INPUT, std::string(what) + ": offsets must start at 0");
    // PCFs [i0, i1): the first invalid one, or i1; its error in *msg.
    auto check = [&s, what](uint64_t i0, uint64_t i1, std::string* msg) -> uint64_t {
      for (uint64_t i = i0; i < i1; ++i)
      {
        const uint64_t a = s.off[i], b = s.off[i + 1];
        if (b <= a) { *msg = std::string(what) + ": PCF " + std::to_string(i) + " has no breakpoints"; return i; }
        if (b - a > 0xffffffffull) { *msg = std::string(what) + ": PCF " + std::to_string(i) + " is too long"; return i; }
        const T* p = s.pts + 2 * a;
        if (p[0] != T(0))
        {
          *msg = std::string(what) + ": PCF " + std::to_string(i) +
                 ": the first breakpoint must have time t=0 (got t=" + std::to_string((double)p[0]) + ").";
          return i;
        }
        for (uint64_t k = 0; k < b - a; ++k)
        {
          const T t = p[2 * k];
          if (!std::isfinite(t))
          {
            *msg = std::string(what) + ": PCF " + std::to_string(i) + ": breakpoint times must be finite";
            return i;
          }
          if (k > 0 && !(p[2 * (k - 1)] <= t))
          {
            *msg = std::string(what) + ": PCF " + std::to_string(i) + ": Breakpoints must be given in non-decreasing time order.";
            return i;
          }
        }
      }
      return i1;
    };
    // Large inputs are checked in parallel over contiguous ranges of PCFs;
    // the error reported is the first invalid PCF's, as in a serial scan.
    const unsigned parts = s.off[s.n] >= (1ull << 20) && s.n >= 1024 ? host_parts() : 1u;
    if (parts <= 1)
    {
      std::string msg;
      if (check(0, s.n, &msg) < s.n) throw Error(ST_INVALID_INPUT, msg);
      return;
    }
    std::vector<uint64_t> bad(parts, ~0ull);
    std::vector<std::string> msgs(parts);
    host_parallel([&](unsigned k) {
      const uint64_t i0 = s.n * k / parts, i1 = s.n * (k + 1) / parts;
      const uint64_t r = check(i0, i1, &msgs[k]);
      if (r < i1) bad[k] = r;
    });
    for (unsigned k = 0; k < parts; ++k)
      if (bad[k] != ~0ull) throw Error(ST_INVALID_INPUT, msgs[k]);
  }

  template void validate_pcfs<float>(const PcfSet<float>&, const char*);
  template void validate_pcfs<double>(const PcfSet<double>&, const char*);

  // ---- planning ---------------------------------------------------------------

  int op_kind(int op, double p)
  {
    if (op == 0) return OPK_L1;
    if (op == 1)
    {
      if (p == 1.0) return OPK_L1;
      if (p == 2.0) return OPK_L2DIST;
      return OPK_LP;
    }
    if (op == 2) return OPK_INNER;
    throw Error(ST_INVALID_ARGUMENT, "unknown op " + std::to_string(op));
  }

  // The kernel an automatic call launches; a forced variant keeps pow().
  static int launch_kind(int opk, double p) { return settings().variant.load() == 0 ? power_kind(opk, p) : opk; }

  uint64_t output_count(int mode, uint64_t nr, uint64_t nc)
  {
    if (mode == MODE_PDIST) return nr == 0 ? 0 : nr * (nr - 1) / 2;
    if (mode == MODE_KERNEL) return nr * (nr + 1) / 2;
    return nr * nc;
  }

  uint64_t row_output_start(int mode, uint64_t r, uint64_t nc)
  {
    if (mode == MODE_PDIST) return r == 0 ? 0 : r * (r - 1) / 2;
    if (mode == MODE_KERNEL) return r * (r + 1) / 2;
    return r * nc;
  }

  static uint64_t items_for(int mode, uint64_t rb, uint64_t re, uint64_t nc, uint32_t q)
  {
    ProblemDesc<float> d{};
    d.mode = mode; d.nc = nc; d.row_begin = rb; d.row_end = re; d.q = q;
    return problem_item_count(d);
  }

  // ---- launch-shape cache (sbg_autotune_device) ---------------------------------

  static std::mutex g_tune_mu;
  static std::map<TuneKey, std::pair<int, int>> g_tune_cache;

  static int floor_log2(uint64_t x)
  {
    int r = -1;
    while (x) { x >>= 1; ++r; }
    return r;
  }

  TuneKey tune_key(int elem_bytes, int opk, int mode, uint64_t n, uint32_t lmax)
  {
    return TuneKey{elem_bytes, opk, mode, floor_log2(n), floor_log2(lmax)};
  }

  bool tune_cache_get(const TuneKey& k, int* warps, int* q)
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tune_cache.find(k);
    if (it == g_tune_cache.end()) return false;
    *warps = it->second.first;
    *q = it->second.second;
    return true;
  }

  void tune_cache_put(const TuneKey& k, int warps, int q)
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tune_cache[k] = {warps, q};
  }

  void tune_cache_clear()
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tune_cache.clear();
  }

  template <typename T>
  Plan make_plan(int mode, uint64_t nr, uint64_t nc, const LengthStats& rs, const LengthStats& cs, const DeviceInfo& dev,
                 int opk)
  {
    Plan pl;
    const int U = kernel_unroll(sizeof(T) == 8);
    const size_t es = sizeof(Elem<T>);
    const size_t reserve = 2048;  // static shared memory + slack
    const size_t usable = dev.smem_optin > reserve ? dev.smem_optin - reserve : 0;
    const uint32_t lmax_c = std::max<uint32_t>(cs.lmax, 1);
    const uint32_t lmax_r = std::max<uint32_t>(rs.lmax, 1);
    const int variant = settings().variant.load();
    // Row buffer: the row, then sentinel copies for the advances past its
    // end.  The default walk (variant 5) pulls the row address back every
    // block, so U copies do; the others need one per step of the longest
    // column.
#ifndef SBG_ROW_PAD_FULL
    const bool short_pad = variant == 0 || variant == 5;
#else
    const bool short_pad = false;
#endif
    const uint32_t row_cap_full = lmax_r + lmax_c + (uint32_t)U + 1;
    const uint32_t row_cap = short_pad ? lmax_r + (uint32_t)U + 1 : row_cap_full;
    auto smem_for = [&](int w) { return (size_t)32 * lmax_c * es + (size_t)w * row_cap * es; };

    const int want_w = settings().warps.load();
    // Shared-memory variants (rows and columns staged): the most warps that fit.
    auto most_warps = [&](uint32_t cap) {
      const int cands[] = {32, 24, 16, 12, 8, 4};
      for (int w : cands)
      {
        if (want_w > 0 && w > want_w) continue;
        if ((size_t)32 * lmax_c * es + (size_t)w * cap * es <= usable) return w;
      }
      return 0;
    };
    int warps = 0;
    if (variant == 0 || variant == 1 || variant == 3 || variant == 5) warps = most_warps(row_cap);
    if ((variant == 1 || variant == 3 || variant == 5) && warps == 0)
      throw Error(ST_INVALID_ARGUMENT, "shared-memory variant requested but the PCFs do not fit in shared memory");
    // The automatic choice between this kernel and the time-windowed one is
    // made on the layout with full row padding (at least 16 warps): with the
    // short padding, L ~ U{16..512} also fits 16 warps, but there (N = 4096)
    // the plain kernel measured 2.89 / 2.95 ms against 2.86 / 2.88 ms for the
    // windowed one (L2 kernel / L2 distance).
    const bool plain_auto = variant == 0 && most_warps(row_cap_full) >= 16;

    if (plain_auto || variant == 1 || variant == 3 || variant == 5)
    {
      pl.smem = true;
      pl.packed = false;
      pl.kvar = variant == 3 ? 1 : (variant == 1 ? 2 : 5);  // auto: row times and values apart
      pl.warps = warps;
      pl.lmax_c = lmax_c;
      pl.row_cap = row_cap;
      pl.smem_bytes = smem_for(warps);
    }
    else if (variant == 7 || variant == 8)
    {
      // the float32 measurement variants (pair_variants.cu); never automatic
      if (sizeof(T) != 4) throw Error(ST_INVALID_ARGUMENT, "variants 7 and 8 are float32 only");
      pl.smem = true;
      pl.packed = false;
      pl.kvar = variant;
      size_t fixed, per_warp;
      if (variant == 7)
      {
        pl.lmax_c = lmax_c;
        pl.row_cap = lmax_r + (uint32_t)U;                   // the row, then U sentinel elements
        fixed = (size_t)32 * lmax_c * es;                     // 32 columns, 8 bytes per element
        per_warp = (size_t)pl.row_cap * 16 * es;              // 16 copies of every row element
      }
      else
      {
        pl.lmax_c = (uint32_t)padded_words((int)lmax_c - 1) + 1;  // padded column stride (words)
        pl.row_cap = (uint32_t)padded_words((int)lmax_r - 1) + 1;
        fixed = (size_t)2 * 32 * pl.lmax_c * sizeof(T);
        per_warp = (size_t)2 * pl.row_cap * sizeof(T);
      }
      int w = 0;
      for (int cand : {32, 24, 20, 16, 12, 8, 4})
      {
        if (want_w > 0 && cand > want_w) continue;
        if (fixed + (size_t)cand * per_warp <= usable) { w = cand; break; }
      }
      if (w == 0) throw Error(ST_INVALID_ARGUMENT, "variant " + std::to_string(variant) +
                                                       ": the PCFs do not fit in shared memory");
      pl.warps = w;
      pl.smem_bytes = fixed + (size_t)w * per_warp;
    }
    else if (variant == 2)
    {
      pl.smem = false;
      pl.packed = true;
      pl.kvar = 0;
      pl.warps = want_w > 0 ? std::min(want_w, 32) : 16;
      pl.lmax_c = lmax_c;
      pl.row_cap = 0;
      pl.smem_bytes = 0;
    }
    else if (variant == 4 || (variant == 0 && sizeof(T) == 8))
    {
      // hybrid: columns staged when the group fits, rows through L1 (the
      // automatic choice for long double PCFs, where the FP64 pipe bounds
      // both and the time-windowed walk measured slower)
      pl.smem = true;
      pl.packed = true;
      pl.kvar = 3;
      pl.warps = want_w > 0 ? std::min(want_w, 32) : 32;
      const uint32_t cap = (uint32_t)std::min<size_t>(usable / (32 * es), 0xffffffffu);
      pl.lmax_c = std::min(lmax_c, cap);
      pl.row_cap = 0;
      pl.smem_bytes = (size_t)32 * pl.lmax_c * es;
    }
    else
    {
      // time-windowed shared memory (float PCFs too long for the plain
      // layout); the layout is sized below, once the rows per item are known
      pl.smem = true;
      pl.packed = false;
      pl.kvar = 6;
      // 32 warps, with windows of up to 440 elements beside their row
      // buffers: N = 1021, L ~ U{16..512} 207 us, N = 4096 2.45 ms, N = 3000,
      // L ~ U{8..1024} 2.61 ms; with 24 warps and row buffers padded for the
      // longest column slice, which leave 344 elements: 237 us, 2.61 ms, 2.85
      // ms; 32 warps and such buffers (280 elements): 213 us, 2.61, 2.79 ms.
      pl.warps = want_w > 0 ? std::min(want_w, 32) : 32;
    }

    // Two CTAs of 16 warps per SM, where their shared memory fits, overlap one
    // CTA's column staging and row fills with the other's merges: small
    // problems, up to 256 rows per item, take them (below).
    const bool two_ctas = settings().warps.load() == 0 && settings().rowChunk.load() == 0 && pl.kvar == 5 &&
                          pl.warps > 16 && ctas_per_sm(dev, 16, smem_for(16)) >= 2;
    // Rows per item = 32 q: as large as possible (fewer column reloads) while
    // enough items per SM are left to end evenly.  At most 1024 rows, one
    // processing-order window, so that bands of whole windows start on item
    // boundaries.  Six items per SM are enough for two CTAs on each; with one,
    // small q gain more from their next doubling than uneven ends cost (plain,
    // L ~ U{10..200} held to one CTA: N = 1500 177 us at q = 2, 3.9 items per
    // SM, 230 at 1; N = 2500 397 at q = 4, 5.5 items, 466 at 2; windowed, L ~
    // U{16..512}: N = 1500 373 us at q = 2, 3.9 items, 460 at 1; N = 2400 906
    // at q = 4, 5.0 items, 940 at 2), and the long items of the windowed
    // variant want more of them at large q (N = 6000 4.64 ms at q = 8, 4.75 at
    // 16, 7.9 items; N = 7500 7.19 at 16, 7.64 at 32, 6.5 items; L ~
    // Poisson(512): N = 9000 20.6 at 16, 20.9 at 32, 9.2 items, N = 20,000
    // 99.6 at 16, 98.3 at 32, 43 items).  In tenths of an item:
    // The hybrid kernel reads rows through L1 and restages only its 32
    // columns per item, so big items buy it little but a ragged tail on
    // uneven lengths: at most 64 rows (f64 stable-rank N = 20,000, L2 kernel
    // / pdist: 1921 / 2458 ms against 2048 / 2533 ms with 1024 rows).
    const uint32_t q_top = pl.kvar == 3 ? 2u : 32u;
    auto tenths = [&](uint32_t cand) -> uint64_t {
      if (pl.kvar == 6) return cand == 2 ? 35 : cand == 4 ? 50 : cand == 16 ? 100 : cand == 32 ? 200 : 60;
      if (pl.kvar == 5 && !two_ctas) return cand == 2 ? 20 : cand == 4 ? 30 : cand == 8 ? 40 : 60;
      return 60;
    };
    uint32_t q = (uint32_t)std::max(0, settings().rowChunk.load());
    if (q == 0)
    {
      q = 1;
      for (uint32_t cand = q_top; cand >= 1; cand /= 2)
      {
        if (10 * items_for(mode, 0, nr, nc, cand) >= (uint64_t)dev.sms * tenths(cand)) { q = cand; break; }
      }
    }
    pl.q = q;
    // L ~ U{10..200}: N = 1000 88 us against 112 with one CTA of 32 warps, N =
    // 1500 162 against 218, N = 2500 376 against 450, N = 4000 892 against
    // 911; with more rows per item there is no difference to rely on (N =
    // 3000, 30,000 and 60,000 2-4 % faster, N = 10,000 2 % slower).
    if (two_ctas && q <= 8)
    {
      pl.warps = 16;
      pl.smem_bytes = smem_for(16);
    }
    if (pl.kvar == 6)
    {
      bool fit = false;
      const bool cap_ok = window_cap_allowed(es, pl.warps, 32 * q, usable);
      for (int w = pl.warps; w >= 4 && !fit && cap_ok; w -= 4)
        fit = window_layout(pl, es, w, 32 * q, std::max(lmax_r, lmax_c), usable);
      if (!fit) throw Error(ST_INVALID_ARGUMENT, "time-windowed variant: the window setting does not fit in shared memory");
    }
    // A launch shape sbg_autotune_device measured for problems of this
    // shape bucket, unless the caller fixed warps or rows per item.  Only
    // the warps and rows per item change; the time-windowed kernel keeps the
    // window cap of the default plan, so no result changes by a bit.
    if (opk >= 0 && settings().warps.load() == 0 && settings().rowChunk.load() == 0)
    {
      int tw = 0, tq = 0;
      if (tune_cache_get(tune_key((int)sizeof(T), opk, mode, nr, std::max(lmax_r, lmax_c)), &tw, &tq) && tw > 0 &&
          tq > 0 && tq <= 32)
      {
        Plan trial = pl;
        bool ok = true;
        if (pl.kvar == 6)
          ok = window_layout(trial, es, tw, 32u * (uint32_t)tq, std::max(lmax_r, lmax_c), usable, pl.win_r);
        else if (pl.kvar == 5 || pl.kvar == 1 || pl.kvar == 2)
        {
          ok = smem_for(tw) <= usable;
          trial.warps = tw;
          trial.smem_bytes = smem_for(tw);
        }
        else
          trial.warps = tw;
        if (ok)
        {
          trial.q = (uint32_t)tq;
          pl = trial;
          q = pl.q;
        }
      }
    }
    const uint64_t items = items_for(mode, 0, nr, nc, q);
    const int per_sm = (pl.kvar == 0) ? 2 : ctas_per_sm(dev, pl.warps, pl.smem_bytes);
    pl.grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(items, (uint64_t)dev.sms * per_sm));
    return pl;
  }

  bool window_cap_allowed(size_t es, int warps, uint32_t rows_per_item, size_t usable)
  {
    const size_t X = (size_t)std::max(0, settings().windowCap.load());
    if (X == 0) return true;
    if (warps < 4) return false;
    const size_t slots = ((size_t)rows_per_item * 4 + 15) / 16 * 16;
    const size_t row = 2 * X + (size_t)kernel_unroll(es == 16) + 1;
    return 32 * X * es + (size_t)(4 + warps % 4) * row * es + slots <= usable;
  }

  bool window_layout(Plan& pl, size_t es, int warps, uint32_t rows_per_item, uint32_t lmax, size_t usable,
                     uint32_t cap)
  {
    const uint32_t U = (uint32_t)kernel_unroll(es == 16);
    const size_t slots = ((size_t)rows_per_item * 4 + 15) / 16 * 16;
    auto bytes = [&](uint32_t X) { return (size_t)32 * X * es + (size_t)warps * (X + U + 1) * es + slots; };
    const uint32_t top = std::max<uint32_t>(8, (lmax + 7) / 8 * 8);
    uint32_t X = cap ? cap : (uint32_t)std::max(0, settings().windowCap.load());
    if (X == 0)
    {
      // bytes(X) is linear in X: the largest multiple of 8 that fits
      const size_t fixed = bytes(0), per = bytes(1) - bytes(0);
      if (usable < fixed + 8 * per) return false;
      X = (uint32_t)std::min<size_t>((usable - fixed) / per / 8 * 8, top);
    }
    if (bytes(X) > usable) return false;
    pl.warps = warps;
    pl.lmax_c = X;
    pl.win_r = X;
    pl.row_cap = X + U + 1;
    pl.row_slots = rows_per_item;
    pl.smem_bytes = bytes(X);
    return true;
  }

  template Plan make_plan<float>(int, uint64_t, uint64_t, const LengthStats&, const LengthStats&, const DeviceInfo&,
                                  int);
  template Plan make_plan<double>(int, uint64_t, uint64_t, const LengthStats&, const LengthStats&, const DeviceInfo&,
                                   int);

  static LengthStats host_length_stats(const uint64_t* off, uint64_t n)
  {
    LengthStats s;
    if (n == 0) return s;
    uint64_t mx = 0, mn = ~0ull, sum = 0;
    for (uint64_t i = 0; i < n; ++i)
    {
      uint64_t l = off[i + 1] - off[i];
      mx = std::max(mx, l);
      mn = std::min(mn, l);
      sum += l;
    }
    s.lmax = (uint32_t)mx;
    s.lmin = (uint32_t)mn;
    s.mean = (double)sum / (double)n;
    return s;
  }


  // ---- device entry -------------------------------------------------------------

  namespace
  {
    template <typename T>
    struct AsyncBuf
    {
      void* p = nullptr;
      size_t n = 0;
      cudaStream_t s = nullptr;
      AsyncBuf(size_t bytes, cudaStream_t st) : n(bytes), s(st)
      {
        if (bytes) p = device_malloc_async(bytes, st);
      }
      ~AsyncBuf()
      {
        if (p) device_free_async(p, n, s);
      }
      AsyncBuf(const AsyncBuf&) = delete;
      AsyncBuf& operator=(const AsyncBuf&) = delete;
    };

    // Max length over a CSR held on the device (one small reduction + sync).
    __global__ void max_len_kernel(const uint64_t* off, uint64_t n, unsigned int* out)
    {
      uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
      unsigned int v = 0;
      for (; i < n; i += (uint64_t)gridDim.x * blockDim.x)
      {
        uint64_t l = off[i + 1] - off[i];
        v = max(v, (unsigned int)(l < 0xffffffffull ? l : 0xffffffffull));
      }
      v = __reduce_max_sync(0xffffffffu, v);
      if ((threadIdx.x & 31) == 0) atomicMax(out, v);
    }
  }

  template <typename T>
  static uint32_t device_max_len(const uint64_t* off, uint64_t n, cudaStream_t st, const DeviceInfo& dev)
  {
    AsyncBuf<T> buf(sizeof(unsigned int), st);
    SBG_CUDA(cudaMemsetAsync(buf.p, 0, sizeof(unsigned int), st));
    unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)dev.sms * 4);
    if (blocks == 0) blocks = 1;
    max_len_kernel<<<blocks, 256, 0, st>>>(off, n, (unsigned int*)buf.p);
    SBG_CUDA(launched());
    unsigned int h = 0;
    SBG_CUDA(cudaMemcpyAsync(&h, buf.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    SBG_CUDA(cudaStreamSynchronize(st));
    return h;
  }

  // One launch of the persistent kernel over rows [d.row_begin, d.row_end)
  // of one problem.  The queue counter is stream-ordered scratch.
  template <typename T>
  static void launch_problem(ProblemDesc<T> d, const Plan& pl, int opk, cudaStream_t st,
                             unsigned long long* given_queue = nullptr, const unsigned* gate = nullptr)
  {
    d.item_begin = 0;
    d.n_items = problem_item_count(d);
    if (d.n_items == 0) return;
    std::unique_ptr<AsyncBuf<T>> own;
    unsigned long long* queue = given_queue;
    if (!queue)
    {
      own.reset(new AsyncBuf<T>(sizeof(unsigned long long), st));
      queue = static_cast<unsigned long long*>(own->p);
    }
    if (!gate) SBG_CUDA(cudaMemsetAsync(queue, 0, sizeof(unsigned long long), st));  // else zeroed with the gate's own
    LaunchParams<T> L{};
    L.one = d;
    L.probs = nullptr;
    L.n_probs = 1;
    L.total_items = d.n_items;
    L.queue = queue;
    L.lmax_c = pl.lmax_c;
    L.row_cap = pl.row_cap;
    L.win_r = pl.win_r;
    L.row_slots = pl.row_slots;
    L.gate = gate;
    // Few items (fewer than twelve per SM): in length order a window's longest
    // rows come last, and the longest items have to start first (L ~
    // U{10..200}: N = 1000 88 us against 107, N = 1500 162 against 181, N =
    // 2000 253 against 277; windowed, L ~ U{16..512}: N = 1500 373 against
    // 431, N = 4096 2376 against 2450).  With many items, or large ones in the
    // plain variant (where they hide what is staged next, and the last chunk's
    // diagonal items are the small ones), the last items end the launch more
    // evenly (N = 3200, q = 4, two CTAs: 592 against 607; N = 4000, q = 8: 891
    // against 928; N = 5000, q = 1: 3.03 ms against 3.06).
    // Where the SMs would run dry, halves of 16 rows spread better than they
    // cost in columns staged twice: up to 2.5 items per SM with two CTAs on
    // each (N = 300: 38 us against 49, N = 800: 68 against 74; N = 1000, 3.5
    // per SM: 95 against 88; quarters are behind halves everywhere), up to
    // 0.75 with one, whose 32 warps have a row each already (L ~ U{16..512}:
    // N = 300 77 us against 105, N = 600, 1.25 per SM, 121 against 107).  No
    // pair's arithmetic depends on either.
    const uint64_t sms = (uint64_t)device_info().sms;
    const uint64_t resident = (uint64_t)ctas_per_sm(device_info(), pl.warps, pl.smem_bytes);
    L.last_first = d.n_items < 12 * sms && (pl.kvar == 6 || (pl.kvar == 5 && d.q <= (resident > 1 ? 2 : 4)));
    L.parts = L.last_first && d.q == 1 && 4 * d.n_items <= (resident > 1 ? 10 : 3) * sms ? 2 : 1;
    L.total_items = d.n_items * L.parts;
    uint64_t ctas = (uint64_t)pl.grid;  // what is resident, at most one per item
    if (L.parts > 1) ctas = std::max<uint64_t>(ctas, sms * resident);
    const int grid = (int)std::min<uint64_t>(ctas, L.total_items);
    SBG_CUDA(launch_pairs<T>(L, opk, pl.kvar, pl.warps, grid, pl.smem_bytes, st));
  }

  // ---- double precision in fixed point (fixed_point.cu) ---------------------------

  bool takes_fixed_point(int opk)
  {
    if (settings().variant.load() != 0 || settings().windowCap.load() != 0) return false;
    return opk == OPK_L1 || opk == OPK_L2DIST || opk == OPK_INNER;
  }

  namespace
  {
    // One call's fixed-point run: the record of its data, the packed arrays
    // and the launches, in one device buffer.  The direct kernel of the plan
    // is launched behind every fixed one, gated by the record.
    struct FixedRun
    {
      int opk = 0, sms = 0, warps = FIXED_WARPS;
      uint32_t q = 1, smem = 0, longest = 0;
      uint64_t rcap = 0, ccap = 0;
      bool cross = false;
      bool used[2] = {false, false};  // whose queue counters are no longer zero
      char* base = nullptr;
      size_t rpack = 0, rshape = 0, rlens = 0, cpack = 0, cshape = 0, clens = 0, carry = 0, carry_bytes = 0, total = 0;

      static constexpr size_t GATE = 128, QUEUES = 192;  // the record at 0
      static constexpr int SLOTS = 2;                    // launches in flight (one per stream)

      // Queue counters of the fixed and the gated direct launch.
      unsigned long long* queue(int slot) const { return reinterpret_cast<unsigned long long*>(base + QUEUES) + 2 * slot; }
      FixedRecord* record() const { return reinterpret_cast<FixedRecord*>(base); }
      unsigned* gate() const { return reinterpret_cast<unsigned*>(base + GATE); }
      void* rows() const { return base + rpack; }
      void* cols() const { return cross ? base + cpack : base + rpack; }
      uint32_t* row_lens() const { return reinterpret_cast<uint32_t*>(base + rlens); }
      uint32_t* col_lens() const { return reinterpret_cast<uint32_t*>(base + (cross ? clens : rlens)); }
      Shape* row_shapes() const { return reinterpret_cast<Shape*>(base + rshape); }
      Shape* col_shapes() const { return reinterpret_cast<Shape*>(base + (cross ? cshape : rshape)); }

      // Whether a call takes this path: every automatic one, whatever its
      // size (30 PCFs of L ~ U{16..200}, L1 on the device: 116 us a call
      // against 304 with the direct kernel, whose chain of FP64 latencies
      // alone is longer than all the launches here).
      static bool wanted(int opk) { return takes_fixed_point(opk); }
      void layout(int opk_, int mode, uint64_t nr, uint64_t nc, uint32_t lmax, uint64_t row_points, uint64_t col_points,
                  uint64_t row_begin, const DeviceInfo& dev, int slots)
      {
        opk = opk_;
        sms = dev.sms;
        longest = std::min(lmax, 0x3fffffffu);  // a pair's breakpoints and words are counted in 32 bits
        cross = mode == MODE_CROSS;
        rcap = std::max<uint64_t>(row_points, 1);
        ccap = cross ? std::max<uint64_t>(col_points, 1) : rcap;
        // The launch shape the caller fixed, or the one measured for problems
        // of this shape bucket; no sum depends on it.
        int w = settings().warps.load(), chunk = settings().rowChunk.load();
        if (w == 0 && chunk == 0) tune_cache_get(tune_key(8, opk, mode, nr, lmax), &w, &chunk);
        if (w > 0) warps = std::min(w, FIXED_WARPS);
        q = (uint32_t)std::min(chunk, 32);
        if (q == 0)
        {
          q = 1;
          for (uint32_t cand : {4u, 2u})
            if (row_begin % (32 * cand) == 0 && items_for(mode, 0, nr, nc, cand) >= (uint64_t)dev.sms * 6)
            {
              q = cand;
              break;
            }
        }
        smem = (uint32_t)(dev.smem_optin - 2048);
        auto up = [](size_t x) { return (x + 255) / 256 * 256; };
        rpack = 256;
        rshape = rpack + up(rcap * 16);
        rlens = rshape + up(nr * sizeof(Shape));
        cpack = rlens + up(nr * sizeof(uint32_t));
        cshape = cpack + up(ccap * 16);
        clens = cshape + up(nc * sizeof(Shape));
        carry = cross ? clens + up(nc * sizeof(uint32_t)) : cpack;
        // one window takes every PCF, in the larger of the two element sizes:
        // no sums pass from one to the next (a longer PCF than lmax does not
        // get there, by the record)
        const uint32_t slots_bytes = (32 * q * 4 + 15) / 16 * 16;
        const bool one = lmax <= fixed_slice_cap(smem - slots_bytes, (uint32_t)warps, 16);
        carry_bytes = one ? 0 : up((size_t)sms * 32 * q * FIXED_CARRY * 32 * 8);
        total = carry + slots * carry_bytes;
      }
      // The record and the packed arrays (elements for the direct kernel
      // where the record asks for it and that kernel reads them).
      // rperm / cperm: where the processing order by packed lengths goes, or
      // null.
      void prepare(char* at, const PcfSet<double>& r, const PcfSet<double>& c, bool elements, uint32_t* rperm,
                   uint32_t* cperm, cudaStream_t st)
      {
        base = at;
        SBG_CUDA(cudaMemsetAsync(base, 0, 256, st));
        SBG_CUDA(launch_fixed_record(r.pts, r.off, r.n, rcap, longest, record(), sms, st));
        if (cross) SBG_CUDA(launch_fixed_record(c.pts, c.off, c.n, ccap, longest, record(), sms, st));
        SBG_CUDA(launch_fixed_pack(r.pts, r.off, r.n, rcap, record(), opk, rows(), row_shapes(), row_lens(), elements, gate(), sms, st));
        if (cross) SBG_CUDA(launch_fixed_pack(c.pts, c.off, c.n, ccap, record(), opk, cols(), col_shapes(), col_lens(), elements, gate(), sms, st));
        if (rperm) length_order_device(r.off, r.n, rperm, nullptr, st, row_lens());
        if (cross && cperm) length_order_device(c.off, c.n, cperm, nullptr, st, col_lens());
      }
      // One launch over the rows and output of `d` (points: the callers' CSR),
      // and the direct kernel behind it.
      void launch(ProblemDesc<double> d, const double* rpts, const double* cpts, const Plan& pl, int slot,
                  cudaStream_t st)
      {
        FixedParams P{};
        P.rec = record();
        P.r = FixedSet{rpts, d.roff, d.rperm, d.nr, static_cast<const uint64_t*>(rows()), rcap, row_shapes(), row_lens()};
        P.c = FixedSet{cpts, d.coff, d.cperm, d.nc, static_cast<const uint64_t*>(cols()), ccap, col_shapes(), col_lens()};
        P.out = d.out; P.out_base = d.out_base; P.out_count = d.out_count; P.ld = d.ld;
        P.row_begin = d.row_begin; P.row_end = d.row_end;
        P.mode = d.mode;
        P.q = q;
        P.rows_per_item = 32 * q;
        P.smem_bytes = smem;
        P.gate = gate();
        P.elements = pl.packed;
        P.carry = reinterpret_cast<uint64_t*>(base + carry + (size_t)slot * carry_bytes);
        P.n_items = items_for(d.mode, d.row_begin, d.row_end, d.nc, q);
        if (P.n_items == 0) return;
        P.queue = queue(slot);
        if (used[slot]) SBG_CUDA(cudaMemsetAsync(P.queue, 0, 2 * sizeof(unsigned long long), st));
        used[slot] = true;
        SBG_CUDA(launch_fixed_pairs(P, opk, warps, (int)std::min<uint64_t>(P.n_items, (uint64_t)sms), st));
        if (pl.packed)
        {
          d.rpts = static_cast<const double*>(rows());
          d.cpts = static_cast<const double*>(cols());
          d.rcap = rcap;
          d.ccap = ccap;
        }
        launch_problem<double>(d, pl, opk, st, queue(slot) + 1, gate());
      }
    };
  }

  template <typename T>
  void compute_device(int mode, int op, double p, const PcfSet<T>& rows, const PcfSet<T>* cols,
                      const uint32_t* rperm, const uint32_t* cperm, uint32_t lmax, T* out, uint64_t out_base,
                      uint64_t row_begin, uint64_t row_end, cudaStream_t st)
  {
    const DeviceInfo dev = device_info();
    if (mode == MODE_CROSS && !cols) throw Error(ST_INVALID_ARGUMENT, "cdist needs a column set");
    const PcfSet<T>& cs = (mode == MODE_CROSS) ? *cols : rows;
    if (row_end > rows.n) row_end = rows.n;
    if (row_begin >= row_end || cs.n == 0) return;
    const int opk = op_kind(op, p);

    if (lmax == 0)
    {
      lmax = device_max_len<T>(rows.off, rows.n, st, dev);
      if (mode == MODE_CROSS) lmax = std::max(lmax, device_max_len<T>(cs.off, cs.n, st, dev));
    }
    LengthStats ls;
    ls.lmax = lmax;
    ls.lmin = 1;
    ls.mean = lmax;
    const Plan pl = make_plan<T>(mode, rows.n, cs.n, ls, ls, dev, opk);
    if (row_begin % (32ull * pl.q) != 0)
      throw Error(ST_INVALID_ARGUMENT, "row_begin must be a multiple of the row chunk (32*q)");

    // Processing order: by breakpoint count within windows of
    // LENGTH_ORDER_WINDOW PCFs, computed on the stream, unless the caller or
    // the order setting fixed one.  The band must be whole windows: the
    // order permutes PCFs only inside a window, so such a band holds the
    // same rows in either order and its results stay in the band's
    // contiguous output range.  The permutation is the one the host entry
    // uses, so both give the same bits.
    std::unique_ptr<AsyncBuf<T>> order_buf;
    size_t order_perm_bytes = 0;
    const bool windows = row_begin % LENGTH_ORDER_WINDOW == 0 &&
                         (row_end % LENGTH_ORDER_WINDOW == 0 || row_end == rows.n);
    const bool caller_perm = rperm || cperm;
    if (!caller_perm && windows && settings().order.load() != 1 && rows.n <= 0xffffffffull &&
        cs.n <= 0xffffffffull)
    {
      const uint64_t nr = rows.n, nc = (mode == MODE_CROSS) ? cs.n : 0;
      const size_t perm_bytes = order_perm_bytes = ((nr + nc) * sizeof(uint32_t) + 255) / 256 * 256;
      const size_t key_bytes = std::max(length_order_scratch_bytes(nr), length_order_scratch_bytes(nc));
      order_buf.reset(new AsyncBuf<T>(perm_bytes + key_bytes, st));
      uint32_t* rp = static_cast<uint32_t*>(order_buf->p);
      rperm = rp;
      if (mode == MODE_CROSS) cperm = rp + nr;
    }
    auto order_by_points = [&] {
      if (!order_buf) return;
      void* keys = static_cast<char*>(order_buf->p) + order_perm_bytes;
      length_order_device(rows.off, rows.n, const_cast<uint32_t*>(rperm), keys, st);
      if (mode == MODE_CROSS) length_order_device(cs.off, cs.n, const_cast<uint32_t*>(cperm), keys, st);
    };

    ProblemDesc<T> d{};
    d.rpts = rows.pts; d.roff = rows.off; d.rperm = rperm; d.nr = rows.n;
    d.cpts = cs.pts; d.coff = cs.off; d.cperm = (mode == MODE_CROSS) ? cperm : rperm; d.nc = cs.n;
    d.out = out; d.out_base = out_base; d.ld = cs.n;
    d.row_begin = row_begin; d.row_end = row_end;
    d.q = pl.q; d.mode = mode; d.p = (T)p;
    {
      // rows [row_begin, row_end) in caller order, or in the windowed length
      // order, own one contiguous range; with a caller's order the results
      // may land anywhere in the matrix
      const uint64_t hi = caller_perm ? output_count(mode, rows.n, cs.n) : row_output_start(mode, row_end, cs.n);
      d.out_count = hi > out_base ? hi - out_base : 0;
    }

    // Packed layouts need the point totals: read back with one
    // synchronisation for the global-memory and hybrid variants; the
    // fixed-point path of a call that needs none otherwise sizes its buffer
    // for PCFs of the longest length.
    uint64_t rtot = 0, ctot = 0;
    if (pl.packed)
    {
      SBG_CUDA(cudaMemcpyAsync(&rtot, rows.off + rows.n, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
      if (mode == MODE_CROSS)
        SBG_CUDA(cudaMemcpyAsync(&ctot, cs.off + cs.n, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
      SBG_CUDA(cudaStreamSynchronize(st));
    }
    if constexpr (sizeof(T) == 8)
    {
      if (FixedRun::wanted(opk))
      {
        FixedRun run;
        run.layout(opk, mode, rows.n, cs.n, lmax, pl.packed ? rtot : rows.n * lmax, pl.packed ? ctot : cs.n * lmax,
                   row_begin, dev, 1);
        std::unique_ptr<AsyncBuf<T>> buf;
        try { buf.reset(new AsyncBuf<T>(run.total, st)); }
        catch (const Error& e)
        {
          if (e.status != ST_OUT_OF_MEMORY) throw;  // the direct path needs less
        }
        if (buf)
        {
          run.prepare(static_cast<char*>(buf->p), rows, cs, pl.packed,
                      order_buf ? const_cast<uint32_t*>(rperm) : nullptr,
                      order_buf ? const_cast<uint32_t*>(cperm) : nullptr, st);
          run.launch(d, rows.pts, cs.pts, pl, 0, st);
          return;
        }
      }
    }
    order_by_points();
    std::unique_ptr<AsyncBuf<T>> rpack, cpack;
    if (pl.packed)
    {
      rpack.reset(new AsyncBuf<T>(sizeof(Elem<T>) * std::max<uint64_t>(rtot, 1), st));
      SBG_CUDA(launch_pack<T>(rows.pts, rows.off, rows.n, (Elem<T>*)rpack->p, rtot, dev.sms, st));
      d.rpts = reinterpret_cast<const T*>(rpack->p);
      d.cpts = d.rpts;
      d.rcap = rtot;
      d.ccap = rtot;
      if (mode == MODE_CROSS)
      {
        cpack.reset(new AsyncBuf<T>(sizeof(Elem<T>) * std::max<uint64_t>(ctot, 1), st));
        SBG_CUDA(launch_pack<T>(cs.pts, cs.off, cs.n, (Elem<T>*)cpack->p, ctot, dev.sms, st));
        d.cpts = reinterpret_cast<const T*>(cpack->p);
        d.ccap = ctot;
      }
    }
    launch_problem<T>(d, pl, launch_kind(opk, p), st);
  }

  template void compute_device<float>(int, int, double, const PcfSet<float>&, const PcfSet<float>*, const uint32_t*,
                                      const uint32_t*, uint32_t, float*, uint64_t, uint64_t, uint64_t, cudaStream_t);
  template void compute_device<double>(int, int, double, const PcfSet<double>&, const PcfSet<double>*,
                                       const uint32_t*, const uint32_t*, uint32_t, double*, uint64_t, uint64_t,
                                       uint64_t, cudaStream_t);

  template <typename T>
  size_t scratch_needed(int mode, uint64_t n_rows, uint64_t n_cols, uint32_t lmax, uint64_t row_points,
                        uint64_t col_points)
  {
    const DeviceInfo dev = device_info();
    LengthStats ls;
    ls.lmax = lmax; ls.lmin = 1; ls.mean = lmax;
    const Plan pl = make_plan<T>(mode, n_rows, mode == MODE_CROSS ? n_cols : n_rows, ls, ls, dev, -1);
    size_t need = 256;  // work-queue counter
    if (pl.packed)
    {
      need += ((sizeof(Elem<T>) * row_points + 255) / 256) * 256;
      if (mode == MODE_CROSS) need += ((sizeof(Elem<T>) * col_points + 255) / 256) * 256;
    }
    return need;
  }

  template <typename T>
  void compute_device_scratch(int mode, int op, double p, const PcfSet<T>& rows, const PcfSet<T>* cols,
                              const uint32_t* rperm, const uint32_t* cperm, uint32_t lmax, uint64_t row_points,
                              uint64_t col_points, T* out, uint64_t out_base, uint64_t row_begin, uint64_t row_end,
                              void* scratch, size_t scratch_bytes, cudaStream_t st)
  {
    const DeviceInfo dev = device_info();
    if (mode == MODE_CROSS && !cols) throw Error(ST_INVALID_ARGUMENT, "cdist needs a column set");
    if (lmax == 0) throw Error(ST_INVALID_ARGUMENT, "max_points must be given (measuring it would allocate)");
    const PcfSet<T>& cs = (mode == MODE_CROSS) ? *cols : rows;
    if (row_end == 0 || row_end > rows.n) row_end = rows.n;
    if (row_begin >= row_end || cs.n == 0) return;
    const int opk = op_kind(op, p);
    LengthStats ls;
    ls.lmax = lmax; ls.lmin = 1; ls.mean = lmax;
    const Plan pl = make_plan<T>(mode, rows.n, cs.n, ls, ls, dev, opk);
    if (row_begin % (32ull * pl.q) != 0)
      throw Error(ST_INVALID_ARGUMENT, "row_begin must be a multiple of the row chunk (32*q)");
    const size_t need = scratch_needed<T>(mode, rows.n, cs.n, lmax, row_points, col_points);
    if (need > scratch_bytes)
      throw Error(ST_INVALID_ARGUMENT, "problem needs " + std::to_string(need) + " bytes of scratch; the limit is " +
                  std::to_string(scratch_bytes) + " bytes");

    ProblemDesc<T> d{};
    d.rpts = rows.pts; d.roff = rows.off; d.rperm = rperm; d.nr = rows.n;
    d.cpts = cs.pts; d.coff = cs.off; d.cperm = (mode == MODE_CROSS) ? cperm : rperm; d.nc = cs.n;
    d.out = out; d.out_base = out_base; d.ld = cs.n;
    d.row_begin = row_begin; d.row_end = row_end;
    d.q = pl.q; d.mode = mode; d.p = (T)p;
    {
      const uint64_t hi = (rperm || cperm) ? output_count(mode, rows.n, cs.n) : row_output_start(mode, row_end, cs.n);
      d.out_count = hi > out_base ? hi - out_base : 0;
    }
    char* base = static_cast<char*>(scratch);
    if (pl.packed)
    {
      Elem<T>* rp = reinterpret_cast<Elem<T>*>(base + 256);
      SBG_CUDA(launch_pack<T>(rows.pts, rows.off, rows.n, rp, row_points, dev.sms, st));
      d.rpts = reinterpret_cast<const T*>(rp);
      d.cpts = d.rpts;
      d.rcap = row_points;
      d.ccap = row_points;
      if (mode == MODE_CROSS)
      {
        Elem<T>* cp = reinterpret_cast<Elem<T>*>(base + 256 + ((sizeof(Elem<T>) * row_points + 255) / 256) * 256);
        SBG_CUDA(launch_pack<T>(cs.pts, cs.off, cs.n, cp, col_points, dev.sms, st));
        d.cpts = reinterpret_cast<const T*>(cp);
        d.ccap = col_points;
      }
    }
    launch_problem<T>(d, pl, launch_kind(opk, p), st, reinterpret_cast<unsigned long long*>(base));
  }

  template size_t scratch_needed<float>(int, uint64_t, uint64_t, uint32_t, uint64_t, uint64_t);
  template size_t scratch_needed<double>(int, uint64_t, uint64_t, uint32_t, uint64_t, uint64_t);
  template void compute_device_scratch<float>(int, int, double, const PcfSet<float>&, const PcfSet<float>*,
                                              const uint32_t*, const uint32_t*, uint32_t, uint64_t, uint64_t, float*,
                                              uint64_t, uint64_t, uint64_t, void*, size_t, cudaStream_t);
  template void compute_device_scratch<double>(int, int, double, const PcfSet<double>&, const PcfSet<double>*,
                                               const uint32_t*, const uint32_t*, uint32_t, uint64_t, uint64_t,
                                               double*, uint64_t, uint64_t, uint64_t, void*, size_t, cudaStream_t);

  // ---- host pipeline ----------------------------------------------------------

  namespace
  {
    // With the device-verbose setting on, the host entry reports on stderr
    // when each of its phases ended (host clock, ms since the call began);
    // declared first in the call, it reports last, after the buffers are
    // freed.
    struct PhaseLog
    {
      bool on = settings().deviceVerbose.load();
      std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
      std::string text;
      void mark(const char* what, long k = -1)
      {
        if (!on) return;
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        char buf[64];
        if (k >= 0) std::snprintf(buf, sizeof buf, " %s%ld %.1f", what, k, ms);
        else std::snprintf(buf, sizeof buf, " %s %.1f", what, ms);
        text += buf;
      }
      ~PhaseLog()
      {
        if (!on) return;
        mark("freed");
        std::fprintf(stderr, "sbgpu host entry, ms since start:%s\n", text.c_str());
      }
    };

    struct StreamGuard
    {
      cudaStream_t s = nullptr;
      StreamGuard() { SBG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)); }
      ~StreamGuard() { if (s) cudaStreamDestroy(s); }
    };
    struct EventGuard
    {
      cudaEvent_t e = nullptr;
      EventGuard() { SBG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); }
      ~EventGuard() { if (e) cudaEventDestroy(e); }
    };

    // A buffer of the host entry: stream-ordered, from the device's pool.
    struct CallBuffer
    {
      std::unique_ptr<StreamBuffer> buf;
      void reset(size_t bytes, cudaStream_t st) { buf.reset(new StreamBuffer(bytes, st)); }
      void* get() const { return buf ? buf->get() : nullptr; }
      template <typename U> U* as() const { return static_cast<U*>(get()); }
    };

    // Waits, before the buffers declared in front of it go, for every stream
    // that may use them (also where an exception ends the call).
    struct Quiesce
    {
      std::vector<cudaStream_t> streams;
      ~Quiesce()
      {
        for (cudaStream_t s : streams) cudaStreamSynchronize(s);
      }
    };

    template <typename T>
    struct DeviceSet
    {
      CallBuffer pts, off;
      PcfSet<T> view;
      void upload(const PcfSet<T>& h, cudaStream_t s)
      {
        const uint64_t npts = h.n ? h.off[h.n] : 0;
        pts.reset(std::max<uint64_t>(1, npts) * 2 * sizeof(T), s);
        off.reset((h.n + 1) * sizeof(uint64_t), s);
        if (npts) upload_pageable(pts.get(), h.pts, npts * 2 * sizeof(T), s);
        SBG_CUDA(cudaMemcpyAsync(off.get(), h.off, (h.n + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
        view.pts = pts.as<T>();
        view.off = off.as<uint64_t>();
        view.n = h.n;
      }
    };
  }

  template <typename T>
  void compute_host(int mode, int op, double p, const PcfSet<T>& rows, const PcfSet<T>* cols, T* out, bool validate,
                    const RunControl& ctl)
  {
    PhaseLog phases;
    if (mode == MODE_CROSS && !cols) throw Error(ST_INVALID_ARGUMENT, "cdist needs a column set");
    const PcfSet<T>& cs = (mode == MODE_CROSS) ? *cols : rows;
    if (validate)
    {
      validate_pcfs(rows, mode == MODE_CROSS ? "X" : "input");
      if (mode == MODE_CROSS) validate_pcfs(cs, "Y");
    }
    phases.mark("checked");
    (void)op_kind(op, p);
    const uint64_t total = output_count(mode, rows.n, cs.n);
    if (total == 0) return;
    if (!out) throw Error(ST_INVALID_ARGUMENT, "null output");

    const DeviceInfo dev = device_info();
    const LengthStats rstat = host_length_stats(rows.off, rows.n);
    const LengthStats cstat = (mode == MODE_CROSS) ? host_length_stats(cs.off, cs.n) : rstat;
    const uint32_t lmax = std::max(rstat.lmax, cstat.lmax);

    StreamGuard compute, copy, compute2;
    // every buffer is allocated, and given back, on the first stream
    DeviceSet<T> drows, dcols;
    CallBuffer drperm, dcperm, obuf[2], rpack, cpack, fixed_buf;
    Quiesce quiesce{{compute.s, copy.s, compute2.s}};
    drows.upload(rows, compute.s);
    if (mode == MODE_CROSS) dcols.upload(cs, compute.s);
    phases.mark("uploaded");

    // Processing order: by length within windows (unless the order setting
    // asks for the caller's), the permutation the device entry computes on
    // the GPU, so both entries give the same bits.
    size_t freeb = 0, totalb = 0;
    SBG_CUDA(cudaMemGetInfo(&freeb, &totalb));
    const size_t out_bytes = (size_t)total * sizeof(T);
    const size_t budget = (size_t)((double)freeb * 0.8);
    int order = settings().order.load();
    const bool sorted = order != 1 && rows.n <= 0xffffffffull && cs.n <= 0xffffffffull;
    if (sorted)
    {
      // computed on the stream from the uploaded offsets (one launch)
      drperm.reset(std::max<uint64_t>(1, rows.n) * sizeof(uint32_t), compute.s);
      length_order_device(drows.view.off, rows.n, drperm.as<uint32_t>(), nullptr, compute.s);
      if (mode == MODE_CROSS)
      {
        dcperm.reset(std::max<uint64_t>(1, cs.n) * sizeof(uint32_t), compute.s);
        length_order_device(dcols.view.off, cs.n, dcperm.as<uint32_t>(), nullptr, compute.s);
      }
    }

    const Plan pl = make_plan<T>(mode, rows.n, cs.n, rstat, cstat, dev, op_kind(op, p));
    const uint64_t chunk_rows = 32ull * pl.q;
    phases.mark("ordered");

    // Output route.  Direct: on coherent hosts (Grace + NVLink-C2C, where the
    // device walks the host page tables) the kernel stores straight into the
    // caller's matrix, one launch, no device output buffer and no copies.
    // Staged: bands of whole row chunks into two device buffers, each band
    // copied out while the next band computes (HostStager).
    int out_mode = settings().outputMode.load();
    bool direct = false;
    if (out_mode == 2)
    {
      int pageable = 0, hpt = 0;
      host_memory_access(&pageable, &hpt);
      if (!(pageable && hpt))
        throw Error(ST_INVALID_ARGUMENT, "direct host output needs a device that uses the host page tables");
      direct = true;
    }

    // Bands of whole row chunks.  One band when writing directly or when the
    // output is small.  In length order the bands are also whole order
    // windows: the order only permutes PCFs inside a window, so the rows of
    // a band of windows are the same set in either order, and every pair
    // with its later PCF in the band lands in the band's contiguous range
    // of the condensed (or dense) output.
    uint64_t band_bytes = settings().bandBytes.load();
    const bool auto_bands = band_bytes == 0;
    if (band_bytes == 0) band_bytes = out_bytes > (512ull << 20) ? out_bytes / 8 + 1 : out_bytes;
    band_bytes = std::min<uint64_t>(band_bytes, budget / 2 > 0 ? budget / 2 : band_bytes);
    std::vector<std::pair<uint64_t, uint64_t>> bands;
    uint64_t align = chunk_rows;
    if (sorted)
    {
      uint64_t g = align, h = LENGTH_ORDER_WINDOW;
      while (h) { const uint64_t r = g % h; g = h; h = r; }
      align = align / g * LENGTH_ORDER_WINDOW;  // lcm(chunk_rows, window)
    }
    if (direct || band_bytes >= out_bytes)
    {
      if (!direct && out_bytes > budget) throw Error(ST_OUT_OF_MEMORY, "output does not fit in device memory");
      bands.emplace_back(0, rows.n);
    }
    else
    {
      // Bands of whole row units, from the last row down.  Nothing overlaps
      // the copy-out of the band computed last, and in a triangle the first
      // rows hold the least output, so the schedule ends on them.  With
      // automatic sizes the two lowest bands are cut into parts of about
      // 1/2, 1/4, ... of their output, top part first, so the last copy is
      // the first unit's output (about 2 MB for 1024 rows in float32), not
      // a full band's.
      const uint64_t units = (rows.n + align - 1) / align;
      auto ustart = [&](uint64_t u) { return std::min<uint64_t>(rows.n, u * align); };
      uint64_t ue = units;
      while (ue > 0)
      {
        uint64_t ub = ue - 1;
        while (ub > 0)
        {
          const uint64_t bytes =
              (row_output_start(mode, ustart(ue), cs.n) - row_output_start(mode, ustart(ub - 1), cs.n)) * sizeof(T);
          if (bytes > band_bytes) break;
          --ub;
        }
        bands.emplace_back(ustart(ub), ustart(ue));
        ue = ub;
      }
      if (auto_bands && bands.size() > 1)
      {
        // The two lowest bands are cut again into parts of about half the
        // remaining output each: every part's copy-out (about 3x faster than
        // the kernel writes it) then hides behind the compute of the next,
        // which is at least half its size, and the last part is unit 0.
        bands.pop_back();
        const auto above = bands.back();  // the lowest two end here
        bands.pop_back();
        uint64_t top = (above.second + align - 1) / align;
        auto out_of = [&](uint64_t u0, uint64_t u1) {
          return row_output_start(mode, ustart(u1), cs.n) - row_output_start(mode, ustart(u0), cs.n);
        };
        while (top > 1)
        {
          const uint64_t half = out_of(0, top) / 2;
          uint64_t ub = top - 1;
          while (ub > 1 && out_of(ub, top) < half) --ub;
          bands.emplace_back(ustart(ub), ustart(top));
          top = ub;
        }
        bands.emplace_back(0, ustart(top));
      }
    }
    uint64_t max_band = 0;
    for (auto& b : bands)
      max_band = std::max<uint64_t>(max_band, row_output_start(mode, b.second, cs.n) - row_output_start(mode, b.first, cs.n));
    const int nbuf = direct ? 0 : (bands.size() > 1 ? 2 : 1);
    for (int b = 0; b < nbuf; ++b) obuf[b].reset(std::max<uint64_t>(1, max_band) * sizeof(T), compute.s);
    EventGuard computed[2], copied[2];
    phases.mark("buffers");

    // Packed segment layout, once, for the global-memory variant; or the
    // fixed-point path's arrays.
    const T* kr_pts = drows.view.pts;
    const T* kc_pts = (mode == MODE_CROSS) ? dcols.view.pts : drows.view.pts;
    FixedRun fixed;
    if constexpr (sizeof(T) == 8)
    {
      const int k = op_kind(op, p);
      if (FixedRun::wanted(k))
      {
        fixed.layout(k, mode, rows.n, cs.n, lmax, rows.off[rows.n], cs.off[cs.n], 0, dev, FixedRun::SLOTS);
        try { fixed_buf.reset(fixed.total, compute.s); }
        catch (const Error& e)
        {
          if (e.status != ST_OUT_OF_MEMORY) throw;  // the direct path needs less
        }
        if (fixed_buf.get())
        {
          fixed.prepare(fixed_buf.as<char>(), drows.view, mode == MODE_CROSS ? dcols.view : drows.view, pl.packed,
                        sorted ? drperm.as<uint32_t>() : nullptr,
                        sorted && mode == MODE_CROSS ? dcperm.as<uint32_t>() : nullptr, compute.s);
        }
      }
    }
    if (pl.packed && !fixed_buf.get())
    {
      rpack.reset(sizeof(Elem<T>) * std::max<uint64_t>(1, rows.off[rows.n]), compute.s);
      SBG_CUDA(launch_pack<T>(drows.view.pts, drows.view.off, rows.n, rpack.as<Elem<T>>(), rows.off[rows.n], dev.sms,
                              compute.s));
      kr_pts = reinterpret_cast<const T*>(rpack.get());
      kc_pts = kr_pts;
      if (mode == MODE_CROSS)
      {
        cpack.reset(sizeof(Elem<T>) * std::max<uint64_t>(1, cs.off[cs.n]), compute.s);
        SBG_CUDA(launch_pack<T>(dcols.view.pts, dcols.view.off, cs.n, cpack.as<Elem<T>>(), cs.off[cs.n], dev.sms,
                                compute.s));
        kc_pts = reinterpret_cast<const T*>(cpack.get());
      }
    }
    const int opk = op_kind(op, p);

    // Bands alternate between two compute streams, one per output buffer:
    // a band's CTAs start on the SMs that the previous band's last wave
    // leaves idle, instead of after its last item.  Bands share nothing but
    // the inputs, which the second stream waits for.
    EventGuard inputs_ready;
    SBG_CUDA(cudaEventRecord(inputs_ready.e, compute.s));
    SBG_CUDA(cudaStreamWaitEvent(compute2.s, inputs_ready.e, 0));
    auto band_stream = [&](size_t k) { return (k % 2) ? compute2.s : compute.s; };

    auto launch_band = [&](size_t k) {
      const int b = (int)(k % 2);
      const cudaStream_t bs = band_stream(k);
      if (k >= 2) SBG_CUDA(cudaStreamWaitEvent(bs, copied[b].e, 0));
      ProblemDesc<T> d{};
      d.rpts = kr_pts; d.roff = drows.view.off; d.nr = rows.n;
      d.cpts = kc_pts; d.coff = (mode == MODE_CROSS) ? dcols.view.off : drows.view.off; d.nc = cs.n;
      d.rperm = sorted ? drperm.as<uint32_t>() : nullptr;
      d.cperm = sorted ? (mode == MODE_CROSS ? dcperm.as<uint32_t>() : drperm.as<uint32_t>()) : nullptr;
      d.out = direct ? out : obuf[b].as<T>();
      d.out_base = direct ? 0 : row_output_start(mode, bands[k].first, cs.n);
      d.out_count = direct ? total : row_output_start(mode, bands[k].second, cs.n) - d.out_base;
      d.ld = cs.n;
      d.row_begin = bands[k].first; d.row_end = bands[k].second;
      d.q = pl.q; d.mode = mode; d.p = (T)p;
      d.rcap = rows.off[rows.n];
      d.ccap = cs.off[cs.n];
      // The small bands at the end of the schedule take fewer rows per item,
      // so that each still gives the planner's 6 items per SM instead of
      // ending on a ragged last wave.  Only an even q is halved, so the new
      // row chunk divides the old one and the band starts stay multiples of
      // it.  No pair's arithmetic depends on the item shape.
      if (!direct)
        while (d.q % 2 == 0 && problem_item_count(d) < 6ull * (uint64_t)dev.sms) d.q /= 2;
      if constexpr (sizeof(T) == 8)
      {
        if (fixed_buf.get())
        {
          fixed.launch(d, drows.view.pts, mode == MODE_CROSS ? dcols.view.pts : drows.view.pts, pl, b, bs);
          SBG_CUDA(cudaEventRecord(computed[b].e, bs));
          return;
        }
      }
      launch_problem<T>(d, pl, launch_kind(opk, p), bs);
      SBG_CUDA(cudaEventRecord(computed[b].e, bs));
    };

    bool cancelled = false;
    if (direct)
    {
      launch_band(0);
      SBG_CUDA(cudaStreamSynchronize(compute.s));
      if (ctl.progress) ctl.progress(total);
      return;
    }
    launch_band(0);
    if (bands.size() == 1 && host_pages_mapped())
    {
      // One band, on a host whose page tables the device walks: the copy
      // engine writes the caller's pages as fast as pinned ones (180 GB/s)
      // once they exist, and the host makes them while the kernel runs.
      // Through the staging buffers, 8 MB of fresh pages cost 420 us of one
      // thread's memcpy on top of the 52 of the transfer, 72 MB 1.3 ms of
      // sixteen threads'.
      const uint64_t hi = row_output_start(mode, bands[0].second, cs.n);
      if (make_pages(out, hi * sizeof(T)))
      {
        SBG_CUDA(cudaStreamWaitEvent(copy.s, computed[0].e, 0));
        if (hi) SBG_CUDA(cudaMemcpyAsync(out, obuf[0].as<T>(), hi * sizeof(T), cudaMemcpyDeviceToHost, copy.s));
        SBG_CUDA(cudaStreamSynchronize(copy.s));
        phases.mark("band", 0);
        if (ctl.progress) ctl.progress(hi);
        if (ctl.stop && ctl.stop->load()) throw Error(ST_CANCELLED, "task was cancelled");
        return;
      }
    }
    HostStager stager(std::min<uint64_t>(std::max<uint64_t>(max_band * sizeof(T), 1), 256ull << 20));
    for (size_t k = 0; k < bands.size(); ++k)
    {
      const int b = (int)(k % 2);
      if (k + 1 < bands.size() && !(ctl.stop && ctl.stop->load())) launch_band(k + 1);
      const uint64_t rb = bands[k].first, re = bands[k].second;
      const uint64_t lo = row_output_start(mode, rb, cs.n);
      const uint64_t hi = row_output_start(mode, re, cs.n);
      SBG_CUDA(cudaStreamWaitEvent(copy.s, computed[b].e, 0));
      if (hi > lo) stager.copy(out + lo, obuf[b].as<T>(), (hi - lo) * sizeof(T), copy.s);
      stager.flush();
      phases.mark("band", (long)k);
      SBG_CUDA(cudaEventRecord(copied[b].e, copy.s));
      if (ctl.progress) ctl.progress(hi - lo);
      if (ctl.stop && ctl.stop->load()) { cancelled = true; break; }
    }
    stager.flush();
    SBG_CUDA(cudaStreamSynchronize(compute.s));
    SBG_CUDA(cudaStreamSynchronize(compute2.s));
    SBG_CUDA(cudaStreamSynchronize(copy.s));
    phases.mark("synced");
    if (cancelled) throw Error(ST_CANCELLED, "task was cancelled");
  }

  template void compute_host<float>(int, int, double, const PcfSet<float>&, const PcfSet<float>*, float*, bool,
                                    const RunControl&);
  template void compute_host<double>(int, int, double, const PcfSet<double>&, const PcfSet<double>*, double*, bool,
                                     const RunControl&);
}
