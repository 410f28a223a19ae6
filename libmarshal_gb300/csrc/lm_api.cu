// lm_api.cu -- host dispatch, planner and the exported C ABI.
//
// Drop-in surface (see include/marshal.h and include/lm_marshal.h):
//   gpu_aos_asta_bs_float/double, gpu_aos_asta_pttwac, gpu_soa_asta_pttwac
//       -- include/marshal.h:26-31 of the reference, same signatures;
//   lm_* -- one entry per cl_* function of include/cl_marshal.h:26-49 with
//       (cl_command_queue, cl_mem) replaced by (cudaStream_t, void *buf, int
//       elem_bytes); same argument order, same meaning, same error convention:
//       false on success, true on error (API.wiki:12,20), with the message
//       available from lm_last_error().
//
// Everything is stream ordered.  Scratch (done bits, ticket words) comes from
// the device's stream-ordered memory pool (cudaMallocAsync / cudaFreeAsync on
// the caller's stream), so concurrent calls on different streams never share
// it and repeated calls reuse pooled memory instead of allocating.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "lm_core.cuh"
#include "lm_internal.h"
#include "../../include/lm_marshal.h"
#include "../../include/marshal.h"

namespace lm {

// ---- device info ------------------------------------------------------------

const DeviceInfo &device_info() {
  static DeviceInfo cache[64];
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  DeviceInfo &d = cache[dev & 63];
  if (d.device != dev) {
    std::lock_guard<std::mutex> lock(mu);
    if (d.device != dev) {
      DeviceInfo n;
      n.device = dev;
      cudaDeviceGetAttribute(&n.sms, cudaDevAttrMultiProcessorCount, dev);
      cudaDeviceGetAttribute(&n.max_smem_optin,
                             cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      cudaDeviceGetAttribute(&n.max_smem_per_sm,
                             cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
      cudaDeviceGetAttribute(&n.cc_major, cudaDevAttrComputeCapabilityMajor, dev);
      cudaDeviceGetAttribute(&n.cc_minor, cudaDevAttrComputeCapabilityMinor, dev);
      if (n.sms <= 0) n.sms = 1;
      if (n.max_smem_optin <= 0) n.max_smem_optin = 48 * 1024;
      d = n;
    }
  }
  return d;
}

// ---- errors -----------------------------------------------------------------

static thread_local std::string g_err;

static bool fail(const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  if (getenv("LM_VERBOSE")) fprintf(stderr, "libmarshal_gb300: %s\n", buf);
  return true;
}

bool set_error(const char *msg) {
  cudaGetLastError();  // (as in cuda_fail)
  return fail("%s", msg);
}

static bool cuda_fail(cudaError_t e, const char *what) {
  cudaGetLastError();  // reported here, not by the next call's check
  return fail("%s: %s", what, cudaGetErrorString(e));
}

// ---- scratch ----------------------------------------------------------------

void pool_keep_memory() {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (done[dev & 63].load(std::memory_order_acquire)) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    uint64_t thr = ~0ull;  // keep freed blocks pooled between calls
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
  }
  done[dev & 63].store(true, std::memory_order_release);
}

struct Scratch {
  void *p = nullptr;
  cudaStream_t s = nullptr;
  ~Scratch() {
    if (p) cudaFreeAsync(p, s);
  }
};

// Like get_scratch, but a failed allocation only returns false (no error
// recorded): for plans that have a fallback.
static bool try_scratch(Scratch &sc, size_t bytes, cudaStream_t s) {
  pool_keep_memory();
  sc.s = s;
  if (cudaMallocAsync(&sc.p, bytes ? bytes : 4, s) != cudaSuccess) {
    cudaGetLastError();
    sc.p = nullptr;
    return false;
  }
  return true;
}

// Memory for a list of cycles that is not kept, asked for where there is
// such a list alone.
static auto list_scratch(Scratch &sc, cudaStream_t s) {
  return [&sc, s](size_t bytes) -> void * {
    return try_scratch(sc, bytes, s) ? sc.p : nullptr;
  };
}

static bool get_scratch(Scratch &sc, size_t bytes, cudaStream_t s) {
  pool_keep_memory();
  sc.s = s;
  cudaError_t e = cudaMallocAsync(&sc.p, bytes ? bytes : 4, s);
  if (e != cudaSuccess) {
    sc.p = nullptr;
    return cuda_fail(e, "scratch allocation");
  }
  return false;
}

static bool get_zeroed(Scratch &sc, size_t bytes, cudaStream_t s) {
  pool_keep_memory();
  sc.s = s;
  cudaError_t e = cudaMallocAsync(&sc.p, bytes ? bytes : 4, s);
  if (e != cudaSuccess) {
    sc.p = nullptr;
    return cuda_fail(e, "scratch allocation");
  }
  e = cudaMemsetAsync(sc.p, 0, bytes ? bytes : 4, s);
  if (e != cudaSuccess) return cuda_fail(e, "scratch clear");
  return false;
}

// ---- persistent status word (failures of waiting kernels) ---------------

uint32_t *device_status_word() {
  static std::mutex mu;
  static uint32_t *words[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!words[dev]) {
    void *p = nullptr;
    if (cudaMalloc(&p, 4) != cudaSuccess || cudaMemset(p, 0, 4) != cudaSuccess) {
      cudaGetLastError();  // the callers have other ways
      return nullptr;
    }
    words[dev] = (uint32_t *)p;
  }
  return words[dev];
}

// A zeroed word of pinned host memory for one call's kernel, from a page
// kept for the process (as many words as calls ever wait at once).
struct HostWord {
  static std::mutex &mu() {
    static std::mutex m;
    return m;
  }
  static std::vector<uint32_t *> &pool() {
    static std::vector<uint32_t *> v;
    return v;
  }
  uint32_t *p = nullptr;
  bool lost = false;  // not to be given back
  HostWord() {
    std::lock_guard<std::mutex> lock(mu());
    if (pool().empty()) {
      void *page = nullptr;
      constexpr int kWords = 64;
      if (cudaHostAlloc(&page, kWords * 64, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return;
      }
      for (int i = 0; i < kWords; ++i)
        pool().push_back((uint32_t *)((char *)page + 64 * i));
    }
    p = pool().back();
    pool().pop_back();
    *(volatile uint32_t *)p = 0;
  }
  ~HostWord() {
    if (!p || lost) return;
    std::lock_guard<std::mutex> lock(mu());
    pool().push_back(p);
  }
};

// The task flags of one padding call.  Blocks of kWords words are kept per
// device (kKept at most, until lm_marshal_finalize) and never cleared: a call
// hands its kernel an epoch that no word holds yet and the ticket word's
// value.  A block is given back when the call has waited for its kernel; one
// whose kernel failed is not.  Larger calls allocate theirs.
struct PadBlock {
  static constexpr uint64_t kWords = 16 * 1024;
  static constexpr size_t kKept = 16;
  struct Kept {
    uint32_t *p;
    uint32_t ticket, epoch;
  };
  static std::mutex &mu() {
    static std::mutex m;
    return m;
  }
  static std::vector<Kept> &pool(int dev) {
    static std::vector<Kept> v[64];
    return v[dev & 63];
  }
  PadFlags f;
  Scratch own;        // not from the pool
  int dev = 0;
  bool kept = false;  // from the pool
  bool done = false;  // the kernel has finished without a failure
  uint64_t started = 0;  // tasks of the kernel, which take a ticket each
  // false: no memory
  bool take(uint64_t n, cudaStream_t s) {
    cudaGetDevice(&dev);
    kept = n + 2 <= kWords;
    if (kept) {
      std::lock_guard<std::mutex> lock(mu());
      if (!pool(dev).empty()) {
        const Kept k = pool(dev).back();
        pool(dev).pop_back();
        f.p = k.p;
        f.words = kWords;
        f.ticket = k.ticket;
        f.epoch = k.epoch + 1;
        return true;
      }
    }
    f.words = kept ? kWords : n + 2;
    if (get_zeroed(own, f.words * 4, s)) return false;
    f.p = (uint32_t *)own.p;
    if (kept) own.p = nullptr;
    return true;
  }
  ~PadBlock() {
    if (!kept || !f.p) return;
    std::lock_guard<std::mutex> lock(mu());
    if (done && pool(dev).size() < kKept && f.epoch != 0xffffffffu)
      pool(dev).push_back({f.p, f.ticket + (uint32_t)started, f.epoch});
    else
      cudaFreeAsync(f.p, own.s);  // (the call has waited for its stream)
  }
  static void clear(int dev) {
    std::lock_guard<std::mutex> lock(mu());
    for (const Kept &k : pool(dev)) cudaFree(k.p);
    pool(dev).clear();
  }
};

// Reads and clears the status word after the stream's work has finished.
static bool check_status(cudaStream_t s, const char *what) {
  uint32_t *w = device_status_word();
  if (!w) return fail("%s: no status word", what);
  uint32_t v = 0;
  cudaError_t e = cudaMemcpyAsync(&v, w, 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, what);
  if (v != kStatusOk) {
    cudaMemsetAsync(w, 0, 4, s);
    return fail("%s: an inter-CTA wait timed out (status %u)", what, v);
  }
  return false;
}

// ---- timing (the reference's elapsed_time accumulator) ----------------------

struct OpTimer {
  unsigned long long *et;
  cudaStream_t s;
  cudaEvent_t a = nullptr, b = nullptr;
  OpTimer(unsigned long long *et_, cudaStream_t s_) : et(et_), s(s_) {
    if (et) {
      cudaEventCreate(&a);
      cudaEventCreate(&b);
      cudaEventRecord(a, s);
    }
  }
  // Adds the elapsed kernel time in ns (blocks, like Profiling::Report).
  bool finish() {
    if (!et) return false;
    cudaEventRecord(b, s);
    cudaError_t e = cudaEventSynchronize(b);
    if (e != cudaSuccess) return cuda_fail(e, "timing");
    if (check_status(s, "status")) return true;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    *et += (unsigned long long)((double)ms * 1.0e6);
    return false;
  }
  ~OpTimer() {
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
  }
};

static bool valid_e(int e) { return e == 1 || e == 2 || e == 4 || e == 8; }

// Elements are moved as e-byte words, so the buffer must be e-byte aligned.
static bool misaligned(const void *buf, int e) {
  return ((uintptr_t)buf & (uintptr_t)(e - 1)) != 0;
}

// Limit for every inter-CTA wait (LM_WAIT_TIMEOUT_MS overrides, default 2 s).
static uint64_t wait_timeout_ns() {
  const char *v = getenv("LM_WAIT_TIMEOUT_MS");
  const long long ms = v ? atoll(v) : 2000;
  return (uint64_t)(ms > 0 ? ms : 2000) * 1000000ull;
}

// ---- planner ----------------------------------------------------------------

constexpr uint64_t kWalkMinBytes = 16ull << 20;
constexpr uint64_t kWalkUnkeptBytes = 80ull << 20;

// Whether the ordered form (3 x payload, k_wave) is faster than the staged one
// (4 x, but no waits, and a copy back out of L2 up to 208 MB): its slack is
// 20 MB of blocks in flight.  Microseconds, staged and ordered: floats of 401
// columns, 90 MB 58 and 62, 120 MB 79 and 80, 150 MB 97 and 93; doubles of
// 2001, 90 MB 57 and 55, 150 MB 97 and 86; half-words of 1001, 120 MB 88 and
// 92, 150 MB 110 and 110; bytes of 5001, 120 MB 95 and 100, 150 MB 121 and
// 119.  Output rows of whole vectors: floats 88 MB 57 and 56, 109 MB 73 and
// 66; bytes 104 MB 70 and 72, 131 MB 91 and 87; units of 32 bytes, 81 MB 50
// and 50, 101 MB 65 and 60.  Short rows make more blocks per byte: rows of
// 46 bytes, 190 MB 138 and 151, 300 MB 223 and 226; 17 floats, 150 MB 99 and
// 107, 300 MB 201 and 190; 11 floats, 600 MB 404 and 423; 3 doubles 513 and
// 663.  Several instances run in the ordered form one after another, in the
// staged one at once: 3 of 100 MB of floats 199 and 197, 3 of 168 MB 330 and
// 300, 2 of 268 MB 351 and 282; 3 of 117 MB of bytes 279 and 291.
// Units of several elements that are no whole vectors are written one element
// at a time: blocks that take longer and of which fewer are in flight, so the
// form pays later (20000 rows and 40, wave and staged: 12-byte units 130 MB 124
// and 113, 110 and 114, 200 MB 167 and 175, 160 and 172; 66-byte ones 200 MB 273
// and 270, 251 and 264, 300 MB 398 and 409, 370 and 402; 9-byte ones 130 MB 285
// and 290, 278 and 292; 24-byte ones of doubles 110 MB 80 and 76, 72 and 73, 160
// MB 107 and 109, 99 and 108).
static bool wave_preferred(const void *buf, uint64_t T, uint64_t a, uint64_t B,
                           uint64_t b, int e) {
  const uint64_t U = b * e, bytes = a * B * U, row = B * U;
  const bool vectors = ((uintptr_t)buf & 15) == 0 && a * U % 16 == 0;
  uint64_t least = (U < 4 ? (vectors ? 104ull : 144ull)
                          : (vectors ? 88ull : 112ull)) << 20;
  if (U < 4 && row <= 304) least = 208ull << 20;
  if (U >= 4 && row < 96) least = 192ull << 20;
  if (U >= 4 && row < 64) return false;
  if (b > 1 && (U % 16 || ((uintptr_t)buf & 15)))
    least = std::max<uint64_t>(least, (e == 1   ? 160ull
                                       : e == 2 ? 256ull
                                       : e == 4 ? 208ull
                                                : 144ull) << 20);
  if (T > 1) least = std::max<uint64_t>(least, 128ull << 20);
  return bytes >= least;
}

// Whether a walk is the faster form for units that it takes: against the
// ordered form by the lines that it reads, beyond L2 (walk_by_lines; 128 MB: 66
// and 79 us at 140 MB for 128-byte units on lines, 57 and 57 at 100 and 87 and
// 78 at 140 off them); against the staged form always where the list of its
// cycles is kept (60 MB of 128-byte units 27 and 33, of 320-byte ones 33 and
// 35), and from 80 MB on where it is found on every call, as under stream
// capture (34 MB 29 and 23, 60 MB 35 to 48 and 35, 84 MB 44 to 49 and 52).
// Units of 1 KB and more have neither (34 MB 19 and 33 by done bits).
static bool walk_preferred(const void *buf, uint64_t T, uint64_t a, uint64_t B,
                           uint64_t U, bool may_keep, bool wave) {
  const uint64_t bytes = T * a * B * U;
  if (U >= kStagedMaxUnit) return true;
  if (bytes < kWalkUnkeptBytes && !(may_keep && walk_list_kept(a, B)))
    return false;
  return bytes < (128ull << 20) || !wave || walk_by_lines(buf, U);
}

// Scratch of the ordered form for T instances one after another (the same plan
// for every instance, but for its place in 16 bytes); 0 where it does not
// take them.
static size_t wave_scratch(void *buf, uint64_t T, uint64_t a, uint64_t B,
                           uint64_t b, int e) {
  const uint64_t step = a * B * b * e;
  size_t need = 0;
  for (uint64_t t = 0; t < T && t < 16; ++t) {
    const size_t n = wave0100_scratch((char *)buf + t * step, a, B, b, e);
    if (n == 0) return 0;
    need = std::max(need, n);
  }
  return need;
}

// The stash plan before the forms through scratch, where its wavefront has the
// rows (kStashRowsPerSm).  Its writers go down a column of rows, the blocks of
// the others write units of several elements one element at a time, if those are
// no whole vectors.  Microseconds, stash and the better of staged and ordered (with
// the row offsets of the stash kept; found on each call, as where 16 shapes are
// kept already, they cost 12 more):
//  * units of several bytes or half-words, at every size: 20000 rows of 9-byte
//    units, 34 / 100 / 200 MB, 51 / 127 / 234 and 88 / 230 / 424, 7400 rows of
//    10-byte ones 50 / 126 / 238 and 59 / 134 / 267;
//  * of several words too: 15001 rows of 12-byte units, 48 / 112 / 300 MB, 43 / 79 /
//    173 and 50 / 98 / 237, 8000 of 44-byte ones 41 / 79 / 177 and 50 / 98 / 234;
//  * of several doubles from 128 MB on: 12298 rows of 40-byte units, 64 / 112 / 160 /
//    600 MB, 51 / 76 / 99 / 316 and 45 / 76 / 112 / 338;
//  * half-words in tall matrices whose output rows are no whole vectors long: at
//    13530 columns level with the ordered form at 20000 rows, and faster above
//    (23001 372 and 384, 28775 443 and 478, 38902 554 and 639); with fewer columns
//    it loses some of that (28775 x 7003 239 and 254, 4005 152 and 155, 2005 92 and
//    85).  Rows 2 bytes past whole vectors take it 13-15 % longer at every height,
//    for no cause that could be shown; those of the seven other places do not
//    differ.  (Bytes, 28775 x 27060: 657 and 514.)
// Strips of fewer than 384 bytes, in very tall matrices, are for narrow elements.
static bool stash_preferred(const void *buf, uint64_t T, uint64_t a, uint64_t B,
                            uint64_t b, int e) {
  if (T != 1 || b * e >= 128 || a * B < (1ull << 20) ||
      a < kStashRowsPerSm * (uint64_t)device_info().sms)
    return false;
  const bool vectors = b * e % 16 == 0 && ((uintptr_t)buf & 15) == 0;
  if (b == 1 ? e != 2 || a < 23000 || B < 4000 || B * 2 % 16 == 2 ||
                   a * 2 % 16 == 0 || !wave_preferred(buf, T, a, B, 1, 2)
             : vectors || (e == 8 && a * B * b * e < (128ull << 20)))
    return false;
  if (getenv("LM_NO_STASH")) return false;
  const StashPlan p = plan_stash(a, B, (uint32_t)b, e);
  return p.feasible && (e < 4 || p.g * b * e >= 384);
}

// Whether a conversion in on-chip tiles by `p` is slower than what takes it
// otherwise, in nanoseconds fitted to 2500 shapes of 4 KB to 28 MB (the choice
// costs 0.4 to 0.8 % on average over the faster of the two, and 20 % in one of
// a hundred).  A CTA moves its elements one by one, at about 0.32 ns each and
// half that where the bands of a cluster do, tile after tile where there are more
// than fit (a GPC has room for one cluster of 16): 41 x 1598 bytes 25.0 us, held in the
// shared memory of all SMs 12.2, 362 x 362 half-words in a cluster of four 18.8
// and 11.9, 9 tiles of 327 x 38 units of 210 bytes 52 and 39.  The held form
// takes 6 to 10 us, and
//  * for units of one element 0.3 to 0.6 us per MB, and some for each tile and
//    row (22 tiles of 246 x 74 doubles 10.3 and 8.3, 66 of 363 x 17 8.3 and 10.4,
//    2108 of 2679 x 2 half-words 23.2 and 37.6), but 0.4 to 2.6 us per MB where a
//    column is a vector or two or a part of one (62 tiles of 8 x 8266 floats 8.8
//    and 17.0, 27 of 4 x 107368 half-words 24.6 and 51.0);
//  * for units of several, which it writes one element at a time too, the time
//    of an SM's share of them and of the tiles' rows: 2 tiles of 92 x 30 units of
//    45 bytes 49.5 and 10.1, but 148 of 91 x 2 of 163 bytes 16.5 and 24.7, 35 of
//    3 x 2405 of 86 bytes 23.2 and 33.4.
// Units of 64 bytes and more whose cycles are short go to those instead: 9 us
// where their list is kept, 14.5 where not (4 x 40 units of 1536 bytes 8.3 and
// 15.2), and 0.5 per MB of doubles to 4 per MB of bytes (314 tiles of 5 x 38 units
// of 347 bytes 56.9 and 70.5); where it is kept with half of the SMs idle from
// 512 KB on in any case (21 tiles of 8 x 2 units of 6776 bytes 8.3 and 7.4).
static bool held_preferred(const void *buf, uint64_t T, uint64_t a, uint64_t B,
                           uint64_t b, int e, const BsPlan &p) {
  const uint64_t sms = (uint64_t)device_info().sms, C = (uint64_t)p.cluster;
  const uint64_t chunks = (T + p.tiles_per_chunk - 1) / p.tiles_per_chunk;
  const uint64_t all = T * a * B * b, bytes = all * (uint64_t)e;
  const uint64_t rows = T * a / sms;
  const bool vectors = ((uintptr_t)buf & 15) == 0;
  // elements of an SM, or of a CTA of a cluster for as many rounds as it takes
  // (one cluster of 16 to a GPC of about 20 SMs, two of 8, ...)
  const uint64_t fit = std::max<uint64_t>(
      1, sms * (C == 2 ? 76 : C == 4 ? 36 : C == 8 ? 15 : 7) / 152);
  const uint64_t elems =
      C == 1 ? a * B * b * p.tiles_per_chunk * std::max(chunks, sms) / sms
             : a * b * p.rows_per_cta * ((chunks + fit - 1) / fit);
  if (b == 1) {
    const uint64_t out = a * e;  // bytes of an output row
    const uint64_t ps = !vectors || out % 16 ? 180 : e == 1 ? 50 : e == 2 ? 80 : 100;
    const uint64_t tile = C == 1   ? 3800 + elems * 32 / 100
                          : e == 8 ? 4400 + elems * 28 / 100 + a * 2
                                   : 5300 + elems * ps / 1000 + a * 2;
    if ((out == 4 || out == 8 || out == 16 || out == 32) &&
        ((uintptr_t)buf & 3) == 0 && (a >= 4 || e == 8))
      return tile > (e == 1   ? 20000 + bytes / 450
                     : e == 2 ? 12500 + bytes / 550
                     : e == 4 ? 9500 + bytes / 1000
                              : 7400 + bytes / 1000);
    return tile > T * 350 / sms + (e == 1   ? 9300 + bytes / 1700 + rows * 35 / 100
                                   : e == 2 ? 8200 + bytes / 2000 + rows * 35 / 100
                                   : e == 4 ? 6700 + bytes / 3000 + rows * 3
                                            : 6500 + bytes / 3300 + rows * 3);
  }
  const uint64_t tile = C == 1  ? 3400 + elems * 36 / 100
                        : e < 8 ? 6500 + elems * 18 / 100 + a * 2
                                : 4800 + elems * 26 / 100 + a * 2;
  const uint64_t share = std::max<uint64_t>(all / sms, 8192 / (uint64_t)e);
  if (tile <= (e == 1   ? 8000 + share * 32 / 100 + bytes / 20000 + rows * 2
               : e == 2 ? 8300 + share * 33 / 100 + bytes / 10000 + rows * 6
               : e == 4 ? 7100 + share * 26 / 100 + bytes / 6000 + rows * 4
                        : 6400 + bytes / 5000 + rows * 8 +
                              share * (vectors && b % 2 == 0 ? 13 : 18) / 100))
    return false;
  if (b * e < 64 || getenv("LM_NO_CYCLES") || a * B - 1 > (1ull << 28) ||
      !cycle_order(a, B, kCycleMaxLen))
    return true;
  const bool kept = cycle_list_kept(a, B, 0);
  return tile > (kept ? 9000 : 14500) + bytes / (e == 1   ? 500
                                                 : e == 2 ? 900
                                                 : e == 4 ? 1300
                                                          : 2000) ||
         (kept && bytes >= (512ull << 10) && chunks * C * 2 < sms);
}

enum class Method { Auto, BS, Pttwac, Stash, TwoPass, Cycles, Staged, Resident };

TuneParams &tune_params() {
  static thread_local TuneParams p;
  return p;
}

bool &planner_beside_other_work() {
  static thread_local bool v = false;
  return v;
}

// A tuned choice: the method, and the variant of it (an index into the
// table below) in bits 8-15.
struct TuneVariant {
  Method m;
  TuneParams p;
};
static const TuneVariant kVariants[] = {
    {Method::Auto, {}},
    {Method::Staged, {16u << 10, 0}},
    {Method::Staged, {0, 0}},            // 32 KB blocks (built-in)
    {Method::Staged, {64u << 10, 0}},
    {Method::Cycles, {}},
    {Method::Stash, {0, 0}},             // the planner's CTAs per SM
    {Method::Stash, {0, 1}},
    {Method::Stash, {0, 2}},
    {Method::TwoPass, {}},
    {Method::Pttwac, {}},
};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));

static bool check_launch(cudaError_t e, const char *what) {
  if (e != cudaSuccess) return cuda_fail(e, what);
  return false;
}

static bool run_pttwac_direct(cudaStream_t s, void *buf, int e, uint64_t T,
                              uint64_t a, uint64_t B, uint64_t b) {
  const size_t fb = pttwac_flag_bytes(buf, T, (uint32_t)a, (uint32_t)B,
                                      (uint32_t)b, e);
  if (fb == 0) return fail("PTTWAC: shape exceeds 2^32 units per instance");
  Scratch flags;
  if (get_zeroed(flags, fb, s)) return true;
  return check_launch(launch_pttwac0100(s, buf, e, T, (uint32_t)a,
                                        (uint32_t)B, (uint32_t)b,
                                        (uint32_t *)flags.p),
                      "PTTWAC launch");
}

// Largest-unit-first search for a two-pass split of one 100(a, B, b):
// returns a2 | a with a2*U in [128, 1024] bytes whose tile a2 x B x b fits BS.
static uint64_t split_a(uint64_t a, uint64_t B, uint64_t b, int e) {
  const uint64_t U = b * e;
  uint64_t best = 0;
  for (uint64_t d = 2; d <= a && d * U <= 1024; ++d) {
    if (a % d) continue;
    if (d * U < 128) continue;
    BsPlan p = plan_bs0100(1, (uint32_t)d, (uint32_t)B, (uint32_t)b, e);
    if (!p.feasible) continue;
    best = d;
    break;  // smallest d with a >= 128-byte unit
  }
  return best;
}

static uint64_t split_B(uint64_t a, uint64_t B, uint64_t b, int e) {
  const uint64_t U = b * e;
  for (uint64_t c = 2; c <= B && c * U <= 1024; ++c) {
    if (B % c) continue;
    if (c * U < 128) continue;
    BsPlan p = plan_bs0100(1, (uint32_t)a, (uint32_t)c, (uint32_t)b, e);
    if (!p.feasible) continue;
    return c;
  }
  return 0;
}

// 0100(T, a, B, b): [T][a][B][b] -> [T][B][a][b] with e-byte elements.
static bool do_0100(cudaStream_t s, void *buf, int e, uint64_t T, uint64_t a,
                    uint64_t B, uint64_t b, Method m) {
  if (!valid_e(e)) return fail("element size must be 1, 2, 4 or 8 (got %d)", e);
  if (T == 0 || a == 0 || B == 0 || b == 0) return false;  // empty
  if (a == 1 || B == 1) return false;                      // identity
  if (buf == nullptr) return fail("null buffer");
  if (misaligned(buf, e)) return fail("buffer must be aligned to the element size");
  if (a * B >= 0xffffffffull) return fail("a*B must be < 2^32");
  widen_units(buf, &e, &b);
  if (m == Method::Auto && a == B && !getenv("LM_NO_SQUARE") &&
      square0100_applies(buf, T, a, B, b, e)) {
    uint32_t *status = device_status_word();
    return check_launch(launch_square0100(s, buf, e, T, a, b, status,
                                          wait_timeout_ns()),
                        "square launch");
  }
  if (m == Method::Auto || m == Method::BS) {
    BsPlan p = plan_bs0100(T, (uint32_t)a, (uint32_t)B, (uint32_t)b, e);
    // a megabyte or more in fewer tile chunks (or clusters) than SMs leaves
    // most of the GPU idle: the methods below spread any shape over blocks
    const uint64_t chunks = (T + p.tiles_per_chunk - 1) / p.tiles_per_chunk;
    // (the 16-byte tile kernel sizes its own chunks to the GPU)
    const bool t010 = b == 1 && p.feasible && p.cluster == 1 &&
                      tile010_applies(buf, e, T, a, B);
    const uint64_t bytes = T * a * B * b * (uint64_t)e;
    const uint64_t ctas = chunks * (uint64_t)p.cluster;
    const uint64_t sms = (uint64_t)device_info().sms;
    bool thin = m == Method::Auto && !t010 && bytes >= (1ull << 20) &&
                ctas < sms;
    // (under stream capture the resident form does not run)
    if (m == Method::Auto && !t010 && p.feasible &&
        !planner_beside_other_work() && !getenv("LM_NO_RESIDENT")) {
      const bool held = held_preferred(buf, T, a, B, b, e, p);
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      if ((thin || held) && resident0100_applies(T, a, B, b, e) &&
          cudaStreamIsCapturing(s, &cs) == cudaSuccess &&
          cs == cudaStreamCaptureStatusNone)
        thin = held;
    }
    if (p.feasible && !thin)
      return check_launch(launch_bs0100(s, buf, e, T, (uint32_t)a,
                                        (uint32_t)B, (uint32_t)b, p),
                          "BS launch");
    if (m == Method::BS)
      return fail("BS: tile of %llu bytes exceeds on-chip capacity",
                  (unsigned long long)(a * B * b * e));
  }
  const uint64_t U = b * e;
  // all cycles short (multiplicative order of a modulo a*B - 1 at most
  // kCycleMaxLen): whole-cycle moves, 2 x payload, no flags (lm_cycles.cu)
  if (m == Method::Cycles ||
      (m == Method::Auto && U >= 64 && !getenv("LM_NO_CYCLES"))) {
    const uint32_t L = cycle_order(a, B, kCycleMaxLen);
    if (L && a * B - 1 <= (1ull << 28)) {
      // leader lists are cached per shape, except under stream capture
      // (where the list is computed into per-call scratch)
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      cudaStreamIsCapturing(s, &cs);
      Scratch list;
      return check_launch(
          launch_cycles100(s, buf, e, T, (uint32_t)a, (uint32_t)B,
                           (uint32_t)b, L, list_scratch(list, s),
                           cs == cudaStreamCaptureStatusNone),
          "cycles launch");
    }
    if (m == Method::Cycles)
      return fail("cycles: the cycles of 100(%llu, %llu) are longer than %u",
                  (unsigned long long)a, (unsigned long long)B,
                  (unsigned)kCycleMaxLen);
  }
  // a payload that fits the shared memory of all SMs: one cooperative
  // launch at 2 x payload (not beside other work, where it would wait for
  // every SM to drain, nor under stream capture); where bytes would be written
  // one by one, near that limit, the staged form first, if its scratch can be had
  // (11675 x 2179 38.1 us and 29.3, 20854 x 1455 49.4 and 31.0)
  const bool may_hold = m == Method::Auto && !planner_beside_other_work() &&
                        !getenv("LM_NO_RESIDENT");
  const bool hold_last = may_hold && !getenv("LM_NO_STAGED") &&
                         T * a * B * b * e >= (16ull << 20) &&
                         resident0100_by_elements(buf, T, a, B, b, e);
  auto hold = [&]() {
    uint32_t *status = device_status_word();
    return status ? launch_resident0100(s, buf, e, T, a, B, b, status,
                                        wait_timeout_ns())
                  : cudaErrorNotSupported;
  };
  if (m == Method::Resident || (may_hold && !hold_last)) {
    const cudaError_t err = hold();
    if (err == cudaSuccess) return false;
    if (err != cudaErrorNotSupported) return cuda_fail(err, "resident launch");
    if (m == Method::Resident)
      return fail("resident: 0100(%llu, %llu, %llu, %llu) does not fit shared "
                  "memory (or the stream is being captured)",
                  (unsigned long long)T, (unsigned long long)a,
                  (unsigned long long)B, (unsigned long long)b);
  }
  const bool stash_first =
      m == Method::Auto && stash_preferred(buf, T, a, B, b, e);
  const size_t wave_need =
      m == Method::Auto && U < kStagedMaxUnit && !stash_first &&
              wave_preferred(buf, T, a, B, b, e) && !getenv("LM_NO_WAVE")
          ? wave_scratch(buf, T, a, B, b, e)
          : 0;
  // longer cycles of units of 128 bytes and of 192 and more, cut into segments
  if (m == Method::Auto && T * a * B * U >= kWalkMinBytes &&
      !getenv("LM_NO_WALK") && walk_applies(buf, T, a, B, U)) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cs);
    Scratch sc, list;
    if (walk_preferred(buf, T, a, B, U, cs == cudaStreamCaptureStatusNone,
                       wave_need != 0) &&
        try_scratch(sc, walk_scratch_bytes(buf, T, a, B, U), s)) {
      const cudaError_t err =
          launch_walk100(s, buf, T, a, B, U, sc.p, list_scratch(list, s),
                         cs == cudaStreamCaptureStatusNone);
      if (err != cudaErrorMemoryAllocation) return check_launch(err, "walk launch");
    }
  }
  // a large matrix at 3 x payload: half of its blocks in place, the others
  // through scratch (lm_batch.cu, k_wave)
  if (wave_need) {
    uint32_t *status = device_status_word();
    Scratch sc;
    if (status && try_scratch(sc, wave_need, s)) {
      cudaError_t err = cudaSuccess;
      for (uint64_t t = 0; t < T && err == cudaSuccess; ++t)
        err = launch_wave0100(s, (char *)buf + t * a * B * U, e, a, B, b, sc.p,
                              status, wait_timeout_ns());
      return check_launch(err, "wave launch");
    }
  }
  // any shape through scratch: block transposes out of place, then a copy
  // back (4 x payload, but every access in whole sectors); falls through
  // when the scratch cannot be had
  // (units of 512 bytes and more move as whole lines in cycle following,
  // which needs no scratch and is as fast or faster)
  // (also larger units when the tiles are many and small: cycle following
  // on 18 tiles of 72 x 100 1600-byte units ran 2.3 TB/s, the staged form
  // 2.9 TB/s)
  if (m == Method::Staged ||
      (m == Method::Auto && !stash_first &&
       (U < kStagedMaxUnit || (T > 1 && a * B < 65536)) &&
       T * a * B * b * e >= (1ull << 20) &&
       !getenv("LM_NO_STAGED"))) {
    if (staged0100_applies(T, a, B, b, e)) {
      // the scratch copy sits at the buffer's address modulo 16, so the
      // copy back runs in aligned 16-byte vectors
      Scratch sc;
      if (try_scratch(sc, T * a * B * b * e + 16, s))
        return check_launch(
            launch_staged0100(s, buf, e, T, a, B, b,
                              (char *)sc.p + ((uintptr_t)buf & 15)),
            "staged launch");
      if (m == Method::Staged) return fail("staged: no scratch for this size");
    } else if (m == Method::Staged) {
      return fail("staged: units above 32 KB or too many blocks");
    }
  }
  if (hold_last) {
    const cudaError_t err = hold();
    if (err == cudaSuccess) return false;
    if (err != cudaErrorNotSupported) return cuda_fail(err, "resident launch");
  }
  // the stash plan moves 3 x payload with half the scratch, where the forms
  // above could not have theirs.  Its wavefront spreads rows over all CTAs:
  // with too few rows per SM its steps are too small to keep HBM busy
  const uint64_t stash_min_rows = kStashRowsPerSm * (uint64_t)device_info().sms;
  const bool want_stash =
      m == Method::Stash ||
      (m == Method::Auto && T == 1 && U < 128 && a * B >= (1ull << 20) &&
       a >= stash_min_rows && !getenv("LM_NO_STASH"));
  if (want_stash) {
    // 100 on small units: the 3 x payload streaming plan (lm_stash.cu).
    StashPlan sp = T == 1 ? plan_stash(a, B, (uint32_t)b, e) : StashPlan();
    uint32_t *status = sp.feasible ? device_status_word() : nullptr;
    if (sp.feasible && status) {
      // the stash (about half the payload) may not be available: then the
      // plans below, which need less scratch, take over
      Scratch sc;
      if (try_scratch(sc, stash_scratch_bytes(sp), s))
        return check_launch(launch_stash100(s, buf, e, a, B, (uint32_t)b, sp,
                                            sc.p, status, wait_timeout_ns()),
                            "stash launch");
      if (m == Method::Stash) return fail("stash: no scratch for this size");
    }
    if (m == Method::Stash)
      return fail("stash plan not applicable to 0100(%llu, %llu, %llu, %llu)",
                  (unsigned long long)T, (unsigned long long)a,
                  (unsigned long long)B, (unsigned long long)b);
  }
  if ((m == Method::Auto && U < 128) || m == Method::TwoPass) {
    // Aggregate small super-elements into >=128-byte units first so the
    // cycle-following pass moves whole cache lines.
    uint64_t a2 = split_a(a, B, b, e);
    if (a2) {
      const uint64_t a1 = a / a2;
      if (do_0100(s, buf, e, T * a1, a2, B, b, Method::BS)) return true;
      return do_0100(s, buf, e, T, a1, B, a2 * b, Method::Pttwac);
    }
    uint64_t c = split_B(a, B, b, e);
    if (c) {
      const uint64_t B1 = B / c;
      if (do_0100(s, buf, e, T, a, B1, c * b, Method::Pttwac)) return true;
      return do_0100(s, buf, e, T * B1, a, c, b, Method::BS);
    }
    if (m == Method::TwoPass) return fail("no two-pass split for this shape");
  }
  return run_pttwac_direct(s, buf, e, T, a, B, b);
}

// ---- autotuner ----------------------------------------------------------------
// Shape class = (element bytes, log2 of a, B and b, and whether the op has
// several instances).  For each class met by a tuned call the candidate plans
// are timed once on a scratch buffer of the job's size and the fastest is
// remembered; LM_TUNE_FILE names a text file that is loaded at first use and
// appended to ("e la lB lb multi method" per line).

struct TuneKey {
  int e, la, lB, lb, multi;
  bool operator<(const TuneKey &o) const {
    return std::tie(e, la, lB, lb, multi) <
           std::tie(o.e, o.la, o.lB, o.lb, o.multi);
  }
};

static int ilog2(uint64_t v) {
  int l = 0;
  while (v > 1) {
    v >>= 1;
    ++l;
  }
  return l;
}

static std::mutex g_tune_mu;
static std::map<TuneKey, int> g_tune;
static bool g_tune_loaded = false;

static void tune_load_locked() {
  if (g_tune_loaded) return;
  g_tune_loaded = true;
  const char *f = getenv("LM_TUNE_FILE");
  if (!f) return;
  FILE *fp = fopen(f, "r");
  if (!fp) return;
  // lines "v2 e log2a log2B log2b multi variant"; other lines are skipped
  char line[256];
  while (fgets(line, sizeof(line), fp)) {
    TuneKey k;
    int m;
    if (sscanf(line, "v2 %d %d %d %d %d %d", &k.e, &k.la, &k.lB, &k.lb,
               &k.multi, &m) == 6)
      g_tune[k] = m;
  }
  fclose(fp);
}

static void tune_save_locked(const TuneKey &k, int m) {
  const char *f = getenv("LM_TUNE_FILE");
  if (!f) return;
  FILE *fp = fopen(f, "a");
  if (!fp) return;
  fprintf(fp, "v2 %d %d %d %d %d %d\n", k.e, k.la, k.lB, k.lb, k.multi, m);
  fclose(fp);
}

// Whether a forced method applies to this exact shape (a tuned choice is
// shared by every shape of its class, whose factors may differ).
static bool method_applies(Method m, int e, uint64_t T, uint64_t a,
                           uint64_t B, uint64_t b) {
  switch (m) {
    case Method::Stash:
      return T == 1 && plan_stash(a, B, (uint32_t)b, e).feasible;
    case Method::TwoPass:
      return b * e < 128 && (split_a(a, B, b, e) || split_B(a, B, b, e));
    case Method::BS:
      return plan_bs0100(T, (uint32_t)a, (uint32_t)B, (uint32_t)b, e).feasible;
    case Method::Cycles:
      return cycle_order(a, B, kCycleMaxLen) != 0 && a * B - 1 <= (1ull << 28);
    case Method::Staged:
      return staged0100_applies(T, a, B, b, e);
    case Method::Resident:
      return resident0100_applies(T, a, B, b, e);
    default:
      return true;
  }
}

// The tuned variant (index into kVariants) of a shape class: every variant
// that applies is timed once on a scratch buffer of the job's shape (after
// a warm-up run), the fastest is kept, in memory and in LM_TUNE_FILE.
static int tuned_variant(cudaStream_t s, int e, uint64_t T, uint64_t a,
                         uint64_t B, uint64_t b) {
  const TuneKey key{e, ilog2(a), ilog2(B), ilog2(b), T > 1 ? 1 : 0};
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    tune_load_locked();
    auto it = g_tune.find(key);
    if (it != g_tune.end() && it->second >= 0 && it->second < kNumVariants)
      return it->second;
  }
  const uint64_t bytes = T * a * B * b * (uint64_t)e;
  void *tmp = nullptr;
  int best = 0;
  if (cudaMallocAsync(&tmp, bytes, s) == cudaSuccess) {
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float best_ms = 1e30f;
    for (int i = 0; i < kNumVariants; ++i) {
      const TuneVariant &v = kVariants[i];
      if (v.m == Method::TwoPass && b * e >= 128) continue;
      TuneScope scope(v.p);
      const std::string saved = g_err;
      if (!method_applies(v.m, e, T, a, B, b) ||
          do_0100(s, tmp, e, T, a, B, b, v.m)) {  // warm-up
        g_err = saved;
        continue;
      }
      cudaEventRecord(e0, s);
      do_0100(s, tmp, e, T, a, B, b, v.m);
      cudaEventRecord(e1, s);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best_ms) {
        best_ms = ms;
        best = i;
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFreeAsync(tmp, s);
  }
  std::lock_guard<std::mutex> lock(g_tune_mu);
  g_tune[key] = best;
  tune_save_locked(key, best);
  return best;
}

bool run_0100_planned(cudaStream_t s, void *buf, int e, uint64_t T,
                      uint64_t a, uint64_t B, uint64_t b, int tune) {
  if (valid_e(e)) widen_units(buf, &e, &b);  // the tuned class is the wide one
  if (tune && valid_e(e) && T > 0 && a > 1 && B > 1 && b > 0 &&
      T * a * B * b * (uint64_t)e >= (1ull << 20)) {
    const TuneVariant &v = kVariants[tuned_variant(s, e, T, a, B, b)];
    TuneScope scope(v.p);
    if (method_applies(v.m, e, T, a, B, b))
      return do_0100(s, buf, e, T, a, B, b, v.m);
  }
  return do_0100(s, buf, e, T, a, B, b, Method::Auto);
}

static bool do_010_pttwac(cudaStream_t s, void *buf, int e, uint64_t A,
                          uint64_t a, uint64_t B, int R, int P) {
  if (!valid_e(e)) return fail("element size must be 1, 2, 4 or 8 (got %d)", e);
  if (A == 0 || a <= 1 || B <= 1) return false;
  if (buf == nullptr) return fail("null buffer");
  if (misaligned(buf, e)) return fail("buffer must be aligned to the element size");
  if (R < 1 || R > 32 || (R & (R - 1))) return fail("R must be a power of two in [1, 32]");
  if (P < 0) return fail("P must be >= 0");
  if (a * B < 0xffffffffull && pttwac010_smem_fits((uint32_t)a, (uint32_t)B, R, P))
    return check_launch(launch_pttwac010_smem(s, buf, e, A, (uint32_t)a,
                                              (uint32_t)B, R, P),
                        "010 PTTWAC launch");
  // tile larger than the shared-memory done-bit map: done bits in HBM
  return do_0100(s, buf, e, A, a, B, 1, Method::Pttwac);
}

static bool do_pad(cudaStream_t s, void *buf, int e, int64_t x, int64_t y,
                   int64_t pad, bool padding, uint64_t timeout_ns,
                   int64_t stall_block) {
  if (!valid_e(e)) return fail("element size must be 1, 2, 4 or 8 (got %d)", e);
  if (x < 0 || y < 0 || pad < x) return fail("padding needs 0 <= x <= pad, y >= 0");
  if ((y == 0 || pad == x) && stall_block < 0) return false;
  if (buf == nullptr) return fail("null buffer");
  if (misaligned(buf, e)) return fail("buffer must be aligned to the element size");
  const uint64_t tasks = pad_tasks(buf, e, y, pad);
  if (tasks == 0) return false;  // an empty layout, with a stall asked for
  PadBlock block;
  if ((tasks > 1 || stall_block >= 0) && !block.take(tasks, s)) return true;
  // (a word of host memory, so that no copy follows the kernel)
  HostWord st;
  if (!st.p) return fail("padding: no status word");
  cudaError_t err =
      padding ? launch_padding(s, buf, e, x, y, pad, block.f, st.p,
                               timeout_ns, stall_block, &block.started)
              : launch_unpadding(s, buf, e, x, y, pad, block.f, st.p,
                                 timeout_ns, stall_block, &block.started);
  if (err != cudaSuccess) return cuda_fail(err, padding ? "padding" : "unpadding");
  err = cudaStreamSynchronize(s);
  if (err != cudaSuccess) {
    st.lost = true;  // the kernel may still write it
    return cuda_fail(err, "padding status");
  }
  const uint32_t status = *(volatile uint32_t *)st.p;
  if (status != kStatusOk)
    return fail("%s: an inter-CTA wait timed out (status %u)",
                padding ? "padding" : "unpadding", status);
  block.done = true;
  return false;
}

// Staged full transposition [A*a][B*b] -> [B*b][A*a] (src/cl_marshal.cc:561-776).
static bool do_transpose(cudaStream_t s, void *buf, int e, int64_t A,
                         int64_t a, int64_t B, int64_t b, int R, int stages,
                         int variant010) {
  if (!valid_e(e)) return fail("element size must be 1, 2, 4 or 8 (got %d)", e);
  if (A <= 0 || a <= 0 || B <= 0 || b <= 0) return fail("dimensions must be positive");
  auto t010 = [&](int64_t AA, int64_t aa, int64_t BB) -> bool {
    if (variant010 == 2) return do_010_pttwac(s, buf, e, AA, aa, BB, R, 1);
    Method m = variant010 == 1 ? Method::BS : Method::Auto;
    BsPlan p = plan_bs0100(AA, (uint32_t)aa, (uint32_t)BB, 1, e);
    if (!p.feasible && variant010 == 0)
      return do_010_pttwac(s, buf, e, AA, aa, BB, R, 1);
    return do_0100(s, buf, e, AA, aa, BB, 1, m);
  };
  auto t100 = [&](int64_t AA, int64_t BB, int64_t bb) {
    return do_0100(s, buf, e, 1, AA, BB, bb, Method::Auto);
  };
  auto t0100 = [&](int64_t AA, int64_t aa, int64_t BB, int64_t bb) {
    return do_0100(s, buf, e, AA, aa, BB, bb, Method::Auto);
  };
  // Every stage code yields the same final layout, the full transpose
  // [A*a][B*b] -> [B*b][A*a]: with the 010 variant left to the library it
  // runs as one planned 100, which moves 2-4 x payload where the staged
  // sequences move 2 x payload per stage (7200 x 1800: 2.4-7.7 x faster,
  // int8 and fp16 in one launch held in shared memory).  Forced variants run
  // the reference's stages.
  if (variant010 == 0) return t100(A * a, B * b, 1);
  switch (stages) {
    case 2:  // 010(A, a, B*b) -> 100(A, B*b, a)            (:569-601)
      if (a > 1 && t010(A, a, B * b)) return true;
      return t100(A, B * b, a);
    case 22:  // 100(A*a, B, b) -> 010(B, A*a, b)           (:602-634)
      if (t100(A * a, B, b)) return true;
      return b > 1 ? t010(B, A * a, b) : false;
    case 3:  // 100(A*a,B,b) -> 010(B*A,a,b) -> 0100(B,A,b,a) (:636-677)
      if (t100(A * a, B, b)) return true;
      if (a > 1 && t010(B * A, a, b)) return true;
      return t0100(B, A, b, a);
    case 32:  // 0100(A,a,B,b) -> 010(A*B,a,b) -> 100(A,B*b,a) (:679-720)
      if (t0100(A, a, B, b)) return true;
      if (a > 1 && t010(A * B, a, b)) return true;
      return t100(A, B * b, a);
    case 4:  // 0100 -> 010 -> 100(A,B,b*a) -> 0100(B,A,b,a)  (:722-767)
      if (t0100(A, a, B, b)) return true;
      if (t010(B * A, a, b)) return true;
      if (t100(A, B, b * a)) return true;
      return t0100(B, A, b, a);
    default:  // element-wise fallback 0100(1, A*a, B*b, 1)  (:769-775)
      return t0100(1, A * a, B * b, 1);
  }
}

// ---- full transposition of an arbitrary M x N matrix ------------------------
// The reference's flow for general matrices (test/cl_unittest.cc:396-640):
// "Algorithm 5" picks the super-element sizes a | M' and b | N' as the
// largest divisors within [24, floor(sqrt(MAX_MEM))] of M' = M + pad_h and
// N' = N + pad_w, growing each dimension by one until it has such a divisor
// (the test sorts the divisors and takes the largest in range, :420-463);
// "Algorithm 3" picks the stage code (:515-617): 2 if a >= 6 and a*B*b fits
// MAX_MEM, else 22 if b >= 6 and b*A*a fits, else 3 (a <= b) or 32.  MAX_MEM
// is the reference's 48 KB of local memory in elements (12288 for 4-byte,
// 6144 for 8-byte elements, :22-28; 12288 for narrower ones here).
struct FullPlan {
  int64_t A = 0, a = 0, B = 0, b = 0, pad_h = 0, pad_w = 0;
  int stages = 0;
};

static int64_t largest_divisor_in(int64_t n, int64_t lo, int64_t hi) {
  for (int64_t d = std::min(hi, n); d >= lo; --d)
    if (n % d == 0) return d;
  return 0;
}

static FullPlan plan_full(int64_t M, int64_t N, int e) {
  const int64_t max_mem = 49152 / std::max(e, 4);
  int64_t hi = 1;
  while ((hi + 1) * (hi + 1) <= max_mem) ++hi;
  const int64_t lo = 24;
  FullPlan p;
  int64_t h = M, w = N;
  while ((p.a = largest_divisor_in(h, lo, hi)) == 0) ++h;
  while ((p.b = largest_divisor_in(w, lo, hi)) == 0) ++w;
  p.pad_h = h - M;
  p.pad_w = w - N;
  p.A = h / p.a;
  p.B = w / p.b;
  if (p.a >= 6 && p.a * p.B * p.b <= max_mem) p.stages = 2;
  else if (p.b >= 6 && p.b * p.A * p.a <= max_mem) p.stages = 22;
  else p.stages = p.a <= p.b ? 3 : 32;
  return p;
}

}  // namespace lm

using namespace lm;

// ============================================================================
// C ABI
// ============================================================================

extern "C" {

const char *lm_last_error(void) { return g_err.c_str(); }

const char *lm_version(void) { return "libmarshal_gb300 1.0 (sm_103a)"; }

void lm_marshal_finalize(void) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  cycle_cache_clear();
  stash_cache_clear();
  PadBlock::clear(dev);
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess)
    cudaMemPoolTrimTo(pool, 0);
}

// reference: cl_marshal_finalize (src/cl_marshal.cc:116-119)
void cl_marshal_finalize(void) { lm_marshal_finalize(); }

bool lm_transpose_010_bs(lm_stream_t stream, void *buf, int elem_bytes,
                         int A, int a, int B, unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (A < 0 || a < 0 || B < 0) return fail("dimensions must be >= 0");
  if (do_0100((cudaStream_t)stream, buf, elem_bytes, (uint64_t)A, (uint64_t)a,
              (uint64_t)B, 1, Method::BS))
    return true;
  return t.finish();
}

bool lm_transpose_010_pttwac(lm_stream_t stream, void *buf, int elem_bytes,
                             int A, int a, int B, unsigned long long *et,
                             int R, int P) {
  OpTimer t(et, (cudaStream_t)stream);
  if (A < 0 || a < 0 || B < 0) return fail("dimensions must be >= 0");
  if (do_010_pttwac((cudaStream_t)stream, buf, elem_bytes, (uint64_t)A,
                    (uint64_t)a, (uint64_t)B, R, P))
    return true;
  return t.finish();
}

bool lm_transpose_100(lm_stream_t stream, void *buf, int elem_bytes, int A,
                      int B, int b, unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (A < 0 || B < 0 || b < 0) return fail("dimensions must be >= 0");
  if (do_0100((cudaStream_t)stream, buf, elem_bytes, 1, (uint64_t)A,
              (uint64_t)B, (uint64_t)b, Method::Auto))
    return true;
  return t.finish();
}

bool lm_transpose_0100(lm_stream_t stream, void *buf, int elem_bytes, int A,
                       int a, int B, int b, unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (A < 0 || a < 0 || B < 0 || b < 0) return fail("dimensions must be >= 0");
  if (do_0100((cudaStream_t)stream, buf, elem_bytes, (uint64_t)A, (uint64_t)a,
              (uint64_t)B, (uint64_t)b, Method::Auto))
    return true;
  return t.finish();
}

bool lm_transpose_0100_method(lm_stream_t stream, void *buf, int elem_bytes,
                              int A, int a, int B, int b, int method,
                              unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (A < 0 || a < 0 || B < 0 || b < 0) return fail("dimensions must be >= 0");
  if (method < 0 || method > 7) return fail("method must be 0..7");
  const Method m = method == 1   ? Method::BS
                   : method == 2 ? Method::Pttwac
                   : method == 3 ? Method::Stash
                   : method == 4 ? Method::TwoPass
                   : method == 5 ? Method::Cycles
                   : method == 6 ? Method::Staged
                   : method == 7 ? Method::Resident
                                 : Method::Auto;
  if (do_0100((cudaStream_t)stream, buf, elem_bytes, (uint64_t)A, (uint64_t)a,
              (uint64_t)B, (uint64_t)b, m))
    return true;
  return t.finish();
}

bool lm_transpose(lm_stream_t stream, void *buf, int elem_bytes, int A, int a,
                  int B, int b, int R, int stages, unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (do_transpose((cudaStream_t)stream, buf, elem_bytes, A, a, B, b, R,
                   stages, 0))
    return true;
  return t.finish();
}

bool lm_transpose_ex(lm_stream_t stream, void *buf, int elem_bytes, int A,
                     int a, int B, int b, int R, int stages, int variant010,
                     unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (variant010 < 0 || variant010 > 2) return fail("variant010 must be 0, 1 or 2");
  if (do_transpose((cudaStream_t)stream, buf, elem_bytes, A, a, B, b, R,
                   stages, variant010))
    return true;
  return t.finish();
}

bool lm_full_transpose_plan(int M, int N, int elem_bytes, int *plan7,
                            long long *padded_elems) {
  if (!valid_e(elem_bytes))
    return fail("element size must be 1, 2, 4 or 8 (got %d)", elem_bytes);
  if (M <= 0 || N <= 0) return fail("full transpose: M and N must be > 0");
  const FullPlan p = plan_full(M, N, elem_bytes);
  if (plan7) {
    const int64_t v[7] = {p.A, p.a, p.B, p.b, p.pad_h, p.pad_w, p.stages};
    for (int k = 0; k < 7; ++k) plan7[k] = (int)v[k];
  }
  if (padded_elems)
    *padded_elems = (long long)((M + p.pad_h) * (int64_t)(N + p.pad_w));
  return false;
}

bool lm_full_transpose(lm_stream_t stream, void *buf, int elem_bytes, int M,
                       int N, long long capacity_elems, int variant010,
                       unsigned long long *et) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!valid_e(elem_bytes))
    return fail("element size must be 1, 2, 4 or 8 (got %d)", elem_bytes);
  if (M <= 0 || N <= 0) return fail("full transpose: M and N must be > 0");
  if (variant010 < 0 || variant010 > 2)
    return fail("full transpose: variant010 must be 0, 1 or 2");
  if (buf == nullptr) return fail("null buffer");
  if (misaligned(buf, elem_bytes))
    return fail("buffer must be aligned to the element size");
  const FullPlan p = plan_full(M, N, elem_bytes);
  const int64_t need = variant010 == 0
                           ? (int64_t)M * N
                           : (M + p.pad_h) * (int64_t)(N + p.pad_w);
  if (capacity_elems < need)
    return fail("full transpose: the buffer must hold %lld elements (has %lld)",
                (long long)need, capacity_elems);
  OpTimer t(et, s);
  if (variant010 == 0) {
    // the same permutation without padding: one planned 100
    if (do_0100(s, buf, elem_bytes, 1, M, N, 1, Method::Auto)) return true;
    return t.finish();
  }
  // [M][N] -> [M][N + pad_w] -> transposed [N + pad_w][M + pad_h] (rows past
  // M were never written: their columns become rows past N) -> [N][M]
  if (p.pad_w > 0 && do_pad(s, buf, elem_bytes, N, M, N + p.pad_w, true,
                            2000000000ull, -1))
    return true;
  if (do_transpose(s, buf, elem_bytes, p.A, p.a, p.B, p.b, 1, p.stages,
                   variant010))
    return true;
  if (p.pad_h > 0 && do_pad(s, buf, elem_bytes, M, N, M + p.pad_h, false,
                            2000000000ull, -1))
    return true;
  return t.finish();
}

bool lm_aos_asta_bs(lm_stream_t stream, void *buf, int elem_bytes, int height,
                    int width, int tile_size) {
  if (tile_size <= 0 || height < 0 || width < 0 || height % tile_size)
    return fail("height must be a multiple of tile_size");
  return lm_transpose_010_bs(stream, buf, elem_bytes, height / tile_size,
                             tile_size, width, nullptr);
}

bool lm_aos_asta_pttwac(lm_stream_t stream, void *buf, int elem_bytes,
                        int height, int width, int tile_size, int R, int P) {
  if (tile_size <= 0 || height < 0 || width < 0 || height % tile_size)
    return fail("height must be a multiple of tile_size");
  return lm_transpose_010_pttwac(stream, buf, elem_bytes, height / tile_size,
                                 tile_size, width, nullptr, R, P);
}

bool lm_aos_asta(lm_stream_t stream, void *buf, int elem_bytes, int height,
                 int width, int tile_size, int R) {
  // src/cl_marshal.cc:814-818: BS, and PTTWAC only if BS reported an error.
  return lm_aos_asta_bs(stream, buf, elem_bytes, height, width, tile_size) &&
         lm_aos_asta_pttwac(stream, buf, elem_bytes, height, width, tile_size,
                            R, 1);
}

bool lm_padding(lm_stream_t stream, void *buf, int elem_bytes, int x_size,
                int y_size, int pad_size, unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (do_pad((cudaStream_t)stream, buf, elem_bytes, x_size, y_size, pad_size,
             true, 2000000000ull, -1))
    return true;
  return t.finish();
}

bool lm_unpadding(lm_stream_t stream, void *buf, int elem_bytes, int x_size,
                  int y_size, int pad_size, unsigned long long *et) {
  OpTimer t(et, (cudaStream_t)stream);
  if (do_pad((cudaStream_t)stream, buf, elem_bytes, x_size, y_size, pad_size,
             false, 2000000000ull, -1))
    return true;
  return t.finish();
}

// Failure-detection hook: runs padding (or unpadding) with task `stall_block`
// waiting on a flag that is never set, bounded by timeout_ns.  Must return
// true (error) with a timeout message and leave the context usable.
bool lm_debug_pad_stall(lm_stream_t stream, void *buf, int elem_bytes,
                        int x_size, int y_size, int pad_size, int unpad,
                        long long stall_block, unsigned long long timeout_ns) {
  return do_pad((cudaStream_t)stream, buf, elem_bytes, x_size, y_size,
                pad_size, unpad == 0, timeout_ns, stall_block);
}

// Failure-detection hook: the resident form of 0100(A, a, B, b) with its
// grid barrier waiting for one arrival more than there are CTAs, bounded by
// timeout_ns.  Must return true (error) with a timeout message, leave the
// buffer as it was (no CTA writes) and the context usable.
bool lm_debug_resident_stall(lm_stream_t stream, void *buf, int elem_bytes,
                             int A, int a, int B, int b,
                             unsigned long long timeout_ns) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!valid_e(elem_bytes))
    return fail("element size must be 1, 2, 4 or 8 (got %d)", elem_bytes);
  if (A <= 0 || a <= 1 || B <= 1 || b <= 0) return fail("dimensions must be positive");
  if (buf == nullptr) return fail("null buffer");
  if (misaligned(buf, elem_bytes))
    return fail("buffer must be aligned to the element size");
  uint32_t *status = device_status_word();
  if (!status) return fail("resident: no status word");
  const cudaError_t err =
      launch_resident0100(s, buf, elem_bytes, (uint64_t)A, (uint64_t)a,
                          (uint64_t)B, (uint64_t)b, status, timeout_ns, 1);
  if (err == cudaErrorNotSupported)
    return fail("resident: the shape does not fit shared memory");
  if (err != cudaSuccess) return cuda_fail(err, "resident launch");
  return check_status(s, "resident");
}

// Failure-detection hook: the ordered form of 100(a, B, b) whose blocks wait
// for one block more of each step than there are, bounded by timeout_ns.  Must
// return true (error) with a timeout message and leave the context usable.
bool lm_debug_wave_stall(lm_stream_t stream, void *buf, int elem_bytes, int a,
                         int B, int b, unsigned long long timeout_ns) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!valid_e(elem_bytes))
    return fail("element size must be 1, 2, 4 or 8 (got %d)", elem_bytes);
  if (a <= 1 || B <= 1 || b <= 0) return fail("dimensions must be positive");
  if (buf == nullptr) return fail("null buffer");
  if (misaligned(buf, elem_bytes))
    return fail("buffer must be aligned to the element size");
  const size_t need = wave0100_scratch(buf, (uint64_t)a, (uint64_t)B,
                                       (uint64_t)b, elem_bytes);
  if (need == 0) return fail("wave: the ordered form does not take this shape");
  uint32_t *status = device_status_word();
  if (!status) return fail("wave: no status word");
  Scratch sc;
  if (get_scratch(sc, need, s)) return true;
  if (check_launch(launch_wave0100(s, buf, elem_bytes, (uint64_t)a, (uint64_t)B,
                                   (uint64_t)b, sc.p, status, timeout_ns, 1),
                   "wave launch"))
    return true;
  return check_status(s, "wave");
}

// Waits for `stream` and returns (then clears) the accumulated status of
// waiting kernels on the current device: 0 = ok.
unsigned lm_device_status(lm_stream_t stream) {
  uint32_t *w = device_status_word();
  if (!w) return 0xffffffffu;
  uint32_t v = 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(&v, w, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return 0xffffffffu;
  if (v) cudaMemsetAsync(w, 0, 4, s);
  return v;
}

int lm_tune_entries(void) {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  tune_load_locked();
  return (int)g_tune.size();
}

// Pins (variant >= 0) or reads (variant < 0) the tuned variant of the shape
// class of 0100(T, a, B, b) on elem_bytes elements; returns the class's
// variant afterwards, or -1 when it has none (or the arguments are bad).
int lm_tune_variant(int elem_bytes, long long T, long long a, long long B,
                    long long b, int variant) {
  if (!valid_e(elem_bytes) || T <= 0 || a <= 0 || B <= 0 || b <= 0 ||
      variant >= kNumVariants)
    return -1;
  int e = elem_bytes;
  uint64_t bb = (uint64_t)b;
  widen_units(nullptr, &e, &bb);  // the class is keyed on the wide unit
  const TuneKey key{e, ilog2((uint64_t)a), ilog2((uint64_t)B), ilog2(bb),
                    T > 1 ? 1 : 0};
  std::lock_guard<std::mutex> lock(g_tune_mu);
  tune_load_locked();
  if (variant >= 0) g_tune[key] = variant;
  auto it = g_tune.find(key);
  return it == g_tune.end() ? -1 : it->second;
}

// Planner query used by the Python API's IsFeasible(): 1 when the 0100 tile
// [a][B][b] of elem_bytes elements can be staged on chip (BS), else 0.
int lm_bs_feasible(long long T, int a, int B, int b, int elem_bytes) {
  if (!valid_e(elem_bytes) || T <= 0 || a <= 0 || B <= 0 || b <= 0) return 0;
  return plan_bs0100((uint64_t)T, (uint32_t)a, (uint32_t)B, (uint32_t)b,
                     elem_bytes).feasible ? 1 : 0;
}

// ---- reference CUDA drop-ins (include/marshal.h:26-31) ----------------------
// Same signatures; launch on the legacy default stream like the reference
// (src/marshal.cu:27-80).  `timer` is accepted and left untouched, as the
// reference kernels never write it.

bool gpu_aos_asta_bs_float(float *src, int height, int width, int tile_size,
                           clock_t *timer) {
  (void)timer;
  return lm_aos_asta_bs(nullptr, src, 4, height, width, tile_size);
}

bool gpu_aos_asta_bs_double(double *src, int height, int width, int tile_size,
                            clock_t *timer) {
  (void)timer;
  return lm_aos_asta_bs(nullptr, src, 8, height, width, tile_size);
}

bool gpu_aos_asta_pttwac(float *src, int height, int width, int tile_size,
                         clock_t *timer) {
  (void)timer;
  return lm_aos_asta_pttwac(nullptr, src, 4, height, width, tile_size, 1, 0);
}

bool gpu_soa_asta_pttwac(float *src, int height, int width, int tile_size,
                         clock_t *timer) {
  (void)timer;
  // [w][h/t][t] -> [h/t][w][t] == 100(A=w, B=h/t, b=t)
  if (tile_size <= 0 || height < 0 || width < 0 || height % tile_size)
    return fail("height must be a multiple of tile_size");
  return lm_transpose_100(nullptr, src, 4, width, height / tile_size,
                          tile_size, nullptr);
}

}  // extern "C"
