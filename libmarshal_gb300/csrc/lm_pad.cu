// lm_pad.cu -- in-place row padding and unpadding.
//
// Reference: kernels `padding` / `unpadding` (src/cl/cl_aos_asta.cl:813-938)
// and hosts cl_padding / cl_unpadding (src/cl_marshal.cc:821-956).
//   padding   [y][x]   -> [y][pad], columns x..pad-1 become zero;
//   unpadding [y][pad] -> [y][x],   elements y*x..y*pad-1 become zero.
// The reference orders its work-groups in a chain: every group waits, with an
// unbounded spin, until its predecessor has stored (cl_aos_asta.cl:855-858,
// 914-917), so the stores of the whole buffer are serialised.
//
// GB300 design: a task is a range of the padded layout (16 KB, less where the
// buffer is small), cut at 16-byte addresses, and the compact bytes that
// belong to it, one range too.  A CTA takes a task from a ticket counter
// (padding from the back, unpadding from the front), brings its source into
// shared memory with bulk copies, publishes "loaded" with a release store,
// then waits -- with an acquire load, a backoff and a time limit -- only for
// the tasks whose SOURCES lie where it writes.  Those tasks always have
// smaller tickets, and a task never waits before publishing its own flag, so
// the waits cannot form a cycle and the stores of independent tasks overlap.
// A wait that runs out sets a status word (the host reports an error) and the
// CTA skips its stores; nothing spins forever.
//
// Output is written in the 16-byte vectors of its address: inside a row,
// which is a shift by a constant, four words from five shared ones; across a
// row's end, two of those, masked (a row end handled element by element kept
// one warp lane busy for sixteen bytes while the rest waited: 5,195,000 rows
// of 28 bytes to 32 took 192 us, now 86; 519,500 of 280 to 288 178, now 82).
// Bound by DRAM and the rate at which tasks start: 8192 x 12289 floats to
// 12320 columns (806 MB moved) 173 us = 4.7 TB/s (313 us with tasks of single
// elements in registers), 7382 x 30496 bytes back to 30484 columns 103 us
// (596).
#include <algorithm>

#include "lm_core.cuh"
#include "lm_internal.h"

namespace lm {

constexpr int kPadThreads = 128;
constexpr uint64_t kPadTask = 16 * 1024;
constexpr uint64_t kPadMinTask = 2 * 1024;

struct PadArgs {
  char *buf;
  uint64_t x, pad;   // row bytes, compact and padded
  uint64_t yx, O;    // bytes of all rows, compact and padded
  uint64_t ntasks;
  uint32_t P;        // buf modulo 16; task k: padded bytes k*task - P and on
  uint32_t task;     // bytes of a task, a multiple of 16
  uint32_t rows;     // unpadding: 1 = copy the rows of a task one by one
  uint32_t *ticket;  // scratch[0]; counts up from ticket0
  uint32_t *loaded;  // scratch[1 .. ntasks]: `epoch` once loaded
  uint32_t *never;   // the last word, never set
  uint32_t ticket0, epoch;
  uint32_t *status;  // host memory, read when the stream has finished
  uint64_t timeout_ns;
  int64_t stall_block;
  FastDiv div_x, div_pad;  // where rows are no longer than a task
};

__device__ __forceinline__ bool wait_flag(const uint32_t *f, uint32_t epoch,
                                          uint64_t t0, uint64_t timeout_ns) {
  unsigned ns = 32;
  while (ld_acquire_gpu(f) != epoch) {
    if (global_timer_ns() - t0 > timeout_ns) return false;
    __nanosleep(ns);
    if (ns < 4096) ns <<= 1;
  }
  return true;
}

// Bytes before padded byte o of the rows' own, and their number up to it.
__device__ __forceinline__ uint64_t pad_compact(uint64_t o, const PadArgs &g) {
  const uint64_t r = o / g.pad, c = o - r * g.pad;
  return r * g.x + min64(c, g.x);
}

// Rows that byte t lies past the row at whose start t counts from zero (t <
// row + task bytes).
__device__ __forceinline__ uint32_t pad_rows(uint64_t t, uint64_t row,
                                             uint32_t task,
                                             const FastDiv &div) {
  return row > task ? (t >= row ? 1u : 0u) : fdiv((uint32_t)t, div);
}

// 16 bytes of shared memory at any byte offset.
__device__ __forceinline__ uint4 pad_read16(const unsigned char *p,
                                            uint32_t off) {
  const uint32_t *q = reinterpret_cast<const uint32_t *>(p + (off & ~3u));
  const uint32_t a = q[0], b = q[1], c = q[2], d = q[3], e = q[4];
  const uint32_t s = off * 8;
  return make_uint4(__funnelshift_r(a, b, s), __funnelshift_r(b, c, s),
                    __funnelshift_r(c, d, s), __funnelshift_r(d, e, s));
}

// A task: padded bytes [lo, hi), compact bytes [c0, c1), the rows of lo and
// c0; its source bytes are [s0, s1), byte s at stage + s - base.
struct PadTask {
  uint64_t k, lo, hi, c0, c1, lo_row, c0_row, s0, s1;
  int64_t base;
};

template <bool PAD>
__device__ __forceinline__ void pad_claim(const PadArgs &g, PadTask &t) {
  // (a single task has no one to wait for and no flags)
  const uint64_t n = g.ticket ? atomicAdd(g.ticket, 1u) - g.ticket0 : 0;
  const uint64_t k = t.k = PAD ? g.ntasks - 1 - n : n;
  t.lo = k * g.task > g.P ? k * g.task - g.P : 0;
  t.hi = min64(g.O, (k + 1) * g.task - g.P);
  t.lo_row = t.lo / g.pad;
  t.c0 = t.lo_row * g.x + min64(t.lo - t.lo_row * g.pad, g.x);
  t.c1 = pad_compact(t.hi, g);
  t.c0_row = t.lo_row;  // (c0 starts the next row where lo is in padding)
  if (t.lo - t.lo_row * g.pad >= g.x) t.c0_row += 1;
  t.s0 = PAD ? t.c0 : t.lo;
  t.s1 = PAD ? t.c1 : t.hi;
  t.base = (int64_t)((t.s0 + g.P) & ~(uint64_t)15) - g.P;
}

// One warp: the task's source into `stage`, completion on `bar`.
template <bool PAD>
__device__ __forceinline__ void pad_load(const PadArgs &g, const PadTask &t,
                                         unsigned char *stage, uint64_t *bar) {
  const uint32_t lane = threadIdx.x & 31;
  if (PAD || !g.rows) {
    if (lane) return;
    const uint32_t bytes =
        t.s1 > t.s0 ? (uint32_t)((t.s1 - t.base + 15) & ~(uint64_t)15) : 0u;
    mbar_arrive_expect_tx(bar, bytes);
    if (bytes) {
      fence_proxy_async_smem();
      bulk_g2s(stage, g.buf + t.base, bytes, bar);
    }
    return;
  }
  // one copy for each row's own bytes (long rows, much padding)
  const uint64_t r1 = (t.hi - 1) / g.pad;
  uint32_t bytes = 0;
  for (int pass = 0; pass < 2; ++pass) {
    for (uint64_t r = t.lo_row + lane; r <= r1; r += 32) {
      const uint64_t a = max(t.lo, r * g.pad), b = min64(t.hi, r * g.pad + g.x);
      if (a >= b) continue;
      const uint64_t a0 = (a + g.P) & ~(uint64_t)15;
      const uint64_t b0 = (b + g.P + 15) & ~(uint64_t)15;
      if (pass == 0)
        bytes += (uint32_t)(b0 - a0);
      else
        bulk_g2s(stage + (a0 - g.P - t.base), g.buf + a0 - g.P,
                 (uint32_t)(b0 - a0), bar);
    }
    if (pass == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(kFull, bytes, o);
      if (lane == 0) mbar_arrive_expect_tx(bar, bytes);
      __syncwarp();
      fence_proxy_async_smem();
    }
  }
}

// Mask of the first n of 16 bytes (n <= 16).
__device__ __forceinline__ uint4 pad_low(uint32_t n) {
  auto word = [n](uint32_t w) {
    const uint32_t t = n <= 4 * w ? 0u : min(n - 4 * w, 4u);
    return (uint32_t)((1ull << (8 * t)) - 1);
  };
  return make_uint4(word(0), word(1), word(2), word(3));
}

// One task per CTA.  (Persistent CTAs that load their next task's source
// meanwhile publish it only after the current task, so the waits of all
// others grow into a convoy: 420 us where this form takes 175.)
template <int E, bool PAD>
__global__ void __launch_bounds__(kPadThreads) k_pad(PadArgs g) {
  using T = typename Elem<E>::T;
  // (reads of masked vectors reach 16 bytes to either side of the source)
  extern __shared__ __align__(128) unsigned char stage[];
  unsigned char *smem = stage + 16;
  __shared__ __align__(8) uint64_t bar;
  __shared__ PadTask tk;
  __shared__ int s_ok;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    s_ok = 1;
    pad_claim<PAD>(g, tk);
  }
  __syncthreads();
  if (tid < 32) pad_load<PAD>(g, tk, smem, &bar);
  const uint64_t k = tk.k;
  const uint64_t lo = tk.lo, hi = tk.hi, c0 = tk.c0, c1 = tk.c1;
  const int64_t base = tk.base;
  const uint64_t t0 = global_timer_ns();
  while (!mbar_try_wait(&bar, 0))
    if (global_timer_ns() - t0 > g.timeout_ns) {
      s_ok = 0;
      break;
    }
  __syncthreads();
  if (tid == 0 && s_ok && g.ticket) st_release_gpu(g.loaded + k, g.epoch);

  // ---- wait for the tasks whose sources lie where this one writes
  if (tid < 32) {
    int64_t k0 = 0, k1 = -1;
    if (PAD) {
      const uint64_t e1 = min64(hi, g.yx);
      if (lo < e1) {
        const uint64_t o0 = (lo / g.x) * g.pad + lo % g.x;
        const uint64_t o1 = ((e1 - 1) / g.x) * g.pad + (e1 - 1) % g.x;
        k0 = (int64_t)((o0 + g.P) / g.task);
        k1 = (int64_t)((o1 + g.P) / g.task);
      }
    } else if (c0 < c1) {
      // compact bytes [c0, c1) hold the padded bytes of the same numbers
      k0 = (int64_t)((c0 + g.P) / g.task);
      k1 = (int64_t)((c1 - 1 + g.P) / g.task);
    }
    const uint64_t t1 = global_timer_ns();
    bool good = true;
    if ((int64_t)k == g.stall_block) good = wait_flag(g.never, g.epoch, t1, g.timeout_ns);
    for (int64_t w = k0 + tid; good && w <= k1; w += 32)
      if (w != (int64_t)k) good = wait_flag(g.loaded + w, g.epoch, t1, g.timeout_ns);
    if (!good) s_ok = 0;
  }
  __syncthreads();
  if (!s_ok) {
    if (tid == 0) {
      *reinterpret_cast<volatile uint32_t *>(g.status) = kStatusWaitTimeout;
      // nothing may still be landing in shared memory when the CTA exits
      const uint64_t t2 = global_timer_ns();
      while (!mbar_try_wait(&bar, 0) && global_timer_ns() - t2 < g.timeout_ns) {
      }
    }
    return;
  }

  // ---- write: padded bytes [lo, hi), or compact ones [c0, c1) and zeros
  const uint64_t d0 = PAD ? lo : c0, d1 = PAD ? hi : c1;
  const uint64_t row = PAD ? g.pad : g.x;    // of the written layout
  const uint64_t from = PAD ? g.x : g.pad;   // of the source
  const uint64_t row0 = PAD ? tk.lo_row : tk.c0_row;
  const FastDiv &div = PAD ? g.div_pad : g.div_x;
  const uint64_t in_row = d0 - row0 * row;   // d0's place in its row
  // source byte of column c, row0 + r: smem[r*from + c + at0]
  const int64_t at0 = (int64_t)(row0 * from) - base;
  const int64_t v0 = (int64_t)((d0 + g.P) & ~(uint64_t)15) - g.P;
  const uint32_t nv = d1 > d0 ? (uint32_t)((d1 - v0 + 15) / 16) : 0u;
  for (uint32_t v = tid; v < nv; v += kPadThreads) {
    const int64_t o = v0 + (int64_t)v * 16;
    const bool whole = o >= (int64_t)d0 && o + 16 <= (int64_t)d1;
    const uint64_t ob = whole ? (uint64_t)o : max((uint64_t)max(o, (int64_t)0), d0);
    const uint64_t t = ob - d0 + in_row;
    uint32_t r = pad_rows(t, row, g.task, div);
    uint64_t c = t - r * row;
    if constexpr (E == 8) {
      // two elements, each of a row or of its padding: a vector across a row's
      // end costs no more than another (a row end in most warps' steps, by the
      // masks below: rows of 4 doubles to 5, 315 MB, 208 us, of 12 to 14 at 8
      // past a vector 208, back 188)
      if (whole) {
        uint2 h[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          h[k] = make_uint2(0, 0);
          if (!PAD || c < g.x)
            h[k] = *reinterpret_cast<const uint2 *>(
                smem + (at0 + (int64_t)(r * from + c)));
          c += 8;
          if (c >= row) {
            c = 0;
            ++r;
          }
        }
        *reinterpret_cast<uint4 *>(g.buf + o) =
            make_uint4(h[0].x, h[0].y, h[1].x, h[1].y);
        continue;
      }
    }
    if (whole && c + 16 <= g.x) {
      *reinterpret_cast<uint4 *>(g.buf + o) =
          pad_read16(smem, (uint32_t)(at0 + (int64_t)(r * from + c)));
      continue;
    }
    if (PAD && whole && c >= g.x && c + 16 <= g.pad) {
      *reinterpret_cast<uint4 *>(g.buf + o) = make_uint4(0, 0, 0, 0);
      continue;
    }
    if (whole && row >= 16) {
      // across a row's end: the rest of row r, and the start of the next
      uint4 a = make_uint4(0, 0, 0, 0);
      const uint64_t next = row - c;  // bytes up to the next row's place
      if (c < g.x) {
        const uint4 m = pad_low((uint32_t)min64(16, g.x - c));
        a = pad_read16(smem, (uint32_t)(at0 + (int64_t)(r * from + c)));
        a = make_uint4(a.x & m.x, a.y & m.y, a.z & m.z, a.w & m.w);
      }
      if (next < 16) {
        const uint32_t n = (uint32_t)next;
        const uint4 lo4 = pad_low(n),
                    hi4 = pad_low((uint32_t)min64(16, next + g.x));
        const uint4 b = pad_read16(
            stage, (uint32_t)(at0 + 16 + (int64_t)((r + 1) * from) - n));
        a.x |= b.x & hi4.x & ~lo4.x;
        a.y |= b.y & hi4.y & ~lo4.y;
        a.z |= b.z & hi4.z & ~lo4.z;
        a.w |= b.w & hi4.w & ~lo4.w;
      }
      *reinterpret_cast<uint4 *>(g.buf + o) = a;
      continue;
    }
    // rows of a few bytes, or an end of the task: element by element
    T e[16 / E];
    const uint64_t oe = min64((uint64_t)(o + 16), d1);
    uint32_t n = (uint32_t)((oe - ob) / E);
#pragma unroll
    for (uint32_t i = 0; i < 16 / E; ++i) {
      e[i] = T(0);
      if (i < n) {
        if (!PAD || c < g.x)
          e[i] = *reinterpret_cast<const T *>(
              smem + (at0 + (int64_t)(r * from + c)));
        c += E;
        if (c >= row) {
          c = 0;
          ++r;
        }
      }
    }
    if (whole) {
      *reinterpret_cast<uint4 *>(g.buf + o) = pack16<E>(e);
    } else {
#pragma unroll
      for (uint32_t i = 0; i < 16 / E; ++i)
        if (i < n) *reinterpret_cast<T *>(g.buf + ob + i * E) = e[i];
    }
  }
  if (!PAD && hi > g.yx) {
    // zeros behind the rows, where this task's own source was: elements up
    // to a vector boundary, vectors (hi is one, or the buffer's end)
    const uint64_t z0 = max(lo, g.yx);
    const uint64_t za = min64(((z0 + g.P + 15) & ~(uint64_t)15) - g.P, hi);
    const uint64_t zb = za + (hi - za) / 16 * 16;
    const uint32_t nh = (uint32_t)(za - z0) / E, nt = (uint32_t)(hi - zb) / E;
    if (tid < nh) *reinterpret_cast<T *>(g.buf + z0 + tid * E) = T(0);
    if (tid < nt) *reinterpret_cast<T *>(g.buf + zb + tid * E) = T(0);
    for (uint64_t z = za + tid * 16; z < zb; z += kPadThreads * 16)
      *reinterpret_cast<uint4 *>(g.buf + z) = make_uint4(0, 0, 0, 0);
  }
}

// Bytes of a task: at least two tasks per SM where the buffer has them.
static uint32_t pad_task_bytes(uint64_t bytes) {
  const uint64_t per = bytes / (2 * (uint64_t)device_info().sms);
  return (uint32_t)(std::max(kPadMinTask, std::min(kPadTask, per)) / 128 * 128);
}

uint64_t pad_tasks(const void *buf, int e, uint64_t y, uint64_t pad) {
  const uint64_t O = y * pad * e, task = pad_task_bytes(O);
  if (O == 0) return 0;
  return (O + ((uintptr_t)buf & 15) + task - 1) / task;
}

template <bool PAD>
static cudaError_t run_pad(cudaStream_t s, void *buf, int e, uint64_t x,
                           uint64_t y, uint64_t pad, const PadFlags &flags,
                           uint32_t *status, uint64_t timeout_ns,
                           int64_t stall_block, uint64_t *started) {
  if (pad < x) return cudaErrorInvalidValue;
  PadArgs g;
  g.buf = reinterpret_cast<char *>(buf);
  g.x = x * e;
  g.pad = pad * e;
  g.yx = y * g.x;
  g.O = y * g.pad;
  if (g.O == 0 || (pad == x && stall_block < 0)) return cudaSuccess;
  g.P = (uint32_t)((uintptr_t)buf & 15);
  g.task = pad_task_bytes(g.O);
  g.ntasks = (g.O + g.P + g.task - 1) / g.task;
  if (g.ntasks >= 0x7fffffffull) return cudaErrorInvalidValue;
  // rows of 1 KB and more with an eighth or more of padding
  g.rows = g.x >= 1024 && (g.pad - g.x) * 8 >= g.pad ? 1u : 0u;
  if (flags.p ? flags.words < g.ntasks + 2 : g.ntasks > 1)
    return cudaErrorInvalidValue;
  g.ticket = flags.p;
  g.loaded = flags.p + 1;
  g.never = flags.p + flags.words - 1;
  g.ticket0 = flags.ticket;
  g.epoch = flags.epoch;
  g.status = status;
  g.timeout_ns = timeout_ns;
  g.stall_block = stall_block;
  g.div_x = make_fastdiv((uint32_t)std::min<uint64_t>(g.x ? g.x : 1, 1u << 30));
  g.div_pad = make_fastdiv((uint32_t)std::min<uint64_t>(g.pad, 1u << 30));
  // the task's bytes, the rest of its first and last 16, and what masked
  // vectors read around them
  const size_t smem = g.task + 128;
  const unsigned grid = (unsigned)g.ntasks;
  ProfScope ps(s, PAD ? "padding" : "unpadding");
  switch (e) {
    case 1: k_pad<1, PAD><<<grid, kPadThreads, smem, s>>>(g); break;
    case 2: k_pad<2, PAD><<<grid, kPadThreads, smem, s>>>(g); break;
    case 4: k_pad<4, PAD><<<grid, kPadThreads, smem, s>>>(g); break;
    case 8: k_pad<8, PAD><<<grid, kPadThreads, smem, s>>>(g); break;
    default: return cudaErrorInvalidValue;
  }
  const cudaError_t err = cudaGetLastError();
  if (err == cudaSuccess) *started = g.ntasks;
  return err;
}

cudaError_t launch_padding(cudaStream_t s, void *buf, int e, uint64_t x,
                           uint64_t y, uint64_t pad, const PadFlags &flags,
                           uint32_t *status, uint64_t timeout_ns,
                           int64_t stall_block, uint64_t *started) {
  return run_pad<true>(s, buf, e, x, y, pad, flags, status, timeout_ns,
                       stall_block, started);
}

cudaError_t launch_unpadding(cudaStream_t s, void *buf, int e, uint64_t x,
                             uint64_t y, uint64_t pad, const PadFlags &flags,
                             uint32_t *status, uint64_t timeout_ns,
                             int64_t stall_block, uint64_t *started) {
  return run_pad<false>(s, buf, e, x, y, pad, flags, status, timeout_ns,
                        stall_block, started);
}

}  // namespace lm
