// lm_walk.cu -- 100/0100 of units of whole lines by walking segments of the
// permutation's cycles: 2 x payload, no done bits, no claims.
//
// The reference moves units along the cycles of 100(A, B) one dependent step
// at a time, with a done flag per unit and an atomic claim per step
// (_transpose_100, src/cl/cl_aos_asta.cl:352-717; Transposition::Next,
// include/plan.hpp:54-56).  Here the cycles are cut into segments beforehand:
//  * every block of m consecutive positions holds one START, at an offset
//    hashed from the block's index, so whether a position is a start (and
//    which) is arithmetic; k_walk_save copies the units at the starts to
//    scratch (1/m of the payload);
//  * k_walk gives each start to one group of lanes (a lane per vector of the
//    unit).  The group fills the hole at its start from the position whose
//    unit belongs there, which is the next hole, and so on backwards along
//    the cycle, until the unit it needs is that of a start: that one it takes
//    from scratch.  Every position between two starts is read and then
//    written by one lane of one group, so the order needs nothing but the
//    lane's own program order, and the positions ahead are known by
//    arithmetic: K loads are in flight per lane;
//  * cycles that hold no start (short ones) are found by k_walk_leaders, once
//    per shape: the smallest position of each, whose unit its group keeps in
//    registers meanwhile.
//
// Bound by DRAM at random lines: 100(24, 187500) of 128-byte units (576 MB)
// 222 us = 5.2 TB/s (the staged form, 4 x payload: 368 us = 3.1), 100(24,
// 20001) of 1 KB units 179 us = 5.5 TB/s (cycle following with done bits: 262
// us).  m = 8: the starts cost a quarter of the payload more (read and written
// once more; the read back stands for that of their places), but segments of 8 positions on average (their lengths are
// geometric, the longest about m * ln(segments)) leave a short tail: m = 4 /
// 8 / 16 / 32 / 64 took 281 / 222 / 228 / 270 / 520 us on the first shape.
// K = 8 loads in flight at 3 CTAs per SM (80 registers, no spills); K = 4, 6
// and 12 or 4 to 8 CTAs were 3-50 % slower.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "lm_core.cuh"
#include "lm_internal.h"

namespace lm {

namespace {

constexpr int kWalkThreads = 256;
constexpr uint32_t kWalkLogBlock = 3;

struct WalkMap {
  uint32_t N;      // positions of one tile: a*B
  uint32_t a, B;
  uint32_t lm;     // log2 m
  uint32_t nS;     // blocks of m positions (a start each, the last maybe none)
  FastDiv div_a;
};

// The position whose unit belongs at q: q = j*a + i holds input (i, j).
__device__ __forceinline__ uint32_t walk_src(uint32_t q, const WalkMap &m) {
  const uint32_t j = fdiv(q, m.div_a);
  return (q - j * m.a) * m.B + j;
}

__device__ __forceinline__ uint32_t walk_start(uint32_t k, uint32_t lm) {
  return (k << lm) + ((k * 0x9E3779B1u) >> (32 - lm));
}

__device__ __forceinline__ bool walk_is_start(uint32_t p, uint32_t lm) {
  return walk_start(p >> lm, lm) == p;
}

// Smallest positions of the cycles (of two positions and more) that hold no
// start.  From every position: back along its cycle until a start or a
// smaller position shows that it is none.
__global__ void __launch_bounds__(kWalkThreads)
    k_walk_leaders(WalkMap m, uint32_t *list, uint32_t *count) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * kWalkThreads;
  const uint64_t iters = (m.N + stride - 1) / stride;  // the same for all (ballot)
  uint64_t x = (uint64_t)blockIdx.x * kWalkThreads + threadIdx.x;
  for (uint64_t it = 0; it < iters; ++it, x += stride) {
    bool lead = false;
    if (x < m.N && !walk_is_start((uint32_t)x, m.lm)) {
      const uint32_t q = (uint32_t)x;
      uint32_t p = walk_src(q, m);
      lead = p != q;
      while (lead && p != q) {
        lead = p > q && !walk_is_start(p, m.lm);
        p = walk_src(p, m);
      }
    }
    const unsigned mask = __ballot_sync(kFull, lead);
    if (mask) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(count, (uint32_t)__popc(mask));
      base = __shfl_sync(kFull, base, 0);
      if (lead) list[base + __popc(mask & ((1u << lane) - 1))] = (uint32_t)x;
    }
  }
}

// A unit is cut into `slices` of `lanes` V-byte vectors (the last may have
// fewer); an instance is one slice of all units of one tile.
struct WalkArgs {
  char *base;
  char *scratch;        // slot (instance, start): lanes * V bytes
  uint64_t tile_bytes;
  uint32_t U;           // unit bytes
  uint32_t nvec;        // vectors of a unit: U / V
  uint32_t lanes, slices;
  uint32_t inst;        // tiles * slices
  WalkMap m;
  FastDiv div_nS, div_slices;
  const uint32_t *list, *count;  // cycles without a start
};

template <int V>
__global__ void __launch_bounds__(kWalkThreads) k_walk_save(WalkArgs g) {
  using T = typename Vec<V>::T;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t per = 32 / g.lanes;  // groups of a warp
  const uint32_t grp = lane / g.lanes, gl = lane - grp * g.lanes;
  if (grp >= per) return;
  const uint32_t w0 =
      ((blockIdx.x * kWalkThreads + threadIdx.x) >> 5) * per + grp;
  const uint32_t nw = gridDim.x * (kWalkThreads / 32) * per;
  const uint64_t n = (uint64_t)g.inst * g.m.nS;
  constexpr int K = 4;
  for (uint64_t w = w0; w < n; w += (uint64_t)nw * K) {
    T v[K] = {};
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const uint64_t x = w + (uint64_t)u * nw;
      if (x >= n) continue;
      const uint32_t in = fdiv((uint32_t)x, g.div_nS);
      const uint32_t p = walk_start((uint32_t)x - in * g.m.nS, g.m.lm);
      const uint32_t t = fdiv(in, g.div_slices);
      const uint32_t vec = (in - t * g.slices) * g.lanes + gl;
      if (p < g.m.N && vec < g.nvec)
        v[u] = __ldcs(reinterpret_cast<const T *>(
            g.base + t * g.tile_bytes + (uint64_t)p * g.U + vec * V));
    }
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const uint64_t x = w + (uint64_t)u * nw;
      if (x < n)  // (an unused slot where the unit has no such vector)
        *reinterpret_cast<T *>(g.scratch + (x * g.lanes + gl) * V) = v[u];
    }
  }
}

template <int V, int K>
__global__ void __launch_bounds__(kWalkThreads, 3) k_walk(WalkArgs g) {
  using T = typename Vec<V>::T;
  __shared__ uint32_t s_next;
  __shared__ FastDiv s_div;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t per = 32 / g.lanes;
  const uint32_t grp = lane / g.lanes, gl = lane - grp * g.lanes;
  // segments of an instance: one per block of m positions, then one per
  // cycle without a start
  const uint32_t nseg = g.m.nS + *g.count;
  if (threadIdx.x == 0) {
    s_next = 0;
    s_div = make_fastdiv(nseg);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the saved starts
  __syncthreads();
  const FastDiv div_seg = s_div;
  // this CTA's segments: blockIdx.x + gridDim.x * 0, 1, ..., mine - 1, taken
  // by its groups as they come free
  const uint32_t total = nseg * g.inst;
  const uint32_t mine =
      blockIdx.x < total ? (total - blockIdx.x - 1) / gridDim.x + 1 : 0;
  bool more = grp < per, active = false, mover = false;
  uint32_t q = 0;                  // the hole
  uint32_t own = 0xffffffffu;      // a cycle without a start: its leader
  T held = T();                    // and the leader's unit
  char *tb = nullptr;              // this lane's vector of position 0
  const char *sb = nullptr;        // this lane's vector of slot 0
  for (;;) {
    // a free group takes the next segment
    uint32_t n = 0;
    if (!active && more && gl == 0) n = atomicAdd(&s_next, 1u);
    n = __shfl_sync(kFull, n, (grp * g.lanes) & 31);
    if (!active && more) {
      if (n >= mine) {
        more = false;
      } else {
        const uint32_t w = blockIdx.x + gridDim.x * n;
        const uint32_t in = fdiv(w, div_seg);
        const uint32_t k = w - in * nseg;
        const uint32_t t = fdiv(in, g.div_slices);
        const uint32_t vec = (in - t * g.slices) * g.lanes + gl;
        mover = vec < g.nvec;
        tb = g.base + t * g.tile_bytes + vec * V;
        sb = g.scratch + ((uint64_t)in * g.m.nS * g.lanes + gl) * V;
        own = 0xffffffffu;
        if (k < g.m.nS) {
          q = walk_start(k, g.m.lm);
          active = q < g.m.N;
        } else {
          q = own = g.list[k - g.m.nS];
          active = true;
          if (mover) held = *reinterpret_cast<const T *>(tb + (uint64_t)q * g.U);
        }
      }
    }
    if (!__any_sync(kFull, active || more)) break;
    // the next K positions back along the cycle, up to the segment's end
    uint32_t p[K];
    uint32_t cnt = 0;
    bool end = !active;
    uint32_t cur = q;
#pragma unroll
    for (int u = 0; u < K; ++u) {
      p[u] = cur;
      if (!end) {
        cur = walk_src(cur, g.m);
        p[u] = cur;
        cnt = u + 1;
        end = walk_is_start(cur, g.m.lm) || cur == own;
      }
    }
    // (the leader's unit is chosen at its store: chosen here, the register
    // of each load would be written twice and each load waited for)
    const bool back = end && own != 0xffffffffu;  // ends at its own leader
    T v[K];
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const bool last = end && u + 1 == cnt;
      const char *from = last ? sb + (uint64_t)(p[u] >> g.m.lm) * (g.lanes * V)
                              : tb + (uint64_t)p[u] * g.U;
      if (u < cnt && mover && !(last && back))
        v[u] = __ldcs(reinterpret_cast<const T *>(from));
    }
#pragma unroll
    for (int u = 0; u < K; ++u)
      if (u < cnt && mover)
        __stcs(reinterpret_cast<T *>(tb + (uint64_t)(u ? p[u - 1] : q) * g.U),
               back && u + 1 == cnt ? held : v[u]);
    q = cur;
    if (end) active = false;
  }
}

template <int V>
cudaError_t run_walk(cudaStream_t s, const WalkArgs &g) {
  const DeviceInfo &di = device_info();
  const uint64_t n = (uint64_t)g.inst * g.m.nS;
  const uint32_t per = kWalkThreads / 32 * (32 / g.lanes);
  {
    ProfScope ps(s, "walk_save");
    const uint64_t want = (n + per * 4 - 1) / (per * 4);
    k_walk_save<V><<<(unsigned)std::min<uint64_t>(want, (uint64_t)di.sms * 8),
                     kWalkThreads, 0, s>>>(g);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
  }
  ProfScope ps(s, "walk");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<uint64_t>((n + per - 1) / per,
                                                  (uint64_t)di.sms * 3));
  cfg.blockDim = dim3(kWalkThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_walk<V, 8>, g);
}

// Geometry of a walk; false where it does not apply.
bool walk_args(const void *buf, uint64_t T, uint64_t a, uint64_t B, uint64_t U,
               WalkArgs *g) {
  // units of whole 16-byte vectors.  Moved one at a time, smaller units or
  // ones that straddle lines fetch more than they hold: 64 bytes 2.4-3.1
  // TB/s, 80 1.8, 112 2.2, 144 2.5, 208 3.2, 128 and 192 and more in whole
  // half lines 4.4-5.6, against 2.9-3.1 of the staged form (walk_by_lines has
  // the line against the ordered one)
  if (T == 0 || a < 2 || B < 2 || (U != 128 && U < 192) || U % 16 ||
      ((uintptr_t)buf & 15))
    return false;
  if (a * B >= 0xffffffffull || U > (1u << 30)) return false;
  g->nvec = (uint32_t)(U / 16);
  g->slices = (g->nvec + 31) / 32;
  g->lanes = (g->nvec + g->slices - 1) / g->slices;
  g->U = (uint32_t)U;
  g->tile_bytes = a * B * U;
  if (T * g->slices > 0xffffffull) return false;
  g->inst = (uint32_t)(T * g->slices);
  g->m.N = (uint32_t)(a * B);
  g->m.a = (uint32_t)a;
  g->m.B = (uint32_t)B;
  g->m.lm = kWalkLogBlock;
  g->m.nS = (uint32_t)((a * B + (1u << kWalkLogBlock) - 1) >> kWalkLogBlock);
  // segments (cycles without a start are at most half the positions) are
  // numbered in 32 bits
  if ((uint64_t)g->inst * (g->m.nS + (uint64_t)g->m.N / 2 + 1) >= 0xffffffffull)
    return false;
  g->m.div_a = make_fastdiv(g->m.a);
  g->div_nS = make_fastdiv(g->m.nS);
  g->div_slices = make_fastdiv(g->slices);
  return true;
}

}  // namespace

bool walk_applies(const void *buf, uint64_t T, uint64_t a, uint64_t B,
                  uint64_t U) {
  WalkArgs g;
  return walk_args(buf, T, a, B, U, &g);
}

size_t walk_scratch_bytes(const void *buf, uint64_t T, uint64_t a, uint64_t B,
                          uint64_t U) {
  WalkArgs g;
  if (!walk_args(buf, T, a, B, U, &g)) return 0;
  return (size_t)g.inst * g.m.nS * g.lanes * 16;
}

// A group of lanes reads its slice of a unit at a random place, so what it
// costs is the lines that the slice touches and the sectors that it touches in
// part, and what it hides is the bytes that a warp has in flight.  At 300 MB
// (walk and ordered form, us): slices of 128 bytes on lines 125 and 155, 64 past
// them 199 and 155; of 192, 146 and 160 on halves of lines, 169 and 161 on
// sectors; of 256 off lines 155 and 154; of 320 (and 640, which are two of
// them) 150 and 159 on sectors, 162 and 161 off them; of 352 off them 157 and
// 160; 17 lanes (272 bytes, 528) 172 and 159.  Up to about 100 MB, in L2, the
// walk is the faster one anyhow.
bool walk_by_lines(const void *buf, uint64_t U) {
  WalkArgs g;
  if (!walk_args(buf, 1, 2, 2, U, &g)) return false;
  const uint64_t slice = (uint64_t)g.lanes * 16;
  const uint64_t at = (uint64_t)(uintptr_t)buf | U | (g.slices > 1 ? slice : 0);
  const uint64_t least = at % 128 == 0  ? 128
                         : at % 64 == 0 ? 192
                         : at % 32 == 0 ? 320
                                        : 352;
  return slice >= least;
}

bool walk_list_kept(uint64_t a, uint64_t B) {
  return cycle_list_kept(a, B, kWalkLogBlock);
}

cudaError_t launch_walk100(cudaStream_t s, void *buf, uint64_t T, uint64_t a,
                           uint64_t B, uint64_t U, void *scratch,
                           const std::function<void *(size_t)> &list_scratch,
                           bool may_cache) {
  WalkArgs g;
  if (!walk_args(buf, T, a, B, U, &g)) return cudaErrorInvalidValue;
  g.base = reinterpret_cast<char *>(buf);
  g.scratch = reinterpret_cast<char *>(scratch);
  const WalkMap m = g.m;
  void *mem = nullptr;
  cudaError_t err = cycle_list_for(
      s, a, B, m.lm, list_scratch, may_cache, &mem,
      [&](uint32_t *list, uint32_t *count) {
        const unsigned grid = (unsigned)std::min<uint64_t>(
            (m.N + kWalkThreads - 1) / kWalkThreads,
            (uint64_t)device_info().sms * 8);
        ProfScope ps(s, "walk_leaders");
        k_walk_leaders<<<grid, kWalkThreads, 0, s>>>(m, list, count);
        return cudaGetLastError();
      });
  if (err != cudaSuccess) return err;
  g.count = reinterpret_cast<const uint32_t *>(mem);
  g.list = reinterpret_cast<const uint32_t *>((const char *)mem + 256);
  return run_walk<16>(s, g);
}

}  // namespace lm
