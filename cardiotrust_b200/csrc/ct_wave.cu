// The two recursions through time of one beat, as one dataflow kernel.
//
// Forward (innovate_system_states_v1 + add_control_function,
// src/core/algorithm/estimation/prediction.rs:40-106), per item (voxel v, offset n, neighbour j):
//   ap[t] = fma(c, x[t-d, j] - ap[t-1], x[t-d-1, j])
//   x[t, 3v+a] = sum_k g[3v+a, k] ap[t][v, k] + u[t] B[3v+a]          (k = 3n + b, in order)
// Adjoint: the exact gradient of the stated loss
//   L = sum_t (mse/M)/2 |H x_t - z_t|^2 + reg/2 sum_v relu(|x_v|_1 - thr)^2
// with respect to the states. With lx = dL/dx, per item (voxel j, offset n) with source
// v = rev[j, n] (the voxel whose offset n points at j), coefficient and gains those of (v, n):
//   lap[t][b]    = sum_a g[3v+a, 3n+b] lx[t, 3v+a] - c lap[t+1][b]              (t = s + d)
//   lx[s, 3j+b]  = (mse/M) (H^T r_s)[3j+b] + reg f_j sign(x_{3j+b}) + sum_n (c lap[t][b] + lap[t+1][b])
// The reference crate has no counterpart of the adjoint: its derivation (derivation.rs:173-229) keeps
// only the per-step terms. Every item gathers the delayed row of its source, advances three chains
// and adds to its voxel's three sums, in either direction, so both run through the kernel below
// (the adjoint in the time tau = T-1-s); the parameter gradients are a sweep over the
// stored rows afterwards (ct_derive.cu). Gathering at the receiver replaces the scatter of one cell
// per (step, item) into per-voxel inboxes that the adjoint used before: only three floats per
// voxel-step cross between tiles instead of 78, and nothing of the all-pass history is stored
// or recomputed (20x20x20 cuboid, T = 2,000: the inbox form moved 24.6 GB through HBM in 11.2 ms).
//
// Compiled with -fmad=false: in the forward every `x + g * a` below rounds the product and the sum
// separately and in column order k = 0..77, and fmaf() stands exactly where the reference calls
// mul_add, so the states are bit-identical to the reference CPU loop.
//
// Design
//   * A tile is 32 consecutive device voxels (4x4x2 bricks, see ct_api.cu). One CTA of eight warps
//     works on it: lane = voxel; compute warp w owns offsets 4w .. 4w+3 (the last 24, 25) with their
//     gains, coefficients and chain states in registers, and passes the voxel's three partial sums
//     to warp w+1 through shared memory (a systolic chain: the column order of the sums is kept, and
//     no all-pass output leaves its warp). The last warp finishes the rows; warp 7 stages history.
//   * No grid barrier: a finished row goes to an exchange ring in global memory (L2) as one 16-byte entry
//     {x0, x1, x2, step + 1} per voxel, and the readers look at the entry itself until its tag is the step
//     they need: a 128-bit relaxed access is one access, so no fence separates data and flag. That is the
//     programming model's word for the polls (ld.relaxed.b128); the staging warp's cp.async of 16 aligned
//     bytes relies on the hardware, which moves such a piece of one 32-byte sector as a whole. Every read
//     is of a row at least dmin steps back, so tiles run up to dmin steps apart, and the latency of the
//     exchange overlaps the work on the steps between. (The former kernels met at a grid barrier every 8
//     steps, staged a block's rows after it and ran their producer and consumer phases one after the
//     other.)
//   * History. The staging warp copies the tile's halo (at most kHaloSlots - 1 voxels) row by row into
//     a ring of kRingRows rows in shared memory. A voxel's slot is chosen so that (slot mod 8) =
//     (2 y + z) mod 8: the eight lanes of a quarter warp are 4 x 2 neighbouring (y, z), so their 16-byte
//     reads fall into eight different bank groups whatever the offset. Where the spread of a tile's delays does
//     not fit the ring, or its halo is too large, the compute warps poll the exchange ring themselves. That way has a
//     kernel of its own (ANY), launched where such tiles may occur: the polling loops in every warp's code cost the staged
//     tiles 15 % (instruction fetch; as a second copy of the visit behind a call, which saves 60 registers in local
//     memory each time, the polled tiles took twice as long). The delays change on the device; where the host's bounds do not
//     tell, both kernels are launched and the one that is not meant leaves (4 us). Shell of 47,264 voxels, T = 1,000, a
//     slow layer of 100 to 173 steps and a fast one of 2 to 4: forward 30.3 ms with every tile polling, 22.1 so; with
//     the slow layer alone 20.4 and 12.0.
//   * Two steps are handed over together where no delay is shorter (one set of waits and arrivals for both: 1.33 ->
//     1.25 ms on the 20x20x20 cuboid), each step's sums as soon as they are there (1.25 -> 1.18 ms with the
//     smaller staging batches).
//   * A CTA that visits several tiles in turn, min(dmin, 64) steps each (the scenario's smallest delay), keeps their
//     registers in packed records (60 floats per lane) between visits. All rows that a visit reads belong to
//     earlier blocks of steps, so its staging warp waits once for the progress that the tiles around have
//     published and starts all copies (64x64x48 shell, T = 4,000: 27.4 -> 24.3 ms). Work is ordered by (phase, block
//     of steps) in every CTA and a row depends on earlier blocks only, so the cooperative launch (all CTAs
//     resident) cannot deadlock.
//   * Every wait is bounded: a wait that sees neither its data nor any progress of the launch (a
//     heartbeat counter) for 2 s records CT_ERR_TIMEOUT and the CTA leaves.
// What bounds it: the cycle of a row through the chain of warps, the exchange and the halo's staging, once
// per dmin steps (20x20x20 cuboid, dmin = 8: 1.18 ms are 9,300 clock cycles for each; issue slots 51 % used, DRAM 1.7 %).
// The forward's 128 registers do not hold everything: 204 bytes per thread are stored outside the loop over steps and ten
// loads per pair of steps and CTA take them back, 0.4 % of the instructions; the adjoint keeps all in registers.
// Measured, ms before -> now: forward 2.87 -> 1.18 (20x20x20, T = 2,000), 0.56 -> 0.23 (8x8x8, T = 500), 54.6 ->
// 24.5 (64x64x48 shell, T = 4,000); adjoint recursion 1.05 and 23 on the first and the last, where the
// inbox form took 11.2 and 145 with the gradients in it.
#include <cuda_runtime.h>

#include <algorithm>

#include "ct_internal.cuh"
#include "ct_sync.cuh"

namespace ct {
namespace {

constexpr int kTile = kFwdTileVoxels;
constexpr int kItems = 4;        // offsets per compute warp (the last one: 2)
constexpr int kComputeWarps = 7;
constexpr int kLastItems = kOffsets - kItems * (kComputeWarps - 1);
constexpr int kThreads = 32 * (kComputeWarps + 1);  // and the staging warp
constexpr int kHaloSlots = kFwdHaloMax;  // slots per ring row; the last one stays zero (absent neighbours)
constexpr int kZeroSlot = kHaloSlots - 1;
constexpr int kRingRows = 32;            // power of two
constexpr int kHand = 2;                 // hand-over buffers between consecutive warps, power of two
constexpr int kGroup = 2;                // steps per hand-over, where no delay is shorter
constexpr int kBatch = 4;                // rows that the staging warp copies together (two at first)
constexpr int kOwn = 4;                  // steps of the last warp's global reads in flight, power of two
constexpr int kMaxVisit = 64;            // steps per visit of a CTA that owns several tiles
constexpr int kPerLane = kHaloSlots / 32;  // halo voxels per lane of the staging warp
constexpr int kSmemPerCta = 233472 / 2 - 1024;  // two CTAs per SM
constexpr unsigned long long kWaitNs = 2000000000ull;
// the rows of one group of steps and of the batch that is staged beside it
static_assert(kFwdRingSpread + 2 + kGroup + kBatch <= kRingRows, "a tile's history fits the ring");
static_assert(kTile == 32 && kLastItems == 2 && kHaloSlots % 32 == 0, "lane = voxel");

struct WaveSmem {
  uint4 ring[kRingRows][kHaloSlots];          // {x0, x1, x2, -}
  uint4 hand[kComputeWarps - 1][kHand][kGroup][32];  // {sum0, sum1, sum2, group number + 1} from warp w to w + 1
  float own[kOwn][6][32];                     // the last warp's global reads per step
  uint64_t full[kRingRows];                   // the slot's row is staged (every lane of the staging warp)
  uint64_t empty[kRingRows];                  // no later step reads the slot's row
  uint64_t taken[kComputeWarps - 1][kHand];   // warp w + 1 has taken the entry
  int abort;
  WaveScn single;
};
static_assert(sizeof(WaveSmem) <= kSmemPerCta, "two CTAs per SM");

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Shared-memory hand-overs go through mbarriers: their arrive orders the shared-memory accesses before it at
// a few cycles, where a release store waited for the thread's global accesses as well (~1,000 cycles
// in the staging warp).
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Entries in shared memory: one 128-bit access each way, so the tag vouches for the data.
__device__ __forceinline__ uint4 lds_entry(uint32_t addr) {
  unsigned long long lo, hi;
  asm volatile(
      "{\n\t.reg .b128 e;\n\t"
      "ld.relaxed.cta.shared.b128 e, [%2];\n\t"
      "mov.b128 {%0, %1}, e;\n\t}"
      : "=l"(lo), "=l"(hi)
      : "r"(addr)
      : "memory");
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
__device__ __forceinline__ void sts_entry(uint32_t addr, const uint4& v) {
  const unsigned long long lo = (unsigned long long)v.x | ((unsigned long long)v.y << 32);
  const unsigned long long hi = (unsigned long long)v.z | ((unsigned long long)v.w << 32);
  asm volatile(
      "{\n\t.reg .b128 e;\n\t"
      "mov.b128 e, {%1, %2};\n\t"
      "st.relaxed.cta.shared.b128 [%0], e;\n\t}" ::"r"(addr),
      "l"(lo), "l"(hi)
      : "memory");
}
__device__ __forceinline__ uint32_t lds_tag(uint32_t addr) {
  uint32_t w;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(w) : "r"(addr + 12) : "memory");
  return w;
}
// One exchange entry {x0, x1, x2, tag}: a single 128-bit access each way.
__device__ __forceinline__ uint4 ld_entry(const uint4* p) {
  unsigned long long lo, hi;
  asm volatile(
      "{\n\t.reg .b128 e;\n\t"
      "ld.relaxed.gpu.global.b128 e, [%2];\n\t"
      "mov.b128 {%0, %1}, e;\n\t}"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
__device__ __forceinline__ void st_entry(uint4* p, float a, float b, float c, uint32_t tag) {
  const unsigned long long lo = (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
  const unsigned long long hi = (unsigned long long)__float_as_uint(c) | ((unsigned long long)tag << 32);
  asm volatile(
      "{\n\t.reg .b128 e;\n\t"
      "mov.b128 e, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], e;\n\t}" ::"l"(p),
      "l"(lo), "l"(hi)
      : "memory");
}

// Steps that a tile has finished (one word per 128 bytes, behind the exchange ring).
__device__ __forceinline__ int* progress_of(const WaveScn& p, int tile) {
  return reinterpret_cast<int*>(p.xch + (size_t)p.xrows * p.V) + 32 * (size_t)tile;
}
__device__ __forceinline__ int ld_progress(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_progress(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Limit of a wait. `since` is 0 at its first call and then what the last call returned; 0 ends the wait.
// It lasts while the launch makes progress: the heartbeat's lowest bits are part of the value.
__device__ __noinline__ unsigned long long may_wait(unsigned long long since, int* abort, int32_t* status,
                                                    const unsigned int* heartbeat) {
  if (*(volatile int*)abort) return 0;
  if (*(volatile int32_t*)status != 0) {
    *(volatile int*)abort = 1;
    return 0;
  }
  const unsigned long long now = (global_ns() & ~255ull) | (ld_acquire_gpu(heartbeat) & 255u);
  if (since == 0 || (since & 255u) != (now & 255u)) return now ? now : 1;
  if (now - since > kWaitNs) {
    atomicCAS(status, 0, (int32_t)CT_ERR_TIMEOUT);
    *(volatile int*)abort = 1;
    return 0;
  }
  return since;
}
// Every `mask` + 1 spins of a wait: whether it may go on. Lanes decide for themselves, and one whose wait is lost leaves the
// kernel on the shortest way, without another vote or barrier. The others find sm.abort at their next look; until
// then their votes, shuffles and reductions count the threads that have not exited, and no mbarrier phase can
// complete without the arrivals that are missing now, so that they end in waits that look. (One decision per warp, by a
// vote in every wait, cost 1 % on the 20x20x20 cuboid and 11 % on the shell's forward.)
__device__ __forceinline__ bool go_on(WaveSmem& sm, const WaveLaunch& L, int& spins, unsigned long long& since, int mask) {
  if ((++spins & mask) != 0) return true;
  since = may_wait(since, &sm.abort, L.status, &L.heartbeat->count);
  return since != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, WaveSmem& sm, const WaveLaunch& L) {
  if (mbar_try(bar, parity)) return true;
  int spins = 0;
  unsigned long long since = 0;
  while (!mbar_try(bar, parity))
    if (!go_on(sm, L, spins, since, 15)) return false;
  return true;
}
// Phase parity of the n-th use (0, 1, ...) of a ring entry at position pos.
__device__ __forceinline__ uint32_t row_parity(int pos) { return (uint32_t)(pos / kRingRows) & 1u; }

// Steps per visit of a CTA with several tiles: the scenario's smallest delay at most, so that every row that a visit
// reads belongs to an earlier block of steps.
__device__ __forceinline__ int visit_steps(const WaveScn& p) {
  return p.dmin[0] > p.dmin[1] ? kMaxVisit : min(p.dmin[0], kMaxVisit);  // nothing connected: nothing is read
}

// Delay range of a tile's own items: one slow or fast layer of tissue leaves the other tiles their pairs and rings.
struct Geometry {
  int dmin, dmax;
  bool pairs; // no step reads the step before: two steps may be handed over together
  bool ring;  // the rows of one step and of two batches fit the shared ring
};
__device__ __forceinline__ Geometry geometry(const WaveScn& p, int tile) {
  Geometry g;
  g.dmin = p.range[2 * tile];
  g.dmax = p.range[2 * tile + 1];
  if (g.dmin > g.dmax) g.dmin = g.dmax = visit_steps(p);  // no connected pair: only rows of its readers are followed, if any
  g.pairs = g.dmin >= kGroup;
  g.ring = (long long)g.dmax - g.dmin <= kFwdRingSpread;
  return g;
}
// The CTA's visits, in the order that every warp of it follows.
struct Visit {
  int tile, scn, v0, t0, t1;
  bool whole;  // the CTA stays with this tile for the whole beat
  bool shared; // some CTA of the phase visits several tiles
};
struct Walk {
  int phase = -1, begin = 0, end = 0, tile = 0, block = 0;
  bool several = false, live = false;
};
__device__ __forceinline__ const WaveScn& scenario_of(const WaveSmem& sm, const WaveLaunch& L, int s) {
  return L.scns ? L.scns[s] : sm.single;
}
__device__ __forceinline__ bool next_visit(const WaveSmem& sm, const WaveLaunch& L, Walk& w, Visit& v) {
  for (;;) {
    if (w.tile < w.end) {
      v.tile = w.tile;
      w.tile += gridDim.x;
      if (L.tiles) {
        const int2 t = L.tiles[v.tile];
        v.scn = t.x;
        v.v0 = t.y;
      } else {
        v.scn = 0;
        v.v0 = v.tile * kTile;
      }
      const WaveScn& p = scenario_of(sm, L, v.scn);
      v.whole = !w.several;
      v.shared = w.end - w.begin > (int)gridDim.x;
      v.t0 = 0;
      v.t1 = p.T;
      if (v.whole) return true;
      const int len = visit_steps(p);
      if (w.block > (p.T - 1) / len) continue;
      w.live = true;
      v.t0 = w.block * len;
      v.t1 = min(p.T, v.t0 + len);
      return true;
    }
    if (w.several && w.live) {
      ++w.block;
      w.live = false;
      w.tile = w.begin + blockIdx.x;
      continue;
    }
    if (++w.phase >= L.nphases) return false;
    w.begin = L.phase_begin ? L.phase_begin[w.phase] : 0;
    w.end = L.phase_begin ? L.phase_begin[w.phase + 1] : L.ntiles;
    w.tile = w.begin + blockIdx.x;
    w.several = w.tile + (int)gridDim.x < w.end;
    w.block = 0;
    w.live = false;
  }
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Copies n rows from r into positions from pos on and returns how many of them, from the first one on,
// carry their tags. PARTS: entries per lane (the halo's length over 32).
template <int PARTS>
__device__ __forceinline__ int copy_rows(const uint4* const (&from)[kPerLane], const uint32_t (&to)[kPerLane], uint32_t ring, int V,
                                         int mask, int r, int pos, int n) {
  for (int j = 0; j < n; ++j) {
    const size_t row = (size_t)((r + j) & mask) * V;
    const uint32_t at = ring + (uint32_t)((pos + j) & (kRingRows - 1)) * (kHaloSlots * 16);
#pragma unroll
    for (int i = 0; i < PARTS; ++i) cp_async16(at + to[i], from[i] + row);
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  uint32_t miss = 1u << n;  // bit j: row r + j is not complete
#pragma unroll 2
  for (int j = 0; j < n; ++j) {
    const uint32_t at = ring + (uint32_t)((pos + j) & (kRingRows - 1)) * (kHaloSlots * 16);
    uint32_t bad = 0;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) bad |= lds_tag(at + to[i]) ^ ((uint32_t)(r + j) + 1u);
    if (bad) miss |= 1u << j;
  }
  return __ffs(__reduce_or_sync(0xffffffffu, miss)) - 1;
}

// The staging warp: rows [t0 - dmax - 1, t1 - 1 - dmin] of every visit, from the exchange ring into the shared
// ring. It copies a few rows' entries with cp.async and then looks at their tags: an entry is one
// aligned 16-byte word, written by one access, and a row whose tags are not all there is copied again. Lanes take
// the halo in device order (runs of neighbouring entries). Two rows at a time while it waits for rows to
// be finished, a few more while it finds them ready (3 against 4 with one tile per CTA: 1.18 against 1.23 ms on
// the 20x20x20 cuboid; always 2: 1.20, and 7 % slower on the shell). Loads into
// registers were slower.
template <bool ANY>
__device__ __forceinline__ void stage_history(WaveSmem& sm, const WaveLaunch& L) {
  const int lane = threadIdx.x & 31;
  Walk walk;
  Visit v;
  int pos = 0;
  // waits until the ring slots of positions up to `at` may be written (rows are released in order)
  auto room = [&](int at) -> bool {
    return at < kRingRows || mbar_wait(&sm.empty[at & (kRingRows - 1)], row_parity(at) ^ 1u, sm, L);
  };
  // this lane's entries of rows [from, to) are stored
  auto publish = [&](int from, int to) {
    for (; from < to; ++from) mbar_arrive(&sm.full[from & (kRingRows - 1)]);
  };
  const uint32_t ring = smem_u32(&sm.ring[0][0]);
  while (next_visit(sm, L, walk, v)) {
    const WaveScn& p = scenario_of(sm, L, v.scn);
    const int tile = v.v0 / kTile;
    const Geometry geo = geometry(p, tile);
    const int nh = p.nhalo[tile];
    if (ANY && (!geo.ring || nh < 0)) continue;
    int r = v.t0 - geo.dmax - 1;
    const int end = v.t1 - geo.dmin;  // rows [r, end)
    const int after = pos + end - r;
    if (nh > 0) {
      const uint4* from[kPerLane];  // the lane's voxels' entries in exchange row 0
      uint32_t to[kPerLane];        // their slots
#pragma unroll
      for (int i = 0; i < kPerLane; ++i) {
        const size_t e = (size_t)tile * kHaloSlots + 32 * i + lane;  // the table repeats its last voxel
        from[i] = p.xch + p.halo[e];
        to[i] = 16u * p.hpos[e];
      }
      const bool zeros = r < 0;
      for (; r < min(0, end); ++r, ++pos) {  // rows before the beat
        if (!room(pos)) return;
#pragma unroll
        for (int i = 0; i < kPerLane; ++i)
          sts_entry(ring + (uint32_t)(pos & (kRingRows - 1)) * (kHaloSlots * 16) + to[i], make_uint4(0, 0, 0, 0));
        publish(pos, pos + 1);
      }
      const int V = p.V, mask = p.xrows - 1;
      const int parts = (nh + 31) / 32;
      const int* near = p.near + (size_t)tile * kNearTiles;
      if (!v.whole && near[0] >= 0 && !zeros) {
        // All rows of the visit belong to earlier blocks: once the tiles around have published these, the copies
        // need no look at their tags, and each row's arrival is counted by the copies themselves. Such an arrival stands for
        // the copies alone: zero rows stored before it, which readers do not wait for one by one, would not be ordered by
        // it, so the few visits that begin before the beat take the other way.
        const int *a = progress_of(p, near[lane]), *b = progress_of(p, near[lane + 32]);
        int spins = 0;
        unsigned long long since = 0;
        while (!__all_sync(0xffffffffu, ld_progress(a) >= end && ld_progress(b) >= end))
          if (!go_on(sm, L, spins, since, 63)) return;
        __syncwarp();  // every lane's acquires before any lane's copies
        for (; r < end; ++r, ++pos) {
          if (!room(pos)) return;
          const size_t row = (size_t)(r & mask) * V;
          const uint32_t at = ring + (uint32_t)(pos & (kRingRows - 1)) * (kHaloSlots * 16);
#pragma unroll
          for (int i = 0; i < kPerLane; ++i)
            if (i < parts) cp_async16(at + to[i], from[i] + row);
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(
                           smem_u32(&sm.full[pos & (kRingRows - 1)]))
                       : "memory");
        }
      }
      // one tile per CTA: rows come one by one, and copying rows that are not there delays the next look
      const int most = v.whole ? kBatch - 1 : kBatch;
      int batch = most, spins = 0;
      unsigned long long since = 0;
      while (r < end) {
        const int n = min(batch, end - r);
        if (!room(pos + n - 1)) return;
        const int got = parts <= 4   ? copy_rows<4>(from, to, ring, V, mask, r, pos, n)
                        : parts == 5 ? copy_rows<5>(from, to, ring, V, mask, r, pos, n)
                                     : copy_rows<6>(from, to, ring, V, mask, r, pos, n);
        if (got > 0) {
          publish(pos, pos + got);
          pos += got;
          r += got;
          since = 0;
        } else if (!go_on(sm, L, spins, since, 63)) {
          return;
        }
        batch = got == n ? most : 2;
      }
    } else {
      for (; pos < after; ++pos) {  // nothing to read
        if (!room(pos)) return;
        publish(pos, pos + 1);
      }
    }
    pos = after;
  }
}

// Counters that run through all of a warp's visits.
struct Cursor {
  int group = 0;  // hand-overs
  int pos = 0;   // ring position of the visit's first row
};

enum { kFirst = 0, kMiddle = 1, kLast = 2 };

// What a compute warp keeps in registers during a visit: its items, and the visit's constants.
template <int NI>
struct Tile {
  float g[NI][3][3], st[NI][3], prev[NI][3], c[NI];
  uint32_t at[NI];  // ring: shared address of the item's slot in row 0; else the source voxel, ~0 if absent
  int off[NI];      // ring: position of the item's row for step t, minus t; else minus the delay
  const uint4* src;     // exchange ring
  uint4* dst;           // the voxel's entry of exchange row 0
  float* out;           // the voxel's state in row 0 of the finished rows
  float* part;          // the tile's regularisation term of step 0
  const float* X;       // adjoint: the voxel's states and mapped residuals in row 0
  const float* MR;
  const float* u;
  float* ap_last;
  float ctrl[3], threshold, mse, reg;
  int V, S, T, mask, ntiles, lane;
  int floor, need;  // ring positions of rows t - dmax - 1 and t - dmin, minus t
  bool live, ring;
};

// The items' delayed rows for steps [t, t + N), from the shared ring or polled from the exchange ring.
template <int N, bool ANY, int NI>
__device__ __forceinline__ bool fetch(WaveSmem& sm, const WaveLaunch& L, const Tile<NI>& k, int t, float (&x)[N][NI][3]) {
  if (!ANY || k.ring) {
    const int pos = k.need + t + N - 1;  // rows are staged in order
    if (!mbar_wait(&sm.full[pos & (kRingRows - 1)], row_parity(pos), sm, L)) return false;
#pragma unroll
    for (int s = 0; s < N; ++s)
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const uint4 e = lds_entry(k.at[i] + ((uint32_t)(k.off[i] + t + s) & (kRingRows - 1)) * (kHaloSlots * 16));
        x[s][i][0] = __uint_as_float(e.x);
        x[s][i][1] = __uint_as_float(e.y);
        x[s][i][2] = __uint_as_float(e.z);
      }
    return true;
  }
  bool good = true;
#pragma unroll
  for (int s = 0; s < N; ++s) {
    int spins = 0;
    unsigned long long since = 0;
    for (;;) {
      uint4 e[NI];
      bool there = true;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int r = t + s + k.off[i];
        const bool reads = (int)k.at[i] >= 0 && r >= 0;
        e[i] = ld_entry(reads ? k.src + (size_t)(r & k.mask) * k.V + k.at[i] : k.src);
        if (!reads) e[i] = make_uint4(0, 0, 0, (uint32_t)r + 1u);
        there = there && e[i].w == (uint32_t)r + 1u;
      }
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        x[s][i][0] = __uint_as_float(e[i].x);
        x[s][i][1] = __uint_as_float(e[i].y);
        x[s][i][2] = __uint_as_float(e[i].z);
      }
      if (there) break;
      if (!go_on(sm, L, spins, since, 63)) {
        good = false;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, good);
}

// Last warp: its global reads for steps [t, t + n) into shared memory, one cp.async group (every lane reads
// back its own words only).
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
template <bool ADJ, int NI>
__device__ __forceinline__ void read_own(WaveSmem& sm, const Tile<NI>& k, int t, int n) {
  for (int s = t; s < t + n && s < k.T; ++s) {
    float(*q)[32] = sm.own[s & (kOwn - 1)];
    if (ADJ) {
      const size_t o = (size_t)(k.T - 1 - s) * k.S;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        cp_async4(&q[b][k.lane], k.X + o + b);
        cp_async4(&q[3 + b][k.lane], k.MR + o + b);
      }
    } else {
      cp_async4(&q[0][k.lane], k.u + s);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Steps [t, t + N) of one warp's items. False: a wait ran out.
template <int N, int NI, int POS, bool ADJ, bool ANY>
__device__ __forceinline__ bool compute_group(WaveSmem& sm, const WaveLaunch& L, Tile<NI>& k, Cursor& cur, int w, int t) {
  float x[N][NI][3];
  if (!fetch<N, ANY>(sm, L, k, t, x)) return false;
  // the items' chains; x becomes the all-pass outputs (forward)
  float sum[N][3];  // adjoint: the items' contributions
#pragma unroll
  for (int s = 0; s < N; ++s) {
    sum[s][0] = sum[s][1] = sum[s][2] = 0.0f;
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (ADJ) {
          const float gl = fmaf(k.g[i][2][b], x[s][i][2], fmaf(k.g[i][1][b], x[s][i][1], k.g[i][0][b] * x[s][i][0]));
          const float lap = fmaf(-k.c[i], k.st[i][b], gl);
          sum[s][b] = sum[s][b] + fmaf(k.c[i], lap, k.st[i][b]);
          k.st[i][b] = lap;
        } else {
          const float in = x[s][i][b];
          k.st[i][b] = fmaf(k.c[i], in - k.st[i][b], k.prev[i][b]);
          k.prev[i][b] = in;
          x[s][i][b] = k.st[i][b];
        }
      }
    if (!ADJ && t + s == k.T - 2 && k.live) {
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int b = 0; b < 3; ++b) k.ap_last[3 * i + b] = k.st[i][b];
    }
  }
  if (POS == kLast) {  // the next group's global reads; this group's have landed
    read_own<ADJ>(sm, k, t + N, kGroup);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
  }
  // the voxel's sums: from warp w - 1, plus this warp's columns, to warp w + 1, step by step. What the seven warps
  // do between taking and passing them on is the latency of a step; everything else comes before or after.
  const int buf = cur.group & (kHand - 1);
  const uint32_t tag = (uint32_t)cur.group + 1u;
  if (POS != kLast && cur.group >= kHand &&
      !mbar_wait(&sm.taken[w][buf], ((uint32_t)(cur.group / kHand) & 1u) ^ 1u, sm, L))
    return false;
  float y[N][3];  // last warp: the finished rows
#pragma unroll
  for (int s = 0; s < N; ++s) {
    float acc[3] = {0.0f, 0.0f, 0.0f};
    if (POS != kFirst) {
      const uint32_t from = smem_u32(&sm.hand[w - 1][buf][s][k.lane]);
      const volatile uint32_t* flag = &sm.hand[w - 1][buf][s][0].w;
      int spins = 0;
      unsigned long long since = 0;
      for (;;) {
        while (*flag != tag)  // one word, then the entries
          if (!go_on(sm, L, spins, since, 1023)) return false;
        const uint4 h = lds_entry(from);
        acc[0] = __uint_as_float(h.x);
        acc[1] = __uint_as_float(h.y);
        acc[2] = __uint_as_float(h.z);
        if (__all_sync(0xffffffffu, h.w == tag)) break;
      }
    }
    if (ADJ) {
#pragma unroll
      for (int b = 0; b < 3; ++b) acc[b] = acc[b] + sum[s][b];
    } else {
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int a = 0; a < 3; ++a) acc[a] = acc[a] + k.g[i][a][b] * x[s][i][b];
    }
    if (POS != kLast) {
      sts_entry(smem_u32(&sm.hand[w][buf][s][k.lane]),
                make_uint4(__float_as_uint(acc[0]), __float_as_uint(acc[1]), __float_as_uint(acc[2]), tag));
    } else {
      const float(*q)[32] = sm.own[(t + s) & (kOwn - 1)];
      if (ADJ) {
        const float xr[3] = {q[0][k.lane], q[1][k.lane], q[2][k.lane]};
        const float l1 = fabsf(xr[0]) + fabsf(xr[1]) + fabsf(xr[2]);
        const float f = l1 > k.threshold ? l1 - k.threshold : 0.0f;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const float pull = f > 0.0f ? f * copysignf(1.0f, xr[b]) : 0.0f;
          y[s][b] = k.mse * q[3 + b][k.lane] + k.reg * pull + acc[b];
        }
      } else {
        const float u = q[0][k.lane];
#pragma unroll
        for (int a = 0; a < 3; ++a) y[s][a] = acc[a] + u * k.ctrl[a];
      }
      if (k.live) st_entry(k.dst + (size_t)((t + s) & k.mask) * k.V, y[s][0], y[s][1], y[s][2], (uint32_t)(t + s) + 1u);
    }
  }
  if (POS == kLast) {
    if (k.live) {
#pragma unroll
      for (int s = 0; s < N; ++s) {
        float* out = k.out + (size_t)(ADJ ? k.T - 1 - t - s : t + s) * k.S;
        out[0] = y[s][0];
        out[1] = y[s][1];
        out[2] = y[s][2];
      }
    }
    if (!ADJ) {
      // the tile's max-regularisation term of each step, reduced in lane order
      float f2[N], any = 0.0f;
#pragma unroll
      for (int s = 0; s < N; ++s) {
        const float l1 = fabsf(y[s][0]) + fabsf(y[s][1]) + fabsf(y[s][2]);
        const float f = l1 - k.threshold;
        f2[s] = k.live && l1 > k.threshold ? f * f : 0.0f;
        any = any + f2[s];
      }
      if (__any_sync(0xffffffffu, any != 0.0f)) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
#pragma unroll
          for (int s = 0; s < N; ++s) f2[s] = f2[s] + __shfl_down_sync(0xffffffffu, f2[s], d);
      }
      if (k.lane == 0)
#pragma unroll
        for (int s = 0; s < N; ++s) k.part[(size_t)(t + s) * k.ntiles] = f2[s];
    }
  }
  if (POS != kFirst) {
    __syncwarp();
    if (k.lane == 0) mbar_arrive(&sm.taken[w - 1][buf]);
    // every warp has read what steps before t + N need: no later step reads rows before t + N - dmax - 1
    if (POS == kLast && (!ANY || k.ring) && k.lane < N) mbar_arrive(&sm.empty[(k.floor + t + k.lane) & (kRingRows - 1)]);
  }
  ++cur.group;
  if (POS == kLast && (cur.group & 127) == 0 && k.lane == 0) atomicAdd(&L.heartbeat->count, 1u);
  return true;
}

// One visit of a compute warp: NI offsets from 4 w for steps [v.t0, v.t1). False: a wait ran out.
template <int NI, int POS, bool ADJ, bool ANY>
__device__ __forceinline__ bool compute_visit(WaveSmem& sm, const WaveLaunch& L, const WaveScn& p, const Geometry& geo,
                                              const Visit& v, Cursor& cur, int w) {
  const int lane = threadIdx.x & 31;
  const int n0 = w * kItems;
  const int tile = v.v0 / kTile;
  constexpr int kFloats = NI * 15, kVecs = (kFloats + 3) / 4;
  float4* rec = L.record ? L.record + ((size_t)v.tile * kComputeWarps + w) * 15 * 32 + lane : nullptr;
  Tile<NI> k;
  k.lane = lane;
  k.V = p.V;
  k.S = 3 * p.V;
  k.T = p.T;
  k.live = lane < min(kTile, k.V - v.v0);
  k.ring = !ANY || (geo.ring && p.nhalo[tile] >= 0);
  const int vox = v.v0 + (k.live ? lane : 0);
  k.mask = p.xrows - 1;
  k.src = p.xch;
  if (POS == kLast) {
    k.dst = p.xch + vox;
    k.out = p.rows + 3 * vox;
    if (ADJ) {
      k.X = p.X + 3 * vox;
      k.MR = p.MR + 3 * vox;
      k.mse = p.mse_scaling;
      k.reg = p.reg_scaling;
    } else {
      k.part = p.part + tile;
      k.ntiles = p.ntiles;
      k.u = p.u;
#pragma unroll
      for (int a = 0; a < 3; ++a) k.ctrl[a] = p.ctrl[3 * vox + a];
    }
    k.threshold = p.threshold;
    read_own<ADJ>(sm, k, v.t0, kGroup);
  }
  if (!ADJ) k.ap_last = p.ap_last + (size_t)vox * kGainCols + 3 * n0;

  if (v.whole || v.t0 == 0) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const size_t it = (size_t)vox * kOffsets + n0 + i;
      const int32_t src = k.live ? p.src[it] : -1;
      const bool ok = src >= 0;
      const size_t own = ADJ ? (size_t)(ok ? src : 0) * kOffsets + n0 + i : it;
      const float* gr = p.gains + (size_t)3 * (ADJ ? (ok ? src : 0) : vox) * kGainCols + 3 * (n0 + i);
      k.c[i] = ok ? p.coefs[own] : 0.0f;
      k.off[i] = -(ok ? p.delays[own] : geo.dmin);
      k.at[i] = k.ring ? (ok ? (uint32_t)p.hslot[((size_t)tile * kTile + lane) * kOffsets + n0 + i] : (uint32_t)kZeroSlot)
                     : (uint32_t)src;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        k.st[i][b] = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) k.g[i][a][b] = ok ? gr[a * kGainCols + b] : 0.0f;
      }
    }
  } else {
    float f[kVecs * 4];
#pragma unroll
    for (int q = 0; q < kVecs; ++q) {
      const float4 r = rec[q * 32];
      f[4 * q] = r.x;
      f[4 * q + 1] = r.y;
      f[4 * q + 2] = r.z;
      f[4 * q + 3] = r.w;
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
#pragma unroll
      for (int q = 0; q < 9; ++q) k.g[i][q / 3][q % 3] = f[3 * NI + 9 * i + q];
#pragma unroll
      for (int b = 0; b < 3; ++b) k.st[i][b] = f[3 * i + b];
      k.c[i] = f[12 * NI + i];
      k.at[i] = (uint32_t)__float_as_int(f[13 * NI + i]);
      k.off[i] = __float_as_int(f[14 * NI + i]);
    }
  }
  // the record: chain states first (rewritten at the end of every visit), then the constants
  auto save = [&](int from, int to) {
    float f[kVecs * 4] = {};
#pragma unroll
    for (int i = 0; i < NI; ++i) {
#pragma unroll
      for (int b = 0; b < 3; ++b) f[3 * i + b] = k.st[i][b];
#pragma unroll
      for (int q = 0; q < 9; ++q) f[3 * NI + 9 * i + q] = k.g[i][q / 3][q % 3];
      f[12 * NI + i] = k.c[i];
      f[13 * NI + i] = __int_as_float((int)k.at[i]);
      f[14 * NI + i] = __int_as_float(k.off[i]);
    }
#pragma unroll
    for (int q = 0; q < kVecs; ++q)
      if (q >= from && q < to) rec[q * 32] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
  };
  if (!v.whole && v.t0 == 0 && v.t1 < k.T) save(0, kVecs);
  k.floor = cur.pos - v.t0;
  k.need = k.floor + geo.dmax - geo.dmin + 1;
  const int base = k.floor + geo.dmax + 1;
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (k.ring) {
      k.at[i] = smem_u32(&sm.ring[0][k.at[i]]);
      k.off[i] += base;
    }
    k.prev[i][0] = k.prev[i][1] = k.prev[i][2] = 0.0f;
  }
  if (!ADJ) {
    float x[1][NI][3];
    if (!fetch<1, ANY>(sm, L, k, v.t0 - 1, x)) return false;
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int b = 0; b < 3; ++b) k.prev[i][b] = x[0][i][b];
  }

  int t = v.t0, said = v.t0;
  const int step = visit_steps(p);
  // last warp: the rows before t are finished, for the staging warps that ask for the progress of tiles
  auto say = [&](bool now) {
    if (POS != kLast || !v.shared || (!now && t - said < step)) return;
    said = t;
    __syncwarp();
    if (lane == 0) st_progress(progress_of(p, tile), t);
  };
  if (geo.pairs)
    for (; t + kGroup <= v.t1;) {
      if (!compute_group<kGroup, NI, POS, ADJ, ANY>(sm, L, k, cur, w, t)) return false;
      t += kGroup;
      say(false);
    }
  for (; t < v.t1;) {
    if (!compute_group<1, NI, POS, ADJ, ANY>(sm, L, k, cur, w, t)) return false;
    ++t;
    say(false);
  }
  say(true);
  if (POS == kLast) {
    asm volatile("cp.async.wait_all;" ::: "memory");  // the next visit reuses the buffers
    if (k.ring && lane == 0)  // the visit's remaining rows
      for (int q = 0; q < geo.dmax - geo.dmin + 1; ++q) mbar_arrive(&sm.empty[(k.floor + v.t1 + q) & (kRingRows - 1)]);
  }
  if (k.ring) cur.pos += v.t1 - v.t0 + geo.dmax - geo.dmin + 1;
  if (v.t1 < k.T) {
    save(0, (3 * NI + 3) / 4);
  } else if (!ADJ && k.live) {
    float* ap = p.ap + (size_t)vox * kGainCols + 3 * n0;
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        ap[3 * i + b] = k.st[i][b];
        if (k.T < 2) k.ap_last[3 * i + b] = 0.0f;
      }
  }
  return true;
}
template <int NI, int POS, bool ADJ, bool ANY>
__device__ __forceinline__ void compute(WaveSmem& sm, const WaveLaunch& L, int w) {
  Walk walk;
  Visit v;
  Cursor cur;
  while (next_visit(sm, L, walk, v)) {
    const WaveScn& p = scenario_of(sm, L, v.scn);
    const Geometry geo = geometry(p, v.v0 / kTile);
    if (!compute_visit<NI, POS, ADJ, ANY>(sm, L, p, geo, v, cur, w)) return;
  }
}

template <bool ADJ, bool ANY>
__global__ void __launch_bounds__(kThreads, 2) wave_kernel(const __grid_constant__ WaveLaunch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WaveSmem& sm = *reinterpret_cast<WaveSmem*>(smem_raw);
  for (int i = threadIdx.x; i < kRingRows * kHaloSlots; i += kThreads) (&sm.ring[0][0])[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < (kComputeWarps - 1) * kHand * kGroup * 32; i += kThreads)
    (&sm.hand[0][0][0][0])[i] = make_uint4(0, 0, 0, 0);
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRingRows; ++i) {
      mbar_init(&sm.full[i], 32);
      mbar_init(&sm.empty[i], 1);
    }
    for (int w = 0; w < kComputeWarps - 1; ++w)
      for (int i = 0; i < kHand; ++i) mbar_init(&sm.taken[w][i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sm.abort = 0;
    if (!L.scns) sm.single = L.single;
  }
  __syncthreads();
  // Which of the two kernels is meant: where the host cannot know it is launched with both, and one leaves. And every
  // exchange ring must hold the rows that a reader may still want, or all of them: when a tile writes step t, its neighbours
  // have finished step t - dmax at least, and from there on they read back to t - 2 dmax.
  bool apart = false, fits = true;
  for (int s = 0; s < L.nscn; ++s) {
    const WaveScn& p = scenario_of(sm, L, s);
    if (p.dmin[0] > p.dmin[1]) continue;  // nothing is connected
    apart = apart || (long long)p.dmin[1] - p.dmin[0] > kFwdRingSpread;
    fits = fits && (p.xrows >= p.T || 2ll * p.dmin[1] + 2 <= p.xrows);
  }
  if (L.routes == kDecide && apart != ANY) return;
  if (!fits || (L.routes == kStaged && apart)) {  // every CTA leaves here
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(L.status, 0, (int32_t)CT_ERR_NOT_SUPPORTED);
    return;
  }
  const int w = threadIdx.x / 32;
  if (w >= kComputeWarps)
    stage_history<ANY>(sm, L);
  else if (w == 0)
    compute<kItems, kFirst, ADJ, ANY>(sm, L, w);
  else if (w < kComputeWarps - 1)
    compute<kItems, kMiddle, ADJ, ANY>(sm, L, w);
  else
    compute<kLastItems, kLast, ADJ, ANY>(sm, L, w);
  asm volatile("cp.async.wait_all;" ::: "memory");  // no thread leaves before its copies have landed, after a lost wait either
}

const void* const kKernels[4] = {(const void*)wave_kernel<false, false>, (const void*)wave_kernel<true, false>,
                                 (const void*)wave_kernel<false, true>, (const void*)wave_kernel<true, true>};

bool configure(int device) {
  static bool done[128] = {};
  if (device < 0 || device >= 128) return false;
  if (!done[device]) {
    for (const void* f : kKernels)
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WaveSmem)) != cudaSuccess) return false;
    done[device] = true;
  }
  return true;
}

}  // namespace

int wave_capacity(int device) {
  configure(device);
  int sms = 0, per_sm = 1 << 10;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  for (const void* f : kKernels) {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, kThreads, sizeof(WaveSmem));
    per_sm = std::min(per_sm, n);
  }
  return sms * std::max(per_sm, 1);
}

size_t wave_record_bytes() { return sizeof(float4) * kComputeWarps * 15 * 32; }

WaveScn wave_scenario(const DeviceScenario& d, bool adjoint, const WaveScalars& s, float* part) {
  WaveScn a;
  a.V = (int)d.V;
  a.T = (int)d.T;
  a.ntiles = (int)d.tiles;
  a.xrows = d.xrows;
  a.src = adjoint ? d.rev : d.nbr;
  a.halo = adjoint ? d.rhalo : d.halo;
  a.hpos = adjoint ? d.rhpos : d.hpos;
  a.hslot = adjoint ? d.rhslot : d.hslot;
  a.near = adjoint ? d.rnear : d.near;
  a.nhalo = adjoint ? d.rnhalo : d.nhalo;
  a.coefs = d.coefs;
  a.delays = d.delays;
  a.gains = d.gains;
  a.dmin = d.dmin;
  a.range = adjoint ? d.rrange : d.range;
  a.xch = d.xch;
  a.rows = adjoint ? d.LX : d.X;
  a.ctrl = d.ctrl;
  a.u = d.u;
  a.ap = d.ap;
  a.ap_last = d.ap_last;
  a.part = part;
  a.X = d.X;
  a.MR = d.MR;
  a.threshold = s.threshold;
  a.mse_scaling = s.mse_scaling;
  a.reg_scaling = s.reg_scaling;
  return a;
}

cudaError_t launch_wave(const WaveLaunch& launch, bool adjoint, int grid, cudaStream_t stream) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  if (!configure(device)) return cudaErrorInvalidValue;
  WaveLaunch l = launch;
  void* args[] = {&l};
  err = cudaSuccess;
  for (int any = 0; any < 2 && err == cudaSuccess; ++any)
    if (launch.routes == kDecide || (launch.routes == kEvery) == (any == 1))
      err = launch_cooperative(kKernels[2 * any + (adjoint ? 1 : 0)], grid, kThreads, args, sizeof(WaveSmem), stream);
  return err;
}

// Empty the exchange ring (tag 0: no step) and the tiles' progress.
cudaError_t clear_exchange(DeviceScenario& d, cudaStream_t stream) {
  return cudaMemsetAsync(d.xch, 0, sizeof(uint4) * ((size_t)d.xrows * d.V + 8 * (size_t)d.tiles), stream);
}

namespace {
cudaError_t launch_single(DeviceScenario& d, bool adjoint, const WaveScalars& s, cudaStream_t stream) {
  cudaError_t err = clear_exchange(d, stream);
  if (err != cudaSuccess) return err;
  WaveLaunch l;
  l.scns = nullptr;
  l.single = wave_scenario(d, adjoint, s, d.stepsum_part);
  l.nscn = 1;
  l.tiles = nullptr;
  l.phase_begin = nullptr;
  l.nphases = 1;
  l.ntiles = (int)d.tiles;
  l.record = d.record;
  l.routes = adjoint ? d.rroutes : d.routes;
  l.status = d.status;
  l.heartbeat = d.heartbeat;
  return launch_wave(l, adjoint, d.wave_grid, stream);
}
}  // namespace

cudaError_t launch_forward(DeviceScenario& d, float threshold, cudaStream_t stream) {
  WaveScalars s;
  s.threshold = threshold;
  return launch_single(d, false, s, stream);
}

cudaError_t launch_adjoint_states(DeviceScenario& d, const WaveScalars& s, cudaStream_t stream) {
  return launch_single(d, true, s, stream);
}

}  // namespace ct
