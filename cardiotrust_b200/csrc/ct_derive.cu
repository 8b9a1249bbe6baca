// Parameter gradients of one beat: a sweep over its stored rows, one thread per (voxel, offset) item.
//
// Reference mode: the per-step accumulation of calculate_step_derivatives
// (src/core/algorithm/refinement/derivation.rs:173-229) run for all steps of the beat after the
// forward pass. The reference derivative at step t uses only quantities of steps <= t (the
// all-pass outputs of t and t-1, the states x[t] and x[t-d], the mapped residuals of t) and never
// feeds the states, so every item is an independent sequential sweep over t once the states and
// mapped residuals of the beat exist: the three all-pass / fir / iir chains (v, n, b), the nine gain
// derivatives dG[3v+a, 3n+b] and the coefficient derivative dC[v, n].
//
// Rounding follows the reference exactly (-fmad=false, fmaf where the reference calls mul_add, the
// same operand order), so for identical mapped residuals the gradients are bit-identical to the CPU loop:
//   gains     dG += ap * fma(mr, mse/M, maxreg * reg)                 derivation.rs:307-329
//   textbook  fir = fma(-c, fir, x[t-d]) ; iir = fma(-c, iir, ap_last) derivation.rs:418-465
//             dC += fma((fir - iir) * g * mr, mse/M, diff * delta^5)   derivation.rs:467-498
//   simple    dC += fma((x[t-d] - ap_last) * g * mr, mse/M, diff * delta^5)  derivation.rs:346-395
//   maxreg    f = |x0|+|x1|+|x2| - thr if positive, times signum(x_a)  derivation.rs:509-535
// The dC update visits (a, b) in the reference's row-major (state, column) order.
//
// Adjoint mode: the gradients of the stated loss from its state gradient lx (ct_wave.cu):
//   dG[3v+a, 3n+b] = sum_t lx[t, 3v+a] ap[t][b]
//   dC[v, n]       = sum_t sum_b (sum_a g[3v+a, 3n+b] lx[t, 3v+a]) z[t][b],
//   z[t] = dap[t]/dc = (x[t-d] - ap[t-1]) - c z[t-1]
// The tangent z runs forward in time like ap itself, so neither the adjoint chain nor the
// all-pass history has to be stored or recomputed for the coefficients.
//
// What bounds it: FP32 issue (69 operations per item-step in textbook mode, 33 in adjoint mode, of 89 and
// 48 instructions), and the waits of a block's warps for each other at each chunk.
// Layout: a CTA owns up to 8 consecutive voxels (4 x 2 neighbours in y and z inside a grid), 208 items. The history
// that the items gather comes from a ring of rows in shared memory, one 16-byte entry {x0, x1, x2, -} per halo voxel,
// staged by cp.async one chunk of 8 steps ahead; thread e works on voxel e mod 8, offset e / 8, and a voxel's slot has
// (slot mod 8) = (2 y + z) mod 8, so a quarter warp's eight entries lie in eight different bank groups. The factor
// fma(mr, mse/M, maxreg * reg) is the same for a voxel's 26 offsets and is formed once per (voxel, step). Blocks end
// early where their halo would not fit. Where a block's delays spread too far for the ring (a tissue of less than 0.25
// m/s at 2.5 mm and 2 kHz) its items read the rows from global memory, two steps ahead; that way has a kernel of its
// own (ANY), launched where the host's bounds do not rule it out, and a loop with registers of its own. 20x20x20
// cuboid, T = 1,000, 0.2 m/s everywhere: 1.42 ms with each read waiting for its answer, 1.35 one step ahead, 1.14 so,
// 1.05 four ahead, which is slower where the rows are scattered (shell of 47,264 voxels, T = 500, each pair's delay
// drawn from 8 to 60: 4.23, 4.01, 3.66 and 3.89; by cp.async into the ring's place, eight ahead, 1.21 and 4.76); one
// thread per item took 1.19 and 3.07 there. A slow layer in that shell: 2.42, now 2.34. Without that way the other
// blocks' kernel is smaller: 0.787 -> 0.777 on the cuboid at 0.6 m/s. Three CTAs per SM with 80 registers and 112 slots
// beat four with 72 and 96, which keep some values in local memory and cut more blocks. 20x20x20 cuboid, T = 2,000,
// textbook: 2.28 ms with one thread per item gathering single floats through L1, 1.83 with four CTAs and blocks of
// exactly 8 voxels, 1.66 with addresses that do not wrap inside a chunk, 1.56 so. Ellipsoidal shell of 47,264 voxels, T
// = 4,000, adjoint sweep: 15, then 7.3. (Two items per thread in paired multiply-adds, 16 voxels per block: 1.77 and
// 7.6; a pair of FP32 operations with three operands takes 2.4 cycles. Two mbarriers instead of the CTA barrier, so
// that warps may be steps apart: 1.70.)
#include <cuda_runtime.h>

#include <type_traits>

#include "ct_internal.cuh"

namespace ct {
namespace {

constexpr int kVox = kSweepVoxels;
constexpr int kThreads = kVox * kOffsets;  // 208
constexpr int kSlots = kSweepHaloMax;      // per ring row; the last one stays zero
constexpr int kRows = 32;   // power of two
constexpr int kRowBytes = kSlots * 16;
constexpr int kChunk = 8;   // steps staged together
constexpr int kAhead = 2;   // steps that a block without a ring reads ahead, divides kChunk
static_assert(kSweepRingSpread + 2 * kChunk <= kRows && kChunk % kAhead == 0, "a block's history fits the ring");
constexpr int kCols = (3 * (kSlots - 1) + kThreads - 1) / kThreads;  // halo words per thread and row

enum { kTextbook = 0, kSimple = 1, kAdjoint = 2 };

struct SweepArgs {
  int V, S, T;
  const int32_t* nbr;
  const float* coefs;
  const int32_t* delays;
  const float* init_delays;
  const float* gains;
  const float* X;
  const float* rows;  // reference: mapped residuals MR; adjoint: LX
  float* dG;
  float* dC;
  float* fir;
  float* iir;
  int32_t* status;
  int blocks;
  const int32_t* start;  // [blocks + 1] first voxel of each block
  const int32_t* halo;   // [blocks, kSlots] voxels of the halo
  const int16_t* hpos;   // [blocks, kSlots] their slots
  const int16_t* hslot;  // [blocks, kVox * 26], slot of the item's neighbour, kZero if absent
  const int32_t* nhalo;  // [blocks] voxels of the halo, -1 if it is too large
  const int32_t* range;  // [blocks, 2] smallest and largest delay of the block's connected items
  DeriveScalars s;
  int simple;
  bool any;
};

struct SweepSmem {
  float4 ring[kRows][kSlots];
  float4 x[3][kChunk][kVox];    // the voxels' states (reference mode)
  float4 row[3][kChunk][kVox];  // mapped residuals or lx
  float4 q[2][kChunk][kVox];    // reference mode: fma(mr, mse/M, maxreg * reg)
};
static_assert(sizeof(SweepSmem) <= 233472 / kSweepPerSm - 1024, "blocks per SM");

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// What a thread keeps through the sweep.
struct Item {
  float g[3][3], dG[3][3], sG[3][3];
  float ap[3], prev[3], fir[3], iir[3];  // adjoint: fir is the tangent z
  float c, minus_fir, minus_iir, dr_dd, mse, dC, sC;
  bool valid;
};

// One step of an item. in: its delayed input (zero before the beat); r: the voxel's mapped residuals or lx; q:
// their factor of the gain gradients; on: t >= d.
template <int MODE, bool GAINS, bool COEFS>
__device__ __forceinline__ void sweep_step(Item& k, const float (&in)[3], const float (&r)[3], const float (&q)[3], bool on) {
  constexpr bool kAdj = MODE == kAdjoint;
  float last[3];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    last[b] = k.ap[b];
    k.ap[b] = fmaf(k.c, in[b] - k.ap[b], k.prev[b]);
    k.prev[b] = in[b];
  }
  if (GAINS) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (kAdj)
          k.sG[a][b] = fmaf(q[a], k.ap[b], k.sG[a][b]);
        else
          k.dG[a][b] = k.dG[a][b] + k.ap[b] * q[a];
      }
  }
  if (!COEFS) return;
  if (kAdj) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      k.fir[b] = fmaf(-k.c, k.fir[b], in[b] - last[b]);
      const float gl = fmaf(k.g[2][b], r[2], fmaf(k.g[1][b], r[1], k.g[0][b] * r[0]));
      k.sC = fmaf(gl, k.fir[b], k.sC);
    }
    return;
  }
  float u[3];
  if (MODE == kTextbook) {
    if (on) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        k.fir[b] = fmaf(k.minus_fir, k.fir[b], in[b]);
        k.iir[b] = fmaf(k.minus_iir, k.iir[b], last[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b) u[b] = k.fir[b] - k.iir[b];
  } else {
#pragma unroll
    for (int b = 0; b < 3; ++b) u[b] = in[b] - last[b];
  }
  if (MODE == kTextbook || (k.valid && on)) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) k.dC = k.dC + fmaf(u[b] * k.g[a][b] * r[a], k.mse, k.dr_dd);
  }
}

// MODE, which of the two gradients are wanted, and whether blocks may come whose delays do not fit the ring.
template <int MODE, bool GAINS, bool COEFS, bool ANY>
__global__ void __launch_bounds__(kThreads, kSweepPerSm) sweep_kernel(const __grid_constant__ SweepArgs p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepSmem& sm = *reinterpret_cast<SweepSmem*>(smem_raw);
  constexpr bool kAdj = MODE == kAdjoint;
  constexpr bool kNeedQ = !kAdj && GAINS;
  const int tid = threadIdx.x;
  const int v0 = p.start[blockIdx.x], nv = p.start[blockIdx.x + 1] - v0;
  const int vl = tid % kVox, n = tid / kVox;
  const bool live = vl < nv;
  const int v = live ? v0 + vl : v0;
  const int T = p.T, S = p.S;
  const int64_t idx = (int64_t)v * kOffsets + n;
  const int32_t nb = p.nbr[idx];
  const int d = p.delays[idx];
  const float c_own = p.coefs[idx];
  Item k;
  k.valid = live && nb >= 0;
  k.c = k.valid ? c_own : 0.0f;
  k.minus_fir = k.valid ? -c_own : 0.0f;
  k.minus_iir = -c_own;
  k.mse = p.s.mse_scaling;

  // the block's own delays decide what its ring holds: a slow or fast layer of tissue leaves the others their rings
  int dmin = p.range[2 * blockIdx.x], dmax = p.range[2 * blockIdx.x + 1];
  if (dmin > dmax) dmin = dmax = 1;  // no connected pair
  if (dmin < 1) dmin = 1;
  const int nh = p.nhalo[blockIdx.x];
  const bool fits = (int64_t)dmax - dmin <= kSweepRingSpread && nh >= 0;
  if (!ANY && !fits) {
    if (tid == 0) atomicCAS(p.status, 0, (int32_t)CT_ERR_NOT_SUPPORTED);
    return;
  }
  const bool ring = !ANY || fits;
  const int late = k.valid ? d - dmin : 0;  // how far behind the newest row the item reads
  // from here on t >= d holds (for absent items too: their stored delay gates nothing but zeros)
  const int settled = MODE == kTextbook ? max(dmax, d) : dmax;

  // delay_delta^5 (powi(5) = x * ((x*x)*(x*x)))
  const float delay = (float)d + (1.0f - c_own) / (c_own + 1.0f);
  const float dx = p.init_delays[idx] - delay;
  const float dx2 = dx * dx;
  const float dx4 = dx2 * dx2;
  k.dr_dd = p.s.diffreg * (dx * dx4);

  k.dC = k.sC = 0.0f;
#pragma unroll
  for (int b = 0; b < 3; ++b) k.ap[b] = k.prev[b] = k.fir[b] = k.iir[b] = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const size_t o = (size_t)(3 * v + a) * kGainCols + 3 * n + b;
      if (COEFS) k.g[a][b] = p.gains[o];
      if (GAINS) k.dG[a][b] = kAdj ? 0.0f : p.dG[o];
      k.sG[a][b] = 0.0f;
    }
  if (COEFS && !kAdj) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      k.fir[b] = p.fir[(size_t)v * kGainCols + 3 * n + b];
      k.iir[b] = p.iir[(size_t)v * kGainCols + 3 * n + b];
    }
    k.dC = p.dC[idx];
  }

  // Staging: this thread's halo words (column of X, address in ring row 0) and its word of the own rows. Row r
  // lies at ring position (r + dmin) mod kRows, so that a chunk's rows do not wrap.
  int col[kCols];
  uint32_t dst[kCols];
  const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(&sm.ring[0][0]);
#pragma unroll
  for (int i = 0; i < kCols; ++i) {
    const int w = tid + i * kThreads, s = w / 3, b = w - 3 * s;
    const bool ok = ring && s < nh;
    const size_t e = (size_t)blockIdx.x * kSlots + (ok ? s : 0);
    col[i] = ok ? 3 * p.halo[e] + b : -1;
    dst[i] = ring0 + 4u * (4u * p.hpos[e] + b);
  }
  auto stage_history = [&](int t0) {  // the rows that the chunk at t0 adds; rows before the beat stay zero
    if (t0 >= T) return;
    const int lo = t0 - dmin;
    const uint32_t at = (uint32_t)(t0 & (kRows - 1)) * kRowBytes;
#pragma unroll
    for (int i = 0; i < kCols; ++i) {
      if (col[i] < 0) continue;
      const float* from = p.X + (int64_t)lo * S + col[i];
      if (lo >= 0 && t0 + kChunk <= T) {
#pragma unroll
        for (int j = 0; j < kChunk; ++j, from += S) cp_async4(dst[i] + at + j * kRowBytes, from);
      } else {
        for (int j = 0; j < min(kChunk, T - t0); ++j, from += S)
          if (lo + j >= 0) cp_async4(dst[i] + at + j * kRowBytes, from);
      }
    }
  };
  const int own_s = tid / (3 * kVox), own_w = tid % (3 * kVox);  // 192 words per chunk, one per thread
  const bool own = tid < kChunk * 3 * kVox && own_w < 3 * nv;
  const uint32_t own_dst = 4u * (uint32_t)(4 * (own_s * kVox + own_w / 3) + own_w % 3);
  const uint32_t x0 = (uint32_t)__cvta_generic_to_shared(&sm.x[0][0][0]);
  const uint32_t row0 = (uint32_t)__cvta_generic_to_shared(&sm.row[0][0][0]);
  constexpr uint32_t kOwnBytes = sizeof(sm.x[0]);
  int64_t own_at = (int64_t)own_s * S + 3 * v0 + own_w;  // moves on a chunk with every call
  auto stage_own = [&](int t0, int buf) {
    const int64_t at = own_at;
    own_at += (int64_t)kChunk * S;
    if (!own || t0 + own_s >= T) return;
    cp_async4(row0 + buf * kOwnBytes + own_dst, p.rows + at);
    if (kNeedQ) cp_async4(x0 + buf * kOwnBytes + own_dst, p.X + at);
  };
  const float reg_s = p.s.reg_scaling, thr = p.s.threshold;
  auto factors = [&](int buf, int to) {  // one (step, voxel) each, on two warps that stage less
    constexpr int kFirst = 128;
    if (!kNeedQ || tid < kFirst || tid >= kFirst + kChunk * kVox) return;
    const int s = (tid - kFirst) / kVox, w = tid % kVox;
    const float4 x4 = sm.x[buf][s][w], m4 = sm.row[buf][s][w];
    const float x[3] = {x4.x, x4.y, x4.z}, m[3] = {m4.x, m4.y, m4.z};
    const float sum = fabsf(x[0]) + fabsf(x[1]) + fabsf(x[2]);
    const bool over = sum > thr;
    const float f = sum - thr;
    float q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float mreg = over ? f * copysignf(1.0f, x[a]) : 0.0f;
      q[a] = fmaf(m[a], k.mse, mreg * reg_s);
    }
    sm.q[to][s][w] = make_float4(q[0], q[1], q[2], 0.0f);
  };

  // slots no halo voxel owns (the zero slot among them) stay zero; so do the rows of voxels beyond V
  for (int e = tid; e < (int)(sizeof(SweepSmem) / 16); e += kThreads)
    reinterpret_cast<float4*>(smem_raw)[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();

  // Pipeline per chunk: the history arrives one chunk ahead, the voxels' own rows two, and their factors are
  // formed one ahead, so that one barrier per chunk is enough.
  stage_own(0, 0);
  stage_history(0);
  cp_async_commit();
  stage_own(kChunk, 1);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  factors(0, 0);
  // address of the neighbour in ring row 0; without a ring its column of X
  const uint32_t slot = ring ? ring0 + 16u * (uint32_t)p.hslot[(size_t)blockIdx.x * kThreads + vl * kOffsets + n] : 3u * (uint32_t)max(nb, 0);
  auto gather = [&](int t, float (&x)[3]) {
    const bool on = k.valid && t >= d && t < T;
    const float* from = p.X + (int64_t)(t - d) * S + slot;
#pragma unroll
    for (int b = 0; b < 3; ++b) x[b] = on ? __ldg(from + b) : 0.0f;
  };
  // with and without a ring, each with registers of its own
  auto steps = [&](auto with_ring) {
    constexpr bool kRing = decltype(with_ring)::value;
    int buf = 0;  // t0 / kChunk mod 3
    for (int t0 = 0; t0 < T; t0 += kChunk) {
      float ahead[kAhead][3];  // without a ring: the next steps' inputs, under way over the barrier and the steps before
      if (!kRing) {
#pragma unroll
        for (int s = 0; s < kAhead; ++s) gather(t0 + s, ahead[s]);
      }
      cp_async_wait<0>();
      // this chunk's history, factors and the next chunk's own rows are there for all; the previous chunk's
      // buffers and the ring rows older than t0 - dmax are free (kRows >= spread + 2 chunks)
      __syncthreads();
      const int next = buf == 2 ? 0 : buf + 1, after = next == 2 ? 0 : next + 1;
      if (kRing) stage_history(t0 + kChunk);
      stage_own(t0 + 2 * kChunk, after);
      cp_async_commit();
      if (t0 + kChunk < T) factors(next, ((t0 / kChunk) + 1) & 1);
      const float4* rows = &sm.row[buf][0][vl];
      const float4* facs = &sm.q[(t0 / kChunk) & 1][0][vl];
      const int tn = min(kChunk, T - t0);
      auto one = [&](int s, const float (&in)[3], bool on) {
        const float4 r4 = rows[s * kVox];
        const float r[3] = {r4.x, r4.y, r4.z};
        float q[3] = {r[0], r[1], r[2]};
        if (kNeedQ) {
          const float4 q4 = facs[s * kVox];
          q[0] = q4.x;
          q[1] = q4.y;
          q[2] = q4.z;
        }
        sweep_step<MODE, GAINS, COEFS>(k, in, r, q, on);
      };
      if (kRing && tn == kChunk && t0 >= settled) {
        // the chunk's rows are consecutive but for one wrap: an immediate offset from one of two addresses
        const int first = (t0 - late) & (kRows - 1);
        const uint32_t low = slot + (uint32_t)first * kRowBytes, high = low - kRows * kRowBytes;
#pragma unroll
        for (int s = 0; s < kChunk; ++s) {
          const uint32_t at = (first + s >= kRows ? high : low) + s * kRowBytes;
          float in[3];
          float pad;
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(in[0]), "=f"(in[1]), "=f"(in[2]), "=f"(pad) : "r"(at));
          one(s, in, true);
        }
      } else if (kRing) {
        for (int s = 0; s < tn; ++s) {
          const int t = t0 + s;
          const float4 h = *reinterpret_cast<const float4*>(smem_raw + (slot - ring0) + (uint32_t)((t - late) & (kRows - 1)) * kRowBytes);
          const float in[3] = {h.x, h.y, h.z};
          one(s, in, t >= d);
        }
      } else {
#pragma unroll 1
        for (int s0 = 0; s0 < tn; s0 += kAhead) {
#pragma unroll
          for (int i = 0; i < kAhead; ++i) {
            const int t = t0 + s0 + i;
            if (t >= T) break;
            const float in[3] = {ahead[i][0], ahead[i][1], ahead[i][2]};
            if (s0 + kAhead < kChunk) gather(t + kAhead, ahead[i]);
            one(s0 + i, in, t >= d);
          }
        }
      }
      if (kAdj) {
        // chunk sums into the totals: the error of a long sum stays that of its T / 8 partial sums
        if (GAINS) {
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              k.dG[a][b] = k.dG[a][b] + k.sG[a][b];
              k.sG[a][b] = 0.0f;
            }
        }
        k.dC = k.dC + k.sC;
        k.sC = 0.0f;
      }
      buf = next;
    }
  };
  if (ring)
    steps(std::true_type{});
  else
    steps(std::false_type{});
  const int w = p.start[blockIdx.x] + vl;  // the voxel, read again rather than kept in a register
  if (w >= p.start[blockIdx.x + 1]) return;
  if (GAINS) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        float* o = p.dG + (size_t)(3 * w + a) * kGainCols + 3 * n + b;
        if (!kAdj)
          *o = k.dG[a][b];
        else if (k.valid)
          *o = *o + k.dG[a][b];
      }
  }
  if (COEFS) {
    if (kAdj) {
      float count = 9.0f * (float)T;
      if (p.simple) count = k.valid ? 9.0f * (float)max(0, T - d) : 0.0f;
      const float sum = (k.valid ? k.dC : 0.0f) + count * k.dr_dd;
      p.dC[(int64_t)w * kOffsets + n] = p.dC[(int64_t)w * kOffsets + n] + sum;
    } else {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        p.fir[(size_t)w * kGainCols + 3 * n + b] = k.fir[b];
        p.iir[(size_t)w * kGainCols + 3 * n + b] = k.iir[b];
      }
      p.dC[(int64_t)w * kOffsets + n] = k.dC;
    }
  }
}

template <int MODE, bool GAINS, bool COEFS, bool ANY>
cudaError_t launch_form(const SweepArgs& a, cudaStream_t stream) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  static bool done[128] = {};
  if (device < 0 || device >= 128) return cudaErrorInvalidValue;
  if (!done[device]) {
    err = cudaFuncSetAttribute(sweep_kernel<MODE, GAINS, COEFS, ANY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(SweepSmem));
    if (err != cudaSuccess) return err;
    done[device] = true;
  }
  sweep_kernel<MODE, GAINS, COEFS, ANY><<<(unsigned)a.blocks, kThreads, sizeof(SweepSmem), stream>>>(a);
  return cudaGetLastError();
}
template <int MODE, bool GAINS, bool COEFS>
cudaError_t launch(const SweepArgs& a, cudaStream_t stream) {
  return a.any ? launch_form<MODE, GAINS, COEFS, true>(a, stream) : launch_form<MODE, GAINS, COEFS, false>(a, stream);
}

template <int MODE>
cudaError_t launch_mode(const SweepArgs& a, cudaStream_t stream) {
  if (a.s.freeze_delays) return launch<MODE == kAdjoint ? kAdjoint : kTextbook, true, false>(a, stream);
  if (a.s.freeze_gains) return launch<MODE, false, true>(a, stream);
  return launch<MODE, true, true>(a, stream);
}

SweepArgs sweep_args(DeviceScenario& d, const DeriveScalars& s) {
  SweepArgs a;
  a.V = (int)d.V;
  a.S = (int)d.S;
  a.T = (int)d.T;
  a.nbr = d.nbr;
  a.coefs = d.coefs;
  a.delays = d.delays;
  a.init_delays = d.init_delays;
  a.gains = d.gains;
  a.X = d.X;
  a.rows = d.MR;
  a.dG = d.dG;
  a.dC = d.dC;
  a.fir = d.fir;
  a.iir = d.iir;
  a.status = d.status;
  a.any = d.sweep_any;
  a.blocks = d.sweep_blocks;
  a.start = d.sstart;
  a.halo = d.shalo;
  a.hpos = d.shpos;
  a.hslot = d.shslot;
  a.nhalo = d.snhalo;
  a.range = d.srange;
  a.s = s;
  a.simple = s.ap_derivative == CT_AP_SIMPLE;
  return a;
}

}  // namespace

cudaError_t launch_derive(DeviceScenario& d, const DeriveScalars& s, cudaStream_t stream) {
  const SweepArgs a = sweep_args(d, s);
  return s.ap_derivative == CT_AP_SIMPLE ? launch_mode<kSimple>(a, stream) : launch_mode<kTextbook>(a, stream);
}

cudaError_t launch_adjoint_gradients(DeviceScenario& d, const DeriveScalars& s, cudaStream_t stream) {
  SweepArgs a = sweep_args(d, s);
  a.rows = d.LX;
  return launch_mode<kAdjoint>(a, stream);
}

}  // namespace ct
