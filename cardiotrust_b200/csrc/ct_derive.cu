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
// What bounds it: FP32 issue (69 operations per item-step in textbook mode, 30 in adjoint mode).
// Layout: a CTA owns 8 voxels (4 x 2 neighbours in y and z), 208 items, four CTAs per SM. The history that
// the items gather comes from a ring of rows in shared memory, one 16-byte entry {x0, x1, x2, -}
// per halo voxel, staged by cp.async one chunk of 8 steps ahead; thread e works on voxel e mod 8, offset
// e / 8, and a voxel's slot has (slot mod 8) = (2 y + z) mod 8, so a quarter warp's eight entries lie in
// eight different bank groups. The factor fma(mr, mse/M, maxreg * reg) is the same for a voxel's 26
// offsets and is formed once per (voxel, step). (One thread per item gathering single floats through L1
// issued 161 instructions per item-step: 2.28 ms on the 20x20x20 cuboid, T = 2,000.) Items whose delays spread
// too far for the ring, or whose halo is too large, read the rows from global memory.
#include <cuda_runtime.h>

#include "ct_internal.cuh"

namespace ct {
namespace {

constexpr int kVox = kSweepVoxels;
constexpr int kThreads = kVox * kOffsets;  // 208
constexpr int kSlots = kSweepHaloMax;      // per ring row; the last one stays zero
constexpr int kZero = kSlots - 1;
constexpr int kRows = 32;   // power of two
constexpr int kChunk = 8;   // steps staged together
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
  const int32_t* halo;   // [blocks, kSlots] voxels of the halo
  const int16_t* hpos;   // [blocks, kSlots] their slots
  const int16_t* hslot;  // [blocks, kVox * 26], slot of the item's neighbour, kZero if absent
  const int32_t* nhalo;  // [blocks], -1 if the halo is too large
  const int32_t* dmin;   // [2]
  DeriveScalars s;
  int simple;
};

struct SweepSmem {
  float4 ring[kRows][kSlots];
  float4 x[2][kChunk][kVox];    // the voxels' states (reference mode)
  float4 row[2][kChunk][kVox];  // mapped residuals or lx
  float4 q[kChunk][kVox];       // reference mode: fma(mr, mse/M, maxreg * reg)
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// MODE, and which of the two gradients are wanted.
template <int MODE, bool GAINS, bool COEFS>
__global__ void __launch_bounds__(kThreads, 4) sweep_kernel(const SweepArgs p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepSmem& sm = *reinterpret_cast<SweepSmem*>(smem_raw);
  constexpr bool kAdj = MODE == kAdjoint;
  const int tid = threadIdx.x;
  const int v0 = blockIdx.x * kVox;
  const int vl = tid % kVox, n = tid / kVox;
  const bool live = v0 + vl < p.V;
  const int v = live ? v0 + vl : v0;
  const int T = p.T, S = p.S;
  const int64_t idx = (int64_t)v * kOffsets + n;
  const int32_t nb = p.nbr[idx];
  const bool valid = live && nb >= 0;
  const int d = p.delays[idx];
  const float c_own = p.coefs[idx];
  const float c = valid ? c_own : 0.0f;
  const float minus_fir = valid ? -c_own : 0.0f, minus_iir = -c_own;

  int dmin = p.dmin[0], dmax = p.dmin[1];
  if (dmin > dmax) dmin = dmax = 1;  // no connected pair
  if (dmin < 1) dmin = 1;
  const int nh = p.nhalo[blockIdx.x];
  const bool ring = nh >= 0 && (int64_t)dmax - dmin + 2 * kChunk <= kRows;
  const int slot = ring ? p.hslot[(size_t)blockIdx.x * kThreads + vl * kOffsets + n] : 0;
  const int dr = valid ? d : dmin;  // the delay that the ring row follows

  // delay_delta^5 (powi(5) = x * ((x*x)*(x*x)))
  const float delay = (float)d + (1.0f - c_own) / (c_own + 1.0f);
  const float dx = p.init_delays[idx] - delay;
  const float dx2 = dx * dx;
  const float dx4 = dx2 * dx2;
  const float dr_dd = p.s.diffreg * (dx * dx4);
  const float mse_s = p.s.mse_scaling, reg_s = p.s.reg_scaling, thr = p.s.threshold;

  float g[3][3], dG[3][3], sG[3][3];
  float ap[3] = {0.0f, 0.0f, 0.0f}, prev[3] = {0.0f, 0.0f, 0.0f};
  float fir[3] = {0.0f, 0.0f, 0.0f}, iir[3] = {0.0f, 0.0f, 0.0f};  // adjoint: fir is the tangent z
  float dC = 0.0f, sC = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const size_t o = (size_t)(3 * v + a) * kGainCols + 3 * n + b;
      if (COEFS) g[a][b] = p.gains[o];
      if (GAINS) dG[a][b] = kAdj ? 0.0f : p.dG[o];
      sG[a][b] = 0.0f;
    }
  if (COEFS && !kAdj) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      fir[b] = p.fir[(size_t)v * kGainCols + 3 * n + b];
      iir[b] = p.iir[(size_t)v * kGainCols + 3 * n + b];
    }
    dC = p.dC[idx];
  }

  // staging: this thread's halo words (column of X, offset in a ring row) and its own-row words
  int col[kCols], dst[kCols];
#pragma unroll
  for (int i = 0; i < kCols; ++i) {
    const int w = tid + i * kThreads, s = w / 3, b = w - 3 * s;
    const bool ok = ring && s < nh;
    const size_t e = (size_t)blockIdx.x * kSlots + (ok ? s : 0);
    col[i] = ok ? 3 * p.halo[e] + b : -1;
    dst[i] = 4 * p.hpos[e] + b;
  }
  const int nv = min(kVox, p.V - v0);
  auto stage = [&](int t0) {
    const int buf = (t0 / kChunk) & 1;
    const int tn = min(kChunk, T - t0);
    if (ring) {
      const int lo = t0 == 0 ? -dmax : t0 - dmin, hi = t0 + tn - 1 - dmin;
      for (int r = lo; r <= hi; ++r) {
        float* to = reinterpret_cast<float*>(sm.ring[r & (kRows - 1)]);
        const float* from = p.X + (int64_t)r * S;
#pragma unroll
        for (int i = 0; i < kCols; ++i) {
          if (col[i] < 0) continue;
          if (r < 0)
            to[dst[i]] = 0.0f;
          else
            cp_async4(to + dst[i], from + col[i]);
        }
      }
    }
    // the voxels' own rows: 3 nv words per step
    for (int e = tid; e < tn * 3 * kVox; e += kThreads) {
      const int s = e / (3 * kVox), w = e - s * (3 * kVox);
      if (w >= 3 * nv) continue;
      const size_t o = (size_t)(t0 + s) * S + 3 * v0 + w;
      cp_async4(reinterpret_cast<float*>(&sm.row[buf][s][w / 3]) + w % 3, p.rows + o);
      if (!kAdj) cp_async4(reinterpret_cast<float*>(&sm.x[buf][s][w / 3]) + w % 3, p.X + o);
    }
    cp_async_commit();
  };

  // slots no halo voxel owns (the zero slot among them) stay zero; so do the rows of voxels beyond V
  for (int e = tid; e < kRows * kSlots; e += kThreads) (&sm.ring[0][0])[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int e = tid; e < 2 * kChunk * kVox; e += kThreads) {
    (&sm.x[0][0][0])[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    (&sm.row[0][0][0])[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  __syncthreads();

  stage(0);
  for (int t0 = 0; t0 < T; t0 += kChunk) {
    const int tn = min(kChunk, T - t0);
    const int buf = (t0 / kChunk) & 1;
    // the next chunk's rows overwrite ring rows older than t0 - dmax (kRows >= spread + 2 chunks) and
    // the buffer that the previous chunk read (the barrier at its end)
    if (t0 + kChunk < T) {
      stage(t0 + kChunk);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (!kAdj && GAINS) {
      if (tid < tn * kVox) {
        const int s = tid / kVox, w = tid % kVox;
        const float4 x4 = sm.x[buf][s][w], m4 = sm.row[buf][s][w];
        const float x[3] = {x4.x, x4.y, x4.z}, m[3] = {m4.x, m4.y, m4.z};
        const float sum = fabsf(x[0]) + fabsf(x[1]) + fabsf(x[2]);
        const bool over = sum > thr;
        const float f = sum - thr;
        float q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float mreg = over ? f * copysignf(1.0f, x[a]) : 0.0f;
          q[a] = fmaf(m[a], mse_s, mreg * reg_s);
        }
        sm.q[s][w] = make_float4(q[0], q[1], q[2], 0.0f);
      }
      __syncthreads();
    }
    auto step = [&](int s, bool on) {  // on: t >= d
      const int t = t0 + s;
      float in[3];
      if (ring) {
        const float4 h = sm.ring[(t - dr) & (kRows - 1)][slot];
        in[0] = h.x;
        in[1] = h.y;
        in[2] = h.z;
      } else {
#pragma unroll
        for (int b = 0; b < 3; ++b) in[b] = (valid && t >= d) ? __ldg(p.X + (int64_t)(t - d) * S + 3 * nb + b) : 0.0f;
      }
      float last[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        last[b] = ap[b];
        ap[b] = fmaf(c, in[b] - ap[b], prev[b]);
        prev[b] = in[b];
      }
      const float4 r4 = sm.row[buf][s][vl];
      const float r[3] = {r4.x, r4.y, r4.z};
      if (GAINS) {
        float q[3] = {r[0], r[1], r[2]};
        if (!kAdj) {
          const float4 q4 = sm.q[s][vl];
          q[0] = q4.x;
          q[1] = q4.y;
          q[2] = q4.z;
        }
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            if (kAdj)
              sG[a][b] = fmaf(q[a], ap[b], sG[a][b]);
            else
              dG[a][b] = dG[a][b] + ap[b] * q[a];
          }
      }
      if (COEFS) {
        if (kAdj) {
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            fir[b] = fmaf(-c, fir[b], in[b] - last[b]);
            const float gl = fmaf(g[2][b], r[2], fmaf(g[1][b], r[1], g[0][b] * r[0]));
            sC = fmaf(gl, fir[b], sC);
          }
        } else {
          float u[3];
          if (MODE == kTextbook) {
            if (on) {
#pragma unroll
              for (int b = 0; b < 3; ++b) {
                fir[b] = fmaf(minus_fir, fir[b], in[b]);
                iir[b] = fmaf(minus_iir, iir[b], last[b]);
              }
            }
#pragma unroll
            for (int b = 0; b < 3; ++b) u[b] = fir[b] - iir[b];
          } else {
#pragma unroll
            for (int b = 0; b < 3; ++b) u[b] = in[b] - last[b];
          }
          if (MODE == kTextbook || (valid && on)) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
              for (int b = 0; b < 3; ++b) dC = dC + fmaf(u[b] * g[a][b] * r[a], mse_s, dr_dd);
          }
        }
      }
    };
    // past every delay (of absent items too: their stored delay gates nothing but zeros)
    if (tn == kChunk && t0 >= dmax && (MODE != kTextbook || valid || d <= t0)) {
#pragma unroll 4
      for (int s = 0; s < kChunk; ++s) step(s, true);
    } else {
      for (int s = 0; s < tn; ++s) step(s, t0 + s >= d);
    }
    if (kAdj) {
      // chunk sums into the totals: the error of a long sum stays that of its T / 8 partial sums
      if (GAINS) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            dG[a][b] = dG[a][b] + sG[a][b];
            sG[a][b] = 0.0f;
          }
      }
      dC = dC + sC;
      sC = 0.0f;
    }
    __syncthreads();
  }
  if (!live) return;
  if (GAINS) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        float* o = p.dG + (size_t)(3 * v + a) * kGainCols + 3 * n + b;
        if (!kAdj)
          *o = dG[a][b];
        else if (valid)
          *o = *o + dG[a][b];
      }
  }
  if (COEFS) {
    if (kAdj) {
      float count = 9.0f * (float)T;
      if (p.simple) count = valid ? 9.0f * (float)max(0, T - d) : 0.0f;
      const float sum = (valid ? dC : 0.0f) + count * dr_dd;
      p.dC[idx] = p.dC[idx] + sum;
    } else {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        p.fir[(size_t)v * kGainCols + 3 * n + b] = fir[b];
        p.iir[(size_t)v * kGainCols + 3 * n + b] = iir[b];
      }
      p.dC[idx] = dC;
    }
  }
}

template <int MODE, bool GAINS, bool COEFS>
cudaError_t launch(const SweepArgs& a, cudaStream_t stream) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  static bool done[128] = {};
  if (device < 0 || device >= 128) return cudaErrorInvalidValue;
  if (!done[device]) {
    err = cudaFuncSetAttribute(sweep_kernel<MODE, GAINS, COEFS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(SweepSmem));
    if (err != cudaSuccess) return err;
    done[device] = true;
  }
  const unsigned blocks = (unsigned)((a.V + kVox - 1) / kVox);
  sweep_kernel<MODE, GAINS, COEFS><<<blocks, kThreads, sizeof(SweepSmem), stream>>>(a);
  return cudaGetLastError();
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
  a.halo = d.shalo;
  a.hpos = d.shpos;
  a.hslot = d.shslot;
  a.nhalo = d.snhalo;
  a.dmin = d.dmin;
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
