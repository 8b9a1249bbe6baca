// Measurement products of one beat over all steps:
//   y[t, m]  = sum_s H[beat, m, s] x[t, s]      predict_measurements, prediction.rs:112-130
//   r[t, m]  = y[t, m] - z[beat, t, m]          calculate_residuals, estimation.rs:146-153
//   mr[t, s] = sum_m H[beat, m, s] r[t, m]      calculate_mapped_residuals, derivation.rs:538-551
// plus the per-step MSE metric (metrics.rs:189-190).
//
// Neither product feeds the state recurrence, so each is one GEMM over the
// whole beat instead of T matrix-vector products. The k-order of these sums
// differs from the reference's (ndarray/matrixmultiply), so their results are
// compared with a tolerance. The reductions are deterministic: split-K
// partials are summed in a fixed order.
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "ct_internal.cuh"

namespace ct {
namespace {

constexpr int BK = 16;
constexpr int kPart = 64;  // row and column step of the split-K rule, column multiple of the partials

__device__ __forceinline__ uint64_t twice(float v) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}

// C[m, n] = sum_{k in [k0, k1)} A[m*lda + k] * B(k, n), with B(k, n) at B[n*ldb + k] (kBKContig) or
// B[k*ldb + n]; one fused multiply-add per term, in order of k.
// What bounds it: FP32 issue. A thread computes TM x TN outputs from 16-byte shared-memory reads, two rows per
// instruction (outer products reach 50 TFLOP/s here with scalar multiply-adds and 58 with paired ones); the slabs of 16 k
// that follow are loaded while one is worked on, two ahead for H x, whose blocks are few and long, one for
// H^T r, whose blocks have few slabs. kVec: 16-byte global accesses, where rows and pitches are multiples of
// four floats.
// Forms: H x in 64 x 64 blocks, since its splits (and with them the order of its sums) are counted in such pieces;
// 47,264 voxels, T = 1,000, 111 rows: 3.0 ms with 4 x 4 outputs per thread and loads between two barriers, 1.50 with them
// overlapped, 1.31 with 8 x 4, 1.15 two slabs ahead (32 x 64 blocks 1.38, 64 x 128 1.61). H^T r in 128 x 128 blocks of 16 x 4
// outputs; 6,468 voxels, T = 1,500, 111 rows, three beats: 0.84 ms before, 0.58 with scalar 8 x 8, 0.51 so.
template <bool kBKContig, int BM, int BN, int TM, int TN, bool kVec>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM * TN == 64 ? 2 : 0)
    gemm_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ Bm, int64_t ldb,
                float* __restrict__ C, int64_t ldc, int64_t c_split_stride, int64_t Mrows, int64_t Ncols, int64_t K,
                int64_t kchunk) {
  constexpr int kTx = BN / TN, kThreads = (BM / TM) * kTx;
  constexpr int kRowStep = BM / (TM / 4), kColStep = BN / (TN / 4);  // distance of a thread's groups of four
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Bs[2][BK][BN + 4];
  const int64_t m0 = (int64_t)blockIdx.y * BM;
  const int64_t n0 = (int64_t)blockIdx.x * BN;
  const int64_t k0 = (int64_t)blockIdx.z * kchunk;
  const int64_t k1 = (k0 + kchunk < K) ? k0 + kchunk : K;
  const int tid = threadIdx.x;
  const int tx = tid % kTx, ty = tid / kTx;
  constexpr int kLoadsA = BM * BK / 4 / kThreads, kLoadsB = BN * BK / 4 / kThreads;
  constexpr int kAhead = kBKContig ? 2 : 1;
  float4 ra[kAhead][kLoadsA], rb[kAhead][kLoadsB];
  // four consecutive k of a row (zero past the end)
  auto four_k = [&](const float* base, int64_t ld, int64_t row, int64_t rows, int64_t k) -> float4 {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row >= rows) return v;
    const float* q = base + row * ld + k;
    if (kVec && k + 3 < k1) return *reinterpret_cast<const float4*>(q);
    if (k < k1) v.x = q[0];
    if (k + 1 < k1) v.y = q[1];
    if (k + 2 < k1) v.z = q[2];
    if (k + 3 < k1) v.w = q[3];
    return v;
  };
  auto load = [&](int64_t kb, int set) {
#pragma unroll
    for (int i = 0; i < kLoadsA; ++i) ra[set][i] = four_k(A, lda, m0 + (tid + i * kThreads) / 4, Mrows, kb + 4 * (tid % 4));
#pragma unroll
    for (int i = 0; i < kLoadsB; ++i) {
      if (kBKContig) {
        rb[set][i] = four_k(Bm, ldb, n0 + (tid + i * kThreads) / 4, Ncols, kb + 4 * (tid % 4));
      } else {
        const int e = tid + i * kThreads;
        const int64_t k = kb + e / (BN / 4), n = n0 + 4 * (e % (BN / 4));
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k < k1) {
          const float* q = Bm + k * ldb + n;
          if (kVec && n + 3 < Ncols) {
            v = *reinterpret_cast<const float4*>(q);
          } else {
            if (n < Ncols) v.x = q[0];
            if (n + 1 < Ncols) v.y = q[1];
            if (n + 2 < Ncols) v.z = q[2];
            if (n + 3 < Ncols) v.w = q[3];
          }
        }
        rb[set][i] = v;
      }
    }
  };
  auto store = [&](int buf, int set) {
#pragma unroll
    for (int i = 0; i < kLoadsA; ++i) {
      const int r = (tid + i * kThreads) / 4, c = 4 * (tid % 4);
      As[buf][c][r] = ra[set][i].x;
      As[buf][c + 1][r] = ra[set][i].y;
      As[buf][c + 2][r] = ra[set][i].z;
      As[buf][c + 3][r] = ra[set][i].w;
    }
#pragma unroll
    for (int i = 0; i < kLoadsB; ++i) {
      if (kBKContig) {
        const int r = (tid + i * kThreads) / 4, c = 4 * (tid % 4);
        Bs[buf][c][r] = rb[set][i].x;
        Bs[buf][c + 1][r] = rb[set][i].y;
        Bs[buf][c + 2][r] = rb[set][i].z;
        Bs[buf][c + 3][r] = rb[set][i].w;
      } else {
        const int e = tid + i * kThreads;
        *reinterpret_cast<float4*>(&Bs[buf][e / (BN / 4)][4 * (e % (BN / 4))]) = rb[set][i];
      }
    }
  };
  uint64_t acc[TM / 2][TN] = {};  // rows in pairs
  if (k0 < k1) {
    load(k0, 0);
    store(0, 0);
    if (kAhead == 2 && k0 + BK < k1) load(k0 + BK, 1);
  }
  __syncthreads();
  for (int64_t kb = k0; kb < k1; kb += 2 * BK) {
#pragma unroll
    for (int buf = 0; buf < 2; ++buf) {
      const int64_t slab = kb + buf * BK;
      if (slab + kAhead * BK < k1) load(slab + kAhead * BK, buf % kAhead);
      if (slab < k1) {
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
          uint64_t a[TM / 2], b[TN];
#pragma unroll
          for (int h = 0; h < TM / 4; ++h) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&As[buf][kk][kRowStep * h + 4 * ty]);
            a[2 * h] = v.x;
            a[2 * h + 1] = v.y;
          }
#pragma unroll
          for (int h = 0; h < TN / 4; ++h) {
            const float4 v = *reinterpret_cast<const float4*>(&Bs[buf][kk][kColStep * h + 4 * tx]);
            b[4 * h] = twice(v.x);
            b[4 * h + 1] = twice(v.y);
            b[4 * h + 2] = twice(v.z);
            b[4 * h + 3] = twice(v.w);
          }
#pragma unroll
          for (int i = 0; i < TM / 2; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j)
              asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a[i]), "l"(b[j]));
        }
      }
      if (slab + BK < k1) store(buf ^ 1, (buf + 1) % kAhead);
      __syncthreads();
    }
  }
  float* Cz = C + (int64_t)blockIdx.z * c_split_stride;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int64_t gm = m0 + kRowStep * (i / 4) + 4 * ty + i % 4;
    if (gm >= Mrows) continue;
    float row[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) row[j] = __uint_as_float((uint32_t)(acc[i / 2][j] >> (i % 2 * 32)));
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
      const int64_t gn = n0 + kColStep * h + 4 * tx;
      float* q = Cz + gm * ldc + gn;
      if (kVec && gn + 3 < Ncols) {
        *reinterpret_cast<float4*>(q) = make_float4(row[4 * h], row[4 * h + 1], row[4 * h + 2], row[4 * h + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (gn + j < Ncols) q[j] = row[4 * h + j];
      }
    }
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// 16-byte accesses where every row of every operand starts on 16 bytes.
template <bool kBKContig, int BM, int BN, int TM, int TN>
void launch_gemm(const float* A, int64_t lda, const float* B, int64_t ldb, float* C, int64_t ldc, int64_t c_split_stride,
                 int64_t M, int64_t N, int64_t K, int64_t kchunk, int splits, cudaStream_t stream) {
  const bool vec = aligned16(A) && aligned16(B) && aligned16(C) && lda % 4 == 0 && ldb % 4 == 0 && ldc % 4 == 0 &&
                   c_split_stride % 4 == 0;
  const dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM), (unsigned)splits);
  constexpr int kThreads = (BM / TM) * (BN / TN);
  if (vec)
    gemm_kernel<kBKContig, BM, BN, TM, TN, true>
        <<<grid, kThreads, 0, stream>>>(A, lda, B, ldb, C, ldc, c_split_stride, M, N, K, kchunk);
  else
    gemm_kernel<kBKContig, BM, BN, TM, TN, false>
        <<<grid, kThreads, 0, stream>>>(A, lda, B, ldb, C, ldc, c_split_stride, M, N, K, kchunk);
}

// The partial sums of H x in split order.
void launch_partials(const float* X, const float* H, float* part, int64_t T, int64_t S, int64_t M, int64_t mpad,
                     int64_t kchunk, int splits, cudaStream_t stream) {
  launch_gemm<true, 64, 64, 8, 4>(X, S, H, S, part, mpad, T * mpad, T, M, S, kchunk, splits, stream);
}

// Sum split-K partials in split order; write Y[beat], R, and optionally the residuals.
__global__ void reduce_measure_kernel(const float* __restrict__ part, int ksplit, int64_t T, int64_t M, int64_t ldp,
                                      float* __restrict__ Y, const float* __restrict__ Z, float* __restrict__ R) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= T * M) return;
  const int64_t t = idx / M, m = idx - (idx / M) * M;
  float y = 0.0f;
  for (int z = 0; z < ksplit; ++z) y = y + part[((int64_t)z * T + t) * ldp + m];
  Y[idx] = y;
  if (R) R[idx] = y - Z[idx];
}

// loss_mse[t] = sum_m r^2 / M with ndarray's eight-accumulator order (metrics.rs:189-190).
__global__ void mse_kernel(const float* __restrict__ R, int64_t T, int64_t M, float* __restrict__ loss_mse) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  const float* r = R + t * M;
  float p[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int64_t i = 0;
  for (; M - i >= 8; i += 8) {
#pragma unroll
    for (int q = 0; q < 8; ++q) p[q] = p[q] + r[i + q] * r[i + q];
  }
  float acc = 0.0f;
  acc = acc + (p[0] + p[4]);
  acc = acc + (p[1] + p[5]);
  acc = acc + (p[2] + p[6]);
  acc = acc + (p[3] + p[7]);
  for (; i < M; ++i) acc = acc + r[i] * r[i];
  loss_mse[t] = acc / (float)M;
}

}  // namespace

int measure_ksplit(int64_t T, int64_t S, int64_t M, int sms) {
  // two 64 x 64 pieces of a split per SM, at least 256 states per split
  const int64_t pieces = ((M + kPart - 1) / kPart) * ((T + kPart - 1) / kPart);
  int64_t ks = (2 * (int64_t)sms + pieces - 1) / pieces;
  ks = ks < S / 256 ? ks : (S / 256 > 1 ? S / 256 : 1);
  return (int)(ks < 64 ? ks : 64);
}

cudaError_t launch_measure(DeviceScenario& d, int64_t beat, bool with_residuals, cudaStream_t stream) {
  const int64_t T = d.T, M = d.M, S = d.S;
  const float* H = d.H + beat * M * S;
  const int64_t mpad = ((M + kPart - 1) / kPart) * kPart;
  const int64_t kchunk = ((S + d.ksplit - 1) / d.ksplit + BK - 1) / BK * BK;
  launch_partials(d.X, H, d.gemm_part, T, S, M, mpad, kchunk, d.ksplit, stream);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  const int64_t n = T * M;
  reduce_measure_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(
      d.gemm_part, d.ksplit, T, M, mpad, d.Y + beat * T * M, with_residuals ? d.meas + beat * T * M : nullptr,
      with_residuals ? d.R : nullptr);
  err = cudaGetLastError();
  if (err != cudaSuccess || !with_residuals) return err;
  return launch_mse(d, stream);
}

cudaError_t launch_mse(DeviceScenario& d, cudaStream_t stream) {
  mse_kernel<<<(unsigned)((d.T + 127) / 128), 128, 0, stream>>>(d.R, d.T, d.M, d.loss_mse);
  return cudaGetLastError();
}

cudaError_t launch_map_residuals(DeviceScenario& d, int64_t beat, cudaStream_t stream) {
  const int64_t T = d.T, M = d.M, S = d.S;
  const float* H = d.H + beat * M * S;
  launch_gemm<false, 128, 128, 16, 4>(d.R, M, H, S, d.MR, S, 0, T, S, M, M, 1, stream);
  return cudaGetLastError();
}

// ---- allocation-free variant of the H x product -------------------------------------------
//
// For callers that must not see device allocations from this library: hosts
// that place every device buffer in their own pool or arena, or run under a
// fixed device-memory budget, and callers for which the implicit device
// synchronisation of cudaMalloc / cudaFree is not acceptable. The split-K
// partial sums live in one file-scope device array instead of a per-scenario
// cudaMalloc'd buffer. Every GPU that loads the library holds this array
// (8 MiB) until the process exits.

namespace {

constexpr int64_t kStaticScratchFloats = int64_t(1) << 21;  // 2,097,152 floats = 8 MiB
__device__ __align__(256) float g_measure_scratch[kStaticScratchFloats];

constexpr int kMaxDevices = 128;
std::mutex g_scratch_mutex;
float* g_scratch_address[kMaxDevices] = {};

// Device address of g_measure_scratch on the current device. In host code the
// array's name is only a host-side stand-in, so the address is looked up once
// per device with that device current, and cached.
int scratch_address(int device, float** out) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_address[device]) {
    void* p = nullptr;
    const cudaError_t err = cudaGetSymbolAddress(&p, g_measure_scratch);
    if (err != cudaSuccess) {
      char msg[256];
      std::snprintf(msg, sizeof(msg), "cudaGetSymbolAddress of the static scratch failed: %s", cudaGetErrorString(err));
      return report_error(CT_ERR_CUDA, msg);
    }
    g_scratch_address[device] = static_cast<float*>(p);
  }
  *out = g_scratch_address[device];
  return CT_OK;
}

}  // namespace
}  // namespace ct

extern "C" int ct_predict_measurements_noalloc(const float* states, const float* measurement_matrix,
                                               const float* actual, float* predicted, float* residuals,
                                               int64_t num_steps, int64_t num_states, int64_t num_sensors,
                                               void* stream) {
  using namespace ct;
  if (!states || !measurement_matrix || !predicted)
    return report_error(CT_ERR_INVALID_ARGUMENT, "states, measurement_matrix and predicted must be device pointers");
  if (residuals && !actual) return report_error(CT_ERR_INVALID_ARGUMENT, "residuals need the actual measurements");
  const int64_t T = num_steps, S = num_states, M = num_sensors;
  if (T <= 0 || S <= 0 || M <= 0) return report_error(CT_ERR_INVALID_ARGUMENT, "num_steps, num_states and num_sensors must be positive");
  const int64_t mpad = ((M + kPart - 1) / kPart) * kPart;
  if (T * mpad > kStaticScratchFloats) {
    char msg[256];
    std::snprintf(msg, sizeof(msg),
                  "num_steps x ceil64(num_sensors) = %lld x %lld exceeds the static scratch of %lld floats",
                  (long long)T, (long long)mpad, (long long)kStaticScratchFloats);
    return report_error(CT_ERR_INVALID_ARGUMENT, msg);
  }
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess || device < 0 || device >= kMaxDevices)
    return report_error(CT_ERR_CUDA, "cudaGetDevice failed or device index out of range");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (st) {
    // the scratch address below is the current device's; a stream of another device would make the
    // kernels write into memory that device does not own
    int stream_device = -1;
    err = cudaStreamGetDevice(st, &stream_device);
    if (err != cudaSuccess) return report_error(CT_ERR_INVALID_ARGUMENT, "cudaStreamGetDevice failed on the stream");
    if (stream_device != device) {
      char msg[160];
      std::snprintf(msg, sizeof(msg), "the stream belongs to device %d but device %d is current", stream_device,
                    device);
      return report_error(CT_ERR_INVALID_ARGUMENT, msg);
    }
  }
  float* scratch = nullptr;
  int rc = scratch_address(device, &scratch);
  if (rc) return rc;
  int sms = 0;
  err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (err != cudaSuccess) return report_error(CT_ERR_CUDA, "cudaDeviceGetAttribute failed");
  // split-K factor: as for the scenario path, but bounded by the scratch capacity
  int64_t ks = measure_ksplit(T, S, M, sms);
  const int64_t by_scratch = kStaticScratchFloats / (T * mpad);
  if (ks > by_scratch) ks = by_scratch;
  if (ks < 1) ks = 1;
  const int64_t kchunk = ((S + ks - 1) / ks + BK - 1) / BK * BK;
  // every (split, step, sensor) partial read below is written first, so nothing is cleared
  launch_partials(states, measurement_matrix, scratch, T, S, M, mpad, kchunk, (int)ks, st);
  err = cudaGetLastError();
  if (err != cudaSuccess) return report_error(CT_ERR_CUDA, cudaGetErrorString(err));
  const int64_t n = T * M;
  reduce_measure_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(scratch, (int)ks, T, M, mpad, predicted,
                                                                    residuals ? actual : nullptr, residuals);
  err = cudaGetLastError();
  if (err != cudaSuccess) return report_error(CT_ERR_CUDA, cudaGetErrorString(err));
  return CT_OK;
}
