// Internal declarations shared by the library's translation units.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "../../include/cardiotrust_cuda.h"

namespace ct {

constexpr int kOffsets = 26;   // neighbour offsets per voxel
constexpr int kGainCols = 78;  // 26 offsets x 3 neighbour components
constexpr int kFwdTileVoxels = 32;  // voxels per tile of the recursions (consecutive in device order)
constexpr int kFwdHaloMax = 192;    // halo slots of a tile; the last one stands for absent neighbours
constexpr int kFwdRingSpread = 24;  // largest difference of delays that a tile's staged history holds
constexpr int kNearTiles = 64;      // tiles of a halo that its staging warp can follow
constexpr int kSweepVoxels = 8;     // most voxels per block of the gradient sweep
constexpr int kSweepHaloMax = 112;  // halo slots of such a block
constexpr int kSweepPerSm = 3;        // blocks per SM
constexpr int kSweepRingSpread = 16;  // largest difference of delays that its staged history holds

// Which tiles a launch of the recursions meets: only such whose history fits the staged ring (the kernel without the direct
// way), such and others (the kernel with both), or what the delays on the device say (both, one of which leaves).
enum WaveRoutes { kStaged, kDecide, kEvery };

// Counts the progress of a launch, so that a bounded wait can tell a long wait from a lost one.
struct Heartbeat {
  unsigned int count;
};

// Everything of one scenario that lives on the device.
struct DeviceScenario {
  int64_t S, V, M, T, B, NB;
  // model
  float* gains;          // [S,78]
  int32_t* nbr;          // [V,26] neighbour voxel, -1 = none (derived from output_state_indices)
  float* coefs;          // [V,26]
  int32_t* delays;       // [V,26]
  float* init_delays;    // [V,26]
  float* H;              // [B,M,S]
  float* ctrl;           // [S]
  float* u;              // [T]
  float* meas;           // [B,T,M] actual measurements
  // estimations
  float* X;              // [T,S] states of the beat being processed
  float* Y;              // [B,T,M] predicted measurements
  float* R;              // [T,M] residuals of the beat being processed
  float* MR;             // [T,S] mapped residuals of the beat being processed
  float* ap;             // [V,78] all-pass state (deduplicated over the row component)
  float* ap_last;        // [V,78] all-pass output of step T-2
  float* avg_delays;     // [V]
  // derivatives
  float* derivatives;    // dG, dC, fir, iir and mreg_sum, each on a multiple of 64 floats
  int64_t derivatives_len;
  float* dG;             // [S,78]
  float* dC;             // [V,26]
  float* fir;            // [V,78]
  float* iir;            // [V,78]
  float* mG1, *mG2;      // [S,78] Adam moments
  float* mC1, *mC2;      // [V,26]
  float* mreg_sum;       // [1] running maximum-regularisation sum
  // metrics
  float* loss, *loss_mse, *loss_mr;          // [T]
  float* loss_b, *loss_mse_b, *loss_mr_b;    // [NB]
  // scratch
  float* stepsum_part;   // [T, tiles] per-tile max-regularisation sums
  float* gemm_part;      // [ksplit, T, Mpad] split-K partials of H x
  int tiles;             // tiles of kFwdTileVoxels voxels
  int wave_grid;         // CTAs of the recursion kernels
  int ksplit;            // split-K factor of the H x product (CUDA-core form)
  // tensor-core form (ct_umma.cu); null when the scenario does not support it
  bool umma;             // S % 4 == 0 and the TMA encoder is available
  int ksplit_umma;       // split-K factor of the tensor-core H x
  int64_t kpad;          // M rounded up to 32 (K extent of H^T r)
  int64_t spad;          // S rounded up to 4: row pitch of H_hi, H_lo and Xpad (16-byte TMA rows)
  float* H_hi, *H_lo;    // [B,M,spad] TF32 split of H, zero beyond S
  float* Xpad;           // [T,spad] copy of X for the H x operand when S % 4 != 0 (else null)
  float* Ht_hi, *Ht_lo;  // [B,S,kpad] TF32 split of H^T, zero padded
  float* R_hi, *R_lo;    // [T,kpad] TF32 split of the residuals
  // sliced BF16 form (ct_slice.cu), allocated on first use; sp = S and kpm = M rounded up to 64
  int ksplit_slice;          // split-K factor of the sliced H x (whole 512-element groups per split)
  bool slice_ready;          // H_sl / Ht_sl hold the slices of the current H
  __nv_bfloat16* H_sl;       // [B][3][M][sp] slices of H
  float* H_sc;               // [B][ceil(sp/512)][M] scales (group-major)
  __nv_bfloat16* Ht_sl;      // [B][3][S][kpm] slices of H^T
  float* Ht_sc;              // [B][ceil(kpm/512)][S]
  __nv_bfloat16* X_sl;       // [3][T][sp] slices of the beat's states
  float* X_sc;               // [T][ceil(sp/512)]
  __nv_bfloat16* R_sl;       // [3][T][kpm] slices of the beat's residuals
  float* R_sc;               // [T][ceil(kpm/512)]
  int32_t* dmin;         // [2] smallest and largest delay of a connected (voxel, offset) pair
  // exchange ring of the recursion kernels: [xrows, V] entries {x0, x1, x2, step + 1}, then the number of
  // steps that each tile has finished, 128 bytes apart
  uint4* xch;
  int xrows;             // power of two; grows with the delays
  int routes, rroutes;   // WaveRoutes of the forward and of the adjoint's direction
  float4* record;        // packed registers of tiles that share a CTA, null when every tile has its own
  // halo tables: slots of each tile's (and each sweep block's) neighbourhood
  int32_t* halo;         // [tiles, kFwdHaloMax] device voxels of the halo in order, the last one repeated
  int16_t* hpos;         // [tiles, kFwdHaloMax] their slots
  int16_t* hslot;        // [tiles, 26 * kFwdTileVoxels] slot of each item's neighbour
  int32_t* near;         // [tiles, kNearTiles] tiles of the halo, the last one repeated
  int32_t* nhalo;        // [tiles] voxels of the halo, -1 if it is too large for the slots
  int32_t* range;        // [tiles, 2] smallest and largest delay of the tile's connected items
  bool sweep_any;        // blocks of the gradient sweep may come whose delays or halo their ring does not hold
  int sweep_blocks;      // blocks of the gradient sweep: consecutive voxels
  int32_t* sstart;       // [sweep blocks + 1] their first voxels
  int32_t* shalo;        // [sweep blocks, kSweepHaloMax]
  int16_t* shpos;
  int16_t* shslot;       // [sweep blocks, 26 * kSweepVoxels]
  int32_t* snhalo;       // [sweep blocks] -1 if it does not fit
  int32_t* srange;       // [sweep blocks, 2]
  // adjoint mode, allocated on first use
  int32_t* rev;          // [V,26] voxel whose offset n points at this voxel, -1 if none
  int32_t* rhalo;        // the tiles' halo tables of that direction (on a lattice the forward's but for rhslot)
  int16_t* rhpos;
  int16_t* rhslot;
  int32_t* rnear;
  int32_t* rnhalo;
  int32_t* rrange;
  float* LX;             // [T,S] gradient of the loss with respect to the states
  // plain form (ct_plain.cu), allocated on first use
  float* plain_mreg;     // [S] maximum regularisation of the current step
  float* plain_part;     // [ceil(V / 256)] per-block sums of the step's regularisation terms
  int32_t* status;       // [1] device-side error code (0 = ok)
  Heartbeat* heartbeat;  // [1]
};

// Records `message` as the calling thread's last error (read by ct_last_error); returns status.
int report_error(int status, const char* message);

// ---- launchers (all enqueue on `stream`, return cudaError_t of the launch)

// One scenario as the recursion kernel sees it, in one direction (ct_wave.cu).
struct WaveScn {
  int V, T, ntiles;
  int xrows;
  const int32_t* src;  // [V,26] voxel whose rows item (v, n) gathers, -1 = none
  const int32_t* halo;
  const int16_t* hpos;
  const int16_t* hslot;
  const int32_t* near;
  const int32_t* nhalo;
  const float* coefs;
  const int32_t* delays;
  const float* gains;
  const int32_t* dmin;   // the scenario's smallest and largest delay
  const int32_t* range;  // [tiles, 2] those of each tile's items
  uint4* xch;
  float* rows;         // [T,S] finished rows: states, or their gradient
  // forward
  const float* ctrl;
  const float* u;
  float* ap;
  float* ap_last;
  float* part;         // [T, ntiles]
  // adjoint
  const float* X;
  const float* MR;
  float threshold, mse_scaling, reg_scaling;
};
struct WaveScalars {
  float threshold = 0.0f, mse_scaling = 0.0f, reg_scaling = 0.0f;
};
// One cooperative launch over the tiles of one or more scenarios. The tiles come in phases; a CTA
// owns every gridDim-th tile of a phase and goes on to the next phase by itself.
struct WaveLaunch {
  const WaveScn* scns;     // device array of nscn scenarios, or null: `single` is the only one
  WaveScn single;
  int nscn;
  const int2* tiles;       // (scenario, first voxel) per tile, or null: tiles of 32 voxels of scenario 0
  const int* phase_begin;  // [nphases + 1] first tile of each phase, or null: one phase
  int nphases;
  int ntiles;
  int routes;              // WaveRoutes
  float4* record;          // [ntiles] packed registers, null if no CTA owns two tiles of a phase
  int32_t* status;
  Heartbeat* heartbeat;
};
WaveScn wave_scenario(const DeviceScenario& d, bool adjoint, const WaveScalars& s, float* part);
// How many CTAs of the recursion kernel are co-resident, and the bytes of one tile's record.
int wave_capacity(int device);
size_t wave_record_bytes();
// The caller clears every scenario's exchange ring first.
cudaError_t launch_wave(const WaveLaunch& launch, bool adjoint, int grid, cudaStream_t stream);
cudaError_t clear_exchange(DeviceScenario& d, cudaStream_t stream);
// Forward propagation of one beat: X[t,:] for t in [0,T).
cudaError_t launch_forward(DeviceScenario& d, float threshold, cudaStream_t stream);
// Back-propagation through time of one beat (needs X and MR): LX = dL/dX.
cudaError_t launch_adjoint_states(DeviceScenario& d, const WaveScalars& s, cudaStream_t stream);

// Split-K factor of the FP32 H x product.
int measure_ksplit(int64_t T, int64_t S, int64_t M, int sms);
// y = H[beat] x for all steps; Y[beat] = y, R = y - meas[beat], loss_mse[t].
cudaError_t launch_measure(DeviceScenario& d, int64_t beat, bool with_residuals, cudaStream_t stream);
// MR[t,:] = H[beat]^T R[t,:] for all steps.
cudaError_t launch_map_residuals(DeviceScenario& d, int64_t beat, cudaStream_t stream);
// loss_mse[t] from R.
cudaError_t launch_mse(DeviceScenario& d, cudaStream_t stream);

// Tensor-core (tcgen05) forms, ct_umma.cu.
bool umma_supported(int64_t M);
int umma_yn(int64_t M);
int umma_ksplit(int64_t T, int64_t S, int64_t M, int sms);
cudaError_t umma_prepare(DeviceScenario& d, cudaStream_t stream);
cudaError_t launch_measure_umma(DeviceScenario& d, int64_t beat, bool with_residuals, int precision,
                                cudaStream_t stream);
cudaError_t launch_map_residuals_umma(DeviceScenario& d, int64_t beat, int precision, cudaStream_t stream);
// Sliced BF16 forms (ct_slice.cu): K extents rounded up to whole 64-element chunks, scale groups of
// 512 elements, the split-K factor of H x, the slicing of H and H^T (after every change of H;
// allocates and frees a temporary [S, kpm] buffer on the stream), and the two products.
int64_t slice_pitch(int64_t k);
int64_t slice_groups(int64_t k);
int slice_ksplit(int64_t T, int64_t S, int64_t M, int sms);
cudaError_t slice_prepare(DeviceScenario& d, cudaStream_t stream);
cudaError_t launch_measure_sliced(DeviceScenario& d, int64_t beat, bool with_residuals, cudaStream_t stream);
cudaError_t launch_map_residuals_sliced(DeviceScenario& d, int64_t beat, cudaStream_t stream);

struct DeriveScalars {
  float mse_scaling, reg_scaling, threshold, diffreg;
  int freeze_gains, freeze_delays, ap_derivative;
};
// Per-(voxel, offset) sweep over the steps of one beat: dG, dC, fir, iir.
cudaError_t launch_derive(DeviceScenario& d, const DeriveScalars& s, cudaStream_t stream);
// The same sweep for the gradients of the stated loss, from LX: dG, dC.
cudaError_t launch_adjoint_gradients(DeviceScenario& d, const DeriveScalars& s, cudaStream_t stream);

struct PlainScalars {
  float mse_scaling, reg_scaling, threshold, diffreg;
  int freeze_gains, freeze_delays, ap_derivative;
};
// Plain form of one beat (prediction, reference derivation and step metrics), launched per step.
cudaError_t launch_plain_beat(DeviceScenario& d, int64_t beat, const PlainScalars& s, cudaStream_t stream);
int plain_step_launches(const PlainScalars& s);

// Step metrics of one beat: loss_mr[t] (running), loss[t]; advances mreg_sum.
cudaError_t launch_step_metrics(DeviceScenario& d, float reg_strength, cudaStream_t stream);
// Batch metrics into slot `index`; the _dev form reads the slot on the device (graph replay).
cudaError_t launch_batch_metrics(DeviceScenario& d, int64_t index, cudaStream_t stream);
cudaError_t launch_batch_metrics_dev(DeviceScenario& d, const int64_t* index_dev, cudaStream_t stream);
// Step metrics from `parts` per-step partial sums (the forward's per-tile partials).
cudaError_t launch_step_metrics_parts(DeviceScenario& d, const float* part, int parts, float reg_strength,
                                      cudaStream_t stream);

cudaError_t launch_average_delays(DeviceScenario& d, cudaStream_t stream);
cudaError_t launch_smoothness(DeviceScenario& d, float strength, cudaStream_t stream);

struct UpdateScalars {
  int optimizer, freeze_gains, freeze_delays;
  float lr_over_bs, bias1, bias2;
  const float* bias_dev = nullptr;  // if set: {bias1, bias2} read on the device (graph replay)
};
cudaError_t launch_update(DeviceScenario& d, const UpdateScalars& s, cudaStream_t stream);
// Delay ranges of the scenario, its tiles and its sweep blocks: after every change of the delays, and once the adjoint's
// tables exist.
cudaError_t launch_delay_ranges(DeviceScenario& d, cudaStream_t stream);
// rev and rhslot of a lattice: nbr and hslot with the offsets in opposite order.
cudaError_t launch_mirror_tables(DeviceScenario& d, cudaStream_t stream);

// Voxel blocks of `words` 32-bit words between reference and device voxel order (perm[u] = the
// reference voxel of device voxel u): gather dst[u] = src[perm[u]], else scatter dst[perm[u]] = src[u].
cudaError_t launch_permute_blocks(const void* src, void* dst, const int32_t* perm, int64_t V, int64_t words,
                                  bool gather, cudaStream_t stream);
// Model construction (ct_model.cu). The lead-field factor of measurement.rs:85-88 for a voxel size.
float lead_field_factor(float voxel_size_mm);
// H[b * M + m, col[i] + a] for every beat b, sensor row m, voxel-list entry i (position vpos[i]) and
// component a, with row pitch ldh.
cudaError_t launch_lead_field(const float* vpos, const int32_t* col, int64_t nv, const float* spos,
                              const float* sori, const float* off, int64_t M, int64_t B, float cf, float* H,
                              int64_t ldh, int num_sms, cudaStream_t stream);
// Delay samples, integer delays and coefficients [V, 26] from the voxel grid; *first_bad (preset to
// all ones) receives the first failing cell * 26 + offset column.
cudaError_t launch_delay_samples(const int32_t* types, const int32_t* numbers, const float* pos, int64_t nx,
                                 int64_t ny, int64_t nz, const float* vel, float rate, float* samples,
                                 int32_t* delays, float* coefs, unsigned long long* first_bad, int num_sms,
                                 cudaStream_t stream);
// connect_voxels (allpass.rs:295-494) on the host: gains [S,78] (zeroed by the caller) and activation
// times in ms [cells] (NaN = never activated).
void connect_voxels_host(const int32_t* types, const int32_t* numbers, const float* pos, int64_t nx, int64_t ny,
                         int64_t nz, const float* vel, float factor, float* gains, float* activation_ms);
// init_output_state_indicies (allpass.rs:212-289) on the host: [S,78], cell_of[v] = the cell of voxel v.
void output_state_indices_host(const int32_t* types, const int32_t* numbers, int64_t nx, int64_t ny, int64_t nz,
                               const std::vector<int64_t>& cell_of, int32_t* out);
// Expand the deduplicated [V,78] all-pass/fir/iir state into the reference [S,78] layout.
cudaError_t launch_expand_rows(const float* src, float* dst, int64_t V, cudaStream_t stream);
// Last-step maximum regularisation [S] from X[T-1].
cudaError_t launch_last_max_reg(DeviceScenario& d, float threshold, float* out, cudaStream_t stream);

// ---- post-run arrays and segmentation metrics (ct_post.cu)
struct PostPlan {
  int parts = 1;           // blocks of steps each voxel's scan is split into
  int steps_per_part = 1;
};
PostPlan post_plan(int64_t V, int64_t T, int sms);
// Device buffers of the post-run pass; the spherical arrays are reference voxel order.
struct PostBuffers {
  int32_t* inv = nullptr;          // [V] device voxel of each reference voxel
  float* mag = nullptr;            // [T,V] |x| + |y| + |z|
  float* theta = nullptr;          // [T,V]
  float* phi = nullptr;            // [T,V]
  float* mag_max = nullptr;        // [V] at the first maximum of the magnitude
  float* theta_max = nullptr;      // [V]
  float* phi_max = nullptr;        // [V]
  float* activation_ms = nullptr;  // [V]
  float* maxmag = nullptr;         // [V] largest magnitude, NaN when every step is NaN
  float* part_val = nullptr;       // [parts,V] per block of steps: largest magnitude
  int32_t* part_idx = nullptr;     // [parts,V] and its first step (-1: all NaN)
};
// Scan of X: maxmag always; with `write`, the spherical arrays, their maxima and the activation
// times (a voxel whose magnitude is NaN at every step sets CT_ERR_NO_MAXIMUM in d.status).
cudaError_t launch_spherical(const DeviceScenario& d, const PostBuffers& b, const PostPlan& plan, bool write,
                             float sample_rate_hz, cudaStream_t stream);
// Threshold sweep over `cells` grid cells (types, numbers in grid order) into `out`
// (the ct_final_metrics layout); hist is 2 x (CT_THRESHOLDS + 1) device counters.
cudaError_t launch_final_metrics(const PostBuffers& b, const int32_t* types, const int32_t* numbers, int64_t cells,
                                 unsigned long long* hist, float* out, int sms, cudaStream_t stream);

}  // namespace ct
