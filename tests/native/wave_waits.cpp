// Launches of the recursion kernel whose rows never all come: tiles of a small scenario wait for a tile that the launch
// leaves out, or the exchange ring is too short. Every wait is bounded, so the launch ends by itself with a status.
// wave_waits(form, status, ms): 0, or the line of the call that failed.
#include <cuda_runtime.h>

#include <vector>

#include "../../cardiotrust_b200/csrc/ct_internal.cuh"

namespace {

std::vector<void*> g_blocks;
template <typename T>
T* device(const std::vector<T>& v) {
  void* p = nullptr;
  if (cudaMalloc(&p, sizeof(T) * v.size()) != cudaSuccess) return nullptr;
  g_blocks.push_back(p);
  return cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice) == cudaSuccess ? static_cast<T*>(p) : nullptr;
}

#define TRY(call) \
  if ((call) != cudaSuccess) return __LINE__

}  // namespace

enum Form {
  kAllTiles,        // every tile runs: status 0
  kStagedTile,  // one tile of two, its history staged
  kDirect,     // the same with delays too far apart for the staging ring
  kShared,     // two tiles of three in one CTA, which asks for the progress of the third
  kShortRing,  // every tile runs, in a ring that could lose rows before they are read
};

extern "C" int wave_waits(int form, int* status, float* ms) {
  constexpr int kTile = ct::kFwdTileVoxels, kHalo = ct::kFwdHaloMax;
  const bool wide = form == kDirect;
  const int tiles = form == kShared ? 3 : 2, V = tiles * kTile, S = 3 * V, T = 200;
  // voxel u reads its counterpart in the next tile (the last tile: in the first) along offset 0, and in the tile before along 1
  std::vector<int32_t> src(V * ct::kOffsets, -1), delays(V * ct::kOffsets, 1), halo(tiles * kHalo), nhalo(tiles),
      near(tiles * ct::kNearTiles), dmin = {wide || form == kShortRing ? 2 : 6, wide ? 60 : 9};
  std::vector<int16_t> hpos(tiles * kHalo), hslot(tiles * kTile * ct::kOffsets, kHalo - 1);
  for (int t = 0; t < tiles; ++t) {
    const int next = (t + 1) % tiles, last = (t + tiles - 1) % tiles;
    nhalo[t] = next == last ? kTile : 2 * kTile;
    for (int i = 0; i < kHalo; ++i) {
      const int at = i < nhalo[t] ? i : nhalo[t] - 1;
      halo[t * kHalo + i] = (at < kTile ? next : last) * kTile + at % kTile;
      hpos[t * kHalo + i] = (int16_t)at;
    }
    for (int i = 0; i < ct::kNearTiles; ++i) near[t * ct::kNearTiles + i] = i == 0 ? next : last;
    for (int l = 0; l < kTile; ++l) {
      const int u = t * kTile + l;
      src[u * ct::kOffsets] = next * kTile + l;
      src[u * ct::kOffsets + 1] = last * kTile + l;
      delays[u * ct::kOffsets] = dmin[0];
      delays[u * ct::kOffsets + 1] = dmin[1];
      hslot[u * ct::kOffsets] = (int16_t)l;
      hslot[u * ct::kOffsets + 1] = (int16_t)(next == last ? l : kTile + l);
    }
  }
  ct::WaveScn p{};
  p.V = V;
  p.T = T;
  p.ntiles = tiles;
  p.xrows = form == kShortRing ? 16 : 128;
  p.src = device(src);
  p.halo = device(halo);
  p.hpos = device(hpos);
  p.hslot = device(hslot);
  p.near = device(near);
  p.nhalo = device(nhalo);
  p.coefs = device(std::vector<float>(V * ct::kOffsets, 0.5f));
  p.delays = device(delays);
  p.gains = device(std::vector<float>((size_t)S * ct::kGainCols, 0.01f));
  p.dmin = device(dmin);
  std::vector<int32_t> range;
  for (int t = 0; t < tiles; ++t) range.insert(range.end(), dmin.begin(), dmin.end());
  p.range = device(range);
  const size_t ring = sizeof(uint4) * ((size_t)p.xrows * V + 8 * tiles);
  p.xch = reinterpret_cast<uint4*>(device(std::vector<char>(ring, 0)));
  p.rows = device(std::vector<float>((size_t)T * S));
  p.ctrl = device(std::vector<float>(S, 1.0f));
  p.u = device(std::vector<float>(T, 1.0f));
  p.ap = device(std::vector<float>((size_t)V * ct::kGainCols));
  p.ap_last = device(std::vector<float>((size_t)V * ct::kGainCols));
  p.part = device(std::vector<float>((size_t)T * tiles));
  p.threshold = 1.0f;
  std::vector<int2> list;
  for (int t = 0; t < tiles; ++t)
    if (form == kAllTiles || form == kShortRing || t + 1 < tiles) list.push_back(make_int2(0, t * kTile));
  ct::WaveLaunch l{};
  l.scns = device(std::vector<ct::WaveScn>(1, p));
  l.nscn = 1;
  l.tiles = device(list);
  l.phase_begin = device(std::vector<int>{0, (int)list.size()});
  l.nphases = 1;
  l.routes = wide ? ct::kDecide : ct::kStaged;
  l.ntiles = (int)list.size();
  l.record = reinterpret_cast<float4*>(device(std::vector<char>(list.size() * ct::wave_record_bytes(), 0)));
  l.status = device(std::vector<int32_t>(1, 0));
  l.heartbeat = device(std::vector<ct::Heartbeat>(1));
  const void* all[] = {p.src, p.halo, p.hpos, p.hslot, p.near, p.nhalo, p.coefs, p.delays, p.gains, p.dmin, p.range, p.xch, p.rows, p.ctrl,
                       p.u, p.ap, p.ap_last, p.part, l.scns, l.tiles, l.phase_begin, l.record, l.status, l.heartbeat};
  for (const void* q : all)
    if (!q) return __LINE__;
  cudaEvent_t e0, e1;
  TRY(cudaEventCreate(&e0));
  TRY(cudaEventCreate(&e1));
  TRY(cudaEventRecord(e0));
  TRY(ct::launch_wave(l, false, form == kShared ? 1 : l.ntiles, nullptr));
  TRY(cudaEventRecord(e1));
  TRY(cudaDeviceSynchronize());
  TRY(cudaEventElapsedTime(ms, e0, e1));
  TRY(cudaMemcpy(status, l.status, sizeof(int32_t), cudaMemcpyDeviceToHost));
  for (void* q : g_blocks) TRY(cudaFree(q));
  g_blocks.clear();
  return 0;
}
