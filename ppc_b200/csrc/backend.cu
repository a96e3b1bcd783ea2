// Hit back end on the device (Engine::accept): the acceptance of gpu/f2k.cxx:247-363 applied
// to kernel-level hits on the GPU.  For every hit, in the reference's order of decisions:
//   1. wavelength x RDE acceptance: a DOM with high voltage and an acceptance table for its
//      (module type, variant) keeps the hit with probability rat[z] x rde / rmax;
//   2. the sensor's PMT choice (getPMT, gpu/ini.cxx:210-280): for a standard DOM a
//      polynomial in the cosine between the photon direction and the sensor axis against
//      mas x u, or the impact point's height along the axis against a threshold; for a
//      multi-PMT module one PMT by its angular response; for a wavelength-shifting tube the
//      readout end and its transit delay (backend.cuh);
//   3. cable shadow (gpu/f2k.cxx:314-335);
//   4. wavelength sampled uniformly in the hit's wavelength bin.
// The reference draws the three uniform numbers from one host stream in hit order; here
// every hit has its own stream keyed by (seed, hit index), so the decisions are the same in
// distribution, not hit by hit.  Output is in input order (a scan of the accept flags within
// and over tiles of hits), so a call is deterministic for a given seed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "backend.cuh"
#include "engine.h"

namespace ppcb {

namespace {

constexpr int kBlock = 256;
constexpr int kPerThread = 2;      // hits of a thread of the deciding kernel
constexpr int kTile = kPerThread * kBlock;  // hits per tile
constexpr int kChunk = 8;          // tiles per thread and turn of the scan over tiles
constexpr int kScanThreads = 1024;
constexpr uint64_t kSumTiles = 4096;
constexpr int kWords = 14;         // a record in 4-byte words
static_assert(sizeof(ppcb_acc_hit) == kWords * 4, "record of 14 words of 4 bytes");

// Decides every hit: a bit per hit and a count per tile.  Bound by issue and by the L1's
// gathers (a DOM record and an acceptance per hit, 52% of their peaks, 18 us for 1.38e6 hits);
// two hits per thread, one after the other: one costs 30% more (blocks that end too soon),
// four 3% (a last wave that is nearly empty).  The whole back end, 1.38e6 hits 64 -> 34.5 us,
// 5e6 191 -> 113, with multi-PMT modules 141 -> 76 (their PMT is kept, not searched again).
__global__ void __launch_bounds__(kBlock) k_accept_decide(const __grid_constant__ BackArgs A, uint32_t* bits,
                                                          unsigned int* cnt, uint16_t* pmts) {
  __shared__ unsigned int s_count;
  if (threadIdx.x == 0) s_count = 0;
  __syncthreads();
  const uint64_t tile = blockIdx.x;
#pragma unroll 1
  for (int r = 0; r < kPerThread; r++) {
    const uint64_t k = tile * kTile + r * kBlock + threadIdx.x;
    ppcb_acc_hit o;
    const bool f = k < A.n && accept_one(A, k, o);
    if (pmts && f) pmts[k] = (uint16_t)o.pmt;
    const unsigned int b = __ballot_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0) {
      bits[k >> 5] = b;
      atomicAdd(&s_count, __popc(b));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) cnt[tile] = s_count;
}

// Exclusive scan of the tiles' counts, kChunk per thread and turn (one block; only for calls
// of more than kSumTiles tiles).
__global__ void __launch_bounds__(kScanThreads) k_accept_scan(const unsigned int* cnt, uint64_t ntiles,
                                                              unsigned long long* off) {
  __shared__ unsigned long long s_warp[kScanThreads / 32];
  const unsigned int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long base = 0;
  for (uint64_t t0 = 0; t0 < ntiles; t0 += kChunk * kScanThreads) {
    const uint64_t t = t0 + kChunk * threadIdx.x;
    unsigned int c[kChunk];
    unsigned long long sum = 0;
#pragma unroll
    for (int q = 0; q < kChunk; q++) {
      c[q] = t + q < ntiles ? cnt[t + q] : 0;
      sum += c[q];
    }
    unsigned long long up = sum;
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long x = __shfl_up_sync(0xffffffffu, up, d);
      if ((int)lane >= d) up += x;
    }
    if (lane == 31) s_warp[w] = up;
    __syncthreads();
    up += base - sum;
    for (int j = 0; j < kScanThreads / 32; j++) {
      if (j < (int)w) up += s_warp[j];
      base += s_warp[j];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kChunk; q++) {
      if (t + q < ntiles) off[t + q] = up;
      up += c[q];
    }
  }
}

// Writes a tile's accepted hits, after those of the tiles before it (`off`, or without it the
// sum of their counts, which for up to kSumTiles tiles costs a block a few loads per thread
// and saves a launch and its wait: a scan in the last block of the deciding kernel made every
// block wait for its ticket, 47 us in all, and look-back over the tiles' counts 59 us).  The
// accepted ones are listed first, so that every lane
// computes a record; a block's records are staged in shared memory and copied out as one
// contiguous run with coalesced 4-byte stores (the caller's buffer needs only the record's
// own 4-byte alignment).
__global__ void __launch_bounds__(kBlock) k_accept_write(const __grid_constant__ BackArgs A, const uint32_t* bits,
                                                         const unsigned int* cnt, const unsigned long long* off,
                                                         const uint16_t* pmts, ppcb_acc_hit* out,
                                                         unsigned long long* count) {
  __shared__ uint16_t list[kTile];
  __shared__ unsigned int before[kTile / 32 + 1];
  __shared__ uint32_t stage[kBlock * kWords];
  __shared__ unsigned int s_sum[kBlock / 32];
  const uint64_t tile = blockIdx.x;
  const unsigned int lane = threadIdx.x & 31;
  constexpr int kWordsOfBits = kTile / 32;
  static_assert(kWordsOfBits <= 32, "one word of bits per lane");
  if (threadIdx.x < 32) {
    const unsigned int c = lane < kWordsOfBits ? __popc(bits[tile * kWordsOfBits + lane]) : 0;
    unsigned int v = c;
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned int x = __shfl_up_sync(0xffffffffu, v, d);
      if ((int)lane >= d) v += x;
    }
    if (lane < kWordsOfBits) before[lane] = v - c;
    if (lane == 31) before[kWordsOfBits] = v;
  }
  unsigned long long first = 0;
  if (off) {
    first = off[tile];
  } else {
    unsigned int sum = 0;
    for (unsigned int t = threadIdx.x; t < tile; t += kBlock) sum += cnt[t];
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_sum[threadIdx.x >> 5] = sum;
  }
  __syncthreads();
  if (!off)
    for (int j = 0; j < kBlock / 32; j++) first += s_sum[j];
  for (int i = threadIdx.x; i < kTile; i += kBlock) {
    const uint32_t b = bits[tile * kWordsOfBits + (i >> 5)];
    if (b >> lane & 1u) list[before[i >> 5] + __popc(b & ((1u << lane) - 1u))] = (uint16_t)i;
  }
  __syncthreads();
  const unsigned int n = before[kWordsOfBits];
  if (threadIdx.x == 0 && tile == gridDim.x - 1) *count = first + n;
  uint32_t* dst = reinterpret_cast<uint32_t*>(out + first);
  for (unsigned int r = 0; r < n; r += kBlock) {
    if (r + threadIdx.x < n) {
      ppcb_acc_hit o;
      const uint64_t k = tile * kTile + list[r + threadIdx.x];
      accept_one<true>(A, k, o, pmts ? pmts[k] : 0);
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&o);
#pragma unroll
      for (int q = 0; q < kWords; q++) stage[threadIdx.x * kWords + q] = src[q];
    }
    __syncthreads();
    const unsigned int words = min(n - r, (unsigned int)kBlock) * kWords;
    for (unsigned int q = threadIdx.x; q < words; q += kBlock) dst[r * kWords + q] = stage[q];
    __syncthreads();
  }
}

}  // namespace


BackArgs back_args(Engine& e, int d, const ppcb_hit* dhits, uint64_t n, uint32_t seed) {
  BackendTables& T = e.backend_tables(d);
  const DeviceCtx& g = e.devs.at(d);
  BackArgs A;
  A.hits = dhits; A.n = n;
  A.doms = T.doms; A.keys = T.keys; A.sensors = T.sensors; A.rat = T.rat; A.wvs = T.wvs; A.dirs = T.dirs;
  A.rm = g.rm; A.nmul = (uint32_t)std::max(1, std::min(g.T, 1024)); A.seed = seed; A.gsize = e.cfg.p.gsize;
  A.wide = reinterpret_cast<uintptr_t>(dhits) % 32 == 0;
  return A;
}

BackendTables& Engine::backend_tables(int d) {
  DeviceCtx& g = devs.at(d);
  if (g.back) return *g.back;
  const Config& c = cfg;
  std::vector<BackDom> doms(c.p.gsize);
  std::vector<int2> keys(c.p.gsize);
  std::vector<BackSensor> sensors;
  std::vector<float3> pmt_dirs;
  bool multi = false;
  std::map<int, int> sensor_index;
  std::vector<float> rat;
  std::map<std::pair<int, int>, int> acc_index;
  for (int k = 0; k < c.p.gsize; k++) {
    const OMName& n = c.names[k];
    BackDom& D = doms[k];
    for (int j = 0; j < 3; j++) D.tilt[j] = n.tilt[j];
    D.azi = n.azi;
    D.R = c.oms[k].R;
    D.F = c.oms[k].F;
    keys[k] = make_int2(n.k.str, n.k.dom);
    D.acc = -1;
    D.sensor = -1;
    D.scale = 0;
    if (n.hv > 0) {
      auto it = c.irdes.find(std::make_pair(n.omt, n.type));
      if (it != c.irdes.end() && it->second.rde > 0) {
        auto ai = acc_index.find(it->first);
        if (ai == acc_index.end()) {
          ai = acc_index.insert(std::make_pair(it->first, (int)acc_index.size())).first;
          std::vector<float> r(PPCB_WNUM, 0.f);
          for (int z = 0; z < PPCB_WNUM && z < (int)it->second.rat.size(); z++) r[z] = it->second.rat[z];
          rat.insert(rat.end(), r.begin(), r.end());
        }
        D.acc = (int16_t)ai->second;
        D.scale = n.rde / it->second.rmax;
      }
    }
    auto ti = c.types.find(n.omt);
    if (ti != c.types.end()) {
      const SensorType& T = ti->second;
      auto si = sensor_index.find(n.omt);
      if (si == sensor_index.end()) {
        si = sensor_index.insert(std::make_pair(n.omt, (int)sensors.size())).first;
        BackSensor S{};
        S.beta = T.beta;
        S.fx = T.fx;
        S.Rr = T.Rr;
        S.Rz = T.Rz;
        S.cable = T.cable;
        if (T.beta == -2) {  // the getPMT branches in the reference's order (gpu/ini.cxx:210-280)
          S.kind = kSensorTube;
        } else if (T.def) {
          if ((int)T.s.size() > kMaxPoly)
            throw Error("the device back end takes angular polynomials of at most 16 coefficients", 7);
          S.kind = kSensorStandard;
          S.mas = T.mas;
          S.ns = (int)T.s.size();
          for (int i = 0; i < S.ns; i++) S.s[i] = T.s[i];
          if (S.ns == 0) { S.ns = 1; S.s[0] = T.mas > 0 ? 0.f : 1.f; }
        } else {
          S.kind = kSensorMultiPMT;
          S.dir0 = (int)pmt_dirs.size();
          S.ndir = (int)T.dirs.size();
          multi = true;
          for (const Vec3& v : T.dirs) pmt_dirs.push_back(make_float3(v[0], v[1], v[2]));
        }
        sensors.push_back(S);
      }
      D.sensor = (int16_t)si->second;
    }
  }
  if (sensors.size() > 32767 || acc_index.size() > 32767) throw Error("back end: too many sensor types", 7);
  if (rat.empty()) rat.assign(PPCB_WNUM, 0.f);
  if (sensors.empty()) sensors.push_back(BackSensor{});
  std::vector<float2> wvs(PPCB_WNUM);
  for (int z = 0; z < PPCB_WNUM; z++) wvs[z] = make_float2(c.wvs[z].i, c.wvs[z].f);
  check(cudaSetDevice(g.dev), "cudaSetDevice");
  auto T = std::make_shared<BackendTables>();
  T->multi_pmt = multi;
  check(cudaMalloc((void**)&T->doms, doms.size() * sizeof(BackDom)), "back end tables");
  check(cudaMalloc((void**)&T->keys, keys.size() * sizeof(int2)), "back end tables");
  check(cudaMalloc((void**)&T->sensors, sensors.size() * sizeof(BackSensor)), "back end tables");
  check(cudaMalloc((void**)&T->rat, rat.size() * sizeof(float)), "back end tables");
  check(cudaMalloc((void**)&T->wvs, wvs.size() * sizeof(float2)), "back end tables");
  if (pmt_dirs.empty()) pmt_dirs.push_back(make_float3(0, 0, 1));
  check(cudaMalloc((void**)&T->dirs, pmt_dirs.size() * sizeof(float3)), "back end tables");
  check(cudaMemcpy(T->dirs, pmt_dirs.data(), pmt_dirs.size() * sizeof(float3), cudaMemcpyHostToDevice), "H2D");
  check(cudaMemcpy(T->doms, doms.data(), doms.size() * sizeof(BackDom), cudaMemcpyHostToDevice), "H2D");
  check(cudaMemcpy(T->keys, keys.data(), keys.size() * sizeof(int2), cudaMemcpyHostToDevice), "H2D");
  check(cudaMemcpy(T->sensors, sensors.data(), sensors.size() * sizeof(BackSensor), cudaMemcpyHostToDevice), "H2D");
  check(cudaMemcpy(T->rat, rat.data(), rat.size() * sizeof(float), cudaMemcpyHostToDevice), "H2D");
  check(cudaMemcpy(T->wvs, wvs.data(), wvs.size() * sizeof(float2), cudaMemcpyHostToDevice), "H2D");
  g.back = T;
  return *g.back;
}

void Engine::accept(int d, const ppcb_hit* dhits, uint64_t n, uint32_t seed, ppcb_acc_hit* dout,
                    unsigned long long* dcount, cudaStream_t st) {
  if (!inited_) throw Error("ini() must come before the back end", 6);
  BackendTables& T = backend_tables(d);
  DeviceCtx& g = devs.at(d);
  check(cudaSetDevice(g.dev), "cudaSetDevice");
  if (n == 0) {
    check(cudaMemsetAsync(dcount, 0, sizeof(unsigned long long), st), "memset");
    return;
  }
  const uint64_t nt = (n + kTile - 1) / kTile;
  if ((n + kBlock - 1) / kBlock > 0x7fffffffull) throw Error("back end: too many hits in one call", 7);
  if (nt > T.tiles_cap) {
    for (void** p : {(void**)&T.tile_off, (void**)&T.tile_cnt, (void**)&T.bits, (void**)&T.pmts})
      if (*p) {
        cudaFree(*p);
        *p = nullptr;
      }
    T.tiles_cap = 0;
    check(cudaMalloc((void**)&T.tile_off, nt * sizeof(unsigned long long)), "back end scratch");
    check(cudaMalloc((void**)&T.tile_cnt, nt * sizeof(unsigned int)), "back end scratch");
    check(cudaMalloc((void**)&T.bits, nt * (kTile / 32) * sizeof(uint32_t)), "back end scratch");
    if (T.multi_pmt) check(cudaMalloc((void**)&T.pmts, nt * kTile * sizeof(uint16_t)), "back end scratch");
    T.tiles_cap = nt;
  }
  const BackArgs A = back_args(*this, d, dhits, n, seed);
  k_accept_decide<<<(unsigned int)nt, kBlock, 0, st>>>(A, T.bits, T.tile_cnt, T.pmts);
  check(cudaGetLastError(), "back end decisions");
  if (nt > kSumTiles) {
    k_accept_scan<<<1, kScanThreads, 0, st>>>(T.tile_cnt, nt, T.tile_off);
    check(cudaGetLastError(), "back end scan");
  }
  k_accept_write<<<(unsigned int)nt, kBlock, 0, st>>>(A, T.bits, T.tile_cnt, nt > kSumTiles ? T.tile_off : nullptr,
                                                      T.pmts, dout, dcount);
  check(cudaGetLastError(), "back end write");
}

}  // namespace ppcb
