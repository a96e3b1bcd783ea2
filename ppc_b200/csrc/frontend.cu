// Source front end on the device (Engine::sources): the library's sources become photon
// bunches on the GPU, as the host front end makes them:
//   light yield per particle type       gpu/f2k.cxx:17-167 (muon segments, EM and hadronic
//                                        cascades with the hadronic light fluctuation)
//   Poisson photon count                gpu/f2k.cxx:387-433 (poidev)
//   addp / addp_clst / addp_mopo / ph   gpu/f2k.cxx:478-528
//   bunching                            gpu/f2k.cxx:377-385 (addh)
// Three kernels: k_src_count (one thread per source: its bunch template, the light
// fluctuation and the Poisson count, from the source's own random stream; bunch and photon
// totals per block of 128 sources), k_src_scan (offsets of the blocks), k_src_write (offsets
// within the block by a CTA scan; the bunches and their first-photon indices).  A source
// makes ceil(count / 2^31) bunches.  This file is compiled without fast-math and without
// contraction, so the bunch templates follow the host front end's float arithmetic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "backend.cuh"
#include "engine.h"

namespace ppcb {

struct FrontScratch {
  unsigned long long* num = nullptr;      // photons per source
  ulonglong2* tot = nullptr;              // bunches and photons per block of kThreads sources
  ulonglong2* off = nullptr;              // [blocks + 1] first bunch and photon of each block
  int* errors = nullptr;
  uint64_t cap = 0;
  ~FrontScratch() {
    for (void* p : {(void*)num, (void*)tot, (void*)off, (void*)errors})
      if (p) cudaFree(p);
  }
};

namespace {

constexpr int kThreads = 128;
constexpr unsigned long long kMaxBunch = 1ull << 31;  // photons per bunch record
constexpr int kMaxTries = 100000;                     // bound on every rejection loop
constexpr float kRho = 0.9216f;                       // density of ice [mwe]
constexpr float kM0 = 0.105658389f;                   // muon rest mass [GeV]

struct SrcRng {
  uint32_t x, y, a;
  __device__ float u() { return bxrnd(x, y, a); }  // (0, 1]
};

// the source's stream: a SplitMix64 hash (Steele, Lea, Flood 2014) of (seed, k) seeds an
// MWC generator with one of the configuration's multipliers
__device__ SrcRng src_stream(uint32_t seed, uint64_t k, const uint32_t* rm, uint32_t nmul) {
  uint64_t z = ((uint64_t)seed << 32 | 0x3c6ef372u) + (k + 1) * 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  SrcRng r;
  r.a = __ldg(&rm[(nmul & (nmul - 1)) ? (uint32_t)(k % nmul) : (uint32_t)k & (nmul - 1)]);
  r.x = (uint32_t)z;
  r.y = __umulhi((uint32_t)(z >> 32), r.a);
  return r;
}

__device__ float src_grnd(SrcRng& r) {  // gpu/f2k.cxx:8-10
  const float a = sqrtf(-2 * logf(r.u()));
  return a * sinf(2 * PPCB_FPI * r.u());
}

// log Gamma(xx) by the Lanczos series the reference uses (gpu/f2k.cxx:387-400)
__device__ double src_gammln(double xx) {
  const double stp = 2.5066282746310005;
  const double cof[6] = {76.18009172947146, -86.50532032941677, 24.01409824083091,
                         -1.231739572450155, 0.1208650973866179e-2, -0.5395239384953e-5};
  double ser = 1, x = xx - 1;
  double tmp = x + 5.5;
  tmp -= (x + 0.5) * log(tmp);
  for (int j = 0; j <= 5; j++) {
    x++;
    ser += cof[j] / x;
  }
  return -tmp + log(stp * ser);
}

// One proposal of the rejection sampler in the reference's double precision: the count
// proposed by tan(x), or -1 when it is negative; its acceptance t in *t.
__device__ __noinline__ double src_proposal(double xm, float x, double* t) {
  const double sq = sqrt(2 * xm), alxm = log(xm), g = xm * alxm - src_gammln(xm + 1);
  const double y = tan((double)x), em = sq * y + xm;
  if (em < 0) return -1;
  const double um = floor(em);
  *t = 0.9 * (1 + y * y) * exp(um * alxm - src_gammln(um + 1) - g);
  return um;
}

struct SrcCount {
  unsigned long long num;
  bool err;
};

// The reference's rejection loop (gpu/f2k.cxx:412-431), for means from 12.  The stream is not
// drawn from again, so it goes by value: by reference it would live in memory, here and in the
// screened loop.
__device__ __noinline__ SrcCount src_poisson_exact(double xm, SrcRng r) {
  const double sq = sqrt(2 * xm), alxm = log(xm), g = xm * alxm - src_gammln(xm + 1);
  for (int it = 0; it < kMaxTries; it++) {
    double y, em;
    int k = 0;
    do {
      y = tan((double)(PPCB_FPI * r.u()));
      em = sq * y + xm;
    } while (em < 0 && ++k < kMaxTries);
    if (em < 0) break;
    const double um = floor(em);
    const double t = 0.9 * (1 + y * y) * exp(um * alxm - src_gammln(um + 1) - g);
    if (!(r.u() > t)) return SrcCount{(unsigned long long)um, false};
  }
  return SrcCount{(unsigned long long)floor(xm + 0.5), true};
}

// Means from which the screening below leaves so many proposals open that a warp with a few such
// lanes is better off without it.  1e6 sources with and without it: means around 3.6e7 200 and 200
// us, 7.2e7 220 and 197, 1.2e8 237 and 200, 3.6e8 312 and 198, log-uniform from 1e6 to 1e9 259 and 204.
// At 4e7 mixtures that reach little beyond lose (1e1 to 1e8: 150 and 188).  Lanes of a warp
// (log-uniform 1e4 to 1e9, 1e0 to 1e9): from 3 lanes 198 and 222, 4 209 and 232, 6 232 and 234, never
// 230 and 204.
constexpr double kExactMean = 1e8;
constexpr int kExactLanes = 3;

// Poisson sample of mean xm (gpu/f2k.cxx:402-433): multiplication of uniforms below 12,
// rejection from a Lorentzian above.  A proposal is first evaluated in single precision, with
// bounds on its error: y = tan(x) to 4 units in the last place (7e-7 with its product by
// sqrt(2 xm)), so the count floor(sqrt(2 xm) y + xm) is certain unless the sum lies that close
// to an integer; and the logarithm of the Poisson ratio, by Stirling's series, as
//   L = B - A + 1/(12 xm) - 1/(12 um),  A = (um + 1/2) log1p(B / xm),  B = um - xm,
// to 7e-7 |A| + 1e-7 |B| + 1e-5 (the quotient's and the logarithm's roundings, the series' next
// term for um >= 8).  Below means of 1e9 the double-precision sums round by less than that.
// Where the count, or the comparison of the uniform number with the acceptance, is not certain,
// src_proposal evaluates the reference's expressions (one proposal in 2e3 at a mean of 1000).
// So the samples are those of the double-precision sampler, which spends 500 instructions on
// a proposal (a double-precision tangent, exponential and six divisions) to 130 here.
// Bound by issue and by lanes that wait for the unluckiest of their warp: the counts of 1e6
// sources take 80 us instead of 157 (a thread that goes on to its next source while others
// still reject: 95 us, the loop's state costs more than the waiting).
// `exact_warp`: without the screening.
__device__ unsigned long long src_poisson(double xm, bool exact_warp, SrcRng& r, bool& err) {
  if (isnan(xm)) {
    err = true;
    return 0;
  }
  if (xm < 12) {
    const double g = exp(-xm);
    unsigned long long um = 0;
    double t = r.u();
    for (int it = 0; t > g; it++) {
      if (it >= kMaxTries) {
        err = true;
        break;
      }
      um++;
      t *= r.u();
    }
    return um;
  }
  if (exact_warp) {
    const SrcCount c = src_poisson_exact(xm, r);
    err |= c.err;
    return c.num;
  }
  const float mf = (float)xm, sq = sqrtf(2 * mf), rx = 1 / mf;
  int negative = 0;  // proposals below zero in a row
  for (int it = 0; it < kMaxTries;) {
    const float x = PPCB_FPI * r.u();
    const float y = tanf(x), p = sq * y;
    const double em = xm + (double)p;
    double um = floor(em);
    const float away = (float)(em - um);  // from the next integer below
    const float slack = 1e-6f * fabsf(p) + 1e-6f;
    double t = 0;
    bool exact = !(away > slack && away < 1 - slack && (um >= 8 || em < 0) && xm < 1e9);
    if (exact) um = src_proposal(xm, x, &t);
    if (um < 0) {
      if (++negative >= kMaxTries) break;
      continue;
    }
    negative = 0;
    it++;
    const float u = r.u();
    if (!exact) {
      const float uf = (float)um, B = (float)(um - xm);
      const float A = (uf + 0.5f) * log1pf(B * rx);
      const float L = (B - A) + (rx - 1 / uf) * (1.f / 12);
      const float margin = 1e-6f * fabsf(A) + 2e-7f * fabsf(B) + 3e-5f;
      const float tf = 0.9f * (1 + y * y) * expf(L);
      if (margin < 0.1f && u < tf * (1 - 2 * margin)) return (unsigned long long)um;
      // a tiny ratio: exp(L) is below the smallest uniform number, whatever its error
      if ((margin < 0.1f && u > tf * (1 + 2 * margin)) || (L + 1.001f * logf(1 + y * y) < -20 - 2 * margin)) continue;
      um = src_proposal(xm, x, &t);
      if (um < 0) continue;
    }
    if (!(u > t)) return (unsigned long long)um;
  }
  err = true;
  return (unsigned long long)floor(xm + 0.5);
}

// The bunch template of a source (everything but its count).  Returns the mean photon
// count, or -1 for an exact count (`amount`).  `r` (null: template only) draws the
// hadronic light fluctuation.
__device__ double src_bunch(const ppcb_source& s, float eff, float ovr, ppcb_bunch& p, SrcRng* r, bool& err) {
  for (int i = 0; i < 4; i++) p.u.c[i] = 0;
  p.r[0] = s.r[0];
  p.r[1] = s.r[1];
  p.r[2] = s.r[2];
  p.r[3] = s.r[3];
  p.n[0] = s.n[0];
  p.n[1] = s.n[1];
  p.n[2] = s.n[2];
  p.n[3] = 0;
  p.q = s.q;
  p.num = 0;
  p.f = 0;
  switch (s.kind) {
    case PPCB_SRC_PARTICLE: {
      const int type = s.type;
      const float E = (float)s.amount, dr = s.dr;
      p.type = -type;
      p.u.p.beta = 1;
      p.u.p.tau = 0;
      p.n[3] = dr;
      if (type < 0) {
        err = true;
        return 0;
      }
      float nph;
      const float logE = logf(fmaxf(kM0, E));
      if (type < 10) {  // bare muon (0) or its end point (1)
        const float extr = 1 + fmaxf(0.0f, 0.1880f + 0.0206f * (logE - type)) * 0.910f / kRho;
        nph = dr > 0 ? dr * extr : 0;
        p.f = 1 / extr;
        p.u.p.a = 0;
        p.u.p.b = 0;
      } else {  // cascades
        const float Lrad = 0.39652 * 0.910f / kRho;
        const float em = 5.321 * 0.910f / kRho;
        nph = em * E;
        if (type < 100) {
          switch (type) {
            default:
            case 10: case 11: case 12:
              p.u.p.a = 2.01849f + 0.63176f * logE; p.u.p.b = Lrad / 0.63207f; break;
            case 13:
              p.u.p.a = 2.00035f + 0.63190f * logE; p.u.p.b = Lrad / 0.63008f; break;
            case 14:
              p.u.p.a = 2.83923f + 0.58209f * logE; p.u.p.b = Lrad / 0.64526f; break;
          }
        } else {
          float E0, m, f0, rms0, gamma;
          switch (type) {
            default:
            case 101: case 102:
              p.u.p.a = 1.58357292f + 0.41886807f * logE; p.u.p.b = Lrad / 0.33833116f;
              E0 = 0.18791678f; m = 0.16267529f; f0 = 0.30974123f; rms0 = 0.95899551f; gamma = 1.35589541f; break;
            case 103:
              p.u.p.a = 1.69176636f + 0.40803489f * logE; p.u.p.b = Lrad / 0.34108075f;
              E0 = 0.19826506f; m = 0.16218006f; f0 = 0.31859323f; rms0 = 0.94033488f; gamma = 1.35070162f; break;
            case 104:
              p.u.p.a = 1.95948974f + 0.34934666f * logE; p.u.p.b = Lrad / 0.34535151f;
              E0 = 0.21687243f; m = 0.16861530f; f0 = 0.27724987f; rms0 = 1.00318874f; gamma = 1.37528605f; break;
            case 105:
              p.u.p.a = 1.47495778f + 0.40450398f * logE; p.u.p.b = Lrad / 0.35226706f;
              E0 = 0.29579368f; m = 0.19373018f; f0 = 0.02455403f; rms0 = 1.01619344f; gamma = 1.45477346f; break;
            case 106:
              p.u.p.a = 1.57739060f + 0.40631102f * logE; p.u.p.b = Lrad / 0.35269455f;
              E0 = 0.66725124f; m = 0.19263595f; f0 = 0.17559033f; rms0 = 1.01414337f; gamma = 1.45086895f; break;
            case 107:
              p.u.p.a = 1.92249171f + 0.33701751f * logE; p.u.p.b = Lrad / 0.34969748f;
              E0 = 0.29579368f; m = 0.19373018f; f0 = 0.02455403f; rms0 = 1.01094637f; gamma = 1.50438415f; break;
          }
          if (r) {  // hadronic light-yield fluctuation, truncated to [0, 1.1]
            const float e = fmaxf(2.71828183f, E);
            const float F = 1 - powf(e / E0, -m) * (1 - f0);
            const float dF = F * rms0 * powf(logf(e), -gamma);
            float f;
            int it = 0;
            do f = F + dF * src_grnd(*r);
            while ((f < 0 || 1.1 < f) && ++it < kMaxTries);
            if (f < 0 || 1.1 < f) err = true;
            nph *= f;
          }
        }
        p.f = 0;
        if (dr > 0) {
          p.u.p.a = 0;
          p.u.p.b = 0;
        }
      }
      const float y = eff * nph;
      return (double)(s.scale * y / ovr);
    }
    case PPCB_SRC_CLST:
      p.type = 0;
      p.n[3] = s.dr;
      p.f = 1.f;
      p.u.p.beta = s.beta;
      return -1;
    case PPCB_SRC_MOPO:
      p.type = 0;
      p.n[3] = s.dr;
      p.f = s.fr;
      p.u.p.beta = s.beta;
      p.u.p.tau = s.tau;
      return (double)((float)s.amount * eff / ovr);
    case PPCB_SRC_POINT:
      p.type = 1;
      p.u.l.ka = 0;
      p.u.l.up = 0;
      p.u.l.fldr = -1;
      p.u.l.fla = -1;
      p.u.l.ofla = -1;
      p.n[3] = 1;
      return -1;
    default:
      err = true;
      return 0;
  }
}

struct SrcArgs {
  const ppcb_source* src;
  uint64_t n;
  const uint32_t* rm;
  uint32_t nmul, seed;
  float eff, ovr;
  unsigned long long* num;
  ulonglong2* tot;
  int* errors;
};

// Exclusive prefix sums over the CTA of two per-thread values (warp shuffles, then the warp
// totals); returns the CTA totals in *ta, *tb.
__device__ void cta_scan2(unsigned long long& a, unsigned long long& b, unsigned long long* ta,
                          unsigned long long* tb) {
  __shared__ unsigned long long wa[kThreads / 32], wb[kThreads / 32];
  const unsigned int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long ia = a, ib = b;
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long xa = __shfl_up_sync(0xffffffffu, ia, d), xb = __shfl_up_sync(0xffffffffu, ib, d);
    if ((int)lane >= d) {
      ia += xa;
      ib += xb;
    }
  }
  if (lane == 31) {
    wa[w] = ia;
    wb[w] = ib;
  }
  __syncthreads();
  unsigned long long oa = 0, ob = 0, sa = 0, sb = 0;
  for (int j = 0; j < kThreads / 32; j++) {
    if (j < (int)w) {
      oa += wa[j];
      ob += wb[j];
    }
    sa += wa[j];
    sb += wb[j];
  }
  a = oa + ia - a;
  b = ob + ib - b;
  *ta = sa;
  *tb = sb;
}

__device__ __forceinline__ unsigned long long src_bunches(unsigned long long num) {
  return (num + kMaxBunch - 1) / kMaxBunch;
}

constexpr unsigned int kSrcWords = sizeof(ppcb_source) / 4;

// Copies n 4-byte words from global to shared memory, 16 bytes at a time where the global
// address allows it.
__device__ __forceinline__ void copy_words(uint32_t* dst, const uint32_t* src, unsigned int n) {
  unsigned int done = 0;
  if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
    const unsigned int q = n / 4;
    for (unsigned int i = threadIdx.x; i < q; i += kThreads)
      reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    done = 4 * q;
  }
  for (unsigned int i = done + threadIdx.x; i < n; i += kThreads) dst[i] = src[i];
}

__global__ void __launch_bounds__(kThreads) k_src_count(SrcArgs A) {
  __shared__ __align__(16) uint32_t in[kThreads * kSrcWords];
  const uint64_t k0 = (uint64_t)blockIdx.x * kThreads, k = k0 + threadIdx.x;
  copy_words(in, reinterpret_cast<const uint32_t*>(A.src + k0),
             (unsigned int)min((uint64_t)kThreads, A.n - k0) * kSrcWords);
  __syncthreads();
  unsigned long long num = 0;
  const ppcb_source& s = reinterpret_cast<const ppcb_source*>(in)[threadIdx.x];
  SrcRng r{0, 0, 0};
  double mean = 0;
  bool err = false;
  if (k < A.n) {
    r = src_stream(A.seed, k, A.rm, A.nmul);
    ppcb_bunch p;
    mean = src_bunch(s, A.eff, A.ovr, p, &r, err);
  }
  const bool exact_warp = __popc(__ballot_sync(0xffffffffu, mean >= kExactMean)) >= kExactLanes;
  if (k < A.n) {
    if (mean < 0) {  // exact count
      if (!(s.amount >= 0) || s.amount >= 1.8e19) err = true;
      else num = (unsigned long long)s.amount;
    } else {
      num = src_poisson(mean, exact_warp, r, err);
    }
    A.num[k] = num;
    if (err) atomicAdd(A.errors, 1);
  }
  unsigned long long nr = src_bunches(num), np = num, tr, tp;
  cta_scan2(nr, np, &tr, &tp);
  if (threadIdx.x == 0) A.tot[blockIdx.x] = make_ulonglong2(tr, tp);
}

// Exclusive scans of the blocks' bunch and photon totals (one block, kChunk blocks of sources
// per thread and turn).
constexpr int kScanThreads = 1024, kChunk = 4;
static_assert(kScanThreads == 32 * 32, "one warp scans the warps' totals");
__global__ void __launch_bounds__(kScanThreads) k_src_scan(const ulonglong2* tot, uint64_t n, ulonglong2* off,
                                                           uint64_t* counts) {
  __shared__ unsigned long long wr[kScanThreads / 32], wp[kScanThreads / 32];
  const unsigned int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long br = 0, bp = 0;
  for (uint64_t t0 = 0; t0 < n; t0 += kChunk * kScanThreads) {
    const uint64_t t = t0 + kChunk * threadIdx.x;
    ulonglong2 c[kChunk];
    unsigned long long sr = 0, sp = 0;
#pragma unroll
    for (int q = 0; q < kChunk; q++) {
      c[q] = t + q < n ? tot[t + q] : make_ulonglong2(0, 0);
      sr += c[q].x;
      sp += c[q].y;
    }
    unsigned long long ur = sr, up = sp;
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long xr = __shfl_up_sync(0xffffffffu, ur, d), xp = __shfl_up_sync(0xffffffffu, up, d);
      if ((int)lane >= d) {
        ur += xr;
        up += xp;
      }
    }
    if (lane == 31) {
      wr[w] = ur;
      wp[w] = up;
    }
    __syncthreads();
    ur += br - sr;
    up += bp - sp;
    if (w == 0) {  // the warps' totals
      unsigned long long r = wr[lane], p = wp[lane];
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long xr = __shfl_up_sync(0xffffffffu, r, d), xp = __shfl_up_sync(0xffffffffu, p, d);
        if ((int)lane >= d) {
          r += xr;
          p += xp;
        }
      }
      wr[lane] = r;
      wp[lane] = p;
    }
    __syncthreads();
    if (w > 0) {
      ur += wr[w - 1];
      up += wp[w - 1];
    }
    br += wr[31];
    bp += wp[31];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kChunk; q++) {
      if (t + q < n) off[t + q] = make_ulonglong2(ur, up);
      ur += c[q].x;
      up += c[q].y;
    }
  }
  if (threadIdx.x == 0) {
    off[n] = make_ulonglong2(br, bp);
    counts[0] = br;
    counts[1] = bp;
  }
}

// Where the 16-byte word e of the staged bunches lies: records four words apart, written by
// eight threads at a time, then fall on eight different banks.
__device__ __forceinline__ unsigned int swizzle(unsigned int e) { return e ^ ((e >> 3) & 7); }

// The block's sources come in, and its bunches go out, as coalesced runs through shared memory
// (a thread's own 72-byte loads and 64-byte stores touch a sector or two each: 77 us for 1e6
// sources, 36 us this way, 24 us at the memory's rate).  A block with a source of several bunches (2^31 photons and
// more) or at the end of the caller's buffer writes its records one by one.
__global__ void __launch_bounds__(kThreads) k_src_write(SrcArgs A, const ulonglong2* off, uint64_t nblk,
                                                        ppcb_bunch* out, uint64_t* bstart, uint64_t cap) {
  __shared__ __align__(16) uint32_t in[kThreads * kSrcWords];
  __shared__ uint4 stage[kThreads * 4];
  static_assert(sizeof(ppcb_bunch) == 4 * sizeof(uint4), "a bunch is four 16-byte words");
  const uint64_t k0 = (uint64_t)blockIdx.x * kThreads, k = k0 + threadIdx.x;
  const unsigned int mine = (unsigned int)min((uint64_t)kThreads, A.n - k0);
  copy_words(in, reinterpret_cast<const uint32_t*>(A.src + k0), mine * kSrcWords);
  const unsigned long long num = k < A.n ? A.num[k] : 0, nrec = src_bunches(num);
  unsigned long long b0 = nrec, ph0 = num, tr, tp;
  cta_scan2(b0, ph0, &tr, &tp);  // a barrier: `in` is complete
  const ulonglong2 o = off[blockIdx.x];
  const bool run = tr <= kThreads && o.x + tr <= cap && !__syncthreads_or(nrec > 1);
  if (nrec > 0) {
    const ppcb_source& s = reinterpret_cast<const ppcb_source*>(in)[threadIdx.x];
    __align__(16) ppcb_bunch p;
    bool err = false;
    src_bunch(s, A.eff, A.ovr, p, nullptr, err);
    if (run) {
      p.num = (uint32_t)num;
      const uint4* w = reinterpret_cast<const uint4*>(&p);
#pragma unroll
      for (unsigned int q = 0; q < 4; q++) stage[swizzle(4 * (unsigned int)b0 + q)] = w[q];
      bstart[o.x + b0] = o.y + ph0;
    } else {
      for (unsigned long long j = 0; j < nrec; j++) {
        const unsigned long long b = o.x + b0 + j;
        if (b >= cap) break;
        const unsigned long long left = num - j * kMaxBunch;
        p.num = (uint32_t)(left < kMaxBunch ? left : kMaxBunch);
        out[b] = p;
        bstart[b] = o.y + ph0 + j * kMaxBunch;
      }
    }
  }
  if (run) {
    __syncthreads();
    const unsigned int n = 4 * (unsigned int)tr;
    if (reinterpret_cast<uintptr_t>(out) % 16 == 0) {
      uint4* dst = reinterpret_cast<uint4*>(out + o.x);
      for (unsigned int e = threadIdx.x; e < n; e += kThreads) dst[e] = stage[swizzle(e)];
    } else {  // the caller's records need only their own 4-byte alignment
      uint32_t* dst = reinterpret_cast<uint32_t*>(out + o.x);
      for (unsigned int i = threadIdx.x; i < 4 * n; i += kThreads)
        dst[i] = reinterpret_cast<const uint32_t*>(&stage[swizzle(i / 4)])[i % 4];
    }
  }
  if (k == A.n - 1 && off[nblk].x <= cap) bstart[off[nblk].x] = off[nblk].y;
}

}  // namespace

void Engine::sources(int d, const ppcb_source* dsrc, uint64_t ns, uint32_t seed, ppcb_bunch* dout, uint64_t* dbstart,
                     uint64_t cap, uint64_t* dcounts, cudaStream_t st) {
  if (!inited_) throw Error("ini() must come before the front end", 6);
  DeviceCtx& g = devs.at(d);
  check(cudaSetDevice(g.dev), "cudaSetDevice");
  if (ns == 0) {
    check(cudaMemsetAsync(dcounts, 0, 2 * sizeof(uint64_t), st), "memset");
    check(cudaMemsetAsync(dbstart, 0, sizeof(uint64_t), st), "memset");
    return;
  }
  const uint64_t grid = (ns + kThreads - 1) / kThreads;
  if (grid > 0x7fffffffull) throw Error("front end: too many sources in one call", 7);
  if (!g.front) {
    g.front = std::make_shared<FrontScratch>();
    check(cudaMalloc((void**)&g.front->errors, sizeof(int)), "front end scratch");
    check(cudaMemset(g.front->errors, 0, sizeof(int)), "front end scratch");
  }
  FrontScratch& F = *g.front;
  if (ns > F.cap) {
    for (void** p : {(void**)&F.num, (void**)&F.tot, (void**)&F.off})
      if (*p) {
        cudaFree(*p);
        *p = nullptr;
      }
    F.cap = 0;
    check(cudaMalloc((void**)&F.num, ns * sizeof(unsigned long long)), "front end scratch");
    check(cudaMalloc((void**)&F.tot, grid * sizeof(ulonglong2)), "front end scratch");
    check(cudaMalloc((void**)&F.off, (grid + 1) * sizeof(ulonglong2)), "front end scratch");
    F.cap = ns;
  }
  SrcArgs A;
  A.src = dsrc;
  A.n = ns;
  A.rm = g.rm;
  A.nmul = (uint32_t)std::max(1, std::min(g.T, 1024));
  A.seed = seed;
  A.eff = cfg.eff;
  A.ovr = cfg.ovr;
  A.num = F.num;
  A.tot = F.tot;
  A.errors = F.errors;
  k_src_count<<<(unsigned int)grid, kThreads, 0, st>>>(A);
  check(cudaGetLastError(), "front end count");
  k_src_scan<<<1, kScanThreads, 0, st>>>(F.tot, grid, F.off, dcounts);
  check(cudaGetLastError(), "front end scan");
  k_src_write<<<(unsigned int)grid, kThreads, 0, st>>>(A, F.off, grid, dout, dbstart, cap);
  check(cudaGetLastError(), "front end write");
}

const int* Engine::front_errors(int d) const {
  const DeviceCtx& g = devs.at(d);
  return g.front ? g.front->errors : nullptr;
}

}  // namespace ppcb
