// Simulated side of DirectFit's likelihood on the GPU:
//   k_llh_count   per kernel-level hit the back end's acceptance (backend.cuh, the same
//                 per-hit streams as Engine::accept), then for each time shift the hit's bin
//                 round((t + dt - t0) / lbin) and, when it lies in the DOM's window and
//                 outside its errata windows, +1 on that bin's block (dat::fill, dat::join,
//                 llh/llh.cxx:469-482, 614-621), in counters of the CTA's own in shared
//                 memory.  Simulated hits on DOMs without observed pulses count toward the
//                 no-hit total (cascade::ppc, llh/llh.cxx:1694-1700).
//   k_llh_count_global  the same where the counters do not fit there.
//   k_llh_terms   one thread per (shift, block): llf (llh/llh.cxx:637-662) in FP64, a
//                 fixed-order tree sum per CTA; the last CTA of a shift adds the CTA sums in
//                 a fixed order, the no-hit term and divides by ndof (fllh,
//                 llh/llh.cxx:1075-1082).
// Counts are integers (one per accepted hit), so the binning is exact; every sum runs in a
// fixed order, so an evaluation is deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "backend.cuh"
#include "engine.h"
#include "llh.h"

namespace ppcb {

struct LlhDevice {
  int32_t* dom_slot = nullptr;
  LlhDom* doms = nullptr;
  int32_t* bin_block = nullptr;
  double* block_dat = nullptr;
  int32_t* block_dom = nullptr;
  double2* win = nullptr;
  // counters of an evaluation, cleared by one memset: the no-hit total, one ticket per shift,
  // simulated counts per (block, shift), and (norm) counts in the DOMs' windows per (DOM, shift)
  unsigned int* work = nullptr;
  double* partial = nullptr;         // [shift][CTA] sums of llf terms
  int* errors = nullptr;
  CallBuffers io;                    // host-pointer evaluations
  ~LlhDevice() {
    for (void* p : {(void*)dom_slot, (void*)doms, (void*)bin_block, (void*)block_dat, (void*)block_dom, (void*)win,
                    (void*)work, (void*)partial, (void*)errors})
      if (p) cudaFree(p);
  }
};

void LlhDeviceFree::operator()(LlhDevice* p) const { delete p; }

namespace {

constexpr int kThreads = 256;
constexpr int kMaxNewton = 200;

constexpr int kCountThreads = 1024;
constexpr size_t kCountSmem = 192 << 10;  // shared memory of the counters of one CTA, at most
// Counters that do not fit in one CTA's shared memory: up to this many per shift the shifts are
// shared out over the CTAs (k_llh_count), from there on the counters are in global memory
// (k_llh_count_global).  1.4e6 hits, 64 shifts: 2400 blocks (four parts) 215 and 229 us, with
// half of the hits on one DOM 206 and 326; 4800 blocks (seven parts) 389 and 227, 368 and 332;
// 5 shifts, 16000 blocks (two parts) 108 and 66.
constexpr size_t kPartCounters = 3072;

struct CountArgs {
  BackArgs A;
  const int32_t* dom_slot;
  const LlhDom* doms;
  const int32_t* bin_block;
  const double2* win;
  unsigned int* simc;   // [block][shift], from k_llh_count_global [shift][block]
  unsigned int* stot;   // [DOM][shift], [shift][DOM]
  unsigned long long* nohit;
  double t0, lbin;
  int nblocks, ndom, ndt, unh, norm;
  int parts, step;      // k_llh_count: CTA c counts shifts [c % parts * step, + step) of ndt
  double dt[PPCB_LLH_MAX_SHIFTS];
};

// What a lane knows of its accepted hit.
struct BinnedHit {
  int slot;       // DOM slot; -1: no observed pulses there, -2: not accepted or left out
  float t;
};

__device__ __forceinline__ BinnedHit llh_hit(const BackArgs& A, const int32_t* dom_slot, uint64_t k) {
  BinnedHit h{-2, 0.f};
  ppcb_acc_hit o;
  if (k < A.n && accept_one(A, k, o)) {
    h.slot = dom_slot[o.i];
    h.t = o.t;
  }
  return h;
}

// The reference's bin of time t shifted by dt, relative to the DOM's window: in [0, n2 - n1)
// when the hit takes part.  `q` is the quotient in single precision, a sum of two numbers
// below kMaxQuot (or a NaN): each of them carries three roundings (operand, 1 / lbin, product;
// 7.2e-4), their sum one more (2.4e-4), so q is within 1.7e-3 of it.  At least 2e-3 from the
// middle between two bins it decides; otherwise, and always with errata windows, the
// double-precision expressions of llh/llh.cxx:469-482 do.
constexpr float kMaxQuot = 4000.f;
__device__ __forceinline__ float quot_part(float q) { return fabsf(q) < kMaxQuot ? q : __int_as_float(0x7fffffff); }

__device__ __forceinline__ int llh_bin(const CountArgs& F, float q, float t, double dt, int n1, int n2, int win0,
                                       int nwin) {
  const float near = q + 12582912.f;  // 1.5 x 2^23: the nearest integer in the low mantissa bits
  if (fabsf(q - (near - 12582912.f)) < 0.498f && nwin == 0)
    return __float_as_int(near) - 0x4b400000 - n1;
  const double x = (double)t + dt;
  for (int w = 0; w < nwin; w++) {
    const double2 e = F.win[win0 + w];
    if (e.x <= x && x < e.y) return -1;
  }
  const double b = round((x - F.t0) / F.lbin);
  return b >= n1 && b < n2 ? (int)b - n1 : -1;  // also drops NaN times
}

// An accepted hit on a DOM with observed pulses, as the warp shares it out.
struct __align__(16) SharedHit {
  float t, q;             // time; its part of the quotient
  int slot, base;         // DOM slot; the DOM's bins in the bin -> block table
  int n1, n2, win0, nwin; // bins that take part, errata windows
};

// A thread accepts a hit; then the warp takes its accepted hits a few at a time, 2^k lanes
// per hit and a lane per shift, so that the lanes have work whatever was accepted and the
// counters of a hit's shifts lie side by side ([block][shift]: no bank conflicts, where
// hits of one block in all lanes would queue for one counter).  Where the counters of all
// shifts do not fit, the CTAs share the shifts out and each part accepts the hits for itself.
// What bounds it is instruction issue: the acceptance (about 250 instructions per hit) and about 15 per
// (accepted hit, shift), against 60 of one thread's loop with a double-precision division and
// a global atomic each.  Whole evaluation, 1.38e6 hits (0.55e6 accepted): 64 shifts 222 ->
// 58 us, 16 shifts 90 -> 43, 5 shifts 63 -> 41, one 50 -> 39.
__global__ void __launch_bounds__(kCountThreads, 1) k_llh_count(const __grid_constant__ CountArgs F) {
  extern __shared__ unsigned int cnt[];  // [block][shift], then with norm [DOM][shift]
  __shared__ unsigned int s_nohit;
  __shared__ double s_dt[PPCB_LLH_MAX_SHIFTS];
  __shared__ float s_q[PPCB_LLH_MAX_SHIFTS];
  const float inv = (float)(1 / F.lbin);
  __shared__ SharedHit s_hits[kCountThreads];
  SharedHit* mine = s_hits + (threadIdx.x & ~31);
  const int part = blockIdx.x % F.parts, j0 = part * F.step, nj = min(F.step, F.ndt - j0);
  const int group = nj > 16 ? 32 : nj > 8 ? 16 : nj > 4 ? 8 : nj > 1 ? 4 : 1;  // lanes per hit
  const int sims = F.nblocks * nj, counters = sims + (F.norm ? F.ndom * nj : 0);
  for (int i = threadIdx.x; i < counters; i += kCountThreads) cnt[i] = 0;
  if (threadIdx.x == 0) s_nohit = 0;
  if (threadIdx.x < nj) {
    s_dt[threadIdx.x] = F.dt[j0 + threadIdx.x];
    s_q[threadIdx.x] = quot_part((float)s_dt[threadIdx.x] * inv);
  }
  __syncthreads();
  const unsigned int lane = threadIdx.x & 31;
  unsigned int nohit = 0;
  const uint64_t tiles = (F.A.n + 31) / 32, warps = (uint64_t)(gridDim.x / F.parts) * (kCountThreads / 32);
  for (uint64_t tile = (uint64_t)(blockIdx.x / F.parts) * (kCountThreads / 32) + (threadIdx.x >> 5); tile < tiles;
       tile += warps) {
    const BinnedHit h = llh_hit(F.A, F.dom_slot, tile * 32 + lane);
    if (F.unh && part == 0 && h.slot == -1) nohit++;
    const unsigned int m = __ballot_sync(0xffffffffu, h.slot >= 0);
    if (h.slot >= 0) {
      const LlhDom& D = F.doms[h.slot];
      mine[__popc(m & ((1u << lane) - 1u))] =
          SharedHit{h.t, quot_part((float)((double)h.t - F.t0) * inv), h.slot, D.bin0, D.n1, D.n2, D.win0, D.nwin};
    }
    __syncwarp();
    const int hits = __popc(m);
    for (int i = lane / group; i < hits; i += 32 / group) {
      const SharedHit x = mine[i];
      for (int j = lane & (group - 1); j < nj; j += group) {
        const int bin = llh_bin(F, x.q + s_q[j], x.t, s_dt[j], x.n1, x.n2, x.win0, x.nwin);
        if ((unsigned)bin < (unsigned)(x.n2 - x.n1)) {
          atomicAdd(&cnt[F.bin_block[x.base + bin] * nj + j], 1u);
          if (F.norm) atomicAdd(&cnt[sims + x.slot * nj + j], 1u);  // only norm reads it
        }
      }
    }
    __syncwarp();
  }
  if (nohit) atomicAdd(&s_nohit, nohit);
  __syncthreads();
  for (int i = threadIdx.x; i < counters; i += kCountThreads) {
    const unsigned int c = cnt[i];
    const int b = i / nj, j = j0 + i - b * nj;  // the DOMs' counters follow the blocks'
    if (c) atomicAdd(b < F.nblocks ? &F.simc[(size_t)b * F.ndt + j] : &F.stot[(size_t)(b - F.nblocks) * F.ndt + j], c);
  }
  if (threadIdx.x == 0 && s_nohit) atomicAdd(F.nohit, (unsigned long long)s_nohit);
}

// Where the counters do not fit in shared memory: a thread per hit, a loop over the shifts,
// counters in global memory.  Bound by additions to the same counters, as hits crowd on a few
// DOMs: lanes that add to one address at a time go out as one addition, and every warp starts
// with another shift.  1.4e6 hits, 64 shifts, 16000 blocks: 240 us, with half of the hits on one
// DOM 359 (a lane per shift, as above, 202 and 829).
__global__ void __launch_bounds__(kThreads) k_llh_count_global(const __grid_constant__ CountArgs F) {
  __shared__ unsigned int s_nohit;
  __shared__ double s_dt[PPCB_LLH_MAX_SHIFTS];
  __shared__ float s_q[PPCB_LLH_MAX_SHIFTS];
  const float inv = (float)(1 / F.lbin);
  if (threadIdx.x == 0) s_nohit = 0;
  if (threadIdx.x < F.ndt) {
    s_dt[threadIdx.x] = F.dt[threadIdx.x];
    s_q[threadIdx.x] = quot_part((float)s_dt[threadIdx.x] * inv);
  }
  __syncthreads();
  const BinnedHit h = llh_hit(F.A, F.dom_slot, (uint64_t)blockIdx.x * kThreads + threadIdx.x);
  if (F.unh && h.slot == -1) atomicAdd(&s_nohit, 1u);
  LlhDom D;
  D.n1 = D.n2 = D.nwin = 0;  // no bin is taken
  float q = 0;
  if (h.slot >= 0) {
    D = F.doms[h.slot];
    q = quot_part((float)((double)h.t - F.t0) * inv);
  }
  int j = (int)((blockIdx.x * (kThreads / 32) + threadIdx.x / 32) % F.ndt);
  for (int i = 0; i < F.ndt; i++, j = j + 1 < F.ndt ? j + 1 : 0) {
    const int bin = llh_bin(F, q + s_q[j], h.t, s_dt[j], D.n1, D.n2, D.win0, D.nwin);
    const bool in = (unsigned)bin < (unsigned)(D.n2 - D.n1);
    __syncwarp();  // lanes that took either way of llh_bin add together
    if (in) {
      atomicAdd(&F.simc[(size_t)j * F.nblocks + F.bin_block[D.bin0 + bin]], 1u);
      if (F.norm) atomicAdd(&F.stot[(size_t)j * F.ndom + h.slot], 1u);  // only norm reads it
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_nohit) atomicAdd(F.nohit, (unsigned long long)s_nohit);
}

// llf of llh/llh.cxx:637-662: the saturated likelihood of s simulated (nsim repetitions)
// against d observed (ndat repetitions) with a log-normal model error sig; the common rate
// is found by Newton's method.  A step that leaves the domain (the reference stops the
// program there) or that has not converged in kMaxNewton steps gives NaN and sets `err`.
__device__ double llf(double s, double d, double nsim, double ndat, double sig, bool& err) {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (s < 0 || d < 0) {
    err = true;
    return nan;
  }
  if (s == 0 && d == 0) return 0;
  const double s2 = sig * sig, is2 = 1 / s2, tol = 1.e-8;
  const double sd = s + d, ntot = ndat + nsim;
  double ls = sd / ntot, ld = ls, llx = 0;
  if (sig > 0) {
    double dls;
    int it = 0;
    do {
      // the reference's step -f / (nsim (1 + (1 / b + 1 / a) / s2)) with a + b = s + d, over one
      // denominator: two divisions per iteration instead of six
      const double a = nsim * ls, b = ndat * ld;
      const double f = a - s - log(ld / ls) * is2;
      dls = -f * (a * b) / (nsim * (a * b + sd * is2));
      ls += dls;
      ld = (sd - nsim * ls) / ndat;
      if (ls < 0 || ld < 0 || ++it > kMaxNewton) {
        err = true;
        return nan;
      }
    } while (fabs(dls) > tol * ls);
    const double lr = log(ld / ls);
    llx = lr * lr / (2 * s2);
  }
  double lls = 0, lld = 0;
  if (s > 0) lls = s * log((s / nsim) / ls);
  if (d > 0) lld = d * log((d / ndat) / ld);
  return llx + lls + lld;
}

__device__ double cta_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  return sh[0];
}

struct TermArgs {
  const unsigned int* simc;   // count of (block b, shift j): [b * block_step + j * shift_step]
  const unsigned int* stot;   // of (DOM d, shift j): [d * block_step + j * dom_shift_step]
  const unsigned long long* nohit;
  unsigned int* ticket;       // [shift] CTAs done
  const double* block_dat;
  const int32_t* block_dom;
  const LlhDom* doms;
  double* partial;
  int* errors;
  double* out;
  double nsim, ndat, sig;
  int nblocks, ndt, norm, ndof;
  int block_step, shift_step, dom_shift_step;
};

__global__ void __launch_bounds__(kThreads) k_llh_terms(TermArgs T) {
  __shared__ double sh[kThreads];
  __shared__ bool last;
  const int b = blockIdx.x * kThreads + threadIdx.x, j = blockIdx.y;
  double v = 0;
  bool err = false;
  if (b < T.nblocks) {
    const double s = T.simc[(size_t)b * T.block_step + (size_t)j * T.shift_step];
    double nsim = T.nsim;
    bool use = true;
    if (T.norm) {
      const int slot = T.block_dom[b];
      const double st = T.stot[(size_t)slot * T.block_step + (size_t)j * T.dom_shift_step];
      if (st > 0) nsim = st * T.ndat / T.doms[slot].dtot;
      else use = false;  // dat::llh returns 0 for a DOM without simulated hits
    }
    if (use) v = llf(s, T.block_dat[b], nsim, T.ndat, T.sig, err);
  }
  if (err) atomicAdd(T.errors, 1);
  const double sum = cta_sum(v, sh);
  // the last CTA of the shift to get here adds up the CTAs' sums (each of them written, and
  // made visible, before its ticket)
  if (threadIdx.x == 0) {
    T.partial[(size_t)j * gridDim.x + blockIdx.x] = sum;
    __threadfence();
    last = atomicAdd(&T.ticket[j], 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  v = 0;
  for (int c = threadIdx.x; c < gridDim.x; c += kThreads) v += __ldcg(&T.partial[(size_t)j * gridDim.x + c]);
  const double total = cta_sum(v, sh);
  if (threadIdx.x == 0) {
    double nh = 0;
    err = false;
    if (!T.norm) nh = llf((double)*T.nohit, 0, T.nsim, T.ndat, T.sig, err);
    if (err) atomicAdd(T.errors, 1);
    T.out[j] = (nh + total) / T.ndof;
  }
}

template <class T>
T* upload_vec(const std::vector<T>& v, const char* what) {
  T* p = nullptr;
  const size_t n = std::max<size_t>(1, v.size());
  check(cudaMalloc((void**)&p, n * sizeof(T)), what);
  if (!v.empty()) check(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice), what);
  return p;
}

// The counting kernel's shared-memory limit, once per device (a function attribute; before
// any stream capture that launches it there).
void count_prepare() {
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  const uint64_t bit = 1ull << (dev & 63);
  if (done.load() & bit) return;
  check(cudaFuncSetAttribute(k_llh_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCountSmem),
        "likelihood attribute");
  done.fetch_or(bit);
}

// CTAs of k_llh_terms per shift.
int term_ctas(int nblocks) { return std::max(1, (nblocks + kThreads - 1) / kThreads); }

// The counters of an evaluation of ndt shifts in 4-byte words: no-hit total, tickets, blocks x
// shifts, DOMs x shifts (ndom = 0 without norm).
size_t work_words(int ndt, int nblocks, int ndom) {
  return 2 + (size_t)(ndt + 1) / 2 * 2 + ((size_t)ndt * nblocks + 1) / 2 * 2 + (size_t)ndt * ndom;
}

}  // namespace

void Likelihood::upload() {
  cuda_dev_ = eng_.devs.at(dev_).dev;
  check(cudaSetDevice(cuda_dev_), "cudaSetDevice");
  std::unique_ptr<LlhDevice, LlhDeviceFree> d(new LlhDevice);
  LlhDevice& D = *d;
  std::vector<double> dat(blocks.size());
  for (size_t k = 0; k < blocks.size(); k++) dat[k] = blocks[k].dat;
  D.dom_slot = upload_vec(dom_slot, "likelihood tables");
  D.doms = upload_vec(doms, "likelihood tables");
  D.bin_block = upload_vec(bin_block, "likelihood tables");
  D.block_dat = upload_vec(dat, "likelihood tables");
  D.block_dom = upload_vec(block_dom, "likelihood tables");
  std::vector<double2> w(win.size() / 2);
  for (size_t k = 0; k < w.size(); k++) w[k] = make_double2(win[2 * k], win[2 * k + 1]);
  D.win = upload_vec(w, "likelihood tables");
  check(cudaMalloc((void**)&D.errors, sizeof(int)), "likelihood scratch");
  check(cudaMemset(D.errors, 0, sizeof(int)), "likelihood scratch");
  // scratch for any number of shifts: what a graph holds stays as long as the object
  const int nblocks = (int)blocks.size();
  check(cudaMalloc((void**)&D.work, work_words(PPCB_LLH_MAX_SHIFTS, nblocks, opts.norm ? (int)doms.size() : 0) *
                                        sizeof(unsigned int)), "likelihood scratch");
  check(cudaMalloc((void**)&D.partial, (size_t)PPCB_LLH_MAX_SHIFTS * term_ctas(nblocks) * sizeof(double)),
        "likelihood scratch");
  count_prepare();
  d_ = std::move(d);
}

Likelihood::~Likelihood() {
  if (d_) {
    cudaSetDevice(cuda_dev_);
    d_.reset();
  }
}

void Likelihood::eval_device(const ppcb_hit* dhits, uint64_t n, uint32_t seed, const double* dts, int ndt,
                             double nsim, double* dout, cudaStream_t st) {
  if (ndt < 1 || ndt > PPCB_LLH_MAX_SHIFTS) throw Error("likelihood: 1 to 64 time shifts per evaluation", 7);
  if (n > 0 && !dhits) throw Error("likelihood: null hits", 7);
  if (!(nsim > 0)) throw Error("likelihood: nsim must be positive", 7);
  require_device();
  check(cudaSetDevice(eng_.devs.at(dev_).dev), "cudaSetDevice");
  LlhDevice& D = *d_;
  const int nblocks = (int)blocks.size(), ndom = (int)doms.size();
  const int parts = term_ctas(nblocks);
  const size_t ntick = (ndt + 1) / 2 * 2, nsimc = ((size_t)ndt * nblocks + 1) / 2 * 2;
  unsigned long long* nohit = reinterpret_cast<unsigned long long*>(D.work);
  unsigned int* ticket = D.work + 2;
  unsigned int* simc = ticket + ntick;
  unsigned int* stot = simc + nsimc;
  check(cudaMemsetAsync(D.work, 0, work_words(ndt, nblocks, opts.norm ? ndom : 0) * sizeof(unsigned int), st),
        "memset");
  // where the counters are: with all shifts or a part of them in shared memory, or in global memory
  const size_t per_shift = std::max(1, nblocks + (opts.norm ? ndom : 0));
  const size_t parts_needed = (per_shift * ndt * sizeof(unsigned int) + kCountSmem - 1) / kCountSmem;
  const bool fits = parts_needed == 1 || per_shift <= kPartCounters;
  if (n > 0) {
    const uint64_t grid = (n + kThreads - 1) / kThreads;
    if (grid > 0x7fffffffull) throw Error("likelihood: too many hits in one call", 7);
    CountArgs F;
    F.A = back_args(eng_, dev_, dhits, n, seed);
    F.dom_slot = D.dom_slot;
    F.doms = D.doms;
    F.bin_block = D.bin_block;
    F.win = D.win;
    F.simc = simc;
    F.stot = stot;
    F.nohit = nohit;
    F.t0 = t0;
    F.lbin = lbin;
    F.nblocks = nblocks;
    F.ndom = ndom;
    F.ndt = ndt;
    F.unh = opts.unh;
    F.norm = opts.norm;
    for (int j = 0; j < PPCB_LLH_MAX_SHIFTS; j++) F.dt[j] = j < ndt ? dts[j] : 0.0;
    if (fits) {
      F.step = (int)((ndt + parts_needed - 1) / parts_needed);
      F.parts = (ndt + F.step - 1) / F.step;
      // a CTA per SM, fewer when there are less than 256 hits for each: every CTA clears and
      // adds up counters of its own (3e4 hits, 64 shifts: 45 us with 2048 hits per CTA)
      const uint64_t sms = eng_.devs.at(dev_).prop.multiProcessorCount;
      const unsigned int ctas = (unsigned int)std::max<uint64_t>(1, std::min(sms / F.parts, grid)) * F.parts;
      k_llh_count<<<ctas, kCountThreads, F.step * per_shift * sizeof(unsigned int), st>>>(F);
    } else {
      k_llh_count_global<<<(unsigned int)grid, kThreads, 0, st>>>(F);
    }
    check(cudaGetLastError(), "likelihood count");
  }
  TermArgs T;
  T.simc = simc;
  T.stot = stot;
  T.nohit = nohit;
  T.ticket = ticket;
  T.block_dat = D.block_dat;
  T.block_dom = D.block_dom;
  T.doms = D.doms;
  T.partial = D.partial;
  T.errors = D.errors;
  T.out = dout;
  T.nsim = nsim;
  T.ndat = opts.drep;
  T.sig = opts.sig;
  T.nblocks = nblocks;
  T.ndt = ndt;
  T.block_step = fits ? ndt : 1;
  T.shift_step = fits ? 1 : nblocks;
  T.dom_shift_step = fits ? 1 : ndom;
  T.norm = opts.norm;
  T.ndof = ndof;
  k_llh_terms<<<dim3(parts, ndt), kThreads, 0, st>>>(T);
  check(cudaGetLastError(), "likelihood terms");
}

CallBuffers& Likelihood::io() { return d_->io; }

const int* Likelihood::device_errors() {
  check(cudaSetDevice(eng_.devs.at(dev_).dev), "cudaSetDevice");
  return d_->errors;
}

void Likelihood::require_device() {
  if (d_) return;
  if (!eng_.ready()) throw Error("ppcb_ini() must come before a likelihood evaluation", 6);
  if (dev_ >= (int)eng_.devs.size()) throw Error("bad device index", 7);
  upload();
}

int Likelihood::errors() {
  if (!d_) return 0;
  check(cudaSetDevice(eng_.devs.at(dev_).dev), "cudaSetDevice");
  int e = 0;
  check(cudaMemcpy(&e, d_->errors, sizeof(int), cudaMemcpyDeviceToHost), "likelihood errors");
  return e;
}

}  // namespace ppcb
