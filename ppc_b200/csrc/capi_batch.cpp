// C ABI of the batched launch (declarations: include/ppc_b200.h, "batched events").
#include <algorithm>
#include <cstring>
#include <memory>
#include <exception>
#include <string>

#include "../../include/ppc_b200.h"
#include "batch.h"
#include "ctx.h"
#include "session.h"

struct ppcb_batch {
  ppcb::Batch* b = nullptr;
  ppcb::BatchResult last;
  uint32_t events = 0;
};

template <class F>
static int bguard(F&& f) {
  try {
    f();
    return PPCB_OK;
  } catch (const ppcb::Error& e) {
    ppcb_internal_set_error(e.what());
    return e.code ? e.code : PPCB_ECONFIG;
  } catch (const std::exception& e) {
    ppcb_internal_set_error(e.what());
    return PPCB_EARG;
  }
}

extern "C" {

int ppcb_batch_create(ppcb_ctx* c, int device, uint32_t max_events, uint32_t max_bunches, uint64_t hit_capacity,
                      ppcb_batch** out) {
  if (!c || !out) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    ppcb_batch* x = new ppcb_batch();
    try {
      x->b = new ppcb::Batch(c->s.eng, device, max_events, max_bunches, hit_capacity);
    } catch (...) {
      delete x;
      throw;
    }
    *out = x;
  });
}

int ppcb_batch_destroy(ppcb_batch* x) {
  if (!x) return PPCB_OK;
  int r = bguard([&] { delete x->b; });
  delete x;
  return r;
}

int ppcb_batch_set_graph(ppcb_batch* x, int use_graph) {
  if (!x) { ppcb_internal_set_error("null batch"); return PPCB_EARG; }
  x->b->use_graph = use_graph != 0;
  return PPCB_OK;
}

int ppcb_batch_run(ppcb_batch* x, const ppcb_bunch* bunches, int32_t nb, uint32_t events, double hits_per_photon,
                   ppcb_batch_info* info) {
  if (!x || !bunches) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    x->b->run(bunches, nb, events, x->last, hits_per_photon);
    x->events = events;
    if (info) {
      memset(info, 0, sizeof(*info));
      info->photons = x->last.photons;
      info->steps = x->last.steps;
      info->kept = x->last.hits.size();
      uint64_t produced = 0;
      for (uint32_t v : x->last.produced) produced += v;
      info->hits = produced;
      info->overflowed = x->last.overflowed;
      info->device_ms = x->last.device_ms;
      info->graph_ms = x->last.graph_ms;
    }
  });
}

int ppcb_batch_counts(ppcb_batch* x, uint32_t* produced, uint64_t* offsets) {
  if (!x) { ppcb_internal_set_error("null batch"); return PPCB_EARG; }
  if (produced) memcpy(produced, x->last.produced.data(), x->events * sizeof(uint32_t));
  if (offsets) memcpy(offsets, x->last.offset.data(), (x->events + 1) * sizeof(uint64_t));
  return PPCB_OK;
}

int ppcb_batch_hits(ppcb_batch* x, ppcb_hit* out, uint64_t cap, uint64_t* n) {
  if (!x) { ppcb_internal_set_error("null batch"); return PPCB_EARG; }
  uint64_t k = std::min<uint64_t>(cap, x->last.hits.size());
  if (k && out) memcpy(out, x->last.hits.data(), k * sizeof(ppcb_hit));
  if (n) *n = x->last.hits.size();
  return PPCB_OK;
}

int ppcb_batch_autotune(ppcb_batch* x, const ppcb_bunch* bunches, int32_t nb, uint32_t events, uint64_t sample_photons,
                        ppcb_tune_info* out) {
  if (!x || !bunches) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    ppcb::TuneResult t = x->b->autotune(bunches, nb, events, sample_photons);
    if (out) {
      out->threads = t.threads;
      out->blocks_per_sm = t.blocks_per_sm;
      out->refill_below = t.refill_below;
      out->photons_per_s = t.photons_per_s;
    }
  });
}

int ppcb_set_ice(ppcb_ctx* c, const float* be, const float* ba) {
  if (!c) { ppcb_internal_set_error("null context"); return PPCB_EARG; }
  return bguard([&] { c->s.eng.set_ice(be, ba); });
}

int ppcb_get_ice(ppcb_ctx* c, float* be, float* ba, int32_t* size) {
  if (!c) { ppcb_internal_set_error("null context"); return PPCB_EARG; }
  return bguard([&] {
    const ppcb::Config& f = c->s.eng.cfg;
    if (size) *size = f.p.size;
    for (int j = 0; j < f.p.size; j++) {
      if (be) be[j] = f.be[j];
      if (ba) ba[j] = f.ba[j];
    }
  });
}

int ppcb_gradient(ppcb_ctx* c, const ppcb_bunch* bunches, int32_t nb, uint32_t events, const float* observed,
                  const float* weights, double scale, uint64_t hit_cap, uint32_t* counts, double* g_be, double* g_ba,
                  ppcb_grad_info* info) {
  if (!c || !bunches) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    ppcb::Engine::Grad r = c->s.eng.gradient(bunches, nb, events, observed, weights, scale, hit_cap);
    const int size = c->s.eng.cfg.p.size;
    if (counts) memcpy(counts, r.counts.data(), r.counts.size() * sizeof(uint32_t));
    if (g_be) memcpy(g_be, r.g_be.data(), size * sizeof(double));
    if (g_ba) memcpy(g_ba, r.g_ba.data(), size * sizeof(double));
    if (info) {
      info->ll = r.ll;
      info->photons = r.photons;
      info->hits = r.hits;
      info->replayed = r.replayed;
      info->unmatched = r.unmatched;
      info->steps = r.steps;
      info->forward_ms = r.forward_ms;
      info->backward_ms = r.backward_ms;
    }
  });
}

struct ppcb_gradgraph {
  ppcb_ctx* c;
  std::unique_ptr<ppcb::GradGraph> g;
};

int ppcb_gradgraph_create(ppcb_ctx* c, const ppcb_bunch* bunches, int32_t nb, uint32_t events, const float* observed,
                          double scale, uint64_t hit_cap, ppcb_gradgraph** out) {
  if (!c || !bunches || !observed || !out) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    std::unique_ptr<ppcb_gradgraph> h(new ppcb_gradgraph{c, nullptr});
    h->g.reset(new ppcb::GradGraph(c->s.eng, bunches, nb, events, observed, scale, hit_cap));
    *out = h.release();
  });
}

int ppcb_gradgraph_run(ppcb_gradgraph* g, const float* be, const float* ba, uint32_t* counts, double* g_be,
                       double* g_ba, ppcb_grad_info* info) {
  if (!g) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    ppcb::Engine::Grad r = g->g->run(be, ba, counts != nullptr);
    const int size = g->c->s.eng.cfg.p.size;
    if (counts) memcpy(counts, r.counts.data(), r.counts.size() * sizeof(uint32_t));
    if (g_be) memcpy(g_be, r.g_be.data(), size * sizeof(double));
    if (g_ba) memcpy(g_ba, r.g_ba.data(), size * sizeof(double));
    if (info) {
      info->ll = r.ll;
      info->photons = r.photons;
      info->hits = r.hits;
      info->replayed = r.replayed;
      info->unmatched = r.unmatched;
      info->steps = r.steps;
      info->forward_ms = r.forward_ms;
      info->backward_ms = r.backward_ms;
    }
  });
}

int ppcb_gradgraph_destroy(ppcb_gradgraph* g) {
  if (!g) return PPCB_OK;
  return bguard([&] { delete g; });
}

}  // extern "C"

extern "C" {

int ppcb_accept_device(ppcb_ctx* c, int device, const ppcb_hit* hits, uint64_t n, uint32_t seed, ppcb_acc_hit* out,
                       unsigned long long* count, void* stream) {
  if (!c || (n > 0 && (!hits || !out)) || !count) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    if (device < 0 || device >= (int)c->s.eng.devs.size()) throw ppcb::Error("bad device index", PPCB_EARG);
    c->s.eng.accept(device, hits, n, seed, out, count, static_cast<cudaStream_t>(stream));
  });
}

int ppcb_accept(ppcb_ctx* c, const ppcb_hit* hits, uint64_t n, uint32_t seed, ppcb_acc_hit* out, uint64_t cap,
                uint64_t* nout) {
  if (!c || (n > 0 && !hits) || !nout) { ppcb_internal_set_error("null argument"); return PPCB_EARG; }
  return bguard([&] {
    ppcb::Engine& e = c->s.eng;
    if (!e.ready()) throw ppcb::Error("ppcb_ini() must come before the back end", PPCB_ESTATE);
    ppcb::check(cudaSetDevice(e.devs[0].dev), "cudaSetDevice");
    const std::shared_ptr<ppcb::CallBuffers> io = e.devs[0].io;
    const ppcb::CallBuffers::Use use(*io);
    const size_t in = n * sizeof(ppcb_hit), res = n * sizeof(ppcb_acc_hit), cnt = sizeof(unsigned long long);
    ppcb_hit* dh = static_cast<ppcb_hit*>(io->device(0, in));
    // the records, then (on its 8-byte boundary) their number
    unsigned char* dout = static_cast<unsigned char*>(io->device(1, res + cnt));
    unsigned char* h = io->stage(in + res + cnt);
    unsigned long long k = 0;
    if (h) {  // a small call: staged both ways, one wait; the records come back uncounted
      if (n) std::memcpy(h, hits, in);
      if (n) ppcb::check(cudaMemcpyAsync(dh, h, in, cudaMemcpyHostToDevice, 0), "H2D hits");
      e.accept(0, dh, n, seed, reinterpret_cast<ppcb_acc_hit*>(dout), reinterpret_cast<unsigned long long*>(dout + res),
               0);
      ppcb::check(cudaMemcpyAsync(h + in, dout, res + cnt, cudaMemcpyDeviceToHost, 0), "D2H hits");
      io->wait(0);
      std::memcpy(&k, h + in + res, cnt);
      const uint64_t w = std::min<uint64_t>(k, cap);
      if (w && out) std::memcpy(out, h + in, w * sizeof(ppcb_acc_hit));
    } else {
      ppcb::check(cudaMemcpy(dh, hits, in, cudaMemcpyHostToDevice), "H2D hits");
      e.accept(0, dh, n, seed, reinterpret_cast<ppcb_acc_hit*>(dout), reinterpret_cast<unsigned long long*>(dout + res),
               0);
      ppcb::check(cudaMemcpy(&k, dout + res, cnt, cudaMemcpyDeviceToHost), "D2H count");
      const uint64_t w = std::min<uint64_t>(k, cap);
      if (w && out) ppcb::check(cudaMemcpy(out, dout, w * sizeof(ppcb_acc_hit), cudaMemcpyDeviceToHost), "D2H");
    }
    *nout = k;
  });
}

}  // extern "C"

extern "C" {

int ppcb_sources_device(ppcb_ctx* c, int device, const ppcb_source* src, uint64_t ns, uint32_t seed,
                        ppcb_bunch* out, uint64_t* bstart, uint64_t cap, uint64_t* counts, void* stream) {
  if (!c || (ns > 0 && !src) || (cap > 0 && !out) || !bstart || !counts) {
    ppcb_internal_set_error("null argument");
    return PPCB_EARG;
  }
  return bguard([&] {
    if (device < 0 || device >= (int)c->s.eng.devs.size()) throw ppcb::Error("bad device index", PPCB_EARG);
    c->s.eng.sources(device, src, ns, seed, out, bstart, cap, counts, static_cast<cudaStream_t>(stream));
  });
}

int ppcb_sources(ppcb_ctx* c, const ppcb_source* src, uint64_t ns, uint32_t seed, ppcb_bunch* out, uint64_t* bstart,
                 uint64_t cap, uint64_t* nb, uint64_t* num) {
  if (!c || (ns > 0 && !src) || (cap > 0 && (!out || !bstart)) || !nb || !num) {
    ppcb_internal_set_error("null argument");
    return PPCB_EARG;
  }
  return bguard([&] {
    ppcb::Engine& e = c->s.eng;
    if (!e.ready()) throw ppcb::Error("ppcb_ini() must come before the front end", PPCB_ESTATE);
    ppcb::check(cudaSetDevice(e.devs[0].dev), "cudaSetDevice");
    const std::shared_ptr<ppcb::CallBuffers> io = e.devs[0].io;
    const ppcb::CallBuffers::Use use(*io);
    const size_t in = ns * sizeof(ppcb_source), res = cap * sizeof(ppcb_bunch), off = (cap + 1) * sizeof(uint64_t);
    ppcb_source* ds = static_cast<ppcb_source*>(io->device(0, in));
    ppcb_bunch* dout = static_cast<ppcb_bunch*>(io->device(1, res));
    uint64_t* dbs = static_cast<uint64_t*>(io->device(2, off));
    uint64_t* dcnt = static_cast<uint64_t*>(io->device(3, 2 * sizeof(uint64_t)));
    // staging: counts and the error counter before and after, then (in a small call, which
    // waits once and brings the records back uncounted) the sources, records and offsets
    unsigned char* h = io->stage(64 + in + res + off);
    const bool small = h != nullptr;
    if (!small) h = io->stage(64);
    uint64_t* cnt = reinterpret_cast<uint64_t*>(h);
    int* err = reinterpret_cast<int*>(h + 16);
    err[0] = err[1] = 0;
    auto fetch = [&](void* to, const void* from, size_t bytes, const char* what) {
      if (bytes) ppcb::check(cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToHost, 0), what);
    };
    if (const int* p = e.front_errors(0)) fetch(&err[0], p, sizeof(int), "D2H errors");
    if (small) {
      if (ns) std::memcpy(h + 64, src, in);
      if (ns) ppcb::check(cudaMemcpyAsync(ds, h + 64, in, cudaMemcpyHostToDevice, 0), "H2D sources");
    } else if (ns) {
      ppcb::check(cudaMemcpy(ds, src, in, cudaMemcpyHostToDevice), "H2D sources");
    }
    e.sources(0, ds, ns, seed, dout, dbs, cap, dcnt, 0);
    fetch(cnt, dcnt, 2 * sizeof(uint64_t), "D2H counts");
    if (const int* p = e.front_errors(0)) fetch(&err[1], p, sizeof(int), "D2H errors");
    if (small) {
      fetch(h + 64 + in, dout, res, "D2H bunches");
      fetch(h + 64 + in + res, dbs, off, "D2H bunch starts");
    }
    io->wait(0);
    const uint64_t w = std::min<uint64_t>(cnt[0], cap);
    const size_t starts = (w + (cnt[0] <= cap ? 1 : 0)) * sizeof(uint64_t);
    const bool want = bstart && (cap > 0 || cnt[0] == 0);
    if (small) {
      if (w) std::memcpy(out, h + 64 + in, w * sizeof(ppcb_bunch));
      if (want) std::memcpy(bstart, h + 64 + in + res, starts);
    } else {
      if (w) ppcb::check(cudaMemcpy(out, dout, w * sizeof(ppcb_bunch), cudaMemcpyDeviceToHost), "D2H bunches");
      if (want) ppcb::check(cudaMemcpy(bstart, dbs, starts, cudaMemcpyDeviceToHost), "D2H bunch starts");
    }
    *nb = cnt[0];
    *num = cnt[1];
    if (err[0] != err[1])
      throw ppcb::Error("front end: a source's sampling failed (negative type, bad count or no convergence)",
                        PPCB_EARG);
  });
}

int ppcb_f2k_sources(const char* text, uint64_t len, uint32_t first_segment, ppcb_source* out, uint64_t cap,
                     uint64_t* n, uint64_t* lines) {
  if ((len > 0 && !text) || (cap > 0 && !out) || !n || !lines) {
    ppcb_internal_set_error("null argument");
    return PPCB_EARG;
  }
  return bguard([&] {
    uint64_t k = 0, line = 0, pos = 0;
    while (pos < len) {
      uint64_t end = pos;
      while (end < len && text[end] != '\n') end++;
      const std::string in(text + pos, end - pos);
      pos = end + 1;
      const uint32_t seg = first_segment + (uint32_t)line++;
      ppcb::F2kTrack tr;
      if (!ppcb::parse_f2k_track(in, tr) || tr.type == -1) continue;
      if (k < cap) {
        ppcb_source s;
        std::memset(&s, 0, sizeof(s));
        s.r[0] = tr.x; s.r[1] = tr.y; s.r[2] = tr.z; s.r[3] = tr.t;
        s.n[0] = tr.n[0]; s.n[1] = tr.n[1]; s.n[2] = tr.n[2];
        s.q = seg;
        if (tr.type == -2) {
          s.kind = PPCB_SRC_POINT;
          s.amount = (double)(unsigned long long)tr.E;
        } else {
          s.kind = PPCB_SRC_PARTICLE;
          s.type = tr.type;
          s.amount = tr.E;
          s.dr = tr.l;
          s.scale = 1;
        }
        out[k] = s;
      }
      k++;
    }
    *n = k;
    *lines = line;
  });
}

}  // extern "C"
