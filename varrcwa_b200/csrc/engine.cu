// Host engine of the varRCWA B200 path: memory pools, descriptor staging,
// batched stages (assembly, eigensolve, segments, projections, star
// products) and the three integrator drivers.  All arithmetic runs in the
// device kernels; the host only evaluates geometry rules and schedules.
#include "engine.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstdlib>
#include <cstring>
#include <tuple>
#include <list>
#include <mutex>
#include <numeric>
#include <stdexcept>

namespace vrc {

// ---------------------------------------------------------------------------
// Geometry helpers
// ---------------------------------------------------------------------------
// Natural cubic spline: on [z_i, z_(i+1)] (h = z_(i+1) - z_i, a = (z_(i+1) - z) / h,
// b = 1 - a) x = a y_i + b y_(i+1) + ((a^3 - a) M_i + (b^3 - b) M_(i+1)) h^2 / 6,
// with second derivatives M from the tridiagonal system
// h_(i-1) M_(i-1) + 2 (h_(i-1) + h_i) M_i + h_i M_(i+1) = 6 (slope_i - slope_(i-1)),
// M_0 = M_(K-1) = 0.  M is linear in y: M = D y, D formed column by column.
void PwlRule::prepare() {
  const size_t K = zs.size();
  D.clear();
  if (interp != 1 || K < 3) return;
  D.assign(K * K, 0.0);
  std::vector<double> h(K - 1), c(K), d(K), r(K);
  for (size_t i = 0; i + 1 < K; ++i) h[i] = zs[i + 1] - zs[i];
  for (size_t col = 0; col < K; ++col) {
    auto y = [&](size_t i) { return i == col ? 1.0 : 0.0; };
    // Thomas algorithm on the interior unknowns M_1 .. M_(K-2)
    for (size_t i = 1; i + 1 < K; ++i) {
      const double rhs = 6.0 * ((y(i + 1) - y(i)) / h[i] - (y(i) - y(i - 1)) / h[i - 1]);
      const double diag = 2.0 * (h[i - 1] + h[i]);
      if (i == 1) {
        c[i] = h[i] / diag;
        d[i] = rhs / diag;
      } else {
        const double m = diag - h[i - 1] * c[i - 1];
        c[i] = h[i] / m;
        d[i] = (rhs - h[i - 1] * d[i - 1]) / m;
      }
    }
    r[0] = r[K - 1] = 0.0;
    for (size_t i = K - 2; i >= 1; --i) {
      r[i] = d[i] - (i + 2 < K ? c[i] * r[i + 1] : 0.0);
      if (i == 1) break;
    }
    for (size_t i = 0; i < K; ++i) D[i * K + col] = r[i];
  }
}

void PwlRule::weights(double z, std::vector<double>& w) const {
  const size_t K = zs.size();
  w.assign(K, 0.0);
  if (K == 0) return;
  if (z <= zs[0]) {
    w[0] = 1.0;
    return;
  }
  if (z >= zs[K - 1]) {
    w[K - 1] = 1.0;
    return;
  }
  const size_t hi = std::upper_bound(zs.begin(), zs.end(), z) - zs.begin(), lo = hi - 1;
  const double h = zs[hi] - zs[lo];
  const double b = (z - zs[lo]) / h, a = 1.0 - b;
  w[lo] += a;
  w[hi] += b;
  if (interp == 1 && !D.empty()) {
    const double ca = (a * a * a - a) * h * h / 6.0, cb = (b * b * b - b) * h * h / 6.0;
    for (size_t k = 0; k < K; ++k) w[k] += ca * D[lo * K + k] + cb * D[hi * K + k];
  }
}

double PwlRule::eval(double z) const {
  const size_t k = zs.size();
  if (k == 0) return 0.0;
  if (z <= zs[0]) return vals[0];
  if (z >= zs[k - 1]) return vals[k - 1];
  size_t hi = std::upper_bound(zs.begin(), zs.end(), z) - zs.begin();
  size_t lo = hi - 1;
  if (interp == 1 && !D.empty()) {
    std::vector<double> w;
    weights(z, w);
    double x = 0.0;
    for (size_t q = 0; q < k; ++q) x += w[q] * vals[q];
    return x;
  }
  double t = (z - zs[lo]) / (zs[hi] - zs[lo]);
  return (1.0 - t) * vals[lo] + t * vals[hi];
}

void CellSpec::geometry(double z, std::vector<double>& xo, std::vector<double>& yo) const {
  if (kind == GEOM_PLANAR) {
    planar_section(z, xo, yo, nullptr);
    return;
  }
  if (kind == GEOM_SAMPLER) {  // only the period: the caller's sampler forms P, Q
    xo = x;
    yo = y;
    return;
  }
  if (kind == GEOM_PILLAR) {
    xo.resize(npx + 1);
    yo.resize(npy + 1);
    for (int i = 0; i <= npx; ++i) xo[i] = Lx * i / npx;
    for (int j = 0; j <= npy; ++j) yo[j] = Ly * j / npy;
    return;
  }
  xo = x;
  yo = y;
  for (const auto& r : xrules) xo[r.index] = r.eval(z);
  for (const auto& r : yrules) yo[r.index] = r.eval(z);
  if (geom_cb) geom_cb(z, xo.data(), yo.data());
}

bool CellSpec::mirrored(double z) const {
  if ((kind != GEOM_GRID && kind != GEOM_PIXELS && kind != GEOM_PLANAR) || geom_cb) return false;
  std::vector<double> xs, ys;
  std::vector<cplx> sect;
  if (kind == GEOM_PLANAR) planar_section(z, xs, ys, &sect);
  else geometry(z, xs, ys);
  // ascending coordinates (crossed ones are refilled in painter's order), each
  // the mirror image of its counterpart to rounding, about a point that is the
  // origin up to half periods
  auto even = [](const std::vector<double>& v) {
    const double a = v.front(), b = v.back(), L = b - a;
    const double tol = 2e-15 * std::max(std::fabs(a), std::fabs(b));
    if (!(L > 0.0)) return false;
    const double half = (a + b) / L;
    if (std::fabs(half - std::round(half)) * L > tol) return false;
    const size_t n = v.size();
    for (size_t i = 0; i < n; ++i) {
      if (i && v[i] < v[i - 1]) return false;
      if (std::fabs((v[i] - a) - (b - v[n - 1 - i])) > tol) return false;
    }
    return true;
  };
  if (xs.size() < 2 || ys.size() < 2 || !even(xs) || !even(ys)) return false;
  const std::vector<cplx>& e = kind == GEOM_PLANAR ? sect : eps;
  const size_t nc = xs.size() - 1, nr = ys.size() - 1;
  if (e.size() != nc * nr) return false;
  for (size_t r = 0; r < nr; ++r)
    for (size_t c = 0; c < nc; ++c) {
      const cplx v = e[r * nc + c], x = e[r * nc + nc - 1 - c], y = e[(nr - 1 - r) * nc + c];
      if (v.x != x.x || v.y != x.y || v.x != y.x || v.y != y.y) return false;
    }
  return true;
}

double CellSpec::radius(double z) const {
  double t = (z1 == z0) ? 0.0 : (z - z0) / (z1 - z0);
  return r0 + (r1 - r0) * t;
}

// ---------------------------------------------------------------------------
// Memory
// ---------------------------------------------------------------------------
BlockPool::~BlockPool() {
  for (auto& c : chunks_) cudaFree(c.first);
}

size_t BlockPool::release_free(cudaStream_t st) {
  if (free_.empty()) return 0;
  std::vector<void*> fr(free_);
  std::sort(fr.begin(), fr.end());
  std::vector<std::pair<void*, size_t>> keep;
  size_t released = 0;
  for (auto& c : chunks_) {
    char* lo = (char*)c.first;
    char* hi = lo + c.second * bytes_;
    const size_t nfree = std::lower_bound(fr.begin(), fr.end(), (void*)hi) - std::lower_bound(fr.begin(), fr.end(), (void*)lo);
    if (nfree == c.second && cudaFree(c.first) == cudaSuccess) {
      released += c.second * bytes_;
      blocks_ -= c.second;
    } else {
      keep.push_back(c);
    }
  }
  if (released) {
    std::vector<void*> nf;
    for (void* p : free_) {
      bool kept = false;
      for (auto& c : keep)
        if ((char*)p >= (char*)c.first && (char*)p < (char*)c.first + c.second * bytes_) {
          kept = true;
          break;
        }
      if (kept) nf.push_back(p);
    }
    free_.swap(nf);
    chunks_.swap(keep);
  }
  return released;
}

namespace {
// host time spent in cudaMalloc/cudaFree (all engines), in microseconds
std::atomic<long long> g_host_alloc_us{0};
std::atomic<long long> g_host_alloc_calls{0};
struct AllocTimer {
  std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
  AllocTimer() { ++g_host_alloc_calls; }
  ~AllocTimer() {
    g_host_alloc_us += (long long)std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0)
                           .count();
  }
};
}  // namespace

void* BlockPool::get(cudaStream_t) {
  if (free_.empty()) {
    AllocTimer at;
    // A pool doubles, up to 64 MB a chunk: the parity classes of many cells fill
    // pools of small blocks (10 KB at 7 x 7 orders), and a cudaMalloc takes 0.2 ms,
    // far more beside other lanes' kernels.  By 256 blocks each time, the first
    // RCWA solve of 400 such cells (four slices, one lane) made 528 calls and took
    // 245 ms; 63 and 100 now (the general way, with 256 blocks, 166 and 209).
    size_t per = std::max<size_t>(1, (size_t)(64u << 20) / bytes_);
    per = std::min(per, std::max<size_t>(256, blocks_));
    void* chunk = nullptr;
    for (;;) {
      if (cudaMalloc(&chunk, per * bytes_) == cudaSuccess) break;
      (void)cudaGetLastError();
      if (per == 1) return nullptr;
      per = per > 256 ? 256 : 1;
    }
    chunks_.push_back({chunk, per});
    blocks_ += per;
    for (size_t i = 0; i < per; ++i) free_.push_back((char*)chunk + i * bytes_);
  }
  void* p = free_.back();
  free_.pop_back();
  return p;
}

Engine::Engine(int device) : device_(device) {
  VRC_CUDA_CHECK(cudaSetDevice(device));
  VRC_CUDA_CHECK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
  own_stream_ = true;
  stage_cap_ = (size_t)128 << 20;  // two halves of 64 MB
  VRC_CUDA_CHECK(cudaMallocHost(&h_stage_, stage_cap_));
  VRC_CUDA_CHECK(cudaMalloc(&d_stage_, stage_cap_));
}

Engine::~Engine() {
  cudaSetDevice(device_);
  cudaStreamSynchronize(stream_);
  pools_.clear();
  for (auto& p : pend_prof_) {
    cudaEventDestroy(p.a);
    cudaEventDestroy(p.b);
  }
  for (auto e : ev_pool_) cudaEventDestroy(e);
  if (ext_ev_) cudaEventDestroy(ext_ev_);
  if (ext_host_) cudaFreeHost(ext_host_);
  if (ws_) cudaFree(ws_);
  if (d_stage_) cudaFree(d_stage_);
  if (h_stage_) cudaFreeHost(h_stage_);
  if (own_stream_) cudaStreamDestroy(stream_);
}

static double host_now_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

void Engine::sync() {
  const double t0 = host_now_ms();
  VRC_CUDA_CHECK(cudaStreamSynchronize(stream_));
  gemm_bulk_check();
  t_sync_ret_ = host_now_ms();
  sync_ms_ += t_sync_ret_ - t0;
  ++nsync_;
  stage_off_ = 0;
  if (!pend_prof_.empty()) resolve_prof();
}

cudaEvent_t Engine::take_event() {
  if (ev_pool_.empty()) {
    cudaEvent_t e;
    VRC_CUDA_CHECK(cudaEventCreate(&e));
    return e;
  }
  cudaEvent_t e = ev_pool_.back();
  ev_pool_.pop_back();
  return e;
}

void Engine::resolve_prof() {
  for (auto& p : pend_prof_) {
    float ms = 0.f;
    VRC_CUDA_CHECK(cudaEventElapsedTime(&ms, p.a, p.b));
    FamStat& f = fam_[p.fam];
    f.ms += ms;
    if (origin_) {  // the launch's interval on the time line shared by all engines
      float t0 = 0.f, t1 = 0.f;
      VRC_CUDA_CHECK(cudaEventElapsedTime(&t0, origin_, p.a));
      VRC_CUDA_CHECK(cudaEventElapsedTime(&t1, origin_, p.b));
      f.iv.push_back({t0, t1});
    }
    f.launches += p.nl;
    f.flops += p.flops;
    f.bytes += p.bytes;
    if (last_b_) {
      // GPU time between the previous profiled family and this one (idle,
      // or small unprofiled copies): a diagnostic of host-side bubbles
      float gap = 0.f;
      VRC_CUDA_CHECK(cudaEventElapsedTime(&gap, last_b_, p.a));
      gap_[last_fam_ + " -> " + p.fam] += gap;
      ev_pool_.push_back(last_b_);
    }
    ev_pool_.push_back(p.a);
    last_b_ = p.b;
    last_fam_ = p.fam;
  }
  pend_prof_.clear();
}

void Engine::set_profiling(bool on) {
  sync();
  profiling_ = on;
}
std::map<std::string, Engine::FamStat>& Engine::fam_stats() {
  sync();
  fam_["host_alloc"].ms = 1e-3 * (double)g_host_alloc_us.load() - alloc_ms0_;
  fam_["host_alloc"].bytes = (double)(g_host_alloc_calls.load() - alloc_calls0_);  // the number of calls
  return fam_;
}
void Engine::reset_fam_stats() {
  sync();
  fam_.clear();
  alloc_ms0_ = 1e-3 * (double)g_host_alloc_us.load();
  alloc_calls0_ = g_host_alloc_calls.load();
}

Engine::Prof::Prof(Engine& eng, const char* f, double fl, double by, int nlaunch)
    : e(eng), fam(f), flops(fl), bytes(by), nl(nlaunch) {
  if (e.t_sync_ret_ >= 0.0) {
    e.bubble_ms_ += host_now_ms() - e.t_sync_ret_;
    e.t_sync_ret_ = -1.0;
  }
  if (e.profiling_) {
    a = e.take_event();
    VRC_CUDA_CHECK(cudaEventRecord(a, e.stream_));
  }
}
Engine::Prof::~Prof() {
  e.launches += nl;
  if (a) {
    cudaEvent_t b = e.take_event();
    cudaEventRecord(b, e.stream_);
    e.pend_prof_.push_back({fam, a, b, flops, bytes, nl});
  }
}

BlockPool& Engine::pool(size_t bytes) {
  auto it = pools_.find(bytes);
  if (it == pools_.end()) it = pools_.emplace(bytes, std::make_unique<BlockPool>(bytes)).first;
  return *it->second;
}

// A block of a size class; when the device has no room for a new chunk, the
// chunks of every size class of this engine that hold no handed-out block
// are freed (memory kept by one workload's pools is then available to the
// next) and the allocation is tried once more.
void* Engine::take(size_t bytes) {
  BlockPool& p = pool(bytes);
  void* b = p.get(stream_);
  if (b) return b;
  if (trim_idle()) b = p.get(stream_);
  if (!b) throw StatusError(ST_ENOMEM, "device memory exhausted");
  return b;
}
size_t Engine::trim_idle() {
  size_t rel = 0;
  for (auto& kv : pools_) rel += kv.second->release_free(stream_);
  return rel;
}
cplx* Engine::mat(int n) { return (cplx*)take((size_t)n * n * 16); }
cplx* Engine::vec(int n) { return (cplx*)take((size_t)((n + 15) / 16) * 256); }
void Engine::free_mat(cplx* p, int n) {
  if (p) pool((size_t)n * n * 16).put(p);
}
void Engine::free_vec(cplx* p, int n) {
  if (p) pool((size_t)((n + 15) / 16) * 256).put(p);
}
// Size classes of untyped blocks (descriptor arrays, status words, scratch):
// quarter-octave steps (at most 25% over the request), so that requests
// whose size follows the batch (every level and wave has its own) share a
// few pools instead of opening one, with its own chunk, per distinct size.
static size_t byte_class(size_t b) {
  b = std::max<size_t>(b, 256);
  int e = 63 - __builtin_clzll((unsigned long long)b);  // 2^e <= b < 2^(e+1)
  const size_t unit = (size_t)1 << (e - 2);             // e >= 8
  size_t c = (b + unit - 1) / unit * unit;
  return (c + 255) / 256 * 256;
}
void* Engine::bytes(size_t b) { return take(byte_class(b)); }
void Engine::free_bytes(void* p, size_t b) {
  if (p) pool(byte_class(b)).put(p);
}

// Launch arguments (descriptor and pointer arrays) are staged in two halves
// of a pinned ring.  When the current half is full the engine synchronises
// and continues in the other half, so arguments already staged for the
// launch being prepared (the earlier operands of one call) stay intact; the
// half they sit in is reused only after the next synchronisation.
void* Engine::stage(const void* data, size_t nbytes) {
  const size_t need = (nbytes + 255) / 256 * 256;
  const size_t half = stage_cap_ / 2;
  if (need > half) throw StatusError(ST_EINVAL, "descriptor batch too large");
  if (stage_off_ + need > half) {
    const int next = stage_half_ ^ 1;
    sync();  // every launch so far has completed: both halves are free
    stage_half_ = next;
  }
  char* h = h_stage_ + stage_half_ * half + stage_off_;
  char* d = d_stage_ + stage_half_ * half + stage_off_;
  std::memcpy(h, data, nbytes);
  VRC_CUDA_CHECK(cudaMemcpyAsync(d, h, nbytes, cudaMemcpyHostToDevice, stream_));
  stage_off_ += need;
  return d;
}

void* Engine::workspace(size_t nbytes) {
  if (nbytes > ws_cap_) {
    sync();
    AllocTimer at;
    if (ws_) cudaFree(ws_);
    ws_ = nullptr;
    size_t cap = nbytes + nbytes / 4;
    cudaError_t e = cudaMalloc(&ws_, cap);
    if (e != cudaSuccess) {  // free the pools' idle chunks and try once more
      (void)cudaGetLastError();
      e = trim_idle() ? cudaMalloc(&ws_, cap) : e;
    }
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      ws_cap_ = 0;
      throw StatusError(ST_ENOMEM, "workspace allocation failed");
    }
    ws_cap_ = cap;
  }
  return ws_;
}

void Engine::pool_report(size_t* held, size_t* out, size_t* npools, size_t* ws) const {
  *held = *out = 0;
  *npools = pools_.size();
  for (const auto& kv : pools_) {
    *held += kv.second->blocks() * kv.first;
    *out += (kv.second->blocks() - kv.second->free_blocks()) * kv.first;
  }
  *ws = ws_cap_;
}

size_t Engine::batch_budget_bytes() const {
  size_t fr = 0, tot = 0;
  cudaMemGetInfo(&fr, &tot);
  size_t b = fr / 4;
  const size_t cap = (size_t)8 << 30;  // per engine: the lanes each hold one workspace
  if (b > cap) b = cap;
  if (b < ((size_t)256 << 20)) b = (size_t)256 << 20;
  return b;
}

// Items of `per` bytes to take at once.  What fits the budget's lower bound,
// or the workspace already held, needs no look at the free memory:
// cudaMemGetInfo is a call into the kernel driver, 64 us on an idle host and
// far more while other processes allocate, and every stage of a solve asks.
size_t Engine::batch_chunk(size_t count, size_t per, size_t most, bool in_workspace) const {
  const size_t take = std::min(count, most);
  const size_t held = std::max<size_t>((size_t)256 << 20, in_workspace ? ws_cap_ : 0);
  if (take <= held / per) return std::max<size_t>(1, take);
  return std::min(most, std::max<size_t>(1, batch_budget_bytes() / per));
}

// ---------------------------------------------------------------------------
// Batched primitives
// ---------------------------------------------------------------------------
void ensure_smem(const void* kernel, size_t bytes) {
  // A launch has 48 KB without asking, what the kernel declares itself included
  // (at most 8.5 KB here).
  if (bytes <= 32 * 1024) return;
  static std::mutex mu;
  static std::map<const void*, size_t> limit;
  std::lock_guard<std::mutex> lock(mu);
  size_t& cur = limit[kernel];
  if (bytes > cur) {
    VRC_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    cur = bytes;
  }
}

int Engine::gemm_tile() const {
  const char* e = std::getenv("VRC_GEMM_TILE");
  return e ? (std::atoi(e) == 32 ? 32 : 64) : 0;
}

void Engine::gemm(std::vector<GemmDesc>& d, int n, cplx alpha, cplx beta, double delta, int opA, int opB) {
  if (d.empty()) return;
  const int tile = gemm_tile();
  const size_t per = 16384;
  for (size_t b0 = 0; b0 < d.size(); b0 += per) {
    size_t nb = std::min(per, d.size() - b0);
    GemmDesc* dd = upload(d.data() + b0, nb);
    const double nn3 = (double)n * n * n;
    Prof pr(*this, "zgemm", 8.0 * nn3 * nb, 48.0 * n * (double)n * nb);
    zgemm_batched(dd, (int)nb, n, alpha, beta, delta, stream_, -1, opA, opB, tile);
  }
}

void Engine::inverse(const std::vector<cplx*>& mats, int n, std::vector<int>* status) {
  if (mats.empty()) return;
  cplx* const* dm = upload(mats);
  int* dst = nullptr;
  if (status) {
    dst = (int*)bytes(mats.size() * sizeof(int));
    VRC_CUDA_CHECK(cudaMemsetAsync(dst, 0, mats.size() * sizeof(int), stream_));
  }
  {
    const double nn3 = (double)n * n * n;
    const int W = zinv_blocked_width(n);
    if (n > zinv_small_maxn()) {
      // blocked: rank-W updates on the tensor cores, in chunks of a fixed
      // number of matrices so that the scratch block is reused
      const size_t per = zinv_blocked_scratch(n);
      const size_t CH = 512;
      char* scr = (char*)bytes(CH * per);
      for (size_t c0 = 0; c0 < mats.size(); c0 += CH) {
        const size_t B = std::min(CH, mats.size() - c0);
        std::vector<GemmDesc> g(B);
        for (size_t b = 0; b < B; ++b) {
          cplx* Mb = (cplx*)(scr + b * per);
          g[b] = {Mb, Mb + (size_t)n * W, mats[c0 + b], mats[c0 + b], nullptr, nullptr};
        }
        const GemmDesc* dd = upload(g);
        Prof pr(*this, "zinv", 8.0 * nn3 * B, 48.0 * n * (double)n * B * ((n + W - 1) / W));
        zinv_blocked_batched(dm + c0, (int)B, n, dst ? dst + c0 : nullptr, scr, dd, stream_);
      }
      free_bytes(scr, CH * per);
    } else {
      Prof pr(*this, "zinv", 8.0 * nn3 * mats.size(), 32.0 * n * (double)n * mats.size());
      zinv_small_batched(dm, (int)mats.size(), n, dst, stream_);
    }
  }
  if (status) {
    std::vector<int> h(mats.size());
    VRC_CUDA_CHECK(cudaMemcpyAsync(h.data(), dst, h.size() * sizeof(int), cudaMemcpyDeviceToHost, stream_));
    sync();
    free_bytes(dst, mats.size() * sizeof(int));
    if (status->size() < h.size()) status->resize(h.size(), 0);
    for (size_t i = 0; i < h.size(); ++i)
      if (h[i]) (*status)[i] = h[i];
  }
}

void Engine::copy(const std::vector<cplx*>& src, const std::vector<cplx*>& dst, int n) {
  std::vector<const cplx*> a(src.begin(), src.end()), b(src.size(), nullptr);
  axpby(a, b, dst, mk(1.0, 0.0), mk(0.0, 0.0), 0.0, n);
}

void Engine::axpby(const std::vector<const cplx*>& A, const std::vector<const cplx*>& B,
                   const std::vector<cplx*>& C, cplx alpha, cplx beta, double delta, int n) {
  if (A.empty()) return;
  const size_t per = 60000;
  for (size_t b0 = 0; b0 < A.size(); b0 += per) {
    size_t nb = std::min(per, A.size() - b0);
    const cplx* const* da = upload(A.data() + b0, nb);
    const cplx* const* db = upload(B.data() + b0, nb);
    cplx* const* dc = upload(C.data() + b0, nb);
    Prof pr(*this, "elementwise", 0.0, 48.0 * n * (double)n * nb);
    axpby_batched(da, db, dc, alpha, beta, delta, (int)nb, n, stream_);
  }
}

// ---------------------------------------------------------------------------
// Per-cell constants
// ---------------------------------------------------------------------------
namespace {
const double PI_H = 3.1415926535897932;

inline cplx fromc(std::complex<double> a) { return mk(a.real(), a.imag()); }

double sinc_h(double x) { return x == 0.0 ? 1.0 : std::sin(PI_H * x) / (PI_H * x); }

// PMLSolver1D::solve, src/rcwa/PMLSolver1D.cpp:15-30
std::complex<double> pml1d(double b0, double b1, double L, std::complex<double> gamma, int n, double coeff) {
  auto expipi = [](double x) { return std::exp(std::complex<double>(0.0, PI_H * x)); };
  double bm = (b1 - b0) / L, bp = (b1 + b0) / L;
  std::complex<double> r = 4.0 * sinc_h(n * bm - 0.5) * expipi(-(n * bp + coeff * 0.5));
  r += 8.0 * expipi(-(n * bp)) * sinc_h(n * bm);
  r += -2.0 * gamma * expipi(-(n * bp)) * sinc_h(n * bm);
  r += 4.0 * sinc_h(n * bm + 0.5) * expipi(-(n * bp - coeff * 0.5));
  r += gamma * sinc_h(n * bm - 1.0) * expipi(-(n * bp + coeff * 1.0));
  r += gamma * sinc_h(n * bm + 1.0) * expipi(-(n * bp - coeff * 1.0));
  r *= bm / 16.0;
  return r;
}

// Block-Toeplitz dense F[(m,n),(j,l)] = mat[nx-1+m-j][ny-1+n-l] (column-major out).
void block_toeplitz(const std::vector<std::complex<double>>& mat /* (2nx-1) x (2ny-1) row-major */, int nx,
                    int ny, std::vector<std::complex<double>>& out) {
  int m = nx * ny, Q = 2 * ny - 1;
  out.assign((size_t)m * m, 0.0);
  for (int c = 0; c < m; ++c)
    for (int r = 0; r < m; ++r) {
      int i = r / ny, j = r % ny, k = c / ny, l = c % ny;
      out[(size_t)c * m + r] = mat[(size_t)(nx - 1 + i - k) * Q + (ny - 1 + j - l)];
    }
}
}  // namespace

Engine::CellDev* Engine::prepare_cell(const CellSpec& c) {
  auto* cd = new CellDev();
  cd->nx = c.nx;
  cd->ny = c.ny;
  cd->m = c.m();
  cd->n = c.n();
  cd->k0 = c.k0();
  cd->pml = c.pml;
  std::vector<double> x, y;
  c.geometry(c.z0, x, y);
  const double Lx = x.back() - x.front(), Ly = y.back() - y.front();
  // alpha, beta: src/core/LayerSampler.cpp:9-32
  const int m = cd->m;
  cd->h_alpha.resize(m);
  cd->h_beta.resize(m);
  const int Nx = (c.nx - 1) / 2, Ny = (c.ny - 1) / 2;
  for (int i = 0; i < c.nx; ++i)
    for (int j = 0; j < c.ny; ++j) {
      cd->h_alpha[c.ny * i + j] = (2 * PI_H / Lx) * (double)(i - Nx);
      cd->h_beta[c.ny * i + j] = (2 * PI_H / Ly) * (double)(j - Ny);
    }
  cd->alpha = (double*)bytes(m * sizeof(double));
  cd->beta = (double*)bytes(m * sizeof(double));
  VRC_CUDA_CHECK(cudaMemcpyAsync(cd->alpha, cd->h_alpha.data(), m * sizeof(double), cudaMemcpyHostToDevice, stream_));
  VRC_CUDA_CHECK(cudaMemcpyAsync(cd->beta, cd->h_beta.data(), m * sizeof(double), cudaMemcpyHostToDevice, stream_));
  if (c.pml) {
    // src/core/LayerSampler.cpp:34-111 (region from VarLayerSampler.cpp:23-39)
    const double b0 = y[0], b1 = y[1], u0 = y[y.size() - 2], u1 = y[y.size() - 1];
    const double l0 = x[0], l1 = x[1], r0 = x[x.size() - 2], r1 = x[x.size() - 1];
    const std::complex<double> gamma = 1.0 / std::complex<double>(1.0, -1.0);
    const int nPx = 2 * c.nx - 1, nPy = 2 * c.ny - 1;
    const int maxPx = (nPx - 1) / 2, maxPy = (nPy - 1) / 2;
    std::vector<std::complex<double>> fyy(nPy), fxx(nPx), fyx(nPx), fxy(nPy);
    for (int i = 0; i < nPy; ++i) {
      int nn = i - maxPy;
      fyy[i] = (u0 - b1) / Ly * sinc_h(nn * (u0 - b1) / Ly) /
               std::exp(std::complex<double>(0, PI_H) * std::complex<double>(nn * (b1 + u0) / Ly));
      fyy[i] += pml1d(b0, b1, Ly, gamma, nn, 1.0);
      fyy[i] += pml1d(u0, u1, Ly, gamma, nn, -1.0);
    }
    for (int i = 0; i < nPx; ++i) {
      int mm = i - maxPx;
      fxx[i] = (r0 - l1) * sinc_h(mm * (r0 - l1) / Lx) / Lx /
               std::exp(std::complex<double>(0, PI_H * mm * (l1 + r0) / Lx));
      fxx[i] += pml1d(l0, l1, Lx, gamma, mm, 1.0);
      fxx[i] += pml1d(r0, r1, Lx, gamma, mm, -1.0);
    }
    for (int i = 0; i < nPx; ++i) {
      int mm = i - maxPx;
      if (mm == 0) fyx[i] = r1 - l0;
      else
        fyx[i] = (std::exp(std::complex<double>(0., -2 * PI_H / Lx * mm * r1)) -
                  std::exp(std::complex<double>(0., -2 * PI_H / Lx * mm * l0))) *
                 std::complex<double>(0., Lx * Lx / (mm * 2 * PI_H));
    }
    for (int i = 0; i < nPy; ++i) {
      int nn = i - maxPy;
      if (nn == 0) fxy[i] = u1 - b0;
      else
        fxy[i] = (std::exp(std::complex<double>(0., -2 * PI_H / Ly * nn * u1)) -
                  std::exp(std::complex<double>(0., -2 * PI_H / Ly * nn * b0))) *
                 std::complex<double>(0., Ly * Ly / (2 * nn * PI_H));
    }
    std::vector<std::complex<double>> fy((size_t)nPx * nPy), fx((size_t)nPx * nPy);
    for (int i = 0; i < nPx; ++i)
      for (int j = 0; j < nPy; ++j) {
        fy[(size_t)i * nPy + j] = 1.0 / Lx * fyx[i] * fyy[j];
        fx[(size_t)i * nPy + j] = 1.0 / Ly * fxx[i] * fxy[j];
      }
    std::vector<std::complex<double>> Fx, Fy;
    block_toeplitz(fx, c.nx, c.ny, Fx);
    block_toeplitz(fy, c.nx, c.ny, Fy);
    std::vector<cplx> hKx((size_t)m * m), hKy((size_t)m * m);
    for (int col = 0; col < m; ++col)
      for (int r = 0; r < m; ++r) {
        hKx[(size_t)col * m + r] = fromc(Fx[(size_t)col * m + r] * cd->h_alpha[col]);
        hKy[(size_t)col * m + r] = fromc(Fy[(size_t)col * m + r] * cd->h_beta[col]);
      }
    cd->Kx = mat(m);
    cd->Ky = mat(m);
    VRC_CUDA_CHECK(cudaMemcpyAsync(cd->Kx, hKx.data(), hKx.size() * 16, cudaMemcpyHostToDevice, stream_));
    VRC_CUDA_CHECK(cudaMemcpyAsync(cd->Ky, hKy.data(), hKy.size() * 16, cudaMemcpyHostToDevice, stream_));
    sync();  // host vectors go out of scope
    cd->KxKy = mat(m);
    cd->KxKx = mat(m);
    cd->KyKy = mat(m);
    cd->KyKx = mat(m);
    std::vector<GemmDesc> g = {{cd->Kx, cd->Ky, cd->KxKy, nullptr, nullptr, nullptr},
                               {cd->Kx, cd->Kx, cd->KxKx, nullptr, nullptr, nullptr},
                               {cd->Ky, cd->Ky, cd->KyKy, nullptr, nullptr, nullptr},
                               {cd->Ky, cd->Kx, cd->KyKx, nullptr, nullptr, nullptr}};
    gemm(g, m, mk(1, 0), mk(0, 0), 0.0);
  }
  if (c.kind != GEOM_PILLAR && c.kind != GEOM_PLANAR && c.kind != GEOM_SAMPLER) {  // planar: per sample
    cd->eps_count = c.eps.size();
    cd->eps_dev = (cplx*)bytes(cd->eps_count * 16);
    VRC_CUDA_CHECK(cudaMemcpyAsync(cd->eps_dev, c.eps.data(), cd->eps_count * 16, cudaMemcpyHostToDevice, stream_));
  }
  if (c.kind == GEOM_GRID && !c.geom_cb && !std::getenv("VRC_HOST_GEOMETRY") &&
      (!c.xrules.empty() || !c.yrules.empty())) {
    // rule tables for the device geometry: bases, then per rule its knots,
    // values and (spline) second derivatives M = D vals
    std::vector<double> gd(c.x.begin(), c.x.end());
    gd.insert(gd.end(), c.y.begin(), c.y.end());
    std::vector<int> gi;
    size_t off = 0;
    for (int axis = 0; axis < 2; ++axis)
      for (const PwlRule& r : axis == 0 ? c.xrules : c.yrules) {
        const size_t K = r.zs.size();
        if (r.index < 0 || r.index >= (int)(axis == 0 ? c.x.size() : c.y.size()) || K < 1 || r.vals.size() != K)
          throw StatusError(ST_EINVAL, "coordinate rule out of range");
        const int spline = (r.interp == 1 && !r.D.empty()) ? 1 : 0;
        gi.insert(gi.end(), {axis, r.index, (int)K, (int)off, spline});
        gd.insert(gd.end(), r.zs.begin(), r.zs.end());
        gd.insert(gd.end(), r.vals.begin(), r.vals.end());
        for (size_t i = 0; i < K; ++i) {
          double mi = 0.0;
          if (spline)
            for (size_t k = 0; k < K; ++k) mi += r.D[i * K + k] * r.vals[k];
          gd.push_back(mi);
        }
        off += 3 * K;
      }
    cd->dev_geom = true;
    cd->nrules = (int)(gi.size() / 5);
    cd->geo_nd = gd.size();
    cd->geo_ni = gi.size();
    cd->geo_d = (double*)bytes(gd.size() * sizeof(double));
    cd->geo_i = (int*)bytes(std::max<size_t>(1, gi.size()) * sizeof(int));
    VRC_CUDA_CHECK(cudaMemcpyAsync(cd->geo_d, gd.data(), gd.size() * sizeof(double), cudaMemcpyHostToDevice, stream_));
    VRC_CUDA_CHECK(cudaMemcpyAsync(cd->geo_i, gi.data(), gi.size() * sizeof(int), cudaMemcpyHostToDevice, stream_));
  }
  sync();
  return cd;
}

void Engine::release_cell(CellDev* cd) {
  if (!cd) return;
  free_bytes(cd->alpha, cd->m * sizeof(double));
  free_bytes(cd->beta, cd->m * sizeof(double));
  free_mat(cd->Kx, cd->m);
  free_mat(cd->Ky, cd->m);
  free_mat(cd->KxKy, cd->m);
  free_mat(cd->KxKx, cd->m);
  free_mat(cd->KyKy, cd->m);
  free_mat(cd->KyKx, cd->m);
  if (cd->eps_dev) free_bytes(cd->eps_dev, cd->eps_count * 16);
  if (cd->geo_d) free_bytes(cd->geo_d, cd->geo_nd * sizeof(double));
  if (cd->geo_i) free_bytes(cd->geo_i, std::max<size_t>(1, cd->geo_ni) * sizeof(int));
  delete cd;
}

// ---------------------------------------------------------------------------
// Assembly (A1-A6)
// ---------------------------------------------------------------------------
namespace {
struct AsmKey {
  int nx, ny, ncx, ncy, pml, pillar, devgeom, mirrored;
  bool operator<(const AsmKey& o) const {
    return std::tie(nx, ny, ncx, ncy, pml, pillar, devgeom, mirrored) <
           std::tie(o.nx, o.ny, o.ncx, o.ncy, o.pml, o.pillar, o.devgeom, o.mirrored);
  }
};
}  // namespace

// Samples of cells driven by the caller's own sampler (LayerSampler::sample
// or sampleOnGPU of the reference, src/core/LayerSampler.h:49-55): a device
// callback writes the engine's n x n buffers directly, in stream order; a
// host callback fills pinned host memory, which is copied to the device
// buffers asynchronously (the staging is reused only after the previous
// copies have completed).
void Engine::sample_external(const std::vector<SampleReq*>& rs) {
  if (rs.empty()) return;
  if (!ext_ev_) VRC_CUDA_CHECK(cudaEventCreateWithFlags(&ext_ev_, cudaEventDisableTiming));
  VRC_CUDA_CHECK(cudaEventSynchronize(ext_ev_));  // staging free
  size_t off = 0;
  bool copied = false;
  for (SampleReq* r : rs) {
    const CellSpec& s = *r->spec;
    const int n = s.n();
    const size_t nn = (size_t)n * n;
    int rc = 0;
    if (s.dev_sample) {
      rc = s.dev_sample(r->z, r->P, r->Q, stream_);
    } else {
      const size_t need = 2 * nn * sizeof(cplx);
      if (off + need > ext_cap_) {
        if (copied) {
          VRC_CUDA_CHECK(cudaEventRecord(ext_ev_, stream_));
          VRC_CUDA_CHECK(cudaEventSynchronize(ext_ev_));
        }
        off = 0;
        if (need > ext_cap_) {
          if (ext_host_) VRC_CUDA_CHECK(cudaFreeHost(ext_host_));
          ext_host_ = nullptr;
          ext_cap_ = std::max(need, (size_t)64 << 20);
          VRC_CUDA_CHECK(cudaMallocHost(&ext_host_, ext_cap_));
        }
      }
      cplx* hp = reinterpret_cast<cplx*>(ext_host_ + off);
      rc = s.host_sample(r->z, hp, hp + nn);
      if (rc == 0) {
        VRC_CUDA_CHECK(cudaMemcpyAsync(r->P, hp, nn * sizeof(cplx), cudaMemcpyHostToDevice, stream_));
        VRC_CUDA_CHECK(cudaMemcpyAsync(r->Q, hp + nn, nn * sizeof(cplx), cudaMemcpyHostToDevice, stream_));
        copied = true;
      }
      off += need;
    }
    if (rc != 0)
      throw StatusError(ST_EINVAL, "sampler callback failed (returned " + std::to_string(rc) + ") at z = " +
                                       std::to_string(r->z));
  }
  VRC_CUDA_CHECK(cudaEventRecord(ext_ev_, stream_));
}

void Engine::assemble(std::vector<SampleReq>& reqs_in, std::vector<int>* status) {
  if (reqs_in.empty()) return;
  // caller-sampler cells first; the rest (and their half-space ends) below
  std::vector<SampleReq*> ext;
  std::vector<int> keep;
  for (size_t i = 0; i < reqs_in.size(); ++i) {
    if (reqs_in[i].spec->kind == GEOM_SAMPLER && !reqs_in[i].homogeneous) ext.push_back(&reqs_in[i]);
    else keep.push_back((int)i);
  }
  sample_external(ext);
  if (status && status->size() < reqs_in.size()) status->resize(reqs_in.size(), 0);
  if (keep.empty()) return;
  std::vector<SampleReq> reqs;
  for (int i : keep) reqs.push_back(reqs_in[i]);
  std::vector<int> sub_status;
  assemble_grid(reqs, status ? &sub_status : nullptr);
  if (status)
    for (size_t q = 0; q < keep.size() && q < sub_status.size(); ++q)
      if (sub_status[q]) (*status)[keep[q]] = sub_status[q];
}

void Engine::assemble_grid(std::vector<SampleReq>& reqs, std::vector<int>* status) {
  if (reqs.empty()) return;
  std::map<AsmKey, std::vector<int>> groups;
  for (size_t i = 0; i < reqs.size(); ++i) {
    const auto& r = reqs[i];
    AsmKey k;
    k.nx = r.spec->nx;
    k.ny = r.spec->ny;
    k.pml = r.spec->pml ? 1 : 0;
    k.mirrored = r.mirrored ? 1 : 0;
    // a perturbed copy (the geometric adjoint's, with a host callback) shares
    // its structure's CellDev but not its rules: it stays on the host path
    k.devgeom = (!r.homogeneous && r.cd && r.cd->dev_geom && r.spec->kind == GEOM_GRID && !r.spec->geom_cb) ? 1 : 0;
    if (r.homogeneous) {
      k.ncx = 2;
      k.ncy = 2;
      k.pillar = 0;
    } else if (r.spec->kind == GEOM_PLANAR) {  // the cross-section's size depends on z
      std::vector<double> xs, ys;
      r.spec->planar_section(r.z, xs, ys, nullptr);
      k.ncx = (int)xs.size();
      k.ncy = (int)ys.size();
      k.pillar = 0;
    } else {
      k.ncx = r.spec->ncx();
      k.ncy = r.spec->ncy();
      k.pillar = r.spec->kind == GEOM_PILLAR ? 1 : 0;
    }
    groups[k].push_back((int)i);
  }
  for (auto& kv : groups) {
    const AsmKey& k = kv.first;
    const std::vector<int>& idx = kv.second;
    const int nx = k.nx, ny = k.ny, ncx = k.ncx, ncy = k.ncy;
    const int nc = ncx - 1, nr = ncy - 1, P = 2 * nx - 1, Q = 2 * ny - 1, m = nx * ny;
    // per-sample workspace (complex elements)
    const size_t o_eps = 0;
    const size_t o_inv = o_eps + ((k.pillar || k.devgeom) ? (size_t)nr * nc : 0);
    const size_t o_ex = o_inv + (size_t)nr * nc;
    const size_t o_exs = o_ex + (size_t)P * nc;
    const size_t o_ey = o_exs + (size_t)P * nc;
    const size_t o_ax = o_ey + (size_t)Q * nr;
    const size_t o_bx = o_ax + (size_t)P * nr;
    const size_t o_ay = o_bx + (size_t)P * nr;
    const size_t o_f2 = o_ay + (size_t)Q * nc;
    const size_t o_ti = o_f2 + (size_t)P * Q;
    const size_t o_tj = o_ti + (size_t)nx * nx * nr;
    const size_t o_g11 = o_tj + (size_t)ny * ny * nc;
    const size_t o_g22 = o_g11 + (size_t)nx * nx * Q;
    const size_t o_fe11 = o_g22 + (size_t)P * ny * ny;
    const size_t o_fe22 = o_fe11 + (size_t)m * m;
    const size_t o_fe33 = o_fe22 + (size_t)m * m;
    const size_t o_pml = o_fe33 + (size_t)m * m;
    const size_t per = (o_pml + (k.pml ? 6 * (size_t)m * m : 0) + 15) / 16 * 16;
    const size_t chunk = batch_chunk(idx.size(), per * 16, 8192, true);
    for (size_t c0 = 0; c0 < idx.size(); c0 += chunk) {
      const size_t B = std::min(chunk, idx.size() - c0);
      cplx* ws = (cplx*)workspace(B * per * 16);
      // host geometry
      std::vector<double> coords((size_t)B * (2 * ncx + ncy));
      std::vector<double> k0sq(B);
      std::vector<RasterDesc> rasters;  // pillars: one per sample
      std::vector<const cplx*> epsp(B), invp(B);
      std::vector<const double*> xp(B), xsp(B), yp(B);
      std::vector<cplx> homog_eps(B);
      std::vector<std::vector<cplx>> refilled;  // keep alive until sync
      std::vector<double> xv, yv;
      std::vector<GridGeomJob> gjobs;  // samples whose geometry the device forms
      for (size_t b = 0; b < B; ++b) {
        const SampleReq& r = reqs[idx[c0 + b]];
        const CellSpec& s = *r.spec;
        double* xo = coords.data() + b * (2 * ncx + ncy);
        double* xso = xo + ncx;
        double* yo = xso + ncx;
        k0sq[b] = s.k0() * s.k0();
        cplx* base = ws + b * per;
        if (r.homogeneous) {
          std::vector<double> x0, y0;
          s.geometry(r.z, x0, y0);
          xo[0] = x0.front();
          xo[1] = x0.back();
          yo[0] = y0.front();
          yo[1] = y0.back();
          xso[0] = xo[0];
          xso[1] = xo[1];
          homog_eps[b] = r.eps_h;
          epsp[b] = nullptr;  // set after upload
        } else if (k.devgeom) {
          gjobs.push_back({r.z, r.cd->geo_d, r.cd->geo_i, r.cd->nrules, (int)b, r.cd->eps_dev, base + o_eps, nullptr});
          epsp[b] = nullptr;  // set on the device
        } else {
          s.geometry(r.z, xv, yv);
          std::memcpy(xo, xv.data(), ncx * sizeof(double));
          std::memcpy(yo, yv.data(), ncy * sizeof(double));
          // sorted copy and painter's-order refill (FourierSolver1D.cpp:145-193)
          std::vector<int> index(ncx);
          std::iota(index.begin(), index.end(), 0);
          std::stable_sort(index.begin(), index.end(), [&](int a, int c) { return xv[a] < xv[c]; });
          std::vector<int> rindex(ncx);
          for (int i = 0; i < ncx; ++i) rindex[index[i]] = i;
          bool need = false;
          for (int i = 0; i + 1 < ncx; ++i)
            if (rindex[i] != i) need = true;
          for (int i = 0; i < ncx; ++i) xso[i] = xv[index[i]];
          if (k.pillar) {
            rasters.push_back({base + o_eps, s.radius(r.z), s.Lx, s.Ly, s.eps_in, s.eps_out});
            epsp[b] = base + o_eps;
          } else if (s.kind == GEOM_PLANAR) {  // crossings come sorted: no refill
            std::vector<double> px, py;
            refilled.emplace_back();
            s.planar_section(r.z, px, py, &refilled.back());
            epsp[b] = upload(refilled.back());
          } else if (need) {
            refilled.emplace_back(s.eps);
            std::vector<cplx>& nf = refilled.back();
            for (int row = 0; row < nr; ++row)
              for (int i = 0; i < nc; ++i) {
                if (xv[i] >= xv[i + 1]) continue;
                for (int j = 0; j < nc; ++j)
                  if (rindex[i] <= j && rindex[i + 1] >= j + 1) nf[(size_t)row * nc + j] = s.eps[(size_t)row * nc + i];
              }
            epsp[b] = upload(nf);
          } else {
            epsp[b] = r.cd->eps_dev;
          }
        }
        invp[b] = base + o_inv;
      }
      double* dcoords = upload(coords);
      for (size_t b = 0; b < B; ++b) {
        double* xo = dcoords + b * (2 * ncx + ncy);
        xp[b] = xo;
        xsp[b] = xo + ncx;
        yp[b] = xo + 2 * ncx;
        const SampleReq& r = reqs[idx[c0 + b]];
        if (r.homogeneous) epsp[b] = upload(&homog_eps[b], 1);
      }
      for (auto& j : gjobs) j.coords = dcoords + (size_t)j.slot * (2 * ncx + ncy);
      // one device array of eps pointers: the host's, completed on the device
      const cplx** d_eps = (const cplx**)upload(epsp);
      auto ptrs = [&](size_t off) {
        std::vector<cplx*> v(B);
        for (size_t b = 0; b < B; ++b) v[b] = ws + b * per + off;
        return v;
      };
      // Fourier/Toeplitz stage (A1-A4) timed as one family; algorithmic
      // bytes: eps raster in, fe11/fe22/fe33 out.
      const double asm_flops =
          8.0 * B * ((double)P * nr * nc * 2 + (double)Q * nc * nr + (double)P * Q * nr + (double)nx * nx * Q * nr +
                     (double)P * ny * ny * nc + (double)nr * nx * nx * nx + (double)nc * ny * ny * ny);
      const double asm_bytes = 16.0 * B * ((double)nr * nc + 3.0 * m * m);
      std::unique_ptr<Prof> asm_prof(
          new Prof(*this, "assembly", asm_flops, asm_bytes, 12 + (k.pillar ? 1 : 0) + (gjobs.empty() ? 0 : 1)));
      if (!gjobs.empty()) grid_geometry(upload(gjobs), (int)gjobs.size(), ncx, ncy, d_eps, stream_);
      if (k.pillar) pillar_raster(upload(rasters), (int)B, nc, nr, stream_);
      int* dstat = nullptr;
      if (status) {
        dstat = (int*)bytes(B * sizeof(int));
        VRC_CUDA_CHECK(cudaMemsetAsync(dstat, 0, B * sizeof(int), stream_));
      }
      auto ex = ptrs(o_ex), exs = ptrs(o_exs), ey = ptrs(o_ey);
      twiddles(upload(xp), upload(ex), (int)B, ncx, P, stream_);
      twiddles(upload(xsp), upload(exs), (int)B, ncx, P, stream_);
      twiddles(upload(yp), upload(ey), (int)B, ncy, Q, stream_);
      std::vector<cplx*> invv(B);
      for (size_t b = 0; b < B; ++b) invv[b] = const_cast<cplx*>(invp[b]);
      reciprocal(const_cast<cplx* const*>(d_eps), upload(invv), (int)B, nr * nc, stream_);
      auto cst = [](const std::vector<cplx*>& v) { return std::vector<const cplx*>(v.begin(), v.end()); };
      auto ax = ptrs(o_ax), bx = ptrs(o_bx), ay = ptrs(o_ay), f2 = ptrs(o_f2);
      // AX = Ex * inv_cm (nc x nr), BX = Ex * eps_cm
      small_gemm(P, nr, nc, upload(cst(ex)), P, upload(cst(invv)), nc, 0, upload(ax), P, (int)B, stream_);
      small_gemm(P, nr, nc, upload(cst(ex)), P, d_eps, nc, 0, upload(bx), P, (int)B, stream_);
      // AY = Ey * inv_cm^T  (Q x nc)
      small_gemm(Q, nc, nr, upload(cst(ey)), Q, upload(cst(invv)), nc, 1, upload(ay), Q, (int)B, stream_);
      // F2 = BX * Ey^T (P x Q)
      small_gemm(P, Q, nr, upload(cst(bx)), P, upload(cst(ey)), Q, 1, upload(f2), P, (int)B, stream_);
      auto ti = ptrs(o_ti), tj = ptrs(o_tj);
      toeplitz_inverses(upload(cst(ax)), upload(ti), nx, nr, (int)B, dstat, stream_);
      toeplitz_inverses(upload(cst(ay)), upload(tj), ny, nc, (int)B, dstat, stream_);
      auto g11 = ptrs(o_g11), g22 = ptrs(o_g22);
      small_gemm(nx * nx, Q, nr, upload(cst(ti)), nx * nx, upload(cst(ey)), Q, 1, upload(g11), nx * nx, (int)B,
                 stream_);
      small_gemm(P, ny * ny, nc, upload(cst(exs)), P, upload(cst(tj)), ny * ny, 1, upload(g22), P, (int)B, stream_);
      auto fe11 = ptrs(o_fe11), fe22 = ptrs(o_fe22), fe33 = ptrs(o_fe33);
      gather_fe(upload(cst(g11)), upload(cst(g22)), upload(cst(f2)), upload(fe11), upload(fe22), upload(fe33), nx,
                ny, (int)B, stream_);
      // (after the inverses: an asymmetric raster stays one whatever they report)
      if (k.pillar && k.mirrored && dstat) mirror_check(d_eps, (int)B, nc, nr, dstat, stream_);
      asm_prof.reset();
      // fe33^{-1} (BDCSVD solve of the square system, Layer.cpp:84-86)
      std::vector<int> inv_status;
      inverse(fe33, m, status ? &inv_status : nullptr);
      {
        std::vector<cplx*> ks, kd;
        for (size_t b = 0; b < B; ++b)
          if (reqs[idx[c0 + b]].keep_fe33inv) {
            ks.push_back(fe33[b]);
            kd.push_back(reqs[idx[c0 + b]].keep_fe33inv);
          }
        copy(ks, kd, m);
      }
      std::vector<cplx*> Pp(B), Qp(B);
      for (size_t b = 0; b < B; ++b) {
        Pp[b] = reqs[idx[c0 + b]].P;
        Qp[b] = reqs[idx[c0 + b]].Q;
      }
      if (!k.pml) {
        // all samples of a group share nx,ny but may belong to cells of
        // different periods: alpha/beta per sample
        std::vector<double> ab((size_t)B * 2 * m);
        for (size_t b = 0; b < B; ++b) {
          const CellDev* cd = reqs[idx[c0 + b]].cd;
          std::memcpy(ab.data() + b * 2 * m, cd->h_alpha.data(), m * sizeof(double));
          std::memcpy(ab.data() + b * 2 * m + m, cd->h_beta.data(), m * sizeof(double));
        }
        double* dab = upload(ab);
        double* dk = upload(k0sq);
        std::vector<const cplx*> fi(fe33.begin(), fe33.end()), f1(fe11.begin(), fe11.end()),
            f2v(fe22.begin(), fe22.end());
        Prof pr(*this, "assembly", 0.0, 16.0 * B * (3.0 * m * m + 8.0 * m * m));
        assemble_periodic(upload(fi), upload(f1), upload(f2v), dab, dk, upload(Pp), upload(Qp), m, (int)B, stream_);
      } else {
        auto F1h = ptrs(o_pml), F2h = ptrs(o_pml + (size_t)m * m), KxF2h = ptrs(o_pml + 2 * (size_t)m * m),
             KxF1h = ptrs(o_pml + 3 * (size_t)m * m), KyF2h = ptrs(o_pml + 4 * (size_t)m * m),
             KyF1h = ptrs(o_pml + 5 * (size_t)m * m);
        std::vector<GemmDesc> g1, g2;
        for (size_t b = 0; b < B; ++b) {
          const CellDev* cd = reqs[idx[c0 + b]].cd;
          g1.push_back({fe33[b], cd->Kx, F1h[b], nullptr, nullptr, nullptr});
          g1.push_back({fe33[b], cd->Ky, F2h[b], nullptr, nullptr, nullptr});
        }
        gemm(g1, m, mk(1, 0), mk(0, 0), 0.0);
        for (size_t b = 0; b < B; ++b) {
          const CellDev* cd = reqs[idx[c0 + b]].cd;
          g2.push_back({cd->Kx, F2h[b], KxF2h[b], nullptr, nullptr, nullptr});
          g2.push_back({cd->Kx, F1h[b], KxF1h[b], nullptr, nullptr, nullptr});
          g2.push_back({cd->Ky, F2h[b], KyF2h[b], nullptr, nullptr, nullptr});
          g2.push_back({cd->Ky, F1h[b], KyF1h[b], nullptr, nullptr, nullptr});
        }
        gemm(g2, m, mk(1, 0), mk(0, 0), 0.0);
        double* dk = upload(k0sq);
        std::vector<const cplx*> kxky(B), kxkx(B), kyky(B), kykx(B);
        for (size_t b = 0; b < B; ++b) {
          const CellDev* cd = reqs[idx[c0 + b]].cd;
          kxky[b] = cd->KxKy;
          kxkx[b] = cd->KxKx;
          kyky[b] = cd->KyKy;
          kykx[b] = cd->KyKx;
        }
        auto cv = [](const std::vector<cplx*>& v) { return std::vector<const cplx*>(v.begin(), v.end()); };
        Prof pr(*this, "assembly", 0.0, 16.0 * B * (6.0 * m * m + 8.0 * m * m));
        assemble_dense(upload(cv(KxF2h)), upload(cv(KxF1h)), upload(cv(KyF2h)), upload(cv(KyF1h)), upload(cv(fe11)),
                       upload(cv(fe22)), upload(kxky), upload(kxkx), upload(kyky), upload(kykx), dk, upload(Pp),
                       upload(Qp), m, (int)B, stream_);
      }
      if (status) {
        std::vector<int> h(B);
        VRC_CUDA_CHECK(cudaMemcpyAsync(h.data(), dstat, B * sizeof(int), cudaMemcpyDeviceToHost, stream_));
        sync();
        free_bytes(dstat, B * sizeof(int));
        if (status->size() < reqs.size()) status->resize(reqs.size(), 0);
        for (size_t b = 0; b < B; ++b) {
          int st = h[b] ? h[b] : (b < inv_status.size() ? inv_status[b] : 0);
          if (st) (*status)[idx[c0 + b]] = st;
        }
      } else {
        sync();  // refilled host tables must outlive their uploads
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Eigen-decomposition of PQ (A7)
// ---------------------------------------------------------------------------
// Blocked Hessenberg reduction (panels + DMMA GEMM updates) from the order up at
// which the matrix no longer fits the shared memory of one CTA: one / 600
// matrices in ms, shared memory against blocked, n = 61 0.21 / 0.73 against 0.49 /
// 1.6, n = 98 0.58 / 2.9 against 0.93 / 4.1, n = 115 0.76 / 3.9 against 1.02 / 5.3;
// from global memory, against blocked, 2.65 / 1.48 for eight at n = 126.
// VRC_HESS_BLOCKED=0 / 1 turns it off / on for every order.
static bool use_blocked_hessenberg(int n) {
  if (const char* e = std::getenv("VRC_HESS_BLOCKED")) return std::atoi(e) != 0 && n >= 3;
  return n > hessenberg_smem_maxn();
}

void Engine::eig(std::vector<EigReq>& reqs, int n, std::vector<int>* status) {
  if (reqs.empty()) return;
  const size_t logc = schur_log_bytes(n) / 16;  // rotation log, complex units
  const size_t per = (size_t)3 * n * n + 2 * (size_t)((n + 15) / 16 * 16) + logc;
  const size_t chunk = batch_chunk(reqs.size(), per * 16, 16384, true);
  if (status && status->size() < reqs.size()) status->resize(reqs.size(), 0);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    cplx* ws = (cplx*)workspace(B * per * 16);
    std::vector<cplx*> H(B), Z(B), Y(B), lam(B), ig(B), W(B), V(B), gam(B);
    std::vector<void*> logs(B);
    std::vector<GemmDesc> g;
    for (size_t b = 0; b < B; ++b) {
      cplx* base = ws + b * per;
      H[b] = base;
      Z[b] = base + (size_t)n * n;
      Y[b] = base + 2 * (size_t)n * n;
      lam[b] = base + 3 * (size_t)n * n;
      ig[b] = lam[b] + (n + 15) / 16 * 16;
      logs[b] = ig[b] + (n + 15) / 16 * 16;
      const EigReq& r = reqs[c0 + b];
      W[b] = r.W;
      V[b] = r.V;
      gam[b] = r.gam;
      if (r.Q) g.push_back({r.P, r.Q, H[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // PQ = P*Q
    {
      // a request without Q asks for the eigenpairs of P itself
      std::vector<cplx*> src, dst;
      for (size_t b = 0; b < B; ++b)
        if (!reqs[c0 + b].Q) {
          src.push_back(const_cast<cplx*>(reqs[c0 + b].P));
          dst.push_back(H[b]);
        }
      if (!src.empty()) copy(src, dst, n);
    }
    // nominal LAPACK counts (real flops): zgehrd 40/3 n^3 + zunghr 16/3 n^3,
    // complex Schur with Z ~ 80 n^3, ztrevc 4/3 n^3
    const double nn3 = (double)n * n * n, mbytes = 16.0 * n * (double)n;
    {
      Prof pr(*this, "hessenberg", (56.0 / 3.0) * nn3 * B, 3.0 * mbytes * B);
      if (use_blocked_hessenberg(n)) {
        // panels with DMMA GEMM updates; the panel scratch lives in each
        // matrix's Y block (free until the back substitution) when it fits
        const size_t need = hessenberg_blocked_scratch(n);
        const bool in_y = need <= (size_t)n * n * 16;
        for (size_t b0 = 0; b0 < B; b0 += 65535) {
          const size_t nb = std::min<size_t>(65535, B - b0);
          void* scr = in_y ? (void*)Y[b0] : bytes(nb * need);
          void* dd = bytes(hessenberg_blocked_descs((int)nb));
          std::vector<cplx*> hb(H.begin() + b0, H.begin() + b0 + nb), zb(Z.begin() + b0, Z.begin() + b0 + nb);
          hessenberg_blocked_batched(upload(hb), upload(zb), (int)nb, n, scr, in_y ? per * 16 : need, dd, stream_);
          free_bytes(dd, hessenberg_blocked_descs((int)nb));
          if (!in_y) free_bytes(scr, nb * need);
        }
      } else {
        hessenberg_batched(upload(H), upload(Z), (int)B, n, stream_);
      }
    }
    int* dstat = (int*)bytes(B * sizeof(int));
    VRC_CUDA_CHECK(cudaMemsetAsync(dstat, 0, B * sizeof(int), stream_));
    {
      cplx* const* dH = upload(H);
      cplx* const* dZ = upload(Z);
      cplx* const* dL = upload(lam);
      void* const* dG = upload(logs);
      {
        // nominal LAPACK count for the complex Schur form with vectors (~80 n^3
        // real), half for T's active windows, half for the replay onto Z and
        // the rest of T
        Prof pr(*this, "schur_qr", 40.0 * nn3 * B, 4.0 * mbytes * B);
        schur_batched(dH, dZ, dL, dG, (int)B, n, dstat, stream_, SCHUR_ITERATE);
      }
      Prof pr(*this, "schur_replay", 40.0 * nn3 * B, 4.0 * mbytes * B, 2);
      schur_batched(dH, dZ, dL, dG, (int)B, n, dstat, stream_, SCHUR_REPLAY);
    }
    if (std::getenv("VRC_QR_STATS")) {
      // diagnostic: per-matrix QR counters from the rotation-log headers
      double tot[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
      for (size_t b = 0; b < B; ++b) {
        int hh[4];
        long long tt[6];
        VRC_CUDA_CHECK(cudaMemcpyAsync(hh, logs[b], sizeof(hh), cudaMemcpyDeviceToHost, stream_));
        VRC_CUDA_CHECK(cudaMemcpyAsync(tt, (char*)logs[b] + 16, sizeof(tt), cudaMemcpyDeviceToHost, stream_));
        sync();
        for (int q = 0; q < 4; ++q) tot[q] += hh[q];
        for (int q = 0; q < 6; ++q) tot[4 + q] += (double)tt[q];
      }
      {
        // sweep-size profile of the first matrix: rounds spent in sweeps on
        // windows of each size class
        int hh[4];
        VRC_CUDA_CHECK(cudaMemcpyAsync(hh, logs[0], sizeof(hh), cudaMemcpyDeviceToHost, stream_));
        sync();
        std::vector<int> rec((size_t)hh[0] * 8);
        if (hh[0] > 0)
          VRC_CUDA_CHECK(cudaMemcpyAsync(rec.data(), (char*)logs[0] + 64, rec.size() * sizeof(int),
                                         cudaMemcpyDeviceToHost, stream_));
        sync();
        double cls[6] = {0, 0, 0, 0, 0, 0};
        int cnt[6] = {0, 0, 0, 0, 0, 0};
        for (int q = 0; q < hh[0]; ++q) {
          const int w = rec[q * 8 + 1] - rec[q * 8] + 1, R = rec[q * 8 + 3];
          const int c = w <= 8 ? 0 : w <= 16 ? 1 : w <= 32 ? 2 : w <= 64 ? 3 : w <= 128 ? 4 : 5;
          cls[c] += R;
          cnt[c] += 1;
        }
        fprintf(stderr, "[vrc qr] first matrix: window<=8: %d sweeps %.0f rounds; <=16: %d %.0f; <=32: %d %.0f; "
                        "<=64: %d %.0f; <=128: %d %.0f; >128: %d %.0f\n",
                cnt[0], cls[0], cnt[1], cls[1], cnt[2], cls[2], cnt[3], cls[3], cnt[4], cls[4], cnt[5], cls[5]);
      }
      fprintf(stderr,
              "[vrc qr] n=%d matrices=%zu per matrix: log entries=%.1f (deflation windows %.1f) rounds=%.0f "
              "rotation slots=%.0f (%.2f n^2) Mcycles defl=%.2f shift+window=%.2f (window Schur %.2f, "
              "window deflation %.2f) rounds=%.2f far=%.2f\n",
              n, B, tot[0] / B, tot[3] / B, tot[2] / B, tot[1] / B, tot[1] / B / ((double)n * n), tot[4] / B / 1e6,
              tot[5] / B / 1e6, tot[8] / B / 1e6, tot[9] / B / 1e6, tot[6] / B / 1e6, tot[7] / B / 1e6);
    }
    {
      Prof pr(*this, "trevc", (4.0 / 3.0) * nn3 * B, 1.5 * mbytes * B);
      trevc_batched(upload(H), upload(Y), (int)B, n, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({Z[b], Y[b], W[b], nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // X = Z Y
    {
      Prof pr(*this, "elementwise", 0.0, 2.0 * mbytes * B, 2);
      vecnorm_batched(upload(W), (int)B, n, stream_);
      std::vector<const cplx*> lamc(lam.begin(), lam.end());
      gamma_batched(upload(lamc), upload(gam), upload(ig), (int)B, n, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b)
      if (reqs[c0 + b].Q) g.push_back({reqs[c0 + b].Q, W[b], V[b], nullptr, nullptr, ig[b]});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // V = Q W diag(1/gamma)
    // W^-1 by inversion; V^-1 = Gamma^-1 W^-1 P (from V = Q W Gamma^-1 and
    // P Q = W Gamma^2 W^-1: (Gamma^-1 W^-1 P)(Q W Gamma^-1) = I), one GEMM
    // instead of a second inversion
    std::vector<cplx*> srcs, dsts;
    std::vector<size_t> inv_req;  // request of each inverted matrix
    for (size_t b = 0; b < B; ++b) {
      const bool wi = reqs[c0 + b].Winv || (reqs[c0 + b].Vinv && reqs[c0 + b].Q);
      if (wi) {
        srcs.push_back(W[b]);
        dsts.push_back(reqs[c0 + b].Winv ? reqs[c0 + b].Winv : H[b]);  // H is free scratch by now
        inv_req.push_back(b);
      } else if (reqs[c0 + b].Vinv) {
        srcs.push_back(V[b]);
        dsts.push_back(reqs[c0 + b].Vinv);
        inv_req.push_back(b);
      }
    }
    copy(srcs, dsts, n);
    std::vector<int> ist;
    inverse(dsts, n, status ? &ist : nullptr);
    g.clear();
    for (size_t q = 0; q < inv_req.size(); ++q) {
      const size_t b = inv_req[q];
      if (reqs[c0 + b].Vinv && reqs[c0 + b].Q && srcs[q] == W[b])
        g.push_back({dsts[q], reqs[c0 + b].P, reqs[c0 + b].Vinv, nullptr, ig[b], nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // V^-1 = diag(1/gamma) W^-1 P
    for (size_t b = 0; b < B; ++b)
      if (reqs[c0 + b].lam)
        VRC_CUDA_CHECK(cudaMemcpyAsync(reqs[c0 + b].lam, lam[b], (size_t)n * 16, cudaMemcpyDeviceToDevice, stream_));
    std::vector<int> h(B);
    VRC_CUDA_CHECK(cudaMemcpyAsync(h.data(), dstat, B * sizeof(int), cudaMemcpyDeviceToHost, stream_));
    sync();
    free_bytes(dstat, B * sizeof(int));
    if (status) {
      for (size_t b = 0; b < B; ++b)
        if (h[b]) (*status)[c0 + b] = h[b];
      for (size_t q = 0; q < inv_req.size() && q < ist.size(); ++q)
        if (ist[q] && !(*status)[c0 + inv_req[q]]) (*status)[c0 + inv_req[q]] = ist[q];
    }
  }
}

// ---------------------------------------------------------------------------
// Perturbative segments (A8)
// ---------------------------------------------------------------------------
void Engine::segments(std::vector<SegReq>& reqs, int n) {
  if (reqs.empty()) return;
  const size_t nn = (size_t)n * n;
  const size_t per = 6 * nn;
  const size_t chunk = batch_chunk(reqs.size(), per * 16, 16384, true);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    cplx* ws = (cplx*)workspace(B * per * 16);
    std::vector<const cplx*> A1, A2;
    std::vector<cplx*> D(B), T(B), X0(B), Y0(B), X2(B), Y2(B);
    for (size_t b = 0; b < B; ++b) {
      cplx* base = ws + b * per;
      D[b] = base;
      T[b] = base + nn;
      X0[b] = base + 2 * nn;
      Y0[b] = base + 3 * nn;
      X2[b] = base + 4 * nn;
      Y2[b] = base + 5 * nn;
    }
    auto one = [&](int side, int pq) {
      // D = S_k - S_ref ; T = D * (V | W) ; out = (Winv | Vinv) * T
      std::vector<const cplx*> a(B), r(B);
      std::vector<GemmDesc> g1, g2;
      for (size_t b = 0; b < B; ++b) {
        const SegReq& s = reqs[c0 + b];
        a[b] = pq == 0 ? (side == 0 ? s.Pa : s.Pb) : (side == 0 ? s.Qa : s.Qb);
        r[b] = pq == 0 ? s.Pr : s.Qr;
        cplx* out = side == 0 ? (pq == 0 ? X0[b] : Y0[b]) : (pq == 0 ? X2[b] : Y2[b]);
        g1.push_back({D[b], pq == 0 ? s.V : s.W, T[b], nullptr, nullptr, nullptr});
        g2.push_back({pq == 0 ? s.Winv : s.Vinv, T[b], out, nullptr, nullptr, nullptr});
      }
      {
        Prof pr(*this, "elementwise", 0.0, 48.0 * nn * B);
        sub_batched(upload(a), upload(r), upload(D), (int)B, (long long)nn, stream_);
      }
      gemm(g1, n, mk(1, 0), mk(0, 0), 0.0);
      gemm(g2, n, mk(1, 0), mk(0, 0), 0.0);
    };
    one(0, 0);
    one(0, 1);
    one(1, 0);
    one(1, 1);
    std::vector<SegDesc> sd(B);
    for (size_t b = 0; b < B; ++b) {
      const SegReq& s = reqs[c0 + b];
      sd[b] = {X0[b], Y0[b], X2[b], Y2[b], s.gam, s.tdd, s.tuu, s.rud, s.rdu, s.err, s.z0, s.z1, s.k0};
    }
    {
      Prof pr(*this, "simpson", 0.0, 16.0 * 8.0 * nn * B);
      simpson_batched(upload(sd), (int)B, n, stream_);
    }
  }
}

// ---------------------------------------------------------------------------
// Projections (A9) and star products (A10)
// ---------------------------------------------------------------------------
void Engine::project_left(std::vector<ProjReq>& reqs, int n, std::vector<int>* status) {
  if (reqs.empty()) return;
  const size_t nn = (size_t)n * n;
  const size_t per = 6 * nn;
  const size_t chunk = batch_chunk(reqs.size(), per * 16, 16384, true);
  if (status && status->size() < reqs.size()) status->resize(reqs.size(), 0);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    cplx* ws = (cplx*)workspace(B * per * 16);
    std::vector<cplx*> A(B), Bm(B), M(B), T1(B), T2(B), T3(B);
    for (size_t b = 0; b < B; ++b) {
      cplx* base = ws + b * per;
      A[b] = base;
      Bm[b] = base + nn;
      M[b] = base + 2 * nn;
      T1[b] = base + 3 * nn;
      T2[b] = base + 4 * nn;
      T3[b] = base + 5 * nn;
    }
    std::vector<GemmDesc> g;
    for (size_t b = 0; b < B; ++b) {
      const ProjReq& r = reqs[c0 + b];
      g.push_back({r.Winv, r.leftW, A[b], nullptr, nullptr, nullptr});
      g.push_back({r.Vinv, r.leftV, Bm[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    {
      Prof pr(*this, "elementwise", 0.0, 64.0 * nn * B);
      ab_batched(upload(A), upload(Bm), (int)B, (long long)nn, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].rdu, Bm[b], M[b], A[b], nullptr, nullptr});
    gemm(g, n, mk(-1, 0), mk(1, 0), 0.0);  // M = A - rdu B
    std::vector<int> ist;
    inverse(M, n, status ? &ist : nullptr);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].rdu, A[b], T1[b], Bm[b], nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(-1, 0), 0.0);  // T1 = rdu A - B
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const ProjReq& r = reqs[c0 + b];
      g.push_back({M[b], T1[b], r.rdu, nullptr, nullptr, nullptr});  // rdu' = M^-1 T1
      g.push_back({M[b], r.tdd, T2[b], nullptr, nullptr, nullptr});  // T2 = M^-1 tdd
      g.push_back({r.tuu, Bm[b], T3[b], nullptr, nullptr, nullptr});  // T3 = tuu B
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    std::vector<cplx*> src, dst;
    for (size_t b = 0; b < B; ++b) {
      src.push_back(T2[b]);
      dst.push_back(reqs[c0 + b].tdd);
    }
    copy(src, dst, n);  // tdd' = T2
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const ProjReq& r = reqs[c0 + b];
      g.push_back({T3[b], r.tdd, r.rud, r.rud, nullptr, nullptr});  // rud' = tuu B tdd' + rud
      g.push_back({r.tuu, A[b], T1[b], nullptr, nullptr, nullptr});  // T1 = tuu A
    }
    gemm(g, n, mk(1, 0), mk(1, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({T3[b], reqs[c0 + b].rdu, reqs[c0 + b].tuu, T1[b], nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(1, 0), 0.0);  // tuu' = tuu B rdu' + tuu A
    if (status)
      for (size_t b = 0; b < ist.size(); ++b)
        if (ist[b]) (*status)[c0 + b] = ist[b];
  }
}

void Engine::project_right(std::vector<ProjRReq>& reqs, int n, std::vector<int>* status) {
  if (reqs.empty()) return;
  const size_t nn = (size_t)n * n;
  const size_t per = 6 * nn;
  const size_t chunk = batch_chunk(reqs.size(), per * 16, 16384, true);
  if (status && status->size() < reqs.size()) status->resize(reqs.size(), 0);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    cplx* ws = (cplx*)workspace(B * per * 16);
    std::vector<cplx*> A(B), Bm(B), M(B), T1(B), T2(B), T3(B);
    for (size_t b = 0; b < B; ++b) {
      cplx* base = ws + b * per;
      A[b] = base;
      Bm[b] = base + nn;
      M[b] = base + 2 * nn;
      T1[b] = base + 3 * nn;
      T2[b] = base + 4 * nn;
      T3[b] = base + 5 * nn;
    }
    std::vector<GemmDesc> g;
    for (size_t b = 0; b < B; ++b) {
      const ProjRReq& r = reqs[c0 + b];
      g.push_back({r.leftWinv, r.W1, A[b], nullptr, nullptr, nullptr});
      g.push_back({r.leftVinv, r.V1, Bm[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    {
      Prof pr(*this, "elementwise", 0.0, 64.0 * nn * B);
      ab_batched(upload(A), upload(Bm), (int)B, (long long)nn, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].Rud, Bm[b], M[b], A[b], nullptr, nullptr});
    gemm(g, n, mk(-1, 0), mk(1, 0), 0.0);  // M = A - Rud B
    std::vector<int> ist;
    inverse(M, n, status ? &ist : nullptr);
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const ProjRReq& r = reqs[c0 + b];
      g.push_back({M[b], r.Tuu, T1[b], nullptr, nullptr, nullptr});  // Tuu' = M^-1 Tuu
      g.push_back({r.Tdd, Bm[b], T3[b], nullptr, nullptr, nullptr});  // T3 = Tdd B
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].Rud, A[b], T2[b], Bm[b], nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(-1, 0), 0.0);  // T2 = Rud A - B
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({M[b], T2[b], reqs[c0 + b].Rud, nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // Rud' = M^-1 T2
    std::vector<cplx*> src, dst;
    for (size_t b = 0; b < B; ++b) {
      src.push_back(T1[b]);
      dst.push_back(reqs[c0 + b].Tuu);
    }
    copy(src, dst, n);
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const ProjRReq& r = reqs[c0 + b];
      g.push_back({T3[b], r.Tuu, r.Rdu, r.Rdu, nullptr, nullptr});  // Rdu' = Rdu + Tdd B Tuu'
      g.push_back({Bm[b], r.Rud, T2[b], A[b], nullptr, nullptr});    // T2 = B Rud' + A
    }
    gemm(g, n, mk(1, 0), mk(1, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].Tdd, T2[b], T1[b], nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // T1 = Tdd (B Rud' + A)
    src.clear();
    dst.clear();
    for (size_t b = 0; b < B; ++b) {
      src.push_back(T1[b]);
      dst.push_back(reqs[c0 + b].Tdd);
    }
    copy(src, dst, n);
    if (status)
      for (size_t b = 0; b < ist.size(); ++b)
        if (ist[b]) (*status)[c0 + b] = ist[b];
  }
}

void Engine::project_left_end(std::vector<ProjLEReq>& reqs, int n, std::vector<int>* status) {
  std::vector<ProjReq> p;
  for (auto& r : reqs) p.push_back({r.W1inv, r.V1inv, r.W0, r.V0, r.Tdd, r.Tuu, r.Rud, r.Rdu});
  project_left(p, n, status);
}

void Engine::star(std::vector<StarReq>& reqs, int n, std::vector<int>* status) {
  if (reqs.empty()) return;
  const size_t nn = (size_t)n * n;
  const size_t per = 7 * nn;
  const size_t chunk = batch_chunk(reqs.size(), per * 16, 16384, true);
  if (status && status->size() < reqs.size()) status->resize(reqs.size(), 0);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    cplx* ws = (cplx*)workspace(B * per * 16);
    std::vector<cplx*> X1(B), X2(B), X3(B), X4(B), X5(B), X6(B), X7(B);
    for (size_t b = 0; b < B; ++b) {
      cplx* base = ws + b * per;
      X1[b] = base;
      X2[b] = base + nn;
      X3[b] = base + 2 * nn;
      X4[b] = base + 3 * nn;
      X5[b] = base + 4 * nn;
      X6[b] = base + 5 * nn;
      X7[b] = base + 6 * nn;
    }
    std::vector<GemmDesc> g;
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].rdu, reqs[c0 + b].Rud, X1[b], nullptr, nullptr, nullptr});
    gemm(g, n, mk(-1, 0), mk(0, 0), 1.0);  // X1 = I - rdu Rud
    std::vector<int> ist;
    inverse(X1, n, status ? &ist : nullptr);  // C1
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const StarReq& r = reqs[c0 + b];
      g.push_back({r.Rud, X1[b], X2[b], nullptr, nullptr, nullptr});  // X2 = Rud C1
      g.push_back({X1[b], r.tdd, X4[b], nullptr, nullptr, nullptr});  // X4 = C1 tdd
      g.push_back({r.tuu, r.Rud, X5[b], nullptr, nullptr, nullptr});  // X5 = tuu Rud
      g.push_back({r.Tdd, r.rdu, X7[b], nullptr, nullptr, nullptr});  // X7 = Tdd rdu
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({X2[b], reqs[c0 + b].rdu, X3[b], nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 1.0);  // C2 = I + Rud C1 rdu
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const StarReq& r = reqs[c0 + b];
      g.push_back({r.Tdd, X4[b], r.oTdd, nullptr, nullptr, nullptr});  // Tdd' = Tdd C1 tdd
      g.push_back({X3[b], r.Tuu, X6[b], nullptr, nullptr, nullptr});   // X6 = C2 Tuu
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const StarReq& r = reqs[c0 + b];
      g.push_back({X5[b], X4[b], r.oRud, r.rud, nullptr, nullptr});  // Rud' = rud + tuu Rud C1 tdd
      g.push_back({X7[b], X6[b], r.oRdu, r.Rdu, nullptr, nullptr});  // Rdu' = Rdu + Tdd rdu C2 Tuu
    }
    gemm(g, n, mk(1, 0), mk(1, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].tuu, X6[b], reqs[c0 + b].oTuu, nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // Tuu' = tuu C2 Tuu
    if (status)
      for (size_t b = 0; b < ist.size(); ++b)
        if (ist[b]) (*status)[c0 + b] = ist[b];
  }
}

void Engine::star_reduce(std::vector<std::vector<SBlocks>>& lists, int n, std::vector<int>* cell_status) {
  while (true) {
    std::vector<StarReq> reqs;
    std::vector<std::pair<int, int>> where;  // (cell, pair index)
    std::vector<std::vector<SBlocks>> next(lists.size());
    for (size_t c = 0; c < lists.size(); ++c) {
      auto& L = lists[c];
      for (size_t i = 0; i + 1 < L.size(); i += 2) {
        SBlocks o{mat(n), mat(n), mat(n), mat(n)};
        reqs.push_back({L[i].tdd, L[i].tuu, L[i].rud, L[i].rdu, L[i + 1].tdd, L[i + 1].tuu, L[i + 1].rud,
                        L[i + 1].rdu, o.tdd, o.tuu, o.rud, o.rdu});
        where.push_back({(int)c, (int)next[c].size()});
        next[c].push_back(o);
      }
      if (L.size() % 2 == 1) next[c].push_back(L.back());
    }
    if (reqs.empty()) break;
    std::vector<int> st;
    star(reqs, n, cell_status ? &st : nullptr);
    if (cell_status)
      for (size_t i = 0; i < st.size(); ++i)
        if (st[i]) (*cell_status)[where[i].first] = st[i];
    // release consumed inputs (stream order keeps them valid for the kernels)
    for (auto& r : reqs) {
      free_mat(const_cast<cplx*>(r.Tdd), n);
      free_mat(const_cast<cplx*>(r.Tuu), n);
      free_mat(const_cast<cplx*>(r.Rud), n);
      free_mat(const_cast<cplx*>(r.Rdu), n);
      free_mat(const_cast<cplx*>(r.tdd), n);
      free_mat(const_cast<cplx*>(r.tuu), n);
      free_mat(const_cast<cplx*>(r.rud), n);
      free_mat(const_cast<cplx*>(r.rdu), n);
    }
    lists.swap(next);
  }
}

// ---------------------------------------------------------------------------
// RCWA slab (A12) and differential slice (A13)
// ---------------------------------------------------------------------------
void Engine::rcwa_slabs(std::vector<SlabReq>& reqs, int n, std::vector<int>* status) {
  if (reqs.empty()) return;
  const size_t nn = (size_t)n * n;
  // eigen outputs are pool-allocated per request; temps are pooled too
  if (status && status->size() < reqs.size()) status->resize(reqs.size(), 0);
  const size_t per_bytes = 16 * nn * 16;
  const size_t chunk = batch_chunk(reqs.size(), per_bytes, 4096, false);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    std::vector<EigReq> er(B);
    std::vector<cplx*> W(B), V(B), Wi(B), Vi(B), gam(B), A(B), Bm(B), Ai(B), iAB(B), XA(B), XB(B), iAXA(B),
        iAXB(B), M(B), T1(B);
    for (size_t b = 0; b < B; ++b) {
      W[b] = mat(n); V[b] = mat(n); Wi[b] = mat(n); Vi[b] = mat(n); gam[b] = vec(n);
      A[b] = mat(n); Bm[b] = mat(n); Ai[b] = mat(n); iAB[b] = mat(n); XA[b] = mat(n); XB[b] = mat(n);
      iAXA[b] = mat(n); iAXB[b] = mat(n); M[b] = mat(n); T1[b] = mat(n);
      er[b] = {reqs[c0 + b].P, reqs[c0 + b].Q, W[b], V[b], Wi[b], Vi[b], gam[b]};
    }
    std::vector<int> est;
    eig(er, n, status ? &est : nullptr);
    std::vector<GemmDesc> g;
    for (size_t b = 0; b < B; ++b) {
      g.push_back({Wi[b], reqs[c0 + b].W1, A[b], nullptr, nullptr, nullptr});
      g.push_back({Vi[b], reqs[c0 + b].V1, Bm[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    // A, B = (F0 +- G0)/2; the common factor 1/2 is exact and cancels
    {
      Prof pr(*this, "elementwise", 0.0, 64.0 * nn * B);
      ab_batched(upload(A), upload(Bm), (int)B, (long long)nn, stream_);
    }
    copy(A, Ai, n);
    std::vector<int> ist;
    inverse(Ai, n, status ? &ist : nullptr);
    std::vector<double> ts(B);
    for (size_t b = 0; b < B; ++b) ts[b] = reqs[c0 + b].dz / reqs[c0 + b].k0;
    double* dts = upload(ts);
    std::vector<const cplx*> Ac(A.begin(), A.end()), Bc(Bm.begin(), Bm.end()), gc(gam.begin(), gam.end());
    {
      Prof pr(*this, "elementwise", 0.0, 64.0 * nn * B, 2);
      phase_rows_batched(upload(Ac), upload(gc), dts, upload(XA), (int)B, n, stream_);
      phase_rows_batched(upload(Bc), upload(gc), dts, upload(XB), (int)B, n, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      g.push_back({Ai[b], Bm[b], iAB[b], nullptr, nullptr, nullptr});
      g.push_back({Ai[b], XA[b], iAXA[b], nullptr, nullptr, nullptr});
      g.push_back({Ai[b], XB[b], iAXB[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({iAXB[b], iAXB[b], M[b], nullptr, nullptr, nullptr});
    gemm(g, n, mk(-1, 0), mk(0, 0), 1.0);  // M = I - (A^-1 X B)^2
    std::vector<int> mst;
    inverse(M, n, status ? &mst : nullptr);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({iAXB[b], iAXA[b], T1[b], iAB[b], nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(-1, 0), 0.0);  // T1 = iAXB iAXA - iAB
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({M[b], T1[b], reqs[c0 + b].rud, nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // Rud
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({iAXB[b], iAB[b], T1[b], iAXA[b], nullptr, nullptr});
    gemm(g, n, mk(-1, 0), mk(1, 0), 0.0);  // T1 = iAXA - iAXB iAB
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({M[b], T1[b], reqs[c0 + b].tuu, nullptr, nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);  // Tuu
    if (status)
      for (size_t b = 0; b < B; ++b) {
        int s = (b < est.size() && est[b]) ? est[b] : ((b < ist.size() && ist[b]) ? ist[b] : (b < mst.size() ? mst[b] : 0));
        if (s) (*status)[c0 + b] = s;
      }
    for (size_t b = 0; b < B; ++b) {
      free_mat(W[b], n); free_mat(V[b], n); free_mat(Wi[b], n); free_mat(Vi[b], n); free_vec(gam[b], n);
      free_mat(A[b], n); free_mat(Bm[b], n); free_mat(Ai[b], n); free_mat(iAB[b], n); free_mat(XA[b], n);
      free_mat(XB[b], n); free_mat(iAXA[b], n); free_mat(iAXB[b], n); free_mat(M[b], n); free_mat(T1[b], n);
    }
  }
}

void Engine::diff_slices(std::vector<DiffReq>& reqs, int n, std::vector<int>* status) {
  if (reqs.empty()) return;
  if (status && status->size() < reqs.size()) status->resize(reqs.size(), 0);
  const size_t nn = (size_t)n * n;
  const size_t chunk = batch_chunk(reqs.size(), 24 * nn * 16, 4096, false);
  for (size_t c0 = 0; c0 < reqs.size(); c0 += chunk) {
    const size_t B = std::min(chunk, reqs.size() - c0);
    const int NT = 20;
    std::vector<std::vector<cplx*>> t(NT, std::vector<cplx*>(B));
    for (int k = 0; k < NT; ++k)
      for (size_t b = 0; b < B; ++b) t[k][b] = mat(n);
    auto& P1Q0 = t[0]; auto& P1Q1 = t[1]; auto& P2Q1 = t[2]; auto& X4 = t[3];
    auto& L11 = t[4]; auto& L12 = t[5]; auto& L21 = t[6]; auto& L22 = t[7];
    auto& Q1P0 = t[8]; auto& Q1P1 = t[9]; auto& Q2P1 = t[10]; auto& Y4 = t[11];
    auto& U1 = t[12]; auto& U2 = t[13]; auto& U3 = t[14]; auto& U4 = t[15];
    auto& T11 = t[16]; auto& T12 = t[17]; auto& T21 = t[18]; auto& T22 = t[19];
    std::vector<GemmDesc> g;
    for (size_t b = 0; b < B; ++b) {
      const DiffReq& r = reqs[c0 + b];
      g.push_back({r.P1, r.Q0, P1Q0[b], nullptr, nullptr, nullptr});
      g.push_back({r.P1, r.Q1, P1Q1[b], nullptr, nullptr, nullptr});
      g.push_back({r.P2, r.Q1, P2Q1[b], nullptr, nullptr, nullptr});
      g.push_back({r.Q1, r.P0, Q1P0[b], nullptr, nullptr, nullptr});
      g.push_back({r.Q1, r.P1, Q1P1[b], nullptr, nullptr, nullptr});
      g.push_back({r.Q2, r.P1, Q2P1[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    // L11 = I - a2 (P1Q0 + P1Q1 + P2Q1 - b2 P2Q1 P1Q0)
    // L22 = I - a2 (Q1P0 + Q1P1 + Q2P1 - b2 Q2P1 Q1P0)
    // (src/core/DifferentialIntegrator.cpp:58-65)
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const DiffReq& r = reqs[c0 + b];
      g.push_back({P2Q1[b], P1Q0[b], X4[b], nullptr, nullptr, nullptr});
      g.push_back({Q2P1[b], Q1P0[b], Y4[b], nullptr, nullptr, nullptr});
      g.push_back({P1Q1[b], r.P0, U1[b], nullptr, nullptr, nullptr});   // P1Q1P0
      g.push_back({P2Q1[b], r.P1, U2[b], nullptr, nullptr, nullptr});   // P2Q1P1
      g.push_back({Q1P1[b], r.Q0, U3[b], nullptr, nullptr, nullptr});   // Q1P1Q0
      g.push_back({Q2P1[b], r.Q1, U4[b], nullptr, nullptr, nullptr});   // Q2P1Q1
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    // S = P1Q0 + P1Q1 + P2Q1 - b2 X4 ; L11 = I - a2 S (L22 alike from Q)
    // L12 = c (P0 + 4 P1 + P2 - h2 (P1Q1P0 + P2Q1P1)) (L21 alike from Q)
    {
      std::vector<DiffDesc> dd;
      for (size_t b = 0; b < B; ++b) {
        const DiffReq& r = reqs[c0 + b];
        dd.push_back({P1Q0[b], P1Q1[b], P2Q1[b], X4[b], r.P0, r.P1, r.P2, U1[b], U2[b], L11[b], L12[b], r.k0, r.dz});
        dd.push_back({Q1P0[b], Q1P1[b], Q2P1[b], Y4[b], r.Q0, r.Q1, r.Q2, U3[b], U4[b], L22[b], L21[b], r.k0, r.dz});
      }
      Prof pr(*this, "elementwise", 0.0, 16.0 * 11.0 * nn * dd.size());
      diff_combine_batched(upload(dd), (int)dd.size(), n, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const DiffReq& r = reqs[c0 + b];
      g.push_back({r.W1inv, L11[b], U1[b], nullptr, nullptr, nullptr});
      g.push_back({r.W1inv, L12[b], U2[b], nullptr, nullptr, nullptr});
      g.push_back({r.V1inv, L21[b], U3[b], nullptr, nullptr, nullptr});
      g.push_back({r.V1inv, L22[b], U4[b], nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    // A11 = (U1+U3)/2, A21 = (U1-U3)/2, A12 = (U2+U4)/2, A22 = (U2-U4)/2
    {
      Prof pr(*this, "elementwise", 0.0, 128.0 * nn * B, 2);
      ab_batched(upload(U1), upload(U3), (int)B, (long long)nn, stream_);
      ab_batched(upload(U2), upload(U4), (int)B, (long long)nn, stream_);
    }
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const DiffReq& r = reqs[c0 + b];
      g.push_back({U1[b], r.W1, P1Q0[b], nullptr, nullptr, nullptr});  // A11 W1
      g.push_back({U2[b], r.V1, P1Q1[b], nullptr, nullptr, nullptr});  // A12 V1
      g.push_back({U3[b], r.W1, P2Q1[b], nullptr, nullptr, nullptr});  // A21 W1
      g.push_back({U4[b], r.V1, Q1P0[b], nullptr, nullptr, nullptr});  // A22 V1
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    {
      std::vector<const cplx*> a, bb;
      std::vector<cplx*> c;
      for (size_t b = 0; b < B; ++b) { a.push_back(P1Q0[b]); bb.push_back(P1Q1[b]); c.push_back(T11[b]); }
      axpby(a, bb, c, mk(1, 0), mk(1, 0), 0.0, n);
      c.clear();
      for (size_t b = 0; b < B; ++b) c.push_back(T12[b]);
      axpby(a, bb, c, mk(1, 0), mk(-1, 0), 0.0, n);
      a.clear(); bb.clear(); c.clear();
      for (size_t b = 0; b < B; ++b) { a.push_back(P2Q1[b]); bb.push_back(Q1P0[b]); c.push_back(T21[b]); }
      axpby(a, bb, c, mk(1, 0), mk(1, 0), 0.0, n);
      c.clear();
      for (size_t b = 0; b < B; ++b) c.push_back(T22[b]);
      axpby(a, bb, c, mk(1, 0), mk(-1, 0), 0.0, n);
    }
    // tdd = T22^-1 ; rud = T12 tdd ; rdu = -T22^-1 T21 ; tuu = T11 + T12 rdu
    std::vector<cplx*> tdd(B);
    for (size_t b = 0; b < B; ++b) tdd[b] = reqs[c0 + b].tdd;
    copy(T22, tdd, n);
    std::vector<int> ist;
    inverse(tdd, n, status ? &ist : nullptr);
    g.clear();
    for (size_t b = 0; b < B; ++b) {
      const DiffReq& r = reqs[c0 + b];
      g.push_back({T12[b], r.tdd, r.rud, nullptr, nullptr, nullptr});
    }
    gemm(g, n, mk(1, 0), mk(0, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({reqs[c0 + b].tdd, T21[b], reqs[c0 + b].rdu, nullptr, nullptr, nullptr});
    gemm(g, n, mk(-1, 0), mk(0, 0), 0.0);
    g.clear();
    for (size_t b = 0; b < B; ++b) g.push_back({T12[b], reqs[c0 + b].rdu, reqs[c0 + b].tuu, T11[b], nullptr, nullptr});
    gemm(g, n, mk(1, 0), mk(1, 0), 0.0);
    if (status)
      for (size_t b = 0; b < ist.size(); ++b)
        if (ist[b]) (*status)[c0 + b] = ist[b];
    sync();
    for (int k = 0; k < NT; ++k)
      for (size_t b = 0; b < B; ++b) free_mat(t[k][b], n);
  }
}

}  // namespace vrc
