// Sweep planner: turns the reference's per-block call sequences into batched
// launches (one launch per recursion step over all systems).
#include "engine.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <tuple>

namespace negf {

cudaError_t zgj_prepare(size_t smem);

namespace {
thread_local std::string g_last_error;

inline ZGemmProblem gp(const cplx* A, int lda, const cplx* B, int ldb, cplx* C, int ldc, int m, int n, int k,
                       cplx alpha, const cplx* Cin = nullptr, int ldcin = 1, cplx beta = {0.0, 0.0},
                       cplx diag = {0.0, 0.0}) {
  ZGemmProblem p;
  p.A = A; p.B = B; p.Cin = Cin; p.C = C; p.diag_ptr = nullptr; p.alpha_ptr = nullptr;
  p.m = m; p.n = n; p.k = k;
  p.lda = lda > 0 ? lda : 1; p.ldb = ldb > 0 ? ldb : 1; p.ldc = ldc; p.ldcin = ldcin > 0 ? ldcin : 1;
  p.pad_ = 0;
  p.alpha = alpha; p.beta = beta; p.diag = diag;
  return p;
}
constexpr cplx ONE{1.0, 0.0};
constexpr cplx MONE{-1.0, 0.0};
constexpr cplx ZERO{0.0, 0.0};
inline cplx cscale(cplx a, double s) { return make_double2(a.x * s, a.y * s); }
}  // namespace

std::string& last_error() { return g_last_error; }
void set_error(const std::string& msg) { g_last_error = msg; }

int gj_panel_width(int max_n) {
  if (max_n <= 112) return max_n;
  if (max_n <= 400) return 32;
  if (max_n <= 800) return 16;
  return 8;
}

// A requested width is taken in whole sub-panels of 8 (a partial one costs as
// much shared memory) and up to the widest that the update kernel holds; the
// inverse does not depend on it beyond rounding.
int Plan::panel_width(int max_n) const {
  if (gj_nb_ <= 0 || max_n <= 112) return gj_panel_width(max_n);
  const int nb = std::min(gj_nb_, kGjMaxNb);
  return nb < 8 ? nb : nb & ~7;
}

int TriSystem::maxb() const {
  int m = 0;
  for (int x : b) m = std::max(m, x);
  return m;
}

// ---------------------------------------------------------------------------
// Plan

namespace {
// Per-device cache of freed plan chunks, keyed by size.  It holds at most half
// of the device's memory; a chunk that does not fit is freed.
struct ChunkCache {
  std::mutex mu;
  std::map<int, std::multimap<size_t, void*>> free_by_dev;
  std::map<int, size_t> bytes;
  std::map<int, size_t> total;  // device memory, read once per device
};
ChunkCache& chunk_cache() {
  static ChunkCache* c = new ChunkCache();  // kept until exit: chunks may be returned during teardown
  return *c;
}
int current_device() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}
// a non-blocking stream per device for plans finalised without one (no legacy-stream work)
cudaStream_t zero_stream() {
  static std::mutex mu;
  static std::map<int, cudaStream_t> streams;
  std::lock_guard<std::mutex> lk(mu);
  const int d = current_device();
  auto it = streams.find(d);
  if (it != streams.end()) return it->second;
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) s = nullptr;
  streams[d] = s;
  return s;
}
// a cached chunk of at least `bytes` and at most 5/4 of it, or null
void* cache_take(size_t bytes, size_t* got) {
  ChunkCache& c = chunk_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  const int d = current_device();
  auto& m = c.free_by_dev[d];
  auto it = m.lower_bound(bytes);
  if (it == m.end() || it->first > bytes + bytes / 4) return nullptr;
  void* p = it->second;
  *got = it->first;
  c.bytes[d] -= it->first;
  m.erase(it);
  return p;
}
void cache_put(void* p, size_t bytes) {
  ChunkCache& c = chunk_cache();
  const int d = current_device();
  {
    std::lock_guard<std::mutex> lk(c.mu);
    size_t& tot = c.total[d];
    if (tot == 0) {
      size_t fr = 0;
      if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) tot = 0;
    }
    if (c.bytes[d] + bytes <= tot / 2) {
      c.free_by_dev[d].emplace(bytes, p);
      c.bytes[d] += bytes;
      return;
    }
  }
  cudaFree(p);
}
void cache_flush(int d) {
  ChunkCache& c = chunk_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  for (auto& kv : c.free_by_dev[d]) cudaFree(kv.second);
  c.free_by_dev[d].clear();
  c.bytes[d] = 0;
}
}  // namespace

size_t cached_bytes(int device) {
  ChunkCache& c = chunk_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  auto it = c.bytes.find(device);
  return it == c.bytes.end() ? 0 : it->second;
}

void release_cached_memory() {
  int n = 0, cur = 0;
  cudaGetDevice(&cur);
  if (cudaGetDeviceCount(&n) != cudaSuccess) return;
  for (int d = 0; d < n; ++d) {
    if (cached_bytes(d) == 0) continue;
    cudaSetDevice(d);
    cache_flush(d);
  }
  cudaSetDevice(cur);
}

Plan::~Plan() {
  if (gexec_) cudaGraphExecDestroy(gexec_);
  if (graph_) cudaGraphDestroy(graph_);
  // The chunks go back to the cache once the last recorded use on every
  // stream is complete.  Only those uses are waited for: a device-wide
  // synchronisation would invalidate CUDA-graph captures that other threads
  // have in progress.  A plan without recorded uses, or whose wait fails,
  // frees its chunks (cudaFree waits for the device itself).
  bool idle = !fences_.empty();
  for (auto& f : fences_) {
    if (cudaEventSynchronize(f.second) != cudaSuccess) idle = false;
    cudaEventDestroy(f.second);
  }
  if (!idle) cudaGetLastError();
  for (auto& c : owned_) {
    if (idle) cache_put(c.first, c.second);
    else cudaFree(c.first);
  }
}

void Plan::fence(cudaStream_t s) {
  cudaEvent_t ev = nullptr;
  for (auto& f : fences_)
    if (f.first == s) ev = f.second;
  if (!ev) {
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return;
    fences_.push_back({s, ev});
  }
  cudaEventRecord(ev, s);
}

// Workspace comes from a bump arena of zeroed chunks: the first is 1 MiB and
// each next one doubles up to 64 MiB, so a plan of thousands of small blocks
// costs a handful of cudaMalloc calls instead of one per block; a request of
// 32 MiB or more gets a chunk of its own.  Every piece is 256-byte aligned.
void* Plan::take_chunk(size_t bytes) {
  size_t got = bytes;
  void* p = cache_take(bytes, &got);
  if (!p) {
    got = bytes;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
      cudaGetLastError();  // clear the allocation error, then retry without the cache
      cache_flush(current_device());
      if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        throw std::bad_alloc();
      }
    }
  }
  owned_.push_back({p, got});
  return p;
}

void* Plan::raw_alloc(size_t bytes) {
  void* p = take_chunk(bytes);
  owned_bytes_ += owned_.back().second;
  to_zero_.push_back({p, bytes});
  return p;
}

void* Plan::alloc(size_t bytes) {
  constexpr size_t kFirst = size_t(1) << 20, kCap = size_t(64) << 20;
  bytes = (std::max<size_t>(bytes, 16) + 255) & ~size_t(255);
  if (bytes >= kCap / 2) return raw_alloc(bytes);
  if (chunk_left_ < bytes) {
    chunk_size_ = chunk_size_ ? std::min(kCap, 2 * chunk_size_) : kFirst;
    while (chunk_size_ < bytes) chunk_size_ *= 2;
    chunk_ = static_cast<unsigned char*>(raw_alloc(chunk_size_));
    chunk_left_ = chunk_size_;
  }
  void* p = chunk_;
  chunk_ += bytes;
  chunk_left_ -= bytes;
  return p;
}

size_t Plan::push_bytes(const void* p, size_t n) {
  size_t off = (blob_.size() + 255) & ~size_t(255);
  blob_.resize(off + n);
  if (n) std::memcpy(blob_.data() + off, p, n);
  return off;
}

void Plan::gemm(char opA, char opB, const std::vector<ZGemmProblem>& probs) {
  if (!mixed_) {
    gemm_fp64(opA, opB, probs);
    return;
  }
  std::vector<ZGemmProblem> dbl, mix;
  for (const auto& p : probs) (p.k > 0 ? mix : dbl).push_back(p);
  gemm_fp64(opA, opB, dbl);
  gemm_mixed(opA, opB, mix);
}

namespace {
// views of the operands as R x K real-and-imaginary matrices (K = contraction)
struct OzKey {
  const cplx* X;
  long long sr, sk;
  int rows, cols, conj, side;
  bool operator<(const OzKey& o) const {
    return std::tie(X, sr, sk, rows, cols, conj, side) < std::tie(o.X, o.sr, o.sk, o.rows, o.cols, o.conj, o.side);
  }
};
inline int round_up(int x, int m) { return (x + m - 1) / m * m; }
}  // namespace

void Plan::gemm_mixed(char opA, char opB, const std::vector<ZGemmProblem>& probs, int pairs) {
  if (probs.empty()) return;
  if (!err_) err_ = static_cast<int*>(alloc(sizeof(int)));
  std::map<OzKey, int> index;
  std::vector<OzKey> keys;
  std::vector<std::pair<int, int>> which(probs.size());
  auto key_of = [&](const ZGemmProblem& p, bool A) {
    OzKey k;
    if (A) {  // Y = op(A): m x k
      k.X = p.A; k.rows = p.m; k.cols = p.k; k.side = 0;
      if (opA == 'N') { k.sr = 1; k.sk = p.lda; k.conj = 0; }
      else { k.sr = p.lda; k.sk = 1; k.conj = opA == 'C'; }
    } else {  // Y = op(B)^T: n x k
      k.X = p.B; k.rows = p.n; k.cols = p.k; k.side = 1;
      if (opB == 'N') { k.sr = p.ldb; k.sk = 1; k.conj = 0; }
      else { k.sr = 1; k.sk = p.ldb; k.conj = opB == 'C'; }
    }
    return k;
  };
  auto get = [&](const OzKey& k) {
    auto it = index.find(k);
    if (it != index.end()) return it->second;
    int id = (int)keys.size();
    index[k] = id;
    keys.push_back(k);
    return id;
  };
  for (size_t i = 0; i < probs.size(); ++i) which[i] = {get(key_of(probs[i], true)), get(key_of(probs[i], false))};
  // Digits the previous mixed step made are used again when no other step
  // came in between, the operand view is the same (pointer, strides, shape,
  // conjugation, side) and none of that step's products wrote into it.
  if (steps.size() != oz_prev_steps_) {
    oz_prev_.clear();
    oz_prev_out_.clear();
    oz_prev_end_ = 0;
  }
  auto view_key = [](const OzKey& k) {
    return std::vector<long long>{(long long)(uintptr_t)k.X, k.sr, k.sk, k.rows, k.cols, k.conj, k.side};
  };
  auto written_before = [&](const OzKey& k) {
    const char* lo = reinterpret_cast<const char*>(k.X);
    const char* hi = lo + sizeof(cplx) * ((size_t)(k.rows - 1) * k.sr + (size_t)(k.cols - 1) * k.sk + 1);
    for (const auto& r : oz_prev_out_)
      if (lo < r.second && r.first < hi) return true;
    return false;
  };
  const size_t nk = keys.size();
  std::vector<int> rpad(nk), kpad(nk);
  std::vector<int8_t*> slc(nk, nullptr);
  std::vector<int*> exs(nk, nullptr);
  bool any_reuse = false;
  for (size_t i = 0; i < nk; ++i) {
    rpad[i] = round_up(std::max(keys[i].rows, 1), keys[i].side == 0 ? 128 : 64);
    kpad[i] = round_up(std::max(keys[i].cols, 1), 32);
    auto it = oz_prev_.find(view_key(keys[i]));
    if (it != oz_prev_.end() && it->second.rpad == rpad[i] && it->second.kpad == kpad[i] && !written_before(keys[i])) {
      slc[i] = it->second.slices;
      exs[i] = it->second.exps;
      any_reuse = true;
    }
  }
  // new digits: 3 real operands x 7 digit slices, then a scale per row; they go
  // after the reused ones when those are in the pool and there is room, else
  // the pool is laid out afresh (and grown as needed) without reuse
  std::vector<size_t> off_s(nk, 0), off_e(nk, 0);
  auto layout = [&](size_t base) {
    size_t need = base;
    for (size_t i = 0; i < nk; ++i) {
      if (slc[i]) continue;
      off_s[i] = need;
      need += (size_t)21 * rpad[i] * kpad[i];
      need = (need + 255) & ~size_t(255);
      off_e[i] = need;
      need += sizeof(int) * (size_t)rpad[i];
      need = (need + 255) & ~size_t(255);
    }
    return need;
  };
  size_t base = 0, need = 0;
  if (any_reuse && oz_prev_pool_ == oz_pool_ && layout(oz_prev_end_) <= oz_pool_bytes_) {
    base = oz_prev_end_;
  } else if (any_reuse) {
    any_reuse = false;
    for (size_t i = 0; i < nk; ++i) {
      slc[i] = nullptr;
      exs[i] = nullptr;
    }
  }
  need = layout(base);
  if (need > oz_pool_bytes_) {
    oz_pool_ = static_cast<unsigned char*>(alloc(need));
    oz_pool_bytes_ = need;
  }
  std::vector<OzSplitProblem> sp;
  int max_rows = 0, max_kpad = 0;
  double split_bytes = 0.0;
  for (size_t i = 0; i < nk; ++i) {
    if (slc[i]) continue;
    slc[i] = reinterpret_cast<int8_t*>(oz_pool_ + off_s[i]);
    exs[i] = reinterpret_cast<int*>(oz_pool_ + off_e[i]);
    OzSplitProblem q;
    q.X = keys[i].X; q.sr = keys[i].sr; q.sk = keys[i].sk;
    q.rows = keys[i].rows; q.cols = keys[i].cols; q.rows_pad = rpad[i]; q.k_pad = kpad[i];
    q.conj = keys[i].conj; q.tile_rows = keys[i].side == 0 ? 128 : 64;
    q.slices = slc[i];
    q.exps = exs[i];
    sp.push_back(q);
    max_rows = std::max(max_rows, rpad[i]);
    max_kpad = std::max(max_kpad, kpad[i]);
    split_bytes += 16.0 * keys[i].rows * keys[i].cols + 21.0 * rpad[i] * kpad[i] + 4.0 * rpad[i];
  }
  if (!sp.empty()) {
    Step s1;
    s1.kind = Step::OZ_SPLIT;
    s1.off = push_bytes(sp.data(), sp.size() * sizeof(OzSplitProblem));
    s1.count = (int)sp.size();
    s1.max_m = max_rows;
    s1.max_n = max_kpad;
    s1.bytes = split_bytes;
    steps.push_back(s1);
  }
  std::vector<OzMmaProblem> mp;
  std::vector<int> tmap;  // 4 ints per output tile, see launch_ozaki_mma
  int total = 0;
  double fl = 0.0;
  for (size_t i = 0; i < probs.size(); ++i) {
    const ZGemmProblem& p = probs[i];
    const int a = which[i].first, b = which[i].second;
    OzMmaProblem q;
    q.SA = slc[a]; q.eA = exs[a]; q.SB = slc[b]; q.eB = exs[b];
    q.C = p.C; q.Cin = p.Cin; q.diag_ptr = p.diag_ptr; q.alpha_ptr = p.alpha_ptr;
    q.m = p.m; q.n = p.n; q.m_pad = rpad[a]; q.n_pad = rpad[b]; q.k_pad = kpad[a];
    q.ldc = p.ldc; q.ldcin = p.ldcin; q.pad_ = 0;
    q.alpha = p.alpha; q.beta = p.beta; q.diag = p.diag;
    const int tm = q.m_pad / 128, tn = q.n_pad / 64, kc = q.k_pad / 32;
    for (int t = 0; t < tm * tn; ++t) {
      tmap.push_back((int)i);
      tmap.push_back((t / tn) | ((t % tn) << 16));
      tmap.push_back(kc | (tm << 16));
      tmap.push_back(tn);
    }
    total += tm * tn;
    fl += 8.0 * p.m * (double)p.n * p.k;
    mp.push_back(q);
  }
  Step s2;
  s2.kind = Step::OZ_MMA;
  s2.off = push_bytes(mp.data(), mp.size() * sizeof(OzMmaProblem));
  s2.tiles_off = push_bytes(tmap.data(), tmap.size() * sizeof(int));
  s2.count = (int)mp.size();
  s2.total_tiles = total;
  s2.flops = fl;
  s2.form = pairs == 28 || pairs == 34 ? pairs : oz_pairs_;
  steps.push_back(s2);
  // what the next mixed step may use again
  oz_prev_.clear();
  for (size_t i = 0; i < nk; ++i) oz_prev_[view_key(keys[i])] = OzSplitDone{slc[i], exs[i], rpad[i], kpad[i]};
  oz_prev_out_.clear();
  for (const auto& p : probs) {
    if (p.m <= 0 || p.n <= 0) continue;
    const char* lo = reinterpret_cast<const char*>(p.C);
    oz_prev_out_.push_back({lo, lo + sizeof(cplx) * ((size_t)(p.n - 1) * p.ldc + p.m)});
  }
  oz_prev_end_ = need;
  oz_prev_pool_ = oz_pool_;
  oz_prev_steps_ = steps.size();
}

void Plan::gemm_fp64(char opA, char opB, const std::vector<ZGemmProblem>& probs) {
  std::vector<ZGemmProblem> v;
  std::vector<int> starts;
  int total = 0;
  double fl = 0.0;
  bool pre = true;
  const int form = zgemm_choose_form(gemm_form_, probs.data(), (int)probs.size(), fixed_order_);
  for (const auto& p : probs) {
    int t = zgemm_tiles_form(form, p.m, p.n);
    if (t == 0) continue;
    v.push_back(p);
    starts.push_back(total);
    total += t;
    fl += 8.0 * p.m * (double)p.n * p.k;
    pre = pre && zgemm_preload_ok(p);
  }
  if (v.empty()) return;
  Step s;
  s.kind = Step::GEMM;
  s.opA = opA;
  s.opB = opB;
  s.preload = pre && form == 1;
  s.form = form;
  s.uniform_tiles = total / (int)v.size();
  if ((long long)s.uniform_tiles * (long long)v.size() != total) s.uniform_tiles = 0;
  for (size_t i = 1; i < starts.size() && s.uniform_tiles; ++i)
    if (starts[i] - starts[i - 1] != s.uniform_tiles) s.uniform_tiles = 0;
  s.off = push_bytes(v.data(), v.size() * sizeof(ZGemmProblem));
  s.tiles_off = push_bytes(starts.data(), starts.size() * sizeof(int));
  s.count = static_cast<int>(v.size());
  s.total_tiles = total;
  s.flops = fl;
  steps.push_back(s);
}

void Plan::inv(const std::vector<InvSpec>& specs) {
  std::vector<ZInvProblem> v;
  int max_n = 0;
  for (const auto& sp : specs) {
    if (sp.n <= 0) continue;
    ZInvProblem p;
    p.W = sp.W; p.F = sp.F; p.Bbuf = sp.Bbuf; p.used = sp.used; p.piv = sp.piv; p.out = sp.out;
    p.info = sp.info; p.n = sp.n; p.ld = sp.ld; p.ldo = sp.ldo; p.pad_ = 0;
    v.push_back(p);
    max_n = std::max(max_n, sp.n);
  }
  if (v.empty()) return;
  int nb = panel_width(max_n);
  bool blocked = nb < max_n;
  size_t off = push_bytes(v.data(), v.size() * sizeof(ZInvProblem));
  double gj_flops = 0.0;
  for (const auto& p : v) gj_flops += 8.0 * p.n * (double)p.n * p.n;
  if (!blocked) {
    Step s;
    s.kind = Step::GJ_PANEL;
    s.off = off; s.count = (int)v.size(); s.k0 = 0; s.nb = nb; s.blocked = 0;
    s.smem = zgj_panel_smem_bytes(max_n, nb);
    s.max_n = max_n;
    s.flops = gj_flops;
    steps.push_back(s);
    return;
  }
  for (int k0 = 0; k0 < max_n; k0 += nb) {
    Step s;
    s.kind = Step::GJ_PANEL;
    s.off = off; s.count = (int)v.size(); s.k0 = k0; s.nb = nb; s.blocked = gj_update_int8() ? 2 : 1;
    s.smem = zgj_panel_smem_bytes(max_n, nb);
    s.max_n = max_n;
    steps.push_back(s);
    if (!gj_update_int8()) {
      s.kind = Step::GEMM;
      s.form = 4;
      for (const auto& p : v) s.flops += 8.0 * p.n * (double)p.n * std::max(0, std::min(nb, p.n - k0));
      steps.push_back(s);
      continue;
    }
    std::vector<ZGemmProblem> g;
    for (const auto& p : v) {
      if (p.n <= k0) continue;
      int w = std::min(nb, p.n - k0);
      g.push_back(gp(p.F, p.n, p.Bbuf, w, p.W, p.ld, p.n, p.n, w, ONE, p.W, p.ld, ONE));
    }
    // W += F Bbuf as INT8 digit products at FP64 accuracy (the panels stay in FP64)
    gemm_mixed('N', 'N', g, 34);
  }
  // the GEMM updates carry their own flop count; the panel work is the rest
  Step u;
  u.kind = Step::GJ_UNPERMUTE;
  u.off = off; u.count = (int)v.size(); u.max_n = max_n;
  steps.push_back(u);
}

int lu_panel_width(int max_n) {
  if (max_n <= 96) return max_n;
  if (max_n <= 400) return 32;
  if (max_n <= 800) return 16;
  return 8;
}

void Plan::getrf(const std::vector<LuSpec>& specs) {
  std::vector<ZLuProblem> v;
  int max_n = 0;
  for (const auto& s : specs) {
    if (s.n <= 0) continue;
    ZLuProblem p;
    p.A = s.A; p.ipiv = s.ipiv; p.Linv = s.Linv; p.T = s.T; p.info = s.info;
    p.n = s.n; p.ld = s.ld;
    v.push_back(p);
    max_n = std::max(max_n, s.n);
  }
  if (v.empty()) return;
  const int nb = lu_panel_width(max_n);
  size_t off = push_bytes(v.data(), v.size() * sizeof(ZLuProblem));
  for (int k0 = 0; k0 < max_n; k0 += nb) {
    Step s;
    s.kind = Step::LU_PANEL;
    s.off = off; s.count = (int)v.size(); s.k0 = k0; s.nb = nb; s.max_n = max_n;
    s.smem = zgetrf_panel_smem_bytes(max_n - k0, nb);
    steps.push_back(s);
    if (nb >= max_n) break;
    Step w = s;
    w.kind = Step::LU_SWAP;
    w.smem = 0;
    steps.push_back(w);
    // A12 = L11^{-1} T ;  A22 -= A21 A12
    std::vector<ZGemmProblem> g1, g2;
    for (const auto& p : v) {
      if (p.n <= k0 + nb) continue;
      int wd = std::min(nb, p.n - k0);
      int rest = p.n - k0 - wd;
      cplx* A12 = p.A + k0 + (size_t)(k0 + wd) * p.ld;
      g1.push_back(gp(p.Linv, wd, p.T, wd, A12, p.ld, wd, rest, wd, ONE));
      const cplx* A21 = p.A + (k0 + wd) + (size_t)k0 * p.ld;
      cplx* A22 = p.A + (k0 + wd) + (size_t)(k0 + wd) * p.ld;
      g2.push_back(gp(A21, p.ld, A12, p.ld, A22, p.ld, rest, rest, wd, MONE, A22, p.ld, ONE));
    }
    gemm_fp64('N', 'N', g1);  // factorisations stay in FP64
    gemm_fp64('N', 'N', g2);
  }
}

// Scratch of the joins: the products of all pairs of a level, or of one block column.
size_t tri_scratch(int n) { return (size_t)std::max(n, kTriJoin) * kTriJoin; }

// With the diagonal blocks of 32 inverted, neighbouring blocks are joined to
// blocks of kTriJoin (upper: X12 = -(X11 U12) X22, lower: X21 = -X22 (L21 X11)),
// two launches per doubling over all pairs of all matrices; then block columns
// (upper) and rows (lower) of that width follow one after the other, two
// launches each.  Joining all the way up would take fewer launches, but
// compounds the rounding of each level.
void Plan::tri_join(const std::vector<TriSpec>& up, const std::vector<TriSpec>& lo) {
  int max_n = 0;
  for (const auto* v : {&up, &lo})
    for (const auto& p : *v) max_n = std::max(max_n, p.n);
  // one join: block rows / columns [j, j + s) and [k, k + s2), k = j + s
  auto join = [&](const TriSpec& p, bool upper, int j, int s, int s2, cplx* T, std::vector<ZGemmProblem>& g1,
                  std::vector<ZGemmProblem>& g2) {
    const int k = j + s;
    cplx* X11 = p.X + j + (size_t)j * p.ldx;
    cplx* X22 = p.X + k + (size_t)k * p.ldx;
    if (upper) {
      g1.push_back(gp(X11, p.ldx, p.A + j + (size_t)k * p.lda, p.lda, T, s, s, s2, s, ONE));
      g2.push_back(gp(T, s, X22, p.ldx, p.X + j + (size_t)k * p.ldx, p.ldx, s, s2, s2, MONE));
    } else {
      g1.push_back(gp(p.A + k + (size_t)j * p.lda, p.lda, X11, p.ldx, T, s2, s2, s, s, ONE));
      g2.push_back(gp(X22, p.ldx, T, s2, p.X + k + (size_t)j * p.ldx, p.ldx, s2, s, s2, MONE));
    }
  };
  for (int s = kTriNb; s < std::min(max_n, kTriJoin); s *= 2) {
    std::vector<ZGemmProblem> g1, g2;
    for (const auto* v : {&up, &lo})
      for (const auto& p : *v) {
        size_t t = 0;
        for (int j = 0; j + s < p.n; j += 2 * s) {
          const int s2 = std::min(s, p.n - j - s);
          join(p, v == &up, j, s, s2, p.T + t, g1, g2);
          t += (size_t)s * s2;
        }
      }
    gemm_fp64('N', 'N', g1);
    gemm_fp64('N', 'N', g2);
  }
  for (int s = kTriJoin; s < max_n; s += kTriJoin) {
    std::vector<ZGemmProblem> g1, g2;
    for (const auto* v : {&up, &lo})
      for (const auto& p : *v)
        if (s < p.n) join(p, v == &up, 0, s, std::min(kTriJoin, p.n - s), p.T, g1, g2);
    gemm_fp64('N', 'N', g1);
    gemm_fp64('N', 'N', g2);
  }
}

void Plan::trtri(const std::vector<TriSpec>& up, const std::vector<TriSpec>& lo) {
  std::vector<ZBlockOp> zero;
  for (const auto* list : {&up, &lo})
    for (const auto& s : *list) {
      if (s.n <= 0) continue;
      ZBlockOp z{};
      z.C = s.X; z.ldc = s.ldx; z.m = z.n = s.n; z.kind = ZOP_FILL;
      zero.push_back(z);
    }
  if (zero.empty()) return;
  blockops(zero);
  for (const auto* list : {&up, &lo}) {
    std::vector<ZTriProblem> v;
    int max_n = 0;
    for (const auto& s : *list) {
      if (s.n <= 0) continue;
      ZTriProblem p;
      p.A = s.A; p.X = s.X; p.n = s.n; p.lda = s.lda; p.ldx = s.ldx; p.pad_ = 0;
      v.push_back(p);
      max_n = std::max(max_n, s.n);
    }
    if (v.empty()) continue;
    Step s;
    s.kind = Step::TRI_DIAG;
    s.off = push_bytes(v.data(), v.size() * sizeof(ZTriProblem));
    s.count = (int)v.size(); s.nb = kTriNb; s.blocked = list == &up ? 1 : 0; s.max_n = max_n;
    s.smem = ztrtri_smem_bytes(kTriNb);
    steps.push_back(s);
  }
  tri_join(up, lo);
}

// Unpivoted LU in panels of 32, three launches each: the diagonal block with the
// inverses of its factors, F21 = A21 U^{-1} and F12 = L^{-1} A12 by substitution,
// A22 -= F21 F12; then the joins of the triangular inverses.  A 512 block with its
// inverses: 62 launches, 1.2 ms for 8 systems (panels of 16 whole columns, row
// swaps and inverses in columns of 32: 190 launches, 3.7 ms); bound by the latency
// of the launches' serial substitutions.
void Plan::lu_nopiv(const std::vector<LuInvSpec>& specs) {
  constexpr int nb = kTriNb;
  std::vector<ZLuDiagProblem> v;
  std::vector<ZBlockOp> zero, back;
  std::vector<TriSpec> up, lo;
  int max_n = 0;
  for (const auto& s : specs) {
    ZLuDiagProblem p;
    p.A = s.A; p.F = s.F; p.Xu = s.Xu; p.Xl = s.Xl; p.info = s.info;
    p.n = s.n; p.ld = s.ld; p.ldf = s.n; p.pad_ = 0;
    v.push_back(p);
    max_n = std::max(max_n, s.n);
    for (cplx* X : {s.Xu, s.Xl}) {
      ZBlockOp z{};
      z.C = X; z.ldc = z.m = z.n = s.n; z.kind = ZOP_FILL;
      zero.push_back(z);
    }
    ZBlockOp c{};
    c.A = s.F; c.lda = s.n; c.C = s.A; c.ldc = s.ld; c.m = c.n = s.n; c.kind = ZOP_COPY;
    back.push_back(c);
    up.push_back({s.F, s.n, s.n, s.Xu, s.n, s.T});
    lo.push_back({s.F, s.n, s.n, s.Xl, s.n, s.T + tri_scratch(s.n)});
  }
  if (v.empty()) return;
  blockops(zero);
  const size_t off = push_bytes(v.data(), v.size() * sizeof(ZLuDiagProblem));
  for (int k0 = 0; k0 < max_n; k0 += nb) {
    Step d;
    d.kind = Step::LU_PANEL;
    d.off = off; d.count = (int)v.size(); d.k0 = k0; d.nb = 0;
    steps.push_back(d);
    if (max_n <= k0 + nb) break;
    d.nb = -1;
    d.max_n = max_n;
    steps.push_back(d);
    std::vector<ZGemmProblem> g;
    for (const auto& s : specs) {
      const int k1 = k0 + nb, rest = s.n - k1;
      if (rest <= 0) continue;
      cplx* A22 = s.A + k1 + (size_t)k1 * s.ld;
      g.push_back(gp(s.F + k1 + (size_t)k0 * s.n, s.n, s.F + k0 + (size_t)k1 * s.n, s.n, A22, s.ld, rest, rest, nb,
                     MONE, A22, s.ld, ONE));
    }
    gemm_fp64('N', 'N', g);
  }
  blockops(back);
  tri_join(up, lo);
}

void Plan::blockops(const std::vector<ZBlockOp>& ops) {
  if (ops.empty()) return;
  Step s;
  s.kind = Step::BLOCKOP;
  s.off = push_bytes(ops.data(), ops.size() * sizeof(ZBlockOp));
  s.count = (int)ops.size();
  for (const auto& o : ops) { s.max_m = std::max(s.max_m, o.m); s.max_n = std::max(s.max_n, o.n); }
  steps.push_back(s);
}

void Plan::trace(const std::vector<ZTraceProblemHost>& probs) {
  if (probs.empty()) return;
  Step s;
  s.kind = Step::TRACE;
  s.off = push_bytes(probs.data(), probs.size() * sizeof(ZTraceProblemHost));
  s.count = (int)probs.size();
  steps.push_back(s);
}

cudaError_t Plan::finalize() {
  if (finalized_) return cudaSuccess;
  cudaStream_t zs = zero_stream();
  if (!zs) return cudaErrorInitializationError;
  cudaError_t e = finalize(zs);
  return e == cudaSuccess ? cudaStreamSynchronize(zs) : e;
}

// The descriptors take a chunk of the cache and, like the zeroing, go in order
// on the stream of the run: a call on the host's critical path then has no
// cudaMalloc, no cudaFree (both synchronise the device) and no host wait before
// its launches.  be_inv_batched_ of four blocks of 24: 83 -> 66 us.
cudaError_t Plan::finalize(cudaStream_t stream) {
  if (finalized_) return cudaSuccess;
  for (const auto& c : to_zero_) {
    cudaError_t e = cudaMemsetAsync(c.first, 0, c.second, stream);
    if (e != cudaSuccess) return e;
  }
  to_zero_.clear();
  if (!blob_.empty()) {
    constexpr size_t kGrain = size_t(64) << 10;  // size classes of the cache
    try {
      dblob_ = take_chunk((blob_.size() + kGrain - 1) / kGrain * kGrain);
    } catch (const std::bad_alloc&) {
      return cudaErrorMemoryAllocation;
    }
    cudaError_t e = cudaMemcpyAsync(dblob_, blob_.data(), blob_.size(), cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
  }
  std::set<std::pair<char, char>> ops;
  size_t max_smem = 0, lu_smem = 0, tri_smem = 0;
  for (const auto& s : steps) {
    if (s.kind == Step::GEMM && s.form == 1) ops.insert({s.opA, s.opB});
    if (s.kind == Step::GJ_PANEL) max_smem = std::max(max_smem, s.smem);
    if (s.kind == Step::LU_PANEL) lu_smem = std::max(lu_smem, s.smem);
    if (s.kind == Step::TRI_DIAG) tri_smem = std::max(tri_smem, s.smem);
  }
  if (lu_smem || tri_smem) {
    cudaError_t e = zlu_prepare(lu_smem, tri_smem);
    if (e != cudaSuccess) return e;
  }
  for (const auto& s : steps)
    if (s.kind == Step::OZ_MMA) {
      cudaError_t e = ozaki_prepare();
      if (e != cudaSuccess) return e;
      break;
    }
  for (auto& o : ops) {
    cudaError_t e = zgemm_prepare(o.first, o.second);
    if (e != cudaSuccess) return e;
  }
  if (max_smem) {
    cudaError_t e = zgj_prepare(max_smem);
    if (e != cudaSuccess) return e;
  }
  finalized_ = true;
  return cudaSuccess;
}

double Plan::flops() const {
  double f = 0.0;
  for (const auto& s : steps) f += s.flops;
  return f;
}

size_t Plan::num_launches() const { return steps.size(); }

cudaError_t Plan::run_events(cudaStream_t stream, const std::vector<cudaEvent_t>& events) {
  if (events.size() < steps.size() + 1) return cudaErrorInvalidValue;
  cudaError_t e = finalize(stream);
  if (e != cudaSuccess) return e;
  e = cudaEventRecord(events[0], stream);
  if (e != cudaSuccess) return e;
  const unsigned char* base = static_cast<const unsigned char*>(dblob_);
  for (size_t i = 0; i < steps.size(); ++i) {
    e = launch_step(steps[i], base, stream);
    if (e == cudaSuccess) e = cudaEventRecord(events[i + 1], stream);
    if (e != cudaSuccess) break;
  }
  fence(stream);
  return e;
}

cudaError_t Plan::run_marked(cudaStream_t stream, const std::function<cudaError_t(int)>& at_mark) {
  cudaError_t e = finalize(stream);
  if (e != cudaSuccess) return e;
  const unsigned char* base = static_cast<const unsigned char*>(dblob_);
  size_t m = 0;
  for (size_t i = 0; i <= steps.size() && e == cudaSuccess; ++i) {
    for (; m < marks_.size() && marks_[m].first == i && e == cudaSuccess; ++m) e = at_mark(marks_[m].second);
    if (i == steps.size() || e != cudaSuccess) break;
    e = launch_step(steps[i], base, stream);
  }
  fence(stream);
  return e;
}

cudaError_t Plan::run(cudaStream_t stream, bool use_graph) {
  cudaError_t e = finalize(stream);
  if (e != cudaSuccess) return e;
  if (use_graph && gexec_ && graph_stream_ == stream) {
    e = cudaGraphLaunch(gexec_, stream);
    fence(stream);
    return e;
  }
  if (use_graph) {
    e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
  }
  const unsigned char* base = static_cast<const unsigned char*>(dblob_);
  if (!use_graph) chain_ctas = 1 << 30;  // the first launch waits as usual
  for (const auto& s : steps) {
    e = launch_step(s, base, stream);
    if (e != cudaSuccess) break;
  }
  chain_ctas = -1;
  if (use_graph) {
    cudaGraph_t g = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(stream, &g);
    if (e != cudaSuccess) {
      if (g) cudaGraphDestroy(g);
      return e;
    }
    if (e2 != cudaSuccess) return e2;
    if (gexec_) cudaGraphExecDestroy(gexec_);
    if (graph_) cudaGraphDestroy(graph_);
    graph_ = g;
    e = cudaGraphInstantiate(&gexec_, graph_, 0);
    if (e != cudaSuccess) return e;
    graph_stream_ = stream;
    e = cudaGraphLaunch(gexec_, stream);
    fence(stream);
    return e;
  }
  fence(stream);
  return e;
}

cudaError_t Plan::launch_step(const Step& s, const unsigned char* base, cudaStream_t stream) {
  cudaError_t e = cudaSuccess;
  {
    switch (s.kind) {
      case Step::GEMM:
        if (s.form == 4) {
          e = launch_zgj_update(reinterpret_cast<const ZInvProblem*>(base + s.off), s.count, s.k0, s.nb, s.max_n, stream);
          break;
        }
        e = launch_zgemm_batched_ex(s.opA, s.opB, s.preload, reinterpret_cast<const ZGemmProblem*>(base + s.off),
                                    reinterpret_cast<const int*>(base + s.tiles_off), s.count, s.total_tiles, stream, s.form,
                                    s.uniform_tiles);
        break;
      case Step::GJ_PANEL:
        e = launch_zgj_panel(reinterpret_cast<const ZInvProblem*>(base + s.off), s.count, s.k0, s.nb, s.blocked,
                             s.smem, stream, s.max_n);
        break;
      case Step::GJ_UNPERMUTE:
        e = launch_zgj_unpermute(reinterpret_cast<const ZInvProblem*>(base + s.off), s.count, s.max_n, stream);
        break;
      case Step::BLOCKOP:
        e = launch_zblockops(reinterpret_cast<const ZBlockOp*>(base + s.off), s.count, s.max_m, s.max_n, stream);
        break;
      case Step::TRACE:
        e = launch_ztrace_prod(base + s.off, s.count, stream);
        break;
      case Step::LU_PANEL:
        if (s.nb <= 0) {
          e = s.nb == 0 ? launch_zlu_diag(base + s.off, s.count, s.k0, stream)
                        : launch_zlu_solve(base + s.off, s.count, s.k0, s.max_n, stream);
          break;
        }
        e = launch_zgetrf_panel(base + s.off, s.count, s.k0, s.nb, s.smem, stream);
        break;
      case Step::LU_SWAP:
        e = launch_zlaswp_copy(base + s.off, s.count, s.k0, s.nb, s.max_n, stream);
        break;
      case Step::TRI_DIAG:
        e = launch_ztrtri_diag(base + s.off, s.count, s.nb, s.blocked, s.max_n, s.smem, stream);
        break;
      case Step::OZ_SPLIT:
        e = launch_ozaki_split(base + s.off, s.count, s.max_m, s.max_n, stream);
        break;
      case Step::OZ_MMA:
        e = launch_ozaki_mma(base + s.off, base + s.tiles_off, s.total_tiles, err_, stream, s.form);
        break;
    }
  }
  return e;
}

// ---------------------------------------------------------------------------
// RGF

void alloc_rgf_work(Plan& plan, const TriSystem& s, RgfWork& w) {
  int n = s.npl();
  int mb = s.maxb();
  int nb = std::max(plan.panel_width(mb), mb > 112 ? 32 : 0);  // room for any tuned width
  w.g.assign(n, nullptr);
  w.R.assign(n > 0 ? n - 1 : 0, nullptr);
  w.L.assign(n > 0 ? n - 1 : 0, nullptr);
  size_t total = 0;
  for (int i = 0; i < n; ++i) total += (size_t)s.b[i] * s.b[i];
  for (int i = 0; i + 1 < n; ++i) total += 2 * (size_t)s.b[i] * s.b[i + 1];
  total += (size_t)mb * mb;              // W
  total += 2 * (size_t)mb * nb;          // F, Bbuf
  cplx* arena = plan.alloc_c(total);
  size_t o = 0;
  for (int i = 0; i < n; ++i) { w.g[i] = arena + o; o += (size_t)s.b[i] * s.b[i]; }
  for (int i = 0; i + 1 < n; ++i) {
    w.R[i] = arena + o; o += (size_t)s.b[i] * s.b[i + 1];
    w.L[i] = arena + o; o += (size_t)s.b[i] * s.b[i + 1];
  }
  w.W = arena + o; o += (size_t)mb * mb;
  w.F = arena + o; o += (size_t)mb * nb;
  w.Bbuf = arena + o; o += (size_t)mb * nb;
  w.used = static_cast<uint8_t*>(plan.alloc(mb));
  w.piv = static_cast<int*>(plan.alloc(sizeof(int) * mb));
}

static InvSpec inv_spec(const TriSystem& s, RgfWork& w, int i) {
  InvSpec sp;
  sp.W = w.W; sp.n = s.b[i]; sp.ld = s.b[i];
  sp.out = w.g[i]; sp.ldo = s.b[i];
  sp.F = w.F; sp.Bbuf = w.Bbuf; sp.used = w.used; sp.piv = w.piv; sp.info = s.info;
  return sp;
}

void build_rgf_upward(Plan& plan, const std::vector<TriSystem>& sys, std::vector<RgfWork>& work, GnUpward* gn) {
  int maxN = 0;
  for (const auto& s : sys) maxN = std::max(maxN, s.npl());
  // bottom layer: X_{N-1} = M[N-1,N-1]  (rgf.jl:144)
  {
    std::vector<ZGemmProblem> pr;
    std::vector<InvSpec> iv;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      int i = s.npl() - 1;
      if (i < 0) continue;
      pr.push_back(gp(nullptr, 1, nullptr, 1, work[k].W, s.b[i], s.b[i], s.b[i], 0, ZERO, s.D[i], s.ldD[i],
                      s.dscale, s.shift));
      pr.back().diag_ptr = s.shift_ptr;
      iv.push_back(inv_spec(s, work[k], i));
    }
    plan.gemm('N', 'N', pr);
    plan.inv(iv);
  }
  // the last round only finishes the operator of the topmost layers (gn)
  for (int j = 1; j < maxN + (gn ? 1 : 0); ++j) {
    // R_i = M[i,i+1] g_{i+1}  (rgf.jl:152-154) and L_{i+1} = g_{i+1} M[i+1,i]  (rgf.jl:157)
    std::vector<ZGemmProblem> rN, lN, lC;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      int i = s.npl() - 1 - j;
      if (gn && i >= -1) gn->after(s, work[k], k, i + 1, lC);
      if (i < 0) continue;
      RgfWork& w = work[k];
      rN.push_back(gp(s.U[i], s.ldU[i], w.g[i + 1], s.b[i + 1], w.R[i], s.b[i], s.b[i], s.b[i + 1], s.b[i + 1],
                      s.uscale));
      auto p = gp(w.g[i + 1], s.b[i + 1], s.Lw[i], s.ldL[i], w.L[i], s.b[i + 1], s.b[i + 1], s.b[i], s.b[i + 1],
                  s.lscale);
      (s.lop == 'N' ? lN : lC).push_back(p);
    }
    std::vector<ZGemmProblem> nn = rN;
    nn.insert(nn.end(), lN.begin(), lN.end());
    plan.gemm('N', 'N', nn);
    if (gn)
      for (size_t k = 0; k < sys.size(); ++k) {
        int i = sys[k].npl() - 1 - j;
        if (i >= 0) gn->before(sys[k], work[k], k, i, lC);
      }
    plan.gemm('N', 'C', lC);
    // X_i = M[i,i] - M[i,i+1] L_{i+1}  (rgf.jl:159-160), then its inverse (rgf.jl:161)
    std::vector<ZGemmProblem> xp;
    std::vector<InvSpec> iv;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      int i = s.npl() - 1 - j;
      if (i < 0) continue;
      RgfWork& w = work[k];
      xp.push_back(gp(s.U[i], s.ldU[i], w.L[i], s.b[i + 1], w.W, s.b[i], s.b[i], s.b[i], s.b[i + 1],
                      cscale(s.uscale, -1.0), s.D[i], s.ldD[i], s.dscale, s.shift));
      xp.back().diag_ptr = s.shift_ptr;
      if (gn) gn->off(s, w, k, i, xp);
      iv.push_back(inv_spec(s, w, i));
    }
    plan.gemm('N', 'N', xp);
    plan.inv(iv);
  }
}

void build_rgf_downward(Plan& plan, const std::vector<TriSystem>& sys, std::vector<RgfWork>& work,
                        std::vector<TriOut>& out, const std::function<void(int)>& on_final) {
  int maxN = 0;
  for (const auto& s : sys) maxN = std::max(maxN, s.npl());
  // G_11 = X_1^{-1}  (rgf.jl:169)
  {
    std::vector<ZBlockOp> ops;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      if (s.npl() == 0) continue;
      ZBlockOp o{};
      o.A = work[k].g[0]; o.lda = s.b[0]; o.C = out[k].d[0]; o.ldc = out[k].ldd[0];
      o.m = o.n = s.b[0]; o.kind = ZOP_COPY;
      ops.push_back(o);
    }
    plan.blockops(ops);
  }
  if (on_final && maxN > 0) on_final(0);
  for (int i = 1; i < maxN; ++i) {
    // G[i-1,i] = -G[i-1,i-1] R_{i-1};  G[i,i-1] = -L_i G[i-1,i-1]  (rgf.jl:174,177)
    std::vector<ZGemmProblem> pr;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      if (i >= s.npl()) continue;
      RgfWork& w = work[k];
      TriOut& o = out[k];
      pr.push_back(gp(o.d[i - 1], o.ldd[i - 1], w.R[i - 1], s.b[i - 1], o.u[i - 1], o.ldu[i - 1], s.b[i - 1], s.b[i],
                      s.b[i - 1], MONE));
      if (o.l[i - 1])
        pr.push_back(gp(w.L[i - 1], s.b[i], o.d[i - 1], o.ldd[i - 1], o.l[i - 1], o.ldl[i - 1], s.b[i], s.b[i - 1],
                        s.b[i - 1], MONE));
    }
    plan.gemm('N', 'N', pr);
    // G[i,i] = X_i^{-1} - L_i G[i-1,i]  (rgf.jl:180-181)
    std::vector<ZGemmProblem> dp;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      if (i >= s.npl()) continue;
      RgfWork& w = work[k];
      TriOut& o = out[k];
      dp.push_back(gp(w.L[i - 1], s.b[i], o.u[i - 1], o.ldu[i - 1], o.d[i], o.ldd[i], s.b[i], s.b[i], s.b[i - 1],
                      MONE, w.g[i], s.b[i], ONE));
    }
    plan.gemm('N', 'N', dp);
    if (on_final) on_final(i);
  }
}

void build_rgf_full_inverse(Plan& plan, const std::vector<TriSystem>& sys, std::vector<RgfWork>& work,
                            std::vector<std::vector<cplx*>>& full) {
  // G[i,j] = -G[i,j-1] R_{j-1};  G[j,i] = -L_j G[j-1,i]  for j >= i+2  (rgf.jl:185-199)
  int maxN = 0;
  for (const auto& s : sys) maxN = std::max(maxN, s.npl());
  for (int d = 2; d < maxN; ++d) {
    std::vector<ZGemmProblem> pr;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      int n = s.npl();
      auto& F = full[k];
      RgfWork& w = work[k];
      for (int i = 0; i + d < n; ++i) {
        int j = i + d;
        if (F[i * n + j] && F[i * n + j - 1])
          pr.push_back(gp(F[i * n + j - 1], s.b[i], w.R[j - 1], s.b[j - 1], F[i * n + j], s.b[i], s.b[i], s.b[j],
                          s.b[j - 1], MONE));
        if (F[j * n + i] && F[(j - 1) * n + i])
          pr.push_back(gp(w.L[j - 1], s.b[j], F[(j - 1) * n + i], s.b[j - 1], F[j * n + i], s.b[j], s.b[j], s.b[i],
                          s.b[j - 1], MONE));
      }
    }
    plan.gemm('N', 'N', pr);
  }
}

// ---------------------------------------------------------------------------
// RKD (recursive Keldysh), src/keldyshndiag.jl:221-317, with every
// be_mldivide!('N', ., ., LU(X_i)) applied as a product with g_i = X_i^{-1}.

namespace {
// Upward pass of a general Hermitian S (diagonal and upper blocks, in place,
// keldyshndiag.jl:230-234), merged into the launches of the RGF upward pass:
//   S[i,i] -= R_i S[i,i+1]^H;  S[i,i+1] -= R_i S[i+1,i+1];  S[i,i] -= S[i,i+1] R_i^H
struct RkdUpward : GnUpward {
  std::vector<HermBlocks>& S;
  explicit RkdUpward(std::vector<HermBlocks>& s) : S(s) {}
  void before(const TriSystem& s, RgfWork& w, size_t k, int i, std::vector<ZGemmProblem>& nc) override {
    HermBlocks& h = S[k];
    nc.push_back(gp(w.R[i], s.b[i], h.u[i], h.ldu[i], h.d[i], h.ldd[i], s.b[i], s.b[i], s.b[i + 1], MONE, h.d[i],
                    h.ldd[i], ONE));
  }
  void off(const TriSystem& s, RgfWork& w, size_t k, int i, std::vector<ZGemmProblem>& nn) override {
    HermBlocks& h = S[k];
    nn.push_back(gp(w.R[i], s.b[i], h.d[i + 1], h.ldd[i + 1], h.u[i], h.ldu[i], s.b[i], s.b[i + 1], s.b[i + 1], MONE,
                    h.u[i], h.ldu[i], ONE));
  }
  void after(const TriSystem& s, RgfWork& w, size_t k, int i, std::vector<ZGemmProblem>& nc) override {
    if (i + 1 >= s.npl()) return;
    HermBlocks& h = S[k];
    nc.push_back(gp(h.u[i], h.ldu[i], w.R[i], s.b[i], h.d[i], h.ldd[i], s.b[i], s.b[i], s.b[i + 1], MONE, h.d[i],
                    h.ldd[i], ONE));
  }
};

// Upward pass of the lead operator S = Gamma_R on the last layer alone: with no
// off-diagonal blocks the recursion is S_i = R_i S_{i+1} R_i^H, two products.
struct LeadUpward : GnUpward {
  std::vector<LeadSystem>& Q;
  explicit LeadUpward(std::vector<LeadSystem>& q) : Q(q) {}
  const cplx* op(size_t k, int i) { return i + 1 == (int)Q[k].gl.size() ? Q[k].gamR : Q[k].gl[i]; }
  void off(const TriSystem& s, RgfWork& w, size_t k, int i, std::vector<ZGemmProblem>& nn) override {
    nn.push_back(gp(w.R[i], s.b[i], op(k, i + 1), s.b[i + 1], Q[k].v, s.b[i], s.b[i], s.b[i + 1], s.b[i + 1], ONE));
  }
  void after(const TriSystem& s, RgfWork& w, size_t k, int i, std::vector<ZGemmProblem>& nc) override {
    if (i + 1 >= s.npl()) return;
    nc.push_back(gp(Q[k].v, s.b[i], w.R[i], s.b[i], Q[k].gl[i], s.b[i], s.b[i], s.b[i], s.b[i + 1], ONE));
  }
};
}  // namespace

void build_rkd(Plan& plan, const std::vector<TriSystem>& sys, std::vector<RgfWork>& work,
               std::vector<HermBlocks>& S) {
  int maxN = 0;
  for (const auto& s : sys) maxN = std::max(maxN, s.npl());
  RkdUpward up(S);
  build_rgf_upward(plan, sys, work, &up);
  // workspace: G_ii of M^{-1} (y), one off-diagonal block, and a temporary per layer
  std::vector<std::vector<cplx*>> y(sys.size()), t(sys.size());
  std::vector<cplx*> yo(sys.size());
  for (size_t k = 0; k < sys.size(); ++k) {
    const auto& s = sys[k];
    const size_t bb = (size_t)s.maxb() * s.maxb();
    cplx* a = plan.alloc_c((2 * (size_t)s.npl() + 1) * bb);
    for (int i = 0; i < s.npl(); ++i) {
      y[k].push_back(i == 0 ? work[k].g[0] : a + 2 * i * bb);
      t[k].push_back(a + (2 * i + 1) * bb);
    }
    yo[k] = a + 2 * (size_t)s.npl() * bb;
  }
  // central pass (keldyshndiag.jl:257-291): its chain X_i = I + M[i,i-1] g_{i-1}
  // X_{i-1} R_{i-1}, multiplied by g_i, is the diagonal of the inverse itself,
  // g_i X_i = g_i + L_i (g_{i-1} X_{i-1}) R_{i-1} = G_ii: two products per layer
  for (int i = 1; i + 1 < maxN; ++i) {
    std::vector<ZGemmProblem> a1, a2;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      if (i + 1 >= s.npl()) continue;
      RgfWork& w = work[k];
      a1.push_back(gp(y[k][i - 1], s.b[i - 1], w.R[i - 1], s.b[i - 1], yo[k], s.b[i - 1], s.b[i - 1], s.b[i],
                      s.b[i - 1], ONE));
      a2.push_back(gp(w.L[i - 1], s.b[i], yo[k], s.b[i - 1], y[k][i], s.b[i], s.b[i], s.b[i], s.b[i - 1], ONE,
                      w.g[i], s.b[i], ONE));
    }
    plan.gemm('N', 'N', a1);
    plan.gemm('N', 'N', a2);
  }
  // S[i,i+1] = G_ii S[i,i+1] g_{i+1}^H (:285-291) and the diagonal rescale
  // S[i,i] = g_i S[i,i] g_i^H (:296-301), all layers at once
  {
    std::vector<ZGemmProblem> p1, p2;
    std::vector<std::vector<cplx*>> t2(sys.size());
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      const size_t bb = (size_t)s.maxb() * s.maxb();
      cplx* a = s.npl() > 1 ? plan.alloc_c((size_t)(s.npl() - 1) * bb) : nullptr;
      for (int i = 0; i + 1 < s.npl(); ++i) t2[k].push_back(a + i * bb);
    }
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      RgfWork& w = work[k];
      HermBlocks& h = S[k];
      for (int i = 0; i < s.npl(); ++i) {
        p1.push_back(gp(w.g[i], s.b[i], h.d[i], h.ldd[i], t[k][i], s.b[i], s.b[i], s.b[i], s.b[i], ONE));
        p2.push_back(gp(t[k][i], s.b[i], w.g[i], s.b[i], h.d[i], h.ldd[i], s.b[i], s.b[i], s.b[i], ONE));
        if (i + 1 == s.npl()) continue;
        p1.push_back(gp(y[k][i], s.b[i], h.u[i], h.ldu[i], t2[k][i], s.b[i], s.b[i], s.b[i + 1], s.b[i], ONE));
        p2.push_back(gp(t2[k][i], s.b[i], w.g[i + 1], s.b[i + 1], h.u[i], h.ldu[i], s.b[i], s.b[i + 1], s.b[i + 1],
                        ONE));
      }
    }
    plan.gemm('N', 'N', p1);
    plan.gemm('N', 'C', p2);
  }
  // downward RKD pass (keldyshndiag.jl:313-317), ix = 0 .. N-2:
  //   S[i+1,i+1] -= S[i,i+1]^H L_{i+1}^H, for all layers at once (it takes
  //   S[i,i+1] as the central pass left it), then layer by layer
  //   S[i,i+1] -= S[i,i] L_{i+1}^H;  S[i+1,i+1] -= L_{i+1} S[i,i+1]
  {
    std::vector<ZGemmProblem> d1;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      RgfWork& w = work[k];
      HermBlocks& h = S[k];
      for (int i = 0; i + 1 < s.npl(); ++i)
        d1.push_back(gp(h.u[i], h.ldu[i], w.L[i], s.b[i + 1], h.d[i + 1], h.ldd[i + 1], s.b[i + 1], s.b[i + 1], s.b[i],
                        MONE, h.d[i + 1], h.ldd[i + 1], ONE));
    }
    plan.gemm('C', 'C', d1);
  }
  for (int i = 0; i + 1 < maxN; ++i) {
    std::vector<ZGemmProblem> d2, d3;
    for (size_t k = 0; k < sys.size(); ++k) {
      const auto& s = sys[k];
      if (i + 1 >= s.npl()) continue;
      RgfWork& w = work[k];
      HermBlocks& h = S[k];
      d2.push_back(gp(h.d[i], h.ldd[i], w.L[i], s.b[i + 1], h.u[i], h.ldu[i], s.b[i], s.b[i + 1], s.b[i], MONE,
                      h.u[i], h.ldu[i], ONE));
      d3.push_back(gp(w.L[i], s.b[i + 1], h.u[i], h.ldu[i], h.d[i + 1], h.ldd[i + 1], s.b[i + 1], s.b[i + 1], s.b[i],
                      MONE, h.d[i + 1], h.ldd[i + 1], ONE));
    }
    plan.gemm('N', 'C', d2);
    plan.gemm('N', 'N', d3);
  }
}

// ---------------------------------------------------------------------------
// G^R and G^< diagonals and the transmission of lead-driven systems.
//
// Sigma^in = f_L Gamma_L on layer 0 and f_R Gamma_R on layer N-1, so the
// Hermitian operator of keldyshndiag! has no off-diagonal blocks and stays a
// chain (S_i = R_i .. R_{N-2} Gamma_R (..)^H); its products share work with
// those of G^R.  Per layer 13 products of 8 b^3 flops (21 in the general
// sequence with the blocks of G^R below the diagonal: 32 x 256, 64 energies,
// FP64 194 -> 134 ms, mixed 131 -> 87 ms), in 4 + 4 launches:
//   up (with the RGF pass): v = R_i S_{i+1};  S_i = v R_i^H
//   all layers:             t_i = f_R S_i g_i^H (i = 0: + f_L Gamma_L g_0^H);  n_i = g_i t_i
//   down:                   G_{i,i+1} = -G_ii R_i;  G_{i+1,i+1} = g_{i+1} - L_{i+1} G_{i,i+1}
//                           A = G_{i,i+1} t_{i+1} - G^n_ii L_{i+1}^H / 2
//                           G^n_{i+1,i+1} = n_{i+1} - L_{i+1} A - (L_{i+1} A)^H
// (the last two are keldyshndiag.jl:313-317 with both updates of S[i+1,i+1] as
// one product and its conjugate transpose), and beside them G_{0,i+1} =
// -G_{0,i} R_i for T = Re Tr[Gamma_L G_{0,N-1} Gamma_R G_{0,N-1}^H] (from S_0,
// T would need no chain, but its error doubled).
void build_lead_pass(Plan& plan, const std::vector<TriSystem>& sys, std::vector<RgfWork>& work,
                     std::vector<LeadSystem>& Q, const std::function<void(int)>& gr_final,
                     const std::function<void(int)>& gl_final) {
  int maxN = 0;
  const size_t ns = sys.size();
  for (const auto& s : sys) maxN = std::max(maxN, s.npl());
  std::vector<std::vector<cplx*>> t(ns);
  std::vector<cplx*> u(ns), ub(ns), q(ns);
  std::vector<std::vector<cplx*>> y(ns);  // G_{0,i} (two in turn), and the two factors of the trace
  std::vector<std::vector<cplx*>> G(ns);
  for (size_t k = 0; k < ns; ++k) {
    const auto& s = sys[k];
    const size_t bb = (size_t)s.maxb() * s.maxb();
    Q[k].v = plan.alloc_c(bb);
    u[k] = plan.alloc_c(bb);
    ub[k] = plan.alloc_c(bb);
    q[k] = plan.alloc_c((size_t)s.b[0] * s.b[0]);
    if (Q[k].t_out)
      for (int c = 0; c < 4; ++c) y[k].push_back(plan.alloc_c((size_t)s.b[0] * s.maxb()));
    cplx* ring = Q[k].gr.empty() ? plan.alloc_c(2 * bb) : nullptr;
    for (int i = 0; i < s.npl(); ++i) {
      t[k].push_back(plan.alloc_c((size_t)s.b[i] * s.b[i]));
      G[k].push_back(ring ? ring + (i & 1) * bb : Q[k].gr[i]);
    }
  }
  LeadUpward up(Q);
  build_rgf_upward(plan, sys, work, &up);
  auto block = [](ZOpKind kind, const cplx* A, cplx* C, int b, cplx alpha, cplx beta, const cplx* alpha_ptr) {
    ZBlockOp o{};
    o.A = A; o.C = C; o.alpha_ptr = alpha_ptr; o.m = o.n = o.lda = o.ldc = b; o.kind = kind;
    o.alpha = alpha; o.beta = beta;
    return o;
  };
  {
    std::vector<ZGemmProblem> tp, np;
    std::vector<ZBlockOp> t0, g0, l0;
    for (size_t k = 0; k < ns; ++k) {
      const auto& s = sys[k];
      RgfWork& w = work[k];
      for (int i = 0; i < s.npl(); ++i) {
        const int b = s.b[i];
        tp.push_back(gp(up.op(k, i), b, w.g[i], b, i == 0 ? q[k] : t[k][i], b, b, b, b, ONE));
        if (i > 0) tp.back().alpha_ptr = Q[k].fR;
        np.push_back(gp(w.g[i], b, t[k][i], b, Q[k].gl[i], b, b, b, b, ONE));
      }
      const int b0 = s.b[0];
      tp.push_back(gp(Q[k].gamL, b0, w.g[0], b0, t[k][0], b0, b0, b0, b0, ONE));
      tp.back().alpha_ptr = Q[k].fL;
      t0.push_back(block(ZOP_AXPBY, q[k], t[k][0], b0, ONE, ONE, Q[k].fR));
      if (!Q[k].gr.empty()) g0.push_back(block(ZOP_COPY, w.g[0], Q[k].gr[0], b0, ONE, ZERO, nullptr));
      l0.push_back(block(ZOP_AXPBY, Q[k].gl[0], Q[k].gl[0], b0, make_double2(0.0, 1.0), ZERO, nullptr));
      G[k][0] = w.g[0];
    }
    plan.gemm('N', 'C', tp);
    plan.blockops(t0);
    plan.gemm('N', 'N', np);
    plan.blockops(g0);
    if (!g0.empty() && gr_final) gr_final(0);
    plan.blockops(l0);  // G^< = i G^n
    if (gl_final) gl_final(0);
  }
  auto g0 = [&](size_t k, int i) -> cplx* { return i == 0 ? work[k].g[0] : y[k][i & 1]; };
  auto push_u = [&](int i, std::vector<ZGemmProblem>& v) {
    for (size_t k = 0; k < ns; ++k) {
      const auto& s = sys[k];
      if (i + 1 >= s.npl()) continue;
      v.push_back(gp(G[k][i], s.b[i], work[k].R[i], s.b[i], u[k], s.b[i], s.b[i], s.b[i + 1], s.b[i], MONE));
      if (Q[k].t_out)  // beside the product with the same R_i: one digit split of it
        v.push_back(gp(g0(k, i), s.b[0], work[k].R[i], s.b[i], g0(k, i + 1), s.b[0], s.b[0], s.b[i + 1], s.b[i], MONE));
    }
  };
  {
    std::vector<ZGemmProblem> v;
    push_u(0, v);
    plan.gemm('N', 'N', v);
  }
  for (int i = 0; i + 1 < maxN; ++i) {
    std::vector<ZGemmProblem> a, c, x;
    std::vector<ZBlockOp> h;
    bool any_gr = false;
    for (size_t k = 0; k < ns; ++k) {
      const auto& s = sys[k];
      if (i + 1 >= s.npl()) continue;
      RgfWork& w = work[k];
      const int b = s.b[i], b1 = s.b[i + 1];
      a.push_back(gp(w.L[i], b1, u[k], b, G[k][i + 1], b1, b1, b1, b, MONE, w.g[i + 1], b1, ONE));
      a.push_back(gp(u[k], b, t[k][i + 1], b1, ub[k], b, b, b1, b1, ONE));
      // gl[i] = i G^n_ii, so -G^n_ii / 2 is (i / 2) gl[i]
      c.push_back(gp(Q[k].gl[i], b, w.L[i], b1, ub[k], b, b, b1, b, make_double2(0.0, 0.5), ub[k], b, ONE));
      // t_{i+1} is done with: it takes n_{i+1} / 2 - L_{i+1} A
      x.push_back(gp(w.L[i], b1, ub[k], b, t[k][i + 1], b1, b1, b1, b, MONE, Q[k].gl[i + 1], b1,
                     make_double2(0.5, 0.0)));
      h.push_back(block(ZOP_HERM_SUM, t[k][i + 1], Q[k].gl[i + 1], b1, make_double2(0.0, 1.0), ZERO, nullptr));
      any_gr = any_gr || !Q[k].gr.empty();
    }
    plan.gemm('N', 'N', a);
    if (any_gr && gr_final) gr_final(i + 1);
    plan.gemm('N', 'C', c);
    push_u(i + 1, x);
    plan.gemm('N', 'N', x);
    plan.blockops(h);
    if (gl_final) gl_final(i + 1);
  }
  std::vector<ZGemmProblem> p1, p2;
  std::vector<ZTraceProblemHost> tr;
  for (size_t k = 0; k < ns; ++k) {
    if (!Q[k].t_out) continue;
    const auto& s = sys[k];
    const int n = s.npl(), b0 = s.b[0], bN = s.b[n - 1];
    p1.push_back(gp(Q[k].gamL, b0, g0(k, n - 1), b0, y[k][2], b0, b0, bN, b0, ONE));
    p2.push_back(gp(Q[k].gamR, bN, g0(k, n - 1), b0, y[k][3], bN, bN, b0, bN, ONE));
    ZTraceProblemHost x{};
    x.X = y[k][2]; x.ldx = b0; x.Y = y[k][3]; x.ldy = bN; x.n = b0; x.out = Q[k].t_out;
    tr.push_back(x);
  }
  plan.gemm('N', 'N', p1);
  plan.gemm('N', 'C', p2);
  plan.trace(tr);
}

}  // namespace negf
