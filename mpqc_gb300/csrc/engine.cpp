// Contraction planner and executor (see engine.h).
#include "engine.h"

#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <mutex>
#include <sstream>

namespace gbcc {

// Autotune choices shared by every handle of the process, by contraction
// shape: a handle whose contractions were timed before (by another handle, or
// in an earlier process whose table was saved and loaded) takes the stored
// tile instead of timing its candidates again.
namespace {
struct TuneChoice {
  int bn, ksplit, sps, group;
  int64_t kps;
};
std::mutex g_tune_mu;
std::map<std::string, TuneChoice>& tune_table() {
  static std::map<std::string, TuneChoice> t;
  return t;
}
}  // namespace

bool tune_save(const std::string& path) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  std::ofstream f(path);
  if (!f) return false;
  f << "gbcc-autotune 1\n";
  for (const auto& kv : tune_table())
    f << kv.first << ' ' << kv.second.bn << ' ' << kv.second.ksplit << ' ' << kv.second.kps << ' '
      << kv.second.sps << ' ' << kv.second.group << '\n';
  return static_cast<bool>(f);
}

bool tune_load(const std::string& path) {
  std::ifstream f(path);
  if (!f) return false;
  std::string line;
  if (!std::getline(f, line) || line != "gbcc-autotune 1") return false;
  std::map<std::string, TuneChoice> add;
  while (std::getline(f, line)) {
    if (line.empty()) continue;
    std::istringstream is(line);
    std::string key;
    TuneChoice c{};
    if (!(is >> key >> c.bn >> c.ksplit >> c.kps >> c.sps >> c.group)) return false;
    std::string extra;
    if (is >> extra) return false;
    if (c.bn <= 0 || c.bn > 256 || c.ksplit < 1 || c.kps < 0 || c.sps < 1 || c.sps > 2 || c.group < 1) return false;
    add[key] = c;
  }
  std::lock_guard<std::mutex> lk(g_tune_mu);
  for (const auto& kv : add) tune_table()[kv.first] = kv.second;
  return true;
}

void tune_clear() {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  tune_table().clear();
}

// test hooks (gbcc_testing_fail_alloc): device allocations made so far, and
// how many more succeed before one fails as if the device were full (-1: all)
std::atomic<int64_t> g_alloc_count{0};
std::atomic<int64_t> g_fail_alloc_after{-1};

// test hooks: lanes of plans made from now on (gbcc_testing_lanes_mode: -1 as
// finalize() decides, 0 one, 1 the program's), and the free bytes that lanes_fit
// is told of (gbcc_testing_free_bytes, -1: the device's)
std::atomic<int> g_lanes_mode{-1};
std::atomic<int64_t> g_free_bytes{-1};

size_t device_bytes_free() {
  const int64_t told = g_free_bytes.load();
  if (told >= 0) return static_cast<size_t>(told);
  size_t free = 0, total = 0;
  if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return free;
}

// test hook (gbcc_testing_fail_site): the operation of an EXEC pass that fails
// instead of being launched, once (-1: none)
std::atomic<int64_t> g_fail_site{-1};

void* dev_alloc(size_t bytes) {
  if (bytes == 0) bytes = 256;
  ++g_alloc_count;
  int64_t left = g_fail_alloc_after.load();
  while (left >= 0 && !g_fail_alloc_after.compare_exchange_weak(left, left - 1)) {
  }
  if (left == 0)
    throw Error(GBCC_ERR_OOM, "cudaMalloc of " + std::to_string(bytes) + " bytes failed: injected failure (test hook)");
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error(GBCC_ERR_OOM, "cudaMalloc of " + std::to_string(bytes) + " bytes failed: " +
                                  cudaGetErrorString(e));
  }
  return p;
}

void dev_free(void* p) {
  if (p) cudaFree(p);
}

namespace {

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

using Extents = std::map<char, int64_t>;

int label_pos(const std::string& lab, char c) {
  auto p = lab.find(c);
  return p == std::string::npos ? -1 : static_cast<int>(p);
}

void check_ix(const Ix& x) {
  if (!x.t) throw Error(GBCC_ERR_STATE, "engine: null tensor");
  if (static_cast<int>(x.lab.size()) != x.t->rank)
    throw Error(GBCC_ERR_STATE, "engine: label count mismatch for " + x.t->name + "(" + x.lab + ")");
}

void add_extents(Extents& e, const Ix& x) {
  check_ix(x);
  for (int k = 0; k < x.t->rank; ++k) {
    char c = x.lab[k];
    auto it = e.find(c);
    if (it == e.end())
      e[c] = x.t->dim[k];
    else if (it->second != x.t->dim[k])
      throw Error(GBCC_ERR_STATE, std::string("engine: extent mismatch for index ") + c + " in " +
                                      x.t->name);
  }
}

int64_t extent_of(const Extents& e, const std::string& labs) {
  int64_t n = 1;
  for (char c : labs) n *= e.at(c);
  return n;
}

int64_t stride_in(const Ix& x, char c) {
  int p = label_pos(x.lab, c);
  return p < 0 ? 0 : x.t->stride(p);
}

// offsets of the composite index over `order` (row-major) into tensor x
std::vector<int64_t> offsets(const std::string& order, const Extents& e, const Ix& x) {
  const int64_t n = extent_of(e, order);
  std::vector<int64_t> out(static_cast<size_t>(n));
  const int d = static_cast<int>(order.size());
  std::vector<int64_t> ext(d), str(d), idx(d, 0);
  for (int k = 0; k < d; ++k) {
    ext[k] = e.at(order[k]);
    str[k] = stride_in(x, order[k]);
  }
  int64_t off = 0;
  for (int64_t i = 0; i < n; ++i) {
    out[static_cast<size_t>(i)] = off;
    for (int k = d - 1; k >= 0; --k) {
      ++idx[k];
      off += str[k];
      if (idx[k] < ext[k]) break;
      off -= str[k] * ext[k];
      idx[k] = 0;
    }
  }
  return out;
}

// labels of `set` in the order they appear in `ref`
std::string order_by(const std::string& set, const std::string& ref) {
  std::string out;
  for (char c : ref)
    if (set.find(c) != std::string::npos) out.push_back(c);
  return out;
}

std::string set_minus(const std::string& a, const std::string& b) {
  std::string out;
  for (char c : a)
    if (b.find(c) == std::string::npos) out.push_back(c);
  return out;
}

std::string set_and(const std::string& a, const std::string& b) {
  std::string out;
  for (char c : a)
    if (b.find(c) != std::string::npos) out.push_back(c);
  return out;
}

// Gather direction: read along R (and transpose in shared memory) when the
// first term is unit-stride along R but not along C.
int pick_transpose(const std::vector<int64_t>& ra, const std::vector<int64_t>& ca) {
  const bool r_unit = ra.size() > 1 && ra[1] - ra[0] == 1;
  const bool c_unit = ca.size() > 1 && ca[1] - ca[0] == 1;
  return (r_unit && !c_unit && ra.size() >= 32) ? 1 : 0;
}

bool same_set(const std::string& a, const std::string& b) {
  std::string x = a, y = b;
  std::sort(x.begin(), x.end());
  std::sort(y.begin(), y.end());
  return x == y;
}

}  // namespace

// ---------------------------------------------------------------------------

struct OperandPlan {
  std::vector<Lin> terms;
  std::string ext;    // ordered external labels (GEMM rows)
  std::string kord;   // ordered contracted labels
  int64_t rows = 0, K = 0;
  bool constant = false;
  bool direct = false;  // FP64: tensor storage used as the panel
  bool inplace = false;  // small-K stream kernel: the one source read in place through its gather tables
  const double* dptr = nullptr;
  int64_t ld = 0;
  GatherArgs gather{};  // packing (FP64 panel or split slices)
  int slices = 0;
  int64_t rows_pad = 0, Kpad = 0;
  __nv_bfloat16* packed = nullptr;  // dedicated split buffer (constants)
  size_t pack_elems = 0;
  // reuse of one split pack by several contractions within a residual
  std::string sig;        // non-empty: sources are not written during a residual
  bool cache_first = false;  // packs into cache_buf
  bool cache_reuse = false;  // reads cache_buf packed by an earlier contraction
  __nv_bfloat16* cache_buf = nullptr;
  int lane = 0;
  cudaEvent_t packed_ev = nullptr;  // first use: recorded after the pack when another lane reads it
  OperandPlan* first_use = nullptr;  // reuse in another lane: the operand to wait for
  // FP64_TC: fixed-point slices under per-row exponents (rows_pad words)
  bool fixed = false;
  unsigned* rowexp = nullptr;
};

// The in-place FP64 kernel (gemm_small.cu) takes a contraction whose estimated
// time is at most this many microseconds: in the FP64 plan, where the panel
// GEMM needs two packs first (500^3: 230 us, the panel GEMM alone 347 us;
// 741^3: 711 against 780 us; beyond that each operand is read too many times);
// in the mixed plan, where a tensor-core launch costs 15-30 us and its packs
// 5-10 us each however small the product; in the FP64_TC plan, with six
// slices to pack.
constexpr double kSmallUs = 800.0;
constexpr double kSmallUsMixed = 20.0;
constexpr double kSmallUsFixed = 80.0;
// While slice counts are chosen (set_trial) the mixed plan runs in FP64 only
// contractions below this many FLOPs, so that the choice is made from the split
// error of the same contractions at every size and does not loosen where a
// size runs some of them in FP64.
constexpr double kTrialFlops = 1.0e6;

struct GemmPlan {
  bool use_tc = false;
  bool smallk = false;     // mixed precision, K <= kSmallK: FP32 CUDA-core kernel on FP64 panels
  bool small = false;      // FP64, operands read in place (gemm_small.cu)
  GemmSmallArgs sg{};
  bool a_is_first = true;  // GEMM M side is the call's A operand
  int64_t M = 0, N = 0, K = 0;
  OperandPlan P[2];        // [0] = M side, [1] = N side
  const int64_t* cm = nullptr;
  const int64_t* cn = nullptr;
  double alpha = 1.0, beta = 0.0;
  double* C = nullptr;
  int slices = 0, npairs = 0, bn = 0;
  bool emu = false;        // FP64_TC: fixed-point slices (gemm_multi.cu)
  int ksplit = 1;         // K split over CTAs (deterministic two-pass reduction)
  bool m_major = false;   // C unit-stride along M
  int64_t k_per_split = 0;  // FP64: K elements per split; tensor cores: k-blocks (FP64_TC: halves of them) per split
  int pa[kMaxPairs] = {}, pb[kMaxPairs] = {};
  double flops = 0.0;
  int sps = 1;             // tensor cores: slices per pipeline stage (2: both slices of a k-block)
  int group = 1;           // tensor cores: M tiles per band of the tile order (1: rows)
  // tensor cores: (tile width, K split, slices per stage, band) candidates
  // for the tuner, the plan's heuristic choice first
  static constexpr int kMaxCand = 24;
  int ncand = 0;
  int cand_bn[kMaxCand] = {}, cand_ks[kMaxCand] = {}, cand_sps[kMaxCand] = {}, cand_group[kMaxCand] = {};
  int64_t cand_kps[kMaxCand] = {};
};

struct Site {
  int kind = 0;  // 0 assign, 1 contract, 2 custom kernels
  TermClass cls = kClassOther;
  GatherArgs gather{};
  GemmPlan plan[3];  // by plan_index(precision)
  cudaEvent_t e0 = nullptr, e1 = nullptr, eg = nullptr;  // profiling: start, end, GEMM start
  bool has_gemm = false;
  int lane = 0;
  std::string label;  // NVTX range name: the operation and its operands
  ~Site() {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (eg) cudaEventDestroy(eg);
    for (const GemmPlan& p : plan)
      for (const OperandPlan& op : p.P)
        if (op.packed_ev) cudaEventDestroy(op.packed_ev);
  }
};

// NVTX ranges around every operation of an EXEC pass when GBCC_NVTX is set in
// the environment (a profiler then shows them; graph replays record none, so
// profile with use_graphs = 0)
static bool nvtx_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("GBCC_NVTX");
    return e && *e && std::strcmp(e, "0") != 0;
  }();
  return on;
}

void Engine::prof_begin(Site& s) {
  if (nvtx_enabled()) nvtxRangePushA(s.label.c_str());
  if (!profile_) return;
  if (!s.e0) GBCC_CK(cudaEventCreate(&s.e0));
  if (!s.e1) GBCC_CK(cudaEventCreate(&s.e1));
  if (!s.eg) GBCC_CK(cudaEventCreate(&s.eg));
  GBCC_CK(cudaEventRecord(s.e0, run_));
  s.has_gemm = false;
}

void Engine::prof_gemm(Site& s) {
  if (!profile_) return;
  GBCC_CK(cudaEventRecord(s.eg, run_));
  s.has_gemm = true;
}

void Engine::prof_end(Site& s) {
  if (profile_) GBCC_CK(cudaEventRecord(s.e1, run_));
  if (nvtx_enabled()) nvtxRangePop();
}

std::vector<SiteStat> Engine::site_stats(int precision) {
  std::vector<SiteStat> out;
  GBCC_CK(cudaStreamSynchronize(stream_));
  for (auto& sp : sites_) {
    SiteStat st;
    if (sp->e0 && sp->e1) {
      float ms = 0.f;
      GBCC_CK(cudaEventElapsedTime(&ms, sp->e0, sp->e1));
      st.ms = ms;
      if (sp->has_gemm) {
        GBCC_CK(cudaEventElapsedTime(&ms, sp->eg, sp->e1));
        st.gemm_ms = ms;
      }
    }
    if (sp->kind == 1) {
      const GemmPlan& p = sp->plan[plan_index(precision)];
      st.flops = p.flops;
      st.pairs = p.use_tc ? p.npairs : 0;
      st.cls = sp->cls;
      st.M = p.M;
      st.N = p.N;
      st.K = p.K;
      st.bn = p.use_tc ? p.bn : (p.smallk ? -1 : 0);
      st.ksplit = p.ksplit;
      st.sps = p.use_tc ? p.sps : 0;
      st.group = p.use_tc ? p.group : 0;
    } else {
      st.M = sp->gather.R;
      st.N = sp->gather.C;
    }
    out.push_back(st);
  }
  return out;
}

Engine::Engine() = default;

Engine::~Engine() {
  for (void* p : owned_) dev_free(p);
  for (auto& kv : tensors_) dev_free(kv.second->d);
  free_workspaces();
  for (cudaEvent_t e : marks_) cudaEventDestroy(e);
  for (int k = 1; k < kLanes; ++k)
    if (lane_ws_[k].stream) cudaStreamDestroy(lane_ws_[k].stream);
}

// every pointer is cleared before any new allocation: one that fails leaves no
// pointer to freed memory behind
void Engine::free_workspaces() {
  if (scratch_) bytes_ -= workspace_bytes();
  scratch_ = false;
  for (Lane& w : lane_ws_) {
    for (void** p : {reinterpret_cast<void**>(&w.w64a), reinterpret_cast<void**>(&w.w64b),
                     reinterpret_cast<void**>(&w.wbfa), reinterpret_cast<void**>(&w.wbfb),
                     reinterpret_cast<void**>(&w.wpart), reinterpret_cast<void**>(&w.wcount)}) {
      dev_free(*p);
      *p = nullptr;
    }
  }
}

void Engine::alloc_workspaces() {
  free_workspaces();
  for (int k = 0; k < nlanes_; ++k) {
    Lane& w = lane_ws_[k];
    if (k > 0 && !w.stream) GBCC_CK(cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking));
    w.w64a = static_cast<double*>(dev_alloc(w.n64a * sizeof(double)));
    w.w64b = static_cast<double*>(dev_alloc(w.n64b * sizeof(double)));
    w.wbfa = static_cast<__nv_bfloat16*>(dev_alloc(w.nbfa * sizeof(__nv_bfloat16)));
    w.wbfb = static_cast<__nv_bfloat16*>(dev_alloc(w.nbfb * sizeof(__nv_bfloat16)));
    w.wpart = static_cast<double*>(dev_alloc(w.npart * sizeof(double)));
    w.wcount = static_cast<unsigned*>(dev_alloc(w.ncount * sizeof(unsigned)));
    GBCC_CK(cudaMemsetAsync(w.wcount, 0, std::max<size_t>(w.ncount, 1) * sizeof(unsigned), stream_));
  }
  bytes_ += workspace_bytes();
  scratch_ = true;
}

bool Engine::one_lane() {
  if (nlanes_ <= 1) return false;
  release_scratch();
  merge_lanes();
  return true;
}

bool Engine::release_scratch() {
  if (!scratch_ || workspace_bytes() == 0) return false;
  abandon();
  GBCC_CK(cudaStreamSynchronize(stream_));
  free_workspaces();
  return true;
}

void Engine::lane(int k) {
  lane_ = k;
  if (mode_ == Mode::kPlan) nlanes_ = std::max(nlanes_, k + 1);
}

int Engine::mark(int k) {
  const int m = mark_cursor_++;
  if (mode_ == Mode::kPlan) {
    if (m >= static_cast<int>(marks_.size())) {
      cudaEvent_t e = nullptr;
      GBCC_CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      marks_.push_back(e);
    }
  } else if (concurrent()) {
    GBCC_CK(cudaEventRecord(marks_.at(m), lane_ws_[k].stream));
  }
  return m;
}

void Engine::wait(int k, int m) {
  if (mode_ == Mode::kExec && concurrent()) GBCC_CK(cudaStreamWaitEvent(lane_ws_[k].stream, marks_.at(m), 0));
}

void Engine::abandon() noexcept {
  for (int k = 1; k < nlanes_; ++k) {
    cudaStream_t s = lane_ws_[k].stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (s && cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
      cudaStreamSynchronize(s);
  }
  cudaGetLastError();
  lane_ = 0;
  run_ = stream_;
  ws_ = &lane_ws_[0];
}

size_t Engine::lane_bytes(const Lane& w) {
  return w.ncount * sizeof(unsigned) + (w.n64a + w.n64b + w.npart) * sizeof(double) +
         (w.nbfa + w.nbfb) * sizeof(__nv_bfloat16);
}

size_t Engine::workspace_bytes() const {
  size_t n = 0;
  for (int k = 0; k < nlanes_; ++k) n += lane_bytes(lane_ws_[k]);
  return n;
}

// one workspace that serves every lane's operations in turn
Engine::Lane Engine::merged_lane() const {
  Lane m = lane_ws_[0];
  for (int k = 1; k < nlanes_; ++k) {
    const Lane& w = lane_ws_[k];
    m.n64a = std::max(m.n64a, w.n64a);
    m.n64b = std::max(m.n64b, w.n64b);
    m.nbfa = std::max(m.nbfa, w.nbfa);
    m.nbfb = std::max(m.nbfb, w.nbfb);
    m.npart = std::max(m.npart, w.npart);
    m.ncount = std::max(m.ncount, w.ncount);
  }
  return m;
}

void Engine::merge_lanes() {
  lane_ws_[0] = merged_lane();
  for (int k = 1; k < nlanes_; ++k) {
    Lane& w = lane_ws_[k];
    w.n64a = w.n64b = w.nbfa = w.nbfb = w.npart = w.ncount = 0;
  }
  nlanes_ = 1;
  for (auto& sp : sites_) {
    sp->lane = 0;
    for (GemmPlan& p : sp->plan)
      for (OperandPlan& op : p.P) op.lane = 0;
  }
}

// Whether the lanes' workspaces beyond one lane's leave room for what the handle may
// still allocate beside them: this plan's shared and constant packs in the precisions
// it runs, and the owner's reserve.  (Up to 32 MB the device is not asked: that takes
// 0.3 ms, an eighth of a small handle's set-up.)
bool Engine::lanes_fit() const {
  if (g_free_bytes.load() < 0 && workspace_bytes() - lane_bytes(merged_lane()) <= size_t{32} << 20) return true;
  size_t need = reserve_ + workspace_bytes();
  for (const auto& sp : sites_)
    for (int pm = mixed_ ? 1 : 2; pm < 3; ++pm)
      for (const OperandPlan& op : sp->plan[pm].P)
        if (sp->plan[pm].use_tc && op.constant) need += op.pack_elems * sizeof(__nv_bfloat16);
  for (const auto& kv : pack_uses_)
    if (kv.second.size() > 1) need += kv.second.front()->pack_elems * sizeof(__nv_bfloat16);
  return need <= device_bytes_free();
}

int Engine::lanes_busy() const {
  int n = 0;
  for (int k = 1; k < nlanes_; ++k)
    if (lane_ws_[k].stream && cudaStreamQuery(lane_ws_[k].stream) == cudaErrorNotReady) ++n;
  return n;
}

Tensor& Engine::tensor(const std::string& name, std::initializer_list<int64_t> dims, bool constant) {
  auto it = tensors_.find(name);
  if (it != tensors_.end()) {
    Tensor& t = *it->second;
    int k = 0;
    bool same = static_cast<int>(dims.size()) == t.rank;
    for (int64_t dval : dims) same = same && (k < t.rank && t.dim[k++] == dval);
    if (!same) throw Error(GBCC_ERR_STATE, "engine: tensor " + name + " re-requested with new shape");
    return t;
  }
  auto t = std::make_unique<Tensor>();
  t->name = name;
  t->rank = static_cast<int>(dims.size());
  int k = 0;
  for (int64_t dval : dims) t->dim[k++] = dval;
  t->constant = constant;
  const size_t bytes = static_cast<size_t>(t->size()) * sizeof(double);
  t->d = static_cast<double*>(dev_alloc(bytes));
  GBCC_CK(cudaMemsetAsync(t->d, 0, bytes, stream_));
  bytes_ += bytes;
  Tensor& ref = *t;
  tensors_[name] = std::move(t);
  return ref;
}

void Engine::release(Tensor& t) {
  if (!t.d) return;
  GBCC_CK(cudaStreamSynchronize(stream_));
  dev_free(t.d);
  t.d = nullptr;
  bytes_ -= static_cast<size_t>(t.size()) * sizeof(double);
}

void Engine::acquire(Tensor& t) {
  if (t.d) return;
  const size_t bytes = static_cast<size_t>(t.size()) * sizeof(double);
  t.d = static_cast<double*>(dev_alloc(bytes));
  GBCC_CK(cudaMemsetAsync(t.d, 0, bytes, stream_));
  bytes_ += bytes;
}

Tensor* Engine::find(const std::string& name) {
  auto it = tensors_.find(name);
  return it == tensors_.end() ? nullptr : it->second.get();
}

void Engine::reset_plans() {
  pack_uses_.clear();
  sites_.clear();
  for (void* p : owned_) dev_free(p);
  owned_.clear();
  tables_.clear();
  planned_ = false;
  free_workspaces();
  for (Lane& w : lane_ws_) w.n64a = w.n64b = w.nbfa = w.nbfb = w.npart = w.ncount = 0;
  nlanes_ = 1;
}

void Engine::begin(Mode m, int precision) {
  if (m == Mode::kExec && !planned_) throw Error(GBCC_ERR_STATE, "engine: EXEC before PLAN");
  mode_ = m;
  prec_ = precision;
  cursor_ = 0;
  flops_ = 0.0;
  n_tc_ = 0;
  n_launch_ = 0;
  lane_ = 0;
  mark_cursor_ = 0;
  run_ = stream_;
  ws_ = &lane_ws_[0];
  if (m == Mode::kPlan) {
    (void)mark(0);  // mark 0: the lanes' common start
  } else {
    lane_ws_[0].stream = stream_;
    const int m0 = mark(0);
    for (int k = 1; k < nlanes_; ++k) wait(k, m0);
  }
}

void Engine::end() {
  if (mode_ == Mode::kPlan) {
    for (int k = 1; k < nlanes_; ++k) (void)mark(k);
    planned_ = true;
  } else {
    if (cursor_ != sites_.size()) throw Error(GBCC_ERR_STATE, "engine: program ended early");
    for (int k = 1; k < nlanes_; ++k) wait(0, mark(k));
  }
  lane_ = 0;
  run_ = stream_;
  ws_ = &lane_ws_[0];
}

Site& Engine::site() {
  if (mode_ == Mode::kPlan) {
    sites_.push_back(std::make_unique<Site>());
    ++cursor_;
    sites_.back()->lane = lane_;
    ws_ = &lane_ws_[lane_];
    return *sites_.back();
  }
  if (cursor_ >= sites_.size()) throw Error(GBCC_ERR_STATE, "engine: program longer than its plan");
  if (g_fail_site.load() == static_cast<int64_t>(cursor_)) {
    g_fail_site.store(-1);
    throw Error(GBCC_ERR_CUDA, "operation not launched: injected failure (test hook)");
  }
  Site& s = *sites_[cursor_++];
  ws_ = &lane_ws_[s.lane];
  run_ = concurrent() ? ws_->stream : stream_;
  return s;
}

// Offset tables are small and many (several per operand and plan): they share
// chunks of device memory, filled on the host while planning and copied once
// each in finalize().
DevTable Engine::upload(const std::vector<int64_t>& v) {
  constexpr size_t kChunk = 1 << 17, kAlign = 32;  // elements; 256-byte aligned tables
  const size_t need = (std::max<size_t>(v.size(), 1) + kAlign - 1) / kAlign * kAlign;
  if (tables_.empty() || tables_.back().host.size() + need > tables_.back().cap) {
    TableChunk c;
    c.cap = std::max(need, kChunk);
    c.d = static_cast<int64_t*>(dev_alloc(c.cap * sizeof(int64_t)));
    owned_.push_back(c.d);
    bytes_ += c.cap * sizeof(int64_t);
    tables_.push_back(std::move(c));
  }
  TableChunk& c = tables_.back();
  DevTable t;
  t.n = static_cast<int64_t>(v.size());
  t.d = c.d + c.host.size();
  c.host.insert(c.host.end(), v.begin(), v.end());
  c.host.resize(static_cast<size_t>(t.d - c.d) + need, 0);
  return t;
}

int Engine::slices_for(TermClass cls) const {
  return slices_[cls];
}

// ---------------------------------------------------------------------------

void Engine::assign(const Ix& c, double beta, const std::vector<Factor>& terms) {
  Site& s = site();
  if (mode_ == Mode::kExec) {
    if (s.kind != 0) throw Error(GBCC_ERR_STATE, "engine: site kind mismatch");
    prof_begin(s);
    launch_gather(s.gather, run_);
    ++n_launch_;
    prof_end(s);
    return;
  }
  s.kind = 0;
  s.label = "assign " + c.t->name + "(" + c.lab + ")";
  check_ix(c);
  if (terms.empty() || terms.size() > static_cast<size_t>(kMaxTerms))
    throw Error(GBCC_ERR_STATE, "engine: assign needs 1..4 terms");
  Extents e;
  add_extents(e, c);
  for (const auto& f : terms) {
    add_extents(e, f.a);
    if (f.b.t) add_extents(e, f.b);
    for (char ch : f.a.lab)
      if (c.lab.find(ch) == std::string::npos)
        throw Error(GBCC_ERR_STATE, std::string("engine: assign index ") + ch + " not in output");
    for (char ch : f.b.lab)
      if (c.lab.find(ch) == std::string::npos)
        throw Error(GBCC_ERR_STATE, std::string("engine: assign index ") + ch + " not in output");
  }
  // split output dims into rows [0,split) and columns [split,rank)
  const int rank = c.t->rank;
  int split = rank;
  int64_t cols = 1;
  while (split > 0 && cols < 1024) {
    --split;
    cols *= c.t->dim[split];
  }
  const std::string rlab = c.lab.substr(0, split), clab = c.lab.substr(split);
  GatherArgs& g = s.gather;
  std::memset(&g, 0, sizeof(g));
  g.nterms = static_cast<int>(terms.size());
  for (size_t t = 0; t < terms.size(); ++t) {
    GatherTerm& T = g.t[t];
    gather_set_coef(T, terms[t].coef);
    T.a = terms[t].a.t->d;
    const std::vector<int64_t> hra = offsets(rlab, e, terms[t].a), hca = offsets(clab, e, terms[t].a);
    if (t == 0) g.transpose = pick_transpose(hra, hca);
    gather_set_c4(T, hca.data(), static_cast<int64_t>(hca.size()));
    T.ra = upload(hra).d;
    T.ca = upload(hca).d;
    if (terms[t].b.t) {
      g.products = 1;
      T.b = terms[t].b.t->d;
      T.rb = upload(offsets(rlab, e, terms[t].b)).d;
      T.cb = upload(offsets(clab, e, terms[t].b)).d;
    }
  }
  g.R = g.Rpad = extent_of(e, rlab);
  g.C = g.Cpad = extent_of(e, clab);
  g.out = c.t->d;
  g.ldo = g.C;
  g.beta = beta;
  gather_finish(g);
}

// ---------------------------------------------------------------------------

namespace {

bool storage_is_panel(const Ix& x, const std::string& ext) {
  // storage order = [ext labels...][K labels...]
  const int ne = static_cast<int>(ext.size());
  for (int k = 0; k < x.t->rank; ++k) {
    const bool is_ext = ext.find(x.lab[k]) != std::string::npos;
    if ((k < ne) != is_ext) return false;
  }
  return true;
}

}  // namespace

// The split panel of one operand of a tensor-core contraction: its constant
// pack, the pack cache, or a fresh pack into the workspace.
__nv_bfloat16* Engine::tc_panel(OperandPlan& op, int side) {
  if (op.constant) {
    if (!op.packed) throw Error(GBCC_ERR_STATE, "engine: constant operand not packed");
    return op.packed;
  }
  if (op.cache_reuse) {
    if (op.first_use && concurrent() && mode_ == Mode::kExec)
      GBCC_CK(cudaStreamWaitEvent(run_, op.first_use->packed_ev, 0));
    return op.cache_buf;
  }
  __nv_bfloat16* out = op.cache_first ? op.cache_buf : (side == 0 ? ws_->wbfa : ws_->wbfb);
  pack_panel(op, out);
  if (op.packed_ev && concurrent() && mode_ == Mode::kExec) GBCC_CK(cudaEventRecord(op.packed_ev, run_));
  return out;
}

// Split pack of an operand into `out`: one gather, or for fixed-point slices
// the row exponents (zeroed, then the exponent pass) and the digit pass.
void Engine::pack_panel(const OperandPlan& op, __nv_bfloat16* out) {
  GatherArgs g = op.gather;
  g.outs = out;
  if (op.fixed) {
    GBCC_CK(cudaMemsetAsync(op.rowexp, 0, static_cast<size_t>(op.rows_pad) * sizeof(unsigned), run_));
    g.fixed = 1;
    launch_gather(g, run_);
    g.fixed = 2;
    ++n_launch_;  // the exponent pass (the memset is not a kernel)
  }
  launch_gather(g, run_);
  ++n_launch_;
}

GemmTcArgs Engine::tc_args(const GemmPlan& p, TermClass cls, __nv_bfloat16* const panel[2]) const {
  GemmTcArgs t{};
  t.M = p.M;
  t.N = p.N;
  t.Mpad = p.P[0].rows_pad;
  t.Npad = round_up(p.N, p.bn);
  t.a_rows = p.P[0].rows_pad;
  t.b_rows = p.P[1].rows_pad;  // padded for every candidate tile width
  t.Kpad = p.P[0].Kpad;
  t.A = panel[0];
  t.a_slices = p.slices;
  t.B = panel[1];
  t.b_slices = p.slices;
  // a slice limit below the packed count keeps the pairs p + q < limit: the
  // split is sequential, so these are exactly the products of a
  // limit-slice split (used to measure the error of fewer slices)
  const int lim = slice_limit_[cls];
  t.npairs = 0;
  for (int q = 0; q < p.npairs; ++q) {
    if (lim > 0 && p.pa[q] + p.pb[q] >= lim) continue;
    t.pa[t.npairs] = p.pa[q];
    t.pb[t.npairs] = p.pb[q];
    ++t.npairs;
  }
  t.C = p.C;
  t.cm = p.cm;
  t.cn = p.cn;
  t.alpha = p.alpha;
  t.beta = p.beta;
  t.bn = p.bn;
  // the accumulation length of the slice count in effect (a calibration trial
  // under a slice limit measures the error the smaller plan will have)
  const int eff_slices = (lim > 0 && lim < p.slices) ? lim : p.slices;
  t.chunk = eff_slices >= 3 ? chunk_ : chunk_lo_;
  t.err = err_;
  t.ksplit = p.ksplit;
  t.kb_per_split = static_cast<int>(p.k_per_split);
  t.partial = ws_->wpart;
  t.m_major = p.m_major ? 1 : 0;
  // a slice limit makes the packed slices a superset of the used ones: one
  // pair per stage then
  t.sps = (lim > 0 && lim < p.slices) ? 1 : p.sps;
  t.group = p.group;
  return t;
}

void Engine::launch_tc(const GemmPlan& p, const GemmTcArgs& t) {
  if (!launch_gemm_tc(t, run_)) throw Error(GBCC_ERR_CUDA, "tcgen05 GEMM launch rejected (tensor map or size)");
  ++n_tc_;
  ++tc_total_;
  ++n_launch_;
  if (p.ksplit > 1) {
    launch_splitk_reduce(p.M, p.N, p.ksplit, ws_->wpart, t.Mpad, t.Npad, p.C, p.cm, p.cn, t.alpha, t.beta, run_);
    ++n_launch_;
  }
}

// FP64_TC: every weight class in one launch (gemm_multi.cu)
void Engine::launch_fixed(const GemmPlan& p, __nv_bfloat16* const panel[2]) {
  GemmMultiArgs t{};
  t.M = p.M;
  t.N = p.N;
  t.K = p.K;
  t.kblocks = p.P[0].Kpad / kTcBK;
  t.A = panel[0];
  t.a_rows = p.P[0].rows_pad;
  t.B = panel[1];
  t.b_rows = p.P[1].rows_pad;
  t.bn = p.bn;
  t.C = p.C;
  t.cm = p.cm;
  t.cn = p.cn;
  t.alpha = p.alpha;
  t.beta = p.beta;
  t.m_major = p.m_major ? 1 : 0;
  t.ksplit = p.ksplit;
  t.hb_per_split = static_cast<int>(p.k_per_split);
  t.partial = ws_->wpart;
  t.err = err_;
  const int n = launch_gemm_fixed(t, run_);
  if (n < 1) throw Error(GBCC_ERR_CUDA, "tcgen05 GEMM launch rejected (tensor map or size)");
  n_tc_ += n;
  tc_total_ += n;
  n_launch_ += n;
  if (p.ksplit > 1) {
    launch_splitk_reduce(p.M, p.N, p.ksplit, ws_->wpart, round_up(p.M, kTcBM), round_up(p.N, p.bn), p.C, p.cm, p.cn,
                         p.alpha, p.beta, run_);
    ++n_launch_;
  }
}

// Tile width and K split of every tensor-core contraction chosen by timing
// its candidates (plan-time lists) on its own operands: each candidate runs
// once untimed and `reps` times between CUDA events, the fastest is kept.
// The outputs of the timed launches are scratch (a residual recomputes them).
void Engine::autotune(int reps) {
  if (!planned_) throw Error(GBCC_ERR_STATE, "engine: autotune before PLAN");
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  GBCC_CK(cudaEventCreate(&e0));
  GBCC_CK(cudaEventCreate(&e1));
  struct Ev {
    cudaEvent_t a, b;
    ~Ev() {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  } ev{e0, e1};
  for (auto& sp : sites_) {
    if (sp->kind != 1) continue;
    GemmPlan& p = sp->plan[1];
    if (!p.use_tc || p.ncand < 2) continue;
    // shape key: SM count, class, M x N x K, slices, output orientation
    const std::string key = std::to_string(num_sms()) + ":c" + std::to_string(static_cast<int>(sp->cls)) + ":" +
                            std::to_string(p.M) + "x" + std::to_string(p.N) + "x" + std::to_string(p.K) + ":s" +
                            std::to_string(p.slices) + (p.m_major ? ":m" : ":n");
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      auto it = tune_table().find(key);
      int hit = -1;
      if (it != tune_table().end())
        for (int c = 0; c < p.ncand && hit < 0; ++c)
          if (p.cand_bn[c] == it->second.bn && p.cand_ks[c] == it->second.ksplit &&
              p.cand_kps[c] == it->second.kps && p.cand_sps[c] == it->second.sps &&
              p.cand_group[c] == it->second.group)
            hit = c;
      if (hit >= 0) {
        p.bn = p.cand_bn[hit];
        p.ksplit = p.cand_ks[hit];
        p.k_per_split = p.cand_kps[hit];
        p.sps = p.cand_sps[hit];
        p.group = p.cand_group[hit];
        continue;
      }
    }
    ws_ = &lane_ws_[sp->lane];
    __nv_bfloat16* panel[2];
    for (int side = 0; side < 2; ++side) panel[side] = tc_panel(p.P[side], side);
    float best = 0.f;
    int pick = -1;
    for (int c = 0; c < p.ncand; ++c) {
      GemmPlan q = p;
      q.bn = p.cand_bn[c];
      q.ksplit = p.cand_ks[c];
      q.k_per_split = p.cand_kps[c];
      q.sps = p.cand_sps[c];
      q.group = p.cand_group[c];
      const GemmTcArgs t = tc_args(q, sp->cls, panel);
      if (!launch_gemm_tc(t, run_)) continue;
      ++tc_total_;
      if (q.ksplit > 1)
        launch_splitk_reduce(q.M, q.N, q.ksplit, ws_->wpart, t.Mpad, t.Npad, q.C, q.cm, q.cn, q.alpha, q.beta, run_);
      GBCC_CK(cudaEventRecord(e0, stream_));
      for (int r = 0; r < reps; ++r) launch_tc(q, t);
      GBCC_CK(cudaEventRecord(e1, stream_));
      GBCC_CK(cudaEventSynchronize(e1));
      float ms = 0.f;
      GBCC_CK(cudaEventElapsedTime(&ms, e0, e1));
      if (pick < 0 || ms < best) {
        best = ms;
        pick = c;
      }
    }
    if (pick >= 0) {
      p.bn = p.cand_bn[pick];
      p.ksplit = p.cand_ks[pick];
      p.k_per_split = p.cand_kps[pick];
      p.sps = p.cand_sps[pick];
      p.group = p.cand_group[pick];
      std::lock_guard<std::mutex> lk(g_tune_mu);
      tune_table()[key] = TuneChoice{p.bn, p.ksplit, p.sps, p.group, p.k_per_split};
    }
  }
  GBCC_CK(cudaStreamSynchronize(stream_));
}

void Engine::custom(const std::function<void(cudaStream_t)>& fn, int launches) {
  Site& s = site();
  if (mode_ == Mode::kExec) {
    if (s.kind != 2) throw Error(GBCC_ERR_STATE, "engine: site kind mismatch");
    prof_begin(s);
    fn(run_);
    n_launch_ += launches;
    prof_end(s);
    return;
  }
  s.kind = 2;
  s.label = "kernels (site " + std::to_string(sites_.size() - 1) + ")";
}

void Engine::contract(const Ix& c, double beta, double alpha, const std::vector<Lin>& A,
                      const std::vector<Lin>& B, TermClass cls) {
  Site& s = site();
  if (mode_ == Mode::kExec) {
    if (s.kind != 1) throw Error(GBCC_ERR_STATE, "engine: site kind mismatch");
    GemmPlan& p = s.plan[plan_index(prec_)];
    flops_ += p.flops;
    prof_begin(s);
    if (p.use_tc) {
      __nv_bfloat16* panel[2];
      for (int side = 0; side < 2; ++side) panel[side] = tc_panel(p.P[side], side);
      prof_gemm(s);
      if (p.emu) {
        launch_fixed(p, panel);
      } else {
        const GemmTcArgs t = tc_args(p, cls, panel);
        launch_tc(p, t);
      }
    } else if (p.small) {
      GemmSmallArgs g = p.sg;
      g.partial = ws_->wpart;
      g.count = ws_->wcount;
      prof_gemm(s);
      launch_gemm_small(g, run_);
      ++n_launch_;
    } else {
      const double* panel[2];
      for (int side = 0; side < 2; ++side) {
        OperandPlan& op = p.P[side];
        if (op.direct) {
          panel[side] = op.dptr;
        } else if (op.inplace) {
          panel[side] = op.gather.t[0].a;
        } else {
          double* w = side == 0 ? ws_->w64a : ws_->w64b;
          GatherArgs g = op.gather;
          g.out = w;
          launch_gather(g, run_);
          ++n_launch_;
          panel[side] = w;
        }
      }
      GemmF64Args f{};
      f.M = p.M;
      f.N = p.N;
      f.K = p.K;
      f.A = panel[0];
      f.lda = p.P[0].direct ? p.P[0].ld : p.K;
      f.B = panel[1];
      f.ldb = p.P[1].direct ? p.P[1].ld : p.K;
      f.C = p.C;
      f.cm = p.cm;
      f.cn = p.cn;
      f.alpha = p.alpha;
      f.beta = p.beta;
      f.ksplit = p.ksplit;
      f.k_per_split = p.k_per_split;
      f.partial = ws_->wpart;
      f.m_major = p.m_major ? 1 : 0;
      if (p.P[0].inplace) {
        f.a_ra = p.P[0].gather.t[0].ra;
        f.a_ca = p.P[0].gather.t[0].ca;
        f.lda = 0;
      }
      prof_gemm(s);
      if (p.smallk) {
        if (!launch_gemm_smallk(f, run_)) throw Error(GBCC_ERR_STATE, "engine: in-place small-K operand off the stream kernel");
        ++n_launch_;
      } else {
        launch_gemm_f64(f, run_);
        n_launch_ += p.ksplit > 1 ? 2 : 1;
      }
    }
    prof_end(s);
    return;
  }

  // ---------------- PLAN ----------------
  s.kind = 1;
  s.cls = cls;
  check_ix(c);
  static const char* const kClassName[3] = {"ladder", "ring", "other"};
  s.label = "contract " + c.t->name + "(" + c.lab + ") <- " + A.at(0).x.t->name + "(" + A.at(0).x.lab + ") " +
            B.at(0).x.t->name + "(" + B.at(0).x.lab + ") [" + kClassName[static_cast<int>(cls)] + "]";
  if (A.empty() || B.empty() || A.size() > static_cast<size_t>(kMaxTerms) ||
      B.size() > static_cast<size_t>(kMaxTerms))
    throw Error(GBCC_ERR_STATE, "engine: contract needs 1..4 terms per operand");
  Extents e;
  add_extents(e, c);
  for (const auto* ops : {&A, &B})
    for (const auto& l : *ops) {
      add_extents(e, l.x);
      if (l.y.t) add_extents(e, l.y);
    }
  // the first term of an operand is a single factor carrying all its indices
  auto term_labels = [](const Lin& l) { return l.y.t ? l.x.lab + l.y.lab : l.x.lab; };
  if (A[0].y.t || B[0].y.t) throw Error(GBCC_ERR_STATE, "engine: the first operand term must be one factor");
  for (const auto& l : A)
    if (!same_set(term_labels(l), A[0].x.lab)) throw Error(GBCC_ERR_STATE, "engine: A terms differ in indices");
  for (const auto& l : B)
    if (!same_set(term_labels(l), B[0].x.lab)) throw Error(GBCC_ERR_STATE, "engine: B terms differ in indices");
  const std::string la = A[0].x.lab, lb = B[0].x.lab;
  const std::string kset = set_and(la, lb);
  const std::string aext = set_minus(la, kset), bext = set_minus(lb, kset);
  for (char ch : kset)
    if (c.lab.find(ch) != std::string::npos)
      throw Error(GBCC_ERR_STATE, "engine: Hadamard indices are not supported");
  if (!same_set(aext + bext, c.lab))
    throw Error(GBCC_ERR_STATE, "engine: output indices must be exactly the external ones (" + c.lab + ")");
  const int64_t rowsA = extent_of(e, aext), rowsB = extent_of(e, bext), K = extent_of(e, kset);
  bool constA = true, constB = true;
  for (const auto& l : A) constA = constA && l.x.t->constant && (!l.y.t || l.y.t->constant);
  for (const auto& l : B) constB = constB && l.x.t->constant && (!l.y.t || l.y.t->constant);
  const double flops = 2.0 * static_cast<double>(rowsA) * rowsB * K;

  for (int pm = 0; pm < (emu_ ? 3 : 2); ++pm) {
    GemmPlan& p = s.plan[pm];
    p = GemmPlan{};
    p.flops = flops;
    const bool emu = pm == 2;
    p.sg.M = std::max(rowsA, rowsB);
    p.sg.N = std::min(rowsA, rowsB);
    p.sg.K = K;
    p.small = plan_gemm_small(p.sg) <= (pm == 0 ? kSmallUs : (emu ? kSmallUsFixed : kSmallUsMixed));
    if (trial_ && pm == 1) p.small = flops < kTrialFlops;
    int slices = p.small || pm == 0 ? 0 : (emu ? kFixedSlices : slices_for(cls));
    // a short contraction into a large output is memory-bound: CUDA cores
    // (measured faster for N > 32; the tensor-core kernel wins below).  The
    // FP64-grade plan keeps such contractions on the FP64 kernel.
    if (slices > 0 && !emu && K <= kSmallK && std::min(rowsA, rowsB) >= 32 &&
        static_cast<double>(rowsA) * static_cast<double>(rowsB) >= 1048576.0) {
      slices = 0;
      p.smallk = true;
    }
    // the larger operand on M: it is then re-read once per N tile, and N
    // tiles are up to 256 wide (less padding alone, with the large operand on
    // N, measured slower: more L2 re-reads of it)
    p.a_is_first = rowsA >= rowsB;
    const std::vector<Lin>& Ms = p.a_is_first ? A : B;
    const std::vector<Lin>& Ns = p.a_is_first ? B : A;
    const std::string mext = p.a_is_first ? aext : bext;
    const std::string next = p.a_is_first ? bext : aext;
    const bool constM = p.a_is_first ? constA : constB;
    const bool constN = p.a_is_first ? constB : constA;
    p.M = extent_of(e, mext);
    p.N = extent_of(e, next);
    p.K = K;
    p.beta = beta;
    p.C = c.t->d;
    p.use_tc = slices > 0;
    OperandPlan& PM = p.P[0];
    OperandPlan& PN = p.P[1];
    PM.terms = Ms;
    PN.terms = Ns;
    PM.constant = constM;
    PN.constant = constN;
    PM.rows = p.M;
    PN.rows = p.N;
    PM.K = PN.K = K;
    PM.ext = order_by(mext, c.lab);
    PN.ext = order_by(next, c.lab);
    // contracted-index order
    const Ix& bigM = Ms[0].x;
    const Ix& bigN = Ns[0].x;
    if (p.small) {
      const Ix& ref = bigM.t->size() >= bigN.t->size() ? bigM : bigN;
      PM.kord = order_by(kset, ref.lab);
    } else if (!p.use_tc) {
      const bool dM = Ms.size() == 1 && !Ms[0].y.t && storage_is_panel(bigM, mext);
      const bool dN = Ns.size() == 1 && !Ns[0].y.t && storage_is_panel(bigN, next);
      if (dM && (!dN || bigM.t->size() >= bigN.t->size())) {
        PM.direct = true;
        PM.ext = order_by(mext, bigM.lab);
        PM.kord = order_by(kset, bigM.lab);
        if (dN && order_by(kset, bigN.lab) == PM.kord) {
          PN.direct = true;
          PN.ext = order_by(next, bigN.lab);
        }
      } else if (dN) {
        PN.direct = true;
        PN.ext = order_by(next, bigN.lab);
        PM.kord = order_by(kset, bigN.lab);
      } else {
        const Ix& ref = bigM.t->size() >= bigN.t->size() ? bigM : bigN;
        PM.kord = order_by(kset, ref.lab);
      }
    } else {
      // pack reads are cheapest along the storage order of the per-iteration operand;
      // a vector's order is free and lets a contraction name the order of a pack
      // that another one makes
      const Ix* ref = nullptr;
      if (!constM && !constN && p.N == 1) ref = &bigN;
      else if (!constM && !constN) ref = bigM.t->size() >= bigN.t->size() ? &bigM : &bigN;
      else if (!constM) ref = &bigM;
      else if (!constN) ref = &bigN;
      else ref = &bigM;
      PM.kord = order_by(kset, ref->lab);
    }
    PN.kord = PM.kord;
    double coef_direct = 1.0;
    for (int side = 0; side < 2; ++side) {
      OperandPlan& op = p.P[side];
      if (op.direct) {
        op.dptr = op.terms[0].x.t->d;
        op.ld = op.K;
        coef_direct *= op.terms[0].coef;
        continue;
      }
      GatherArgs& g = op.gather;
      std::memset(&g, 0, sizeof(g));
      g.nterms = static_cast<int>(op.terms.size());
      // a single one-factor term packs as a plain copy; its coefficient scales alpha
      const bool single = op.terms.size() == 1 && !op.terms[0].y.t;
      if (single) coef_direct *= op.terms[0].coef;
      g.plain = single ? 1 : 0;
      for (size_t t = 0; t < op.terms.size(); ++t) {
        gather_set_coef(g.t[t], single ? 1.0 : op.terms[t].coef);
        g.t[t].a = op.terms[t].x.t->d;
        const std::vector<int64_t> hra = offsets(op.ext, e, op.terms[t].x), hca = offsets(op.kord, e, op.terms[t].x);
        if (t == 0) g.transpose = pick_transpose(hra, hca);
        gather_set_c4(g.t[t], hca.data(), static_cast<int64_t>(hca.size()));
        g.t[t].ra = upload(hra).d;
        g.t[t].ca = upload(hca).d;
        if (op.terms[t].y.t) {
          g.products = 1;
          g.t[t].b = op.terms[t].y.t->d;
          g.t[t].rb = upload(offsets(op.ext, e, op.terms[t].y)).d;
          g.t[t].cb = upload(offsets(op.kord, e, op.terms[t].y)).d;
        }
      }
      gather_finish(g);
      g.R = op.rows;
      g.C = op.K;
      if (!p.use_tc && !p.small) {
        g.Rpad = op.rows;
        g.Cpad = op.K;
        g.ldo = op.K;
        g.beta = 0.0;
        size_t need = static_cast<size_t>(op.rows * op.K);
        if (side == 0) ws_->n64a = std::max(ws_->n64a, need);
        else ws_->n64b = std::max(ws_->n64b, need);
      }
    }
    p.alpha = alpha * coef_direct;
    {
      Ix cx = c;
      const std::vector<int64_t> hm = offsets(p.P[0].ext, e, cx), hn = offsets(p.P[1].ext, e, cx);
      // epilogue lane direction: along M when C is unit-stride in M but not in N
      const bool m_unit = hm.size() > 1 && hm[1] - hm[0] == 1;
      const bool n_unit = hn.size() > 1 && hn[1] - hn[0] == 1;
      p.m_major = m_unit && !n_unit;
      p.cm = upload(hm).d;
      p.cn = upload(hn).d;
    }
    // a single-factor M operand contiguous along M (its pack would transpose)
    // is read in place by the stream kernel: no FP64 panel written and read back
    if (p.smallk && !p.P[0].direct && p.P[0].gather.plain && p.P[0].gather.transpose &&
        smallk_streams(p.N, K, p.m_major))
      p.P[0].inplace = true;
    if (p.small) {
      GemmSmallArgs& g = p.sg;
      g.a = p.P[0].gather;
      g.b = p.P[1].gather;
      g.C = p.C;
      g.cm = p.cm;
      g.cn = p.cn;
      g.alpha = p.alpha;
      g.beta = p.beta;
      p.ksplit = g.ksplit;
      ws_->npart = std::max(ws_->npart, g.partial_elems);
      if (g.ksplit > 1) ws_->ncount = std::max(ws_->ncount, static_cast<size_t>(g.tiles));
    } else if (!p.use_tc && !p.smallk) {
      // fewer 64 x 64 output tiles than two per SM: split K over blocks (one SM
      // runs FP64 at ~1/150 of the GPU's already low FP64 rate, so even a
      // 1 MFLOP contraction is slow on a single block)
      const int64_t tiles = ((p.M + 63) / 64) * ((p.N + 63) / 64);
      const int64_t sms = num_sms();
      if (tiles < 2 * sms && K >= 32) {
        int64_t ks = std::min<int64_t>((2 * sms + tiles - 1) / tiles, K / 16);
        if (ks > 1) {
          int64_t kps = (K + ks - 1) / ks;
          kps = (kps + 15) / 16 * 16;
          ks = (K + kps - 1) / kps;
          p.ksplit = static_cast<int>(ks);
          p.k_per_split = kps;
          ws_->npart = std::max(ws_->npart, static_cast<size_t>(ks * p.M * p.N));
        }
      }
    }
    if (p.use_tc) {
      p.slices = slices;
      p.emu = emu;
      // the ladder and ring contractions take the faster 192/256-wide tiles
      // (FP64_TC has its own kernel and tile: gemm_multi_bn)
      const bool wide = !emu && (cls == kClassLadder || cls == kClassRing);
      int bns[4];
      int nbn = 1;
      if (emu) bns[0] = gemm_multi_bn(p.N);
      else nbn = gemm_tc_bn_candidates(p.N, wide, bns);
      int64_t npanel = 0;  // N-side panel rows: room for every candidate tile width
      for (int c = 0; c < nbn; ++c) npanel = std::max<int64_t>(npanel, round_up(p.N, bns[c]));
      p.npairs = 0;
      if (emu) {
        p.npairs = slices * (slices + 1) / 2;
      } else {
        for (int a = 0; a < slices; ++a)
          for (int b = 0; b < slices; ++b)
            if (a + b < slices) {
              p.pa[p.npairs] = a;
              p.pb[p.npairs] = b;
              ++p.npairs;
            }
      }
      const int64_t Kpad = round_up(std::max<int64_t>(K, 1), kTcBK);
      for (int side = 0; side < 2; ++side) {
        OperandPlan& op = p.P[side];
        op.lane = lane_;
        op.slices = slices;
        op.Kpad = Kpad;
        // (the FP64_TC kernel's tensor maps end at the last row)
        op.rows_pad = emu ? op.rows : (side == 0 ? round_up(op.rows, kTcBM) : npanel);
        if (!emu && side == 0 && p.N == 1) {
          // the matrix of a vector product is padded as on the N side of a wide
          // product, whose pack it can then share
          int wbns[4];
          const int nw = gemm_tc_bn_candidates(op.rows, true, wbns);
          int64_t wide_rows = op.rows_pad;
          for (int c = 0; c < nw; ++c) wide_rows = std::max(wide_rows, round_up(op.rows, wbns[c]));
          op.rows_pad = round_up(wide_rows, kTcBM);
        }
        GatherArgs& g = op.gather;
        g.Rpad = op.rows_pad;
        g.Cpad = Kpad;
        g.ldo = Kpad;
        g.out = nullptr;
        g.nslices = slices;
        g.slice_stride = op.rows_pad * Kpad;
        if (emu) {
          op.fixed = true;
          op.rowexp = static_cast<unsigned*>(dev_alloc(static_cast<size_t>(op.rows_pad) * sizeof(unsigned)));
          owned_.push_back(op.rowexp);
          bytes_ += static_cast<size_t>(op.rows_pad) * sizeof(unsigned);
          g.rowexp = op.rowexp;
          g.fixed = 2;
        }
        const size_t need = static_cast<size_t>(slices) * op.rows_pad * Kpad;
        if (!op.constant) {
          bool frozen = true;
          // labels by their place among rows and columns, so that packs of the same
          // elements match whatever their contractions call the indices
          auto place = [&](const std::string& lab) {
            const std::string order = op.ext + op.kord;
            std::string out;
            for (char ch : lab) out += static_cast<char>('A' + order.find(ch));
            return out;
          };
          std::string sig;
          for (const auto& l : op.terms) {
            frozen = frozen && frozen_.count(l.x.t) > 0 && (!l.y.t || frozen_.count(l.y.t) > 0);
            // a single one-factor term is packed unscaled (plain copy)
            const double coef = (op.terms.size() == 1 && !l.y.t) ? 1.0 : l.coef;
            sig += l.x.t->name + "(" + place(l.x.lab) + ")";
            if (l.y.t) sig += l.y.t->name + "(" + place(l.y.lab) + ")";
            sig += "*" + std::to_string(coef) + ";";
          }
          if (frozen) {
            op.sig = sig + std::to_string(op.ext.size()) + "|" + (emu ? "fixed" : "float") + std::to_string(slices) + "|" +
                     std::to_string(op.rows_pad) + "|" + std::to_string(Kpad);
            op.pack_elems = need;
            pack_uses_[op.sig].push_back(&op);
          }
        }
        if (op.constant) {
          op.pack_elems = need;  // allocated and packed by prepack()
        } else if (side == 0) {
          ws_->nbfa = std::max(ws_->nbfa, need);
        } else {
          ws_->nbfb = std::max(ws_->nbfb, need);
        }
      }
      // fewer output tiles than SMs and a long K: split K over CTAs.  The
      // candidates: every tile width with that split, and unsplit where it splits
      const int64_t kblocks = Kpad / kTcBK;
      const int64_t sms = num_sms();
      p.ncand = 0;
      if (emu) {
        // fewer tiles than SMs: splits of at least 10 stages (two chunks), as
        // many as fill the chip
        p.bn = bns[0];
        const int64_t hbs = (K + 31) / 32;
        const int64_t tiles = ((p.M + kTcBM - 1) / kTcBM) * ((p.N + p.bn - 1) / p.bn);
        int64_t ks = tiles < sms ? std::min<int64_t>(sms / tiles, hbs / 10) : 1;
        if (ks > 1) {
          p.k_per_split = (hbs + ks - 1) / ks;
          ks = (hbs + p.k_per_split - 1) / p.k_per_split;
        }
        p.ksplit = static_cast<int>(std::max<int64_t>(ks, 1));
        if (p.ksplit > 1)
          ws_->npart = std::max(ws_->npart, static_cast<size_t>(ks * round_up(p.M, kTcBM) * round_up(p.N, p.bn)));
        continue;
      }
      for (int c = 0; c < nbn; ++c) {
        const int64_t npad = round_up(p.N, bns[c]);
        const int64_t tiles = (p.P[0].rows_pad / kTcBM) * (npad / bns[c]);
        int64_t ks = 1, kbps = 0;
        if (tiles < sms && kblocks >= 16) {
          ks = std::min<int64_t>((sms + tiles - 1) / tiles, kblocks / 8);
        } else if (tiles < 3 * sms && kblocks >= 64) {
          // one to three waves: a split that fills the last wave better (the
          // Giabc pair products at o = 32, v = 320: 240 tiles on 152 SMs fill
          // 79 % of two waves, split in three 95 % of five)
          auto fill = [&](int64_t k) {
            const int64_t n = tiles * k;
            return static_cast<double>(n) / static_cast<double>((n + sms - 1) / sms * sms);
          };
          double best = fill(1) + 0.05;
          for (int64_t k = 2; k <= 4 && kblocks / k >= 16; ++k)
            if (fill(k) > best) {
              best = fill(k);
              ks = k;
            }
        }
        if (ks > 1) {
          kbps = (kblocks + ks - 1) / ks;
          ks = (kblocks + kbps - 1) / kbps;
        } else {
          ks = 1;
        }
        if (ks > 1) ws_->npart = std::max(ws_->npart, static_cast<size_t>(ks * p.P[0].rows_pad * npad));
        // both slices of a k-block per stage: two slices, tiles up to 192 wide;
        // every slice per stage on CTA pairs: 256 x 256 tiles, where the padding
        // of M to 256 is small
        const int nsps = ((slices == 2 && bns[c] >= 64 && bns[c] <= 192) || (slices > 1 && bns[c] == 256 && p.M >= 512))
                             ? 2
                             : 1;
        // bands of 8 M tiles: many N tiles per row and enough rows
        const bool banded = npad / bns[c] >= 8 && p.P[0].rows_pad / kTcBM >= 16;
        for (int sp = 1; sp <= nsps; ++sp) {
          for (int split = 0; split < (ks > 1 ? 2 : 1); ++split) {
            for (int band = 0; band < (banded && (split == 1 || ks == 1) ? 2 : 1); ++band) {
              if (p.ncand >= GemmPlan::kMaxCand) break;
              p.cand_bn[p.ncand] = bns[c];
              p.cand_ks[p.ncand] = split == 0 ? static_cast<int>(ks) : 1;
              p.cand_kps[p.ncand] = split == 0 ? kbps : 0;
              p.cand_sps[p.ncand] = sp;
              p.cand_group[p.ncand] = band ? 8 : 1;
              ++p.ncand;
            }
          }
        }
      }
      // the heuristic choice: the first candidate
      p.bn = p.cand_bn[0];
      p.ksplit = p.cand_ks[0];
      p.k_per_split = p.cand_kps[0];
      p.sps = p.cand_sps[0];
      p.group = p.cand_group[0];
    }
  }
}

void Engine::finalize() {
  if (!planned_) throw Error(GBCC_ERR_STATE, "engine: finalize before PLAN");
  for (const TableChunk& c : tables_)
    GBCC_CK(cudaMemcpy(c.d, c.host.data(), c.host.size() * sizeof(int64_t), cudaMemcpyHostToDevice));
  tables_.clear();
  const int mode = g_lanes_mode.load();
  if (nlanes_ > 1 && (mode < 0 ? !lanes_fit() : mode == 0)) merge_lanes();
  alloc_workspaces();
  // packs shared by several contractions of a residual get their own buffer
  for (auto& kv : pack_uses_) {
    if (kv.second.size() < 2) continue;
    OperandPlan* first = kv.second.front();
    if (!first->cache_buf) {
      first->cache_buf = static_cast<__nv_bfloat16*>(dev_alloc(first->pack_elems * sizeof(__nv_bfloat16)));
      owned_.push_back(first->cache_buf);
      bytes_ += first->pack_elems * sizeof(__nv_bfloat16);
    }
    first->cache_first = true;
    for (size_t i = 1; i < kv.second.size(); ++i) {
      kv.second[i]->cache_reuse = true;
      kv.second[i]->cache_buf = first->cache_buf;
      if (kv.second[i]->lane != first->lane) {
        kv.second[i]->first_use = first;
        if (!first->packed_ev) GBCC_CK(cudaEventCreateWithFlags(&first->packed_ev, cudaEventDisableTiming));
      }
    }
  }
  packed_[0] = packed_[1] = packed_[2] = false;
}

void Engine::prepack(int precision) {
  const int pi = plan_index(precision);
  if (!planned_) throw Error(GBCC_ERR_STATE, "engine: prepack before PLAN");
  if (!scratch_) alloc_workspaces();  // given up by release_scratch()
  if (pi == 0 || packed_[pi]) return;
  if (pi == 2 && !emu_) throw Error(GBCC_ERR_STATE, "engine: no FP64_TC plan");
  for (auto& sp : sites_) {
    if (sp->kind != 1) continue;
    GemmPlan& p = sp->plan[pi];
    if (!p.use_tc) continue;
    for (int side = 0; side < 2; ++side) {
      OperandPlan& op = p.P[side];
      if (!op.constant) continue;
      if (!op.packed) {
        op.packed = static_cast<__nv_bfloat16*>(dev_alloc(op.pack_elems * sizeof(__nv_bfloat16)));
        owned_.push_back(op.packed);
        bytes_ += op.pack_elems * sizeof(__nv_bfloat16);
      }
      pack_panel(op, op.packed);
    }
  }
  GBCC_CK(cudaGetLastError());
  packed_[pi] = true;
}

}  // namespace gbcc

extern "C" int gbcc_testing_lanes_mode(int mode) {
  if (mode < -1 || mode > 1) return GBCC_ERR_INVALID_ARG;
  gbcc::g_lanes_mode.store(mode);
  return GBCC_OK;
}

extern "C" int gbcc_testing_free_bytes(int64_t bytes) {
  if (bytes < -1) return GBCC_ERR_INVALID_ARG;
  gbcc::g_free_bytes.store(bytes);
  return GBCC_OK;
}

extern "C" int gbcc_testing_fail_site(int64_t site) {
  if (site < -1) return GBCC_ERR_INVALID_ARG;
  gbcc::g_fail_site.store(site);
  return GBCC_OK;
}

extern "C" int gbcc_testing_fail_alloc(int64_t after, int64_t* count) {
  if (after < -1) return GBCC_ERR_INVALID_ARG;
  if (count) *count = gbcc::g_alloc_count.load();
  gbcc::g_fail_alloc_after.store(after);
  return GBCC_OK;
}
