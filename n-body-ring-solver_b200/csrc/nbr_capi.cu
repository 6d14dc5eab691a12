// nbr_capi.cu -- the C ABI (include/nbr.h): contexts, device state, the
// leapfrog launch sequences and their CUDA-graph capture, diagnostics and the
// autotune cache.  Host code; the kernels live in nbr_kernels.cu and
// nbr_batch.cu.
#include "nbr.h"
#include "nbr_ctx.h"
#include "nbr_device.cuh"
#include "nbr_kernels.cuh"

#include <dlfcn.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <mutex>
#include <new>
#include <sstream>
#include <string>
#include <vector>

using namespace nbr;

namespace nbr {

thread_local std::string t_err;

int fail(nbr_ctx* c, int code, const std::string& msg) {
  if (c) c->err = msg;
  t_err = msg;
  return code;
}

int cuda_fail(nbr_ctx* c, cudaError_t e, const char* where) {
  std::string m = std::string(where) + ": " + cudaGetErrorString(e);
  cudaGetLastError();  // clear a sticky launch error where possible
  return fail(c, e == cudaErrorMemoryAllocation ? NBR_ERR_NO_MEMORY : NBR_ERR_CUDA, m);
}

void dfree(void* p) {
  if (p) cudaFree(p);
}

// Allocates and zeroes device memory.  cudaMemset runs on the legacy default
// stream, which does not order with the contexts' non-blocking streams, so the
// zeroing is completed here before any kernel can see the memory (a counter
// array zeroed late once left split-arrival counters non-zero).  Allocation is
// rare (buffers only grow), so the device-wide wait costs nothing in a step.
//
// Test hook (fault injection on the host, no GPU fault): with
// NBR_TEST_FAIL_ALLOC=k set, the k-th allocation counted from the moment the
// variable took its current value reports cudaErrorMemoryAllocation instead of
// allocating.
cudaError_t dalloc(void** p, size_t bytes) {
  *p = nullptr;
  if (bytes == 0) bytes = 256;
  {
    static std::mutex mu;
    static std::string armed;
    static long count = 0;
    const char* v = std::getenv("NBR_TEST_FAIL_ALLOC");
    std::lock_guard<std::mutex> lock(mu);
    if (v && *v) {
      if (armed != v) {
        armed = v;
        count = 0;
      }
      if (++count == std::atol(v)) return cudaErrorMemoryAllocation;
    } else {
      armed.clear();
    }
  }
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) return e;
  e = cudaMemset(*p, 0, bytes);
  if (e != cudaSuccess) return e;
  return cudaDeviceSynchronize();
}

bool RunKey::operator==(const RunKey& o) const {
  if (precision != o.precision || scheme != o.scheme || order != o.order || dt != o.dt ||
      G != o.G || eps2 != o.eps2 || steps != o.steps || n != o.n || cap != o.cap ||
      fsal != o.fsal || cur != o.cur || rec_ok[0] != o.rec_ok[0] || rec_ok[1] != o.rec_ok[1] ||
      cfg.ni != o.cfg.ni || cfg.warps != o.cfg.warps || cfg.split != o.cfg.split ||
      cfg.tile != o.cfg.tile || cfg.unroll != o.cfg.unroll ||
      wait_ns != o.wait_ns || skip_tile != o.skip_tile || strips != o.strips || bands != o.bands)
    return false;
  for (int i = 0; i < 7; ++i)
    if (ptr[i] != o.ptr[i]) return false;
  return true;
}

void RunGraph::release() {
  if (exec) cudaGraphExecDestroy(exec);
  *this = RunGraph();
}

bool give_back(nbr_ctx* c) {
  bool any = c->bat.d_flat != nullptr;
  dfree(c->bat.d_flat);
  c->bat.d_flat = nullptr;
  for (RunGraph& g : c->run_graph) {
    any |= g.exec != nullptr;
    g.release();
  }
  return any;
}

bool finite_array(const double* a, size_t n) {
  bool ok = true;
  for (size_t i = 0; i < n; ++i) ok &= std::isfinite(a[i]);
  return ok;
}

void SysState::release() {
  for (int b = 0; b < 2; ++b) {
    for (int d = 0; d < 3; ++d) dfree(pos[b][d]);
    dfree(rec[b]);
    dfree(org[b]);
  }
  for (int d = 0; d < 3; ++d) { dfree(vel[d]); dfree(acc[d]); }
  dfree(mass);
  *this = SysState();
}

cudaError_t SysState::reserve(size_t n_) {
  const size_t np = ((n_ + 1023) / 1024) * 1024;
  // Per-particle arrays carry kRangeSlack zeroed entries past n_pad: a force
  // launch over a receiver range [i0, i0 + count) reads receivers in whole
  // chunks (up to 1023 past the range end), and an all-gather of equal
  // 128-aligned shards may write up to 8 x 127 entries past n.
  const size_t na = np + kRangeSlack;
  if (np <= cap) {
    n = n_;
    n_pad = np;
    ntiles = (int)((n_ + kTile - 1) / kTile);
    return cudaSuccess;
  }
  release();
  cudaError_t e = cudaSuccess;
  auto A = [&](void** p, size_t bytes) {
    if (e == cudaSuccess) e = dalloc(p, bytes);
  };
  for (int b = 0; b < 2; ++b) {
    for (int d = 0; d < 3; ++d) A((void**)&pos[b][d], na * sizeof(double));
    A((void**)&rec[b], np * 3 * sizeof(float4));
    A((void**)&org[b], (np / kTile) * sizeof(double4));
  }
  for (int d = 0; d < 3; ++d) {
    A((void**)&vel[d], na * sizeof(double));
    A((void**)&acc[d], na * sizeof(double));
  }
  A((void**)&mass, na * sizeof(double));
  if (e != cudaSuccess) {
    release();
    return e;
  }
  cap = np;
  n = n_;
  n_pad = np;
  ntiles = (int)((n_ + kTile - 1) / kTile);
  return cudaSuccess;
}

// Zeroes the padding of every per-particle array (entries n .. cap +
// kRangeSlack - 1), so padding particles have zero mass and sit at the origin
// of both buffers.
cudaError_t SysState::clear_padding(cudaStream_t st) {
  const size_t tail = cap + kRangeSlack - n;
  cudaError_t e = cudaSuccess;
  auto Z = [&](double* p) {
    if (e == cudaSuccess && tail) e = cudaMemsetAsync(p + n, 0, tail * sizeof(double), st);
  };
  for (int b = 0; b < 2; ++b)
    for (int d = 0; d < 3; ++d) Z(pos[b][d]);
  for (int d = 0; d < 3; ++d) { Z(vel[d]); Z(acc[d]); }
  Z(mass);
  return e;
}

cudaError_t Scratch::need_part(size_t doubles) {
  if (doubles <= part_cap) return cudaSuccess;
  dfree(part);
  part = nullptr;
  part_cap = 0;
  cudaError_t e = dalloc((void**)&part, doubles * sizeof(double));
  if (e == cudaSuccess) part_cap = doubles;
  return e;
}
cudaError_t Scratch::need_counters(size_t count) {
  if (count <= cnt_cap) return cudaSuccess;
  dfree(cnt);
  cnt = nullptr;
  cnt_cap = 0;
  cudaError_t e = dalloc((void**)&cnt, count * sizeof(unsigned));
  if (e == cudaSuccess) cnt_cap = count;
  return e;
}
cudaError_t Scratch::need_red(size_t doubles) {
  if (doubles <= red_cap) return cudaSuccess;
  dfree(red);
  red = nullptr;
  red_cap = 0;
  cudaError_t e = dalloc((void**)&red, doubles * sizeof(double));
  if (e == cudaSuccess) red_cap = doubles;
  return e;
}
void Scratch::release() {
  dfree(part);
  dfree(cnt);
  dfree(red);
  *this = Scratch();
}

// --------------------------------------------------------------- tuning ----
namespace {

std::mutex g_tune_mu;
std::map<std::string, ForceConfig>* g_tune = nullptr;
std::string g_tune_path;

std::string lib_dir() {
  Dl_info info;
  if (dladdr((void*)&nbr_version, &info) && info.dli_fname) {
    std::string p = info.dli_fname;
    size_t s = p.find_last_of('/');
    if (s != std::string::npos) return p.substr(0, s);
  }
  return ".";
}

// Sizes by powers of two.  Where the Newton-3 default begins inside one (at 4097)
// its part of it has a key of its own (":n3"): a result for a system below it,
// or an entry from before the default began there, says nothing about the
// sizes above.
std::string tune_key(int precision, long long n_i, int ntiles, bool excl) {
  int bucket = 0;
  while ((1LL << (bucket + 1)) <= n_i) ++bucket;
  int jb = 0;
  while ((1LL << (jb + 1)) <= (long long)ntiles) ++jb;
  std::ostringstream k;
  k << (precision == kFP32C ? "fp32c" : "fp64") << ":i" << bucket << ":j" << jb
    << (excl ? ":e0" : "") << (n_i >= kN3MinN && (1LL << bucket) < kN3MinN ? ":n3" : "");
  return k.str();
}

// The cache is a flat JSON object {"key": [ni, warps, split, tile, unroll], ...}
// (entries with three numbers leave tile and unroll at their defaults).
void load_tune_locked() {
  if (g_tune) return;
  g_tune = new std::map<std::string, ForceConfig>();
  const char* env = std::getenv("NBR_TUNE_CACHE");
  g_tune_path = env && *env ? env : lib_dir() + "/nbr_tune_cache.json";
  std::ifstream f(g_tune_path);
  if (!f) return;
  std::stringstream ss;
  ss << f.rdbuf();
  std::string s = ss.str();
  size_t p = 0;
  while ((p = s.find('"', p)) != std::string::npos) {
    size_t q = s.find('"', p + 1);
    if (q == std::string::npos) break;
    std::string key = s.substr(p + 1, q - p - 1);
    size_t lb = s.find('[', q), rb = s.find(']', q);
    if (lb == std::string::npos || rb == std::string::npos) break;
    ForceConfig c{0, 0, 0};
    const int got = std::sscanf(s.c_str() + lb + 1, "%d , %d , %d , %d , %d", &c.ni, &c.warps,
                                &c.split, &c.tile, &c.unroll);
    const int prec = key.compare(0, 5, "fp32c") == 0 ? kFP32C : kFP64;
    if (got < 5) c.tile = c.unroll = 0;
    if (got >= 3 && force_config_supported(prec, c)) (*g_tune)[key] = c;
    p = rb + 1;
  }
}

void save_tune_locked() {
  std::ofstream f(g_tune_path);
  if (!f) return;
  f << "{\n";
  size_t k = 0;
  for (auto& kv : *g_tune) {
    f << "  \"" << kv.first << "\": [" << kv.second.ni << ", " << kv.second.warps << ", "
      << kv.second.split << ", " << kv.second.tile << ", " << kv.second.unroll << "]"
      << (++k < g_tune->size() ? ",\n" : "\n");
  }
  f << "}\n";
}

}  // namespace

bool tune_get(const std::string& key, ForceConfig* out) {
  std::lock_guard<std::mutex> g(g_tune_mu);
  load_tune_locked();
  auto it = g_tune->find(key);
  if (it == g_tune->end()) return false;
  *out = it->second;
  return true;
}

void tune_put(const std::string& key, const ForceConfig& cfg) {
  std::lock_guard<std::mutex> g(g_tune_mu);
  load_tune_locked();
  (*g_tune)[key] = cfg;
  save_tune_locked();
}

// Heuristic split.  Finer (chunk, split) units balance the SMs better; a B200
// sweep (N = 32768 .. 1048576) found throughput rising with the split up to
// 8 tiles (1024 sources) per split range and at most 64 splits.  Small systems
// get at least ~4 waves of resident CTAs, down to 2 tiles per range.
int auto_split(int precision, double eps2, const ForceConfig& c, long long n_i, int ntiles,
               int sms) {
  const long long chunk = force_chunk(c);
  const long long chunks = (n_i + chunk - 1) / chunk;
  int per_sm = force_blocks_per_sm(precision, eps2, c);
  if (per_sm < 1) per_sm = 1;
  const long long slots = (long long)sms * per_sm;
  const long long waves4 = (4 * slots + chunks - 1) / chunks;
  long long s = std::max<long long>(ntiles / 8, std::min<long long>(ntiles / 2, waves4));
  s = std::max<long long>(1, std::min<long long>(s, 64));
  return (int)s;
}

// whole: an evaluation of the whole system, which the Newton-3 strips can
// take; receiver ranges and separate receiver and source sets cannot.
ForceConfig choose_config(nbr_ctx* c, int precision, double eps2, long long n_i, int ntiles,
                          bool whole = true) {
  ForceConfig cfg = c->override_cfg[precision];
  if (cfg.ni == kPersistNI) cfg = ForceConfig{0, 0, 0};  // a run-level choice: evaluations use the default
  if (cfg.ni == 0) {
    std::lock_guard<std::mutex> g(g_tune_mu);
    load_tune_locked();
    auto it = g_tune->find(tune_key(precision, n_i, ntiles, eps2 == 0.0));
    // Defaults from a configuration sweep on B200 (N = 32768 .. 262144):
    // FP32C is FMA-pipe bound and gains from 4 receiver pairs per thread;
    // FP64 has twice the registers per receiver and prefers 4 per thread.
    ForceConfig dflt = precision == kFP32C ? ForceConfig{8, 2, 0} : ForceConfig{4, 4, 0};
    // Small systems, receiver ranges and separate sets: the warp-splitting
    // kernel.  Lane groups per warp from a B200 sweep: FP32C 8 up to 4096
    // receivers, 2 up to 8192; FP64 8 up to 16384, 4 up to 32768.  Ranges and
    // separate sets of 8192 to 32768 receivers went to the large kernels before
    // inv_cube; with it, us per FP64 evaluation of n receivers and n sources, this
    // kernel / the large one: 8192 82 / 104, 12288 165 / 185, 16384 277 / 302, 24576 611 /
    // 658, 32768 1058 / 1123; with 262144 sources 16384 4176 / 4321, 32768 8239 /
    // 8472.  (Above it the large kernel is at most 4 % slower, up to 65536.)
    const int F = precision == kFP32C ? (n_i <= 4096 ? 8 : n_i <= 8192 ? 2 : 0)
                                      : (n_i <= 16384 ? 8 : n_i <= 32768 ? 4 : 0);
    // From there to 2^23 particles: Newton-3 (B200, us per KDK step, the best
    // kernel above against the strips: FP32C 6000 42.6 / 20.8, 8192 53.6 / 32.0,
    // 12001 108.6 / 58.5; FP64 56.1 / 33.2, 87.8 / 55.0, 164 / 111; and larger
    // systems, see uses_strips and nbr_strip.cu).
    if (whole && n_i >= kN3MinN && n_i <= kN3MaxN) dflt = ForceConfig{3, kN3Warps, 0};
    else if (F) dflt = ForceConfig{1, F, 0};
    // (a Newton-3 result is of no use to a range or separate sets)
    cfg = it != g_tune->end() && (whole || it->second.ni != 3) ? it->second : dflt;
  }
  if (cfg.split <= 0) cfg.split = auto_split(precision, eps2, cfg, n_i, ntiles, c->sms);
  // at most one split per ring stage of sources (j-tile: 128 by default)
  const int tj = (cfg.ni == 4 || cfg.ni == 8) && cfg.tile > 0 ? cfg.tile : kTile;
  const int stages = (int)(((long long)ntiles * kTile + tj - 1) / tj);
  if (cfg.split > stages) cfg.split = std::max(1, stages);
  return cfg;
}

// The large-kernel default for callers that cannot take the Newton-3 kernels
// (a receiver range, separate receiver and source sets).
ForceConfig choose_config_large(nbr_ctx* c, int precision, double eps2, long long n_i, int ntiles) {
  ForceConfig cfg = precision == kFP32C ? ForceConfig{8, 2, 0} : ForceConfig{4, 4, 0};
  cfg.split = std::max(1, std::min(auto_split(precision, eps2, cfg, n_i, ntiles, c->sms), ntiles));
  return cfg;
}

// Test hook: NBR_TEST_N3_SLICES=k forces k launches of a Newton-3 evaluation on
// any system, so that the banded path (partial sums accumulated launch by
// launch, then the epilogue) runs on systems small enough to check against
// the oracle.  0: not set.
int forced_bands() {
  const char* f = std::getenv("NBR_TEST_N3_SLICES");
  return f ? std::max(0, std::atoi(f)) : 0;
}

// Slices of a banded evaluation of nb blocks by the CTA-grid kernel (1: one
// launch).
int n3_bands(long long nb) {
  if (const int k = forced_bands()) return k;
  const long long total = n3_scratch_doubles(nb);
  if (total <= kN3SingleMaxDoubles) return 1;
  int V = (int)((total + kN3SliceMaxDoubles - 1) / kN3SliceMaxDoubles);
  // slices are balanced by CTAs: grow V until the largest one fits
  while (V < (1 << 16)) {
    long long worst = 0;
    for (int v = 0; v < V; ++v) worst = std::max(worst, n3_slice_scratch_doubles(nb, v, V));
    if (worst <= kN3SliceMaxDoubles) break;
    ++V;
  }
  return V;
}

// Scratch of a banded Newton-3 evaluation: the largest slice's partial sums,
// then the FP64 accumulator [3][n_pad].
long long n3_banded_doubles(long long nb, int V, long long n_pad, long long* acc_off) {
  long long worst = 0;
  for (int v = 0; v < V; ++v) worst = std::max(worst, n3_slice_scratch_doubles(nb, v, V));
  *acc_off = (worst + 31) / 32 * 32;
  return *acc_off + 3 * n_pad;
}

// The launch-order table of the whole-system Newton-3 grid for nb blocks
// (n3_launch_order) followed by its inverse, written when nb changes.  Called
// outside stream capture (prepare_split runs before nbr_run captures).
cudaError_t n3_order_prepare(nbr_ctx* c, long long nb) {
  if (c->n3_order && c->n3_order_nb == nb) return cudaSuccess;
  std::vector<int> order;
  n3_launch_order(nb, n3_cols(nb), order);
  const size_t C = order.size();
  order.resize(2 * C);
  for (size_t i = 0; i < C; ++i) order[C + order[i]] = (int)i;
  cudaError_t e = cudaSuccess;
  if ((long long)order.size() > c->n3_order_cap) {
    dfree(c->n3_order);
    c->n3_order = nullptr;
    c->n3_order_cap = 0;
    c->n3_order_nb = -1;
    e = dalloc((void**)&c->n3_order, order.size() * sizeof(int));
    if (e != cudaSuccess) return e;
    c->n3_order_cap = (long long)order.size();
  }
  e = cudaMemcpyAsync(c->n3_order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice,
                      c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  c->n3_order_nb = e == cudaSuccess ? nb : -1;
  return e;
}

// The launches of a Newton-3 evaluation of the context's system in strips:
// receivers per lane, the row blocks at which they begin and end, and the
// scratch: the largest launch's partial sums, then, where there are several
// launches, the FP64 accumulator [3][n_pad].
struct StripLaunches {
  int ni = 0;
  std::vector<int> cut;
  long long acc_off = 0, doubles = 0;
};
StripLaunches strip_launches(nbr_ctx* c, int precision) {
  StripLaunches L;
  const long long n = (long long)c->sys.n;
  L.ni = strip_choose(precision, n, c->sms);
  L.cut = strip_bands(precision, n, c->sms, L.ni, forced_bands(), c->strip_single);
  for (size_t v = 0; v + 1 < L.cut.size(); ++v)
    L.doubles = std::max(
        L.doubles, strip_plan(precision, n, L.cut[v], L.cut[v + 1], c->sms, L.ni).doubles);
  if (L.cut.size() > 2) {
    L.acc_off = (L.doubles + 31) / 32 * 32;
    L.doubles = L.acc_off + 3 * (long long)c->sys.n_pad;
  }
  return L;
}
// FP32C: every whole system.  FP64: up to kStripMaxN64 particles (us per
// evaluation on B200, CTA grid against strips: 32768 812 / 719, 65536 2904 /
// 2828, 131072 11323 / 11293, 262144 44156 / 44625, 2^20 705 / 718 ms: the
// strips' 24 B of reactions per (320 rows, particle) take more launches).
// Test hook: NBR_TEST_N3_GRID set, FP64 takes the CTA grid at any size, so that
// systems small enough for the oracle reach it.
bool uses_strips(int precision, const ForceConfig& cfg, long long n) {
  if (cfg.ni != 3 || cfg.warps != kN3Warps) return false;
  return precision == kFP32C || (n <= kStripMaxN64 && !std::getenv("NBR_TEST_N3_GRID"));
}

// Prepares scratch for a force launch of `cfg` over n_i receivers.
int prepare_split(nbr_ctx* c, int precision, const ForceConfig& cfg, long long n_pad_i) {
  if (uses_strips(precision, cfg, (long long)c->sys.n)) {  // (the context's whole system only)
    const StripLaunches L = strip_launches(c, precision);
    const StripKernel k{precision, L.ni, (long long)c->sys.n};
    if (!(k == c->strip_ready)) {
      const cudaError_t e = prepare_strips(precision, k.n, k.ni);
      if (e != cudaSuccess) return cuda_fail(c, e, "Newton-3 kernel setup");
      c->strip_ready = k;
    }
    long long doubles = L.doubles;
    cudaError_t e = with_room(c, [&] { return c->scr.need_part((size_t)doubles); });
    if (e == cudaErrorMemoryAllocation && doubles > kN3SliceMaxDoubles &&
        c->strip_single > kN3SliceMaxDoubles) {
      // No room for one launch's scratch (up to 9 GiB; the CTA grid, which
      // took 0.6 of it, may have found room): several launches of 2 GiB.  (No
      // graph captured with the larger scratch is left to run on the smaller.)
      cudaGetLastError();
      give_back(c);
      c->strip_single = kN3SliceMaxDoubles;
      doubles = strip_launches(c, precision).doubles;
      e = c->scr.need_part((size_t)doubles);
    }
    return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "Newton-3 scratch");
  }
  if (cfg.ni == 3) {  // Newton-3 (the context's whole system only): its own partial sums
    (void)n_pad_i;
    const long long nb = ((long long)c->sys.n + kN3Block - 1) / kN3Block;
    const int V = n3_bands(nb);
    long long acc_off = 0;
    const long long need =
        V == 1 ? n3_scratch_doubles(nb) : n3_banded_doubles(nb, V, (long long)c->sys.n_pad, &acc_off);
    cudaError_t e = with_room(c, [&] { return c->scr.need_part((size_t)need); });
    if (e == cudaSuccess && V == 1) e = n3_order_prepare(c, nb);
    return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "Newton-3 scratch");
  }
  if (cfg.split <= 1) return NBR_OK;
  cudaError_t e =
      with_room(c, [&] { return c->scr.need_part((size_t)cfg.split * 3 * (size_t)n_pad_i); });
  if (e == cudaSuccess)
    e = with_room(c, [&] { return c->scr.need_counters((size_t)(n_pad_i / 64 + 1)); });
  return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "split scratch");
}

// Bounded-wait limit and the test hook of the tile pipeline, from the
// environment: NBR_WAIT_LIMIT_MS (default 4000) and NBR_TEST_SKIP_TILE
// (CTA-local tile index whose copy is never issued, so that its wait expires
// and the launch reports NBR_ERR_TIMEOUT; default off).
void pipeline_params(JStream& js) {
  js.wait_ns = kWaitLimitNs;
  js.skip_tile = -1;
  if (const char* w = std::getenv("NBR_WAIT_LIMIT_MS")) {
    const long long ms = std::atoll(w);
    if (ms > 0) js.wait_ns = (unsigned long long)ms * 1000000ull;
  }
  if (const char* k = std::getenv("NBR_TEST_SKIP_TILE")) {
    if (*k) js.skip_tile = std::atoi(k);
  }
}

// Reads and clears the device error word; maps it to a status.
int check_device_error(nbr_ctx* c) {
  int h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "kernel execution");
  return device_error_status(c, h);
}

bool stage_host(nbr_ctx* c, size_t doubles) {
  if (c->h_stage.size() >= doubles) return true;
  try {
    c->h_stage.resize(doubles);
  } catch (const std::bad_alloc&) {
    return false;
  }
  return true;
}

bool stage_ready(nbr_ctx* c, size_t doubles) {
  if (!stage_host(c, doubles)) return false;
  if (c->scr.need_red(doubles) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

cudaError_t stage_fetch(nbr_ctx* c, const StageArrays& a, double* dst, int words[2]) {
  size_t total = 0;
  for (int k = 0; k < a.count; ++k) total += (size_t)a.n[k];
  if (!stage_host(c, total + 1)) return cudaErrorMemoryAllocation;
  cudaError_t e = launch_stage_out(a, dst, c->d_err, c->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c->h_stage.data(), dst, (total + 1) * sizeof(double),
                        cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) std::memcpy(words, c->h_stage.data() + total, 2 * sizeof(int));
  return e;
}

cudaError_t stage_download(nbr_ctx* c, int count, const double* const* src, double* const* out,
                           size_t n, int* err, int* flags) {
  StageArrays a{};
  double* to[8];
  for (int k = 0; k < count; ++k) {
    if (!out[k]) continue;
    a.dev[a.count] = const_cast<double*>(src[k]);
    a.n[a.count] = (long long)n;
    to[a.count++] = out[k];
  }
  const int arrays = a.count;
  if (a.count == 0) a.count = 1;  // the error words alone
  cudaError_t e = c->scr.need_red(arrays * n + 2);
  int words[2] = {0, 0};
  if (e == cudaSuccess) e = stage_fetch(c, a, c->scr.red, words);
  if (e != cudaSuccess) return e;
  if (err) *err = words[0];
  if (flags) *flags = words[1];
  if (!(err && *err != kErrNone) && !(flags && *flags))
    for (int k = 0; k < arrays; ++k)
      std::memcpy(to[k], c->h_stage.data() + (size_t)k * n, n * sizeof(double));
  return cudaSuccess;
}

int device_error_status(nbr_ctx* c, int h) {
  if (h != kErrNone) {
    cudaMemsetAsync(c->d_err, 0, sizeof(int), c->stream);
    if (c->scr.cnt) cudaMemsetAsync(c->scr.cnt, 0, c->scr.cnt_cap * sizeof(unsigned), c->stream);
    cudaStreamSynchronize(c->stream);
    c->acc_ok = false;
    if (h == kErrBounds)
      return fail(c, NBR_ERR_BOUNDS, "a kernel index was outside its array (checked build); "
                                     "the access was skipped");
    return fail(c, NBR_ERR_TIMEOUT,
                h == kErrTileWait ? "a j-tile copy did not complete within the wait limit"
                                  : "device wait limit exceeded (code " + std::to_string(h) + ")");
  }
  return NBR_OK;
}

// Makes the FP32C records of position buffer b valid.
cudaError_t ensure_records(nbr_ctx* c, int b, int* kernels) {
  SysState& s = c->sys;
  if (s.rec_ok[b]) return cudaSuccess;
  cudaError_t e = launch_kick_drift((long long)s.n, (long long)s.n_pad, s.pos[b][0], s.pos[b][1],
                                    s.pos[b][2], s.mass, nullptr, nullptr, nullptr, 0.0, 0.0,
                                    nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, s.rec[b],
                                    s.org[b], c->stream);
  if (kernels) ++*kernels;
  if (e == cudaSuccess) s.rec_ok[b] = true;
  return e;
}

// One force evaluation of the uploaded system on its current buffer with the
// given epilogue (mode 1 writes the next buffer, which becomes current).
// Receivers are particles [r0, r0 + rn) (rn < 0: all n); sources are always
// all n.  With a receiver range only the range's entries of the next buffer
// are written, so no FP32C records are packed for it.
int eval_system(nbr_ctx* c, int precision, double G, double eps2, int mode, double kick,
                double drift, int want_force, int* kernels, long long r0 = 0, long long rn = -1) {
  SysState& s = c->sys;
  const int a = s.cur, b = 1 - s.cur;
  const bool ranged = rn >= 0;
  if (!ranged) {
    r0 = 0;
    rn = (long long)s.n;
  }
  const long long np_i = ((rn + 1023) / 1024) * 1024;
  cudaError_t e = cudaSuccess;
  ForceConfig cfg = choose_config(c, precision, eps2, rn, s.ntiles, !ranged);
  if (cfg.ni == 3 && ranged)  // needs the whole system
    cfg = choose_config_large(c, precision, eps2, rn, s.ntiles);
  const bool strips = uses_strips(precision, cfg, rn);  // these read the FP64 positions: no records
  if (precision == kFP32C && !strips) e = ensure_records(c, a, kernels);
  if (e != cudaSuccess) return cuda_fail(c, e, "pack");
  int rc = prepare_split(c, precision, cfg, np_i);
  if (rc) return rc;
  IParticles ip{s.pos[a][0] + r0, s.pos[a][1] + r0, s.pos[a][2] + r0, s.mass + r0, rn};
  JStream js{s.pos[a][0], s.pos[a][1], s.pos[a][2], s.mass, s.rec[a], s.org[a], s.ntiles, 0, -1};
  pipeline_params(js);
  Epilogue ep{};
  ep.mode = mode;
  ep.G = G;
  ep.ax = s.acc[0] + r0; ep.ay = s.acc[1] + r0; ep.az = s.acc[2] + r0;
  ep.want_force = want_force;
  ep.kick = kick;
  ep.drift = drift;
  ep.vx = s.vel[0] + r0; ep.vy = s.vel[1] + r0; ep.vz = s.vel[2] + r0;
  ep.xn = s.pos[b][0] + r0; ep.yn = s.pos[b][1] + r0; ep.zn = s.pos[b][2] + r0;
  // neither the small-N kernel nor the strips pack records
  const bool packs = precision == kFP32C && !ranged && cfg.ni != 1 && !strips;
  ep.rec_next = mode != 0 && packs ? s.rec[b] : nullptr;
  ep.origin_next = s.org[b];
  ep.part = c->scr.part;
  ep.counters = c->scr.cnt;
  ep.n_pad = np_i;
  ep.err = c->d_err;
  NBR_CHECKED_ONLY(
      ip.len = (long long)(s.cap + kRangeSlack) - r0; js.len = (long long)s.cap;
      ep.part_len = (long long)c->scr.part_cap; ep.cnt_len = (long long)c->scr.cnt_cap;
      ep.rec_len = (long long)s.cap;
      // test hook: under-report the receivers' length so that the check trips
      if (std::getenv("NBR_TEST_SHRINK_BOUNDS")) ip.len = rn - 1;)
  if (strips) {
    const StripLaunches L = strip_launches(c, precision);
    const bool one = L.cut.size() == 2;
    const long long np = (long long)s.n_pad;
    double* acc = c->scr.part + L.acc_off;
    for (size_t v = 0; v + 1 < L.cut.size() && e == cudaSuccess; ++v) {
      const StripPlan sp = strip_plan(precision, rn, L.cut[v], L.cut[v + 1], c->sms, L.ni);
      e = launch_strips(precision, sp, eps2, ip, js, ep, c->scr.part, c->sms,
                        one ? 0 : v == 0 ? 1 : 2, acc, np, c->stream);
      if (kernels) *kernels += 2;
    }
    if (!one) {
      if (e == cudaSuccess) e = launch_sum_finish(ip, ep, acc, 1, 0, np, 3 * np, c->stream);
      if (kernels) *kernels += 1;
    }
  } else if (cfg.ni == 3) {
    const long long nb = (rn + kN3Block - 1) / kN3Block;
    const int V = n3_bands(nb);
    if (V == 1) {
      e = launch_force_n3(precision, cfg.warps, eps2, ip, js, ep, c->scr.part,
                          (long long)c->scr.part_cap, c->n3_order, c->stream);
      if (kernels) *kernels += 2;
    } else {
      // banded: the slices' partial accelerations accumulate in slice order in
      // an FP64 buffer behind the largest slice's scratch, then the epilogue
      long long acc_off = 0;
      n3_banded_doubles(nb, V, (long long)s.n_pad, &acc_off);
      double* acc = c->scr.part + acc_off;
      const long long np = (long long)s.n_pad;
      for (int v = 0; v < V && e == cudaSuccess; ++v) {
        e = launch_n3_slice(precision, cfg.warps, eps2, ip, js, ep.err, v, V, c->scr.part, acc_off,
                            acc, np, 3 * np, v > 0, c->stream);
        if (kernels) *kernels += 2;
      }
      if (e == cudaSuccess) e = launch_sum_finish(ip, ep, acc, 1, 0, np, 3 * np, c->stream);
      if (kernels) *kernels += 1;
    }
  } else {
    e = launch_force(precision, eps2, cfg, ip, js, ep, c->stream);
    if (kernels) ++*kernels;
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "force launch");
  if (mode != 0) {
    s.cur = b;
    s.rec_ok[b] = packs;
    s.rec_ok[a] = false;
  }
  return NBR_OK;
}

// Standalone kick (v += kick a) + drift (x' = x + drift v into the other
// buffer), packing records of x' when the next evaluation is FP32C.
int kick_drift_system(nbr_ctx* c, bool pack, double kick, double drift, bool use_acc,
                      int* kernels) {
  SysState& s = c->sys;
  const int a = s.cur, b = 1 - s.cur;
  cudaError_t e = launch_kick_drift(
      (long long)s.n, (long long)s.n_pad, s.pos[a][0], s.pos[a][1], s.pos[a][2], s.mass,
      use_acc ? s.acc[0] : nullptr, use_acc ? s.acc[1] : nullptr, use_acc ? s.acc[2] : nullptr,
      kick, drift, s.vel[0], s.vel[1], s.vel[2], s.pos[b][0], s.pos[b][1], s.pos[b][2],
      pack ? s.rec[b] : nullptr, pack ? s.org[b] : nullptr, c->stream);
  if (kernels) ++*kernels;
  if (e != cudaSuccess) return cuda_fail(c, e, "kick-drift launch");
  s.cur = b;
  s.rec_ok[b] = pack;
  s.rec_ok[a] = false;
  return NBR_OK;
}

// Softened potential of the uploaded system on the context stream: phi into
// dphi (device, may be null) and U = 1/2 sum m_i phi_i as *dU (device) times
// *factor.  Without phi the pairs are evaluated once each (launch_energy).
// Uses red[red_off ..] for the per-chunk sums: at most potential_sums(c) + 16.
size_t potential_sums(const nbr_ctx* c) {
  return std::max<size_t>((c->sys.n + 127) / 128, (size_t)kEnergyStrips * c->sms);
}
int potential_system(nbr_ctx* c, double G, double eps2, double* dphi, size_t red_off,
                     double** dU, double* factor) {
  SysState& s = c->sys;
  const int a = s.cur;
  IParticles ip{s.pos[a][0], s.pos[a][1], s.pos[a][2], s.mass, (long long)s.n};
  JStream js{s.pos[a][0], s.pos[a][1], s.pos[a][2], s.mass, nullptr, nullptr, s.ntiles, 0, -1};
  pipeline_params(js);
  NBR_CHECKED_ONLY(ip.len = (long long)(s.cap + kRangeSlack); js.len = (long long)s.cap;)
  if (!dphi && (long long)s.n <= kEnergyMaxN) {
    cudaError_t e = with_room(c, [&] { return c->scr.need_red(red_off + potential_sums(c) + 16); });
    if (e != cudaSuccess) return cuda_fail(c, e, "potential scratch");
    double* sums = c->scr.red + red_off;
    int strips = 0;
    e = launch_energy((long long)s.n, eps2, ip, js, c->d_err, sums, c->sms, &strips, c->stream);
    if (e == cudaSuccess) e = launch_scaled_sum(sums, strips, kInvDistScale, sums + strips, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "energy launch");
    *dU = sums + strips;
    *factor = -G;
    return NBR_OK;
  }
  *factor = 1.0;
  const ForceConfig pc{kPotNI, kPotWarps, 0};
  int split = auto_split(kFP64, eps2, pc, (long long)s.n, s.ntiles, c->sms);
  split = std::max(1, std::min(split, s.ntiles));
  const ForceConfig cfg{kPotNI, kPotWarps, split};
  int rc = prepare_split(c, kFP64, cfg, (long long)s.n_pad);
  if (rc) return rc;
  const long long chunk = 32LL * kPotNI * kPotWarps;
  const int chunks = (int)(((long long)s.n + chunk - 1) / chunk);
  cudaError_t e = with_room(c, [&] { return c->scr.need_red(red_off + (size_t)chunks + 16); });
  if (e != cudaSuccess) return cuda_fail(c, e, "potential scratch");
  PotentialOut po{};
  po.G = G;
  po.phi = dphi;
  po.blocksum = c->scr.red + red_off;
  po.part = c->scr.part;
  po.counters = c->scr.cnt;
  po.n_pad = (long long)s.n_pad;
  po.err = c->d_err;
  NBR_CHECKED_ONLY(
      po.part_len = (long long)c->scr.part_cap; po.cnt_len = (long long)c->scr.cnt_cap;
      po.blocksum_len = (long long)(c->scr.red_cap - red_off);)
  e = launch_potential(split, ip, js, po, eps2, c->stream);
  if (e == cudaSuccess)
    e = launch_rowsum(po.blocksum, chunks, 1, po.blocksum + chunks, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "potential launch");
  *dU = po.blocksum + chunks;
  return NBR_OK;
}

int diag_system(nbr_ctx* c, double G, double eps2, nbr_diag* out) {
  SysState& s = c->sys;
  const int a = s.cur;
  const int nb = (int)((s.n + 127) / 128);
  // moments (8 x nb), their sums (16), then the potential's sums and U, then
  // the results packed: sized once here so that nothing below reallocates.
  const size_t used = (size_t)nb * 9 + 32 + potential_sums(c);
  cudaError_t e = with_room(c, [&] { return c->scr.need_red(used + 16); });
  if (e != cudaSuccess) return cuda_fail(c, e, "diag scratch");
  double* part = c->scr.red;
  double* res = c->scr.red + (size_t)nb * 8;
  e = launch_moments((long long)s.n, (long long)s.n_pad, s.pos[a][0], s.pos[a][1], s.pos[a][2],
                     s.vel[0], s.vel[1], s.vel[2], s.mass, part, c->stream);
  if (e == cudaSuccess) e = launch_rowsum(part, nb, 8, res, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "diagnostics");
  double *dU = nullptr, factor = 1.0;
  int rc = potential_system(c, G, eps2, nullptr, (size_t)nb * 9 + 16, &dU, &factor);
  if (rc) return rc;
  StageArrays sa{};
  sa.count = 2;
  sa.dev[0] = res; sa.n[0] = 8;
  sa.dev[1] = dU; sa.n[1] = 1;
  int words[2];
  e = stage_fetch(c, sa, c->scr.red + used, words);
  if (e != cudaSuccess) return cuda_fail(c, e, "diagnostics");
  rc = device_error_status(c, words[0]);
  if (rc) return rc;
  const double* h = c->h_stage.data();
  out->T = h[0];
  out->P[0] = h[1]; out->P[1] = h[2]; out->P[2] = h[3];
  out->L[0] = h[4]; out->L[1] = h[5]; out->L[2] = h[6];
  out->M = h[7];
  out->U = factor * h[8];
  out->E = out->T + out->U;
  return NBR_OK;
}

// Yoshida weights -> c/d (order 2/4/6/8), the construction of omp_main
// (CPU/omp_solver.cpp:677-726): c_0 = c_{2w-1} = w_{w-1}/2,
// c_i = c_{2w-1-i} = (w_{w-i} + w_{w-1-i})/2, d_i = d_{2w-2-i} = w_{w-1-i}.
int yoshida(int order, double* c, double* d) {
  const double cb = std::cbrt(2.0);
  double w2[1] = {1.0};
  double w4[2] = {-cb / (2.0 - cb), 1.0 / (2.0 - cb)};
  double w6[4] = {1.0, -1.17767998417887, 0.235573213359357, 0.78451361047756};
  double w8[8] = {1.0, -0.161582374150097e1, -0.244699182370524e1, -0.716989419708120e-2,
                  0.244002732616735e1, 0.157739928123617, 0.182020630970714e1,
                  0.104242620869991e1};
  for (int i = 1; i < 4; ++i) w6[0] -= 2.0 * w6[i];
  for (int i = 1; i < 8; ++i) w8[0] -= 2.0 * w8[i];
  const double* w;
  int ws;
  switch (order) {
    case 2: w = w2; ws = 1; break;
    case 4: w = w4; ws = 2; break;
    case 6: w = w6; ws = 4; break;
    case 8: w = w8; ws = 8; break;
    default: return 0;
  }
  for (int i = 0; i < ws; ++i) {
    const double ci = i == 0 ? w[ws - 1] / 2.0 : (w[ws - i] + w[ws - 1 - i]) / 2.0;
    c[i] = c[2 * ws - 1 - i] = ci;
    d[i] = d[2 * ws - 2 - i] = w[ws - 1 - i];
  }
  return 2 * ws;
}

}  // namespace nbr

// ===================================================================== ABI ==
extern "C" {

int nbr_version(void) { return 1000; }

int nbr_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

const char* nbr_last_error_string(const nbr_ctx* c) {
  return c ? c->err.c_str() : t_err.c_str();
}

int nbr_ctx_create(int device, nbr_ctx** out) {
  if (!out) return fail(nullptr, NBR_ERR_INVALID_ARG, "out is NULL");
  *out = nullptr;
  int nd = nbr_device_count();
  if (nd == 0) return fail(nullptr, NBR_ERR_UNSUPPORTED, "no CUDA device");
  if (device < 0 || device >= nd) return fail(nullptr, NBR_ERR_INVALID_ARG, "bad device index");
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaSetDevice");
  cudaDeviceProp prop;
  e = cudaGetDeviceProperties(&prop, device);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDeviceProperties");
  if (prop.major < 10)
    return fail(nullptr, NBR_ERR_UNSUPPORTED,
                std::string("needs an sm_100 device, found ") + prop.name);
  nbr_ctx* c = new nbr_ctx();
  c->device = device;
  c->sms = prop.multiProcessorCount;
  c->coop = prop.cooperativeLaunch != 0;
  e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&c->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&c->ev1);
  if (e == cudaSuccess) e = dalloc((void**)&c->d_err, sizeof(int) * 4);
  if (e == cudaSuccess) e = configure_kernels();
  if (e != cudaSuccess) {
    int rc = cuda_fail(nullptr, e, "context setup");
    nbr_ctx_destroy(c);
    return rc;
  }
  *out = c;
  return NBR_OK;
}

int nbr_ctx_destroy(nbr_ctx* c) {
  if (!c) return NBR_OK;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  for (RunGraph& g : c->run_graph) g.release();
  c->sys.release();
  c->bat.release();
  c->scr.release();
  c->ij.release();
  dfree(c->n3_order);
  dfree(c->d_err);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return NBR_OK;
}

void* nbr_ctx_stream(nbr_ctx* c) { return c ? (void*)c->stream : nullptr; }

int nbr_ctx_synchronize(nbr_ctx* c) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  cudaSetDevice(c->device);
  cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "synchronize");
  // A bounded wait that gave up in an asynchronous call surfaces here.
  return check_device_error(c);
}

size_t nbr_system_size(const nbr_ctx* c) { return c ? c->sys.n : 0; }

int nbr_system_upload(nbr_ctx* c, size_t n, const double* x, const double* y, const double* z,
                      const double* vx, const double* vy, const double* vz, const double* m) {
  TraceRange trace_range("nbr_system_upload");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (n == 0 || !x || !y || !z || !m) return fail(c, NBR_ERR_INVALID_ARG, "empty system or NULL array");
  if ((vx || vy || vz) && !(vx && vy && vz))
    return fail(c, NBR_ERR_INVALID_ARG, "velocities must be all given or all NULL");
  if (n > (size_t)1 << 31) return fail(c, NBR_ERR_INVALID_ARG, "n above 2^31");
  cudaSetDevice(c->device);
  SysState& s = c->sys;
  const size_t cap0 = s.cap;
  cudaError_t e = with_room(c, [&] { return s.reserve(n); });
  if (s.cap != cap0)  // their buffers are gone
    for (RunGraph& g : c->run_graph) g.release();
  if (e != cudaSuccess) return cuda_fail(c, e, "system allocation");
  s.cur = 0;
  s.rec_ok[0] = s.rec_ok[1] = false;
  c->strip_single = kN3SingleMaxDoubles;
  c->acc_ok = false;
  const size_t B = n * sizeof(double);
  auto H = [&](double* d, const double* h) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(d, h, B, cudaMemcpyHostToDevice, c->stream);
  };
  H(s.pos[0][0], x); H(s.pos[0][1], y); H(s.pos[0][2], z);
  H(s.mass, m);
  if (vx) { H(s.vel[0], vx); H(s.vel[1], vy); H(s.vel[2], vz); }
  else {
    for (int d = 0; d < 3 && e == cudaSuccess; ++d)
      e = cudaMemsetAsync(s.vel[d], 0, B, c->stream);
  }
  // NaN / Inf / negative-mass check on the device copy (one pass over the
  // uploaded bytes at HBM speed instead of a host loop over them).
  int* flags = c->d_err + 1;
  int h_flags = 0;
  if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0, sizeof(int), c->stream);
  if (e == cudaSuccess)
    e = launch_validate((long long)n, s.pos[0][0], s.pos[0][1], s.pos[0][2], vx ? s.vel[0] : nullptr,
                        s.vel[1], s.vel[2], s.mass, flags, c->sms, c->stream);
  if (e == cudaSuccess) e = s.clear_padding(c->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&h_flags, flags, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    s.n = 0;  // no half-copied system is kept
    return cuda_fail(c, e, "upload");
  }
  if (h_flags) {
    s.n = 0;  // the rejected system is not kept
    return (h_flags & 1) ? fail(c, NBR_ERR_NONFINITE, "input contains NaN or Inf")
                         : fail(c, NBR_ERR_INVALID_ARG, "negative mass");
  }
  return NBR_OK;
}

int nbr_system_download(nbr_ctx* c, double* x, double* y, double* z, double* vx, double* vy,
                        double* vz) {
  TraceRange trace_range("nbr_system_download");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  const size_t B = s.n * sizeof(double);
  cudaError_t e = cudaSuccess;
  if (stage_fits(6 * s.n) && stage_ready(c, 6 * s.n + 2)) {
    const double* src[6] = {s.pos[s.cur][0], s.pos[s.cur][1], s.pos[s.cur][2],
                            s.vel[0], s.vel[1], s.vel[2]};
    double* out[6] = {x, y, z, vx, vy, vz};
    e = stage_download(c, 6, src, out, s.n, nullptr);
    return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "download");
  }
  auto D = [&](double* h, const double* d) {
    if (h && e == cudaSuccess) e = cudaMemcpyAsync(h, d, B, cudaMemcpyDeviceToHost, c->stream);
  };
  D(x, s.pos[s.cur][0]); D(y, s.pos[s.cur][1]); D(z, s.pos[s.cur][2]);
  D(vx, s.vel[0]); D(vy, s.vel[1]); D(vz, s.vel[2]);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "download");
}

int nbr_forces(nbr_ctx* c, int precision, double G, double eps2, int want_force, double* ax,
               double* ay, double* az) {
  TraceRange trace_range("nbr_forces");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (!(eps2 >= 0.0) || !std::isfinite(eps2) || !std::isfinite(G))
    return fail(c, NBR_ERR_INVALID_ARG, "eps2 must be finite and >= 0, G finite");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  int rc = eval_system(c, precision, G, eps2, 0, 0.0, 0.0, want_force, nullptr);
  if (rc) return rc;
  const bool staged = stage_fits(3 * s.n) && stage_ready(c, 3 * s.n + 2);
  if (staged) {
    const double* src[3] = {s.acc[0], s.acc[1], s.acc[2]};
    double* out[3] = {ax, ay, az};
    int err = 0;
    const cudaError_t e = stage_download(c, 3, src, out, s.n, &err);
    if (e != cudaSuccess) return cuda_fail(c, e, "kernel execution");
    rc = device_error_status(c, err);
  } else {
    rc = check_device_error(c);
  }
  if (rc) return rc;
  c->acc_ok = !want_force;
  c->acc_prec = precision;
  c->acc_G = G;
  c->acc_eps2 = eps2;
  if (staged) return NBR_OK;
  const size_t B = s.n * sizeof(double);
  cudaError_t e = cudaSuccess;
  auto D = [&](double* h, const double* d) {
    if (h && e == cudaSuccess) e = cudaMemcpyAsync(h, d, B, cudaMemcpyDeviceToHost, c->stream);
  };
  D(ax, s.acc[0]); D(ay, s.acc[1]); D(az, s.acc[2]);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "forces download");
}

int nbr_forces_device(nbr_ctx* c, int precision, double G, double eps2) {
  TraceRange trace_range("nbr_forces_device");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (!(eps2 >= 0.0) || !std::isfinite(eps2) || !std::isfinite(G))
    return fail(c, NBR_ERR_INVALID_ARG, "eps2 must be finite and >= 0, G finite");
  if (c->sys.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  const int rc = eval_system(c, precision, G, eps2, 0, 0.0, 0.0, 0, nullptr);
  if (rc) return rc;
  c->acc_ok = true;
  c->acc_prec = precision;
  c->acc_G = G;
  c->acc_eps2 = eps2;
  return NBR_OK;
}

int nbr_forces_download(nbr_ctx* c, double* ax, double* ay, double* az) {
  TraceRange trace_range("nbr_forces_download");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  int rc = check_device_error(c);
  if (rc) return rc;
  const size_t B = s.n * sizeof(double);
  cudaError_t e = cudaSuccess;
  auto D = [&](double* h, const double* d) {
    if (h && e == cudaSuccess) e = cudaMemcpyAsync(h, d, B, cudaMemcpyDeviceToHost, c->stream);
  };
  D(ax, s.acc[0]); D(ay, s.acc[1]); D(az, s.acc[2]);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "forces download");
}

// ------------------------------------------------ multi-GPU i-partition ----

int nbr_step_range(nbr_ctx* c, int precision, int scheme, size_t i0, size_t count, double kick,
                   double drift, double G, double eps2) {
  TraceRange trace_range("nbr_step_range");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (scheme != NBR_KDK && scheme != NBR_DKD && scheme != NBR_EULER)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown scheme");
  if (!std::isfinite(kick) || !std::isfinite(drift) || !(eps2 >= 0.0) || !std::isfinite(eps2) ||
      !std::isfinite(G))
    return fail(c, NBR_ERR_INVALID_ARG, "kick, drift, G must be finite, eps2 finite and >= 0");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  if (i0 % kTile != 0) return fail(c, NBR_ERR_INVALID_ARG, "i0 must be a multiple of 128");
  if (count == 0 || i0 >= s.n) return fail(c, NBR_ERR_INVALID_ARG, "empty receiver range");
  const size_t rn = std::min(count, s.n - i0);
  cudaSetDevice(c->device);
  const int rc = eval_system(c, precision, G, eps2, scheme == NBR_EULER ? 2 : 1, kick, drift, 0,
                             nullptr, (long long)i0, (long long)rn);
  c->acc_ok = false;
  return rc;
}

int nbr_n3_grid_plan(size_t n, int sms, int nslices, int* cols, int* slice_cols,
                     double* efficiency, long long* ctas, int* order, long long order_cap) {
  if (n < 1 || sms < 1 || nslices < 1)
    return fail(nullptr, NBR_ERR_INVALID_ARG, "need n >= 1, sms >= 1, nslices >= 1");
  const long long nb = ((long long)n + kN3Block - 1) / kN3Block;
  const int c = n3_cols_for(nb, sms);
  if (cols) *cols = c;
  if (slice_cols) *slice_cols = n3_slice_cols_for(nb, nslices, sms);
  if (efficiency) *efficiency = n3_grid_efficiency_for(nb, sms);
  if (ctas) *ctas = n3_ctas(nb, c);
  if (order && order_cap > 0) {
    std::vector<int> o;
    n3_launch_order(nb, c, o);
    const size_t k = std::min((size_t)order_cap, o.size());
    std::copy(o.begin(), o.begin() + (long)k, order);
  }
  return NBR_OK;
}

int nbr_n3_slice_accel(nbr_ctx* c, int precision, double eps2, int slice_begin, int slice_end,
                       int nslices, double* dst, size_t ld) {
  TraceRange trace_range("nbr_n3_slice_accel");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (!(eps2 >= 0.0) || !std::isfinite(eps2))
    return fail(c, NBR_ERR_INVALID_ARG, "eps2 must be finite and >= 0");
  if (nslices < 1 || slice_begin < 0 || slice_end <= slice_begin || slice_end > nslices)
    return fail(c, NBR_ERR_INVALID_ARG, "need 0 <= slice_begin < slice_end <= nslices");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  if (!dst || ld < s.n_pad)
    return fail(c, NBR_ERR_INVALID_ARG, "dst is NULL or ld below the padded particle count");
  cudaSetDevice(c->device);
  const int a = s.cur;
  cudaError_t e = precision == kFP32C ? ensure_records(c, a, nullptr) : cudaSuccess;
  if (e != cudaSuccess) return cuda_fail(c, e, "pack");
  const long long nb = ((long long)s.n + kN3Block - 1) / kN3Block;
  const long long need = n3_slices_scratch_doubles(nb, slice_begin, slice_end, nslices);
  e = with_room(c, [&] { return c->scr.need_part((size_t)std::max<long long>(need, 1)); });
  if (e != cudaSuccess) return cuda_fail(c, e, "Newton-3 slice scratch");
  ForceConfig cfg = choose_config(c, precision, eps2, (long long)s.n, s.ntiles);
  const int warps = cfg.ni == 3 ? cfg.warps : kN3Warps;
  IParticles ip{s.pos[a][0], s.pos[a][1], s.pos[a][2], s.mass, (long long)s.n};
  JStream js{s.pos[a][0], s.pos[a][1], s.pos[a][2], s.mass, s.rec[a], s.org[a], s.ntiles, 0, -1};
  pipeline_params(js);
  NBR_CHECKED_ONLY(ip.len = (long long)(s.cap + kRangeSlack); js.len = (long long)s.cap;)
  e = launch_n3_slices(precision, warps, eps2, ip, js, c->d_err, slice_begin, slice_end, nslices,
                       c->scr.part, (long long)c->scr.part_cap, dst, (long long)ld,
                       3 * (long long)ld * (slice_end - slice_begin), false, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "Newton-3 slice launch");
  c->acc_ok = false;
  return NBR_OK;
}

int nbr_step_range_sum(nbr_ctx* c, int precision, int scheme, size_t i0, size_t count, double kick,
                       double drift, double G, const double* src, int nslices, size_t vstride,
                       size_t ld) {
  TraceRange trace_range("nbr_step_range_sum");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (scheme != NBR_KDK && scheme != NBR_DKD && scheme != NBR_EULER)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown scheme");
  if (!std::isfinite(kick) || !std::isfinite(drift) || !std::isfinite(G))
    return fail(c, NBR_ERR_INVALID_ARG, "kick, drift, G must be finite");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  if (i0 % kTile != 0) return fail(c, NBR_ERR_INVALID_ARG, "i0 must be a multiple of 128");
  if (count == 0 || i0 >= s.n) return fail(c, NBR_ERR_INVALID_ARG, "empty receiver range");
  const size_t rn = std::min(count, s.n - i0);
  const size_t rpad = (rn + kTile - 1) / kTile * kTile;
  if (!src || nslices < 1 || ld < rpad || (nslices > 1 && vstride < 3 * ld))
    return fail(c, NBR_ERR_INVALID_ARG, "src layout: ld >= count rounded up to 128, vstride >= 3 ld");
  cudaSetDevice(c->device);
  const int a = s.cur, b = 1 - s.cur;
  IParticles ip{s.pos[a][0] + i0, s.pos[a][1] + i0, s.pos[a][2] + i0, s.mass + i0, (long long)rn};
  Epilogue ep{};
  ep.mode = scheme == NBR_EULER ? 2 : 1;
  ep.G = G;
  ep.ax = s.acc[0] + i0; ep.ay = s.acc[1] + i0; ep.az = s.acc[2] + i0;
  ep.kick = kick;
  ep.drift = drift;
  ep.vx = s.vel[0] + i0; ep.vy = s.vel[1] + i0; ep.vz = s.vel[2] + i0;
  ep.xn = s.pos[b][0] + i0; ep.yn = s.pos[b][1] + i0; ep.zn = s.pos[b][2] + i0;
  ep.rec_next = nullptr;
  ep.err = c->d_err;
  NBR_CHECKED_ONLY(ip.len = (long long)(s.cap + kRangeSlack) - (long long)i0;)
  const long long src_len = (long long)(nslices - 1) * (long long)vstride + 3 * (long long)ld;
  cudaError_t e = launch_sum_finish(ip, ep, src, nslices, (long long)vstride, (long long)ld, src_len,
                                    c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "slice sum launch");
  s.cur = b;
  s.rec_ok[0] = s.rec_ok[1] = false;
  c->acc_ok = false;
  return NBR_OK;
}

int nbr_state_pointers(nbr_ctx* c, double** x, double** y, double** z, double** vx, double** vy,
                       double** vz, size_t* len) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  if (x) *x = s.pos[s.cur][0];
  if (y) *y = s.pos[s.cur][1];
  if (z) *z = s.pos[s.cur][2];
  if (vx) *vx = s.vel[0];
  if (vy) *vy = s.vel[1];
  if (vz) *vz = s.vel[2];
  if (len) *len = s.n_pad + kRangeSlack;
  return NBR_OK;
}

int nbr_state_changed(nbr_ctx* c) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  SysState& s = c->sys;
  s.rec_ok[0] = s.rec_ok[1] = false;
  c->acc_ok = false;
  return NBR_OK;
}

int nbr_accel_ij(nbr_ctx* c, int precision, size_t n_i, const double* xi, const double* yi,
                 const double* zi, const double* mi, size_t n_j, const double* xj,
                 const double* yj, const double* zj, const double* mj, double G, double eps2,
                 int want_force, double* ax, double* ay, double* az) {
  TraceRange trace_range("nbr_accel_ij");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (n_i == 0) return NBR_OK;
  if (!xi || !yi || !zi || !ax || !ay || !az || (want_force && !mi))
    return fail(c, NBR_ERR_INVALID_ARG, "NULL receiver array");
  if (n_j > 0 && (!xj || !yj || !zj || !mj)) return fail(c, NBR_ERR_INVALID_ARG, "NULL source array");
  if (!(eps2 >= 0.0) || !std::isfinite(eps2) || !std::isfinite(G))
    return fail(c, NBR_ERR_INVALID_ARG, "eps2 must be finite and >= 0, G finite");
  if (n_i > (size_t)1 << 31 || n_j > (size_t)1 << 31) return fail(c, NBR_ERR_INVALID_ARG, "size above 2^31");
  // small sets: one transfer each way, the check on the device
  const size_t total = (mi ? 4 : 3) * n_i + 4 * n_j;
  bool staged = n_j > 0 && stage_fits(total);
  if (staged) {
    cudaSetDevice(c->device);
    staged = stage_ready(c, total + 2);  // (3 n_i + 2 come back)
  }
  if (!staged &&
      (!finite_array(xi, n_i) || !finite_array(yi, n_i) || !finite_array(zi, n_i) ||
       (mi && !finite_array(mi, n_i)) || !finite_array(xj, n_j) || !finite_array(yj, n_j) ||
       !finite_array(zj, n_j) || !finite_array(mj, n_j)))
    return fail(c, NBR_ERR_NONFINITE, "input contains NaN or Inf");
  if (n_j == 0) {
    std::fill(ax, ax + n_i, 0.0); std::fill(ay, ay + n_i, 0.0); std::fill(az, az + n_i, 0.0);
    return NBR_OK;
  }
  cudaSetDevice(c->device);
  // Receivers live in ij.pos[0] (+ mass), sources in ij.pos[1] (+ j_mass).
  SysState& r = c->ij;
  const size_t nmax = std::max(n_i, n_j);
  cudaError_t e = with_room(c, [&] { return r.reserve(nmax); });
  if (e != cudaSuccess) return cuda_fail(c, e, "ij allocation");
  const long long npi = (long long)(((n_i + 1023) / 1024) * 1024);
  const long long npj = (long long)(((n_j + 1023) / 1024) * 1024);
  auto H = [&](double* d, const double* h, size_t n, long long np) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(d, h, n * sizeof(double), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess && (long long)n < np)
      e = cudaMemsetAsync(d + n, 0, (np - n) * sizeof(double), c->stream);
  };
  if (staged) {
    StageArrays sa{};
    size_t off = 0;
    auto put = [&](double* d, const double* h, size_t n, long long np) {
      if (!h) return;
      std::memcpy(c->h_stage.data() + off, h, n * sizeof(double));
      off += n;
      sa.dev[sa.count] = d;
      sa.n[sa.count] = (long long)n;
      sa.n_pad[sa.count++] = np;
    };
    put(r.pos[0][0], xi, n_i, npi); put(r.pos[0][1], yi, n_i, npi); put(r.pos[0][2], zi, n_i, npi);
    put(r.mass, mi, n_i, npi);
    put(r.pos[1][0], xj, n_j, npj); put(r.pos[1][1], yj, n_j, npj); put(r.pos[1][2], zj, n_j, npj);
    put(r.vel[0], mj, n_j, npj);  // source masses
    e = cudaMemcpyAsync(c->scr.red, c->h_stage.data(), total * sizeof(double),
                        cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_err + 1, 0, sizeof(int), c->stream);
    if (e == cudaSuccess) e = launch_stage_in(sa, c->scr.red, c->d_err + 1, c->stream);
  } else {
    H(r.pos[0][0], xi, n_i, npi); H(r.pos[0][1], yi, n_i, npi); H(r.pos[0][2], zi, n_i, npi);
    if (mi) H(r.mass, mi, n_i, npi);
    H(r.pos[1][0], xj, n_j, npj); H(r.pos[1][1], yj, n_j, npj); H(r.pos[1][2], zj, n_j, npj);
    H(r.vel[0], mj, n_j, npj);  // source masses
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "ij upload");
  const int ntiles = (int)((n_j + kTile - 1) / kTile);
  if (precision == kFP32C) {
    e = launch_kick_drift((long long)n_j, npj, r.pos[1][0], r.pos[1][1], r.pos[1][2], r.vel[0],
                          nullptr, nullptr, nullptr, 0.0, 0.0, nullptr, nullptr, nullptr, nullptr,
                          nullptr, nullptr, r.rec[1], r.org[1], c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "ij pack");
  }
  ForceConfig cfg = choose_config(c, precision, eps2, (long long)n_i, ntiles, false);
  if (cfg.ni == 3) cfg = choose_config_large(c, precision, eps2, (long long)n_i, ntiles);
  int rc = prepare_split(c, precision, cfg, npi);
  if (rc) return rc;
  IParticles ip{r.pos[0][0], r.pos[0][1], r.pos[0][2], r.mass, (long long)n_i};
  // (the source masses are staged in r.vel[0])
  JStream js{r.pos[1][0], r.pos[1][1], r.pos[1][2], r.vel[0], r.rec[1], r.org[1], ntiles, 0, -1};
  pipeline_params(js);
  Epilogue ep{};
  ep.mode = 0;
  ep.G = G;
  ep.ax = r.acc[0]; ep.ay = r.acc[1]; ep.az = r.acc[2];
  ep.want_force = want_force;
  ep.part = c->scr.part;
  ep.counters = c->scr.cnt;
  ep.n_pad = npi;
  ep.err = c->d_err;
  NBR_CHECKED_ONLY(
      ip.len = (long long)(r.cap + kRangeSlack); js.len = (long long)r.cap;
      ep.part_len = (long long)c->scr.part_cap; ep.cnt_len = (long long)c->scr.cnt_cap;)
  e = launch_force(precision, eps2, cfg, ip, js, ep, c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "ij force launch");
  if (staged) {
    const double* src[3] = {r.acc[0], r.acc[1], r.acc[2]};
    double* out[3] = {ax, ay, az};
    int err = 0, flags = 0;
    e = stage_download(c, 3, src, out, n_i, &err, &flags);
    if (e != cudaSuccess) return cuda_fail(c, e, "kernel execution");
    rc = device_error_status(c, err);
    if (rc) return rc;
    return flags ? fail(c, NBR_ERR_NONFINITE, "input contains NaN or Inf") : NBR_OK;
  }
  rc = check_device_error(c);
  if (rc) return rc;
  const size_t B = n_i * sizeof(double);
  e = cudaMemcpyAsync(ax, r.acc[0], B, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(ay, r.acc[1], B, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(az, r.acc[2], B, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? NBR_OK : cuda_fail(c, e, "ij download");
}

int nbr_potential(nbr_ctx* c, double G, double eps2, double* phi, double* U) {
  TraceRange trace_range("nbr_potential");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (!(eps2 >= 0.0) || !std::isfinite(eps2)) return fail(c, NBR_ERR_INVALID_ARG, "bad eps2");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  // phi goes to the (otherwise idle) acceleration x array only when requested.
  double* dphi = phi ? s.acc[0] : nullptr;
  if (phi) c->acc_ok = false;
  double *dU = nullptr, factor = 1.0;
  int rc = potential_system(c, G, eps2, dphi, 0, &dU, &factor);
  if (rc) return rc;
  double u = 0.0;
  cudaError_t e = cudaMemcpyAsync(&u, dU, sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess && phi)
    e = cudaMemcpyAsync(phi, dphi, s.n * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "potential");
  rc = check_device_error(c);
  if (rc) return rc;
  if (U) *U = factor * u;
  return NBR_OK;
}

int nbr_diagnostics(nbr_ctx* c, double G, double eps2, nbr_diag* out) {
  TraceRange trace_range("nbr_diagnostics");
  if (!c || !out) return fail(c, NBR_ERR_INVALID_ARG, "NULL argument");
  if (!(eps2 >= 0.0) || !std::isfinite(eps2)) return fail(c, NBR_ERR_INVALID_ARG, "bad eps2");
  if (c->sys.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  return diag_system(c, G, eps2, out);
}

int nbr_yoshida_coefficients(int order, double* cc, double* dd) {
  if (!cc || !dd) return 0;
  return yoshida(order, cc, dd);
}

int nbr_run(nbr_ctx* c, int precision, int scheme, int order, double dt, size_t steps, double G,
            double eps2, nbr_diag* diag, nbr_run_stats* stats) {
  TraceRange trace_range("nbr_run");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (scheme != NBR_KDK && scheme != NBR_DKD && scheme != NBR_EULER)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown scheme");
  if (scheme == NBR_KDK && order != 2) return fail(c, NBR_ERR_INVALID_ARG, "KDK is second order");
  double cc[16], dd[16];
  const int lf = scheme == NBR_DKD ? yoshida(order, cc, dd) : 2;
  if (lf == 0) return fail(c, NBR_ERR_INVALID_ARG, "order must be 2, 4, 6 or 8");
  if (!std::isfinite(dt) || !(eps2 >= 0.0) || !std::isfinite(eps2) || !std::isfinite(G))
    return fail(c, NBR_ERR_INVALID_ARG, "dt, G must be finite, eps2 finite and >= 0");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  int rc;
  if (diag) {
    rc = diag_system(c, G, eps2, &diag[0]);
    if (rc) return rc;
  }
  nbr_run_stats st{};
  if (steps > 0 && persistent_run_applies(c, precision, s.n)) {
    // small systems: every step in one cooperative launch
    const bool fsal = (scheme == NBR_KDK) && c->acc_ok && c->acc_prec == precision &&
                      c->acc_G == G && c->acc_eps2 == eps2;
    rc = run_persistent(c, precision, scheme, dt, steps, G, eps2, fsal, cc, dd, lf, &st);
    if (rc) {
      c->acc_ok = false;
      return rc;
    }
    c->acc_ok = scheme == NBR_KDK;
    c->acc_prec = precision;
    c->acc_G = G;
    c->acc_eps2 = eps2;
  } else if (steps > 0) {
    // Allocate everything the sequence needs before capture.
    ForceConfig cfg = choose_config(c, precision, eps2, (long long)s.n, s.ntiles);
    rc = prepare_split(c, precision, cfg, (long long)s.n_pad);
    if (rc) return rc;
    const bool fsal = (scheme == NBR_KDK) && c->acc_ok && c->acc_prec == precision &&
                      c->acc_G == G && c->acc_eps2 == eps2;
    // A repeated call (same arguments, starting state and buffers) replays the
    // graph captured last time instead of capturing and instantiating again.
    RunKey key;
    key.precision = precision; key.scheme = scheme; key.order = order;
    key.dt = dt; key.G = G; key.eps2 = eps2; key.steps = steps;
    key.n = s.n; key.cap = s.cap; key.fsal = fsal; key.cur = s.cur;
    key.rec_ok[0] = s.rec_ok[0]; key.rec_ok[1] = s.rec_ok[1];
    key.cfg = cfg;
    key.strips = uses_strips(precision, cfg, (long long)s.n);
    key.bands = forced_bands();
    {
      JStream probe{};
      pipeline_params(probe);
      key.wait_ns = probe.wait_ns;
      key.skip_tile = probe.skip_tile;
    }
    key.ptr[0] = s.pos[0][0]; key.ptr[1] = s.rec[0]; key.ptr[2] = s.vel[0];
    key.ptr[3] = c->scr.part; key.ptr[4] = c->scr.cnt; key.ptr[5] = c->d_err;
    key.ptr[6] = c->n3_order;
    // the matching graph to the front; none: the oldest makes room
    int at = 0;
    while (at < kRunGraphs - 1 && !(c->run_graph[at].exec && c->run_graph[at].key == key)) ++at;
    std::rotate(c->run_graph, c->run_graph + at, c->run_graph + at + 1);
    RunGraph& rg = c->run_graph[0];
    int kernels = 0;
    double evals = 0;
    cudaError_t e = cudaSuccess;
    if (rg.exec && rg.key == key) {
      s.cur = rg.cur_after;
      s.rec_ok[0] = rg.rec_after[0];
      s.rec_ok[1] = rg.rec_after[1];
      kernels = rg.kernels;
      evals = rg.evals;
    } else {
      rg.release();
      cudaGraph_t graph = nullptr;
      e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
      if (e != cudaSuccess) return cuda_fail(c, e, "begin capture");
      const int cur0 = s.cur;
      const bool rec0 = s.rec_ok[0], rec1 = s.rec_ok[1];
      rc = NBR_OK;
      const bool fp32 = precision == kFP32C && !uses_strips(precision, cfg, (long long)s.n);
      if (scheme == NBR_KDK) {
        if (fsal) {
          rc = kick_drift_system(c, fp32, 0.5 * dt, dt, true, &kernels);
        } else {
          rc = eval_system(c, precision, G, eps2, 1, 0.5 * dt, dt, 0, &kernels);
          evals += 1;
        }
        for (size_t k = 1; k < steps && rc == NBR_OK; ++k) {
          rc = eval_system(c, precision, G, eps2, 1, dt, dt, 0, &kernels);
          evals += 1;
        }
        if (rc == NBR_OK) {
          rc = eval_system(c, precision, G, eps2, 1, 0.5 * dt, 0.0, 0, &kernels);
          evals += 1;
        }
      } else if (scheme == NBR_EULER) {
        for (size_t k = 0; k < steps && rc == NBR_OK; ++k) {
          rc = eval_system(c, precision, G, eps2, 2, dt, dt, 0, &kernels);
          evals += 1;
        }
      } else {
        rc = kick_drift_system(c, fp32, 0.0, cc[0] * dt, false, &kernels);
        for (size_t k = 0; k < steps && rc == NBR_OK; ++k) {
          for (int sub = 0; sub < lf - 1 && rc == NBR_OK; ++sub) {
            double drift;
            if (sub < lf - 2) drift = cc[sub + 1];
            else drift = (k + 1 < steps) ? cc[lf - 1] + cc[0] : cc[lf - 1];
            rc = eval_system(c, precision, G, eps2, 1, dd[sub] * dt, drift * dt, 0, &kernels);
            evals += 1;
          }
        }
      }
      cudaError_t ee = cudaStreamEndCapture(c->stream, &graph);
      if (rc != NBR_OK || ee != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        s.cur = cur0;
        s.rec_ok[0] = rec0;
        s.rec_ok[1] = rec1;
        return rc != NBR_OK ? rc : cuda_fail(c, ee, "end capture");
      }
      long long kept = kernels;
      for (int k = 1; k < kRunGraphs; ++k) {
        kept += c->run_graph[k].kernels;
        if (k >= 2 && kept > kRunGraphKernels) c->run_graph[k].release();
      }
      cudaGraphExec_t exec = nullptr;
      e = with_room(c, [&] { return cudaGraphInstantiate(&exec, graph, 0); });
      cudaGraphDestroy(graph);
      if (e != cudaSuccess) {
        s.cur = cur0;
        s.rec_ok[0] = rec0;
        s.rec_ok[1] = rec1;
        return cuda_fail(c, e, "graph instantiate");
      }
      rg.exec = exec;
      rg.key = key;
      rg.cur_after = s.cur;
      rg.rec_after[0] = s.rec_ok[0];
      rg.rec_after[1] = s.rec_ok[1];
      rg.kernels = kernels;
      rg.evals = evals;
    }
    e = cudaEventRecord(c->ev0, c->stream);
    if (e == cudaSuccess) e = cudaGraphLaunch(rg.exec, c->stream);
    if (e == cudaSuccess) e = cudaEventRecord(c->ev1, c->stream);
    if (e != cudaSuccess) {
      rg.release();
      c->acc_ok = false;
      return cuda_fail(c, e, "graph launch");
    }
    rc = check_device_error(c);  // waits for the stream
    if (rc) {
      if (rc == NBR_ERR_CUDA) rg.release();
      c->acc_ok = false;
      return rc;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    st.gpu_ms = ms;
    st.kernels = kernels;
    st.force_evals = evals;
    st.pairs = evals * double(s.n) * double(s.n - 1);
    if (scheme == NBR_KDK) {
      c->acc_ok = true;
      c->acc_prec = precision;
      c->acc_G = G;
      c->acc_eps2 = eps2;
    } else {
      c->acc_ok = false;
    }
  }
  if (diag) {
    rc = diag_system(c, G, eps2, &diag[1]);
    if (rc) return rc;
  }
  if (stats) *stats = st;
  return NBR_OK;
}

int nbr_set_force_config(nbr_ctx* c, int precision, int ni, int warps, int split) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  if (ni == 0) {
    c->override_cfg[precision] = ForceConfig{0, 0, 0};
    return NBR_OK;
  }
  ForceConfig cfg{ni, warps, split < 1 ? 1 : split};
  if (!force_config_supported(precision, cfg))
    return fail(c, NBR_ERR_INVALID_ARG, "unsupported (ni, warps)");
  cfg.split = split;
  c->override_cfg[precision] = cfg;
  return NBR_OK;
}

int nbr_set_force_tiling(nbr_ctx* c, int precision, int tile, int unroll) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  ForceConfig cfg = c->override_cfg[precision];
  if (cfg.ni != 4 && cfg.ni != 8 && cfg.ni != kPersistNI)
    return fail(c, NBR_ERR_INVALID_ARG,
                "force a large-kernel (ni 4 or 8) or persistent (ni 2) configuration first");
  cfg.tile = tile;
  cfg.unroll = unroll;
  ForceConfig probe = cfg;
  if (probe.split < 1) probe.split = 1;
  if (!force_config_supported(precision, probe))
    return fail(c, NBR_ERR_INVALID_ARG, "unsupported (tile, unroll) for this configuration");
  c->override_cfg[precision] = cfg;
  return NBR_OK;
}

int nbr_get_force_tiling(nbr_ctx* c, int precision, double eps2, int* tile, int* unroll) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  ForceConfig cfg = choose_config(c, precision, eps2, (long long)s.n, s.ntiles);
  const bool large = cfg.ni == 4 || cfg.ni == 8;
  if (tile) *tile = large ? (cfg.tile > 0 ? cfg.tile : kDefaultTileJ) : 0;
  if (unroll) *unroll = large ? (cfg.unroll > 0 ? cfg.unroll : default_unroll(precision)) : 0;
  return NBR_OK;
}

int nbr_get_force_config(nbr_ctx* c, int precision, double eps2, int* ni, int* warps, int* split) {
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  ForceConfig cfg = choose_config(c, precision, eps2, (long long)s.n, s.ntiles);
  if (ni) *ni = cfg.ni;
  if (warps) *warps = cfg.warps;
  if (split) *split = cfg.split;
  return NBR_OK;
}

const char* nbr_tune_cache_path(void) {
  std::lock_guard<std::mutex> g(g_tune_mu);
  load_tune_locked();
  return g_tune_path.c_str();
}

int nbr_autotune(nbr_ctx* c, int precision, double eps2) {
  TraceRange trace_range("nbr_autotune");
  if (!c) return fail(nullptr, NBR_ERR_INVALID_ARG, "ctx is NULL");
  if (precision != NBR_FP64 && precision != NBR_FP32C)
    return fail(c, NBR_ERR_INVALID_ARG, "unknown precision");
  SysState& s = c->sys;
  if (s.n == 0) return fail(c, NBR_ERR_NO_SYSTEM, "no system uploaded");
  cudaSetDevice(c->device);
  const ForceConfig saved = c->override_cfg[precision];
  const int cand[][2] = {{4, 2}, {4, 4}, {4, 8}, {8, 2}, {8, 4}, {1, 2},
                         {1, 4}, {1, 8}, {3, 8}, {3, 16}};
  ForceConfig best{0, 0, 0};
  float best_ms = 1e30f;
  for (auto& cw : cand) {
    if (cw[0] == 1 && s.n > 65536) continue;  // the small-N kernel only competes on small systems
    // Newton-3 wherever it can be the default; two warps per row block only compete
    // on larger systems
    if (cw[0] == 3 && (long long)s.n < (cw[1] == kN3Warps ? kN3MinN : 8192)) continue;
    if (cw[0] == 3 && cw[1] == 16 && precision != kFP32C) continue;  // FP64 has one Newton-3 layout
    ForceConfig base{cw[0], cw[1], 1};
    const int s0 = auto_split(precision, eps2, base, (long long)s.n, s.ntiles, c->sms);
    const int splits[] = {std::max(1, s0 / 2), s0, s0 * 2};
    for (int sp : splits) {
      if (sp > s.ntiles) continue;
      c->override_cfg[precision] = ForceConfig{cw[0], cw[1], sp};
      float tot = 0.f;
      bool ok = true;
      for (int rep = 0; rep < 3 && ok; ++rep) {
        cudaEventRecord(c->ev0, c->stream);
        ok = eval_system(c, precision, 1.0, eps2, 0, 0.0, 0.0, 0, nullptr) == NBR_OK;
        cudaEventRecord(c->ev1, c->stream);
        ok = ok && check_device_error(c) == NBR_OK;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->ev0, c->ev1);
        if (rep > 0) tot += ms;  // first repetition warms up
      }
      if (ok && tot < best_ms) {
        best_ms = tot;
        best = ForceConfig{cw[0], cw[1], sp};
      }
    }
  }
  // The j-tile (sources per ring stage) and the unroll depth of the source
  // loop, for the large kernel's default configuration when it won.
  const bool large_default = (precision == kFP32C && best.ni == 8 && best.warps == 2) ||
                             (precision == kFP64 && best.ni == 4 && best.warps == 4);
  if (large_default) {
    for (int tj : {64, 128, 256})
      for (int u : {2, 4, 8}) {
        ForceConfig cand = best;
        cand.tile = tj;
        cand.unroll = u;
        if (!force_config_supported(precision, cand)) continue;
        c->override_cfg[precision] = cand;
        float tot = 0.f;
        bool ok = true;
        for (int rep = 0; rep < 3 && ok; ++rep) {
          cudaEventRecord(c->ev0, c->stream);
          ok = eval_system(c, precision, 1.0, eps2, 0, 0.0, 0.0, 0, nullptr) == NBR_OK;
          cudaEventRecord(c->ev1, c->stream);
          ok = ok && check_device_error(c) == NBR_OK;
          float ms = 0.f;
          cudaEventElapsedTime(&ms, c->ev0, c->ev1);
          if (rep > 0) tot += ms;
        }
        if (ok && tot < best_ms) {
          best_ms = tot;
          best = cand;
        }
      }
  }
  c->override_cfg[precision] = saved;
  c->acc_ok = false;
  if (best.ni == 0) return fail(c, NBR_ERR_CUDA, "no configuration ran");
  std::lock_guard<std::mutex> g(g_tune_mu);
  load_tune_locked();
  (*g_tune)[tune_key(precision, (long long)s.n, s.ntiles, eps2 == 0.0)] = best;
  save_tune_locked();
  return NBR_OK;
}

}  // extern "C"
