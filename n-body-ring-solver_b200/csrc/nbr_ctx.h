// nbr_ctx.h -- internal definition of nbr_ctx and its device state.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "nbr.h"
#include "nbr_kernels.cuh"

namespace nbr {

// Device state of one particle system (or of a batch of systems stored back to
// back).  Positions are double-buffered: a force evaluation reads buffer
// `cur` and its fused kick/drift epilogue writes buffer 1 - cur.  Every array
// holds n_pad entries (per-particle arrays kRangeSlack more); entries >= n are
// zero-mass padding at the origin.
// Zeroed entries allocated past n_pad in every per-particle array (see
// SysState::reserve).
constexpr size_t kRangeSlack = 1024;

struct SysState {
  size_t n = 0, n_pad = 0, cap = 0;
  int ntiles = 0;
  double* pos[2][3] = {{nullptr, nullptr, nullptr}, {nullptr, nullptr, nullptr}};
  double* vel[3] = {nullptr, nullptr, nullptr};
  double* acc[3] = {nullptr, nullptr, nullptr};
  double* mass = nullptr;
  float4* rec[2] = {nullptr, nullptr};     // FP32C source records of each buffer
  double4* org[2] = {nullptr, nullptr};    // FP64 tile origins of each buffer
  int cur = 0;
  bool rec_ok[2] = {false, false};

  cudaError_t reserve(size_t n);
  cudaError_t clear_padding(cudaStream_t st);
  void release();
};

// Scratch reused across calls: split partial sums, split arrival counters,
// diagnostic partial sums.
struct Scratch {
  double* part = nullptr;
  size_t part_cap = 0;
  unsigned* cnt = nullptr;
  size_t cnt_cap = 0;
  double* red = nullptr;
  size_t red_cap = 0;

  cudaError_t need_part(size_t doubles);
  cudaError_t need_counters(size_t count);
  cudaError_t need_red(size_t doubles);
  void release();
};

// Batched independent systems (nbr_batch_*).  Each system is padded to whole
// tiles, so a tile never mixes systems.
struct BatchState {
  SysState s;                        // all systems' particles (padded layout)
  size_t nsys = 0;
  size_t n_real = 0;                 // sum of the real sizes
  std::vector<size_t> off;           // real offsets (host), nsys + 1
  std::vector<long long> poff;       // padded offsets (host), nsys + 1
  long long* d_poff = nullptr;       // padded offsets (device), nsys + 1
  int* d_nreal = nullptr;            // real size of each system (device)
  long long* d_off = nullptr;        // real offsets (device), nsys + 1
  double* d_flat = nullptr;          // one array, or six small ones, without padding (first download)
  int* d_sys_of_tile = nullptr;      // system index of every padded tile
  // Work queues of (system | kWideItem flag, first receiver tile), cost
  // ordered: [0] one-tile items only, [1] two-tile items where a system has
  // two tiles left.
  int2* d_items[2] = {nullptr, nullptr};
  int n_items[2] = {0, 0};
  // Newton-3 work per precision ([0] FP64: one-tile row blocks of the systems
  // of two tiles or more, the others' items as in list 0; [1] FP32C: two-tile
  // row blocks of the systems of three tiles or more, the others' items as in
  // list 1): the queue of (system | kN3Item, row block) and other items, the
  // Newton-3 systems' tiles (system, local tile) for the epilogue kernel, each
  // system's first reaction slot (-1: none), the slot count, and the slots
  // [slots][3][128] (allocated at first use).
  struct N3List {
    int2* d_items = nullptr;
    int n_items = 0;
    double cost = 0.0, cost_max = 0.0;  // of all items and of the largest one
    int2* d_tiles = nullptr;
    int n_tiles = 0;
    long long* d_rea_off = nullptr;
    long long slots = 0;
    double* d_rea = nullptr;
  };
  N3List n3[2];
  double* d_act = nullptr;           // Newton-3 action sums [3][n_pad] (at first use)
  int max_ns = 0;                    // largest system
  unsigned* d_head = nullptr;        // work-queue heads
  double* d_red = nullptr;           // per-system diagnostic sums
  bool acc_ok = false;
  int acc_prec = 0;
  double acc_G = 0.0, acc_eps2 = 0.0;
  double pairs_per_eval = 0.0;
  // Kernel configuration per precision: wide items, resident CTAs per SM
  // (0: the occupancy limit); chosen from the autotune cache or the default
  // at first use.
  bool cfg_ok[2] = {false, false};
  int wide[2] = {1, 1};
  int per_sm[2] = {0, 0};
  int occ[2][2][3] = {};              // occupancy limit per (precision, eps == 0, wide)

  void release();
};

// An NVTX range around a public call (visible to Nsight tools; a no-op when
// none is attached).
struct TraceRange {
  explicit TraceRange(const char* name) { nvtxRangePushA(name); }
  ~TraceRange() { nvtxRangePop(); }
  TraceRange(const TraceRange&) = delete;
  TraceRange& operator=(const TraceRange&) = delete;
};

// Autotune cache (a JSON file shared by the processes on a host).
bool tune_get(const std::string& key, ForceConfig* out);
void tune_put(const std::string& key, const ForceConfig& cfg);

int fail(nbr_ctx* c, int code, const std::string& msg);
int cuda_fail(nbr_ctx* c, cudaError_t e, const char* where);
cudaError_t dalloc(void** p, size_t bytes);
void dfree(void* p);
// Gives back what a context keeps for speed alone: the graphs of nbr_run and the
// batch's copy without padding.  False if there was nothing.
bool give_back(nbr_ctx* c);
// alloc(), and where it finds no room once more with that given back.
template <class F>
cudaError_t with_room(nbr_ctx* c, F alloc) {
  cudaError_t e = alloc();
  if (e == cudaErrorMemoryAllocation && give_back(c)) {
    cudaGetLastError();
    e = alloc();
  }
  return e;
}
bool finite_array(const double* a, size_t n);
int check_device_error(nbr_ctx* c);
// The status of a device error word already on the host (0: NBR_OK).
int device_error_status(nbr_ctx* c, int h);
// Arrays of up to kStageBytes in all travel between the host and the device in
// one transfer, packed in Scratch::red on the device and in nbr_ctx::h_stage on
// the host.
constexpr size_t kStageBytes = 1 << 20;
inline bool stage_fits(size_t doubles) { return doubles * sizeof(double) <= kStageBytes; }
// Whether both sides hold `doubles` (allocated here where they do not): a call
// whose staging finds no memory makes its transfers one by one.
bool stage_ready(nbr_ctx* c, size_t doubles);
// The arrays of a, packed at dst (device scratch), into c->h_stage, and the
// device error block's first two words into words; waits for the stream.
cudaError_t stage_fetch(nbr_ctx* c, const StageArrays& a, double* dst, int words[2]);
// count arrays of n doubles each into out[k] (null: left out), unless *err (the
// device error word) or *flags (the input flags) is set.  err null: whatever the
// error word, which stays for the next call that checks it.
cudaError_t stage_download(nbr_ctx* c, int count, const double* const* src, double* const* out,
                           size_t n, int* err, int* flags = nullptr);
// Bounded-wait limit and tile-skip test hook from the environment.
void pipeline_params(JStream& js);
// The persistent small-system run (nbr_persist.cu): whether it serves an
// nbr_run of this system, and the run itself (the schedule of nbr_run's
// launch sequence; cc/dd/lf the Yoshida tables for DKD).
bool persistent_run_applies(nbr_ctx* c, int precision, size_t n);
int run_persistent(nbr_ctx* c, int precision, int scheme, double dt, size_t steps, double G,
                   double eps2, bool fsal, const double* cc, const double* dd, int lf,
                   nbr_run_stats* st);

}  // namespace nbr

namespace nbr {
// Identity of a captured nbr_run launch sequence: the call's arguments, the
// host-side state it starts from and every device address it bakes in.
struct RunKey {
  int precision = -1, scheme = -1, order = 0;
  double dt = 0.0, G = 0.0, eps2 = 0.0;
  size_t steps = 0, n = 0, cap = 0;
  bool fsal = false;
  int cur = 0;
  bool rec_ok[2] = {false, false};
  ForceConfig cfg{0, 0, 0};
  unsigned long long wait_ns = 0;
  int skip_tile = -1;
  bool strips = false;  // Newton-3: strips (else the CTA grid), and the launches
  int bands = 0;        // forced by the test hook
  const void* ptr[7] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  bool operator==(const RunKey& o) const;
};
// What decides the kernels of an evaluation in strips (but for the softening).
struct StripKernel {
  int precision = -1, ni = 0;
  long long n = 0;
  bool operator==(const StripKernel& o) const {
    return precision == o.precision && ni == o.ni && n == o.n;
  }
};
// A captured nbr_run graph, replayed while the key matches.  The last two stay; the
// two before them only while all hold at most kRunGraphKernels launches (2.5 KB of
// device and 6.6 KB of host memory each).
constexpr int kRunGraphs = 4;
constexpr int kRunGraphKernels = 16384;
struct RunGraph {
  cudaGraphExec_t exec = nullptr;
  RunKey key;
  int cur_after = 0;
  bool rec_after[2] = {false, false};
  int kernels = 0;
  double evals = 0.0;
  void release();
};
}  // namespace nbr

struct nbr_ctx {
  int device = 0;
  int sms = 148;
  bool coop = false;       // the device supports cooperative launches
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::string err;
  nbr::SysState sys;       // the uploaded system
  nbr::SysState ij;        // scratch for nbr_accel_ij
  nbr::Scratch scr;
  nbr::BatchState bat;
  int* d_err = nullptr;    // device error word (nbr::kErr*)
  // First-same-as-last: sys.acc holds G-scaled accelerations of the current
  // positions for (acc_prec, acc_G, acc_eps2).
  bool acc_ok = false;
  int acc_prec = 0;
  double acc_G = 0.0, acc_eps2 = 0.0;
  nbr::ForceConfig override_cfg[2] = {{0, 0, 0}, {0, 0, 0}};
  // The last graphs of nbr_run, most recent first: a run of an odd number of
  // position updates ends in the other buffer, so a repeated call alternates
  // between two.
  nbr::RunGraph run_graph[nbr::kRunGraphs];
  std::vector<double> h_stage;
  // Most scratch of an evaluation in strips that runs as one launch, lowered
  // when that much could not be allocated, until the next upload.
  long long strip_single = nbr::kN3SingleMaxDoubles;
  nbr::StripKernel strip_ready;  // the last kernels whose attributes were set
  // The last persistent launch configuration whose attributes were set, and its
  // resident CTAs per SM.
  const void* persist_fn = nullptr;
  size_t persist_smem = 0;
  int persist_per_sm = 0;
  // Launch order of the whole-system Newton-3 CTA grid (longest CTA first) for
  // n3_order_nb blocks, then its inverse; written before any graph capture
  // (n3_order_prepare, the only writer), read by the pair and reduce kernels.
  int* n3_order = nullptr;
  long long n3_order_cap = 0;    // ints allocated
  long long n3_order_nb = -1;    // blocks the table holds the order of
};
