// Host-side internals shared by the translation units of the C ABI:
// bfe_plan.cpp (matrix conversion, operator formation, plan building),
// bfe_run.cpp (the time loop of bfe_run / bfe_run_batched / bfe_run_device /
// bfe_run_field / bfe_run_v5) and bfe_adjoint_host.cpp (bfe_adjoint_gradient).
#pragma once
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <new>
#include <numeric>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>

#include "bfe_internal.h"
#include "../../include/bfe_gb300.h"

namespace bfe_host {

// Message returned by bfe_last_error() on the calling thread.
extern thread_local std::string g_last_error;

// Record a formatted message for bfe_last_error() and return code.
int fail(int code, const char* fmt, ...);

// Host threads for plan building: the machine's hardware threads (at most
// 64), and at most one per `grain` work items.
inline int plan_threads(int64_t items, int64_t grain) {
  const unsigned hc = std::thread::hardware_concurrency();
  int64_t t = std::min<int64_t>(hc ? hc : 1, 64);
  return (int)std::max<int64_t>(1, std::min<int64_t>(t, items / std::max<int64_t>(grain, 1)));
}

// Runs f(t, begin, end) for the nt even chunks of [0, items), chunk t on a
// thread of its own (on the calling thread if a thread cannot be started).
// No exception leaves a worker: false if any chunk threw (allocation).
template <typename F>
bool parallel_chunks(int64_t items, int nt, F&& f) {
  std::atomic<bool> ok{true};
  auto run = [&](int t) {
    try {
      f(t, items * t / nt, items * (t + 1) / nt);
    } catch (...) {
      ok = false;
    }
  };
  std::vector<std::thread> th;
  int started = 1;
  try {
    th.reserve(nt);
    for (; started < nt; ++started) th.emplace_back(run, started);
  } catch (...) {
  }
  run(0);
  for (int t = started; t < nt; ++t) run(t);
  for (auto& x : th) x.join();
  return ok;
}

#define CUDA_TRY(expr)                                                                \
  do {                                                                                \
    cudaError_t e_ = (expr);                                                          \
    if (e_ != cudaSuccess)                                                            \
      return fail(e_ == cudaErrorMemoryAllocation ? BFE_ERR_OOM : BFE_ERR_CUDA,       \
                  "%s failed: %s", #expr, cudaGetErrorString(e_));                    \
  } while (0)

// Row-compressed FP64 matrix used during plan construction.
struct Csr {
  int64_t n = 0, m = 0;
  std::vector<int64_t> ptr, idx;
  std::vector<double> val;
};

// Copy a bfe_sparse view into sorted, duplicate-summed CSR.
int to_csr(const bfe_sparse* A, const char* name, Csr& out);
double max_abs(const Csr& A);

template <typename T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  ~DevBuf() { if (p) cudaFree(p); }
  cudaError_t alloc(size_t count) {
    if (p) { cudaFree(p); p = nullptr; }
    n = count;
    if (count == 0) return cudaSuccess;
    return cudaMalloc(&p, count * sizeof(T));
  }
  cudaError_t upload(const std::vector<T>& h) {
    cudaError_t e = alloc(h.size());
    if (e != cudaSuccess || h.empty()) return e;
    return cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
  }
};

size_t elem_size(int prec);

template <typename T>
inline void push_val(std::vector<unsigned char>& buf, double v) {
  T x = (T)v;
  const unsigned char* b = reinterpret_cast<const unsigned char*>(&x);
  buf.insert(buf.end(), b, b + sizeof(T));
}

// count doubles converted to T, as bytes
template <typename T>
inline std::vector<unsigned char> cast_bytes(const double* v, int64_t count) {
  std::vector<T> x(v, v + count);
  std::vector<unsigned char> b((size_t)count * sizeof(T));
  if (count) std::memcpy(b.data(), x.data(), b.size());
  return b;
}

std::vector<unsigned char> cast_bytes(int prec, const double* v, int64_t count);
int upload_bytes(DevBuf<unsigned char>& d, const std::vector<unsigned char>& h);

// Partition of a plan's operator for the one-source march that stays on the
// chip (bfe_onchip_host.cpp), built on the first run that can use it.
struct Onchip {
  int state = 0;                    // 0: not built, 1: usable, -1: does not fit
  bfe::OnchipArgs args{};
  std::vector<int32_t> part_slice;  // n_parts + 1
  std::vector<int64_t> need;        // shared memory of each part without forcing and cached operator
  std::vector<int32_t> op_bytes;    // and of its operator
  uint32_t next_tag = 0;
  DevBuf<int32_t> d_part, d_off, d_word, d_bytes, d_cnt, d_halo, d_vptr, d_vhalo;
  DevBuf<uint16_t> flags, order, z_lcol;
  DevBuf<unsigned char> blocks, xch, xchv;
  DevBuf<int32_t> row_of;           // tiled parts: the plan's row of each row here, and its inverse
  std::vector<int32_t> place;
  DevBuf<uint4> xchm;               // exchange words of marches with several sources
  std::vector<int32_t> halo_cnt;
  DevBuf<ushort4> lref;
  int64_t device_bytes() const;
};

}  // namespace bfe_host

struct bfe_plan {
  bfe_plan() = default;
  bfe_plan(const bfe_plan&) = delete;
  ~bfe_plan() { if (stream) cudaStreamDestroy(stream); }
  int64_t n = 0;
  int32_t mode = 0, prec = 0;
  double dt = 0;
  int device = 0;
  cudaStream_t stream = nullptr;
  // operator
  int32_t n_slices = 0;
  int32_t max_slice_entries = 0;
  bfe_host::DevBuf<int32_t> slice_ptr;
  bfe_host::DevBuf<uint32_t> col;
  bfe_host::DevBuf<unsigned char> val;        // double or float
  bfe_host::DevBuf<unsigned char> rowc;       // double or float
  std::vector<int32_t> h_slice_ptr;
  std::unique_ptr<bfe_host::Onchip> onchip{new bfe_host::Onchip()};
  std::unique_ptr<bfe_host::Onchip> tiled{new bfe_host::Onchip()};   // several sources, 2D: parts cut as tiles
  std::vector<uint32_t> h_base;     // node-block base per row
  std::vector<double> h_acoef;      // forcing coefficient per row (diagonal of A)
  // interface correction
  int32_t n_int = 0;
  int32_t int_base_prev = 1;
  std::vector<int32_t> h_int_row;
  bfe_host::DevBuf<int32_t> int_row, z_ptr, z_col;
  bfe_host::DevBuf<unsigned char> z_val;
  std::vector<int32_t> h_z_ptr, h_z_col;
  // statistics
  int64_t nnz_operator = 0;         // stored (unpadded) entries
  int64_t nnz_padded = 0;
  int64_t n_direct_rows = 0;
  bool timing = false;
  double time_limit_s = 0.0;        // wall-clock limit of a run (0 = none)
  int32_t march_fault = 0;          // BFE_MARCH_FAULT_*, for tests
  int64_t partitions_built = 0;     // on-chip partitions begun
  bool packed_on_gpu = false;       // the sliced-ELL operator (bfe_pack.cu)
  int64_t steps_marched = 0;        // towards the first (onchip_due)
  int32_t mid_neighbours = 0, mid_last = 0;   // of the first group's middle node: neighbours, first row of the last
  bfe_host::DevBuf<int> d_flag;     // non-finite flag of the last run, and a march's wait-ran-out flag
  bfe_stats last{};
  // autotuned batched-kernel variant per R (chosen on the first run with that R)
  std::map<int64_t, int> variant_of_R;
  int32_t n_nodes = 0;              // nodes given by dof_node / dof_type
  // group block-sparse operator (FP32 difference form)
  bool have_groups = false;
  bfe::GroupArgs groups{};
  bfe_host::DevBuf<int32_t> g_nptr[bfe::kMaxGroups], g_nrow[bfe::kMaxGroups];
  bfe_host::DevBuf<int4> g_rec[bfe::kMaxGroups];
  bfe_host::DevBuf<float> g_coef[bfe::kMaxGroups];
  bfe_host::DevBuf<double> g_coef64[bfe::kMaxGroups];
  // BFE_MODE_V5: K, C (FP64 CSR) and the lumped mass, for the
  // prescribed-displacement rows of bfe_run_v5
  bfe_host::Csr hK, hC;
  std::vector<double> h_m;
};

namespace bfe_host {

// ---------------------------------------------------------------------------
// Run machinery (bfe_run.cpp) shared with the adjoint.

struct ForceEntry {
  int32_t row, rhs, sig;
  double w;
};

// Host lists behind V5Args: rows and slots of the listed entries, K and C
// rows of the slots.
struct V5Lists {
  std::vector<int32_t> ent_row, ent_slot, kp, kc, cp, cc, slot_row;
  std::vector<double> kv, cv;
  bool corrections = false;        // rows coupled by C to a prescribed DOF
};

// Whether the launch of a later piece of an on-chip march is to be refused
// (bfe_plan_set_march_fault).
inline bool refuse_piece(const bfe_plan* pl, bool later) { return later && pl->march_fault == BFE_MARCH_FAULT_LAUNCH; }

struct RunSpec {
  int64_t R = 1, n_t = 0, ti_start = 0;
  std::vector<ForceEntry> frc;     // one per (row, rhs) after last-wins dedupe
  int64_t n_sig = 0;
  const double* d_sig64 = nullptr; // device [n_t][n_sig]
  std::vector<int64_t> hist_idx;
  double* d_hist = nullptr;        // device [q][n_t][R] column-major (slot fastest)
  int64_t every_n = 0;             // R == 1 only
  int32_t field_is_vel = 1;
  double* d_fld = nullptr;
  std::vector<double>* fld_time = nullptr;
  const double* time = nullptr;    // host time samples (for frame times)
  const bfe::FieldArgs* field = nullptr;  // frames reduced to element values (bfe_run_field)
  double* d_el = nullptr;          // device n_el x n_frames
  const bfe::V5Args* v5 = nullptr; // prescribed-displacement rows (bfe_run_v5)
  const V5Lists* v5_lists = nullptr;
  double* d_ud[2] = {nullptr, nullptr};
};

// Device arrays of one run (forcing, monitors, per-row info, FP32 signals,
// interface staging) and the StepArgs template; the states are set per step.
struct RunArrays {
  DevBuf<int32_t> frow, frhs, fsig, mrow, mslot;
  DevBuf<unsigned char> fcoef, vint;
  DevBuf<uint32_t> info;
  DevBuf<float> sig32;
};

int prepare_run(bfe_plan* pl, std::vector<ForceEntry>& frc, const std::vector<int64_t>& hist_idx,
                int64_t R, int64_t n_t, int64_t n_sig, const double* d_sig64, double* d_hist,
                cudaStream_t st, RunArrays& ra, bfe::StepArgs& a);
int execute(bfe_plan* pl, RunSpec& rs, cudaStream_t st);
// Builds the plan's on-chip partition if it has none yet (state says whether
// it is usable afterwards); with the run's forced rows, its shared memory and
// thread count are set. false: this run does not fit.
int onchip_prepare(bfe_plan* pl, cudaStream_t st);
bool onchip_fit(bfe_plan* pl, const std::vector<ForceEntry>& frc, const std::vector<int64_t>& v5_bytes,
                const std::vector<int32_t>& v5_count, bfe::OnchipArgs& o);
// Shared memory, threads and exchange buffer of a march with several sources
// (a: its forcing, monitors and padded R). false: it does not fit, or the step
// kernels (against_graph: replayed from a graph) are faster.
bool onchip_multi_fit(bfe_plan* pl, Onchip& oc, const bfe::StepArgs& a, const std::vector<int32_t>& frc_rows,
                      const std::vector<int32_t>& mon_rows, bool against_graph, cudaStream_t st, bfe::OnchipArgs& o);
// The partition a march with several sources uses, built at its first use:
// tiles where the model has them, else the one-source partition; nullptr: none.
Onchip* onchip_for_several(bfe_plan* pl, cudaStream_t st);
// The forced and monitored rows of such a march in its partition's order, and
// (tiles) as a's device lists.
struct MultiLists {
  DevBuf<int32_t> ints;
  DevBuf<unsigned char> coef;
  std::vector<int32_t> forced, frows, mrows, mslots;
};
void onchip_multi_rows(const Onchip& oc, const std::vector<ForceEntry>& frc, const std::vector<int64_t>& hist_idx,
                       MultiLists& L);
int onchip_multi_lists(const bfe_plan* pl, const Onchip& oc, const std::vector<ForceEntry>& frc, MultiLists& L,
                       bfe::StepArgs& a);
// Frees a partition whose march gave up (the stream is idle) and keeps the plan
// from building it again.
void onchip_give_up(bfe_plan* pl, const Onchip* oc);
// BFE_MARCH_FAULT_WAIT: one row of the partition is published no more.
int onchip_meet_fault(const bfe_plan* pl, Onchip& oc);
// Whether the plan has decided about its partition, or has marched enough steps
// with these to build it.
bool onchip_due(bfe_plan* pl, int64_t steps, bool several);
// Whether that is worth building the partition for.
bool onchip_multi_may_fit(const bfe_plan* pl, int64_t R, bool against_graph);
// Step numbers for n steps that the exchange buffers do not hold yet.
int onchip_tags(Onchip& oc, int64_t n, cudaStream_t st, uint32_t& tag0);
// Device data of a run's prescribed displacements for the on-chip march, and
// what each part needs for them; fits = false: they do not fit the form.
struct OnchipV5 {
  DevBuf<int32_t> ptr, ent, row, kptr;
  DevBuf<uint16_t> kcol;
  DevBuf<double> kval, c;
  std::vector<int64_t> bytes;
  std::vector<int32_t> count;
};
int onchip_v5(bfe_plan* pl, const V5Lists& L, OnchipV5& d, bool& fits);
bool outputs_valid(int rc);
int64_t first_nonzero_column(const double* frcs, int64_t rows, int64_t n_t, int64_t R);
int check_time(bfe_plan* pl, int64_t n_t, const double* time);
int build_forcing(bfe_plan* pl, int64_t R, int64_t p, const int64_t* frc_idx, int64_t frc_rows,
                  std::vector<ForceEntry>& out);
int run_one(bfe_plan* plan, const bfe_field* field, int64_t n_t, const double* time,
            int64_t p, const int64_t* frc_idx, int64_t frc_rows, const double* frcs,
            int64_t q, const int64_t* hist_idx, int64_t every_n, int32_t field_is_vel,
            double* hist_out, double* fld_out, double* fld_time_out);

}  // namespace bfe_host
