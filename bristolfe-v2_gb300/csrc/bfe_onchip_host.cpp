// Host side of the one-source march that stays on the chip (bfe_onchip.cu):
// cutting a plan's rows into one part per SM, the device data of the parts,
// and what a run needs of shared memory and threads.
#include "bfe_host.h"

using namespace bfe_host;

namespace {

constexpr int64_t kSmemLimit = bfe::kOnchipSmem;
// Slices per part below which a part is not split further: one warp of rows
// for each of an SM's four schedulers.
constexpr int64_t kMinSlices = 4;
// Largest operator, as blocks: three quarters of the 129 MB L2. Above it the
// streamed chunks come from HBM as the step kernels' operator does: FP64
// bricks of 202,878 DOF (163 MB) took 39 us per step against 35.5 with one
// launch per step. FP64, whose blocks are known before they are built, stops
// a little lower. Us per step on chip / step kernels (MB of 2^20): coupled
// 592,202 DOF (57 MB) 14.8 / 18.0, 696,719 (67) 18.0 / 20.2, plate of 642,402 DOF (78)
// 18.0 / 19.4, bricks of 122,034 DOF (83) 25.5 / 27.4, coupled 961,641 DOF (92) 27.6 /
// 25.6.
constexpr int64_t kMaxOperator = (int64_t)96 << 20, kMaxOperator64 = (int64_t)88 << 20;

// FP32 rows of many entries (3D) whose blocks alone exceed the SMs' shared
// memory (35 MB) stream too much of them: the step kernel is faster as long as
// its operator, 8 bytes an entry, comes from L2. Us per step on chip / step
// kernels, bricks: 73,872 DOF (blocks of 24 MB) 6.6 / 10.9, 100,800 DOF (34) 7.7
// / 11.5, 105,903 DOF (35.4) 11.9 / 11.1, 122,034 DOF (39; 65 MB of entries) 12.6
// / 11.2, 133,584 DOF (76 MB) 13.1 / 14.5, 202,878 DOF 14.7 / 29.0. Rows of a few
// entries gain either way: coupled 961,641 DOF (50 MB) 10.8 / 17.
constexpr int64_t kStepOperator = (int64_t)70 << 20, kWideRow = 32;

inline int64_t align2(int64_t x) { return (x + 1) & ~(int64_t)1; }

// Lists of the interface correction: which interface values each part reads
// from others (made symmetric), which are read, local columns of Z.
struct InterfaceLists {
  std::vector<int32_t> ptr, list;
  std::vector<uint16_t> z_lcol;
  std::vector<uint8_t> exported;
  std::vector<int32_t> first;        // first interface number of each part (n_parts + 1)
};

bool interface_lists(const bfe_plan* pl, const std::vector<int32_t>& part, InterfaceLists& L) {
  const int P = (int)part.size() - 1;
  const int32_t ni = pl->n_int;
  L.first.resize(P + 1);
  for (int p = 0; p <= P; ++p)
    L.first[p] = (int32_t)(std::lower_bound(pl->h_int_row.begin(), pl->h_int_row.end(), part[p] * bfe::kSlice) -
                           pl->h_int_row.begin());
  std::vector<int32_t> owner(ni);
  for (int p = 0; p < P; ++p)
    for (int32_t t = L.first[p]; t < L.first[p + 1]; ++t) owner[t] = p;
  std::vector<std::vector<int32_t>> need(P);
  std::vector<char> adj((size_t)P * P, 0);
  std::vector<int32_t> at(ni, -1);   // the last part that noted a column, later its local number there
  for (int p = 0; p < P; ++p) {
    for (int32_t e = pl->h_z_ptr[L.first[p]]; e < pl->h_z_ptr[L.first[p + 1]]; ++e) {
      const int32_t c = pl->h_z_col[e];
      if (owner[c] == p || at[c] == p) continue;
      at[c] = p;
      need[p].push_back(c);
      adj[(size_t)p * P + owner[c]] = 1;
    }
    std::sort(need[p].begin(), need[p].end());
  }
  std::vector<size_t> real(P);
  for (int p = 0; p < P; ++p) real[p] = need[p].size();
  for (int p = 0; p < P; ++p)
    for (int q = 0; q < P; ++q)
      if (adj[(size_t)p * P + q] && !adj[(size_t)q * P + p]) need[q].push_back(L.first[p]);
  L.exported.assign(ni, 0);
  L.ptr.assign(1, 0);
  L.z_lcol.assign(pl->h_z_col.size(), 0);
  for (int p = 0; p < P; ++p) {
    for (int32_t c : need[p]) L.exported[c] = 1;
    L.list.insert(L.list.end(), need[p].begin(), need[p].end());
    L.ptr.push_back((int32_t)L.list.size());
    const int32_t own = L.first[p + 1] - L.first[p];
    if (own + (int64_t)need[p].size() > 65535) return false;
    for (size_t k = 0; k < real[p]; ++k) at[need[p][k]] = own + (int32_t)k;
    for (int32_t e = pl->h_z_ptr[L.first[p]]; e < pl->h_z_ptr[L.first[p + 1]]; ++e) {
      const int32_t c = pl->h_z_col[e];
      L.z_lcol[e] = (uint16_t)(owner[c] == p ? c - L.first[p] : at[c]);
    }
  }
  return true;
}

}  // namespace

namespace {

// The operator the parts are cut from: the plan's, or the same in tile order.
struct PartView {
  const std::vector<int32_t>* sp;    // slice offsets, here and on the device
  const int32_t* slice_ptr;
  const uint32_t* col;
  const void *val, *rowc;
};

// How P parts of S slices are cut from M mesh columns of len nodes: px strips of
// py parts, and the halo nodes of the largest. A row costs about twice what a
// halo row does. py = 1: tiles are not worth it.
struct TileCut {
  int64_t px, py, halo;
};
TileCut tile_cut(int64_t S, int64_t P, int64_t M, double len, int64_t bs) {
  auto halo = [&](int64_t px, int64_t py) {
    const double w = (double)M / (double)px, h = len / (double)py;
    return (px > 1 ? 2 * h : 0) + (py > 1 ? 2 * w : 0) + 4;
  };
  auto cost = [&](int64_t px, int64_t py) {
    return (double)((S + px * py - 1) / (px * py) * bfe::kSlice) + 0.5 * halo(px, py) * (double)bs;
  };
  int64_t px = P, py = 1;
  for (int64_t x = 1; x <= std::min(P, M); ++x)
    for (int64_t y = 1; x * y <= P && y <= (int64_t)len; ++y)
      if (cost(x, y) < cost(px, py)) px = x, py = y;
  if (cost(px, py) > 0.9 * cost(P, 1)) px = P, py = 1;
  const int64_t w = (M + px - 1) / px, h = (int64_t)std::ceil(len / (double)py);
  return {px, py, (px > 1 ? 2 * h : 0) + (py > 1 ? 2 * w : 0) + 4};
}

// Tiles for a 2D model. Contiguous ranges of the caller's node order (column
// by column) are strips of a mesh column or two when a part is small, and then
// all of their rows are read by other parts. Here the nodes are put in an
// order whose contiguous ranges are tiles: the columns are the runs of
// consecutive nodes that are neighbours; a node's height is its place in its
// run, levelled to the run on its left by one neighbour there; the columns are
// cut into px strips, and a strip's nodes sorted by height and cut into py
// parts. Any order is correct; models that are not so numbered only gain less.
// perm: row of the plan of each row in tile order. False: not worth it.
bool tile_order(const bfe_plan* pl, int64_t P, std::vector<int32_t>& perm, std::vector<int32_t>& parts) {
  const int64_t bs = pl->groups.bs[0], N = pl->groups.n_nodes[0], S = pl->n_slices;
  if (!pl->have_groups || pl->groups.n_groups != 1 || bs > 2 || N * bs != pl->n) return false;
  std::vector<int32_t> nptr(N + 1);
  if (cudaMemcpy(nptr.data(), pl->g_nptr[0].p, nptr.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
  std::vector<int32_t> nrow(nptr[N]);
  if (cudaMemcpy(nrow.data(), pl->g_nrow[0].p, nrow.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
  std::vector<int32_t> start, run(N), level;
  for (int64_t q = 0; q < N; ++q) {
    const auto b = nrow.begin() + nptr[q], e = nrow.begin() + nptr[q + 1];
    if (q == 0 || !std::binary_search(b, e, (int32_t)((q - 1) * bs))) start.push_back((int32_t)q);
    run[q] = (int32_t)start.size() - 1;
  }
  const int64_t M = (int64_t)start.size();
  level.assign(M, 0);
  for (int64_t r = 1; r < M; ++r) {
    const int64_t q0 = start[r], q1 = r + 1 < M ? start[r + 1] : N;
    for (int64_t d = 0; d < q1 - q0; ++d) {
      // a node near the middle of the run with neighbours on both sides of its left one
      const int64_t q = q0 + ((q1 - q0) / 2 + d) % (q1 - q0);
      int64_t hi = -1, lo = 0;
      for (int32_t e = nptr[q]; e < nptr[q + 1] && nrow[e] / bs < q0; ++e) {
        const int64_t j = nrow[e] / bs;
        if (hi < 0 || run[j] != run[hi]) lo = j;
        hi = j;
      }
      if (hi - lo != 2) continue;
      level[r] = (int32_t)(level[run[hi]] + (lo + 1 - start[run[hi]]) - (q - q0));
      break;
    }
  }
  const TileCut cut = tile_cut(S, P, M, (double)N / (double)M, bs);
  const int64_t px = cut.px, py = cut.py;
  if (py == 1) return false;
  perm.resize(pl->n);
  parts.assign(1, 0);
  std::vector<int32_t> first, node;
  for (int64_t x = 0; x < px; ++x) {
    const int64_t s0 = S * x / px, s1 = S * (x + 1) / px;
    const int64_t a = s0 * bfe::kSlice / bs, b = std::min<int64_t>(N, s1 * bfe::kSlice / bs);
    auto height = [&](int64_t q) { return (int64_t)q - start[run[q]] + level[run[q]]; };
    int64_t lo = INT64_MAX, hi = INT64_MIN;
    for (int64_t q = a; q < b; ++q) lo = std::min(lo, height(q)), hi = std::max(hi, height(q));
    if (hi - lo > 8 * N) return false;
    first.assign(hi - lo + 2, 0);
    for (int64_t q = a; q < b; ++q) ++first[height(q) - lo + 1];
    std::partial_sum(first.begin(), first.end(), first.begin());
    node.resize(b - a);
    for (int64_t q = a; q < b; ++q) node[first[height(q) - lo]++] = (int32_t)q;
    for (int64_t k = 0; k < b - a; ++k)
      for (int64_t l = 0; l < bs; ++l) perm[(a + k) * bs + l] = (int32_t)(node[k] * bs + l);
    for (int64_t y = 0; y < py; ++y) parts.push_back((int32_t)(s0 + (s1 - s0) * (y + 1) / py));
  }
  return true;
}

}  // namespace

namespace bfe_host {

// Sources up to which a march on the chip is the faster one (onchip_multi_fit);
// FP64 multiply-adds weigh as much as a launch: 1,722 DOF R = 16 9.6 us per
// step on chip against 8.2.
static int64_t most_sources(int prec, bool against_graph) {
  return !against_graph ? 16 : prec == BFE_PREC_DOUBLE ? 8 : 64;
}

// Least bytes of an FP32 operator's blocks, from the slices' widths alone: every
// slice in the smallest form (3D rows: three entries a node, else two), no node
// short of entries.
static int64_t least_operator(const std::vector<int32_t>& sp, bool wide) {
  int64_t total = 0;
  for (size_t s = 0; s + 1 < sp.size(); ++s)
    total += bfe::onchip_block_least((sp[s + 1] - sp[s]) / bfe::kSlice, wide ? 3 : 2);
  return total;
}

static int64_t max_parts(int64_t slices) {
  return std::min<int64_t>(bfe::sm_count(), (slices + kMinSlices - 1) / kMinSlices);
}


// Builds the partition oc; parts already in part_slice are kept. Its state
// becomes 1 when it fits.
static int build_parts(bfe_plan* pl, Onchip& oc, const PartView& view, const std::vector<uint32_t>& h_base,
                       cudaStream_t st) {
  const int64_t n = pl->n, S = pl->n_slices;
  const int prec = pl->prec;
  const int64_t es = (int64_t)elem_size(prec);
  int coop = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, pl->device));
  const bool given = !oc.part_slice.empty();
  const int64_t P = given ? (int64_t)oc.part_slice.size() - 1 : max_parts(S);
  // 16-bit window indices; FP32 entries use two bits to name a reference value
  const int64_t max_window = std::min<int64_t>(kSmemLimit / (2 * es), es == 8 ? 65535 : 16383);
  if (!coop || P < 1 || n > P * max_window) return BFE_OK;
  // contiguous parts of even cost: a slice costs its width (one load of
  // operator and state per entry) and a fixed part for the row's update
  const std::vector<int32_t>& sp = *view.sp;
  auto cost = [&](int64_t s) { return (double)((sp[s + 1] - sp[s]) / bfe::kSlice) + 4.0; };
  double total = 0;
  for (int64_t s = 0; s < S; ++s) total += cost(s);
  if (!given) {
    oc.part_slice.assign(1, 0);
    double run = 0;
    int64_t s = 0;
    for (int64_t p = 0; p < P; ++p) {
      const double target = total * (double)(p + 1) / (double)P;
      const int64_t must = S - (P - 1 - p);          // leave a slice for every later part
      run += cost(s++);
      while (s < must && run + 0.5 * cost(s) <= target) run += cost(s++);
      if (p == P - 1) {
        s = S;
      } else if (prec == BFE_PREC_SINGLE) {
        // FP32 rows of a node that an edge cuts take the slow form: move the
        // edge to a node's first row where one is near (3D: every 96 rows)
        for (int64_t d : {0, 1, -1, 2, -2}) {
          const int64_t x = s + d;
          if (x <= oc.part_slice.back() || x > must || (int64_t)h_base[x * bfe::kSlice] != x * bfe::kSlice) continue;
          for (; s < x; ++s) run += cost(s);
          for (; s > x; --s) run -= cost(s - 1);
          break;
        }
      }
      oc.part_slice.push_back((int32_t)s);
    }
  }
  std::vector<int32_t> boff(S + 1, 0);
  int64_t max_slices = 0, off = 0;
  for (int64_t p = 0; p < P; ++p)
    max_slices = std::max<int64_t>(max_slices, oc.part_slice[p + 1] - oc.part_slice[p]);
  for (int64_t s = 0; s < S; ++s) {
    boff[s] = (int32_t)(off / 16);
    off += bfe::onchip_block_bound(prec, (sp[s + 1] - sp[s]) / bfe::kSlice);
    if (off / 16 > INT32_MAX) return BFE_OK;
  }
  const bool wide = sp[S] >= n * kWideRow;
  // What cannot fit is not built: blocks, halo lists and exchange words of a
  // 1,560,753-DOF brick in FP32 cost 3.4 ms of a plan's first run. FP64 sizes
  // are exact.
  if (prec == BFE_PREC_DOUBLE && off > kMaxOperator64) return BFE_OK;
  if (prec == BFE_PREC_SINGLE && off > kMaxOperator && least_operator(sp, wide) > kMaxOperator) return BFE_OK;
  if (max_slices * bfe::kSlice > max_window) return BFE_OK;
  if (prec == BFE_PREC_SINGLE && off > P * kSmemLimit && wide && (int64_t)sp[S] * 8 <= kStepOperator &&
      least_operator(sp, wide) > P * kSmemLimit)
    return BFE_OK;
  InterfaceLists L;
  if (pl->n_int && !interface_lists(pl, oc.part_slice, L)) return BFE_OK;

  ++pl->partitions_built;
  bfe::OnchipBuild b{};
  b.n = (int32_t)n;
  b.n_parts = (int32_t)P;
  b.max_part_slices = (int32_t)max_slices;
  b.max_words = (int32_t)std::min<int64_t>((n + 31) / 32 + 1, bfe::kOnchipMaxWords);
  b.max_window = (int32_t)max_window;
  b.halo_cap = (int32_t)std::min<int64_t>(max_window, n + P);
  b.n_int = pl->n_int;
  DevBuf<uint8_t> scratch, vexp;
  DevBuf<uint32_t> base;
  DevBuf<int> misfit;
  CUDA_TRY(oc.d_part.upload(oc.part_slice));
  CUDA_TRY(oc.d_off.upload(boff));
  CUDA_TRY(oc.d_bytes.alloc(P));
  CUDA_TRY(oc.d_word.alloc(S));
  CUDA_TRY(oc.d_cnt.alloc(P));
  CUDA_TRY(oc.d_halo.alloc((size_t)P * b.halo_cap));
  CUDA_TRY(oc.flags.alloc(n));
  CUDA_TRY(oc.order.alloc(S));
  CUDA_TRY(oc.blocks.alloc(off));
  if (pl->march_fault == BFE_MARCH_FAULT_MEMORY) return fail(BFE_ERR_OOM, "no memory for a partition (injected)");
  if (prec == BFE_PREC_SINGLE) {
    CUDA_TRY(oc.lref.alloc(n));
    CUDA_TRY(base.upload(h_base));
  }
  CUDA_TRY(scratch.alloc((size_t)n * 2 + (size_t)P * P));
  CUDA_TRY(cudaMemsetAsync(scratch.p, 0, (size_t)n * 2 + (size_t)P * P, st));
  CUDA_TRY(misfit.alloc(2));
  CUDA_TRY(cudaMemsetAsync(misfit.p, 0, 2 * sizeof(int), st));
  if (pl->n_int) {
    CUDA_TRY(vexp.upload(L.exported));
    CUDA_TRY(oc.d_vptr.upload(L.ptr));
    CUDA_TRY(oc.d_vhalo.upload(L.list));
    CUDA_TRY(oc.z_lcol.upload(L.z_lcol));
    CUDA_TRY(oc.xchv.alloc((size_t)pl->n_int * 4 * es));
    CUDA_TRY(cudaMemsetAsync(oc.xchv.p, 0, (size_t)pl->n_int * 4 * es, st));
  }
  if (!given) {
    CUDA_TRY(oc.xch.alloc((size_t)n * 4 * es));
    CUDA_TRY(cudaMemsetAsync(oc.xch.p, 0, (size_t)n * 4 * es, st));
  }
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));     // the uploads, before st reads them
  b.part_slice = oc.d_part.p;
  b.slice_ptr = view.slice_ptr;
  b.block_off = oc.d_off.p;
  b.col = view.col;
  b.val = view.val;
  b.rowc = view.rowc;
  b.base = base.p;
  b.int_row = pl->int_row.p;
  b.v_exported = vexp.p;
  b.halo_cnt = oc.d_cnt.p;
  b.halo_row = oc.d_halo.p;
  b.exported = scratch.p;
  if (prec == BFE_PREC_SINGLE) b.pos = scratch.p + n;
  b.adj = scratch.p + 2 * n;
  b.flags = oc.flags.p;
  b.order = oc.order.p;
  b.blocks = oc.blocks.p;
  b.slice_word = oc.d_word.p;
  b.op_bytes = oc.d_bytes.p;
  b.lref = oc.lref.p;
  b.fail = misfit.p;
  b.slot_bytes = misfit.p + 1;
  CUDA_TRY(bfe::launch_onchip_build(b, prec, st));
  int flags[2] = {0, 0};
  std::vector<int32_t> cnt(P), obytes(P);
  CUDA_TRY(cudaMemcpyAsync(flags, misfit.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaMemcpyAsync(cnt.data(), oc.d_cnt.p, P * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaMemcpyAsync(obytes.data(), oc.d_bytes.p, P * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaStreamSynchronize(st));
  bool failed = flags[0] != 0;
  int64_t max_halo = 0, op_total = 0;
  for (int32_t x : obytes) op_total += x;
  failed = failed || op_total > kMaxOperator;
  oc.need.assign(P, 0);
  for (int64_t p = 0; p < P && !failed; ++p) {
    const int64_t ns = oc.part_slice[p + 1] - oc.part_slice[p], rp = ns * bfe::kSlice;
    const int64_t W = (rp + cnt[p] + 5) & ~(int64_t)3;
    int64_t need = 2 * W * es + ns * 8 + rp * 2 + 32;
    if (pl->n_int) {
      const int64_t own = L.first[p + 1] - L.first[p];
      const int64_t nz = pl->h_z_ptr[L.first[p + 1]] - pl->h_z_ptr[L.first[p]];
      need += (align2(own + L.ptr[p + 1] - L.ptr[p]) + align2(nz)) * es + (own + 1) * 4 + (align2(nz) + align2(own)) * 2;
    }
    oc.need[p] = need;
    max_halo = std::max<int64_t>(max_halo, cnt[p]);
    if (need > kSmemLimit || rp + cnt[p] > max_window) failed = true;
  }
  if (failed) return BFE_OK;
  oc.op_bytes = obytes;
  oc.halo_cnt = cnt;
  bfe::OnchipArgs& o = oc.args;
  o.n_parts = (int32_t)P;
  // a warp per slice where that is enough, else as many warps as give each the
  // same number of slices; and enough threads to poll the halo together
  const int64_t turns = (max_slices + 31) / 32, warps = (max_slices + turns - 1) / turns;
  const int64_t poll = turns == 1 ? std::min<int64_t>(max_slices <= 16 ? 512 : 1024, (max_halo / 2 + 31) / 32 * 32) : 0;
  o.threads = (int32_t)std::max<int64_t>({128, warps * 32, poll});
  o.slot_bytes = flags[1];
  o.part_slice = oc.d_part.p;
  o.halo_cnt = oc.d_cnt.p;
  o.halo_row = oc.d_halo.p;
  o.halo_cap = b.halo_cap;
  o.flags = oc.flags.p;
  o.order = oc.order.p;
  o.blocks = oc.blocks.p;
  o.block_off = oc.d_off.p;
  o.slice_word = oc.d_word.p;
  o.op_bytes = oc.d_bytes.p;
  o.row_of = oc.row_of.p;
  o.lref = oc.lref.p;
  o.vhalo_ptr = oc.d_vptr.p;
  o.vhalo = oc.d_vhalo.p;
  o.z_lcol = oc.z_lcol.p;
  o.xch = oc.xch.p;
  o.x_stride = 2 * n;
  o.xchv = oc.xchv.p;
  o.xv_stride = 2 * (int64_t)pl->n_int;
  oc.next_tag = 1;
  oc.state = 1;
  return BFE_OK;
}

static void discard(std::unique_ptr<Onchip>& holder) {
  holder.reset(new Onchip());
  holder->state = -1;
}

void onchip_give_up(bfe_plan* pl, const Onchip* oc) {
  for (auto* holder : {&pl->tiled, &pl->onchip})
    if (holder->get() == oc) discard(*holder);
}

// Builds a partition once per plan. Nothing is kept of one that does not fit
// or could not be built.
template <typename Build>
static int prepare(std::unique_ptr<Onchip>& holder, cudaStream_t st, Build&& build) {
  if (holder->state) return BFE_OK;
  int rc;
  try {
    rc = build();
  } catch (const std::bad_alloc&) {
    rc = fail(BFE_ERR_OOM, "host allocation failed while building a partition");
  }
  if (rc == BFE_OK && holder->state == 1) return BFE_OK;
  if (rc) {
    cudaStreamSynchronize(st);                         // work on the buffers about to go
    cudaGetLastError();
  }
  discard(holder);
  return rc;
}

int onchip_prepare(bfe_plan* pl, cudaStream_t st) {
  return prepare(pl->onchip, st, [&] {
    const PartView view{&pl->h_slice_ptr, pl->slice_ptr.p, pl->col.p, pl->val.p, pl->rowc.p};
    return build_parts(pl, *pl->onchip, view, pl->h_base, st);
  });
}

int64_t Onchip::device_bytes() const {
  int64_t b = 0;
  auto add = [&](const auto& d) { if (d.p) b += (int64_t)(d.n * sizeof(*d.p)); };
  for (auto* d : {&d_part, &d_off, &d_word, &d_bytes, &d_cnt, &d_halo, &d_vptr, &d_vhalo, &row_of}) add(*d);
  for (auto* d : {&flags, &order, &z_lcol}) add(*d);
  for (auto* d : {&blocks, &xch, &xchv}) add(*d);
  add(xchm);
  add(lref);
  return b;
}

int onchip_meet_fault(const bfe_plan* pl, Onchip& oc) {
  if (pl->march_fault != BFE_MARCH_FAULT_WAIT) return BFE_OK;
  std::vector<uint16_t> f(oc.flags.n);
  CUDA_TRY(cudaMemcpy(f.data(), oc.flags.p, f.size() * sizeof(uint16_t), cudaMemcpyDeviceToHost));
  auto it = std::find_if(f.begin(), f.end(), [](uint16_t x) { return x & 1; });     // bit 0: other parts read the row
  if (it == f.end()) return BFE_OK;
  *it &= (uint16_t)~1u;
  CUDA_TRY(cudaMemcpy(oc.flags.p, f.data(), f.size() * sizeof(uint16_t), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
  return BFE_OK;
}

// The tiled partition, if the model has one.
static int build_tiled(bfe_plan* pl, cudaStream_t st) {
  Onchip& oc = *pl->tiled;
  const int64_t n = pl->n, S = pl->n_slices;
  std::vector<int32_t> perm;
  if (!tile_order(pl, max_parts(S), perm, oc.part_slice)) return BFE_OK;
  oc.place.resize(n);
  for (int64_t i = 0; i < n; ++i) oc.place[perm[i]] = (int32_t)i;
  std::vector<uint32_t> base;
  if (pl->prec == BFE_PREC_SINGLE) {
    base.resize(n);
    for (int64_t i = 0; i < n; ++i) base[i] = (uint32_t)oc.place[pl->h_base[perm[i]]];
  }
  std::vector<int32_t> sp(S + 1, 0);
  for (int64_t s = 0; s < S; ++s) {
    int32_t w = 0;
    for (int64_t i = s * bfe::kSlice; i < std::min<int64_t>(n, (s + 1) * bfe::kSlice); ++i) {
      const int32_t o = perm[i] / bfe::kSlice;
      w = std::max(w, pl->h_slice_ptr[o + 1] - pl->h_slice_ptr[o]);
    }
    if ((int64_t)sp[s] + w > INT32_MAX) return BFE_OK;
    sp[s + 1] = sp[s] + w;
  }
  const int64_t es = (int64_t)elem_size(pl->prec);
  DevBuf<int32_t> place, slice_ptr;
  DevBuf<uint32_t> col;
  DevBuf<unsigned char> val, rowc;
  CUDA_TRY(oc.row_of.upload(perm));
  CUDA_TRY(place.upload(oc.place));
  CUDA_TRY(slice_ptr.upload(sp));
  CUDA_TRY(col.alloc(sp[S]));
  CUDA_TRY(val.alloc((size_t)sp[S] * es));
  CUDA_TRY(rowc.alloc((size_t)n * es));
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));     // the uploads, before st reads them
  bfe::OnchipReorder r{(int32_t)n, (int32_t)S, oc.row_of.p, place.p, pl->slice_ptr.p, pl->col.p, pl->val.p, pl->rowc.p,
                       slice_ptr.p, col.p, val.p, rowc.p};
  CUDA_TRY(bfe::launch_onchip_reorder(r, pl->prec, st));
  const PartView view{&sp, slice_ptr.p, col.p, val.p, rowc.p};
  return build_parts(pl, oc, view, base, st);            // synchronises before it returns
}

Onchip* onchip_for_several(bfe_plan* pl, cudaStream_t st) {
  if (prepare(pl->tiled, st, [&] { return build_tiled(pl, st); }) != BFE_OK) g_last_error.clear();
  if (pl->tiled->state == 1) return pl->tiled.get();
  if (onchip_prepare(pl, st) != BFE_OK) g_last_error.clear();
  return pl->onchip->state == 1 ? pl->onchip.get() : nullptr;
}

// Steps a plan marches before its partition is built: about as many as win back
// what that costs, so that a plan of one short run does not pay for it and one
// of many short runs soon has it. One source: 0.3 to 1.4 ms, for 2 to 5 us a
// step and 0.3 ms a run (no graph). Samples at which a first run breaks even:
// plate of 161,202 DOF FP32 115, coupled 241,579 DOF FP64 165, 961,641 DOF FP32
// 215 (96 samples there: 3.28 ms on the chip, 2.71 in steps). Several sources:
// 0.6 ms at 10,000 DOF, 1.0 at 40,602, 1.5 at 90,902, for 3.4 to 5.7 us a step:
// 40,602 DOF R = 16 breaks even at 200 samples, 90,902 DOF R = 4 at 270. Rows of
// many entries (3D) gain up to 30 us a step and break even below 96.
bool onchip_due(bfe_plan* pl, int64_t steps, bool several) {
  if (pl->onchip->state || (several && pl->tiled->state)) return true;
  pl->steps_marched += steps;
  const int64_t n = pl->n;
  const bool wide = pl->h_slice_ptr.back() >= n * kWideRow;
  return pl->steps_marched >= (wide ? 0 : several ? 70 + n / 350 : 80 + n / 4500);
}

bool onchip_fit(bfe_plan* pl, const std::vector<ForceEntry>& frc, const std::vector<int64_t>& v5_bytes,
                const std::vector<int32_t>& v5_count, bfe::OnchipArgs& o) {
  const Onchip& oc = *pl->onchip;
  o = oc.args;
  const int P = o.n_parts;
  std::vector<int32_t> rows(frc.size());
  for (size_t k = 0; k < frc.size(); ++k) rows[k] = frc[k].row;
  std::sort(rows.begin(), rows.end());
  if (std::adjacent_find(rows.begin(), rows.end()) != rows.end()) return false;
  // prescribed entries get warps of their own where there are some left
  if (!v5_count.empty()) {
    const int32_t most = *std::max_element(v5_count.begin(), v5_count.end());
    o.threads = std::min(o.threads <= 512 ? 512 : 1024, o.threads + (most + 31) / 32 * 32);
    if (most > o.threads) return false;
  }
  // slots per warp for streamed chunks: up to four as long as they take no
  // more than half of the memory the operator has
  const int64_t warps = o.threads / 32;
  int64_t room = kSmemLimit;
  std::vector<int64_t> need(P);
  bool stream = false;
  for (int p = 0; p < P; ++p) {
    const int64_t nf =
        std::lower_bound(rows.begin(), rows.end(), oc.part_slice[p + 1] * bfe::kSlice) -
        std::lower_bound(rows.begin(), rows.end(), oc.part_slice[p] * bfe::kSlice);
    if (nf > o.threads) return false;
    need[p] = oc.need[p] + 2 * nf * (int64_t)elem_size(pl->prec) + 16 + nf * 4 + (warps * 4 + 1) * 8 + 16 +
              (v5_bytes.empty() ? 0 : v5_bytes[p]);
    room = std::min(room, kSmemLimit - need[p]);
    stream = stream || need[p] + oc.op_bytes[p] > kSmemLimit;
  }
  const int64_t ring = warps * o.slot_bytes;
  if (room < (stream ? ring : 0)) return false;
  o.depth = (int32_t)std::max<int64_t>(1, std::min<int64_t>(4, room / 2 / std::max<int64_t>(ring, 1)));
  int64_t smem = 0;
  for (int p = 0; p < P; ++p) smem = std::max(smem, std::min<int64_t>(kSmemLimit, need[p] + oc.op_bytes[p]));
  o.smem = (int32_t)(smem & ~(int64_t)15);
  return true;
}

// The form serves prescribed DOFs whose C row is at most its diagonal (no
// fluid-solid coupling), without correction rows, with K rows inside the
// part's window.
int onchip_v5(bfe_plan* pl, const V5Lists& L, OnchipV5& d, bool& fits) {
  fits = false;
  if (L.corrections) return BFE_OK;
  const Onchip& oc = *pl->onchip;
  const int P = oc.args.n_parts;
  const int64_t ne = (int64_t)L.ent_row.size();
  std::vector<int32_t> ord(ne), ptr(P + 1, 0), row(ne), kptr(1, 0), cnt(P);
  std::iota(ord.begin(), ord.end(), 0);
  std::stable_sort(ord.begin(), ord.end(), [&](int32_t x, int32_t y) { return L.ent_row[x] < L.ent_row[y]; });
  std::vector<uint16_t> kcol;
  std::vector<double> kval, c(ne, 0.0);
  CUDA_TRY(cudaMemcpy(cnt.data(), oc.d_cnt.p, P * sizeof(int32_t), cudaMemcpyDeviceToHost));
  d.bytes.assign(P, 0);
  d.count.assign(P, 0);
  int64_t e = 0;
  for (int p = 0; p < P; ++p) {
    const int64_t r0 = (int64_t)oc.part_slice[p] * bfe::kSlice, rpad = (int64_t)oc.part_slice[p + 1] * bfe::kSlice - r0;
    const int64_t r1 = std::min<int64_t>(pl->n, r0 + rpad);
    std::vector<int32_t> halo;
    std::map<int32_t, int32_t> at;             // halo row -> window index
    const size_t k0 = kcol.size();
    for (; e < ne && L.ent_row[ord[e]] < r1; ++e) {
      const int32_t s = L.ent_slot[ord[e]];
      row[e] = (int32_t)(L.ent_row[ord[e]] - r0);
      for (int32_t x = L.cp[s]; x < L.cp[s + 1]; ++x) {
        if (L.cc[x] != L.slot_row[s]) return BFE_OK;
        c[e] = L.cv[x];
      }
      if (halo.empty() && cnt[p]) {
        halo.resize(cnt[p]);
        CUDA_TRY(cudaMemcpy(halo.data(), oc.d_halo.p + (size_t)p * oc.args.halo_cap, cnt[p] * sizeof(int32_t),
                            cudaMemcpyDeviceToHost));
        for (int32_t k = 0; k < cnt[p]; ++k) at.emplace(halo[k], (int32_t)rpad + k);
      }
      for (int32_t x = L.kp[s]; x < L.kp[s + 1]; ++x) {
        const int32_t col = L.kc[x];
        int64_t w = col - r0;
        if (col < r0 || col >= r1) {
          auto it = at.find(col);
          if (it == at.end()) return BFE_OK;
          w = it->second;
        }
        kcol.push_back((uint16_t)w);
        kval.push_back(L.kv[x]);
      }
      kptr.push_back((int32_t)kcol.size());
      ++d.count[p];
    }
    ptr[p + 1] = (int32_t)e;
    d.bytes[p] = (int64_t)(kcol.size() - k0) * 8 + align2(kcol.size() - k0) * 2;
  }
  CUDA_TRY(d.ptr.upload(ptr));
  CUDA_TRY(d.ent.upload(ord));
  CUDA_TRY(d.row.upload(row));
  CUDA_TRY(d.kptr.upload(kptr));
  CUDA_TRY(d.kcol.upload(kcol));
  CUDA_TRY(d.kval.upload(kval));
  CUDA_TRY(d.c.upload(c));
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
  fits = true;
  return BFE_OK;
}

// Whether the exchange of so many halo rows takes longer than a step from a graph
// (the figures are in onchip_multi_fit).
static bool too_many_words(int prec, int64_t R, int64_t halo) {
  return halo * (prec == BFE_PREC_DOUBLE ? R : R / 2) > 3300 && R > (prec == BFE_PREC_DOUBLE ? 4 : 8);
}

bool onchip_multi_may_fit(const bfe_plan* pl, int64_t R, bool against_graph) {
  if (pl->n_int || R < 2 || R > most_sources(pl->prec, against_graph) || R % bfe::onchip_multi_rv(pl->prec)) return false;
  // the states alone must fit in the SMs' shared memory
  const int64_t es = (int64_t)elem_size(pl->prec);
  if (2 * (double)pl->n * (double)R * (double)es > (double)kSmemLimit * bfe::sm_count()) return false;
  // On a 2D model whose tiles are not cut yet, what onchip_multi_fit would
  // find: tiles cost 1 to 2 ms, and 161,202 DOF, R = 16 had them cut in vain in
  // every plan's first run (3.1 -> 5.3 ms for 200 samples). A mesh column is as
  // long as a node in the middle is far from its last neighbour, and other nodes
  // have as many neighbours.
  const auto& g = pl->groups;
  if (pl->tiled->state || !pl->have_groups || g.n_groups != 1 || g.bs[0] > 2 || (int64_t)g.n_nodes[0] * g.bs[0] != pl->n)
    return true;
  const int64_t bs = g.bs[0], N = g.n_nodes[0], q = N / 2, S = pl->n_slices, P = max_parts(S);
  // (a part of a few rows fits with twice its rows as halo)
  const int64_t most = 3 * ((S + P - 1) / P) * bfe::kSlice;
  if (2 * R * most * es <= kSmemLimit / 2 && !(against_graph && too_many_words(pl->prec, R, most))) return true;
  if (pl->mid_neighbours == 0) return true;
  const int64_t len = std::max<int64_t>(1, pl->mid_last / bs - q), M = (N + len - 1) / len;
  const TileCut cut = tile_cut(S, P, M, (double)len, bs);
  const int64_t rows = (S + cut.px * cut.py - 1) / (cut.px * cut.py) * bfe::kSlice, halo = cut.halo * bs;
  const int width = es == 8 ? (int)(pl->h_slice_ptr[S] / (S * bfe::kSlice)) : pl->mid_neighbours * (int)bs;
  const int64_t block = es == 8 ? bfe::onchip_block_bound(pl->prec, width) : bfe::onchip_block_least(width, (int)bs);
  return 2 * R * (rows + halo) * es + 6 * rows + 4 * halo + rows / bfe::kSlice * block <= kSmemLimit &&
         !(against_graph && too_many_words(pl->prec, R, halo));
}

void onchip_multi_rows(const Onchip& oc, const std::vector<ForceEntry>& frc, const std::vector<int64_t>& hist_idx,
                       MultiLists& L) {
  auto at = [&](int64_t row) { return oc.place.empty() ? (int32_t)row : oc.place[row]; };
  L.forced.resize(frc.size());
  std::iota(L.forced.begin(), L.forced.end(), 0);
  std::stable_sort(L.forced.begin(), L.forced.end(),
                   [&](int32_t x, int32_t y) { return at(frc[x].row) < at(frc[y].row); });
  std::vector<std::pair<int32_t, int32_t>> mons;
  for (size_t k = 0; k < hist_idx.size(); ++k)
    if (hist_idx[k] >= 0) mons.emplace_back(at(hist_idx[k]), (int32_t)k);
  std::sort(mons.begin(), mons.end());
  for (int32_t k : L.forced) L.frows.push_back(at(frc[k].row));
  for (auto& x : mons) {
    L.mrows.push_back(x.first);
    L.mslots.push_back(x.second);
  }
}

int onchip_multi_lists(const bfe_plan* pl, const Onchip& oc, const std::vector<ForceEntry>& frc, MultiLists& L,
                       bfe::StepArgs& a) {
  if (oc.place.empty()) return BFE_OK;             // the run's own lists serve
  std::vector<int32_t> ints(L.frows);
  for (int32_t k : L.forced) ints.push_back(frc[k].rhs);
  for (int32_t k : L.forced) ints.push_back(frc[k].sig);
  ints.insert(ints.end(), L.mrows.begin(), L.mrows.end());
  ints.insert(ints.end(), L.mslots.begin(), L.mslots.end());
  std::vector<unsigned char> coef;
  for (int32_t k : L.forced) {
    const double c = pl->h_acoef[frc[k].row] * frc[k].w;
    if (pl->prec == BFE_PREC_DOUBLE) push_val<double>(coef, c); else push_val<float>(coef, c);
  }
  CUDA_TRY(L.ints.upload(ints));
  CUDA_TRY(L.coef.upload(coef));
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));     // before the run's stream reads them
  const size_t nf = L.frows.size(), nm = L.mrows.size();
  a.frc_row = L.ints.p;
  a.frc_rhs = L.ints.p + nf;
  a.frc_sig = L.ints.p + 2 * nf;
  a.frc_coef = L.coef.p;
  a.mon_row = L.ints.p + 3 * nf;
  a.mon_slot = L.ints.p + 3 * nf + nm;
  return BFE_OK;
}

bool onchip_multi_fit(bfe_plan* pl, Onchip& oc, const bfe::StepArgs& a, const std::vector<int32_t>& frc_rows,
                      const std::vector<int32_t>& mon_rows, bool against_graph, cudaStream_t st, bfe::OnchipArgs& o) {
  o = oc.args;
  const int P = o.n_parts;
  const int64_t R = a.R, es = (int64_t)elem_size(pl->prec), rv = bfe::onchip_multi_rv(pl->prec);
  if (!onchip_multi_may_fit(pl, R, against_graph)) return false;
  int64_t smem = 0, tasks = 0, words = 0;
  const int64_t wpr = pl->prec == BFE_PREC_DOUBLE ? R : R / 2;
  auto in_part = [&](const std::vector<int32_t>& v, int p) {
    return std::lower_bound(v.begin(), v.end(), oc.part_slice[p + 1] * bfe::kSlice) -
           std::lower_bound(v.begin(), v.end(), oc.part_slice[p] * bfe::kSlice);
  };
  for (int p = 0; p < P; ++p) {
    const int64_t ns = oc.part_slice[p + 1] - oc.part_slice[p], rp = ns * bfe::kSlice, H = oc.halo_cnt[p];
    const int64_t nf = in_part(frc_rows, p), nm = in_part(mon_rows, p);
    const int64_t W = bfe::onchip_multi_window((int)(rp + H));
    const int64_t need = 2 * R * W * es + 3 * align2(nf) * es + ns * 8 + (2 * nf + 2 * nm + H + rp) * 4 + rp * 2 + 16 +
                         oc.op_bytes[p];
    if (need > kSmemLimit || nf > 1024) return false;
    smem = std::max(smem, need);
    tasks = std::max(tasks, ns * (R / rv));
    words = std::max(words, H * wpr);
  }
  // Against step kernels replayed from a graph (8 to 12 us per step for models
  // that fit) the exchange decides, about 2 us per 1,000 words of a part. Us
  // per step on chip / graph, in tiles: plate of 40,602 DOF FP32 R = 4 2.8 /
  // 8.1, R = 16 4.7 / 9.1, R = 32 7.2 / 10.2, R = 48 10.3 / 12.2; 90,902 DOF
  // R = 16 7.1 / 10.6, R = 24 9.8 / 13.0; 1,722 DOF R = 64 7.6 / 9.7; FP64
  // 40,602 DOF R = 8 10.1 / 13.9. In strips (a model without tiles): bricks of
  // 14,553 DOF R = 8 8.6 / 9.9, of 46,128 R = 4 8.0 / 12.0; a plate in strips
  // 40,602 DOF R = 16 9.3 / 9.1 (3,232 words), R = 32 14.1 / 9.9. One launch
  // per step, which the adjoint would make, is slower wherever this fits up to
  // R = 16 (17 us per step of 90,902 DOF, R = 16, against 7.5).
  if (against_graph && too_many_words(pl->prec, R, words / wpr)) return false;
  const int64_t turns = (tasks + 31) / 32, warps = (tasks + turns - 1) / turns;
  o.threads = (int32_t)std::max<int64_t>({128, warps * 32, std::min<int64_t>(1024, (words / 4 + 31) / 32 * 32)});
  for (int p = 0; p < P; ++p)
    if (in_part(frc_rows, p) > o.threads) o.threads = 1024;
  o.smem = (int32_t)((smem + 15) & ~(int64_t)15);
  const size_t need_words = (size_t)pl->n * wpr * 2;
  if (oc.xchm.n < need_words) {
    if (oc.xchm.alloc(need_words) != cudaSuccess ||
        cudaMemsetAsync(oc.xchm.p, 0, need_words * sizeof(uint4), st) != cudaSuccess) {
      cudaGetLastError();
      oc.xchm.alloc(0);
      return false;
    }
  }
  o.xch = oc.xchm.p;
  o.x_stride = (int64_t)pl->n * wpr;
  return true;
}

int onchip_tags(Onchip& oc, int64_t n, cudaStream_t st, uint32_t& tag0) {
  if ((uint64_t)oc.next_tag + (uint64_t)n + 2 > 0xffffffffull) {
    if (oc.xch.n) CUDA_TRY(cudaMemsetAsync(oc.xch.p, 0, oc.xch.n, st));
    if (oc.xchv.n) CUDA_TRY(cudaMemsetAsync(oc.xchv.p, 0, oc.xchv.n, st));
    if (oc.xchm.n) CUDA_TRY(cudaMemsetAsync(oc.xchm.p, 0, oc.xchm.n * sizeof(uint4), st));
    oc.next_tag = 1;
  }
  tag0 = oc.next_tag;
  oc.next_tag += (uint32_t)n + 2;
  return BFE_OK;
}

}  // namespace bfe_host
