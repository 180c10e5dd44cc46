// Sliced-ELL operator of a one-source plan, packed on the GPU from the
// caller's CSR arrays (fn_explicit_dynamic_solver_v6.m:130-159).
//
// A drop-in call makes a plan per load step, and packing its operator on the
// host (validating, copying and re-ordering K's entries) took half of the
// call: 5.3 of 11.8 ms on a 40,602-DOF plate, 105 ms on 961,641 DOF. Here K's
// arrays are copied as they are and one warp per slice (a lane per row) first
// counts and validates, then packs; both passes read each entry once, which
// at 16 bytes an entry is a few tens of microseconds. Anything irregular
// (unsorted or repeated columns, an index out of range, a non-finite value)
// only raises a flag: the host path then converts the matrix or reports the
// error. The values are the host path's, operation for operation.
#include <cuda_runtime.h>
#include <cstdint>

#include "bfe_internal.h"

namespace bfe {

namespace {

// Type sums of an FP32 row: true when every column type exists in the row's
// node block and its entries sum to zero (the difference form applies).
__device__ bool row_is_difference(const PackArgs& p, int64_t i, int64_t e0, int64_t e1) {
  int32_t ty[16];
  double sm[16], sa[16];
  int nty = 0;
  for (int64_t e = e0; e < e1; ++e) {
    const double v = p.val[e];
    if (v == 0.0) continue;
    const int32_t t = p.dof_type[p.idx[e]];
    int k = 0;
    while (k < nty && ty[k] != t) ++k;
    if (k == nty) {
      if (nty == 16) return false;
      ty[nty] = t;
      sm[nty] = 0.0;
      sa[nty] = 0.0;
      ++nty;
    }
    sm[k] += v;
    sa[k] += fabs(v);
  }
  const int32_t b0 = p.blk_base[i], b1 = b0 + p.blk_len[i];
  for (int k = 0; k < nty; ++k) {
    bool found = false;
    for (int32_t b = b0; b < b1; ++b) found = found || p.dof_type[b] == ty[k];
    if (!found || fabs(sm[k]) > __dmul_rn(1e-9, sa[k])) return false;
  }
  return true;
}

template <bool F64>
__global__ void __launch_bounds__(256) pack_count(PackArgs p) {
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= p.n_slices) return;
  const int lane = threadIdx.x & 31;
  const int64_t i = s * kSlice + lane;
  int count = 0;
  bool direct = false;
  if (i < p.n) {
    const int64_t e0 = p.ptr[i], e1 = p.ptr[i + 1];
    bool ok = e0 >= 0 && e1 >= e0 && e1 <= p.nnz && e1 - e0 <= INT32_MAX;
    int64_t prev = -1;
    bool has_diag = false;
    for (int64_t e = e0; ok && e < e1; ++e) {
      const int64_t b = p.idx[e];
      const double v = p.val[e];
      ok = b > prev && b < p.n && isfinite(v);
      prev = b;
      if (v != 0.0) {
        ++count;
        has_diag = has_diag || b == i;
      }
    }
    if (!ok) {
      atomicExch(p.irregular, 1);
      count = 0;
    } else if (F64) {
      count += has_diag ? 0 : 1;
    } else {
      const bool diff = p.blk_base && row_is_difference(p, i, e0, e1);
      p.base[i] = diff ? (uint32_t)p.blk_base[i] : 0u;
      p.diff[i] = diff;
      direct = !diff;
      if (diff)
        for (int64_t e = e0; e < e1; ++e)
          if (p.val[e] != 0.0 && p.dof_node[p.idx[e]] == p.dof_node[i]) --count;
    }
  }
  int w = count;
  long long stored = count;
  for (int d = 16; d > 0; d >>= 1) {
    w = max(w, __shfl_xor_sync(0xffffffffu, w, d));
    stored += __shfl_xor_sync(0xffffffffu, stored, d);
  }
  const unsigned nd = __ballot_sync(0xffffffffu, direct);
  if (lane == 0) {
    p.width[s] = w;
    atomicAdd(reinterpret_cast<unsigned long long*>(p.totals), (unsigned long long)stored);
    atomicAdd(reinterpret_cast<unsigned long long*>(p.totals + 1), (unsigned long long)__popc(nd));
  }
}

template <bool F64>
__global__ void __launch_bounds__(256) pack_write(PackArgs p) {
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= p.n_slices) return;
  const int lane = threadIdx.x & 31;
  const int64_t i = s * kSlice + lane;
  const int32_t off = p.slice_ptr[s], w = (p.slice_ptr[s + 1] - off) / kSlice;
  uint32_t* col = p.col + off + lane;
  double* vd = static_cast<double*>(p.out) + off + lane;
  float* vf = static_cast<float*>(p.out) + off + lane;
  int k = 0;
  auto put = [&](uint32_t c, double v) {
    col[32 * k] = c;
    if (F64) vd[32 * k] = v;
    else vf[32 * k] = (float)v;
    ++k;
  };
  if (i < p.n) {
    const int64_t e0 = p.ptr[i], e1 = p.ptr[i + 1];
    const double ls = p.lscale[i];
    if (F64) {
      bool has_diag = false;
      for (int64_t e = e0; e < e1 && !has_diag; ++e) has_diag = p.idx[e] == i && p.val[e] != 0.0;
      bool due = !has_diag;                            // a diagonal of its own, in column order
      for (int64_t e = e0; e < e1; ++e) {
        const int64_t j = p.idx[e];
        if (p.val[e] == 0.0) continue;
        if (due && j > i) {
          put((uint32_t)i, p.diag[i]);
          due = false;
        }
        double v = __dmul_rn(-ls, p.val[e]);
        if (j == i) v = __dadd_rn(v, p.diag[i]);
        put((uint32_t)j, v);
      }
      if (due) put((uint32_t)i, p.diag[i]);
    } else if (p.diff[i]) {
      const int32_t b0 = p.blk_base[i], b1 = b0 + p.blk_len[i];
      for (int64_t e = e0; e < e1; ++e) {
        const int64_t j = p.idx[e];
        if (p.val[e] == 0.0 || p.dof_node[j] == p.dof_node[i]) continue;
        uint32_t slot = 0;
        for (int32_t b = b0; b < b1; ++b)
          if (p.dof_type[b] == p.dof_type[j]) slot = (uint32_t)(b - b0);
        put((uint32_t)j | (slot << kSlotShift), __dmul_rn(ls, p.val[e]));
      }
    } else {
      for (int64_t e = e0; e < e1; ++e)
        if (p.val[e] != 0.0) put((uint32_t)p.idx[e] | kDirect, __dmul_rn(ls, p.val[e]));
    }
  }
  while (k < w) put((uint32_t)(i < p.n ? i : p.n - 1) | (F64 ? 0u : kDirect), 0.0);
}

}  // namespace

cudaError_t launch_pack_count(const PackArgs& p, int precision, cudaStream_t st) {
  const unsigned blocks = (unsigned)((p.n_slices * 32 + 255) / 256);
  if (precision == 0) pack_count<true><<<blocks, 256, 0, st>>>(p);
  else pack_count<false><<<blocks, 256, 0, st>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_pack_write(const PackArgs& p, int precision, cudaStream_t st) {
  const unsigned blocks = (unsigned)((p.n_slices * 32 + 255) / 256);
  if (precision == 0) pack_write<true><<<blocks, 256, 0, st>>>(p);
  else pack_write<false><<<blocks, 256, 0, st>>>(p);
  return cudaGetLastError();
}

}  // namespace bfe
