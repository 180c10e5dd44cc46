// Device helpers shared by the step kernels (bfe_kernels.cu,
// bfe_group_kernels.cu, bfe_group4_kernels.cu): forcing and monitor lookups on the
// sorted per-run lists, and the error-free sums of the compensated update.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "bfe_internal.h"

namespace bfe {

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

__device__ __forceinline__ int lower_bound_i32(const int32_t* a, int n, int key) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (__ldg(a + mid) < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Sum of coef * signal over the forcing entries of row i for right-hand side r.
template <typename T>
__device__ __forceinline__ T forcing_sum(const StepArgs& a, int i, int r) {
  const T* coef = static_cast<const T*>(a.frc_coef);
  const T* sig = static_cast<const T*>(a.sig) + (size_t)step_index(a) * a.n_sig;
  T f = T(0);
  for (int e = lower_bound_i32(a.frc_row, a.n_frc, i); e < a.n_frc && __ldg(a.frc_row + e) == i; ++e) {
    if (__ldg(a.frc_rhs + e) == r) f += __ldg(coef + e) * __ldg(sig + __ldg(a.frc_sig + e));
  }
  return f;
}

// The same for N consecutive right-hand sides from r0, in one pass over the
// row's entries, which are sorted by right-hand side. A receiver of the adjoint
// is forced in every source, and a pass for each right-hand side of a lane was a
// chain of loads that a step waits for: 6,642 DOF FP32 R = 24, 600 samples 24.2 ->
// 21.1 ms. (In the FP64 group kernels it costs registers: coupled 241,579 DOF R =
// 64 281 -> 309 us per step.)
template <typename T, int N>
__device__ __forceinline__ void forcing_sums(const StepArgs& a, int i, int r0, T (&f)[N]) {
  const T* coef = static_cast<const T*>(a.frc_coef);
  const T* sig = static_cast<const T*>(a.sig) + (size_t)step_index(a) * a.n_sig;
#pragma unroll
  for (int j = 0; j < N; ++j) f[j] = T(0);
  for (int e = lower_bound_i32(a.frc_row, a.n_frc, i); e < a.n_frc && __ldg(a.frc_row + e) == i; ++e) {
    const int k = __ldg(a.frc_rhs + e) - r0;
    if (k >= N) break;
    if (k < 0) continue;
    const T c = __ldg(coef + e), s = __ldg(sig + __ldg(a.frc_sig + e));
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (j == k) f[j] += c * s;
  }
}

__device__ __forceinline__ void write_history(const StepArgs& a, int i, int r, double v) {
  if (r >= a.R_out) return;
  for (int k = lower_bound_i32(a.mon_row, a.n_mon, i); k < a.n_mon && __ldg(a.mon_row + k) == i; ++k) {
    int slot = __ldg(a.mon_slot + k);
    a.hist[(size_t)slot + (size_t)a.q * ((size_t)step_index(a) + (size_t)a.n_t * r)] = v;
  }
}

// Error-free transformation: s + e == a + b exactly (Knuth two-sum).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Asks L2 for [p, p + bytes), cut to 16-byte boundaries and to the end of the
// array: one bulk instruction of one thread.
__device__ __forceinline__ void prefetch_l2(const void* p, size_t bytes, const void* end) {
  const uintptr_t b = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15);
  const uintptr_t lim = reinterpret_cast<uintptr_t>(end);
  uintptr_t e = reinterpret_cast<uintptr_t>(p) + bytes;
  e = (e < lim ? e : lim) & ~uintptr_t(15);
  if (e > b) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"((uint32_t)(e - b)) : "memory");
}

// One thread of a group kernel's CTA, whose first node is `node` of npc:
// requests to L2 for what the CTA will read last (its rows of u_{n-1}) and for
// what the CTA gr.ahead further on will read first (its rows of u_n, its
// neighbour lists and blocks). A node's loads are a chain, record -> neighbour
// row -> state, in which each DRAM miss costs about a microsecond; with the
// requests made early they are L2 hits. Rows and blocks of a group follow the
// order of its nodes, so the place of the later CTA's is estimated from this
// one's: a request that misses its aim only costs its bytes.
__device__ __forceinline__ void prefetch_group(const StepArgs& a, const GroupArgs& gr, int gi, int node, int npc) {
  const int4 rec = __ldg(gr.rec[gi] + node);
  const int bs = gr.bs[gi], dn = gr.ahead * npc;
  const size_t R = (size_t)a.R, state = (size_t)a.n * R, bytes = (size_t)(npc * bs) * R * sizeof(float);
  const float* up = static_cast<const float*>(a.u_prev);
  const float* un = static_cast<const float*>(a.u_n);
  prefetch_l2(up + (size_t)rec.x * R, bytes, up + state);
  const int64_t row = (int64_t)rec.x + (int64_t)dn * bs;
  if (row < a.n) prefetch_l2(un + (size_t)row * R, bytes, un + state);
  if (node + dn >= gr.n_nodes[gi]) return;
  const size_t e = (size_t)rec.y + (size_t)rec.z * dn, n_blk = (size_t)__ldg(gr.nptr[gi] + gr.n_nodes[gi]);
  if (e >= n_blk) return;
  const size_t cnt = (size_t)rec.z * npc, bb = (size_t)(bs * bs);
  prefetch_l2(gr.coef[gi] + e * bb, cnt * bb * sizeof(float), gr.coef[gi] + n_blk * bb);
  prefetch_l2(gr.nrow[gi] + e, cnt * sizeof(int32_t), gr.nrow[gi] + n_blk);
  prefetch_l2(gr.rec[gi] + node + dn, npc * sizeof(int4), gr.rec[gi] + gr.n_nodes[gi]);
}

// Packed FP32x2 forms (__ffma2_rn / __fadd2_rn: IEEE round-to-nearest per
// component, the same results as two scalar operations).
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) {        // a - b, exact rounding
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e) {
  s = __fadd2_rn(a, b);
  const float2 bb = f2sub(s, a);
  e = __fadd2_rn(f2sub(a, f2sub(s, bb)), f2sub(b, bb));
}

}  // namespace bfe
