// The FP64 group block-sparse step kernels (sm_103a, step_f64_group), with the
// launcher the batched dispatch in bfe_kernels.cu calls by variant number. The
// FP32 forms are in bfe_group4_kernels.cu.
#include <cuda_runtime.h>
#include <cstdint>

#include "bfe_device.cuh"
#include "bfe_internal.h"

namespace bfe {

// FP64 group block-sparse kernel (direct form, the reference's arithmetic):
// u_new = sum over the node's blocks (its own included) of B_block u_n
// + D u_{n-1} + forcing, summed in column order like the one-source kernel.
// LPN lanes per node, VEC doubles (right-hand sides) per lane and pass; UNROLL
// neighbours in flight (0: the compiler's choice).
template <int BS, int VEC, int UNROLL>
__device__ __forceinline__ void group64_node(const StepArgs& a, const GroupArgs& gr, int gi, int node,
                                             int c0, int stride) {
  const int4 rec = __ldg(gr.rec[gi] + node);
  const int row0 = rec.x, p0 = rec.y, p1 = rec.y + rec.z;
  const int R = a.R;
  const size_t rs = (size_t)R;
  const double* un = static_cast<const double*>(a.u_n);
  const int32_t* nrow = gr.nrow[gi];
  const double* cf = gr.coef64[gi];
  for (int c = c0; c < R; c += stride) {
    double acc[BS][VEC];
#pragma unroll
    for (int k = 0; k < BS; ++k)
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[k][v] = 0.0;
    auto add = [&](int e) {
      const double* nb = un + (size_t)__ldg(nrow + e) * rs + c;
      double g[BS][VEC];
#pragma unroll
      for (int l = 0; l < BS; ++l)
#pragma unroll
        for (int v = 0; v < VEC; v += 2) {
          const double2 x = __ldg(reinterpret_cast<const double2*>(nb + l * rs + v));
          g[l][v] = x.x;
          g[l][v + 1] = x.y;
        }
      double cv[BS * BS];
#pragma unroll
      for (int t = 0; t < BS * BS; ++t) cv[t] = __ldg(cf + (size_t)e * (BS * BS) + t);
#pragma unroll
      for (int l = 0; l < BS; ++l)
#pragma unroll
        for (int k = 0; k < BS; ++k)
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc[k][v] = fma(cv[k * BS + l], g[l][v], acc[k][v]);
    };
    if constexpr (UNROLL == 0) {
      for (int e = p0; e < p1; ++e) add(e);
    } else {
#pragma unroll UNROLL
      for (int e = p0; e < p1; ++e) add(e);
    }
    double* unew = static_cast<double*>(a.u_new);
    const double* upv = static_cast<const double*>(a.u_prev);
#pragma unroll
    for (int k = 0; k < BS; ++k) {
      const int row = row0 + k;
      const uint32_t info = __ldg(a.rowinfo + row);
      const double dk = __ldg(static_cast<const double*>(a.rowc) + row);
      const size_t o = (size_t)row * rs + c;
      double res[VEC], upk[VEC];
#pragma unroll
      for (int v = 0; v < VEC; v += 2) {
        const double2 x = __ldcs(reinterpret_cast<const double2*>(upv + o + v));
        upk[v] = x.x;
        upk[v + 1] = x.y;
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        double r = acc[k][v] + dk * upk[v];
        if (info & kRowForced) r += forcing_sum<double>(a, row, c + v);
        res[v] = r;
      }
#pragma unroll
      for (int v = 0; v < VEC; v += 2)
        *reinterpret_cast<double2*>(unew + o + v) = make_double2(res[v], res[v + 1]);
      if (info & kRowInterface) {
        const int t = lower_bound_i32(a.int_row, a.n_int, row);
        double* vi = static_cast<double*>(a.v_int) + (size_t)t * R + c;
#pragma unroll
        for (int v = 0; v < VEC; ++v) vi[v] = a.int_base_prev ? (res[v] - upk[v]) : (un[o + v] - upk[v]);
      } else if (info & kRowMonitored) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) write_history(a, row, c + v, res[v]);
      }
    }
  }
}

template <int LPN, int VEC, int MINB, int MAXBS, int UNROLL = 0>
__global__ void __launch_bounds__(128, MINB) step_f64_group(StepArgs a, GroupArgs gr) {
  const int b = blockIdx.x;
  int gi = 0;
#pragma unroll
  for (int k = 1; k < kMaxGroups; ++k)
    if (k < gr.n_groups && b >= gr.blk_begin[k]) gi = k;
  // LPN lanes per node, or gr.lpn of them (LPN = 0: any R)
  const int lpn = LPN ? LPN : gr.lpn, npc = 128 / lpn, ln = threadIdx.x / lpn;
  const int node = (b - gr.blk_begin[gi]) * npc + ln;
  if (ln >= npc || node >= gr.n_nodes[gi]) return;
  const int c0 = (threadIdx.x - ln * lpn) * VEC, stride = lpn * VEC;
  if (gr.bs[gi] == 1) group64_node<1, VEC, UNROLL>(a, gr, gi, node, c0, stride);
  else if (MAXBS == 2 || gr.bs[gi] == 2) group64_node<(MAXBS >= 2 ? 2 : 1), VEC, UNROLL>(a, gr, gi, node, c0, stride);
  else group64_node<MAXBS, VEC, UNROLL>(a, gr, gi, node, c0, stride);
}

// FP64 variants: 1 = 16 lanes x 4 right-hand sides (R a multiple of 64),
// 2 = 16 x 2 (R a multiple of 32), 3 = 8 x 2 (R a multiple of 16), 4 and 5 =
// any even R, two right-hand sides per lane, one or two neighbours in flight
// (us per step, slice kernel / variant 4: coupled 241,579 DOF R = 5 154.5 /
// 35.1, R = 21 157.5 / 111.5; the FP64 pipe bounds both). Skipping the absent
// entries of a block (one in seven) by a branch made variant 1 slower, 359 us
// against 272 at R = 64. One neighbour at a time suits variants 1 and 2 on 2D
// nodes (us per step with the compiler's choice / one: coupled 241,579 DOF R = 64
// 286.4 / 283.2); variant 3 and 3D nodes want the compiler's choice (bricks of
// 14,553 DOF R = 48 100.9 / 102.5, R = 64 129.8 / 131.7, plate of 40,602 DOF R = 48
// 57.7 / 58.4).
static cudaError_t launch_group64(const StepArgs& a, const GroupArgs& gr, int variant, cudaStream_t st) {
  const int pairs = a.R / 2, passes = (pairs + 15) / 16;
  const int lpn = variant >= 4 ? (pairs + passes - 1) / passes : variant == 3 ? 8 : 16;
  GroupArgs g = gr;
  g.lpn = lpn;
  int blocks = 0;
  for (int k = 0; k < g.n_groups; ++k) {
    g.blk_begin[k] = blocks;
    blocks += (g.n_nodes[k] + 128 / lpn - 1) / (128 / lpn);
  }
  g.blk_begin[g.n_groups] = blocks;
  int maxbs = 1;
  for (int k = 0; k < g.n_groups; ++k) maxbs = g.bs[k] > maxbs ? g.bs[k] : maxbs;
  if (maxbs <= 2) {
    if (variant == 1) step_f64_group<16, 4, 8, 2, 1><<<blocks, 128, 0, st>>>(a, g);
    else if (variant == 2) step_f64_group<16, 2, 10, 2, 1><<<blocks, 128, 0, st>>>(a, g);
    else if (variant == 3) step_f64_group<8, 2, 10, 2><<<blocks, 128, 0, st>>>(a, g);
    else if (variant == 4) step_f64_group<0, 2, 8, 2, 1><<<blocks, 128, 0, st>>>(a, g);
    else step_f64_group<0, 2, 6, 2, 2><<<blocks, 128, 0, st>>>(a, g);
  } else {
    if (variant == 1) step_f64_group<16, 4, 6, 3><<<blocks, 128, 0, st>>>(a, g);
    else if (variant == 2) step_f64_group<16, 2, 8, 3><<<blocks, 128, 0, st>>>(a, g);
    else if (variant == 3) step_f64_group<8, 2, 8, 3><<<blocks, 128, 0, st>>>(a, g);
    else if (variant == 4) step_f64_group<0, 2, 6, 3, 1><<<blocks, 128, 0, st>>>(a, g);
    else step_f64_group<0, 2, 4, 3, 2><<<blocks, 128, 0, st>>>(a, g);
  }
  return cudaGetLastError();
}

cudaError_t launch_group64_variant(const StepArgs& a, const GroupArgs& gr, int variant, cudaStream_t st) {
  return launch_group64(a, gr, variant, st);
}

}  // namespace bfe
