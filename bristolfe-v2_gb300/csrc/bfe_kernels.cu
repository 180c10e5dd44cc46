// Time-step kernels of the GB300 explicit solver (sm_103a).
//
// One time step of fn_explicit_dynamic_solver_v6.m:180-218 is
//     u_{n+1} = A f + B u_n + D u_{n-1}
// (v6.m:185). The operator is stored as a sliced ELL matrix (slices of 32
// rows, entries column-major inside a slice) so that a warp of consecutive
// rows reads its matrix entries with coalesced loads.
//
//  * FP64 plans keep the reference's arithmetic: B (with its diagonal) in
//    the slice entries, the diagonal D in rowc, forcing coefficients of the
//    diagonal A in the forcing list.
//  * FP32 plans use the equivalent increment form
//        u_{n+1} = u_n + q (u_n - u_{n-1}) - Lp u_n + forcing
//    where Lp = P^-1 dt^2 M^-1 K and q = P^-1 (1 - dt/2 M^-1 C) for the
//    diagonal part of P. The stiffness product is evaluated in the
//    difference form sum_j Lp_ij (u_j - u_{node(i), dof(j)}), which is exact
//    for rigid translations whatever the FP32 rounding of Lp, and the update
//    is evaluated with an error-free two-sum of (u_n - u_{n-1}).
//  * Interface rows (fluid-solid coupling in C) get the exact implicit part
//    in a second small kernel: v = (u_hat - u_{n-1}) or (u_n - u_{n-1})
//    is staged per interface row, then u_new = base + Z v.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "bfe_device.cuh"
#include "bfe_internal.h"

namespace bfe {

// Read-only loads that take no L1 space: the one-source FP64 kernel's
// column words and values are each read once per step by one thread, so
// leaving them out of L1 keeps it for the gathered u_n values (C1, 961,641
// DOF: 27.2 us per step against 31.2). The FP32 kernel keeps the default
// loads, which measured faster for it (17.6 us against 22.7).
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* a) {
  uint32_t r;
  asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(r) : "l"(a));
  return r;
}
__device__ __forceinline__ double ld_stream(const double* a) {
  double r;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(r) : "l"(a));
  return r;
}

// ---------------------------------------------------------------------------
// FP64, one right-hand side: one thread per row.
__global__ void __launch_bounds__(256) step_f64_r1(StepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const int s = i >> 5, lane = i & 31;
  const int off = __ldg(a.slice_ptr + s);
  const int w = (__ldg(a.slice_ptr + s + 1) - off) >> 5;
  const uint32_t* col = a.col + off + lane;
  const double* val = static_cast<const double*>(a.val) + off + lane;
  const double* un = static_cast<const double*>(a.u_n);
  double acc = 0.0;
#pragma unroll 4
  for (int k = 0; k < w; ++k) {
    acc = fma(ld_stream(val + 32 * k), __ldg(un + ld_stream(col + 32 * k)), acc);
  }
  const uint32_t info = __ldg(a.rowinfo + i);
  const double up = static_cast<const double*>(a.u_prev)[i];
  double r = acc + __ldg(static_cast<const double*>(a.rowc) + i) * up;
  if (info & kRowForced) r += forcing_sum<double>(a, i, 0);
  static_cast<double*>(a.u_new)[i] = r;
  if (info & kRowInterface) {
    const int t = lower_bound_i32(a.int_row, a.n_int, i);
    static_cast<double*>(a.v_int)[t] = a.int_base_prev ? (r - up) : (un[i] - up);
    return;
  }
  if (info & kRowMonitored) write_history(a, i, 0, r);
  if (a.fld) write_frame<double>(a, i, r, un[i]);
}

// ---------------------------------------------------------------------------
// FP32, one right-hand side: one thread per row, difference form.
__global__ void __launch_bounds__(256) step_f32_r1(StepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const int s = i >> 5, lane = i & 31;
  const int off = __ldg(a.slice_ptr + s);
  const int w = (__ldg(a.slice_ptr + s + 1) - off) >> 5;
  const uint32_t* col = a.col + off + lane;
  const float* val = static_cast<const float*>(a.val) + off + lane;
  const float* un = static_cast<const float*>(a.u_n);
  const uint32_t info = __ldg(a.rowinfo + i);
  const uint32_t base = info & kBaseMask;
  float acc = 0.f;
#pragma unroll 4
  for (int k = 0; k < w; ++k) {
    const uint32_t e = __ldg(col + 32 * k);
    const float uj = __ldg(un + (e & kColMask));
    const float ur = (e & kDirect) ? 0.f : __ldg(un + base + ((e >> kSlotShift) & kSlotMask));
    acc = fmaf(__ldg(val + 32 * k), uj - ur, acc);
  }
  const float ui = un[i];
  const float up = static_cast<const float*>(a.u_prev)[i];
  const float q = __ldg(static_cast<const float*>(a.rowc) + i);
  float d, err;
  two_sum(ui, -up, d, err);
  float inc = fmaf(q, d, -acc);
  if (info & kRowForced) inc += forcing_sum<float>(a, i, 0);
  inc = fmaf(q, err, inc);
  const float r = ui + inc;
  static_cast<float*>(a.u_new)[i] = r;
  if (info & kRowInterface) {
    const int t = lower_bound_i32(a.int_row, a.n_int, i);
    static_cast<float*>(a.v_int)[t] = a.int_base_prev ? (d + err + inc) : (d + err);
    return;
  }
  if (info & kRowMonitored) write_history(a, i, 0, (double)r);
  if (a.fld) write_frame<float>(a, i, r, ui);
}

// ---------------------------------------------------------------------------
// Batched (R right-hand sides, state [n][R]). One CTA per slice of 32 rows:
// the slice's matrix entries are staged in shared memory with coalesced
// loads, then each warp takes rows of the slice and its lanes take the
// right-hand sides, so every gathered state row is one contiguous R-vector.
template <typename T, int VEC>
__global__ void __launch_bounds__(256) step_batched(StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int s = blockIdx.x;
  const int off = __ldg(a.slice_ptr + s);
  const int ne = __ldg(a.slice_ptr + s + 1) - off;
  const int w = ne >> 5;
  uint32_t* scol = reinterpret_cast<uint32_t*>(smem_raw);
  T* sval = reinterpret_cast<T*>(smem_raw + ((ne * sizeof(uint32_t) + 15) & ~size_t(15)));
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    scol[e] = __ldg(a.col + off + e);
    sval[e] = __ldg(static_cast<const T*>(a.val) + off + e);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5;
  const int R = a.R;
  const T* un = static_cast<const T*>(a.u_n);
  const T* upv = static_cast<const T*>(a.u_prev);
  T* unew = static_cast<T*>(a.u_new);
  for (int rr = warp; rr < kSlice; rr += nwarps) {
    const int i = s * kSlice + rr;
    if (i >= a.n) break;
    const uint32_t info = __ldg(a.rowinfo + i);
    const uint32_t base = info & kBaseMask;
    const T rc = __ldg(static_cast<const T*>(a.rowc) + i);
    for (int c0 = lane * VEC; c0 < R; c0 += 32 * VEC) {
      T acc[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] = T(0);
#pragma unroll 2
      for (int k = 0; k < w; ++k) {
        const uint32_t e = scol[k * kSlice + rr];
        const T lv = sval[k * kSlice + rr];
        const size_t j = (size_t)(e & kColMask);
        if constexpr (sizeof(T) == 4) {
          const size_t jr = (size_t)base + ((e >> kSlotShift) & kSlotMask);
          const bool direct = (e & kDirect) != 0;
          if constexpr (VEC == 2) {
            const float2 uj = __ldg(reinterpret_cast<const float2*>(un + j * R + c0));
            float2 ur = make_float2(0.f, 0.f);
            if (!direct) ur = __ldg(reinterpret_cast<const float2*>(un + jr * R + c0));
            acc[0] = fmaf(lv, uj.x - ur.x, acc[0]);
            acc[1] = fmaf(lv, uj.y - ur.y, acc[1]);
          } else {
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
              const float uj = __ldg(un + j * R + c0 + v);
              const float ur = direct ? 0.f : __ldg(un + jr * R + c0 + v);
              acc[v] = fmaf(lv, uj - ur, acc[v]);
            }
          }
        } else {
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc[v] = fma(lv, __ldg(un + j * R + c0 + v), acc[v]);
        }
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int c = c0 + v;
        const size_t o = (size_t)i * R + c;
        const T ui = un[o];
        const T up = upv[o];
        T r, vint;
        if constexpr (sizeof(T) == 4) {
          float d, err;
          two_sum(ui, -up, d, err);
          float inc = fmaf(rc, d, -acc[v]);
          if (info & kRowForced) inc += forcing_sum<float>(a, i, c);
          inc = fmaf(rc, err, inc);
          r = ui + inc;
          vint = a.int_base_prev ? (d + err + inc) : (d + err);
        } else {
          r = acc[v] + rc * up;
          if (info & kRowForced) r += forcing_sum<double>(a, i, c);
          vint = a.int_base_prev ? (r - up) : (ui - up);
        }
        unew[o] = r;
        if (info & kRowInterface) {
          const int t = lower_bound_i32(a.int_row, a.n_int, i);
          static_cast<T*>(a.v_int)[(size_t)t * R + c] = vint;
        } else if (info & kRowMonitored) {
          write_history(a, i, c, (double)r);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Interface correction: u_new[row] = base + sum_z Z[t, z] v[z], one thread
// per (interface row, right-hand side).
template <typename T>
__global__ void __launch_bounds__(256) interface_fixup(StepArgs a) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int R = a.R;
  if (g >= (int64_t)a.n_int * R) return;
  const int t = (int)(g / R), c = (int)(g % R);
  const int row = __ldg(a.int_row + t);
  const T* z = static_cast<const T*>(a.z_val);
  const T* v = static_cast<const T*>(a.v_int);
  T acc = T(0);
  for (int e = __ldg(a.z_ptr + t); e < __ldg(a.z_ptr + t + 1); ++e) {
    acc += __ldg(z + e) * v[(size_t)__ldg(a.z_col + e) * R + c];
  }
  const size_t o = (size_t)row * R + c;
  T* unew = static_cast<T*>(a.u_new);
  const T base = a.int_base_prev ? static_cast<const T*>(a.u_prev)[o] : unew[o];
  const T r = base + acc;
  unew[o] = r;
  if (__ldg(a.rowinfo + row) & kRowMonitored) write_history(a, row, c, (double)r);
}

// Interface correction with VEC consecutive right-hand sides per thread (R
// a multiple of VEC): each Z entry and column index is loaded once for VEC
// values. The sums are interface_fixup's, term for term in the same order.
// A few thousand threads, so bound by the latency of the loads: eight
// entries are loaded before they are summed (R = 64, 961,641 DOF coupled
// FP64 run: 286.5 us per step with one entry at a time, 281.1 with eight).
template <typename T, typename V, int VEC>
__global__ void __launch_bounds__(256) interface_fixup_vec(StepArgs a) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int RV = a.R / VEC;
  if (g >= (int64_t)a.n_int * RV) return;
  const int t = (int)(g / RV), c = (int)(g % RV) * VEC;
  const int row = __ldg(a.int_row + t);
  const T* z = static_cast<const T*>(a.z_val);
  const T* v = static_cast<const T*>(a.v_int);
  T acc[VEC];
#pragma unroll
  for (int j = 0; j < VEC; ++j) acc[j] = T(0);
  const int e1 = __ldg(a.z_ptr + t + 1);
#pragma unroll 8
  for (int e = __ldg(a.z_ptr + t); e < e1; ++e) {
    const T zv = __ldg(z + e);
    const V x = *reinterpret_cast<const V*>(v + (size_t)__ldg(a.z_col + e) * a.R + c);
    const T* xs = reinterpret_cast<const T*>(&x);
#pragma unroll
    for (int j = 0; j < VEC; ++j) acc[j] = fma(zv, xs[j], acc[j]);
  }
  const size_t o = (size_t)row * a.R + c;
  T* unew = static_cast<T*>(a.u_new);
  const V bv = a.int_base_prev ? *reinterpret_cast<const V*>(static_cast<const T*>(a.u_prev) + o)
                               : *reinterpret_cast<const V*>(unew + o);
  const T* bs = reinterpret_cast<const T*>(&bv);
  V rv;
  T* rs = reinterpret_cast<T*>(&rv);
#pragma unroll
  for (int j = 0; j < VEC; ++j) rs[j] = bs[j] + acc[j];
  *reinterpret_cast<V*>(unew + o) = rv;
  if (__ldg(a.rowinfo + row) & kRowMonitored)
    for (int j = 0; j < VEC; ++j) write_history(a, row, c + j, (double)rs[j]);
}

// Interface correction for one right-hand side: one warp per interface row,
// lanes stride over the row of Z and reduce with shuffles. Bound by the chain
// of dependent loads, so what does not depend on the sum is loaded before it.
template <typename T>
__global__ void __launch_bounds__(256) interface_fixup_r1(StepArgs a) {
  const int t = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= a.n_int) return;
  const int row = __ldg(a.int_row + t);
  const int e0 = __ldg(a.z_ptr + t), e1 = __ldg(a.z_ptr + t + 1);
  const T* z = static_cast<const T*>(a.z_val);
  const T* v = static_cast<const T*>(a.v_int);
  T* unew = static_cast<T*>(a.u_new);
  const T base = a.int_base_prev ? static_cast<const T*>(a.u_prev)[row] : unew[row];
  const uint32_t info = __ldg(a.rowinfo + row);
  T acc = T(0);
#pragma unroll 4
  for (int e = e0 + lane; e < e1; e += 32) acc += __ldg(z + e) * v[__ldg(a.z_col + e)];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if (lane == 0) {
    const T r = base + acc;
    unew[row] = r;
    if (info & kRowMonitored) write_history(a, row, 0, (double)r);
    if (a.fld) write_frame<T>(a, row, r, static_cast<const T*>(a.u_n)[row]);
  }
}

// Field frame: fld[i + n * frame] = (u_new - u_n) / dt or u_new (R = 1).
template <typename T>
__global__ void frame_kernel(StepArgs a, double* fld, int64_t frame, int is_vel, double dt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double un = (double)static_cast<const T*>(a.u_new)[i];
  const double uo = (double)static_cast<const T*>(a.u_n)[i];
  fld[(size_t)i + (size_t)a.n * frame] = is_vel ? (un - uo) / dt : un;
}

// v5 prescribed-displacement rows (V5Args): one thread per listed entry,
// then one per correction row. Reads u_n, u_{n-1} and ud_old, writes u_new
// at prescribed and correction rows only (disjoint), ud_new and frc_out.
template <typename T>
__global__ void __launch_bounds__(128) v5_kernel(StepArgs a, V5Args v) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const T* un = static_cast<const T*>(a.u_n);
  const T* up = static_cast<const T*>(a.u_prev);
  T* unew = static_cast<T*>(a.u_new);
  const int64_t ti = step_index(a);
  const double dt = v.dt;
  if (g < v.n_ent) {
    const int s = __ldg(v.ent_slot + g);
    double ku = 0.0;
    for (int e = __ldg(v.k_ptr + s); e < __ldg(v.k_ptr + s + 1); ++e)
      ku = fma(__ldg(v.k_val + e), (double)un[__ldg(v.k_col + e)], ku);
    const double m = __ldg(v.slot_m + s);
    v.frc_out[(size_t)g + (size_t)v.n_ent * ti] = m * __ldg(v.accn + (size_t)ti * v.n_ent + g) + ku;
    if (!__ldg(v.ent_last + g)) return;
    // udd = (f - K u - C ud) / m  (v5.m:150), ud += dt udd  (v5.m:153)
    double cv = 0.0;
    for (int e = __ldg(v.c_ptr + s); e < __ldg(v.c_ptr + s + 1); ++e) {
      const int k = __ldg(v.c_col + e);
      const int ks = __ldg(v.c_cslot + e);
      const double udk = ks >= 0 ? v.ud_old[ks] : ((double)un[k] - (double)up[k]) / dt;
      cv = fma(__ldg(v.c_val + e), udk, cv);
    }
    double f = 0.0;
    const int fs = __ldg(v.f_sig + s);
    if (fs >= 0) f = __ldg(v.f_w + s) * (double)static_cast<const T*>(a.sig)[(size_t)ti * a.n_sig + fs];
    const double ud = v.ud_old[s] + dt * ((f - ku - cv) / m);
    v.ud_new[s] = ud;
    const int row = __ldg(v.ent_row + g);
    const T u = (T)__ldg(v.dsp + (size_t)ti * v.n_ent + g);
    unew[row] = u;
    for (int h = __ldg(v.h_ptr + s); h < __ldg(v.h_ptr + s + 1); ++h)
      a.hist[(size_t)__ldg(v.h_slot + h) + (size_t)a.q * (size_t)ti] = (double)u;
    if (v.fld) v.fld[row] = ud;
    return;
  }
  const int t = g - v.n_ent;
  if (t >= v.n_cor) return;
  const int row = __ldg(v.cor_row + t);
  double corr = 0.0;
  for (int e = __ldg(v.cor_ptr + t); e < __ldg(v.cor_ptr + t + 1); ++e) {
    const int s = __ldg(v.cor_slot + e);
    const int j = __ldg(v.slot_row + s);
    corr = fma(__ldg(v.cor_val + e), dt * v.ud_old[s] - ((double)un[j] - (double)up[j]), corr);
  }
  const T u = (T)((double)unew[row] + corr);
  unew[row] = u;
  const int hs = v.n_slot + t;
  for (int h = __ldg(v.h_ptr + hs); h < __ldg(v.h_ptr + hs + 1); ++h)
    a.hist[(size_t)__ldg(v.h_slot + h) + (size_t)a.q * (size_t)ti] = (double)u;
  if (v.fld) v.fld[row] = ((double)u - (double)un[row]) / dt;
}

__global__ void advance_kernel(int64_t* ti_dev, int64_t k) { *ti_dev += k; }

__global__ void cast_kernel(const double* in, float* out, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)in[i];
}

// ---------------------------------------------------------------------------
cudaError_t launch_step(const StepArgs& a, int precision, cudaStream_t st) {
  // Blocks of 128: the last wave ends sooner than with 256 (coupled 961,641
  // DOF FP64 27.0 us per step against 27.6, 2.7 M DOF 75.5 against 77.3, FP32
  // 57.7 against 59.5); 64 is the same, 32 is slower (32.4).
  const int threads = 128;
  const int blocks = (a.n + threads - 1) / threads;
  if (precision == 0) step_f64_r1<<<blocks, threads, 0, st>>>(a);
  else step_f32_r1<<<blocks, threads, 0, st>>>(a);
  return cudaGetLastError();
}

size_t batched_smem_bytes(int precision, int max_slice_entries) {
  const size_t elem = precision == 0 ? sizeof(double) : sizeof(float);
  return ((size_t(max_slice_entries) * 4 + 15) & ~size_t(15)) + size_t(max_slice_entries) * elem;
}

// Kernel variants of batched runs (the numbers are the names BFE_VARIANT and
// the benchmark use); R is the padded number of right-hand sides:
//   0        slice-staged row kernel step_batched: every plan and R
//   FP64 plans with the group form:
//   1, 2, 3  FP64 group kernel with 4, 2 or 1 right-hand side pairs per lane
//            (R % 64, R % 32, R % 16)
//   4, 5     the same for any R, one or two pairs of neighbours in flight
//   FP32 plans with the group form:
//   20, 22   half-warp float4 kernel step_f32_group4 (raw coefficient
//            loads) at 12 or 10 CTAs per SM: node blocks of at most 2 DOFs,
//            R a multiple of 64 or R = 16, 32
//   24 - 26  the float4 form for any R and block size, one, two or four
//            neighbours in flight
//            (forced numbers from 9 on that name no kernel run 24)
// The first candidate is the default; the autotuner keeps it unless another
// is clearly faster on the live operator.
int batched_candidates(int precision, int R, bool have_groups, int max_bs, int* out) {
  int k = 0;
  if (precision == 0) {
    if (have_groups && R % 16 == 0) {
      if (R % 64 == 0) out[k++] = 1;
      if (R % 32 == 0) out[k++] = 2;
      out[k++] = 3;
      out[k++] = 5;
    } else if (have_groups) {
      // a slice kernel's warp with 28 or more of its 32 lanes busy loses less
      // than the blocks' zeros cost on all-solid models, so it is the default
      // there and the group form has to be clearly faster (us per step, slice /
      // group: five sub-domains of 108,752 DOF R = 60 178.9 / 181.9, R = 28 91.3
      // / 83.6; coupled 60,891 DOF R = 60 105.7 / 87.2, R = 29 59.2 / 51.5)
      if (R % 32 >= 28) out[k++] = 0;
      out[k++] = 4;
      out[k++] = 5;
      if (R % 32 >= 28) return k;
    }
    out[k++] = 0;
    return k;
  }
  if (have_groups && max_bs <= 2 && (R % 64 == 0 || R == 16 || R == 32)) {
    for (int v : {20, 22}) out[k++] = v;
    return k;
  }
  // (3D nodes too, us per step of 24 / 25 / 26, bricks R = 64: 14,553 DOF 23.2 / 22.2
  // / 18.5, 46,128 DOF 36.5 / 37.0 / 34.4, 202,878 DOF 123.8 / 139.8 / 135.8; the best
  // of a warp-per-node form with packed pairs of coefficients took 21.1, 45.6 and
  // 195.8 there)
  if (have_groups) {
    for (int v : {24, 25, 26}) out[k++] = v;
    return k;
  }
  out[k++] = 0;
  return k;
}

// A step of one wave of CTAs waits for its chains of loads, and more neighbours
// in flight shorten them: adjoint of 6,642 DOF FP32 R = 24, 600 samples 21.1 ms
// with variant 24, 19.6 with 26 (20.3 in the slice kernel), 26,082 DOF R = 40, 400
// samples 21.8 / 20.6; 90,902 DOF R = 52 (5 waves of 12 CTAs per SM) 23.7 / 23.8,
// 361,802 DOF 49.8 / 53.0.
int untimed_candidate(int precision, int R, int n, bool have_groups, int max_bs) {
  int cand[8];
  batched_candidates(precision, R, have_groups, max_bs, cand);
  const int64_t lanes = (int64_t)(n / max_bs) * ((R + 3) / 4);
  return cand[0] == 24 && lanes <= (int64_t)sm_count() * 12 * 128 ? 26 : cand[0];
}

int settled_variant(int precision, int64_t R, bool have_groups, int max_bs) {
  if (!have_groups) return 0;
  if (precision == 0) return R % 16 ? 0 : R % 32 ? 3 : R % 64 ? 2 : 1;
  if (max_bs <= 2 && (R % 64 == 0 || R == 16 || R == 32)) return 20;
  return R % 64 ? 0 : 24;
}

// Prefetching pays where the three states do not fit in L2, so that a step's
// first touch of a row is a DRAM miss in a node's chain of loads; below that
// the requests are only extra work. Us per step without / with, FP32: coupled
// 961,641 DOF R = 16 65.7 / 63.4, R = 32 107.2 / 97.9, R = 64 166.7 / 150.0; bricks
// of 1,778,478 DOF R = 8 268.2 / 258.7, R = 24 571.9 / 534.8, of 202,878 R = 64
// 132.4 / 120.3, R = 256 453.5 / 443.3; states of 139 to 186 MB gain 1 to 10 %.
// Where it loses: fewer than 16 right-hand sides of one- and two-DOF nodes
// (R = 8, 2,674,573 DOF: 96.8 / 98.4: a request costs as much as the load),
// several uneven passes over R on models of up to 360,000 DOF (R = 80 plate of
// 161,202 DOF 51.1 / 55.1, R = 96 coupled 241,579 DOF 91.6 / 93.4; 961,641 DOF would
// gain, 312 / 297, as bricks of 202,878 DOF, 207 / 200 at 200), and it does nothing
// for FP64, which the FP64 pipe bounds (R = 64 271.2 / 272.4). The
// distance is long enough for a DRAM miss and short enough that the data are
// still in L2: 800 CTAs of 1,824 resident (400: 156.7, 1,200: 150.6, 2,000: 161 at
// R = 64); the wide blocks of three-DOF nodes want 200 (R = 16, 1,778,478 DOF: 363
// us, 400: 379, 800: 429).
// Above 64 right-hand sides a CTA's rows are as many times larger, and the
// distance shorter. None / 400 / 800: R = 128 plate of 161,202 DOF 61.3 / 61.5 /
// 63.0, coupled 241,579 DOF 101.5 / 98.8 / 102.8, 961,641 DOF 325 / 295 / 296; R = 192
// 161,202 DOF (371 MB of states) 90.8 / 94.4 / 100.1, 241,579 DOF (557 MB) 141.2 /
// 139.0 / 144.4, plate of 1,003,002 DOF 514 / 464 / 527. R = 256 none / 200 / 800:
// plate of 361,802 DOF (1.1 GB) 238.4 / 239.6 / 274.4, 961,641 DOF 644 / 600 / 641.
// R = 320 only loses (361,802 DOF 295.5 / 306.5 at 200; bricks of 46,128 DOF 157.6 /
// 161.6).
int group_ahead(const StepArgs& a, const GroupArgs& g) {
  const size_t state = 3 * (size_t)a.n * (size_t)a.R * sizeof(float), l2 = (size_t)l2_bytes();
  if (l2 == 0 || state <= l2 || (a.R > 64 && a.R % 64 != 0) || a.R > 256) return 0;
  if (group_max_bs(g) > 2) return a.R < 8 ? 0 : 200;
  if (a.R <= 128) return a.R < 16 ? 0 : a.R <= 64 ? 800 : 400;
  return a.R == 192 ? (state >= 4 * l2 ? 400 : 0) : (state >= 12 * l2 ? 200 : 0);
}

int group_max_bs(const GroupArgs& g) {
  int maxbs = 1;
  for (int k = 0; k < g.n_groups; ++k) maxbs = g.bs[k] > maxbs ? g.bs[k] : maxbs;
  return maxbs;
}

cudaError_t launch_step_batched(const StepArgs& a, const GroupArgs* gr, int precision, int max_slice_entries,
                                int variant, cudaStream_t st) {
  const int threads = 256;
  const size_t smem = batched_smem_bytes(precision, max_slice_entries);
  if (precision == 0) {
    if (variant >= 1 && variant <= 5 && gr) return launch_group64_variant(a, *gr, variant, st);
    step_batched<double, 1><<<a.n_slices, threads, smem, st>>>(a);
    return cudaGetLastError();
  }
  const int maxbs = gr ? group_max_bs(*gr) : 0;
  const bool r64 = a.R % 64 == 0, r1632 = a.R == 16 || a.R == 32;
  const bool half_warp = variant == 20 || variant == 22;
  if (gr && variant >= 24 && variant <= 26) {
    launch_groupn_variant(maxbs, a, *gr, variant, st);
  } else if (gr && half_warp && maxbs <= 2 && (r64 || r1632)) {
    launch_group4_variant(r64 ? 16 : a.R == 32 ? 8 : 4, a, *gr, variant, st);
  } else if (gr && variant >= 9) {                    // 20 and 22 where they do not apply
    launch_groupn_variant(maxbs, a, *gr, 24, st);
  } else if (r64) {
    step_batched<float, 2><<<a.n_slices, threads, smem, st>>>(a);
  } else {
    step_batched<float, 1><<<a.n_slices, threads, smem, st>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t set_batched_smem_limit(int precision) {
  const int smem = (int)kBatchedSmem;
  cudaError_t e;
  if (precision == 0) {
    e = cudaFuncSetAttribute(step_batched<double, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  } else {
    e = cudaFuncSetAttribute(step_batched<float, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(step_batched<float, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  }
  return e;
}

cudaError_t launch_interface_fixup(const StepArgs& a, int precision, cudaStream_t st) {
  if (a.n_int == 0) return cudaSuccess;
  const int threads = 256;
  if (a.R == 1) {
    const int blocks = (int)(((int64_t)a.n_int * 32 + threads - 1) / threads);
    if (precision == 0) interface_fixup_r1<double><<<blocks, threads, 0, st>>>(a);
    else interface_fixup_r1<float><<<blocks, threads, 0, st>>>(a);
    return cudaGetLastError();
  }
  if (precision != 0 && a.R % 4 == 0) {
    const int64_t total = (int64_t)a.n_int * (a.R / 4);
    interface_fixup_vec<float, float4, 4><<<(int)((total + threads - 1) / threads), threads, 0, st>>>(a);
    return cudaGetLastError();
  }
  if (precision == 0 && a.R % 2 == 0) {
    const int64_t total = (int64_t)a.n_int * (a.R / 2);
    interface_fixup_vec<double, double2, 2><<<(int)((total + threads - 1) / threads), threads, 0, st>>>(a);
    return cudaGetLastError();
  }
  const int64_t total = (int64_t)a.n_int * a.R;
  const int blocks = (int)((total + threads - 1) / threads);
  if (precision == 0) interface_fixup<double><<<blocks, threads, 0, st>>>(a);
  else interface_fixup<float><<<blocks, threads, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename T>
__global__ void nonfinite_kernel(const T* __restrict__ u, int64_t count, int* flag) {
  bool bad = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    bad |= !isfinite(u[i]);
  if (__syncthreads_or(bad) && threadIdx.x == 0) *flag = 1;
}

cudaError_t launch_nonfinite_check(const void* u, int64_t count, int precision, int* flag, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const int threads = 256;
  const int64_t need = (count + threads - 1) / threads;
  const int blocks = (int)std::min<int64_t>(need, (int64_t)sm_count() * 8);
  if (precision == 0) nonfinite_kernel<double><<<blocks, threads, 0, st>>>(static_cast<const double*>(u), count, flag);
  else nonfinite_kernel<float><<<blocks, threads, 0, st>>>(static_cast<const float*>(u), count, flag);
  return cudaGetLastError();
}

cudaError_t launch_frame(const StepArgs& a, int precision, double* fld, int64_t frame,
                         int field_is_vel, double dt, cudaStream_t st) {
  const int threads = 256;
  const int blocks = (a.n + threads - 1) / threads;
  if (precision == 0) frame_kernel<double><<<blocks, threads, 0, st>>>(a, fld, frame, field_is_vel, dt);
  else frame_kernel<float><<<blocks, threads, 0, st>>>(a, fld, frame, field_is_vel, dt);
  return cudaGetLastError();
}

cudaError_t launch_v5(const StepArgs& a, const V5Args& v, int precision, cudaStream_t st) {
  const int total = v.n_ent + v.n_cor;
  if (total == 0) return cudaSuccess;
  const int threads = 128;
  const int blocks = (total + threads - 1) / threads;
  if (precision == 0) v5_kernel<double><<<blocks, threads, 0, st>>>(a, v);
  else v5_kernel<float><<<blocks, threads, 0, st>>>(a, v);
  return cudaGetLastError();
}

cudaError_t launch_advance(int64_t* ti_dev, int64_t k, cudaStream_t st) {
  advance_kernel<<<1, 1, 0, st>>>(ti_dev, k);
  return cudaGetLastError();
}

cudaError_t launch_cast_f64_to_f32(const double* in, float* out, int64_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int threads = 256;
  cast_kernel<<<(int)((n + threads - 1) / threads), threads, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

}  // namespace bfe
