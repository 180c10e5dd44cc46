// March of several sources that stays on the chip (sm_103a): the one-source
// form (bfe_onchip.cu) with R right-hand sides, for models whose R states, halo
// and operator all fit in shared memory (R n up to about 2 million values in
// FP32), without interface rows.
//
// Such a march is as short of work per step as a one-source one: a step kernel
// of 90,902 DOF and 16 sources takes 9.6 us from a graph, most of it launch
// and one chain of dependent loads, and 15.8 us when every state goes to a
// slot of its own in HBM (the adjoint). A warp takes a slice (lane = row) and
// RV right-hand sides, so an entry's value and index are loaded once for RV
// multiply-adds; states are planes [R][window], so lanes of a gather fall on
// neighbouring words. Exchange words hold two FP32 values or one FP64 value,
// each 4 bytes beside their step number. Its volume, R words a halo row, bounds
// the march for many sources, so 2D models are cut into tiles (o.row_of,
// bfe_onchip_host.cpp) where contiguous rows would be strips of a mesh column
// or two, all read by other parts: 90,902 DOF, R = 16 12.0 us per step in
// strips (604 halo rows a part), 7.1 in tiles (about 150); 40,602 DOF R = 16
// 8.8 / 4.7, R = 4 3.3 / 2.8. With m.out every new state is also
// written to global memory, [n][R] at m.out + k m.out_stride.
//
// Arithmetic and order are those of the group kernels (step_f32_groupn,
// step_f64_group), so the results are the same bits while the state is finite.
// 90,902 DOF, R = 16 in tiles (ncu): 60 % of the issue slots, 46 % of the
// shared-memory pipe.
#include <cuda_runtime.h>
#include <cstdint>

#include "bfe_onchip.cuh"

namespace bfe {

namespace {

// A state element of 8 bytes: two FP32 right-hand sides (packed arithmetic,
// rounded per component as the scalar operations) or one FP64 one.
template <typename T> struct Elem;
template <> struct Elem<float> { using E = float2; static constexpr int kPer = 2; };
template <> struct Elem<double> { using E = double; static constexpr int kPer = 1; };
constexpr int kRe = 2;                                  // elements per thread
constexpr int kSlPaired = kSlResident;                  // (all slices are resident here)

__device__ __forceinline__ float2 e_sub(float2 a, float2 b) { return f2sub(a, b); }
__device__ __forceinline__ float2 e_fma(float c, float2 x, float2 acc) {
  return __ffma2_rn(make_float2(c, c), x, acc);
}
__device__ __forceinline__ double e_fma(double c, double x, double acc) { return fma(c, x, acc); }
__device__ __forceinline__ void e_zero(float2& x) { x = make_float2(0.f, 0.f); }
__device__ __forceinline__ void e_zero(double& x) { x = 0.0; }
// component y of an element
__device__ __forceinline__ float& e_at(float2& x, int y) { return y ? x.y : x.x; }
__device__ __forceinline__ double& e_at(double& x, int) { return x; }
// New values of a row (row_update): acc is its sum, f its forcing.
__device__ __forceinline__ double e_update(double acc, double, double up, double rc, bool forced, double f) {
  double r = acc + rc * up;
  if (forced) r += f;
  return r;
}
__device__ __forceinline__ float2 e_update(float2 acc, float2 ui, float2 up, float rc, bool forced, float2 f) {
  float2 d, err;
  two_sum2(ui, make_float2(-up.x, -up.y), d, err);
  const float2 q = make_float2(rc, rc);
  float2 inc = __ffma2_rn(q, d, make_float2(-acc.x, -acc.y));
  if (forced) inc = __fadd2_rn(inc, f);
  inc = __ffma2_rn(q, err, inc);
  return __fadd2_rn(ui, inc);
}

// Exchange words of 16 bytes: an element, each half with the step number.
__device__ __forceinline__ void wput(uint4* w, float2 v, uint32_t tag) {
  put_words(w, word(__float_as_uint(v.x), tag), word(__float_as_uint(v.y), tag));
}
__device__ __forceinline__ void wput(uint4* w, double v, uint32_t tag) {
  xput(reinterpret_cast<double*>(w), 0, v, tag);
}
__device__ __forceinline__ bool wtry(const uint4* w, uint32_t tag, float2& v) {
  uint32_t lo, hi;
  const bool ok = get_words(w, tag, lo, hi);
  v = make_float2(__uint_as_float(lo), __uint_as_float(hi));
  return ok;
}
__device__ __forceinline__ bool wtry(const uint4* w, uint32_t tag, double& v) {
  return xtry(reinterpret_cast<const double*>(w), 0, tag, v);
}
template <typename E>
__device__ __noinline__ bool wwait(const uint4* w, uint32_t tag, E& v, int* err) {
  long long t0 = 0;
  E x;
  for (uint32_t spin = 1; !wtry(w, tag, x); ++spin) {
    if ((spin & 255u) == 0) {
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (now - t0 > kSpinClocks) atomicExch(err, 1);
      if (*reinterpret_cast<volatile int*>(err)) return false;
    }
  }
  v = x;
  return true;
}

// Adds a chunk's entries to the row sums; au: byte offset of the first plane,
// ws: bytes of a plane. The forms of row_sum (bfe_onchip.cuh).
__device__ __forceinline__ void row_sums(double (&acc)[kRe], const unsigned char* blk, int lane, int, int w,
                                         const unsigned char* sm, uint32_t au, uint32_t ws, const double (&)[3][kRe]) {
  const int np = (w + 1) >> 1;
  const double2* v = reinterpret_cast<const double2*>(blk) + lane;
  const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + np * 512) + lane;
#pragma unroll 2
  for (int k = 0; k < np; ++k) {
    const double2 x = v[32 * k];
    const uint32_t cc = c[32 * k], c0 = au + 8 * (cc & 0xffffu), c1 = au + 8 * (cc >> 16);
#pragma unroll
    for (int r = 0; r < kRe; ++r) acc[r] = fma(x.x, sm_at<double>(sm, c0 + r * ws), acc[r]);
    if (2 * k + 1 < w) {
#pragma unroll
      for (int r = 0; r < kRe; ++r) acc[r] = fma(x.y, sm_at<double>(sm, c1 + r * ws), acc[r]);
    }
  }
}
// Slices whose nodes all start at an even place of the window: both DOFs of a
// neighbour (kind 2) come with one 16-byte load, fewer instructions and
// shared-memory wavefronts (two lanes of a node read the same words, so 16
// distinct ones per load either way): 6.5 instead of 10.5 wavefronts a neighbour, 90,902 DOF R = 16
// 16,000 -> 13,700 clocks of rows per step. Eight right-hand sides per lane in
// place of four: no faster at R = 16 (12.3 us per step both), slower at R = 8
// (6.7 / 5.7).
__device__ __forceinline__ void row_sums_paired(float2 (&acc)[kRe], const unsigned char* blk, int lane, int u,
                                                const unsigned char* sm, uint32_t au, uint32_t ws,
                                                const float2 (&ref)[3][kRe]) {
  const float2* v = reinterpret_cast<const float2*>(blk) + lane;
  const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * 256) + lane;
#pragma unroll 4
  for (int k = 0; k < u; ++k) {
    const uint32_t cc = c[32 * (k >> 1)], c0 = au + 2 * (k & 1 ? cc >> 16 : cc & 0xffffu);
    const float2 x = v[32 * k];
#pragma unroll
    for (int r = 0; r < kRe; ++r) {
      const float4 n = sm_at<float4>(sm, c0 + r * ws);
      acc[r] = e_fma(x.x, e_sub(make_float2(n.x, n.y), ref[0][r]), acc[r]);
      acc[r] = e_fma(x.y, e_sub(make_float2(n.z, n.w), ref[1][r]), acc[r]);
    }
  }
}
__device__ __forceinline__ void row_sums_paired(double (&)[kRe], const unsigned char*, int, int, const unsigned char*,
                                                uint32_t, uint32_t, const double (&)[3][kRe]) {}
__device__ __forceinline__ void split4(const float4& n, float2& lo, float2& hi) {
  lo = make_float2(n.x, n.y);
  hi = make_float2(n.z, n.w);
}
__device__ __forceinline__ void split4(const float4&, double&, double&) {}

__device__ __forceinline__ void row_sums(float2 (&acc)[kRe], const unsigned char* blk, int lane, int kind, int u,
                                         const unsigned char* sm, uint32_t au, uint32_t ws, const float2 (&ref)[3][kRe]) {
  auto add = [&](float x, uint32_t at, const float2 (&rf)[kRe]) {
#pragma unroll
    for (int r = 0; r < kRe; ++r) acc[r] = e_fma(x, e_sub(sm_at<float2>(sm, at + r * ws), rf[r]), acc[r]);
  };
  // the blocks' byte offsets are of 4-byte values, elements take 8
  if (kind >= 2) {
    const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * kind * 128) + lane;
    const float* v = reinterpret_cast<const float*>(blk);
#pragma unroll 2
    for (int k = 0; k < u; ++k) {
      const uint32_t cc = c[32 * (k >> 1)], c0 = au + 2 * (k & 1 ? cc >> 16 : cc & 0xffffu);
      if (kind == 2) {
        const float2 x = reinterpret_cast<const float2*>(v)[32 * k + lane];
        add(x.x, c0, ref[0]);
        add(x.y, c0 + 8, ref[1]);
      } else {
        add(v[96 * k + lane], c0, ref[0]);
        add(v[96 * k + 32 + lane], c0 + 8, ref[1]);
        add(v[96 * k + 64 + lane], c0 + 16, ref[2]);
      }
    }
    return;
  }
  const float2* v = reinterpret_cast<const float2*>(blk) + lane;
  const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * 256) + lane;
  for (int k = 0; k < u; ++k) {
    const float2 x = v[32 * k];
    const uint32_t cc = c[32 * k];
    if (kind == 1) {
      add(x.x, au + 2 * (cc & 0xffffu), ref[0]);
      add(x.y, au + 2 * (cc >> 16), ref[0]);
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t ch = h ? cc >> 16 : cc & 0xffffu, s = ch & 3u;
        float2 rf[kRe];
#pragma unroll
        for (int r = 0; r < kRe; ++r) {
          rf[r].x = (s & 2u) ? ((s & 1u) ? 0.f : ref[2][r].x) : ((s & 1u) ? ref[1][r].x : ref[0][r].x);
          rf[r].y = (s & 2u) ? ((s & 1u) ? 0.f : ref[2][r].y) : ((s & 1u) ? ref[1][r].y : ref[0][r].y);
        }
        add(h ? x.y : x.x, au + 2 * (ch & 0xfffcu), rf);
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(1024, 1) march_onchip_multi(OnchipArgs o, StepArgs a, OnchipMulti m, int64_t n_steps,
                                                              int fresh) {
  using E = typename Elem<T>::E;
  constexpr int PER = Elem<T>::kPer, RV = kRe * PER;
  struct alignas(16) Pack { E e[kRe]; };
  extern __shared__ __align__(16) unsigned char sm[];
  const int p = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  const int s0 = o.part_slice[p], s1 = o.part_slice[p + 1];
  const int ns = s1 - s0, row0 = s0 * kSlice, rpad = ns * kSlice;
  const int rows = min(a.n - row0, rpad);
  const int R = a.R, nc = R / RV, wpr = R / PER;        // chunks and exchange words of a row
  const int H = o.halo_cnt[p];
  const int W = onchip_multi_window(rpad + H);
  const uint32_t ws = (uint32_t)(W * sizeof(E));        // bytes of a plane (of PER right-hand sides)
  const int f0 = lower_bound_i32(a.frc_row, a.n_frc, row0);
  const int nf = lower_bound_i32(a.frc_row, a.n_frc, row0 + rows) - f0;
  const int m0 = lower_bound_i32(a.mon_row, a.n_mon, row0);
  const int nm = lower_bound_i32(a.mon_row, a.n_mon, row0 + rows) - m0;
  T* U = reinterpret_cast<T*>(sm);
  T* fco = U + 2 * R * W;                               // forcing: coefficients, signals of two steps
  T* fs = fco + ((nf + 1) & ~1);
  int2* sd = reinterpret_cast<int2*>(fs + 2 * ((nf + 1) & ~1));
  int32_t* frw = reinterpret_cast<int32_t*>(sd + ns);   // its rows and right-hand sides
  int32_t* frr = frw + nf;
  int32_t* mrow = frr + nf;
  int32_t* mslot = mrow + nm;
  int32_t* hr = mslot + nm;                             // halo rows
  int32_t* orow = hr + H;                               // the rows' places in the caller's states
  uint16_t* fl = reinterpret_cast<uint16_t*>(orow + rpad);
  unsigned char* cache = sm + ((reinterpret_cast<unsigned char*>(fl + rpad) - sm + 15) & ~15);

  for (int r = tid; r < rpad; r += nt) {
    fl[r] = r < rows ? __ldg(o.flags + row0 + r) : 0;
    orow[r] = r < rows && o.row_of ? __ldg(o.row_of + row0 + r) : row0 + r;
  }
  for (int k = tid; k < nf; k += nt) {
    frw[k] = __ldg(a.frc_row + f0 + k) - row0;
    frr[k] = __ldg(a.frc_rhs + f0 + k);
    fco[k] = __ldg(static_cast<const T*>(a.frc_coef) + f0 + k);
  }
  for (int k = tid; k < nm; k += nt) {
    mrow[k] = __ldg(a.mon_row + m0 + k) - row0;
    mslot[k] = __ldg(a.mon_slot + m0 + k);
  }
  for (int k = tid; k < H; k += nt) hr[k] = __ldg(o.halo_row + (size_t)p * o.halo_cap + k);
  for (int j = tid; j < ns; j += nt) {
    const int ls = __ldg(o.order + s0 + j), y = __ldg(o.slice_word + s0 + ls);
    sd[j] = make_int2(__ldg(o.block_off + s0 + ls), y | (ls << kSlLocalShift));
  }
  __syncthreads();
  for (int k = tid; k < nf; k += nt)
    if (k == 0 || frw[k] != frw[k - 1]) fl[frw[k]] |= (uint16_t)kOcForced;
  {
    int off = 0;
    for (int j = 0; j < ns; ++j) {
      const int2 d = sd[j];
      const int bytes = block_bytes<T>(sl_kind(d.y), sl_units<T>(d.y));
      if (j % nw == warp) {
        const int4* src = reinterpret_cast<const int4*>(static_cast<const unsigned char*>(o.blocks) + (size_t)d.x * 16);
        for (int k = lane; k < bytes / 16; k += 32) reinterpret_cast<int4*>(cache + off)[k] = __ldg(src + k);
        __syncwarp();
        bool paired = sizeof(T) == 4 && sl_kind(d.y) == 2;
        if (paired) {
          const int r = (d.y >> kSlLocalShift) * kSlice + lane, un = sl_units<T>(d.y), cu = chunk_units<T>(2);
          uint32_t odd = (uint32_t)(r - ((fl[r] >> kOcPosShift) & 7)) << 2;
          for (int k = 0; k < un; k += cu) {
            const int u = min(cu, un - k);
            const uint32_t* c = reinterpret_cast<const uint32_t*>(cache + off + coef_bytes<T>() + k / cu * units_bytes<T>(2, cu) + u * 256);
            for (int h = 0; 2 * h < u; ++h) odd |= c[32 * h + lane] | c[32 * h + lane] >> 16;
          }
          paired = __all_sync(0xffffffffu, !(odd & 4u));
        }
        if (lane == 0) {
          sd[j].x = off;
          if (paired) sd[j].y = d.y | kSlPaired;
        }
      }
      off += bytes;
    }
  }
  for (int k = tid; k < R * W; k += nt) {
    const int r = k / W, x = k - r * W;
    T un = T(0), up = T(0);
    int g = x < rpad ? (x < rows ? orow[x] : -1) : (x < rpad + H ? hr[x - rpad] : -1);
    if (x >= rpad && g >= 0 && o.row_of) g = __ldg(o.row_of + g);
    if (!fresh && g >= 0) {
      un = static_cast<const T*>(a.u_n)[(size_t)g * R + r];
      if (x < rpad) up = static_cast<const T*>(a.u_prev)[(size_t)g * R + r];
    }
    const int at = (r / PER * W + x) * PER + r % PER;
    U[at] = un;
    U[R * W + at] = up;
  }
  // this thread's forcing signal, one step ahead in freg
  const T* fsig = static_cast<const T*>(a.sig);
  T freg = T(0);
  if (tid < nf) {
    fsig += (int64_t)a.n_sig * m.ti0 + __ldg(a.frc_sig + f0 + tid);
    fs[tid] = __ldg(fsig);
    fsig += m.ti_step * a.n_sig;
    if (n_steps > 1) freg = __ldg(fsig);
  }
  uint4* const x0 = static_cast<uint4*>(o.xch);
  uint4* const x1 = x0 + o.x_stride;
  T* out = static_cast<T*>(m.out);
  __syncthreads();

  const uint32_t nc_magic = nc == 1 ? 0u : (uint32_t)((0x100000000ull + nc - 1) / nc);
  uint32_t au = 0, bu = (uint32_t)wpr * ws;             // byte offsets of u_n and of u_{n-1} / u_{n+1}
  bool bad = false;
  for (int64_t k = 0; k <= n_steps; ++k) {
    const uint32_t tag = o.tag0 + (uint32_t)k;
    if (k > 0)                                          // samples of the state just completed
      for (int e = tid; e < nm * a.R_out; e += nt) {
        const int r = e / nm, x = e - r * nm;
        a.hist[(size_t)mslot[x] + (size_t)a.q * ((size_t)(m.ti0 + (k - 1) * m.ti_step) + (size_t)a.n_t * r)] =
            (double)sm_at<T>(sm, au + r / PER * ws + mrow[x] * (uint32_t)sizeof(E) + r % PER * (uint32_t)sizeof(T));
      }
    if (k == n_steps) break;
    if (tid < nf) {
      fs[((k + 1) & 1) * nf + tid] = freg;
      fsig += m.ti_step * a.n_sig;
      if (k + 2 < n_steps) freg = __ldg(fsig);
    }
    uint4* xw = k & 1 ? x1 : x0;
    for (int t = warp; t < ns * nc; t += nw) {
      const int j = nc == 1 ? t : (int)__umulhi((uint32_t)t, nc_magic), c = t - j * nc, r0 = c * RV;
      const int2 d = sd[j];
      const int kind = sizeof(T) == 8 ? 0 : sl_kind(d.y), r = (d.y >> kSlLocalShift) * kSlice + lane;
      const uint32_t ap = au + r0 / PER * ws, at = ap + r * (uint32_t)sizeof(E), bt = at - au + bu;
      const uint32_t f = fl[r];
      E ui[kRe], ref[3][kRe], acc[kRe];
#pragma unroll
      for (int v = 0; v < kRe; ++v) {
        ui[v] = sm_at<E>(sm, at + v * ws);
        ref[0][v] = ui[v];
        e_zero(acc[v]);
      }
      const bool paired = sizeof(T) == 4 && (d.y & kSlPaired);
      if (paired) {
        const uint32_t own = at - 8 * ((f >> kOcPosShift) & 7);
#pragma unroll
        for (int v = 0; v < kRe; ++v) split4(sm_at<float4>(sm, own + v * ws), ref[0][v], ref[1][v]);
      } else if (sizeof(T) == 4 && kind != 1) {
        const int pos = (int)(f >> kOcPosShift) & 7;
        int q0 = r - pos, q1 = q0 + 1, q2 = q0 + 2;
        if (kind == 0 && pos == (int)kOcCut) {
          const ushort4 x = o.lref[row0 + r];
          q0 = x.x, q1 = x.y, q2 = x.z;
        }
        __syncwarp();
#pragma unroll
        for (int v = 0; v < kRe; ++v) {
          ref[0][v] = sm_at<E>(sm, ap + v * ws + 8 * q0);
          ref[1][v] = sm_at<E>(sm, ap + v * ws + 8 * q1);
          ref[2][v] = sm_at<E>(sm, ap + v * ws + 8 * q2);
        }
      }
      const unsigned char* blk = cache + d.x;
      const T rc = reinterpret_cast<const T*>(blk)[lane];
      blk += coef_bytes<T>();
      const int cu = chunk_units<T>(kind), full = sizeof(T) == 8 ? 2 * cu : cu, step = units_bytes<T>(kind, cu);
      if (paired)
        for (int left = sl_width(d.y); left > 0; left -= full, blk += step)
          row_sums_paired(acc, blk, lane, min(left, full), sm, ap, ws, ref);
      else
        for (int left = sl_width(d.y); left > 0; left -= full, blk += step)
          row_sums(acc, blk, lane, kind, min(left, full), sm, ap, ws, ref);
      E ft[kRe];
#pragma unroll
      for (int v = 0; v < kRe; ++v) e_zero(ft[v]);
      if (f & kOcForced) {
        for (int e = lower_bound_sm(frw, nf, r); e < nf && frw[e] == r; ++e)
#pragma unroll
          for (int v = 0; v < RV; ++v)
            if (frr[e] == r0 + v) {
              T& x = e_at(ft[v / PER], v % PER);
              x = fma(fco[e], fs[(k & 1) * nf + e], x);
            }
      }
      Pack pk;
#pragma unroll
      for (int v = 0; v < kRe; ++v) {
        pk.e[v] = e_update(acc[v], ui[v], sm_at<E>(sm, bt + v * ws), rc, (f & kOcForced) != 0, ft[v]);
        *reinterpret_cast<E*>(sm + bt + v * ws) = pk.e[v];
      }
      if (f & kOcExport) {
        uint4* w = xw + (size_t)(row0 + r) * wpr + r0 / PER;
#pragma unroll
        for (int v = 0; v < kRe; ++v) wput(w + v, pk.e[v], tag);
      }
      if (out && r < rows) *reinterpret_cast<Pack*>(out + (size_t)orow[r] * R + r0) = pk;
    }
    out = out ? out + m.out_stride : out;
    if (k + 1 < n_steps) {
      // halo of the new state, four words of a thread in flight
      for (int e0 = tid; e0 < H * wpr; e0 += 4 * nt) {
        const uint4* w[4];
        uint32_t dst[4];
        E v[4];
        bool got[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int e = e0 + i * nt;
          got[i] = e >= H * wpr;
          const int h = got[i] ? 0 : (int)__umulhi((uint32_t)e, m.wpr_magic), x = got[i] ? 0 : e - h * wpr;
          w[i] = xw + (size_t)hr[h] * wpr + x;
          dst[i] = bu + (uint32_t)x * ws + (uint32_t)(rpad + h) * (uint32_t)sizeof(E);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) got[i] = got[i] || wtry(w[i], tag, v[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (e0 + i * nt >= H * wpr) continue;
          if (!got[i] && !bad) bad = !wwait(w[i], tag, v[i], o.err);
          *reinterpret_cast<E*>(sm + dst[i]) = v[i];
        }
      }
    }
    if (__syncthreads_or(bad)) return;
    const uint32_t x = au;
    au = bu;
    bu = x;
  }
  // the two newest states back to global memory (as march_onchip)
  if (!a.u_new) return;
  for (int k = tid; k < rows * R; k += nt) {
    const int x = k / R, r = k - x * R;
    const uint32_t at = r / PER * ws + x * (uint32_t)sizeof(E) + r % PER * (uint32_t)sizeof(T);
    static_cast<T*>(a.u_new)[(size_t)orow[x] * R + r] = sm_at<T>(sm, au + at);
    const_cast<T*>(static_cast<const T*>(a.u_prev))[(size_t)orow[x] * R + r] = sm_at<T>(sm, bu + at);
  }
}

template <typename T>
cudaError_t launch_t(const OnchipArgs& o, const StepArgs& a, const OnchipMulti& m, int64_t n_steps, int fresh,
                     cudaStream_t st) {
  auto* kern = march_onchip_multi<T>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kOnchipSmem);
  if (e != cudaSuccess) return e;
  OnchipArgs oo = o;
  StepArgs aa = a;
  OnchipMulti mm = m;
  const uint32_t wpr = (uint32_t)(a.R / Elem<T>::kPer);      // at least 2: R is a multiple of kRe kPer
  mm.wpr_magic = (uint32_t)((0x100000000ull + wpr - 1) / wpr);
  void* args[] = {&oo, &aa, &mm, &n_steps, &fresh};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kern), dim3(o.n_parts), dim3(o.threads), args,
                                     (size_t)o.smem, st);
}

}  // namespace

int onchip_multi_rv(int precision) { return kRe * (precision == 0 ? Elem<double>::kPer : Elem<float>::kPer); }

cudaError_t launch_onchip_multi(const OnchipArgs& o, const StepArgs& a, const OnchipMulti& m, int precision,
                                int64_t n_steps, int fresh, cudaStream_t st) {
  return precision == 0 ? launch_t<double>(o, a, m, n_steps, fresh, st) : launch_t<float>(o, a, m, n_steps, fresh, st);
}

}  // namespace bfe
