// Device helpers of the marches that stay on the chip (bfe_onchip.cu,
// bfe_onchip_multi.cu): row flags, exchange words, operator blocks.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "bfe_device.cuh"
#include "bfe_internal.h"

namespace bfe {

// Flag word of a row (shared memory): bits 0-3; in 4-6 the row's place in its
// node block (FP32: reference values are the block's rows), kOcCut when the
// block is cut by the part's edge; interface number in 7-15.
constexpr uint32_t kOcExport = 1, kOcInterface = 2, kOcForced = 4, kOcExportV = 8;
constexpr int kOcPosShift = 4, kOcIntShift = 7;
constexpr uint32_t kOcCut = 7, kOcMaxInt = 511;
// A prescribed row of the v5 scheme: an interface number without the
// interface bit (such rows are no interface rows).
__device__ __forceinline__ bool is_slot(uint32_t f) { return !(f & kOcInterface) && (f >> kOcIntShift); }

// ---------------------------------------------------------------------------
// Exchange words. 4 bytes of a value and the step number are the halves of one
// 64-bit word, and every access is of whole 64-bit scalars (as .v2 where two
// words lie side by side), which memory never tears: a reader that sees the
// step number has the value too. Relaxed: nothing else is published by them.
__device__ __forceinline__ uint64_t word(uint32_t v, uint32_t tag) { return (uint64_t)tag << 32 | v; }
__device__ __forceinline__ void put_words(void* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1,%2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ bool get_words(const void* p, uint32_t tag, uint32_t& lo, uint32_t& hi) {
  uint64_t a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  lo = (uint32_t)a;
  hi = (uint32_t)b;
  return (uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag;
}
__device__ __forceinline__ void xput(double* base, size_t i, double v, uint32_t tag) {
  put_words(base + 2 * i, word((uint32_t)__double2loint(v), tag), word((uint32_t)__double2hiint(v), tag));
}
__device__ __forceinline__ void xput(float* base, size_t i, float v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(base + 2 * i), "l"(word(__float_as_uint(v), tag)) : "memory");
}
__device__ __forceinline__ bool xtry(const double* base, size_t i, uint32_t tag, double& v) {
  uint32_t lo, hi;
  const bool ok = get_words(base + 2 * i, tag, lo, hi);
  v = __hiloint2double((int)hi, (int)lo);
  return ok;
}
__device__ __forceinline__ bool xtry(const float* base, size_t i, uint32_t tag, float& v) {
  uint64_t a;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(base + 2 * i) : "memory");
  v = __uint_as_float((uint32_t)a);
  return (uint32_t)(a >> 32) == tag;
}

// About two seconds of the SM clock: far above any wait of a running march.
constexpr long long kSpinClocks = 4000000000ll;

// A value from exchange slot i, polled until it carries tag. false: gave up.
template <typename T>
__device__ __noinline__ bool xwait(const T* xbuf, uint32_t i, uint32_t tag, T& v, int* err) {
  long long t0 = 0;
  T x;
  for (uint32_t spin = 1; !xtry(xbuf, i, tag, x); ++spin) {
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
// The values of exchange slots idx[tid], idx[tid + nt], ... into dst. The
// thread's first N slots are held in registers (ix) and their first polls are
// in flight together.
template <typename T, int N>
__device__ __forceinline__ bool receive(const T* xbuf, const int32_t* __restrict__ idx, int count, const int (&ix)[N],
                                        uint32_t tag, T* dst, int tid, int nt, int* err) {
  if (tid >= count) return true;
  T v[N];
  bool got[N], ok = true;
#pragma unroll
  for (int j = 0; j < N; ++j) got[j] = tid + j * nt >= count || xtry(xbuf, (uint32_t)ix[j], tag, v[j]);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (!got[j]) ok &= xwait(xbuf, (uint32_t)ix[j], tag, v[j], err);
    if (tid + j * nt < count) dst[tid + j * nt] = v[j];
  }
  for (int k = tid + N * nt; k < count && ok; k += nt) {
    T x;
    ok = xwait(xbuf, (uint32_t)__ldg(idx + k), tag, x, err);
    dst[k] = x;
  }
  return ok;
}

__device__ __forceinline__ int lower_bound_sm(const int32_t* a, int n, int key) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Bulk copies of operator chunks into shared memory, completion on an
// mbarrier (one phase per copy).
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tfence.mbarrier_init.release.cluster;" ::"r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // after the warp's reads of the old contents
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
// Wait for the phase with this parity; false after about two seconds.
static __device__ bool bar_wait(uint64_t* bar, uint32_t parity, int* err) {
  long long t0 = 0;
  for (uint32_t spin = 1;; ++spin) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((spin & 63u) == 0) {
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (now - t0 > kSpinClocks) {
        atomicExch(err, 1);
        return false;
      }
    }
  }
}

// Operator blocks. The block of a slice (32 rows, lane = row) is the rows'
// update coefficients followed by chunks of entries; a chunk is what one bulk
// copy moves, about 3 KB. The entries of a slice are of one kind:
//   0, 1  single entries in pairs: values as T2 per lane, then the pair's two
//         window indices in one word. Kind 0 is any row (FP64: all rows).
//         FP32 kind 0 names in the index's low bits which of the row's three
//         reference values is subtracted (3: none); kind 1 are rows whose
//         entries all subtract the row's own value (fluid).
//   2, 3  FP32 rows whose entries subtract the matching DOF of the row's own
//         node, by neighbour node: the node's 2 or 3 values (absent entries
//         as zeros), one window index for all of them.
// FP32 indices are byte offsets into the window (4 x index, at most 64 KB).
// An entry of kind 0 takes about 14 instructions, one of kind 2 under 4, and
// FP32 rows are bound by instruction issue: C1's 961,641 rows took 12.4 us of
// a step as kind 0.
template <typename T> __host__ __device__ constexpr int coef_bytes() { return 32 * (int)sizeof(T); }
// Units (pairs or nodes) of a full chunk, bytes of a chunk of u units.
template <typename T>
__host__ __device__ inline int chunk_units(int kind) { return sizeof(T) == 8 ? 4 : kind == 3 ? 6 : 8; }
template <typename T>
__host__ __device__ inline int units_bytes(int kind, int u) {
  if (kind < 2) return u * 64 * ((int)sizeof(T) + 2);
  return u * kind * 128 + ((u + 1) >> 1) * 128;
}
// Units of a slice of so many entries (kinds 0, 1) or nodes per row.
__host__ __device__ inline int slice_units(int kind, int width) { return kind < 2 ? (width + 1) >> 1 : width; }
template <typename T>
__host__ __device__ inline int block_bytes(int kind, int units) {
  const int cu = chunk_units<T>(kind);
  return coef_bytes<T>() + units / cu * units_bytes<T>(kind, cu) + units_bytes<T>(kind, units % cu);
}
// Space kept for the block of a slice of this many entries per row; a slice
// that would need more as kind 2 or 3 (many absent entries) stays kind 0.
template <typename T>
__host__ __device__ inline int block_bound(int width) {
  const int b = block_bytes<T>(0, slice_units(0, width));
  return sizeof(T) == 8 ? b : (b + b / 4 + 512) & ~15;
}
// Offset and bytes of chunk c in its block; chunk 0 includes the coefficients.
template <typename T>
__device__ __forceinline__ int chunk_offset(int kind, int c) {
  return c == 0 ? 0 : coef_bytes<T>() + c * units_bytes<T>(kind, chunk_units<T>(kind));
}
template <typename T>
__device__ __forceinline__ int chunk_bytes(int kind, int c, int units) {
  const int cu = chunk_units<T>(kind);
  return units_bytes<T>(kind, min(cu, units - c * cu)) + (c == 0 ? coef_bytes<T>() : 0);
}
// Slice word: width (FP64: entries, FP32: units), kind, resident, more than
// one chunk, local slice.
__device__ __forceinline__ int sl_width(int y) { return y & 0x7ff; }
__device__ __forceinline__ int sl_kind(int y) { return (y >> 11) & 3; }
template <typename T>
__device__ __forceinline__ int sl_units(int y) { return sizeof(T) == 8 ? (sl_width(y) + 1) >> 1 : sl_width(y); }
constexpr int kSlResident = 1 << 13, kSlChunks = 1 << 14, kSlLocalShift = 15, kSlMaxWidth = 0x7ff;

// Value at a byte offset of shared memory.
template <typename T>
__device__ __forceinline__ T sm_at(const unsigned char* sm, uint32_t bytes) {
  return *reinterpret_cast<const T*>(sm + bytes);
}

// Adds the entries of a chunk (blk: its first value) to a row's sum; au is
// the byte offset of the state in shared memory, w the entries (FP64) or
// units (FP32) of the chunk.
__device__ __forceinline__ double row_sum(double acc, const unsigned char* blk, int lane, int, int w,
                                          const unsigned char* sm, uint32_t au, const float*) {
  const int np = w >> 1;
  const double2* v = reinterpret_cast<const double2*>(blk) + lane;
  const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + ((w + 1) >> 1) * 512) + lane;
#pragma unroll 4
  for (int k = 0; k < np; ++k) {
    const double2 x = v[32 * k];
    const uint32_t cc = c[32 * k];
    acc = fma(x.x, sm_at<double>(sm, au + 8 * (cc & 0xffffu)), acc);
    acc = fma(x.y, sm_at<double>(sm, au + 8 * (cc >> 16)), acc);
  }
  if (w & 1) acc = fma(v[32 * np].x, sm_at<double>(sm, au + 8 * (c[32 * np] & 0xffffu)), acc);
  return acc;
}
__device__ __forceinline__ float ref_of(uint32_t s, const float* ref) {
  const float lo = (s & 1u) ? ref[1] : ref[0], hi = (s & 1u) ? 0.f : ref[2];
  return (s & 2u) ? hi : lo;
}
__device__ __forceinline__ float row_sum(float acc, const unsigned char* blk, int lane, int kind, int u,
                                         const unsigned char* sm, uint32_t au, const float* ref) {
  if (kind == 2) {
    const float2* v = reinterpret_cast<const float2*>(blk) + lane;
    const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * 256) + lane;
    const float r0 = ref[0], r1 = ref[1];
#pragma unroll 3
    for (int k = 0; k < u >> 1; ++k, v += 64, c += 32) {
      const uint32_t c0 = au + (*c & 0xffffu), c1 = au + (*c >> 16);
      const float2 x = v[0], y = v[32];
      acc = fmaf(x.x, sm_at<float>(sm, c0) - r0, acc);
      acc = fmaf(x.y, sm_at<float>(sm, c0 + 4) - r1, acc);
      acc = fmaf(y.x, sm_at<float>(sm, c1) - r0, acc);
      acc = fmaf(y.y, sm_at<float>(sm, c1 + 4) - r1, acc);
    }
    if (u & 1) {
      const uint32_t c0 = au + (*c & 0xffffu);
      acc = fmaf(v->x, sm_at<float>(sm, c0) - r0, acc);
      acc = fmaf(v->y, sm_at<float>(sm, c0 + 4) - r1, acc);
    }
  } else if (kind == 1) {
    const float2* v = reinterpret_cast<const float2*>(blk) + lane;
    const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * 256) + lane;
    const float r0 = ref[0];
#pragma unroll 3
    for (int k = 0; k < u; ++k, v += 32, c += 32) {
      const float2 x = *v;
      const uint32_t c0 = au + (*c & 0xffffu), c1 = au + (*c >> 16);
      acc = fmaf(x.x, sm_at<float>(sm, c0) - r0, acc);
      acc = fmaf(x.y, sm_at<float>(sm, c1) - r0, acc);
    }
  } else if (kind == 3) {
    const float* v = reinterpret_cast<const float*>(blk) + lane;
    const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * 384) + lane;
    const float r0 = ref[0], r1 = ref[1], r2 = ref[2];
#pragma unroll 3
    for (int k = 0; k < u >> 1; ++k, v += 192, c += 32) {
      const uint32_t c0 = au + (*c & 0xffffu), c1 = au + (*c >> 16);
      acc = fmaf(v[0], sm_at<float>(sm, c0) - r0, acc);
      acc = fmaf(v[32], sm_at<float>(sm, c0 + 4) - r1, acc);
      acc = fmaf(v[64], sm_at<float>(sm, c0 + 8) - r2, acc);
      acc = fmaf(v[96], sm_at<float>(sm, c1) - r0, acc);
      acc = fmaf(v[128], sm_at<float>(sm, c1 + 4) - r1, acc);
      acc = fmaf(v[160], sm_at<float>(sm, c1 + 8) - r2, acc);
    }
    if (u & 1) {
      const uint32_t c0 = au + (*c & 0xffffu);
      acc = fmaf(v[0], sm_at<float>(sm, c0) - r0, acc);
      acc = fmaf(v[32], sm_at<float>(sm, c0 + 4) - r1, acc);
      acc = fmaf(v[64], sm_at<float>(sm, c0 + 8) - r2, acc);
    }
  } else {
    const float2* v = reinterpret_cast<const float2*>(blk) + lane;
    const uint32_t* c = reinterpret_cast<const uint32_t*>(blk + u * 256) + lane;
#pragma unroll 2
    for (int k = 0; k < u; ++k, v += 32, c += 32) {
      const uint32_t c0 = *c & 0xffffu, c1 = *c >> 16;
      acc = fmaf(v->x, sm_at<float>(sm, au + (c0 & 0xfffcu)) - ref_of(c0 & 3u, ref), acc);
      acc = fmaf(v->y, sm_at<float>(sm, au + (c1 & 0xfffcu)) - ref_of(c1 & 3u, ref), acc);
    }
  }
  return acc;
}

// New value r of a row from its sum, and what its interface correction
// starts from (v).
__device__ __forceinline__ void row_update(double acc, double ui, double up, double rc, bool forced, double f,
                                           int base_prev, double& r, double& v) {
  r = acc + rc * up;
  if (forced) r += f;
  v = base_prev ? (r - up) : (ui - up);
}
__device__ __forceinline__ void row_update(float acc, float ui, float up, float rc, bool forced, float f,
                                           int base_prev, float& r, float& v) {
  float d, err;
  two_sum(ui, -up, d, err);
  float inc = fmaf(rc, d, -acc);
  if (forced) inc += f;
  inc = fmaf(rc, err, inc);
  r = ui + inc;
  v = base_prev ? (d + err + inc) : (d + err);
}

__device__ __forceinline__ double round_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float round_mul(float a, float b) { return __fmul_rn(a, b); }

}  // namespace bfe
