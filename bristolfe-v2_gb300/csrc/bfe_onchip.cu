// One-source march that stays on the chip (sm_103a).
//
// A march of one source (fn_explicit_dynamic_solver_v6.m:180-218 for one load
// step) on a model of up to about 1.5 million DOFs is short work per step: a
// kernel launch per step spends its few microseconds on the launch, on the
// chain column index -> gathered value, and on reading the same operator
// again. Here ONE cooperative launch marches all steps. Every CTA (one per
// SM) owns a contiguous range of 32-row slices and keeps in shared memory
//   * the two newest states of its rows, and the values of the rows of other
//     CTAs that its rows couple to (halo),
//   * as many slices of its operator as fit; the others stream from L2 by
//     bulk copies into a slot or two per warp. The operator does not change,
//     so a slot's next copy is issued as soon as the slot has been read, also
//     across the end of a step.
// Operator entries carry 16-bit indices into the CTA's shared window, so a
// gather is one shared-memory load.
//
// Exchange: after computing a row that others read, its owner writes the
// value to a global buffer together with the step number, as 64-bit words of 4
// bytes of value and 4 of step number; readers poll the value itself. One L2
// round trip replaces data, fence, flag, poll, read. Two buffers by step
// parity suffice: a CTA publishes step t + 2 only after it has read step
// t + 1 of every CTA that reads from it (reading is made symmetric when the
// partition is built), and those publish t + 1 after having read step t.
// Every poll is bounded in time; when one runs out the kernel sets *err and
// all CTAs leave, and the host marches with one launch per step instead.
//
// The arithmetic of a row is that of step_f64_r1 / step_f32_r1 and
// interface_fixup_r1 (bfe_kernels.cu), term for term in the same order, so
// the results are the same bits while the state is finite (entries that a node
// block lacks are zeros here; execute() in bfe_run.cpp has the rest).
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "bfe_onchip.cuh"

namespace bfe {

namespace {

// ---------------------------------------------------------------------------
// The march, one CTA of NT threads or fewer per part.
//
// What bounds it (ncu): FP64 rows the FP64 pipe (coupled 241,579 DOF: 65 % of
// active cycles; plate of 40,602 DOF 37 %, the rest waits for the exchange, about
// a microsecond from a value's store to its use in another CTA); FP32 rows of
// large models instruction issue (coupled 961,641 DOF: 69 % of the issue slots,
// beside 3.7 TB/s of operator chunks from L2); 3D ones that chunk stream (bricks of
// 73,872 DOF: 3.1 TB/s, 40 % of the slots). Measured per step of a 500-step run
// against one launch per step from a graph, GB300 (us): plate of 40,602 DOF FP64
// 2.9 / 6.2, FP32 2.3 / 6.0; coupled 241,579 DOF FP64 8.3 / 13.1, FP32 4.5 / 9.3;
// coupled 961,641 DOF FP32 12.5 / 17.1; bricks of 202,878 DOF FP32 15.7 / 29.8.
//
// Per step: rows (interface and exported slices first, so that
// their values travel while the others are computed), interface correction,
// halo of the new state. A monitor's sample and a frame of state t are
// written during step t + 1, when both states are still on chip.
// V5: prescribed displacements (v5_kernel's rows and arithmetic): one thread
// per listed entry, from the last thread down, forms K(d,:) u_n, writes the
// reaction, and sets the DOF's value instead of its row's thread. Plate of
// 40,602 DOF, 21 prescribed, 1,500 steps in FP64: 4.8 ms against 15.9 with a
// step kernel (4.6 us) and v5_kernel (5.4 us, one thread walking a K row) per
// step.
template <typename T, bool INT, bool V5, int NT>
__global__ void __launch_bounds__(NT, 1) march_onchip(OnchipArgs o, StepArgs a, V5Args q5, int64_t ti0,
                                                      int64_t n_steps, int fresh) {
  using T2 = typename Vec2<T>::type;
  extern __shared__ __align__(16) unsigned char sm[];
  const int p = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  const int s0 = o.part_slice[p], s1 = o.part_slice[p + 1];
  const int ns = s1 - s0, row0 = s0 * kSlice, rpad = ns * kSlice;
  const int rows = min(a.n - row0, rpad);
  const int H = o.halo_cnt[p];
  const int32_t* hrow = o.halo_row + (size_t)p * o.halo_cap;
  const int W = (rpad + H + 2 + 3) & ~3;            // two rows of slack for unused reference values
  // this CTA's forced rows, monitors and interface rows (sorted global lists)
  const int f0 = lower_bound_i32(a.frc_row, a.n_frc, row0);
  const int nf = lower_bound_i32(a.frc_row, a.n_frc, row0 + rows) - f0;
  const int m0 = lower_bound_i32(a.mon_row, a.n_mon, row0);
  const int nm = lower_bound_i32(a.mon_row, a.n_mon, row0 + rows) - m0;
  int t0 = 0, ni = 0, nv = 0, nz = 0, zb = 0;
  const int32_t* vrow = nullptr;
  if (INT) {
    t0 = lower_bound_i32(a.int_row, a.n_int, row0);
    ni = lower_bound_i32(a.int_row, a.n_int, row0 + rows) - t0;
    nv = o.vhalo_ptr[p + 1] - o.vhalo_ptr[p];
    vrow = o.vhalo + o.vhalo_ptr[p];
    zb = __ldg(a.z_ptr + t0);
    nz = __ldg(a.z_ptr + t0 + ni) - zb;
  }
  int e0 = 0, ne = 0, nk = 0, kb = 0;
  if (V5) {
    e0 = o.v5_ptr[p];
    ne = o.v5_ptr[p + 1] - e0;
    kb = __ldg(o.v5_kptr + e0);
    nk = __ldg(o.v5_kptr + e0 + ne) - kb;
  }
  // shared memory
  T* U0 = reinterpret_cast<T*>(sm);
  T* U1 = U0 + W;
  T* vs = U1 + W;                                   // interface differences: own, then halo
  T* zv = vs + (INT ? ((ni + nv + 1) & ~1) : 0);
  T* fs = zv + (INT ? ((nz + 1) & ~1) : 0);         // forcing terms of two steps
  int2* sd = reinterpret_cast<int2*>(fs + ((2 * nf + 1) & ~1));   // slices in order
  double* kv = reinterpret_cast<double*>(sd + ns);                // K rows of prescribed DOFs
  int32_t* fr = reinterpret_cast<int32_t*>(kv + nk);              // forced rows (local)
  int32_t* zp = fr + nf;
  uint16_t* zc = reinterpret_cast<uint16_t*>(zp + (INT ? ni + 1 : 0));
  uint16_t* zr = zc + (INT ? ((nz + 1) & ~1) : 0);
  uint16_t* kc = zr + (INT ? ((ni + 1) & ~1) : 0);
  uint16_t* fl = kc + (V5 ? ((nk + 1) & ~1) : 0);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + ((reinterpret_cast<unsigned char*>(fl + rpad) - sm + 15) & ~15));
  unsigned char* cache = reinterpret_cast<unsigned char*>(bars + ((nw * o.depth + 1) & ~1));

  for (int r = tid; r < rpad; r += nt) fl[r] = r < rows ? __ldg(o.flags + row0 + r) : 0;
  for (int k = tid; k < nf; k += nt) fr[k] = __ldg(a.frc_row + f0 + k) - row0;
  if (INT) {
    for (int k = tid; k <= ni; k += nt) zp[k] = __ldg(a.z_ptr + t0 + k) - zb;
    for (int k = tid; k < ni; k += nt) zr[k] = (uint16_t)(__ldg(a.int_row + t0 + k) - row0);
    for (int k = tid; k < nz; k += nt) {
      zc[k] = __ldg(o.z_lcol + zb + k);
      zv[k] = __ldg(static_cast<const T*>(a.z_val) + zb + k);
    }
  }
  // slices in order: {block offset / 16, slice word}
  for (int j = tid; j < ns; j += nt) {
    const int ls = __ldg(o.order + s0 + j);
    const int y = __ldg(o.slice_word + s0 + ls);
    sd[j] = make_int2(__ldg(o.block_off + s0 + ls),
                      y | (ls << kSlLocalShift) | (sl_units<T>(y) > chunk_units<T>(sl_kind(y)) ? kSlChunks : 0));
  }
  for (int k = tid; k < nw * o.depth; k += nt) bar_init(bars + k);
  __syncthreads();
  for (int k = tid; k < nf; k += nt) fl[fr[k]] |= (uint16_t)kOcForced;
  if (V5) {
    for (int k = tid; k < nk; k += nt) {
      kv[k] = __ldg(o.v5_kval + kb + k);
      kc[k] = __ldg(o.v5_kcol + kb + k);
    }
    __syncthreads();                                    // forced marks are in
    for (int k = tid; k < ne; k += nt) fl[__ldg(o.v5_row + e0 + k)] |= (uint16_t)(1u << kOcIntShift);
  }
  // Resident slices: all of them when they fit, else what the slots leave
  // room for, spread evenly over the order so that a warp computes a resident
  // slice while its slot is filled.
  const bool stream = __ldg(o.op_bytes + p) > o.smem - (int)(cache - sm);
  unsigned char* ring = cache;
  if (stream) cache += nw * o.depth * o.slot_bytes;
  const unsigned char* gblk = static_cast<const unsigned char*>(o.blocks);
  if (tid == 0) {
    const int room = o.smem - (int)(cache - sm);
    const float share = stream ? (float)room / (float)__ldg(o.op_bytes + p) : 1.f;
    float due = 0.f;
    int used = 0;
    for (int m0 = 0; m0 < ns; m0 += nw) {               // one slice of every warp at a time
      due += share;
      if (stream && due < 1.f) continue;
      due -= 1.f;
      for (int j = m0; j < min(m0 + nw, ns); ++j) {
        const int y = sd[j].y, bytes = block_bytes<T>(sl_kind(y), sl_units<T>(y));
        if (used + bytes > room) break;
        used += bytes;
        sd[j].y = y | kSlResident;
      }
    }
  }
  __syncthreads();
  {
    int off = 0;
    for (int j = 0; j < ns; ++j) {
      const int2 d = sd[j];
      if (!(d.y & kSlResident)) continue;
      const int bytes = block_bytes<T>(sl_kind(d.y), sl_units<T>(d.y));
      if (j % nw == warp) {
        const int4* src = reinterpret_cast<const int4*>(gblk + (size_t)d.x * 16);
        for (int k = lane; k < bytes / 16; k += 32) reinterpret_cast<int4*>(cache + off)[k] = __ldg(src + k);
        __syncwarp();
        if (lane == 0) sd[j].x = off;
      }
      off += bytes;
    }
  }
  __syncthreads();
  // this warp's slots: the chunk (ij, ic) to copy next, copies left to issue
  int ij = warp, ic = 0;
  int64_t to_issue = 0;
  int waiting = 0, w_slot = 0, i_slot = 0;              // copies in flight, slot to read, slot to fill
  uint32_t w_parity = 0;
  bool bad = false;                                     // a wait of this thread ran out
  if (stream)
    for (int j = warp; j < ns; j += nw)
      if (!(sd[j].y & kSlResident)) {
        const int kd = sl_kind(sd[j].y), cu = chunk_units<T>(kd);
        to_issue += max(1, (sl_units<T>(sd[j].y) + cu - 1) / cu) * n_steps;
      }
  // Only lane 0 copies, and none after a wait of its own ran out: its counts
  // are those of the copies in flight.
  auto issue = [&]() {
    if (to_issue == 0 || bad) return;
    while (sd[ij].y & kSlResident) {
      ij += nw;
      if (ij >= ns) ij = warp;
    }
    const int2 d = sd[ij];
    const int kd = sl_kind(d.y), un = sl_units<T>(d.y);
    if (lane == 0)
      bulk_load(ring + (warp * o.depth + i_slot) * o.slot_bytes, gblk + (size_t)d.x * 16 + chunk_offset<T>(kd, ic),
                (uint32_t)chunk_bytes<T>(kd, ic, un), bars + warp * o.depth + i_slot);
    if (++i_slot == o.depth) i_slot = 0;
    if (++ic * chunk_units<T>(kd) >= un) {
      ic = 0;
      ij += nw;
      if (ij >= ns) ij = warp;
    }
    --to_issue;
    ++waiting;
  };
  for (int k = 0; k < o.depth && stream; ++k) issue();
  // the slot just read is free again: fill it, go on to the next
  auto next_slot = [&]() {
    if (!bad) {
      --waiting;
      if (++w_slot == o.depth) {
        w_slot = 0;
        w_parity ^= 1;
      }
    }
    __syncwarp();
    issue();
  };
  // states
  for (int r = tid; r < W; r += nt) {
    T un = T(0), up = T(0);
    if (!fresh) {
      const int g = r < rpad ? (r < rows ? row0 + r : -1) : (r < rpad + H ? __ldg(hrow + r - rpad) : -1);
      if (g >= 0) {
        un = static_cast<const T*>(a.u_n)[g];
        if (r < rpad) up = static_cast<const T*>(a.u_prev)[g];
      }
    }
    U0[r] = un;
    U1[r] = up;
  }
  // forcing terms: those of step k are in fs[k & 1], the signal of the step
  // after next is on its way in freg
  T fcoef = T(0), freg = T(0);
  const T* fsig = static_cast<const T*>(a.sig);
  if (tid < nf) {
    fcoef = __ldg(static_cast<const T*>(a.frc_coef) + f0 + tid);
    fsig += (size_t)ti0 * a.n_sig + __ldg(a.frc_sig + f0 + tid);
    fs[tid] = round_mul(fcoef, __ldg(fsig));
    fsig += a.n_sig;
    if (n_steps > 1) freg = __ldg(fsig);
  }
  // one monitor per thread from the last thread down (the rest in a loop)
  const int mt = nt - 1 - tid;
  int mrow = 0;
  double* hist = a.hist;
  if (mt < nm) {
    mrow = __ldg(a.mon_row + m0 + mt) - row0;
    hist += (size_t)__ldg(a.mon_slot + m0 + mt) + (size_t)a.q * (size_t)ti0;
  }
  // this thread's prescribed entry; displacement and acceleration of the next
  // step are on their way in dreg and areg
  int g5 = -1, r5 = 0, s5 = 0, k5 = 0, k5e = 0, f5 = -1;
  bool set5 = false;
  double m5 = 0, c5 = 0, w5 = 0, ud5 = 0, dreg = 0, areg = 0;
  if (V5 && mt < ne) {
    g5 = __ldg(o.v5_ent + e0 + mt);
    r5 = __ldg(o.v5_row + e0 + mt);
    s5 = __ldg(q5.ent_slot + g5);
    set5 = __ldg(q5.ent_last + g5);
    k5 = __ldg(o.v5_kptr + e0 + mt) - kb;
    k5e = __ldg(o.v5_kptr + e0 + mt + 1) - kb;
    m5 = __ldg(q5.slot_m + s5);
    c5 = __ldg(o.v5_c + e0 + mt);
    f5 = __ldg(q5.f_sig + s5);
    w5 = __ldg(q5.f_w + s5);
    ud5 = fresh ? 0.0 : o.v5_ud[s5];
    dreg = __ldg(q5.dsp + (size_t)ti0 * q5.n_ent + g5);
    areg = __ldg(q5.accn + (size_t)ti0 * q5.n_ent + g5);
  }
  // exchange buffers of even and odd steps, this thread's first slots in them
  T* const xu0 = static_cast<T*>(o.xch);
  T* const xu1 = xu0 + o.x_stride;
  T* const xv0 = static_cast<T*>(o.xchv);
  T* const xv1 = xv0 + o.xv_stride;
  constexpr int kPolls = NT <= 512 ? 4 : 2;
  int hx[kPolls], vx[kPolls];
#pragma unroll
  for (int j = 0; j < kPolls; ++j) {
    hx[j] = tid + j * nt < H ? __ldg(hrow + tid + j * nt) : 0;
    vx[j] = INT && tid + j * nt < nv ? __ldg(vrow + tid + j * nt) : 0;
  }
  // step (from ti0) after which the next frame is due
  int64_t frame = -1;
  double* fcol = a.fld;
  if (a.fld) {
    const int64_t c = (ti0 + a.fld_every - 1) / a.fld_every;
    frame = c * a.fld_every - ti0;
    fcol += (size_t)a.n * (size_t)c;
  }
  __syncthreads();

  uint32_t au = 0, bu = (uint32_t)(W * sizeof(T));      // byte offsets of u_n and of u_{n-1} / u_{n+1}
  for (int64_t k = 0; k <= n_steps; ++k) {
    const T* A = reinterpret_cast<const T*>(sm + au);
    T* B = reinterpret_cast<T*>(sm + bu);
    const uint32_t tag = o.tag0 + (uint32_t)(ti0 + k);
    const bool odd = (ti0 + k) & 1;
    // state ti0 + k - 1 (A): samples and, on frame steps, the frame
    if (k > 0) {
      if (mt < nm) {
        *hist = (double)A[mrow];
        hist += a.q;
      }
      for (int j = mt + nt; j < nm; j += nt)
        a.hist[(size_t)__ldg(a.mon_slot + m0 + j) + (size_t)a.q * (size_t)(ti0 + k - 1)] =
            (double)A[__ldg(a.mon_row + m0 + j) - row0];
      if (k - 1 == frame) {
        for (int j = warp; j < ns; j += nw) {            // each thread the rows it will overwrite
          const int r = (sd[j].y >> kSlLocalShift) * kSlice + lane;
          if (r < rows && !(V5 && is_slot(fl[r])))
            fcol[row0 + r] = a.fld_is_vel ? ((double)A[r] - (double)B[r]) / a.dt : (double)A[r];
        }
        if (V5 && g5 >= 0 && set5) fcol[row0 + r5] = ud5;
        frame += a.fld_every;
        fcol += a.n;
      }
    }
    if (k == n_steps) break;
    if (tid < nf) {
      fs[((k + 1) & 1) * nf + tid] = round_mul(fcoef, freg);
      fsig += a.n_sig;
      if (k + 2 < n_steps) freg = __ldg(fsig);
    }
    T* xu = odd ? xu1 : xu0;
    T* xv = odd ? xv1 : xv0;
    if (V5 && g5 >= 0) {
      const int64_t ti = ti0 + k;
      double ku = 0.0;
      for (int e = k5; e < k5e; ++e) ku = fma(kv[e], (double)A[kc[e]], ku);
      q5.frc_out[(size_t)g5 + (size_t)q5.n_ent * ti] = m5 * areg + ku;
      if (set5) {
        const double cv = c5 != 0.0 ? round_mul(c5, ud5) : 0.0;
        double f = 0.0;
        if (f5 >= 0) f = w5 * (double)static_cast<const T*>(a.sig)[(size_t)ti * a.n_sig + f5];
        ud5 = ud5 + q5.dt * ((f - ku - cv) / m5);
        const T u = (T)dreg;
        B[r5] = u;
        if (fl[r5] & kOcExport) xput(xu, (size_t)(row0 + r5), u, tag);
        for (int h = __ldg(q5.h_ptr + s5); h < __ldg(q5.h_ptr + s5 + 1); ++h)
          a.hist[(size_t)__ldg(q5.h_slot + h) + (size_t)a.q * (size_t)ti] = (double)u;
      }
      if (k + 1 < n_steps) {
        dreg = __ldg(q5.dsp + (size_t)(ti + 1) * q5.n_ent + g5);
        areg = __ldg(q5.accn + (size_t)(ti + 1) * q5.n_ent + g5);
      }
    }
    // rows
    for (int j = warp; j < ns; j += nw) {
      const int2 d = sd[j];
      const int kind = sizeof(T) == 8 ? 0 : sl_kind(d.y), r = (d.y >> kSlLocalShift) * kSlice + lane;
      const bool resident = d.y & kSlResident;
      const T ui = A[r], up = B[r];
      const uint32_t f = fl[r];
      float ref[3];
      if (sizeof(T) == 4) {
        const int pos = (int)(f >> kOcPosShift) & 7;
        ref[0] = (float)ui;
        if (kind != 1) {
          int q0 = r - pos, q1 = q0 + 1, q2 = q0 + 2;
          if (kind == 0 && pos == (int)kOcCut) {
            const ushort4 x = o.lref[row0 + r];
            q0 = x.x, q1 = x.y, q2 = x.z;
          }
          __syncwarp();
          ref[0] = (float)A[q0];
          ref[1] = (float)A[q1];
          ref[2] = (float)A[q2];
        }
      }
      const unsigned char* blk = cache + d.x;
      if (!resident) {
        blk = ring + (warp * o.depth + w_slot) * o.slot_bytes;
        bad = bad || !bar_wait(bars + warp * o.depth + w_slot, w_parity, o.err);
      }
      const T rc = reinterpret_cast<const T*>(blk)[lane];
      blk += coef_bytes<T>();
      T acc = T(0);
      // the indices of a chunk that did not come are not followed
      if (!(d.y & kSlChunks)) {
        acc = row_sum(acc, blk, lane, kind, bad ? 0 : sl_width(d.y), sm, au, ref);
      } else {
        // FP64 counts entries (an odd last one is not paired), FP32 units
        const int cu = chunk_units<T>(kind), full = sizeof(T) == 8 ? 2 * cu : cu, step = units_bytes<T>(kind, cu);
        for (int left = sl_width(d.y);;) {
          acc = row_sum(acc, blk, lane, kind, bad ? 0 : min(left, full), sm, au, ref);
          left -= full;
          if (left <= 0) break;
          blk += step;
          if (!resident) {
            next_slot();
            blk = ring + (warp * o.depth + w_slot) * o.slot_bytes;
            bad = bad || !bar_wait(bars + warp * o.depth + w_slot, w_parity, o.err);
          }
        }
      }
      if (!resident) next_slot();
      T ft = T(0);
      if (f & kOcForced) ft = fs[(k & 1) * nf + lower_bound_sm(fr, nf, r)];
      T rn, v;
      row_update(acc, ui, up, rc, (f & kOcForced) != 0, ft, a.int_base_prev, rn, v);
      if (INT && (f & kOcInterface)) {
        const int li = (int)(f >> kOcIntShift);
        vs[li] = v;
        if (f & kOcExportV) xput(xv, (size_t)(t0 + li), v, tag);
        if (!a.int_base_prev) B[r] = rn;
      } else if (!(V5 && is_slot(f))) {
        B[r] = rn;
        if (f & kOcExport) xput(xu, (size_t)(row0 + r), rn, tag);
      }
    }
    if (INT && ni) {
      bad |= !receive(xv, vrow, nv, vx, tag, vs + ni, tid, nt, o.err);
      __syncthreads();
      for (int t = warp; t < ni; t += nw) {
        T acc = T(0);
        for (int e = zp[t] + lane; e < zp[t + 1]; e += 32) acc += zv[e] * vs[zc[e]];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) {
          const int r = zr[t];
          const T rn = B[r] + acc;
          B[r] = rn;
          if (fl[r] & kOcExport) xput(xu, (size_t)(row0 + r), rn, tag);
        }
      }
    }
    if (k + 1 < n_steps) bad |= !receive(xu, hrow, H, hx, tag, B + rpad, tid, nt, o.err);
    if (__syncthreads_or(bad)) {
      for (; lane == 0 && waiting > 0; --waiting) {     // no copy may outlive the CTA
        if (!bar_wait(bars + warp * o.depth + w_slot, w_parity, o.err)) break;
        if (++w_slot == o.depth) {
          w_slot = 0;
          w_parity ^= 1;
        }
      }
      return;
    }
    const uint32_t x = au;
    au = bu;
    bu = x;
  }
  if (V5 && g5 >= 0 && set5) o.v5_ud[s5] = ud5;
  // the two newest states back to global memory: u_n may still be read by a
  // CTA that is loading, u_prev only by this one
  for (int r = tid; r < rows; r += nt) {
    static_cast<T*>(a.u_new)[row0 + r] = sm_at<T>(sm, au + r * (uint32_t)sizeof(T));
    const_cast<T*>(static_cast<const T*>(a.u_prev))[row0 + r] = sm_at<T>(sm, bu + r * (uint32_t)sizeof(T));
  }
}

// ---------------------------------------------------------------------------
// Building the partition's device data from the sliced-ELL operator.

constexpr int kRankWords = 8;     // bitmap words per stored prefix count

// One CTA per part: the columns its rows read outside the part become its
// halo (ascending rows), and every slice gets its kind and its block.
template <typename T>
__global__ void __launch_bounds__(1024) oc_columns(OnchipBuild b) {
  extern __shared__ __align__(16) unsigned char smb[];
  uint32_t* bits = reinterpret_cast<uint32_t*>(smb);
  __shared__ int cmin, cmax, total, bytes;
  __shared__ int scan[1024];
  constexpr bool F32 = sizeof(T) == 4;
  const int p = blockIdx.x, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  const int s0 = b.part_slice[p], s1 = b.part_slice[p + 1];
  const int row0 = s0 * kSlice, row1 = min(b.n, s1 * kSlice), rpad = (s1 - s0) * kSlice;
  const int e0 = b.slice_ptr[s0], e1 = b.slice_ptr[s1];
  if (tid == 0) { cmin = 0x7fffffff; cmax = -1; bytes = 0; }
  __syncthreads();
  int lo = 0x7fffffff, hi = -1;
  for (int e = e0 + tid; e < e1; e += nt) {
    const int c = (int)(__ldg(b.col + e) & kColMask);
    lo = min(lo, F32 ? max(c - 2, 0) : c);
    hi = max(hi, F32 ? min(c + 2, b.n - 1) : c);
  }
  for (int i = row0 + tid; i < row1; i += nt) {
    const int base = F32 ? (int)__ldg(b.base + i) : i;
    lo = min(lo, base);
    hi = max(hi, min(base + 2, b.n - 1));
  }
  atomicMin(&cmin, lo);
  atomicMax(&cmax, hi);
  __syncthreads();
  const int c0 = cmin & ~31, nwords = (cmax - c0) / 32 + 1;
  if (nwords > b.max_words) {
    if (tid == 0) atomicExch(b.fail, 1);
    return;
  }
  int* pre = reinterpret_cast<int*>(bits + ((b.max_words + kRankWords - 1) / kRankWords) * kRankWords);
  const int ngrp = (nwords + kRankWords - 1) / kRankWords;
  for (int k = tid; k < ngrp * kRankWords; k += nt) bits[k] = 0;
  __syncthreads();
  auto mark = [&](int c) {
    if (c < row0 || c >= row1) atomicOr(bits + ((c - c0) >> 5), 1u << ((c - c0) & 31));
  };
  // padding of the sliced ELL: a direct zero on the row itself
  auto is_pad = [&](uint32_t e, T v, int i) { return (e & kDirect) && v == T(0) && (int)(e & kColMask) == min(i, b.n - 1); };
  // the first row of the node that entry e (of DOF slot s) belongs to, if the
  // node has rows for all of kind's DOFs; else -1
  auto node_of = [&](uint32_t e, int kind) -> int {
    const int c = (int)(e & kColMask), nb = c - (int)((e >> kSlotShift) & kSlotMask);
    if (nb < 0 || nb + kind > b.n || (int)__ldg(b.base + c) != nb || (int)__ldg(b.base + nb) != nb ||
        (int)__ldg(b.base + nb + kind - 1) != nb)
      return -1;
    return nb;
  };
  for (int s = s0 + (tid >> 5); s < s1; s += nt >> 5) {
    const int off = b.slice_ptr[s], w = (b.slice_ptr[s + 1] - off) >> 5, i = s * kSlice + lane;
    if (w > kSlMaxWidth) atomicExch(b.fail, 1);
    if (!F32) {
      for (int k = 0; k < w; ++k) mark((int)(__ldg(b.col + off + 32 * k + lane) & kColMask));
      if (lane == 0) b.slice_word[s] = w;
      continue;
    }
    // kind: which of the forms every row of the slice has
    const int base = i < b.n ? (int)__ldg(b.base + i) : 0, pos = i - base;
    bool k1 = true, k2 = pos < 2 || i >= b.n, k3 = pos < 3 || i >= b.n;
    for (int k = 0; k < w; ++k) {
      const uint32_t e = __ldg(b.col + off + 32 * k + lane);
      if (is_pad(e, __ldg(static_cast<const T*>(b.val) + off + 32 * k + lane), i)) continue;
      const int slot = (int)((e >> kSlotShift) & kSlotMask);
      if (e & kDirect) { k1 = k2 = k3 = false; continue; }
      k1 = k1 && slot == pos;
      k2 = k2 && slot < 2 && node_of(e, 2) >= 0;
      k3 = k3 && slot < 3 && node_of(e, 3) >= 0;
      if (slot > 2) atomicExch(b.fail, 1);
    }
    k2 = k2 && (i >= b.n || (base + 2 <= b.n && (int)__ldg(b.base + base + 1) == base));
    k3 = k3 && (i >= b.n || (base + 3 <= b.n && (int)__ldg(b.base + base + 2) == base));
    const int kind = __all_sync(0xffffffffu, k1) ? 1 : __all_sync(0xffffffffu, k2) ? 2 : __all_sync(0xffffffffu, k3) ? 3 : 0;
    for (int k = 0; k < w; ++k) {
      const uint32_t e = __ldg(b.col + off + 32 * k + lane);
      mark((int)(e & kColMask));
      if ((e & kDirect)) continue;
      mark(base + (int)((e >> kSlotShift) & kSlotMask));
      if (kind >= 2)
        for (int q = 0, nb = node_of(e, kind); q < kind; ++q) mark(nb + q);
    }
    if (kind >= 2 && i < b.n)
      for (int q = 0; q < kind; ++q) mark(base + q);
    if (lane == 0) b.slice_word[s] = w | (kind << 11);
  }
  __syncthreads();
  // prefix counts over groups of words
  int mine = 0;
  const int per = (ngrp + nt - 1) / nt;
  for (int g = tid * per; g < min((tid + 1) * per, ngrp); ++g)
    for (int k = 0; k < kRankWords; ++k) mine += __popc(bits[g * kRankWords + k]);
  scan[tid] = mine;
  __syncthreads();
  for (int d = 1; d < nt; d <<= 1) {
    const int x = tid >= d ? scan[tid - d] : 0;
    __syncthreads();
    scan[tid] += x;
    __syncthreads();
  }
  int run = scan[tid] - mine;
  for (int g = tid * per; g < min((tid + 1) * per, ngrp); ++g) {
    pre[g] = run;
    for (int k = 0; k < kRankWords; ++k) run += __popc(bits[g * kRankWords + k]);
  }
  if (tid == nt - 1) total = scan[tid];
  __syncthreads();
  const int H = total;
  // one slot of the list is kept free per other part for symmetric reading
  if (H + b.n_parts > b.halo_cap || rpad + H > b.max_window) {
    if (tid == 0) atomicExch(b.fail, 1);
    return;
  }
  auto local = [&](int c) -> int {
    if (c >= row0 && c < row1) return c - row0;
    const int w = (c - c0) >> 5, g = w / kRankWords;
    int r = pre[g];
    for (int k = g * kRankWords; k < w; ++k) r += __popc(bits[k]);
    return rpad + r + __popc(bits[w] & ((1u << ((c - c0) & 31)) - 1u));
  };
  // halo rows, their owners and export marks
  for (int w = tid; w < nwords; w += nt) {
    uint32_t m = bits[w];
    while (m) {
      const int c = c0 + 32 * w + __ffs((int)m) - 1;
      m &= m - 1;
      b.halo_row[(size_t)p * b.halo_cap + local(c) - rpad] = c;
      b.exported[c] = 1;
      int a0 = 0, a1 = b.n_parts - 1;                  // the part that owns row c
      while (a0 < a1) {
        const int mid = (a0 + a1 + 1) >> 1;
        if (b.part_slice[mid] * kSlice <= c) a0 = mid; else a1 = mid - 1;
      }
      b.adj[(size_t)p * b.n_parts + a0] = 1;
    }
  }
  if (tid == 0) b.halo_cnt[p] = H;
  for (int s = s0 + (tid >> 5); s < s1; s += nt >> 5) {
    const int off = b.slice_ptr[s], w = (b.slice_ptr[s + 1] - off) >> 5, i = s * kSlice + lane;
    const T* val = static_cast<const T*>(b.val) + off + lane;
    const uint32_t* col = b.col + off + lane;
    unsigned char* blk = static_cast<unsigned char*>(b.blocks) + (size_t)b.block_off[s] * 16;
    reinterpret_cast<T*>(blk)[lane] = __ldg(static_cast<const T*>(b.rowc) + min(i, b.n - 1));
    blk += coef_bytes<T>();
    int kind = 0, pos = 0, units = 0;
    if (F32) {
      kind = b.slice_word[s] >> 11;
      const int base = i < b.n ? (int)__ldg(b.base + i) : i;
      pos = i - base;
      // a node block cut by the part's edge keeps the row's indices in lref;
      // units must lie together in the window
      unsigned used = kind >= 2 && i < b.n ? (1u << kind) - 1u : 0u;
      bool together = true;
      int prev = -1;
      for (int k = 0; k < w; ++k) {
        const uint32_t e = __ldg(col + 32 * k);
        if (e & kDirect) continue;
        used |= 1u << ((e >> kSlotShift) & kSlotMask);
        if (kind >= 2) {
          const int nb = node_of(e, kind);
          together = together && local(nb + kind - 1) == local(nb) + kind - 1;
          if (nb != prev) ++units;
          prev = nb;
        }
      }
      const int top = used ? 31 - __clz((int)used) : 0;
      const bool cut = used && (base < row0 || base + top >= row1 || pos >= (int)kOcCut);
      if (i < b.n) {
        uint16_t x[3];
        for (int q = 0; q < 3; ++q) x[q] = (uint16_t)((used >> q) & 1u ? local(base + q) : i - row0);
        b.lref[i] = make_ushort4(x[0], x[1], x[2], 0);
        b.pos[i] = (uint8_t)(cut ? kOcCut : used ? pos : 0);
      }
      if (kind && !__all_sync(0xffffffffu, !cut && together)) kind = 0;
      for (int d = 16; d > 0; d >>= 1) units = max(units, __shfl_xor_sync(0xffffffffu, units, d));
      if (kind >= 2 && block_bytes<T>(kind, units) > block_bound<T>(w)) kind = 0;
    }
    const int width = kind < 2 ? w : units, un = slice_units(kind, width), cu = chunk_units<T>(kind);
    if (lane == 0) {
      b.slice_word[s] = (F32 ? un : width) | (kind << 11);
      atomicAdd(&bytes, block_bytes<T>(kind, un));
      atomicMax(b.slot_bytes, chunk_bytes<T>(kind, 0, un));
    }
    const int own = (F32 ? 4 : 1) * (min(i, row1 - 1) - row0);       // window index of the row itself
    if (kind < 2) {
      for (int k = 0; k < 2 * un; ++k) {
        uint32_t lc = (uint32_t)own | (F32 && kind == 0 ? 3u : 0u);
        T v = T(0);
        if (k < w) {
          const uint32_t e = __ldg(col + 32 * k);
          v = __ldg(val + 32 * k);
          if (kind == 0) {
            lc = (uint32_t)local((int)(e & kColMask));
            if (F32) lc = lc << 2 | ((e & kDirect) ? 3u : ((e >> kSlotShift) & kSlotMask));
          } else if (!(e & kDirect)) {
            lc = (uint32_t)local((int)(e & kColMask)) << 2;
          }
        }
        const int c = (k >> 1) / cu, q = (k >> 1) - c * cu, npc = min(cu, un - c * cu);
        T* cv = reinterpret_cast<T*>(blk + c * units_bytes<T>(kind, cu));
        cv[64 * q + 2 * lane + (k & 1)] = v;
        reinterpret_cast<uint16_t*>(cv + npc * 64)[64 * q + 2 * lane + (k & 1)] = (uint16_t)lc;
      }
    } else if (F32) {
      int k = 0;
      for (int q = 0; q < un; ++q) {                   // next node of the row, zeros past its last
        float v[3] = {0.f, 0.f, 0.f};
        while (k < w && (__ldg(col + 32 * k) & kDirect)) ++k;
        int nb = -1;
        while (k < w) {
          const uint32_t e = __ldg(col + 32 * k);
          if (e & kDirect) { ++k; continue; }
          const int x = node_of(e, kind);
          if (nb < 0) nb = x;
          if (x != nb) break;
          v[(e >> kSlotShift) & kSlotMask] = (float)__ldg(val + 32 * k);
          ++k;
        }
        // past the last node: the row's own node, so that nothing else enters
        const uint32_t lc = nb >= 0 ? 4u * (uint32_t)local(nb) : i < b.n ? 4u * (uint32_t)(i - pos - row0) : 0u;
        const int c = q / cu, x = q - c * cu, nc = min(cu, un - c * cu);
        float* cv = reinterpret_cast<float*>(blk + c * units_bytes<T>(kind, cu));
        if (kind == 2) reinterpret_cast<float2*>(cv)[32 * x + lane] = make_float2(v[0], v[1]);
        else
          for (int l = 0; l < 3; ++l) cv[96 * x + 32 * l + lane] = v[l];
        uint16_t* ci = reinterpret_cast<uint16_t*>(cv + nc * kind * 32);
        ci[64 * (x >> 1) + 2 * lane + (x & 1)] = (uint16_t)lc;
        if ((nc & 1) && x == nc - 1) ci[64 * (x >> 1) + 2 * lane + 1] = (uint16_t)lc;
      }
    }
  }
  __syncthreads();
  if (tid == 0) b.op_bytes[p] = bytes;
}

// Reading made symmetric: when p reads from q and q not from p, q gets the
// first row of p as one more halo row.
__global__ void oc_symmetric(OnchipBuild b) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= b.n_parts * b.n_parts || *b.fail) return;
  const int p = g / b.n_parts, q = g % b.n_parts;
  if (!b.adj[(size_t)p * b.n_parts + q] || b.adj[(size_t)q * b.n_parts + p]) return;
  const int k = atomicAdd(b.halo_cnt + q, 1);
  if (k >= b.halo_cap) { atomicExch(b.fail, 1); return; }
  const int c = b.part_slice[p] * kSlice;
  b.halo_row[(size_t)q * b.halo_cap + k] = c;
  b.exported[c] = 1;
}

// Row flags, and each part's slices in the order of their work: slices with
// interface rows, then slices that others read from, then the rest, the wide
// ones of each class first. Warps take them in turn, so this also evens out
// the warps' work (in the order of the rows a warp's turns fall on the same
// place of every mesh column: all solid or all fluid; C1 in FP32 then took
// 14.0 us per step).
__global__ void __launch_bounds__(256) oc_order(OnchipBuild b) {
  extern __shared__ int pri[];
  if (*b.fail) return;
  const int p = blockIdx.x, s0 = b.part_slice[p], ns = b.part_slice[p + 1] - s0;
  const int row0 = s0 * kSlice;
  const int t0 = lower_bound_i32(b.int_row, b.n_int, row0);
  for (int j = threadIdx.x; j < ns; j += blockDim.x) pri[j] = 2;
  __syncthreads();
  for (int r = threadIdx.x; r < ns * kSlice && row0 + r < b.n; r += blockDim.x) {
    const int i = row0 + r;
    uint32_t f = (b.exported[i] ? kOcExport : 0u) | (b.pos ? (uint32_t)b.pos[i] << kOcPosShift : 0u);
    if (b.n_int) {
      const int t = lower_bound_i32(b.int_row, b.n_int, i);
      if (t < b.n_int && b.int_row[t] == i) {
        if (t - t0 > (int)kOcMaxInt) atomicExch(b.fail, 1);
        f |= kOcInterface | (b.v_exported[t] ? kOcExportV : 0u) | ((uint32_t)(t - t0) << kOcIntShift);
      }
    }
    b.flags[i] = (uint16_t)f;
    if (f & kOcInterface) atomicMin(pri + r / kSlice, 0);
    else if (f & kOcExport) atomicMin(pri + r / kSlice, 1);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < ns; j += blockDim.x) pri[j] = pri[j] * 4096 + 4095 - (b.slice_ptr[s0 + j + 1] - b.slice_ptr[s0 + j]) / kSlice;
  __syncthreads();
  for (int j = threadIdx.x; j < ns; j += blockDim.x) {
    int rank = 0;
    for (int i = 0; i < ns; ++i) rank += pri[i] < pri[j] || (pri[i] == pri[j] && i < j);
    b.order[s0 + rank] = (uint16_t)j;
  }
}

// One warp per slice of the new order, lane = row.
template <typename T>
__global__ void __launch_bounds__(256) oc_reorder(OnchipReorder r) {
  const int s = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (s >= r.n_slices) return;
  const int i = s * kSlice + lane, off = __ldg(r.slice_ptr + s), w = (__ldg(r.slice_ptr + s + 1) - off) >> 5;
  int from = 0, wf = 0;
  if (i < r.n) {
    const int o = __ldg(r.row_of + i), so = o >> 5;
    from = __ldg(r.old_ptr + so) + (o & 31);
    wf = (__ldg(r.old_ptr + so + 1) - __ldg(r.old_ptr + so)) >> 5;
    static_cast<T*>(r.rowc)[i] = __ldg(static_cast<const T*>(r.old_rowc) + o);
  }
  for (int k = 0; k < w; ++k) {
    uint32_t e = (uint32_t)min(i, r.n - 1) | (sizeof(T) == 8 ? 0u : kDirect);
    T v = T(0);
    if (k < wf) {
      e = __ldg(r.old_col + from + 32 * k);
      e = (e & ~kColMask) | (uint32_t)__ldg(r.place + (e & kColMask));
      v = __ldg(static_cast<const T*>(r.old_val) + from + 32 * k);
    }
    r.col[off + 32 * k + lane] = e;
    static_cast<T*>(r.val)[off + 32 * k + lane] = v;
  }
}

template <typename T>
cudaError_t build_t(const OnchipBuild& b, cudaStream_t st) {
  auto smem_of = [](int max_words) {
    const int words = (max_words + kRankWords - 1) / kRankWords * kRankWords;
    return words * 4 + words / kRankWords * 4;
  };
  const int smem = smem_of(b.max_words);
  cudaError_t e =
      cudaFuncSetAttribute(oc_columns<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_of(kOnchipMaxWords));
  if (e != cudaSuccess) return e;
  oc_columns<T><<<b.n_parts, 1024, smem, st>>>(b);
  const int pairs = b.n_parts * b.n_parts;
  oc_symmetric<<<(pairs + 255) / 256, 256, 0, st>>>(b);
  oc_order<<<b.n_parts, 256, (size_t)b.max_part_slices * sizeof(int), st>>>(b);
  return cudaGetLastError();
}

template <typename T, bool INT, bool V5, int NT>
cudaError_t launch_t(const OnchipArgs& o, const StepArgs& a, const V5Args& v, int64_t ti0, int64_t n_steps, int fresh,
                     cudaStream_t st) {
  auto* kern = march_onchip<T, INT, V5, NT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kOnchipSmem);
  if (e != cudaSuccess) return e;
  OnchipArgs oo = o;
  StepArgs aa = a;
  V5Args vv = v;
  void* args[] = {&oo, &aa, &vv, &ti0, &n_steps, &fresh};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kern), dim3(o.n_parts), dim3(o.threads), args,
                                     (size_t)o.smem, st);
}

}  // namespace

int onchip_block_bound(int precision, int width) {
  return precision == 0 ? block_bound<double>(width) : block_bound<float>(width);
}

int onchip_block_least(int width, int dofs) {
  int least = block_bytes<float>(1, slice_units(1, width));
  for (int kind = 2; kind <= dofs; ++kind) {
    const int b = block_bytes<float>(kind, (width + kind - 1) / kind);
    if (b < least) least = b;
  }
  return least;
}

cudaError_t launch_onchip_reorder(const OnchipReorder& r, int precision, cudaStream_t st) {
  const int blocks = (r.n_slices * 32 + 255) / 256;
  if (precision == 0) oc_reorder<double><<<blocks, 256, 0, st>>>(r);
  else oc_reorder<float><<<blocks, 256, 0, st>>>(r);
  return cudaGetLastError();
}

cudaError_t launch_onchip_build(const OnchipBuild& b, int precision, cudaStream_t st) {
  return precision == 0 ? build_t<double>(b, st) : build_t<float>(b, st);
}

cudaError_t launch_onchip(const OnchipArgs& o, const StepArgs& a, const V5Args& v, int precision, int64_t ti0,
                          int64_t n_steps, int fresh, cudaStream_t st) {
  // parts of at most 16 warps take the form with 128 registers per thread:
  // more of a row's loads in flight
  auto go = [&](auto zero, auto interface, auto v5) {
    using T = decltype(zero);
    constexpr bool kInt = decltype(interface)::value, kV5 = decltype(v5)::value;
    return o.threads <= 512 ? launch_t<T, kInt, kV5, 512>(o, a, v, ti0, n_steps, fresh, st)
                            : launch_t<T, kInt, kV5, 1024>(o, a, v, ti0, n_steps, fresh, st);
  };
  auto pick = [&](auto zero) {
    if (o.v5_ptr) return a.n_int ? go(zero, std::true_type(), std::true_type()) : go(zero, std::false_type(), std::true_type());
    return a.n_int ? go(zero, std::true_type(), std::false_type()) : go(zero, std::false_type(), std::false_type());
  };
  return precision == 0 ? pick(0.0) : pick(0.f);
}

}  // namespace bfe
