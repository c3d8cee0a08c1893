// RoPE (full or partial, NeoX pairing), the f16 KV-cache append and the standalone sigmoid gate.
//
// One small CTA per (column, head); for prefill chunks 64 threads per column (f16) or one CTA per column.
//   PA_ROPE_F64    angle = pos * inv_freq[i] in float64 (inv_freq = theta^(-2i/n_rot) comes from the host's
//                  libm), cos / sin in float64, the two products and their difference / sum rounded one by
//                  one in float64, the result rounded to f32 — the arithmetic of pooled's CPU reference
//                  (tests/reference/ref_q38.mjs:67-79).  cos / sin come from a table that pa_angles_kernel fills
//                  once per (position, width) and every layer of the step reuses; the rotation itself is
//                  rot_exact(): the same bits as the float64 expression at f32 cost.
//   PA_ROPE_TABLE  cos / sin read from the caller's f32 table, products and sums rounded one by one in f32
//                  (the Flash engine's host table, engine/qwen4exp.js:549-553).
// K is rotated, rounded to f32 and then to f16 (round to nearest even) into row pos + col of the K cache;
// V is converted only.  Stands in for rope_part(_mc), kv_store and attn_glue_kv of pooled
// (engine/wgsl/qwen35.js:386-404, :858-906; engine/wgsl/layer_fuse.js:87-146).
#include "pa_params.cuh"

namespace pa {

// grid (n_cols, q heads + k heads + v heads); one thread per pair of elements of the head.  Thread t < n_rot/2
// evaluates its own cos / sin and rotates dims (t, t + n_rot/2); the other threads pass dims n_rot + 2(t - n_rot/2),
// +1 through.  No shared memory and no barrier: every global load of the call is in flight at once, which is what
// the latency of a one-token call consists of.
__global__ void __launch_bounds__(128) pa_rope_append_kernel(const RopeParams p) {
  const uint32_t col = blockIdx.x, half = p.n_rot / 2, hd = p.hd, pr = threadIdx.x;
  // The kernel after this one may start fetching old cache rows while this one runs (it never touches the rows or
  // the rotated q written here before its own wait); this kernel itself writes nothing before its predecessor ends.
  // by-value angles go through shared memory: launch parameters indexed differently by every thread are served one
  // address at a time.  Done ahead of the wait, while the predecessor still runs.
  __shared__ Angle s_ang[64];
  if (p.trigger_early) pdl_trigger();
  if (p.n_ang) {
    if (threadIdx.x < p.n_ang * 2) reinterpret_cast<uint4*>(s_ang)[threadIdx.x] = reinterpret_cast<const uint4*>(p.ang)[threadIdx.x];
    __syncthreads();
  }
  // an angle this thread evaluates itself needs nothing of the predecessor's: ahead of the wait
  const uint32_t pos_c = p.n_items ? p.item_pos[col] : p.pos + col;
  Angle g_own;
  const bool own_angle = p.mode == PA_ROPE_F64 && !p.n_ang && !p.angles && pr < half && (p.q || p.k);
  if (own_angle) {
    double s, c;
    sincos(__dmul_rn((double)pos_c, p.inv_freq[pr]), &s, &c);
    g_own = make_angle(c, s);
  }
  pdl_wait();
  if (!p.trigger_early) pdl_trigger();
  if (pr >= hd / 2) return;
  const uint32_t nq = p.q ? p.q_heads : 0, nk = p.k ? p.kv_heads : 0;
  uint32_t slot = blockIdx.y;
  const uint64_t row_c = p.n_items ? p.item_row[col] : p.cache_row0 + col;
  if (slot >= nq && row_c == ~0ull) return;   // an item whose row another shard holds: nothing to append
  if (slot >= nq + nk) {
    // V head: conversion only
    const uint32_t head = slot - nq - nk, kvd = p.kv_heads * hd;
    const uint64_t so = (uint64_t)col * p.v_col_stride + (uint64_t)head * hd + 2 * pr;
    __half* dst = p.v_cache + row_c * (uint64_t)kvd + (uint64_t)head * hd + 2 * pr;
    dst[0] = f16_rne(ld_act(p.v, so, p.in_f16));
    dst[1] = f16_rne(ld_act(p.v, so + 1, p.in_f16));
    return;
  }
  const bool is_q = slot < nq;
  const uint32_t head = is_q ? slot : slot - nq;
  uint32_t d0, d1;
  const bool rot = p.mode != PA_ROPE_NONE && pr < half;
  if (pr < half) { d0 = pr; d1 = pr + half; } else { d0 = p.n_rot + 2 * (pr - half); d1 = d0 + 1; }
  const void* src = is_q ? p.q : p.k;
  const uint64_t sb = is_q ? (uint64_t)col * p.q_col_stride + (uint64_t)head * p.q_head_stride
                           : (uint64_t)col * p.kv_col_stride + (uint64_t)head * hd;
  const float a = ld_act(src, sb + d0, p.in_f16), b = ld_act(src, sb + d1, p.in_f16);
  float ra = a, rb = b;
  if (rot) {
    if (p.mode == PA_ROPE_F64) {
      Angle g;
      if (p.n_ang) g = s_ang[col * half + pr];
      else if (p.angles) g = p.angles[(uint64_t)col * half + pr];
      else g = g_own;
      ra = rot_exact(a, b, g, true);     // a cos - b sin
      rb = rot_exact(b, a, g, false);    // b cos + a sin
    } else {
      const float c = p.cs_table[(uint64_t)col * p.n_rot + 2 * pr], s = p.cs_table[(uint64_t)col * p.n_rot + 2 * pr + 1];
      ra = __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s));
      rb = __fadd_rn(__fmul_rn(a, s), __fmul_rn(b, c));
    }
  }
  if (is_q) {
    const uint64_t o = (uint64_t)col * p.q_out_col_stride + (uint64_t)head * hd;
    if (p.q_out_f16 == 2) {   // high and low f16 parts for the verify kernel's hi / lo rows
      __half* dst = reinterpret_cast<__half*>(p.q_out) + o;
      const __half ha = __float2half_rn(ra), hb = __float2half_rn(rb);
      dst[d0] = ha; dst[d1] = hb;
      dst[p.q_lo_offset + d0] = __float2half_rn(ra - __half2float(ha)); dst[p.q_lo_offset + d1] = __float2half_rn(rb - __half2float(hb));
    } else if (p.q_out_f16) { __half* dst = reinterpret_cast<__half*>(p.q_out) + o; dst[d0] = __float2half_rn(ra); dst[d1] = __float2half_rn(rb); }
    else { float* dst = reinterpret_cast<float*>(p.q_out) + o; dst[d0] = ra; dst[d1] = rb; }
  } else {
    __half* dst = p.k_cache + row_c * (uint64_t)(p.kv_heads * hd) + (uint64_t)head * hd;
    dst[d0] = f16_rne(ra); dst[d1] = f16_rne(rb);
  }
}

// Many columns (prefill chunks): one 256-thread CTA per column.  The column's n_rot/2 angles are evaluated once and
// shared by every head through shared memory; each thread then takes (head, pair) items four at a time so that its
// loads overlap.  Same arithmetic, element for element, as the per-head kernel above.
__global__ void __launch_bounds__(256) pa_rope_append_cols_kernel(const RopeParams p) {
  __shared__ Angle s_g[128];
  const uint32_t col = blockIdx.x, half = p.n_rot / 2, hd = p.hd, pairs = hd / 2;
  if (p.trigger_early) pdl_trigger();
  pdl_wait();
  if (!p.trigger_early) pdl_trigger();
  if (p.mode == PA_ROPE_F64) {
    for (uint32_t i = threadIdx.x; i < half; i += blockDim.x) {
      if (p.n_ang) s_g[i] = p.ang[col * half + i];
      else if (p.angles) s_g[i] = p.angles[(uint64_t)col * half + i];
      else {
        double sv, cv;
        sincos(__dmul_rn((double)(p.pos + col), p.inv_freq[i]), &sv, &cv);
        s_g[i] = make_angle(cv, sv);
      }
    }
  }
  __syncthreads();
  const uint32_t nq = p.q ? p.q_heads * pairs : 0, nk = p.k ? p.kv_heads * pairs : 0, nv = p.v ? p.kv_heads * pairs : 0;
  const uint32_t total = nq + nk + nv, kvd = p.kv_heads * hd;
  for (uint32_t w0 = threadIdx.x; w0 < total; w0 += 4 * blockDim.x) {
    float a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t w = w0 + u * blockDim.x;
      a[u] = b[u] = 0.f;
      if (w >= total) continue;
      if (w >= nq + nk) {                      // V: elements 2i, 2i+1
        const uint64_t so = (uint64_t)col * p.v_col_stride + 2 * (w - nq - nk);
        a[u] = ld_act(p.v, so, p.in_f16); b[u] = ld_act(p.v, so + 1, p.in_f16);
      } else {
        const bool is_q = w < nq;
        const uint32_t ww = is_q ? w : w - nq, head = ww / pairs, pr = ww % pairs;
        const uint32_t d0 = pr < half ? pr : p.n_rot + 2 * (pr - half), d1 = pr < half ? pr + half : d0 + 1;
        const uint64_t sb = is_q ? (uint64_t)col * p.q_col_stride + (uint64_t)head * p.q_head_stride : (uint64_t)col * p.kv_col_stride + (uint64_t)head * hd;
        a[u] = ld_act(is_q ? p.q : p.k, sb + d0, p.in_f16); b[u] = ld_act(is_q ? p.q : p.k, sb + d1, p.in_f16);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t w = w0 + u * blockDim.x;
      if (w >= total) continue;
      if (w >= nq + nk) {
        __half* dst = p.v_cache + (p.cache_row0 + col) * (uint64_t)kvd + 2 * (w - nq - nk);
        dst[0] = f16_rne(a[u]); dst[1] = f16_rne(b[u]);
        continue;
      }
      const bool is_q = w < nq;
      const uint32_t ww = is_q ? w : w - nq, head = ww / pairs, pr = ww % pairs;
      const uint32_t d0 = pr < half ? pr : p.n_rot + 2 * (pr - half), d1 = pr < half ? pr + half : d0 + 1;
      float ra = a[u], rb = b[u];
      if (p.mode != PA_ROPE_NONE && pr < half) {
        if (p.mode == PA_ROPE_F64) {
          const Angle g = s_g[pr];
          ra = rot_exact(a[u], b[u], g, true);
          rb = rot_exact(b[u], a[u], g, false);
        } else {
          const float c = p.cs_table[(uint64_t)col * p.n_rot + 2 * pr], sn = p.cs_table[(uint64_t)col * p.n_rot + 2 * pr + 1];
          ra = __fsub_rn(__fmul_rn(a[u], c), __fmul_rn(b[u], sn));
          rb = __fadd_rn(__fmul_rn(a[u], sn), __fmul_rn(b[u], c));
        }
      }
      if (is_q) {
        const uint64_t o = (uint64_t)col * p.q_out_col_stride + (uint64_t)head * hd;
        if (p.q_out_f16 == 2) {   // high and low f16 parts for the verify kernel's hi / lo rows
      __half* dst = reinterpret_cast<__half*>(p.q_out) + o;
      const __half ha = __float2half_rn(ra), hb = __float2half_rn(rb);
      dst[d0] = ha; dst[d1] = hb;
      dst[p.q_lo_offset + d0] = __float2half_rn(ra - __half2float(ha)); dst[p.q_lo_offset + d1] = __float2half_rn(rb - __half2float(hb));
    } else if (p.q_out_f16) { __half* dst = reinterpret_cast<__half*>(p.q_out) + o; dst[d0] = __float2half_rn(ra); dst[d1] = __float2half_rn(rb); }
        else { float* dst = reinterpret_cast<float*>(p.q_out) + o; dst[d0] = ra; dst[d1] = rb; }
      } else {
        __half* dst = p.k_cache + (p.cache_row0 + col) * (uint64_t)kvd + (uint64_t)head * hd;
        dst[d0] = f16_rne(ra); dst[d1] = f16_rne(rb);
      }
    }
  }
}


// Prefill chunks of f16 activations with the rotated q stored as f16 (what the prefill kernel consumes): the same
// results as the kernels above.  The rotated dims first, then 16-byte vectors of everything that is only copied (NaNs
// take the pattern the scalar path produces).
__device__ __forceinline__ uint32_t fix_nan2(uint32_t w, bool cache) {
  // per half: NaN -> 0x7fff (q, cvt.rn.f16.f32 of a NaN) or sign | 0x7e00 (cache, f16_rne)
  uint32_t out = w;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const uint32_t h = (w >> (16 * e)) & 0xffffu;
    if ((h & 0x7c00u) == 0x7c00u && (h & 0x03ffu)) {
      const uint32_t r = cache ? ((h & 0x8000u) | 0x7e00u) : 0x7fffu;
      out = (out & ~(0xffffu << (16 * e))) | (r << (16 * e));
    }
  }
  return out;
}
// one output the way of the other kernels, in the few cases rot_h() leaves open: the cache takes f16_rne's NaN pattern
static __device__ __noinline__ uint32_t rot_h_slow(uint32_t xw, uint32_t yw, int shift, const Angle* g, bool minus, bool cache) {
  const float x = __half2float(__ushort_as_half((unsigned short)(xw >> shift))), y = __half2float(__ushort_as_half((unsigned short)(yw >> shift)));
  const float r = rot_exact(x, y, *g, minus);
  return cache ? __half_as_ushort(f16_rne(r)) : __half_as_ushort(__float2half_rn(r));
}
// 64 threads per column, four columns per CTA.  Thread t of a column holds the cos / sin of eight neighbouring dims and
// walks the heads t / (half / 8), + 64 / (half / 8), ...: 16-byte loads and stores on both sides, the angles loaded once,
// rot_h() for the arithmetic, everything of a thread's first turn requested before anything is used.  Eight layers of 2999
// columns of 16 + 8 heads x 128, whole calls: 639 us with one kind of load after the other, two heads at a time, 612 so.  8192
// columns of 24 heads of which 64 dims turn take 47 us for 117 MB: 128-byte pieces of q 1 KB apart.
// half / 8 need not divide 64: the threads past the last whole turn then only copy.
// kRopeU heads and kRopeC copied vectors a thread has in flight: three and four, or, up to kRopeFew columns (one wave of two CTAs an SM),
// one and two.  There a CTA's time is the fetch of its instructions, which the kernels between two of its launches have put out
// of the SM's caches, and three heads' arithmetic is three times as long.  A layer call of 48 columns of 16 / 8 heads x 128: 13.5 us
// with three and four, 12.5 with one and two (two heads one after the other's loads, as before both: 12.9); 300 columns 15.9 and 15.0, 1100 25.7
// and 24.8, 2999 73.8 and 75.2.
constexpr uint32_t kRopeFew = 1184;
template <int kRopeU, int kRopeC>
__global__ void __launch_bounds__(256, 2) pa_rope_append_vec_kernel(const RopeParams p, const uint32_t n_cols) {
  __shared__ float2 s_cs[4][128];
  const uint32_t cl = threadIdx.x >> 6, t = threadIdx.x & 63, col = min(blockIdx.x * 4 + cl, n_cols - 1), half = p.n_rot / 2, hd = p.hd;
  const bool live = blockIdx.x * 4 + cl < n_cols;
  if (p.trigger_early) pdl_trigger();
  const uint32_t kvd = p.kv_heads * hd;
  const __half* qs = reinterpret_cast<const __half*>(p.q) + (uint64_t)col * p.q_col_stride;
  const __half* ks = reinterpret_cast<const __half*>(p.k) + (uint64_t)col * p.kv_col_stride;
  const __half* vs = reinterpret_cast<const __half*>(p.v) + (uint64_t)col * p.v_col_stride;
  __half* qd = reinterpret_cast<__half*>(p.q_out) + (uint64_t)col * p.q_out_col_stride;
  __half* kd = p.k_cache + (p.cache_row0 + col) * (uint64_t)kvd;
  __half* vd = p.v_cache + (p.cache_row0 + col) * (uint64_t)kvd;
  const uint32_t nqh = p.q ? p.q_heads : 0, nh = live ? nqh + (p.k ? p.kv_heads : 0) : 0;
  const uint32_t groups = half / 8, step = 64 / groups, d = (t % groups) * 8;
  // everything but the rotated dims: 16-byte vectors of the unrotated dims of q and k, and all of v
  const uint32_t cv = (hd - p.n_rot) / 8, vv = hd / 8;
  const uint32_t nq = p.q_rot_only ? 0u : nqh * cv, nk = (p.k ? p.kv_heads : 0) * cv, nv = p.v ? p.kv_heads * vv : 0, total = live ? nq + nk + nv : 0;
  uint4 A[kRopeU], B[kRopeU], C[kRopeC];
  auto load_heads = [&](uint32_t h0) {     // dims d .. d + 7 of heads h0, h0 + step, ... with their partners half further on
#pragma unroll
    for (int u = 0; u < kRopeU; ++u) {
      const uint32_t h = h0 + u * step;
      if (h >= nh) continue;
      const __half* src = (h < nqh ? qs + (uint64_t)h * p.q_head_stride : ks + (uint64_t)(h - nqh) * hd) + d;
      A[u] = *reinterpret_cast<const uint4*>(src);
      B[u] = *reinterpret_cast<const uint4*>(src + half);
    }
  };
  auto load_copies = [&](uint32_t w0) {
#pragma unroll
    for (int u = 0; u < kRopeC; ++u) {
      const uint32_t w = w0 + u * 64;
      if (w >= total) continue;
      const __half* src;
      if (w >= nq + nk) src = vs + 8 * (w - nq - nk);
      else {
        const bool is_q = w < nq;
        const uint32_t ww = is_q ? w : w - nq, head = ww / cv, dd = p.n_rot + 8 * (ww % cv);
        src = (is_q ? qs + (uint64_t)head * p.q_head_stride : ks + (uint64_t)head * hd) + dd;
      }
      C[u] = *reinterpret_cast<const uint4*>(src);
    }
  };
  auto store_copies = [&](uint32_t w0) {
#pragma unroll
    for (int u = 0; u < kRopeC; ++u) {
      const uint32_t w = w0 + u * 64;
      if (w >= total) continue;
      __half* dst;
      bool cache = true;
      if (w >= nq + nk) dst = vd + 8 * (w - nq - nk);
      else {
        const bool is_q = w < nq;
        const uint32_t ww = is_q ? w : w - nq, head = ww / cv, dd = p.n_rot + 8 * (ww % cv);
        cache = !is_q;
        dst = (is_q ? qd + (uint64_t)head * hd : kd + (uint64_t)head * hd) + dd;
      }
      uint4 o = C[u];
      o.x = fix_nan2(o.x, cache); o.y = fix_nan2(o.y, cache); o.z = fix_nan2(o.z, cache); o.w = fix_nan2(o.w, cache);
      *reinterpret_cast<uint4*>(dst) = o;
    }
  };
  const uint32_t first_h = t < groups * step ? t / groups : nh;
  pdl_wait();
  if (!p.trigger_early) pdl_trigger();
  // a column's angles, rotated dims and copies are all requested before the first of them is used
  const Angle* ang = p.angles + (uint64_t)col * half;
  for (uint32_t i = t; i < half; i += 64) s_cs[cl][i] = make_float2(ang[i].c_hi, ang[i].s_hi);
  load_heads(first_h);
  load_copies(t);
  __syncthreads();
  float2 cs[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) cs[e] = s_cs[cl][d + e];
  for (uint32_t h0 = first_h; h0 < nh; h0 += kRopeU * step) {
    if (h0 != first_h) load_heads(h0);
#pragma unroll
    for (int u = 0; u < kRopeU; ++u) {
      const uint32_t h = h0 + u * step;
      if (h >= nh) continue;
      const uint32_t aw[4] = {A[u].x, A[u].y, A[u].z, A[u].w}, bw[4] = {B[u].x, B[u].y, B[u].z, B[u].w};
      uint32_t ra[8], rb[8], bad = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 a2 = __half22float2(*reinterpret_cast<const __half2*>(&aw[e >> 1])), b2 = __half22float2(*reinterpret_cast<const __half2*>(&bw[e >> 1]));
        const float x = e & 1 ? a2.y : a2.x, y = e & 1 ? b2.y : b2.x;
        bool ok1, ok2;
        ra[e] = rot_h(x, y, cs[e].x, cs[e].y, true, ok1);
        rb[e] = rot_h(y, x, cs[e].x, cs[e].y, false, ok2);
        bad |= (ok1 ? 0u : 1u << e) | (ok2 ? 0u : 256u << e);
      }
      if (bad) {
        const bool cache = h >= nqh;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (bad & (1u << e)) ra[e] = rot_h_slow(aw[e >> 1], bw[e >> 1], 16 * (e & 1), ang + d + e, true, cache);
          if (bad & (256u << e)) rb[e] = rot_h_slow(bw[e >> 1], aw[e >> 1], 16 * (e & 1), ang + d + e, false, cache);
        }
      }
      __half* dst = (h < nqh ? qd + (uint64_t)h * hd : kd + (uint64_t)(h - nqh) * hd) + d;
      *reinterpret_cast<uint4*>(dst) = make_uint4(ra[0] | (ra[1] << 16), ra[2] | (ra[3] << 16), ra[4] | (ra[5] << 16), ra[6] | (ra[7] << 16));
      *reinterpret_cast<uint4*>(dst + half) = make_uint4(rb[0] | (rb[1] << 16), rb[2] | (rb[3] << 16), rb[4] | (rb[5] << 16), rb[6] | (rb[7] << 16));
    }
  }
  store_copies(t);
  for (uint32_t w0 = t + kRopeC * 64; w0 < total; w0 += kRopeC * 64) {
    load_copies(w0);
    store_copies(w0);
  }
}

// cos / sin of every (column, rotary pair) of a call, evaluated once in float64 and shared by all layers of the step
// (the host keeps the table while position and width stay the same)
__global__ void __launch_bounds__(128) pa_angles_kernel(const AnglesParams p) {
  pdl_wait();        // an earlier kernel may still be reading the table
  pdl_trigger();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n_cols * p.half) return;
  double s, c;
  sincos(__dmul_rn((double)(p.pos0 + i / p.half), p.inv_freq[i % p.half]), &s, &c);
  p.out[i] = make_angle(c, s);
}

// QK head-norm (the step before RoPE in attn_glue, engine/wgsl/qwen35.js:1112-1122), with the bits of the CPU reference
// (tests/reference/ref_q38.mjs:50-57): out = f32((x * inv) * w), inv = 1 / sqrt(ss / hd + eps), ss the float64 sum of the
// squares in index order.  A warp per (column, head), four warps per CTA; a lane holds hd / 32 values.  The squares are
// summed in parallel and head_norm_value() says for each output whether the order of the sum could show in it; only
// then (about one head in 2^12) the warp repeats the sum in index order.  What bounds it is latency: the in-order sum
// alone is 256 dependent float64 additions, and one thread per head made them (eight layers of 203 columns of 24 + 4 heads, whole calls:
// 1695 us so, 1640 us with the parallel sum).
// grid (ceil(columns * heads / 4)).
__global__ void __launch_bounds__(128) pa_head_norm_kernel(const HeadNormParams p) {
  const uint32_t hd = p.hd, lane = threadIdx.x & 31, unit = blockIdx.x * 4 + (threadIdx.x >> 5);
  pdl_wait();
  pdl_trigger();
  if (unit >= p.n_cols * p.n_heads) return;
  const uint32_t col = unit / p.n_heads, slot = unit % p.n_heads;
  const bool second = slot >= p.n_first;
  const uint32_t head = second ? slot - p.n_first : slot;
  const void* x = second ? p.x2 : p.x;
  void* y = second ? p.y2 : p.y;
  const float* w = second ? p.w2 : p.w;
  const uint64_t xo = (uint64_t)col * (second ? p.x2_col_stride : p.x_col_stride) + (uint64_t)head * (second ? p.x2_head_stride : p.x_head_stride);
  const uint64_t yo = (uint64_t)col * (second ? p.y2_col_stride : p.y_col_stride) + (uint64_t)head * (second ? p.y2_head_stride : p.y_head_stride);
  constexpr int MAXV = 16;   // head_dim up to 512
  float xv[MAXV], wv[MAXV];
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const uint32_t d = lane + 32 * i;
    xv[i] = d < hd ? ld_act(x, xo + d, p.f16) : 0.f;
    wv[i] = d < hd ? w[d] : 0.f;
  }
  double ss = 0.0;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) if (32u * i < hd) ss = __fma_rn((double)xv[i], (double)xv[i], ss);   // a product of two f32 is exact in float64
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
  double inv = head_norm_inv(ss, hd, p.eps);
  bool ok = true;
  float r[MAXV];
#pragma unroll
  for (int i = 0; i < MAXV; ++i) if (lane + 32u * i < hd) r[i] = head_norm_value(xv[i], inv, wv[i], ok);
  if (!__all_sync(0xffffffffu, ok)) {
    inv = head_norm_inv(head_norm_sum_in_order(x, xo, hd, p.f16), hd, p.eps);
#pragma unroll
    for (int i = 0; i < MAXV; ++i) r[i] = (float)__dmul_rn(__dmul_rn((double)xv[i], inv), (double)wv[i]);
  }
  __syncwarp();   // in place: every lane of the warp has read its values, and the in-order sum its row
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const uint32_t d = lane + 32 * i;
    if (d >= hd) continue;
    if (p.f16) reinterpret_cast<__half*>(y)[yo + d] = __float2half_rn(r[i]);
    else reinterpret_cast<float*>(y)[yo + d] = r[i];
  }
}

__global__ void __launch_bounds__(256) pa_sigmoid_mul_kernel(const SigmoidParams p) {
  const uint32_t col = blockIdx.x, n = p.n_heads * p.hd;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t h = i / p.hd, d = i % p.hd;
    const uint64_t ao = (uint64_t)col * p.a_col_stride + i, go = (uint64_t)col * p.g_col_stride + (uint64_t)h * p.g_head_stride + d;
    const float gv = ld_act(p.g, go, p.f16);
    const float sg = 1.0f / (1.0f + expf(-gv));
    if (p.f16) reinterpret_cast<__half*>(p.a)[ao] = __float2half_rn(__half2float(reinterpret_cast<__half*>(p.a)[ao]) * sg);
    else reinterpret_cast<float*>(p.a)[ao] = reinterpret_cast<float*>(p.a)[ao] * sg;
  }
}

// whether a call goes to the vectorised kernel (the only one that knows q_rot_only)
bool rope_vec_applies(const RopeParams& p, uint32_t n_cols) {
  auto al16 = [](const void* x) { return ((uintptr_t)x & 15) == 0; };
  return !p.n_items && n_cols >= 16 && p.mode == PA_ROPE_F64 && p.angles && p.in_f16 && p.n_rot % 16 == 0 && p.n_rot <= 256 && p.hd % 8 == 0 &&
         (!p.q || (p.q_out_f16 == 1 && al16(p.q) && al16(p.q_out) && p.q_col_stride % 8 == 0 && p.q_head_stride % 8 == 0 && p.q_out_col_stride % 8 == 0)) &&
         (!p.k || (p.v && al16(p.k) && al16(p.v) && p.kv_col_stride % 8 == 0 && p.v_col_stride % 8 == 0));
}

cudaError_t launch_rope_append(const RopeParams& p, uint32_t n_cols, cudaStream_t st) {
  if (rope_vec_applies(p, n_cols)) {
    const dim3 grid((n_cols + 3) / 4);
    return n_cols <= kRopeFew ? launch_pdl(pa_rope_append_vec_kernel<1, 2>, grid, dim3(256), 0, st, p, n_cols)
                              : launch_pdl(pa_rope_append_vec_kernel<3, 4>, grid, dim3(256), 0, st, p, n_cols);
  }
  if (n_cols >= 16 && !p.n_items) return launch_pdl(pa_rope_append_cols_kernel, dim3(n_cols), dim3(256), 0, st, p);
  const uint32_t slots = (p.q ? p.q_heads : 0) + (p.k ? p.kv_heads : 0) + (p.v ? p.kv_heads : 0);
  return launch_pdl(pa_rope_append_kernel, dim3(n_cols, slots), dim3(128), 0, st, p);
}
cudaError_t launch_angles(const AnglesParams& p, cudaStream_t st) {
  return launch_pdl(pa_angles_kernel, dim3((p.n_cols * p.half + 127) / 128), dim3(128), 0, st, p);
}
cudaError_t launch_head_norm(const HeadNormParams& p, cudaStream_t st) {
  return launch_pdl(pa_head_norm_kernel, dim3((uint32_t)(((uint64_t)p.n_cols * p.n_heads + 3) / 4)), dim3(128), 0, st, p);
}
cudaError_t launch_sigmoid_mul(const SigmoidParams& p, uint32_t n_cols, cudaStream_t st) {
  pa_sigmoid_mul_kernel<<<n_cols, 256, 0, st>>>(p);
  return cudaGetLastError();
}

}  // namespace pa
