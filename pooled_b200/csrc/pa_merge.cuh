// The merge of split records inside the kernel that makes them (f16 decode, f32 tokens).  Not in the kernel of token blocks, whose
// 30 rows x 4 slices over 37 CTAs are two rounds of units that hold every SM (16 layers of a 5-token block over 16384 rows: 355 us with the
// combine kernel, 396 so), nor in pa_q8_kernel (ten layers of a token over 12345 rows: 182 and 181).
#pragma once
#include "pa_params.cuh"

namespace pa {

// acc += x * w, each component one fused multiply-add: the merge inside the decode kernel (merge_slice_128) and the
// combine kernel round the same way, so either path gives the same bits
__device__ __forceinline__ void fma4(float4& acc, const float4& x, float w) {
  acc.x = __fmaf_rn(x.x, w, acc.x); acc.y = __fmaf_rn(x.y, w, acc.y); acc.z = __fmaf_rn(x.z, w, acc.z); acc.w = __fmaf_rn(x.w, w, acc.w);
}

// Records that the CTAs of one call leave for one another say themselves when they are there: every 32-bit word of the buffer holds
// kNoWord until its value is stored, a reader repeats its loads until no word of them does, and puts kNoWord back for the next call
// (whose CTAs write after this call's end).  Both sides use relaxed accesses of whole 32-bit words, which land whole, and nothing else orders them: with a fence behind
// the records, a count and a wait for it ahead of the first load, three more trips to L2 stood between a CTA's last product and its merge
// (ten layers of a token over 32768 rows, 16 / 2 heads x 256, head-norm: 193.5 us with them, 185 without; 16 over 4099 rows, 24 / 4 x 256, host
// buffers: 238 and 209).  A value that has kNoWord's bits (a NaN no instruction here produces) is stored as the ordinary NaN.
constexpr uint32_t kNoWord = 0xffffffffu;
__device__ __forceinline__ uint32_t word_for(float x) { return __float_as_uint(x) == kNoWord ? 0x7fffffffu : __float_as_uint(x); }
__device__ __forceinline__ uint4 ld_words4(const float* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_words2(const float* p) {
  uint2 v;
  asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_words4(float* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void st_words2(float* p, uint32_t a, uint32_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ bool all_words(const uint4& v) { return v.x != kNoWord && v.y != kNoWord && v.z != kNoWord && v.w != kNoWord; }
__device__ __forceinline__ float4 as_float4(const uint4& v) { return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
// named_bar_sync that also says whether any of the threads brought a non-zero value
__device__ __forceinline__ bool named_bar_any(uint32_t id, uint32_t threads, uint32_t v) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\tbar.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(any) : "r"(id), "r"(threads), "r"(v) : "memory");
  return any != 0;
}

// LSE merge of the ns split records of one query row over one 64-dim slice, gate and store, by the 128 consumer threads
// of a decode CTA: the arithmetic of pa_combine_kernel, operation for operation and in the same order (that kernel has
// 256 threads; thread t here does the work of its threads t and t + 128), so a call gives the same bits whether its
// records are merged here or there.  o_rec / ml_rec: the slice of record 0 of the row; records lie `stride` floats apart.  Scratch:
// 6 KB of shared memory no one else uses any more.  bar: the group's named barrier.  Where a record was not there within `limit`
// looks: LEAVE: false, to all threads, the buffer as it was; otherwise the error word is set.  (One form for both cost f16 tokens 3 %: 16 over 4099
// rows, host buffers, 197 -> 203 us.)
struct MergeScratch { float w[512]; float red[8]; float red2[8]; float4 acc[16][16]; };
template <int HD, bool LEAVE>
__device__ __forceinline__ bool merge_slice_128(float* o_rec, float* ml_rec, size_t stride, uint32_t ns, int t, MergeScratch& sc, uint32_t bar, bool gated,
                                                float gv, bool empty_is_zero, int act_f16, void* out, uint64_t oo, uint32_t limit, volatile uint32_t* s_err) {
  const int wv = t >> 5, lane = t & 31, ln = t & 15, gA = t >> 4;
  float* ob = o_rec + ln * 4;
  // everything is requested before the first use, and whatever was not there yet once more
  uint4 xw[16];          // records gA + 8 i of this thread's four dims
  uint2 mw[4];
  uint32_t want = 0;     // bits 0-15: xw, 16-19: mw
#pragma unroll
  for (int i = 0; i < 16; ++i) { xw[i] = make_uint4(0, 0, 0, 0); want |= (gA + 8u * i < ns ? 1u : 0u) << i; }
#pragma unroll
  for (int k = 0; k < 4; ++k) { mw[k] = make_uint2(__float_as_uint(-3.0e38f), 0u); want |= (t + 128u * k < ns ? 1u : 0u) << (16 + k); }
  const uint32_t mine = want;
  for (uint32_t polls = 0; want && polls < limit && !*s_err; ++polls) {
#pragma unroll
    for (int k = 0; k < 4; ++k) if ((want >> (16 + k)) & 1u) mw[k] = ld_words2(ml_rec + (size_t)(t + 128 * k) * stride);
#pragma unroll
    for (int i = 0; i < 16; ++i) if ((want >> i) & 1u) xw[i] = ld_words4(ob + (size_t)(gA + 8 * i) * stride);
#pragma unroll
    for (int k = 0; k < 4; ++k) if (((want >> (16 + k)) & 1u) && mw[k].x != kNoWord && mw[k].y != kNoWord) want &= ~(1u << (16 + k));
#pragma unroll
    for (int i = 0; i < 16; ++i) if (((want >> i) & 1u) && all_words(xw[i])) want &= ~(1u << i);
    if (want && polls > 16) __nanosleep(32);
  }
  float mv[4], lv[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) { mv[k] = __uint_as_float(mw[k].x); lv[k] = __uint_as_float(mw[k].y); }
  auto put_back = [&] {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if ((mine >> (16 + k)) & 1u) st_words2(ml_rec + (size_t)(t + 128 * k) * stride, kNoWord, kNoWord);
#pragma unroll
    for (int i = 0; i < 16; ++i) if ((mine >> i) & 1u) st_words4(ob + (size_t)(gA + 8 * i) * stride, kNoWord, kNoWord, kNoWord, kNoWord);
  };
  if (!LEAVE) {
    if (want) *s_err = WAIT_MERGE;
    put_back();
  }
  float M = fmaxf(fmaxf(mv[0], mv[1]), fmaxf(mv[2], mv[3]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  if (lane == 0) sc.red[wv] = M;
  if (LEAVE) {
    if (named_bar_any(bar, 128, want)) return false;
    put_back();
  } else {
    named_bar_sync(bar, 128);
  }
  M = fmaxf(fmaxf(sc.red[0], sc.red[1]), fmaxf(sc.red[2], sc.red[3]));
  float wk[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t s = t + 128 * k;
    wk[k] = s < ns ? __expf(mv[k] - M) : 0.f;
    sc.w[s] = wk[k];
  }
  // the combine kernel's thread v sums records v and v + 256, then its warp reduces: v = t and v = t + 128 here
  float LpA = __fmaf_rn(lv[2], wk[2], __fmul_rn(lv[0], wk[0])), LpB = __fmaf_rn(lv[3], wk[3], __fmul_rn(lv[1], wk[1]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    LpA = __fadd_rn(LpA, __shfl_xor_sync(0xffffffffu, LpA, o));
    LpB = __fadd_rn(LpB, __shfl_xor_sync(0xffffffffu, LpB, o));
  }
  if (lane == 0) { sc.red2[wv] = LpA; sc.red2[wv + 4] = LpB; }
  named_bar_sync(bar, 128);
  float Lsum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) Lsum = __fadd_rn(Lsum, sc.red2[i]);
  float4 accA = make_float4(0.f, 0.f, 0.f, 0.f), accB = accA;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const uint32_t sa = gA + 16 * u, sb = gA + 8 + 16 * u;
    fma4(accA, as_float4(xw[2 * u]), sa < ns ? sc.w[sa] : 0.f);
    fma4(accB, as_float4(xw[2 * u + 1]), sb < ns ? sc.w[sb] : 0.f);
  }
  for (int h = 0; h < 2; ++h) {
    const uint32_t g = gA + 8 * h;
    float4& acc = h ? accB : accA;
    for (uint32_t s0 = g + 128; s0 < ns; s0 += 64) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t s = s0 + 16 * u;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (s < ns) {
          for (uint32_t polls = 0; !*s_err; ++polls) {
            x = ld_words4(ob + (size_t)s * stride);
            if (all_words(x)) break;
            if (polls > kMergePolls) *s_err = WAIT_MERGE;
            if (polls > 16) __nanosleep(32);
          }
          st_words4(ob + (size_t)s * stride, kNoWord, kNoWord, kNoWord, kNoWord);
        }
        fma4(acc, as_float4(x), s < ns ? sc.w[s] : 0.f);
      }
    }
  }
  sc.acc[gA][ln] = accA; sc.acc[gA + 8][ln] = accB;
  named_bar_sync(bar, 128);
  float tt = 0.f;
  if (t < 64) {
    const float* sa = reinterpret_cast<const float*>(sc.acc);
    tt = sa[t];
#pragma unroll
    for (int i = 1; i < 16; ++i) tt = __fadd_rn(tt, sa[i * 64 + t]);
  }
  if (t < 64) {
    float rv = (empty_is_zero && Lsum == 0.f) ? 0.f : __fdiv_rn(tt, Lsum);
    if (gated) rv = __fmul_rn(rv, __fdiv_rn(1.0f, __fadd_rn(1.0f, __expf(-gv))));
    if (act_f16) reinterpret_cast<__half*>(out)[oo + t] = __float2half_rn(rv);
    else reinterpret_cast<float*>(out)[oo + t] = rv;
  }
  named_bar_sync(bar, 128);   // the scratch is free again
  return true;
}

// A CTA's block of a record buffer: o [rows][HD], then (m, l) once for each 64-dim slice, [rows][HD / 64][2]; whole 16-byte vectors, so
// that every block's rows are aligned for the vector accesses (one row of 64 dims alone is 264 bytes)
__host__ __device__ constexpr size_t merge_block(int hd, int rows) { return ((size_t)rows * (hd + hd / 32) + 3) & ~(size_t)3; }
// row `row` of a CTA's record: four of its values, and beside the first of each 64 (m in natural-log units, l)
template <int HD>
__device__ __forceinline__ void put_record4(float* blk, uint32_t rows, uint32_t row, uint32_t c4, float4 x, float m, float l) {
  static_assert(HD % 4 == 0 && merge_block(HD, 1) % 4 == 0 && merge_block(HD, 2) % 4 == 0, "records are read and written 16 bytes at a time");
  if (c4 % 16 == 0) st_words2(blk + (size_t)rows * HD + (row * (HD / 64) + c4 / 16) * 2, word_for(m), word_for(l));
  st_words4(blk + (size_t)row * HD + c4 * 4, word_for(x.x), word_for(x.y), word_for(x.z), word_for(x.w));
}

}  // namespace pa
