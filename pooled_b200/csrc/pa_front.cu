// The front of a layer call in one launch, a warp per (column, head): QK head-norm (where the layer has one), rotation, and
// the append in the cache's own format.  The arithmetic is that of the kernels it stands for, operation for operation
// (pa_head_norm_kernel, the RoPE kernels, pa_kv_store_q8_kernel, pa_kv_store_f32_kernel): the same bits.
//
// As separate kernels an int8 layer's front was four launches (norm, q, k, store) with the rotated k and the normed q and
// k making a round trip through memory between them; each is a few microseconds of latency and next to no work (a token over
// f32 caches, 28 layers of 16 + 8 heads x 128: 829 us with the separate kernels, 644 us with this one).  Lane i
// holds values i, i + 32, ..., so rotary partners (32 or 64 apart) sit in one lane, a 32-value block of the int8 format is
// one value per lane, and every load and store of the warp is one contiguous run.
#include "pa_params.cuh"

namespace pa {

// HB: 32-value groups of half the rotary width (n_rot = 64 HB); 0: nothing is rotated
template <int HD, int HB>
__global__ void __launch_bounds__(128) pa_front_kernel(const FrontParams p) {
  constexpr int NV = HD / 32;
  __shared__ Angle s_ang[64];
  const uint32_t lane = threadIdx.x & 31, unit = blockIdx.x * 4 + (threadIdx.x >> 5);
  const uint32_t nq = p.q ? p.q_heads : 0, per_col = nq + 2 * p.kv_heads;
  if (HB && p.n_ang) {   // by-value angles go through shared memory (indexed per thread they are served one at a time)
    if (threadIdx.x < p.n_ang * 2) reinterpret_cast<uint4*>(s_ang)[threadIdx.x] = reinterpret_cast<const uint4*>(p.ang)[threadIdx.x];
    __syncthreads();
  }
  pdl_wait();
  pdl_trigger();         // the attention kernel may fetch rows older than this call's now
  if (unit >= per_col * p.n_cols) return;
  const uint32_t col = unit / per_col, slot = unit % per_col;
  const int what = slot < nq ? 0 : slot < nq + p.kv_heads ? 1 : 2;      // q, k or v
  const uint32_t head = what == 0 ? slot : what == 1 ? slot - nq : slot - nq - p.kv_heads;
  const void* src = what == 0 ? p.q : what == 1 ? p.k : p.v;
  const uint64_t so = what == 0 ? (uint64_t)col * p.q_col_stride + (uint64_t)head * p.q_head_stride
                                : (uint64_t)col * (what == 1 ? p.k_col_stride : p.v_col_stride) + (uint64_t)head * HD;
  float x[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) x[i] = ld_act(src, so + lane + 32 * i, p.in_f16);
  const float* nw = what == 0 ? p.qn_w : what == 1 ? p.kn_w : nullptr;
  Angle ang[HB ? HB : 1];
  if (HB && what < 2) {
#pragma unroll
    for (int i = 0; i < HB; ++i) ang[i] = p.n_ang ? s_ang[col * 32 * HB + 32 * i + lane] : p.angles[(uint64_t)col * 32 * HB + 32 * i + lane];
  }
  if (nw) {
    double ss = 0.0;
#pragma unroll
    for (int i = 0; i < NV; ++i) ss = __fma_rn((double)x[i], (double)x[i], ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
    double inv = head_norm_inv(ss, HD, p.norm_eps);
    bool ok = true;
    float y[NV], w[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) { w[i] = nw[lane + 32 * i]; y[i] = head_norm_value(x[i], inv, w[i], ok); }
    if (!__all_sync(0xffffffffu, ok)) {
      inv = head_norm_inv(head_norm_sum_in_order(src, so, HD, p.in_f16), HD, p.norm_eps);
#pragma unroll
      for (int i = 0; i < NV; ++i) y[i] = (float)__dmul_rn(__dmul_rn((double)x[i], inv), (double)w[i]);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) x[i] = p.in_f16 ? __half2float(__float2half_rn(y[i])) : y[i];   // the layer's activation type
  }
  if (HB && what < 2) {
#pragma unroll
    for (int i = 0; i < HB; ++i) {
      const float a = x[i], b = x[i + HB];
      x[i] = rot_exact(a, b, ang[i], true); x[i + HB] = rot_exact(b, a, ang[i], false);
    }
  }
  if (what == 0) {
    const uint64_t o = (uint64_t)col * p.q_out_col_stride + (uint64_t)head * HD + lane;
    if (p.q_out_f16 == 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) reinterpret_cast<float*>(p.q_out)[o + 32 * i] = x[i];
    } else {
      __half* dst = reinterpret_cast<__half*>(p.q_out) + o;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const __half h = __float2half_rn(x[i]);
        dst[32 * i] = h;
        if (p.q_out_f16 == 2) dst[p.q_lo_offset + 32 * i] = __float2half_rn(x[i] - __half2float(h));
      }
    }
    return;
  }
  const uint64_t row = p.cache_row0 + col, kvd = (uint64_t)p.kv_heads * HD, eo = row * kvd + (uint64_t)head * HD + lane;
  void* cache = what == 1 ? p.k_cache : p.v_cache;
  if (p.format == PA_KV_F16) {
#pragma unroll
    for (int i = 0; i < NV; ++i) reinterpret_cast<__half*>(cache)[eo + 32 * i] = f16_rne(x[i]);
  } else if (p.format == PA_KV_F32) {
#pragma unroll
    for (int i = 0; i < NV; ++i) reinterpret_cast<float*>(cache)[eo + 32 * i] = x[i];
  } else {
    float* sc_out = (what == 1 ? p.k_scale : p.v_scale) + row * (kvd / 32) + head * NV;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      // the largest |x| of the block; a NaN does not count, as with fmaxf (non-negative floats order as integers)
      const uint32_t ab = x[i] != x[i] ? 0u : __float_as_uint(x[i]) & 0x7fffffffu;
      const float a = __uint_as_float(__reduce_max_sync(0xffffffffu, ab));
      const float sc = __fdiv_rn(a, 127.0f), inv = sc > 0.f ? __fdiv_rn(1.0f, sc) : 0.f;
      reinterpret_cast<int8_t*>(cache)[eo + 32 * i] = (int8_t)(int)fminf(fmaxf(rintf(__fmul_rn(x[i], inv)), -127.0f), 127.0f);
      if (lane == 0) sc_out[i] = sc;
    }
  }
}

bool front_supported(uint32_t hd, uint32_t n_rot, bool rotates) {
  if (!rotates) return hd == 256 || hd == 128 || hd == 64;
  return (n_rot == 64 && (hd == 256 || hd == 128 || hd == 64)) || (n_rot == 128 && hd == 128);
}
cudaError_t launch_front(const FrontParams& p, uint32_t hd, uint32_t n_rot, cudaStream_t st) {
  const uint64_t units = (uint64_t)p.n_cols * ((p.q ? p.q_heads : 0) + 2 * p.kv_heads);
  const dim3 grid((uint32_t)((units + 3) / 4)), block(128);
  if (hd == 256) return n_rot ? launch_pdl(pa_front_kernel<256, 1>, grid, block, 0, st, p) : launch_pdl(pa_front_kernel<256, 0>, grid, block, 0, st, p);
  if (hd == 128) return n_rot == 128 ? launch_pdl(pa_front_kernel<128, 2>, grid, block, 0, st, p)
                      : n_rot ? launch_pdl(pa_front_kernel<128, 1>, grid, block, 0, st, p) : launch_pdl(pa_front_kernel<128, 0>, grid, block, 0, st, p);
  return n_rot ? launch_pdl(pa_front_kernel<64, 1>, grid, block, 0, st, p) : launch_pdl(pa_front_kernel<64, 0>, grid, block, 0, st, p);
}

}  // namespace pa
