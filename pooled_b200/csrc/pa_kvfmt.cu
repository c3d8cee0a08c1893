// KV caches in the other two formats pooled's engines keep: int8 with one f32 scale per 32 values (kvQ8: kv_store_q8 +
// attn_flash_q8, engine/wgsl/qwen35.js:97-139, :908-946) and f32 (the dense engine, engine/wgsl/dense.js:22-136).
//
// The f16 cache has the TMA / tensor-core kernels of pa_decode.cu and pa_prefill.cu, the int8 cache pa_q8.cu.  The f32
// cache has a split-K kernel of the same outer shape (one CTA per (split, kv head, column), an unnormalised (o, m, l)
// record per (row, split) for pa_combine_kernel) built from plain vector loads: per chunk of 64 positions
//   scores   four threads per K row, a quarter of the head each, the G heads of the group per thread; q in shared memory
//   softmax  32 threads per head, online rescale across chunks (m starts at -3.0e38, as in the reference)
//   values   a thread per four dims and group of positions, the groups summed in a fixed order at the end
// A row of kv_dim values costs kv_dim * 1.125 bytes (int8) or kv_dim * 4 bytes (f32) against kv_dim * 2 for f16.
#include "pa_merge.cuh"

namespace pa {

// ---- append -------------------------------------------------------------------------------------------------

// kv_store_q8 (engine/wgsl/qwen35.js:908-946), operation for operation: per block of 32 values scale = max|x| / 127,
// inv = 1 / scale (0 when the block is all zeros), value = clamp(round_to_nearest_even(x * inv), -127, 127).
// grid (kv_dim / 32 blocks, columns), one thread per (block, K or V).
__global__ void __launch_bounds__(64) pa_kv_store_q8_kernel(const KvStoreParams p) {
  pdl_wait();
  pdl_trigger();
  const uint32_t nb = p.kv_dim / 32, blk = blockIdx.x * 32 + (threadIdx.x & 31), col = blockIdx.y, which = threadIdx.x >> 5;
  if (blk >= nb) return;
  const void* src = which ? p.v : p.k;
  const uint64_t so = (uint64_t)col * (which ? p.v_col_stride : p.k_col_stride) + (uint64_t)blk * 32;
  float x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = (which ? p.v_f16 : p.k_f16) ? __half2float(reinterpret_cast<const __half*>(src)[so + i]) : reinterpret_cast<const float*>(src)[so + i];
  float a = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) a = fmaxf(a, fabsf(x[i]));
  const float sc = __fdiv_rn(a, 127.0f), inv = sc > 0.f ? __fdiv_rn(1.0f, sc) : 0.f;
  const uint64_t row = p.cache_row0 + col;
  (which ? p.vs : p.ks)[row * nb + blk] = sc;
  uint32_t* dst = reinterpret_cast<uint32_t*>((which ? p.v8 : p.k8) + row * p.kv_dim + (uint64_t)blk * 32);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t w = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int q = (int)fminf(fmaxf(rintf(__fmul_rn(x[4 * j + b], inv)), -127.0f), 127.0f);
      w |= ((uint32_t)q & 255u) << (8 * b);
    }
    dst[j] = w;
  }
}

// f32 cache rows: a copy (f16 activations widen exactly)
__global__ void __launch_bounds__(256) pa_kv_store_f32_kernel(const KvStoreParams p) {
  pdl_wait();
  pdl_trigger();
  const uint32_t col = blockIdx.y;
  const uint64_t row = p.cache_row0 + col;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < p.kv_dim; i += gridDim.x * blockDim.x) {
    const uint64_t ko = (uint64_t)col * p.k_col_stride + i, vo = (uint64_t)col * p.v_col_stride + i;
    p.k32[row * p.kv_dim + i] = p.k_f16 ? __half2float(reinterpret_cast<const __half*>(p.k)[ko]) : reinterpret_cast<const float*>(p.k)[ko];
    p.v32[row * p.kv_dim + i] = p.v_f16 ? __half2float(reinterpret_cast<const __half*>(p.v)[vo]) : reinterpret_cast<const float*>(p.v)[vo];
  }
}

cudaError_t launch_kv_store(const KvStoreParams& p, uint32_t n_cols, cudaStream_t st) {
  if (p.format == PA_KV_Q8) return launch_pdl(pa_kv_store_q8_kernel, dim3((p.kv_dim / 32 + 31) / 32, n_cols), dim3(64), 0, st, p);
  return launch_pdl(pa_kv_store_f32_kernel, dim3((p.kv_dim + 255) / 256, n_cols), dim3(256), 0, st, p);
}

// ---- split-K decode / verify / prefill over an f32 cache -----------------------------------------------

constexpr int kAnyChunk = 64;     // positions per chunk
constexpr int kAnyThreads = 256;
constexpr int kAnyMaxG = 16;      // query heads per kv head

// grid (splits, kv heads, columns of one item).  Dynamic shared memory: q [G][hd] f32, then the chunk's scores /
// weights [G][64], then m, l, alpha [G] each, then the values phase's partial sums.
__global__ void __launch_bounds__(kAnyThreads) pa_decode_f32_any_kernel(const AnyDecodeParams p) {
  extern __shared__ float sm[];
  const uint32_t hd = p.hd, G = p.G, split = blockIdx.x, g = blockIdx.y, c = blockIdx.z;
  float* q_s = sm;                               // [G][hd]
  float* s_s = q_s + G * hd;                     // [G][64]
  float* s_m = s_s + G * kAnyChunk;              // [G]
  float* s_l = s_m + G;
  float* s_a = s_l + G;
  float* s_red = sm + ((G * hd + G * kAnyChunk + 3 * G + 3) & ~3u);   // [position groups][G][hd] at the end (16-byte aligned)
  const int tid = threadIdx.x, lane = tid & 31;
  // rows this column sees, and this split's range of them (the plan is the item's: its last column's rows)
  const uint32_t lim = (uint32_t)min(max(p.lim0 + (int32_t)c, 0), (int32_t)p.n_rows);
  const uint32_t tiles = (p.n_rows + kAnyChunk - 1) / kAnyChunk;
  const uint32_t tps = p.tps, t0 = split * tps * kAnyChunk, t1 = min(min(tiles, (split + 1) * tps) * kAnyChunk, lim);
  if (split * tps >= tiles) return;              // no record expected from this split
  pdl_wait();
  pdl_trigger();
  const uint64_t col = p.col0 + c;
  for (uint32_t i = tid; i < G * hd; i += kAnyThreads) {
    const uint64_t off = col * p.q_col_stride + (uint64_t)(g * G + i / hd) * p.q_head_stride + i % hd;
    q_s[i] = p.q_f16 ? __half2float(reinterpret_cast<const __half*>(p.q)[off]) : reinterpret_cast<const float*>(p.q)[off];
  }
  if ((uint32_t)tid < G) { s_m[tid] = -3.0e38f; s_l[tid] = 0.f; }
  // values phase: thread = (group of positions pg, four dims dq)
  const uint32_t quads = hd / 4, n_pg = kAnyThreads / quads, dq = tid % quads, pg = tid / quads;
  float acc[kAnyMaxG][4];
#pragma unroll
  for (int h = 0; h < kAnyMaxG; ++h) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f;
  const float rs = sqrtf((float)hd);
  const uint64_t row0 = (uint64_t)p.seq * p.max_seq;
  __syncthreads();
  for (uint32_t c0 = t0; c0 < t1; c0 += kAnyChunk) {
    const uint32_t n = min((uint32_t)kAnyChunk, t1 - c0);
    // ---- scores: thread (r, part) takes a quarter of row r for all G heads; the four parts are summed in lane order ----
    {
      const uint32_t r = tid >> 2, part = tid & 3, span = hd / 4;
      float s[kAnyMaxG];
#pragma unroll
      for (int h = 0; h < kAnyMaxG; ++h) s[h] = 0.f;
      if (r < n) {
        const float4* src = reinterpret_cast<const float4*>(p.k + (row0 + c0 + r) * p.kv_dim + g * hd + part * span);
        for (uint32_t i = 0; i < span; i += 4) {
          const float4 x = src[i / 4];
#pragma unroll
          for (int h = 0; h < kAnyMaxG; ++h) {
            if ((uint32_t)h >= G) break;
            const float* qp = q_s + h * hd + part * span + i;
            s[h] = __fmaf_rn(qp[3], x.w, __fmaf_rn(qp[2], x.z, __fmaf_rn(qp[1], x.y, __fmaf_rn(qp[0], x.x, s[h]))));
          }
        }
      }
#pragma unroll
      for (int h = 0; h < kAnyMaxG; ++h) {
        if ((uint32_t)h >= G) break;
        float v = s[h];
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (part == 0) s_s[h * kAnyChunk + r] = r < n ? v / rs : -INFINITY;
      }
    }
    __syncthreads();
    // ---- online softmax: warp w takes heads w, w + 8 ----
    for (uint32_t h = tid >> 5; h < G; h += kAnyThreads / 32) {
      const float a = s_s[h * kAnyChunk + lane], b = s_s[h * kAnyChunk + 32 + lane];
      float mx = fmaxf(a, b);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_old = s_m[h], m_new = fmaxf(m_old, mx);
      const float ea = expf(a - m_new), eb = expf(b - m_new);      // exp(-inf) = 0 for rows past the chunk's end
      s_s[h * kAnyChunk + lane] = ea; s_s[h * kAnyChunk + 32 + lane] = eb;
      float sum = ea + eb;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) {
        const float alpha = expf(m_old - m_new);
        s_m[h] = m_new; s_l[h] = s_l[h] * alpha + sum; s_a[h] = alpha;
      }
    }
    __syncthreads();
    // ---- values ----
#pragma unroll
    for (int h = 0; h < kAnyMaxG; ++h) {
      if ((uint32_t)h >= G) break;
      const float a = s_a[h];
      acc[h][0] *= a; acc[h][1] *= a; acc[h][2] *= a; acc[h][3] *= a;
    }
    for (uint32_t t = pg; t < n; t += n_pg) {
      const float4 v = *reinterpret_cast<const float4*>(p.v + (row0 + c0 + t) * p.kv_dim + g * hd + dq * 4);
#pragma unroll
      for (int h = 0; h < kAnyMaxG; ++h) {
        if ((uint32_t)h >= G) break;
        const float w = s_s[h * kAnyChunk + t];
        acc[h][0] = __fmaf_rn(w, v.x, acc[h][0]); acc[h][1] = __fmaf_rn(w, v.y, acc[h][1]);
        acc[h][2] = __fmaf_rn(w, v.z, acc[h][2]); acc[h][3] = __fmaf_rn(w, v.w, acc[h][3]);
      }
    }
    __syncthreads();
  }
  // ---- the position groups' sums, added in group order; one record per (row, split) ----
#pragma unroll
  for (int h = 0; h < kAnyMaxG; ++h) {
    if ((uint32_t)h >= G) break;
    *reinterpret_cast<float4*>(s_red + ((size_t)pg * G + h) * hd + dq * 4) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
  }
  __syncthreads();
  for (uint32_t i = tid; i < G * hd; i += kAnyThreads) {
    const uint32_t h = i / hd, d = i % hd;
    float o = s_red[(size_t)h * hd + d];
    for (uint32_t k = 1; k < n_pg; ++k) o += s_red[((size_t)k * G + h) * hd + d];
    const uint64_t prow = col * p.n_heads + g * G + h;
    p.part_o[(prow * p.n_splits + split) * hd + d] = o;
  }
  if ((uint32_t)tid < G) {
    const uint64_t prow = col * p.n_heads + g * G + tid;
    p.part_ml[(prow * p.n_splits + split) * 2] = s_m[tid];
    p.part_ml[(prow * p.n_splits + split) * 2 + 1] = s_l[tid];
  }
}

size_t any_decode_smem(uint32_t G, uint32_t hd) {
  const size_t n_pg = kAnyThreads / (hd / 4);
  return ((((size_t)G * hd + (size_t)G * kAnyChunk + 3 * G + 3) & ~(size_t)3) + n_pg * G * hd) * sizeof(float);
}

// The same for 1, 2 or 4 heads per kv head (the dense engine's models have 2), straight from memory to registers: HD / 16
// lanes share a row, 16 dims each, so a warp instruction reads whole rows, and a warp requests the K and the V of 16 (head_dim
// 64: 32, 256: 8; with four heads half of that) rows together, 128 registers a thread, before it uses the first: 128 KB
// in flight per SM, which is what HBM's latency takes at full rate.  No barrier and no shared memory until the warps' (o, m, l) are merged at the end.  A CTA's
// rows are one or two such batches per warp at the contexts these caches serve.  28 layers of a token over 2000 rows (16 q / 8 kv
// heads x 128), whole calls: 644 us with the chunked kernel above and a front kernel, 257 us with this one, a front and a merge
// kernel, 218 us with the front in this one, 199 us with the merge in it too (floor 70: 459 MB).
//
// FU: one token whose front the kernel makes itself, as pa_decode_kernel does: the 256 threads rotate the G query rows (rot_exact,
// host cos / sin) into shared memory; the CTA of the sequence's last rows also rotates k, stores the row, and takes it from shared
// memory, not from the cache, into its own sums.  As a kernel of its own ahead of this one the front was 3 us of a layer's 9.2.
constexpr int f32_batch(int hd, int G) { return 512 / hd * (G == 4 ? 2 : 4); }
template <int HD, int G, bool FU>
__global__ void __launch_bounds__(256, 1) pa_decode_f32_kernel(const F32DecodeParams p) {
  constexpr int LPR = HD / 16, RPI = 32 / LPR, BATCH = f32_batch(HD, G), U = BATCH / RPI;   // lanes per row, rows per instruction and per batch
  extern __shared__ float sm[];                                             // [8 warps][G][HD], then m[8][G], l[8][G]
  const uint32_t split = blockIdx.x, g = blockIdx.y, c = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane / LPR, lr = lane % LPR;
  const uint32_t lim = (uint32_t)min(max(p.lim0 + (int32_t)c, 0), (int32_t)p.n_rows);
  const uint32_t r_lo = split * p.rows_per_split, r_hi = min(r_lo + p.rows_per_split, lim);
  if (split >= p.n_splits) return;                                          // (a cluster's size is a power of two)
  const uint64_t base = ((uint64_t)p.seq * p.max_seq) * p.kv_dim + (uint64_t)g * HD + lr * 4;
  float4 k[U][4], v[U][4];
  auto load = [&](uint32_t b0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t row = b0 + u * RPI + sub;
      const float* kp = p.k + base + (uint64_t)row * p.kv_dim;
      const float* vp = p.v + base + (uint64_t)row * p.kv_dim;
#pragma unroll
      for (int i = 0; i < 4; ++i) k[u][i] = row < r_hi ? __ldcg(reinterpret_cast<const float4*>(kp + i * LPR * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[u][i] = row < r_hi ? __ldcg(reinterpret_cast<const float4*>(vp + i * LPR * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  uint32_t b0 = r_lo + warp * BATCH;
  // rows the kernel before this one does not write may be fetched while it runs
  const bool ahead = p.early && b0 + BATCH <= min(p.n_rows - min(p.n_rows, p.n_cols), FU ? p.early_limit : 0xffffffffu);
  if (ahead && b0 < r_hi) load(b0);
  __shared__ Angle s_ang[FU ? 64 : 1];
  __shared__ __align__(16) float s_new[FU ? G + 2 : 1][HD];     // the rotated query rows, the token's own k and v
  if constexpr (FU) {      // (launch parameters indexed per thread are served one address at a time: staged while the predecessor runs)
    if ((uint32_t)tid < 2 * p.half) reinterpret_cast<uint4*>(s_ang)[tid] = reinterpret_cast<const uint4*>(p.ang)[tid];
    __syncthreads();
  }
  pdl_wait();
  pdl_trigger();
  const bool own = FU && r_hi == p.n_rows && r_lo < r_hi;
  if constexpr (FU) {
    constexpr uint32_t P = HD / 2, TURNS = ((G + 2) * P + 255) / 256;
    const uint32_t n_it = (own ? G + 2 : G) * P;
    float a[TURNS], b[TURNS];
    auto dims = [&](uint32_t pr, uint32_t& d0, uint32_t& d1) { d0 = pr < p.half ? pr : 2 * pr; d1 = pr < p.half ? pr + p.half : d0 + 1; };
#pragma unroll
    for (uint32_t t = 0; t < TURNS; ++t) {
      const uint32_t it = tid + 256 * t, hh = it / P;
      if (it >= n_it) continue;
      uint32_t d0, d1;
      dims(it % P, d0, d1);
      const void* src = hh < G ? p.q : hh == G ? p.k_new : p.v_new;
      const uint64_t so = hh < G ? (uint64_t)(g * G + hh) * p.q_head_stride : (uint64_t)g * HD;
      a[t] = ld_act(src, so + d0, p.q_f16); b[t] = ld_act(src, so + d1, p.q_f16);
    }
    if (!ahead && b0 < r_hi) load(b0);
#pragma unroll
    for (uint32_t t = 0; t < TURNS; ++t) {
      const uint32_t it = tid + 256 * t, hh = it / P, pr = it % P;
      if (it >= n_it) continue;
      uint32_t d0, d1;
      dims(pr, d0, d1);
      float x = a[t], y = b[t];
      if (hh <= G && pr < p.half) { x = rot_exact(a[t], b[t], s_ang[pr], true); y = rot_exact(b[t], a[t], s_ang[pr], false); }
      s_new[hh][d0] = x; s_new[hh][d1] = y;
      if (hh >= G) {
        float* dst = const_cast<float*>(hh == G ? p.k : p.v) + ((uint64_t)p.seq * p.max_seq + p.n_rows - 1) * p.kv_dim + (uint64_t)g * HD;
        dst[d0] = x; dst[d1] = y;
      }
    }
    __syncthreads();
  } else if (!ahead && b0 < r_hi) load(b0);
  const uint64_t col = c;
  float4 q[G][4];
#pragma unroll
  for (int h = 0; h < G; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t off = col * p.q_col_stride + (uint64_t)(g * G + h) * p.q_head_stride + i * LPR * 4 + lr * 4;
      if constexpr (FU) q[h][i] = *reinterpret_cast<const float4*>(&s_new[h][i * LPR * 4 + lr * 4]);
      else if (p.q_vec) q[h][i] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.q) + off);
      else q[h][i] = make_float4(ld_act(p.q, off, p.q_f16), ld_act(p.q, off + 1, p.q_f16), ld_act(p.q, off + 2, p.q_f16), ld_act(p.q, off + 3, p.q_f16));
    }
  float m[G], l[G];
  float4 o[G][4];
#pragma unroll
  for (int h = 0; h < G; ++h) {
    m[h] = -FLT_MAX; l[h] = 0.f;      // m in units of q . k : no finite score lies below its start
#pragma unroll
    for (int i = 0; i < 4; ++i) o[h][i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  while (b0 < r_hi) {
    if (FU && own) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b0 + u * RPI + sub == p.n_rows - 1) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            k[u][i] = *reinterpret_cast<const float4*>(&s_new[FU ? G : 0][i * LPR * 4 + lr * 4]);
            v[u][i] = *reinterpret_cast<const float4*>(&s_new[FU ? G + 1 : 0][i * LPR * 4 + lr * 4]);
          }
        }
    }
#pragma unroll
    for (int h = 0; h < G; ++h) {
      float s[U], mx = m[h];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float a = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          a = __fmaf_rn(q[h][i].w, k[u][i].w, __fmaf_rn(q[h][i].z, k[u][i].z, __fmaf_rn(q[h][i].y, k[u][i].y, __fmaf_rn(q[h][i].x, k[u][i].x, a))));
#pragma unroll
        for (int x = LPR / 2; x > 0; x >>= 1) a += __shfl_xor_sync(0xffffffffu, a, x);
        s[u] = b0 + u * RPI + sub < r_hi ? a : -INFINITY;
        mx = fmaxf(mx, s[u]);
      }
#pragma unroll
      for (int x = LPR; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float al = exp2f((m[h] - mx) * p.scale_log2);
      m[h] = mx; l[h] *= al;
#pragma unroll
      for (int i = 0; i < 4; ++i) { o[h][i].x *= al; o[h][i].y *= al; o[h][i].z *= al; o[h][i].w *= al; }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float w = exp2f((s[u] - mx) * p.scale_log2);
        l[h] += w;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o[h][i].x = __fmaf_rn(w, v[u][i].x, o[h][i].x); o[h][i].y = __fmaf_rn(w, v[u][i].y, o[h][i].y);
          o[h][i].z = __fmaf_rn(w, v[u][i].z, o[h][i].z); o[h][i].w = __fmaf_rn(w, v[u][i].w, o[h][i].w);
        }
      }
    }
    b0 += 8 * BATCH;
    if (b0 < r_hi) load(b0);
  }
  // ---- the row groups of a warp, then the warps ----
  float* so = sm + warp * G * HD;
  float* sml = sm + 8 * G * HD;
#pragma unroll
  for (int h = 0; h < G; ++h) {
#pragma unroll
    for (int x = LPR; x < 32; x <<= 1) {
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[h][i].x += __shfl_xor_sync(0xffffffffu, o[h][i].x, x); o[h][i].y += __shfl_xor_sync(0xffffffffu, o[h][i].y, x);
        o[h][i].z += __shfl_xor_sync(0xffffffffu, o[h][i].z, x); o[h][i].w += __shfl_xor_sync(0xffffffffu, o[h][i].w, x);
      }
    }
    if (sub == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(so + h * HD + i * LPR * 4 + lr * 4) = o[h][i];
    }
    if (lane == 0) { sml[warp * G + h] = m[h]; sml[8 * G + warp * G + h] = l[h]; }
  }
  __syncthreads();
  const bool keep = p.cluster || p.merge_rec;      // behind the warps' shares
  for (uint32_t idx = tid; idx < G * HD; idx += 256) {
    const uint32_t h = idx / HD, d = idx % HD;
    float M = sml[h], L = 0.f, a = 0.f;
#pragma unroll
    for (int w = 1; w < 8; ++w) M = fmaxf(M, sml[w * G + h]);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float e = exp2f((sml[w * G + h] - M) * p.scale_log2);
      L = __fmaf_rn(sml[8 * G + w * G + h], e, L);
      a = __fmaf_rn(sm[w * G * HD + idx], e, a);
    }
    if (keep) {
      float* mine = sm + 8 * G * (HD + 2);
      mine[idx] = a;
      if (d == 0) { mine[G * HD + 2 * h] = M; mine[G * HD + 2 * h + 1] = L; }
      continue;
    }
    const uint64_t slot = (col * p.n_heads + g * G + h) * p.n_splits + split;
    p.part_o[slot * HD + d] = a;
    if (d == 0) { p.part_ml[slot * 2] = M * inv_sqrt_hd<HD>(); p.part_ml[slot * 2 + 1] = L; }
  }
  if (p.merge_rec) {
    // one wave of CTAs: those of a (kv head, column) leave their records for one another (see kNoWord) and share out the merge.  Nobody
    // has to wait for a CTA that found no SM, beside another stream's kernels: a unit whose records are not there in time is left to the
    // CTA that comes last, for which all of them are.  ctr[0]: CTAs that have come (back at zero with the last), ctr[1]: units left.  Who leaves
    // one looks for the last one afterwards, and the last one for what was left, with a fence between, so at least one of the two sees the
    // other, and the atomics on ctr[1] give a unit to one of them.  (28 layers of a token over 2000 rows: 197 us with waits alone, 192 so.)
    __shared__ uint32_t s_err, s_take;
    if (tid == 0) s_err = 0;
    __syncthreads();
    if (warp >= 4) return;
    constexpr size_t BLK = merge_block(HD, G);
    const float* mine = sm + 8 * G * (HD + 2);
    float* const blk0 = p.merge_rec + ((size_t)c * gridDim.y + g) * p.n_splits * BLK;
    for (uint32_t idx = tid; idx < G * (HD / 4); idx += 128) {
      const uint32_t h = idx / (HD / 4), c4 = idx % (HD / 4);
      put_record4<HD>(blk0 + split * BLK, G, h, c4, *reinterpret_cast<const float4*>(mine + h * HD + c4 * 4), mine[G * HD + 2 * h] * inv_sqrt_hd<HD>(),
                      mine[G * HD + 2 * h + 1]);
    }
    unsigned int* const ctr = p.merge_ctr + 2 * (c * gridDim.y + g);
    uint32_t come = 0;
    if (tid == 0) come = atomicInc(ctr, p.n_splits - 1);
    named_bar_sync(1, 128);                        // the scratch takes the place of the warps' shares, which nobody reads any more
    constexpr uint32_t UNITS = G * (HD / 64);
    static_assert(UNITS <= 32, "units left are bits of a word");
    auto unit = [&](uint32_t u, uint32_t polls) {
      const uint32_t row = u / (HD / 64), slice = u % (HD / 64), h = g * G + row;
      const float gv = p.gate && tid < 64 ? ld_act(p.gate, col * p.gate_col_stride + (uint64_t)h * p.gate_head_stride + slice * 64 + tid, p.act_f16) : 0.f;
      return merge_slice_128<HD, true>(blk0 + row * HD + slice * 64, blk0 + G * HD + (row * (HD / 64) + slice) * 2, BLK, p.n_splits, tid, *reinterpret_cast<MergeScratch*>(sm), 1,
                                 p.gate != nullptr, gv, false, p.act_f16, p.out, col * p.out_col_stride + (uint64_t)h * HD + slice * 64, polls, &s_err);
    };
    uint32_t left = 0;
    for (uint32_t u = split; u < UNITS; u += p.n_splits) if (!unit(u, p.merge_polls)) left |= 1u << u;
    if (tid == 0) {
      uint32_t take = 0;
      if (come == p.n_splits - 1) {
        __threadfence();
        take = atomicExch(ctr + 1, 0u) | left;
      } else if (left) {
        atomicOr(ctr + 1, left);
        __threadfence();
        if (*reinterpret_cast<volatile unsigned int*>(ctr) == 0) take = atomicAnd(ctr + 1, ~left) & left;
      }
      s_take = take;
    }
    named_bar_sync(1, 128);
    for (uint32_t take = s_take; take; take &= take - 1)
      if (!unit(__ffs(take) - 1, kMergePolls) && tid == 0) s_err = WAIT_MERGE;
    if (tid == 0 && s_err) atomicMax(p.err, s_err);
    return;
  }
  if (!p.cluster) return;
  // at most eight splits: the CTAs of a (kv head, column) are a cluster and merge without another launch
  cluster_sync();
  const uint32_t mine_s = smem_u32(sm + 8 * G * (HD + 2));
  for (uint32_t idx = split * 256 + tid; idx < G * (HD / 4); idx += p.n_splits * 256) {
    const uint32_t h = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
    float L;
    const float4 o4 = cluster_merge4(mine_s + (h * HD + d) * 4, mine_s + (G * HD + 2 * h) * 4, p.n_splits, p.scale_log2, L);
    gate_store4(o4, L, p.gate, col * p.gate_col_stride + (uint64_t)(g * G + h) * p.gate_head_stride + d, p.out,
                col * p.out_col_stride + (uint64_t)(g * G + h) * HD + d, p.act_f16);
  }
  cluster_sync();            // no CTA leaves while another reads its rows
}

template <int HD, int G, bool FU>
static cudaError_t launch_f32_fu(const F32DecodeParams& p, dim3 grid, cudaStream_t st) {
  const size_t smem = std::max((size_t)(9 * G * (HD + 2)) * 4, sizeof(MergeScratch));       // (at most 37 KB)
  if (p.cluster) return launch_pdl_cluster(pa_decode_f32_kernel<HD, G, FU>, grid, dim3(256), smem, st, p.cluster, p);
  return launch_pdl(pa_decode_f32_kernel<HD, G, FU>, grid, dim3(256), smem, st, p);
}
template <int HD, int G>
static cudaError_t launch_f32_t(const F32DecodeParams& p, dim3 grid, cudaStream_t st) {
  return p.k_new ? launch_f32_fu<HD, G, true>(p, grid, st) : launch_f32_fu<HD, G, false>(p, grid, st);
}
bool decode_f32_direct(uint32_t G) { return G == 1 || G == 2 || G == 4; }
uint32_t decode_f32_batch(uint32_t hd, uint32_t G) { return (uint32_t)f32_batch((int)hd, (int)G); }
cudaError_t launch_decode_f32_direct(const F32DecodeParams& p, uint32_t hd, uint32_t G, uint32_t n_kv, cudaStream_t st) {
  const dim3 grid(p.cluster ? p.cluster : p.n_splits, n_kv, p.n_cols);
#define PA_F32_CASE(H) case H: return G == 1 ? launch_f32_t<H, 1>(p, grid, st) : G == 2 ? launch_f32_t<H, 2>(p, grid, st) : launch_f32_t<H, 4>(p, grid, st);
  switch (hd) {
    PA_F32_CASE(256) PA_F32_CASE(128) PA_F32_CASE(64)
    default: return cudaErrorInvalidValue;
  }
#undef PA_F32_CASE
}

cudaError_t launch_decode_f32(const AnyDecodeParams& p, dim3 grid, int dev, cudaStream_t st) {
  const size_t smem = any_decode_smem(p.G, p.hd);
  static bool attr_set[64] = {};
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(pa_decode_f32_any_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    attr_set[dev & 63] = true;
  }
  return launch_pdl(pa_decode_f32_any_kernel, grid, dim3(kAnyThreads), smem, st, p);
}

}  // namespace pa
