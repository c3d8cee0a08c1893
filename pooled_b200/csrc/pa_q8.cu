// Attention over an int8 KV cache (one f32 scale per 32 values) on the tensor cores: decode, blocks and prompts.
//
// The int8 values are exact in f16, so they enter mma.sync m16n8k16 unscaled and the scales are applied in f32 around it:
//   scores   S[row, pos] = sum over 32-dim blocks b of ks[pos][b] * (q . k8)_b : a fresh accumulator per block, scaled
//            and added in f32.  A (16 rows) holds q of eight query rows twice, the f16 high parts in rows 0-7 and the low
//            parts in rows 8-15, B the int8 rows: both halves of the product come from one instruction.
//   values   O^T[dim, row] += v8^T[dim, pos] . (P * vs)^T[pos, row] : the weights take each block's scale before they are
//            split into high and low f16 parts.
// q is first scaled by a power of two per row and 32-dim block so that its largest value lies in [2^12, 2^13) (one for the
// whole row left outputs off by 3e-6 where a block lay 2^-20 below the others, against keys as much larger), P * vs by one per row, block
// and step of 16 positions so that its largest lies in [2^13, 2^14) : high + low are then within 2^-23 of that value and
// within 2^-38 of it of every smaller one (an unscaled P * vs of 1e-4 would sit among f16's subnormals).  The power is a row's
// and a block's own, and positions a row does not see are not in it: with one for all rows and dims of a warp, a large V scale
// anywhere took bits from everything else (a block at 2^-20 of its neighbours was off by 9e-6 of itself, now 3e-7 as with f32
// operands), and an infinite one of a later column made NaN of earlier ones.  It takes 4 shuffles and some 30
// instructions per pair of blocks and step, q's 32 multiplications: 181 us where one power each took 174 (the token below), 348
// where 319 (the prompt, each warp then converting for itself).
//
// A warp owns eight query rows (heads of the GQA group, columns) and runs an online softmax over the positions it takes,
// P in registers from one product to the next; no barrier but the ring's.  A CTA is four or eight warps over a ring of 64-position
// tiles (cp.async): with few query rows the warps share the positions of a tile and merge their (o, m, l)
// at the end, with many each has rows of its own and all positions.  Eight warps fit an SM.
// What bounds it: the latency of two warps per scheduler.  Four warps: each executes some 1400 instructions per 16 positions and eight rows
// (loading its share of the tiles included) against 64 MMAs, most of them conversions, which it makes for its eight rows alone (int8 ->
// f16 costs a byte permute and an f16 subtraction per two values): issue slots 30 %, ALU 25 %, tensor pipe 7 %, HBM 11 % of the active cycles
// of the token below.  Eight warps that share a conversion: some 1000 instructions; issue slots 37 %, ALU 23 %, tensor pipe 19 %, shared
// memory 48 % of those of the prompt below.
// Measured with its front (pa_front.cu) against plain f32 loops, a CTA per column: ten layers of a token over 12345 rows (16 q / 2 kv
// heads x 256, head-norm) 918 -> 181 us, two layers of a 777-token prompt (24 / 4 x 256) 4231 -> 322 us; distance from float64
// no larger: 2.2e-7 against 3.1e-7 (a token over 20000 rows), 1.6e-7 against 2.0e-7 (that prompt), relative.
//
// Stands in for attn_flash_q8 of pooled (engine/wgsl/qwen35.js:946-1010 and its column-wise use in prefill).
#include "pa_params.cuh"

namespace pa {

constexpr int kQ8Tile = 64;

// CV: the CTA converts a tile once, to f16 in shared memory, for all of its warps (see the kernel)
template <int HD, bool CV>
struct Q8Smem {
  static constexpr int NW = CV ? 8 : 4, THREADS = 32 * NW;
  static constexpr int NB = HD / 32;                       // scale blocks per row of a kv head
  static constexpr int KB = kQ8Tile * HD, SB = kQ8Tile * NB * 4;
  // values: K, V (int8); scales: K, V.  CV: two stages of values (a tile is converted while the one before it is used), and
  // four of scales, which are read until the tile's end
  static constexpr int STAGES = CV ? 2 : HD == 256 ? 3 : 4, SC_STAGES = CV ? 4 : STAGES;
  static constexpr int F16 = CV ? 2 * 2 * KB * 2 : 0;      // two tiles of K and V as f16, ahead of the rings
  // (a stage's scales lie behind its values, or, CV, in a ring of their own)
  static constexpr int STAGE = CV ? 2 * KB : 2 * KB + 2 * SB, SC_STAGE = CV ? 2 * SB : STAGE;
  static constexpr int OFF_RAW = F16, OFF_SC = CV ? OFF_RAW + STAGES * STAGE : OFF_RAW + 2 * KB;
  static constexpr int RING = OFF_RAW + STAGES * STAGE + (CV ? SC_STAGES * SC_STAGE : 0);
  static constexpr int MROWS = 8 * NW;                     // most query rows of a CTA
  static constexpr int MERGE = MROWS * (HD + 2) * 4;       // the warps' (o, m, l), over the idle ring
  static constexpr int MINE = MROWS * (HD + 2) * 4;        // the CTA's merged rows behind them, for the cluster's merge
  static constexpr int TOTAL = RING > MERGE + MINE ? RING : MERGE + MINE;
};

// 16-byte chunk c of row r, permuted so that the reads below hit 32 different banks: the score reads take four rows r ..
// r + 3 at a time (8 bytes per lane), the value reads rows r, r + 2, r + 4, r + 6 (4 bytes per lane)
// (CV: the conversion reads one chunk of eight neighbouring rows at a time)
template <int HD> __device__ __forceinline__ uint32_t q8_cv_off(uint32_t r, uint32_t c) {
  return HD == 64 ? r * HD + ((c ^ ((r >> 1) & 3u)) << 4) : r * HD + ((c ^ (r & 7u)) << 4);
}
// 16-byte chunk c (eight values) of row r of an f16 tile: eight neighbouring rows of a chunk hit different banks
template <int HD> __device__ __forceinline__ uint32_t q8_h_off(uint32_t r, uint32_t c) { return r * (HD * 2) + ((c ^ (r & 7u)) << 4); }
template <int HD> __device__ __forceinline__ uint32_t q8_k_off(uint32_t r, uint32_t c) {
  if (HD == 64) return r * HD + ((c ^ ((r >> 1) & 3u)) << 4);
  return r * HD + ((c ^ (((r & 3u) << 1) | ((r >> 2) & 1u))) << 4);
}
template <int HD> __device__ __forceinline__ uint32_t q8_v_off(uint32_t r, uint32_t c) {
  if (HD == 64) return r * HD + ((c ^ ((r >> 1) & 3u)) << 4);
  return r * HD + ((c ^ (r & 7u)) << 4);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// bytes (as v + 128) two at a time to f16: 0x6400 | u is 1024 + u, minus 1152 is v
__device__ __forceinline__ uint32_t u8_h2(uint32_t w, uint32_t sel) {
  const uint32_t x = prmt(w, 0x64646464u, sel);
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&x), __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void split_h2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 b = __half22float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_h2(x - b.x, y - b.y);
}
// a low part is at most 4 here; that of an infinity would be inf - inf (min takes the number)
__device__ __forceinline__ uint32_t h2_min8(uint32_t x) {
  const __half2 r = __hmin2(*reinterpret_cast<const __half2*>(&x), __half2half2(__ushort_as_half(0x4800)));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp8(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(live ? 8 : 0) : "memory");
}

// grid (splits, kv heads, row tiles).  rgw row groups per CTA (of NW warps): warp w has row group w % rgw and takes the
// 16-position steps w / rgw, w / rgw + NW / rgw, ... of a tile.
//
// CV, for more than 16 query rows where it is the faster form (q8_plan): eight warps, and each tile is converted to f16 once for all of them instead of by every
// warp for its own eight rows, then read with ldmatrix: two layers of the 777-token prompt below 350 -> 322 us.
// K's values go to the places the other form's lanes take them from (a score's products meet in the same order) and V's
// stay in theirs, so both forms give the same bits for the same split plan.
template <int HD, bool CV>
__global__ void __launch_bounds__((Q8Smem<HD, CV>::THREADS), CV && HD >= 128 ? 1 : 2) pa_q8_kernel(const Q8Params p) {
  using L = Q8Smem<HD, CV>;
  constexpr int NB = L::NB, NW = L::NW, kQ8Threads = L::THREADS;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sm0 = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, j = lane & 3;
  const uint32_t split = blockIdx.x, g = blockIdx.y, G = p.G, RT = 8 * p.rgw;
  const uint32_t row0 = (gridDim.z - 1 - blockIdx.z) * RT, rows = p.n_cols * G;    // the longest rows first
  const uint32_t rg = warp % p.rgw, pw = warp / p.rgw, n_pw = NW / p.rgw;
  // the plan is the call's (its last column's rows); a row tile stops at what its own last row sees
  const uint32_t tiles = (p.n_rows + kQ8Tile - 1) / kQ8Tile;
  const uint32_t ns_eff = min(p.n_splits, plan_cap(tiles)), tps = (tiles + ns_eff - 1) / max(ns_eff, 1u);
  const uint32_t t_lo = split * tps;
  if (t_lo >= tiles) return;                                  // no record expected from this split
  auto row_lim = [&](uint32_t row) { return (uint32_t)min(max(p.lim0 + (int32_t)(min(row, rows - 1) / G), 0), (int32_t)p.n_rows); };
  const uint32_t t_hi = min(min(tiles, t_lo + tps), (row_lim(row0 + RT - 1) + kQ8Tile - 1) / kQ8Tile);
  const uint32_t n_tiles = t_hi > t_lo ? t_hi - t_lo : 0;
  const uint64_t seq_row0 = (uint64_t)p.seq * p.max_seq;
  const uint32_t kv_dim = p.kv_dim, nbk = kv_dim / 32;

  auto load_tile = [&](uint32_t t) {      // one commit group per call, empty past the range
    if (t < n_tiles) {
      const uint32_t pos0 = (t_lo + t) * kQ8Tile, base = sm0 + L::OFF_RAW + (t % L::STAGES) * L::STAGE,
                     sbase = CV ? sm0 + L::OFF_SC + (t % L::SC_STAGES) * L::SC_STAGE : base + 2 * L::KB;
      constexpr int CPR = HD / 16;
#pragma unroll
      for (int it = 0; it < kQ8Tile * CPR / kQ8Threads; ++it) {
        const uint32_t idx = tid + it * kQ8Threads, rr = idx / CPR, c = idx % CPR;
        const bool live = pos0 + rr < p.n_rows;
        const uint64_t off = (seq_row0 + (live ? pos0 + rr : 0)) * kv_dim + (uint64_t)g * HD + c * 16;
        cp16(base + (CV ? q8_cv_off<HD>(rr, c) : q8_k_off<HD>(rr, c)), p.k + off, live);
        cp16(base + L::KB + (CV ? q8_cv_off<HD>(rr, c) : q8_v_off<HD>(rr, c)), p.v + off, live);
      }
      if (HD >= 128) {
        constexpr int SC = NB >= 4 ? NB / 4 : 1;
        for (uint32_t idx = tid; idx < kQ8Tile * SC; idx += kQ8Threads) {
          const uint32_t rr = idx / SC, c = idx % SC;
          const bool live = pos0 + rr < p.n_rows;
          const uint64_t off = (seq_row0 + (live ? pos0 + rr : 0)) * nbk + g * NB + c * 4;
          cp16(sbase + rr * (NB * 4) + c * 16, p.ks + off, live);
          cp16(sbase + L::SB + rr * (NB * 4) + c * 16, p.vs + off, live);
        }
      } else if (tid < kQ8Tile) {
        const bool live = pos0 + tid < p.n_rows;
        const uint64_t off = (seq_row0 + (live ? pos0 + tid : 0)) * nbk + g * NB;
        cp8(sbase + tid * 8, p.ks + off, live);
        cp8(sbase + L::SB + tid * 8, p.vs + off, live);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // tiles of rows that the kernel before this one does not write may be fetched while it runs
  const uint32_t old_rows = p.early ? p.n_rows - min(p.n_rows, p.n_cols) : 0u;
  bool waited = false;
#pragma unroll
  for (int t = 0; t < (CV ? 2 : L::STAGES - 1); ++t) {
    if (!waited && (t_lo + t + 1) * kQ8Tile > old_rows) { pdl_wait(); waited = true; }
    load_tile(t);
  }
  if (!waited) pdl_wait();
  pdl_trigger();

  // ---- this warp's eight query rows: thread (r, j) holds dims 32 b + 8 j .. + 7 of row r, as high and low f16 pairs ----
  const uint32_t my_row = row0 + 8 * rg + r;
  const bool live_row = my_row < rows;
  uint32_t qa[2 * NB][4];
  float q_down[NB];   // back from the blocks' powers of two
  {
    float x[NB][8];
    const uint32_t qc = live_row ? my_row / G : 0, qh = live_row ? my_row % G : 0;
    const uint64_t off = (uint64_t)qc * p.q_col_stride + (uint64_t)(g * G + qh) * p.q_head_stride + 8 * j;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (!live_row) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[b][e] = 0.f;
      } else if (p.q_vec) {
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.q) + off + 32 * b);
        *reinterpret_cast<float4*>(&x[b][0]) = src[0]; *reinterpret_cast<float4*>(&x[b][4]) = src[1];
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[b][e] = ld_act(p.q, off + 32 * b + e, p.q_f16);
      }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float mx = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) mx = fmaxf(mx, fabsf(x[b][e]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      // times 2^(139 - e) with e the largest value's exponent field (at least 20, so that the factor is finite)
      const uint32_t e = min(max(__float_as_uint(mx) >> 23, 20u), 254u);
      const float up = __uint_as_float((266u - e) << 23);
      q_down[b] = __uint_as_float((e - 12u) << 23);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        split_h2(x[b][4 * h] * up, x[b][4 * h + 1] * up, qa[2 * b + h][0], qa[2 * b + h][1]);
        split_h2(x[b][4 * h + 2] * up, x[b][4 * h + 3] * up, qa[2 * b + h][2], qa[2 * b + h][3]);
      }
    }
  }
  const uint32_t lim = live_row ? row_lim(my_row) : 0u;
  const uint32_t warp_lim = row_lim(row0 + 8 * rg + 7);       // no position at or past it concerns this warp
  const uint32_t first_lim = row_lim(row0 + 8 * rg);          // every row of the warp sees the positions below it
  const bool warp_live = row0 + 8 * rg < rows;

  // Sums in two levels, sixteen steps and the whole: one after the other the 1200 additions of a thread over 5000 rows left
  // 4.3e-7 of the result, where f32 loops over shorter runs leave 3.2e-7 (so 2.1e-7).  At head_dim 256 l alone: there is no room
  // for a second o, and l was the larger part (4.4e-7, f32 loops 3.9e-7, so 3.7e-7).  2 us of the prompt above.
  constexpr bool O2 = HD <= 128;
  float m = -FLT_MAX, l = 0.f, lt = 0.f;                      // m in units of q . k : no finite score lies below its start
  float oacc[2 * NB][4], ot[O2 ? 2 * NB : 1][4];
  auto zero = [](auto& o) {
#pragma unroll
    for (auto& x : o) x[0] = x[1] = x[2] = x[3] = 0.f;
  };
  auto flush = [&]() {
    l += lt;
    lt = 0.f;
    if constexpr (O2) {
#pragma unroll
      for (int i = 0; i < 2 * NB; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) oacc[i][k] += ot[i][k];
      zero(ot);
    }
  };
  zero(oacc); zero(ot);
  uint32_t steps = 0;
  // CV: tile t to f16, a (row, block of 32) of K or V per thread and turn
  auto convert = [&](uint32_t t) {
    const uint8_t* raw = smem + L::OFF_RAW + (t & 1) * 2 * L::KB;
    uint8_t* dst = smem + (t & 1) * 4 * L::KB;
#pragma unroll
    for (int it = 0; it < 2 * kQ8Tile * NB / kQ8Threads; ++it) {
      const uint32_t idx = tid + it * kQ8Threads, rr = idx % kQ8Tile, b = (idx / kQ8Tile) % NB, which = idx / (kQ8Tile * NB);
      const uint8_t* src = raw + which * L::KB;
      const uint4 x = *reinterpret_cast<const uint4*>(src + q8_cv_off<HD>(rr, 2 * b)), y = *reinterpret_cast<const uint4*>(src + q8_cv_off<HD>(rr, 2 * b + 1));
      const uint32_t w[8] = {x.x ^ 0x80808080u, x.y ^ 0x80808080u, x.z ^ 0x80808080u, x.w ^ 0x80808080u,
                             y.x ^ 0x80808080u, y.y ^ 0x80808080u, y.z ^ 0x80808080u, y.w ^ 0x80808080u};
      uint8_t* d = dst + which * 2 * L::KB;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // K: chunk (h, half) of a block holds dims 8 j + 4 h + 2 half, + 1 of j = 0 .. 3, the pairs lane j multiplies
        const uint32_t sel = c & 1 ? 0x4342u : 0x4140u;
        const uint4 v = which ? make_uint4(u8_h2(w[2 * c], 0x4140u), u8_h2(w[2 * c], 0x4342u), u8_h2(w[2 * c + 1], 0x4140u), u8_h2(w[2 * c + 1], 0x4342u))
                              : make_uint4(u8_h2(w[c >> 1], sel), u8_h2(w[2 + (c >> 1)], sel), u8_h2(w[4 + (c >> 1)], sel), u8_h2(w[6 + (c >> 1)], sel));
        *reinterpret_cast<uint4*>(d + q8_h_off<HD>(rr, 4 * b + c)) = v;
      }
    }
  };
  if constexpr (CV) {
    if (n_tiles) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      convert(0);
    }
  }

  for (uint32_t t = 0; t < n_tiles; ++t) {
    if constexpr (CV) {
      // tile t + 1 has landed and tile t is converted for every thread; tile t - 1, whose f16 place the next one takes, is consumed
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      load_tile(t + 2);
      if (t + 1 < n_tiles) convert(t + 1);
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(L::STAGES - 2) : "memory");
      __syncthreads();                                        // tile t has landed for every thread, tile t - 1 is consumed
      load_tile(t + L::STAGES - 1);
    }
    if (!warp_live) continue;
    const uint8_t* kt = smem + (CV ? (t & 1) * 4 * L::KB : L::OFF_RAW + (t % L::STAGES) * L::STAGE);
    const uint8_t* vt = kt + (CV ? 2 : 1) * L::KB;
    const float* kst = reinterpret_cast<const float*>(CV ? smem + L::OFF_SC + (t % L::SC_STAGES) * L::SC_STAGE : kt + 2 * L::KB);
    const float* vst = kst + kQ8Tile * NB;
    const uint32_t kt_s = smem_u32(kt), vt_s = smem_u32(vt);
#pragma unroll 1
    for (uint32_t st = pw; st < kQ8Tile / 16; st += n_pw) {
      const uint32_t pos0 = (t_lo + t) * kQ8Tile + 16 * st;
      if (pos0 >= warp_lim) break;
      // ---- scores of 16 positions: two groups of eight ----
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const uint32_t pr = 16 * st + 8 * n;
        float k0[NB], k1[NB];                                  // scales of positions 2 j, 2 j + 1 of the group
#pragma unroll
        for (int b = 0; b < NB; b += (NB >= 4 ? 4 : 2)) {
          if (NB >= 4) {
            *reinterpret_cast<float4*>(&k0[b]) = *reinterpret_cast<const float4*>(kst + (pr + 2 * j) * NB + b);
            *reinterpret_cast<float4*>(&k1[b]) = *reinterpret_cast<const float4*>(kst + (pr + 2 * j + 1) * NB + b);
          } else {
            *reinterpret_cast<float2*>(&k0[b]) = *reinterpret_cast<const float2*>(kst + (pr + 2 * j) * NB + b);
            *reinterpret_cast<float2*>(&k1[b]) = *reinterpret_cast<const float2*>(kst + (pr + 2 * j + 1) * NB + b);
          }
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          uint32_t k8[4];
          if constexpr (CV) {
            ldsm_x4(kt_s + q8_h_off<HD>(pr + (lane & 7), 4 * b + (lane >> 3)), k8[0], k8[1], k8[2], k8[3]);
          } else {
            uint2 w = *reinterpret_cast<const uint2*>(kt + q8_k_off<HD>(pr + r, 2 * b + (j >> 1)) + (j & 1) * 8);
            w.x ^= 0x80808080u; w.y ^= 0x80808080u;
            k8[0] = u8_h2(w.x, 0x4140u); k8[1] = u8_h2(w.x, 0x4342u); k8[2] = u8_h2(w.y, 0x4140u); k8[3] = u8_h2(w.y, 0x4342u);
          }
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          mma_16816(c, qa[2 * b][0], qa[2 * b][1], qa[2 * b][2], qa[2 * b][3], k8[0], k8[1]);
          mma_16816(c, qa[2 * b + 1][0], qa[2 * b + 1][1], qa[2 * b + 1][2], qa[2 * b + 1][3], k8[2], k8[3]);
          s[2 * n] = __fmaf_rn(k0[b] * q_down[b], c[0] + c[2], s[2 * n]);
          s[2 * n + 1] = __fmaf_rn(k1[b] * q_down[b], c[1] + c[3], s[2 * n + 1]);
        }
      }
      // ---- mask, running maximum, weights ----
      float mx = m;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t pos = pos0 + 8 * (e >> 1) + 2 * j + (e & 1);
        s[e] = pos < lim ? s[e] : -INFINITY;
        mx = fmaxf(mx, s[e]);
      }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      if (__any_sync(0xffffffffu, mx > m)) {
        const float al = exp2f((m - mx) * p.scale_log2);
        l *= al; lt *= al;
        m = mx;
        const float a0 = __shfl_sync(0xffffffffu, al, 8 * j), a1 = __shfl_sync(0xffffffffu, al, 8 * j + 4);   // rows 2 j, 2 j + 1
#pragma unroll
        for (int i = 0; i < 2 * NB; ++i) {
          oacc[i][0] *= a0; oacc[i][1] *= a1; oacc[i][2] *= a0; oacc[i][3] *= a1;
          if constexpr (O2) { ot[i][0] *= a0; ot[i][1] *= a1; ot[i][2] *= a0; ot[i][3] *= a1; }
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = exp2f((s[e] - m) * p.scale_log2);
      lt += (s[0] + s[1]) + (s[2] + s[3]);
      // ---- weights times the V scales of positions 2 j, 2 j + 1, 2 j + 8, 2 j + 9 ----
      float pv[4][NB];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t pr = 16 * st + 8 * (e >> 1) + 2 * j + (e & 1);
#pragma unroll
        for (int b = 0; b < NB; b += (NB >= 4 ? 4 : 2)) {
          if (NB >= 4) *reinterpret_cast<float4*>(&pv[e][b]) = *reinterpret_cast<const float4*>(vst + pr * NB + b);
          else *reinterpret_cast<float2*>(&pv[e][b]) = *reinterpret_cast<const float2*>(vst + pr * NB + b);
        }
      }
      if (pos0 + 16 > first_lim) {      // a position the row does not see counts as nothing, whatever its scale (0 * inf is NaN)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (pos0 + 8 * (e >> 1) + 2 * j + (e & 1) >= lim) {
#pragma unroll
            for (int b = 0; b < NB; ++b) pv[e][b] = 0.f;
          }
      }
      // ---- values, two blocks at a time ----
#pragma unroll
      for (int b2 = 0; b2 < NB; b2 += 2) {
        // a power of two per (row, block): the largest product of the step, over the row's four threads, to 2^13 .. 2^14.
        // dn: 2^(E - 140) of the two blocks as the upper halves of their f32s, E the largest's exponent field
        float mb[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
          for (int e = 0; e < 4; ++e) pv[e][b2 + u] *= s[e];
          mb[u] = fmaxf(fmaxf(fabsf(pv[0][b2 + u]), fabsf(pv[1][b2 + u])), fmaxf(fabsf(pv[2][b2 + u]), fabsf(pv[3][b2 + u])));
        }
        uint32_t dn = prmt(__float_as_uint(mb[0]), __float_as_uint(mb[1]), 0x7632u);
        dn = __vmaxu2(dn, __shfl_xor_sync(0xffffffffu, dn, 1));
        dn = __vmaxu2(dn, __shfl_xor_sync(0xffffffffu, dn, 2));
        dn = (__vmaxu2(dn, 0x07000700u) & 0x7f807f80u) - 0x06800680u;           // E at least 14, so that both factors are normal
        const uint32_t dn0 = __shfl_sync(0xffffffffu, dn, 8 * j), dn1 = __shfl_sync(0xffffffffu, dn, 8 * j + 4);   // rows 2 j, 2 j + 1
#pragma unroll
        for (int b = b2; b < b2 + 2; ++b) {
          auto factor = [&](uint32_t x) { return b & 1 ? x & 0xffff0000u : x << 16; };
          const float up = __uint_as_float(0x7f000000u - factor(dn)), d0 = __uint_as_float(factor(dn0)), d1 = __uint_as_float(factor(dn1));
          uint32_t ph0, pl0, ph1, pl1;
          split_h2(pv[0][b] * up, pv[1][b] * up, ph0, pl0);
          split_h2(pv[2][b] * up, pv[3][b] * up, ph1, pl1);
          pl0 = h2_min8(pl0); pl1 = h2_min8(pl1);
          uint32_t w[4];
#pragma unroll
          for (int e = 0; !CV && e < 4; ++e) {
            const uint32_t pr = 16 * st + 8 * (e >> 1) + 2 * j + (e & 1);
            w[e] = *reinterpret_cast<const uint32_t*>(vt + q8_v_off<HD>(pr, 2 * b + (r >> 2)) + (r & 3) * 4) ^ 0x80808080u;
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t a0, a1, a2, a3;
            if constexpr (CV) {     // rows of the tile: dims 32 b + 16 e .. + 15
              ldsm_x4_t(vt_s + q8_h_off<HD>(16 * st + (lane & 7) + ((lane >> 4) << 3), 4 * b + 2 * e + ((lane >> 3) & 1)), a0, a1, a2, a3);
            } else {                // dims 32 b + 4 i + 2 e, then those + 1
              const uint32_t ta = prmt(w[0], w[1], e ? 0x7362u : 0x5140u), tb = prmt(w[2], w[3], e ? 0x7362u : 0x5140u);
              a0 = u8_h2(ta, 0x4140u); a1 = u8_h2(ta, 0x4342u); a2 = u8_h2(tb, 0x4140u); a3 = u8_h2(tb, 0x4342u);
            }
            // into a fresh accumulator, added in f32: the tensor cores' own accumulation rounds towards zero, and over the
            // 250 steps of 4000 rows the result lost 4.4e-6 of itself (2.9e-7 so, as f32 loops do; a 777-token prompt takes 3 % longer)
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            mma_16816(c, a0, a1, a2, a3, ph0, ph1);
            mma_16816(c, a0, a1, a2, a3, pl0, pl1);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float& o = O2 ? ot[O2 ? 2 * b + e : 0][k] : oacc[2 * b + e][k];
              o = __fmaf_rn(c[k], k & 1 ? d1 : d0, o);
            }
          }
        }
      }
      if ((++steps & 15u) == 0) flush();
    }
  }
  flush();
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();                                            // the ring is idle

  // ---- the warps' (o, m, l) to shared memory, then one record (or the output) per query row ----
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  float* so = reinterpret_cast<float*>(smem) + warp * 8 * (HD + 2);   // [8][HD], then m[8], l[8]
#pragma unroll
  for (int i = 0; i < 2 * NB; ++i) {
    if constexpr (CV) {
      float* a = so + (2 * j) * HD + 16 * i + r;
      a[0] = oacc[i][0]; a[8] = oacc[i][2]; a[HD] = oacc[i][1]; a[HD + 8] = oacc[i][3];
    } else {
      const uint32_t d = 32 * (i >> 1) + 4 * r + 2 * (i & 1);
      *reinterpret_cast<float2*>(so + (2 * j) * HD + d) = make_float2(oacc[i][0], oacc[i][2]);
      *reinterpret_cast<float2*>(so + (2 * j + 1) * HD + d) = make_float2(oacc[i][1], oacc[i][3]);
    }
  }
  if (j == 0) { so[8 * HD + r] = m; so[8 * HD + 8 + r] = l; }
  __syncthreads();
  const uint32_t n_rows_here = min(RT, rows - row0);
  const uint32_t ns_live = (tiles + tps - 1) / tps;
  for (uint32_t idx = tid; idx < n_rows_here * (HD / 4); idx += kQ8Threads) {
    const uint32_t lr = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
    const float* wb = reinterpret_cast<const float*>(smem) + (lr >> 3) * 8 * (HD + 2);      // the row group's first warp
    const uint32_t step = p.rgw * 8 * (HD + 2), rr = lr & 7;
    float M = -FLT_MAX, Ls = 0.f;
    for (uint32_t k = 0; k < n_pw; ++k) M = fmaxf(M, wb[k * step + 8 * HD + rr]);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t k = 0; k < n_pw; ++k) {
      const float w = exp2f((wb[k * step + 8 * HD + rr] - M) * p.scale_log2);
      const float4 x = *reinterpret_cast<const float4*>(wb + k * step + rr * HD + d);
      Ls = __fmaf_rn(wb[k * step + 8 * HD + 8 + rr], w, Ls);
      o.x = __fmaf_rn(x.x, w, o.x); o.y = __fmaf_rn(x.y, w, o.y); o.z = __fmaf_rn(x.z, w, o.z); o.w = __fmaf_rn(x.w, w, o.w);
    }
    const uint32_t row = row0 + lr, c = row / G, h = g * G + row % G;
    if (p.cluster) {       // this CTA's share of the row, for the cluster's merge below
      float* mine = reinterpret_cast<float*>(smem + L::MERGE);
      *reinterpret_cast<float4*>(mine + lr * HD + d) = o;
      if (d == 0) { mine[L::MROWS * HD + 2 * lr] = M; mine[L::MROWS * HD + 2 * lr + 1] = Ls; }
      continue;
    }
    if (ns_live > 1) {
      const uint64_t slot = ((uint64_t)c * p.n_heads + h) * p.n_splits + split;
      *reinterpret_cast<float4*>(p.part_o + slot * HD + d) = o;
      if (d == 0) { p.part_ml[slot * 2] = M * inv_sqrt_hd<HD>(); p.part_ml[slot * 2 + 1] = Ls; }
      continue;
    }
    // a call of one split needs no merge: gate and store here
    gate_store4(o, Ls, p.gate, (uint64_t)c * p.gate_col_stride + (uint64_t)h * p.gate_head_stride + d, p.out, (uint64_t)c * p.out_col_stride + (uint64_t)h * HD + d,
                p.act_f16);
  }
  if (!p.cluster) return;
  // at most eight splits: the CTAs of a row tile are a cluster, share out its outputs and read one another's rows (71
  // columns of 16 q / 8 kv heads x 128 into an empty cache: 15.1 us a layer call with a merge kernel, 14.5 so)
  cluster_sync();
  const uint32_t mine_s = sm0 + L::MERGE;
  for (uint32_t idx = split * kQ8Threads + tid; idx < n_rows_here * (HD / 4); idx += ns_live * kQ8Threads) {
    const uint32_t lr = idx / (HD / 4), d = (idx % (HD / 4)) * 4, row = row0 + lr, c = row / G, h = g * G + row % G;
    float Ls;
    const float4 o = cluster_merge4(mine_s + (lr * HD + d) * 4, mine_s + (L::MROWS * HD + 2 * lr) * 4, ns_live, p.scale_log2, Ls);
    gate_store4(o, Ls, p.gate, (uint64_t)c * p.gate_col_stride + (uint64_t)h * p.gate_head_stride + d, p.out, (uint64_t)c * p.out_col_stride + (uint64_t)h * HD + d,
                p.act_f16);
  }
  cluster_sync();          // no CTA leaves while another reads its rows
}

template <int HD, bool CV>
static cudaError_t launch_q8_t(const Q8Params& p, dim3 grid, int dev, cudaStream_t st) {
  using L = Q8Smem<HD, CV>;
  static_assert(L::TOTAL <= 227 * 1024, "shared memory of one CTA");
  static bool attr_set[64] = {};
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(pa_q8_kernel<HD, CV>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (e != cudaSuccess) return e;
    attr_set[dev & 63] = true;
  }
  if (p.cluster) return launch_pdl_cluster(pa_q8_kernel<HD, CV>, grid, dim3(L::THREADS), (size_t)L::TOTAL, st, p.cluster, p);
  return launch_pdl(pa_q8_kernel<HD, CV>, grid, dim3(L::THREADS), (size_t)L::TOTAL, st, p);
}
cudaError_t launch_q8(const Q8Params& p, uint32_t hd, uint32_t n_kv, int dev, cudaStream_t st) {
  const dim3 grid(p.cluster ? p.cluster : p.n_splits, n_kv, (p.n_cols * p.G + 8 * p.rgw - 1) / (8 * p.rgw));
  switch (hd) {
    case 256: return p.cv ? launch_q8_t<256, true>(p, grid, dev, st) : launch_q8_t<256, false>(p, grid, dev, st);
    case 128: return p.cv ? launch_q8_t<128, true>(p, grid, dev, st) : launch_q8_t<128, false>(p, grid, dev, st);
    case 64: return p.cv ? launch_q8_t<64, true>(p, grid, dev, st) : launch_q8_t<64, false>(p, grid, dev, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace pa
