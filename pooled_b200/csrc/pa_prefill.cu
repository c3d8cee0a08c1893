// Tiled causal prefill attention on the 5th-generation tensor cores: tcgen05.mma with the accumulators in tensor
// memory (TMEM), K/V tiles brought in by TMA.
//
// One CTA takes 128 consecutive query columns of one q head and walks the KV cache in tiles of 128 positions up to
// the causal diagonal.  K/V tiles of the G heads of a GQA group are the same bytes, read by G CTAs that run at about
// the same time; the caches of a prefill fit the 126 MB L2, so HBM sees them once.
//
//   warps 0, 3   TMA producers: K in chunks of 128 keys x 64 dims, V in chunks of 16 KB of keys x all dims, a ring each
//                (whole 64 KB tiles of head_dim 256 would leave room for one of each beside Q)
//   warp 1       issues every MMA, in the order S(j + 1), P V(j), S(j + 2), ... (head_dim 128 and 64: S one tile further ahead), so that the
//                weights of a tile have the time of a score product and of a P V product to be formed in
//   warp 2       allocates and frees tensor memory
//   warps 4-11   (4-19 at head_dim 128 and 64) softmax: warp w and warp w + 4 share the 32 query rows of TMEM lanes 32 (w % 4) ..., 64 keys of the tile each:
//                tcgen05.ld of the scores, causal mask, the row's maximum through shared memory, P = 2^(s - m) as f16 pairs
//                into tensor memory (tcgen05.st); then the epilogue (O / l, sigmoid gate, store)
// What a product overwrites has been read: the order of the issue is promised for products of one accumulator and shape only,
// which scores and P V are not.  At head_dim 256 the next scores take the place of scores that the softmax warps have taken into registers, and P
// has two tiles of its own: no wait in the stream (4 layers of 8192 columns of 24 heads 3270 us, as with two S tiles that P overwrites and
// nothing but that order).  At 128 and 64, where a thread has no room for its scores, P lies over S, and S(j + 2) waits for the P V(j - 1)
// that reads it: 318 -> 338 us (8192 columns of 16 heads x 128; 8 layers of 2999 571 -> 592; scores in registers all the same, with spills, 332), 266 both at 64.
//
// O is rescaled only when a row's running maximum has grown by more than 2^8 since its last rescale (weights stay below
// 2^8, exact in f32 sums and safe in f16); the rescale waits for the previous P V to retire and rewrites the row in TMEM.
//
// What bounds it: at head_dim 256 the chip's power, under whose limit it runs at 1.39 GHz, and the tensor cores, whose 2048 cycles a tile
// takes 2220 for; at 128 the exponentials (1024 cycles a tile of the four units) and the wait above.  Why tiles of 128 keys: an instruction of
// 128 x N x 16 takes no less than 67 cycles, so scores in tiles of 64 keys (N = 64, 32 cycles of work) ran at under half of the
// rate: 1394 cycles per 64 keys of head_dim 256 for both products against 1024 with N = 128, measured with nothing else running.
//
// Measured (whole passes, power-capped; tiles of 64 keys with two groups of four softmax warps on alternate tiles and gate rows fetched
// by the lanes before): 4 layers of 8192 columns of 24 heads x 256 3675 -> 3317 us, 8 layers of 2999 x 16 x 128 676 -> 594 (36 of it
// sixteen softmax warps instead of eight, 27 the rotation kernel's), 8 layers of 203 columns of 24 x 256 behind 9001 rows 595 -> 549.
//
// Stands in for attn_flash_tile + attn_combine_tile + sigmoid_mul_mc of pooled (engine/wgsl/attn_tile.js:108-193,
// engine/wgsl/qwen35.js:877-887); there the pass is 16 columns wide and split over the sequence, here a pass takes
// the whole chunk and needs no split/combine because one CTA walks all of its keys.
#include "pa_tc.cuh"

namespace pa {

constexpr int kPM = 128;   // query rows per CTA
constexpr int kPN = 128;   // keys per tile

template <int HD>
struct PfSmem {
  static constexpr int KC = HD / 64, K_CHUNK = kPN * 128;       // K chunks of a tile: [128 keys][64 dims]
  static constexpr int VK = 8192 / HD < kPN ? 8192 / HD : kPN;  // keys of a V chunk: [HD / 64][VK keys][64 dims]
  static constexpr int VC = kPN / VK, V_CHUNK = VK * HD * 2;
  static constexpr bool ALT = HD <= 128;      // sixteen softmax warps, eight on every other tile (see there)
  static constexpr int NGRP = ALT ? 4 : 2, SOFT = 128 * NGRP;            // groups of four softmax warps
  static constexpr int NK = ALT ? 6 : 5, NV = 5;                         // ring depths in chunks
  // tensor memory.  ALT: three S tiles (128 columns each; P takes the first 32 of each half of its S) | O (HD).  head_dim 256, whose O
  // leaves 256 columns: one S tile, which the softmax warps take into registers at once | two P tiles of 64 columns | O
  static constexpr int SBUF = ALT ? 3 : 1, PBUF = ALT ? SBUF : 2;
  static constexpr int T_S = 0, T_P = ALT ? 0 : kPN, P_COLS = ALT ? kPN : kPN / 2, P_HALF = P_COLS / 2, T_O = T_P + PBUF * P_COLS, TMEM_COLS = 512;
  static_assert(T_O + HD <= 512, "tensor memory columns");
  static constexpr int THREADS = 128 + SOFT;
  static constexpr int OFF_Q = 0, OFF_K = HD * kPM * 2, OFF_V = OFF_K + NK * K_CHUNK, OFF_BAR = OFF_V + NV * V_CHUNK;
  static constexpr int RINGS = NK * K_CHUNK + NV * V_CHUNK;
  // halves' row maxima of a tile, [2 tiles][ALT: tiles' parity][2 halves][128]; ALT: the rows' references after a tile, [2][128]
  static constexpr int OFF_MX = OFF_BAR + 512, OFF_RM = OFF_MX + NGRP * 2 * kPM * 4;
  static constexpr int TOTAL = OFF_RM + (ALT ? 2 * kPM * 4 : 0);
  static_assert(TOTAL <= 227 * 1024, "shared memory of one CTA");
};

// keys of each of ns splits of `keys` keys, in whole 64s
__device__ __forceinline__ uint32_t split_keys(uint32_t keys, uint32_t ns) { return ((keys + 63) / 64 + ns - 1) / ns * 64; }

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// two f32 operations per instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// SPLIT: the keys split over blockIdx.z and a record per (row, split) instead of the output (an instantiation of its own:
// a run-time split cost the unsplit kernel 2.5 % at head_dim 128).
template <int HD, bool SPLIT>
__global__ void __launch_bounds__(PfSmem<HD>::THREADS, 1)
pa_prefill_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_q,
                  const __grid_constant__ CUtensorMap tm_o, const __grid_constant__ CUtensorMap tm_q2, const __grid_constant__ CUtensorMap tm_g,
                  const PrefillParams p) {
  using L = PfSmem<HD>;
  constexpr int NK = L::NK, NV = L::NV, SB = L::SBUF, PB = L::PBUF, NGRP = L::NGRP, SOFT = L::SOFT;
  extern __shared__ __align__(1024) uint8_t base[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + L::OFF_BAR);
  enum { K_FULL = 0, K_EMPTY = NK, V_FULL = 2 * NK, V_EMPTY = 2 * NK + NV, S_FULL = 2 * NK + 2 * NV, P_FULL = S_FULL + SB, PV_DONE = P_FULL + PB, O_DONE = PV_DONE + 2,
         Q_FULL = O_DONE + 1, G_FULL = O_DONE + 2, M_READY = O_DONE + 3, S_READ = M_READY + 2, N_BARS = S_READ + 1 };
  static_assert(N_BARS <= 62, "barrier slots");
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(bars + 62);
  volatile uint32_t* s_err = s_tmem + 1;
  float* s_mx = reinterpret_cast<float*>(base + L::OFF_MX);
  const uint32_t bar0 = smem_u32(bars);
  auto BAR = [&](int which, uint32_t idx) { return bar0 + 8u * ((uint32_t)which + idx); };
  const uint32_t q_s = smem_u32(base + L::OFF_Q), k_s = smem_u32(base + L::OFF_K), v_s = smem_u32(base + L::OFF_V);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Every head's longest q tile first, then every head's next one: with the q tiles of a head following one another the
  // last heads' longest tiles began when the other SMs had run out of work (2048 columns of 24 heads: SMs busy 71 %).
  const uint32_t q_tile = gridDim.y - 1 - blockIdx.y;
  const uint32_t h = blockIdx.x, g = h / p.G, c0 = q_tile * kPM;
  const uint32_t rows_valid = min((uint32_t)kPM, p.n_cols - c0);
  const uint32_t p0 = p.pos + c0;                       // cache row of column c0's own token
  uint32_t key0 = 0, key_end = p0 + rows_valid;         // this CTA's keys
  if constexpr (SPLIT) {
    // a short prompt behind a long context: the keys of a q tile are split over blockIdx.z (see prefill_splits)
    const uint32_t per = split_keys(key_end, p.n_splits);
    key0 = blockIdx.z * per;
    if (key0 >= key_end) return;                        // uniform for the CTA; the merge derives the same count
    key_end = min(key_end, key0 + per);
  }
  const uint32_t n_tiles = (key_end - key0 + kPN - 1) / kPN;
  // f16 q: the 128 query rows land in shared memory, in the layout the score products read, by one TMA copy
  const bool q_by_tma = p.q_tma != 0;
  if (warp == 1 && lane == 0) {
    *s_err = 0;
    for (int i = 0; i < NK; ++i) { mbar_init(BAR(K_FULL, i), 1); mbar_init(BAR(K_EMPTY, i), 1); }
    for (int i = 0; i < NV; ++i) { mbar_init(BAR(V_FULL, i), 1); mbar_init(BAR(V_EMPTY, i), 1); }
    for (int i = 0; i < SB; ++i) mbar_init(BAR(S_FULL, i), 1);
    for (int i = 0; i < PB; ++i) mbar_init(BAR(P_FULL, i), 8);
    mbar_init(BAR(S_READ, 0), 8);
    for (int i = 0; i < 2; ++i) { mbar_init(BAR(PV_DONE, i), 1); mbar_init(BAR(M_READY, i), 8); }
    mbar_init(BAR(O_DONE, 0), 1);
    mbar_init(BAR(G_FULL, 0), 1);
    mbar_init(BAR(Q_FULL, 0), q_by_tma ? 1 : SOFT);
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32((const void*)s_tmem), L::TMEM_COLS);
    tmem_relinquish();
    tc_fence_before();
  }
  pdl_wait();        // q, and the rows the RoPE/append kernel before this one writes
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const uint32_t t_s0 = tmem + L::T_S, t_p0 = tmem + L::T_P, t_o = tmem + L::T_O;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer, Q and K ----
    if (lane == 0) {
      prefetch_tmap(&tm_k);
      if (q_by_tma) {
        mbar_expect_tx(BAR(Q_FULL, 0), HD * kPM * 2);
        tma_load_3d(q_s, &tm_q, 0, (int)c0, (int)(h * (p.q_head_stride / 64)), BAR(Q_FULL, 0));
        if (p.q_tma == 2)   // the chunks no rotation touches come straight from the caller's q
          tma_load_3d(q_s + p.q_rot_chunks * (kPM * 128), &tm_q2, 0, (int)c0, (int)(h * (p.q2_head_stride / 64) + p.q_rot_chunks), BAR(Q_FULL, 0));
      }
      if (!SPLIT && p.gate_tma) tma_prefetch_3d(&tm_g, 0, (int)c0, (int)(h * (p.gate_head_stride / 64)));
      if (!SPLIT && p.q_tma) {
        // the query rows of the CTA that takes this one's place, into L2 (those a kernel wrote just now are there): 128-byte pieces of
        // rows 12 KB and more apart, for which it would wait for HBM at its start.  (The gate's above likewise, for the end.)  8 layers of 2999 columns of 16
        // heads x 128 577 -> 572 us, 4 of 8192 of 24 x 256 3310 -> 3265.
        const uint32_t next = blockIdx.y * gridDim.x + blockIdx.x + p.sms;
        if (next < gridDim.x * gridDim.y) {
          const uint32_t hn = next % gridDim.x, cn = (gridDim.y - 1 - next / gridDim.x) * kPM;
          if (p.q_tma == 2) tma_prefetch_3d(&tm_q2, 0, (int)cn, (int)(hn * (p.q2_head_stride / 64) + p.q_rot_chunks));
          else tma_prefetch_3d(&tm_q, 0, (int)cn, (int)(hn * (p.q_head_stride / 64)));
        }
      }
      uint32_t st = 0, ph = 1;
      for (uint32_t j = 0; j < n_tiles; ++j) {
        for (int c = 0; c < L::KC; ++c) {
          mbar_wait(BAR(K_EMPTY, st), ph, s_err, WAIT_EMPTY);
          mbar_expect_tx(BAR(K_FULL, st), L::K_CHUNK);
          tma_load_3d(k_s + st * L::K_CHUNK, &tm_k, 0, (int)(key0 + j * kPN), (int)(g * L::KC + c), BAR(K_FULL, st));
          if (++st == NK) { st = 0; ph ^= 1; }
        }
      }
      if (!SPLIT && p.gate_tma) {
        // the gate's 128 rows into the K ring as soon as the last scores have read it, while the last tile's weights are formed:
        // the epilogue finds them in shared memory.  (Each lane fetching its own row, 64 bytes 12 KB apart at a time, the epilogue
        // took 17 us of a 67 us CTA of 8192 columns of 24 heads x 256.)
        static_assert(HD * kPM * 2 <= NK * L::K_CHUNK && HD * kPM * 2 <= NV * L::V_CHUNK, "the gate and the output tile fit the rings");
        for (int i = 0; i < NK; ++i) {
          mbar_wait(BAR(K_EMPTY, st), ph, s_err, WAIT_EMPTY);
          if (++st == NK) { st = 0; ph ^= 1; }
        }
        mbar_expect_tx(BAR(G_FULL, 0), HD * kPM * 2);
        tma_load_3d(k_s, &tm_g, 0, (int)c0, (int)(h * (p.gate_head_stride / 64)), BAR(G_FULL, 0));
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ TMA producer, V ----
    if (lane == 0) {
      prefetch_tmap(&tm_v);
      uint32_t st = 0, ph = 1;
      for (uint32_t j = 0; j < n_tiles; ++j) {
        for (int c = 0; c < L::VC && key0 + j * kPN + c * L::VK < key_end; ++c) {      // (every chunk is waited for: the epilogue uses the ring)
          mbar_wait(BAR(V_EMPTY, st), ph, s_err, WAIT_EMPTY);
          mbar_expect_tx(BAR(V_FULL, st), L::V_CHUNK);
          tma_load_3d(v_s + st * L::V_CHUNK, &tm_v, 0, (int)(key0 + j * kPN + c * L::VK), (int)(g * L::KC), BAR(V_FULL, st));
          if (++st == NV) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer ----
    // The whole warp runs the loop and the elected lane issues (operands in uniform registers).
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc_qk = umma_idesc(kPM, kPN, 0), idesc_pv = umma_idesc(kPM, HD, 1);
    const uint64_t q_desc = smem_desc(q_s, 16, 1024), k_desc = smem_desc(k_s, 16, 1024), v_desc = smem_desc(v_s, L::VK * 128, 1024);
    uint32_t kst = 0, kph = 0, vst = 0, vph = 0;
    auto scores = [&](uint32_t j) {      // S(j) = Q K(j)^T
      const uint32_t ts = t_s0 + (j % SB) * kPN;
#pragma unroll
      for (int c = 0; c < L::KC; ++c) {
        mbar_wait(BAR(K_FULL, kst), kph, s_err, WAIT_KFULL);
        tc_fence_after();
        const uint64_t kd = k_desc + (uint64_t)(kst * (L::K_CHUNK >> 4)), qd = q_desc + (uint64_t)(c * ((kPM * 128) >> 4));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma_f16_ss(leader, ts, qd + ks * 2, kd + ks * 2, idesc_qk, (c > 0 || ks > 0) ? 1u : 0u);
        umma_commit_elected(leader, BAR(K_EMPTY, kst));
        if (++kst == NK) { kst = 0; kph ^= 1; }
      }
      umma_commit_elected(leader, BAR(S_FULL, j % SB));
    };
    mbar_wait(BAR(Q_FULL, 0), 0, s_err, WAIT_QFULL);
    tc_fence_after();
    // Nothing rests on the order in which products of different accumulators run: what a product overwrites has been read.
    constexpr uint32_t AHEAD = L::ALT ? SB - 1 : 1;
#pragma unroll 1
    for (uint32_t j = 0; j < AHEAD && j < n_tiles; ++j) scores(j);
    auto ahead = [&](uint32_t j) {
      if (j + AHEAD >= n_tiles) return;
      // ALT: the scores two tiles ahead take the place of the weights P(j - 1), once the product that reads them has retired.  Otherwise
      // the next tile's take the place of S(j), which the softmax warps hold in registers while P V(j - 1) runs
      if (!L::ALT) mbar_wait(BAR(S_READ, 0), j & 1, s_err, WAIT_MMA);
      else if (j > 0) mbar_wait(BAR(PV_DONE, (j - 1) & 1), ((j - 1) >> 1) & 1, s_err, WAIT_MMA);
      scores(j + AHEAD);
    };
    // P(j): packed f16 pairs in the first 32 columns of each half; 16 keys of them
    auto p_at = [&](uint32_t j, int k16) { return t_p0 + (j % PB) * L::P_COLS + (k16 >> 2) * L::P_HALF + (k16 & 3) * 8; };
    // The last tile's product goes no further than the 16 keys that hold the CTA's last: a weight of zero times an infinite value of
    // a later row is NaN.  In a loop of its own, since the others' issue bears no test between products (2999 columns of 16
    // heads x 128, 8 layers: 592 us; 612 with a branch per product, 654 with the test in the product's predicate).
    const uint32_t whole = (key_end - key0 + 15) / kPN;
#pragma unroll 1
    for (uint32_t j = 0; j < whole; ++j) {
      ahead(j);
      mbar_wait(BAR(P_FULL, j % PB), (j / PB) & 1, s_err, WAIT_MMA);
#pragma unroll
      for (int c = 0; c < L::VC; ++c) {              // O += P(j) V(j)
        mbar_wait(BAR(V_FULL, vst), vph, s_err, WAIT_VFULL);
        tc_fence_after();
        const uint64_t vd = v_desc + (uint64_t)(vst * (L::V_CHUNK >> 4));
#pragma unroll
        for (int ks = 0; ks < L::VK / 16; ++ks)
          umma_f16_ts(leader, t_o, p_at(j, c * L::VK / 16 + ks), vd + (uint64_t)((ks * 2048) >> 4), idesc_pv, (j > 0 || c > 0 || ks > 0) ? 1u : 0u);
        umma_commit_elected(leader, BAR(V_EMPTY, vst));
        if (++vst == NV) { vst = 0; vph ^= 1; }
      }
      umma_commit_elected(leader, BAR(PV_DONE, j & 1));
    }
    if (whole < n_tiles) {
      const uint32_t j = whole, steps = (key_end - key0 - j * kPN + 15) / 16;
      mbar_wait(BAR(P_FULL, j % PB), (j / PB) & 1, s_err, WAIT_MMA);
#pragma unroll 1
      for (int k16 = 0; k16 < (int)steps; ++k16) {
        if (k16 % (L::VK / 16) == 0) {
          if (k16 > 0 && ++vst == NV) { vst = 0; vph ^= 1; }
          mbar_wait(BAR(V_FULL, vst), vph, s_err, WAIT_VFULL);
          tc_fence_after();
        }
        umma_f16_ts(leader, t_o, p_at(j, k16), v_desc + (uint64_t)(vst * (L::V_CHUNK >> 4)) + (uint64_t)((k16 % (L::VK / 16) * 2048) >> 4), idesc_pv,
                    (j > 0 || k16 > 0) ? 1u : 0u);
      }
    }
    umma_commit_elected(leader, BAR(O_DONE, 0));
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax + epilogue ----
    const uint32_t wg = (warp - 4) >> 2, half = wg & 1;  // group; half of a tile's keys
    const uint32_t qd = warp & 3, row = qd * 32 + lane;  // a warp reaches the 32 TMEM lanes of its index mod 4
    const uint32_t lane_addr = (qd * 32) << 16;
    const bool live = row < rows_valid;
    const uint32_t lim = min(p0 + row + 1, key_end);     // of the CTA's keys those below lim are visible to this row
    pdl_trigger();
    const __half* gate_row = reinterpret_cast<const __half*>(p.gate) + (uint64_t)(c0 + row) * p.gate_col_stride + (uint64_t)h * p.gate_head_stride;
    const bool by_pieces = p.act_f16 && (!p.gate || p.gate_tma || !(((uintptr_t)p.gate & 15) | (p.gate_col_stride & 7) | (p.gate_head_stride & 7)));
    if (!SPLIT && by_pieces && p.gate && !p.gate_tma && live)      // a lane's own row of the gate, for the end
      for (uint32_t d = wg * 64; d < HD; d += NGRP * 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(gate_row + d));
    if (!q_by_tma) {
      // this thread's share of its Q row as f16 into the layout the score products read
      constexpr int PC = HD / 8 / NGRP;                  // 16-byte pieces
      const uint64_t off = (uint64_t)(c0 + (live ? row : 0)) * p.q_col_stride + (uint64_t)h * p.q_head_stride + wg * (HD / NGRP);
      uint4 x[PC];
#pragma unroll
      for (int i = 0; i < PC; ++i) {
        if (!live) { x[i] = make_uint4(0, 0, 0, 0); continue; }
        if (p.q_f16) { x[i] = reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(p.q) + off)[i]; continue; }
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.q) + off) + 2 * i;
        const float4 a = src[0], b = src[1];
        x[i] = make_uint4(pack_h2(a.x, a.y), pack_h2(a.z, a.w), pack_h2(b.x, b.y), pack_h2(b.z, b.w));
      }
#pragma unroll
      for (int i = 0; i < PC; ++i) {
        const uint32_t pc = wg * PC + i, c = pc >> 3;    // piece of the row, 64-dim chunk
        *reinterpret_cast<uint4*>(base + L::OFF_Q + c * (kPM * 128) + row * 128 + (((pc & 7) ^ (row & 7)) << 4)) = x[i];
      }
      fence_proxy_async();
      mbar_arrive(BAR(Q_FULL, 0));
    }
    // m_st: the row's reference maximum, the same in both halves' threads (the weights of a tile are 2^(s - m_st); it moves only
    // when the maximum of a tile's half passes it by more than 2^8).  (A split that does not begin at key 0 may hold no visible key of a row, hence the finite start.)
    const bool first0 = !SPLIT || key0 == 0;
    float m_st = first0 ? -INFINITY : -1.0e30f;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    // causal mask on tiles that reach this row's diagonal
    auto mask = [&](float* x, int n, uint32_t key0) {
      if (key0 + n > lim) {
#pragma unroll
        for (int i = 0; i < n; ++i) if (key0 + i >= lim) x[i] = -INFINITY;
      }
    };
    auto max32 = [](const float* x, float m) {
      float a = max3(m, x[0], x[1]), b = fmaxf(x[2], x[3]), c = fmaxf(x[4], x[5]), d = fmaxf(x[6], x[7]);
#pragma unroll
      for (int i = 8; i < 32; i += 8) { a = max3(a, x[i], x[i + 1]); b = max3(b, x[i + 2], x[i + 3]); c = max3(c, x[i + 4], x[i + 5]); d = max3(d, x[i + 6], x[i + 7]); }
      return fmaxf(fmaxf(a, b), fmaxf(c, d));
    };
    // the row's reference given the maxima (scaled) of the tile's halves; how much O and the row's sum shrink if it moves.  It is the
    // running reference of 64 keys after 64, whatever the tile: the f16 roundings of the weights depend on it, and with one
    // maximum for the tile a result moved by 2e-4 of itself, as much as all of those roundings.
    auto refer = [&](uint32_t j, float mt0, float mt1, float& alpha) {
      const bool start = first0 && j == 0;                       // key 0 is visible to every row
      const float was = m_st;
      if (start || mt0 > m_st + 8.f) m_st = mt0;
      if (mt1 > m_st + 8.f) m_st = mt1;
      alpha = 1.f;
      if (start || m_st == was) return false;
      alpha = ex2_approx(was - m_st);
      return true;
    };
    // O must not change under the previous P V: wait for it, then rescale this warp's 32 rows in TMEM, chunks c0, c0 + dc, ...
    auto rescale = [&](uint32_t j, float alpha, uint32_t c0, uint32_t dc) {
      mbar_wait(BAR(PV_DONE, (j - 1) & 1), ((j - 1) >> 1) & 1, s_err, WAIT_MMA);
      tc_fence_after();
#pragma unroll 1
      for (uint32_t c = c0; c < HD / 32; c += dc) {
        float o[32];
        tmem_ld32(t_o + c * 32 + lane_addr, o);
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] *= alpha;
        tmem_st32(t_o + c * 32 + lane_addr, o);
      }
    };
    // P = 2^(s - m) of 32 scores as packed f16 pairs, and their sum
    auto weigh = [&](const float* x, uint32_t* w) {
      const float2 nm = make_float2(-m_st, -m_st);
      float2 la = make_float2(0.f, 0.f), lb = la;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 y = fma2(make_float2(x[2 * i], x[2 * i + 1]), sc2, nm);
        const float2 e = make_float2(ex2_approx(y.x), ex2_approx(y.y));
        if (i & 1) lb = add2(lb, e); else la = add2(la, e);
        w[i] = pack_h2(e.x, e.y);
      }
      return add2(la, lb);
    };
    float l_sum;
    if constexpr (L::ALT) {
      // Head_dim 128 and 64: the exponentials of a tile, 1024 cycles of the four units, are as much as its products.  Eight warps on
      // halves of every tile load, compare and exponentiate in step and the units idle in between (1970 cycles a tile of head_dim 128), as
      // do eight on whole rows of alternate tiles (1850); so sixteen, eight on every other tile, four per scheduler.  The scores are
      // read twice, for the maximum and for the weights (40 cycles per 64 columns): 96 registers do.  The reference travels with the tiles.
      const uint32_t par = wg >> 1;
      float* s_rm = reinterpret_cast<float*>(base + L::OFF_RM);
      float m_l = m_st, l = 0.f;       // this thread's share of the row's sum, and the reference it is in
      for (uint32_t j = par; j < n_tiles; j += 2) {
        const uint32_t b = j % SB, kv0 = key0 + j * kPN + half * 64, ts = t_s0 + b * kPN + lane_addr + half * 64;
        mbar_wait(BAR(S_FULL, b), (j / SB) & 1, s_err, WAIT_MMA);
        tc_fence_after();
        float s[32], mt = -INFINITY;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tmem_ld32(ts + c * 32, s);
          mask(s, 32, kv0 + c * 32);
          mt = max32(s, mt);
        }
        float* mx = s_mx + ((j >> 1) & 1) * (4 * kPM) + par * (2 * kPM);
        mx[half * kPM + row] = mt;
        named_bar_sync(2 + par * 4 + qd, 64);
        const float mo = mx[(half ^ 1) * kPM + row];
        if (j > 0) {
          mbar_wait(BAR(M_READY, (j - 1) & 1), ((j - 1) >> 1) & 1, s_err, WAIT_MMA);
          m_st = s_rm[((j - 1) & 1) * kPM + row];
        }
        float alpha;
        const bool grow = refer(j, (half ? mo : mt) * p.scale_log2, (half ? mt : mo) * p.scale_log2, alpha);
        if (half == 0) s_rm[(j & 1) * kPM + row] = m_st;
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(M_READY, j & 1));      // (both halves have read the one before: its place is free for tile j + 1)
        if (j > 0 && __any_sync(0xffffffffu, grow)) rescale(j, alpha, half, 2);
        if (m_st != m_l) { l *= ex2_approx(m_l - m_st); m_l = m_st; }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tmem_ld32(ts + c * 32, s);
          mask(s, 32, kv0 + c * 32);
          uint32_t pw[16];
          const float2 lt = weigh(s, pw);
          tmem_st16u(ts + c * 16, pw);
          l += lt.x + lt.y;
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(P_FULL, b));
      }
      const uint32_t last = n_tiles - 1;
      mbar_wait(BAR(M_READY, last & 1), (last >> 1) & 1, s_err, WAIT_MMA);
      m_st = s_rm[(last & 1) * kPM + row];
      named_bar_sync(1, SOFT);         // the maxima are not read any more
      s_mx[wg * kPM + row] = l * ex2_approx(m_l - m_st);
      named_bar_sync(1, SOFT);
      l_sum = (s_mx[row] + s_mx[kPM + row]) + (s_mx[2 * kPM + row] + s_mx[3 * kPM + row]);
    } else {
      float2 l2 = make_float2(0.f, 0.f);       // this thread's share of the row's sum
      const uint32_t ts = t_s0 + lane_addr + half * 64;
      for (uint32_t j = 0; j < n_tiles; ++j) {
        const uint32_t kv0 = key0 + j * kPN + half * 64;
        mbar_wait(BAR(S_FULL, 0), j & 1, s_err, WAIT_MMA);
        tc_fence_after();
        float s[64];
        tmem_ld32_async(ts, s);
        tmem_ld32_async(ts + 32, s + 32);
        tmem_wait_ld(s);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(S_READ, 0));
        mask(s, 64, kv0);
        // the two halves' maxima through shared memory
        const float m_half = max32(s + 32, max32(s, -INFINITY));
        float* mx = s_mx + (j & 1) * (2 * kPM);
        mx[wg * kPM + row] = m_half;
        named_bar_sync(2 + qd, 64);
        const float mo = mx[(wg ^ 1) * kPM + row];
        float alpha;
        if (__any_sync(0xffffffffu, refer(j, (wg ? mo : m_half) * p.scale_log2, (wg ? m_half : mo) * p.scale_log2, alpha))) {
          l2.x *= alpha; l2.y *= alpha;
          if (j > 0) rescale(j, alpha, wg, 2);            // half of the dims per warp
        }
        uint32_t pw[32];
        float2 lt = weigh(s, pw);
        lt = add2(lt, weigh(s + 32, pw + 16));
        if (j >= 2) {      // P(j - 2), in the same place, has been read
          mbar_wait(BAR(PV_DONE, j & 1), ((j >> 1) - 1) & 1, s_err, WAIT_MMA);
          tc_fence_after();
        }
        tmem_st32u(t_p0 + (j & 1) * L::P_COLS + lane_addr + half * L::P_HALF, pw);
        l2 = add2(l2, lt);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR(P_FULL, j & 1));
      }
      float* s_l = s_mx + ((n_tiles & 1) ? 2 * kPM : 0);   // the slot the last tile's maxima are not in
      s_l[wg * kPM + row] = l2.x + l2.y;
      named_bar_sync(1, 256);
      l_sum = s_l[row] + s_l[kPM + row];
    }
    // ---- epilogue: O / l, gate, store ----
    mbar_wait(BAR(O_DONE, 0), 0, s_err, WAIT_MMA);
    tc_fence_after();
    const float inv_l = 1.f / l_sum;
    const uint32_t col = c0 + row;
    if constexpr (SPLIT) {
      // this split's unnormalised (o, m, l) of every row, by way of shared memory (the rings are idle): a lane holds a row,
      // and stored as they are the 32 lanes of an instruction would write into 32 records 1 KB and more apart
      constexpr int RP = HD / 4 + 1;                                    // row pitch in float4: 16 bytes apart in their bank phase
      static_assert(kPM * RP * 16 <= L::RINGS, "the record tile fits the idle rings");
      float4* xs = reinterpret_cast<float4*>(base + L::OFF_K);
#pragma unroll 1
      for (uint32_t c = wg; c < HD / 32; c += NGRP) {
        float o[32];
        tmem_ld32(t_o + c * 32 + lane_addr, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) xs[row * RP + c * 8 + i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      }
      named_bar_sync(1, SOFT);
      for (uint32_t idx = tid - 128; idx < rows_valid * (HD / 4); idx += SOFT) {
        const uint32_t rr = idx / (HD / 4), c4 = idx % (HD / 4);
        const uint64_t slot = ((uint64_t)(c0 + rr) * p.n_heads + h) * p.n_splits + blockIdx.z;
        reinterpret_cast<float4*>(p.part_o + slot * HD)[c4] = xs[rr * RP + c4];
      }
      if (wg == 0 && row < rows_valid) {
        const uint64_t slot = ((uint64_t)col * p.n_heads + h) * p.n_splits + blockIdx.z;
        p.part_ml[slot * 2] = m_st * 0.6931471805599453f; p.part_ml[slot * 2 + 1] = l_sum;
      }
    } else if (by_pieces) {
      // f16: the output tile leaves as the query tile came: through shared memory in the TMA layout ([64-dim chunk][row][128 B],
      // 16-byte pieces XOR-swizzled by the row), one bulk tensor store for the CTA, from the V ring (every product
      // has retired).  Rows past the prompt's end are not written: the map ends at n_cols.
      // (A lane storing its own row issues 16-byte stores 12 KB apart.)  Where no map takes the output's stride, the threads store whole rows.
      uint8_t* o_s = base + L::OFF_V;
      const uint4* gp = reinterpret_cast<const uint4*>(gate_row);
      if (p.gate_tma) mbar_wait(BAR(G_FULL, 0), 0, s_err, WAIT_QFULL);
#pragma unroll 1
      for (uint32_t c = wg; c < HD / 32; c += NGRP) {            // the groups share the columns out
        const uint32_t at = (c >> 1) * (kPM * 128) + row * 128;
        uint4 gq[4];      // (a gate no tensor map takes: each lane its own row)
        if (p.gate) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            gq[i] = p.gate_tma ? *reinterpret_cast<const uint4*>(base + L::OFF_K + at + ((((c & 1) * 4 + i) ^ (row & 7)) << 4)) : live ? gp[c * 4 + i] : make_uint4(0, 0, 0, 0);
        }
        float o[32];
        tmem_ld32(t_o + c * 32 + lane_addr, o);
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] *= inv_l;
        if (p.gate) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t gw[4] = {gq[i].x, gq[i].y, gq[i].z, gq[i].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 gv = __half22float2(*reinterpret_cast<const __half2*>(&gw[k]));
              o[8 * i + 2 * k] *= 1.0f / (1.0f + __expf(-gv.x));
              o[8 * i + 2 * k + 1] *= 1.0f / (1.0f + __expf(-gv.y));
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(o_s + at + ((((c & 1) * 4 + i) ^ (row & 7)) << 4)) =
              make_uint4(pack_h2(o[8 * i], o[8 * i + 1]), pack_h2(o[8 * i + 2], o[8 * i + 3]), pack_h2(o[8 * i + 4], o[8 * i + 5]), pack_h2(o[8 * i + 6], o[8 * i + 7]));
      }
      if (p.out_tma) fence_proxy_async();
      named_bar_sync(1, SOFT);
      if (!p.out_tma) {
        for (uint32_t idx = tid - 128; idx < rows_valid * (HD / 8); idx += SOFT) {
          const uint32_t rr = idx / (HD / 8), pc = idx % (HD / 8);
          *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.out) + (uint64_t)(c0 + rr) * p.out_col_stride + (uint64_t)h * HD + pc * 8) =
              *reinterpret_cast<const uint4*>(o_s + (pc >> 3) * (kPM * 128) + rr * 128 + (((pc & 7) ^ (rr & 7)) << 4));
        }
      } else if (tid == 128) {
        tma_store_3d(&tm_o, 0, (int)c0, (int)(h * (HD / 64)), smem_u32(o_s));
        tma_store_wait_read();
      }
    } else {
      // f32 activations, or a gate that is not read 16 bytes at a time: the rows by way of shared memory, so that gate loads and output
      // stores are whole rows too
      constexpr int RP = HD / 4 + 1, U = L::ALT ? 4 : 8;
      float4* xs = reinterpret_cast<float4*>(base + L::OFF_K);
#pragma unroll 1
      for (uint32_t c = wg; c < HD / 32; c += NGRP) {
        float o[32];
        tmem_ld32(t_o + c * 32 + lane_addr, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) xs[row * RP + c * 8 + i] = make_float4(o[4 * i] * inv_l, o[4 * i + 1] * inv_l, o[4 * i + 2] * inv_l, o[4 * i + 3] * inv_l);
      }
      named_bar_sync(1, SOFT);
      const bool g_vec = !p.act_f16 && !(((uintptr_t)p.gate & 15) | (p.gate_col_stride & 3) | (p.gate_head_stride & 3));
      const uint32_t n_it = rows_valid * (HD / 4);
      for (uint32_t i0 = tid - 128; i0 < n_it; i0 += SOFT * U) {
        float gv[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t idx = i0 + SOFT * u, rr = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
          if (!p.gate || idx >= n_it) continue;
          const uint64_t go = (uint64_t)(c0 + rr) * p.gate_col_stride + (uint64_t)h * p.gate_head_stride + d;
          if (g_vec) *reinterpret_cast<float4*>(gv[u]) = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.gate) + go);
          else {
#pragma unroll
            for (int k = 0; k < 4; ++k) gv[u][k] = ld_act(p.gate, go + k, p.act_f16);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t idx = i0 + SOFT * u, rr = idx / (HD / 4), d = (idx % (HD / 4)) * 4;
          if (idx >= n_it) continue;
          float4 o = xs[rr * RP + d / 4];
          if (p.gate) {
            o.x *= 1.0f / (1.0f + __expf(-gv[u][0])); o.y *= 1.0f / (1.0f + __expf(-gv[u][1]));
            o.z *= 1.0f / (1.0f + __expf(-gv[u][2])); o.w *= 1.0f / (1.0f + __expf(-gv[u][3]));
          }
          const uint64_t oo = (uint64_t)(c0 + rr) * p.out_col_stride + (uint64_t)h * HD + d;
          if (p.act_f16) *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.out) + oo) = make_uint2(pack_h2(o.x, o.y), pack_h2(o.z, o.w));
          else *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + oo) = o;
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, L::TMEM_COLS);
  }
  if (tid == 0 && *s_err) atomicMax(p.err, *s_err);
}

// LSE merge of the few (2..8) records a split prefill leaves per query row, gate and store: a warp per row, HD / 32 values
// per lane, every record of the row requested at once.  (pa_combine_kernel, 256 threads per row and 64 dims, is made for
// few rows of many records: at 4872 rows x 3 records it would be 19488 CTAs with 48 of 256 lanes at work.)  The
// records were written just now and come from L2.  The same arithmetic: weights e^(m - M), sums in split order.
template <int HD>
__global__ void __launch_bounds__(256) pa_combine_few_kernel(const PrefillParams p) {
  constexpr int NV = HD >= 128 ? HD / 128 : 1, W = HD >= 128 ? 4 : 2;   // vectors of W floats per lane
  const uint32_t prow = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_wait();
  pdl_trigger();
  if (prow >= p.n_cols * p.n_heads) return;
  const uint32_t col = prow / p.n_heads, h = prow % p.n_heads, c0 = col / kPM * kPM;
  const uint32_t keys = p.pos + c0 + min((uint32_t)kPM, p.n_cols - c0), per = split_keys(keys, p.n_splits);
  const uint32_t ns = (keys + per - 1) / per;      // live splits of this q tile
  const float* ml = p.part_ml + (uint64_t)prow * p.n_splits * 2;
  const float* ob = p.part_o + (uint64_t)prow * p.n_splits * HD + lane * W;
  float m[kPrefillSplits], l[kPrefillSplits], x[kPrefillSplits][NV * W];
#pragma unroll
  for (int s = 0; s < kPrefillSplits; ++s) {
    m[s] = -3.0e38f; l[s] = 0.f;
    if ((uint32_t)s >= ns) continue;
    m[s] = ml[2 * s]; l[s] = ml[2 * s + 1];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (W == 4) *reinterpret_cast<float4*>(&x[s][4 * v]) = *reinterpret_cast<const float4*>(ob + s * HD + v * 128);
      else *reinterpret_cast<float2*>(&x[s][0]) = *reinterpret_cast<const float2*>(ob + s * HD);
    }
  }
  float gv[NV * W];
  const uint64_t go = (uint64_t)col * p.gate_col_stride + (uint64_t)h * p.gate_head_stride;
#pragma unroll
  for (int i = 0; i < NV * W; ++i) {
    const uint32_t d = (i / W) * 128 + lane * W + i % W;
    gv[i] = p.gate ? ld_act(p.gate, go + d, p.act_f16) : 0.f;
  }
  float M = m[0];
#pragma unroll
  for (int s = 1; s < kPrefillSplits; ++s) M = fmaxf(M, m[s]);
  float L = 0.f, acc[NV * W];
#pragma unroll
  for (int i = 0; i < NV * W; ++i) acc[i] = 0.f;
#pragma unroll
  for (int s = 0; s < kPrefillSplits; ++s) {
    if ((uint32_t)s >= ns) continue;
    const float w = __expf(m[s] - M);
    L = __fmaf_rn(l[s], w, L);
#pragma unroll
    for (int i = 0; i < NV * W; ++i) acc[i] = __fmaf_rn(x[s][i], w, acc[i]);
  }
  const uint64_t oo = (uint64_t)col * p.out_col_stride + (uint64_t)h * HD;
#pragma unroll
  for (int i = 0; i < NV * W; ++i) {
    acc[i] = __fdiv_rn(acc[i], L);
    if (p.gate) acc[i] = __fmul_rn(acc[i], __fdiv_rn(1.0f, __fadd_rn(1.0f, __expf(-gv[i]))));
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const uint32_t d = v * 128 + lane * W;
    if (p.act_f16) {
      __half* dst = reinterpret_cast<__half*>(p.out) + oo + d;
      if (W == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(pack_h2(acc[4 * v], acc[4 * v + 1]), pack_h2(acc[4 * v + 2], acc[4 * v + 3]));
      else *reinterpret_cast<uint32_t*>(dst) = pack_h2(acc[0], acc[1]);
    } else {
      float* dst = reinterpret_cast<float*>(p.out) + oo + d;
      if (W == 4) *reinterpret_cast<float4*>(dst) = make_float4(acc[4 * v], acc[4 * v + 1], acc[4 * v + 2], acc[4 * v + 3]);
      else *reinterpret_cast<float2*>(dst) = make_float2(acc[0], acc[1]);
    }
  }
}
cudaError_t launch_combine_few(int head_dim, const PrefillParams& p, cudaStream_t st) {
  const dim3 grid((p.n_cols * p.n_heads + 7) / 8);
  switch (head_dim) {
    case 256: return launch_pdl(pa_combine_few_kernel<256>, grid, dim3(256), 0, st, p);
    case 128: return launch_pdl(pa_combine_few_kernel<128>, grid, dim3(256), 0, st, p);
    default: return launch_pdl(pa_combine_few_kernel<64>, grid, dim3(256), 0, st, p);
  }
}

// Key splits of a prefill call.  One CTA per (128 columns, head) leaves most of the chip idle when a short prompt follows
// a long context (203 columns of 24 heads behind 9001: 48 CTAs of 73 tiles on 148 SMs, a third of the rate of three ways
// split).  The count is the one with the least estimated makespan, in units of 64 keys' time (0.6 us): a CTA costs its keys and
// about 8 more for its start and end, equal CTAs run in whole waves, CTAs of a causal triangle (heavy ones first) pack;
// a split call adds the merge launch (6) and its records' way through L2 (1 KB each, about 3 TB/s both ways).
uint32_t prefill_splits(uint32_t pos, uint32_t n_cols, uint32_t n_heads, uint32_t head_dim, uint32_t sms, size_t slots) {
  const uint32_t q_tiles = (n_cols + kPM - 1) / kPM;
  const double longest = (double)((pos + n_cols + 63) / 64), avg = (double)((pos + n_cols / 2 + 63) / 64);
  const uint64_t rows = (uint64_t)n_cols * n_heads, ctas = (uint64_t)q_tiles * n_heads;
  uint32_t best = 1;
  double best_t = 0;
  for (uint32_t ns = 1; ns <= (uint32_t)kPrefillSplits; ++ns) {
    if (ns > 1 && (rows * ns > slots || longest / ns < 4.0)) break;
    const double waves = (double)(ctas * ns) / sms;
    double t;
    if (waves <= 1.0) t = longest / ns + 8.0;
    else if (avg >= 0.8 * longest) t = ceil(waves) * (longest / ns + 8.0);
    else t = waves * (avg / ns + 8.0) + 0.5 * longest / ns;
    if (ns > 1) t += 6.0 + (double)(rows * ns) * (head_dim * 8.0) / 3.0e6 / 0.8;
    if (ns == 1 || t < 0.95 * best_t) { best = ns; best_t = t; }
  }
  return best;
}

int prefill_supported(const pa_ctx* ctx) { return ctx->cfg.head_dim == 256 || ctx->cfg.head_dim == 128 || ctx->cfg.head_dim == 64; }

template <int HD, bool SPLIT>
static cudaError_t launch_pf(const pa_layer* L, const PrefillParams& p, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_q,
                             const CUtensorMap& tm_o, const CUtensorMap& tm_q2, const CUtensorMap& tm_g, dim3 grid, cudaStream_t st) {
  static bool attr_set[64] = {};
  const int dev = L->ctx->device & 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(pa_prefill_kernel<HD, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, PfSmem<HD>::TOTAL);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  return launch_pdl(pa_prefill_kernel<HD, SPLIT>, grid, dim3(PfSmem<HD>::THREADS), (size_t)PfSmem<HD>::TOTAL, st, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, p);
}

// boxes of the K and V maps: 128 keys x 64 dims, and prefill_v_rows() keys x head_dim
uint32_t prefill_v_rows(uint32_t head_dim) { return std::min(8192u / head_dim, (uint32_t)kPN); }
cudaError_t launch_prefill(const pa_layer* L, const PrefillParams& p, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_q,
                           const CUtensorMap& tm_o, const CUtensorMap& tm_q2, const CUtensorMap& tm_g, cudaStream_t st) {
  const dim3 grid(p.n_heads, (p.n_cols + kPM - 1) / kPM, p.n_splits);
  switch (L->ctx->cfg.head_dim) {
    case 256: return p.n_splits > 1 ? launch_pf<256, true>(L, p, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, grid, st) : launch_pf<256, false>(L, p, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, grid, st);
    case 128: return p.n_splits > 1 ? launch_pf<128, true>(L, p, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, grid, st) : launch_pf<128, false>(L, p, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, grid, st);
    case 64: return p.n_splits > 1 ? launch_pf<64, true>(L, p, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, grid, st) : launch_pf<64, false>(L, p, tm_k, tm_v, tm_q, tm_o, tm_q2, tm_g, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace pa
