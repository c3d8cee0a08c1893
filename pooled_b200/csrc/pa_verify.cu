// Attention of a block of a few tokens (an accepted token and its drafts, checked together) on the 5th-generation tensor
// cores: one CTA per (split of the KV sequence, kv head); the rows of its tile are the (column, head of the GQA group) pairs,
// at most 64 of them, and it writes an unnormalised (o, m, l) record per row for the LSE combine.
//
//   warps 0, 3  TMA producers: K tiles and V tiles (64 x head_dim f16, 128-byte swizzle), a ring of three and of two slots
//   warp 1      MMA issuer (one thread) of the scores: S = Q K^T into one of three TMEM tiles (128 x 64 f32)
//   warp 2      allocates / frees tensor memory, and in between is the MMA issuer of O += P V into the TMEM
//               accumulator (128 x head_dim f32).  Both A operands come from tensor memory (the lower half of Q sits there for the
//               CTA's life, P is written over its own S tile); completion is signalled to mbarriers with tcgen05.commit
//   warps 4-11  two softmax groups on alternate KV tiles: thread r of a group owns row r (TMEM lane r): its Q row into TMEM and
//               shared memory as f16 pairs, then per tile tcgen05.ld of its S row, causal mask, running max / sum,
//               P = 2^(s - m) as f16 pairs back into TMEM (tcgen05.st), and the record.  A row's reference maximum travels with
//               the tiles from group to group through shared memory; each group keeps its own share of the row sum
// O is rescaled only when a row's running maximum has grown by more than 2^8 since its last rescale; the rescale
// waits for the previous P V to retire and rewrites the row's TMEM accumulator.  What bounds it: HBM in the loop, and the chain
// of rotation, staging of the query rows and merge around it.
//
// Stands in for attn_dec of pooled in its k-token verify use (engine/wgsl/attn_dec.js:67-200).
#include "pa_tc.cuh"

namespace pa {


constexpr int kBM = 128;   // query rows per CTA
constexpr int kBN = 64;    // keys per tile

// MODE 2 keeps about 22 bits of q and of the softmax weights at no extra tensor work: even rows carry the f16 high parts
// (q_hi, P_hi), odd rows the low parts (q_lo, P_lo) of the same query row, so the two sit in neighbouring lanes of one warp:
// S_hi + S_lo is one shuffle per score in the softmax, O_hi + O_lo one per output in the epilogue, and the split writes a
// single record per query row.  MODE 1: single f16 operands.
template <int HD, int MODE>
struct VfSmem {
  static constexpr int SBUF = 3;                    // S / P tiles in tensor memory
  // three K slots (the scores run two tiles ahead) and two V slots, which leaves 32 KB free so that the CTAs can join SMs that
  // still run a small kernel
  static constexpr int NK = 3, NV = 2;
  static constexpr int KV_BYTES = HD * 128;         // [HD/64][64 rows][128 B]
  // tensor memory columns: the first TQC 64-dim chunks of Q (32 columns of f16 pairs each) | S tiles (64 each; P
  // overwrites the first 32 of its S) | O (HD).  HD 256: 64 + 192 + 256 = 512.
  static constexpr int TQC = HD / 128;
  static constexpr int QS_BYTES = (HD / 64 - TQC) * 128 * 128;   // the chunks of Q not in tensor memory: [chunk][128 rows][128 B]
  // softmax warpgroups, on alternate KV tiles: with one group the softmax of a tile, not the arrival of the tile from HBM, set
  // the pace of the seven-tile loop
  static constexpr int NGRP = 2;
  static constexpr int THREADS = 128 + 128 * NGRP;
  static constexpr int OFF_K = 0, OFF_V = NK * KV_BYTES, OFF_Q = (NK + NV) * KV_BYTES, OFF_BAR = OFF_Q + QS_BYTES;
  static constexpr int OFF_ROW = OFF_BAR + 256;      // per-row hand-over between the softmax groups: the reference maximum, m[128]
  static constexpr int TOTAL = 1024 + OFF_ROW + 128 * 4;
  static_assert(TOTAL <= 227 * 1024, "shared memory of one CTA");
  static constexpr int T_Q = 0, T_S = TQC * 32, T_O = TQC * 32 + SBUF * kBN;
  static_assert(T_O + HD <= 512, "tensor memory columns");
  static constexpr int TMEM_COLS = 512;
};

template <int HD, int MODE>
__global__ void __launch_bounds__(VfSmem<HD, MODE>::THREADS, 1)
pa_verify_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const PrefillParams p) {
  using L = VfSmem<HD, MODE>;
  constexpr int CH = HD / 64;
  constexpr bool PREC = MODE == 2;
  constexpr int NK = L::NK, NV = L::NV, NGRP = L::NGRP, kSBuf = L::SBUF;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + L::OFF_BAR);
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(bars + 31);
  volatile uint32_t* s_err = s_tmem + 1;
  float* s_rm = reinterpret_cast<float*>(base + L::OFF_ROW);   // [128] reference maximum of each query row (scaled, log2 units)
  // [2][128] each group's row sum and [2][128] the reference maximum it is expressed in: exchanged once, after the
  // last tile's scores exist, in the first K slot (every K tile has been multiplied by then)
  float* s_rl = reinterpret_cast<float*>(base + L::OFF_K);
  float* s_rr = s_rl + 256;
  const uint32_t bar0 = smem_u32(bars);
  enum { K_FULL = 0, K_EMPTY = 3, V_FULL = 6, V_EMPTY = 9, S_FULL = 12, P_FULL = 12 + kSBuf, PV_DONE = 12 + 2 * kSBuf, O_DONE = 12 + 3 * kSBuf,
         Q_FULL = O_DONE + 1, Q_ISSUED = O_DONE + 2, Q_SENT = O_DONE + 3,
         M_READY = O_DONE + 4 /* [2]: group g has published the row maxima after its tile */ };
  static_assert(M_READY + 2 <= 31, "barrier slots");
  uint8_t* q_s = base + L::OFF_Q;
  auto BAR = [&](int which, int idx) { return bar0 + 8u * (uint32_t)(which + idx); };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t g = blockIdx.y;
  const uint32_t tiles = (p.n_rows + kBN - 1) / kBN, tps = (tiles + p.n_splits - 1) / p.n_splits;
  const uint32_t tile0 = blockIdx.x * tps;
  if (tile0 >= tiles) return;                           // this split holds no row (uniform for the CTA)
  const uint32_t n_tiles = min(tiles, tile0 + tps) - tile0;

  if (warp == 1 && lane == 0) {
    *s_err = 0;
    for (int i = 0; i < NK; ++i) { mbar_init(BAR(K_FULL, i), 1); mbar_init(BAR(K_EMPTY, i), 1); }
    for (int i = 0; i < NV; ++i) { mbar_init(BAR(V_FULL, i), 1); mbar_init(BAR(V_EMPTY, i), 1); }
    for (int i = 0; i < kSBuf; ++i) { mbar_init(BAR(S_FULL, i), 1); mbar_init(BAR(P_FULL, i), 128); mbar_init(BAR(PV_DONE, i), 1); }
    mbar_init(BAR(O_DONE, 0), 1);
    mbar_init(BAR(Q_FULL, 0), 128 * NGRP);
    mbar_init(BAR(Q_ISSUED, 0), HD >= 256 ? 128 * NGRP : 128);   // every thread that reads the staging area, after its last read
    mbar_init(BAR(Q_SENT, 0), 128 * NGRP);
    mbar_init(BAR(M_READY, 0), 128); mbar_init(BAR(M_READY, 1), 128);
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32((const void*)s_tmem), L::TMEM_COLS);
    tmem_relinquish();
    tc_fence_before();
  }
  // q, and the rows the RoPE/append kernel before this one writes, may only be touched after pdl_wait(); the producers may fetch older K/V tiles ahead of it when the caller allows
  const bool early = p.prefetch_old_rows;
  const uint32_t old_rows = min(p.n_rows - min(p.n_rows, p.n_cols), p.early_limit);
  if (!early) pdl_wait();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const uint32_t t_q = tmem + L::T_Q, t_s0 = tmem + L::T_S, t_o = tmem + L::T_O;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer, K ----
    if (lane == 0) {
      prefetch_tmap(&tm_k);
      bool waited = !early;
      for (uint32_t j = 0; j < n_tiles; ++j) {
        const uint32_t st = j % NK, u = j / NK;
        if (!waited && (tile0 + j + 1) * kBN > old_rows) { pdl_wait(); waited = true; }
        // tile 0 may go out at once (ahead of the wait if the caller allows); the next one only when the
        // requests for the query rows are on their way (a burst of tiles would queue in front of them), and the
        // third, whose slot stages the query rows, when those have been consumed
        if (j == ((early && p.pre_stages == 0) ? 0u : 1u)) mbar_wait(BAR(Q_SENT, 0), 0, s_err, WAIT_QFULL);
        if (j == 2) mbar_wait(BAR(Q_ISSUED, 0), 0, s_err, WAIT_QFULL);
        mbar_wait(BAR(K_EMPTY, st), (u & 1) ^ 1, s_err, WAIT_EMPTY);
        mbar_expect_tx(BAR(K_FULL, st), L::KV_BYTES);
        if (p.kv_evict_first) tma_load_3d_hint(smem_u32(base + L::OFF_K + st * L::KV_BYTES), &tm_k, 0, (int)((tile0 + j) * kBN), (int)(g * CH), BAR(K_FULL, st), l2_policy_evict_first());
        else tma_load_3d(smem_u32(base + L::OFF_K + st * L::KV_BYTES), &tm_k, 0, (int)((tile0 + j) * kBN), (int)(g * CH), BAR(K_FULL, st));
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ TMA producer, V ----
    // (its own thread: behind the K loads in one loop, K(j+1) would wait for the V slot that P V (j-1) still reads)
    if (lane == 0) {
      prefetch_tmap(&tm_v);
      bool waited = !early;
      for (uint32_t j = 0; j < n_tiles; ++j) {
        const uint32_t st = j % NV, u = j / NV;
        if (!waited && (tile0 + j + 1) * kBN > old_rows) { pdl_wait(); waited = true; }
        if (j == 1) mbar_wait(BAR(Q_ISSUED, 0), 0, s_err, WAIT_QFULL);   // slot 1 stages query rows until then
        mbar_wait(BAR(V_EMPTY, st), (u & 1) ^ 1, s_err, WAIT_EMPTY);
        mbar_expect_tx(BAR(V_FULL, st), L::KV_BYTES);
        if (p.kv_evict_first) tma_load_3d_hint(smem_u32(base + L::OFF_V + st * L::KV_BYTES), &tm_v, 0, (int)((tile0 + j) * kBN), (int)(g * CH), BAR(V_FULL, st), l2_policy_evict_first());
        else tma_load_3d(smem_u32(base + L::OFF_V + st * L::KV_BYTES), &tm_v, 0, (int)((tile0 + j) * kBN), (int)(g * CH), BAR(V_FULL, st));
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer, scores ----
    // S(j) = Q K(j)^T.  The whole warp runs the loop and the elected lane issues.  Issuing blocks while the tensor
    // cores' queue is full, so one thread issuing both products of every tile spends its time in turns on each and
    // the waits in between leave the queue empty; with the scores here and P V in warp 2 there are two queues' worth
    // of work in front of the tensor cores.  S(j) goes into the TMEM tile of S(j - 3) / P(j - 3): once that P V has
    // retired (PV_DONE).
    {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_qk = umma_idesc(kBM, kBN, 0);
      // Both A operands live in tensor memory (Q for the whole CTA, P per tile), so a k-step costs shared-memory
      // bandwidth for the K or V slice only.  B descriptors are built once; a k-step adds a byte offset (>> 4).
      uint64_t k_desc[NK];
#pragma unroll
      for (int i = 0; i < NK; ++i) k_desc[i] = smem_desc(smem_u32(base + L::OFF_K + i * L::KV_BYTES), 16, 1024);
      const uint64_t q_desc = smem_desc(smem_u32(q_s), 16, 1024);
      mbar_wait(BAR(Q_FULL, 0), 0, s_err, WAIT_QFULL);
      tc_fence_after();
      for (uint32_t j = 0; j < n_tiles; ++j) {
        const uint32_t sb = j % kSBuf, st = j % NK;
        if (j >= (uint32_t)kSBuf) mbar_wait(BAR(PV_DONE, sb), ((j - kSBuf) / kSBuf) & 1, s_err, WAIT_MMA);
        mbar_wait(BAR(K_FULL, st), (j / NK) & 1, s_err, WAIT_KFULL);
        tc_fence_after();
        const uint64_t kd = st == 0 ? k_desc[0] : (st == 1 ? k_desc[1] : k_desc[NK - 1]);
        const uint32_t ts = t_s0 + sb * kBN;
        // the head dims whose Q chunks sit in tensor memory first, then those whose Q comes from shared memory
        constexpr int TS_STEPS = L::TQC * 4;
#pragma unroll
        for (int ks = 0; ks < TS_STEPS; ++ks)
          umma_f16_ts(leader, ts, t_q + ks * 8, kd + (uint64_t)(((ks >> 2) * (kBN * 128) + (ks & 3) * 32) >> 4), idesc_qk, ks > 0);
#pragma unroll
        for (int ks = TS_STEPS; ks < HD / 16; ++ks)
          umma_f16_ss(leader, ts, q_desc + (uint64_t)(((((ks - TS_STEPS) >> 2)) * (kBM * 128) + (ks & 3) * 32) >> 4),
                      kd + (uint64_t)(((ks >> 2) * (kBN * 128) + (ks & 3) * 32) >> 4), idesc_qk, ks > 0 ? 1u : 0u);
        umma_commit_elected(leader, BAR(K_EMPTY, st));
        umma_commit_elected(leader, BAR(S_FULL, sb));
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ MMA issuer, P V ----
    // O += P(j) V(j), in tile order (this thread's products retire in order, so O is always complete up to a tile)
    {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_pv = umma_idesc(kBM, HD, 1);
      uint64_t v_desc[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) v_desc[i] = smem_desc(smem_u32(base + L::OFF_V + i * L::KV_BYTES), kBN * 128, 1024);
      for (uint32_t j = 0; j < n_tiles; ++j) {
        const uint32_t sb = j % kSBuf, st = j % NV;
        mbar_wait(BAR(P_FULL, sb), (j / kSBuf) & 1, s_err, WAIT_QFULL);
        mbar_wait(BAR(V_FULL, st), (j / NV) & 1, s_err, WAIT_VFULL);
        tc_fence_after();
        const uint64_t vd = st == 0 ? v_desc[0] : (st == 1 ? v_desc[1] : v_desc[NV - 1]);
        const uint32_t tp = t_s0 + sb * kBN;     // P(j): packed f16 pairs in the first 32 columns of S(j)'s tile
#pragma unroll
        for (int ks = 0; ks < kBN / 16; ++ks)
          umma_f16_ts(leader, t_o, tp + ks * 8, vd + (uint64_t)((ks * 2048) >> 4), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
        umma_commit_elected(leader, BAR(V_EMPTY, st));
        umma_commit_elected(leader, BAR(PV_DONE, sb));
      }
      umma_commit_elected(leader, BAR(O_DONE, 0));
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax + epilogue ----
    const uint32_t wg = (warp - 4) >> 2;                 // softmax group: takes KV tiles wg, wg + NGRP, ...
    const uint32_t qd = (warp - 4) & 3, row = qd * 32 + lane;   // a warp reaches the 32 TMEM lanes of its index mod 4
    const uint32_t lane_addr = (qd * 32) << 16;
    // a (column, head-of-group) pair per row; MODE 2: per two rows (even: high parts, odd: low parts)
    const bool is_lo = PREC ? (row & 1u) != 0 : row >= 64;
    const uint32_t lr = PREC ? row >> 1 : (row & 63u);
    const uint32_t sk_c = lr / p.G, sk_hh = lr % p.G;
    const uint32_t head = g * p.G + sk_hh;
    const bool live = lr < p.n_cols * p.G && (PREC || !is_lo);
    // keys [0, lim) are visible to this row
    const uint32_t lim = (uint32_t)min(max(p.lim0 + (int32_t)min(sk_c, p.n_cols - 1), 0), (int32_t)p.n_rows);
    // m_st: the row's reference maximum (the weights of a tile are 2^(s - m_st); it moves only when a tile's maximum
    // passes it by more than 2^8).  With two softmax groups it travels with the tiles: the group that took tile j - 1
    // publishes it in s_rm, the group that takes tile j picks it up there.  l_sum: this group's share of the row sum,
    // expressed in the reference m_l.  (A split may hold no visible key of a row, hence the finite start.)
    // ---- the few query rows are fetched by all 128 threads at once, 16 bytes per request, straight into
    //      shared memory (cp.async: no registers held, every request in flight together), into the K and the V slot
    //      the producers leave alone until Q_ISSUED (32 rows each); a row's chunks are XOR-swizzled so that the
    //      per-row reads below do not all hit one bank.  (One thread loading its own 1 KB row needs the loads in register-sized batches,
    //      a memory round trip each: 4.8 us between the wait and the first MMA.) ----
    auto stage_row = [&](uint32_t pr) {
      return (pr < 32 ? base + L::OFF_K + 2 * L::KV_BYTES : base + L::OFF_V + L::KV_BYTES - (size_t)32 * (HD * 4)) + (size_t)pr * (HD * 4);
    };
    // q as f32 (this kernel splits it), as f16 (no low part), or as two f16 planes, high and low parts, which the
    // RoPE kernel of a layer call writes: then a staged row is [high HD halves][low HD halves] and nothing is left
    // to convert here (the f32 -> f16 conversions of 128 x HD elements took 3 us on four warps)
    const bool planes = p.q_f16 && p.q_lo != nullptr;
    const uint32_t q_es = p.q_f16 ? 2u : 4u, q_ch = planes ? HD * 4 / 16 : HD * q_es / 16;     // 16-byte chunks per staged row
    if (early) pdl_wait();
    pdl_trigger();
    {
      const uint32_t pairs = p.n_cols * p.G, st_tid = tid - 128, total = pairs * q_ch;
      for (uint32_t idx = st_tid; idx < total; idx += 128 * NGRP) {
        const uint32_t pr = idx / q_ch, c = idx % q_ch;
        const uint32_t half_ch = HD * 2 / 16;
        const bool lo_plane = planes && c >= half_ch;
        const uint8_t* src = reinterpret_cast<const uint8_t*>(lo_plane ? p.q_lo : p.q) +
                             ((uint64_t)(p.col0 + pr / p.G) * p.q_col_stride + (uint64_t)(g * p.G + pr % p.G) * p.q_head_stride) * q_es +
                             (uint64_t)(lo_plane ? c - half_ch : c) * 16;
        const uint32_t dst = smem_u32(stage_row(pr) + ((c ^ (pr & 7u)) << 4));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      mbar_arrive(BAR(Q_SENT, 0));
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      named_bar_sync(1, 128 * NGRP);
    }
    const uint8_t* my_stage = stage_row(lr & 63u);
    auto stage_ld = [&](uint32_t c) { return *reinterpret_cast<const uint4*>(my_stage + ((c ^ (lr & 7u)) << 4)); };
    // ---- this thread's Q row -> f16 pairs: lower half of the dims to tensor memory, upper half to shared memory ----
    {
      // ER elements per round (the loads of a round are all in flight together), in 64-dim chunks: the first TQC chunks
      // of the row go to tensor memory (32 columns each), the others to shared memory (one 128-byte row chunk each)
      constexpr int ER = HD >= 128 ? 128 : 64, ROUNDS = HD / ER, HCN = ER / 64;
#pragma unroll 1
      for (int c2 = 0; c2 < ROUNDS; ++c2) {
        // with two softmax groups each stages one round of its rows (head_dim 256); a single round is the first group's
        if (NGRP == 2 && (uint32_t)(ROUNDS == 2 ? c2 : 0) != wg) continue;
        uint32_t w[ER / 2];
        if (p.q_f16) {
#pragma unroll
          for (int i = 0; i < ER / 8; ++i) {
            const uint32_t cb = (planes && is_lo) ? HD * 2 / 16 : 0;
            const uint4 x = (live && (planes || !is_lo)) ? stage_ld(cb + c2 * (ER / 8) + i) : make_uint4(0, 0, 0, 0);   // plain f16 q has no low part
            w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
          }
        } else {
          float4 xs[ER / 4];
#pragma unroll
          for (int i = 0; i < ER / 4; ++i) {
            const uint4 r4 = live ? stage_ld(c2 * (ER / 4) + i) : make_uint4(0, 0, 0, 0);
            xs[i] = *reinterpret_cast<const float4*>(&r4);
          }
#pragma unroll
          for (int i = 0; i < ER / 4; ++i) {
            float4 x = xs[i];
            if (is_lo) {   // what the f16 high part leaves over
              x.x -= __half2float(__float2half_rn(x.x)); x.y -= __half2float(__float2half_rn(x.y));
              x.z -= __half2float(__float2half_rn(x.z)); x.w -= __half2float(__float2half_rn(x.w));
            }
            w[2 * i] = pack_h2(x.x, x.y); w[2 * i + 1] = pack_h2(x.z, x.w);
          }
        }
        if (c2 == ROUNDS - 1 || (NGRP == 2 && ROUNDS == 2)) {
          // this thread is done with the staging area (with two groups and two rounds, each thread reads one round):
          // the producers may fetch into it (and may send the tiles they held back so that the early burst would not
          // queue in front of the q requests)
          fence_proxy_async();
          mbar_arrive(BAR(Q_ISSUED, 0));
        }
#pragma unroll
        for (int hc = 0; hc < HCN; ++hc) {
          const int c = HCN * c2 + hc;
          uint32_t wc[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) wc[i] = w[32 * hc + i];
          if (c < L::TQC) {
            tmem_st32u(t_q + c * 32 + lane_addr, wc);
          } else {
            uint8_t* dst = q_s + (c - L::TQC) * (kBM * 128) + row * 128;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<uint4*>(dst + ((i ^ (row & 7)) << 4)) = make_uint4(wc[4 * i], wc[4 * i + 1], wc[4 * i + 2], wc[4 * i + 3]);
          }
        }
      }
      fence_proxy_async();
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(BAR(Q_FULL, 0));
    }
    float m_st = -1.0e30f, l_sum = 0.f, m_l = m_st;
    for (uint32_t j = wg; j < n_tiles; j += NGRP) {
      const uint32_t b = j % kSBuf, u = j / kSBuf, kv0 = (tile0 + j) * kBN;
      mbar_wait(BAR(S_FULL, b), u & 1, s_err, WAIT_MMA);
      tc_fence_after();
      float s[kBN];
      {
        float t0[32], t1[32];
        tmem_ld32(t_s0 + b * kBN + lane_addr, t0);
        tmem_ld32(t_s0 + b * kBN + 32 + lane_addr, t1);
#pragma unroll
        for (int i = 0; i < 32; ++i) { s[i] = t0[i]; s[32 + i] = t1[i]; }
      }
      if (PREC) {
        // S = S_hi + S_lo: the two rows of a query row are neighbouring lanes
#pragma unroll
        for (int i = 0; i < kBN; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], 1);
      }
      // maximum of the raw scores (the scale is positive), causal mask on tiles that reach this row's diagonal
      if (kv0 + kBN > lim) {
#pragma unroll
        for (int i = 0; i < kBN; ++i) if (kv0 + i >= lim) s[i] = -INFINITY;
      }
      float mt = s[0];
#pragma unroll
      for (int i = 1; i < kBN; ++i) mt = fmaxf(mt, s[i]);
      mt *= p.scale_log2;
      if (NGRP == 2 && j > 0) {
        mbar_wait(BAR(M_READY, (j - 1) & 1), ((j - 1) >> 1) & 1, s_err, WAIT_MMA);
        m_st = s_rm[row];
      }
      float alpha = 1.f;
      bool grow = false;
      if (mt > m_st + 8.f) { alpha = ex2_approx(m_st - mt); m_st = mt; grow = true; }
      if (NGRP == 2) {
        // hand the reference on at once: the other group's next tile needs nothing else from this one
        s_rm[row] = m_st;
        mbar_arrive(BAR(M_READY, j & 1));
      }
      if (m_st != m_l) { l_sum *= ex2_approx(m_l - m_st); m_l = m_st; }
      if (j > 0 && __any_sync(0xffffffffu, grow)) {
        // O must not change under the previous P V: wait for it, then rescale this warp's 32 rows in TMEM
        const uint32_t jb = (j - 1) % kSBuf, ju = (j - 1) / kSBuf;
        mbar_wait(BAR(PV_DONE, jb), ju & 1, s_err, WAIT_MMA);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          float o[32];
          tmem_ld32(t_o + c * 32 + lane_addr, o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= alpha;
          tmem_st32(t_o + c * 32 + lane_addr, o);
        }
      }
      // P = 2^(s - m) as packed f16 pairs over the first 32 columns of this S buffer (its scores are in registers now)
      uint32_t pw[32];
      float ls = 0.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float e0 = ex2_approx(fmaf(s[2 * i], p.scale_log2, -m_st)), e1 = ex2_approx(fmaf(s[2 * i + 1], p.scale_log2, -m_st));
        ls += e0 + e1;
        if (is_lo) { e0 -= __half2float(__float2half_rn(e0)); e1 -= __half2float(__float2half_rn(e1)); }
        pw[i] = pack_h2(e0, e1);
      }
      l_sum += ls;
      tmem_st32u(t_s0 + b * kBN + lane_addr, pw);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(BAR(P_FULL, b));
    }
    // ---- epilogue: the records ----
    if (NGRP == 2) {
      // the row sum is the two groups' shares brought to the final reference; O already is in it
      const uint32_t last = n_tiles - 1;
      mbar_wait(BAR(M_READY, last & 1), (last >> 1) & 1, s_err, WAIT_MMA);   // published after S(last) was complete: the K ring is idle
      s_rl[wg * 128 + row] = l_sum; s_rr[wg * 128 + row] = m_l;
      named_bar_sync(2, 128 * NGRP);
      const float m_fin = s_rm[row];
      l_sum = s_rl[row] * ex2_approx(s_rr[row] - m_fin) + s_rl[128 + row] * ex2_approx(s_rr[128 + row] - m_fin);
    }
    mbar_wait(BAR(O_DONE, 0), 0, s_err, WAIT_MMA);
    tc_fence_after();
    {
      // unnormalised partial (o, m, l) of this split for the LSE combine.  MODE 2: O = O_hi + O_lo, the odd lane's
      // row added to the even lane's, which writes the record (m and l are the same in both)
      const uint64_t prow = (uint64_t)(p.col0 + sk_c) * p.n_heads + head;
      const uint64_t slot = prow * p.n_splits + blockIdx.x;
      const bool writer = live && !is_lo;
      // A lane holds a row: stored as they are, the 32 lanes of an instruction would write 16 bytes each into 32
      // records 1 KB apart.  The rows go to shared memory first (the K ring is idle: every product has retired; rows
      // 16 bytes apart in their bank phase), then all 128 threads write whole records, 16 consecutive bytes per
      // thread and 512 consecutive bytes per warp instruction.
      constexpr int RP = HD / 4 + 1;                                  // row pitch in float4
      float4* xs = reinterpret_cast<float4*>(base + L::OFF_K + 2048);   // [rows][RP], behind the groups' row sums (s_rl, s_rr)
      unsigned long long* xslot = reinterpret_cast<unsigned long long*>(xs + 64 * RP);   // [64] record of each row, ~0: none
      if (!is_lo && lr < 64 && wg == 0) xslot[lr] = writer ? (unsigned long long)slot : ~0ull;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        if (NGRP == 2 && (uint32_t)(c & 1) != wg) continue;   // the groups share the columns out
        float o[32];
        tmem_ld32(t_o + c * 32 + lane_addr, o);
        if (PREC) {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] += __shfl_xor_sync(0xffffffffu, o[i], 1);
        }
        if (writer) {
#pragma unroll
          for (int i = 0; i < 8; ++i) xs[lr * RP + c * 8 + i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        }
      }
      named_bar_sync(1, 128 * NGRP);
      for (uint32_t idx = tid - 128; idx < 64 * (HD / 4); idx += 128 * NGRP) {
        const uint32_t rr = idx / (HD / 4), c4 = idx % (HD / 4);
        const unsigned long long sl = xslot[rr];
        if (sl != ~0ull) reinterpret_cast<float4*>(p.part_o + sl * HD)[c4] = xs[rr * RP + c4];
      }
      if (writer && wg == 0) { p.part_ml[slot * 2] = (NGRP == 2 ? s_rm[row] : m_st) * 0.6931471805599453f; p.part_ml[slot * 2 + 1] = l_sum; }
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

template <int HD, int MODE>
static cudaError_t launch_vf(const pa_layer* L, const PrefillParams& p, const CUtensorMap& tm_k, const CUtensorMap& tm_v, dim3 grid, cudaStream_t st) {
  using S = VfSmem<HD, MODE>;
  static bool attr_set[64] = {};
  const int dev = L->ctx->device & 63;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(pa_verify_kernel<HD, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  return launch_pdl(pa_verify_kernel<HD, MODE>, grid, dim3(S::THREADS), (size_t)S::TOTAL, st, tm_k, tm_v, p);
}

// k-token verify block (more than 8 query rows per kv head) on the tensor cores
cudaError_t launch_verify(const pa_layer* L, const PrefillParams& p, const CUtensorMap& tm_k, const CUtensorMap& tm_v, uint32_t n_kv, cudaStream_t st) {
  const dim3 grid(p.n_splits, n_kv);
  const bool precise = !(L->ctx->cfg.flags & PA_FLAG_FAST);
  if (L->ctx->cfg.head_dim == 256)
    return precise ? launch_vf<256, 2>(L, p, tm_k, tm_v, grid, st) : launch_vf<256, 1>(L, p, tm_k, tm_v, grid, st);
  return precise ? launch_vf<128, 2>(L, p, tm_k, tm_v, grid, st) : launch_vf<128, 1>(L, p, tm_k, tm_v, grid, st);
}

}  // namespace pa
