// Flash-attention forward for sm_100a, head_dim 128, bf16, causal or full, GQA.
//   O = softmax(Q K^T * scale [+ causal mask]) V,   LSE = log-sum-exp per query row (natural log)
// Layout [batch, seq, heads, 128] with arbitrary token/batch strides (q/k/v may be views into one
// packed qkv buffer), as in the reference API (python/paddle/nn/functional/flash_attention.py:358;
// the reference itself calls the external FA2 library: paddle/phi/kernels/gpu/flash_attn_kernel.cu:517).
//
// One CTA per NT (1 or 2) tiles of 128 queries of one head.  Warps 4t .. 4t + 3: softmax of tile t, one query row per thread
// (= one TMEM lane): tcgen05.ld S, online max / exp2 / sum with lazy rescaling of the O accumulator in TMEM, P written back to
// TMEM as packed bf16, at the end O / l through a swizzled staging tile and TMA store.  Then a TMA warp (Q once, K / V tiles
// through two 2-stage rings, 128B swizzle) and an MMA warp (S = Q K^T from shared memory, O += P V with P from TMEM).
//
// Keys are loaded 128 at a time and worked on 64 at a time: a query tile has two 64-column score buffers, so the scores of
// step u + 1 are in TMEM before the softmax of step u ends.  P(u) is written over S(u); the MMAs of a tile are issued in the order
//   QK(0, 1) | PV(0) QK(2) | PV(1) QK(3) | ...
// The first two steps are one product and one softmax step of 128 keys: the row's first reference point is the maximum of both.
// with one MMA warp for each tile, so that the two streams interleave freely.
// What bounds it: per 64 keys the MMAs of a tile take 640 cycles (8 of 48 for a 64-column S, 4 of 64 for O) and its softmax some
// 1000 (ten a column, two warps of a scheduler sharing the special-function unit), and every hand-over between them adds a
// shared-memory round trip of 150 to 200 cycles beside the softmax warps' traffic.  One MMA warp for both tiles ran two steps
// behind: of 950 cycles a step it spent 240 on waits that were long complete.  With a warp for each tile a pair of steps takes
// 1480 cycles instead of 1920.  All waits look once before they spin, and the MMA warps stay converged.
// B=1 S=4096 H=32: 128 us causal, 243 full (1074 / 1131 TFLOP/s; one MMA warp: 142 / 271; one tile per CTA with 128-key steps: 235 /
// 364); B=8 H=32/8 full 2786 -> 1836 us (1198 TFLOP/s).  Measured without gain: 128-key steps (one score buffer per tile), part of the
// exponentials as polynomials on the FMA pipe, looking at the next barrier ahead of the MMAs (7 % slower).
#include <math.h>

#include "host_utils.h"
#include "sm100_prims.cuh"

namespace pd {
namespace fa {

constexpr int BQ = 128, BKV = 128, D = 128;
constexpr int TILE_BYTES = 128 * D * 2;       // 32 KB: two 16 KB swizzled boxes of [128 rows x 64 d]
constexpr int HALF_BYTES = TILE_BYTES / 2;
constexpr int KV_STAGES = 2;

struct Params {
  int B, Sq, Sk, Hq, Hkv;
  int causal;
  float scale_log2;   // softmax scale * log2(e)
  float* lse;         // [B, Hq, Sq]
  int* status;
  // column-sparse mask (flashmask): per key column four query-row bounds {lts, lte, uts, ute}; query row r does not
  // see column c iff lts <= r < lte or uts <= r < ute.  [B, mask_heads, Sk] with mask_heads 1, Hkv or Hq; null = none.
  const int4* bounds;
  int mask_heads;
  // per 128-column key tile: {max lts, min lte, max uts, min ute} over its columns, [B, mask_heads, ceil(Sk / 128)];
  // a (query tile, key tile) pair is skipped when one of the two ranges covers every row of the query tile for every
  // column of the key tile
  const int4* tile_bounds;
};

constexpr int MAX_NT = 2;                       // query tiles per CTA
constexpr int BU = 64;                          // keys per step
constexpr int SPT = BKV / BU;                   // steps per key tile = score buffers per query tile
static_assert(KV_STAGES == 2, "score-buffer parities and the issue loop count on two stages");
constexpr int num_threads(int nt) { return (5 * nt + 1) * 32; }
constexpr int smem_bytes(int nt) { return TILE_BYTES * (nt + 2 * KV_STAGES) + 1024 + 256; }
constexpr uint32_t COL_S = 0, COL_O = 256;      // TMEM columns: S 128 per tile (two buffers), O 128 per tile

struct Barriers {
  uint64_t q_full[MAX_NT];
  uint64_t k_full[KV_STAGES], k_empty[KV_STAGES];
  uint64_t v_full[KV_STAGES], v_empty[KV_STAGES];
  uint64_t s_full[MAX_NT][2], p_full[MAX_NT][2];
  uint64_t o_prev[MAX_NT], o_done[MAX_NT];      // PV of the last step but one / of the last step is complete
  uint64_t drain[MAX_NT];
  uint32_t tmem_base;
  int abort_flag;
  int j_lo, j_hi;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// probabilities of the 32 columns in `r` -> packed bf16; their sum is added to `sum`
__device__ __forceinline__ void probs32(const uint32_t* r, uint64_t scale2, uint64_t neg_m2, uint64_t (&sum)[2], uint32_t* pk) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float a, b;
    unpack_f32x2(fma2(f32x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), scale2, neg_m2), a, b);
    a = fast_exp2(a);
    b = fast_exp2(b);
    sum[i & 1] = add2(sum[i & 1], f32x2(a, b));
    pk[i] = pack_bf16x2(a, b);
  }
}

template <int NT, bool kMask>
__global__ void __launch_bounds__(num_threads(NT), 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, Params p,
                  int head_chunk) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                               // tile t: also its output staging at the end
  uint8_t* sK = sQ + NT * TILE_BYTES;
  uint8_t* sV = sK + KV_STAGES * TILE_BYTES;
  Barriers* bars = reinterpret_cast<Barriers*>(sV + KV_STAGES * TILE_BYTES);
  volatile int* abort_flag = &bars->abort_flag;

  constexpr int kTmaWarp = 4 * NT, kMmaWarp = 4 * NT + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Block order: within a chunk of heads whose keys and values fit the L2 together, all heads of the last (for a causal
  // mask: longest) query block first, so that the short ones fill the end of the last wave.
  const int n_qblocks = (p.Sq + NT * BQ - 1) / (NT * BQ);
  const int chunk = static_cast<int>(blockIdx.x) / (head_chunk * n_qblocks);
  const int in_chunk = static_cast<int>(blockIdx.x) - chunk * head_chunk * n_qblocks;
  const int heads_here = min(head_chunk, p.B * p.Hq - chunk * head_chunk);
  const int qb = n_qblocks - 1 - in_chunk / heads_here;
  const int bh = chunk * head_chunk + in_chunk % heads_here;
  const int head = bh % p.Hq, batch = bh / p.Hq;
  const int kv_head = head / (p.Hq / p.Hkv);
  const int q0 = qb * NT * BQ;
  const int causal_off = p.Sk - p.Sq;                             // key j visible to query i iff j <= i + off
  int n_u[NT];                                                    // 64-key steps of each query tile, from key tile jbase on
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    int kv_len = p.Sk;
    if (p.causal) kv_len = min(p.Sk, q0 + (t + 1) * BQ + causal_off);
    n_u[t] = kv_len > 0 && q0 + t * BQ < p.Sq ? (kv_len + BU - 1) / BU : 0;
  }
  int jbase = 0;

  // The first loads need only the barriers, which the thread that issues them sets up: they run under the rest of the set-up (us
  // without / with: S=65 H=8 8.2 / 6.2, B=2 S=320 H=40 causal 18.5 / 16.9, B=3 S=777 H=40 49.0 / 48.1, B=8 S=700 H=32/8 70.9 / 69.8;
  // long calls alike).  With a mask the first key tile is not known yet.
  auto load_q = [&](int t) {
    if (n_u[t] == 0) return;
    mbar_expect_tx(&bars->q_full[t], TILE_BYTES);
    tma_load_4d(sQ + t * TILE_BYTES, &tmQ, &bars->q_full[t], 0, head, q0 + t * BQ, batch);
    tma_load_4d(sQ + t * TILE_BYTES + HALF_BYTES, &tmQ, &bars->q_full[t], 64, head, q0 + t * BQ, batch);
  };
  auto load_kv = [&](const CUtensorMap* tm, uint8_t* dst, uint64_t* full, int j) {
    mbar_expect_tx(full, TILE_BYTES);
    tma_load_4d(dst, tm, full, 0, kv_head, (jbase + j) * BKV, batch);
    tma_load_4d(dst + HALF_BYTES, tm, full, 64, kv_head, (jbase + j) * BKV, batch);
  };
  auto load_first = [&]() {
    load_q(0);
    load_kv(&tmK, sK, &bars->k_full[0], 0);
    if (NT == 2) load_q(NT - 1);
    load_kv(&tmV, sV, &bars->v_full[0], 0);
  };
  if (threadIdx.x == kTmaWarp * 32) {
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    for (int s = 0; s < KV_STAGES; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->k_empty[s], NT);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->v_empty[s], NT);
    }
    for (int t = 0; t < NT; ++t) {
      mbar_init(&bars->q_full[t], 1);
      for (int b = 0; b < 2; ++b) {
        mbar_init(&bars->s_full[t][b], 1);
        mbar_init(&bars->p_full[t][b], NT == 1 ? 128 : 4);
      }
      mbar_init(&bars->o_prev[t], 1);
      mbar_init(&bars->o_done[t], 1);
      mbar_init(&bars->drain[t], 1);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    if (!kMask && max(n_u[0], n_u[NT - 1]) > 0) load_first();
  }
  if (warp == kMmaWarp) tmem_alloc(&bars->tmem_base, 512);
  if (kMask && warp == 1) {
    // first and last key tile that is not masked out as a whole for both query tiles
    const int mh = p.mask_heads == 1 ? 0 : (p.mask_heads == p.Hq ? head : kv_head);
    const int tiles_k = (p.Sk + BKV - 1) / BKV;
    const int4* tb = p.tile_bounds + (static_cast<size_t>(batch) * p.mask_heads + mh) * tiles_k;
    const int n = (max(n_u[0], n_u[NT - 1]) + SPT - 1) / SPT;
    int lo = n, hi = 0;
    for (int j = lane; j < n; j += 32) {
      const int4 b = __ldg(tb + j);
      bool dead = true;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int r0 = q0 + t * BQ;
        if (SPT * j < n_u[t]) dead = dead && ((b.x <= r0 && b.y >= r0 + BQ) || (b.z <= r0 && b.w >= r0 + BQ));
      }
      if (!dead) {
        lo = min(lo, j);
        hi = max(hi, j + 1);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
      bars->j_lo = lo;
      bars->j_hi = hi;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  if (kMask) {
    jbase = bars->j_lo;
#pragma unroll
    for (int t = 0; t < NT; ++t) n_u[t] = max(0, min(n_u[t], SPT * bars->j_hi) - SPT * jbase);
  }
  const int n_kv = (max(n_u[0], n_u[NT - 1]) + SPT - 1) / SPT;

  if (warp == kTmaWarp) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && n_kv > 0) {
      bool ok = true;
      int k_armed = 1, v_armed = 1;
      if (kMask) load_first();
      for (int j = 1; j < n_kv && ok; ++j) {
        const int s = j % KV_STAGES;
        const uint32_t ph = (j / KV_STAGES) & 1;
        if (!mbar_wait(&bars->k_empty[s], ph ^ 1, abort_flag, p.status, 100 + s)) { ok = false; break; }
        load_kv(&tmK, sK + s * TILE_BYTES, &bars->k_full[s], j);
        k_armed = j + 1;
        if (!mbar_wait(&bars->v_empty[s], ph ^ 1, abort_flag, p.status, 110 + s)) { ok = false; break; }
        load_kv(&tmV, sV + s * TILE_BYTES, &bars->v_full[s], j);
        v_armed = j + 1;
      }
      if (!ok || *abort_flag) {                        // copies in flight must land before the CTA may exit
        if (n_u[0] > 0) mbar_drain(&bars->q_full[0], 0);
        if (NT == 2 && n_u[NT - 1] > 0) mbar_drain(&bars->q_full[NT - 1], 0);
        for (int j = max(0, k_armed - KV_STAGES); j < k_armed; ++j) mbar_drain(&bars->k_full[j % KV_STAGES], (j / KV_STAGES) & 1);
        for (int j = max(0, v_armed - KV_STAGES); j < v_armed; ++j) mbar_drain(&bars->v_full[j % KV_STAGES], (j / KV_STAGES) & 1);
      }
    }
    __syncwarp();
  } else if (warp >= kMmaWarp) {
    // ---------------------------------------------------------------- MMA issuers (whole warps, converged), one for each query tile
    if (n_kv > 0) {
      constexpr uint32_t idesc_qk = make_idesc(BQ, BU, false, false);
      constexpr uint32_t idesc_qk2 = make_idesc(BQ, BKV, false, false);
      constexpr uint32_t idesc_pv = make_idesc(BQ, D, false, true);
      const int t = NT == 1 ? 0 : __shfl_sync(0xffffffffu, warp - kMmaWarp, 0);
      const int n = t == 0 ? n_u[0] : n_u[NT - 1];
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint32_t s_base = tm + COL_S + t * 128, o_tmem = tm + COL_O + t * 128;
      const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ + t * TILE_BYTES), 16, 1024);
      const uint64_t k_desc = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t v_desc = make_smem_desc_sw128(smem_u32(sV), HALF_BYTES, 1024);
      bool ok = true;
      // everything but the loop over pairs of key tiles is unrolled: stage and buffer are constants, so a descriptor is a base
      // plus an immediate.  Scores of step u into buffer b = u % SPT, keys in stage s; the stage is waited for at its first step.
      auto issue_qk = [&](int s, int b, int u, uint32_t parity) -> bool {
        if (b == 0 && !mbar_wait_warp(&bars->k_full[s], parity, abort_flag, p.status, 210 + s)) return false;
        tc_fence_after();
        const uint64_t kd = k_desc + s * (TILE_BYTES >> 4) + b * (BU * 128 >> 4);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = ((ks >> 2) * HALF_BYTES + (ks & 3) * 32) >> 4;
          umma_bf16_ss_if(leader, s_base + b * BU, q_desc + off, kd + off, idesc_qk, ks != 0 ? 1u : 0u);
        }
        umma_commit_if(leader, &bars->s_full[t][b]);
        if (b == SPT - 1 || u == n - 1) umma_commit_if(leader, &bars->k_empty[s]);    // this tile's last use of the stage
        return true;
      };
      // a key tile that only the other query tile works on: hand its stage back once it has arrived
      auto pass = [&](uint64_t* full, uint64_t* empty, uint32_t parity, int site) -> bool {
        if (!mbar_wait_warp(full, parity, abort_flag, p.status, site)) return false;
        mbar_arrive_warp(empty);
        return true;
      };
      if (NT == 1 || n > 0) {
        // the first two steps in one product of 128 columns (512 cycles, two of 64 take 768)
        ok = mbar_wait_warp(&bars->q_full[t], 0, abort_flag, p.status, 200 + t) &&
             mbar_wait_warp(&bars->k_full[0], 0, abort_flag, p.status, 210);
        if (ok) {
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = ((ks >> 2) * HALF_BYTES + (ks & 3) * 32) >> 4;
            umma_bf16_ss_if(leader, s_base, q_desc + off, k_desc + off, idesc_qk2, ks != 0 ? 1u : 0u);
          }
          umma_commit_if(leader, &bars->s_full[t][0]);
          if (n > 1) umma_commit_if(leader, &bars->s_full[t][1]);
          umma_commit_if(leader, &bars->k_empty[0]);
        }
      } else {
        ok = pass(&bars->k_full[0], &bars->k_empty[0], 0, 240);
      }
#pragma unroll 1
      for (int j0 = 0; j0 < n_kv && ok; j0 += KV_STAGES) {
        const uint32_t ph = (j0 / KV_STAGES) & 1;
#pragma unroll
        for (int s = 0; s < KV_STAGES; ++s) {
          const int j = j0 + s;
          const uint32_t ph_next = s == 0 ? ph : ph ^ 1;                              // of key tile j + 1, in the other stage
          if (!ok || j >= n_kv) continue;
          if (NT == 1 || j * SPT < n) {
            ok = mbar_wait_warp(&bars->v_full[s], ph, abort_flag, p.status, 230 + s);
#pragma unroll
            for (int b = 0; b < SPT; ++b) {
              const int u = j * SPT + b;
              if (!ok || u >= n) continue;
              if (!mbar_wait_warp(&bars->p_full[t][b], s & 1, abort_flag, p.status, 220 + t)) { ok = false; continue; }
              tc_fence_after();
              const uint64_t vd = v_desc + s * (TILE_BYTES >> 4) + b * (BU * 128 >> 4);
#pragma unroll
              for (int ks = 0; ks < BU / 16; ++ks)
                umma_bf16_ts_if(leader, o_tmem, s_base + b * BU + ks * 8, vd + ks * (2048 >> 4), idesc_pv, (u | ks) != 0 ? 1u : 0u);
              if (u == n - 2) umma_commit_if(leader, &bars->o_prev[t]);
              if (u == n - 1) umma_commit_if(leader, &bars->o_done[t]);
              if (b == SPT - 1 || u == n - 1) umma_commit_if(leader, &bars->v_empty[s]);
              if (u + SPT < n) ok = issue_qk(s ^ 1, b, u + SPT, ph_next);
            }
          } else {
            ok = pass(&bars->v_full[s], &bars->v_empty[s], ph, 250);
          }
          if (NT > 1 && ok && j + 1 < n_kv && (j + 1) * SPT >= n) ok = pass(&bars->k_full[s ^ 1], &bars->k_empty[s ^ 1], ph_next, 240);
        }
      }
      if (!ok) {
        umma_commit_if(leader, &bars->drain[t]);
        mbar_drain(&bars->drain[t], 0);
      }
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- softmax + epilogue (the first four warps: tile 0, the next four: tile 1)
    const int t = warp >> 2;
    const int row = threadIdx.x & 127;           // query row within the tile == TMEM lane
    const int qi = q0 + t * BQ + row;
    const int n_t = t == 0 ? n_u[0] : n_u[NT - 1];
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t o_tmem = tmem + lane_base + COL_O + t * 128;
    const uint64_t scale2 = f32x2(p.scale_log2, p.scale_log2);
    float m_used = -INFINITY;
    uint64_t sum[2] = {f32x2(0.f, 0.f), f32x2(0.f, 0.f)};
    bool ok = true;
    // the scores of step u from TMEM; hidden keys become -inf, which contributes exp2(-inf) = 0
    auto load_scores = [&](int u, uint32_t (&r)[BU / 32][32]) {
#pragma unroll
      for (int c = 0; c < BU / 32; ++c) tmem_ld_32x32(tmem + lane_base + COL_S + t * 128 + (u % SPT) * BU + c * 32, r[c]);
    };
    auto hide = [&](int u, uint32_t (&r)[BU / 32][32]) {
      const int col0 = jbase * BKV + u * BU;       // first key column of this step
      int col_limit = p.Sk - 1 - col0;             // highest visible key column (local to this step) for this row
      if (p.causal) col_limit = min(col_limit, qi + causal_off - col0);
      if (__any_sync(0xffffffffu, col_limit < BU - 1)) {
#pragma unroll
        for (int c = 0; c < BU / 32; ++c) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (c * 32 + i > col_limit) r[c][i] = 0xff800000u;
          }
        }
      }
      if (kMask) {
        // every lane of the warp reads the same address: one broadcast transaction per column
        const int mh = p.mask_heads == 1 ? 0 : (p.mask_heads == p.Hq ? head : kv_head);
        const int4* bnd = p.bounds + (static_cast<size_t>(batch) * p.mask_heads + mh) * p.Sk + col0;
        const int cols = min(BU, p.Sk - col0);
#pragma unroll
        for (int c = 0; c < BU / 32; ++c) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (c * 32 + i < cols) {
              const int4 b4 = __ldg(bnd + c * 32 + i);
              if ((qi >= b4.x && qi < b4.y) || (qi >= b4.z && qi < b4.w)) r[c][i] = 0xff800000u;
            }
          }
        }
      }
    };
    // row maximum in four chains of three-operand maxima
    auto row_max = [&](const uint32_t (&r)[BU / 32][32]) {
      float mxs[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t* v = &r[c * (BU / 4) / 32][c * (BU / 4) % 32];
        mxs[c] = fmaxf(__uint_as_float(v[0]), __uint_as_float(v[1]));
#pragma unroll
        for (int i = 2; i < BU / 4; i += 2) mxs[c] = max3(mxs[c], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      }
      return fmaxf(max3(mxs[0], mxs[1], mxs[2]), mxs[3]);
    };
    // probabilities of step u over its scores
    auto write_probs = [&](int u, const uint32_t (&r)[BU / 32][32]) {
      const float m_eff = (m_used == -INFINITY) ? 0.f : m_used;
      const uint64_t neg_m2 = f32x2(-m_eff, -m_eff);
#pragma unroll
      for (int c = 0; c < BU / 32; ++c) {
        uint32_t pk[16];
        probs32(r[c], scale2, neg_m2, sum, pk);
        tmem_st_32x16(tmem + lane_base + COL_S + t * 128 + (u % SPT) * BU + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      if (NT == 1) mbar_arrive(&bars->p_full[t][u % SPT]);    // one tile alone: 2 % faster without the warp-wide step
      else mbar_arrive_warp(&bars->p_full[t][u % SPT]);       // two: 128 arrivals one by one hold up the other tile's waits (252 / 241 us)
    };
    int u = 0;
    if (n_t > 1) {
      // The first reference point is the maximum of 128 keys, not of 64: it stays for most rows, and the closer it is to the
      // row's maximum, the more of the large probabilities are near 1, which bf16 holds exactly.  Relative error of O against
      // 64 bits with 64 / 128 keys: S=130 H=40 0.00224 / 0.00217, B=4 S=1024 H=40 causal 0.002055 / 0.002039, S=4096 H=32
      // causal 0.002111 / 0.002098; time 8.2 / 8.2, 65.6 / 67.6, 122.8 / 126.8 us.
      // Both buffers' first phases are observed here: a later wait for the second phase of one would pass over a first that is missing.
      ok = mbar_wait_warp2(&bars->s_full[t][0], &bars->s_full[t][1], 0, abort_flag, p.status, 302 + t);
      if (ok) {
        tc_fence_after();
        uint32_t r0[BU / 32][32], r1[BU / 32][32];
        load_scores(0, r0);
        load_scores(1, r1);
        tmem_ld_wait();
        hide(0, r0);
        hide(1, r1);
        m_used = fmaxf(row_max(r0), row_max(r1)) * p.scale_log2;
        write_probs(0, r0);
        write_probs(1, r1);
      }
      u = SPT;
    }
#pragma unroll 1
    for (; u < n_t && ok; ++u) {
      if (!mbar_wait_warp(&bars->s_full[t][u % SPT], (u / SPT) & 1, abort_flag, p.status, 300 + t)) { ok = false; break; }
      tc_fence_after();
      uint32_t r[BU / 32][32];
      load_scores(u, r);
      tmem_ld_wait();
      hide(u, r);
      const float mx = row_max(r);
      const float m_new = fmaxf(m_used, mx * p.scale_log2);
      // lazy rescale: only when some row of the warp moved its maximum by more than 2^8
      if (__any_sync(0xffffffffu, (u == 0) || (m_new - m_used > 8.f))) {
        const float factor = (m_used == -INFINITY) ? 0.f : fast_exp2(m_used - m_new);
        m_used = m_new;
        sum[0] = mul2(sum[0], f32x2(factor, factor));
        sum[1] = mul2(sum[1], f32x2(factor, factor));
        if (u > 0) {
          // O holds steps 0 .. u - 1 once PV of step u - 1 is complete, and S of step u + 1 was issued right behind that
          ok = u + 1 < n_t ? mbar_wait_warp(&bars->s_full[t][(u + 1) % SPT], ((u + 1) / SPT) & 1, abort_flag, p.status, 310 + t)
                           : mbar_wait_warp(&bars->o_prev[t], 0, abort_flag, p.status, 312 + t);
          if (!ok) break;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 8; ++c) {
            uint32_t o[16];
            tmem_ld_32x16(o_tmem + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
            tmem_st_32x16(o_tmem + c * 16, o);
          }
        }
      }
      write_probs(u, r);
    }
    float l0, l1, l2, l3;
    unpack_f32x2(sum[0], l0, l1);
    unpack_f32x2(sum[1], l2, l3);
    const float l = (l0 + l1) + (l2 + l3);
    // ---- epilogue: O / l -> bf16 -> swizzled staging (this tile's Q buffer) -> TMA store; LSE
    const bool rows_live = q0 + t * BQ < p.Sq;
    if (ok && n_t > 0) ok = mbar_wait_warp(&bars->o_done[t], 0, abort_flag, p.status, 320 + t);
    uint8_t* stage = sQ + t * TILE_BYTES;
    if (ok && rows_live) {
      tc_fence_after();
      const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
      const int sw = row & 7;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        if (n_t > 0) {
          tmem_ld_32x32(o_tmem + c * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        uint8_t* row_ptr = stage + (c >> 1) * HALF_BYTES + row * 128;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          uint4 v;
          v.x = pack_bf16x2(__uint_as_float(r[8 * jj + 0]) * inv_l, __uint_as_float(r[8 * jj + 1]) * inv_l);
          v.y = pack_bf16x2(__uint_as_float(r[8 * jj + 2]) * inv_l, __uint_as_float(r[8 * jj + 3]) * inv_l);
          v.z = pack_bf16x2(__uint_as_float(r[8 * jj + 4]) * inv_l, __uint_as_float(r[8 * jj + 5]) * inv_l);
          v.w = pack_bf16x2(__uint_as_float(r[8 * jj + 6]) * inv_l, __uint_as_float(r[8 * jj + 7]) * inv_l);
          *reinterpret_cast<uint4*>(row_ptr + ((((c & 1) * 4 + jj) ^ sw) << 4)) = v;
        }
      }
      if (qi < p.Sq && p.lse != nullptr) {
        const float lse = (l > 0.f) ? (m_used * 0.6931471805599453f + logf(l)) : -INFINITY;
        p.lse[(static_cast<size_t>(batch) * p.Hq + head) * p.Sq + qi] = lse;
      }
      fence_proxy_async_smem();
    }
    named_bar_sync(1 + t, 128);
    if (ok && rows_live && row == 0) {
      tma_store_4d(&tmO, stage, 0, head, q0 + t * BQ, batch);
      tma_store_4d(&tmO, stage + HALF_BYTES, 64, head, q0 + t * BQ, batch);
      tma_commit_group();
      tma_wait_group<0>();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
}

// 4-D map over [B, S, H, 128] bf16 with element strides (token, batch); box = {64, 1, 128 rows, 1}
static bool make_map(CUtensorMap* m, const void* ptr, int B, int S, int H, int64_t tok_stride,
                     int64_t batch_stride) {
  uint64_t dims[4] = {static_cast<uint64_t>(D), static_cast<uint64_t>(H), static_cast<uint64_t>(S),
                      static_cast<uint64_t>(B)};
  uint64_t strides[3] = {static_cast<uint64_t>(D) * 2, static_cast<uint64_t>(tok_stride) * 2,
                         static_cast<uint64_t>(batch_stride) * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  return encode_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int NT, bool kMask>
static int launch(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmO,
                  const Params& p, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_fwd_kernel<NT, kMask>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(NT)) != cudaSuccess)
      return kErrCuda;
    configured = true;
  }
  // heads whose keys and values (half the 126 MB L2, with room for the other operands) are worked on together
  const int64_t heads = static_cast<int64_t>(p.B) * p.Hq;
  int64_t chunk = (int64_t(48) << 20) / (static_cast<int64_t>(p.Sk) * D * 2 * 2) * (p.Hq / p.Hkv);
  chunk = chunk < 1 ? 1 : (chunk > heads ? heads : chunk);
  const int64_t blocks = static_cast<int64_t>((p.Sq + NT * BQ - 1) / (NT * BQ)) * heads;
  // With a causal mask every chunk starts with long blocks; in a grid of a few waves a last chunk would start them when the
  // others are done, so there all heads form one chunk (S = 4096, H = 32: 167 -> 149 us; more blocks gained nothing).
  if (p.causal && blocks <= 4 * sm_count()) chunk = heads;
  if (blocks > INT32_MAX) return kErrTooLarge;
  flash_fwd_kernel<NT, kMask><<<static_cast<unsigned>(blocks), num_threads(NT), smem_bytes(NT), stream>>>(
      tmQ, tmK, tmV, tmO, p, static_cast<int>(chunk));
  return cudaGetLastError() == cudaSuccess ? kLaunchOk : kErrCuda;
}

}  // namespace fa
}  // namespace pd

// q: [B, Sq, Hq, 128], k/v: [B, Sk, Hkv, 128], o: [B, Sq, Hq, 128] (bf16; strides in elements, head
// stride must be 128), lse: [B, Hq, Sq] fp32.  bounds: optional int32 [B, mask_heads, Sk, 4] column-sparse mask
// (see Params::bounds; python/paddle/nn/functional/flash_attention.py:1299 `flashmask_attention`).
PD_EXPORT int pd_flash_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Sq,
                                int Sk, int Hq, int Hkv, int64_t q_tok, int64_t q_batch, int64_t k_tok,
                                int64_t k_batch, int64_t v_tok, int64_t v_batch, int64_t o_tok, int64_t o_batch,
                                float scale, int causal, const void* bounds, const void* tile_bounds, int mask_heads,
                                int* status, cudaStream_t stream) {
  using namespace pd;
  using namespace pd::fa;
  if (bounds != nullptr && (mask_heads != 1 && mask_heads != Hq && mask_heads != Hkv)) return kErrBadShape;
  if (bounds != nullptr && (!aligned16(bounds) || tile_bounds == nullptr || !aligned16(tile_bounds))) return kErrAlignment;
  if (B <= 0 || Sq <= 0 || Sk <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0) return kErrBadShape;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return kErrAlignment;
  if ((q_tok % 8) || (k_tok % 8) || (v_tok % 8) || (o_tok % 8) || (q_batch % 8) || (k_batch % 8) ||
      (v_batch % 8) || (o_batch % 8))
    return kErrAlignment;
  CUtensorMap tmQ, tmK, tmV, tmO;
  if (!make_map(&tmQ, q, B, Sq, Hq, q_tok, q_batch) || !make_map(&tmK, k, B, Sk, Hkv, k_tok, k_batch) ||
      !make_map(&tmV, v, B, Sk, Hkv, v_tok, v_batch) || !make_map(&tmO, o, B, Sq, Hq, o_tok, o_batch))
    return kErrTensorMap;
  Params p{B, Sq, Sk, Hq, Hkv, causal, scale * 1.4426950408889634f, lse, status, static_cast<const int4*>(bounds),
           mask_heads, static_cast<const int4*>(tile_bounds)};
  // One or two query tiles per CTA, by an estimate of the time in us: a step of 64 keys takes 0.72 with one tile and 1.0 with two,
  // a CTA 4 more for its set-up and output (measured at S = 512 .. 4096), and the CTAs of an SM follow one another: whole waves
  // without a mask, with a causal one (long blocks first) the longest block or the average load.  One tile / two tiles: H=8 S=2048
  // causal 31 / 39, full 32 / 43 us; H=40 S=1000 34 / 27, 52 / 46; B=4 S=512 H=16/4 22 / 19, 26 / 21; H=32 S=4096 189 / 129, 327 / 242.
  auto estimate = [&](int nt, double step_us) {
    const double n = (Sq + nt * BQ - 1) / (nt * BQ), waves = n * B * Hq / sm_count(), full = step_us * ((Sk + BU - 1) / BU);
    return causal ? fmax(full + 4, waves * (full * (n + 1) / (2 * n) + 4)) : ceil(waves) * (full + 4);
  };
  const bool two = estimate(2, 1.0) < estimate(1, 0.72);
  if (two) return bounds != nullptr ? launch<2, true>(tmQ, tmK, tmV, tmO, p, stream) : launch<2, false>(tmQ, tmK, tmV, tmO, p, stream);
  return bounds != nullptr ? launch<1, true>(tmQ, tmK, tmV, tmO, p, stream) : launch<1, false>(tmQ, tmK, tmV, tmO, p, stream);
}
