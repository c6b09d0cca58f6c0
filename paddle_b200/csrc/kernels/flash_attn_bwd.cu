// Flash-attention backward for sm_100a, head_dim 128, bf16, causal or full, GQA.
// (Reference: the external FA2 library behind paddle/phi/kernels/gpu/flash_attn_grad_kernel.cu:317.)
//
// One CTA owns a 128-row K/V tile of one kv head and walks over the query heads of its group and the
// 64-row query sub-tiles that can see it.  Every GEMM has M = 128 = the kv rows of the tile, so the
// per-row softmax threads coincide with TMEM lanes and P^T / dS^T feed the next GEMMs straight from
// TMEM (no shared-memory round trip):
//   (1) S^T  = K  Q_t^T          SS   N = 64      (2) dP^T = V dO_t^T          SS   N = 64
//   softmax warps: P^T = exp2(S^T*c - LSE), dS^T = P^T o (dP^T - Delta) * scale  -> TMEM (bf16) + smem
//   (3) dV  += P^T  dO_t         TS   N = 128     (4) dK  += dS^T Q_t           TS   N = 128
//   (5) dQ_t^T = K^T dS_t^T      SS   N = 64  -> added to an fp32 dQ accumulator in global memory by 4 extra warps
// dK / dV stay in TMEM for the whole walk and are written once.
// (The scale goes into dS before it is rounded to bf16.  Applied in fp32 at the end instead, dQ and dK were 0.3 % further from 64
// bits over 24 draws of S = 130 .. 1024: where in a binade the large values fall decides it, and it costs nothing here.)
// TMEM columns:
//   dK 0-127 | dV 128-255 | work buffer A 256-383 | work buffer B 384-511
// A work buffer holds S^T (cols 0-63) and dP^T (64-127) of one query sub-tile; the softmax warps write P^T and dS^T (packed
// bf16) over the S^T columns they read themselves, and GEMM (5) later puts dQ^T over dP^T.  Sub-tiles alternate between A and
// B, so GEMMs (1),(2) of sub-tile t+1 run on the tensor cores while the softmax warps work on sub-tile t, and GEMMs (3)-(5)
// of t overlap the softmax of t+1.  The per-column LSE / Delta values are staged in shared memory by a warp of their own and read
// as broadcasts.
// Warps: 0-3 softmax of query columns 0-31 (+ final dK/dV store), 12-15 softmax of query columns
// 32-63 (the element-wise work needs no exchange between the halves: the log-sum-exp is an input), 4-7 dQ drain, 8 TMA
// producer, 9 MMA issuer, 10 statistics (11 only fills the warpgroup that gives registers away).
// What bounds it: a sub-tile takes some 2150 cycles.  The five GEMMs are 1664 of them (24 MMAs of 48, 8 of 64; the 64-column ones
// run at the full shared-memory rate), and the dQ additions keep their warps busy for 1800: the L2 takes the 32 KB of a sub-tile
// from every SM in 1400 at best, as plain additions or as TMA reductions.  The next step would be two CTAs that add their dQ^T up
// before it goes to memory.  B=1 S=4096 H=32, whole call (dO o O and the dQ conversion included): causal 663 -> 395 us, full 1089
// -> 687 us (1001 TFLOP/s); B=2 S=1999 H=32/8 causal 529 -> 230, full 649 -> 395 us; S=2048 H=8 134 -> 74; S=1024 H=8/2, whose 16
// (key tile, kv head) pairs are shared by four CTAs each, 186 -> 68 us.
// The rest was latency in the softmax warps, which a trace of their steps showed: a look at a barrier or a broadcast read costs 150
// to 200 cycles each beside the MMAs, so all three barriers of a sub-tile are looked at together and dP^T is read with S^T; a warp of
// its own stages the statistics, where a store and a 256-thread barrier stood in front of every sub-tile (438 -> 395 us causal);
// MMAs issued from a one-lane branch and waits of three steps came before that.  (1) and (2) issued by a warp of their own: 2 % slower.
// Long calls run at the power cap (990 W, 1600 MHz), where shared-memory traffic costs as much as cycles: sub-tiles of 128 queries, which
// run every MMA at its full rate but read dS^T from shared memory for (4), took 416 / 734 us (causal / full) against 397 / 702.
// The dQ accumulator is [B, Hq, Sq, 128], so the 64 additions of a thread share one address; it is cleared by the kernel that makes
// Delta, and the conversion is launched ahead of this kernel's end: forward and backward of B=2 S=1999 H=32/8 599 -> 591 us, of B=1
// S=4096 H=32 causal 625 -> 619 (the layout alone 397 -> 394 and 221 -> 218 for the backward call).
#include <math.h>

#include "host_utils.h"
#include "sm100_prims.cuh"

namespace pd {
namespace fab {

constexpr int BKV = 128, BQ = 64, D = 128;
constexpr int KV_TILE = BKV * D * 2;          // 32 KB (two 16 KB boxes)
constexpr int KV_HALF = KV_TILE / 2;
constexpr int Q_TILE = BQ * D * 2;            // 16 KB (two 8 KB boxes)
constexpr int Q_HALF = Q_TILE / 2;
constexpr int STAGES = 4;
constexpr int DS_BYTES = BKV * BQ * 2;        // 16 KB
constexpr int NUM_THREADS = 512;
constexpr int STATS_BYTES = 2 * 128 * 4;         // [2][lse2 x64 | delta x64]
constexpr int SMEM_BYTES = 2 * KV_TILE + STAGES * 2 * Q_TILE + 2 * DS_BYTES + STATS_BYTES + 1024 + 256;
constexpr uint32_t COL_DK = 0, COL_DV = 128, COL_BUF = 256;
// inside a 128-column work buffer; P^T and dS^T of query half h at OFF_PT + 32 h and OFF_DST + 32 h
constexpr uint32_t OFF_ST = 0, OFF_DPT = 64, OFF_PT = 0, OFF_DST = 16, OFF_DQT = 64;

struct Barriers {
  uint64_t kv_full;
  uint64_t qdo_full[STAGES], qdo_empty[STAGES];
  uint64_t st_full[2], dp_full[2], pds_full[2], stat_full[2], dq_full[2], dq_empty[2], dkv_full, drain;
  uint32_t tmem_base;
  int abort_flag;
};

struct Params {
  int B, Sq, Sk, Hq, Hkv, causal;
  float scale, scale_log2;
  const float* lse;     // [B, Hq, Sq] natural log
  const float* delta;   // [B, Hq, Sq]
  float* dq_acc;        // [B, Hq, Sq, 128], added into
  int parts;            // CTAs that share the query heads of a group; with more than one each writes its own fp32 sums
  float* dkv_part;      // [parts, 2, B, Sk, Hkv, 128]: dK and dV of each part
  int* status;
  const int4* bounds;   // column-sparse mask, as in the forward kernel: [B, mask_heads, Sk] of {lts, lte, uts, ute}
  int mask_heads;
  const int4* tile_bounds;   // [B, mask_heads, ceil(Sk / 128)] of {max lts, min lte, max uts, min ute}
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void red_add_f32(float* p, float v) {
  asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

template <bool kMask>
__global__ void __launch_bounds__(NUM_THREADS, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                 const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                 const __grid_constant__ CUtensorMap tmDK,
                 const __grid_constant__ CUtensorMap tmDV, Params p, int head_chunk) {
  pdl_wait();                                        // Delta and the cleared dQ sums, should this ever start under the kernel that makes them
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + KV_TILE;
  uint8_t* sQ = sV + KV_TILE;                       // STAGES x [Q tile | dO tile]
  uint8_t* sDS = sQ + STAGES * 2 * Q_TILE;
  float* stats = reinterpret_cast<float*>(sDS + 2 * DS_BYTES);
  Barriers* bars = reinterpret_cast<Barriers*>(sDS + 2 * DS_BYTES + STATS_BYTES);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Block order: within a chunk of heads whose operands share the L2, all heads of the first key tile (for a causal mask:
  // the longest walk) first, so that the short walks fill the end of the last wave.
  const int n_jb = (p.Sk + BKV - 1) / BKV;
  const int part = static_cast<int>(blockIdx.x) % p.parts, unit = static_cast<int>(blockIdx.x) / p.parts;
  const int chunk = unit / (head_chunk * n_jb);
  const int in_chunk = unit - chunk * head_chunk * n_jb;
  const int heads_here = min(head_chunk, p.B * p.Hkv - chunk * head_chunk);
  const int jb = in_chunk / heads_here;
  const int bh = chunk * head_chunk + in_chunk % heads_here;
  const int kv_head = bh % p.Hkv, batch = bh / p.Hkv;
  const int group = p.Hq / p.Hkv / p.parts;               // query heads this CTA walks over, from qh0 on
  const int qh0 = kv_head * group * p.parts + part * group;
  const int kv0 = jb * BKV;
  const int causal_off = p.Sk - p.Sq;
  const int n_sub = (p.Sq + BQ - 1) / BQ;
  int t0 = 0;
  if (p.causal) {
    const int first_q = kv0 - causal_off;            // first query row that sees kv row kv0
    t0 = first_q > 0 ? first_q / BQ : 0;
  }
  int t1 = n_sub;
  if (kMask && p.mask_heads != p.Hq) {
    // query sub-tiles outside [t0, t1) are masked as a whole for every column of this key tile: rows from max lts on
    // when the lower range is open-ended, rows below min ute when the upper range starts at row 0.  (With one mask per
    // query head the range would differ between the heads this CTA walks, so it is not narrowed then.)
    const int mh = p.mask_heads == 1 ? 0 : kv_head;
    const int4 tb = __ldg(p.tile_bounds + (static_cast<size_t>(batch) * p.mask_heads + mh) * n_jb + jb);
    if (tb.y >= p.Sq) t1 = min(t1, (max(tb.x, 0) + BQ - 1) / BQ);
    if (tb.z <= 0) t0 = max(t0, min(tb.w, p.Sq) / BQ);
  }
  const int per_head = t1 > t0 ? t1 - t0 : 0;
  const int n_it = per_head * group;

  if (threadIdx.x == 0) {
    pdl_trigger();                                   // after pdl_wait above; the conversion of dQ waits for this kernel before it reads
    mbar_init(&bars->kv_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->qdo_full[s], 1);
      mbar_init(&bars->qdo_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->st_full[b], 1);
      mbar_init(&bars->dp_full[b], 1);
      mbar_init(&bars->pds_full[b], 8);
      mbar_init(&bars->stat_full[b], 1);
      mbar_init(&bars->dq_full[b], 1);
      mbar_init(&bars->dq_empty[b], 4);
    }
    mbar_init(&bars->dkv_full, 1);
    mbar_init(&bars->drain, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 9) tmem_alloc(&bars->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;

  // 512 threads x 128 registers at launch = softmax 256 x 168 + drain 128 x 104 + issuers 128 x 72
  if (warp >= 8 && warp < 12) {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
   if (warp == 8) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      prefetch_tmap(&tmQ);
      prefetch_tmap(&tmDO);
      mbar_expect_tx(&bars->kv_full, 2 * KV_TILE);
      tma_load_4d(sK, &tmK, &bars->kv_full, 0, kv_head, kv0, batch);
      tma_load_4d(sK + KV_HALF, &tmK, &bars->kv_full, 64, kv_head, kv0, batch);
      tma_load_4d(sV, &tmV, &bars->kv_full, 0, kv_head, kv0, batch);
      tma_load_4d(sV + KV_HALF, &tmV, &bars->kv_full, 64, kv_head, kv0, batch);
      bool ok = true;
      int issued = 0, qh = qh0, tq = 0;
      for (int it = 0; it < n_it && ok; ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!mbar_wait(&bars->qdo_empty[s], ph ^ 1, abort_flag, p.status, 100 + s)) { ok = false; break; }
        const int q0 = (t0 + tq) * BQ;
        uint8_t* dst = sQ + s * 2 * Q_TILE;
        mbar_expect_tx(&bars->qdo_full[s], 2 * Q_TILE);
        tma_load_4d(dst, &tmQ, &bars->qdo_full[s], 0, qh, q0, batch);
        tma_load_4d(dst + Q_HALF, &tmQ, &bars->qdo_full[s], 64, qh, q0, batch);
        tma_load_4d(dst + Q_TILE, &tmDO, &bars->qdo_full[s], 0, qh, q0, batch);
        tma_load_4d(dst + Q_TILE + Q_HALF, &tmDO, &bars->qdo_full[s], 64, qh, q0, batch);
        issued = it + 1;
        if (++tq == per_head) tq = 0, ++qh;
      }
      if (!ok || *abort_flag || n_it == 0) {
        mbar_drain(&bars->kv_full, 0);
        for (int it = max(0, issued - STAGES); it < issued; ++it)
          mbar_drain(&bars->qdo_full[it % STAGES], (it / STAGES) & 1);
      }
    }
    __syncwarp();
   } else if (warp == 9) {
    // ---------------------------------------------------------------- MMA issuer (the whole warp, converged)
    if (n_it > 0) {
      constexpr uint32_t idesc_s = make_idesc(BKV, BQ, false, false);   // (1),(2)
      constexpr uint32_t idesc_kv = make_idesc(BKV, D, false, true);    // (3),(4)  A from TMEM
      constexpr uint32_t idesc_dq = make_idesc(D, BQ, true, true);      // (5)
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t k_desc = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t v_desc = make_smem_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t q_desc = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t kt_desc = make_smem_desc_sw128(smem_u32(sK), KV_HALF, 1024);     // K as an MN-major operand
      const uint64_t qt_desc = make_smem_desc_sw128(smem_u32(sQ), Q_HALF, 1024);
      const uint64_t ds_desc = make_smem_desc_sw128(smem_u32(sDS), 16, 1024);
      bool ok = mbar_wait_warp(&bars->kv_full, 0, abort_flag, p.status, 200);
      int s_next = 0;                                    // ring stage and phase of the next sub-tile to start
      uint32_t s_ph = 0;
      // S^T only needs P^T / dS^T of the buffer's previous use to be consumed, which the issue order gives; dP^T goes over
      // dQ^T, which has to be drained first: S^T hides that wait
      auto issue_s = [&](int it) -> bool {
        if (!mbar_wait_warp(&bars->qdo_full[s_next], s_ph, abort_flag, p.status, 210 + s_next)) return false;
        tc_fence_after();
        const uint64_t qd = q_desc + s_next * (2 * Q_TILE >> 4), dod = qd + (Q_TILE >> 4);
        const uint32_t buf = tm + COL_BUF + (it & 1) * 128;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t offa = ((ks >> 2) * KV_HALF + (ks & 3) * 32) >> 4, offb = ((ks >> 2) * Q_HALF + (ks & 3) * 32) >> 4;
          umma_bf16_ss_if(leader, buf + OFF_ST, k_desc + offa, qd + offb, idesc_s, ks != 0 ? 1u : 0u);
        }
        umma_commit_if(leader, &bars->st_full[it & 1]);
        if (!mbar_wait_warp(&bars->dq_empty[it & 1], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 230 + (it & 1))) return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t offa = ((ks >> 2) * KV_HALF + (ks & 3) * 32) >> 4, offb = ((ks >> 2) * Q_HALF + (ks & 3) * 32) >> 4;
          umma_bf16_ss_if(leader, buf + OFF_DPT, v_desc + offa, dod + offb, idesc_s, ks != 0 ? 1u : 0u);
        }
        umma_commit_if(leader, &bars->dp_full[it & 1]);
        if (++s_next == STAGES) s_next = 0, s_ph ^= 1;
        return true;
      };
      if (ok) ok = issue_s(0);
      int s = 0;
#pragma unroll 1
      for (int it = 0; it < n_it && ok; ++it) {
        const int b = it & 1;
        // S^T / dP^T of the NEXT sub-tile go to the other buffer now: they run while the softmax warps work
        if (it + 1 < n_it) {
          if (!issue_s(it + 1)) { ok = false; break; }
        }
        const uint64_t qd = qt_desc + s * (2 * Q_TILE >> 4), dod = qd + (Q_TILE >> 4);
        const uint64_t dsd = ds_desc + b * (DS_BYTES >> 4);
        const uint32_t buf = tm + COL_BUF + b * 128;
        if (!mbar_wait_warp(&bars->pds_full[b], (it >> 1) & 1, abort_flag, p.status, 220 + b)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < BKV / 16; ++ks)  // (5) dQ^T = K^T dS^T  (over this buffer's dP^T, already consumed); first, so
                                               // that its drain runs under (3) and (4)
          umma_bf16_ss_if(leader, buf + OFF_DQT, kt_desc + ks * (2048 >> 4), dsd + ks * (2048 >> 4), idesc_dq, ks != 0 ? 1u : 0u);
        umma_commit_if(leader, &bars->dq_full[b]);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)   // (3) dV += P^T dO
          umma_bf16_ts_if(leader, tm + COL_DV, buf + OFF_PT + (ks >> 1) * 32 + (ks & 1) * 8, dod + ks * (2048 >> 4), idesc_kv,
                          (it | ks) != 0 ? 1u : 0u);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)   // (4) dK += dS^T Q
          umma_bf16_ts_if(leader, tm + COL_DK, buf + OFF_DST + (ks >> 1) * 32 + (ks & 1) * 8, qd + ks * (2048 >> 4), idesc_kv,
                          (it | ks) != 0 ? 1u : 0u);
        umma_commit_if(leader, &bars->qdo_empty[s]);
        if (++s == STAGES) s = 0;
      }
      if (ok) umma_commit_if(leader, &bars->dkv_full);
      else {
        umma_commit_if(leader, &bars->drain);
        mbar_drain(&bars->drain, 0);
      }
    }
    __syncwarp();
   } else if (warp == 10) {
    // ---------------------------------------------------------------- statistics: -LSE (log2 units) and -Delta * scale of a sub-tile's
    // queries -> shared memory, fetched one sub-tile ahead.  The softmax warps are done with a buffer when they have handed
    // over the P^T / dS^T made with it.
    const size_t row0 = static_cast<size_t>(batch) * p.Hq * p.Sq;
    int qh = qh0, tq = 0;
    float v[4];                                          // rows lane, lane + 32 of both
    auto load = [&]() {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const size_t at = row0 + static_cast<size_t>(qh) * p.Sq + min((t0 + tq) * BQ + lane + 32 * i, p.Sq - 1);
        v[i] = __ldg(p.lse + at);
        v[2 + i] = __ldg(p.delta + at);
      }
    };
    if (n_it > 0) load();
#pragma unroll 1
    for (int it = 0; it < n_it; ++it) {
      const int b = it & 1, q0 = (t0 + tq) * BQ;
      if (!mbar_wait_warp(&bars->pds_full[b], ((it >> 1) & 1) ^ 1, abort_flag, p.status, 260 + b)) break;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = lane + 32 * i;
        const bool live = q0 + r < p.Sq;
        stats[b * 128 + r] = live ? v[i] * -1.4426950408889634f : -INFINITY;     // -inf -> p = 0 for padded rows
        stats[b * 128 + 64 + r] = live ? -v[2 + i] * p.scale : 0.f;
      }
      mbar_arrive_warp(&bars->stat_full[b]);
      if (++tq == per_head) tq = 0, ++qh;
      if (it + 1 < n_it) load();
    }
    __syncwarp();
   }
  } else if (warp < 4 || warp >= 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    // ---------------------------------------------------------------- softmax warps: thread = kv row x column half
    // a warp may touch the TMEM lanes of its own quarter (warp index mod 4) only
    const int h = warp < 4 ? 0 : 1;                                 // query columns [32 h, 32 h + 32) of the sub-tile
    const int row = (warp & 3) * 32 + lane;
    const int kvi = kv0 + row;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int sw = row & 7;
    const uint64_t scale2 = f32x2(p.scale_log2, p.scale_log2), dscale2 = f32x2(p.scale, p.scale);
    bool ok = true;
    int qh_next = qh0, tq_next = 0;
#pragma unroll 1
    for (int it = 0; it < n_it; ++it) {
      const int qh = qh_next;
      const int q0 = (t0 + tq_next) * BQ;
      if (++tq_next == per_head) tq_next = 0, ++qh_next;
      const int b = it & 1;
      const uint32_t ph = (it >> 1) & 1;
      // one look at all three; S^T and dP^T are issued a sub-tile ahead
      const bool seen = mbar_try_wait(&bars->st_full[b], ph) & mbar_try_wait(&bars->dp_full[b], ph) & mbar_try_wait(&bars->stat_full[b], ph);
      if (!__all_sync(0xffffffffu, seen)) {
        ok = mbar_wait_warp(&bars->st_full[b], ph, abort_flag, p.status, 300 + b) &&
             mbar_wait_warp(&bars->stat_full[b], ph, abort_flag, p.status, 302 + b) &&
             mbar_wait_warp(&bars->dp_full[b], ph, abort_flag, p.status, 304 + b);
        if (!ok) break;
      }
      tc_fence_after();
      const float* st = stats + b * 128 + h * 32;
      // visible iff kv <= q + off  <=>  q_local >= kvi - off - q0
      // A padded key row (of a last key tile, filled with zeros) is seen by no query: its score 0 against the row's log-sum-exp
      // overflows when all real scores are far below 0 (or the query sees no key), and 0 * inf would reach dQ
      const int first_visible = kvi >= p.Sk ? BQ : (p.causal ? kvi - causal_off - q0 : 0);
      // this thread's key column carries its own masked query-row ranges (made local to the sub-tile here)
      int4 b4 = make_int4(0, 0, 0, 0);
      if (kMask && kvi < p.Sk) {
        const int mh = p.mask_heads == 1 ? 0 : (p.mask_heads == p.Hq ? qh : kv_head);
        b4 = __ldg(p.bounds + (static_cast<size_t>(batch) * p.mask_heads + mh) * p.Sk + kvi);
        b4.x -= q0; b4.y -= q0; b4.z -= q0; b4.w -= q0;
      }
      const uint32_t buf = tmem + lane_base + COL_BUF + b * 128;
      // A half's outputs go over its own S^T columns, so the halves need no agreement
      uint8_t* row_ptr = sDS + b * DS_BYTES + row * 128;
      float pv[32];
      uint32_t dp_r[32];
      {
        uint32_t s_r[32], pk[16];
        tmem_ld_32x32(buf + OFF_ST + h * 32, s_r);
        tmem_ld_32x32(buf + OFF_DPT + h * 32, dp_r);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 nl = *reinterpret_cast<const float4*>(st + 4 * c);          // - LSE
          float x0, x1, x2, x3;
          unpack_f32x2(fma2(f32x2(__uint_as_float(s_r[4 * c]), __uint_as_float(s_r[4 * c + 1])), scale2, f32x2(nl.x, nl.y)), x0, x1);
          unpack_f32x2(fma2(f32x2(__uint_as_float(s_r[4 * c + 2]), __uint_as_float(s_r[4 * c + 3])), scale2, f32x2(nl.z, nl.w)), x2, x3);
          pv[4 * c] = fast_exp2(x0);
          pv[4 * c + 1] = fast_exp2(x1);
          pv[4 * c + 2] = fast_exp2(x2);
          pv[4 * c + 3] = fast_exp2(x3);
        }
        if (kMask || __any_sync(0xffffffffu, first_visible > h * 32)) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const int ql = h * 32 + c;
            if (ql < first_visible || (kMask && ((ql >= b4.x && ql < b4.y) || (ql >= b4.z && ql < b4.w)))) pv[c] = 0.f;
          }
        }
#pragma unroll
        for (int c = 0; c < 32; c += 2) pk[c >> 1] = pack_bf16x2(pv[c], pv[c + 1]);
        tmem_st_32x16(buf + OFF_PT + h * 32, pk);
      }
      {
        uint32_t pk[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 nd = *reinterpret_cast<const float4*>(st + 64 + 4 * c);     // - Delta * scale
          float d0, d1, d2, d3;
          unpack_f32x2(mul2(fma2(f32x2(__uint_as_float(dp_r[4 * c]), __uint_as_float(dp_r[4 * c + 1])), dscale2, f32x2(nd.x, nd.y)),
                            f32x2(pv[4 * c], pv[4 * c + 1])), d0, d1);
          unpack_f32x2(mul2(fma2(f32x2(__uint_as_float(dp_r[4 * c + 2]), __uint_as_float(dp_r[4 * c + 3])), dscale2, f32x2(nd.z, nd.w)),
                            f32x2(pv[4 * c + 2], pv[4 * c + 3])), d2, d3);
          pk[2 * c] = pack_bf16x2(d0, d1);
          pk[2 * c + 1] = pack_bf16x2(d2, d3);
        }
        tmem_st_32x16(buf + OFF_DST + h * 32, pk);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          *reinterpret_cast<uint4*>(row_ptr + (((h * 4 + jj) ^ sw) << 4)) =
              make_uint4(pk[4 * jj], pk[4 * jj + 1], pk[4 * jj + 2], pk[4 * jj + 3]);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive_warp(&bars->pds_full[b]);
    }
    // ---- final (first softmax warpgroup): dK, dV (fp32 in TMEM) -> bf16 -> swizzled staging (Q/dO ring is idle now)
    // -> TMA store
    if (h == 0 && ok && n_it > 0) ok = mbar_wait_warp(&bars->dkv_full, 0, abort_flag, p.status, 310);
    if (p.parts > 1) {
      // several CTAs share this key tile: each stores its fp32 sums, each warpgroup one of dK / dV; dkv_convert_kernel adds the
      // parts up in a fixed order, so dK / dV are the same on every run
      if (h == 1 && ok && n_it > 0) ok = mbar_wait_warp(&bars->dkv_full, 0, abort_flag, p.status, 312);
      if (ok) {
        tc_fence_after();
        const size_t kv_rows = static_cast<size_t>(p.B) * p.Sk * p.Hkv;
        float* dst = p.dkv_part + ((part * 2 + h) * kv_rows + (static_cast<size_t>(batch) * p.Sk + min(kvi, p.Sk - 1)) * p.Hkv + kv_head) * D;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          if (n_it > 0) {
            tmem_ld_32x32(tmem + lane_base + (h == 0 ? COL_DK : COL_DV) + c * 32, r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = 0u;
          }
          if (kvi < p.Sk) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              *reinterpret_cast<uint4*>(dst + c * 32 + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
          }
          __syncwarp();
        }
      }
    } else {
      if (h == 0) named_bar_sync(3, 128);
      if (h == 0 && ok) {
        tc_fence_after();
  #pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          uint8_t* stage = sQ + which * KV_TILE;
  #pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            if (n_it > 0) {
              tmem_ld_32x32(tmem + lane_base + (which == 0 ? COL_DK : COL_DV) + c * 32, r);
              tmem_ld_wait();
            } else {
  #pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0u;
            }
            uint8_t* row_ptr = stage + (c >> 1) * KV_HALF + row * 128;
  #pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[8 * jj + 0]), __uint_as_float(r[8 * jj + 1]));
              v.y = pack_bf16x2(__uint_as_float(r[8 * jj + 2]), __uint_as_float(r[8 * jj + 3]));
              v.z = pack_bf16x2(__uint_as_float(r[8 * jj + 4]), __uint_as_float(r[8 * jj + 5]));
              v.w = pack_bf16x2(__uint_as_float(r[8 * jj + 6]), __uint_as_float(r[8 * jj + 7]));
              *reinterpret_cast<uint4*>(row_ptr + ((((c & 1) * 4 + jj) ^ sw) << 4)) = v;
            }
          }
        }
        fence_proxy_async_smem();
      }
      if (h == 0) named_bar_sync(3, 128);
      if (h == 0 && ok && threadIdx.x == 0) {
        tma_store_4d(&tmDK, sQ, 0, kv_head, kv0, batch);
        tma_store_4d(&tmDK, sQ + KV_HALF, 64, kv_head, kv0, batch);
        tma_store_4d(&tmDV, sQ + KV_TILE, 0, kv_head, kv0, batch);
        tma_store_4d(&tmDV, sQ + KV_TILE + KV_HALF, 64, kv_head, kv0, batch);
        tma_commit_group();
        tma_wait_group<0>();
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    // ---------------------------------------------------------------- dQ drain warps (4..7): thread = d
    // A warp adds 32 neighbouring floats of one query row per instruction, straight from registers.  Through a staging tile
    // and a TMA reduction the same bytes crossed shared memory twice, next to MMAs that use its whole bandwidth, for the
    // same rate: the L2 takes the 32 KB of a sub-tile from every SM in 0.8 us either way.
    const int dr = threadIdx.x - 128;                 // 0..127 = head-dim index = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    constexpr int row_stride = D;                     // rows of a head lie one behind the other: all additions share one address
    int qh = qh0, tq = 0;
#pragma unroll 1
    for (int it = 0; it < n_it; ++it) {
      if (!mbar_wait_warp(&bars->dq_full[it & 1], (it >> 1) & 1, abort_flag, p.status, 400 + (it & 1))) break;
      tc_fence_after();
      uint32_t r0[32], r1[32];
      tmem_ld_32x32(tmem + lane_base + COL_BUF + (it & 1) * 128 + OFF_DQT, r0);
      tmem_ld_32x32(tmem + lane_base + COL_BUF + (it & 1) * 128 + OFF_DQT + 32, r1);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive_warp(&bars->dq_empty[it & 1]);
      const int q0 = (t0 + tq) * BQ;
      float* dst = p.dq_acc + ((static_cast<size_t>(batch) * p.Hq + qh) * p.Sq + q0) * D + dr;
      const int live = p.Sq - q0;                     // rows of this sub-tile inside the matrix
      if (live >= BQ) {
#pragma unroll
        for (int c = 0; c < 32; ++c) red_add_f32(dst + c * row_stride, __uint_as_float(r0[c]));
#pragma unroll
        for (int c = 0; c < 32; ++c) red_add_f32(dst + (32 + c) * row_stride, __uint_as_float(r1[c]));
      } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (c < live) red_add_f32(dst + c * row_stride, __uint_as_float(r0[c]));
          if (32 + c < live) red_add_f32(dst + (32 + c) * row_stride, __uint_as_float(r1[c]));
        }
      }
      if (++tq == per_head) tq = 0, ++qh;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

// delta[b, h, s] = sum_d dO * O, and the row of the dQ accumulator is cleared: 16 lanes of 16 bytes per row, so two rows per warp, and four such pairs in flight (with one
// row of 8-byte loads per warp the 67 MB of S = 4096, H = 32 took 26 us)
constexpr int DELTA_ROWS = 4;
__global__ void __launch_bounds__(256) delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                                    float* __restrict__ delta, float* __restrict__ dq_acc, int64_t rows, int S, int H, int64_t o_tok,
                                                    int64_t o_batch, int64_t do_tok, int64_t do_batch) {
  const int64_t first = (static_cast<int64_t>(blockIdx.x) * 16 + (threadIdx.x >> 4)) * DELTA_ROWS;
  const int c = (threadIdx.x & 15) * 8;
  uint4 a[DELTA_ROWS], g[DELTA_ROWS];
  int64_t at[DELTA_ROWS];
#pragma unroll
  for (int k = 0; k < DELTA_ROWS; ++k) {
    const int64_t w = min(first + k, rows - 1);
    const int64_t bs = w / H;
    const int h = static_cast<int>(w - bs * H);
    const int64_t b = bs / S;
    const int s = static_cast<int>(bs - b * S);
    a[k] = *reinterpret_cast<const uint4*>(o + b * o_batch + s * o_tok + h * D + c);
    g[k] = *reinterpret_cast<const uint4*>(d_o + b * do_batch + s * do_tok + h * D + c);
    at[k] = (b * H + h) * S + s;
  }
#pragma unroll
  for (int k = 0; k < DELTA_ROWS; ++k) {
    if (first + k < rows) {
      float4* z = reinterpret_cast<float4*>(dq_acc + at[k] * D) + (threadIdx.x & 15);
      z[0] = z[16] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int k = 0; k < DELTA_ROWS; ++k) {
    const uint32_t u[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, v[4] = {g[k].x, g[k].y, g[k].z, g[k].w};
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc = fmaf(__uint_as_float(u[i] << 16), __uint_as_float(v[i] << 16), acc);
      acc = fmaf(__uint_as_float(u[i] & 0xffff0000u), __uint_as_float(v[i] & 0xffff0000u), acc);
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 15) == 0 && first + k < rows) delta[at[k]] = acc;
  }
}

// dq (bf16, [B, S, H, 128] with token / batch strides) = dq_acc (fp32 [B, H, S, 128]); 16 threads of 8 values per row
__global__ void __launch_bounds__(256) dq_convert_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int64_t rows,
                                                         int S, int H, int64_t tok, int64_t batch) {
  pdl_wait();
  const int64_t first = (static_cast<int64_t>(blockIdx.x) * 16 + (threadIdx.x >> 4)) * 2;
  const int c = (threadIdx.x & 15) * 8;
  float4 v[2][2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float4* p = reinterpret_cast<const float4*>(src + min(first + k, rows - 1) * D + c);
    v[k][0] = p[0];
    v[k][1] = p[1];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int64_t row = first + k;
    if (row >= rows) break;
    const int64_t bh = row / S, s = row - bh * S;
    const int64_t b = bh / H;
    const int h = static_cast<int>(bh - b * H);
    *reinterpret_cast<uint4*>(dst + b * batch + s * tok + static_cast<int64_t>(h) * D + c) =
        make_uint4(pack_bf16x2(v[k][0].x, v[k][0].y), pack_bf16x2(v[k][0].z, v[k][0].w), pack_bf16x2(v[k][1].x, v[k][1].y),
                   pack_bf16x2(v[k][1].z, v[k][1].w));
  }
}

// dk, dv (blockIdx.y = 0, 1; bf16, token / batch strides) = the sum of the parts in their order; 16 threads of 8 values per row
__global__ void __launch_bounds__(256) dkv_convert_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dk,
                                                          __nv_bfloat16* __restrict__ dv, int parts, int64_t rows, int S, int H,
                                                          int64_t dk_tok, int64_t dk_batch, int64_t dv_tok, int64_t dv_batch) {
  const int which = blockIdx.y;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 16 + (threadIdx.x >> 4);
  if (row >= rows) return;
  const int c = (threadIdx.x & 15) * 8;
  const float* p = src + (which * rows + row) * D + c;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int k = 0; k < parts; ++k, p += 2 * rows * D) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
  }
  const int64_t bs = row / H;
  const int h = static_cast<int>(row - bs * H);
  const int64_t b = bs / S, s = bs - b * S;
  __nv_bfloat16* dst = which == 0 ? dk + b * dk_batch + s * dk_tok : dv + b * dv_batch + s * dv_tok;
  *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(h) * D + c) =
      make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

static bool make_map_bf16(CUtensorMap* m, const void* ptr, int B, int S, int H, int64_t tok, int64_t batch,
                          uint32_t rows) {
  uint64_t dims[4] = {D, static_cast<uint64_t>(H), static_cast<uint64_t>(S), static_cast<uint64_t>(B)};
  uint64_t strides[3] = {D * 2, static_cast<uint64_t>(tok) * 2, static_cast<uint64_t>(batch) * 2};
  uint32_t box[4] = {64, 1, rows, 1};
  return encode_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace fab
}  // namespace pd

// Number of CTAs that should share a (key tile, kv head): the query heads of a group are walked one after the other, so few kv
// heads leave the GPU idle or its last wave empty.  Costs in us, measured: 1.45 per 64-row sub-tile, 3 per CTA, and with more than
// one part the fp32 sums of dK / dV (written and read for each part, converted: 8 parts + 2 bytes per element at 6.6 TB/s, a launch).
// Without a mask whole waves count; with a causal one the longest walk or the average load.  The sums of the parts take no more
// memory than the fp32 accumulator of dQ, or 64 MB.  (Added into one accumulator by reductions instead, the same shapes take as long
// up to S = 4096, S = 8192 H = 16/1 702 instead of 735 us, but dK / dV differed from run to run.)
PD_EXPORT int pd_flash_attn_bwd_parts(int B, int Sq, int Sk, int Hq, int Hkv, int causal) {
  using namespace pd::fab;
  if (B <= 0 || Sq <= 0 || Sk <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0) return 1;
  const int group = Hq / Hkv;
  const double sms = pd::sm_count(), units = static_cast<double>(B) * Hkv * ((Sk + BKV - 1) / BKV), n_sub = (Sq + BQ - 1) / BQ;
  const double kv_elems = 2.0 * B * Sk * Hkv * D, most = fmax(4.0 * B * Sq * Hq * D, 64e6);
  int best = 1;
  double best_cost = 0;
  for (int parts = 1; parts <= group; ++parts) {
    if (group % parts != 0 || (parts > 1 && 4.0 * kv_elems * parts > most)) continue;
    const double walk = 1.45 * n_sub * group / parts + 3.0, waves = units * parts / sms;
    const double cost = walk * (causal ? fmax(1.0, 0.5 * waves) : ceil(waves)) + (parts > 1 ? (8.0 * parts + 2) * kv_elems / 6.6e6 + 6.0 : 0.0);
    if (parts == 1 || cost < 0.97 * best_cost) {
      best = parts;
      best_cost = cost;
    }
  }
  return best;
}

// dkv_part: null, or fp32 scratch [parts, 2, B, Sk, Hkv, 128] for `parts` (a divisor of Hq / Hkv) > 1 CTAs per key tile.
// dq_acc: fp32 scratch [B, Hq, Sq, 128], 16-byte aligned; delta: fp32 [B, Hq, Sq] scratch;
// dq/dk/dv: bf16 outputs [B, S, H, 128] with their own token / batch strides (e.g. views of a packed dqkv).  
PD_EXPORT int pd_flash_attn_bwd(const void* d_o, const void* q, const void* k, const void* v, const void* o,
                                const float* lse, float* delta, float* dq_acc, float* dkv_part, void* dq, void* dk,
                                void* dv, int B, int Sq, int Sk, int Hq, int Hkv, int64_t q_tok, int64_t q_batch,
                                int64_t k_tok, int64_t k_batch, int64_t v_tok, int64_t v_batch, int64_t o_tok,
                                int64_t o_batch, int64_t do_tok, int64_t do_batch, int64_t dq_tok, int64_t dq_batch,
                                int64_t dk_tok, int64_t dk_batch, int64_t dv_tok, int64_t dv_batch, float scale, int causal,
                                const void* bounds, const void* tile_bounds, int mask_heads, int parts, int* status,
                                cudaStream_t stream) {
  using namespace pd;
  using namespace pd::fab;
  if (B <= 0 || Sq <= 0 || Sk <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0) return kErrBadShape;
  if (parts < 1 || (Hq / Hkv) % parts != 0 || (parts > 1 && dkv_part == nullptr)) return kErrBadShape;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o) || !aligned16(d_o) || !aligned16(dkv_part) || !aligned16(dq_acc)) return kErrAlignment;
  if ((q_tok % 8) || (k_tok % 8) || (v_tok % 8) || (o_tok % 8) || (do_tok % 8)) return kErrAlignment;
  CUtensorMap tmQ, tmDO, tmK, tmV, tmDK, tmDV;
  bool ok = make_map_bf16(&tmQ, q, B, Sq, Hq, q_tok, q_batch, BQ) &&
            make_map_bf16(&tmDO, d_o, B, Sq, Hq, do_tok, do_batch, BQ) &&
            make_map_bf16(&tmK, k, B, Sk, Hkv, k_tok, k_batch, BKV) &&
            make_map_bf16(&tmV, v, B, Sk, Hkv, v_tok, v_batch, BKV) &&
            make_map_bf16(&tmDK, dk, B, Sk, Hkv, dk_tok, dk_batch, BKV) &&
            make_map_bf16(&tmDV, dv, B, Sk, Hkv, dv_tok, dv_batch, BKV);
  if (!ok) return kErrTensorMap;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(flash_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
      return kErrCuda;
    configured = true;
  }
  const int64_t rows = static_cast<int64_t>(B) * Sq * Hq;
  delta_kernel<<<static_cast<unsigned>((rows + 16 * DELTA_ROWS - 1) / (16 * DELTA_ROWS)), 256, 0, stream>>>(
      (const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, delta, dq_acc, rows, Sq, Hq, o_tok, o_batch, do_tok, do_batch);
  if (bounds != nullptr && (mask_heads != 1 && mask_heads != Hq && mask_heads != Hkv)) return kErrBadShape;
  if (bounds != nullptr && (!aligned16(bounds) || tile_bounds == nullptr || !aligned16(tile_bounds))) return kErrAlignment;
  Params p{B, Sq, Sk, Hq, Hkv, causal, scale, scale * 1.4426950408889634f, lse, delta, dq_acc, parts, dkv_part, status,
           static_cast<const int4*>(bounds), mask_heads, static_cast<const int4*>(tile_bounds)};
  // kv heads whose operands (q, dO in bf16, dQ in fp32; k, v) share the L2: about 48 MB of them
  const int64_t head_bytes = static_cast<int64_t>(Sq) * (Hq / Hkv) * D * 8 + static_cast<int64_t>(Sk) * D * 4;
  const int64_t heads = static_cast<int64_t>(B) * Hkv;
  int64_t chunk = (int64_t(48) << 20) / head_bytes;
  chunk = chunk < 1 ? 1 : (chunk > heads ? heads : chunk);
  // With a causal mask every chunk starts with long walks; in a grid of a few waves a last chunk would start them when the
  // others are done, so there all heads form one chunk (B = 2, S = 1999, H = 32/8: 373 -> 258 us for the whole call).
  if (causal && (Sk + BKV - 1) / BKV * heads <= 4 * sm_count()) chunk = heads;
  const int64_t grid64 = (Sk + BKV - 1) / BKV * heads * parts;
  if (grid64 > INT32_MAX) return kErrTooLarge;
  const unsigned grid = static_cast<unsigned>(grid64);
  if (bounds != nullptr) flash_bwd_kernel<true><<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(tmQ, tmDO, tmK, tmV, tmDK, tmDV, p, static_cast<int>(chunk));
  else flash_bwd_kernel<false><<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(tmQ, tmDO, tmK, tmV, tmDK, tmDV, p, static_cast<int>(chunk));
  if (cudaGetLastError() != cudaSuccess) return kErrCuda;
  const int rc = launch_pdl(dq_convert_kernel, dim3(static_cast<unsigned>((rows + 31) / 32)), dim3(256), 0, stream, 1, dq_acc,
                            (__nv_bfloat16*)dq, rows, Sq, Hq, dq_tok, dq_batch);
  if (rc != kLaunchOk) return rc;
  if (parts > 1) {
    const int64_t kv_rows = static_cast<int64_t>(B) * Sk * Hkv;
    dkv_convert_kernel<<<dim3(static_cast<unsigned>((kv_rows + 15) / 16), 2), 256, 0, stream>>>(
        dkv_part, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, parts, kv_rows, Sk, Hkv, dk_tok, dk_batch, dv_tok, dv_batch);
  }
  return cudaGetLastError() == cudaSuccess ? kLaunchOk : kErrCuda;
}
