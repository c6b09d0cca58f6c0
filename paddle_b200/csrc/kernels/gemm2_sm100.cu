// Two-SM (cta_group::2) variant of the persistent bf16 GEMM for sm_100a:  C[M,N] (=|+=) op(A)[M,K] * op(B)[K,N]
//
// A cluster of two CTAs (one SM pair) owns a 256 x TN output tile: TN = 256, for products whose tiles all run at once 128, for deep ones
// 512 (tile_n below).  An accumulator holds ACC_N = min(TN, 256) columns; a 512-column tile is two of them side by side.  CTA r of the
// pair loads rows [128 r, 128 r + 128) of the A tile and, of each accumulator's columns, [ACC_N / 2 r, ACC_N / 2 (r + 1)) of the B tile
// into ITS OWN shared memory (plain per-CTA TMA loads, no cluster multicast); the tensor core reads the other half of B from the
// partner SM.  A 64-deep K block fills 32 KB of each SM with TN = 256 (six stages), 24 KB with 128 (eight stages), 48 KB with 512
// (four stages: A 16 KB, B 16 KB for each accumulator); the 128 x 256 single-CTA tile takes 48 KB.  One thread of the leader CTA
// (cluster rank 0; its MMA warp stays converged and predicates the instruction: with a one-lane branch the same tiles took 4 to 12 %
// longer, 4096 x 11008 x 4096 with B transposed 258 against 228 us) issues tcgen05.mma.cta_group::2 (M = 256, N = ACC_N, K = 16); the
// accumulator rows 0-127 live in the leader's TMEM, rows 128-255 in the partner's, and each CTA's four epilogue warps drain their half.
//
// Barriers (all waits bounded, see sm100_prims.cuh):
//   full[s]   leader only, 1 arrival + transaction bytes of BOTH CTAs (the partner's TMA loads complete on the
//             leader's barrier through the .cta_group::2 form of the load)
//   empty[s]  in both CTAs, released by tcgen05.commit.cta_group::2 with a CTA mask of both
//   tfull[a]  in both CTAs, same commit form: accumulator a is complete
//   tempty[a] leader only, 2 arrivals: each CTA's epilogue has drained its half of accumulator a
// Accumulators alternate between tiles; those of a 512-column tile both belong to it.
// Same operand-layout support, epilogues (bf16 store / fp32 store / fp32 reduce-add) and split-K slicing as
// gemm_sm100.cu; replaces the cuBLAS call behind matmul / linear
// (reference: paddle/phi/kernels/funcs/blas/blas_impl.cu.h:426).
#include "host_utils.h"
#include "sm100_prims.cuh"

namespace pd {
namespace gemm2 {

constexpr int BM = 128, BK = 64;
constexpr int TILE_M = 256;
constexpr int A_STAGE_BYTES = BM * BK * 2;        // 16 KB
constexpr int C_CHUNK_BYTES = BM * 128;
constexpr int NUM_THREADS = 192;
// TN: columns of the pair's tile, 512, 256 or 128; each CTA holds half of the columns of each accumulator
constexpr int stages(int tn) { return tn == 512 ? 4 : (tn == 256 ? 6 : 8); }
constexpr int b_stage_bytes(int tn) { return tn / 2 * BK * 2; }
constexpr int smem_bytes(int tn) { return stages(tn) * (A_STAGE_BYTES + b_stage_bytes(tn)) + 2 * C_CHUNK_BYTES + 1024 + 256; }
constexpr uint32_t PEER_BIT_MASK = 0xFEFFFFFFu;   // clears the CTA-pair bit of a shared::cluster address -> leader CTA

enum Epi : int { kStoreBf16 = 0, kStoreF32 = 1, kAccumF32 = 2, kBiasAct = 3, kSwiglu = 4 };
// kBiasAct: C = act(A B + bias) + residual as bf16 (bias bf16 [N], residual bf16 [M, N], each or null; act: 0 none, 1 relu, 2 gelu (erf), 3 gelu (tanh),
// 4 silu) - the reference's fused_gemm_epilogue (paddle/phi/kernels/fusion/gpu/fused_gemm_epilogue_kernel.cu).
// kSwiglu: the N columns hold (gate, up) pairs interleaved; C [M, N / 2] = silu(gate) * up as bf16, i.e. the first
// feed-forward GEMM with its activation, without the [M, N] intermediate ever reaching memory.
__device__ __forceinline__ float apply_act(float x, int act) {
  switch (act) {
    case 1: return fmaxf(x, 0.f);
    case 2: return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
    case 3: return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    case 4: return x / (1.f + __expf(-x));
    default: return x;
  }
}

struct Barriers {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tfull[2];
  uint64_t tempty[2];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
  int epi_decision;
};

// ---- cluster / cta_group::2 primitives
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint64_t* bar, uint32_t cta) {
  uint32_t raddr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(smem_u32(bar)), "r"(cta));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(raddr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_2cta(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_2cta(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// issued by a converged warp, predicated on one lane (see umma_bf16_ss_if)
__device__ __forceinline__ void umma2_bf16_ss_if(uint32_t lead, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// arrive on the barrier at this shared-memory offset in BOTH CTAs of the pair once all MMAs issued so far are complete
__device__ __forceinline__ void umma2_commit_both_if(uint32_t lead, uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n"
      " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n" ::"r"(smem_u32(bar)),
      "h"(mask), "r"(lead)
      : "memory");
}
// per-CTA tiled loads whose completion bytes are counted on the LEADER CTA's barrier (no data multicast)
__device__ __forceinline__ void tma2_load_2d(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar) & PEER_BIT_MASK), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma2_load_3d(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar) & PEER_BIT_MASK), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Tiles go in groups of G row tiles, column by column.
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int G, int& tm, int& tn) {
  const int per_group = G * tiles_n;
  const int g = t / per_group;
  const int first_m = g * G;
  const int gsz = min(G, tiles_m - first_m);
  const int r = t - g * per_group;
  tm = first_m + r % gsz;
  tn = r / gsz;
}

// a ROWS x 64 operand block (rows = M or N index of this CTA's half) into one stage
template <bool MN, int ROWS>
__device__ __forceinline__ void load_half(void* dst, const CUtensorMap* tm, uint64_t* bar, int mn0, int k0, bool use3d) {
  if (!MN) {
    tma2_load_2d(dst, tm, bar, k0, mn0);                        // box {64 k, ROWS rows}
  } else if (use3d) {
    tma2_load_3d(dst, tm, bar, 0, k0, mn0 >> 6);                // one box {64 mn, 64 k, ROWS / 64 chunks}
  } else {
#pragma unroll
    for (int c = 0; c < ROWS / 64; ++c)                                  // boxes {64 mn, 64 k}
      tma2_load_2d(static_cast<uint8_t*>(dst) + c * 8192, tm, bar, mn0 + c * 64, k0);
  }
}

constexpr int MAX_GROUPS = 8;
// The operands of G products of the same M x N, worked on one after the other in one launch; K differs.
template <int G>
struct Operands {
  CUtensorMap a[G], b[G], c[G];
  int k[G];
};

template <bool A_MN, bool B_MN, int EPI, int TILE_N, int G>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm2_bf16_kernel(const __grid_constant__ Operands<G> op, int groups, int M, int N, int mn3d, int splits, int* status,
                  const __nv_bfloat16* bias, int act, const __nv_bfloat16* residual, int ldr, int round_product, int raster) {
  // accumulators hold ACC_N columns; a 512-column tile takes both of one tile, narrower ones alternate between tiles
  constexpr int ACC_N = TILE_N == 512 ? 256 : TILE_N, HALVES = TILE_N / ACC_N;
  constexpr int STAGES = stages(TILE_N), BN_HALF = ACC_N / 2, B_STAGE_BYTES = b_stage_bytes(TILE_N), B_HALF_BYTES = B_STAGE_BYTES / HALVES;
  constexpr uint32_t TM_COLS = 2 * ACC_N;
  extern __shared__ uint8_t smem_raw[];
  // the dynamic shared memory starts at the same offset in both CTAs, so the aligned carve-up is identical in both
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_STAGE_BYTES;
  uint8_t* sC = sB + STAGES * B_STAGE_BYTES;
  Barriers* bars = reinterpret_cast<Barriers*>(sC + 2 * C_CHUNK_BYTES);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();          // 0 = leader
  const bool leader = cta_rank == 0;
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const int tiles_m = (M + TILE_M - 1) / TILE_M, tiles_n = (N + TILE_N - 1) / TILE_N;
  const int group_tiles = tiles_m * tiles_n * splits;
  const int num_tiles = group_tiles * (G == 1 ? 1 : groups);
  // tile t: which product it belongs to, its number in that one, its blocks of K
  auto group_of = [&](int t) { return G == 1 ? 0 : t / group_tiles; };
  // accumulators of a tile that starts at column n0: the second half of a wide one may lie outside the matrix
  auto halves_at = [&](int n0) { return HALVES == 2 && n0 + ACC_N < N ? 2 : 1; };
  auto k_range = [&](int g, int t, int& kb0, int& kb1) {
    const int kb_total = (op.k[g] + BK - 1) / BK, kbs = (kb_total + splits - 1) / splits;
    kb0 = (t % splits) * kbs;
    kb1 = min(kb_total, kb0 + kbs);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bars->tfull[a], 1);
      mbar_init(&bars->tempty[a], 2);
    }
    mbar_init(&bars->drain, 1);
    bars->abort_flag = 0;
    bars->epi_decision = 0;
    fence_mbar_init();
  }
  if (warp == 5) tmem_alloc_2cta(&bars->tmem_base, TM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // both CTAs' barriers are initialised before any remote arrive / remote completion
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp == 4) {
    // ------------------------------------------------------------ TMA producer (one per CTA: its halves of A and B)
    if (lane == 0) {
      prefetch_tmap(&op.a[0]);
      prefetch_tmap(&op.b[0]);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      int issued = 0;
      for (int t = cluster_id; t < num_tiles && ok; t += n_clusters) {
        int tm, tn, kb0, kb1;
        const int g = group_of(t), tg = t - g * group_tiles;
        tile_coords(tg / splits, tiles_m, tiles_n, raster, tm, tn);
        const int m0 = tm * TILE_M + static_cast<int>(cta_rank) * BM;
        const int n0 = tn * TILE_N + static_cast<int>(cta_rank) * BN_HALF, halves = halves_at(tn * TILE_N);
        k_range(g, tg, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&bars->empty[s], ph ^ 1, abort_flag, status, 100 + s)) { ok = false; break; }
          if (leader) mbar_expect_tx(&bars->full[s], 2 * (A_STAGE_BYTES + halves * B_HALF_BYTES));
          const int k0 = kb * BK;
          load_half<A_MN, BM>(sA + s * A_STAGE_BYTES, &op.a[g], &bars->full[s], m0, k0, (mn3d & 1) != 0);
          load_half<B_MN, BN_HALF>(sB + s * B_STAGE_BYTES, &op.b[g], &bars->full[s], n0, k0, (mn3d & 2) != 0);
          if (HALVES == 2 && halves == 2)
            load_half<B_MN, BN_HALF>(sB + s * B_STAGE_BYTES + B_HALF_BYTES, &op.b[g], &bars->full[s], n0 + ACC_N, k0, (mn3d & 2) != 0);
          ++issued;
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      if (!ok && leader) {  // drain the loads that were armed but never consumed before the CTA may exit
        for (int i = 0; i < STAGES && i < issued; ++i) mbar_drain(&bars->full[i], 0), mbar_drain(&bars->full[i], 1);
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only, the whole warp converged)
    if (leader) {
      const uint32_t lead = elect_one() ? 1u : 0u;
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
      constexpr uint32_t idesc = make_idesc(TILE_M, ACC_N, A_MN, B_MN);
      constexpr uint32_t a_kstep = A_MN ? 2048u : 32u;
      constexpr uint32_t b_kstep = B_MN ? 2048u : 32u;
      constexpr uint32_t a_lbo = A_MN ? 8192u : 16u;
      constexpr uint32_t b_lbo = B_MN ? 8192u : 16u;
      const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(sA), a_lbo, 1024), b_desc0 = make_smem_desc_sw128(smem_u32(sB), b_lbo, 1024);
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      bool ok = true;
      if (HALVES == 2) {
        // A batch of K blocks goes into the first accumulator, then into the second.  The first and last batch of a tile are all
        // stages long: the first accumulator is drained under the end of its tile, the second under the beginning of the next.
        int it1 = 0;                                                             // tiles with two halves so far
        for (int t = cluster_id; t < num_tiles && ok; t += n_clusters, ++it) {
          const int g = group_of(t), tg = t - g * group_tiles;
          int tm_, tn, kb0, kb1;
          tile_coords(tg / splits, tiles_m, tiles_n, raster, tm_, tn);
          k_range(g, tg, kb0, kb1);
          const int halves = halves_at(tn * TILE_N);
          if (!mbar_wait_warp(&bars->tempty[0], (it & 1) ^ 1, abort_flag, status, 200)) { ok = false; break; }
          bool first = true;
#pragma unroll 1
          for (int left = kb1 - kb0; left > 0 && ok;) {
            const int n = first || left <= STAGES ? min(STAGES, left) : 1;
            int si = s;
            uint32_t phi = ph;
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
              if (!mbar_wait_warp(&bars->full[si], phi, abort_flag, status, 300 + si)) { ok = false; break; }
              tc_fence_after();
              const uint64_t ad = a_desc0 + si * (A_STAGE_BYTES >> 4), bd = b_desc0 + si * (B_STAGE_BYTES >> 4);
#pragma unroll
              for (int k = 0; k < BK / 16; ++k)
                umma2_bf16_ss_if(lead, tm, ad + k * (a_kstep >> 4), bd + k * (b_kstep >> 4), idesc, !first || (i | k) != 0 ? 1u : 0u);
              if (++si == STAGES) si = 0, phi ^= 1;
            }
            if (!ok) break;
            if (n == left) umma2_commit_both_if(lead, &bars->tfull[0]);
            if (first && halves == 2) {
              if (!mbar_wait_warp(&bars->tempty[1], (it1 & 1) ^ 1, abort_flag, status, 201)) { ok = false; break; }
              tc_fence_after();
            }
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
              const uint64_t ad = a_desc0 + s * (A_STAGE_BYTES >> 4), bd = b_desc0 + ((s * B_STAGE_BYTES + B_HALF_BYTES) >> 4);
              if (halves == 2) {
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                  umma2_bf16_ss_if(lead, tm + ACC_N, ad + k * (a_kstep >> 4), bd + k * (b_kstep >> 4), idesc, !first || (i | k) != 0 ? 1u : 0u);
              }
              umma2_commit_both_if(lead, &bars->empty[s]);
              if (++s == STAGES) s = 0, ph ^= 1;
            }
            if (n == left && halves == 2) umma2_commit_both_if(lead, &bars->tfull[1]);
            left -= n;
            first = false;
          }
          it1 += halves - 1;
        }
      } else
      for (int t = cluster_id; t < num_tiles && ok; t += n_clusters, ++it) {
        const int acc = it & 1;
        const uint32_t acc_ph = (it >> 1) & 1;
        if (!mbar_wait_warp(&bars->tempty[acc], acc_ph ^ 1, abort_flag, status, 200 + acc)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tm + acc * ACC_N;
        const int g = group_of(t);
        int kb0, kb1;
        k_range(g, t - g * group_tiles, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&bars->full[s], ph, abort_flag, status, 300 + s)) { ok = false; break; }
          tc_fence_after();
          const uint64_t ad = a_desc0 + s * (A_STAGE_BYTES >> 4), bd = b_desc0 + s * (B_STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            umma2_bf16_ss_if(lead, d_tmem, ad + k * (a_kstep >> 4), bd + k * (b_kstep >> 4), idesc, ((kb - kb0) | k) != 0 ? 1u : 0u);
          }
          umma2_commit_both_if(lead, &bars->empty[s]);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) umma2_commit_both_if(lead, &bars->tfull[acc]);
      }
      if (!ok) {
        if (lead) asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&bars->drain))
                               : "memory");
        mbar_drain(&bars->drain, 0);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue (warps 0..3 of each CTA: its 128 rows)
    const int epi_tid = threadIdx.x;
    constexpr int CW = (EPI == kStoreBf16 || EPI == kBiasAct) ? 64 : (EPI == kSwiglu ? 128 : 32);
    constexpr int NCHUNK = ACC_N / CW;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const bool bias_vec = (reinterpret_cast<uintptr_t>(bias) & 15u) == 0;
    int it = 0;
    int chunk_counter = 0;
    int it1 = 0;                              // wide tiles with two halves so far
    bool live = true;
    for (int t = cluster_id; t < num_tiles && live; t += n_clusters, ++it) {
      int tm, tn;
      const int g = group_of(t);
      tile_coords((t - g * group_tiles) / splits, tiles_m, tiles_n, raster, tm, tn);
      const int m0 = tm * TILE_M + static_cast<int>(cta_rank) * BM;
      const int halves = halves_at(tn * TILE_N);
#pragma unroll 1
      for (int half = 0; half < halves; ++half) {
      const int n0 = tn * TILE_N + half * ACC_N;
      const int acc = HALVES == 2 ? half : it & 1;
      const uint32_t acc_ph = HALVES == 2 ? (half == 0 ? it : it1) & 1 : (it >> 1) & 1;
      if (epi_tid == 0) {
        const bool ok = mbar_wait(&bars->tfull[acc], acc_ph, abort_flag, status, 400 + acc);
        bars->epi_decision = ok ? 1 : 0;
      }
      named_bar_sync(1, 128);
      if (bars->epi_decision == 0) { live = false; break; }
      tc_fence_after();
      const uint32_t t_acc = tmem_base + lane_base + acc * ACC_N;
      const bool rows_live = m0 < M;          // a partner half entirely below the matrix stores nothing
#pragma unroll 1
      for (int c = 0; c < NCHUNK; ++c, ++chunk_counter) {
        uint8_t* stage = sC + (chunk_counter & 1) * C_CHUNK_BYTES;
        if (epi_tid == 0) tma_wait_group_read<1>();
        named_bar_sync(1, 128);
        uint8_t* row_ptr = stage + epi_tid * 128;
        const int sw = epi_tid & 7;
        if (EPI == kSwiglu) {
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            uint32_t r[32];
            tmem_ld_32x32(t_acc + c * CW + h * 32, r);
            tmem_ld_wait();
            float o[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float g = __uint_as_float(r[2 * i]), u = __uint_as_float(r[2 * i + 1]);
              o[i] = g / (1.f + __expf(-g)) * u;
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint4 v;
              v.x = pack_bf16x2(o[8 * j + 0], o[8 * j + 1]);
              v.y = pack_bf16x2(o[8 * j + 2], o[8 * j + 3]);
              v.z = pack_bf16x2(o[8 * j + 4], o[8 * j + 5]);
              v.w = pack_bf16x2(o[8 * j + 6], o[8 * j + 7]);
              *reinterpret_cast<uint4*>(row_ptr + (((h * 2 + j) ^ sw) << 4)) = v;
            }
          }
        } else if (EPI == kStoreBf16 || EPI == kBiasAct) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld_32x32(t_acc + c * CW + h * 32, r);
            tmem_ld_wait();
            if (EPI == kBiasAct) {
              const int col0 = n0 + c * CW + h * 32;
              if (bias != nullptr) {
                if (bias_vec && col0 + 32 <= N) {      // four 16-byte loads that all threads share, not 32 of two bytes
#pragma unroll
                  for (int q = 0; q < 4; ++q) {
                    const uint4 b4 = __ldg(reinterpret_cast<const uint4*>(bias + col0) + q);
                    const uint32_t w[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                      r[8 * q + 2 * e] = __float_as_uint(__uint_as_float(r[8 * q + 2 * e]) + __uint_as_float(w[e] << 16));
                      r[8 * q + 2 * e + 1] = __float_as_uint(__uint_as_float(r[8 * q + 2 * e + 1]) + __uint_as_float(w[e] & 0xffff0000u));
                    }
                  }
                } else {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    if (col0 + i < N) r[i] = __float_as_uint(__uint_as_float(r[i]) + __bfloat162float(__ldg(bias + col0 + i)));
                }
              }
              if (act != 0) {
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(apply_act(__uint_as_float(r[i]), act));
              }
              // a residual added by a kernel of its own moves the product through memory twice more: a prompt of 3 x 777 tokens
              // through one 13B layer 1507 -> 1481 us, two additions of 14 each.  With
              // round_product the addition starts from what that kernel is given, a product in bf16 (2331 x 5120 x 5120 106.6 / 108.9 us
              // without / with; 113 with the rounding between the loads, which then waited for one another).
              if (residual != nullptr && m0 + epi_tid < M) {      // N % 8 == 0: a group of eight columns is inside or outside
                const uint4* rp = reinterpret_cast<const uint4*>(residual + static_cast<int64_t>(m0 + epi_tid) * ldr + col0);
                uint4 r4[4];                                      // all four in flight before the first use
#pragma unroll
                for (int q = 0; q < 4; ++q) r4[q] = col0 + 8 * q < N ? __ldg(rp + q) : make_uint4(0, 0, 0, 0);
                if (round_product) {
#pragma unroll
                  for (int i = 0; i < 32; i += 2) {
                    const uint32_t y = pack_bf16x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                    r[i] = y << 16, r[i + 1] = y & 0xffff0000u;
                  }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const uint32_t w[4] = {r4[q].x, r4[q].y, r4[q].z, r4[q].w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    r[8 * q + 2 * e] = __float_as_uint(__uint_as_float(r[8 * q + 2 * e]) + __uint_as_float(w[e] << 16));
                    r[8 * q + 2 * e + 1] = __float_as_uint(__uint_as_float(r[8 * q + 2 * e + 1]) + __uint_as_float(w[e] & 0xffff0000u));
                  }
                }
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[8 * j + 0]), __uint_as_float(r[8 * j + 1]));
              v.y = pack_bf16x2(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3]));
              v.z = pack_bf16x2(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5]));
              v.w = pack_bf16x2(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7]));
              *reinterpret_cast<uint4*>(row_ptr + (((h * 4 + j) ^ sw) << 4)) = v;
            }
          }
        } else {
          uint32_t r[32];
          tmem_ld_32x32(t_acc + c * CW, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint4 v = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            *reinterpret_cast<uint4*>(row_ptr + ((j ^ sw) << 4)) = v;
          }
        }
        if (c == NCHUNK - 1) tc_fence_before();
        fence_proxy_async_smem();
        named_bar_sync(1, 128);
        if (epi_tid == 0) {
          if (c == NCHUNK - 1) {   // this CTA's half of the accumulator is drained: tell the leader's MMA thread
            if (leader) mbar_arrive(&bars->tempty[acc]);
            else mbar_arrive_remote(&bars->tempty[acc], 0);
          }
          if (rows_live && n0 + c * CW < N) {
            if (EPI == kAccumF32) tma_reduce_add_2d(&op.c[g], stage, n0 + c * CW, m0);
            else if (EPI == kSwiglu) tma_store_2d(&op.c[g], stage, (n0 + c * CW) / 2, m0);
            else tma_store_2d(&op.c[g], stage, n0 + c * CW, m0);
          }
          tma_commit_group();
        }
      }
      }
      it1 += halves - 1;
    }
    if (epi_tid == 0) tma_wait_group<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // nobody leaves while the partner may still signal this CTA's barriers or read its tiles
  if (warp == 5) tmem_dealloc_2cta(tmem_base, TM_COLS);
}

// CTA pairs that a call may use: all SMs, or as many as the caller leaves it
static int max_clusters(int max_ctas) {
  int clusters = sm_count() / 2;
  if (max_ctas > 0 && clusters > max_ctas / 2) clusters = max_ctas / 2;
  return clusters < 1 ? 1 : clusters;
}

// Row tiles of a raster group (tile_coords): their rows of A stay in the L2 while the columns of B pass once.  Sixteen: under sustained
// load (the power cap), us with 4 / 8 / 16 / 32: 4096 x 12288 x 4096 335 / 316 / 305 / -, its weight gradient 362 / 343 / 331 / -,
// 2331 x 27648 x 5120 - / 552 / 526 / 544; 8 / 16: 8192 x 12288 x 4096 628 / 603, 8192 x 11008 x 4096 561 / 543, 5120 x 12288 x 4096
// 397 / 380, 8192 x 5120 x 5120 330 / 330, 16384 x 4096 x 4096 415 / 414.  Thirty-two lose their own rows (8192 x 4096 x 5120 258 / 263 /
// 289 with 8 / 16 / 32).  Of deep products (K >= 8192) sixteen row tiles of A are 64 MB of the 126 MB and more, so tiles of 256 columns
// take eight there: 8 / 16, 8192 x 4096 x 8192 445 / 450, x 11008 573 / 582, x 13824 721 / 734, 4096 x 22016 x 8200 1221 / 1250, 4096 x
// 5120 x 13824 483 / 488, 22016 x 4096 x 16384 into fp32 2510 / 2581; with K = 7168 483 / 487, with 6144 417 / 413.  Up to fifteen row
// tiles would be cut into two groups: 2331 x 5120 x 13824 301 / 292.  Tiles of 512 columns pass over A half as often: 8192 x 8192 x
// 11008 1106 / 1086, 4096 x 4096 x 22016 575 / 566.
static int raster_rows(int tile_n, int M, int K) { return tile_n == 256 && K >= 8192 && M > 15 * TILE_M ? 8 : 16; }

template <bool A_MN, bool B_MN, int EPI, int TILE_N, int G = 1>
static int launch_variant(const Operands<G>& op, int groups, int M, int N, int mn3d, int* status, cudaStream_t stream, int max_ctas,
                          int splits, const __nv_bfloat16* bias = nullptr, int act = 0, const __nv_bfloat16* residual = nullptr,
                          int ldr = 0, int round_product = 0) {
  auto kfn = gemm2_bf16_kernel<A_MN, B_MN, EPI, TILE_N, G>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(TILE_N)) != cudaSuccess) return kErrCuda;
    configured = true;
  }
  const int tiles = ((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N) * splits * groups;
  int clusters = max_clusters(max_ctas);
  if (clusters > tiles) clusters = tiles;
  kfn<<<clusters * 2, NUM_THREADS, smem_bytes(TILE_N), stream>>>(op, groups, M, N, mn3d, splits, status, bias, act, residual, ldr,
                                                                round_product, raster_rows(TILE_N, M, op.k[0]));
  return cudaGetLastError() == cudaSuccess ? kLaunchOk : kErrCuda;
}

// 256 x 128 tiles when even those all run at once on the pairs that the call may use: every pair then does half the work of a 256 x 256 tile (us, 256 / 128:
// 512 x 1024 x 512 15.3 / 13.3, 818 x 616 x 3064 35.8 / 31.7, 200 x 4096 x 4096 34.8 / 29.7).  With more tiles the other form wins
// although its last wave is emptier: a 64-deep block of a narrow tile is 256 tensor cycles and costs some 350 (4096^3: 96 / 124;
// 1000 x 11008 x 4096, 3 waves against 2.5: 84 / 109).
//
// 256 x 512 tiles for deep products (K >= 8192) where they take no more rounds: a K block then brings 48 KB to an SM for the MMAs that
// two 256 x 256 tiles bring 64 KB for, and at the power cap that is time (without any loads of B the same products ran 10 to 12 %
// faster).  us under sustained load, 256 / 512 columns, groups of 16 row tiles: 4096 x 4096 x 12288 345 / 322, x 22016 610 / 571,
// x 32000 892 / 855, x 11008 311 / 290, x 8192 (into fp32) 238 / 228; but x 4096 111 / 112, and where the rounds come out longer 2331 x
// 5120 x 13824 290 / 321, 8192 x 4096 x 4096 210 / 224.
static int tile_n(int M, int N, int K, int splits, int max_ctas) {
  const int64_t rows = (M + TILE_M - 1) / TILE_M, pairs = max_clusters(max_ctas);
  if (K >= 8192 && splits == 1 && 2 * ((rows * ((N + 511) / 512) + pairs - 1) / pairs) <= (rows * ((N + 255) / 256) + pairs - 1) / pairs) return 512;
  return static_cast<int64_t>((M + TILE_M - 1) / TILE_M) * ((N + 127) / 128) * splits <= max_clusters(max_ctas) ? 128 : 256;
}

}  // namespace gemm2
}  // namespace pd

// Columns of the tiles that pd_gemm_bf16_2cta works in: for K below 8192, and for any K.
PD_EXPORT int pd_gemm_2cta_tile_n(int M, int N, int splits, int max_ctas) { return pd::gemm2::tile_n(M, N, 0, splits, max_ctas); }
PD_EXPORT int pd_gemm_2cta_tile_n_at(int M, int N, int K, int splits, int max_ctas) { return pd::gemm2::tile_n(M, N, K, splits, max_ctas); }

// Same contract as pd_gemm_bf16 / pd_gemm_bf16_splitk (gemm_sm100.cu); splits = 1 for the plain form.
PD_EXPORT int pd_gemm_bf16_2cta(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                                int a_mn_major, int b_mn_major, int epi, int max_ctas, int splits, int* status,
                                cudaStream_t stream) {
  using namespace pd;
  using namespace pd::gemm2;
  if (M <= 0 || N <= 0 || K <= 0 || splits < 1) return kErrBadShape;
  if (splits > 1 && epi != kAccumF32) return kErrBadShape;
  {
    const int kb_total = (K + BK - 1) / BK;
    if (splits > kb_total) splits = kb_total;
    const int kbs = (kb_total + splits - 1) / splits;
    splits = (kb_total + kbs - 1) / kbs;
  }
  if (!aligned16(A) || !aligned16(B) || !aligned16(C)) return kErrAlignment;
  if ((lda % 8) || (ldb % 8) || (epi == kStoreBf16 ? (ldc % 8) : (ldc % 4))) return kErrAlignment;
  const int TN = tile_n(M, N, K, splits, max_ctas), BN_HALF = TN == 512 ? 128 : TN / 2;
  Operands<1> op;
  op.k[0] = K;
  bool ok = true;
  int a3d = 0, b3d = 0;
  if (!a_mn_major) ok &= encode_tmap_2d(&op.a[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, A, K, M, uint64_t(lda) * 2, BK, BM);
  else ok &= encode_tmap_mn(&op.a[0], A, M, K, uint64_t(lda) * 2, BM / 64, BK, &a3d);
  if (!b_mn_major) ok &= encode_tmap_2d(&op.b[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, B, K, N, uint64_t(ldb) * 2, BK, BN_HALF);
  else ok &= encode_tmap_mn(&op.b[0], B, N, K, uint64_t(ldb) * 2, BN_HALF / 64, BK, &b3d);
  if (epi == kStoreBf16) ok &= encode_tmap_2d(&op.c[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, C, N, M, uint64_t(ldc) * 2, 64, BM);
  else ok &= encode_tmap_2d(&op.c[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, C, N, M, uint64_t(ldc) * 4, 32, BM);
  if (!ok) return kErrTensorMap;
#define PD_GEMM2_CASE(AM, BM_, E)                                                                  \
  if (a_mn_major == AM && b_mn_major == BM_ && epi == E)                                           \
    return TN == 512 ? launch_variant<AM, BM_, E, 512>(op, 1, M, N, a3d | (b3d << 1), status, stream, max_ctas, splits) \
         : TN == 128 ? launch_variant<AM, BM_, E, 128>(op, 1, M, N, a3d | (b3d << 1), status, stream, max_ctas, splits) \
                     : launch_variant<AM, BM_, E, 256>(op, 1, M, N, a3d | (b3d << 1), status, stream, max_ctas, splits);
  PD_GEMM2_CASE(0, 0, 0) PD_GEMM2_CASE(0, 1, 0) PD_GEMM2_CASE(1, 0, 0) PD_GEMM2_CASE(1, 1, 0)
  PD_GEMM2_CASE(0, 0, 1) PD_GEMM2_CASE(0, 1, 1) PD_GEMM2_CASE(1, 0, 1) PD_GEMM2_CASE(1, 1, 1)
  PD_GEMM2_CASE(0, 0, 2) PD_GEMM2_CASE(0, 1, 2) PD_GEMM2_CASE(1, 0, 2) PD_GEMM2_CASE(1, 1, 2)
#undef PD_GEMM2_CASE
  return kErrBadShape;
}

// C = act(A B + bias) + residual (swiglu = 0; C bf16 [M, N]; bias and residual may be null; with a residual N and ldr are multiples of
// 8; round_product = 1: what it is added to is rounded to bf16 first) or C = silu(gate) * up over interleaved (gate, up) column pairs
// (swiglu = 1; C bf16 [M, N / 2], N a multiple of 16, bias and residual must be null).  Operand layouts as pd_gemm_bf16_2cta.
PD_EXPORT int pd_gemm_bf16_2cta_epi(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                                    int a_mn_major, int b_mn_major, const void* bias, int act, int swiglu, const void* residual, int ldr,
                                    int round_product, int* status, cudaStream_t stream) {
  using namespace pd;
  using namespace pd::gemm2;
  if (M <= 0 || N <= 0 || K <= 0 || act < 0 || act > 4) return kErrBadShape;
  if (swiglu && (bias != nullptr || residual != nullptr || (N % 16))) return kErrBadShape;
  if (!aligned16(A) || !aligned16(B) || !aligned16(C) || !aligned16(residual)) return kErrAlignment;
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (residual != nullptr && ((ldr % 8) || (N % 8)))) return kErrAlignment;
  const int TN = swiglu ? 256 : tile_n(M, N, K, 1, 0), BN_HALF = TN == 512 ? 128 : TN / 2;
  Operands<1> op;
  op.k[0] = K;
  bool ok = true;
  int a3d = 0, b3d = 0;
  if (!a_mn_major) ok &= encode_tmap_2d(&op.a[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, A, K, M, uint64_t(lda) * 2, BK, BM);
  else ok &= encode_tmap_mn(&op.a[0], A, M, K, uint64_t(lda) * 2, BM / 64, BK, &a3d);
  if (!b_mn_major) ok &= encode_tmap_2d(&op.b[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, B, K, N, uint64_t(ldb) * 2, BK, BN_HALF);
  else ok &= encode_tmap_mn(&op.b[0], B, N, K, uint64_t(ldb) * 2, BN_HALF / 64, BK, &b3d);
  ok &= encode_tmap_2d(&op.c[0], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, C, swiglu ? N / 2 : N, M, uint64_t(ldc) * 2, 64, BM);
  if (!ok) return kErrTensorMap;
  const __nv_bfloat16 *bp = static_cast<const __nv_bfloat16*>(bias), *rp = static_cast<const __nv_bfloat16*>(residual);
#define PD_GEMM2_EPI_CASE(AM, BM_)                                                                              \
  if (a_mn_major == AM && b_mn_major == BM_) {                                                                  \
    if (swiglu) return launch_variant<AM, BM_, kSwiglu, 256>(op, 1, M, N, a3d | (b3d << 1), status, stream, 0, 1); \
    return TN == 512 ? launch_variant<AM, BM_, kBiasAct, 512>(op, 1, M, N, a3d | (b3d << 1), status, stream, 0, 1, bp, act, rp, ldr, round_product) \
         : TN == 128 ? launch_variant<AM, BM_, kBiasAct, 128>(op, 1, M, N, a3d | (b3d << 1), status, stream, 0, 1, bp, act, rp, ldr, round_product) \
                     : launch_variant<AM, BM_, kBiasAct, 256>(op, 1, M, N, a3d | (b3d << 1), status, stream, 0, 1, bp, act, rp, ldr, round_product); \
  }
  PD_GEMM2_EPI_CASE(0, 0) PD_GEMM2_EPI_CASE(0, 1) PD_GEMM2_EPI_CASE(1, 0) PD_GEMM2_EPI_CASE(1, 1)
#undef PD_GEMM2_EPI_CASE
  return kErrBadShape;
}

// Weight gradients of several experts:  C_g[M, N] (=|+=) A_g^T B_g for the rows [starts[g], starts[g] + rows[g]) of A [*, M] and
// B [*, N] (bf16).  C: fp32, added into (accumulate = 1), or bf16, `c_stride` elements apart; starts / rows: host arrays.  A product
// without rows is left out.  One launch takes up to MAX_GROUPS products, the longest first: a launch each pays its own ramp and last
// wave (us, launches each -> one; 8192 rows of 4 experts, 4096 x 8192 into fp32 438 -> 425, 4096 x 4096 241 -> 204; of 8 experts
// 4096 x 7168 568 -> 489; 4096 rows of 8, 2048 x 3584 169 -> 119; 256 rows of 8, 512 x 512 54 -> 9).
PD_EXPORT int pd_gemm_bf16_grouped_tn(const void* A, const void* B, void* C, const int64_t* starts, const int64_t* rows, int groups,
                                      int M, int N, int lda, int ldb, int ldc, int64_t c_stride, int accumulate, int* status,
                                      cudaStream_t stream) {
  using namespace pd;
  using namespace pd::gemm2;
  if (M <= 0 || N <= 0 || groups < 0) return kErrBadShape;
  if (!aligned16(A) || !aligned16(B) || !aligned16(C)) return kErrAlignment;
  if ((lda % 8) || (ldb % 8) || (accumulate ? (ldc % 4) || (c_stride % 4) : (ldc % 8) || (c_stride % 8))) return kErrAlignment;
  const int elem = accumulate ? 4 : 2;
  int left = 0;
  for (int g = 0; g < groups; ++g) {
    if (rows[g] < 0 || rows[g] > INT32_MAX) return kErrBadShape;
    left += rows[g] > 0;
  }
  Operands<MAX_GROUPS> op;
  int64_t below_rows = INT64_MAX;      // of the product taken last; equal ones are taken in their order
  int below_g = -1;
  while (left > 0) {
    const int n = left < MAX_GROUPS ? left : MAX_GROUPS, TN = tile_n(M, N, 0, n, 0);
    int a3d = 0, b3d = 0;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      int best = -1;
      for (int g = 0; g < groups; ++g) {
        const bool open = rows[g] > 0 && (rows[g] < below_rows || (rows[g] == below_rows && g > below_g));
        if (open && (best < 0 || rows[g] > rows[best])) best = g;
      }
      below_rows = rows[best];
      below_g = best;
      op.k[i] = static_cast<int>(rows[best]);
      ok &= encode_tmap_mn(&op.a[i], static_cast<const __nv_bfloat16*>(A) + starts[best] * lda, M, rows[best], uint64_t(lda) * 2, BM / 64, BK, &a3d);
      ok &= encode_tmap_mn(&op.b[i], static_cast<const __nv_bfloat16*>(B) + starts[best] * ldb, N, rows[best], uint64_t(ldb) * 2, TN / 2 / 64, BK, &b3d);
      ok &= encode_tmap_2d(&op.c[i], accumulate ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                           static_cast<char*>(C) + best * c_stride * elem, N, M, uint64_t(ldc) * elem, accumulate ? 32 : 64, BM);
    }
    if (!ok) return kErrTensorMap;
    for (int i = n; i < MAX_GROUPS; ++i) op.a[i] = op.a[0], op.b[i] = op.b[0], op.c[i] = op.c[0], op.k[i] = 0;
    const int mn3d = a3d | (b3d << 1);
    int rc;
    if (accumulate)
      rc = TN == 128 ? launch_variant<true, true, kAccumF32, 128, MAX_GROUPS>(op, n, M, N, mn3d, status, stream, 0, 1)
                     : launch_variant<true, true, kAccumF32, 256, MAX_GROUPS>(op, n, M, N, mn3d, status, stream, 0, 1);
    else
      rc = TN == 128 ? launch_variant<true, true, kStoreBf16, 128, MAX_GROUPS>(op, n, M, N, mn3d, status, stream, 0, 1)
                     : launch_variant<true, true, kStoreBf16, 256, MAX_GROUPS>(op, n, M, N, mn3d, status, stream, 0, 1);
    if (rc != kLaunchOk) return rc;
    left -= n;
  }
  return kLaunchOk;
}
