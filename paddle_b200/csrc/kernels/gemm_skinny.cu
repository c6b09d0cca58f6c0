// Skinny bf16 GEMM for sm_100a:  C[M,N] = x[M,K] * W[K,N] (+ bias) (+ residual), M <= 128: the projections of a decode step and
// linear layers on a handful of tokens.  (Reference: the cuBLAS call behind matmul, paddle/phi/kernels/funcs/blas/blas_impl.cu.h:426.)
//
// Bandwidth-bound: every weight is read once for M rows.  So the tile is made of weights: the tensor core computes
// D[128 n, M] = W^T x^T (A = W tile as an MN-major operand, B = x, MT columns with MT the next of 16, 32, 64, 128), a CTA streams its
// 128 columns through a TMA ring of 16 KB weight blocks, two or more CTAs share an SM (about 100 KB of loads in flight each) and
// K is cut over the CTAs of a cluster until the grid fills the GPU.  The partial tiles are summed in a fixed order through
// distributed shared memory: no workspace, no atomics, no second kernel, and the result does not change from run to run.
//
//   warp 4: TMA producer    warp 5: MMA issuer    warps 0-3: TMEM -> shared memory;    then all: cluster reduction + epilogue
//
// Epilogues: kStore (bias and / or residual added in fp32, bf16 result), kSwiglu (W holds gate columns [0, F) and up columns
// [F, 2F); a tile takes 64 of each and stores silu(gate) * up: the [M, 2F] product never reaches memory), kQkv (a tile is one
// head: bias, rotary embedding, q stored densely, k / v appended to their cache pages).
//
// Launched as a programmatic dependent: set-up, and with `weights_ready` the first weights of each CTA (a full ring: 80 KB up to
// 16 rows, 64 KB up to 64, 48 KB above), run under the end of the kernel before.
// Measured in a replayed decode step: gate / up of a 7B layer (180 MB) with its activation 30.2 us for one row (5.97 TB/s; before,
// 256 x 256 tiles and a separate activation: 72 us); qkv, out and down projections of two layers 89 us (before, 128 x 256 tiles
// with split-K atomics and a finalising kernel each: 123 us).  Two 7B layers and the head for one sequence, 1.07 GB of weights
// (161 us at the copy rate): 382 -> 262 us, with the qkv epilogue, dependent launches and a CTA per row in the norms 216 us;
// two 13B layers and the head, batch 64, 842 -> 760 -> 717 us (attention 387 of it, at the copy rate).
#include "host_utils.h"
#include "sm100_prims.cuh"

namespace pd {
namespace skinny {

constexpr int BN = 128, BK = 64;
constexpr int W_STAGE_BYTES = BN * BK * 2;        // 16 KB
constexpr int NUM_THREADS = 192;
constexpr int MAX_SPLIT = 8;
constexpr int x_stage_bytes(int mt) { return mt * BK * 2; }
// two CTAs on an SM; the ring also holds the fp32 partial tile [MT][128] at the end
constexpr int stages(int mt) { return mt <= 16 ? 5 : (mt <= 64 ? 4 : 3); }
constexpr int smem_bytes(int mt) { return stages(mt) * (W_STAGE_BYTES + x_stage_bytes(mt)) + 1024 + 256; }

enum Epi : int { kStore = 0, kSwiglu = 1, kQkv = 2 };

struct Params {
  int M, N, K;              // N: columns of W (2F for kSwiglu)
  int splits;               // CTAs of a cluster
  int F;                    // kSwiglu: columns of the result
  __nv_bfloat16* out;
  int ldo;
  const __nv_bfloat16* bias;       // [N] or null
  const __nv_bfloat16* residual;   // [M, N] or null
  int ldr;
  int weights_ready;        // W is not written by the kernel before this one: its first blocks are fetched ahead of the wait
  int* status;
  // kQkv: a tile is one head; rotary embedding at the sequences' positions, q to out [M, Hq, 128], k / v to their cache pages
  const float *cos_t, *sin_t;      // [max_pos, 64]
  const int *seq_lens, *block_table;
  __nv_bfloat16 *k_cache, *v_cache;   // [num_blocks, Hkv, 64, 128]
  int Hq, Hkv, table_stride, pages, max_pos;   // pages: entries of a block-table row
};

struct Barriers {
  uint64_t full[8], empty[8];
  uint64_t done;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer_f4(const void* local, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
// eight neighbouring sums of row m from column c on, over all CTAs of the cluster in rank order
__device__ __forceinline__ void reduce8(const float* part, int m, int c, int splits, float (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  const float* p = part + m * BN + c;
  for (int r = 0; r < splits; ++r) {
    const float4 a = ld_peer_f4(p, r), b = ld_peer_f4(p + 4, r);
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
  }
}
__device__ __forceinline__ void add8_bf16(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 q = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] += __uint_as_float(w[i] << 16);
    v[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void store8_bf16(__nv_bfloat16* p, const float (&v)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

template <int MT, int EPI>
__global__ void __launch_bounds__(NUM_THREADS, 2)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, Params p) {
  constexpr int ST = stages(MT), XB = x_stage_bytes(MT);
  constexpr uint32_t TM_COLS = MT < 32 ? 32 : MT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = smem + ST * W_STAGE_BYTES;
  float* part = reinterpret_cast<float*>(smem);                 // [MT][128], over the ring once all MMAs are complete
  Barriers* bars = reinterpret_cast<Barriers*>(sX + ST * XB);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int tile = static_cast<int>(blockIdx.x) / p.splits;
  const int kb_total = (p.K + BK - 1) / BK, kbs = (kb_total + p.splits - 1) / p.splits;
  const int kb0 = rank * kbs, nk = max(0, min(kb_total, kb0 + kbs) - kb0);
  const int n0 = EPI == kSwiglu ? tile * 64 : tile * BN;
  const int n1 = EPI == kSwiglu ? p.F + n0 : n0 + 64;           // the tile's second 64 columns

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    mbar_init(&bars->done, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 5) tmem_alloc(&bars->tmem_base, TM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;

  if (warp == 4) {
    if (lane == 0) {
      // Large weights pass through the L2 without pushing out x and the cached keys.  us, normal / first to leave: behind other kernels of a
      // step 64 rows 5120 x 15360 28.8 / 27.3, 5120 x 32000 52.1 / 49.9, 128 rows 4096 x 22016 38.8 / 37.0, one row 28.8 / 28.6.  The line
      // is a matrix of which no second fits the L2 (126 MB).  Two in turn, 64 rows: 48 MB 15.3 / 15.0, 62 MB 18.6 / 18.5, 68 MB 19.5 /
      // 19.3, 76 MB 19.5 / 19.0, 86 MB 20.5 / 19.8; twelve: 14.9 / 14.8, 17.0 / 16.8, 17.7 / 17.5, 18.1 / 17.8, 19.4 / 19.0; one row 0 to
      // 2 %.  So below it there is little to gain, and a small model, whose weights may stay from token to token, has something to lose:
      // one layer of 1024 and its 65 MB head 47.2 / 49.1.
      const bool pass_through = static_cast<int64_t>(p.K) * p.N * 2 >= (int64_t(72) << 20);
      const uint64_t policy = l2_evict_first();
      prefetch_tmap(&tmW);
      prefetch_tmap(&tmX);
      bool ok = true;
      int armed = 0;
      auto arm_and_load_w = [&](int i) {
        const int s = i % ST, k0 = (kb0 + i) * BK;
        mbar_expect_tx(&bars->full[s], W_STAGE_BYTES + XB);
        uint8_t* dst = sW + s * W_STAGE_BYTES;
        if (pass_through) {
          tma_load_2d(dst, &tmW, &bars->full[s], n0, k0, policy);
          tma_load_2d(dst + W_STAGE_BYTES / 2, &tmW, &bars->full[s], n1, k0, policy);
        } else {
          tma_load_2d(dst, &tmW, &bars->full[s], n0, k0);
          tma_load_2d(dst + W_STAGE_BYTES / 2, &tmW, &bars->full[s], n1, k0);
        }
      };
      const int ahead = p.weights_ready ? min(nk, ST) : 0;
      for (int i = 0; i < ahead; ++i) arm_and_load_w(i);
      pdl_wait();
      for (int i = 0; i < nk && ok; ++i) {
        const int s = i % ST, k0 = (kb0 + i) * BK;
        if (i >= ST && !mbar_wait(&bars->empty[s], ((i / ST) & 1) ^ 1, abort_flag, p.status, 100 + s)) { ok = false; break; }
        if (i >= ahead) arm_and_load_w(i);
        tma_load_2d(sX + s * XB, &tmX, &bars->full[s], k0, 0);
        armed = i + 1;
      }
      if (!ok || *abort_flag)
        for (int i = max(0, armed - ST); i < armed; ++i) mbar_drain(&bars->full[i % ST], (i / ST) & 1);
    }
    __syncwarp();
  } else if (warp == 5) {
    if (nk > 0) {
      constexpr uint32_t idesc = make_idesc(BN, MT, true, false);
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t wd0 = make_smem_desc_sw128(smem_u32(sW), W_STAGE_BYTES / 2, 1024);
      const uint64_t xd0 = make_smem_desc_sw128(smem_u32(sX), 16, 1024);
      bool ok = true;
      int s = 0;
      uint32_t ph = 0;
#pragma unroll 1
      for (int i = 0; i < nk; ++i) {
        if (!mbar_wait_warp(&bars->full[s], ph, abort_flag, p.status, 200 + s)) { ok = false; break; }
        tc_fence_after();
        const uint64_t wd = wd0 + s * (W_STAGE_BYTES >> 4), xd = xd0 + s * (XB >> 4);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16_ss_if(leader, tm, wd + k * (2048 >> 4), xd + k * (32 >> 4), idesc, (i | k) != 0 ? 1u : 0u);
        umma_commit_if(leader, &bars->empty[s]);
        if (++s == ST) s = 0, ph ^= 1;
      }
      umma_commit_if(leader, &bars->done);
      if (!ok) mbar_drain(&bars->done, 0);
    }
    __syncwarp();
  }
  pdl_wait();                                                    // residual, positions; the results are written below
  if (threadIdx.x == 0) pdl_trigger();
  // ---- partial tile -> shared memory (the ring is idle once `done` completes)
  if (warp < 4) {
    const int n = threadIdx.x;                                   // column of the tile = TMEM lane
    const uint32_t t = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const bool ok = nk > 0 && mbar_wait_warp(&bars->done, 0, abort_flag, p.status, 300);
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < MT; c += 16) {
      uint32_t r[16];
      if (ok) {
        tmem_ld_32x16(t + c, r);
        tmem_ld_wait();
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) part[(c + i) * BN + n] = ok ? __uint_as_float(r[i]) : 0.f;
    }
    tc_fence_before();
  }
  cluster_sync();
  // ---- sums over the cluster, dealt out in units of eight columns
  if (*abort_flag == 0) {
    if (EPI == kSwiglu) {
      for (int u = rank * NUM_THREADS + threadIdx.x; u < p.M * 8; u += NUM_THREADS * p.splits) {
        const int m = u >> 3, c = (u & 7) * 8;
        if (n0 + c >= p.F) continue;
        float g[8], up[8];
        reduce8(part, m, c, p.splits, g);
        reduce8(part, m, 64 + c, p.splits, up);
#pragma unroll
        for (int i = 0; i < 8; ++i) g[i] = g[i] / (1.f + __expf(-g[i])) * up[i];
        store8_bf16(p.out + static_cast<size_t>(m) * p.ldo + n0 + c, g);
      }
    } else if (EPI == kQkv) {
      const int head = tile;
      for (int u = rank * NUM_THREADS + threadIdx.x; u < p.M * 8; u += NUM_THREADS * p.splits) {
        const int m = u >> 3, c = (u & 7) * 8;
        const int pos = p.seq_lens[m];
        if (pos < 0 || pos >= p.max_pos || pos / 64 >= p.pages) continue;
        float a[8], b[8];
        reduce8(part, m, c, p.splits, a);
        reduce8(part, m, 64 + c, p.splits, b);
        if (p.bias != nullptr) {
          add8_bf16(p.bias + n0 + c, a);
          add8_bf16(p.bias + n0 + 64 + c, b);
        }
        if (head < p.Hq + p.Hkv) {
          const float* cp = p.cos_t + static_cast<size_t>(pos) * 64 + c;
          const float* sp = p.sin_t + static_cast<size_t>(pos) * 64 + c;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float co = cp[i], si = sp[i], x1 = a[i], x2 = b[i];
            a[i] = x1 * co - x2 * si;
            b[i] = x2 * co + x1 * si;
          }
        }
        __nv_bfloat16* dst;
        if (head < p.Hq) {
          dst = p.out + (static_cast<size_t>(m) * p.Hq + head) * BN;
        } else {
          const int kvh = (head - p.Hq) % p.Hkv;
          const int blk = p.block_table[static_cast<size_t>(m) * p.table_stride + pos / 64];
          dst = (head < p.Hq + p.Hkv ? p.k_cache : p.v_cache) + ((static_cast<size_t>(blk) * p.Hkv + kvh) * 64 + pos % 64) * BN;
        }
        store8_bf16(dst + c, a);
        store8_bf16(dst + 64 + c, b);
      }
    } else {
      for (int u = rank * NUM_THREADS + threadIdx.x; u < p.M * 16; u += NUM_THREADS * p.splits) {
        const int m = u >> 4, c = (u & 15) * 8;
        if (n0 + c >= p.N) continue;
        float v[8];
        reduce8(part, m, c, p.splits, v);
        if (p.bias != nullptr) add8_bf16(p.bias + n0 + c, v);
        if (p.residual != nullptr) add8_bf16(p.residual + static_cast<size_t>(m) * p.ldr + n0 + c, v);
        store8_bf16(p.out + static_cast<size_t>(m) * p.ldo + n0 + c, v);
      }
    }
  }
  cluster_sync();                                                // nobody leaves while a peer may read its partial tile
  if (warp == 5) tmem_dealloc(tmem, TM_COLS);
}

template <int MT, int EPI>
static int launch(const CUtensorMap& tmW, const CUtensorMap& tmX, const Params& p, int tiles, cudaStream_t stream) {
  auto kfn = skinny_gemm_kernel<MT, EPI>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MT)) != cudaSuccess) return kErrCuda;
    configured = true;
  }
  return launch_pdl(kfn, dim3(static_cast<unsigned>(tiles) * p.splits), dim3(NUM_THREADS), smem_bytes(MT), stream, p.splits, tmW, tmX, p);
}

}  // namespace skinny
}  // namespace pd

namespace pd {
namespace skinny {
// Fills in what all entry points share: tile maps, the row tile and the number of K cuts.
static int setup(const void* x, const void* w, int M, int N, int K, int ldx, int ldw, int tiles, int splits, CUtensorMap* tmW,
                 CUtensorMap* tmX, int* mt, Params* p) {
  *mt = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
  if (!encode_tmap_2d(tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w, N, K, uint64_t(ldw) * 2, 64, BK) ||
      !encode_tmap_2d(tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, K, M, uint64_t(ldx) * 2, BK, *mt))
    return kErrTensorMap;
  const int kb = (K + BK - 1) / BK;
  if (splits == 0) {
    // two CTAs per SM in one wave, no CTA with fewer than four blocks of K; at most 4: with 8 the partial tiles cost more than the
    // further loads in flight bring (us with 4 / 8: K = N = 4096, M = 128 14.0 / 20.7; K = 11008, N = 4096, M = 32 18.9 / 19.5).  One row
    // would gain (8.7 / 7.7 and 16.9 / 15.8), but the number of cuts is the order in which a row is summed up: it must not follow M, or
    // a sequence's result changes with the number of those that are decoded beside it.
    splits = 1;
    while (splits < 4 && tiles * splits * 2 <= 2 * sm_count() && kb >= 8 * splits) splits *= 2;
  }
  p->M = M;
  p->N = N;
  p->K = K;
  p->splits = splits > kb ? kb : splits;
  return kLaunchOk;
}
}  // namespace skinny
}  // namespace pd

// out[M, N] (bf16) = x[M, K] W[K, N] (+ bias[N]) (+ residual[M, N]); swiglu = 1: W holds [gate | up] halves, out is [M, N / 2].
// M <= 128; N, K, the leading dimensions multiples of 8, pointers 16-byte aligned.  splits = 0: as many CTAs per tile as fill
// the GPU.  weights_ready = 1 promises that the kernel before this one in the stream does not write W.
PD_EXPORT int pd_gemm_skinny(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldo,
                             const void* bias, const void* residual, int ldr, int swiglu, int splits, int weights_ready,
                             int* status, cudaStream_t stream) {
  using namespace pd;
  using namespace pd::skinny;
  if (M <= 0 || M > 128 || N <= 0 || K <= 0 || (N % 8) || (K % 8) || splits < 0 || splits > MAX_SPLIT) return kErrBadShape;
  if (swiglu && (bias != nullptr || residual != nullptr || (N % 16))) return kErrBadShape;
  if (!aligned16(x) || !aligned16(w) || !aligned16(out) || !aligned16(bias) || !aligned16(residual)) return kErrAlignment;
  if ((ldx % 8) || (ldw % 8) || (ldo % 8) || (residual != nullptr && (ldr % 8))) return kErrAlignment;
  CUtensorMap tmW, tmX;
  Params p = {};
  int MT;
  p.F = N / 2;
  const int tiles = swiglu ? (p.F + 63) / 64 : (N + BN - 1) / BN;
  const int rc = setup(x, w, M, N, K, ldx, ldw, tiles, splits, &tmW, &tmX, &MT, &p);
  if (rc != kLaunchOk) return rc;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ldo = ldo;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.ldr = ldr;
  p.weights_ready = weights_ready;
  p.status = status;
#define PD_SKINNY(MT_)                                                     \
  if (MT == MT_) return swiglu ? launch<MT_, kSwiglu>(tmW, tmX, p, tiles, stream) : launch<MT_, kStore>(tmW, tmX, p, tiles, stream);
  PD_SKINNY(16) PD_SKINNY(32) PD_SKINNY(64) PD_SKINNY(128)
#undef PD_SKINNY
  return kErrBadShape;
}

// The qkv projection of a decode step with everything that follows it up to the attention: x [M, K] times W [K, (Hq + 2 Hkv) * 128]
// (+ bias), rotary embedding of the q and k heads at position seq_lens[m] (cos / sin [max_pos, 64] fp32), q to q_out [M, Hq, 128],
// the new k / v rows into the cache pages that the block table names (`pages` entries a row, rows `table_stride` apart).  A sequence
// whose position is outside the rotary table or its pages is left out.
PD_EXPORT int pd_gemm_skinny_qkv(const void* x, const void* w, const void* bias, const float* cos_t, const float* sin_t,
                                 const int* seq_lens, const int* block_table, void* q_out, void* k_cache, void* v_cache, int M,
                                 int K, int ldx, int ldw, int Hq, int Hkv, int table_stride, int pages, int max_pos, int weights_ready,
                                 int* status, cudaStream_t stream) {
  using namespace pd;
  using namespace pd::skinny;
  if (M <= 0 || M > 128 || K <= 0 || (K % 8) || Hq <= 0 || Hkv <= 0 || pages < 1 || table_stride < 1) return kErrBadShape;
  if (!aligned16(x) || !aligned16(w) || !aligned16(bias) || !aligned16(q_out) || !aligned16(k_cache) || !aligned16(v_cache))
    return kErrAlignment;
  if ((ldx % 8) || (ldw % 8)) return kErrAlignment;
  CUtensorMap tmW, tmX;
  Params p = {};
  int MT;
  const int heads = Hq + 2 * Hkv;
  const int rc = setup(x, w, M, heads * BN, K, ldx, ldw, heads, 0, &tmW, &tmX, &MT, &p);
  if (rc != kLaunchOk) return rc;
  p.out = static_cast<__nv_bfloat16*>(q_out);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.weights_ready = weights_ready;
  p.status = status;
  p.cos_t = cos_t;
  p.sin_t = sin_t;
  p.seq_lens = seq_lens;
  p.block_table = block_table;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.table_stride = table_stride;
  p.pages = pages;
  p.max_pos = max_pos;
#define PD_SKINNY(MT_) \
  if (MT == MT_) return launch<MT_, kQkv>(tmW, tmX, p, heads, stream);
  PD_SKINNY(16) PD_SKINNY(32) PD_SKINNY(64) PD_SKINNY(128)
#undef PD_SKINNY
  return kErrBadShape;
}
