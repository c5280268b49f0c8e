// bfloat16 matrix product on pairs of SMs:  out[t, n] = sum_k X[t, k] * W[n, k]  for many tokens (prefill).
//
// Two CTAs of a cluster share one 256 x BN tile through `tcgen05.mma.cta_group::2`: each CTA stages 128
// weight rows (the M operand) and HALF of the token rows (the N operand) in its own shared memory, the
// leader CTA issues one MMA that reads both halves, and each CTA ends up with its 128 output features
// for all BN tokens in its own tensor memory.  Per SM and k-step that is 16 KB of weights + 16 KB of
// tokens for a 128 x 256 x 64 product, two thirds of what a single-CTA tile of the same shape pulls
// through the L2 -- and the L2 is what bounds the single-CTA kernel (gemm_tc.cu) at these sizes.
//
// Synchronisation: TMA loads of both CTAs complete on the LEADER's full barrier (`cta_group::2` loads may
// signal the peer's barrier; no multicast load is used); the leader's `tcgen05.commit` with
// `multicast::cluster` frees the stage in both CTAs and, at the end, tells both that the accumulators
// are complete.  Every wait is bounded; a CTA that gives up raises the error flag and leaves.
// Epilogues as in gemm_tc.cu: STORE, ADD (float32 residual), SWIGLU, with groups (routed experts), a
// per-token scale and output row scatter; no split-K here.
// The reference has no tensor-core kernel of its own (src/kernels/kernels_ops_matvec.cu:343-418 are
// SIMT GEMVs); this file has no counterpart there.
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include <cuda.h>

namespace cpi {
namespace tc {
int get_map_2d_bf16(const void* ptr, uint64_t inner, uint64_t rows, uint64_t row_stride_bytes, uint32_t box_inner,
                    uint32_t box_rows, CUtensorMap* out);
int get_map_3d_bf16(const void* ptr, uint64_t inner, uint64_t rows, uint64_t groups, uint32_t box_inner,
                    uint32_t box_rows, CUtensorMap* out);
}
namespace tc2 {

constexpr int BM = 128;          // output features per CTA (256 per pair)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr uint32_t kSpinLimit = 1u << 24;
constexpr int kMaxSlots = 512;     // token tiles of a grouped product that the persistent kernel lists
// Two rules for every launch of a kernel on pairs.
// No early start: these kernels are launched without programmatic dependence, after the kernel before them has ended (that one's
// successors may start early as elsewhere).  Started early behind row kernels of many blocks, now and then such a product did
// not return: prompts of 32,768 tokens (query product behind the norm and the page write, 32,768 blocks each) stopped within 11 to 50
// passes, whether two pairs shared an SM pair or one had it alone; without the early start 525 passes ran through.  It costs a
// product 2 to 4 us (a latent prompt's mixer of 2,048 tokens 167 -> 179 us with its four).
// Alone: a CTA takes more than half of an SM's shared memory, so that no second pair and no other CTA with tensor memory shares
// an SM with it.  `tcgen05.alloc.cta_group::2` has no limit and needs both SMs of the pair: of two pairs that start on the same two SMs
// at one time, one may come first on the one SM and the other on the other.
constexpr int kAlone = 116 * 1024;
enum Mode : int { kStore = 0, kAdd = 1, kSwiglu = 2 };

struct Params {
  void* out; long ldo;
  const int* out_rows;
  const float* row_scale;
  const int* group_offsets; int n_groups;      // routed experts: tokens [offsets[g], offsets[g+1]) use W[g]
  int T, bn, N, k_tiles;
  int* error_flag;
  int gate_act;                                // gated mode: the gate's activation (0 silu, 1 gelu in its tanh form, 2 clamped)
  float gate_limit;                            // the clamp of act 2 (see epi::gate_mul)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// loads of a CTA pair: data into this CTA's shared memory, completion on the barrier at cluster address `bar`
__device__ __forceinline__ void tma2_load_2d(void* smem, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(smem)), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma2_load_3d(void* smem, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(smem_u32(smem)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
// arrives on the barrier at the same shared-memory offset in both CTAs of the pair
__device__ __forceinline__ void umma2_commit_both(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, float* v) {      // complete after tcgen05.wait::ld
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ uint32_t instr_desc_pair(int n) {       // M = 256 over the pair
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}
template <typename TO> __device__ __forceinline__ void store_out(TO* p, float v);
template <> __device__ __forceinline__ void store_out<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void store_out<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// The epilogue of a thread (one output feature n, the tile's tokens in tensor memory from `acc` on, the second accumulator's from
// `acc2` on) for rows that do not start on 16 bytes and for narrow tiles: straight from the registers.
template <int MODE, typename TO>
__device__ __forceinline__ void direct(const Params& p, uint32_t acc, uint32_t acc2, int n, int t0, int n_valid_t, int n_cols) {
  const bool row_ok = n < p.N;
  TO* out = reinterpret_cast<TO*>(p.out);
  if (MODE == kAdd) {
    float* outf = reinterpret_cast<float*>(p.out);
    float old[2][16];
    auto fetch = [&](int c, float* dst) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int col = c + j;
        dst[j] = (row_ok && col < n_valid_t) ? outf[(size_t)(p.out_rows ? p.out_rows[t0 + col] : t0 + col) * p.ldo + n] : 0.f;
      }
    };
    fetch(0, old[0]);
#pragma unroll 1
    for (int c = 0; c < n_cols; c += 32) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cc = c + 16 * h;
        if (cc >= n_cols) break;
        if (cc + 16 < n_cols) fetch(cc + 16, old[h ^ 1]);
        float v[16];
        tmem_ld16(acc + cc, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int col = cc + j;
          if (row_ok && col < n_valid_t) {
            const float s = p.row_scale ? p.row_scale[t0 + col] : 1.0f;
            outf[(size_t)(p.out_rows ? p.out_rows[t0 + col] : t0 + col) * p.ldo + n] = old[h][j] + v[j] * s;
          }
        }
      }
    }
    return;
  }
#pragma unroll 1
  for (int c = 0; c < n_cols; c += 16) {
    float v[16], u[16];
    tmem_ld16(acc + c, v);
    if (MODE == kSwiglu) tmem_ld16(acc2 + c, u);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int col = c + j;
      if (!row_ok || col >= n_valid_t) continue;
      const float s = p.row_scale ? p.row_scale[t0 + col] : 1.0f;
      float x = v[j] * s;
      if (MODE == kSwiglu) x = epi::gate_mul(x, u[j] * s, p.gate_act, p.gate_limit);
      if (MODE == kStore) x = epi::store_act(x, p.gate_act);
      store_out<TO>(out + (size_t)(p.out_rows ? p.out_rows[t0 + col] : t0 + col) * p.ldo + n, x);
    }
  }
}

template <int BN, int MODE, typename TO, int STAGES>
__global__ void __launch_bounds__(128) gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_w,
                                                           const __grid_constant__ CUtensorMap map_x, Params p) {
  constexpr int ACC = MODE == kSwiglu ? 2 : 1;
  constexpr int HALF = BN / 2;                                   // token rows this CTA stages, at most
  constexpr uint32_t A_BYTES = BM * BK * 2, B_BYTES = HALF * BK * 2;
  constexpr uint32_t STAGE_BYTES = ACC * A_BYTES + B_BYTES;
  constexpr int BOX_ROWS = 64;
  constexpr uint32_t BOX_BYTES = BOX_ROWS * BK * 2;
  constexpr uint32_t TMEM_COLS = ACC * BN;
  static_assert(BN % 128 == 0 && TMEM_COLS <= 512, "pair tiles are 128 or 256 tokens wide");
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], accum_bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  __shared__ int offs_s[257], tiles_s[256], found_s[2];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t rank = cluster_rank();                          // 0: leader (issues the MMAs), 1: peer

  // ---- which tile (both CTAs of a pair share blockIdx.y, so they find the same one) ----
  int group = 0, t_begin = 0, t_end = p.T, tile_t = blockIdx.y;
  if (p.group_offsets) {
    pdl_wait();
    for (int g = tid; g < p.n_groups; g += 128) {
      const int b = p.group_offsets[g], e = p.group_offsets[g + 1];
      offs_s[g] = b;
      tiles_s[g] = (e - b + p.bn - 1) / p.bn;
      if (g == p.n_groups - 1) offs_s[g + 1] = e;
    }
    __syncthreads();
    if (tid == 0) {
      int rest = tile_t, hit = -1;
      for (int g = 0; g < p.n_groups; ++g) {
        if (rest < tiles_s[g]) { hit = g; break; }
        rest -= tiles_s[g];
      }
      found_s[0] = hit;
      found_s[1] = rest;
    }
    __syncthreads();
    if (found_s[0] < 0) return;                                  // both CTAs of the pair leave together
    group = found_s[0]; tile_t = found_s[1]; t_begin = offs_s[group]; t_end = offs_s[group + 1];
  }
  int pair_n = blockIdx.x >> 1;                                  // which 256 output features
  if (!p.group_offsets) {
    // Dense product: pairs are handed out (x fastest, then y) so that the ones running at the same time
    // cover a band of up to 8 token tiles times as many weight tiles as fit: a wave then pulls about
    // 8 + 9 operand strips through the L2 instead of 28 + 3, and the weights come from DRAM once.
    const int n_pairs = gridDim.x >> 1, n_tok = gridDim.y, W = 8;
    const int pid = blockIdx.y * n_pairs + pair_n;
    const int band = pid / (W * n_pairs), rem = pid - band * W * n_pairs;
    const int w_eff = min(W, n_tok - band * W);
    tile_t = band * W + rem % w_eff;
    pair_n = rem / w_eff;
  }
  const int n0 = (pair_n * 2 + (int)rank) * BM;                  // this CTA's output features
  const int t0 = t_begin + tile_t * p.bn;
  const int n_valid_t = min(p.bn, t_end - t0);
  const int n_mma = min(BN, (n_valid_t + 31) & ~31);             // MMA width: both halves stay multiples of 16
  const int half = n_mma / 2;                                    // token rows of the tile staged by each CTA
  const int n_boxes = (half + BOX_ROWS - 1) / BOX_ROWS;
  const uint32_t cta_tx = ACC * A_BYTES + (uint32_t)n_boxes * BOX_BYTES;
  const int n_kt = p.k_tiles;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&accum_bar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();                                                // the peer's barriers exist before anyone signals them
  fence_after_sync();
  pdl_launch_dependents();                                       // (not before the tensor memory is ours: see common.cuh)
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort_flag = &abort_s;

  if (warp == 0 && lane == 0) {
    // ---- TMA producer (both CTAs): weights before the wait on the preceding kernel, tokens after ----
    const int n_early = p.group_offsets ? 0 : min(n_kt, STAGES);
    for (int i = 0; i < n_early; ++i) {
      uint8_t* st = smem + (size_t)i * STAGE_BYTES;
      const uint32_t bar = map_to_cta(smem_u32(&full_bar[i]), 0);
      if (rank == 0) mbar_expect_tx(&full_bar[i], 2 * cta_tx);
      tma2_load_3d(st, &map_w, bar, i * BK, n0, group);
      if (ACC == 2) tma2_load_3d(st + A_BYTES, &map_w, bar, i * BK, p.N + n0, group);
    }
    pdl_wait();
    for (int i = 0; i < n_early; ++i) {
      const uint32_t bar = map_to_cta(smem_u32(&full_bar[i]), 0);
      for (int b = 0; b < n_boxes; ++b)
        tma2_load_2d(smem + (size_t)i * STAGE_BYTES + ACC * A_BYTES + b * BOX_BYTES, &map_x, bar, i * BK,
                     t0 + (int)rank * half + b * BOX_ROWS);
    }
    for (int i = n_early; i < n_kt; ++i) {
      const int s = i % STAGES;
      if (i >= STAGES && !mbar_wait(&empty_bar[s], ((i / STAGES) - 1) & 1, abort_flag)) break;
      uint8_t* st = smem + (size_t)s * STAGE_BYTES;
      const uint32_t bar = map_to_cta(smem_u32(&full_bar[s]), 0);
      if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * cta_tx);
      tma2_load_3d(st, &map_w, bar, i * BK, n0, group);
      if (ACC == 2) tma2_load_3d(st + A_BYTES, &map_w, bar, i * BK, p.N + n0, group);
      for (int b = 0; b < n_boxes; ++b)
        tma2_load_2d(st + ACC * A_BYTES + b * BOX_BYTES, &map_x, bar, i * BK, t0 + (int)rank * half + b * BOX_ROWS);
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer (leader only): one instruction spans both CTAs ----
    const uint32_t idesc = instr_desc_pair(n_mma);
    bool ok = true;
    for (int i = 0; i < n_kt && ok; ++i) {
      const int s = i % STAGES;
      ok = mbar_wait(&full_bar[s], (i / STAGES) & 1, abort_flag);
      if (!ok) break;
      fence_after_sync();
      const uint32_t a_addr = smem_u32(smem + (size_t)s * STAGE_BYTES);
      const uint64_t da = smem_desc_sw128(a_addr), db = smem_desc_sw128(a_addr + ACC * A_BYTES);
#pragma unroll
      for (int j = 0; j < BK / UMMA_K; ++j) {
        const uint32_t acc = (i > 0 || j > 0) ? 1u : 0u;
        umma2_bf16(tmem_base, da + 2 * j, db + 2 * j, idesc, acc);
        if (ACC == 2) umma2_bf16(tmem_base + BN, smem_desc_sw128(a_addr + A_BYTES) + 2 * j, db + 2 * j, idesc, acc);
      }
      umma2_commit_both(&empty_bar[s]);
    }
    if (ok) umma2_commit_both(&accum_bar);
  }
  __syncwarp();

  // ---- epilogue: each CTA stores its 128 features of all the tile's tokens ----
  pdl_wait();
  bool ok = mbar_wait(&accum_bar, 0, abort_flag);
  fence_after_sync();
  ok = __syncthreads_and(ok && !abort_s) != 0;                   // one decision for the CTA
  const int row = warp * 32 + lane;
  const int n = n0 + row;
  const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
  const int n_cols = min(BN, (n_valid_t + 15) & ~15);
  TO* out = reinterpret_cast<TO*>(p.out);
  if (ok && epi::staged_ok<TO>(p.out, p.ldo, n_valid_t)) {
    // the tile is turned in shared memory (the stages are idle: every MMA has completed) and leaves in
    // whole rows
    constexpr int kFit = (int)((size_t)STAGES * STAGE_BYTES / (128 * sizeof(TO))) / 16 * 16;   // columns the idle stages hold
      constexpr int kStageCols = kFit < BN ? kFit : BN;
      auto ld = [&](int c, float* d) { tmem_ld16(lane_addr + c, d); };
    auto ldu = [&](int c, float* d) { tmem_ld16(lane_addr + BN + c, d); };
    epi::staged<MODE, TO, kStageCols>(smem, ld, ldu, warp, lane, n0, p.N, t0, n_valid_t, n_cols, out, p.ldo, p.out_rows, p.row_scale, epi::CtaSync(), p.gate_act, p.gate_limit);
  } else if (ok) {
    direct<MODE, TO>(p, lane_addr, ACC == 2 ? lane_addr + BN : 0u, n, t0, n_valid_t, n_cols);
  }
  if (!ok) {
    if (tid == 0 && p.error_flag) atomicExch(p.error_flag, 3);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();                                                // neither CTA leaves while the other may still use it
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
}

// ---------------------------------------------------------------------------------------------- two tiles at a time
// Dense products with one accumulator: a pair of CTAs per SM pair whose two halves of 128 threads work on a tile each, with
// rings, barriers and 256 columns of tensor memory of their own, so that one's fill and epilogue run under the other's
// products.  Tiles go round the halves: c, then c + clusters, .. for the halves of cluster c, so with fewer tiles than SM
// pairs every tile has one to itself.  (Two pairs of CTAs that shared an SM pair did the same work; see kAlone for what was wrong.)
struct HalfSync {
  int id;
  __device__ __forceinline__ void operator()() const { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
};

template <int BN, int MODE, typename TO, int STAGES>
__global__ void __launch_bounds__(256) gemm_tc_pair_dual_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                const __grid_constant__ CUtensorMap map_x, Params p, int n_pairs,
                                                                int n_tok) {
  constexpr uint32_t A_BYTES = BM * BK * 2, STAGE_BYTES = A_BYTES + (BN / 2) * BK * 2, RING = STAGES * STAGE_BYTES;
  constexpr int BOX_ROWS = 64;
  constexpr uint32_t BOX_BYTES = BOX_ROWS * BK * 2;
  constexpr uint32_t TMEM_COLS = 2 * BN;
  static_assert(MODE != kSwiglu && TMEM_COLS <= 512, "two tiles with one accumulator each");
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_all[2][STAGES], empty_all[2][STAGES], accum_all[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s[2];

  const int tid = threadIdx.x, half_no = tid >> 7, warp = (tid >> 5) & 3, lane = tid & 31;
  const uint32_t rank = cluster_rank();                          // 0: leader (issues the MMAs), 1: peer
  if (tid == 0) {
    for (int h = 0; h < 2; ++h) {
      for (int s = 0; s < STAGES; ++s) { mbar_init(&full_all[h][s], 1); mbar_init(&empty_all[h][s], 1); }
      mbar_init(&accum_all[h], 1);
      abort_s[h] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();                                                // the peer's barriers exist before anyone signals them
  fence_after_sync();
  pdl_launch_dependents();                                       // (not before the tensor memory is ours: see common.cuh)
  uint64_t *full_bar = full_all[half_no], *empty_bar = empty_all[half_no], *accum_bar = &accum_all[half_no];
  uint8_t* ring = smem + half_no * RING;
  const uint32_t tmem = tmem_base_s + half_no * BN;
  volatile int* abort_flag = &abort_s[half_no];
  const HalfSync sync{1 + half_no};
  const int n_clusters = gridDim.x >> 1, n_tiles = n_pairs * n_tok, n_kt = p.k_tiles;
  int it = 0, j = 0;                                             // k steps and tiles of this half before the present tile
  for (int pid = (blockIdx.x >> 1) + half_no * n_clusters; pid < n_tiles; pid += 2 * n_clusters, ++j, it += n_kt) {
    // bands of up to 8 token tiles times as many weight tiles as run at one time: see the kernel above
    const int W = 8, band = pid / (W * n_pairs), rem = pid - band * W * n_pairs, w_eff = min(W, n_tok - band * W);
    const int t0 = (band * W + rem % w_eff) * p.bn, n_valid_t = min(p.bn, p.T - t0);
    const int n0 = ((rem / w_eff) * 2 + (int)rank) * BM;         // this CTA's output features
    const int n_mma = min(BN, (n_valid_t + 31) & ~31), half = n_mma / 2;
    const int n_boxes = (half + BOX_ROWS - 1) / BOX_ROWS;
    const uint32_t cta_tx = A_BYTES + (uint32_t)n_boxes * BOX_BYTES;
    auto load_w = [&](int i) {
      const int s = (it + i) % STAGES;
      if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * cta_tx);
      tma2_load_3d(ring + (size_t)s * STAGE_BYTES, &map_w, map_to_cta(smem_u32(&full_bar[s]), 0), i * BK, n0, 0);
    };
    auto load_x = [&](int i) {
      const int s = (it + i) % STAGES;
      for (int b = 0; b < n_boxes; ++b)
        tma2_load_2d(ring + (size_t)s * STAGE_BYTES + A_BYTES + b * BOX_BYTES, &map_x, map_to_cta(smem_u32(&full_bar[s]), 0), i * BK,
                     t0 + (int)rank * half + b * BOX_ROWS);
    };
    if (warp == 0 && lane == 0) {
      // ---- TMA producer (both CTAs): the first tile's weights before the wait on the preceding kernel, tokens after ----
      const int n_early = j == 0 ? min(n_kt, STAGES) : 0;
      for (int i = 0; i < n_early; ++i) load_w(i);
      if (j == 0) pdl_wait();
      for (int i = 0; i < n_early; ++i) load_x(i);
      for (int i = n_early; i < n_kt; ++i) {
        const int g = it + i;
        if (g >= STAGES && !mbar_wait(&empty_bar[g % STAGES], ((g / STAGES) - 1) & 1, abort_flag)) break;
        load_w(i);
        load_x(i);
      }
    } else if (warp == 1 && lane == 0 && rank == 0) {
      // ---- MMA issuer (leader only): one instruction spans both CTAs ----
      const uint32_t idesc = instr_desc_pair(n_mma);
      bool ok = true;
      for (int i = 0; i < n_kt && ok; ++i) {
        const int g = it + i, s = g % STAGES;
        ok = mbar_wait(&full_bar[s], (g / STAGES) & 1, abort_flag);
        if (!ok) break;
        fence_after_sync();
        const uint32_t a_addr = smem_u32(ring + (size_t)s * STAGE_BYTES);
        const uint64_t da = smem_desc_sw128(a_addr), db = smem_desc_sw128(a_addr + A_BYTES);
#pragma unroll
        for (int q = 0; q < BK / UMMA_K; ++q) umma2_bf16(tmem, da + 2 * q, db + 2 * q, idesc, (i > 0 || q > 0) ? 1u : 0u);
        umma2_commit_both(&empty_bar[s]);
      }
      if (ok) umma2_commit_both(accum_bar);
    }
    __syncwarp();
    // ---- epilogue: this half of each CTA stores its 128 features of the tile's tokens ----
    if (j == 0) pdl_wait();
    mbar_wait(accum_bar, j & 1, abort_flag);
    sync();                                                      // one decision for the half: nobody sets its flag from here on
    if (abort_s[half_no]) break;
    fence_after_sync();
    const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
    const int n_cols = min(BN, (n_valid_t + 15) & ~15);
    TO* out = reinterpret_cast<TO*>(p.out);
    if (epi::staged_ok<TO>(p.out, p.ldo, n_valid_t)) {
      // turned in the half's stages, which are idle: every MMA has completed
      constexpr int kFit = (int)((size_t)RING / (128 * sizeof(TO))) / 16 * 16, kStageCols = kFit < BN ? kFit : BN;
      auto ld = [&](int c, float* d) { tmem_ld16(lane_addr + c, d); };
      epi::staged<MODE, TO, kStageCols>(ring, ld, ld, warp, lane, n0, p.N, t0, n_valid_t, n_cols, out, p.ldo, p.out_rows, p.row_scale,
                                        sync, p.gate_act, p.gate_limit);
    } else {
      direct<MODE, TO>(p, lane_addr, 0u, n0 + warp * 32 + lane, t0, n_valid_t, n_cols);
    }
    // The next tile's loads overwrite the stages (through the async proxy), its products the accumulator: they wait for this
    // CTA's loads, the loads for all of this half.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    fence_before_sync();
    sync();
  }
  __syncwarp();
  if (abort_s[half_no]) {
    if ((tid & 127) == 0 && p.error_flag) atomicExch(p.error_flag, 3);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();                                                // neither CTA leaves while the other may still use it
  if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_s), "r"(TMEM_COLS));
}

// ---------------------------------------------------------------------------------------------- persistent
// The same product with one pair per SM pair that works through a list of tiles (dense products only).
// Warps 0-3 own the accumulator's lanes and run the epilogue, warp 4 issues the TMA loads, warp 5 (of the leading CTA) the
// MMAs; the gated form has twelve warps, 8-11 a second group of the epilogue.  The stage ring runs on across tiles, and with one accumulator per
// tile there are two accumulator buffers in tensor memory: the MMAs of tile j+1 run while tile j is turned
// in shared memory and written out, so an SM pair's tiles follow each other at the tensor pipe's rate
// instead of each paying fill, drain and epilogue.  With two accumulators, SwiGLU, the tensor memory
// holds one tile, whose successor's MMAs wait until it has been read (its loads do not): two groups of four warps take half of
// the tokens each, keep their gated products as packed bfloat16 in registers (64 a thread), give the accumulators
// back and turn and store the tile under the next one's MMAs.  A pair with one tile takes the loop over 16 tokens at a time that
// the other forms take: all of that unrolled code, run once, costs more than it saves.  By four warps that gave the accumulators
// back with the last token stored / by two groups / by two groups with the loop, in us: gate/up of 16 experts of 2,048 x 2,048
// at 512 rows each 141 / 132 / 134; one tile a pair, 512 x 2,048 -> 8,192 pairs 34.0 / 36.0 / 32.9, 2,048 x 1,024 -> 2,048 24.2 / 25.6 /
// 22.7, 8 experts of 2,048 x 1,024 at 192 rows 36.0 / 39.1 / 33.9.
//   full[s] / empty[s]            stage ring, as above
//   acc_full[b]                   MMA -> epilogue warps of both CTAs (commit with multicast)
//   acc_empty[b] (in the leader)  epilogue warps of both CTAs -> MMA: one arrival per warp, 8 in all (16 with two groups)
// The gated products of a group's tokens (up to 128 of the tile, from `acc` on), packed two tokens a register.
__device__ __forceinline__ void gated_read(uint32_t acc, uint32_t acc2, int n_cols, int n_valid_t, const float* scale, int act, float limit,
                                           uint32_t (&packed)[64]) {
#pragma unroll
  for (int c = 0; c < 128; c += 16) {
    if (c >= n_cols) continue;
    float v[16], u[16];
    tmem_ld16_issue(acc + c, v);
    tmem_ld16_issue(acc2 + c, u);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) asm volatile("" : "+f"(v[j]), "+f"(u[j]));      // (not before the wait)
    if (scale) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float f = scale[min(c + j, n_valid_t - 1)];
        v[j] *= f;
        u[j] *= f;
      }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = epi::gate_mul(v[j], u[j], act, limit);
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const __nv_bfloat162 two = __floats2bfloat162_rn(v[j], v[j + 1]);
      packed[(c + j) / 2] = *reinterpret_cast<const uint32_t*>(&two);
    }
  }
}
// Turned in shared memory 32 tokens at a time (a thread has a feature's), and out in rows; 128 threads, `sync` their barrier.
template <typename Sync>
__device__ __forceinline__ void gated_store(const uint32_t (&packed)[64], __nv_bfloat16* stage, int warp, int lane, int n0, int N, int t0,
                                            int n_valid_t, __nv_bfloat16* out, long ldo, const int* out_rows, Sync sync) {
  const int n = n0 + 4 * lane;
#pragma unroll
  for (int p0 = 0; p0 < 128; p0 += 32) {
    if (p0 >= n_valid_t) continue;
    if (p0 > 0) sync();                                          // the pass before has been copied out
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const uint32_t w = packed[(p0 + j) / 2];
      const __nv_bfloat162 two = *reinterpret_cast<const __nv_bfloat162*>(&w);
      stage[j * 128 + warp * 32 + lane] = two.x;
      stage[(j + 1) * 128 + warp * 32 + lane] = two.y;
    }
    sync();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int col = p0 + warp + 4 * q;
      if (col >= n_valid_t) break;
      const uint2 x = *reinterpret_cast<const uint2*>(stage + (col - p0) * 128 + 4 * lane);
      __nv_bfloat16* to = out + (size_t)(out_rows ? out_rows[t0 + col] : t0 + col) * ldo + n;
      if (n + 4 <= N) {
        *reinterpret_cast<uint2*>(to) = x;
      } else {
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&x);
        for (int i = 0; i < 4 && n + i < N; ++i) to[i] = e[i];
      }
    }
  }
}
// One decision of 128 threads that meet at barrier `id`: whether any of them says so.
__device__ __forceinline__ bool any_of_group(int id, bool x) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(r) : "r"((uint32_t)x), "r"(id) : "memory");
  return r != 0;
}

template <int BN, int MODE, typename TO, int STAGES>
__global__ void __launch_bounds__(MODE == kSwiglu ? 384 : 192) gemm_tc_pair_persistent_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                      const __grid_constant__ CUtensorMap map_x,
                                                                      Params p, int n_pairs, int n_tok) {
  constexpr int ACC = MODE == kSwiglu ? 2 : 1;
  constexpr int NB = ACC == 1 ? 2 : 1;                           // accumulator buffers in tensor memory
  constexpr int GROUPS = ACC;                                    // groups of four epilogue warps: 0 to 3, and 8 to 11
  constexpr int HALF = BN / 2;
  constexpr uint32_t A_BYTES = BM * BK * 2, B_BYTES = HALF * BK * 2;
  constexpr uint32_t STAGE_BYTES = ACC * A_BYTES + B_BYTES;
  constexpr int BOX_ROWS = 64;
  constexpr uint32_t BOX_BYTES = BOX_ROWS * BK * 2;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr int EPI_COLS = 64;                                   // columns turned at a time
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[NB], acc_empty[NB];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s, n_live_s;
  __shared__ int slot_group[kMaxSlots], slot_t0[kMaxSlots], slot_rows[kMaxSlots];     // groups: the token tiles that hold rows
  __shared__ short slot_first[kMaxSlots], slot_count[kMaxSlots];                     // ... and their group's first tile and tile count

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* ring = smem;
  uint8_t* epi = smem + (size_t)STAGES * STAGE_BYTES;
  const uint32_t rank = cluster_rank();
  const bool grouped = p.group_offsets != nullptr;
  if (grouped) {
    // the row lists come from the kernel before this one; one thread walks the groups and lists their tiles
    pdl_wait();
    if (tid == 0) {
      int n = 0;
      for (int g = 0; g < p.n_groups; ++g) {
        const int b = p.group_offsets[g], e = p.group_offsets[g + 1], first = n;
        // a group with more rows than a tile takes is cut into tiles of about equal size (a multiple of 32 rows):
        // the tile numbers go round the SM pairs, and a full tile beside a nearly empty one would give every
        // second pair the full ones
        const int count = (e - b + p.bn - 1) / p.bn;
        const int per = count > 0 ? (((e - b + count - 1) / count + 31) & ~31) : p.bn;
        for (int t = b; t < e && n < kMaxSlots; t += per) { slot_group[n] = g; slot_t0[n] = t; slot_rows[n] = min(per, e - t); ++n; }
        for (int i = first; i < n; ++i) { slot_first[i] = (short)first; slot_count[i] = (short)(n - first); }
      }
      n_live_s = n;
    }
    __syncthreads();
  }
  const int n_tok_live = grouped ? n_live_s : n_tok;
  const int n_tiles = n_pairs * n_tok_live;
  const int n_clusters = gridDim.x >> 1, cluster_id = blockIdx.x >> 1;
  const int n_kt = p.k_tiles;
  // tile number -> (first token row, rows, weight pair, group).  Dense: bands of 8 token tiles as in the kernel
  // above.  Groups: group after group, within a group weight pair after weight pair, and the group's token tiles
  // for one weight pair next to each other: the SM pairs that run them at the same time share the weights' way
  // through the L2, so a group's weights are read from memory once however many token tiles it has, and its rows
  // (a few MB) stay in the L2 while its weight pairs go by.
  auto tile_of = [&](int pid, int& t0, int& n_valid_t, int& pair_n, int& group) {
    if (grouped) {
      const int s = pid / n_pairs;                       // a tile of the group (its tiles own n_pairs numbers each)
      const int first = slot_first[s], count = slot_count[s];
      const int local = pid - first * n_pairs;
      pair_n = local / count;
      const int slot = first + (local - pair_n * count);
      group = slot_group[slot]; t0 = slot_t0[slot]; n_valid_t = slot_rows[slot];
      return;
    }
    const int W = 8;
    const int band = pid / (W * n_pairs), rem = pid - band * W * n_pairs;
    const int w_eff = min(W, n_tok - band * W);
    const int tile_t = band * W + rem % w_eff;
    pair_n = rem / w_eff;
    group = 0; t0 = tile_t * p.bn; n_valid_t = min(p.bn, p.T - t0);
  };

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < NB; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8 * GROUPS); }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();
  fence_after_sync();
  pdl_launch_dependents();                                       // (not before the tensor memory is ours: see common.cuh)
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort_flag = &abort_s;

  if (warp == 4) {
    if (lane == 0) {
      // ---- TMA producer (both CTAs); weights need no wait on the preceding kernel, tokens do ----
      bool waited = false;
      int it = 0;
      for (int pid = cluster_id; pid < n_tiles; pid += n_clusters) {
        int t0, n_valid_t, pair_n, group;
        tile_of(pid, t0, n_valid_t, pair_n, group);
        const int n0 = (pair_n * 2 + (int)rank) * BM;
        const int half = min(BN, (n_valid_t + 31) & ~31) / 2;
        const int n_boxes = (half + BOX_ROWS - 1) / BOX_ROWS;
        const uint32_t cta_tx = ACC * A_BYTES + (uint32_t)n_boxes * BOX_BYTES;
        bool ok = true;
        for (int kt = 0; kt < n_kt; ++kt, ++it) {
          const int s = it % STAGES;
          if (it >= STAGES && !mbar_wait(&empty_bar[s], ((it / STAGES) - 1) & 1, abort_flag)) { ok = false; break; }
          uint8_t* st = ring + (size_t)s * STAGE_BYTES;
          const uint32_t bar = map_to_cta(smem_u32(&full_bar[s]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * cta_tx);
          tma2_load_3d(st, &map_w, bar, kt * BK, n0, group);
          if (ACC == 2) tma2_load_3d(st + A_BYTES, &map_w, bar, kt * BK, p.N + n0, group);
          if (!waited) { pdl_wait(); waited = true; }
          for (int b = 0; b < n_boxes; ++b)
            tma2_load_2d(st + ACC * A_BYTES + b * BOX_BYTES, &map_x, bar, kt * BK, t0 + (int)rank * half + b * BOX_ROWS);
        }
        if (!ok) break;
      }
    }
  } else if (warp == 5) {
    if (lane == 0 && rank == 0) {
      // ---- MMA issuer (leader only) ----
      int it = 0, j = 0;
      bool ok = true;
      for (int pid = cluster_id; pid < n_tiles && ok; pid += n_clusters, ++j) {
        int t0, n_valid_t, pair_n, group;
        tile_of(pid, t0, n_valid_t, pair_n, group);
        const uint32_t idesc = instr_desc_pair(min(BN, (n_valid_t + 31) & ~31));
        const int b = j % NB;
        if (j >= NB) ok = mbar_wait(&acc_empty[b], ((j / NB) - 1) & 1, abort_flag);     // the epilogue has read it
        if (!ok) break;
        fence_after_sync();
        const uint32_t d0 = tmem_base + b * (ACC * BN);
        for (int kt = 0; kt < n_kt; ++kt, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(&full_bar[s], (it / STAGES) & 1, abort_flag);
          if (!ok) break;
          fence_after_sync();
          const uint32_t a_addr = smem_u32(ring + (size_t)s * STAGE_BYTES);
          const uint64_t da = smem_desc_sw128(a_addr), db = smem_desc_sw128(a_addr + ACC * A_BYTES);
          const uint64_t da2 = smem_desc_sw128(a_addr + A_BYTES);
#pragma unroll
          for (int q = 0; q < BK / UMMA_K; ++q) {
            const uint32_t acc = (kt > 0 || q > 0) ? 1u : 0u;
            umma2_bf16(d0, da + 2 * q, db + 2 * q, idesc, acc);
            if (ACC == 2) umma2_bf16(d0 + BN, da2 + 2 * q, db + 2 * q, idesc, acc);
          }
          umma2_commit_both(&empty_bar[s]);
        }
        if (ok) umma2_commit_both(&acc_full[b]);
      }
    }
  } else if (warp < 4 || warp >= 8) {
    // ---- epilogue: each CTA stores its 128 features of the tile's tokens ----
    pdl_wait();
    const int group_no = warp >> 3, wq = warp & 3;               // (a warp reads the lanes of its number mod 4)
    const uint32_t leader_empty0 = map_to_cta(smem_u32(&acc_empty[0]), 0);
    int j = 0;
    for (int pid = cluster_id; pid < n_tiles; pid += n_clusters, ++j) {
      int t0, n_valid_t, pair_n, group;
      tile_of(pid, t0, n_valid_t, pair_n, group);
      const int n0 = (pair_n * 2 + (int)rank) * BM;
      const int n_cols = min(BN, (n_valid_t + 15) & ~15);
      const int b = j % NB;
      mbar_wait(&acc_full[b], (j / NB) & 1, abort_flag);
      // one decision for the four warps (a named barrier has no time limit: nobody may leave alone); it also
      // keeps the turning buffer of the tile before from being overwritten while a warp still copies it out
      if (any_of_group(1 + group_no, abort_s != 0)) break;
      fence_after_sync();
      const uint32_t lane_addr = tmem_base + b * (ACC * BN) + ((uint32_t)(wq * 32) << 16);
      // the accumulator has been read: one arrival per warp
      auto give_back = [&] {
        fence_before_sync();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];"
                       ::"r"(leader_empty0 + (uint32_t)(b * sizeof(uint64_t))) : "memory");
      };
      TO* out = reinterpret_cast<TO*>(p.out);
      if constexpr (MODE == kSwiglu) {
        const int mid = min((n_cols / 2 + 15) & ~15, n_valid_t), from = group_no ? mid : 0, valid = group_no ? n_valid_t - mid : mid;
        uint8_t* stage = epi + group_no * (EPI_COLS / GROUPS * 128 * sizeof(TO));
        if (j > 0 || pid + n_clusters < n_tiles) {
          uint32_t packed[64];
          gated_read(lane_addr + from, lane_addr + BN + from, valid, valid, p.row_scale ? p.row_scale + t0 + from : nullptr, p.gate_act,
                     p.gate_limit, packed);
          give_back();
          gated_store(packed, reinterpret_cast<__nv_bfloat16*>(stage), wq, lane, n0, p.N, t0 + from, valid, out, p.ldo, p.out_rows,
                      HalfSync{1 + group_no});
        } else {                                                 // the pair's only tile: nothing waits for the accumulators
          auto ld = [&](int c, float* d) { tmem_ld16(lane_addr + from + c, d); };
          auto ldu = [&](int c, float* d) { tmem_ld16(lane_addr + BN + from + c, d); };
          epi::staged<MODE, TO, EPI_COLS / GROUPS>(stage, ld, ldu, wq, lane, n0, p.N, t0 + from, valid, (valid + 15) & ~15, out, p.ldo,
                                                   p.out_rows, p.row_scale, HalfSync{1 + group_no}, p.gate_act, p.gate_limit);
        }
      } else {
        auto ld = [&](int c, float* d) { tmem_ld16(lane_addr + c, d); };
        epi::staged<MODE, TO, EPI_COLS>(epi, ld, ld, warp, lane, n0, p.N, t0, n_valid_t, n_cols, out, p.ldo, p.out_rows,
                                        p.row_scale, epi::NamedSync<1, 128>(), p.gate_act, p.gate_limit);
        give_back();                                             // (its last load precedes the last barrier above)
      }
    }
  }
  __syncwarp();
  if (abort_s) {
    if (tid == 0 && p.error_flag) atomicExch(p.error_flag, 4);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();                                                // neither CTA leaves while the other may still use it
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
}

// A launch of one pair of CTAs per SM pair, or per tile if there are fewer.
template <typename Kernel>
static int launch_clusters(Kernel kern, int smem, int threads, bool& attr_set, const char* name, const CUtensorMap& mw, const CUtensorMap& mx,
                           const Params& p, int n_pairs, int n_tok, cudaStream_t stream) {
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      set_error("%s: cannot reserve %d bytes of shared memory", name, smem);
      return 1;
    }
    attr_set = true;
  }
  int dev = 0, n_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  int clusters = n_sm / 2;
  if (clusters > n_pairs * n_tok) clusters = n_pairs * n_tok;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];                                   // (no early start: see above kAlone)
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  cudaLaunchKernelEx(&cfg, kern, mw, mx, p, n_pairs, n_tok);
  return check_launch(name);
}

template <int MODE, typename TO>
static int launch_dual(const CUtensorMap& mw, const CUtensorMap& mx, const Params& p, int n_pairs, int n_tok, cudaStream_t stream) {
  constexpr int STAGES = 3;
  constexpr int SMEM = 2 * STAGES * (BM + 128) * BK * 2;
  static_assert(SMEM >= kAlone, "a pair has its SM pair to itself");
  static bool attr_set = false;
  return launch_clusters(gemm_tc_pair_dual_kernel<256, MODE, TO, STAGES>, SMEM, 256, attr_set, "gemm_tc_pair_dual", mw, mx, p, n_pairs, n_tok, stream);
}

template <int BN, int MODE, typename TO>
static int launch_persistent(const CUtensorMap& mw, const CUtensorMap& mx, const Params& p, int n_pairs, int n_tok,
                             cudaStream_t stream) {
  constexpr int ACC = MODE == kSwiglu ? 2 : 1;
  constexpr int STAGE = ACC * BM * BK * 2 + (BN / 2) * BK * 2;
  constexpr int EPI = 64 * 128 * (int)sizeof(TO);
  constexpr int S0 = (222 * 1024 - EPI) / STAGE;
  constexpr int STAGES = S0 > 8 ? 8 : S0;
  constexpr int SMEM = STAGES * STAGE + EPI;
  static_assert(SMEM >= kAlone, "a pair has its SM pair to itself");
  static bool attr_set = false;
  return launch_clusters(gemm_tc_pair_persistent_kernel<BN, MODE, TO, STAGES>, SMEM, MODE == kSwiglu ? 384 : 192, attr_set, "gemm_tc_pair_persistent", mw, mx, p, n_pairs,
                         n_tok, stream);
}

template <int BN, int MODE, typename TO>
static int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Params& p, dim3 grid, cudaStream_t stream) {
  constexpr int ACC = MODE == kSwiglu ? 2 : 1;
  constexpr int STAGE = ACC * BM * BK * 2 + (BN / 2) * BK * 2;
  constexpr int S0 = 196 * 1024 / STAGE;
  constexpr int STAGES = S0 > 8 ? 8 : S0;
  constexpr int SMEM = STAGES * STAGE + 1024;
  static_assert(SMEM >= kAlone, "a pair has its SM pair to itself");
  auto kern = gemm_tc_pair_kernel<BN, MODE, TO, STAGES>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
      set_error("gemm_tc_pair: cannot reserve %d bytes of shared memory", SMEM);
      return 1;
    }
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];                                   // (no early start: see above kAlone)
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  count_launch();
  cudaLaunchKernelEx(&cfg, kern, mw, mx, p);
  return check_launch("gemm_tc_pair");
}

}  // namespace tc2
}  // namespace cpi

using namespace cpi;

// Whether the paired kernel takes this product, and the token-tile width it would use (0: not taken).
// Three kernels: a list of tiles one after another (persistent; 2: always), two tiles at a time or, with groups or two
// accumulators, a launch slot per tile (0: always), or by shape (1, the default).  All run at what the L2 can deliver to the SMs (a
// 256 x 256 pair tile at the tensor pipe's full rate would pull 64 bytes per cycle and SM, ~15 TB/s over the GPU; the MMA thread of
// the list kernel waits for operands a third of the time), and two tiles at a time hide that latency better for one accumulator:
// list / two at a time in us, bfloat16 stored: 2,048 x 2,048 -> 3,072 34 / 25, -> 5,120 47 / 42, 2,048 x 5,120 -> 7,168 148 / 115, 8,192 x
// 5,120 -> 7,168 467 / 439 (two pairs of CTAs that shared an SM pair took 110 and 414 there).  The list wins where two
// accumulators leave no room for a second tile, and where ADD's epilogue is long against the products.
static int g_persistent = 1;
extern "C" void cpi_gemm_tc_pair_persistent(int mode) { g_persistent = mode; }

// The token tile of a dense product, and what it costs: one pair per two SMs at a time, time ~ waves x (weight rows + half the
// tile width) per SM.
static int dense_tile(int T, int N, int swiglu, long* cost_out) {
  const long sm_pairs = cpi::sm_count() / 2 > 0 ? cpi::sm_count() / 2 : 1;
  long best_cost = -1;
  int bn = 0;
  const long pairs_x = (N + 255) / 256;
  const int w_rows = swiglu ? 256 : 128;
  for (int cand = 256; cand >= 160; cand -= 32) {
    const long pairs = pairs_x * ((T + cand - 1) / cand);
    const long waves = (pairs + sm_pairs - 1) / sm_pairs;
    const long cost = waves * (w_rows + cand / 2 + 16);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; bn = cand; }
  }
  *cost_out = best_cost;
  return bn;
}

extern "C" int cpi_gemm_tc_pair_plan(int T, int N, int K, int swiglu, int n_groups) {
  // Features that are no multiple of 256 leave part of the last pair's rows idle (their loads give zeros, their results are not
  // stored): at most a fifth of the work from 1,024 on.  Where such a product is faster here, `cpi_gemm_tc_pair_pays` says.
  if ((N % 256 != 0 && (N < 1024 || n_groups > 0)) || K % 8 != 0) return 0;
  if (n_groups > 0) {
    // experts: one token tile per expert (its weights are then read once), sized for 1.5 x the mean rows
    if (n_groups > 256 || T < 64 * n_groups) return 0;
    const int want = (3 * ((T + n_groups - 1) / n_groups) + 1) / 2;
    return want > 128 ? 256 : 128;
  }
  if (T < 512) return 0;
  long cost;
  return dense_tile(T, N, swiglu, &cost);
}

// Whether a dense product of features that are no multiple of 256 is faster on the pairs than on single CTAs.  Measured over
// 512 to 8,192 tokens, 1,025 to 32,008 features and K of 512 to 8,192 (single / pairs in us, float32 stored unless said):
//   single CTAs in one wave without splits lose little or win: 2,048 x 2,048 -> 2,056 23 / 22, -> 1,288 17 / 21;
//   more than a wave loses what the last one leaves idle: 2,048 x 2,048 -> 3,144 36 / 25, 512 -> 10,304 37 / 24, but
//     not below 1,152 features, where the pairs' idle rows weigh as much (8,192 x 1,024 -> 1,032 32 / 31, 8,192 deep 0.93 times)
//     (ADD 512 deep at 4,096 tokens and more is the exception: 0.87 to 1.2 times);
//   two accumulators leave one CTA an SM on either side, so there the two costs decide: 2,048 x 2,048 -> 4,104 62 / 61 at a ratio of
//     1.28, 3,000 -> 2,056 49 / 52 at 1.22, 4,096 -> 1,160 43 / 48 at 1.0;
//   splits meet in a reduction that the pairs don't have, for a shorter loop: 1,024 x 2,048 -> 1,032 in two splits 36 / 23, 5,120 deep
//     42 / 42; in three 1,024 deep 21 / 14, 5,120 deep 35 / 48.  Outputs whose rows do not start on 16 bytes cost the pairs more:
//     half that depth.
extern "C" int cpi_gemm_tc_plan(int T, int N, int K, int n_groups, int swiglu, int* bn_out, int* splits_out, int* live_y_out);
extern "C" int cpi_gemm_tc_pair_pays(int T, int N, int K, int swiglu) {
  int bn = 0, splits = 1, live = 0;
  if (T < 512 || N < 1024 || cpi_gemm_tc_plan(T, N, K, 0, swiglu, &bn, &splits, &live)) return 0;
  if (splits > 1) return (long)K * splits <= (N % 4 == 0 ? 9216 : 4608);
  const long sms = cpi::sm_count();
  const long waves = ((long)((N + 127) / 128) * ((T + bn - 1) / bn) + sms - 1) / sms;
  if (waves < 2 || N < 1152) return 0;
  if (!swiglu) return 1;
  long pairs_cost;
  dense_tile(T, N, swiglu, &pairs_cost);
  return waves * (bn + 256) * 40 > pairs_cost * 49;
}

// x [T, K] bf16 (row stride ldx), w [N or 2N][K] bf16 contiguous, out [T, N]; bn from cpi_gemm_tc_pair_plan.
extern "C" int cpi_gemm_tc_pair(const void* x, long ldx, const void* w, void* out, int out_dtype, long ldo,
                                const int* out_rows, const float* row_scale, const int* group_offsets, int n_groups,
                                int T, int N, int K, int mode, int bn, int* error_flag, float gate_limit,
                                cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  // modes 3, 4: the gated mode with a gelu / a clamped gate; modes 5, 6: the storing mode with a squared relu / a gelu
  const int gate_act = mode == 3 ? 1 : mode == 4 ? 2 : mode == 5 ? 3 : mode == 6 ? 4 : 0;
  if (mode == 3 || mode == 4) mode = 2;
  if (mode == 5 || mode == 6) mode = 0;
  CPI_REQUIRE((N % 256 == 0 || n_groups == 0) && K % 8 == 0 && ldx % 8 == 0, "gemm_tc_pair: K (%d) and the row stride must be multiples of 8, N (%d) in groups of 256", K, N);
  CPI_REQUIRE(bn >= 32 && bn <= 256 && bn % 32 == 0, "gemm_tc_pair: token tile %d (multiples of 32 up to 256)", bn);
  CPI_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0, "gemm_tc_pair: operands must be 16-byte aligned");
  CPI_REQUIRE(mode != tc2::kAdd || out_dtype == kF32, "gemm_tc_pair: ADD mode needs a float32 output");
  CPI_REQUIRE(mode != tc2::kSwiglu || out_dtype == kBF16, "gemm_tc_pair: SWIGLU mode writes bfloat16");
  const int acc = mode == tc2::kSwiglu ? 2 : 1;
  CUtensorMap mw, mx;
  CPI_REQUIRE(n_groups <= 256, "gemm_tc_pair: %d groups (at most 256)", n_groups);
  if (tc::get_map_3d_bf16(w, (uint64_t)K, (uint64_t)acc * N, (uint64_t)(n_groups > 0 ? n_groups : 1), tc2::BK, tc2::BM, &mw)) return 1;
  if (tc::get_map_2d_bf16(x, (uint64_t)K, (uint64_t)T, (uint64_t)ldx * 2, tc2::BK, 64, &mx)) return 1;
  tc2::Params p{out, ldo, out_rows, row_scale, group_offsets, n_groups, T, bn, N, (K + tc2::BK - 1) / tc2::BK, error_flag, gate_act, gate_limit};
  const int n_pairs = (N + 255) / 256;
  dim3 grid(2 * n_pairs, (T + bn - 1) / bn + (n_groups > 0 ? (T < n_groups ? T : n_groups) : 0), 1);
  CPI_REQUIRE(grid.y <= 65535, "gemm_tc_pair: too many token tiles (%u)", grid.y);
  const int cap = bn <= 128 ? 128 : 256;
  // (ADD, list / two at a time: 4,096 x 2,048 -> 5,120 76 / 86, 8,192 x 1,024 -> 5,120 88 / 111; 4,096 x 5,120 -> 7,168 253 / 242)
  // (the list kernel stores whole 16-byte groups of a row only: rows that do not start on 16 bytes take another one)
  const bool rows16 = (reinterpret_cast<uintptr_t>(out) & 15) == 0 && ldo % (out_dtype == kF32 ? 4 : 8) == 0;
  const bool persistent = g_persistent == 2 || (g_persistent == 1 && (mode == tc2::kSwiglu ||
                                                (mode == tc2::kAdd && T >= 4096 && K <= 3072)));
  const int n_slots = (T + bn - 1) / bn + (n_groups > 0 ? (T < n_groups ? T : n_groups) : 0);
  // (groups: one accumulator with at least 192 rows a group; 16 experts of 2,048 x 2,048, list / slots in us: 512 rows 82 / 101, 256
  // 54 / 61, 128 41 / 45; 32 of 1,024 x 768: 512 rows 57 / 68, 256 39 / 41, 128 30 / 27)
  const bool persistent_groups = (g_persistent == 2 || (g_persistent == 1 && (mode == tc2::kSwiglu || T >= 192 * n_groups))) &&
                                 n_groups > 0 && n_slots <= tc2::kMaxSlots;
  if ((n_groups == 0 ? persistent : persistent_groups) && cap == 256 && rows16) {
    const int n_tok = n_slots;
    if (mode == tc2::kStore && out_dtype == kBF16) return tc2::launch_persistent<256, tc2::kStore, __nv_bfloat16>(mw, mx, p, n_pairs, n_tok, stream);
    if (mode == tc2::kStore && out_dtype == kF32) return tc2::launch_persistent<256, tc2::kStore, float>(mw, mx, p, n_pairs, n_tok, stream);
    if (mode == tc2::kAdd) return tc2::launch_persistent<256, tc2::kAdd, float>(mw, mx, p, n_pairs, n_tok, stream);
    if (mode == tc2::kSwiglu) return tc2::launch_persistent<256, tc2::kSwiglu, __nv_bfloat16>(mw, mx, p, n_pairs, n_tok, stream);
  }
  if (n_groups == 0 && cap == 256 && mode != tc2::kSwiglu) {
    if (mode == tc2::kAdd) return tc2::launch_dual<tc2::kAdd, float>(mw, mx, p, n_pairs, n_slots, stream);
    if (out_dtype == kBF16) return tc2::launch_dual<tc2::kStore, __nv_bfloat16>(mw, mx, p, n_pairs, n_slots, stream);
    return tc2::launch_dual<tc2::kStore, float>(mw, mx, p, n_pairs, n_slots, stream);
  }
#define CPI_PAIR(CAP)                                                                                         \
  if (mode == tc2::kStore && out_dtype == kBF16) return tc2::launch<CAP, tc2::kStore, __nv_bfloat16>(mw, mx, p, grid, stream); \
  if (mode == tc2::kStore && out_dtype == kF32) return tc2::launch<CAP, tc2::kStore, float>(mw, mx, p, grid, stream);         \
  if (mode == tc2::kAdd) return tc2::launch<CAP, tc2::kAdd, float>(mw, mx, p, grid, stream);                                  \
  if (mode == tc2::kSwiglu) return tc2::launch<CAP, tc2::kSwiglu, __nv_bfloat16>(mw, mx, p, grid, stream);
  if (cap == 128) { CPI_PAIR(128) } else { CPI_PAIR(256) }
#undef CPI_PAIR
  set_error("gemm_tc_pair: unsupported mode %d with output dtype %d", mode, out_dtype);
  return 1;
}
