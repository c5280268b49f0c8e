// Attention over a cached latent for prompts, with the heads' keys and values formed once per step.
//
// `latent_attention.cu` takes the queries through W_uk and attends over the cached rows [c | r] themselves: 2 (rank + rot)
// + 2 rank operations per query, head and key (2,176 at rank 512 and a rotated part of 64).  When many queries meet the
// same keys it is cheaper to form every head's key W_uk c and value W_uv c once, as one matrix product over the cached
// rows, and to attend with heads of 128 + 64 elements: 2 (128 + 64) + 2 128 = 640 operations.  The steps here:
//
//   latent_key_rows    the cached rows that a step's queries can see, sequence after sequence, out of their pages into one
//                      dense matrix [R, rank + rot] (the products' operand, and the rotated parts that all heads share)
//   latent_q_rows      the query heads [plain | rotated] in bfloat16, rotated by position
//   latent_prefill     the attention: tcgen05, two tiles of 128 queries of one head per CTA
//
// The attention kernel is laid out as `attention_prefill.cu` is (see there for the issue order, the softmax and the
// rescaling).  What differs is what shared memory holds: a query tile is three 64-column blocks of 16 KB (two plain, one
// rotated), 96 KB for the two tiles; what is left takes a ring of FIVE key blocks (a key tile of 128 positions is three of
// them) and a ring of THREE value blocks (64 positions x 128 columns; a value tile is two).  Blocks are freed and filled
// one by one, so that the next key tile's first two blocks and the next value tile's first one arrive under the products
// of this one.  Keys and values come from the matrix product's dense rows, the rotated block from the gathered rows.
//
// Bound: the products of a query tile (12 + 8 MMAs of 128 x 128 x 16 per key tile) and, at a few thousand tokens, the last
// wave: 16 heads x 8 tiles of 256 queries are 128 CTAs whose longest meets 16 key tiles and whose mean meets 9.  A mixer of
// 16 heads and rank 512, device time: a prompt of 2,048 tokens 723 -> 180 us, 4,096 tokens 2,188 -> 309 us (with 32 heads
// 3,996 -> 517 us), of which attention over the cached rows had 575 us and this kernel has about 60.
#include "prefill_tc.cuh"

namespace cpi {
namespace latent_pre {

using namespace pre;

constexpr int PAGE = 64;
constexpr int DK = 128, DR = 64, DV = 128;              // plain key, rotated key, value elements of a head
constexpr int QB = (DK + DR) / 64;                      // 64-column blocks of a query or key row
constexpr uint32_t BLOCK = 128 * 128;                   // bytes of a block
constexpr int NK = 5, NV = 3;                           // blocks of the key ring, of the value ring
constexpr int SMEM = (2 * QB + NK + NV) * BLOCK;
constexpr uint32_t TMEM_COLS = 512;                     // S of tile A, S of tile B, O of A, O of B

// First position whose row a step's queries on a sequence need: whole pages, from the one that holds the oldest position
// that the window lets its first query see.
__device__ __forceinline__ int first_row_pos(int start, int window) {
  return window > 0 ? max(0, start - window + 1) / PAGE * PAGE : 0;
}
// Rows of the sequences before `s` in the dense matrix (all lanes of a warp call it; every lane gets the sum).
__device__ __forceinline__ int rows_before(const int* seq_start, const int* seq_new, int s, int window) {
  const int lane = threadIdx.x & 31;
  int n = 0;
  for (int i = lane; i < s; i += 32) n += seq_start[i] + seq_new[i] - first_row_pos(seq_start[i], window);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}

struct Params {
  __nv_bfloat16* out;                                   // [T, out_heads * DV]; this launch's heads start at head0
  const int* token_pos; const int* token_seq;
  const int* seq_start; const int* seq_new;
  const int* tile_tok0; const int* tile_rows;           // per query tile: first packed token, valid rows
  int out_heads, head0, window;                         // window 0: none
  float scale_log2;
  const float* sink;                                    // [out_heads] or null
  int* error_flag;
};

__global__ void __launch_bounds__(kThreads) latent_prefill_kernel(const __grid_constant__ CUtensorMap map_q,
                                                             const __grid_constant__ CUtensorMap map_k,
                                                             const __grid_constant__ CUtensorMap map_r,
                                                             const __grid_constant__ CUtensorMap map_v, Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t q_full, k_full[NK], k_empty[NK], v_full[NV], v_empty[NV], s_full[2], p_full[2], o_done[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* q_s = smem_raw;                              // [2 query tiles][QB blocks]
  uint8_t* k_s = q_s + 2 * QB * BLOCK;                  // [NK]
  uint8_t* v_s = k_s + NK * BLOCK;                      // [NV]

  if (tid == 0) {
    mbar_init(&q_full, 1);
    for (int s = 0; s < NK; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < NV; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 4); mbar_init(&o_done[s], 1); }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  pdl_launch_dependents();                              // (not before the tensor memory is ours: see common.cuh)
  pdl_wait();
  const int tile = blockIdx.y, head = blockIdx.x;       // heads are the fast axis: all heads of the longest tile start first
  const int tok0 = p.tile_tok0[tile], rows = p.tile_rows[tile];
  const int seq = p.token_seq[tok0];
  // the tile's rows are consecutive positions of one sequence; rows 0-127 are query tile A, the rest tile B
  const int pos_first = p.token_pos[tok0], pos_last = pos_first + rows - 1;
  const int rows_x[2] = {min(rows, BQ), max(rows - BQ, 0)};
  const bool has_b = rows_x[1] > 0;
  const int p0_x[2] = {pos_first, pos_first + BQ};
  const int p1_x[2] = {pos_first + rows_x[0] - 1, pos_last};
  auto low = [&](int pos) { return p.window > 0 ? max(0, pos - p.window + 1) : 0; };
  // Key tiles are counted in dense rows from the page that holds the oldest position tile A sees, so a tile starts on a
  // page that the sequence's rows hold.  B's first tile is A's or a later one, its last is the union's last.
  const int key_first = low(p0_x[0]) / PAGE * PAGE;
  const int kb_x[2] = {0, has_b ? (low(p0_x[1]) - key_first) / BKV : 0};
  const int ke_x[2] = {(p1_x[0] - key_first) / BKV + 1, has_b ? (p1_x[1] - key_first) / BKV + 1 : 0};
  const int kt1 = has_b ? ke_x[1] : ke_x[0];
  const uint32_t tmem_s = tmem_base_s, tmem_o = tmem_base_s + 256;        // + 128 for tile B, both
  volatile int* abort_flag = &abort_s;
  bool ok = true;

  if (warp == 8) {
    // ---- TMA producer: Q of both tiles, then per key tile its three key blocks and its two value blocks ----
    const int row_first = rows_before(p.seq_start, p.seq_new, seq, p.window) +
                          key_first - first_row_pos(p.seq_start[seq], p.window);      // dense row of position key_first
    if (lane == 0) {
      mbar_expect_tx(&q_full, QB * BLOCK * (has_b ? 2 : 1));
      for (int x = 0; x < (has_b ? 2 : 1); ++x)
        for (int b = 0; b < QB; ++b)
          tma_load_2d(q_s + (x * QB + b) * BLOCK, &map_q, &q_full, head * (DK + DR) + b * 64, tok0 + x * BQ);
      int ks = 0, kph = 1, vs = 0, vph = 1;              // (a slot's first fill waits for nobody: parity of the phase before)
      for (int kt = 0; kt < kt1 && ok; ++kt) {
        const int row = row_first + kt * BKV;
        for (int b = 0; b < QB && ok; ++b) {
          ok = mbar_wait(&k_empty[ks], kph, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&k_full[ks], BLOCK);
          if (b < DK / 64) tma_load_2d(k_s + ks * BLOCK, &map_k, &k_full[ks], head * (DK + DV) + b * 64, row);
          else tma_load_2d(k_s + ks * BLOCK, &map_r, &k_full[ks], 0, row);
          if (++ks == NK) { ks = 0; kph ^= 1; }
        }
        for (int h = 0; h < 2 && ok; ++h) {
          ok = mbar_wait(&v_empty[vs], vph, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&v_full[vs], BLOCK);
          for (int c = 0; c < DV / 64; ++c)
            tma_load_2d(v_s + vs * BLOCK + c * (BLOCK / 2), &map_v, &v_full[vs], head * (DK + DV) + DK + c * 64, row + 64 * h);
          if (++vs == NV) { vs = 0; vph ^= 1; }
        }
      }
    }
  } else if (warp == 9) {
    // ---- MMA issuer: per key tile  O_A += P_A V;  S_A = Q_A K'^T;  O_B += P_B V;  S_B = Q_B K'^T  (K' the next tile) ----
    constexpr uint32_t idesc_s = instr_desc(BQ, BKV, 0);
    constexpr uint32_t idesc_o = instr_desc(BQ, DV, 1);
    constexpr uint64_t kBlockUnits = BLOCK >> 4;         // a block further, in the descriptor's 16-byte units
    const uint64_t dq[2] = {smem_desc(smem_u32(q_s), 16, 1024), smem_desc(smem_u32(q_s + QB * BLOCK), 16, 1024)};
    const uint64_t dk0 = smem_desc(smem_u32(k_s), 16, 1024), dv0 = smem_desc(smem_u32(v_s), BLOCK / 2, 1024);
    int ks[2], kph[2], vs[2], vph[2], pph[2] = {0, 0}, first_pv[2] = {1, 1};
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int nk = QB * kb_x[x], nv = 2 * kb_x[x];
      ks[x] = nk % NK; kph[x] = (nk / NK) & 1;
      vs[x] = nv % NV; vph[x] = (nv / NV) & 1;
    }
    // S_x = Q_x K^T, block by block as the blocks arrive; `release`: no later product reads this key tile
    auto issue_qk = [&](int x, bool release) -> bool {
#pragma unroll
      for (int b = 0; b < QB; ++b) {
        if (!__all_sync(0xffffffffu, mbar_wait(&k_full[ks[x]], kph[x], abort_flag))) return false;
        fence_after_sync();
        if (elect_one()) {
          const uint64_t dk = dk0 + (uint64_t)ks[x] * kBlockUnits, da = dq[x] + (uint64_t)b * kBlockUnits;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (b == 0 && k == 0) umma_bf16_c<false>(tmem_s + x * 128, da, dk, idesc_s);
            else umma_bf16_c<true>(tmem_s + x * 128, da + (uint64_t)(k * 2), dk + (uint64_t)(k * 2), idesc_s);
          }
          if (b == QB - 1) umma_commit(&s_full[x]);
          if (release) umma_commit(&k_empty[ks[x]]);
        }
        __syncwarp();
        if (++ks[x] == NK) { ks[x] = 0; kph[x] ^= 1; }
      }
      return true;
    };
    // O_x += P_x V, the tile's two value blocks of 64 positions one after the other
    auto issue_pv = [&](int x, bool release) -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait(&p_full[x], pph[x], abort_flag))) return false;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!__all_sync(0xffffffffu, mbar_wait(&v_full[vs[x]], vph[x], abort_flag))) return false;
        fence_after_sync();
        if (elect_one()) {
          const uint64_t dv = dv0 + (uint64_t)vs[x] * kBlockUnits;
          const uint32_t pa = tmem_s + x * 128 + h * 32, od = tmem_o + x * 128;
          if (h == 0 && first_pv[x]) umma_bf16_a_tmem_c<false>(od, pa, dv, idesc_o);
          else umma_bf16_a_tmem_c<true>(od, pa, dv, idesc_o);
#pragma unroll
          for (int j = 1; j < 4; ++j) umma_bf16_a_tmem_c<true>(od, pa + j * 8, dv + (uint64_t)(j * (2048 >> 4)), idesc_o);
          if (release) umma_commit(&v_empty[vs[x]]);
        }
        __syncwarp();
        if (++vs[x] == NV) { vs[x] = 0; vph[x] ^= 1; }
      }
      first_pv[x] = 0;
      pph[x] ^= 1;
      return true;
    };
    ok = __all_sync(0xffffffffu, mbar_wait(&q_full, 0, abort_flag));
    const int kb_b = has_b ? kb_x[1] : 0x7fffffff, ke_a = ke_x[0];
    ok = ok && issue_qk(0, kb_b != 0);
    if (ok && kb_b == 0) ok = issue_qk(1, true);
    for (int kt = 0; kt < kt1 && ok; ++kt) {
      // which query tiles meet key tile kt, and kt + 1 (B's range ends with the union's, A's begins with it)
      const bool a_now = kt < ke_a, b_now = kt >= kb_b;
      const bool a_next = kt + 1 < ke_a, b_next = kt + 1 >= kb_b && kt + 1 < kt1;
      if (a_now) {
        ok = issue_pv(0, !b_now);
        if (ok && a_next) ok = issue_qk(0, !b_next);
      }
      if (ok && b_now) ok = issue_pv(1, true);
      if (ok && b_next) ok = issue_qk(1, true);
    }
    if (ok && elect_one()) { umma_commit(&o_done[0]); umma_commit(&o_done[1]); }
    __syncwarp();
  } else {
    // ---- softmax: warps 0-3 own query tile A, warps 4-7 tile B; thread r of a group owns query row r ----
    const int x = warp >> 2, row = tid & 127;
    const bool live = row < rows_x[x];
    const int qp = live ? p0_x[x] + row : -1;
    const int lo = live ? low(qp) : 0, lo_last = low(p1_x[x]);
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_row = tmem_s + x * 128 + lane_addr, o_row = tmem_o + x * 128 + lane_addr;
    float m_ref = -1e30f, l_run = 0.f;                  // reference maximum of the exponentials; the row's sum
    const float sc = p.scale_log2;
    // Rows beyond the newest position (another sequence's, or what a shorter matrix left) are zeroed in the last value
    // tile by the group whose product reads it first: 0 * NaN would reach the output.
    const bool zero_duty = x == 0 ? kt1 - 1 < ke_x[0] : !(kt1 - 1 < ke_x[0]);
    int j = 0;
    bool okl = rows_x[x] > 0;
    for (int kt = kb_x[x]; kt < ke_x[x] && okl; ++kt, ++j) {
      const int key0 = key_first + kt * BKV;
      okl = __all_sync(0xffffffffu, mbar_wait(&s_full[x], j & 1, abort_flag));
      if (okl && kt == kt1 - 1 && zero_duty) {
        const int n = 2 * kt + (row >> 6), sl = n % NV;  // (a warp's rows lie in one of the two blocks)
        okl = __all_sync(0xffffffffu, mbar_wait(&v_full[sl], (n / NV) & 1, abort_flag));
        if (okl && key0 + row > pos_last) {
#pragma unroll
          for (int c = 0; c < DV / 64; ++c) {
            uint4* r4 = reinterpret_cast<uint4*>(v_s + sl * BLOCK + c * (BLOCK / 2) + (row & 63) * 128);
#pragma unroll
            for (int q = 0; q < 8; ++q) r4[q] = make_uint4(0, 0, 0, 0);
          }
        }
        fence_async_proxy();                             // the MMA reads V through the async proxy
      }
      if (!okl) break;
      fence_after_sync();
      const bool no_mask = key0 + BKV - 1 <= p0_x[x] && key0 >= lo_last;
      uint32_t w[BKV / 32][16];
      float mx, ls;
      // (the first tile's maximum alone, then optimistic passes: see there)
      if (j == 0) {
        mx = -INFINITY;
#pragma unroll 1
        for (int c = 0; c < BKV; c += 32) {
          float v[32], mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
          tmem_ld32(s_row + c, v);
          const uint32_t in = visible(qp, lo, 0, key0 + c);
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            mx4[e & 3] = fmaxf(mx4[e & 3], (in >> e) & 1u ? v[e] : -INFINITY);
          }
          mx = fmaxf(mx, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
        }
        m_ref = fmaxf(mx * sc, m_ref);
      }
      auto pass = [&](const float ref) {
        const float nref = -ref;
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, ls4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t raw[2][32];
        tmem_ld32_issue(s_row, raw[0]);
        tmem_ld32_issue(s_row + 32, raw[1]);
        tmem_wait_ld();
#pragma unroll
        for (int cc = 0; cc < BKV / 32; ++cc) {
          float v[32];
          if (no_mask) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              float sv = __uint_as_float(raw[cc & 1][e]);
              mx4[e & 3] = fmaxf(mx4[e & 3], sv);
              v[e] = exp2_fast(fmaf(sv, sc, nref));
            }
          } else {
            const uint32_t in = visible(qp, lo, 0, key0 + cc * 32);
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              float sv = __uint_as_float(raw[cc & 1][e]);
              mx4[e & 3] = fmaxf(mx4[e & 3], (in >> e) & 1u ? sv : -INFINITY);
              v[e] = (in >> e) & 1u ? exp2_fast(fmaf(sv, sc, nref)) : 0.f;
            }
          }
          if (cc + 2 < BKV / 32) tmem_ld32_issue(s_row + (cc + 2) * 32, raw[cc & 1]);     // this buffer is consumed
#pragma unroll
          for (int e = 0; e < 32; ++e) ls4[e & 3] += v[e];
#pragma unroll
          for (int g = 0; g < 16; ++g) w[cc][g] = pack_bf16(v[2 * g], v[2 * g + 1]);
          if (cc == 1) tmem_wait_ld();
        }
        mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sc;
        ls = (ls4[0] + ls4[1]) + (ls4[2] + ls4[3]);
      };
      pass(m_ref);
      const bool grow = mx > m_ref + (m_ref < -1e29f ? 0.f : kRescaleSlack);
      if (__any_sync(0xffffffffu, grow)) {
        const float m_new = grow ? mx : m_ref;
        const float f = exp2f(m_ref - m_new);
        // Every P V issued so far for this query tile has landed: the Q K^T whose S was waited for above was
        // issued after the last of them, and its arrival covers everything issued before it.
#pragma unroll 1
        for (int c = 0; c < DV; c += 32) {
          float v[32];
          tmem_ld32(o_row + c, v);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] *= f;
          tmem_st32(o_row + c, v);
        }
        l_run *= f;
        m_ref = m_new;
        pass(m_ref);
      }
#pragma unroll
      for (int cc = 0; cc < BKV / 32; ++cc) tmem_st16_nowait(s_row + cc * 16, w[cc]);
      l_run += ls;
      tmem_wait_st();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[x]);            // one arrival per warp
    }
    ok = okl && !abort_s && j > 0;
    ok = __all_sync(0xffffffffu, ok && mbar_wait(&o_done[x], 0, abort_flag));
    fence_after_sync();
    if (ok) {
      const int oh = p.head0 + head;
      if (p.sink) l_run += exp2f(fminf(p.sink[oh] * 1.4426950408889634f - m_ref, 120.f));
      const float inv = 1.0f / fmaxf(l_run, 1e-20f);
      __nv_bfloat16* dst = p.out + ((size_t)(tok0 + x * BQ + row) * p.out_heads + oh) * DV;
#pragma unroll 1
      for (int c = 0; c < DV; c += 32) {
        float v[32];
        tmem_ld32(o_row + c, v);
        if (live) {
#pragma unroll
          for (int e = 0; e < 32; e += 8)
            *reinterpret_cast<uint4*>(dst + c + e) =
                make_uint4(pack_bf16(v[e] * inv, v[e + 1] * inv), pack_bf16(v[e + 2] * inv, v[e + 3] * inv),
                           pack_bf16(v[e + 4] * inv, v[e + 5] * inv), pack_bf16(v[e + 6] * inv, v[e + 7] * inv));
        }
      }
    }
    fence_before_sync();
  }
  if (abort_s) {
    if (tid == 0 && p.error_flag) atomicExch(p.error_flag, 2);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_s), "r"(TMEM_COLS));
}

// ---- the cached rows of a step's sequences into one dense matrix ---------------------------------------------------
struct RowsParams {
  const uint4* cache; uint4* out; int row16;            // 16-byte pieces of a row
  const int* page_table; int max_blocks;
  const int* seq_slot; const int* seq_start; const int* seq_new;
  int window;
};
constexpr int ROWS_PER_BLOCK = 16;

// A block copies 16 rows of one sequence (blockIdx.y); a page holds 64, so they lie in one page.
__global__ void __launch_bounds__(256) latent_key_rows_kernel(RowsParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = blockIdx.y, first = first_row_pos(p.seq_start[s], p.window), end = p.seq_start[s] + p.seq_new[s];
  const int pos0 = first + blockIdx.x * ROWS_PER_BLOCK, n = min(ROWS_PER_BLOCK, end - pos0);
  if (n <= 0) return;
  const int base = rows_before(p.seq_start, p.seq_new, s, p.window);
  const int page = p.page_table[(size_t)p.seq_slot[s] * p.max_blocks + pos0 / PAGE];
  const uint4* src = p.cache + ((size_t)page * PAGE + pos0 % PAGE) * p.row16;
  uint4* dst = p.out + (size_t)(base + pos0 - first) * p.row16;
  for (int i = threadIdx.x; i < n * p.row16; i += blockDim.x) dst[i] = src[i];
}

// ---- query heads in bfloat16, their last `rot` elements rotated ----------------------------------------------------
struct QRowsParams {
  const float* q; long q_stride;                        // [T, H (D + R)]
  __nv_bfloat16* out;                                   // [T, H (D + R)]
  const float* inv_freq; int interleaved; float amplitude;       // [R / 2] or null
  const int* token_pos;
  int n_heads, dim, rot;
};

// A block per token; a thread takes four neighbouring elements of a row (a head's parts are multiples of four).  The
// sines and cosines of the position are taken once per pair, not once per pair and head.
__global__ void __launch_bounds__(256) latent_q_rows_kernel(QRowsParams p) {
  pdl_launch_dependents();
  extern __shared__ float2 turn[];                      // [R / 2] (cosine, sine)
  const int t = blockIdx.x, half = p.rot >> 1, W = p.dim + p.rot;
  pdl_wait();
  const int pos = p.token_pos[t];
  for (int f = threadIdx.x; f < half; f += blockDim.x) {
    float sn = 0.f, cs = 1.f;
    if (p.inv_freq) {
      sincosf((float)pos * p.inv_freq[f], &sn, &cs);
      sn *= p.amplitude; cs *= p.amplitude;
    }
    turn[f] = make_float2(cs, sn);
  }
  __syncthreads();
  const float* q = p.q + (size_t)t * p.q_stride;
  __nv_bfloat16* out = p.out + (size_t)t * p.n_heads * W;
  for (int i = 4 * threadIdx.x; i < p.n_heads * W; i += 4 * blockDim.x) {
    const int d = i % W;
    const float4 v = *reinterpret_cast<const float4*>(q + i);
    float y[4] = {v.x, v.y, v.z, v.w};
    if (d >= p.dim && p.inv_freq) {
      const int r = d - p.dim;
      if (p.interleaved) {
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const float2 cs = turn[(r + e) >> 1];
          const float a = y[e], b = y[e + 1];
          y[e] = a * cs.x - b * cs.y;
          y[e + 1] = b * cs.x + a * cs.y;
        }
      } else {
        const bool first = r < half;
        const float4 u = *reinterpret_cast<const float4*>(q + i + (first ? half : -half));
        const float o[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 cs = turn[(first ? r : r - half) + e];
          y[e] = first ? y[e] * cs.x - o[e] * cs.y : y[e] * cs.x + o[e] * cs.y;
        }
      }
    }
    *reinterpret_cast<uint2*>(out + i) = make_uint2(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]));
  }
}

}  // namespace latent_pre
}  // namespace cpi

using namespace cpi;

extern "C" int cpi_latent_prefill_supported(int dim, int rot, int value_dim, int kv_rank, int page_size) {
  return dim == latent_pre::DK && rot == latent_pre::DR && value_dim == latent_pre::DV && kv_rank % 8 == 0 && kv_rank > 0 &&
         page_size == latent_pre::PAGE;
}

// cache [pages, 1, 64, row] bfloat16 -> out [R, row]: per sequence the positions from the first its window needs to its newest.
extern "C" int cpi_latent_key_rows(const void* cache, void* out, int row, const int* page_table, int max_blocks,
                                   const int* seq_slot, const int* seq_start, const int* seq_new, int n_seqs, int most_rows,
                                   int window, cudaStream_t stream) {
  if (n_seqs == 0 || most_rows <= 0) return 0;
  CPI_REQUIRE(row % 8 == 0 && ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15) == 0,
              "latent_key_rows: rows of %d elements must be whole 16-byte pieces", row);
  CPI_REQUIRE(n_seqs <= 65535, "latent_key_rows: %d sequences", n_seqs);
  latent_pre::RowsParams p{reinterpret_cast<const uint4*>(cache), reinterpret_cast<uint4*>(out), row / 8, page_table, max_blocks,
                           seq_slot, seq_start, seq_new, window};
  const dim3 grid((most_rows + latent_pre::ROWS_PER_BLOCK - 1) / latent_pre::ROWS_PER_BLOCK, n_seqs);
  cpi::launch_pdl(latent_pre::latent_key_rows_kernel, grid, dim3(256), 0, stream, p);
  return check_launch("latent_key_rows");
}

extern "C" int cpi_latent_q_rows(const float* q, long q_stride, const float* inv_freq, int interleaved, float amplitude, void* out,
                                 const int* token_pos, int n_tokens, int n_heads, int dim, int rot, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  CPI_REQUIRE(dim % 4 == 0 && rot % 8 == 0 && q_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0 &&
              (reinterpret_cast<uintptr_t>(out) & 7) == 0, "latent_q_rows: heads of %d + %d elements", dim, rot);
  latent_pre::QRowsParams p{q, q_stride, reinterpret_cast<__nv_bfloat16*>(out), inv_freq, interleaved, amplitude, token_pos,
                            n_heads, dim, rot};
  cpi::launch_pdl(latent_pre::latent_q_rows_kernel, dim3(n_tokens), dim3(256), (size_t)(rot / 2) * sizeof(float2), stream, p);
  return check_launch("latent_q_rows");
}

// The heads head0 .. head0 + n_heads - 1 of q [T, out_heads (128 + 64)] against kv [n_rows, n_heads (128 + 128)] (a head's key
// then its value) and the rotated parts rows[:, rank : rank + 64] of rows [n_rows, rank + 64]; out [T, out_heads 128].
extern "C" int cpi_latent_prefill(const void* q, const void* kv, const void* rows, int rank, void* out, long n_rows,
                                  const int* token_seq, const int* token_pos, const int* seq_start, const int* seq_new,
                                  const int* tile_tok0, const int* tile_rows, int n_tiles, int n_tokens, int n_heads, int out_heads,
                                  int head0, int window, float scale, const float* sink, int* error_flag, cudaStream_t stream) {
  using namespace latent_pre;
  if (n_tiles == 0 || n_heads == 0) return 0;
  CPI_REQUIRE(n_tiles <= 65535, "latent_prefill: too many query tiles in one launch (%d)", n_tiles);
  CPI_REQUIRE(rank % 8 == 0 && head0 >= 0 && head0 + n_heads <= out_heads && n_rows > 0, "latent_prefill: heads %d .. of %d, rank %d",
              head0, out_heads, rank);
  CUtensorMap mq, mk, mr, mv;
  const uint64_t qw = (uint64_t)out_heads * (DK + DR), kw = (uint64_t)n_heads * (DK + DV);
  const __nv_bfloat16* q0 = reinterpret_cast<const __nv_bfloat16*>(q) + (size_t)head0 * (DK + DR);
  if (tc::get_map_2d_bf16(q0, (uint64_t)n_heads * (DK + DR), (uint64_t)n_tokens, qw * 2, 64, BQ, &mq)) return 1;
  if (tc::get_map_2d_bf16(kv, kw, (uint64_t)n_rows, kw * 2, 64, BKV, &mk)) return 1;
  if (tc::get_map_2d_bf16(kv, kw, (uint64_t)n_rows, kw * 2, 64, 64, &mv)) return 1;
  const __nv_bfloat16* r0 = reinterpret_cast<const __nv_bfloat16*>(rows) + rank;
  if (tc::get_map_2d_bf16(r0, DR, (uint64_t)n_rows, (uint64_t)(rank + DR) * 2, 64, BKV, &mr)) return 1;
  Params p{reinterpret_cast<__nv_bfloat16*>(out), token_pos, token_seq, seq_start, seq_new, tile_tok0, tile_rows, out_heads, head0,
           window, scale * 1.4426950408889634f, sink, error_flag};
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(latent_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
      cpi::set_error("latent_prefill: %d bytes of shared memory were refused", SMEM);
      return 1;
    }
    set = true;
  }
  cpi::launch_pdl(latent_prefill_kernel, dim3(n_heads, n_tiles), dim3(kThreads), SMEM, stream, mq, mk, mr, mv, p);
  return check_launch("latent_prefill");
}
