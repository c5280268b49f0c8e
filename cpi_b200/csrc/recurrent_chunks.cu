// The recurrences of `linear_scan` (recurrent.cu) over a prompt, in chunks of 64 tokens that are worked on side by side.
//
// A token-by-token scan of 2,048 tokens is a chain of 2,048 dependent steps in which one block per SM waits for its own
// shuffles.  Over a chunk that starts from the state S, with a_t the decays (per row n of the state), the same outputs are
//
//     o_i = sum_n q~_i[n] S[n] + sum_{j <= i} A_ij v_j          q~_i = q_i * prod_{t <= i} a_t
//     S' = D S + sum_j k~_j v_j^T                               k~_j = k_j * prod_{t > j} a_t,  D = prod_t a_t
//     A_ij = sum_n q_i[n] k_j[n] prod_{j < t <= i} a_t[n]
//
// so what depends on the chunk alone (A, q~, k~, D and U = k~^T v) is formed for all chunks at once, the states between
// the chunks by one pass over them (S' = D S + U), and the outputs for all chunks at once again.  With the delta rule
// (u_i = beta_i (v_i - S_i^T k_i) is written instead of v_i) the chunk's u solve a unit lower-triangular system:
//
//     u = T (beta v) - T (beta K^) S,   (I + beta M) T = I,  M_ij = sum_n k_i[n] k_j[n] prod_{j < t <= i} a_t[n],  K^_i = k_i * prod_{t <= i} a_t
//
// whose right-hand sides are solved for all chunks at once; the pass over the chunks then is u = U^ - W S, S' = D S + k~^T u.
//
// Everything is float32 on the FP32 pipe, as in the scan.  Products of decays are always taken forward, one factor after
// another, never as a quotient or as the exponential of a sum of logarithms: they lose no digits however strong the decays
// are and underflow to the zero that the scan reaches too.  A token's output reads nothing of later tokens.
//
// Why not the tensor cores: the operands are float32 (three bfloat16 terms each), which takes six products for one; at the
// rate of mma.sync that is what the FP32 pipe does without any splitting.
//
// Measured (one prompt of 2,048 tokens, width 2,048): the recurrence of gated linear attention with 8 heads of 128 x 256
// 480 -> 114 us (prepare_rows 34, chunk_state 24, chain 14, chunk_out 40; the FP32 pipe's floor is 36), the delta rule at
// 1,500 tokens 435 -> 176 us (48, solve 21, delta_chain 76, 31), the state-space form with 64 heads of 128 x 64 at 1,855 tokens
// 507 -> 183 us (prepare_step 15, 53, 35, 80; floor 64).
//
//   prepare_rows   the decays per row (their transform too), and A, q~, k~, D (and M, K^) of a chunk and head
//   prepare_step   C_i . B_j and C transposed, of a chunk and group of heads: one decay per head and token
//   solve          W and U^ of the delta rule: 128 right-hand sides a block, 16 x 16 blocks of the triangle in registers
//   chunk_state    U = k~^T v, 128 x 64 (or 64 x 64) a block, 8 x 8 a thread
//   chain          the states between the chunks; `delta_chain` with the delta rule, 16 columns a block
//   chunk_out      the outputs, 64 tokens x 64 columns a block, 8 x 8 a thread, the triangle's dead part left out
//
// A long step runs in segments of chunks so that the scratch stays within what the caller gives.
#include "decay.cuh"
#include <type_traits>

namespace cpi {
namespace chunks {

constexpr int C = 64;

struct Params {
  const float* k; long k_stride; const float* q; long q_stride; const float* v; long v_stride;
  const float* z; long z_stride;                 // row decays before their transform [T, H N]
  const void* z_bias; float inv_tau; int decay_kind;             // the transform: see row_decay_f in decay.cuh
  const float* dt; long dt_stride;               // raw step sizes [T, H]
  const void* dt_bias; const void* a_log; const void* skip; int small_dtype;
  const float* beta; long beta_stride;           // [T, H] before the sigmoid (the delta rule)
  float q_scale;
  float* state;                                  // [slots, H, N, Dv]
  float* out; long out_stride;
  const int* seq_slot; const int* seq_tok0; const int* seq_new;
  int H, hpg, N, Dv, n_seqs;
  int seg0, seg_chunks;                          // this launch's chunks, counted over all sequences: seg0 .. seg0 + seg_chunks - 1
  // scratch, per chunk of the segment and head (AT and QT of the step flavour: and group)
  float *U, *KT, *QT, *AT, *DC, *MT, *KP, *WT, *UH;
};

struct Place { int tok, n; size_t item; };
// The chunk of block x, counted from the segment's first over the sequences one after another; n = 0: past the last one.
// (Every warp finds it by itself: 32 sequences at a time, their chunks summed up across the lanes.)
__device__ __forceinline__ Place place(const Params& p, int x, int h, int H) {
  const int lane = threadIdx.x & 31;
  Place c{0, 0, (size_t)x * H + h};
  int at = p.seg0 + x;                           // chunks still to skip
  for (int s0 = 0; s0 < p.n_seqs; s0 += 32) {
    const int s = s0 + lane, n = s < p.n_seqs ? p.seq_new[s] : 0, own = (n + C - 1) / C;
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    const unsigned here = __ballot_sync(0xffffffffu, at < upto);
    if (here) {
      const int l = __ffs(here) - 1, first = (at - __shfl_sync(0xffffffffu, upto - own, l)) * C;
      c.n = min(C, __shfl_sync(0xffffffffu, n, l) - first);
      c.tok = p.seq_tok0[s0 + l] + first;
      return c;
    }
    at -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return c;
}
// The chunks of sequence s in the segment: the first one's number there, and how many (all lanes of a warp call it).
__device__ __forceinline__ void chunks_of(const Params& p, int s, int& first, int& n) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int i = lane; i < s; i += 32) before += (p.seq_new[i] + C - 1) / C;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  const int lo = max(before, p.seg0), hi = min(before + (p.seq_new[s] + C - 1) / C, p.seg0 + p.seg_chunks);
  first = lo - p.seg0;
  n = hi - lo;
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float2 two(float x) { return make_float2(x, x); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }

// ---- row decays: A, q~, k~, D (and M, K^) --------------------------------------------------------------------------
// Thread (j, kk) of the scores carries k_j[n] prod a_t[n] for its eighth of the rows (n / 4 mod 8 = kk: eight lanes read
// 128 neighbouring bytes) forward over the tokens i; the warps
// with the late j, which are done first, then take q~ and k~ while the others go on.  What is waited for is the longest
// warp's chain (an instruction every 13 cycles), hence sixteen warps of four j; with eight of eight j 42 us instead of
// 34 for 2,048 tokens of 8 heads, 128 rows.
template <int NPT, bool DELTA>
struct PrepShape {
  static constexpr int N = 8 * NPT;
  static constexpr size_t bytes = ((DELTA ? 3 : 2) * C * N + C + N) * sizeof(float);
};

// Of four numbers per lane: their sums over eight neighbouring lanes, the (kk mod 4)-th of them for lane kk.
__device__ __forceinline__ float sum4(const float (&s)[4], int kk) {
  const bool hi = kk & 2, odd = kk & 1;
  float a = hi ? s[2] : s[0], b = hi ? s[3] : s[1], c = hi ? s[0] : s[2], d = hi ? s[1] : s[3];
  a += __shfl_xor_sync(0xffffffffu, c, 2);
  b += __shfl_xor_sync(0xffffffffu, d, 2);
  a = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
  return a + __shfl_xor_sync(0xffffffffu, a, 4);
}

template <int NPT, bool DELTA>
__global__ void __launch_bounds__(512) prepare_rows_kernel(Params p) {
  using Sh = PrepShape<NPT, DELTA>;
  constexpr int N = Sh::N, PIECES = C * N / 4 / 512;
  extern __shared__ __align__(16) float sm[];
  float *qs = sm, *as = qs + C * N, *ks = as + C * N, *bs = DELTA ? ks + C * N : ks, *zb = bs + C;
  const int h = blockIdx.y, g = h / p.hpg, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float rate = p.decay_kind == 1 ? expf(load_any(p.a_log, p.small_dtype, h)) : 0.f;
  if (tid < N) zb[tid] = p.z_bias ? load_any(p.z_bias, p.small_dtype, (size_t)h * N + tid) : 0.f;
  pdl_wait();
  const Place c = place(p, blockIdx.x, h, p.H);
  if (c.n <= 0) return;
  const float *q = p.q + (size_t)c.tok * p.q_stride + (size_t)g * N, *k = p.k + (size_t)c.tok * p.k_stride + (size_t)g * N,
              *a = p.z + (size_t)c.tok * p.z_stride + (size_t)h * N;
  // rows past the chunk's tokens: zeros, and decays of one
  float4 d[PIECES];
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int e = tid + i * 512, j = e / (N / 4), n = e % (N / 4) * 4, to = j * N + n;
    const bool live = j < c.n;
    if (live) d[i] = ld4(a + (size_t)j * p.z_stride + n);
    copy16(qs + to, live ? q + (size_t)j * p.q_stride + n : p.q, live);
    if (DELTA) copy16(ks + to, live ? k + (size_t)j * p.k_stride + n : p.k, live);
  }
  copy_commit();
  if (DELTA && tid < C) bs[tid] = tid < c.n ? 1.0f / (1.0f + expf(-p.beta[(size_t)(c.tok + tid) * p.beta_stride + h])) : 0.f;
  __syncthreads();                                             // the biases are in place
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int e = tid + i * 512, j = e / (N / 4), n = e % (N / 4) * 4, to = j * N + n;
    float4 y = make_float4(1.f, 1.f, 1.f, 1.f);
    if (j < c.n) {
      const float* b = zb + n;
      y = make_float4(row_decay_f(d[i].x, b[0], p.inv_tau, p.decay_kind, rate), row_decay_f(d[i].y, b[1], p.inv_tau, p.decay_kind, rate),
                      row_decay_f(d[i].z, b[2], p.inv_tau, p.decay_kind, rate), row_decay_f(d[i].w, b[3], p.inv_tau, p.decay_kind, rate));
    }
    *reinterpret_cast<float4*>(as + to) = y;
  }
  const int j = 4 * warp + (lane >> 3), kk = lane & 7;
  float w[NPT];
#pragma unroll
  for (int r = 0; r < NPT; r += 4) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < c.n) x = ld4(k + (size_t)j * p.k_stride + 8 * r + 4 * kk);
    w[r] = x.x; w[r + 1] = x.y; w[r + 2] = x.z; w[r + 3] = x.w;
  }
  copy_wait<0>();
  __syncthreads();
  {
    float *AT = p.AT + c.item * (size_t)(C * C) + (size_t)j * C, *MT = DELTA ? p.MT + c.item * (size_t)(C * C) + (size_t)j * C : nullptr;
    auto decay = [&](int i) {
      const float* ai = as + i * N + 4 * kk;
#pragma unroll
      for (int r = 0; r < NPT; r += 4) {
        const float4 y = ld4(ai + 8 * r);
        const float2 lo = __fmul2_rn(make_float2(w[r], w[r + 1]), make_float2(y.x, y.y));
        const float2 hi = __fmul2_rn(make_float2(w[r + 2], w[r + 3]), make_float2(y.z, y.w));
        w[r] = lo.x; w[r + 1] = lo.y; w[r + 2] = hi.x; w[r + 3] = hi.y;
      }
    };
    auto dot = [&](const float* rows, int i) -> float {        // this thread's eighth of row i . w
      const float* y = rows + i * N + 4 * kk;
      float2 s2[2] = {two(0.f), two(0.f)};
#pragma unroll
      for (int r = 0; r < NPT; r += 4) {
        const float4 x = ld4(y + 8 * r);
        s2[0] = __ffma2_rn(make_float2(x.x, x.y), make_float2(w[r], w[r + 1]), s2[0]);
        s2[1] = __ffma2_rn(make_float2(x.z, x.w), make_float2(w[r + 2], w[r + 3]), s2[1]);
      }
      return (s2[0].x + s2[0].y) + (s2[1].x + s2[1].y);
    };
    // Four tokens at a time, their sums over the eight lanes side by side, after which lane kk holds token kk's.  A j's own
    // tokens begin at i = j: before that the decays are left out (what is stored above the diagonal is not read).  The rows
    // past the chunk's tokens are zeros, which the delta rule's right-hand sides rely on.
    for (int i = 4 * warp; i < C; i += 4) {
      float s[4], m[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (i + e > j) decay(i + e);
        s[e] = dot(qs, i + e);
        if (DELTA) m[e] = dot(ks, i + e);
      }
      const float y = sum4(s, kk), z = DELTA ? sum4(m, kk) : 0.f;
      if (kk < 4) {
        AT[i + kk] = y * p.q_scale;
        if (DELTA) MT[i + kk] = z * bs[i + kk];
      }
    }
  }
  // forward over the tokens: q~, K^; backward: k~, D
  if (tid >= 256 && tid < 256 + N) {
    const int n = tid - 256;
    float P = 1.f;
    float *QT = p.QT + c.item * (size_t)(N * C) + (size_t)n * C, *KP = DELTA ? p.KP + c.item * (size_t)(N * C) + n : nullptr;
#pragma unroll 4
    for (int i = 0; i < C; i += 4) {
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        P *= as[(i + e) * N + n];
        y[e] = qs[(i + e) * N + n] * P * p.q_scale;
        if (DELTA) KP[(size_t)(i + e) * N] = ks[(i + e) * N + n] * P;
      }
      st4(QT + i, y[0], y[1], y[2], y[3]);
    }
  } else if (tid >= 512 - N) {
    const int n = tid - (512 - N);
    float R = 1.f;
    float* KT = p.KT + c.item * (size_t)(N * C) + n;
#pragma unroll 16
    for (int t = C - 1; t >= 0; --t) {
      const float x = DELTA ? ks[t * N + n] : t < c.n ? k[(size_t)t * p.k_stride + n] : 0.f;
      KT[(size_t)t * N] = x * R;
      R *= as[t * N + n];
    }
    p.DC[c.item * N + n] = R;
  }
}

// ---- one decay per head and token: C_i . B_j and C transposed, once per group of heads ---------------------------------
template <int N>
__global__ void __launch_bounds__(256) prepare_step_kernel(Params p) {
  constexpr int LD = N + 4;
  extern __shared__ __align__(16) float sm[];
  float *cs = sm, *bs = cs + C * LD;
  pdl_wait();
  const int g = blockIdx.y, G = p.H / p.hpg, tid = threadIdx.x;
  const Place c = place(p, blockIdx.x, g, G);
  if (c.n <= 0) return;
  for (int e = tid; e < C * N / 4; e += 256) {
    const int j = e / (N / 4), n = e % (N / 4) * 4;
    const bool live = j < c.n;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(cs + j * LD + n) = live ? ld4(p.q + (size_t)(c.tok + j) * p.q_stride + (size_t)g * N + n) : zero;
    *reinterpret_cast<float4*>(bs + j * LD + n) = live ? ld4(p.k + (size_t)(c.tok + j) * p.k_stride + (size_t)g * N + n) : zero;
  }
  __syncthreads();
  // thread: tokens i0, i0 + 16, .. of C against tokens j0, j0 + 16, .. of B
  const int i0 = tid & 15, j0 = tid >> 4;
  float acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = 0.f;
#pragma unroll 4
  for (int n = 0; n < N; n += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) { a[x] = ld4(cs + (i0 + 16 * x) * LD + n); b[x] = ld4(bs + (j0 + 16 * x) * LD + n); }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y)
        acc[x][y] = fmaf(a[x].w, b[y].w, fmaf(a[x].z, b[y].z, fmaf(a[x].y, b[y].y, fmaf(a[x].x, b[y].x, acc[x][y]))));
  }
  float* AT = p.AT + c.item * (size_t)(C * C);
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) AT[(j0 + 16 * y) * C + i0 + 16 * x] = acc[x][y] * p.q_scale;
  float* QT = p.QT + c.item * (size_t)(N * C);
  for (int e = tid; e < N * C / 4; e += 256) {
    const int n = e % N, i = e / N * 4;
    st4(QT + (size_t)n * C + i, cs[i * LD + n] * p.q_scale, cs[(i + 1) * LD + n] * p.q_scale, cs[(i + 2) * LD + n] * p.q_scale,
        cs[(i + 3) * LD + n] * p.q_scale);
  }
}

// The step sizes and decays of a chunk's tokens: one warp, lane l holds the tokens 2 l and 2 l + 1 (a = 1, dt = 0 past them).
__device__ __forceinline__ void step_of(const Params& p, const Place& c, int h, int lane, float (&dt)[2], float (&a)[2]) {
  const float rate = -expf(load_any(p.a_log, p.small_dtype, h)), bias = p.dt_bias ? load_any(p.dt_bias, p.small_dtype, h) : 0.f;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int j = 2 * lane + e;
    dt[e] = j < c.n ? softplus_f(p.dt[(size_t)(c.tok + j) * p.dt_stride + h] + bias) : 0.f;
    a[e] = j < c.n ? expf(rate * dt[e]) : 1.f;
  }
}

// ---- the delta rule's right-hand sides -----------------------------------------------------------------------------------
// Columns 0 .. N - 1: W = T (beta K^), stored transposed; N ..: U^ = T (beta V).  A thread owns a column.
__global__ void __launch_bounds__(128) solve_kernel(Params p) {
  __shared__ __align__(16) float mt[C * C];
  __shared__ float bs[C];
  extern __shared__ __align__(16) float us[];                 // [C][128]
  pdl_wait();
  const int h = blockIdx.y, tid = threadIdx.x, N = p.N, col = blockIdx.z * 128 + tid;
  const Place c = place(p, blockIdx.x, h, p.H);
  if (c.n <= 0) return;
  const float* MT = p.MT + c.item * (size_t)(C * C);
  for (int e = tid; e < C * C / 4; e += 128) copy16(mt + 4 * e, MT + 4 * e, true);
  copy_commit();
  if (tid < C) bs[tid] = tid < c.n ? 1.0f / (1.0f + expf(-p.beta[(size_t)(c.tok + tid) * p.beta_stride + h])) : 0.f;
  copy_wait<0>();
  __syncthreads();
  if (col >= N + p.Dv) return;
  const bool is_w = col < N;
  const float* src = is_w ? p.KP + c.item * (size_t)(N * C) + col : p.v + (size_t)c.tok * p.v_stride + (size_t)h * p.Dv + (col - N);
  const size_t step = is_w ? (size_t)N : (size_t)p.v_stride;
  float* WT = p.WT + c.item * (size_t)(N * C) + (size_t)col * C;
  float* UH = p.UH + c.item * (size_t)(C * p.Dv) + (col - N);
  for (int I = 0; I < C; I += 16) {
    float acc[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) acc[r] = I + r < c.n ? bs[I + r] * src[(size_t)(I + r) * step] : 0.f;
#pragma unroll 2
    for (int j = 0; j < I; ++j) {
      const float u = us[j * 128 + tid];
#pragma unroll
      for (int r = 0; r < 16; r += 4) {
        const float4 m = ld4(mt + j * C + I + r);
        acc[r] = fmaf(-m.x, u, acc[r]); acc[r + 1] = fmaf(-m.y, u, acc[r + 1]);
        acc[r + 2] = fmaf(-m.z, u, acc[r + 2]); acc[r + 3] = fmaf(-m.w, u, acc[r + 3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) {
#pragma unroll
      for (int x = r + 1; x < 16; ++x) acc[x] = fmaf(-mt[(I + r) * C + I + x], acc[r], acc[x]);
      us[(I + r) * 128 + tid] = acc[r];
    }
    if (is_w) {
#pragma unroll
      for (int r = 0; r < 16; r += 4) st4(WT + I + r, acc[r], acc[r + 1], acc[r + 2], acc[r + 3]);
    } else {
#pragma unroll
      for (int r = 0; r < 16; ++r) UH[(size_t)(I + r) * p.Dv] = acc[r];
    }
  }
}

// A thread's eight columns of a 64-column row: x0 .. x0 + 3 and 32 further (eight lanes read 128 neighbouring bytes), as
// pairs for the packed float32 instructions (each half rounds as the single instruction does; 122 against 92 FMA per clock
// and SM measured at 16 warps).
__device__ __forceinline__ void load_cols(const float* p, float2 (&b)[4]) {
  const float4 u = ld4(p), v = ld4(p + 32);
  b[0] = make_float2(u.x, u.y); b[1] = make_float2(u.z, u.w); b[2] = make_float2(v.x, v.y); b[3] = make_float2(v.z, v.w);
}
__device__ __forceinline__ void store_cols(float* p, const float2 (&a)[4]) {
  st4(p, a[0].x, a[0].y, a[1].x, a[1].y);
  st4(p + 32, a[2].x, a[2].y, a[3].x, a[3].y);
}

// ---- U = k~^T v ------------------------------------------------------------------------------------------------------------
template <int N, bool STEP>
__global__ void __launch_bounds__(128) chunk_state_kernel(Params p) {
  constexpr int RT = N / 16;                                  // rows of a thread: 8 or 4
  extern __shared__ __align__(16) float sm[];
  float *ks = sm, *vs = ks + C * N, *ws = vs + C * 64;
  pdl_wait();
  const int h = blockIdx.y, c0 = blockIdx.z * 64, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Place c = place(p, blockIdx.x, h, p.H);
  if (c.n <= 0) return;
  const float* k = STEP ? p.k + (size_t)c.tok * p.k_stride + (size_t)(h / p.hpg) * N : p.KT + c.item * (size_t)(N * C);
  const size_t kstep = STEP ? (size_t)p.k_stride : (size_t)N;
  const float* v = p.v + (size_t)c.tok * p.v_stride + (size_t)h * p.Dv + c0;
  for (int e = tid; e < C * N / 4; e += 128) {
    const int j = e / (N / 4), n = e % (N / 4) * 4;
    const bool live = j < c.n;
    copy16(ks + j * N + n, live ? k + j * kstep + n : p.v, live);
  }
  for (int e = tid; e < C * 16; e += 128) {
    const int j = e / 16, x = e % 16 * 4;
    const bool live = j < c.n;
    copy16(vs + j * 64 + x, live ? v + (size_t)j * p.v_stride + x : p.v, live);
  }
  copy_commit();
  if (STEP && warp == 0) {
    // v_j is written with dt_j prod_{t > j} a_t
    float dt[2], a[2];
    step_of(p, c, h, lane, dt, a);
    float suf = a[0] * a[1];                                   // product over the lanes from this one on
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float x = __shfl_down_sync(0xffffffffu, suf, o);
      if (lane + o < 32) suf *= x;
    }
    float after = __shfl_down_sync(0xffffffffu, suf, 1);
    if (lane == 31) after = 1.f;
    ws[2 * lane] = dt[0] * (a[1] * after);
    ws[2 * lane + 1] = dt[1] * after;
    if (lane == 0 && blockIdx.z == 0) p.DC[c.item] = suf;
  }
  copy_wait<0>();
  __syncthreads();
  const int r0 = warp * (4 * RT) + (lane >> 3) * RT, x0 = (lane & 7) * 4;
  float2 acc[RT][4];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[r][x] = two(0.f);
#pragma unroll 4
  for (int j = 0; j < C; ++j) {
    float a[RT];
    float2 b[4];
#pragma unroll
    for (int r = 0; r < RT; r += 4) *reinterpret_cast<float4*>(a + r) = ld4(ks + j * N + r0 + r);
    load_cols(vs + j * 64 + x0, b);
    if (STEP) {
      const float2 w = two(ws[j]);
#pragma unroll
      for (int x = 0; x < 4; ++x) b[x] = __fmul2_rn(b[x], w);
    }
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const float2 ar = two(a[r]);
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[r][x] = __ffma2_rn(ar, b[x], acc[r][x]);
    }
  }
  float* U = p.U + (c.item * N + r0) * (size_t)p.Dv + c0 + x0;
#pragma unroll
  for (int r = 0; r < RT; ++r) store_cols(U + (size_t)r * p.Dv, acc[r]);
}

// ---- the states between the chunks: U of a chunk becomes the state it starts from -----------------------------------------
__device__ __forceinline__ float4 next_state(float d, float4 s, float4 u) {
  return make_float4(fmaf(d, s.x, u.x), fmaf(d, s.y, u.y), fmaf(d, s.z, u.z), fmaf(d, s.w, u.w));
}
template <bool STEP>
__global__ void __launch_bounds__(256) chain_kernel(Params p) {
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y, N = p.N, Dv = p.Dv;
  const int e = (blockIdx.z * 256 + threadIdx.x) * 4, n = e / Dv;
  int first, live;
  chunks_of(p, s, first, live);
  if (live <= 0 || e >= N * Dv) return;
  float* st = p.state + ((size_t)p.seq_slot[s] * p.H + h) * N * Dv + e;
  const size_t item = (size_t)first * p.H + h;
  float* U = p.U + item * N * Dv + e;
  const float* D = STEP ? p.DC + item : p.DC + item * N + n;
  const size_t ustep = (size_t)p.H * N * Dv, dstep = STEP ? (size_t)p.H : (size_t)p.H * N;
  float4 S = *reinterpret_cast<const float4*>(st);
  for (int c0 = 0; c0 < live; c0 += 4) {                      // four chunks' loads in flight
    float4 u[4];
    float d[4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (c0 + x < live) {
        u[x] = *reinterpret_cast<const float4*>(U + (c0 + x) * ustep);
        d[x] = D[(c0 + x) * dstep];
      }
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (c0 + x < live) {
        *reinterpret_cast<float4*>(U + (c0 + x) * ustep) = S;
        S = next_state(d[x], S, u[x]);
      }
  }
  *reinterpret_cast<float4*>(st) = S;
}

// The delta rule's pass: a block owns 16 columns of one head's state and walks over the chunks; u = U^ - W S, then S' = D S +
// k~^T u.  Both products are taken in shares of their sums (a warp per share of W S: 8 x 4 outputs a thread), whose parts
// meet in shared memory: what bounds a chunk is then the FP32 pipe (1,300 cycles a product), not the operands' loads.
template <int N>
struct ChainShape {
  static constexpr int BUF = 2 * N * C + C * 16 + N, PARTS = 8 * C * 16;
  static constexpr size_t bytes = (2 * BUF + N * 16 + PARTS + C * 16) * sizeof(float);
};
// acc[r][x] += a[k][r] b[k][x] for K neighbouring k, eight rows and four columns a thread
template <int K>
__device__ __forceinline__ void share_product(const float* a, int lda, const float* b, float2 (&acc)[8][2]) {
#pragma unroll
  for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = two(0.f);
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    const float4 u = ld4(a + k * lda), v = ld4(a + k * lda + 4), y = ld4(b + k * 16);
    const float f[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    const float2 lo = make_float2(y.x, y.y), hi = make_float2(y.z, y.w);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      acc[r][0] = __ffma2_rn(two(f[r]), lo, acc[r][0]);
      acc[r][1] = __ffma2_rn(two(f[r]), hi, acc[r][1]);
    }
  }
}
template <int N>
__global__ void __launch_bounds__(256) delta_chain_kernel(Params p) {
  constexpr int T = 256, BUF = ChainShape<N>::BUF, PER_S = N / 2, S_SHARES = T / PER_S, OWN = N * 16 / (4 * T);
  extern __shared__ __align__(16) float sm[];
  float *ss = sm + 2 * BUF, *part = ss + N * 16, *us = part + ChainShape<N>::PARTS;      // state [N][16], shares, u [C][16]
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * 16, Dv = p.Dv, tid = threadIdx.x;
  int first, live;
  chunks_of(p, s, first, live);
  if (live <= 0) return;
  auto load = [&](int c, float* b) {
    const size_t item = (size_t)(first + c) * p.H + h;
    const float *W = p.WT + item * (size_t)(N * C), *K = p.KT + item * (size_t)(N * C), *H = p.UH + item * (size_t)(C * Dv) + c0;
    for (int e = tid; e < N * C / 4; e += T) { copy16(b + 4 * e, W + 4 * e, true); copy16(b + N * C + 4 * e, K + 4 * e, true); }
    for (int e = tid; e < C * 4; e += T) copy16(b + 2 * N * C + 4 * e, H + (size_t)(e / 4) * Dv + e % 4 * 4, true);
    for (int e = tid; e < N / 4; e += T) copy16(b + 2 * N * C + C * 16 + 4 * e, p.DC + item * N + 4 * e, true);
  };
  load(0, sm);
  copy_commit();
  // this thread's four columns of OWN rows of the state, in registers from the first chunk to the last
  float* st = p.state + (((size_t)p.seq_slot[s] * p.H + h) * N) * Dv + c0;
  float4 S[OWN];
#pragma unroll
  for (int o = 0; o < OWN; ++o) {
    const int e = tid + o * T, n = e / 4, x = e % 4 * 4;
    S[o] = ld4(st + (size_t)n * Dv + x);
    *reinterpret_cast<float4*>(ss + 4 * e) = S[o];
  }
  for (int c = 0; c < live; ++c) {
    float* b = sm + (c & 1) * BUF;
    const float *W = b, *K = b + N * C, *H = K + N * C, *D = H + C * 16;
    if (c + 1 < live) load(c + 1, sm + ((c + 1) & 1) * BUF);
    copy_commit();
    copy_wait<1>();
    __syncthreads();                                          // the chunk is here; the state of everybody is in place
    const size_t item = (size_t)(first + c) * p.H + h;
    float2 acc[8][2];
    {
      const int share = tid / 32, i0 = tid % 32 / 4 * 8, x0 = tid % 4 * 4;
      share_product<N / 8>(W + share * (N / 8) * C + i0, C, ss + share * (N / 8) * 16 + x0, acc);
#pragma unroll
      for (int r = 0; r < 8; ++r) st4(part + (share * C + i0 + r) * 16 + x0, acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
    }
#pragma unroll
    for (int o = 0; o < OWN; ++o) {                           // the state that the chunk starts from
      const int e = tid + o * T;
      *reinterpret_cast<float4*>(p.U + (item * N + e / 4) * (size_t)Dv + c0 + e % 4 * 4) = S[o];
    }
    __syncthreads();
    {
      float4 u = ld4(H + 4 * tid);
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const float4 y = ld4(part + x * C * 16 + 4 * tid);
        u = make_float4(u.x - y.x, u.y - y.y, u.z - y.z, u.w - y.w);
      }
      *reinterpret_cast<float4*>(us + 4 * tid) = u;
      *reinterpret_cast<float4*>(p.UH + item * (size_t)(C * Dv) + c0 + (size_t)(tid / 4) * Dv + tid % 4 * 4) = u;
    }
    __syncthreads();
    {
      const int share = tid / PER_S, n0 = tid % PER_S / 4 * 8, x0 = tid % 4 * 4;
      share_product<C / S_SHARES>(K + share * (C / S_SHARES) * N + n0, N, us + share * (C / S_SHARES) * 16 + x0, acc);
#pragma unroll
      for (int r = 0; r < 8; ++r) st4(part + (share * N + n0 + r) * 16 + x0, acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
      const int e = tid + o * T;
      float4 y = ld4(part + 4 * e);
#pragma unroll
      for (int x = 1; x < S_SHARES; ++x) {
        const float4 z = ld4(part + x * N * 16 + 4 * e);
        y = make_float4(y.x + z.x, y.y + z.y, y.z + z.z, y.w + z.w);
      }
      S[o] = next_state(D[e / 4], S[o], y);
      *reinterpret_cast<float4*>(ss + 4 * e) = S[o];
    }
    __syncthreads();                                          // this buffer may be copied into again
  }
  copy_wait<0>();
#pragma unroll
  for (int o = 0; o < OWN; ++o) {
    const int e = tid + o * T;
    *reinterpret_cast<float4*>(st + (size_t)(e / 4) * Dv + e % 4 * 4) = S[o];
  }
}

// ---- the outputs -----------------------------------------------------------------------------------------------------------
// The contraction runs over the state's rows and then over the chunk's tokens, in slices of 16 that come through three
// buffers.  A block is two warps of 8 x 8 outputs a thread (4 x 8 was bound by its shared-memory loads, 75 % of their
// pipe), and eight blocks share an SM: a scheduler needs three or four warps to issue packed instructions back to back.
constexpr int SLICE = 16, STAGES = 3;
template <bool STEP>
struct OutShape {
  static constexpr int LDA = STEP ? C + 4 : C;
  static constexpr size_t bytes = (STAGES * SLICE * (LDA + 64) + 3 * C) * sizeof(float);
};
template <int N, bool STEP, bool DELTA>
__global__ void __launch_bounds__(64) chunk_out_kernel(Params p) {
  constexpr int LDA = OutShape<STEP>::LDA, BUF = SLICE * (LDA + 64), NS = N / SLICE, SLICES = NS + C / SLICE;
  extern __shared__ __align__(16) float sm[];
  float *dts = sm + STAGES * BUF, *as = dts + C, *pre = as + C;
  pdl_wait();
  const int h = blockIdx.y, c0 = blockIdx.z * 64, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, Dv = p.Dv;
  const Place c = place(p, blockIdx.x, h, p.H);
  if (c.n <= 0) return;
  const size_t gi = STEP ? (size_t)blockIdx.x * (p.H / p.hpg) + h / p.hpg : c.item;
  const float *QT = p.QT + gi * (size_t)(N * C), *AT = p.AT + gi * (size_t)(C * C);
  const float* U = p.U + c.item * (size_t)N * Dv + c0;
  const float* v = DELTA ? p.UH + c.item * (size_t)(C * Dv) + c0 : p.v + (size_t)c.tok * p.v_stride + (size_t)h * Dv + c0;
  const size_t vstep = DELTA ? (size_t)Dv : (size_t)p.v_stride;
  auto load = [&](int sl) {
    float *a = sm + sl % STAGES * BUF, *b = a + SLICE * LDA;
    if (sl < NS) {
#pragma unroll
      for (int e = tid; e < SLICE * 16; e += 64) {
        const int n = e / 16, x = e % 16 * 4;
        copy16(a + n * LDA + x, QT + (size_t)(sl * SLICE + n) * C + x, true);
        copy16(b + n * 64 + x, U + (size_t)(sl * SLICE + n) * Dv + x, true);
      }
    } else if (sl < SLICES) {
#pragma unroll
      for (int e = tid; e < SLICE * 16; e += 64) {
        const int j = e / 16, x = e % 16 * 4, t = (sl - NS) * SLICE + j;
        const bool live = t < c.n;
        copy16(a + j * LDA + x, AT + (size_t)t * C + x, true);
        copy16(b + j * 64 + x, live ? v + t * vstep + x : p.v, live);
      }
    }
    copy_commit();
  };
  load(0);
  load(1);
  if (STEP && warp == 0) {
    float dt[2], a[2];
    step_of(p, c, h, lane, dt, a);
    float upto = a[0] * a[1];                                  // product over the lanes up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto *= x;
    }
    float before = __shfl_up_sync(0xffffffffu, upto, 1);
    if (lane == 0) before = 1.f;
#pragma unroll
    for (int e = 0; e < 2; ++e) { dts[2 * lane + e] = dt[e]; as[2 * lane + e] = a[e]; }
    pre[2 * lane] = before * a[0];
    pre[2 * lane + 1] = upto;
  }
  const int i0 = 32 * warp + 8 * (lane >> 3), x0 = 4 * (lane & 7);
  float2 acc[8][4];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[r][x] = two(0.f);
  for (int sl = 0; sl < SLICES; ++sl) {
    copy_wait<1>();
    __syncthreads();                                           // the slice is here; everybody is done with the one before
    load(sl + 2);
    float *a = sm + sl % STAGES * BUF, *b = a + SLICE * LDA;
    const int t0 = (sl - NS) * SLICE;                          // the slice's first token, once the state's rows are done
    if (STEP && sl >= NS) {
      if (sl == NS) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float2 w = two(pre[i0 + r]);
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[r][x] = __fmul2_rn(acc[r][x], w);
        }
      }
      // (C_i . B_j) dt_j prod_{j < t <= i} a_t: a thread takes one j and a quarter of the tokens i, four at a time
      const int j = t0 + tid % SLICE, from = tid / SLICE * 16;
      float L = dts[j];
      for (int t = j + 1; t < from; ++t) L *= as[t];
#pragma unroll
      for (int i = from; i < from + 16; i += 4) {
        float* at = a + tid % SLICE * LDA + i;
        const float4 f = ld4(at);
        float y[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (i + e > j) L *= as[i + e];
          y[e] *= L;
        }
        st4(at, y[0], y[1], y[2], y[3]);
      }
      __syncthreads();
    }
    // a warp's own 32 tokens under their diagonal (nothing of a later token is read), later ones not at all
    if (sl >= NS && t0 >= 32 * warp + 32) continue;
    const bool whole = sl < NS || t0 < 32 * warp;
    auto product = [&](auto masked) {
#pragma unroll 4
      for (int k = 0; k < SLICE; ++k) {
        float av[8];
        float2 bv[4];
        *reinterpret_cast<float4*>(av) = ld4(a + k * LDA + i0);
        *reinterpret_cast<float4*>(av + 4) = ld4(a + k * LDA + i0 + 4);
        load_cols(b + k * 64 + x0, bv);
#pragma unroll
        for (int r = 0; r < 8; ++r)
          if (!masked || t0 + k <= i0 + r) {
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[r][x] = __ffma2_rn(two(av[r]), bv[x], acc[r][x]);
          }
      }
    };
    if (whole) product(std::false_type{});
    else product(std::true_type{});
  }
  // (the skip adds v itself, also with the delta rule, whose products above take the corrected u)
  const float skip = p.skip ? load_any(p.skip, p.small_dtype, h) : 0.f;
  const float* raw = p.v + (size_t)c.tok * p.v_stride + (size_t)h * Dv + c0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int i = i0 + r;
    if (i >= c.n) continue;
    if (p.skip) {
      float2 b[4];
      load_cols(raw + i * p.v_stride + x0, b);
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[r][x] = __ffma2_rn(two(skip), b[x], acc[r][x]);
    }
    store_cols(p.out + (size_t)(c.tok + i) * p.out_stride + (size_t)h * Dv + c0 + x0, acc[r]);
  }
}

// ---- launches --------------------------------------------------------------------------------------------------------------
template <typename K>
static int allow(K kernel, size_t bytes, bool& done) {
  if (!done && bytes > 16 * 1024) {                           // (with the static part some pass the default limit of 48 KB)
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
      set_error("linear_chunks: %zu bytes of shared memory were refused", bytes);
      return 1;
    }
    done = true;
  }
  return 0;
}
#define CPI_CHUNK_LAUNCH(kernel, grid, threads, bytes)                    \
  do {                                                                    \
    static bool done = false;                                             \
    if (allow(kernel, bytes, done)) return 1;                             \
    cpi::launch_pdl(kernel, grid, dim3(threads), bytes, stream, p);       \
    if (int rc = check_launch("linear_chunks")) return rc;                \
  } while (0)

template <int N>
static int run(const Params& p, cudaStream_t stream) {
  const dim3 items(p.seg_chunks, p.H), tiles(p.seg_chunks, p.H, p.Dv / 64);
  const dim3 chain(p.n_seqs, p.H, (N * p.Dv / 4 + 255) / 256);
  constexpr size_t state_bytes = (C * N + C * 64 + C) * sizeof(float);
  if (p.dt) {
    CPI_CHUNK_LAUNCH(prepare_step_kernel<N>, dim3(p.seg_chunks, p.H / p.hpg), 256, 2 * C * (N + 4) * sizeof(float));
    CPI_CHUNK_LAUNCH((chunk_state_kernel<N, true>), tiles, 128, state_bytes);
    CPI_CHUNK_LAUNCH(chain_kernel<true>, chain, 256, (size_t)0);
    CPI_CHUNK_LAUNCH((chunk_out_kernel<N, true, false>), tiles, 64, OutShape<true>::bytes);
  } else if (p.beta) {
    CPI_CHUNK_LAUNCH((prepare_rows_kernel<N / 8, true>), items, 512, (PrepShape<N / 8, true>::bytes));
    CPI_CHUNK_LAUNCH(solve_kernel, dim3(p.seg_chunks, p.H, (N + p.Dv + 127) / 128), 128, C * 128 * sizeof(float));
    CPI_CHUNK_LAUNCH(delta_chain_kernel<N>, dim3(p.n_seqs, p.H, p.Dv / 16), 256, ChainShape<N>::bytes);
    CPI_CHUNK_LAUNCH((chunk_out_kernel<N, false, true>), tiles, 64, OutShape<false>::bytes);
  } else {
    CPI_CHUNK_LAUNCH((prepare_rows_kernel<N / 8, false>), items, 512, (PrepShape<N / 8, false>::bytes));
    CPI_CHUNK_LAUNCH((chunk_state_kernel<N, false>), tiles, 128, state_bytes);
    CPI_CHUNK_LAUNCH(chain_kernel<false>, chain, 256, (size_t)0);
    CPI_CHUNK_LAUNCH((chunk_out_kernel<N, false, false>), tiles, 64, OutShape<false>::bytes);
  }
  return 0;
}

// floats of scratch per chunk: {U, KT, QT, AT, DC, MT, KP, WT, UH} one after another
static void sizes(int kind, int H, int groups, int N, int Dv, long (&n)[9]) {
  const long rows = (long)H * N * C, tri = (long)H * C * C;
  n[0] = (long)H * N * Dv;
  n[1] = kind == 0 ? 0 : rows;
  n[2] = kind == 0 ? (long)groups * N * C : rows;
  n[3] = kind == 0 ? (long)groups * C * C : tri;
  n[4] = kind == 0 ? (H + 3) / 4 * 4 : (long)H * N;
  n[5] = kind == 2 ? tri : 0;
  n[6] = n[7] = kind == 2 ? rows : 0;
  n[8] = kind == 2 ? (long)H * C * Dv : 0;
}

}  // namespace chunks
}  // namespace cpi

using namespace cpi;

// kind 0: one decay per head and token; 1: a decay per row; 2: the delta rule.
extern "C" int cpi_linear_chunks_supported(int n_rows, int n_cols) {
  return (n_rows == 64 || n_rows == 128) && n_cols >= 64 && n_cols % 64 == 0 && n_cols <= 1024;
}

extern "C" long cpi_linear_chunks_scratch(int kind, int n_heads, int groups, int n_rows, int n_cols) {
  long n[9], sum = 0;
  chunks::sizes(kind, n_heads, groups, n_rows, n_cols, n);
  for (long x : n) sum += x;
  return sum;
}

// total_chunks: sum of ceil(tokens / 64) over the sequences.  scratch: at least seg_chunks * cpi_linear_chunks_scratch floats; the
// step runs in segments of seg_chunks chunks.
extern "C" int cpi_linear_chunks(const float* k, long k_stride, const float* q, long q_stride, const float* v, long v_stride,
                                 const float* z, long z_stride, const void* z_bias, float inv_tau, int decay_kind, const float* dt, long dt_stride, const void* dt_bias,
                                 const void* a_log, const void* skip, int small_dtype, const float* beta, long beta_stride,
                                 float q_scale, float* state, float* out, long out_stride, const int* seq_slot,
                                 const int* seq_tok0, const int* seq_new, int n_seqs, int total_chunks, int n_heads,
                                 int heads_per_group, int n_rows, int n_cols, float* scratch, int seg_chunks,
                                 cudaStream_t stream) {
  if (n_seqs == 0 || total_chunks <= 0) return 0;
  CPI_REQUIRE(cpi_linear_chunks_supported(n_rows, n_cols), "linear_chunks: a state of %d x %d is not supported", n_rows, n_cols);
  CPI_REQUIRE((z != nullptr) + (dt != nullptr) == 1 && (dt == nullptr || (a_log != nullptr && beta == nullptr)),
              "linear_chunks: give row decays or step sizes (with the heads' rates); the delta rule comes with row decays");
  CPI_REQUIRE(n_heads > 0 && n_heads <= 65535 && heads_per_group > 0 && n_heads % heads_per_group == 0 && seg_chunks > 0,
              "linear_chunks: heads %d by %d, segments of %d chunks", n_heads, heads_per_group, seg_chunks);
  CPI_REQUIRE(decay_kind == 0 || (decay_kind == 1 && z != nullptr && a_log != nullptr), "linear_chunks: decay kind %d needs row "
              "decays and the heads' rates", decay_kind);
  auto aligned = [](const void* x, long stride) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0 && stride % 4 == 0; };
  CPI_REQUIRE(aligned(k, k_stride) && aligned(q, q_stride) && aligned(v, v_stride) && (!z || aligned(z, z_stride)) &&
              aligned(out, out_stride) && aligned(scratch, 0) && aligned(state, 0), "linear_chunks: rows must start on 16 bytes");
  chunks::Params p{};
  p.k = k; p.k_stride = k_stride; p.q = q; p.q_stride = q_stride; p.v = v; p.v_stride = v_stride;
  p.z = z; p.z_stride = z_stride; p.z_bias = z_bias; p.inv_tau = inv_tau; p.decay_kind = decay_kind; p.dt = dt; p.dt_stride = dt_stride; p.dt_bias = dt_bias; p.a_log = a_log; p.skip = skip;
  p.small_dtype = small_dtype; p.beta = beta; p.beta_stride = beta_stride; p.q_scale = q_scale; p.state = state; p.out = out;
  p.out_stride = out_stride; p.seq_slot = seq_slot; p.seq_tok0 = seq_tok0; p.seq_new = seq_new;
  p.H = n_heads; p.hpg = heads_per_group; p.N = n_rows; p.Dv = n_cols; p.n_seqs = n_seqs;
  const int kind = dt ? 0 : beta ? 2 : 1;
  long n[9];
  chunks::sizes(kind, n_heads, n_heads / heads_per_group, n_rows, n_cols, n);
  float** parts[9] = {&p.U, &p.KT, &p.QT, &p.AT, &p.DC, &p.MT, &p.KP, &p.WT, &p.UH};
  for (int i = 0; i < 9; ++i) { *parts[i] = scratch; scratch += n[i] * seg_chunks; }
  for (p.seg0 = 0; p.seg0 < total_chunks; p.seg0 += seg_chunks) {
    p.seg_chunks = total_chunks - p.seg0 < seg_chunks ? total_chunks - p.seg0 : seg_chunks;
    if (int rc = n_rows == 64 ? chunks::run<64>(p, stream) : chunks::run<128>(p, stream)) return rc;
  }
  return 0;
}
