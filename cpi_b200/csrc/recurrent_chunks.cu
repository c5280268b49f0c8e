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
// Everything is float32, as in the scan; the two large products (U, and the outputs) run on the tensor cores with each operand
// as three bfloat16 terms, which loses no more than the float32 sums (see there), the rest on the FP32 pipe.  Products of
// decays are always taken forward, one factor after another, never as a quotient or as the exponential of a sum of logarithms:
// they lose no digits however strong the decays are and underflow to the zero that the scan reaches too.  A token's output
// reads nothing of later tokens.
//
// Measured (one prompt of 2,048 tokens, width 2,048), the scan, all on the FP32 pipe, here: the recurrence of gated linear
// attention with 8 heads of 128 x 256 480, 114, 72 us (prepare_rows 34 -> 23, chunk_state 25 -> 15, chain 15, chunk_out 41 -> 19; its bytes
// through the L2 take about 20), the delta rule at 1,500 tokens 435, 176, 153 us (48 -> 35, solve 21, delta_chain 77, 31 -> 19), the
// state-space form with 64 heads of 128 x 64 at 1,855 tokens 507, 187, 134 us (prepare_step 18, 53 -> 26, 31, 80 -> 57).
//
//   prepare_rows   the decays per row (their transform too), and A, q~, k~, D (and M, K^) of a chunk and head
//   prepare_step   C_i . B_j of a chunk and group of heads, and the heads' decays: one per head and token
//   solve          W and U^ of the delta rule: 128 right-hand sides a block, 16 x 16 blocks of the triangle in registers
//   chunk_state    U = k~^T v, tiles of 64 columns
//   chain          the states between the chunks; `delta_chain` with the delta rule, 16 columns a block
//   chunk_out      the outputs, 64 tokens x 128 (or 64) columns a tile; `chunk_out_step` with one decay per head and token
//
// A long step runs in segments of chunks so that the scratch stays within what the caller gives.
#include "decay.cuh"
#include "prefill_tc.cuh"

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
  int* error_flag;                               // raised by a tensor-core kernel whose wait ran out
  int seg0, seg_chunks;                          // this launch's chunks, counted over all sequences: seg0 .. seg0 + seg_chunks - 1
  // scratch, per chunk of the segment and head (AT of the step flavour: and group; its MT: the heads' Decays)
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
// Over the whole chunk, carrying each key forward past every later token costs a multiplication and a multiply-add per pair
// of tokens and row, and a load of decay and query for both (34 us for 2,048 tokens of 8 heads of 128 rows; delta rule 45).  So
// the chunk is taken in four runs of 16.  Within a run the keys are carried forward token by token: thread (j, kk) has k_j[n]
// prod a_t[n] for its eighth of the rows (n / 4 mod 8 = kk: eight lanes read 128 neighbouring bytes).  Then every thread takes
// a row and a run: q_i and k_i times the decays from the run's begin to i, k_j times those from j to the run's end, and the
// run's whole product, still one factor after another.  A pair in different runs is the plain product of two such rows, with
// the whole runs between them: 4 x 4 pairs a thread over a quarter of the rows.  Here 23 (delta rule 35) us, of 14 a block 5 the decays (delta rule 8: their exponentials and logarithms), 5 the pairs within runs, 3 those between.
constexpr int RUN = 16, RUNS = C / RUN;
template <int NPT, bool DELTA>
struct PrepShape {
  static constexpr int N = 8 * NPT, LD = N + 4;
  static constexpr size_t bytes = (3 * C * LD + C + N + RUNS * N) * sizeof(float);
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
__global__ void __launch_bounds__(512, 2) prepare_rows_kernel(Params p) {
  using Sh = PrepShape<NPT, DELTA>;
  constexpr int N = Sh::N, LD = Sh::LD, PIECES = C * N / 4 / 512;
  extern __shared__ __align__(16) float sm[];
  float *qs = sm, *as = qs + C * LD, *ks = as + C * LD, *bs = ks + C * LD, *zb = bs + C, *whole = zb + N;
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
    const int e = tid + i * 512, j = e / (N / 4), n = e % (N / 4) * 4, to = j * LD + n;
    const bool live = j < c.n;
    if (live) d[i] = ld4(a + (size_t)j * p.z_stride + n);
    copy16(qs + to, live ? q + (size_t)j * p.q_stride + n : p.q, live);
    copy16(ks + to, live ? k + (size_t)j * p.k_stride + n : p.k, live);
  }
  copy_commit();
  if (DELTA && tid < C) bs[tid] = tid < c.n ? 1.0f / (1.0f + expf(-p.beta[(size_t)(c.tok + tid) * p.beta_stride + h])) : 0.f;
  __syncthreads();                                             // the biases are in place
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int e = tid + i * 512, j = e / (N / 4), n = e % (N / 4) * 4, to = j * LD + n;
    float4 y = make_float4(1.f, 1.f, 1.f, 1.f);
    if (j < c.n) {
      const float* b = zb + n;
      y = make_float4(row_decay_f(d[i].x, b[0], p.inv_tau, p.decay_kind, rate), row_decay_f(d[i].y, b[1], p.inv_tau, p.decay_kind, rate),
                      row_decay_f(d[i].z, b[2], p.inv_tau, p.decay_kind, rate), row_decay_f(d[i].w, b[3], p.inv_tau, p.decay_kind, rate));
    }
    *reinterpret_cast<float4*>(as + to) = y;
  }
  copy_wait<0>();
  __syncthreads();
  float *AT = p.AT + c.item * (size_t)(C * C), *MT = DELTA ? p.MT + c.item * (size_t)(C * C) : nullptr;      // A by rows i, M by rows j
  // ---- pairs within a run
  {
    const int j = 4 * warp + (lane >> 3), kk = lane & 7, end = warp / 4 * RUN + RUN;
    float w[NPT];
#pragma unroll
    for (int r = 0; r < NPT; r += 4) *reinterpret_cast<float4*>(w + r) = ld4(ks + j * LD + 8 * r + 4 * kk);
    auto decay = [&](int i) {
      const float* ai = as + i * LD + 4 * kk;
#pragma unroll
      for (int r = 0; r < NPT; r += 4) {
        const float4 y = ld4(ai + 8 * r);
        const float2 lo = __fmul2_rn(make_float2(w[r], w[r + 1]), make_float2(y.x, y.y));
        const float2 hi = __fmul2_rn(make_float2(w[r + 2], w[r + 3]), make_float2(y.z, y.w));
        w[r] = lo.x; w[r + 1] = lo.y; w[r + 2] = hi.x; w[r + 3] = hi.y;
      }
    };
    auto dot = [&](const float* rows, int i) -> float {        // this thread's eighth of row i . w
      const float* y = rows + i * LD + 4 * kk;
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
    for (int i = 4 * warp; i < end; i += 4) {
      float s[4], m[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (i + e > j) decay(i + e);
        s[e] = dot(qs, i + e);
        if (DELTA) m[e] = dot(ks, i + e);
      }
      const float y = sum4(s, kk), z = DELTA ? sum4(m, kk) : 0.f;
      if (kk < 4) {
        AT[(i + kk) * C + j] = y * p.q_scale;
        if (DELTA) MT[j * C + i + kk] = z * bs[i + kk];
      }
    }
  }
  __syncthreads();
  // ---- a row n and a run b: queries (and keys, for the delta rule) from the run's begin, keys to its end in place of the decays
  const int n = tid % N, b = tid / N;
  if (b < RUNS) {
    float *qc = qs + b * RUN * LD + n, *ac = as + b * RUN * LD + n, *kc = ks + b * RUN * LD + n, key[RUN], P = 1.f, R = 1.f;
#pragma unroll
    for (int t = 0; t < RUN; ++t) {
      P *= ac[t * LD];
      key[t] = kc[t * LD];
      qc[t * LD] *= P;
      if (DELTA) kc[t * LD] = key[t] * P;
    }
    whole[b * N + n] = P;
#pragma unroll
    for (int t = RUN - 1; t >= 0; --t) {
      const float x = ac[t * LD];
      ac[t * LD] = key[t] * R;
      R *= x;
    }
  }
  __syncthreads();
  // ---- what the other kernels read: the same from the chunk's begin, to its end
  if (b < RUNS) {
    const float *qc = qs + b * RUN * LD + n, *ac = as + b * RUN * LD + n, *kc = ks + b * RUN * LD + n;
    float before = 1.f, after = 1.f;
#pragma unroll
    for (int r = 0; r < RUNS; ++r) {
      const float x = whole[r * N + n];
      if (r < b) before *= x;
      if (r > b) after *= x;
    }
    const size_t at = c.item * (size_t)(N * C) + (size_t)b * RUN * N + n;
#pragma unroll 8
    for (int t = 0; t < RUN; ++t) {
      p.QT[at + t * N] = qc[t * LD] * before * p.q_scale;
      p.KT[at + t * N] = ac[t * LD] * after;
      if (DELTA) p.KP[at + t * N] = kc[t * LD] * before;
    }
    if (b == 0) p.DC[c.item * N + n] = whole[n] * after;
  }
  // ---- pairs in different runs I > J: four lanes have 4 x 4 of them, a quarter of the rows each
  if (tid < 6 * 16 * 4) {
    const int pair = tid / 64, l = tid % 4, I = pair < 3 ? pair + 1 : pair < 5 ? pair - 1 : 3, J = pair < 3 ? pair : pair < 5 ? pair - 3 : 0;
    const int i0 = I * RUN + tid / 16 % 4 * 4, j0 = J * RUN + tid / 4 % 4 * 4;
    auto cross = [&](const float* rows, float (&sum)[4]) {     // lane l: rows[i0 + l] . the four keys
      float acc[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[r][x] = 0.f;
#pragma unroll 2
      for (int m = 4 * l; m < N; m += 16) {
        float4 f = make_float4(1.f, 1.f, 1.f, 1.f), y[4];
        for (int r = J + 1; r < I; ++r) {                      // the whole runs between
          const float4 x = ld4(whole + r * N + m);
          f = make_float4(f.x * x.x, f.y * x.y, f.z * x.z, f.w * x.w);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float4 u = ld4(as + (j0 + x) * LD + m);
          y[x] = make_float4(u.x * f.x, u.y * f.y, u.z * f.z, u.w * f.w);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float4 u = ld4(rows + (i0 + r) * LD + m);
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[r][x] = fmaf(u.w, y[x].w, fmaf(u.z, y[x].z, fmaf(u.y, y[x].y, fmaf(u.x, y[x].x, acc[r][x]))));
        }
      }
      const bool hi = l & 2, odd = l & 1;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float u = hi ? acc[2][x] : acc[0][x], v = hi ? acc[3][x] : acc[1][x];
        u += __shfl_xor_sync(0xffffffffu, hi ? acc[0][x] : acc[2][x], 2);
        v += __shfl_xor_sync(0xffffffffu, hi ? acc[1][x] : acc[3][x], 2);
        sum[x] = (odd ? v : u) + __shfl_xor_sync(0xffffffffu, odd ? u : v, 1);
      }
    };
    float sum[4];
    cross(qs, sum);
    st4(AT + (i0 + l) * C + j0, sum[0] * p.q_scale, sum[1] * p.q_scale, sum[2] * p.q_scale, sum[3] * p.q_scale);
    if (DELTA) {
      cross(ks, sum);
#pragma unroll
      for (int x = 0; x < 4; ++x) MT[(j0 + x) * C + i0 + l] = sum[x] * bs[i0 + l];
    }
  }
}

// ---- one decay per head and token: C_i . B_j, once per group of heads, and the decays of its heads ------------------------
// A chunk's decays, one per token: step sizes, decays, what the token's value is written with into the chunk's state (dt_j
// prod_{t > j} a_t), products of decays from the chunk's begin and from the begin of the token's run of eight to the token, and
// of the whole runs between two.  Formed here once and read by every block that needs them: the chain of loads, exponentials
// and scans (5,000 cycles) would stand at the begin of each.
struct Decays { float dt[C], a[C], w[C], upto[C], run[C], mid[8][8]; };
constexpr int DECAYS = sizeof(Decays) / sizeof(float);
__device__ __forceinline__ void decays_of(const Params& p, const Place& c, int h, int lane) {      // one warp; lane: tokens 2 lane, 2 lane + 1
  const float rate = -expf(load_any(p.a_log, p.small_dtype, h)), bias = p.dt_bias ? load_any(p.dt_bias, p.small_dtype, h) : 0.f;
  const size_t item = (size_t)blockIdx.x * p.H + h;
  float dt[2], a[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int j = 2 * lane + e;
    dt[e] = j < c.n ? softplus_f(p.dt[(size_t)(c.tok + j) * p.dt_stride + h] + bias) : 0.f;
    a[e] = j < c.n ? expf(rate * dt[e]) : 1.f;
  }
  // over the lanes up to this one, from this one on, and within its run of eight tokens
  float upto = a[0] * a[1], from = upto, run = upto;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float x = __shfl_up_sync(0xffffffffu, upto, o), y = __shfl_up_sync(0xffffffffu, run, o), z = __shfl_down_sync(0xffffffffu, from, o);
    if (lane >= o) upto *= x;
    if (lane + o < 32) from *= z;
    if (o < 4 && (lane & 3) >= o) run *= y;
  }
  float before = __shfl_up_sync(0xffffffffu, upto, 1), run_before = __shfl_up_sync(0xffffffffu, run, 1), after = __shfl_down_sync(0xffffffffu, from, 1);
  if (lane == 0) before = 1.f;
  if ((lane & 3) == 0) run_before = 1.f;
  if (lane == 31) after = 1.f;
  Decays& D = reinterpret_cast<Decays*>(p.MT)[item];
  auto put = [&](float* to, float x, float y) { reinterpret_cast<float2*>(to)[lane] = make_float2(x, y); };
  put(D.dt, dt[0], dt[1]);
  put(D.a, a[0], a[1]);
  put(D.w, dt[0] * (a[1] * after), dt[1] * after);
  put(D.upto, before * a[0], upto);
  put(D.run, run_before * a[0], run);
  float whole[8];                                              // of each run
#pragma unroll
  for (int r = 0; r < 8; ++r) whole[r] = __shfl_sync(0xffffffffu, run, 4 * r + 3);
  const int x = lane / 4, y = lane % 4 * 2;                    // mid[x][y], mid[x][y + 1]: the runs x + 1 .. y - 1
  float m0 = 1.f, m1 = 1.f;
#pragma unroll
  for (int r = 1; r < 8; ++r) {
    if (r > x && r < y) m0 *= whole[r];
    if (r > x && r < y + 1) m1 *= whole[r];
  }
  put(&D.mid[0][0], m0, m1);
  if (lane == 0) p.DC[item] = from;
}
template <int N>
__global__ void __launch_bounds__(256) prepare_step_kernel(Params p) {
  constexpr int LD = N + 4;
  extern __shared__ __align__(16) float sm[];
  float *cs = sm, *bs = cs + C * LD;
  pdl_wait();
  const int g = blockIdx.y, G = p.H / p.hpg, tid = threadIdx.x;
  const Place c = place(p, blockIdx.x, g, G);
  if (c.n <= 0) return;
  for (int h = g * p.hpg + (tid >> 5); h < (g + 1) * p.hpg; h += 8) decays_of(p, c, h, tid & 31);
  for (int e = tid; e < C * N / 4; e += 256) {
    const int j = e / (N / 4), n = e % (N / 4) * 4;
    const bool live = j < c.n;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(cs + j * LD + n) = live ? ld4(p.q + (size_t)(c.tok + j) * p.q_stride + (size_t)g * N + n) : zero;
    *reinterpret_cast<float4*>(bs + j * LD + n) = live ? ld4(p.k + (size_t)(c.tok + j) * p.k_stride + (size_t)g * N + n) : zero;
  }
  __syncthreads();
  // thread: tokens i0, i0 + 16, .. of C against tokens j0, j0 + 16, .. of B
  const int j0 = tid & 15, i0 = tid >> 4;
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
    for (int y = 0; y < 4; ++y) AT[(i0 + 16 * x) * C + j0 + 16 * y] = acc[x][y] * p.q_scale;
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

// ---- products on the tensor cores -----------------------------------------------------------------------------------------
// A float32 operand enters as three bfloat16 terms, x = h + m + l to 2^-25 of it (8 bits a term).  Of the nine products of
// terms the six above 2^-24 are taken.  h h has an accumulator of its own and the small ones another: a product adds into its
// accumulator with one truncation, so what counts is how many of them the large sum sees, K / 16 for the 64 to 192 terms
// here, no more than a float32 sum of that length loses, and what truncation takes on average is given back (OUT_LOST).  Against
// 64 bits, four heads of 128 x 256 at 1,500 tokens, decays as layers are initialised: outputs 2.05e-7 and states 1.74e-7 off with
// float32 sums, 1.71e-7 and 1.66e-7 with these; with one decay per token 2.98e-7 and 2.37e-7, 2.74e-7 and 2.33e-7; outputs of the
// delta rule 2.03e-7, 1.99e-7.
//
// The operand with a row a lane (M) is loaded a lane's row a thread, its neighbours' beside it, split in registers and left in
// tensor memory; the other goes to shared memory as it lies in memory, a tile of 64 rows of 64 columns per term, 128 bytes a
// row in the 128-byte swizzle, read MN-major where its rows are k, else K-major.  With both in shared memory a product of 64
// columns waits for its operands (83 cycles instead of 32), and writing and reading them fill that memory's pipe: blocks of 256
// threads, three an SM, took 28 us for the outputs of 8 heads of 128 x 256 at 2,048 tokens, a stream of warps with a task each
// (splitting, issuing, writing out) 33, the form here 19.  What bounds it now is latency: a slice of 64 k takes two blocks an SM
// 4,000 cycles (splitting 700, loads' issue 900, 24 products 1,100, waits) of which the tensor pipe works 1,500.  Two blocks an SM leave
// 128 registers a thread: the outputs of 128 columns keep 29 to 31 of their numbers in memory, the step flavour's 9 to 12.
using pre::smem_u32;
constexpr uint32_t TILE = 64 * 128;
constexpr int TC_THREADS = 256;
constexpr uint32_t TC_COLUMNS = 256;                           // tensor memory: h h, small products (64 each), three terms of M (96)
constexpr uint32_t SMALL = 64, TERMS = 128;
// The share of a sum that the truncation of its K / 16 additions takes from it on average (2 to 4e-8 measured, by the mean of (result - exact)
// sign(exact) against that of float32 sums), given back where the two accumulators are added, before that rounding.
constexpr float STATE_LOST = 1.5f / (1 << 25), OUT_LOST = 1.f / (1 << 25);

// A float32 that is no finite number, or so large that its first term is none (from 2^128 - 2^119 on), has no such terms: its last
// one is NaN, and so are the sums that it enters, whatever it meets there.  A sum that comes out as NaN is formed again in
// float32, as one chain of multiply-adds, by the thread that writes it: it is then the infinity or NaN of float32 sums.
// Values, which would also reach the sums of earlier tokens through the zeros above the diagonal, are taken as zero
// instead, and the sums that they belong to are formed again.
__device__ __forceinline__ bool has_terms(float x) { return fabsf(x) < 3.3961775292304601e38f; }      // 2^128 - 2^119
// h, m and l of a pair, packed
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pre::pack_bf16(a, b);
  a -= __uint_as_float(h << 16);
  b -= __uint_as_float(h & 0xffff0000u);
  m = pre::pack_bf16(a, b);
  a -= __uint_as_float(m << 16);
  b -= __uint_as_float(m & 0xffff0000u);
  l = pre::pack_bf16(a, b);
}
// The M operand, 128 lanes x 64 k: a thread has 32 k of a lane's row (warps 0 to 3 the first ones).  Element k of a lane's row is
// src[k * stride] with src at the lane's column.
struct LaneOperand {
  float x[32];
  __device__ __forceinline__ void load(const float* src, size_t stride, int n) {     // n of the thread's k; the rest are zeros
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      x[k] = k < n ? *src : 0.f;
      src += stride;
      asm volatile("" : "+l"(src));                            // (32 addresses at a time would not fit in registers)
    }
  }
  __device__ __forceinline__ void split(uint32_t (&w)[3][16]) const {
#pragma unroll
    for (int e = 0; e < 16; ++e) split2(x[2 * e], x[2 * e + 1], w[0][e], w[1][e], w[2][e]);
  }
  // The same for values of the tokens from `token` on: those without terms become zeros, and `first` the first such token.
  __device__ __forceinline__ void split_values(uint32_t (&w)[3][16], int token, int* first) {
    split(w);
    __nv_bfloat162 none = __floats2bfloat162_rn(0.f, 0.f);      // not zero if any last term is NaN
#pragma unroll
    for (int e = 0; e < 16; ++e) none = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w[2][e]), __floats2bfloat162_rn(0.f, 0.f), none);
    if ((*reinterpret_cast<const uint32_t*>(&none) & 0x7fff7fffu) == 0) return;
#pragma unroll
    for (int e = 0; e < 32; ++e)
      if (!has_terms(x[e])) { atomicMin(first, token + e); x[e] = 0.f; }
    split(w);
  }
};
__device__ __forceinline__ void put_lanes(uint32_t tmem, int warp, const uint32_t (&w)[3][16]) {
  const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + TERMS + (warp >> 2) * 16;
#pragma unroll
  for (int t = 0; t < 3; ++t) pre::tmem_st16_nowait(at + t * 32, w[t]);
  pre::tmem_wait_st();
}
// The other operand, 64 x 64: two groups of eight columns a thread.
struct TileOperand {
  float4 x[2][2];
  // rows from src, `stride` floats apart, n of them; the rest are zeros
  __device__ __forceinline__ void load(const float* src, size_t stride, int n, int tid) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int row = tid / 8 + u * 32, col = tid % 8 * 8;
      x[u][0] = x[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < n) {
        const float* at = src + row * stride + col;
        x[u][0] = ld4(at);
        x[u][1] = ld4(at + 4);
      }
    }
  }
  // fix(row, first column, the eight values)
  template <typename Fix> __device__ __forceinline__ void put(uint8_t* tile, int tid, Fix fix) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int row = tid / 8 + u * 32, col = tid % 8 * 8;
      float y[8] = {x[u][0].x, x[u][0].y, x[u][0].z, x[u][0].w, x[u][1].x, x[u][1].y, x[u][1].z, x[u][1].w};
      fix(row, col, y);
      uint32_t w[3][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) split2(y[2 * e], y[2 * e + 1], w[0][e], w[1][e], w[2][e]);
      uint8_t* to = tile + row * 128 + (((col >> 3) ^ (row & 7)) << 4);
#pragma unroll
      for (int t = 0; t < 3; ++t) *reinterpret_cast<uint4*>(to + t * TILE) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
    }
  }
};
// acc += A B over 64 k, one thread.  `fresh`: the accumulators hold nothing yet.
template <bool B_MN>
__device__ __forceinline__ void products(uint32_t tmem, uint32_t tile, bool fresh) {
  constexpr uint32_t idesc = pre::instr_desc(128, 64, B_MN);
  const uint64_t b = pre::smem_desc(tile, B_MN ? TILE : 16, 1024);
  auto mma = [&](uint32_t d, uint32_t a, uint64_t bb, bool first) {
    if (first) pre::umma_bf16_a_tmem_c<false>(d, a, bb, idesc);
    else pre::umma_bf16_a_tmem_c<true>(d, a, bb, idesc);
  };
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t h = tmem + TERMS + k * 8, m = h + 32, l = h + 64, s = tmem + SMALL;
    const uint64_t bh = b + (uint64_t)(k * (B_MN ? 2048 >> 4 : 32 >> 4)), bm = bh + (TILE >> 4), bl = bm + (TILE >> 4);
    mma(tmem, h, bh, fresh && k == 0);
    mma(s, l, bh, fresh && k == 0);
    mma(s, h, bl, false);
    mma(s, m, bm, false);
    mma(s, m, bh, false);
    mma(s, h, bm, false);
  }
}
// The same for sums of which the large part holds something already, in a half of the 128 lanes or in all of them.
enum Lanes : int { kAllLanes, kLowerLanes, kUpperLanes };
__device__ __forceinline__ void products_onto(uint32_t tmem, uint32_t tile, Lanes lanes) {
  constexpr uint32_t idesc = pre::instr_desc(128, 64, false);
  const uint64_t b = pre::smem_desc(tile, 16, 1024);
  const uint32_t lo = lanes == kUpperLanes ? ~0u : 0u, hi = lanes == kLowerLanes ? ~0u : 0u;      // lanes that stay as they are
  auto mma = [&](uint32_t d, uint32_t a, uint64_t bb, uint32_t onto) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %6, %6}, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bb), "r"(idesc), "r"(onto), "r"(lo), "r"(hi) : "memory");
  };
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t h = tmem + TERMS + k * 8, m = h + 32, l = h + 64, s = tmem + SMALL;
    const uint64_t bh = b + (uint64_t)(k * (32 >> 4)), bm = bh + (TILE >> 4), bl = bm + (TILE >> 4);
    mma(tmem, h, bh, 1);
    mma(s, l, bh, k > 0);
    mma(s, h, bl, 1);
    mma(s, m, bm, 1);
    mma(s, m, bh, 1);
    mma(s, h, bm, 1);
  }
}
// COLUMNS (16 or 32) of both accumulators, added; whether any sum is no finite number.  `lost`: see OUT_LOST, or 0.
template <int COLUMNS>
__device__ __forceinline__ bool tmem_sum(uint32_t at, float lost, float (&v)[COLUMNS]) {
  uint32_t a[COLUMNS], b[COLUMNS];
  if constexpr (COLUMNS == 32) {
    pre::tmem_ld32_issue(at, a);
    pre::tmem_ld32_issue(at + SMALL, b);
  } else {
    pre::tmem_ld16_issue(at, a);
    pre::tmem_ld16_issue(at + SMALL, b);
  }
  pre::tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < COLUMNS; ++i) {
    asm volatile("" : "+r"(a[i]), "+r"(b[i]));                 // (not before the wait)
    const float large = __uint_as_float(a[i]), small = __uint_as_float(b[i]);
    v[i] = large + (lost == 0.f ? small : fmaf(large, lost, small));
  }
  float zero = 0.f;
#pragma unroll
  for (int i = 0; i < COLUMNS; ++i) zero = fmaf(v[i], 0.f, zero);
  return zero != 0.f;
}
// What a block of the two kernels begins and ends with; two share an SM.
struct Tensor { uint64_t bar; uint32_t base; int gave_up; };
__device__ __forceinline__ void tensor_begin(Tensor& t, int tid) {
  if (tid == 0) {
    pre::mbar_init(&t.bar, 1);
    t.gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&t.base)), "r"(TC_COLUMNS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  pre::fence_before_sync();
  __syncthreads();
  pre::fence_after_sync();
}
__device__ __forceinline__ void tensor_end(Tensor& t, int tid, bool ok, int* error_flag) {
  if (!ok) {
    if (tid == 0 && error_flag) atomicExch(error_flag, 1);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);          // products in flight may still read shared memory
  }
  pre::fence_before_sync();
  __syncthreads();
  if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t.base), "r"(TC_COLUMNS));
}
// All operands of a slice are in place: the products of a slice begin.
template <bool B_MN>
__device__ __forceinline__ bool tensor_issue(Tensor& t, int tid, uint8_t* tile, bool ok, bool fresh) {
  pre::fence_async_proxy();
  pre::fence_before_sync();
  ok = __syncthreads_and(ok) != 0;
  if (ok && tid < 32) {
    pre::fence_after_sync();
    if (pre::elect_one()) {
      products<B_MN>(t.base, smem_u32(tile), fresh);
      pre::umma_commit(&t.bar);
    }
    __syncwarp();
  }
  return ok;
}
// Scores times values onto the state's products: one head's for all lanes, or those of two heads for a half of the lanes each.
__device__ __forceinline__ bool tensor_issue_heads(Tensor& t, int tid, uint8_t* tile, bool ok, bool two_heads) {
  pre::fence_async_proxy();
  pre::fence_before_sync();
  ok = __syncthreads_and(ok) != 0;
  if (ok && tid < 32) {
    pre::fence_after_sync();
    if (pre::elect_one()) {
      products_onto(t.base, smem_u32(tile), two_heads ? kLowerLanes : kAllLanes);
      if (two_heads) products_onto(t.base, smem_u32(tile + 3 * TILE), kUpperLanes);
      pre::umma_commit(&t.bar);
    }
    __syncwarp();
  }
  return ok;
}

// ---- U = k~^T v ------------------------------------------------------------------------------------------------------------
// The state's rows are the product's lanes, so that what depends on the keys alone is split once for all columns that see
// them: a block takes up to eight tiles of 64 columns, of one head or (one decay per head) of a group's heads.
constexpr int MOST_TILES = 8;
// The tiles of a block: of one unit (the heads whose keys are the same), `per_block` of them.
template <int DT, bool STEP>
struct Tiles {
  int unit, heads, per_head, first, count;
  __device__ __forceinline__ Tiles(const Params& p, int per_block)
      : unit(blockIdx.y), heads(STEP ? p.hpg : 1), per_head(p.Dv / DT), first(blockIdx.z * per_block) {
    count = min(per_block, heads * per_head - first);
  }
  __device__ __forceinline__ int head(int i) const { return unit * heads + (first + i) / per_head; }
  __device__ __forceinline__ int column(int i) const { return (first + i) % per_head * DT; }
};
// Two buffers of the values' terms, and rows of U on their way out (a lane has a row of the state, a row of U goes out whole).
template <int N> constexpr size_t STATE_BYTES = 6 * TILE + N * 64 * sizeof(float);
template <int N, bool STEP>
__global__ void __launch_bounds__(TC_THREADS, 2) chunk_state_kernel(Params p, int per_block) {
  extern __shared__ __align__(1024) uint8_t tile[];
  __shared__ Tensor t;
  __shared__ float ws[STEP ? MOST_TILES : 1][C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n = (warp & 3) * 32 + lane, half = warp >> 2;
  tensor_begin(t, tid);
  pdl_launch_dependents();                                    // (tensor memory is ours: see common.cuh)
  pdl_wait();
  const Tiles<64, STEP> tiles(p, per_block);
  const int count = tiles.count;
  const Place c = place(p, blockIdx.x, tiles.unit * tiles.heads, p.H);
  bool ok = true;
  if (c.n > 0 && count > 0) {
    auto item = [&](int h) { return (size_t)blockIdx.x * p.H + h; };
    LaneOperand k;
    TileOperand v;
    const float* keys = STEP ? p.k + (size_t)c.tok * p.k_stride + (size_t)tiles.unit * N : p.KT + c.item * (size_t)(N * C);
    const size_t step = STEP ? (size_t)p.k_stride : (size_t)N;
    if (n < N) k.load(keys + half * 32 * step + n, step, c.n - half * 32);
    auto values = [&](int i) { return p.v + (size_t)c.tok * p.v_stride + (size_t)tiles.head(i) * p.Dv + tiles.column(i); };
    auto load = [&](int i) { v.load(values(i), p.v_stride, c.n, tid); };
    load(0);
    if (STEP) {                                                // v_j is written with dt_j prod_{t > j} a_t
      for (int e = tid; e < count * C; e += TC_THREADS) ws[e / C][e % C] = reinterpret_cast<const Decays*>(p.MT)[item(tiles.head(e / C))].w[e % C];
      __syncthreads();
    }
    auto put = [&](int i) {
      v.put(tile + (i & 1) * 3 * TILE, tid, [&](int row, int, float* y) {
        if (STEP) {
          const float f = ws[STEP ? i : 0][row];
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] *= f;
        }
      });
    };
    if (n < N) {
      uint32_t w[3][16];
      k.split(w);
      put_lanes(t.base, warp, w);
    }
    put(0);
    if (count > 1) load(1);
    ok = tensor_issue<true>(t, tid, tile, ok, true);
    for (int i = 0; i < count && ok; ++i) {
      if (i + 1 < count) put(i + 1);
      if (i + 2 < count) load(i + 2);
      ok = pre::mbar_wait(&t.bar, i & 1, &t.gave_up);
      pre::fence_after_sync();
      if (__all_sync(0xffffffffu, ok) && n < N) {
        float y[32];
        const bool again = tmem_sum<32>(t.base + ((uint32_t)((warp & 3) * 32) << 16) + half * 32, STATE_LOST, y);
        // 16 bytes at a time, rows of 256 turned by their number; each warp reads what it wrote
        uint8_t* rows = tile + 6 * TILE;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          st4(reinterpret_cast<float*>(rows + n * 256 + (((half * 8 + e) ^ (n & 15)) << 4)), y[4 * e], y[4 * e + 1], y[4 * e + 2], y[4 * e + 3]);
        __syncwarp();
        float* U = p.U + item(tiles.head(i)) * N * (size_t)p.Dv + tiles.column(i);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int r = (warp & 3) * 32 + e * 4 + lane / 8, x = half * 8 + lane % 8;
          *reinterpret_cast<float4*>(U + (size_t)r * p.Dv + x * 4) = ld4(reinterpret_cast<const float*>(rows + r * 256 + ((x ^ (r & 15)) << 4)));
        }
        __syncwarp();
#pragma unroll 1
        for (int x = half * 32; again && x < half * 32 + 32; ++x) {      // (sums of numbers without terms)
          float* at = U + (size_t)n * p.Dv + x;
          if (*at == *at) continue;
          float sum = 0.f;
          for (int j = 0; j < c.n; ++j) {
            const float y = values(i)[j * p.v_stride + x];
            sum = fmaf(keys[j * step + n], STEP ? y * ws[STEP ? i : 0][j] : y, sum);
          }
          *at = sum;
        }
      }
      if (i + 1 < count) ok = tensor_issue<true>(t, tid, tile + ((i + 1) & 1) * 3 * TILE, ok, true);
    }
    ok = __syncthreads_and(ok) != 0;
  }
  tensor_end(t, tid, ok, p.error_flag);
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
// The contraction runs over the state's rows and then over the chunk's tokens, 64 at a time; a slice's loads are on the way
// while the slice before is split and multiplied.  Columns are the product's lanes, tokens its columns.
// DT columns a tile: 128, or 64 (the upper lanes then do the same as the lower ones, and are not read).  A block takes up to
// eight tiles; the queries and scores of one head are split for the first one only.
template <int N> constexpr size_t OUT_BYTES = (N / 64 + 1) * 3 * TILE;
template <int N, int DT, bool DELTA>
__global__ void __launch_bounds__(TC_THREADS, 2) chunk_out_kernel(Params p, int per_block) {
  constexpr int SLICES = N / 64 + 1;
  extern __shared__ __align__(1024) uint8_t tile[];
  __shared__ Tensor t;
  __shared__ int bad[2][DT];                                   // per column the first token whose value has no terms
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, Dv = p.Dv;
  const int x = ((warp & 3) * 32 + lane) % DT, half = warp >> 2;      // column of the tile
  if (tid < DT) bad[0][tid] = bad[1][tid] = C;
  tensor_begin(t, tid);
  pdl_launch_dependents();                                    // (tensor memory is ours: see common.cuh)
  pdl_wait();
  const Tiles<DT, false> tiles(p, per_block);
  const int count = tiles.count;
  const Place c = place(p, blockIdx.x, tiles.unit * tiles.heads, p.H);
  bool ok = true;
  if (c.n > 0 && count > 0) {
    const float* AT = p.AT + c.item * (size_t)(C * C);
    const size_t vstep = DELTA ? (size_t)Dv : (size_t)p.v_stride;
    auto values = [&](int i) {
      return (DELTA ? p.UH + c.item * (size_t)(C * Dv) : p.v + (size_t)c.tok * p.v_stride + (size_t)tiles.head(i) * Dv) + tiles.column(i);
    };
    LaneOperand a;
    TileOperand b;
    auto load_a = [&](int i, int sl) {
      if (sl < SLICES - 1) a.load(p.U + (c.item * N + sl * 64 + half * 32) * (size_t)Dv + tiles.column(i) + x, Dv, 32);
      else a.load(values(i) + half * 32 * vstep + x, vstep, c.n - half * 32);
    };
    auto load_b = [&](int i, int sl) {
      if (i > 0) return;
      if (sl == SLICES - 1) b.load(AT, C, c.n, tid);
      else b.load(p.QT + c.item * (size_t)(N * C) + sl * 64, N, c.n, tid);
    };
    load_a(0, 0);
    load_b(0, 0);
    int round = 0;                                             // products begun
    for (int i = 0; i < count && ok; ++i) {
      // (the skip adds v itself, also with the delta rule, whose products take the corrected u)
      const float skip = p.skip ? load_any(p.skip, p.small_dtype, tiles.head(i)) : 0.f;
#pragma unroll
      for (int sl = 0; sl < SLICES; ++sl) {
        const bool last = sl == SLICES - 1;
        uint32_t w[3][16];
        if (last) a.split_values(w, half * 32, &bad[i & 1][x]);
        else a.split(w);
        if (sl > 0) {
          ok = ok && pre::mbar_wait(&t.bar, (round - 1) & 1, &t.gave_up);
          pre::fence_after_sync();
        }
        put_lanes(t.base, warp, w);
        if (!last) load_a(i, sl + 1);
        else if (i + 1 < count) load_a(i + 1, 0);
        if (i == 0)
          b.put(tile + sl * 3 * TILE, tid, [&](int r, int j0, float* y) {
            if (!last) return;
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = j0 + e > r ? 0.f : y[e];
          });
        if (!last) load_b(i, sl + 1);
        else if (i + 1 < count) load_b(i + 1, 0);
        ok = tensor_issue<false>(t, tid, tile + sl * 3 * TILE, ok, sl == 0);
        ++round;
        if (!ok) break;
      }
      // (with 64 columns two warps hold the same sums: each writes half of the tokens)
      constexpr int ROWS = DT / 4;
      const int i0 = half * 32 + (DT == 64 ? (warp >> 1 & 1) * 16 : 0);
      float raw[ROWS];
      if (p.skip) {
        const float* from = p.v + (size_t)(c.tok + i0) * p.v_stride + (size_t)tiles.head(i) * Dv + tiles.column(i) + x;
#pragma unroll
        for (int e = 0; e < ROWS; ++e) {
          raw[e] = i0 + e < c.n ? *from : 0.f;
          from += p.v_stride;
          asm volatile("" : "+l"(from));
        }
      }
      ok = ok && pre::mbar_wait(&t.bar, (round - 1) & 1, &t.gave_up);
      pre::fence_after_sync();
      if (__all_sync(0xffffffffu, ok) && i0 < c.n) {
        const int first = bad[i & 1][x];
        float y[ROWS];
        const bool again = tmem_sum<ROWS>(t.base + ((uint32_t)((warp & 3) * 32) << 16) + i0, OUT_LOST, y) || first < C;
        float* out = p.out + (size_t)(c.tok + i0) * p.out_stride + (size_t)tiles.head(i) * Dv + tiles.column(i) + x;
        float* to = out;
#pragma unroll
        for (int e = 0; e < ROWS; ++e) {
          if (i0 + e < c.n) *to = p.skip ? fmaf(skip, raw[e], y[e]) : y[e];
          to += p.out_stride;
          asm volatile("" : "+l"(to));                         // (32 addresses at a time would not fit in registers)
        }
#pragma unroll 1
        for (int r = i0; again && r < min(i0 + ROWS, c.n); ++r) {      // (sums of numbers without terms)
          float* at = out + (r - i0) * p.out_stride;
          if (r < first && *at == *at) continue;
          const float *query = p.QT + (c.item * C + r) * (size_t)N, *states = p.U + c.item * N * (size_t)Dv + tiles.column(i) + x;
          float o = 0.f;
          for (int n = 0; n < N; ++n) o = fmaf(query[n], states[(size_t)n * Dv], o);
          for (int j = 0; j <= r; ++j) o = fmaf(AT[r * C + j], values(i)[j * vstep + x], o);
          if (p.skip) o = fmaf(skip, p.v[(size_t)(c.tok + r) * p.v_stride + (size_t)tiles.head(i) * Dv + tiles.column(i) + x], o);
          *at = o;
        }
      }
      ok = __syncthreads_and(ok) != 0;                         // (one decision; everybody has read what the next tiles' values may change)
      if (half == 0) bad[i & 1][x] = C;
    }
    ok = __syncthreads_and(ok) != 0;
  }
  tensor_end(t, tid, ok, p.error_flag);
}

// The same with one decay per head and token, for 128 neighbouring columns of a group's heads a tile, each half of 64 of one
// head.  The queries are the group's, so their terms are formed once for a block's tiles and the decays up to each token are put
// on the sums of the state's products in tensor memory.  The scores are a head's own: of a tile with two heads either's products
// leave the other's lanes alone (the instruction's lane mask: nothing of one head reaches the other, whatever its values).
// A tile per 64 columns, with every lane's work done twice and the queries' terms formed for each head, took 72 us for 64 heads
// of 128 x 64 at 1,855 tokens, this form 57 (a block's tiles: four there; two or one take 60).
template <int N> constexpr size_t STEP_OUT_BYTES = (N / 64 + 2) * 3 * TILE;
template <int N>
__global__ void __launch_bounds__(TC_THREADS, 2) chunk_out_step_kernel(Params p, int per_block) {
  constexpr int SLICES = N / 64;
  extern __shared__ __align__(1024) uint8_t tile[];
  __shared__ Tensor t;
  __shared__ __align__(16) Decays decays[2][2];                // this tile's, the next one's: of either half's head
  __shared__ int bad[2][128];                                  // as above
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, Dv = p.Dv;
  const int x = (warp & 3) * 32 + lane, half = warp >> 2, side = x >> 6;      // column of the tile, tokens' half, the column's half
  if (tid < 128) bad[0][tid] = bad[1][tid] = C;
  tensor_begin(t, tid);
  pdl_launch_dependents();                                    // (tensor memory is ours: see common.cuh)
  pdl_wait();
  const int unit = blockIdx.y, columns = p.hpg * Dv, first = blockIdx.z * per_block;
  const int count = min(per_block, (columns + 127) / 128 - first);
  const Place c = place(p, blockIdx.x, unit * p.hpg, p.H);
  bool ok = true;
  if (c.n > 0 && count > 0) {
    // the last tile may hold one half; its other lanes work on zeros and are not stored
    auto column = [&](int i) { return (first + i) * 128 + x; };
    auto live = [&](int i) { return column(i) < columns; };
    auto head = [&](int i, int s) { return unit * p.hpg + min((first + i) * 128 + s * 64, columns - 64) / Dv; };
    auto item = [&](int h) { return (size_t)blockIdx.x * p.H + h; };
    const float* AT = p.AT + ((size_t)blockIdx.x * (p.H / p.hpg) + unit) * (size_t)(C * C);
    auto values = [&](int i) { return p.v + (size_t)c.tok * p.v_stride + (size_t)unit * columns + column(i); };
    LaneOperand a;
    TileOperand b;                                             // the queries' slices (for the first tile), the scores
    auto load_a = [&](int i, int sl) {
      if (sl < SLICES) a.load(p.U + (item(head(i, side)) * N + sl * 64 + half * 32) * (size_t)Dv + column(i) % Dv, Dv, live(i) ? 32 : 0);
      else a.load(values(i) + half * 32 * p.v_stride, p.v_stride, live(i) ? c.n - half * 32 : 0);
    };
    auto load_b = [&](int sl) {
      if (sl < SLICES) b.load(p.q + (size_t)c.tok * p.q_stride + (size_t)unit * N + sl * 64, p.q_stride, c.n, tid);
      else b.load(AT, C, c.n, tid);
    };
    auto ask_decays = [&](int i) {
      for (int e = tid; e < DECAYS / 2; e += TC_THREADS) {
        const int s = e / (DECAYS / 4), at = e % (DECAYS / 4) * 4;
        copy16(reinterpret_cast<float*>(&decays[i & 1][s]) + at, p.MT + item(head(i, s)) * DECAYS + at, true);
      }
      copy_commit();
    };
    ask_decays(0);
    load_a(0, 0);
    load_b(0);
    int round = 0;                                             // products begun
    const uint32_t sums = t.base + ((uint32_t)((warp & 3) * 32) << 16) + half * 32;
    for (int i = 0; i < count && ok; ++i) {
      const int h = head(i, side);
      const Decays& D = decays[i & 1][side];
      const float skip = p.skip ? load_any(p.skip, p.small_dtype, h) : 0.f;
#pragma unroll
      for (int sl = 0; sl < SLICES; ++sl) {
        uint32_t w[3][16];
        a.split(w);
        if (sl > 0) {
          ok = ok && pre::mbar_wait(&t.bar, (round - 1) & 1, &t.gave_up);
          pre::fence_after_sync();
        }
        put_lanes(t.base, warp, w);
        load_a(i, sl + 1);
        if (i == 0) {
          b.put(tile + sl * 3 * TILE, tid, [&](int, int, float* y) {
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] *= p.q_scale;
          });
        }
        if (i == 0 || sl == SLICES - 1) load_b(sl + 1);
        if (sl == SLICES - 1) copy_wait<0>();                  // this tile's decays
        ok = tensor_issue<false>(t, tid, tile + sl * 3 * TILE, ok, sl == 0);
        ++round;
        if (!ok) break;
      }
      if (!ok) break;
      if (i + 1 < count) ask_decays(i + 1);                    // (everybody is done with the tile before)
      const bool two_heads = head(i, 0) != head(i, 1);
      for (int s = 0; s <= (two_heads ? 1 : 0); ++s) {
        const Decays& E = decays[i & 1][s];
        b.put(tile + (SLICES + s) * 3 * TILE, tid, [&](int r, int j0, float* y) {
          if (r >= j0) {
            // (C_i . B_j) dt_j prod_{j < t <= i} a_t, from the row's end of this run of eight backwards
            const int from = j0 / 8, to = r / 8;
            float L = to > from ? E.run[r] * E.mid[from][to] : 1.f, dt[8], d[8];
#pragma unroll
            for (int e = 0; e < 8; e += 4) {
              *reinterpret_cast<float4*>(dt + e) = ld4(E.dt + j0 + e);
              *reinterpret_cast<float4*>(d + e) = ld4(E.a + j0 + e);
            }
#pragma unroll
            for (int e = 7; e >= 0; --e) {
              y[e] *= dt[e] * L;
              L = j0 + e > r ? 1.f : L * d[e];
            }
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] = j0 + e > r ? 0.f : y[e];
        });
      }
      ok = pre::mbar_wait(&t.bar, (round - 1) & 1, &t.gave_up);
      pre::fence_after_sync();
#pragma unroll
      for (int e = 0; e < 32; e += 16) {                       // the decays up to each token, on the state's products
        float y[16];
        uint32_t u[16];
        tmem_sum<16>(sums + e, 0.f, y);
#pragma unroll
        for (int r = 0; r < 16; r += 4) {
          const float4 f = ld4(D.upto + half * 32 + e + r);
          u[r] = __float_as_uint(y[r] * f.x); u[r + 1] = __float_as_uint(y[r + 1] * f.y);
          u[r + 2] = __float_as_uint(y[r + 2] * f.z); u[r + 3] = __float_as_uint(y[r + 3] * f.w);
        }
        pre::tmem_st16_nowait(sums + e, u);
      }
      {
        uint32_t w[3][16];
        a.split_values(w, half * 32, &bad[i & 1][x]);
        put_lanes(t.base, warp, w);
      }
      if (i + 1 < count) load_a(i + 1, 0);
      ok = tensor_issue_heads(t, tid, tile + SLICES * 3 * TILE, ok, two_heads);
      ++round;
      const int i0 = half * 32;
      float raw[16];
      const float* from = values(i) + i0 * p.v_stride;
      auto load_raw = [&](int first_token) {
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          raw[e] = live(i) && first_token + e < c.n ? *from : 0.f;
          from += p.v_stride;
          asm volatile("" : "+l"(from));                       // (16 addresses at a time would not fit in registers)
        }
      };
      if (p.skip) load_raw(i0);
      ok = ok && pre::mbar_wait(&t.bar, (round - 1) & 1, &t.gave_up);
      pre::fence_after_sync();
      if (__all_sync(0xffffffffu, ok) && live(i) && i0 < c.n) {      // (a warp's columns are of one half)
        const int wrong = bad[i & 1][x];
        bool again = wrong < C;
        float* out = p.out + (size_t)(c.tok + i0) * p.out_stride + (size_t)unit * columns + column(i);
        float* to = out;
#pragma unroll
        for (int q = 0; q < 32; q += 16) {
          float y[16];
          again |= tmem_sum<16>(sums + q, OUT_LOST, y);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            if (i0 + q + e < c.n) *to = p.skip ? fmaf(skip, raw[e], y[e]) : y[e];
            to += p.out_stride;
            asm volatile("" : "+l"(to));
          }
          if (q == 0 && p.skip) load_raw(i0 + 16);
        }
#pragma unroll 1
        for (int r = i0; again && r < min(i0 + 32, c.n); ++r) {      // (sums of numbers without terms)
          float* at = out + (r - i0) * p.out_stride;
          if (r < wrong && *at == *at) continue;
          const float* query = p.q + (size_t)(c.tok + r) * p.q_stride + (size_t)unit * N;
          const float* states = p.U + item(h) * N * (size_t)Dv + column(i) % Dv;
          float o = 0.f;
          for (int n = 0; n < N; ++n) o = fmaf(query[n] * p.q_scale, states[(size_t)n * Dv], o);
          o *= D.upto[r];
          for (int j = 0; j <= r; ++j) {
            float f = D.dt[j];
            for (int s = j + 1; s <= r; ++s) f *= D.a[s];
            o = fmaf(AT[r * C + j] * f, values(i)[j * p.v_stride], o);
          }
          if (p.skip) o = fmaf(skip, values(i)[r * p.v_stride], o);
          *at = o;
        }
      }
      ok = __syncthreads_and(ok) != 0;                         // (one decision; everybody has read what the next tiles' values may change)
      if (half == 0) bad[i & 1][x] = C;
    }
    copy_wait<0>();
    ok = __syncthreads_and(ok) != 0;
  }
  tensor_end(t, tid, ok, p.error_flag);
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

// A block's tiles: as many as leave two blocks an SM, up to eight.
static int tiles_of_block(const Params& p, int units, int tiles) {
  int n = 1;
  while (n < MOST_TILES && n < tiles && (long)p.seg_chunks * units * ((tiles + n - 1) / n) > 2 * sm_count()) n *= 2;
  return n;
}
#define CPI_TILES_LAUNCH(kernel, units, tiles, bytes)                                                       \
  do {                                                                                                      \
    static bool done = false;                                                                               \
    if (allow(kernel, bytes, done)) return 1;                                                               \
    const int n = tiles_of_block(p, units, tiles);                                                          \
    cpi::launch_pdl(kernel, dim3(p.seg_chunks, units, ((tiles) + n - 1) / n), dim3(TC_THREADS), bytes, stream, p, n); \
    return check_launch("linear_chunks");                                                                   \
  } while (0)
template <int N, bool STEP>
static int state_products(const Params& p, cudaStream_t stream) {
  const int units = STEP ? p.H / p.hpg : p.H;
  CPI_TILES_LAUNCH((chunk_state_kernel<N, STEP>), units, p.H / units * (p.Dv / 64), STATE_BYTES<N>);
}
// column tiles of 128 where they come out even, else of 64
template <int N, bool DELTA>
static int output_products(const Params& p, cudaStream_t stream) {
  if (p.Dv % 128 == 0) CPI_TILES_LAUNCH((chunk_out_kernel<N, 128, DELTA>), p.H, p.Dv / 128, OUT_BYTES<N>);
  else CPI_TILES_LAUNCH((chunk_out_kernel<N, 64, DELTA>), p.H, p.Dv / 64, OUT_BYTES<N>);
}
template <int N>
static int output_products_step(const Params& p, cudaStream_t stream) {
  CPI_TILES_LAUNCH(chunk_out_step_kernel<N>, p.H / p.hpg, (p.hpg * p.Dv + 127) / 128, STEP_OUT_BYTES<N>);
}

template <int N>
static int run(const Params& p, cudaStream_t stream) {
  const dim3 items(p.seg_chunks, p.H);
  const dim3 chain(p.n_seqs, p.H, (N * p.Dv / 4 + 255) / 256);
  if (p.dt) {
    CPI_CHUNK_LAUNCH(prepare_step_kernel<N>, dim3(p.seg_chunks, p.H / p.hpg), 256, 2 * C * (N + 4) * sizeof(float));
    if (int rc = state_products<N, true>(p, stream)) return rc;
    CPI_CHUNK_LAUNCH(chain_kernel<true>, chain, 256, (size_t)0);
    if (int rc = output_products_step<N>(p, stream)) return rc;
  } else if (p.beta) {
    CPI_CHUNK_LAUNCH((prepare_rows_kernel<N / 8, true>), items, 512, (PrepShape<N / 8, true>::bytes));
    CPI_CHUNK_LAUNCH(solve_kernel, dim3(p.seg_chunks, p.H, (N + p.Dv + 127) / 128), 128, C * 128 * sizeof(float));
    CPI_CHUNK_LAUNCH(delta_chain_kernel<N>, dim3(p.n_seqs, p.H, p.Dv / 16), 256, ChainShape<N>::bytes);
    if (int rc = output_products<N, true>(p, stream)) return rc;
  } else {
    CPI_CHUNK_LAUNCH((prepare_rows_kernel<N / 8, false>), items, 512, (PrepShape<N / 8, false>::bytes));
    if (int rc = state_products<N, false>(p, stream)) return rc;
    CPI_CHUNK_LAUNCH(chain_kernel<false>, chain, 256, (size_t)0);
    if (int rc = output_products<N, false>(p, stream)) return rc;
  }
  return 0;
}

// floats of scratch per chunk: {U, KT, QT, AT, DC, MT, KP, WT, UH} one after another
static void sizes(int kind, int H, int groups, int N, int Dv, long (&n)[9]) {
  const long rows = (long)H * N * C, tri = (long)H * C * C;
  n[0] = (long)H * N * Dv;
  n[1] = kind == 0 ? 0 : rows;
  n[2] = kind == 0 ? 0 : rows;
  n[3] = kind == 0 ? (long)groups * C * C : tri;
  n[4] = kind == 0 ? (H + 3) / 4 * 4 : (long)H * N;
  n[5] = kind == 2 ? tri : kind == 0 ? (long)H * DECAYS : 0;     // (the step flavour's decays)
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
                                 int* error_flag, cudaStream_t stream) {
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
  p.error_flag = error_flag;
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
