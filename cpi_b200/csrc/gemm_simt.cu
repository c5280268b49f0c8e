// General matrix product on the FP32 pipe (FFMA): out[m, n] = sum_k A[row(m), k] * W[g(m)][n, k].
//
// This is the true 32-bit contraction of the library: float accumulation in a fixed k order
// (no tensor cores, no tf32), for any mix of float32 / bfloat16 activations and weights (bfloat16
// widens exactly, as src/engine/llama4_cpu_engine.cpp:24-29 does).  The bfloat16 path uses it for
// shapes that the tensor-core kernels refuse.  The reference's counterparts are its GEMV kernels
// (src/kernels/kernels_ops_matvec.cu:343-418) and one cublasGemmEx call
// (src/engine/llama4_cuda_engine_setup.cu:579-605), all batch 1.
//
// Modes:  STORE   out = acc * scale(m)
//         ADD     out += acc * scale(m)                      (out is the float32 residual stream)
//         SWIGLU  out = silu(g) * u,  g = scale(m) * sum_k A W[n, k],  u = scale(m) * sum_k A W[N + n, k]
// Optional row gather (a_rows), output row scatter (out_rows), per-row scale, and groups: logical
// rows [offsets[g], offsets[g+1]) use the weight matrix W + g * w_group_stride (routed experts).
#include "common.cuh"

namespace cpi {

enum GemmMode : int { kStore = 0, kAdd = 1, kSwiglu = 2 };

struct GemmParams {
  const void* a; long lda; const int* a_rows;
  const void* w; long ldw; long w_group_stride;
  void* out; long ldo; const int* out_rows;
  const float* row_scale;
  const int* group_offsets; int n_groups;
  int M, N, K;
  int gate_act;      // gated mode: the gate's activation (0 silu, 1 gelu in its tanh form, 2 the clamped form below)
  int vec_a, vec_w, vec_o;      // every row starts on 16 bytes (on 8 for bfloat16)
  float gate_limit;  // act 2: g' = min(g, limit), u' = clamp(u, -limit, limit), out = g' sigmoid(1.702 g') (u' + 1)
};

constexpr int BN = 64, BK = 16, NT = 256;

// One output: v is the (gate's) sum, u the up projection's in the gated mode, both scaled.
template <int MODE, typename TO>
__device__ __forceinline__ void put(const GemmParams& p, TO* o, float v, float u) {
  if (MODE == kSwiglu) {
    if (p.gate_act == 2) {
      v = fminf(v, p.gate_limit);
      u = fminf(fmaxf(u, -p.gate_limit), p.gate_limit) + 1.0f;
      v = v / (1.0f + expf(-1.702f * v)) * u;
    } else {
      v = (p.gate_act ? 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)))
                      : v / (1.0f + expf(-v))) * u;
    }
  } else if (MODE == kAdd) {
    v = to_f32(*o) + v;
  } else {
    if (p.gate_act == 3) { v = fmaxf(v, 0.f); v *= v; }      // the storing mode with a squared relu
    if (p.gate_act == 4) v = 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));   // ... a gelu
  }
  *o = from_f32<TO>(v);
}

template <typename TA, typename TW, typename TO, int MODE>
__global__ void __launch_bounds__(NT) gemm_simt_kernel(GemmParams p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int BM = 16;
  constexpr bool GLU = MODE == kSwiglu;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[GLU ? 2 : 1][BK][BN + 4];

  int m_begin = 0, m_end = p.M;
  const TW* w = reinterpret_cast<const TW*>(p.w);
  int tile_m = blockIdx.y;
  if (p.group_offsets) {
    // map blockIdx.y to (group, tile in group): groups are visited in order
    int g = 0, found = 0;
    for (; g < p.n_groups; ++g) {
      const int b = p.group_offsets[g], e = p.group_offsets[g + 1];
      const int tiles = (e - b + BM - 1) / BM;
      if (tile_m < tiles) { m_begin = b; m_end = e; found = 1; break; }
      tile_m -= tiles;
    }
    if (!found) return;
    w += (size_t)g * p.w_group_stride;
  }
  const int m0 = m_begin + tile_m * BM;
  if (m0 >= m_end) return;
  const int n0 = blockIdx.x * BN;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;

  float acc[4], acc2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j] = acc2[j] = 0.f;

  const TA* a = reinterpret_cast<const TA*>(p.a);
  // loader mapping: A tile BM x BK, 4 consecutive k per thread
  const int la_row = tid >> 2, la_k = (tid & 3) * 4;        // valid for tid < BM*4
  const bool la_active = la_row < BM && (m0 + la_row) < m_end;
  const TA* a_ptr = nullptr;
  if (la_active) {
    const int lr = m0 + la_row;
    a_ptr = a + (size_t)(p.a_rows ? p.a_rows[lr] : lr) * p.lda;
  }
  const int lw_row = tid >> 2, lw_k = (tid & 3) * 4;          // W tile BN x BK: 64 rows x 4 threads
  const bool lw_active = (n0 + lw_row) < p.N;
  const TW* w_ptr = w + (size_t)(n0 + lw_row) * p.ldw;
  const TW* w2_ptr = w + (size_t)(p.N + n0 + lw_row) * p.ldw;

  for (int k0 = 0; k0 < p.K; k0 += BK) {
    if (la_row < BM) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = k0 + la_k + j;
        As[la_k + j][la_row] = (la_active && k < p.K) ? to_f32(a_ptr[k]) : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lw_k + j;
      const bool ok = lw_active && k < p.K;
      Ws[0][lw_k + j][lw_row] = ok ? to_f32(w_ptr[k]) : 0.f;
      if (GLU) Ws[1][lw_k + j][lw_row] = ok ? to_f32(w2_ptr[k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float av = As[k][ty];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[j] = fmaf(av, Ws[0][k][tx * 4 + j], acc[j]);
        if (GLU) acc2[j] = fmaf(av, Ws[1][k][tx * 4 + j], acc2[j]);
      }
    }
    __syncthreads();
  }

  TO* out = reinterpret_cast<TO*>(p.out);
  const int lr = m0 + ty;
  if (lr >= m_end) return;
  const float s = p.row_scale ? p.row_scale[lr] : 1.0f;
  TO* o = out + (size_t)(p.out_rows ? p.out_rows[lr] : lr) * p.ldo;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + tx * 4 + j;
    if (n < p.N) put<MODE>(p, o + n, acc[j] * s, GLU ? acc2[j] * s : 0.f);
  }
}

// ---- many rows per group -------------------------------------------------------------------------------------------
// The same sums in the same order (an output is one chain of fused multiply-adds over k, so its bits do not depend on
// which of the two kernels made it), from register tiles of RT x 8 with the packed float32 instructions.  A CTA takes 64 rows
// and COLS weight rows (in the gated mode half of them are gate rows, half up rows): a thread has RT rows and four columns in
// either half, so that the eight distinct addresses of a warp's weight loads and the four of its activation loads each take
// two cycles of the shared-memory pipe (32 distinct ones take eight).  DEPTH sixteens of k are on the way through registers
// while 16 are multiplied, and a step's operands are read from shared memory one step ahead.  The k 8 to 15 of a sixteen lie
// with their rows' eights exchanged: without it a warp's writes of four k at a time meet two and two in the same banks.
// Bound: the issue of packed multiply-adds and of the moves that double an activation for them (3.0 cycles a multiply-add where
// the pipe takes 2), and whole CTAs an SM; 509 x 2,048 -> 3,072 and 2,048 in float32: 335 -> 298 us together (floor 148), 2,048 x
// 2,048 -> 6,144 1,092 -> 1,007 (716), 17 x 2,048 -> 2,048 108 -> 77.
// Four neighbouring elements of a row as they lie in memory; they are widened on their way to shared memory, so that nothing
// waits for a load while the 16 k before are multiplied.  64 rows, 2,048 x 2,048: bfloat16 weights widened at the load 205 us,
// here 107 (float32 weights 117); with 4 x 4 outputs a thread and 64 rows a tile it was 169 (177).
template <typename T> struct Four;
template <> struct Four<float> {
  float v[4];
  __device__ __forceinline__ void clear() { v[0] = v[1] = v[2] = v[3] = 0.f; }
  __device__ __forceinline__ void whole(const float* p) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
  __device__ __forceinline__ void some(const float* p, int k, int K) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = k + j < K ? p[k + j] : 0.f;
  }
  __device__ __forceinline__ float at(int e) const { return v[e]; }
};
template <> struct Four<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void clear() { v = make_uint2(0u, 0u); }
  __device__ __forceinline__ void whole(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void some(const __nv_bfloat16* p, int k, int K) {
    const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
    uint32_t x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = k + j < K ? u[k + j] : 0u;
    v = make_uint2(x[0] | x[1] << 16, x[2] | x[3] << 16);
  }
  __device__ __forceinline__ float at(int e) const {                 // (a bfloat16 is the upper half of its float32)
    const uint32_t w = e < 2 ? v.x : v.y;
    return __uint_as_float(e & 1 ? w & 0xffff0000u : w << 16);
  }
};
template <typename T>
__device__ __forceinline__ void load4(const T* p, bool live, bool vec, int k, int K, Four<T>& v) {
  if (!live) v.clear();
  else if (vec && k + 4 <= K) v.whole(p + k);
  else v.some(p, k, K);
}

constexpr int TILE_ROWS = 64;
constexpr int tile_threads(int RT, int COLS) { return TILE_ROWS / (4 * RT) * (COLS / 64) * 32; }

template <typename TA, typename TW, typename TO, int MODE, int RT, int COLS, int DEPTH, bool SHORT>
__global__ void __launch_bounds__(tile_threads(RT, COLS)) gemm_simt_tile_kernel(GemmParams p) {
  constexpr bool GLU = MODE == kSwiglu;
  constexpr int TILE_THREADS = tile_threads(RT, COLS);
  constexpr int HALF = COLS / 2, OUT = GLU ? HALF : COLS;                      // halves of the weight rows, output columns
  constexpr int LDM = TILE_ROWS + 4, LDC = COLS + 4, LA = TILE_ROWS * BK / 4 / TILE_THREADS, LW = COLS * BK / 4 / TILE_THREADS;
  __shared__ __align__(16) float As[2][BK][LDM], Ws[2][BK][LDC];
  pdl_wait();
  int m_begin = 0, m_end = p.M;
  const TW* w = reinterpret_cast<const TW*>(p.w);
  int tile_m = blockIdx.y;
  if (p.group_offsets) {
    int g = 0, found = 0;
    for (; g < p.n_groups; ++g) {
      const int b = p.group_offsets[g], e = p.group_offsets[g + 1];
      const int tiles = (e - b + TILE_ROWS - 1) / TILE_ROWS;
      if (tile_m < tiles) { m_begin = b; m_end = e; found = 1; break; }
      tile_m -= tiles;
    }
    if (!found) return;
    w += (size_t)g * p.w_group_stride;
  }
  const int m0 = m_begin + tile_m * TILE_ROWS;
  if (m0 >= m_end) return;
  const int n0 = blockIdx.x * OUT, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int WARPS_M = TILE_ROWS / (4 * RT);
  const int r0 = (warp % WARPS_M) * (4 * RT) + (lane >> 3) * RT, x0 = (warp / WARPS_M) * 32 + (lane & 7) * 4;

  // loaders: piece e of a tile is row e / 4, k's 4 (e % 4) ..
  const TA* a = reinterpret_cast<const TA*>(p.a);
  const TA* a_ptr[LA];
  bool a_live[LA];
#pragma unroll
  for (int i = 0; i < LA; ++i) {
    const int lr = m0 + (tid + i * TILE_THREADS) / 4;
    a_live[i] = lr < m_end;
    a_ptr[i] = a + (size_t)(a_live[i] ? (p.a_rows ? p.a_rows[lr] : lr) : 0) * p.lda;
  }
  const TW* w_ptr[LW];
  bool w_live[LW];
#pragma unroll
  for (int i = 0; i < LW; ++i) {
    const int c = (tid + i * TILE_THREADS) / 4;              // weight row of the tile: its output column, and which matrix
    const int n = GLU ? n0 + c % HALF : n0 + c;
    w_live[i] = n < p.N;
    w_ptr[i] = w + (size_t)(w_live[i] ? (GLU && c >= HALF ? p.N + n : n) : 0) * p.ldw;
  }
  const int kq = (tid & 3) * 4;
  const bool va = p.vec_a, vw = p.vec_w;
  struct Set { Four<TA> a[LA]; Four<TW> w[LW]; };
  auto fetch = [&](int k0, Set& r) {
#pragma unroll
    for (int i = 0; i < LA; ++i) load4(a_ptr[i], a_live[i], va, k0 + kq, p.K, r.a[i]);
#pragma unroll
    for (int i = 0; i < LW; ++i) load4(w_ptr[i], w_live[i], vw, k0 + kq, p.K, r.w[i]);
  };
  auto stash = [&](int b, const Set& r) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
      for (int i = 0; i < LA; ++i) As[b][kq + e][(tid + i * TILE_THREADS) / 4 ^ (kq & 8)] = r.a[i].at(e);
#pragma unroll
      for (int i = 0; i < LW; ++i) Ws[b][kq + e][(tid + i * TILE_THREADS) / 4 ^ (kq & 8)] = r.w[i].at(e);
    }
  };
  float2 acc[RT][4];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[r][x] = make_float2(0.f, 0.f);
  // DEPTH sixteens of k on the way: slot i % DEPTH of the registers, buffer i % 2 of shared memory
  // (SHORT: see launch_simt)
  static_assert(!SHORT || DEPTH == 1, "a loop of one step has one set of registers");
  constexpr int UNROLL = SHORT ? 1 : DEPTH % 2 ? 2 * DEPTH : DEPTH;
  Set ring[DEPTH];
#pragma unroll
  for (int d = 0; d < DEPTH; ++d) fetch(d * BK, ring[d]);
  stash(0, ring[0]);
  __syncthreads();
  auto step = [&](int k0, int b, Set& next, Set& free) {
    if (k0 + DEPTH * BK < p.K) fetch(k0 + DEPTH * BK, free);
    // the operands of a step of k, one step ahead of its products
    float av[2][RT], wv[2][8];
    auto read = [&](int k, int to) {
#pragma unroll
      for (int r = 0; r < RT; r += 4) *reinterpret_cast<float4*>(av[to] + r) = *reinterpret_cast<const float4*>(&As[b][k][(r0 ^ (k & 8)) + r]);
      *reinterpret_cast<float4*>(wv[to]) = *reinterpret_cast<const float4*>(&Ws[b][k][x0 ^ (k & 8)]);
      *reinterpret_cast<float4*>(wv[to] + 4) = *reinterpret_cast<const float4*>(&Ws[b][k][HALF + (x0 ^ (k & 8))]);
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      if (k + 1 < BK) read(k + 1, (k + 1) & 1);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float2 ar = make_float2(av[k & 1][r], av[k & 1][r]);
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[r][x] = __ffma2_rn(ar, make_float2(wv[k & 1][2 * x], wv[k & 1][2 * x + 1]), acc[r][x]);
      }
    }
    if (k0 + BK < p.K) stash(b ^ 1, next);
    __syncthreads();
  };
  for (int k0 = 0; k0 < p.K; k0 += UNROLL * BK)
#pragma unroll
    for (int i = 0; i < UNROLL; ++i)
      if (k0 + i * BK < p.K) step(k0 + i * BK, SHORT ? (k0 / BK) & 1 : i & 1, ring[(i + 1) % DEPTH], ring[i % DEPTH]);
  // (not earlier: blocks of the next kernel that wait beside the running ones slow them down, 343 us became 699 when the two
  // products of the figure above took 343)
  pdl_launch_dependents();

  TO* out = reinterpret_cast<TO*>(p.out);
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int lr = m0 + r0 + r;
    if (lr >= m_end) continue;
    const float s = p.row_scale ? p.row_scale[lr] : 1.0f;
    TO* o = out + (size_t)(p.out_rows ? p.out_rows[lr] : lr) * p.ldo;
    const float v[8] = {acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y, acc[r][2].x, acc[r][2].y, acc[r][3].x, acc[r][3].y};
#pragma unroll
    for (int h = 0; h < (GLU ? 1 : 2); ++h) {
      const int n = n0 + h * HALF + x0;
      if constexpr (MODE != kSwiglu && sizeof(TO) == 4) {
        if (p.vec_o && n + 4 <= p.N && p.gate_act == 0) {
          float4 y = make_float4(v[4 * h] * s, v[4 * h + 1] * s, v[4 * h + 2] * s, v[4 * h + 3] * s);
          float4* dst = reinterpret_cast<float4*>(o + n);
          if (MODE == kAdd) { const float4 z = *dst; y = make_float4(z.x + y.x, z.y + y.y, z.z + y.z, z.w + y.w); }
          *dst = y;
          continue;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < p.N) put<MODE>(p, o + n + j, v[4 * h + j] * s, GLU ? v[4 + j] * s : 0.f);
    }
  }
}

template <typename TA, typename TW, typename TO, int MODE>
int launch_simt(const GemmParams& p, int m_tiles_hint, cudaStream_t stream) {
  // 16 rows per tile when few rows are expected per group, else the register tiles of 64 (17 rows already, 2,048 x 2,048: 114 us,
  // with 4 x 4 outputs a thread and 64 rows a tile 176; bfloat16 weights 104, 162; 17 rows in each of 16 experts of
  // 2 x 2,048 x 2,048 471, 651)
  if (m_tiles_hint <= 16) {
    const int m_tiles = (p.M + 15) / 16 + (p.group_offsets ? p.n_groups : 0);
    const dim3 grid((p.N + BN - 1) / BN, m_tiles);
    if (grid.y > 65535) { set_error("gemm: too many row tiles (%u)", grid.y); return 1; }
    cpi::launch_pdl(gemm_simt_kernel<TA, TW, TO, MODE>, grid, NT, 0, stream, p);
    return check_launch("gemm_simt");
  }
  const int m_tiles = (p.M + TILE_ROWS - 1) / TILE_ROWS + (p.group_offsets ? p.n_groups : 0);
  if (m_tiles > 65535) { set_error("gemm: too many row tiles (%d)", m_tiles); return 1; }
  constexpr int per = MODE == kSwiglu ? 2 : 1;
  auto go = [&](auto kernel, int cols, int threads) { cpi::launch_pdl(kernel, dim3((per * p.N + cols - 1) / cols, m_tiles), threads, 0, stream, p); };
  // Two tiles: 128 weight rows a CTA with 8 x 8 outputs a thread, 64 with 4 x 8.  The wide one needs CTAs enough for the SMs and,
  // up to two and a half an SM, a sum long enough for its longer begin and end; with bfloat16 weights it gains less.  Wide /
  // narrow in us, wide CTAs an SM: float32 weights, K = 2,048, 0.9 167 / 123, 1.3 209 / 175, 1.7 212 / 234, 2.2 294 / 297, 2.6 289 / 345,
  // K = 128, 1.7 16.5 / 16.7, K = 96, 1.7 12.8 / 12.9; bfloat16 weights, K = 2,048, 1.7 239 / 232, 2.2 313 / 352, K = 4,096, 1.7 440 / 460.
  // Sums over soon, and the wide tile's with bfloat16 weights, take the loop of one step, the first since its code is there sooner:
  // wide, one step / two, 10 an SM, K = 64 39.6 / 42.9, K = 128 71.7 / 70.7; bfloat16 38.5 / 44.3, 70.5 / 76.6, K = 4,096, 2.6 an SM 598 / 622.
  // The narrow tile has two sixteens of k on the way (one / two: 509 x 16 -> 64 2.9 / 2.6, 2,048 ->
  // 3,072 187 / 175); bfloat16 weights one, which widening four at a time leaves no room to do better (K = 256, 1.3 an SM 24.4, two
  // 29.1, three 26.4), or three where the sum is long (K = 2,048 179, 199, 174; half an SM's CTA, K = 256 15.4, 16.6, 14.7).
  const long sms = sm_count(), ctas = (long)m_tiles * ((per * p.N + 127) / 128);
  constexpr bool f32 = sizeof(TW) == 4;
  if (2 * ctas >= 5 * sms || (p.K >= 128 && 2 * ctas >= (f32 || p.K >= 4096 ? 3 : 4) * sms)) {
    if (p.K <= 64) go(gemm_simt_tile_kernel<TA, TW, TO, MODE, 8, 128, 1, true>, 128, tile_threads(8, 128));
    else go(gemm_simt_tile_kernel<TA, TW, TO, MODE, 8, 128, 1, !f32>, 128, tile_threads(8, 128));
  } else if constexpr (f32) {
    go(gemm_simt_tile_kernel<TA, TW, TO, MODE, 4, 64, 2, false>, 64, tile_threads(4, 64));
  } else {
    if (p.K <= 64) go(gemm_simt_tile_kernel<TA, TW, TO, MODE, 4, 64, 1, true>, 64, tile_threads(4, 64));
    else if (p.K <= (2 * ctas <= sms ? 192 : 384)) go(gemm_simt_tile_kernel<TA, TW, TO, MODE, 4, 64, 1, false>, 64, tile_threads(4, 64));
    else go(gemm_simt_tile_kernel<TA, TW, TO, MODE, 4, 64, 3, false>, 64, tile_threads(4, 64));
  }
  return check_launch("gemm_simt");
}

template <typename TA, typename TW, typename TO>
int launch_mode(const GemmParams& p, int mode, int hint, cudaStream_t s) {
  switch (mode) {
    case kStore:  return launch_simt<TA, TW, TO, kStore>(p, hint, s);
    case kAdd:    return launch_simt<TA, TW, TO, kAdd>(p, hint, s);
    case kSwiglu: return launch_simt<TA, TW, TO, kSwiglu>(p, hint, s);
  }
  set_error("gemm: unknown mode %d", mode);
  return 1;
}

}  // namespace cpi

using namespace cpi;

// a [*, K] (lda), w [N or 2N (SWIGLU), K] (ldw) per group, out [*, N] (ldo).
// M = number of logical rows (over all groups); rows_per_group_hint sizes the row tile.
extern "C" int cpi_gemm_simt(const void* a, int a_dtype, long lda, const int* a_rows,
                             const void* w, int w_dtype, long ldw, long w_group_stride,
                             void* out, int out_dtype, long ldo, const int* out_rows,
                             const float* row_scale, const int* group_offsets, int n_groups,
                             int M, int N, int K, int mode, int rows_per_group_hint, float gate_limit,
                             cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  // modes 3, 4: the gated mode with a gelu / a clamped gate; modes 5, 6: the storing mode with a squared relu / a gelu
  const int gate_act = mode == 3 ? 1 : mode == 4 ? 2 : mode == 5 ? 3 : mode == 6 ? 4 : 0;
  if (mode == 3 || mode == 4) mode = 2;
  if (mode == 5 || mode == 6) mode = 0;
  CPI_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  CPI_REQUIRE(mode != kAdd || out_dtype == kF32, "gemm: ADD mode needs a float32 output");
  auto vec = [](const void* x, int dtype, long ld) {
    return (reinterpret_cast<uintptr_t>(x) & (dtype == kF32 ? 15 : 7)) == 0 && ld % 4 == 0 ? 1 : 0;
  };
  GemmParams p{a, lda, a_rows, w, ldw, w_group_stride, out, ldo, out_rows, row_scale, group_offsets, n_groups, M, N, K, gate_act,
               vec(a, a_dtype, lda), vec(w, w_dtype, ldw) && w_group_stride % 4 == 0, vec(out, out_dtype, ldo), gate_limit};
  CPI_DISPATCH_DTYPE(a_dtype, TA, CPI_DISPATCH_DTYPE(w_dtype, TW, CPI_DISPATCH_DTYPE(out_dtype, TO,
      return (launch_mode<TA, TW, TO>(p, mode, rows_per_group_hint, stream)))));
  return 0;
}
