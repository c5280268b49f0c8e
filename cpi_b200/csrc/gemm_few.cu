// bfloat16 matrix product for a handful of tokens:  out[t, n] = sum_k X[t, k] * W[n, k]  with up to 32 tokens.
//
// Such a product is one pass over the weights.  8 MB at the copy bandwidth take 1.3 us, less than a kernel with a pipeline
// needs to begin and to end (tensor memory, barriers, a ring of TMA stages, a cluster's merge of split sums: gemm_tc.cu,
// 4.9 us).  Here a warp loads its weights straight into the registers that `mma.sync` takes them from: a lane's 16 bytes of
// a row are eight neighbouring k, which two instructions use as the k slots (2t, 2t + 1) and (2t + 8, 2t + 9) of theirs; the
// activations are loaded the same way, so every factor meets its partner and only the order of k differs from memory's.
// A block owns 16 features (gated: 16 pairs); its warps share K in contiguous parts, summed in warp order.  A warp's first
// weights are asked for before the wait on the preceding kernel (no kernel writes weights), and nothing here is held that a
// successor waits for, so a decode step's next product has its weights on the way while this one ends.
//
// What bounds it is bytes in flight: D steps of 32 k a warp, and up to a block an SM, or up to three or four of the smaller forms,
// resident at once (see plan(); with more the launch takes rounds).
// Measured on a chain of products over different weights, one token, gemm_tc.cu / here / floor in us: 2,048 x 2,048 4.9 / 2.4 /
// 1.3, 2,048 x 8,192 (N x K) 10.4 / 6.6 / 5.1, 3,072 x 2,048 6.2 / 2.9 / 1.9, 5,120 x 5,120 12.3 / 9.4 / 8.0, 8,192 pairs x 2,048
// 14.3 / 11.1 / 10.2, 32,000 x 2,048 23.4 / 21.5 / 20.0; 16 tokens: 2,048 x 2,048 5.7 / 3.1, 5,120 x 5,120 13.1 / 12.3.
//
// Groups of equally many rows (the heads of latent attention: 16 of 8 rows, 512 x 128 and 128 x 512, 6.1 -> 2.0 us each) have their
// weights side by side.
//
// Epilogues as in gemm_tc.cu: STORE (with its activations), ADD (float32 residual, one writer per element), gated pairs.
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "mma_frag.cuh"

namespace cpi {
namespace few {

struct Params {
  const __nv_bfloat16* x; long ldx;
  const __nv_bfloat16* w;
  void* out; long ldo;
  const int* out_rows;           // where row r of all groups' goes; null: to r
  int T, N, K;                   // T tokens a group: blockIdx.y takes rows from T blockIdx.y on and weights of its own
  int gate_act; float gate_limit;
};

__device__ __forceinline__ uint4 load_weights(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// NB: octets of tokens.  A step is 32 k; D steps of weights and DX of activations are in flight per warp.
template <int MODE, typename TO, int NB, int WARPS, int D, int DX, int PER_SM>
__global__ void __launch_bounds__(WARPS * 32, PER_SM) gemm_few_kernel(Params p) {
  static_assert(D % DX == 0, "the activations' ring turns with the weights'");
  constexpr int ACC = MODE == epi::kSwiglu ? 2 : 1;
  constexpr int CH = WARPS < 8 && ACC * NB < 4 ? 2 : 1;   // a warp's long share is summed in two chains (registers allow it)
  __shared__ float part[WARPS][ACC][NB * 8][17];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16, row0 = blockIdx.y * p.T;
  const __nv_bfloat16 *px = p.x + (size_t)row0 * p.ldx, *pw = p.w + (size_t)blockIdx.y * ACC * p.N * p.K;
  const int steps = (p.K + 31) / 32, per = (steps + WARPS - 1) / WARPS;
  const int s0 = warp * per, s1 = min(steps, s0 + per);
  // rows past the last feature repeat it; their sums are not stored
  const __nv_bfloat16* w[ACC][2];
#pragma unroll
  for (int a = 0; a < ACC; ++a)
#pragma unroll
    for (int h = 0; h < 2; ++h) w[a][h] = pw + (size_t)(a * p.N + min(n0 + g + 8 * h, p.N - 1)) * p.K + 8 * t;
  const __nv_bfloat16* x[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) x[b] = px + (size_t)(b * 8 + g) * p.ldx + 8 * t;

  uint4 wr[D][ACC][2], xr[DX][NB];
  float acc[CH][ACC][NB][4];
#pragma unroll
  for (int c = 0; c < CH; ++c)
#pragma unroll
    for (int a = 0; a < ACC; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[c][a][b][e] = 0.f;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  auto in = [&](int s) { return s < s1 && s * 32 + 8 * t < p.K; };
  auto ask_w = [&](int d, int s) {
#pragma unroll
    for (int a = 0; a < ACC; ++a)
#pragma unroll
      for (int h = 0; h < 2; ++h) wr[d][a][h] = in(s) ? load_weights(w[a][h] + (size_t)s * 32) : zero;
  };
  auto ask_x = [&](int d, int s) {
#pragma unroll
    for (int b = 0; b < NB; ++b) xr[d][b] = in(s) && b * 8 + g < p.T ? *reinterpret_cast<const uint4*>(x[b] + (size_t)s * 32) : zero;
  };
#pragma unroll
  for (int d = 0; d < D; ++d) ask_w(d, s0 + d);
  pdl_launch_dependents();
  pdl_wait();
#pragma unroll
  for (int d = 0; d < DX; ++d) ask_x(d, s0 + d);
  // the residual's old values, while the weights are on the way: thread tid adds to feature tid % 16 of token tid / 16
  constexpr int OUT = NB * 8 * 16, PER = (OUT + WARPS * 32 - 1) / (WARPS * 32);
  float old[PER];
  TO *out = reinterpret_cast<TO*>(p.out), *at[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = tid + i * WARPS * 32, tok = e / 16, n = n0 + e % 16;
    const bool live = e < OUT && tok < p.T && n < p.N;
    at[i] = !live ? nullptr : out + (size_t)(p.out_rows ? p.out_rows[row0 + tok] : row0 + tok) * p.ldo + n;
    old[i] = MODE == epi::kAdd && live ? to_f32(*at[i]) : 0.f;
  }
  for (int s = s0; s < s1; s += D) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
      for (int a = 0; a < ACC; ++a) {
        const uint4 lo = wr[d][a][0], hi = wr[d][a][1];
        const uint32_t f0[4] = {lo.x, hi.x, lo.y, hi.y}, f1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          frag::mma_bf16(acc[0][a][b], f0, xr[d % DX][b].x, xr[d % DX][b].y);
          frag::mma_bf16(acc[CH - 1][a][b], f1, xr[d % DX][b].z, xr[d % DX][b].w);
        }
      }
      ask_w(d, s + D + d);
      ask_x(d % DX, s + d + DX);
    }
  }
#pragma unroll
  for (int a = 0; a < ACC; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[warp][a][b * 8 + 2 * t + (e & 1)][g + 8 * (e >> 1)] = CH == 2 ? acc[0][a][b][e] + acc[CH - 1][a][b][e] : acc[0][a][b][e];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = tid + i * WARPS * 32, tok = e / 16, f = e % 16;
    if (at[i] == nullptr) continue;
    float v = part[0][0][tok][f], u = ACC == 2 ? part[0][ACC - 1][tok][f] : 0.f;
#pragma unroll
    for (int q = 1; q < WARPS; ++q) {
      v += part[q][0][tok][f];
      if (ACC == 2) u += part[q][ACC - 1][tok][f];
    }
    if (MODE == epi::kSwiglu) v = epi::gate_mul(v, u, p.gate_act, p.gate_limit);
    else if (MODE == epi::kAdd) v = old[i] + v;
    else v = epi::store_act(v, p.gate_act);
    *at[i] = from_f32<TO>(v);
  }
}

// The forms: blocks that share an SM.  One of 16 warps, two of eight with eight steps in flight, three of eight with four, four
// of four with eight.
enum Form : int { kNone = 0, kOne = 1, kTwo = 2, kThree = 3, kFour = 4 };

// The form for a product, or kNone where the tensor-memory kernel is faster.  A launch takes as long as the SM with the most
// blocks, so the form whose rounds hold the fewest blocks per SM is taken, of equals the one with more blocks in flight.  One
// token, forms two / three / four in us: 192 blocks (3,072 x 2,048) 2.9 / 3.9 / 3.9, 320 (5,120 x 5,120) 14.2 / 9.4 / 10.8, 448
// (7,168 x 5,120) 15.5 / 14.7 / 12.8, 2,000 (32,000 x 2,048) 22.9 / 21.5 / 21.8: beyond six a place the last round no longer
// counts.
// The lines, as this kernel's time over gemm_tc.cu's at one to eight, nine to 16 and 17 to 32 tokens (K of 64 to 16,384; gated
// products, twice the weights a block, in brackets):
//   up to 8 tokens, up to six blocks an SM: 0.3 to 1.0 (1.02).  More blocks: a block's begin and end count again and again, 1,024
//     blocks K 256 1.16 (1.12), 512 0.83 (0.77), 4,096 0.96 (1.02), 12,288 1.04; 2,000 blocks K 512 1.23 (1.02), 1,024 0.93 (1.11);
//   up to 16, up to a block an SM: 0.3 to 0.9.  To two: K 8,192 0.96 (0.94), 12,288 1.05 (1.01).  To three: K 2,048 0.73 (0.90),
//     4,096 0.91 (1.06), 8,192 1.04 (1.15).  More: 512 blocks K 2,048 0.80 (0.88), 8,192 1.02 (1.01), not taken;
//   up to 32, up to a block an SM: registers for the tokens leave fewer weights in flight.  K 4,096 0.82 to 0.91 (0.87 to 1.07, but
//     0.95 from half of the SMs on), 8,192 1.0 to 1.1 (1.0 to 1.4; up to 24 tokens 0.9 to 1.04).  More blocks: 1.0 to 1.8.
static int plan(int T, int N, int K, bool gated, int sms) {
  const int blocks = (N + 15) / 16;
  if (T > 32) return kNone;
  if (blocks <= sms) {
    const int deepest = gated ? (2 * blocks > sms ? 4096 : 2048) : T > 24 ? 4096 : 8192;
    return T > 16 && K > deepest ? kNone : kOne;
  }
  if (T > 16) return kNone;
  if (T > 8 && (blocks > 3 * sms || K > (blocks <= 2 * sms ? 8192 : gated ? 2048 : 4096))) return kNone;
  if (blocks > 6 * sms) return K < 512 || K > (gated ? 2048 : 4096) || (blocks > 8 * sms && (K < 1024 || gated)) ? kNone : kThree;
  int best = kNone, least = 0;
  for (int f = kFour; f >= kTwo; --f) {
    const int load = (blocks + f * sms - 1) / (f * sms) * f;
    if (best == kNone || load < least) { best = f; least = load; }
  }
  return best;
}

// Loads in flight sit in the L1, so the shared memory is held to 64 KB of the 228 (left to the runtime, or with all of it as
// shared memory, a request's eight decode steps took 1,185 and 1,300 us, with 32 to 100 KB 990).
constexpr int kSharedPercent = 28;
template <int MODE, typename TO, int NB, int WARPS, int D, int DX, int PER_SM>
static void go(dim3 grid, cudaStream_t stream, const Params& p) {
  auto kernel = gemm_few_kernel<MODE, TO, NB, WARPS, D, DX, PER_SM>;
  static bool done[64] = {false};                              // per device, as the attribute is
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !done[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, kSharedPercent) != cudaSuccess)
      cudaGetLastError();                                      // (a preference: the kernel runs without it)
    done[dev] = true;
  }
  cpi::launch_pdl(kernel, grid, WARPS * 32, 0, stream, p);
}

template <int MODE, typename TO, int NB>
static int launch(const Params& p, int groups, int form, cudaStream_t stream) {
  const dim3 grid((p.N + 15) / 16, groups);
  constexpr int A = MODE == epi::kSwiglu ? 2 : 1;              // (a pair's weights take twice the registers a step)
  constexpr int X = NB > 1 ? 2 : 4 / A;
  if constexpr (NB < 4) {
    if (form == kTwo) go<MODE, TO, NB, 8, 8 / A, 2, 2>(grid, stream, p);
    if (form == kThree) go<MODE, TO, NB, 8, 4 / A, X, 3>(grid, stream, p);
    if (form == kFour) go<MODE, TO, NB, 4, 8 / A, 2, 4>(grid, stream, p);
  }
  if (form == kOne) {
    if constexpr (A * NB < 8) go<MODE, TO, NB, 16, 4 / A, X, 1>(grid, stream, p);
    else go<MODE, TO, NB, 8, 4, 2, 1>(grid, stream, p);     // (its shares' sums in 48 KB)
  }
  return check_launch("gemm_few");
}

}  // namespace few
}  // namespace cpi

using namespace cpi;

// The form that a product of T tokens (a group) and N features takes (0: it is left to gemm_tc).  Of groups it takes those of up
// to 16 rows whose blocks are all resident; short sums (up to eight steps of 32 k) need no more than four warps a block.
extern "C" int cpi_gemm_few_plan(int T, int N, int K, int gated, int groups) {
  if (T <= 0 || N <= 0) return few::kNone;
  if (groups <= 1) return few::plan(T, N, K, gated != 0, sm_count());
  const long blocks = (long)((N + 15) / 16) * groups;
  return T > 16 || groups > 65535 || blocks > 4l * sm_count() ? few::kNone : K > 256 && blocks <= sm_count() ? few::kOne : few::kFour;
}

// x [groups T, K] bf16 (row stride ldx), w [groups][N or 2N][K] bf16 contiguous, out [groups T, N] or its rows out_rows; modes as in
// cpi_gemm_tc; form as cpi_gemm_few_plan gives it.
extern "C" int cpi_gemm_few(const void* x, long ldx, const void* w, void* out, int out_dtype, long ldo, const int* out_rows, int groups, int T,
                            int N, int K, int mode, int form, float gate_limit, cudaStream_t stream) {
  if (T == 0 || N == 0) return 0;
  const int gate_act = mode == 3 ? 1 : mode == 4 ? 2 : mode == 5 ? 3 : mode == 6 ? 4 : 0;
  if (mode == 3 || mode == 4) mode = 2;
  if (mode == 5 || mode == 6) mode = 0;
  CPI_REQUIRE(T > 0 && T <= 32 && N > 0 && K > 0, "gemm_few: bad sizes T=%d N=%d K=%d", T, N, K);
  CPI_REQUIRE(groups >= 1 && groups <= 65535, "gemm_few: %d groups", groups);
  CPI_REQUIRE(form == few::kOne || (form > few::kOne && form <= few::kFour && T <= 16), "gemm_few: no form %d for %d tokens", form, T);
  CPI_REQUIRE(K % 8 == 0 && ldx % 8 == 0, "gemm_few: K (%d) and the activation row stride (%ld) must be multiples of 8", K, ldx);
  CPI_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
              "gemm_few: operands must be 16-byte aligned");
  CPI_REQUIRE(mode != epi::kAdd || out_dtype == kF32, "gemm_few: ADD mode needs a float32 output");
  CPI_REQUIRE(mode != epi::kSwiglu || out_dtype == kBF16, "gemm_few: gated modes write bfloat16");
  few::Params p{reinterpret_cast<const __nv_bfloat16*>(x), ldx, reinterpret_cast<const __nv_bfloat16*>(w), out, ldo, out_rows, T, N, K, gate_act, gate_limit};
#define CPI_FEW(MODE, TO) return T <= 8 ? few::launch<MODE, TO, 1>(p, groups, form, stream) : T <= 16 ? few::launch<MODE, TO, 2>(p, groups, form, stream) : few::launch<MODE, TO, 4>(p, groups, form, stream)
  if (mode == epi::kStore && out_dtype == kBF16) CPI_FEW(epi::kStore, __nv_bfloat16);
  if (mode == epi::kStore && out_dtype == kF32) CPI_FEW(epi::kStore, float);
  if (mode == epi::kAdd) CPI_FEW(epi::kAdd, float);
  if (mode == epi::kSwiglu) CPI_FEW(epi::kSwiglu, __nv_bfloat16);
#undef CPI_FEW
  set_error("gemm_few: unsupported mode %d with output dtype %d", mode, out_dtype);
  return 1;
}
