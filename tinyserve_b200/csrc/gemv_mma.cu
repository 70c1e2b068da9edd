// out[M, N] = x[M, K] W[N, K]^T for up to 8 tokens and weights that the whole device holds in registers at once
// (up to 16 MB in blocks that all have a place; 119 registers a thread, 16 warps a multiprocessor): the products of a decode
// step of a small model, bfloat16.
//
// Such a product takes longer to start and to end than to read its weights, so nothing here is staged: a warp owns 16
// weight rows and 256 columns of K and loads them before the dependency wait straight into the registers from which
// mma.sync takes them (64 a lane); after the wait there is one trip to memory for x, 16 MMAs in four accumulators, one
// meeting of the block's warps in shared memory (K is cut over the warps of a block, never over blocks) and the epilogue.
// The tcgen05 kernel (gemm_tcgen05.cu) has x brought by TMA, MMAs committed to a barrier, tensor memory read back and a
// cluster that meets twice behind its wait.  In a decode step at the 0.6B shapes (weights of 4 to 13 MB) a product takes
// 2.8 us of the critical path, 5.1 by that kernel; the step, us: 1 request of 90 tokens 810 -> 622, 8 of 300 932 -> 808.
// A lane's 16 bytes of a row are eight neighbouring k; the MMA's k are dealt to lanes in another order, but x is loaded
// in the same one, and a sum does not depend on the names of its terms.
//
// Forms (as in gemm_tcgen05.cu): plain (bfloat16 or float; or float tiles as a split-K product of one part leaves them),
// x whose rows lack their RMSNorm factor, gated, residual.
#include "common.cuh"

TS_DEFINE_LAST_ERROR()

namespace {

using bf16 = __nv_bfloat16;
constexpr int ROWS = 16;             // weight rows of a warp (MMA M)
constexpr int TOKENS = 8;            // MMA N
constexpr int KW = 256;              // columns of K of a warp
constexpr int CHUNKS = KW / 32;      // 16-byte pieces of a lane and row
constexpr int MAX_WARPS = 16;        // K up to 4096
constexpr int RED = 20;              // floats of a token's 16 sums in shared memory: no bank conflicts
constexpr int SUMSQ_STRIDE = 16;

struct GemvParams {
  const bf16* x;        // [M, ldx]
  const bf16* w;        // [N, ldw]
  void* out;            // [M, ldc] bfloat16 or float, or null
  float* partials;      // or null: [N / 128][16][128]
  int M, N, K, out_f32;
  long long ldx, ldw, ldc;
  int k_warps, groups;  // warps along K, groups of 16 rows of a block
  const float* x_sumsq; // [x_tiles][16], or null
  int x_tiles;
  float x_eps;
  float* residual;      // [M, N] or null
  VecParam norm_w;
  bf16* hprime;         // [M, N]
  float* sumsq_out;     // [N / 16][16]
  int gated_act;        // 0: off; else the activation's code + 1
  float gated_limit;
};

__device__ __forceinline__ uint4 load_weight(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(32 * MAX_WARPS, 1) gemv_mma_kernel(const __grid_constant__ GemvParams p) {
  __shared__ float red[MAX_WARPS][TOKENS * RED];
  __shared__ float factor_part[MAX_WARPS][TOKENS];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int group = warp / p.k_warps, ks = warp - group * p.k_warps, warps = blockDim.x >> 5;
  // gated: a block has 16 gate rows and the 16 up rows that belong to them, 64 further on
  auto row_of = [&](int grp) {
    return p.gated_act ? (int)(blockIdx.x >> 2) * 128 + grp * 64 + (int)(blockIdx.x & 3) * ROWS : ((int)blockIdx.x * p.groups + grp) * ROWS;
  };
  const int row = row_of(group), k0 = ks * KW + 8 * t;
  uint4 wa[CHUNKS], wb[CHUNKS];
  {
    const bf16* ra = p.w + (size_t)(row + g) * p.ldw + k0;
    const bf16* rb = ra + 8 * p.ldw;
    const bool a_in = row + g < p.N, b_in = row + g + 8 < p.N;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const bool in = k0 + 32 * c < p.K;
      wa[c] = in && a_in ? load_weight(ra + 32 * c) : make_uint4(0u, 0u, 0u, 0u);
      wb[c] = in && b_in ? load_weight(rb + 32 * c) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  // the element this thread finishes: row `er` of group `eg`, token `em` (row fastest)
  const int er = threadIdx.x & 15, em = (threadIdx.x >> 4) & 7, eg = threadIdx.x >> 7;
  const int en = row_of(eg) + er;
  const bool mine = eg < (p.gated_act ? 1 : p.groups) && em < p.M && en < p.N;
  const float wn = p.residual && mine ? p.norm_w[en] : 0.f;
  pdl_wait();
  const float before = p.residual && mine ? __ldcg(p.residual + (size_t)em * p.N + en) : 0.f;
  uint4 xv[CHUNKS];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
    xv[c] = g < p.M && k0 + 32 * c < p.K ? __ldcg(reinterpret_cast<const uint4*>(p.x + (size_t)g * p.ldx + k0 + 32 * c)) : make_uint4(0u, 0u, 0u, 0u);
  if (p.x_sumsq) {
    const int m = threadIdx.x & 7;
    float sum = 0.f;
    if (m < p.M)
      for (int i = threadIdx.x >> 3; i < p.x_tiles; i += blockDim.x >> 3) sum += __ldcg(p.x_sumsq + (size_t)i * SUMSQ_STRIDE + m);
    sum += __shfl_xor_sync(0xffffffffu, sum, 8);
    sum += __shfl_xor_sync(0xffffffffu, sum, 16);
    if (lane < TOKENS) factor_part[warp][lane] = sum;
  }
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[a][e] = 0.f;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    mma(acc[2 * c & 3], wa[c].x, wb[c].x, wa[c].y, wb[c].y, xv[c].x, xv[c].y);
    mma(acc[(2 * c + 1) & 3], wa[c].z, wb[c].z, wa[c].w, wb[c].w, xv[c].z, xv[c].w);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)        // e & 1: the token 2t or 2t + 1; e & 2: the row g or g + 8
    red[warp][(2 * t + (e & 1)) * RED + g + 4 * (e & 2)] = (acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]);
  __syncthreads();
  if (eg >= (p.gated_act ? 1 : p.groups)) return;      // (whole warps: 128 threads a group)
  auto total = [&](int grp) {
    float sum = 0.f;
    for (int s = 0; s < p.k_warps; ++s) sum += red[grp * p.k_warps + s][em * RED + er];
    return sum;
  };
  float factor = 1.f;
  if (p.x_sumsq) {
    float sum = 0.f;
    for (int i = 0; i < warps; ++i) sum += factor_part[i][em];
    factor = rsqrtf(sum / (float)p.K + p.x_eps);
  }
  if (p.residual) {
    const float v = before + total(eg) * factor;
    float sq = mine ? v * v : 0.f;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (mine) {
      p.residual[(size_t)em * p.N + en] = v;
      p.hprime[(size_t)em * p.N + en] = __float2bfloat16_rn(v * wn);
      if (er == 0) p.sumsq_out[(size_t)(en / ROWS) * SUMSQ_STRIDE + em] = sq;
    }
  } else if (p.gated_act) {
    const float y = gated_value(total(0) * factor, total(1) * factor, p.gated_act - 1, p.gated_limit);
    if (mine) static_cast<bf16*>(p.out)[(size_t)em * p.ldc + (blockIdx.x >> 2) * 64 + (blockIdx.x & 3) * ROWS + er] = __float2bfloat16_rn(y);
  } else if (mine) {
    const float y = total(eg) * factor;
    if (p.partials) p.partials[((size_t)(en >> 7) * 16 + em) * 128 + (en & 127)] = y;
    else if (p.out_f32) static_cast<float*>(p.out)[(size_t)em * p.ldc + en] = y;
    else static_cast<bf16*>(p.out)[(size_t)em * p.ldc + en] = __float2bfloat16_rn(y);
  }
}

}  // namespace

// x [M, K] (M up to 8, leading dimension ldx), w [N, K] (ldw), bfloat16, K a multiple of 8 up to 4096.  One of:
// out [M, N] (ldc; float where out_f32); partials [N / 128 rounded up][16][128] floats (a split-K product of one part);
// gated_act != 0: out [M, N / 2] bfloat16, the rows of w alternate in blocks of 64 gate and 64 up rows, N a multiple of 128;
// residual [M, N] float (contiguous) += the result, hprime [M, N] = bfloat16(residual * norm_w), sumsq_out [N / 16][16] = the
// sums of residual^2 over each 16 columns (N a multiple of 16).
// x_sumsq [x_tiles][16] (or null): every token's result is scaled by rsqrt(sum / K + x_eps).
TS_EXPORT int ts_gemv_mma(const void* x, const void* w, void* out, float* partials, int M, int N, int K, long long ldx, long long ldw,
                          long long ldc, int out_f32, const float* x_sumsq, int x_tiles, float x_eps, float* residual,
                          const void* norm_w, int norm_w_is_f32, void* hprime, float* sumsq_out, int gated_act, float gated_limit,
                          cudaStream_t stream) {
  TS_REQUIRE(M > 0 && M <= TOKENS && N > 0 && K > 0 && K <= KW * MAX_WARPS, "gemv_mma: %d tokens, %d rows, K %d", M, N, K);
  TS_REQUIRE(K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0, "gemv_mma: operands must be 16-byte aligned, K a multiple of 8");
  TS_REQUIRE((out != nullptr) + (partials != nullptr) + (residual != nullptr) == 1, "gemv_mma: one output form");
  TS_REQUIRE(gated_act == 0 || (out && !out_f32 && N % 128 == 0 && K <= KW * MAX_WARPS / 2 && gated_act <= ACT_COUNT && (gated_act - 1 != ACT_BOUNDED_SWISH || gated_limit > 0.f)),
             "gemv_mma: the gated form takes a bfloat16 output, whole blocks of 128 rows and K up to %d", KW * MAX_WARPS / 2);
  TS_REQUIRE(residual == nullptr || (norm_w && hprime && sumsq_out && N % ROWS == 0), "gemv_mma: the residual form needs the norm's weight, both outputs and whole groups of 16 rows");
  TS_REQUIRE(x_sumsq == nullptr || x_tiles > 0, "gemv_mma: sums of squares without their tile count");
  GemvParams p = {};
  p.x = static_cast<const bf16*>(x); p.w = static_cast<const bf16*>(w); p.out = out; p.partials = partials;
  p.M = M; p.N = N; p.K = K; p.out_f32 = out_f32; p.ldx = ldx; p.ldw = ldw; p.ldc = ldc;
  p.x_sumsq = x_sumsq; p.x_tiles = x_tiles; p.x_eps = x_eps;
  p.residual = residual; p.norm_w = VecParam{norm_w, norm_w_is_f32}; p.hprime = static_cast<bf16*>(hprime); p.sumsq_out = sumsq_out;
  p.gated_act = gated_act; p.gated_limit = gated_limit;
  // (128 threads finish a group of 16 rows: never fewer than four warps of it)
  p.k_warps = (K + KW - 1) / KW;
  if (p.k_warps < 4) p.k_warps = 4;
  p.groups = gated_act ? 2 : 1;
  const int warps = p.k_warps * p.groups, blocks = gated_act ? N / 32 : (N + ROWS - 1) / ROWS;
  TS_LAUNCH("gemv_mma", gemv_mma_kernel, blocks, warps * 32, 0, stream, p);
  return 0;
}
