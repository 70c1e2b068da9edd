// C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) with 32-bit FMA on the CUDA cores.
//
// This is the matrix product of the true 32-bit path: no tensor cores, no reduced
// precision mode.  Every output element is summed in the same order whatever the tile shape
// or M is, so a row's result does not depend on what else is in the batch: k runs in order,
// in chains of fmaf over SUM_BLOCK = 64 consecutive k, and the chains' results are added in
// order.  (One chain over all of K loses about sqrt(K) roundings of the running sum; two levels
// lose sqrt(64) + sqrt(K / 64): at K = 4,096 an eighth of the error, which 36 layers of four
// products each need to stay within 1e-4 of a float64 reference.)  Inputs may also be bfloat16
// (products and sums still 32-bit).
// tinyserve uses cuBLAS through nn.Linear for all of these (serve.py:828-829, 912-913, 1263).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"

TS_DEFINE_LAST_ERROR()

namespace {

constexpr int BK = 16;
constexpr int SUM_BLOCK = 64;        // k of one fmaf chain
constexpr int THREADS = 256;

template <typename T> struct Load4;
template <> struct Load4<float> {
  static __device__ __forceinline__ void run(const float* p, float (&v)[4]) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  }
};
template <> struct Load4<__nv_bfloat16> {
  static __device__ __forceinline__ void run(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&q.x);
    const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&q.y);
    v[0] = __low2float(lo); v[1] = __high2float(lo); v[2] = __low2float(hi); v[3] = __high2float(hi);
  }
};

// rows x BK tile of a [rows_total, K] matrix (leading dimension ld) -> smem[k][row]
template <typename T, int ROWS, bool VEC>
__device__ __forceinline__ void load_tile(const T* __restrict__ src, int row0, int rows_total, int k0,
                                          int K, size_t ld, float (*dst)[ROWS + 4]) {
  if (VEC) {
    for (int i = threadIdx.x; i < ROWS * (BK / 4); i += THREADS) {
      const int r = i / (BK / 4), kq = (i % (BK / 4)) * 4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (row0 + r < rows_total && k0 + kq < K) Load4<T>::run(src + (size_t)(row0 + r) * ld + k0 + kq, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[kq + j][r] = v[j];
    }
  } else {
    for (int i = threadIdx.x; i < ROWS * BK; i += THREADS) {
      const int r = i / BK, k = i % BK;
      dst[k][r] = (row0 + r < rows_total && k0 + k < K)
                      ? to_f32<T>(src[(size_t)(row0 + r) * ld + k0 + k]) : 0.f;
    }
  }
}

// index of the j-th of a thread's TX values along a tile edge of length B: chunks of 4
// spread over the edge so that shared-memory reads of neighbouring threads do not collide
template <int B, int TX>
__device__ __forceinline__ int spread(int t, int j) {
  return (j / 4) * (B / (TX / 4)) + t * 4 + (j % 4);
}

template <typename TI, typename TO, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(THREADS)
gemm_nt_kernel(const TI* A, const TI* W, const TI* bias,
               TO* __restrict__ C, int M, int N, int K, size_t lda, size_t ldw, size_t ldc) {
  static_assert((BM / TM) * (BN / TN) == THREADS, "tile does not match the block");
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  pdl_trigger();
  pdl_wait();
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN], part[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = part[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    load_tile<TI, BM, VEC>(A, m0, M, k0, K, lda, As);
    load_tile<TI, BN, VEC>(W, n0, N, k0, K, ldw, Ws);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[k][spread<BM, TM>(ty, i)];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Ws[k][spread<BN, TN>(tx, j)];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) part[i][j] = fmaf(a[i], b[j], part[i][j]);
    }
    if ((k0 + BK) % SUM_BLOCK == 0 || k0 + BK >= K) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          acc[i][j] += part[i][j];
          part[i][j] = 0.f;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + spread<BM, TM>(ty, i);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + spread<BN, TN>(tx, j);
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += to_f32<TI>(bias[n]);
      C[(size_t)m * ldc + n] = from_f32<TO>(v);
    }
  }
}

// The tiled product with the chains of k dealt to CHAIN_GROUPS groups of threads, for float operands: a
// block has a tile of 64 x 64 outputs, 64 threads of 8 x 8 outputs each take one chain of SUM_BLOCK k
// of it, and four chains are under way side by side.  After every four chains the groups' results
// meet in shared memory, where each output is added up in the order of k: the sums are those of the other kernels
// bit by bit.  Slices of 16 k of every chain come through a ring of stages by cp.async, K fastest, in
// rows of 64 bytes whose 16-byte unit u lies at u ^ (row / 2 & 3).
// Bound by the multiply-add units (half of their rate: 36 TFLOP/s at 24576 x 4096 by 1,024 rows, where the tiled
// kernel reached 21) and, for few tiles, by the chain of a block.  227 rows: 6144 x 1024 209 -> 109 us, 4096 x 1024
// 217 -> 74; 1,024 rows of 1024 x 3072 588 -> 214.
constexpr int CHAIN_GROUPS = 4, TILE = 64, SLICE = 16, SPLIT_STAGES = 2;
constexpr int SPLIT_THREADS = 64 * CHAIN_GROUPS;
constexpr int SLICE_BYTES = TILE * SLICE * 4;                        // of one operand and chain
constexpr int SPLIT_STAGE_BYTES = 2 * CHAIN_GROUPS * SLICE_BYTES;    // 32 KB
constexpr size_t SPLIT_SMEM = (size_t)SPLIT_STAGES * SPLIT_STAGE_BYTES;       // the ring; behind it the chains' results, a quarter of the tile
constexpr size_t SPLIT_RED_BYTES = (size_t)CHAIN_GROUPS * 16 * TILE * 4;
constexpr size_t SPLIT_TOTAL_BYTES = (size_t)TILE * TILE * 4;        // and the outputs' sums so far

__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0));
}

__global__ void __launch_bounds__(SPLIT_THREADS, 2)
gemm_nt_chains_kernel(const float* A, const float* W, const float* bias,
                      float* __restrict__ C, int M, int N, int K, size_t lda, size_t ldw, size_t ldc, bool constant_w) {
  extern __shared__ __align__(16) char smem[];
  pdl_trigger();
  const int tid = threadIdx.x, grp = tid >> 6, t = tid & 63;
  // 8 x 8 outputs of a thread: rows ty + 8 i, columns tx + 8 j
  const int tx = t & 7, ty = t >> 3;
  const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
  const int chains = (K + SUM_BLOCK - 1) / SUM_BLOCK;
  const int rounds = (chains + CHAIN_GROUPS - 1) / CHAIN_GROUPS;
  constexpr int PER_ROUND = SUM_BLOCK / SLICE;
  const int stages = rounds * PER_ROUND;
  auto load = [&](int st, bool of_w) {
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem + (st % SPLIT_STAGES) * SPLIT_STAGE_BYTES)) +
                          (of_w ? CHAIN_GROUPS * SLICE_BYTES : 0);
    const float* src = of_w ? W : A;
    const size_t ld = of_w ? ldw : lda;
    const int row0 = of_w ? n0 : m0, rows = of_w ? N : M;
#pragma unroll
    for (int i = tid; i < CHAIN_GROUPS * TILE * SLICE / 4; i += SPLIT_THREADS) {
      const int u = i & 3, r = (i >> 2) & (TILE - 1), c = i >> 8;
      const int k = ((st / PER_ROUND) * CHAIN_GROUPS + c) * SUM_BLOCK + (st % PER_ROUND) * SLICE + u * 4;
      const bool ok = row0 + r < rows && k < K;
      copy16_async(base + c * SLICE_BYTES + r * (SLICE * 4) + ((u ^ ((r >> 1) & 3)) << 4), src + (ok ? (size_t)(row0 + r) * ld + k : 0), ok);
    }
  };
  // (W is read ahead of the predecessors only where the caller says that none of them may have made it; a
  // second wait returns at once)
  if (!constant_w) pdl_wait();
  for (int st = 0; st < SPLIT_STAGES - 1; ++st)
    if (st < stages) load(st, true);
  pdl_wait();
  for (int st = 0; st < SPLIT_STAGES - 1; ++st) {
    if (st < stages) load(st, false);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  float part[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) part[i][j] = 0.f;
  float* red = reinterpret_cast<float*>(smem + SPLIT_SMEM);        // [CHAIN_GROUPS][16][TILE]
  float* totals = red + SPLIT_RED_BYTES / 4;                       // [TILE][TILE], an element always by the same thread
  for (int rd = 0; rd < rounds; ++rd) {
#pragma unroll 1
    for (int q = 0; q < PER_ROUND; ++q) {
      const int st = rd * PER_ROUND + q;
      asm volatile("cp.async.wait_group %0;\n" ::"n"(SPLIT_STAGES - 2));
      __syncthreads();
      // (the stage that everybody is done with)
      if (st + SPLIT_STAGES - 1 < stages) {
        load(st + SPLIT_STAGES - 1, true);
        load(st + SPLIT_STAGES - 1, false);
      }
      asm volatile("cp.async.commit_group;\n" ::);
      const char* as = smem + (st % SPLIT_STAGES) * SPLIT_STAGE_BYTES + grp * SLICE_BYTES;
      const char* ws = as + CHAIN_GROUPS * SLICE_BYTES;
#pragma unroll
      for (int u = 0; u < SLICE / 4; ++u) {
        // (half of the rows at a time: the registers hold two blocks a multiprocessor)
#pragma unroll
        for (int half = 0; half < 8; half += 4) {
          float4 a[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = (half + i) * 8 + ty;
            a[i] = *reinterpret_cast<const float4*>(as + r * (SLICE * 4) + ((u ^ ((r >> 1) & 3)) << 4));
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = j * 8 + tx;
            const float4 w = *reinterpret_cast<const float4*>(ws + r * (SLICE * 4) + ((u ^ ((r >> 1) & 3)) << 4));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              part[half + i][j] = fmaf(a[i].x, w.x, part[half + i][j]);
              part[half + i][j] = fmaf(a[i].y, w.y, part[half + i][j]);
              part[half + i][j] = fmaf(a[i].z, w.z, part[half + i][j]);
              part[half + i][j] = fmaf(a[i].w, w.w, part[half + i][j]);
            }
          }
        }
      }
    }
    // a chain of every group is complete: its results go through shared memory, a quarter of the tile's
    // rows (16) at a time, to the thread that adds up the output
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      if (h > 0) __syncthreads();
#pragma unroll
      for (int i2 = 0; i2 < 2; ++i2) {
        const int i = h * 2 + i2;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          red[(grp * 16 + i2 * 8 + ty) * TILE + j * 8 + tx] = part[i][j];
          part[i][j] = 0.f;
        }
      }
      __syncthreads();
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const int at = o * SPLIT_THREADS + tid;
        float sum = rd == 0 ? 0.f : totals[h * 16 * TILE + at];
#pragma unroll
        for (int c = 0; c < CHAIN_GROUPS; ++c) sum += red[c * 16 * TILE + at];
        totals[h * 16 * TILE + at] = sum;
      }
    }
  }
  // output o of quarter h: row h * 16 + at / TILE of the tile
#pragma unroll
  for (int h = 0; h < 4; ++h)
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const int at = o * SPLIT_THREADS + tid;
      const int m = m0 + h * 16 + at / TILE, n = n0 + at % TILE;
      if (m < M && n < N) {
        const float sum = totals[h * 16 * TILE + at];
        C[(size_t)m * ldc + n] = bias ? sum + bias[n] : sum;
      }
    }
}

// Lets a kernel have this much dynamic shared memory, once per device of the process.
template <typename Kernel>
cudaError_t allow_shared(Kernel* kernel, size_t bytes, std::atomic<unsigned long long>& devices) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = device < 64 ? 1ull << device : 0ull;
  if (devices.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

int launch_chains(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, size_t lda, size_t ldw,
                  size_t ldc, bool constant_w, cudaStream_t stream) {
  constexpr size_t smem = SPLIT_SMEM + SPLIT_RED_BYTES + SPLIT_TOTAL_BYTES;
  static std::atomic<unsigned long long> devices;
  const cudaError_t e = allow_shared(gemm_nt_chains_kernel, smem, devices);
  if (e != cudaSuccess) return ts_fail("gemm_simt: %s", cudaGetErrorString(e));
  dim3 grid((N + TILE - 1) / TILE, (M + TILE - 1) / TILE);
  if (grid.y > 65535) return ts_fail("gemm: M = %d is too large", M);
  TS_LAUNCH("gemm_simt", gemm_nt_chains_kernel, grid, SPLIT_THREADS, smem, stream, A, W, bias, C, M, N, K, lda, ldw, ldc, constant_w);
  return 0;
}

// The product of a few rows of A (decode steps, the last rows before the vocabulary projection), in
// which W is nearly all the bytes.  A thread owns one chain of SUM_BLOCK k (a "slot") of RT rows of W
// for all of the MT rows of A, so that the sums are those of the tiled kernel bit by bit, and a block
// covers CS chains of a row at a time: its threads are CS chains x 128 / CS groups of RT rows.  Slices
// of STAGE_K k of every slot come through a ring of shared-memory stages (cp.async, 16 bytes a thread,
// neighbouring threads on neighbouring bytes of a row); with a constant W its first stages do not
// wait for the predecessor kernels.  The 16-byte unit u of slot s lies at u ^ (s & 7), so that
// eight threads that read the same unit of eight slots touch all banks.  After the last slice of a
// chain the chains' results go through shared memory to one thread per output, which adds them in
// the order of k.
// Bound by the bytes of W where MT is small, by shared-memory reads (1 + MT / RT per four fmaf x MT) above:
// hence RT rows of W share the values of A.
constexpr int SLOTS = 128;           // threads of a block: chains in flight x groups of rows
constexpr int STAGE_K = 32;          // k of a slot that a stage holds: half a chain, 128 bytes
constexpr int STAGE_UNITS = STAGE_K / 4;
constexpr int GEMV_WIDTH = 8;        // most rows of A of a block
constexpr int GEMV_MIN_BLOCKS = 128;
constexpr int MAX_CHAINS_SHIFT = 4;  // up to 16 chains of a row at a time: 8 RT rows a block

template <int MT, int RT, int STAGES>
__global__ void __launch_bounds__(SLOTS)
gemv_nt_kernel(const float* A, const float* W, const float* bias, float* __restrict__ C,
               int M, int N, int K, size_t lda, size_t ldw, size_t ldc, int cs_shift, bool constant_w) {
  extern __shared__ __align__(16) char smem[];
  const int cs = 1 << cs_shift, groups = SLOTS >> cs_shift;      // chains in flight, groups of rows
  const int rows = groups * RT;
  constexpr int W_BYTES = SLOTS * RT * STAGE_K * 4;
  const int x_bytes = MT * cs * STAGE_K * 4;
  const int stage_bytes = W_BYTES + x_bytes;
  float* red = reinterpret_cast<float*>(smem + STAGES * stage_bytes);        // [MT][rows][cs + 1]
  pdl_trigger();
  const int n0 = blockIdx.x * rows, m0 = blockIdx.y * MT;
  const int chains = (K + SUM_BLOCK - 1) / SUM_BLOCK;
  const int passes = (chains + cs - 1) >> cs_shift;              // a pass: cs chains of every row, two stages
  const int stages = 2 * passes;
  const int tid = threadIdx.x;
  const int c = tid & (cs - 1), g = tid >> cs_shift;

  // unit i of a stage: slot i / 8 ((row, chain) with the chain fastest), 16 bytes i % 8 of it
  auto load_w = [&](int st) {
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem + (st % STAGES) * stage_bytes));
    const int k0 = (st >> 1) * cs * SUM_BLOCK + (st & 1) * STAGE_K;
#pragma unroll
    for (int i = tid; i < SLOTS * RT * STAGE_UNITS; i += SLOTS) {
      const int slot = i / STAGE_UNITS, u = i % STAGE_UNITS;
      const int r = slot >> cs_shift, k = k0 + (slot & (cs - 1)) * SUM_BLOCK + u * 4;
      const bool ok = n0 + r < N && k < K;
      copy16_async(base + slot * (STAGE_K * 4) + ((u ^ (slot & 7)) << 4), W + (ok ? (size_t)(n0 + r) * ldw + k : 0), ok);
    }
  };
  auto load_x = [&](int st) {
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem + (st % STAGES) * stage_bytes + W_BYTES));
    const int k0 = (st >> 1) * cs * SUM_BLOCK + (st & 1) * STAGE_K;
    for (int i = tid; i < MT * cs * STAGE_UNITS; i += SLOTS) {
      const int slot = i / STAGE_UNITS, u = i % STAGE_UNITS;
      const int m = m0 + (slot >> cs_shift), k = k0 + (slot & (cs - 1)) * SUM_BLOCK + u * 4;
      const bool ok = m < M && k < K;
      copy16_async(base + slot * (STAGE_K * 4) + ((u ^ (slot & 7)) << 4), A + (ok ? (size_t)m * lda + k : 0), ok);
    }
  };
  // the first stages of W, then (with the predecessor's results) those of A: a group of copies each
  if (!constant_w) pdl_wait();
  for (int st = 0; st < STAGES - 1; ++st)
    if (st < stages) load_w(st);
  pdl_wait();
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < stages) load_x(st);
    asm volatile("cp.async.commit_group;\n" ::);       // (the first group holds every stage of W so far)
  }

  float part[RT][MT];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) part[r][m] = 0.f;
  const int outputs = rows * MT;
  float* totals = red + (size_t)outputs * (cs + 1);              // [MT][rows]
  for (int st = 0; st < stages; ++st) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    __syncthreads();
    // (the stage that everybody is done with)
    if (st + STAGES - 1 < stages) {
      load_w(st + STAGES - 1);
      load_x(st + STAGES - 1);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    const char* ws = smem + (st % STAGES) * stage_bytes;
    const char* xs = ws + W_BYTES + c * (STAGE_K * 4);
#pragma unroll(MT * RT >= 16 ? 2 : 4)
    for (int u = 0; u < STAGE_UNITS; ++u) {
      float4 w[RT];
#pragma unroll
      for (int r = 0; r < RT; ++r)
        w[r] = *reinterpret_cast<const float4*>(ws + (r * SLOTS + tid) * (STAGE_K * 4) + ((u ^ (tid & 7)) << 4));
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        // (slot m * cs + c of A: its low bits are c's, and m's where there are fewer than eight chains)
        const float4 x = *reinterpret_cast<const float4*>(xs + (m << cs_shift) * (STAGE_K * 4) + ((u ^ (((m << cs_shift) + c) & 7)) << 4));
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          part[r][m] = fmaf(x.x, w[r].x, part[r][m]);
          part[r][m] = fmaf(x.y, w[r].y, part[r][m]);
          part[r][m] = fmaf(x.z, w[r].z, part[r][m]);
          part[r][m] = fmaf(x.w, w[r].w, part[r][m]);
        }
      }
    }
    if (st & 1) {
      // a chain of every slot is complete
#pragma unroll
      for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          red[(size_t)(m * rows + r * groups + g) * (cs + 1) + c] = part[r][m];
          part[r][m] = 0.f;
        }
      __syncthreads();
      for (int o = tid; o < outputs; o += SLOTS) {
        float sum = st == 1 ? 0.f : totals[o];
        for (int i = 0; i < cs; ++i) sum += red[(size_t)o * (cs + 1) + i];
        if (st + 1 < stages) {
          totals[o] = sum;
        } else {
          const int m = m0 + o / rows, n = n0 + o % rows;
          if (m < M && n < N) C[(size_t)m * ldc + n] = bias ? sum + bias[n] : sum;
        }
      }
    }
  }
}

template <int MT, int RT, int STAGES>
int launch_gemv(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, size_t lda, size_t ldw,
                size_t ldc, bool constant_w, cudaStream_t stream) {
  const int chains = (K + SUM_BLOCK - 1) / SUM_BLOCK;
  int cs_shift = 0;
  while (cs_shift < MAX_CHAINS_SHIFT && (1 << cs_shift) < chains) ++cs_shift;
  auto smem_of = [](int shift) {
    const int cs = 1 << shift, outputs = (SLOTS >> shift) * RT * MT;
    return (size_t)STAGES * (SLOTS * RT + MT * cs) * STAGE_K * 4 + (size_t)outputs * (cs + 2) * 4;
  };
  size_t most = 0;
  for (int s = 0; s <= MAX_CHAINS_SHIFT; ++s) most = std::max(most, smem_of(s));
  static std::atomic<unsigned long long> devices;
  const cudaError_t e = allow_shared(gemv_nt_kernel<MT, RT, STAGES>, most, devices);
  if (e != cudaSuccess) return ts_fail("gemm_simt: %s", cudaGetErrorString(e));
  const int rows = (SLOTS >> cs_shift) * RT;
  dim3 grid((N + rows - 1) / rows, (M + MT - 1) / MT);
  if (grid.y > 65535) return ts_fail("gemm: M = %d is too large", M);
  TS_LAUNCH("gemm_simt", (gemv_nt_kernel<MT, RT, STAGES>), grid, SLOTS, smem_of(cs_shift), stream, A, W, bias, C, M, N, K,
            lda, ldw, ldc, cs_shift, constant_w);
  return 0;
}

// of the current device (148 if it does not say)
int multiprocessors() {
  constexpr int DEVICES = 64;
  static std::atomic<int> known[DEVICES];
  int device = 0, n = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device >= DEVICES) return 148;
  if ((n = known[device].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) return 148;
  known[device].store(n, std::memory_order_relaxed);
  return n;
}

template <typename TI, typename TO>
int launch(const void* A, const void* W, const void* bias, void* C, int M, int N, int K, size_t lda,
           size_t ldw, size_t ldc, bool constant_w, cudaStream_t stream) {
  const size_t align = 4 * sizeof(TI);
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(A) % align == 0 && reinterpret_cast<uintptr_t>(W) % align == 0;
  const TI* a = static_cast<const TI*>(A);
  const TI* w = static_cast<const TI*>(W);
  const TI* b = static_cast<const TI*>(bias);
  TO* c = static_cast<TO*>(C);
  constexpr bool chained = std::is_same<TI, float>::value && std::is_same<TO, float>::value;
  if constexpr (chained) {
    // (a grid has 65,535 blocks of rows at most: more rows than these kernels' blocks cover go to the wider ones)
    auto fits = [&](int rows) { return ((long long)M + rows - 1) / rows <= 65535; };
    if (vec && fits(TILE)) {
      // Estimates in us; the three kernels give the same bits.
      // few: the kernel for few rows, 13.8 TFLOP/s where it fills the device, for what its blocks compute: whole groups of
      // rows of W, whole passes of chains.  many: the chains kernel, a round of four chains in 10.25 us where a
      // multiprocessor has one block, in 9 a block where it has more (measured: 4096 x 1024 by 48 / 64 / 128 / 512 rows
      // 35 / 42 / 81 / 325 us against 41 / 42 / 65 / 143; 24576 x 4096 by 24 / 48 rows 309 / 609 against 422 / 425).
      const int chains = (K + SUM_BLOCK - 1) / SUM_BLOCK, sms = multiprocessors();
      int cs = 1;
      while (cs < (1 << MAX_CHAINS_SHIFT) && cs < chains) cs *= 2;
      auto blocks = [&](int mt, int rt) { return (long long)((N + SLOTS / cs * rt - 1) / (SLOTS / cs * rt)) * ((M + mt - 1) / mt); };
      const int passes = (chains + cs - 1) / cs, group = SLOTS / cs * 2;
      const double few = 2.0 * M * ((N + group - 1) / group * (double)group) * (passes * cs * SUM_BLOCK) / 13.8e6;
      const long long tiles = (long long)((N + TILE - 1) / TILE) * ((M + TILE - 1) / TILE);
      const double many = (chains + CHAIN_GROUPS - 1) / CHAIN_GROUPS * (tiles <= sms ? 10.25 : 9.0 * ((tiles + sms - 1) / sms));
      // As many rows of A to a block as leave a block for nearly every multiprocessor: they share the reads of W.
      const int width = M > 4 && blocks(GEMV_WIDTH, 2) >= GEMV_MIN_BLOCKS ? GEMV_WIDTH : M > 2 && blocks(4, 2) >= GEMV_MIN_BLOCKS ? 4 : 2;
      const int height = width > 2 || blocks(2, 2) >= GEMV_MIN_BLOCKS ? 2 : 1;
      const bool chained_tiles = M > GEMV_WIDTH && (many < few || !fits(GEMV_WIDTH));
      // Both work in whole chains and rounds, the tiled kernel in slices of 16 k (2.75 us for a tile of 128 x 128; 64 x 64 up
      // to 64 rows): the better one for a short K.  M x N x K, us, the other kernel's first: 100,000 x 8 x 16 314 / 23,
      // 512 x 32,000 x 4 214 / 33, 20,000 x 256 x 96 83 / 54, 4,096 x 64 x 64 16 / 12, but 4,096 x 128 x 128 15 / 24.
      const double ours = chained_tiles ? many : 1.0 + std::max(1.4 * few, 0.45 * passes * width * height);
      const int slices = (K + BK - 1) / BK;
      double tiled;
      if (M > 64) {
        const long long t = (long long)((N + 127) / 128) * ((M + 127) / 128);
        tiled = 2.5 + 2.75 * slices * ((t + sms - 1) / sms) + (double)t / sms;
      } else {
        const double t = (double)((N + 63) / 64) / sms;
        tiled = 1.0 + std::max(1.65, 0.75 * t) * slices + 0.3 * t;
      }
      if (tiled >= 0.95 * ours) {
        if (chained_tiles) return launch_chains(a, w, b, c, M, N, K, lda, ldw, ldc, constant_w, stream);
        if (width == GEMV_WIDTH) return launch_gemv<GEMV_WIDTH, 2, 2>(a, w, b, c, M, N, K, lda, ldw, ldc, constant_w, stream);
        if (width == 4) return launch_gemv<4, 2, 2>(a, w, b, c, M, N, K, lda, ldw, ldc, constant_w, stream);
        if (height == 2) return launch_gemv<2, 2, 3>(a, w, b, c, M, N, K, lda, ldw, ldc, constant_w, stream);
        return launch_gemv<2, 1, 3>(a, w, b, c, M, N, K, lda, ldw, ldc, constant_w, stream);
      }
    }
  }
  if (M > 64) {
    dim3 grid((N + 127) / 128, (M + 127) / 128);
    if (grid.y > 65535) return ts_fail("gemm: M = %d is too large", M);
    if (vec) TS_LAUNCH("gemm_simt", (gemm_nt_kernel<TI, TO, 128, 128, 8, 8, true>), grid, THREADS, 0, stream, a, w, b, c, M, N, K, lda, ldw, ldc);
    else TS_LAUNCH("gemm_simt", (gemm_nt_kernel<TI, TO, 128, 128, 8, 8, false>), grid, THREADS, 0, stream, a, w, b, c, M, N, K, lda, ldw, ldc);
  } else {
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    if (vec) TS_LAUNCH("gemm_simt", (gemm_nt_kernel<TI, TO, 64, 64, 4, 4, true>), grid, THREADS, 0, stream, a, w, b, c, M, N, K, lda, ldw, ldc);
    else TS_LAUNCH("gemm_simt", (gemm_nt_kernel<TI, TO, 64, 64, 4, 4, false>), grid, THREADS, 0, stream, a, w, b, c, M, N, K, lda, ldw, ldc);
  }
  return 0;
}

}  // namespace

// in_dtype: element type of A, W and bias; out_dtype: element type of C; constant_w: no kernel that may still run
// writes W (float32 products then fetch their first tiles of it before the kernels ahead of them are done)
TS_EXPORT int ts_gemm_simt(int in_dtype, int out_dtype, const void* A, const void* W,
                           const void* bias, void* C, int M, int N, int K, long long lda,
                           long long ldw, long long ldc, int constant_w, cudaStream_t stream) {
  TS_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: empty operand (M=%d N=%d K=%d)", M, N, K);
  TS_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm: a leading dimension is smaller than its row");
  if (in_dtype == TS_F32 && out_dtype == TS_F32)
    return launch<float, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, constant_w != 0, stream);
  if (in_dtype == TS_BF16 && out_dtype == TS_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16>(A, W, bias, C, M, N, K, lda, ldw, ldc, constant_w != 0, stream);
  if (in_dtype == TS_BF16 && out_dtype == TS_F32)
    return launch<__nv_bfloat16, float>(A, W, bias, C, M, N, K, lda, ldw, ldc, constant_w != 0, stream);
  return ts_fail("gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}
