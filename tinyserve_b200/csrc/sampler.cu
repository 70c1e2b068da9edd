// Sampling from 32-bit logits, everything on the device.  A row is read by one block or by a cluster of up
// to eight, a range of the vocabulary each, which combine their maxima and histograms through
// distributed shared memory.  All that blocks combine is a maximum or an integer sum, so the result does
// not depend on how many blocks share a row.  One row of 151,936 logits (600 KB) by one block / by eight:
// greedy 9.1 / 4.8 us, with a temperature 66 / 12, with top-p 369 / 65, with top-k 50 and top-p 311 / 64.
//
//   temperature == 0           -> argmax (serve.py:1521-1522)
//   temperature > 0            -> x = logit / temperature, optional top-k (keep the k largest),
//                                 optional top-p (keep a token iff the probability mass of the
//                                 tokens ranked before it is <= top_p), then Gumbel-max over the
//                                 kept tokens: argmax(x + g) (serve.py:1544-1547, 1575-1588;
//                                 tinykernels.py:1813-1859)
//   repetition penalty         -> ts_apply_repetition_penalty, before sampling (serve.py:1488-1497)
//
// The noise is counter-based, so a row's sample does not depend on the rest of the batch:
// token v of a row uses word v % 4 of Philox-4x32-10 with key (seed_lo, seed_hi) and counter
// (v / 4, step, stream_lo, stream_hi); u = ((word >> 9) + 0.5) * 2^-23; g = -log(-log(u)).
// tinyserve draws from torch's global generator instead (serve.py:1546, tinykernels.py:1866).
// Ties go to the lowest token id.  Top-k keeps every token that ties with the k-th largest.
#include <atomic>

#include "common.cuh"

TS_DEFINE_LAST_ERROR()

namespace {

constexpr int THREADS = 1024;
// The longest row of which one block finds the maximum as fast as a cluster (16,384 / 32,000 / 65,536 tokens: 2.6 / 3.6 /
// 4.8 us by one block, 3.6 / 3.9 / 4.1 by the best of two, four and eight).
constexpr int GREEDY_ALONE = 32768;

__device__ __forceinline__ void philox4x32_10(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__device__ __forceinline__ float gumbel(uint32_t word) {
  const float u = ((float)(word >> 9) + 0.5f) * 1.1920928955078125e-07f;   // 2^-23
  return -logf(-logf(u));
}

// order-preserving map from float to unsigned
__device__ __forceinline__ uint32_t sort_key(float x) {
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct Best {
  float value;
  int index;
};
__device__ __forceinline__ Best better(Best a, Best b) {
  if (b.value > a.value || (b.value == a.value && b.index < a.index)) return b;
  return a;
}
__device__ Best block_best(Best v, Best* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best other;
    other.value = __shfl_xor_sync(0xffffffffu, v.value, o);
    other.index = __shfl_xor_sync(0xffffffffu, v.index, o);
    v = better(v, other);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    Best t = lane < (blockDim.x >> 5) ? scratch[lane] : Best{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      Best other;
      other.value = __shfl_xor_sync(0xffffffffu, t.value, o);
      other.index = __shfl_xor_sync(0xffffffffu, t.index, o);
      t = better(t, other);
    }
    if (lane == 0) scratch[0] = t;
  }
  __syncthreads();
  return scratch[0];
}

__device__ __forceinline__ uint32_t cluster_blocks() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned long long cluster_load_u64(const unsigned long long* own_shared, uint32_t rank) {
  uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(own_shared)), remote;
  unsigned long long v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
  return v;
}

__device__ float block_max_f(float v, float* scratch) {
  v = warp_max(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < (blockDim.x >> 5) ? scratch[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

// The histograms of one radix pass: a block counts into its own, every block of the cluster then adds
// up all of them.  Two buffers take turns, so that one cluster barrier per pass is enough: a
// buffer is cleared two passes later, after the barrier that its last readers arrived at.
struct Histogram {
  unsigned long long own[2][256];
  unsigned long long all[256];
  unsigned int chosen;
  unsigned long long before;       // what lies in bins above the chosen one
};

// hist[bin] += weight for the lanes with `on`.  `crowded`: most lanes fall into a few bins; lanes of one
// bin then add up among themselves first (a weight above 2^32, which only infinite logits can have, goes
// its own way).
__device__ __forceinline__ void hist_add(unsigned long long* hist, bool on, uint32_t bin, unsigned long long weight, bool crowded) {
  if (on && (!crowded || weight > (1ull << 32))) {
    atomicAdd(&hist[bin], weight);
    on = false;
  }
  if (!crowded) return;
  const unsigned active = __ballot_sync(0xffffffffu, on);
  if (!on) return;
  const unsigned peers = __match_any_sync(active, bin);
  const uint32_t lo = __reduce_add_sync(peers, (uint32_t)(weight & 0xFFFFFFu));
  const uint32_t hi = __reduce_add_sync(peers, (uint32_t)(weight >> 24));
  if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[bin], ((unsigned long long)hi << 24) + lo);
}

// Sums of the cluster's histograms into h.all (every block for itself); called by all threads.
template <bool CLUSTER>
__device__ void hist_combine(Histogram& h, int buf, uint32_t blocks) {
  if constexpr (CLUSTER) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (threadIdx.x < 256) {
    unsigned long long sum = 0;
    if constexpr (CLUSTER) {
      for (uint32_t r = 0; r < blocks; ++r) sum += cluster_load_u64(&h.own[buf][threadIdx.x], r);
    } else {
      sum = h.own[buf][threadIdx.x];
    }
    h.all[threadIdx.x] = sum;
  }
  __syncthreads();
}

// From the highest bin down: the first bin where before + bins above + the bin reaches `limit` (>= limit, or
// > limit with `beyond`); h.chosen is that bin (0 if there is none), h.before = before + the bins above it
// (all bins if there is none).
__device__ void hist_choose(Histogram& h, unsigned long long before, unsigned long long limit, bool beyond) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    unsigned long long own = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) own += h.all[255 - (lane * 8 + i)];
    unsigned long long upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const unsigned long long total = before + upto;
    const unsigned hit = __ballot_sync(0xffffffffu, beyond ? total > limit : total >= limit);
    if (hit == 0) {
      if (lane == 31) { h.chosen = 0; h.before = total; }
    } else if (lane == __ffs(hit) - 1) {
      unsigned long long cum = total - own;
      for (int i = 0; i < 8; ++i) {
        const int bin = 255 - (lane * 8 + i);
        const unsigned long long next = cum + h.all[bin];
        if (beyond ? next > limit : next >= limit) { h.chosen = bin; h.before = cum; break; }
        cum = next;
      }
    }
  }
  __syncthreads();
}

constexpr int LIST = 1024;            // most tokens of a block that top-k leaves and the passes after it keep apart

struct SampleArgs {
  const float* logits;      // [rows, row_stride]
  long long row_stride;
  int vocab;
  const float* temperature; // [rows]
  const int* top_k;         // [rows] or null; <= 0 means off
  const float* top_p;       // [rows] or null; >= 1 means off
  const unsigned long long* stream;   // [rows] request key of the noise
  const unsigned int* step;           // [rows] position counter of the noise
  unsigned long long seed;
  int* out;                 // [rows]
  int* slot_tokens;         // optional: the token also goes to slot_tokens[slots[row]]
  const int* slots;
};

// CLUSTER false: a row is one block's, which then has nothing to wait for (a cluster of one costs 0.8 to 1 us:
// 512 tokens greedy 1.8 us, 2.8 as a cluster).
template <bool CLUSTER>
__global__ void __launch_bounds__(THREADS) sample_kernel(SampleArgs a) {
  __shared__ Best best_scratch[32];
  __shared__ float f_scratch[33];
  __shared__ Histogram h;
  __shared__ unsigned long long shared_word;      // what this block tells the cluster (a maximum, or its best token)
  // the tokens that top-k leaves of this block's range, where they are so few: the passes after it go over these alone
  // (151,936 tokens, top-k 50 and top-p, us: 1 row 87 -> 64, 16 143 -> 100, 64 249 -> 171)
  __shared__ int list_token[LIST];
  __shared__ float list_value[LIST];
  __shared__ int list_count;

  pdl_trigger();
  pdl_wait();
  const uint32_t blocks = CLUSTER ? cluster_blocks() : 1u, rank = CLUSTER ? cluster_rank() : 0u;
  const int row = blockIdx.x / blocks;
  const float* x = a.logits + (size_t)row * a.row_stride;
  const int V = a.vocab;
  // this block's range of the vocabulary, in whole groups of four tokens (one Philox call each)
  const int per = ((V + 3) / 4 + blocks - 1) / blocks * 4;
  int v0 = min(V, (int)rank * per), v1 = min(V, v0 + per);
  bool alone = false;       // the first block has the row to itself
  const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const float temp = a.temperature[row];

  // tokens v .. v + 3 of the row (v a multiple of four); -inf behind the range
  auto load4 = [&](int v, float (&q)[4]) {
    if (aligned && v + 3 < v1) {
      const float4 t = *reinterpret_cast<const float4*>(x + v);
      q[0] = t.x; q[1] = t.y; q[2] = t.z; q[3] = t.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) q[j] = v + j < v1 ? x[v + j] : -INFINITY;
    }
  };
  // the best of all blocks' tokens; the first block writes it
  auto finish = [&](Best b) {
    b = block_best(b, best_scratch);
    if (CLUSTER && !alone) {
      if (threadIdx.x == 0) shared_word = (unsigned long long)__float_as_uint(b.value) << 32 | (uint32_t)b.index;
      cluster_arrive();
      cluster_wait();
      if (rank == 0 && threadIdx.x == 0)
        for (uint32_t r = 1; r < blocks; ++r) {
          const unsigned long long w = cluster_load_u64(&shared_word, r);
          b = better(b, Best{__uint_as_float((uint32_t)(w >> 32)), (int)(uint32_t)w});
        }
    }
    if (rank == 0 && threadIdx.x == 0) {
      a.out[row] = b.index;
      if (a.slot_tokens) a.slot_tokens[a.slots[row]] = b.index;
    }
    if (CLUSTER && !alone) {
      // no block leaves while the first may still read its shared memory
      cluster_arrive();
      cluster_wait();
    }
  };

  if (!(temp > 0.f)) {   // greedy
    // a short row is the first block's (nobody has met in the cluster so far)
    alone = CLUSTER && V <= GREEDY_ALONE;
    if (alone) {
      if (rank > 0) return;
      v0 = 0;
      v1 = V;
    }
    Best b{-INFINITY, 0x7fffffff};
    int base = v0 + threadIdx.x * 4;
    // four loads in flight per thread
    for (; aligned && base < v1 - 3 * THREADS * 4 - 3; base += 4 * THREADS * 4) {
      float4 t[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) t[i] = *reinterpret_cast<const float4*>(x + base + i * THREADS * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = base + i * THREADS * 4;
        b = better(better(better(better(b, Best{t[i].x, v}), Best{t[i].y, v + 1}), Best{t[i].z, v + 2}), Best{t[i].w, v + 3});
      }
    }
    for (; base < v1; base += THREADS * 4) {
      float q[4];
      load4(base, q);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (base + j < v1) b = better(b, Best{q[j], base + j});
    }
    finish(b);
    return;
  }
  const float inv_temp = 1.f / temp;
  const int k = a.top_k ? a.top_k[row] : 0;
  const float top_p = a.top_p ? a.top_p[row] : 1.f;
  uint32_t keep_from = 0;   // tokens with sort_key(x / temp) >= keep_from are kept
  int buf = 0;
  bool listed = false;

  if (k > 0 && k < V) {
    // radix select of the k-th largest key, one byte per pass
    uint32_t prefix = 0, mask = 0;
    unsigned long long remaining = (unsigned long long)k;
    for (int byte = 3; byte >= 0; --byte, buf ^= 1) {
      if (threadIdx.x < 256) h.own[buf][threadIdx.x] = 0ull;
      __syncthreads();
      for (int base = v0; base < v1; base += THREADS * 4) {
        const int v = base + threadIdx.x * 4;
        float q[4];
        load4(v, q);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t key = sort_key(q[j] * inv_temp);
          hist_add(h.own[buf], v + j < v1 && (key & mask) == prefix, (key >> (8 * byte)) & 255u, 1ull, byte == 3);
        }
      }
      hist_combine<CLUSTER>(h, buf, blocks);
      hist_choose(h, 0ull, remaining, false);
      prefix |= h.chosen << (8 * byte);
      remaining -= h.before;
      mask |= 0xFFu << (8 * byte);
      __syncthreads();
    }
    keep_from = prefix;
    // (More tokens than the blocks' lists hold leave no list, and the pass over the row would be for nothing: k = 9,000 and
    // top-p, with the pass / without, 1 row 103.5 / 100.2, 16 179 / 173, 64 325 / 311; top-k alone 64 rows 211 / 197.)
    if (k <= LIST * (int)blocks) {
      if (threadIdx.x == 0) list_count = 0;
      __syncthreads();
      for (int base = v0 + threadIdx.x * 4; base < v1; base += THREADS * 4) {
        float q[4];
        load4(base, q);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float y = q[j] * inv_temp;
          if (base + j < v1 && sort_key(y) >= keep_from) {
            const int at = atomicAdd(&list_count, 1);
            if (at < LIST) {
              list_token[at] = base + j;
              list_value[at] = y;
            }
          }
        }
      }
      __syncthreads();
      listed = list_count <= LIST;       // (equal logits may leave more than k tokens)
    }
  }
  const int list_n = listed ? list_count : 0;

  if (top_p < 1.f) {
    // weights exp(x - max) as 32.32 fixed point: sums are exact and order-independent
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < list_n; i += THREADS) mx = fmaxf(mx, list_value[i]);
    for (int base = v0 + threadIdx.x * 4; !listed && base < v1; base += THREADS * 4) {
      float q[4];
      load4(base, q);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float y = q[j] * inv_temp;
        if (base + j < v1 && sort_key(y) >= keep_from) mx = fmaxf(mx, y);
      }
    }
    mx = block_max_f(mx, f_scratch);
    if constexpr (CLUSTER) {
      if (threadIdx.x == 0) shared_word = __float_as_uint(mx);
      cluster_arrive();
      cluster_wait();
      for (uint32_t r = 0; r < blocks; ++r) mx = fmaxf(mx, __uint_as_float((uint32_t)cluster_load_u64(&shared_word, r)));
    }
    uint32_t prefix = 0, mask = 0;
    unsigned long long above = 0, limit = 0;
    for (int byte = 3; byte >= 0; --byte, buf ^= 1) {
      if (threadIdx.x < 256) h.own[buf][threadIdx.x] = 0ull;
      __syncthreads();
      for (int i = threadIdx.x; i < list_n; i += THREADS) {
        const uint32_t key = sort_key(list_value[i]);
        const unsigned long long w = (key & mask) == prefix ? (unsigned long long)(expf(list_value[i] - mx) * 4294967296.f) : 0ull;
        if (w != 0ull) atomicAdd(&h.own[buf][(key >> (8 * byte)) & 255u], w);
      }
      for (int base = v0; !listed && base < v1; base += THREADS * 4) {
        const int v = base + threadIdx.x * 4;
        float q[4];
        load4(v, q);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float y = q[j] * inv_temp;
          const uint32_t key = sort_key(y);
          const bool on = v + j < v1 && key >= keep_from && (key & mask) == prefix;
          const unsigned long long w = on ? (unsigned long long)(expf(y - mx) * 4294967296.f) : 0ull;
          hist_add(h.own[buf], on && w != 0ull, (key >> (8 * byte)) & 255u, w, byte == 3);
        }
      }
      hist_combine<CLUSTER>(h, buf, blocks);
      if (byte == 3) {
        unsigned long long total = 0;      // (every warp for itself; a sum of integers)
#pragma unroll
        for (int i = 0; i < 8; ++i) total += h.all[(threadIdx.x & 31) + 32 * i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        limit = (unsigned long long)((double)top_p * (double)total);
      }
      hist_choose(h, above, limit, true);
      prefix |= h.chosen << (8 * byte);
      above = h.before;
      mask |= 0xFFu << (8 * byte);
      __syncthreads();
    }
    keep_from = max(keep_from, prefix);
  }

  // Gumbel-max over the kept tokens
  const uint32_t k0 = (uint32_t)a.seed, k1 = (uint32_t)(a.seed >> 32);
  const unsigned long long stream = a.stream[row];
  const uint32_t step = a.step[row];
  Best b{-INFINITY, 0x7fffffff};
  for (int i = threadIdx.x; i < list_n; i += THREADS) {
    const int v = list_token[i];
    if (sort_key(list_value[i]) < keep_from) continue;
    uint32_t c[4] = {(uint32_t)(v >> 2), step, (uint32_t)stream, (uint32_t)(stream >> 32)};
    philox4x32_10(c, k0, k1);
    const uint32_t noise = (v & 2) ? ((v & 1) ? c[3] : c[2]) : ((v & 1) ? c[1] : c[0]);
    b = better(b, Best{list_value[i] + gumbel(noise), v});
  }
  for (int base = v0 + threadIdx.x * 4; !listed && base < v1; base += THREADS * 4) {
    uint32_t c[4] = {(uint32_t)(base >> 2), step, (uint32_t)stream, (uint32_t)(stream >> 32)};
    philox4x32_10(c, k0, k1);
    float q[4];
    load4(base, q);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = base + j;
      if (v < v1) {
        const float y = q[j] * inv_temp;
        if (sort_key(y) >= keep_from) b = better(b, Best{y + gumbel(c[j]), v});
      }
    }
  }
  finish(b);
}

// logits[row, id] = logit > 0 ? logit / penalty : logit * penalty for every listed id (>= 0);
// the host lists each distinct recent token once.
__global__ void repetition_penalty_kernel(float* logits, long long row_stride, int vocab,
                                          const int* rows, const int* ids, int ids_per_row,
                                          const float* penalty) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  float* x = logits + (size_t)rows[r] * row_stride;
  const float p = penalty[r];
  for (int i = threadIdx.x; i < ids_per_row; i += blockDim.x) {
    const int id = ids[(size_t)r * ids_per_row + i];
    if (id >= 0 && id < vocab) {
      const float v = x[id];
      x[id] = v > 0.f ? v / p : v * p;
    }
  }
}

// how many clusters of this many blocks the current device holds at once (0 if it does not say)
int max_clusters(int blocks) {
  constexpr int DEVICES = 64;
  static std::atomic<int> known[DEVICES][9];       // the number + 1
  int device = 0, n = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return 0;
  if (device < DEVICES && (n = known[device][blocks].load(std::memory_order_relaxed)) > 0) return n - 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(THREADS);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = blocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, sample_kernel<true>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
  if (device < DEVICES) known[device][blocks].store(n + 1, std::memory_order_relaxed);
  return n;
}

}  // namespace

TS_EXPORT int ts_sample(const float* logits, long long row_stride, int num_rows, int vocab,
                        const float* temperature, const int* top_k, const float* top_p,
                        const unsigned long long* stream_ids, const unsigned int* steps,
                        unsigned long long seed, int* out, int* slot_tokens, const int* slots,
                        cudaStream_t stream) {
  TS_REQUIRE(num_rows > 0 && vocab > 0, "sample: empty input");
  TS_REQUIRE(row_stride >= vocab, "sample: row stride smaller than the vocabulary");
  TS_REQUIRE(temperature && stream_ids && steps && out, "sample: missing argument");
  TS_REQUIRE((slot_tokens == nullptr) == (slots == nullptr), "sample: slot_tokens and slots come together");
  SampleArgs a{logits, row_stride, vocab, temperature, top_k, top_p, stream_ids, steps, seed, out, slot_tokens, slots};
  // Blocks per row: as many (1, 2, 4 or 8, the portable cluster) as leave every row's cluster a place at once (a second
  // wave doubles the time: 16 rows of 151,936 tokens with top-k and top-p 101 us in clusters of four, 127 in
  // clusters of eight, of which 15 fit; 64 rows 175 in clusters of two, 204 of four), a range of at least 2,048 tokens each
  // and no cluster below 8,192 (with top-k and top-p 8,192 tokens 31 / 27 us by one block / by four, 4,096 tokens 23 / 27 by
  // one / by two; at a temperature alone 5.9 / 4.7 and 4.3 / 4.7).
  int blocks = 1;
  while (blocks < 8 && vocab >= 8192 && vocab / (2 * blocks) >= 2048 && num_rows <= max_clusters(2 * blocks)) blocks *= 2;
  if (blocks == 1) {
    TS_LAUNCH("sample", sample_kernel<false>, num_rows, THREADS, 0, stream, a);
    return 0;
  }
  cudaError_t e = ts_launch_cluster(sample_kernel<true>, dim3(num_rows * blocks), dim3(THREADS), 0, stream, dim3(blocks, 1, 1), a);
  if (e != cudaSuccess) return ts_fail("sample: %s", cudaGetErrorString(e));
  return 0;
}

TS_EXPORT int ts_apply_repetition_penalty(float* logits, long long row_stride, int vocab,
                                          const int* rows, const int* ids, int num_rows,
                                          int ids_per_row, const float* penalty,
                                          cudaStream_t stream) {
  TS_REQUIRE(num_rows > 0 && ids_per_row > 0, "repetition_penalty: empty input");
  TS_LAUNCH("repetition_penalty", repetition_penalty_kernel, num_rows, 256, 0, stream, logits, row_stride, vocab,
            rows, ids, ids_per_row, penalty);
  return 0;
}
