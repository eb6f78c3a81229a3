// Selection kernels of the top-k search.
//
//   dice_topk_floor    k-th largest of each row of group maxima: a lower bound of the row's k-th best score, because k
//                      different columns reach it
//   dice_topk_select   best k of each row's candidate list, sorted
//   dice_topk_scan     the whole search for a few queries: one pass over the table, one launch
//
// A block of 256 threads selects in two passes: the k-th largest of the threads' maxima is reached by k values, so only what
// reaches it (about k values) is gathered, and each of those counts how many are better.  Where more than 256 values reach
// the bound (ties), a radix search over histograms in shared memory finds the k-th key instead; as the general method it
// took five passes and its atomics on the few bins that similar scores share (29 us for one query against 14 541 rows).
// The work depends on the number of candidates, not on the capacity of the lists.  Scores that are -inf or NaN are never
// selected; missing places hold (-inf, -1).
//
// Measured: top 10 of 1024 queries against 2M rows x 256, everything but the pass over the table 500 -> 80 us (running lists
// per thread over the sample were 346 of it); one query against 14 541 rows 88 -> 21 us, 12 of them on the device (ten
// launches before).
#include "dice_b200.h"
#include "ptx_sm100.cuh"

#include <math_constants.h>

#include <cstddef>

namespace dice {
namespace topk {

constexpr int KMAX = 32;
constexpr int THREADS = 256;

// order-preserving key of a float; 0 marks values that cannot be selected
__device__ __forceinline__ uint32_t key_of(float s) {
  if (!(s > -CUDART_INF_F)) return 0u;
  const uint32_t b = __float_as_uint(s == 0.f ? 0.f : s);   // -0 and +0 compare equal
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t key) {
  if (key == 0u) return -CUDART_INF_F;
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

struct alignas(16) Shared {     // list and place are read four values at a time
  union {
    unsigned int hist[256];
    uint32_t list[THREADS];      // keys of the threads' maxima, then of the gathered values
  };
  int place[THREADS];            // their positions, then their ids
  unsigned int prefix, need, above, ties, count;
  uint32_t key[KMAX];
  int id[KMAX];
};
static_assert(offsetof(Shared, list) % 16 == 0 && offsetof(Shared, place) % 16 == 0, "16-byte loads");

// Number of s.list entries that come before (key, tie) in the order of decreasing keys and increasing ties (s.place, or the
// position where BY_POSITION); n is rounded up to a multiple of four, the list is padded with zeros.
template <bool BY_POSITION>
__device__ __forceinline__ int rank_in_list(const Shared& s, int n, uint32_t key, int tie) {
  int rank = 0;
  for (int j = 0; j < n; j += 4) {
    const uint4 k4 = *reinterpret_cast<const uint4*>(s.list + j);
    const int4 p4 = BY_POSITION ? make_int4(j, j + 1, j + 2, j + 3) : *reinterpret_cast<const int4*>(s.place + j);
    rank += (k4.x > key || (k4.x == key && p4.x < tie)) + (k4.y > key || (k4.y == key && p4.y < tie)) +
            (k4.z > key || (k4.z == key && p4.z < tie)) + (k4.w > key || (k4.w == key && p4.w < tie));
  }
  return rank;
}

// Gathers into s.list / s.place (positions) every value that can be among the best k of get(0 .. n-1), keys of 0 left out;
// returns their number, or -1 where there are more than 256 of them.
template <class Get>
__device__ int gather_best(Shared& s, int n, int k, Get get) {
  uint32_t bound = 1u;
  if (n > THREADS) {
    uint32_t m = 0u;
    for (int i = threadIdx.x; i < n; i += THREADS) m = max(m, get(i));
    s.list[threadIdx.x] = m;
    if (threadIdx.x == 0) s.prefix = 1u;
    __syncthreads();
    const int rank = rank_in_list<true>(s, THREADS, m, threadIdx.x);
    if (rank == k - 1 && m != 0u) s.prefix = m;
    __syncthreads();
    bound = s.prefix;
  }
  s.list[threadIdx.x] = 0u;
  s.place[threadIdx.x] = 0x7fffffff;
  if (threadIdx.x == 0) s.count = 0u;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += THREADS) {
    const uint32_t key = get(i);
    if (key >= bound) {
      const unsigned int at = atomicAdd(&s.count, 1u);
      if (at < THREADS) { s.list[at] = key; s.place[at] = i; }
    }
  }
  __syncthreads();
  return s.count <= THREADS ? static_cast<int>(s.count) : -1;
}

// k-th largest key among get(0 .. n-1), 0 if fewer than k can be selected; *need = how many of the keys equal to it belong
// to the best k.  All threads of the block call it and get the result.
template <class Get>
__device__ uint32_t kth_key(Shared& s, int n, int k, Get get, int* need) {
  if (threadIdx.x == 0) { s.prefix = 0u; s.need = k; }
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += THREADS) s.hist[i] = 0u;
    __syncthreads();
    const uint32_t prefix = s.prefix;
    for (int i = threadIdx.x; i < n; i += THREADS) {
      const uint32_t key = get(i);
      if (key != 0u && (shift == 24 || (key >> (shift + 8)) == (prefix >> (shift + 8))))
        atomicAdd(&s.hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // lane l owns the bins 255 - 8 l .. 248 - 8 l, best first
      const int lane = threadIdx.x;
      unsigned int c[8], sum = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) { c[j] = s.hist[255 - 8 * lane - j]; sum += c[j]; }
      unsigned int before = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += v;
      }
      const unsigned int total = __shfl_sync(0xffffffffu, before, 31);
      before -= sum;
      const unsigned int want = s.need;
      __syncwarp();
      if (total < want) {
        if (lane == 0) s.need = 0u;     // fewer than k values (only possible in the first pass)
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (before < want && before + c[j] >= want) {
            s.prefix = prefix | (static_cast<uint32_t>(255 - 8 * lane - j) << shift);
            s.need = want - before;
          }
          before += c[j];
        }
      }
    }
    __syncthreads();
    if (s.need == 0u) break;
  }
  *need = static_cast<int>(s.need);
  const uint32_t key = s.need == 0u ? 0u : s.prefix;
  __syncthreads();
  return key;
}

// Best k of get(0 .. n-1), sorted (ties by id): put(rank, key, id) is called once per rank by some thread.
template <class Get, class Id, class Put>
__device__ void select_best(Shared& s, int n, int k, Get get, Id id, Put put) {
  const int found = gather_best(s, n, k, get);
  if (found >= 0) {
    const int t = threadIdx.x;
    const uint32_t mine = t < found ? s.list[t] : 0u;
    const int my_id = t < found ? id(s.place[t]) : 0x7fffffff;
    __syncthreads();
    s.place[t] = my_id;
    __syncthreads();
    if (t < found) {
      const int rank = rank_in_list<false>(s, found, mine, my_id);
      if (rank < k) put(rank, mine, my_id);
    } else if (t < k) {
      put(t, 0u, -1);            // fewer than k values
    }
    __syncthreads();
    return;
  }
  int need;
  const uint32_t kth = kth_key(s, n, k, get, &need);
  if (threadIdx.x < KMAX) { s.key[threadIdx.x] = 0u; s.id[threadIdx.x] = -1; }
  if (threadIdx.x == 0) { s.above = 0u; s.ties = 0u; }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += THREADS) {
    const uint32_t key = get(i);
    unsigned int at = KMAX;
    if (key > kth) {
      at = atomicAdd(&s.above, 1u);                        // at most k - need of them
    } else if (key == kth && kth != 0u) {
      const unsigned int t = atomicAdd(&s.ties, 1u);
      if (t < static_cast<unsigned int>(need)) at = k - need + t;
    }
    if (at < KMAX) { s.key[at] = key; s.id[at] = id(i); }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const uint32_t key = lane < k ? s.key[lane] : 0u;
    const int me = lane < k ? s.id[lane] : -1;
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const uint32_t kj = __shfl_sync(0xffffffffu, key, j);
      const int ij = __shfl_sync(0xffffffffu, me, j);
      rank += (kj > key || (kj == key && (ij < me || (ij == me && j < lane)))) ? 1 : 0;
    }
    // places without a candidate (key 0) rank last, in any order
    if (rank < k) put(rank, key, me);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(THREADS) floor_kernel(const float* __restrict__ gmax, int groups, int k, float* __restrict__ floor,
                                                        int* __restrict__ cand_count) {
  __shared__ Shared s;
  const float* row = gmax + static_cast<size_t>(blockIdx.x) * groups;
  int need;
  const uint32_t kth = kth_key(s, groups, k, [&](int i) { return key_of(row[i]); }, &need);   // 9 us for 1024 rows of 1024
  if (threadIdx.x == 0) {                                                                      // maxima; by gathering 17
    floor[blockIdx.x] = value_of(kth);
    cand_count[2 * blockIdx.x] = 0;
    cand_count[2 * blockIdx.x + 1] = 0;
  }
}

__global__ void __launch_bounds__(THREADS) select_kernel(const float* __restrict__ score, const int* __restrict__ idx,
                                                         const int* __restrict__ count, int cand_cap, int tie_cap, int k,
                                                         float* __restrict__ out_s, long long* __restrict__ out_i,
                                                         float* __restrict__ kth_score, int* overflow) {
  __shared__ Shared s;
  const size_t base = static_cast<size_t>(blockIdx.x) * (cand_cap + tie_cap);
  const int found = count[2 * blockIdx.x];
  const int n1 = min(found, cand_cap), n2 = min(count[2 * blockIdx.x + 1], tie_cap);
  if (threadIdx.x == 0 && found > cand_cap) atomicOr(overflow, 1);
  auto slot = [&](int i) -> size_t { return base + (i < n1 ? i : cand_cap + (i - n1)); };
  select_best(
      s, n1 + n2, k, [&](int i) { return key_of(score[slot(i)]); }, [&](int i) { return idx[slot(i)]; },
      [&](int rank, uint32_t key, int id) {
        if (out_s != nullptr) {
          out_s[static_cast<size_t>(blockIdx.x) * k + rank] = value_of(key);
          out_i[static_cast<size_t>(blockIdx.x) * k + rank] = id;
        }
        if (kth_score != nullptr && rank == k - 1) kth_score[blockIdx.x] = value_of(key);
      });
}

// ------------------------------------------------------------------------------------ few queries
// Bound by reading the table once.  Every block scores a contiguous range of rows for all queries (scores stay in shared
// memory), selects its best k per query, and the last block to finish selects among all blocks' winners.
constexpr int SCAN_Q = 4;
constexpr int SCAN_SMEM = 160 * 1024;

struct ScanParams {
  const void* q;               // [B, d] fp32 or bf16, row stride q_stride
  int q_is_bf16;
  long long q_stride;
  int B, d, k;
  const __nv_bfloat16* table;  // [n, D]
  const float* col_bias;
  int n, y_offset, y_stride;
  int chunk;                   // rows per block
  float* part_s;               // [grid, B, k]
  int* part_i;
  unsigned int* done;          // zero-initialised, left zero
  float* out_s;                // [B, k]
  long long* out_i;
};

template <int D>
__global__ void __launch_bounds__(THREADS) scan_kernel(const ScanParams p) {
  extern __shared__ float scores[];       // [B, chunk]
  __shared__ Shared s;
  __shared__ bool last;
  constexpr int PER = D / 32;             // bf16 values of a row per lane: 2, 4 or 8
  constexpr int ROWS = 8;                 // rows of a warp in flight
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float q[SCAN_Q][PER];
#pragma unroll
  for (int b = 0; b < SCAN_Q; ++b)
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int c = lane * PER + u;
      float v = 0.f;
      if (b < p.B && c < p.d)
        v = p.q_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.q)[b * p.q_stride + c])
                        : __bfloat162float(__float2bfloat16_rn(static_cast<const float*>(p.q)[b * p.q_stride + c]));
      q[b][u] = v;
    }
  const int row0 = blockIdx.x * p.chunk;
  const int rows = min(p.chunk, p.n - row0);
  for (int r0 = warp * ROWS; r0 < rows; r0 += (THREADS / 32) * ROWS) {
    uint32_t v[ROWS][PER / 2];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const size_t r = static_cast<size_t>(row0 + min(r0 + j, rows - 1));
      const __nv_bfloat16* src = p.table + r * D + lane * PER;
      if constexpr (PER == 8) {
        const uint4 t = __ldg(reinterpret_cast<const uint4*>(src));
        v[j][0] = t.x; v[j][1] = t.y; v[j][2] = t.z; v[j][3] = t.w;
      } else if constexpr (PER == 4) {
        const uint2 t = __ldg(reinterpret_cast<const uint2*>(src));
        v[j][0] = t.x; v[j][1] = t.y;
      } else {
        v[j][0] = __ldg(reinterpret_cast<const uint32_t*>(src));
      }
    }
#pragma unroll
    for (int b = 0; b < SCAN_Q; ++b) {
      if (b >= p.B) break;
      float a[ROWS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        float x = 0.f;
#pragma unroll
        for (int u = 0; u < PER / 2; ++u) {
          x = fmaf(q[b][2 * u], __uint_as_float(v[j][u] << 16), x);
          x = fmaf(q[b][2 * u + 1], __uint_as_float(v[j][u] & 0xffff0000u), x);
        }
        a[j] = x;
      }
      // sums over the warp: lane l ends up with row l / 4
#pragma unroll
      for (int half = 4, m = 16; half > 0; half >>= 1, m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int j = 0; j < half; ++j) {
          const float keep = up ? a[j + half] : a[j];
          const float give = up ? a[j] : a[j + half];
          a[j] = keep + __shfl_xor_sync(0xffffffffu, give, m);
        }
      }
      float x = a[0];
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      const int r = r0 + (lane >> 2);
      if ((lane & 3) == 0 && r < rows) {
        if (p.col_bias != nullptr) x += p.col_bias[row0 + r];
        scores[b * p.chunk + r] = x;
      }
    }
  }
  __syncthreads();
  for (int b = 0; b < p.B; ++b) {
    const float* mine = scores + b * p.chunk;
    const size_t out = (static_cast<size_t>(blockIdx.x) * p.B + b) * p.k;
    select_best(
        s, rows, p.k, [&](int i) { return key_of(mine[i]); }, [&](int i) { return row0 + i; },
        [&](int rank, uint32_t key, int id) {
          p.part_s[out + rank] = value_of(key);
          p.part_i[out + rank] = id;
        });
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(p.done, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  const int total = static_cast<int>(gridDim.x) * p.k;
  for (int b = 0; b < p.B; ++b) {
    auto slot = [&](int i) -> size_t { return (static_cast<size_t>(i / p.k) * p.B + b) * p.k + i % p.k; };
    for (int i = threadIdx.x; i < total; i += THREADS) scores[i] = __ldcg(p.part_s + slot(i));
    __syncthreads();
    select_best(
        s, total, p.k, [&](int i) { return key_of(scores[i]); },
        [&](int i) { return __ldcg(p.part_i + slot(i)); },
        [&](int rank, uint32_t key, int id) {
          p.out_s[b * p.k + rank] = value_of(key);
          p.out_i[b * p.k + rank] = id < 0 ? -1ll : p.y_offset + static_cast<long long>(id) * p.y_stride;
        });
  }
  if (threadIdx.x == 0) *p.done = 0u;
}

// Blocks of the scan: at least 64 rows each (below that selection outweighs the scores), at most two per SM, and their
// scores must fit shared memory; 0 = the table is too large for this path.
static int scan_grid(int B, int n) {
  if (B < 1 || B > SCAN_Q || n < 1) return 0;
  int grid = (n + 63) / 64;
  if (grid > 148 * 2) grid = 148 * 2;
  const long long chunk = (n + grid - 1) / grid;
  if (chunk * B * 4 > SCAN_SMEM / 2) {   // one block per SM
    grid = 148;
    const long long c1 = (n + grid - 1) / grid;
    if (c1 * B * 4 > SCAN_SMEM) return 0;
  }
  return grid;
}

template <int D>
static int launch_scan(const ScanParams& p, int grid, cudaStream_t s) {
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(scan_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SCAN_SMEM) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  // a block's scores, or in the last block one query's winners of all blocks (148 * 2 * 32 values at most)
  const size_t smem = 4 * static_cast<size_t>(p.B * p.chunk > grid * p.k ? p.B * p.chunk : grid * p.k);
  scan_kernel<D><<<grid, THREADS, smem, s>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace topk
}  // namespace dice

// floor[row] = k-th largest of gmax[row, 0 .. groups) (-inf when there are fewer); clears cand_count [rows, 2].
extern "C" int dice_topk_floor(const float* gmax, int rows, int groups, int k, float* floor, int* cand_count, void* stream) {
  using namespace dice::topk;
  if (rows <= 0) return 0;
  if (k < 1 || k > KMAX || groups < 1) return -7;
  floor_kernel<<<rows, THREADS, 0, static_cast<cudaStream_t>(stream)>>>(gmax, groups, k, floor, cand_count);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// Best k of the lists written by dice_rank_collect (tie_cap > 0): out_s / out_i [rows, k] sorted, best first, and / or
// kth_score [rows].  *overflow is set when a list had no room for a score above the floor.
extern "C" int dice_topk_select(const float* score, const int* idx, const int* count, int rows, int cand_cap, int tie_cap, int k,
                                float* out_s, long long* out_i, float* kth_score, int* overflow, void* stream) {
  using namespace dice::topk;
  if (rows <= 0) return 0;
  if (k < 1 || k > KMAX || (out_s == nullptr) != (out_i == nullptr)) return -7;
  select_kernel<<<rows, THREADS, 0, static_cast<cudaStream_t>(stream)>>>(score, idx, count, cand_cap, tie_cap, k, out_s, out_i,
                                                                         kth_score, overflow);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// Number of blocks dice_topk_scan uses for B queries against n rows (its scratch is [blocks, B, k]), 0 if it cannot.
extern "C" int dice_topk_scan_blocks(int B, int n) { return dice::topk::scan_grid(B, n); }

// Best k rows of table [n, D] for the B <= 4 queries q [B, d] (fp32, rounded to bf16 here, or bf16): out_s / out_i [B, k].
extern "C" int dice_topk_scan(const void* q, int q_is_bf16, long long q_stride, int B, int d, const void* table, int n, int D, int k,
                              const float* col_bias, int y_offset, int y_stride, float* part_s, int* part_i, unsigned int* done,
                              float* out_s, long long* out_i, void* stream) {
  using namespace dice::topk;
  const int grid = scan_grid(B, n);
  if (grid <= 0 || k < 1 || k > KMAX || d < 1 || d > D) return -7;
  if (reinterpret_cast<uintptr_t>(table) & 15) return -5;
  const ScanParams p{q, q_is_bf16, q_stride, B, d, k, static_cast<const __nv_bfloat16*>(table), col_bias, n, y_offset,
                     y_stride > 0 ? y_stride : 1, (n + grid - 1) / grid, part_s, part_i, done, out_s, out_i};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (D) {
    case 256: return launch_scan<256>(p, grid, s);
    case 128: return launch_scan<128>(p, grid, s);
    case 64: return launch_scan<64>(p, grid, s);
    default: return -6;
  }
}
