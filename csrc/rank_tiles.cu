// Scores of queries X against an entity table Y on the tensor cores, consumed where they appear (sm_100a: tcgen05, TMEM, TMA).
//
//   COUNT    greater[row] += number of columns above target[row]
//   BAND     the same above target + margin; columns within +-margin are listed for an exact second pass
//   GMAX     largest score of every group of 32 columns (lower bounds for a top-k search)
//   COLLECT  every column at or above floor[row] goes to the row's candidate list
//
// COUNT and BAND take an optional bit mask of columns to leave out (known answers of the filtered protocol).
//
// What bounds it: one GEMM whose result never leaves the chip.  X stays in tensor memory (read as the A operand from
// there), which leaves shared memory to three Y tiles at D = 256, and the MMA reads only B from shared memory.  With X in
// shared memory there was room for two Y tiles of one GEMM each, and the refill of a stage (1100 - 1600 cycles) took
// longer than the one GEMM (1024 cycles) it had to hide behind: 2370 cycles per 128 x 128 tile.  A CTA holds 256 rows of X
// (two 128-lane planes), so every Y tile serves two GEMMs and the traffic from L2 is 32 B per clock and SM at the full
// MMA rate instead of 64.
//
// SPLIT (BAND only): the operands are sums hi + lo of two bf16 numbers and S = Xhi Yhi + Xlo Yhi + Xhi Ylo, so that S is
// within about 1.7e-4 |x| |y| of the exact product (D = 256) instead of 2^-8, and the undecided band is more than 20 times
// narrower.  The second X plane then holds the lo part of the same 128 rows.
//
// Measured: 8192 queries x 2M rows x 256, COUNT 8855 -> 6808 us, with warp-uniform MMA issue (see mma_ts_warp)
// 4096 x 262144 x 256 441 -> 400 us (1.37 PFLOP/s); 1024 x 2M x 256, COLLECT 1348 -> 1070 us;
// evaluation of 20 466 queries x 14 541 x 256 (band, filters and counts) 15.8 -> 0.56 ms on the device (75 us a batch of 4096
// for the three GEMMs; with the parts of a 64-row tile side by side in one stage 116 us, the MMA being half as wide).
//
// CTA (one per SM, persistent over a range of tiles): warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 epilogue (two per
// TMEM lane quarter, each one half of the columns; warp (quarter, p) also fills plane p of X).  All waits are bounded.
#include "dice_b200.h"
#include "ptx_sm100.cuh"
#include "tile_map.cuh"
#include "tma_host.cuh"

#include <math_constants.h>

namespace dice {
namespace rankk {

enum Mode : int { COUNT = 0, BAND = 1, GMAX = 2, COLLECT = 3 };

constexpr int THREADS = 320;
constexpr int EPI_WARPS = 8;

struct RankParams {
  const __nv_bfloat16* x;      // [x_rows, D]
  const __nv_bfloat16* x_lo;   // SPLIT
  int x_rows, y_rows, nx_tiles, ny_tiles;
  TileMap map;
  const float* target;         // [x_rows]
  const int* target_idx;       // entity never counted; may be null
  const float* col_bias;       // [y_rows] or null
  int y_offset, y_stride;      // column c is entity y_offset + c * y_stride
  const uint32_t* mask;        // bit c of row r: column c is left out; may be null
  long long mask_stride;       // words
  int* greater;
  const float* margin;
  int* band_rows;
  int* band_cols;
  unsigned long long* band_count;
  long long band_cap;
  float* gmax;                 // [x_rows, groups]
  int groups;                  // groups per row: 4 * ny_tiles
  const float* floor;
  int cand_cap, tie_cap;       // list of a row: cand_cap entries above the floor (with ties where tie_cap is 0), then tie_cap equal to it
  float* cand_score;
  int* cand_idx;
  int* cand_count;             // [x_rows] entries above, or with tie_cap > 0 [x_rows, 2]
  int* status;
};

template <int D, bool SPLIT>
struct Cfg {
  static constexpr int NSLAB = D / 64;
  static constexpr int XR = SPLIT ? 128 : 256;         // rows of an X tile
  static constexpr int BY = 128;                       // rows of a Y tile; with SPLIT its hi and lo parts are two stages
  static constexpr int PARTS = SPLIT ? 2 : 1;
  static constexpr int YSLAB = BY * 128;
  static constexpr int Y_BYTES = NSLAB * YSLAB;        // bytes of a stage
  static constexpr int NSTAGE = D == 256 ? 3 : D == 128 ? 6 : 8;
  static constexpr int S_COL = D;                      // two planes of D / 2 columns each come first
  static constexpr int NBUF = (512 - D) / BY > 4 ? 4 : (512 - D) / BY;
  static constexpr int SMEM_BYTES = NSTAGE * Y_BYTES + 1024 + 512;
  static_assert(SMEM_BYTES <= 227 * 1024 && NBUF >= 2, "layout");
};

// bit i set where r[i] > t (false for NaN; t must not be -0): the sign of t - r[i], shifted in from the top column down
__device__ __forceinline__ uint32_t above(const uint32_t (&r)[32], float t) {
  const uint64_t tt = pack2(t, t), minus = pack2(-1.f, -1.f);
  uint32_t hi = 0u, lo = 0u;
#pragma unroll
  for (int i = 14; i >= 0; i -= 2) {
    float a, b;
    unpack2(fma2(pack2(__uint_as_float(r[16 + i]), __uint_as_float(r[17 + i])), minus, tt), a, b);
    hi = __funnelshift_l(__float_as_uint(b), hi, 1);
    hi = __funnelshift_l(__float_as_uint(a), hi, 1);
    unpack2(fma2(pack2(__uint_as_float(r[i]), __uint_as_float(r[1 + i])), minus, tt), a, b);
    lo = __funnelshift_l(__float_as_uint(b), lo, 1);
    lo = __funnelshift_l(__float_as_uint(a), lo, 1);
  }
  return (hi << 16) | lo;
}

__device__ __forceinline__ float pick(const uint32_t (&r)[32], int i) {
  float s = __uint_as_float(r[0]);
#pragma unroll
  for (int u = 1; u < 32; ++u) s = (u == i) ? __uint_as_float(r[u]) : s;
  return s;
}

template <int D, int MODE, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
rank_tiles_kernel(const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ CUtensorMap tmap_ylo, const RankParams p) {
  using C = Cfg<D, SPLIT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sY = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(sY + C::NSTAGE * C::Y_BYTES);
  uint64_t* x_full = bars + 0;
  uint64_t* x_empty = bars + 1;
  uint64_t* s_full = bars + 2;                 // [NBUF]
  uint64_t* s_empty = s_full + C::NBUF;        // [NBUF]
  uint64_t* y_full = s_empty + C::NBUF;        // [NSTAGE]
  uint64_t* y_empty = y_full + C::NSTAGE;      // [NSTAGE]
  uint64_t* words = y_empty + C::NSTAGE;
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(words);
  volatile int* s_abort = reinterpret_cast<volatile int*>(words + 1);   // [0] abort flag, [1] always zero
  static_assert(8 * (4 + 2 * C::NBUF + 2 * C::NSTAGE) <= 512, "barrier area");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long total = static_cast<long long>(p.nx_tiles) * p.ny_tiles;
  const long long w_begin = total * blockIdx.x / gridDim.x;
  const long long w_end = total * (blockIdx.x + 1) / gridDim.x;

  if (threadIdx.x == 0) {
    mbar_init(x_full, EPI_WARPS);
    mbar_init(x_empty, 1);
    for (int i = 0; i < C::NBUF; ++i) {
      mbar_init(s_full + i, 1);
      mbar_init(s_empty + i, EPI_WARPS);
    }
    for (int i = 0; i < C::NSTAGE; ++i) {
      mbar_init(y_full + i, 1);
      mbar_init(y_empty + i, 1);
    }
    *reinterpret_cast<volatile uint64_t*>(words + 1) = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_base_smem, 512);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_y);
    if (SPLIT) tma_prefetch_desc(&tmap_ylo);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;

  auto fail = [&](int code) {
    atomicCAS(p.status, 0, code);
    *s_abort = 1;
  };
  // GEMM units of a Y tile: one per 128 rows of X that hold any query
  auto units_of = [&](int x) -> int {
    if (SPLIT) return 1;
    return p.x_rows - x * C::XR > 128 ? 2 : 1;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------------- TMA producer
    if (lane == 0) {
      uint32_t ycount = 0;
      bool ok = true;
      for (long long w = w_begin; w < w_end && ok && !*s_abort;) {
        int x, y0, run;
        p.map.locate(w, x, y0, run);
        const int n = static_cast<int>(min(static_cast<long long>(run), w_end - w));
        for (int t = 0; t < n * C::PARTS; ++t, ++ycount) {
          const uint32_t st = ycount % C::NSTAGE;
          if (!mbar_wait_bounded(y_empty + st, ((ycount / C::NSTAGE) & 1) ^ 1, s_abort)) { ok = false; break; }
          mbar_arrive_expect_tx(y_full + st, C::Y_BYTES);
          uint8_t* dst = sY + st * C::Y_BYTES;
          const CUtensorMap* tm = SPLIT && (t & 1) ? &tmap_ylo : &tmap_y;
          for (int s = 0; s < C::NSLAB; ++s)
            tma_load_2d(dst + s * C::YSLAB, tm, s * 64, (y0 + t / C::PARTS) * C::BY, y_full + st);
        }
        w += n;
      }
      if (!ok) fail(ST_TIMEOUT_PRODUCER);
      if (*s_abort) {  // every copy issued by this thread must land before the CTA exits
        bool drained = true;
        for (uint32_t i = 0; i < C::NSTAGE && i < ycount; ++i) {
          const uint32_t last = ycount - 1 - i;
          drained &= mbar_wait_bounded(y_full + (last % C::NSTAGE), (last / C::NSTAGE) & 1, s_abort + 1, 1u << 20);
        }
        if (!drained) atomicExch(p.status, ST_TIMEOUT_DRAIN);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------- MMA issuer
    // all lanes run this branch; one elected lane issues each MMA and commit
    {
      constexpr uint32_t IDESC = make_idesc_bf16(128, C::BY, 0, 0);
      const uint64_t ydesc = make_sw128_desc(smem_u32(sY), 16, 1024);
      uint32_t g = 0, ycount = 0, seg = 0;
      bool ok = true;
      auto all = [](bool x) { return __all_sync(0xffffffffu, x) != 0; };   // the same in every lane, and known to be
      // d (+)= (plane of X) . (Y tile at descriptor yd)^T
      auto gemm = [&](uint32_t d_tmem, uint32_t plane, uint64_t yd, bool first) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k >> 2) * (C::YSLAB >> 4) + (k & 3) * 2;
          mma_ts_warp(d_tmem, tmem_base + plane * (D / 2) + k * 8, yd + off, IDESC, (first && k == 0) ? 0u : 1u);
        }
      };
      for (long long w = w_begin; w < w_end && ok && all(*s_abort == 0);) {
        int x, y0, run;
        p.map.locate(w, x, y0, run);
        const int n = static_cast<int>(min(static_cast<long long>(run), w_end - w));
        const int units = units_of(x);
        if (!all(mbar_wait_bounded(x_full, seg & 1, s_abort))) { ok = false; break; }
        for (int t = 0; t < n && ok; ++t, ++ycount) {
          uint32_t st = ycount % C::NSTAGE;
          uint64_t yd = ydesc + st * (C::Y_BYTES >> 4);
          if (!all(mbar_wait_bounded(y_full + st, (ycount / C::NSTAGE) & 1, s_abort))) { ok = false; break; }
          for (int u = 0; u < units; ++u, ++g) {
            const uint32_t b = g % C::NBUF;
            if (!all(mbar_wait_bounded(s_empty + b, ((g / C::NBUF) & 1) ^ 1, s_abort))) { ok = false; break; }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + C::S_COL + b * C::BY;
            gemm(d_tmem, u, yd, true);
            if constexpr (SPLIT) {
              gemm(d_tmem, 1, yd, false);
              tc_commit_warp(y_empty + st);
              ++ycount;                       // the lo part is the next stage
              st = ycount % C::NSTAGE;
              yd = ydesc + st * (C::Y_BYTES >> 4);
              if (!all(mbar_wait_bounded(y_full + st, (ycount / C::NSTAGE) & 1, s_abort))) { ok = false; break; }
              tc_fence_after();
              gemm(d_tmem, 0, yd, false);
            }
            tc_commit_warp(s_full + b);
          }
          if (ok) tc_commit_warp(y_empty + st);
        }
        if (ok) tc_commit_warp(x_empty);
        w += n;
        ++seg;
      }
      if (!ok && lane == 0) fail(ST_TIMEOUT_MMA);
    }
  } else {
    // ------------------------------------------------------------------------- epilogue warps
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    const int row = quarter * 32 + lane;
    constexpr int UN = SPLIT ? 1 : 2;
    constexpr int NCH = C::BY / 64;      // chunks of 32 columns per thread and tile
    uint32_t g = 0, seg = 0;
    bool ok = true;

    for (long long w = w_begin; w < w_end && ok && !*s_abort;) {
      int x, y0, run;
      p.map.locate(w, x, y0, run);
      const int n = static_cast<int>(min(static_cast<long long>(run), w_end - w));
      const int units = units_of(x);

      // X: this warp's 32 rows of plane `half` go to tensor memory once the previous segment's GEMMs are done
      if (!mbar_wait_bounded(x_empty, (seg & 1) ^ 1, s_abort)) { ok = false; break; }
      tc_fence_after();
      {
        const int xr = x * C::XR + (SPLIT ? row : half * 128 + row);
        const __nv_bfloat16* src = (SPLIT && half == 1) ? p.x_lo : p.x;
        const uint4* rowp = reinterpret_cast<const uint4*>(src + static_cast<size_t>(xr < p.x_rows ? xr : 0) * D);
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 q = xr < p.x_rows ? rowp[c * 4 + i] : make_uint4(0u, 0u, 0u, 0u);
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
          }
          tmem_st16(tmem_base + lane_sel + half * (D / 2) + c * 16, v);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(x_full);
      }

      // per-row state of the (one or two) GEMM units
      int x_global[UN], tgt_col[UN], cnt[UN];
      float hi[UN], lo[UN];
      bool valid[UN];
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        x_global[u] = x * C::XR + u * 128 + row;
        valid[u] = x_global[u] < p.x_rows;
        hi[u] = lo[u] = CUDART_INF_F;    // rows past the end: nothing is above
        tgt_col[u] = -1;
        cnt[u] = 0;
        if (valid[u]) {
          // + 0 turns -0 into +0: the sign of -0 - (+0) would count a score of zero as above
          if constexpr (MODE == COUNT) hi[u] = p.target[x_global[u]] + 0.f;
          if constexpr (MODE == BAND) {
            const float t = p.target[x_global[u]], mg = p.margin[x_global[u]];
            hi[u] = t + mg + 0.f;
            lo[u] = t - mg + 0.f;
          }
          if constexpr (MODE == COLLECT) {
            hi[u] = p.floor[x_global[u]];
            // s >= floor  <=>  s > the next smaller float; with a floor of -inf only scores above it
            const int fb = __float_as_int(hi[u]);
            lo[u] = hi[u] == 0.f ? __int_as_float(0x80000001) : hi[u] == -CUDART_INF_F ? hi[u] : __int_as_float(hi[u] > 0.f ? fb - 1 : fb + 1);
          }
          if (p.target_idx != nullptr) {
            const int rel_id = p.target_idx[x_global[u]] - p.y_offset;
            if (rel_id >= 0 && rel_id % p.y_stride == 0) tgt_col[u] = rel_id / p.y_stride;
          }
        }
      }

      for (int t = 0; t < n && ok; ++t) {
        const int col_t = (y0 + t) * C::BY + half * (C::BY / 2);   // first column of this thread's share
#pragma unroll
        for (int u = 0; u < UN; ++u) {
          if (u >= units) continue;
          const uint32_t b = g % C::NBUF;
          uint32_t drop[NCH];
          if constexpr (MODE == COUNT || MODE == BAND) {
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
              drop[c] = 0u;
              const int wd = (col_t >> 5) + c;
              if (p.mask != nullptr && valid[u] && wd < p.mask_stride)
                drop[c] = p.mask[static_cast<size_t>(x_global[u]) * p.mask_stride + wd];
            }
          }
          if (!mbar_wait_bounded(s_full + b, (g / C::NBUF) & 1, s_abort)) { ok = false; break; }
          tc_fence_after();
          const uint32_t s_addr = tmem_base + C::S_COL + b * C::BY + lane_sel + half * (C::BY / 2);
          uint32_t r[NCH][32];
#pragma unroll
          for (int c = 0; c < NCH; ++c) tmem_ld32(s_addr + c * 32, r[c]);
          tc_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_empty + b);   // the scores are in registers: the buffer may be overwritten
          ++g;
#pragma unroll
          for (int c = 0; c < NCH; ++c) {
            const int col0 = col_t + c * 32;
            const int left = p.y_rows - col0;        // columns >= left of this chunk are padding
            if (p.col_bias != nullptr) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (i < left) r[c][i] = __float_as_uint(__uint_as_float(r[c][i]) + p.col_bias[col0 + i]);
            }
            const uint32_t in = left >= 32 ? 0xffffffffu : left <= 0 ? 0u : (1u << left) - 1u;
            if constexpr (MODE == COUNT || MODE == BAND) {
              uint32_t keep = in & ~drop[c];
              const int rel = tgt_col[u] - col0;
              if (static_cast<unsigned>(rel) < 32u) keep &= ~(1u << rel);
              const uint32_t up = above(r[c], hi[u]) & keep;
              cnt[u] += __popc(up);
              if constexpr (MODE == BAND) {
                uint32_t band = above(r[c], lo[u]) & keep & ~up;
                if (__any_sync(0xffffffffu, band != 0u)) {   // undecided pairs: one slot range per warp
                  const int nb = __popc(band);
                  int incl = nb;
#pragma unroll
                  for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                  }
                  unsigned long long base = 0;
                  if (lane == 31) base = atomicAdd(p.band_count, static_cast<unsigned long long>(incl));
                  base = __shfl_sync(0xffffffffu, base, 31);
                  long long at = static_cast<long long>(base) + incl - nb;
                  // what still fits is written: the second pass reads every slot below min(count, capacity)
                  if (band != 0u && at + nb > p.band_cap) atomicCAS(p.status, 0, ST_INBOX_OVERFLOW);
                  while (band != 0u && at < p.band_cap) {
                    const int i = __ffs(band) - 1;
                    band &= band - 1;
                    p.band_rows[at] = x_global[u];
                    p.band_cols[at] = p.y_offset + (col0 + i) * p.y_stride;
                    ++at;
                  }
                }
              }
            }
            if constexpr (MODE == GMAX) {
              float m = -CUDART_INF_F;
              if (in == 0xffffffffu) {
#pragma unroll
                for (int i = 0; i < 32; ++i) m = fmaxf(m, __uint_as_float(r[c][i]));
              } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) m = i < left ? fmaxf(m, __uint_as_float(r[c][i])) : m;
              }
              if (valid[u]) p.gmax[static_cast<size_t>(x_global[u]) * p.groups + (col0 >> 5)] = m;
            }
            if constexpr (MODE == COLLECT) {
              uint32_t take = above(r[c], lo[u]) & in;
              while (take) {
                const int i = __ffs(take) - 1;
                take &= take - 1;
                const float s = pick(r[c], i);
                const size_t base = static_cast<size_t>(x_global[u]) * (p.cand_cap + p.tie_cap);
                int at;
                bool fits;
                if (p.tie_cap == 0) {
                  at = atomicAdd(p.cand_count + x_global[u], 1);
                  fits = at < p.cand_cap;
                } else if (s > hi[u]) {
                  at = atomicAdd(p.cand_count + 2 * x_global[u], 1);
                  fits = at < p.cand_cap;
                } else {       // equal to the floor: any tie_cap of them will do
                  at = atomicAdd(p.cand_count + 2 * x_global[u] + 1, 1);
                  fits = at < p.tie_cap;
                  at += p.cand_cap;
                }
                if (fits) {
                  p.cand_score[base + at] = s;
                  p.cand_idx[base + at] = p.y_offset + (col0 + i) * p.y_stride;
                }
              }
            }
          }
        }
      }
      if (!ok) break;
      if constexpr (MODE == COUNT || MODE == BAND) {
#pragma unroll
        for (int u = 0; u < UN; ++u)
          if (valid[u] && cnt[u] != 0 && p.greater != nullptr) atomicAdd(p.greater + x_global[u], cnt[u]);
      }
      w += n;
      ++seg;
    }
    if (!ok) fail(ST_TIMEOUT_EPILOGUE);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D, int MODE, bool SPLIT>
static int launch(RankParams& p, const void* y, const void* y_lo, int num_ctas, cudaStream_t stream) {
  using C = Cfg<D, SPLIT>;
  auto kern = rank_tiles_kernel<D, MODE, SPLIT>;
  static bool configured[64] = {false};   // the attribute is per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  CUtensorMap ty, tl;
  int rc = make_tmap_bf16(&ty, y, p.y_rows, D, C::BY);
  if (rc) return rc;
  rc = make_tmap_bf16(&tl, SPLIT ? y_lo : y, p.y_rows, D, C::BY);
  if (rc) return rc;
  p.nx_tiles = (p.x_rows + C::XR - 1) / C::XR;
  p.ny_tiles = (p.y_rows + C::BY - 1) / C::BY;
  p.map = TileMap::make(p.nx_tiles, p.ny_tiles, C::PARTS * C::Y_BYTES, 48ll << 20);
  if (num_ctas <= 0) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    num_ctas = sms;
  }
  const long long total = static_cast<long long>(p.nx_tiles) * p.ny_tiles;
  if (num_ctas > total) num_ctas = static_cast<int>(total);
  kern<<<num_ctas, THREADS, C::SMEM_BYTES, stream>>>(ty, tl, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

template <int D>
static int dispatch(RankParams& p, int mode, const void* y, const void* y_lo, int num_ctas, cudaStream_t s) {
  switch (mode) {
    case COUNT: return launch<D, COUNT, false>(p, y, y_lo, num_ctas, s);
    case BAND: return p.x_lo != nullptr ? launch<D, BAND, true>(p, y, y_lo, num_ctas, s) : launch<D, BAND, false>(p, y, y_lo, num_ctas, s);
    case GMAX: return launch<D, GMAX, false>(p, y, y_lo, num_ctas, s);
    default: return launch<D, COLLECT, false>(p, y, y_lo, num_ctas, s);
  }
}

static int rank_tiles(int mode, RankParams& p, const void* y, const void* y_lo, int D, int num_ctas, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(p.x) & 15) || (reinterpret_cast<uintptr_t>(p.x_lo) & 15) ||
      (reinterpret_cast<uintptr_t>(y) & 15) || (reinterpret_cast<uintptr_t>(y_lo) & 15))
    return -5;
  if ((p.x_lo == nullptr) != (y_lo == nullptr)) return -7;
  switch (D) {
    case 256: return dispatch<256>(p, mode, y, y_lo, num_ctas, s);
    case 128: return dispatch<128>(p, mode, y, y_lo, num_ctas, s);
    case 64: return dispatch<64>(p, mode, y, y_lo, num_ctas, s);
    default: return -6;
  }
}

// One warp per query: sets the bits of its known answers.  The answers come either as a CSR over the batch (ptr, cols) or are
// looked up by pair (a, b) in a CSR over sorted keys a * num_b + b.
struct MaskParams {
  int n;
  const long long* ptr;
  const int* cols;
  const long long* ab;         // pairs [n, stride]: a in column 0, b in column 1
  long long ab_stride, num_b;
  const long long* keys;
  long long num_keys;
  const long long* offsets;
  const long long* values;
  uint32_t* mask;
  long long stride;
  int y_rows;
  uint32_t* repeated;          // bits of the entries whose answer their list has named before, list i from word
                               // ptr[i] / 32 + i on; may be null
};

__global__ void __launch_bounds__(256) filter_mask_kernel(const MaskParams p) {
  const int lane = threadIdx.x & 31;
  const long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (i >= p.n) return;
  long long beg, end;
  if (p.ptr != nullptr) {
    beg = p.ptr[i];
    end = p.ptr[i + 1];
  } else {
    const long long key = p.ab[i * p.ab_stride] * p.num_b + p.ab[i * p.ab_stride + 1];
    // 32 probes per step; the first index with keys[index] >= key lies in [lo, hi]
    long long lo = 0, hi = p.num_keys;
    while (hi - lo > 0) {
      const long long step = (hi - lo + 32) / 33;
      const long long at = lo + step * (lane + 1) - 1;
      const bool below = at < hi && p.keys[at] < key;
      const int c = __popc(__ballot_sync(0xffffffffu, below));   // probes below the key form a prefix
      const long long nlo = lo + step * c;
      const long long nhi = c < 32 ? lo + step * (c + 1) - 1 : hi;
      lo = nlo;
      hi = nhi < hi ? nhi : hi;
    }
    if (lo >= p.num_keys || p.keys[lo] != key) return;
    beg = p.offsets[lo];
    end = p.offsets[lo + 1];
  }
  uint32_t* row = p.mask + i * p.stride;
  uint32_t* rep = p.repeated != nullptr ? p.repeated + beg / 32 + i : nullptr;
  for (long long b0 = beg; b0 < end; b0 += 128) {   // four loads in flight: popular pairs have thousands of answers
    long long c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long e = b0 + 32 * j + lane;
      c[j] = e >= end ? -1 : p.ptr != nullptr ? static_cast<long long>(p.cols[e]) : p.values[e];
    }
    bool again[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      again[j] = false;
      if (c[j] >= 0 && c[j] < p.y_rows) {
        const uint32_t bit = 1u << (c[j] & 31);
        if (rep == nullptr) atomicOr(row + (c[j] >> 5), bit);   // no value to wait for (8 us a batch of 4096 popular pairs)
        else again[j] = (atomicOr(row + (c[j] >> 5), bit) & bit) != 0u;
      }
    }
    if (rep != nullptr) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t bits = __ballot_sync(0xffffffffu, again[j]);
        if (lane == 0 && b0 + 32 * j < end) rep[(b0 - beg) / 32 + j] = bits;
      }
    }
  }
}

// Rows of fp32 [n, d] as hi + lo in bf16, zero-padded to d_pad columns, an fp32 copy of that width (optional) and
// margin[row] = |row| * factor + offset (optional).  One warp per row.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ src, long long src_stride, long long n, int d,
                                                         int d_pad, __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo,
                                                         float* __restrict__ copy, float* __restrict__ margin, float factor, float offset) {
  const int lane = threadIdx.x & 31;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long i = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    float sq = 0.f;
    for (int c = lane; c < d_pad; c += 32) {
      const float v = c < d ? src[i * src_stride + c] : 0.f;
      const __nv_bfloat16 h = __float2bfloat16_rn(v);
      const float rest = v - __bfloat162float(h);
      hi[i * d_pad + c] = h;
      lo[i * d_pad + c] = isfinite(rest) ? __float2bfloat16_rn(rest) : __float2bfloat16_rn(0.f);
      if (copy != nullptr) copy[i * d_pad + c] = v;
      sq = fmaf(v, v, sq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0 && margin != nullptr) margin[i] = sqrtf(sq) * factor + offset;
  }
}

}  // namespace rankk
}  // namespace dice

// greater[row] += columns of X Yᵀ (+ col_bias) above target[row]; with margin only those above target + margin, the ones
// within +-margin go to the band list.  x_lo / y_lo: second bf16 terms of the operands (band form only).  The column of
// target_idx[row] and the columns in mask (words of 32 columns, mask_stride per row) are left out.
extern "C" int dice_rank_count(const void* x, const void* x_lo, int x_rows, const void* y, const void* y_lo, int y_rows, int D,
                               const float* target, const int* target_idx, const float* col_bias, int y_offset, int y_stride,
                               const unsigned int* mask, long long mask_stride, int* greater, const float* margin,
                               int* band_rows, int* band_cols, unsigned long long* band_count, long long band_cap,
                               int* status, int num_ctas, void* stream) {
  using namespace dice::rankk;
  if (x_rows <= 0 || y_rows <= 0) return 0;
  if (target == nullptr || (greater == nullptr && margin == nullptr)) return -7;   // a band may be listed without counts
  if (margin != nullptr ? (band_rows == nullptr || band_cols == nullptr || band_count == nullptr) : x_lo != nullptr) return -7;
  RankParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.x_lo = static_cast<const __nv_bfloat16*>(x_lo);
  p.x_rows = x_rows;
  p.y_rows = y_rows;
  p.target = target;
  p.target_idx = target_idx;
  p.col_bias = col_bias;
  p.y_offset = y_offset;
  p.y_stride = y_stride > 0 ? y_stride : 1;
  p.mask = mask;
  p.mask_stride = mask_stride;
  p.greater = greater;
  p.margin = margin;
  p.band_rows = band_rows;
  p.band_cols = band_cols;
  p.band_count = band_count;
  p.band_cap = band_cap;
  p.status = status;
  return rank_tiles(margin != nullptr ? BAND : COUNT, p, y, y_lo, D, num_ctas, static_cast<cudaStream_t>(stream));
}

// gmax[row, g] = largest score of columns [32 g, 32 g + 32) (-inf for padding); groups must be 4 * ceil(y_rows / 128).
extern "C" int dice_rank_group_max(const void* x, int x_rows, const void* y, int y_rows, int D, const float* col_bias,
                                   float* gmax, int groups, int* status, int num_ctas, void* stream) {
  using namespace dice::rankk;
  if (x_rows <= 0 || y_rows <= 0) return 0;
  if (gmax == nullptr || groups != 4 * ((y_rows + 127) / 128)) return -7;
  RankParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.x_rows = x_rows;
  p.y_rows = y_rows;
  p.col_bias = col_bias;
  p.y_stride = 1;
  p.gmax = gmax;
  p.groups = groups;
  p.status = status;
  return rank_tiles(GMAX, p, y, nullptr, D, num_ctas, static_cast<cudaStream_t>(stream));
}

// Appends every column with a score >= floor[row] to the row's list of cand_cap + tie_cap entries: with tie_cap > 0 scores
// above the floor from the front (counted in cand_count[2 row]) and up to tie_cap equal ones behind cand_cap
// (cand_count[2 row + 1]), otherwise all of them from the front (cand_count[row]).
extern "C" int dice_rank_collect(const void* x, int x_rows, const void* y, int y_rows, int D, const float* col_bias, int y_offset,
                                 int y_stride, const float* floor, int cand_cap, int tie_cap, float* cand_score, int* cand_idx,
                                 int* cand_count, int* status, int num_ctas, void* stream) {
  using namespace dice::rankk;
  if (x_rows <= 0 || y_rows <= 0) return 0;
  if (floor == nullptr || cand_cap < 0 || tie_cap < 0 || cand_score == nullptr || cand_idx == nullptr || cand_count == nullptr) return -7;
  RankParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.x_rows = x_rows;
  p.y_rows = y_rows;
  p.col_bias = col_bias;
  p.y_offset = y_offset;
  p.y_stride = y_stride > 0 ? y_stride : 1;
  p.floor = floor;
  p.cand_cap = cand_cap;
  p.tie_cap = tie_cap;
  p.cand_score = cand_score;
  p.cand_idx = cand_idx;
  p.cand_count = cand_count;
  p.status = status;
  return rank_tiles(COLLECT, p, y, nullptr, D, num_ctas, static_cast<cudaStream_t>(stream));
}

// Sets the mask bits of the known answers of n queries: of (ptr [n + 1], cols), or with ptr == null of the pairs ab (two
// leading columns, row stride ab_stride) found in keys / offsets / values.  The mask is cleared by the caller.  repeated (with
// ptr, optional): one bit per entry of cols, set where its list has named the answer before (dice_eval_sparse reads it); the
// words of list i start at ptr[i] / 32 + i, which no two lists share; ptr[n] / 32 + n words, need not be cleared.
extern "C" int dice_filter_mask(int n, const long long* ptr, const int* cols, const long long* ab, long long ab_stride,
                                long long num_b, const long long* keys, long long num_keys, const long long* offsets,
                                const long long* values, unsigned int* mask, long long mask_stride, int y_rows, unsigned int* repeated,
                                void* stream) {
  using namespace dice::rankk;
  if (n <= 0) return 0;
  if (mask == nullptr || mask_stride * 32 < y_rows || (repeated != nullptr && ptr == nullptr)) return -7;
  if (ptr == nullptr ? (ab == nullptr || (num_keys > 0 && (keys == nullptr || offsets == nullptr || values == nullptr))) : cols == nullptr)
    return -7;
  const MaskParams p{n, ptr, cols, ab, ab_stride, num_b, keys, num_keys, offsets, values, mask, mask_stride, y_rows, repeated};
  filter_mask_kernel<<<(n + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int dice_split_rows(const float* src, long long src_stride, long long n, int d, int d_pad, void* hi, void* lo,
                               float* copy, float* margin, float factor, float offset, void* stream) {
  using namespace dice::rankk;
  if (n <= 0) return 0;
  if (d <= 0 || d > d_pad || src == nullptr || hi == nullptr || lo == nullptr) return -6;
  long long blocks = (n + 7) / 8;
  if (blocks > 148 * 16) blocks = 148 * 16;
  split_rows_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      src, src_stride, n, d, d_pad, static_cast<__nv_bfloat16*>(hi), static_cast<__nv_bfloat16*>(lo), copy, margin, factor, offset);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
