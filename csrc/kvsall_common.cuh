// Pieces of the tensor-core scoring kernel (kvsall_fused.cu) that do not depend on its tile sizes: launch parameters, the cursor over
// a CTA's range of tiles, and the epilogue arithmetic that turns logits into loss terms and dS.
#pragma once
#include "dice_b200.h"
#include "ptx_sm100.cuh"
#include "tile_map.cuh"

namespace dice {

struct KvsAllParams {
  float* out;           // [x_rows, D] fp32, accumulated with red.add
  double* loss;         // scalar accumulator (may be null when LOSS == false)
  int* status;          // 0 = ok, otherwise first failure code
  int x_rows, y_rows;   // valid row counts
  int nx_tiles, ny_tiles;
  TileMap map;          // visiting order of the (x tile, y tile) pairs
  float base;           // label value outside the positives (smoothing term)
  float scale;          // factor applied to out (1 / (B * |E|) for a mean-reduced loss)
  const uint32_t* mask; // MASK: bit y of row x set where (x, y) is a positive label; row stride mask_stride words
  int mask_stride;      // (a multiple of 4; a thread reads one word per tile)
  float pos_delta;      // label(positive) - base
  long long* trace;     // optional [64 tiles][8] clock64 stamps written by CTA 0 (pipeline diagnostics), else null
  // SCORE != 0: the logit is a function of the dot product and one scalar per row of X and of Y
  const float* x_bias;  // [x_rows] or null (= 0): SCORE 1 bias of row x; SCORE 2 squared norm of row x
  const float* y_bias;  // the same for the rows of Y, or null (= 0); readable up to the next multiple of 128 rows
  float* x_dsum;        // optional [x_rows]: += scale * sum over y of the value fed to the second GEMM
  float margin;         // SCORE 2: logit = margin - sqrt(|x|^2 + |y|^2 - 2 x.y)
  // Optimiser fused into the drain (opt.param != null): out is then the gradient buffer of the rows of X, and the CTA
  // whose partial sums complete an x tile (tile counters) updates those 128 rows at once: master weights, moments,
  // the bf16 rows that X itself is (no CTA reads a completed tile again) and clears the gradient.
  DiceFusedOptimizer opt;
};

__device__ __forceinline__ float fast_lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_tanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Position of one GEMM stream inside this CTA's range of flattened (x tile, y tile) pairs; a segment is a run of
// tiles sharing the x tile.
struct TileCursor {
  long long w, w_end;
  TileMap map;
  int x, y0, t, n;
  uint32_t seg;
  __device__ __forceinline__ void load() {
    int run;
    map.locate(w, x, y0, run);
    n = static_cast<int>(min(static_cast<long long>(run), w_end - w));
  }
  __device__ __forceinline__ void start(long long wb, long long we, const TileMap& m) {
    w = wb; w_end = we; map = m; t = 0; seg = 0; x = 0; y0 = 0; n = 0;
    if (w < w_end) load();
  }
  __device__ __forceinline__ bool done() const { return w >= w_end; }
  __device__ __forceinline__ bool first() const { return t == 0; }
  __device__ __forceinline__ bool last() const { return t + 1 == n; }
  __device__ __forceinline__ void advance() {
    if (++t == n) {
      w += n;
      ++seg;
      t = 0;
      if (w < w_end) load();
    }
  }
};

// One thread's 32 logits of a tile (bit i of mword is the label of logit i): dS = sigmoid(s) - label packed as bf16 pairs
// (low half = even column) and, with LOSS, the BCE-with-logits terms added to lacc.  FULL: all columns are valid entries
// of Y; otherwise the first y_valid are.
// SCORE selects how the logit follows from the dot product a = x.y of the tensor cores:
//   0  s = a
//   1  s = a + xb + yb[col]                     (per-query scalar terms of the Clifford models)
//   2  s = margin - sqrt(xb + yb[col] - 2 a)    (translational distance; xb, yb are squared norms).  The value handed
//      to the second GEMM is then dS / distance, and the caller subtracts (sum of those values) * x from the result:
//      d s / d x = (y - x) / distance.
// dsum accumulates the values handed to the second GEMM (SCORE != 0 only).
//
// Everything is derived from one hyperbolic tangent per logit, t = tanh(s / 2):
//   dS = sigmoid(s) - label = 0.5 t + c              with c = 0.5 - label (one of two constants)
//   sigmoid(|s|) = 0.5 (1 + |t|)  in [0.5, 1)        (no cancellation)
//   BCE(s, label) = softplus(s) - label s = c s + 0.5 |s| - ln 2 * (lg2(1 + |t|) - 1)
// and the three sums  sum c s,  sum |s|,  sum lg2(sigmoid(|s|))  are kept apart (lacc[0..2]) and combined once per segment.
// The last one is the logarithm of a product: the 32 factors 1 + |t| (each in [1, 2), so the product stays below 2^32)
// are multiplied up and ONE logarithm is taken per call.
//
// The epilogue is bound by instruction issue (all its warps share four schedulers), so it works on pairs of logits with
// the packed fp32 operations (two results per issued instruction), and the label of a logit costs nothing where no lane
// of the warp has a positive among its 32 columns: positives are a few per thousand logits, so most warps take that
// path (`any` is uniform in the warp).  5.5 issued instructions per logit with the loss and 2.5 without, against 15 and 8
// of the scalar form with a select per logit; one of them is the special-function tanh (16 results per clock and SM).
template <bool LOSS, bool LABELS, bool FULL, int SCORE>
__device__ __forceinline__ void epilogue_pairs(const uint32_t (&r)[32], uint32_t mword, float c_base, float delta,
                                               int y_valid, uint32_t (&packed)[16], float (&lacc)[3], float xb,
                                               const float* __restrict__ yb, float margin, float& dsum) {
  const uint64_t half2 = pack2(0.5f, 0.5f), c2 = pack2(c_base, c_base), zero2 = pack2(0.f, 0.f);
  uint64_t s_sum = zero2, prod = pack2(1.f, 1.f), d_sum = zero2;
  float abs0 = 0.f, abs1 = 0.f, pos_sum = 0.f;
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float s0 = __uint_as_float(r[i]), s1 = __uint_as_float(r[i + 1]);
    float g0 = 1.f, g1 = 1.f;
    if constexpr (SCORE == 1) { s0 += xb + yb[i]; s1 += xb + yb[i + 1]; }
    if constexpr (SCORE == 2) {
      const float a0 = fmaxf(fmaf(-2.f, s0, xb + yb[i]), 1e-12f), a1 = fmaxf(fmaf(-2.f, s1, xb + yb[i + 1]), 1e-12f);
      g0 = rsqrtf(a0);
      g1 = rsqrtf(a1);
      s0 = fmaf(-a0, g0, margin);
      s1 = fmaf(-a1, g1, margin);
    }
    if constexpr (!FULL) {   // a padded column counts as s = 0: t = 0, a factor of one, nothing added to the sums
      s0 = i < y_valid ? s0 : 0.f;
      s1 = i + 1 < y_valid ? s1 : 0.f;
    }
    const uint64_t s2 = pack2(s0, s1);
    float h0, h1;
    unpack2(mul2(s2, half2), h0, h1);
    const float t0 = fast_tanh(h0), t1 = fast_tanh(h1);
    uint64_t d2 = fma2(pack2(t0, t1), half2, c2);
    if constexpr (LOSS) {
      s_sum = add2(s_sum, s2);
      abs0 += fabsf(s0);
      abs1 += fabsf(s1);
      prod = mul2(prod, pack2(1.f + fabsf(t0), 1.f + fabsf(t1)));
    }
    float d0, d1;
    unpack2(d2, d0, d1);
    if constexpr (LABELS) {
      const bool p0 = (mword >> i) & 1u, p1 = (mword >> (i + 1)) & 1u;
      if (p0) d0 -= delta;
      if (p1) d1 -= delta;
      if constexpr (LOSS) {
        if (p0) pos_sum += s0;
        if (p1) pos_sum += s1;
      }
    }
    if constexpr (SCORE == 2) { d0 *= g0; d1 *= g1; }
    if constexpr (!FULL) {
      d0 = i < y_valid ? d0 : 0.f;
      d1 = i + 1 < y_valid ? d1 : 0.f;
    }
    if constexpr (SCORE != 0) d_sum = add2(d_sum, pack2(d0, d1));
    __nv_bfloat162 v = __floats2bfloat162_rn(d0, d1);  // .x (low 16 bits) = even K element
    packed[i >> 1] = *reinterpret_cast<uint32_t*>(&v);
  }
  if constexpr (LOSS) {
    float a, b;
    unpack2(s_sum, a, b);
    lacc[0] = fmaf(c_base, a + b, lacc[0]);
    if constexpr (LABELS) lacc[0] = fmaf(-delta, pos_sum, lacc[0]);
    lacc[1] += abs0 + abs1;
    unpack2(prod, a, b);
    lacc[2] += fast_lg2(a * b) - (FULL ? 32.f : static_cast<float>(max(0, min(y_valid, 32))));
  }
  if constexpr (SCORE != 0) {
    float a, b;
    unpack2(d_sum, a, b);
    dsum += a + b;
  }
}

template <bool LOSS, bool MASK, int SCORE>
__device__ __forceinline__ void epilogue_chunk(const uint32_t (&r)[32], uint32_t mword, float base, float delta,
                                               int y_valid, uint32_t (&packed)[16], float (&lacc)[3], float xb,
                                               const float* __restrict__ yb, float margin, float& dsum) {
  const float c_base = 0.5f - base;
  const bool any = MASK && __any_sync(0xffffffffu, mword != 0u);
  if (y_valid >= 32) {
    if (!any) epilogue_pairs<LOSS, false, true, SCORE>(r, mword, c_base, delta, 32, packed, lacc, xb, yb, margin, dsum);
    else epilogue_pairs<LOSS, MASK, true, SCORE>(r, mword, c_base, delta, 32, packed, lacc, xb, yb, margin, dsum);
  } else {
    epilogue_pairs<LOSS, MASK, false, SCORE>(r, mword, c_base, delta, y_valid, packed, lacc, xb, yb, margin, dsum);
  }
}

}  // namespace dice
