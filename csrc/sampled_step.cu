// Training step on sampled candidates (negative sampling, 1vsSample, KvsSample) against one table, in two launches:
//
//   dice_sampled_grad     draws the corruptions (counter-based generator), gathers and composes the query, scores it
//                         against its candidates, BCE-with-logits loss, gradients of all rows
//   dice_sampled_update   optimiser sweep over the entity rows (dense, or only the rows with a gradient), the relations
//                         and the coefficient; closes the step
//
// A *group* is one fixed vector F and its C candidate rows.  With corrupted tails F is the composed query h o r; with
// corrupted heads the score is bilinear in the head, so F is the same product seen from the other side (the chain rule
// of the composition applied to the tail), and the C heads are the candidates.  Either way a triple costs one row read
// and one dot product, and the relation and the fixed entity get ONE gradient row per group instead of one per triple.
//
// What bounds it: the candidate rows (random 4 D-byte reads) and the optimiser's passes over table and moments.  The
// gradient rows of drawn entities are never formed in memory where they have a chain: such an entity's triples are linked
// (list head per row, one 8-byte node {next, g} per triple) and the update adds up g * F (F: [groups, D], resident in
// L2) while it holds the row in registers.  That takes out the read-modify-write of a gradient row per triple and the
// update's read and clear of the gradient table (8 passes over the touched rows become 6).  Only uniformly drawn
// entities are chained, so a chain has a Poisson length; the positives' entities, whose degrees are heavy-tailed, and
// candidates given by the caller go through red.add into the gradient table and a flag per row.
//
// Measured against the launch sequence lookup / score / backward / sweeps (one triple per query, scalar atomics), whole step:
// 10 000 positives x 11, D = 128, 123 182 rows, 37 relations 655 -> 123 us; 1024 x 100 given candidates, D = 256, 14 541 rows
// 132 -> 74 us; 32 768 x 129, D = 128, 5 million rows, sparse 5280 -> 2730 us (the update of 2.9 million rows moves 8.7 GB
// in 1.9 ms).
#include "algebra.cuh"
#include "dice_b200.h"
#include "optim.cuh"
#include "philox.cuh"
#include "ptx_sm100.cuh"

namespace dice {
namespace sampled {

enum Draw : int { DRAW_GIVEN = 0, DRAW_CORRUPT = 1, DRAW_TAILS = 2 };

struct GradParams {
  const long long* h;          // DRAW_GIVEN: head and relation ids, query n at [n * idx_stride]
  const long long* r;
  long long idx_stride;
  const long long* cand;       // DRAW_GIVEN: candidate c of query n at [n * cand_stride + c]
  long long cand_stride;
  const float* labels;         // DRAW_GIVEN: [N, C]
  const long long* pos;        // otherwise: positive triples [N, 3]; candidate 0 is the positive itself
  int N, C, draw;
  unsigned long long seed, offset;
  const long long* step;       // added to offset
  float label_pos, label_neg;
  const float* ent;            // [NE, D]
  float* g_ent;                // [NE, D] red.add
  unsigned char* touched;      // [NE] rows of g_ent that received something
  int* list_head;              // [NE] first node of the row's chain or -1; null = no chains
  int2* nodes;                 // [N * C] {next, g as bits}
  float* fixed;                // [N, D] F of every group (chains only)
  const float* rel;
  float* g_rel;
  const float* coeff;
  float* g_coeff;
  double* loss;
  int* status;
  long long num_entities, num_relations;
  float scale, margin, eps;
  int D, norm_mode, translation, split;
};

// A lane's share of a row: positions (c * 32 + lane) * V + u of each of the K blocks of width w.
template <int K, int V, int NC>
struct Frag {
  float x[K][NC][V];
};

#define FRAG_LOOP(k, c, u)                            \
  _Pragma("unroll") for (int k = 0; k < K; ++k)       \
  _Pragma("unroll") for (int c = 0; c < NC; ++c)      \
  _Pragma("unroll") for (int u = 0; u < V; ++u)

template <int K, int V, int NC>
__device__ __forceinline__ void frag_zero(Frag<K, V, NC>& f) {
  FRAG_LOOP(k, c, u) f.x[k][c][u] = 0.f;
}

template <int K, int V, int NC>
__device__ __forceinline__ void frag_load(const float* __restrict__ row, int w, int lane, Frag<K, V, NC>& f) {
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = (c * 32 + lane) * V;
      if (j < w) {   // w is a multiple of 4
        const float* s = row + k * w + j;
        if constexpr (V == 4) {
          const float4 t = *reinterpret_cast<const float4*>(s);
          f.x[k][c][0] = t.x; f.x[k][c][1] = t.y; f.x[k][c][2] = t.z; f.x[k][c][3] = t.w;
        } else if constexpr (V == 2) {
          const float2 t = *reinterpret_cast<const float2*>(s);
          f.x[k][c][0] = t.x; f.x[k][c][1] = t.y;
        } else {
          f.x[k][c][0] = *s;
        }
      } else {
#pragma unroll
        for (int u = 0; u < V; ++u) f.x[k][c][u] = 0.f;
      }
    }
}

template <int K, int V, int NC>
__device__ __forceinline__ void frag_store(float* __restrict__ row, int w, int lane, const Frag<K, V, NC>& f) {
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = (c * 32 + lane) * V;
      if (j < w) {
        float* s = row + k * w + j;
        if constexpr (V == 4) *reinterpret_cast<float4*>(s) = make_float4(f.x[k][c][0], f.x[k][c][1], f.x[k][c][2], f.x[k][c][3]);
        else if constexpr (V == 2) *reinterpret_cast<float2*>(s) = make_float2(f.x[k][c][0], f.x[k][c][1]);
        else *s = f.x[k][c][0];
      }
    }
}

// row += s * f
template <int K, int V, int NC>
__device__ __forceinline__ void frag_red(float* row, int w, int lane, const Frag<K, V, NC>& f, float s) {
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = (c * 32 + lane) * V;
      if (j < w) {
        float* d = row + k * w + j;
        if constexpr (V == 4) red_add_v4(d, s * f.x[k][c][0], s * f.x[k][c][1], s * f.x[k][c][2], s * f.x[k][c][3]);
        else if constexpr (V == 2) red_add_v2(d, s * f.x[k][c][0], s * f.x[k][c][1]);
        else atomicAdd(d, s * f.x[k][c][0]);
      }
    }
}

// q_k = sum_a sgn(k, a) h_a r_idx(k, a)
template <int K, int V, int NC>
__device__ __forceinline__ void compose(const Frag<K, V, NC>& h, const Frag<K, V, NC>& r, Frag<K, V, NC>& q) {
  FRAG_LOOP(k, c, u) {
    float s = 0.f;
#pragma unroll
    for (int a = 0; a < K; ++a) s = fmaf(Alg<K>::sgn(k, a) * h.x[a][c][u], r.x[Alg<K>::idx(k, a)][c][u], s);
    q.x[k][c][u] = s;
  }
}
// gradient of <dq, h o r> with respect to h, and to r
template <int K, int V, int NC>
__device__ __forceinline__ void compose_dh(const Frag<K, V, NC>& dq, const Frag<K, V, NC>& r, Frag<K, V, NC>& dh) {
  frag_zero(dh);
  FRAG_LOOP(k, c, u) {
#pragma unroll
    for (int a = 0; a < K; ++a)
      dh.x[a][c][u] = fmaf(Alg<K>::sgn(k, a) * dq.x[k][c][u], r.x[Alg<K>::idx(k, a)][c][u], dh.x[a][c][u]);
  }
}
template <int K, int V, int NC>
__device__ __forceinline__ void compose_dr(const Frag<K, V, NC>& dq, const Frag<K, V, NC>& h, Frag<K, V, NC>& dr) {
  frag_zero(dr);
  FRAG_LOOP(k, c, u) {
#pragma unroll
    for (int a = 0; a < K; ++a) {
      const int b = Alg<K>::idx(k, a);
      dr.x[b][c][u] = fmaf(Alg<K>::sgn(k, a) * dq.x[k][c][u], h.x[a][c][u], dr.x[b][c][u]);
    }
  }
}

// Sum of v over the four consecutive positions a 4-tuple consists of (V of them in this lane).
template <int V>
__device__ __forceinline__ float tuple4_sum(float v) {
  if constexpr (V <= 2) v += __shfl_xor_sync(0xffffffffu, v, 1);
  if constexpr (V == 1) v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}

// r -> r / norm, keeping the norms for the way back (positions past the block width w stay zero)
template <int K, int V, int NC>
__device__ __forceinline__ void normalise(int mode, int w, int lane, Frag<K, V, NC>& r, Frag<K, V, NC>& nrm) {
  if (mode == NORM_ACROSS_BLOCKS) {
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int u = 0; u < V; ++u) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) s += r.x[k][c][u] * r.x[k][c][u];
        const float n = (c * 32 + lane) * V < w ? sqrtf(s) : 1.f;
#pragma unroll
        for (int k = 0; k < K; ++k) { r.x[k][c][u] /= n; nrm.x[k][c][u] = n; }
      }
  } else if (mode == NORM_CONSECUTIVE4) {
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float s = 0.f;
#pragma unroll
        for (int u = 0; u < V; ++u) s += r.x[k][c][u] * r.x[k][c][u];
        const float n = fmaxf(sqrtf(tuple4_sum<V>(s)), 1e-12f);
#pragma unroll
        for (int u = 0; u < V; ++u) { r.x[k][c][u] /= n; nrm.x[k][c][u] = n; }
      }
  }
}
// dr = (drh - rh <drh, rh>) / norm, in place
template <int K, int V, int NC>
__device__ __forceinline__ void normalise_bwd(int mode, const Frag<K, V, NC>& rh, const Frag<K, V, NC>& nrm,
                                              Frag<K, V, NC>& d) {
  if (mode == NORM_ACROSS_BLOCKS) {
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int u = 0; u < V; ++u) {
        float dot = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) dot += d.x[k][c][u] * rh.x[k][c][u];
#pragma unroll
        for (int k = 0; k < K; ++k) d.x[k][c][u] = (d.x[k][c][u] - rh.x[k][c][u] * dot) / nrm.x[k][c][u];
      }
  } else if (mode == NORM_CONSECUTIVE4) {
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float dot = 0.f;
#pragma unroll
        for (int u = 0; u < V; ++u) dot += d.x[k][c][u] * rh.x[k][c][u];
        dot = tuple4_sum<V>(dot);
#pragma unroll
        for (int u = 0; u < V; ++u) d.x[k][c][u] = (d.x[k][c][u] - rh.x[k][c][u] * dot) / nrm.x[k][c][u];
      }
  }
}

// Sums of CH values over the warp: afterwards every lane holds the sum of value lane / (32 / CH).  CH - 1 shuffles for
// the first log2(CH) steps instead of CH each.
template <int CH>
__device__ __forceinline__ float transpose_sum(float (&a)[CH], int lane) {
  int m = 16;
#pragma unroll
  for (int half = CH / 2; half > 0; half >>= 1, m >>= 1) {
    const bool up = (lane & m) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = up ? a[i + half] : a[i];
      const float give = up ? a[i] : a[i + half];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
    }
  }
  float v = a[0];
#pragma unroll
  for (int o = 16 / CH; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int GRAD_THREADS = 256;
// Candidate rows in flight (of up to 128 floats) and resident blocks per SM.  Measured (4, 4) / (8, 2): 32 768 x 129 on 5
// million rows, D = 128: 609 / 660 us, 10 000 x 11: 30 / 39 us.  Measured at D = 128 only: four blocks leave 64 registers, at
// which most widths spill (116 to 144 bytes of stores per thread at D = 128, 320 to 400 at 256, up to 830 at 512), and two
// blocks would leave room for all but the widest.
constexpr int GRAD_CH = 4;
constexpr int GRAD_B = 4;

// One warp per part of a group (`split` parts share the candidates of a group where there are few groups).  CH candidate
// rows are in flight at a time.
template <int K, int V, int NC>
__global__ void __launch_bounds__(GRAD_THREADS, GRAD_B) grad_kernel(const GradParams p) {
  using F = Frag<K, V, NC>;
  constexpr int PL = K * V * NC;                       // floats of a row per lane
  constexpr int CH = PL <= 4 ? GRAD_CH : PL <= 8 ? GRAD_CH / 2 : GRAD_CH / 4;
  constexpr int LPC = 32 / CH;                         // lanes that end up with a candidate's score
  const int lane = threadIdx.x & 31;
  const int w = p.D / K;
  const Philox rng(p.seed);
  const unsigned long long offset = p.offset + (p.step != nullptr ? static_cast<unsigned long long>(*p.step) : 0ull);
  const bool heads = p.draw == DRAW_CORRUPT && (rng(~0ull, offset).x & 1u) != 0u;   // one coin per batch
  const bool chained = p.list_head != nullptr;
  const float coef = p.coeff != nullptr ? *p.coeff : 1.f;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const long long items = static_cast<long long>(p.N) * p.split;
  double loss_local = 0.0;
  float dc = 0.f;

  for (long long item = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; item < items; item += warps) {
    const int n = static_cast<int>(item / p.split), part = static_cast<int>(item % p.split);
    const int c_lo = static_cast<int>(static_cast<long long>(p.C) * part / p.split);
    const int c_hi = static_cast<int>(static_cast<long long>(p.C) * (part + 1) / p.split);
    long long fix_id, rel_id, true_id = -1;
    if (p.draw == DRAW_GIVEN) {
      fix_id = p.h[n * p.idx_stride];
      rel_id = p.r[n * p.idx_stride];
    } else {
      const long long* t = p.pos + 3ll * n;
      fix_id = heads ? t[2] : t[0];
      rel_id = t[1];
      true_id = heads ? t[0] : t[2];
    }
    if (fix_id < 0 || fix_id >= p.num_entities || rel_id < 0 || rel_id >= p.num_relations) {
      if (lane == 0) atomicCAS(p.status, 0, ST_BAD_INDEX);
      continue;   // no chain points at the group's nodes
    }

    F fix, rel, nrm, fv, acc;
    frag_load<K, V, NC>(p.ent + fix_id * p.D, w, lane, fix);
    frag_load<K, V, NC>(p.rel + rel_id * p.D, w, lane, rel);
    normalise(p.norm_mode, w, lane, rel, nrm);
    if (p.coeff != nullptr) {   // Keci Cl(0,1): the vector parts of head and relation are scaled by the coefficient
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int u = 0; u < V; ++u) {
          rel.x[K - 1][c][u] *= coef;
          if (!heads) fix.x[K - 1][c][u] *= coef;
        }
    }
    // fix / rel now hold the scaled values.  fv is F of the scores: dot product <F, row> or distance |F - row|
    if (p.translation) {
      FRAG_LOOP(k, c, u) {
        const float f = heads ? fix.x[k][c][u] - (rel.x[k][c][u] + p.eps) : fix.x[k][c][u] + rel.x[k][c][u] + p.eps;
        fv.x[k][c][u] = (c * 32 + lane) * V < w ? f : 0.f;   // positions past the row width must not count as a distance
      }
    } else if (heads) {
      compose_dh(fix, rel, fv);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int u = 0; u < V; ++u) fv.x[K - 1][c][u] *= coef;
    } else {
      compose(fix, rel, fv);
    }
    if (chained && part == 0) frag_store<K, V, NC>(p.fixed + static_cast<size_t>(n) * p.D, w, lane, fv);
    frag_zero(acc);

    for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
      // ids and labels of up to 32 candidates, one per lane
      const int c = c0 + lane;
      long long id = -1;
      float y = 0.f;
      if (c < c_hi) {
        if (p.draw == DRAW_GIVEN) {
          id = p.cand[n * p.cand_stride + c];
          y = p.labels[static_cast<size_t>(n) * p.C + c];
        } else if (c == 0) {
          id = true_id;
          y = p.label_pos;
        } else {
          y = p.label_neg;
          if (p.draw == DRAW_CORRUPT) {
            const uint4 x = rng(static_cast<unsigned long long>(n) + static_cast<unsigned long long>(c) * p.N, offset);
            id = bounded(x.x, x.y, p.num_entities);
          } else {
            const unsigned long long f = static_cast<unsigned long long>(n) * (p.C - 1) + (c - 1);
            const uint4 x = rng(f >> 1, offset);
            id = (f & 1) ? bounded(x.z, x.w, p.num_entities) : bounded(x.x, x.y, p.num_entities);
          }
        }
        if (id < 0 || id >= p.num_entities) {
          atomicCAS(p.status, 0, ST_BAD_INDEX);
          id = -1;
        }
      }
      // a drawn entity's chain: the link is exchanged now, its value is only needed when the node is written
      const bool listed = chained && c > 0 && id >= 0;
      const int node = n * p.C + c;   // N * C fits 31 bits (checked on the host)
      int next = -1;
      if (listed) next = atomicExch(p.list_head + id, node);
      float g_mine = 0.f;
      const int count = min(32, c_hi - c0);
      for (int s0 = 0; s0 < count; s0 += CH) {
        F row[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) {   // -1 past the end or out of range: the group's own fixed row stands in (with g = 0 it
          const long long e = __shfl_sync(0xffffffffu, id, s0 + j);   // adds nothing, unless it is inf or NaN, as is then the group)
          frag_load<K, V, NC>(p.ent + (e < 0 ? fix_id : e) * p.D, w, lane, row[j]);
        }
        float a[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) {
          float s = 0.f;
          if (p.translation) {
            FRAG_LOOP(k, cc, u) { const float x = fv.x[k][cc][u] - row[j].x[k][cc][u]; s = fmaf(x, x, s); }
          } else {
            FRAG_LOOP(k, cc, u) s = fmaf(fv.x[k][cc][u], row[j].x[k][cc][u], s);
          }
          a[j] = s;
        }
        float s = transpose_sum<CH>(a, lane);           // this lane's candidate: s0 + lane / LPC
        const int mine = s0 + lane / LPC;
        const float label = __shfl_sync(0xffffffffu, y, mine);
        const long long my_id = __shfl_sync(0xffffffffu, id, mine);
        float dist = 0.f;
        if (p.translation) {
          dist = sqrtf(s);
          s = p.margin - dist;
        }
        float g = 0.f;
        if (my_id >= 0) {
          const float z = expf(-fabsf(s));
          if (lane % LPC == 0) loss_local += static_cast<double>(fmaxf(s, 0.f) - s * label + log1pf(z));
          const float sig = s >= 0.f ? 1.f / (1.f + z) : z / (1.f + z);
          g = (sig - label) * p.scale;
          if (p.translation) g = dist > 0.f ? -g / dist : 0.f;
        }
        const float spread = __shfl_sync(0xffffffffu, g, (lane % CH) * LPC);
        if (lane / CH == s0 / CH) g_mine = spread;
#pragma unroll
        for (int j = 0; j < CH; ++j) {
          const float gj = __shfl_sync(0xffffffffu, g, j * LPC);
          if (p.translation) {
            FRAG_LOOP(k, cc, u) row[j].x[k][cc][u] = fv.x[k][cc][u] - row[j].x[k][cc][u];
          }
          FRAG_LOOP(k, cc, u) acc.x[k][cc][u] = fmaf(gj, row[j].x[k][cc][u], acc.x[k][cc][u]);
          if (!chained || c0 + s0 + j == 0) {   // uniform
            const long long e = __shfl_sync(0xffffffffu, id, s0 + j);
            if (e >= 0) {
              if (p.translation) frag_red<K, V, NC>(p.g_ent + e * p.D, w, lane, row[j], -gj);
              else frag_red<K, V, NC>(p.g_ent + e * p.D, w, lane, fv, gj);
            }
          }
        }
      }
      if (listed) p.nodes[node] = make_int2(next, __float_as_int(g_mine));
      else if (id >= 0) p.touched[id] = 1;
    }

    // back through F to the fixed entity and the relation
    F dfix, drel;
    if (p.translation) {
      // acc = sum g' (F - row).  tails: dq = acc, dh = dr = dq.  heads: F - row = -(h + r + eps - t), so dq = -acc, dt = acc
      FRAG_LOOP(k, c, u) { dfix.x[k][c][u] = acc.x[k][c][u]; drel.x[k][c][u] = heads ? -acc.x[k][c][u] : acc.x[k][c][u]; }
    } else if (heads) {
      // acc = sum g h (unscaled heads).  F[K-1] carries a factor coef that the derivative with respect to the coefficient
      // does not have
      if (p.coeff != nullptr) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int u = 0; u < V; ++u) {
            float without = 0.f;
#pragma unroll
            for (int k = 0; k < K; ++k)
              without = fmaf(Alg<K>::sgn(k, K - 1) * fix.x[k][c][u], rel.x[Alg<K>::idx(k, K - 1)][c][u], without);
            dc = fmaf(without, acc.x[K - 1][c][u], dc);
            acc.x[K - 1][c][u] *= coef;
          }
      }
      compose(acc, rel, dfix);
      compose_dr(fix, acc, drel);
    } else {
      compose_dh(acc, rel, dfix);
      compose_dr(acc, fix, drel);
      if (p.coeff != nullptr) {
        const float* raw = p.ent + fix_id * p.D + (K - 1) * w;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int u = 0; u < V; ++u) {
            const int j = (c * 32 + lane) * V + u;
            if (j < w) dc = fmaf(dfix.x[K - 1][c][u], raw[j], dc);
            dfix.x[K - 1][c][u] *= coef;
          }
      }
    }
    if (p.coeff != nullptr) {
      const float* raw = p.rel + rel_id * p.D + (K - 1) * w;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int u = 0; u < V; ++u) {
          const int j = (c * 32 + lane) * V + u;
          if (j < w) dc = fmaf(drel.x[K - 1][c][u], raw[j], dc);
          drel.x[K - 1][c][u] *= coef;
        }
    }
    normalise_bwd(p.norm_mode, rel, nrm, drel);
    frag_red<K, V, NC>(p.g_ent + fix_id * p.D, w, lane, dfix, 1.f);
    frag_red<K, V, NC>(p.g_rel + rel_id * p.D, w, lane, drel, 1.f);
    if (lane == 0) p.touched[fix_id] = 1;
  }

  // one reduction per block for the loss and the coefficient
  __shared__ double s_loss[GRAD_THREADS / 32];
  __shared__ float s_dc[GRAD_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    loss_local += __shfl_xor_sync(0xffffffffu, loss_local, o);
    dc += __shfl_xor_sync(0xffffffffu, dc, o);
  }
  if (lane == 0) {
    s_loss[threadIdx.x >> 5] = loss_local;
    s_dc[threadIdx.x >> 5] = dc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double l = 0.0;
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < GRAD_THREADS / 32; ++i) { l += s_loss[i]; d += s_dc[i]; }
    if (l != 0.0) atomicAdd(p.loss, l * p.scale);
    if (p.g_coeff != nullptr && d != 0.f) atomicAdd(p.g_coeff, d);
  }
}

// ------------------------------------------------------------------------------------------------ update
struct UpdateParams {
  float* E;
  float* gE;
  float* mE;
  float* vE;
  unsigned char* touched;
  int* list_head;            // or null
  const int2* nodes;
  const float* fixed;
  long long rows;
  int D, C, translation, chunk;
  float* P[2];               // relation table, coefficient (or null)
  float* gP[2];
  float* mP[2];
  float* vP[2];
  long long nP[2];
  float lr, beta1, beta2, eps, weight_decay;
  double* loss;
  float* loss_out;
  long long* step;
  unsigned int* done;        // zero-initialised; the last block closes the step and clears it
};

constexpr int UPDATE_THREADS = 256;
// Resident blocks per SM and float4s in flight per thread.  Measured (8, 1) / (6, 1) / (5, 1) / (4, 2): 123 182 rows x 128
// 82 / 102 / 96 / 117 us, 14 541 x 256 25 / 35 / 34 / 38 us, sparse 2.9 of 5 million rows x 128 1893 / 1994 / 1937 / 2147 us.
constexpr int UPDATE_B = 8;
constexpr int UPDATE_R = 1;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

template <int KIND>
__device__ __forceinline__ void update4(const UpdateParams& p, const OptStepConsts& c, float4& w, const float4& g, float4& m,
                                        float4& v) {
  w.x = opt_update(KIND, w.x, g.x, m.x, v.x, p.lr, p.beta1, p.beta2, p.eps, p.weight_decay, c.inv_bc1, c.inv_sqrt_bc2, c.clip, c.first_step);
  w.y = opt_update(KIND, w.y, g.y, m.y, v.y, p.lr, p.beta1, p.beta2, p.eps, p.weight_decay, c.inv_bc1, c.inv_sqrt_bc2, c.clip, c.first_step);
  w.z = opt_update(KIND, w.z, g.z, m.z, v.z, p.lr, p.beta1, p.beta2, p.eps, p.weight_decay, c.inv_bc1, c.inv_sqrt_bc2, c.clip, c.first_step);
  w.w = opt_update(KIND, w.w, g.w, m.w, v.w, p.lr, p.beta1, p.beta2, p.eps, p.weight_decay, c.inv_bc1, c.inv_sqrt_bc2, c.clip, c.first_step);
}

// g += s * F, or for distances -s * (F - w) with the row's own values w
__device__ __forceinline__ void add_triple(bool translation, float s, const float4& f, const float4& w, float4& g) {
  if (translation) {
    g.x = fmaf(-s, f.x - w.x, g.x); g.y = fmaf(-s, f.y - w.y, g.y);
    g.z = fmaf(-s, f.z - w.z, g.z); g.w = fmaf(-s, f.w - w.w, g.w);
  } else {
    g.x = fmaf(s, f.x, g.x); g.y = fmaf(s, f.y, g.y); g.z = fmaf(s, f.z, g.z); g.w = fmaf(s, f.w, g.w);
  }
}

// A block takes `chunk` <= 256 consecutive rows.  One thread per row reads the row's flag and list head, clears them and
// follows the links of the first CHAIN triples (their latencies overlap over the rows); the rows to update (all of them, or
// with SPARSE the ones with a gradient) are compacted into shared memory in row order.  Then the float4s of these rows are
// dealt to the threads, with nothing dependent left to load: walking a chain while holding the row left
// the memory system idle (5M rows x 128, 2.9M of them touched, TransE: 2734 us).
constexpr int CHAIN = 6;

template <bool SPARSE, int KIND>
__device__ __forceinline__ void update_rows(const UpdateParams& p, const OptStepConsts& c) {
  constexpr int R = UPDATE_R;
  __shared__ float s_g[UPDATE_THREADS][CHAIN];
  __shared__ int s_n[UPDATE_THREADS][CHAIN];
  __shared__ int s_rest[UPDATE_THREADS];             // first node of a longer chain's rest, or -1
  __shared__ unsigned short s_row[UPDATE_THREADS];   // row of the chunk; bit 15: has a gradient row; bits 8..10: triples
  __shared__ int s_count[UPDATE_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tpr = p.D / 4;
  for (long long base = static_cast<long long>(blockIdx.x) * p.chunk; base < p.rows;
       base += static_cast<long long>(gridDim.x) * p.chunk) {
    const long long mine = base + threadIdx.x;
    const bool in = threadIdx.x < p.chunk && mine < p.rows;
    bool dense = false;
    int node = -1;
    if (in) {
      dense = p.touched[mine] != 0;
      if (p.list_head != nullptr) node = p.list_head[mine];
      if (dense) p.touched[mine] = 0;
      if (node >= 0) p.list_head[mine] = -1;
    }
    const bool flag = SPARSE ? dense || node >= 0 : in;
    const unsigned int bits = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) s_count[warp] = __popc(bits);
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int i = 0; i < UPDATE_THREADS / 32; ++i) {
      const int n = s_count[i];
      if (i < warp) before += n;
      total += n;
    }
    if (flag) {
      const int at = before + __popc(bits & ((1u << lane) - 1u));
      int links = 0;
#pragma unroll
      for (int l = 0; l < CHAIN; ++l) {
        if (node < 0) break;
        const int2 nd = p.nodes[node];
        s_n[at][l] = node / p.C;
        s_g[at][l] = __int_as_float(nd.y);
        node = nd.x;
        ++links;
      }
      s_rest[at] = node;
      s_row[at] = static_cast<unsigned short>(threadIdx.x | (links << 8) | (dense ? 0x8000 : 0));
    }
    __syncthreads();
    const int items = total * tpr;
    for (int q0 = threadIdx.x; q0 < items; q0 += UPDATE_THREADS * R) {
      float4 w[R], m[R], v[R], g[R];
      size_t off[R];
      int at[R], d[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int q = q0 + j * UPDATE_THREADS < items ? q0 + j * UPDATE_THREADS : q0;
        at[j] = q / tpr;
        d[j] = (q - at[j] * tpr) * 4;
        const int rc = s_row[at[j]];
        off[j] = static_cast<size_t>(base + (rc & 0xff)) * p.D + d[j];
        w[j] = ld4(p.E + off[j]);
        m[j] = v[j] = g[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (KIND != 2) { m[j] = ld4_once(p.mE + off[j]); v[j] = ld4_once(p.vE + off[j]); }
        if ((rc & 0x8000) && (j == 0 || q != q0)) {
          g[j] = ld4(p.gE + off[j]);
          st4(p.gE + off[j], make_float4(0.f, 0.f, 0.f, 0.f));
        }
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int links = (s_row[at[j]] >> 8) & 7;
        for (int l = 0; l < links; ++l)
          add_triple(p.translation, s_g[at[j]][l], ld4(p.fixed + static_cast<size_t>(s_n[at[j]][l]) * p.D + d[j]), w[j], g[j]);
        for (int rest = links == CHAIN ? s_rest[at[j]] : -1; rest >= 0;) {
          const int2 nd = p.nodes[rest];
          add_triple(p.translation, __int_as_float(nd.y), ld4(p.fixed + static_cast<size_t>(rest / p.C) * p.D + d[j]), w[j], g[j]);
          rest = nd.x;
        }
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (j > 0 && q0 + j * UPDATE_THREADS >= items) continue;
        update4<KIND>(p, c, w[j], g[j], m[j], v[j]);
        st4(p.E + off[j], w[j]);
        if (KIND != 2) { st4_once(p.mE + off[j], m[j]); st4_once(p.vE + off[j], v[j]); }
      }
    }
    __syncthreads();   // the lists are rebuilt for the next chunk
  }
}

template <bool SPARSE, int KIND>
__global__ void __launch_bounds__(UPDATE_THREADS, UPDATE_B) update_kernel(const UpdateParams p) {
  const long long t = *p.step + 1;
  const OptStepConsts c = opt_step_consts(KIND, t, p.beta1, p.beta2);
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (p.P[s] == nullptr) continue;
    for (long long i = tid; i < p.nP[s]; i += stride) {
      const float g = p.gP[s][i];
      p.gP[s][i] = 0.f;
      float m = 0.f, v = 0.f;
      if (KIND != 2) { m = p.mP[s][i]; v = p.vP[s][i]; }
      p.P[s][i] = opt_update(KIND, p.P[s][i], g, m, v, p.lr, p.beta1, p.beta2, p.eps, p.weight_decay, c.inv_bc1,
                             c.inv_sqrt_bc2, c.clip, c.first_step);
      if (KIND != 2) { p.mP[s][i] = m; p.vP[s][i] = v; }
    }
  }
  update_rows<SPARSE, KIND>(p, c);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(p.done, 1u) == gridDim.x - 1) {   // every block has read the step counter
      *p.loss_out = static_cast<float>(*p.loss);
      *p.loss = 0.0;
      *p.step = t;
      *p.done = 0u;
    }
  }
}

template <int K, int V, int NC>
static int launch_grad(const GradParams& p, cudaStream_t s) {
  const long long warps = static_cast<long long>(p.N) * p.split;
  long long blocks = (warps * 32 + GRAD_THREADS - 1) / GRAD_THREADS;
  if (blocks > 148 * 64) blocks = 148 * 64;
  grad_kernel<K, V, NC><<<static_cast<unsigned>(blocks), GRAD_THREADS, 0, s>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// The narrowest vector that covers a block with the 32 lanes: V = 1, 2 or 4, then several chunks of V = 4.
template <int K>
static int dispatch_grad(const GradParams& p, cudaStream_t s) {
  const int w = p.D / K;
  if (w <= 32) return launch_grad<K, 1, 1>(p, s);
  if (w <= 64) return launch_grad<K, 2, 1>(p, s);
  if constexpr (K <= 4) {
    if (w <= 128) return launch_grad<K, 4, 1>(p, s);
  }
  if constexpr (K <= 2) {
    if (w <= 256) return launch_grad<K, 4, 2>(p, s);
  }
  if constexpr (K == 1) {
    if (w <= 512) return launch_grad<K, 4, 4>(p, s);
  }
  return -6;
}

}  // namespace sampled
}  // namespace dice

// Gradients of one step.  draw 0: query n = (h[n * idx_stride], r[n * idx_stride]) against cand[n * cand_stride + c] with
// labels [N, C]; 1: positives pos [N, 3], C - 1 corruptions each, one coin per batch replaces all heads or all tails; 2: the
// same with uniformly drawn tails (the numbers of dice_neg_sample mode 0 and of dice_uniform_int for the same seed and
// offset + *step).  model: 0 DistMult, 1 ComplEx, 2 QMult, 3 OMult, 4 Keci Cl(0,1), 5 translation.  Gradients are added to
// g_ent (rows flagged in touched), g_rel and *g_coeff, the loss to *loss; with list_head (draws 1 and 2 only) drawn entities
// are chained for dice_sampled_update instead, which needs nodes [N * C], fixed [N, D] and list_head filled with -1.
extern "C" int dice_sampled_grad(int model, int normalize, int draw, const long long* h, const long long* r,
                                 long long idx_stride, const long long* cand, long long cand_stride, const float* labels,
                                 const long long* pos, int N, int C, unsigned long long seed, unsigned long long offset,
                                 const long long* step, float label_pos, float label_neg, const float* ent, float* g_ent,
                                 unsigned char* touched, int* list_head, void* nodes, float* fixed, long long num_entities,
                                 const float* rel, float* g_rel, long long num_relations, const float* coeff, float* g_coeff,
                                 double* loss, float scale, float margin, float eps, int D, int* status, void* stream) {
  using namespace dice;
  using namespace dice::sampled;
  if (N <= 0 || C <= 0) return 0;
  if (D <= 0 || D > 512 || draw < 0 || draw > 2 || num_entities <= 0 || num_relations <= 0) return -6;
  if (draw == DRAW_GIVEN ? (h == nullptr || r == nullptr || cand == nullptr || labels == nullptr || list_head != nullptr)
                         : pos == nullptr)
    return -6;
  if (list_head != nullptr && (nodes == nullptr || fixed == nullptr || static_cast<long long>(N) * C > 0x7fffffffll)) return -6;
  const uintptr_t al = reinterpret_cast<uintptr_t>(ent) | reinterpret_cast<uintptr_t>(g_ent) | reinterpret_cast<uintptr_t>(rel) |
                       reinterpret_cast<uintptr_t>(g_rel) | reinterpret_cast<uintptr_t>(fixed);
  if ((al & 15) || (reinterpret_cast<uintptr_t>(nodes) & 7)) return -5;
  const int K = model == 1 || model == 4 ? 2 : model == 2 ? 4 : model == 3 ? 8 : 1;
  if (D % (4 * K)) return -6;
  GradParams p{h, r, idx_stride, cand, cand_stride, labels, pos, N, C, draw, seed, offset, step, label_pos, label_neg, ent,
               g_ent, touched, list_head, static_cast<int2*>(nodes), fixed, rel, g_rel, nullptr, nullptr, loss, status,
               num_entities, num_relations, scale, margin, eps, D, NORM_NONE, 0, 1};
  // Few groups: several warps share one, so that about 16 warps per SM have rows in flight, with at least eight
  // candidates per warp (below that the fixed vector and its gradient rows cost more than the candidates).
  while (static_cast<long long>(N) * p.split < 148 * 16 && C / (p.split * 2) >= 8) p.split *= 2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (model) {
    case 0: return dispatch_grad<1>(p, s);
    case 1: return dispatch_grad<2>(p, s);
    case 2: p.norm_mode = normalize ? NORM_CONSECUTIVE4 : NORM_NONE; return dispatch_grad<4>(p, s);
    case 3: p.norm_mode = normalize ? NORM_ACROSS_BLOCKS : NORM_NONE; return dispatch_grad<8>(p, s);
    case 4: p.coeff = coeff; p.g_coeff = g_coeff; return dispatch_grad<2>(p, s);
    case 5: p.translation = 1; return dispatch_grad<1>(p, s);
    default: return -6;
  }
}

// Optimiser step behind dice_sampled_grad (C, D, translation and the chain arguments as there).  sparse != 0 updates only
// rows with a gradient (lazily decayed moments; kinds 0 Adam, 1 AdamW, 2 SGD), otherwise every row (also 3 ADOPT).
// Gradients, flags and list heads are left cleared; *loss_out = *loss, *loss = 0, *step += 1.  done: zero-initialised.
extern "C" int dice_sampled_update(int kind, int sparse, float* E, float* gE, float* mE, float* vE, unsigned char* touched,
                                   int* list_head, const void* nodes, const float* fixed, long long rows, int D, int C,
                                   int translation, float* R, float* gR, float* mR, float* vR, long long nR, float* coeff,
                                   float* gC, float* mC, float* vC, long long nC, float lr, float beta1, float beta2,
                                   float eps, float weight_decay, double* loss, float* loss_out, long long* step,
                                   unsigned int* done, void* stream) {
  using namespace dice;
  using namespace dice::sampled;
  if (rows <= 0 || D <= 0 || D % 4 || D > 512 || C <= 0 || kind < 0 || kind > 3 || (sparse && kind == 3)) return -6;
  const uintptr_t al = reinterpret_cast<uintptr_t>(E) | reinterpret_cast<uintptr_t>(gE) | reinterpret_cast<uintptr_t>(mE) |
                       reinterpret_cast<uintptr_t>(vE) | reinterpret_cast<uintptr_t>(fixed);
  if (al & 15) return -5;
  UpdateParams p{E, gE, mE, vE, touched, list_head, static_cast<const int2*>(nodes), fixed, rows, D, C, translation, 0,
                 {R, coeff}, {gR, gC}, {mR, mC}, {vR, vC}, {nR, nC}, lr, beta1, beta2, eps, weight_decay,
                 loss, loss_out, step, done};
  // as many blocks as are resident (148 SMs x UPDATE_B), each with the same number of equally long chunks: a partial second
  // wave of blocks costs as much as a full one
  const long long resident = 148ll * UPDATE_B;
  const long long passes = (rows + resident * UPDATE_THREADS - 1) / (resident * UPDATE_THREADS);
  p.chunk = static_cast<int>((rows + resident * passes - 1) / (resident * passes));
  long long blocks = (rows + p.chunk - 1) / p.chunk;
  const long long other = (nR + UPDATE_THREADS - 1) / UPDATE_THREADS;
  if (blocks < other) blocks = other;
  if (blocks > resident) blocks = resident;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const dim3 grid(static_cast<unsigned>(blocks));
  switch (sparse ? 4 + kind : kind) {
    case 0: update_kernel<false, 0><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
    case 1: update_kernel<false, 1><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
    case 2: update_kernel<false, 2><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
    case 3: update_kernel<false, 3><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
    case 4: update_kernel<true, 0><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
    case 5: update_kernel<true, 1><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
    default: update_kernel<true, 2><<<grid, UPDATE_THREADS, 0, s>>>(p); break;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
