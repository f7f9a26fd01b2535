// route.cuh - one token's top-k experts and routing weights by one warp
// (src/moe_kernels.rs:1019-1081, src/oss_kernels.rs:15-35, src/ds4.rs:1371-1426,
// src/q4x.rs:2213-2231). Two spellings of one definition, the same operations in the same
// order: pm_route_scores keeps a token's experts in registers (the decode kernel, which ranks
// them itself), pm_route_warp in shared memory with every loop rolled (all other kernels). The
// group selection and the weights are one function for both.
#pragma once

#include "common.cuh"

// float -> unsigned key with the same order (finite values; -0 is folded onto
// +0 first so that equal floats get equal keys). Maxima over keys are maxima
// over the floats, bit for bit.
__device__ __forceinline__ uint32_t pm_fkey(float v) {
  uint32_t u = __float_as_uint(__fadd_rn(v, 0.0f));
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float pm_funkey(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Group-limited selection (this repository's definition): a group's score = the sum of its two largest biased scores, the
// second no lower than PM_NEG; the best topk_group groups stay, ties -> lower group index. These two say it step by
// step, for one thread; the warp-wide forms below give the same and leave what is no number (a NaN in a bias or a router
// row) to them.
__device__ __forceinline__ float pm_group_score(const float *sv, int gs) {
  int i1 = 0;
  float v1 = sv[0], v2 = PM_NEG;
#pragma unroll 1
  for (int i = 1; i < gs; i++)
    if (sv[i] > v1) { v1 = sv[i]; i1 = i; }
#pragma unroll 1
  for (int i = 0; i < gs; i++)
    if (i != i1 && sv[i] > v2) v2 = sv[i];
  return __fadd_rn(v1, v2);
}
__device__ __forceinline__ void pm_group_keep(const float *gsc, int G, int topk_group, unsigned char *keep) {
#pragma unroll 1
  for (int g = 0; g < G; g++) keep[g] = 0;
#pragma unroll 1
  for (int r = 0; r < topk_group; r++) {
    int bg = -1;
    float bv = 0.0f;
#pragma unroll 1
    for (int g = 0; g < G; g++) {
      if (keep[g]) continue;
      const float v = gsc[g];
      if (bg < 0 || v > bv) { bv = v; bg = g; }
    }
    keep[bg] = 1;
  }
}
// the score of a group of 32 from its scores, one a lane (sv: the same in memory); all lanes get it
__device__ __forceinline__ float pm_group_score32(float v, const float *sv) {
  if (__any_sync(PM_FULL, v != v)) return pm_group_score(sv, 32);
  const uint32_t key = pm_fkey(v), m1 = __reduce_max_sync(PM_FULL, key);
  const uint32_t top = __ballot_sync(PM_FULL, key == m1);
  const uint32_t m2 = __reduce_max_sync(PM_FULL, key == m1 && !(top & (top - 1)) ? 0u : key);
  return __fadd_rn(pm_funkey(m1), fmaxf(pm_funkey(m2), PM_NEG));
}
// one warp: which of G groups stay
__device__ __forceinline__ void pm_group_rank(const float *gsc, int G, int topk_group, int lane, unsigned char *keep) {
  bool odd = false;
#pragma unroll 1
  for (int g = lane; g < G; g += 32) {  // kept when fewer than topk_group groups come before it
    const float mine = gsc[g];
    int before = 0;
#pragma unroll 1
    for (int j = 0; j < G; j++) {
      const float v = gsc[j];
      before += v > mine || (v == mine && j < g);
    }
    keep[g] = before < topk_group;
    odd = odd || mine != mine;
  }
  if (__any_sync(PM_FULL, odd)) {
    __syncwarp();
    if (lane == 0) pm_group_keep(gsc, G, topk_group, keep);
  }
}

// Scores of one token by one warp (decode kernel). Lane L holds experts L, L+32, ... (NP per lane,
// NP*32 >= E); `lg` points at the token's E logits (any address space); ssv[E],
// gsc[E/2], keep[E/2] are per-warp scratch in shared memory (group-limited
// selection only). Out: pr[] = the score the weight is taken from, key[] = the
// ordered key of what the selection ranks (score + bias, masked groups lowest).
template <int NP>
__device__ __forceinline__ void pm_route_scores(const pm_layer_desc &D, const float *lg,
                                                const float *__restrict__ sel_bias, int lane,
                                                float *ssv, float *gsc, unsigned char *keep,
                                                float pr[NP], uint32_t key[NP]) {
  const int E = D.n_exp;
  float sv[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) {
    int e = lane + 32 * i;
    pr[i] = e < E ? lg[e] : PM_NEG;
  }
  if (D.gating == PM_GATE_SOFTMAX_ALL) {  // src/moe_kernels.rs:1023-1042
    float mx = PM_NEG;
#pragma unroll
    for (int i = 0; i < NP; i++) mx = fmaxf(mx, pr[i]);
    mx = pm_funkey(__reduce_max_sync(PM_FULL, pm_fkey(mx)));
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < NP; i++) {
      if (lane + 32 * i < E) {
        pr[i] = pm_exp(__fsub_rn(pr[i], mx));
        sum = __fadd_rn(sum, pr[i]);
      }
    }
    sum = pm_warp_sum_16_1(sum);
#pragma unroll
    for (int i = 0; i < NP; i++) pr[i] = __fdiv_rn(pr[i], sum);
  } else if (D.gating == PM_GATE_SIGMOID) {  // src/moe_kernels.rs:1034
#pragma unroll
    for (int i = 0; i < NP; i++)
      if (lane + 32 * i < E) pr[i] = __fdiv_rn(1.0f, __fadd_rn(1.0f, pm_exp(-pr[i])));
  } else if (D.gating == PM_GATE_SQRT_SOFTPLUS) {  // src/ds4.rs:1377-1379
#pragma unroll
    for (int i = 0; i < NP; i++)
      if (lane + 32 * i < E) {
        float v = pr[i];
        float sp = v > 20.0f ? v : pm_log1p(pm_exp(v));
        pr[i] = __fsqrt_rn(sp);
      }
  }
  // what the selection ranks: score (+ bias) (src/moe_kernels.rs:1044-1049)
#pragma unroll
  for (int i = 0; i < NP; i++) {
    int e = lane + 32 * i;
    sv[i] = e < E ? (sel_bias ? __fadd_rn(pr[i], sel_bias[e]) : pr[i]) : PM_NEG;
  }
  if (D.n_group > 0) {
#pragma unroll
    for (int i = 0; i < NP; i++)
      if (lane + 32 * i < E) ssv[lane + 32 * i] = sv[i];
    __syncwarp();
    const int G = D.n_group, gs = E / G;
    if (gs == 32) {  // a group is one register of the warp: two reductions find its two largest scores
#pragma unroll
      for (int i = 0; i < NP; i++)
        if (i < G) {
          const float s = pm_group_score32(sv[i], ssv + 32 * i);
          if (lane == i) gsc[i] = s;
        }
    } else {
      for (int g = lane; g < G; g += 32) gsc[g] = pm_group_score(ssv + g * gs, gs);  // lane g scores groups g, g+32, ...
    }
    __syncwarp();
    pm_group_rank(gsc, G, D.topk_group, lane, keep);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NP; i++) {
      int e = lane + 32 * i;
      if (e < E && !keep[e / gs]) sv[i] = PM_NEG;
    }
  }
#pragma unroll
  for (int i = 0; i < NP; i++) key[i] = pm_fkey(sv[i]);
}

// The routing weight of pick k = lane (< K) from the picked scores in selection
// order sel_p[0..K) (src/moe_kernels.rs:1072-1074, src/oss_kernels.rs:31-32,
// src/ds4.rs:1416-1424). Sums run in k order, every lane repeats them.
__device__ __forceinline__ float pm_route_weight(const pm_layer_desc &D, const float *sel_p,
                                                 int k) {
  const int K = D.top_k;
  float x;
  if (D.gating == PM_GATE_SOFTMAX_SELECTED) {
    float evsum = 0.0f, mine = 0.0f;
    for (int j = 0; j < K; j++) {
      float ev = pm_exp(__fsub_rn(sel_p[j], sel_p[0]));
      evsum = __fadd_rn(evsum, ev);
      if (j == k) mine = ev;
    }
    x = __fdiv_rn(mine, evsum);
  } else {
    float wsum = 0.0f;
    for (int j = 0; j < K; j++) wsum = __fadd_rn(wsum, sel_p[j]);
    x = sel_p[k];
    if (D.gating == PM_GATE_SQRT_SOFTPLUS) x = __fdiv_rn(x, wsum);
    else if (D.norm_w) x = __fdiv_rn(x, fmaxf(wsum, 6.103515625e-5f));
  }
  if (D.w_scale != 0.0f) x = __fmul_rn(x, D.w_scale);
  return x;
}

// The same routing with a token's scores in shared memory and every loop rolled. A kernel that routes a few tokens runs
// each instruction once or a few times, cold: unrolled over registers (256 experts: 8 a lane, with the exponentials and
// divisions of every gating) one token took 8.7 us of waiting for instructions.
// Floats of scratch a token: scores, ranked scores, group scores, group marks, the picks' scores.
__host__ __device__ inline int pm_route_scratch(int E) { return 2 * E + E / 2 + (E / 2 + 3) / 4 + PM_MAX_TOPK; }
// elementwise part of the gating (mx: the largest logit, softmax over all experts only)
__device__ __forceinline__ float pm_route_elem(int gating, float v, float mx) {
  if (gating == PM_GATE_SOFTMAX_ALL) return pm_exp(__fsub_rn(v, mx));
  if (gating == PM_GATE_SIGMOID) return __fdiv_rn(1.0f, __fadd_rn(1.0f, pm_exp(-v)));
  if (gating == PM_GATE_SQRT_SOFTPLUS) return __fsqrt_rn(v > 20.0f ? v : pm_log1p(pm_exp(v)));
  return v;
}
// one warp: the largest of E logits; the sum of E scores (lane L adds L, L + 32, ... in order, then the lanes)
__device__ __forceinline__ float pm_route_max(const float *lg, int E, int lane) {
  float mx = PM_NEG;
#pragma unroll 1
  for (int e = lane; e < E; e += 32) mx = fmaxf(mx, lg[e]);
  return pm_funkey(__reduce_max_sync(PM_FULL, pm_fkey(mx)));
}
__device__ __forceinline__ float pm_route_sum(const float *pr, int E, int lane) {
  float sum = 0.0f;
#pragma unroll 1
  for (int e = lane; e < E; e += 32) sum = __fadd_rn(sum, pr[e]);
  return pm_warp_sum_16_1(sum);
}
// one warp: group mask, K picks and their weights from a token's scores pr[E] and ranked scores sv[E] (sv is used up);
// rest: the scratch behind them. Lane k < K writes ids_out[k], w_out[k].
__device__ __forceinline__ void pm_route_pick(const pm_layer_desc &D, const float *pr, float *sv, float *rest, int lane,
                                              uint32_t *ids_out, float *w_out) {
  const int E = D.n_exp, K = D.top_k;
  float *gsc = rest, *sel_p = rest + E / 2 + (E / 2 + 3) / 4;
  unsigned char *keep = (unsigned char *)(rest + E / 2);
  if (D.n_group > 0) {
    const int G = D.n_group, gs = E / G;
    if (gs == 32) {
#pragma unroll 1
      for (int g = 0; g < G; g++) {
        const float s = pm_group_score32(sv[32 * g + lane], sv + 32 * g);
        if (lane == 0) gsc[g] = s;
      }
    } else {
#pragma unroll 1
      for (int g = lane; g < G; g += 32) gsc[g] = pm_group_score(sv + g * gs, gs);
    }
    __syncwarp();
    pm_group_rank(gsc, G, D.topk_group, lane, keep);
    __syncwarp();
#pragma unroll 1
    for (int e = lane; e < E; e += 32)
      if (!keep[gs == 32 ? e >> 5 : e / gs]) sv[e] = PM_NEG;
  }
  // K rounds of (max, lowest index) (src/moe_kernels.rs:1053-1067) on ordered integer keys; a lane keeps the best of
  // its own experts and looks for the next one only when it has lost it
  uint32_t best = 0, at = 0xffffffffu, mine = 0;
  auto look = [&] {
    best = lane < E ? pm_fkey(sv[lane]) : 0u;
    at = lane < E ? (uint32_t)lane : 0xffffffffu;
#pragma unroll 4
    for (int e = lane + 32; e < E; e += 32) {
      const uint32_t k = pm_fkey(sv[e]);
      if (k > best) {
        best = k;
        at = (uint32_t)e;
      }
    }
  };
  look();
#pragma unroll 1
  for (int k = 0; k < K; k++) {
    const uint32_t m = __reduce_max_sync(PM_FULL, best);
    const uint32_t e = __reduce_min_sync(PM_FULL, best == m ? at : 0xffffffffu);
    if (lane == k) mine = e;
    if (at == e) {
      sv[e] = PM_NEG;
      look();
    }
  }
  if (lane < K) sel_p[lane] = pr[mine];
  __syncwarp();
  if (lane < K) {
    ids_out[lane] = mine;
    w_out[lane] = pm_route_weight(D, sel_p, lane);
  }
}
// the whole routing of one token by one warp; sc: pm_route_scratch(E) floats
__device__ __forceinline__ void pm_route_warp(const pm_layer_desc &D, const float *lg, const float *__restrict__ sel_bias, int lane,
                                              float *sc, uint32_t *ids_out, float *w_out) {
  const int E = D.n_exp;
  float *pr = sc, *sv = sc + E;
  const bool soft = D.gating == PM_GATE_SOFTMAX_ALL;
  const float mx = soft ? pm_route_max(lg, E, lane) : 0.0f;
#pragma unroll 1
  for (int e = lane; e < E; e += 32) pr[e] = pm_route_elem(D.gating, lg[e], mx);
  const float sum = soft ? pm_route_sum(pr, E, lane) : 1.0f;
#pragma unroll 1
  for (int e = lane; e < E; e += 32) {
    const float p = soft ? __fdiv_rn(pr[e], sum) : pr[e];
    pr[e] = p;
    sv[e] = sel_bias ? __fadd_rn(p, sel_bias[e]) : p;
  }
  __syncwarp();
  pm_route_pick(D, pr, sv, sc + 2 * E, lane, ids_out, w_out);
}
