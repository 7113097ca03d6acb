// Routing of the MoE block: parameters of the router kernel and the per-token selection,
// shared with the expert projection kernel, which repeats the selection per CTA for single-row passes.
#pragma once
#include "common.cuh"

namespace b200 {

struct RouterParams {
  const __half* xn;                                // [M][H] ffn_norm output, fp16 (when h is null)
  const float* h; const float* gamma; const float* ss_in; int ss_n; float eps;  // or: normalise the residual rows here
  __half* xn_out;                                  // ... and leave the fp16 rows for the expert kernels (CTA 0)
  DTensor router;                                  // [nE][H], F32 / F16 / Q8_0 (planes)
  const float* sh_gate;                            // [H] F32
  int M, H, nE, used;
  float* logits;       // [M][nE]
  float* probs;        // optional [M][nE]: the softmax, for inspection
  int32_t* topk;       // [M][used]
  float* topk_w;       // [M][used+1] (last = sigmoid(shared gate))
  float* margin;       // [M] optional: (p_k - p_{k+1}) / p_k
  int4* entries; int* n_entries; int* cols;   // expert work list for the grouped kernels
  int* ticket;         // rows routed so far (left zero)
  int* pair_counts;    // [nE] pairs per expert, counted while the rows are routed (left zero)
  int* pair_pos;       // [M][used] place of a pair among its expert's, in the order of the counting
  int gate_done;       // the router kernel has left the shared expert's gate
  int4* gprob;         // optional [nE + 1]: {expert, first sorted row, rows, first sorted row} per expert (GemmProblem), the shared expert last
  int max_entries;
  int defer;           // the expert kernel that follows selects the experts itself
  int ecols;           // columns per work-list entry (8, or 4 for passes of some tens of rows; 0 means 8)
  // expert parallelism: the work list keeps the experts [e_lo, e_hi) only (e_hi == 0: all) and makes shared-expert
  // entries for the rows [sh_lo, sh_hi) only (sh_hi == 0: all rows)
  int e_lo, e_hi, sh_lo, sh_hi;
  int* n_pairs;        // optional: the number of (row, slot) pairs in cols (routed pairs of the kept experts + shared rows)
  int64_t* distinct;   // optional: += the number of experts this pass's work list touches (for the byte count of a step)
  Timeline tl;
};

#ifdef __CUDACC__
// softmax + top-k + weights of one token by one warp; a lane owns experts lane + 32*i in registers
// (reference: llm/moe.go:219-282, 426-443; shaders/llm_moe_route_decode.comp:84-213)
template <int NPL>
__device__ __forceinline__ int route_token(const RouterParams& p, int n, int lane, bool write, float2 (&cand)[32], int want_slot = -1) {
  int wanted = -1;
  const int nE = p.nE, used = p.used;
  float pv[NPL];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < NPL; i++) {
    const int e = lane + 32 * i;
    pv[i] = e < nE ? __ldcg(p.logits + (size_t)n * nE + e) : -INFINITY;
    mx = fmaxf(mx, pv[i]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < NPL; i++) { pv[i] = lane + 32 * i < nE ? expf(pv[i] - mx) : 0.f; sum += pv[i]; }
  sum = warp_sum(sum);
  const float inv = 1.0f / sum;
#pragma unroll
  for (int i = 0; i < NPL; i++) {
    pv[i] = lane + 32 * i < nE ? pv[i] * inv : -1.f;
    if (write && p.probs != nullptr && lane + 32 * i < nE) p.probs[(size_t)n * nE + lane + 32 * i] = pv[i];
  }
  // Logits that are not finite leave no probabilities to order: the first experts then, with weights that show it. The ids index
  // counters, work lists and weights without further checks, so they lie in [0, nE) whatever the logits.
  if (!(sum > 0.f)) {
    if (write) {
      if (lane < used) { p.topk[(size_t)n * used + lane] = lane; p.topk_w[(size_t)n * (used + 1) + lane] = inv; }
      if (lane == 0 && p.margin) p.margin[n] = 0.f;
    }
    return want_slot < used ? want_slot : -1;
  }
  // top-k by descending probability, ties to the lower index (llm/moe.go:249-252). The (used + 1)-th largest of the 32 lanes' own
  // maxima bounds the selection from below, and hardly more than used + 1 values reach that bound: those are put side by side, one
  // per lane in index order, and each finds its rank by comparing with all the others. (Eleven rounds of a warp-wide maximum over
  // 512 values took 5 us of a decode step's layer; this takes under one.)
  {
    float lm = pv[0];
#pragma unroll
    for (int i = 1; i < NPL; i++) lm = fmaxf(lm, pv[i]);
    int above = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const float o = __shfl_sync(0xffffffffu, lm, j);
      above += o > lm || (o == lm && j < lane);
    }
    const float bound = used < 32 ? __shfl_sync(0xffffffffu, lm, __ffs((int)__ballot_sync(0xffffffffu, above == used)) - 1) : -1.f;
    int n_cand = 0;
#pragma unroll
    for (int i = 0; i < NPL; i++) n_cand += __popc(__ballot_sync(0xffffffffu, pv[i] >= bound));
    if (bound >= 0.f && n_cand <= 32) {
      int at = 0;
#pragma unroll
      for (int i = 0; i < NPL; i++) {
        const uint32_t m = __ballot_sync(0xffffffffu, pv[i] >= bound);
        if (pv[i] >= bound) cand[at + __popc(m & ((1u << lane) - 1))] = make_float2(pv[i], __int_as_float(lane + 32 * i));
        at += __popc(m);
      }
      __syncwarp();
      const float v = lane < n_cand ? cand[lane].x : -1.f;
      const int idx = lane < n_cand ? __float_as_int(cand[lane].y) : 0;
      int rank = 0;
      for (int j = 0; j < n_cand; j++) {
        const float o = cand[j].x;
        rank += o > v || (o == v && j < lane);
      }
      if (lane >= n_cand) rank = 64;
      const uint32_t hit = __ballot_sync(0xffffffffu, rank == want_slot);
      const int wanted = __shfl_sync(0xffffffffu, idx, hit != 0 ? __ffs((int)hit) - 1 : 0);
      if (write) {
        __syncwarp();
        if (rank <= used) cand[rank].x = v;
        __syncwarp();
        if (rank < used) p.topk[(size_t)n * used + rank] = idx;
        float wsum = 0.f;
        for (int k = 0; k < used; k++) wsum += cand[k].x;
        if (lane == 0 && p.margin) p.margin[n] = cand[used - 1].x > 0.f ? (cand[used - 1].x - cand[used].x) / cand[used - 1].x : 0.f;
        if (wsum < 6.103515625e-5f) wsum = 6.103515625e-5f;   // normalise the weights (llm/moe.go:256-282)
        if (lane < used) p.topk_w[(size_t)n * (used + 1) + lane] = cand[lane].x / wsum;
        __syncwarp();
      }
      return hit != 0 ? wanted : -1;
    }
  }
  // many equal values, or fewer experts than lanes: one warp-wide maximum after the other. Probabilities are non-negative, so their
  // bit patterns order like unsigned integers: a warp-wide max of the values, then a warp-wide min of the indices that hold it.
  float wsum = 0.f, last_p = 0.f, myw = 0.f;
  for (int k = 0; k <= used; k++) {
    // the lane's maximum by a tree (depth log2 NPL), then the lowest of its slots that holds it
    float t[NPL];
#pragma unroll
    for (int i = 0; i < NPL; i++) t[i] = pv[i];
#pragma unroll
    for (int w = NPL / 2; w >= 1; w >>= 1) {
#pragma unroll
      for (int i = 0; i < w; i++) t[i] = fmaxf(t[i], t[i + w]);
    }
    const float bv = t[0];
    uint32_t eq = 0;
#pragma unroll
    for (int i = 0; i < NPL; i++) eq |= (pv[i] == bv ? 1u : 0u) << i;
    const int bi = __ffs((int)eq) - 1;
    const uint32_t key = bv < 0.f ? 0u : __float_as_uint(bv) + 1u;          // taken / absent entries sort last
    const uint32_t best = __reduce_max_sync(0xffffffffu, key);
    const uint32_t mine = key == best && best != 0u ? (uint32_t)(lane + 32 * bi) : 0x7fffffffu;
    const int widx = (int)__reduce_min_sync(0xffffffffu, mine);
    const float wv = best == 0u ? -1.f : __uint_as_float(best - 1u);
    if (k == used) {
      if (write && lane == 0 && p.margin) p.margin[n] = last_p > 0.f ? (last_p - fmaxf(wv, 0.f)) / last_p : 0.f;
      break;
    }
    if ((widx & 31) == lane) {
#pragma unroll
      for (int i = 0; i < NPL; i++) if (i == (widx >> 5)) pv[i] = -1.f;
    }
    if (k == want_slot) wanted = widx;
    if (lane == k) { myw = wv; if (write) p.topk[(size_t)n * used + k] = widx; }
    wsum += wv; last_p = wv;
  }
  // normalise the weights (llm/moe.go:256-282)
  if (wsum < 6.103515625e-5f) wsum = 6.103515625e-5f;
  if (write && lane < used) p.topk_w[(size_t)n * (used + 1) + lane] = myw / wsum;
  return wanted;
}

// The same selection by a CTA of 256 threads with VPT experts each, of one row whose logits an earlier kernel left; returns the expert
// of slot want_slot (in every thread). In one warp the chain of instructions is what costs (3.6 us for 512 experts); spread over
// eight it is three barriers and about as many hundred instructions.
struct RouteSmem { float mx[8], sum[8], gmax[32]; float2 cand[32]; int n_cand, expert; };
template <int VPT>
__device__ __forceinline__ int route_row_cta(const RouterParams& p, int n, const float (&l)[VPT], bool write, int want_slot, RouteSmem& sm) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, used = p.used;
  float m = l[0];
#pragma unroll
  for (int i = 1; i < VPT; i++) m = fmaxf(m, l[i]);
  int key = __float_as_int(m);                       // order of the floats as signed integers
  key ^= (key >> 31) & 0x7fffffff;
  key = __reduce_max_sync(0xffffffffu, key);
  if (lane == 0) sm.mx[warp] = __int_as_float(key ^ ((key >> 31) & 0x7fffffff));
  if (tid == 0) sm.n_cand = 0;
  __syncthreads();
  m = sm.mx[0];
#pragma unroll
  for (int w = 1; w < 8; w++) m = fmaxf(m, sm.mx[w]);
  float ev[VPT], s = 0.f, gm = -1.f;
#pragma unroll
  for (int i = 0; i < VPT; i++) {
    const bool live = tid + 256 * i < p.nE;
    ev[i] = live ? expf(l[i] - m) : -1.f;
    s += live ? ev[i] : 0.f;
    gm = fmaxf(gm, ev[i]);
  }
  s = warp_sum(s);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
  if (lane == 0) sm.sum[warp] = s;
  if ((lane & 7) == 0) sm.gmax[tid >> 3] = gm;
  __syncthreads();
  s = 0.f;
#pragma unroll
  for (int w = 0; w < 8; w++) s += sm.sum[w];
  const float inv = 1.0f / s;
  // bound: the (used + 1)-th largest of the 32 groups' maxima
  const float g = sm.gmax[lane];
  int above = 0;
#pragma unroll 8
  for (int j = 0; j < 32; j++) { const float o = sm.gmax[j]; above += o > g || (o == g && j < lane); }
  const uint32_t at = __ballot_sync(0xffffffffu, above == used);
  const float be = __shfl_sync(0xffffffffu, g, at != 0 ? __ffs((int)at) - 1 : 0), bound = at != 0 && be >= 0.f ? be * inv : -1.f;
#pragma unroll
  for (int i = 0; i < VPT; i++) {
    const float pv = ev[i] * inv;
    if (ev[i] >= 0.f && pv >= bound) {
      const int c = atomicAdd(&sm.n_cand, 1);
      if (c < 32) sm.cand[c] = make_float2(pv, __int_as_float(tid + 256 * i));
    }
  }
  __syncthreads();
  const int nc = sm.n_cand;
  if (nc > 32 || nc <= used) {   // many equal values, or none comparable (a NaN among the sums leaves no candidate): the one-warp form
    if (warp == 0) {
      const int ex = p.nE <= 512 ? route_token<16>(p, n, lane, write, sm.cand, want_slot) : route_token<32>(p, n, lane, write, sm.cand, want_slot);
      if (lane == 0) sm.expert = ex;
    }
    __syncthreads();
    return sm.expert;
  }
  const float v = lane < nc ? sm.cand[lane].x : -1.f;
  const int idx = lane < nc ? __float_as_int(sm.cand[lane].y) : 0x7fffffff;
  int rank = lane < nc ? 0 : 64;
  for (int j = 0; j < nc; j++) { const float2 o = sm.cand[j]; rank += o.x > v || (o.x == v && __float_as_int(o.y) < idx); }
  const uint32_t hit = __ballot_sync(0xffffffffu, rank == want_slot);
  if (write && warp == 0) {
    if (rank < used) p.topk[(size_t)n * used + rank] = idx;
    // the weights, added in slot order (llm/moe.go:256-282): lane k takes the value of rank k
    float mine = 0.f, wsum = 0.f, last = 0.f, next = 0.f;
    for (int k = 0; k <= used; k++) {
      const float x = __shfl_sync(0xffffffffu, v, __ffs((int)__ballot_sync(0xffffffffu, rank == k)) - 1);
      if (k == lane) mine = x;
      if (k < used) { wsum += x; last = x; } else next = x;
    }
    if (lane == 0 && p.margin) p.margin[n] = last > 0.f ? (last - next) / last : 0.f;
    if (wsum < 6.103515625e-5f) wsum = 6.103515625e-5f;
    if (lane < used) p.topk_w[(size_t)n * (used + 1) + lane] = mine / wsum;
  }
  return __shfl_sync(0xffffffffu, idx, hit != 0 ? __ffs((int)hit) - 1 : 0);
}

#endif

}  // namespace b200
