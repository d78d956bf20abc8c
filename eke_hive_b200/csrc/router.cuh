// Per-row routing by a group of W warps, shared by the stand-alone router kernels (k_router.cu), the fused route + group kernel
// (k_moe_decode.cu) and the expert-parallel route + push kernel (k_ep.cu).  The exp is the portable polynomial form, sums are taken
// per lane of one warp (e = lane, lane+32, …) and then by a 16,8,4,2,1 butterfly, the k picks are summed in pick order — the CPU
// oracle does the same operations in the same order, so ids and weights agree with it to the bit.
//
// What bounds routing in a decode step is the length of one warp's instruction stream: it runs once, a warp on its own issues an
// instruction every 6-9 clocks of straight-line code, and a row of 512 experts in one warp took 9000 clocks (16 rows 14500, eight
// rows of the sigmoid router 27000).  So the scores of a row are worked out by all warps of its group, in loops that are short, and the
// picks are not k dependent rounds over all scores: the k-th largest of the 32 column maxima (column = e mod 32) is a bound that at
// least k experts reach, the dozen or so that reach it are listed, and each counts how many of them come before it.
#pragma once
#include "hb_common.cuh"

namespace hb {

constexpr int kRouteCand = 64;                                            // longer lists (long runs of equal scores) fall back to k rounds
struct RouteShare { uint2 cand[kRouteCand]; uint2 pick[16]; uint32_t red[16]; uint32_t bound; int n; };   // one per row group, in shared memory
struct RouteGroup { int warp, W, bar; };                                  // warp within the group, warps of the group, its named barrier

struct RouteArgs {                                                        // of one call; kind: 1 softmax, 2 sigmoid + bias
  int kind, E, k, renorm, logits_bf16; const float* bias; float scale;
};

__device__ __forceinline__ void route_sync(const RouteGroup& g) {
  if (g.W == 1) __syncwarp();
  else named_bar_sync(g.bar, 32 * g.W);
}
// Scores as unsigned numbers in the same order, 0 = not selectable.  Softmax: a non-negative float orders like its bits, NaN and the
// -1 of a taken expert give 0.  Sigmoid: any finite sum of score and bias (+0 folds -0 into it, as a comparison would), NaN and the
// -inf of a taken expert give 0.
template <bool SIG>
__device__ __forceinline__ uint32_t route_key(float v) {
  if (!SIG) return v >= 0.f ? __float_as_uint(v) + 1u : 0u;
  const uint32_t u = __float_as_uint(__fadd_rn(v, 0.f));
  return v > -INFINITY ? ((u & 0x80000000u) ? ~u : (u | 0x80000000u)) : 0u;
}
__device__ __forceinline__ float route_max(float v, const RouteGroup& g, uint32_t* red, int lane) {   // of the group; v is not NaN
  const uint32_t u = __float_as_uint(v);
  uint32_t o = __reduce_max_sync(0xffffffffu, (u & 0x80000000u) ? ~u : (u | 0x80000000u));
  if (g.W > 1) {
    if (lane == 0) red[g.warp] = o;
    route_sync(g);
    o = __reduce_max_sync(0xffffffffu, lane < g.W ? red[lane] : 0u);
  }
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// The weights of a row's picks, by one warp: lane l < k holds pick l as (key, id); sum: the softmax sum; score(id): the sigmoid of its logit.
template <bool SIG, class SCORE>
__device__ __forceinline__ void route_weights(const RouteArgs& a, uint2 mine, float sum, const SCORE& score, int& id, float& w) {
  id = (int)mine.y;
  float s, tot = 0.f;
  if (!SIG) s = __fmul_rn(mine.x ? __uint_as_float(mine.x - 1u) : -1.f, __fdiv_rn(1.f, sum));
  else {
    if (id == 0x7fffffff) id = 0;                                         // nothing left to pick (NaN): keep a valid id
    s = score(id);
  }
#pragma unroll 4
  for (int r = 0; r < a.k; ++r) tot = __fadd_rn(tot, __shfl_sync(0xffffffffu, s, r));
  if (!SIG) w = __fmul_rn(s, a.renorm ? __fdiv_rn(1.f, tot) : 1.f);
  else w = __fmul_rn(__fmul_rn(s, __fdiv_rn(1.f, __fadd_rn(tot, 1e-20f))), a.scale);
}

// One row of at most 32 experts by one warp, an expert a lane: k rounds over registers instead of the list below.  131072 rows of 8 experts,
// 1 pick: softmax 22 us, sigmoid 29 (with the list 43 and 44); of 32 experts, 4 picks: 29 and 27 (50 and 51).
template <bool SIG>
__device__ __forceinline__ void route_row32(const RouteArgs& a, const float* __restrict__ lr, int lane, int& id, float& w) {
  const bool on = lane < a.E;
  float v = on ? lr[lane] : -INFINITY, sum = 0.f;
  if (!SIG) {
    if (a.logits_bf16) v = bf16r(v);
    float mx = fmaxf(v, -INFINITY);                                       // NaN counts as the smallest
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    v = exp_portable(__fsub_rn(v, mx));
    sum = on ? v : 0.f;
    for (int o = 16; o > 0; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
  }
  const float sg = SIG ? sigmoid_portable(v) : 0.f;
  if (SIG) v = __fadd_rn(sg, on && a.bias ? a.bias[lane] : 0.f);
  uint32_t key = on ? route_key<SIG>(v) : 0u;
  uint2 mine = make_uint2(0u, 0x7fffffffu);
#pragma unroll 1
  for (int r = 0; r < a.k; ++r) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, key), at = __reduce_min_sync(0xffffffffu, m && key == m ? (uint32_t)lane : 0x7fffffffu);
    if (lane == r) mine = make_uint2(m, at);
    if ((uint32_t)lane == at) key = 0u;
  }
  route_weights<SIG>(a, mine, sum, [&](int e) { return __shfl_sync(0xffffffffu, sg, e); }, id, w);
}

// One row (logits lr) by the whole group.  p: E floats of shared memory and rs belong to the group.  Lane l < k of the group's warp 0
// gets pick l in (id, w); the other warps and lanes get nothing.  All warps of the group call it; it ends in step (a group may go on
// to its next row).
template <bool SIG>
__device__ __forceinline__ void route_row(const RouteArgs& a, const float* __restrict__ lr, float* p, RouteShare& rs, const RouteGroup& g, int lane, int& id,
                                          float& w) {
  const int t = g.warp * 32 + lane, T = g.W * 32;
  float sum = 0.f;
  if (!SIG) {
    float mx = -INFINITY;
#pragma unroll 4
    for (int e = t; e < a.E; e += T) {
      const float v = a.logits_bf16 ? bf16r(lr[e]) : lr[e];
      p[e] = v;
      mx = fmaxf(mx, v);
    }
    mx = route_max(mx, g, rs.red, lane);
#pragma unroll 2
    for (int e = t; e < a.E; e += T) p[e] = exp_portable(__fsub_rn(p[e], mx));
  } else {
#pragma unroll 2
    for (int e = t; e < a.E; e += T) {
      const float b = a.bias ? a.bias[e] : 0.f;                           // a score is positive: + 0 leaves it as it is
      p[e] = __fadd_rn(sigmoid_portable(lr[e]), b);
    }
  }
  route_sync(g);
  if (g.warp == 0) {
    uint32_t best = 0u;
#pragma unroll 8
    for (int e = lane; e < a.E; e += 32) { const float v = p[e]; if (!SIG) sum = __fadd_rn(sum, v); best = max(best, route_key<SIG>(v)); }
    if (!SIG) for (int o = 16; o > 0; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
    uint32_t bound = 0u;                                                  // the k-th largest distinct column maximum: no larger than the k-th largest one
#pragma unroll 1
    for (int r = 0; r < a.k; ++r) {
      bound = __reduce_max_sync(0xffffffffu, best);
      if (best == bound) best = 0u;
    }
    bound = max(bound, 1u);                                               // fewer than k distinct ones: every selectable expert is listed
    if (lane == 0) { rs.bound = bound; rs.n = 0; }
    if (lane < 16) rs.pick[lane] = make_uint2(0u, 0x7fffffffu);
  }
  route_sync(g);
  const uint32_t bound = rs.bound;
#pragma unroll 2
  for (int e = t; e < a.E; e += T) {
    const uint32_t key = route_key<SIG>(p[e]);
    if (key >= bound) { const int at = atomicAdd(&rs.n, 1); if (at < kRouteCand) rs.cand[at] = make_uint2(key, (uint32_t)e); }
  }
  route_sync(g);
  if (g.warp == 0) {
    const int n = rs.n;
    if (n <= kRouteCand) {
      for (int c = lane; c < n; c += 32) {
        const uint2 me = rs.cand[c];
        int r = 0;
#pragma unroll 4
        for (int i = 0; i < n; ++i) { const uint2 o = rs.cand[i]; r += o.x > me.x || (o.x == me.x && o.y < me.y); }   // the smaller id first among equals
        if (r < a.k) rs.pick[r] = me;
      }
    } else {
#pragma unroll 1
      for (int r = 0; r < a.k; ++r) {
        uint32_t mx = 0u, at = 0x7fffffffu;
        for (int e = lane; e < a.E; e += 32) { const uint32_t key = route_key<SIG>(p[e]); if (key > mx) { mx = key; at = (uint32_t)e; } }
        const uint32_t m = __reduce_max_sync(0xffffffffu, mx);
        at = __reduce_min_sync(0xffffffffu, mx == m ? at : 0x7fffffffu);
        if (m && (at & 31u) == (uint32_t)lane) p[at] = SIG ? -INFINITY : -1.f;
        if (lane == 0) rs.pick[r] = make_uint2(m, m ? at : 0x7fffffffu);
        __syncwarp();
      }
    }
    __syncwarp();
    route_weights<SIG>(a, rs.pick[lane & 15], sum, [&](int e) { return sigmoid_portable(lr[e]); }, id, w);
  }
  route_sync(g);                                                          // p and rs are free for the group's next row
}

}  // namespace hb
