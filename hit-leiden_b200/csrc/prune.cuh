// prune.cuh — which re-activated vertices need no evaluation.
//
// A movement round re-activates every neighbour of a moved vertex, hubs above
// all, and almost none of them has a positive gain: on the upper levels of a
// 1M-vertex graph 5 moves a round re-activate rows of 7M entries.  Every
// evaluation therefore leaves a bound behind that later rounds keep up to date
// in O(1) per changed edge, and a vertex whose bound stays negative is not
// evaluated again.
//
// In units of weight, the gain of moving v from its community A to C is
//     h(C) = (w(v,C) - w(v,A)) + γ k_v (d_A - k_v - d_C) / 2m,
// the empty community having w = d = 0.  Let H be the largest h at v's last
// evaluation, over its neighbour communities and the empty one.  While v
// itself stays in A:
//   * a neighbour u that moves from X to Y raises w(v,Y) - w(v,A) by w_uv if
//     Y != A, and once more by w_uv if X = A; Y = A and other X raise no h.  A
//     community that v had no edge to starts from w = 0 and d >= 0, so from at
//     most h(empty) <= H;
//   * d_A has gone from its value then to its value now;
//   * no d_C has fallen by more than the sum over the rounds since of the
//     round's largest drop of one community's degree (S now minus S then).
// So every h now is at most
//     b + γ k_v (d_A + S) / 2m,   b = H - γ k_v (d_A + S)_then / 2m + Σ raises,
// (γ >= 0).  The arithmetic behind H, b and the computed gains is off by
// relative errors of order 1e-12 of terms no larger than k_v (1 + γ) (1 + rounds);
// the test leaves 1e-8 of them.  A vertex ruled out has no gain > 0: it gets the
// result its evaluation would give (no candidate), so rounds, candidates and
// moves are those of the full evaluation.
//
// Measured: 1M vertices with f64 weights, a batch whose levels run 73 rounds in
// all: movement 51 -> 29 ms.  On R-MAT graphs the bounds loosen too fast (every
// hub has moving neighbours in every round); they are dropped there after three
// rounds (run_eval).
#pragma once
#include "hl_engine.cuh"

namespace hl {

// Only rows longer than this are worth a bound.
constexpr u32 PRUNE_MIN_DEG = 64;

__device__ __forceinline__ bool prune_valid(const Prune& P, u32 v) {
  return P.b != nullptr && ((P.valid[v >> 5] >> (v & 31)) & 1u);
}

// v's gains are all <= 0 (v holds a valid bound; S now).
__device__ __forceinline__ bool prune_rules_out(const Prune& P, double S, u32 v, double kv,
                                                double d_cur, double tw, double gamma) {
  const double h = P.b[v] + gamma * kv * (d_cur + S) / tw;
  return h < -1e-8 * kv * (1.0 + gamma);
}

// The bound of a fresh evaluation: best computed gain over the neighbour
// communities (if any) and the empty one's.
__device__ __forceinline__ void prune_store(const Prune& P, double S, u32 v, double best,
                                            double kv, double d_cur, double tw, double gamma) {
  P.b[v] = best * tw - gamma * kv * (d_cur + S) / tw;
  const u32 m = 1u << (v & 31);
  if (!(P.valid[v >> 5] & m)) atomicOr(&P.valid[v >> 5], m);
}

// A moved vertex's own bound is void, and its community's degree drops by kv.
__device__ __forceinline__ void prune_moved(const Prune& P, u32 v, u32 from, double kv) {
  if (!P.b) return;
  const u32 m = 1u << (v & 31);
  if (P.valid[v >> 5] & m) atomicAnd(&P.valid[v >> 5], ~m);
  atomicAdd(&P.drop[from], kv);
}

// The round's largest drop (positive doubles order like their bits).
__device__ __forceinline__ void prune_worst(const Prune& P, u32 from) {
  if (P.b) atomicMax(P.worst, (unsigned long long)__double_as_longlong(P.drop[from]));
}
__device__ __forceinline__ double prune_worst_now(const Prune& P) {
  return __longlong_as_double((long long)*P.worst);
}

// Neighbour nb (community fn now) of a vertex that moved from -> to, fn != to.
__device__ __forceinline__ void prune_raise(const Prune& P, u32 nb, u32 fn, u32 from, double w) {
  if (prune_valid(P, nb)) atomicAdd(&P.b[nb], fn == from ? 2.0 * w : w);
}

}  // namespace hl
