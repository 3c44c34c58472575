// det.cu — RunMode::Deterministic on the GPU: the sequential Gauss–Seidel
// movement (hit_leiden.rs:1103-1191) and the sequential singleton merges of
// the refinement (hit_leiden.rs:1392-1548).
//
// Both loops are sequential by definition: each step reads the state the
// previous step wrote.  They run as one persistent block that walks the
// vertices in the reference's order and spreads the work of each step (a
// row's neighbour scan, the candidate argmax, the frontier marks, a T-filter
// sum) over its threads, so a whole stage is one launch with no host round
// trip.  Results are bit-identical to the reference's steps under the
// canonical order used throughout (first CSR encounter for hash order):
//   * per-key sums are exact in any order with integral weights; with f64
//     weights one warp extends every key's sum in CSR order;
//   * strict '>' in first-encounter order = the largest gain, ties to the
//     smallest first CSR position;
//   * d(C), d_S and the sizes are updated in step order by one thread.
// No step waits on another block, and the loops are bounded (max_pops); a
// loop that reaches its bound stops and reports it through a status word.
#include <cstring>

#include "hl_engine.cuh"

namespace hl {

static inline u32 grid_for(u64 n, u32 block = 256) {
  u64 g = (n + block - 1) / block;
  if (g > 148u * 64u) g = 148u * 64u;
  return g ? (u32)g : 1u;
}

constexpr u32 DET_THREADS = 512;
constexpr u32 DET_WARPS = DET_THREADS / 32;
constexpr u32 DET_EMPTY = 0xFFFFFFFEu;  // "the next empty community" before an id is given

enum : u32 { DET_OK = 0, DET_POP_LIMIT = 1, DET_ID_SPACE = 2 };

// Σw and the first CSR position of every key of row [o0, o1) into the dense
// scratch (bw, bp), the distinct keys into klist (count in *nk).  `key(q)`
// returns the entry's key or NONE32 to skip it.  Integral weights: the whole
// block, atomics of the keys of 32 entries each (every order gives the same
// sums; most of a hub's neighbours may share one community, and an atomic an
// entry took 20 us for a row of 1,800).  Otherwise warp 0, in CSR
// order: a 32-entry tile at a time, entries of one key folded by its first
// lane in lane order, tiles in order.
template <typename K>
__device__ __forceinline__ void det_row_sums(u64 o0, u64 o1, const double* w, bool ordered,
                                             K key, double* bw, u32* bp, u32* klist, u32* nk,
                                             double* tile) {
  const u32 tid = threadIdx.x, lane = tid & 31;
  if (!ordered) {
    for (u64 q0 = o0 + (tid - lane); q0 < o1; q0 += 4 * DET_THREADS) {
      u32 c[4];
      double x[4];
#pragma unroll
      for (u32 j = 0; j < 4; ++j) {
        const u64 q = q0 + j * DET_THREADS + lane;
        c[j] = q < o1 ? key(q) : NONE32;
        x[j] = q < o1 ? w[q] : 0.0;
      }
#pragma unroll
      for (u32 j = 0; j < 4; ++j) {
        if (q0 + j * DET_THREADS >= o1) break;  // warp-uniform
        const u64 q = q0 + j * DET_THREADS + lane;
        const u32 grp = __match_any_sync(0xffffffffu, c[j]);
        const bool lead = c[j] != NONE32 && !(grp & ((1u << lane) - 1u));
        const double y = warp_group_sum(grp, lead, x[j]);
        if (!lead) continue;
        atomicAdd(&bw[c[j]], y);
        const u32 old = atomicMin(&bp[c[j]], (u32)(q - o0));
        if (old == NONE32) klist[atomicAdd(nk, 1u)] = c[j];
      }
    }
    return;
  }
  if (tid >= 32) return;
  for (u64 base = o0; base < o1; base += 32) {
    const u64 q = base + lane;
    const u32 c = q < o1 ? key(q) : NONE32;
    const bool ok = c != NONE32;
    tile[lane] = ok ? w[q] : 0.0;
    const u32 grp = __match_any_sync(0xffffffffu, ok ? (unsigned long long)c
                                                     : ((1ull << 32) | lane));
    __syncwarp();
    if (ok && lane == (u32)(__ffs(grp) - 1)) {
      if (bp[c] == NONE32) {
        bp[c] = (u32)(q - o0);
        klist[atomicAdd(nk, 1u)] = c;
      }
      double acc = bw[c];
      for (u32 m = grp; m; m &= m - 1) acc = __dadd_rn(acc, tile[__ffs(m) - 1]);
      bw[c] = acc;
    }
    __syncwarp();
  }
}

// Largest gain over the lanes (g of lanes without a candidate: 0), ties to the
// smallest position; the winning lane, or 32 when no gain is positive.
__device__ __forceinline__ u32 det_warp_best(double g, u32 p) {
  const u64 key = g > 0.0 ? (u64)__double_as_longlong(g) : 0ull;  // positive: bits ascend
  const u32 hi = (u32)(key >> 32), lo = (u32)key;
  const u32 mh = __reduce_max_sync(0xffffffffu, hi);
  if (!mh) return 32;
  const u32 ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const bool best = hi == mh && lo == ml;
  const u32 mp = __reduce_min_sync(0xffffffffu, best ? p : NONE32);
  return __ffs(__ballot_sync(0xffffffffu, best && p == mp)) - 1;
}

// Block argmax of (gain, first position, key) over positive gains (p: NONE32
// without one): the largest gain, ties to the smallest position.  Returns in the
// first warp.
__device__ __forceinline__ void det_argmax(double& g, u32& p, u32& k, double* r_g, u32* r_p,
                                           u32* r_k) {
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  auto warp_best = [&]() {
    const u32 bl = det_warp_best(p != NONE32 ? g : 0.0, p);
    g = __shfl_sync(0xffffffffu, g, bl & 31);
    p = __shfl_sync(0xffffffffu, p, bl & 31);
    k = __shfl_sync(0xffffffffu, k, bl & 31);
    if (bl == 32) p = NONE32;
  };
  warp_best();
  if (lane == 0) {
    r_g[wib] = g;
    r_p[wib] = p;
    r_k[wib] = k;
  }
  __syncthreads();
  if (wib == 0) {
    g = lane < DET_WARPS ? r_g[lane] : 0.0;
    p = lane < DET_WARPS ? r_p[lane] : NONE32;
    k = lane < DET_WARPS ? r_k[lane] : NONE32;
    warp_best();
  }
}

struct DetMoveArgs {
  u32 n;
  const u64* off;
  const u32* col;
  const double* w;
  u32* f;
  const u32* s;
  const double* k;
  double* d;
  u64 dcap;            // entries of d (and of bw / bp): community ids stay below it
  const u32* act;      // active bitset, (n + 31) / 32 words
  u8* changed;
  u8* affected;
  bool mark_moved;
  double* bw;          // dense per-community scratch: Σw (0.0 between rows)
  u32* bp;             // first CSR position (NONE32 between rows)
  u32* klist;          // the row's distinct keys
  double tw, gamma;
  u32 next_empty;      // id of the next empty community (hit_leiden.rs:1104)
  bool ordered;
  bool f_local;        // the labels are kept in shared memory too
  bool d_local;        // ... and d of the ids below n
  u32* gbits;          // the bit sets, when they exceed shared memory
  u64 max_pops;
  unsigned long long* out;  // [0] pops, [1] moves, [2] traversed, [3] status, [4] next_empty
};

// The walk pops the lowest active vertex, evaluates it, perhaps moves it, and
// most pops move nothing (25 pops a move on the 9.9k-vertex graph).  A pop that
// moves nothing changes nothing that later evaluations read, so the next
// vertices in order are evaluated together on the current state, a warp each;
// up to and including the first one that moves they are the reference's pops,
// the rest stay active and are evaluated again after the move.  The number taken
// grows while nothing moves.  The active set is a three-level bit set in shared
// memory, and so are the labels and the community degrees of small levels.
// Rows above DET_WARP_ROW entries take the whole block, one at a time, and end
// the list: where every other pop is such a row, evaluations beyond it would be
// done again and again.
constexpr u32 DET_AHEAD = 128;       // vertices evaluated together at most
constexpr u32 DET_WARP_ROW = 128;
constexpr u32 DET_TAB = 2 * DET_WARP_ROW;
constexpr u32 DET_F_LOCAL = 32768;   // nodes whose labels fit shared memory
constexpr u32 DET_D_LOCAL = 10240;   // ... whose community degrees do, too
constexpr size_t DET_SMEM_MAX = 216 * 1024;
constexpr u32 DET_BITS_LOCAL = 1u << 20;  // nodes whose bit sets fit shared memory

struct DetWarp {
  double tv[DET_TAB];
  double sw[DET_WARP_ROW];
  u32 tk[DET_TAB], tp[DET_TAB];
};
struct DetSmem {
  DetWarp warp[DET_WARPS];
};

// The active set: words of 32 vertices, and one bit per non-zero word, twice.
struct DetBits {
  u32 *l0, *l1, *l2;
  __device__ __forceinline__ void set(u32 v) {
    atomicOr(&l0[v >> 5], 1u << (v & 31));
    atomicOr(&l1[v >> 10], 1u << ((v >> 5) & 31));
    atomicOr(&l2[v >> 15], 1u << ((v >> 10) & 31));
  }
  // Several threads may clear at once, but none may set meanwhile.
  __device__ __forceinline__ void clear(u32 v) {
    const u32 m0 = ~(1u << (v & 31)), m1 = ~(1u << ((v >> 5) & 31));
    if (atomicAnd(&l0[v >> 5], m0) & m0) return;
    if (atomicAnd(&l1[v >> 10], m1) & m1) return;
    atomicAnd(&l2[v >> 15], ~(1u << ((v >> 10) & 31)));
  }
};

__device__ __forceinline__ u32 det_word(const u32* p) { return *(const volatile u32*)p; }

// The lowest active vertex (NONE32: none), by one warp; n2 words at the top.
__device__ __forceinline__ u32 det_lowest(const DetBits& B, u32 n2) {
  const u32 lane = threadIdx.x & 31;
  for (u32 i0 = 0; i0 < n2; i0 += 32) {
    const u32 x = i0 + lane < n2 ? det_word(&B.l2[i0 + lane]) : 0u;
    const u32 m = __ballot_sync(0xffffffffu, x != 0);
    if (!m) continue;
    const u32 j = __ffs(m) - 1;
    const u32 i2 = ((i0 + j) << 5) + (u32)__ffs(__shfl_sync(0xffffffffu, x, j)) - 1;
    const u32 i1 = (i2 << 5) + (u32)__ffs(det_word(&B.l1[i2])) - 1;
    return (i1 << 5) + (u32)__ffs(det_word(&B.l0[i1])) - 1;
  }
  return NONE32;
}

// False when the computed gain of moving to (w_to, d_to) is certainly <= 0: the
// division-free proxy Q = 2m·c·gain lies below zero by more than the rounding
// of both (GainScreen in hl_internal.cuh).  Two divisions cost as much as the
// rest of a step, and few candidates gain.
__device__ __forceinline__ bool det_may_gain(double w_to, double d_to, double w_cur, double tw,
                                             double gamma, double kv, double d_cur) {
  const double p1 = __dmul_rn(__dsub_rn(w_to, w_cur), __dmul_rn(tw, tw));
  const double p2 =
      __dmul_rn(__dmul_rn(__dmul_rn(gamma, kv), __dsub_rn(__dsub_rn(d_cur, kv), d_to)), tw);
  const double t = __dadd_rn(fabs(p1), fabs(p2));
  return !(__dadd_rn(p1, p2) < -__dadd_rn(__dmul_rn(1.7763568394002505e-15, t), 1e-300));
}

// hit_leiden.rs:1103-1191.  What bounds it: the chain of a step (barriers and
// dependent loads, about 6 us) times the moves.  9.9k vertices, 1,672 pops with
// 67 moves: 128 steps, 0.83 ms, against 2.9 ms one pop at a time by the block
// (two divisions, eight barriers and global atomics a pop).
__global__ void __launch_bounds__(DET_THREADS) k_det_move(DetMoveArgs A) {
  extern __shared__ __align__(16) unsigned char det_raw[];
  DetSmem& M = *reinterpret_cast<DetSmem*>(det_raw);
  __shared__ u32 s_list[DET_AHEAD], s_to[DET_AHEAD], s_deg[DET_AHEAD];
  __shared__ u64 s_off[DET_AHEAD];
  __shared__ u32 s_nlist, s_first, s_big, s_nk, s_best, s_stop;
  __shared__ double s_bestg;
  __shared__ double r_g[DET_WARPS];
  __shared__ u32 r_p[DET_WARPS], r_k[DET_WARPS];
  __shared__ double tile[32];
  __shared__ unsigned long long s_pops, s_moves, s_trav;
  __shared__ u32 s_empty;
  const u32 tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const u32 n0 = (A.n + 31) >> 5, n1 = (n0 + 31) >> 5, n2 = (n1 + 31) >> 5;
  u32* local = reinterpret_cast<u32*>(det_raw + sizeof(DetSmem));
  DetBits B;
  B.l0 = A.gbits ? A.gbits : local;
  B.l1 = B.l0 + n0;
  B.l2 = B.l1 + n1;
  u32* fl = A.f_local ? local + (A.gbits ? 0 : n0 + n1 + n2) : nullptr;
  u32* f = fl ? fl : A.f;
  // d of ids below n; written through to A.d
  double* dl = A.d_local ? reinterpret_cast<double*>(
                               det_raw + ((sizeof(DetSmem) + 4 * (size_t)(n0 + n1 + n2 + A.n) + 7) &
                                          ~(size_t)7))
                         : nullptr;
  auto d_of = [&](u32 c) { return dl && c < A.n ? dl[c] : A.d[c]; };
  auto d_put = [&](u32 c, double x) {
    if (dl && c < A.n) dl[c] = x;
    A.d[c] = x;
  };
  for (u32 i = tid; i < n0; i += DET_THREADS) B.l0[i] = A.act[i];
  for (u32 i = tid; i < n1 + n2; i += DET_THREADS) B.l1[i] = 0;
  if (fl)
    for (u32 i = tid; i < A.n; i += DET_THREADS) fl[i] = A.f[i];
  if (dl)
    for (u32 i = tid; i < A.n; i += DET_THREADS) dl[i] = A.d[i];
  if (tid == 0) {
    s_stop = DET_OK;
    s_pops = s_moves = s_trav = 0;
    s_empty = A.next_empty;
  }
  __syncthreads();
  for (u32 i = tid; i < n0; i += DET_THREADS)
    if (det_word(&B.l0[i])) {
      atomicOr(&B.l1[i >> 5], 1u << (i & 31));
      atomicOr(&B.l2[i >> 10], 1u << ((i >> 5) & 31));
    }
  __syncthreads();
  u32 ahead = DET_WARPS;  // vertices taken together
  unsigned long long trav = 0;
  while (true) {
    // ---- the next active vertices in order ----
    if (wib == 0) {
      const u32 first = det_lowest(B, n2);
      u32 cnt = 0;
      if (first != NONE32) {
        u32 w0 = first >> 5;
        for (u32 win = 0; win < 16 && w0 < n0 && cnt < ahead; ++win, w0 += 32) {
          u32 x = w0 + lane < n0 ? det_word(&B.l0[w0 + lane]) : 0u;
          if (!__any_sync(0xffffffffu, x != 0)) continue;
          u32 inc = __popc(x);
#pragma unroll
          for (u32 o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
          }
          for (u32 at = cnt + inc - __popc(x); x && at < ahead; x &= x - 1, ++at)
            s_list[at] = ((w0 + lane) << 5) + (u32)__ffs(x) - 1;
          cnt = min(ahead, cnt + __shfl_sync(0xffffffffu, inc, 31));
        }
      }
      if (lane == 0) {
        s_nlist = cnt;
        s_first = s_big = NONE32;
        s_nk = 0;
      }
    }
    __syncthreads();
    const u32 nlist = s_nlist;
    if (nlist == 0) break;
    // ---- their rows; the first long one ends the list ----
    if (tid < nlist) {
      const u32 v = s_list[tid];
      const u64 o0 = A.off[v], len = A.off[v + 1] - o0;
      s_off[tid] = o0;
      s_deg[tid] = (u32)len;
      if (len > DET_WARP_ROW) atomicMin(&s_big, tid);
    }
    __syncthreads();
    const u32 big = s_big, neval = min(nlist, big);
    // ---- the best moves of those before it on the current state ----
    for (u32 i = wib; i < neval; i += DET_WARPS) {
      const u32 v = s_list[i];
      const u64 o0 = s_off[i];
      const u32 deg = s_deg[i];
      const u32 cur = f[v];
      const double kv = A.k[v];
      const double dcur = d_of(cur);
      // Σw per neighbour community, self-loops included (:1119-1125): this
      // lane's candidate (key, first position, gain)
      double wcur = 0.0, g = 0.0;
      u32 key = NONE32, pos = NONE32;
      DetWarp& T = M.warp[wib];
      if (deg <= 32) {
        u32 c = NONE32;
        if (lane < deg) {
          c = f[A.col[o0 + lane]];
          T.sw[lane] = A.w[o0 + lane];
        }
        __syncwarp();
        const u32 grp = __match_any_sync(0xffffffffu, c);
        const bool lead = c != NONE32 && !(grp & ((1u << lane) - 1u));
        double sum = 0.0, dkey = 0.0;
        if (lead) {
          dkey = d_of(c);
          for (u32 m = grp; m; m &= m - 1) sum = __dadd_rn(sum, T.sw[__ffs(m) - 1]);
        }
        const u32 cm = __ballot_sync(0xffffffffu, lead && c == cur);
        const double wc = __shfl_sync(0xffffffffu, sum, cm ? __ffs(cm) - 1 : 0);
        wcur = cm ? wc : 0.0;
        if (lead && c != cur && det_may_gain(sum, dkey, wcur, A.tw, A.gamma, kv, dcur)) {
          g = move_gain(sum, wcur, A.tw, A.gamma, kv, dcur, dkey);
          key = c;
          pos = lane;
        }
      } else {
        u32 cap = 64;
        while (cap < 2 * deg) cap <<= 1;
        const u32 mask = cap - 1;
        for (u32 x = lane; x < cap; x += 32) T.tk[x] = NONE32;
        u32 cq[DET_WARP_ROW / 32];
#pragma unroll
        for (u32 j = 0; j < DET_WARP_ROW / 32; ++j) {
          const u32 q = 32 * j + lane;
          cq[j] = q < deg ? A.col[o0 + q] : NONE32;
          if (q < deg) T.sw[q] = A.w[o0 + q];
        }
#pragma unroll
        for (u32 j = 0; j < DET_WARP_ROW / 32; ++j)
          if (cq[j] != NONE32) cq[j] = f[cq[j]];
        __syncwarp();
#pragma unroll
        for (u32 j = 0; j < DET_WARP_ROW / 32; ++j) {
          if (32 * j >= deg) break;
          const u32 c = cq[j];
          const u32 grp = __match_any_sync(0xffffffffu, c);
          if (c != NONE32 && !(grp & ((1u << lane) - 1u))) {
            u32 slot = ((c * 2654435761u) >> 7) & mask;
            while (true) {  // the table holds at most deg < cap keys
              const u32 prev = atomicCAS(&T.tk[slot], NONE32, c);
              if (prev == NONE32 || prev == c) {
                double sum = prev == NONE32 ? 0.0 : T.tv[slot];
                for (u32 m = grp; m; m &= m - 1)
                  sum = __dadd_rn(sum, T.sw[32 * j + __ffs(m) - 1]);
                T.tv[slot] = sum;
                if (prev == NONE32) T.tp[slot] = 32 * j + lane;
                break;
              }
              slot = (slot + 1) & mask;
            }
          }
          __syncwarp();
        }
        bool found = false;
        for (u32 x = lane; x < cap; x += 32)
          if (T.tk[x] == cur) {
            wcur = T.tv[x];
            found = true;
          }
        const u32 fm = __ballot_sync(0xffffffffu, found);
        wcur = __shfl_sync(0xffffffffu, wcur, fm ? __ffs(fm) - 1 : 0);
        if (!fm) wcur = 0.0;
        for (u32 x = lane; x < cap; x += 32) {
          const u32 c = T.tk[x];
          if (c == NONE32 || c == cur) continue;
          const double dc = d_of(c);
          if (!det_may_gain(T.tv[x], dc, wcur, A.tw, A.gamma, kv, dcur)) continue;
          const double gn = move_gain(T.tv[x], wcur, A.tw, A.gamma, kv, dcur, dc);
          const u32 pc = T.tp[x];
          if (gn > 0.0 && (pos == NONE32 || gn > g || (gn == g && pc < pos))) {
            g = gn;
            pos = pc;
            key = c;
          }
        }
      }
      // best candidate (:1127-1146), then the empty community (:1150-1162)
      const bool may_empty = det_may_gain(0.0, 0.0, wcur, A.tw, A.gamma, kv, dcur);
      const u32 bl = det_warp_best(g, pos);
      u32 to = NONE32;
      double bestg = 0.0;
      if (bl < 32) {
        bestg = __shfl_sync(0xffffffffu, g, bl);
        to = __shfl_sync(0xffffffffu, key, bl);
      }
      if (may_empty && empty_gain(wcur, A.tw, A.gamma, kv, dcur) > bestg) to = DET_EMPTY;
      if (lane == 0) {
        s_to[i] = to;
        if (to != NONE32) atomicMin(&s_first, i);
      }
      __syncwarp();
    }
    if (neval) __syncthreads();
    // ---- the pops: all up to the first that moves, or the long row ----
    const u32 first = min(s_first, big);
    const u32 popped = first == NONE32 ? nlist : first + 1;
    if (tid < popped) {
      B.clear(s_list[tid]);
      trav += s_deg[tid];
    }
    if (tid == 0) {
      s_pops += popped;
      if (s_pops > A.max_pops) s_stop = DET_POP_LIMIT;
    }
    __syncthreads();
    // a list that ends at a long row was too long by what it listed beyond it
    ahead = first == NONE32 ? min(2 * ahead, DET_AHEAD)
            : first == big  ? min(2 * popped, DET_WARPS)
                            : DET_WARPS;
    if (s_stop != DET_OK) break;
    if (first == NONE32) continue;
    const u32 v = s_list[first];
    const u32 cur = f[v];
    const u64 o0 = s_off[first], o1 = o0 + s_deg[first];
    u32 best = first != big ? s_to[first] : NONE32;
    if (first != big) {
      // ---- the move (:1168-1187), by one warp ----
      if (wib == 0) {
        const double kv = A.k[v];
        if (best == DET_EMPTY) {
          best = s_empty;
          if ((u64)best >= A.dcap) {
            best = NONE32;
            if (lane == 0) s_stop = DET_ID_SPACE;
          }
        }
        if (best != NONE32) {
          const double dcur = d_of(cur), dbest = d_of(best);
          __syncwarp();
          if (lane == 0) {
            if (s_to[first] == DET_EMPTY) s_empty = best + 1;
            A.f[v] = best;
            if (fl) fl[v] = best;
            A.changed[v] = 1;
            if (A.mark_moved) A.affected[v] = 1;
            d_put(cur, __dsub_rn(dcur, kv));
            d_put(best, __dadd_rn(dbest, kv));
            ++s_moves;
          }
          __syncwarp();
          const u32 sv = A.s[v];
          bool any = false;
          for (u64 q = o0 + lane; q < o1; q += 32) {
            const u32 nb = A.col[q];
            if (f[nb] != best) B.set(nb);
            if (A.s[nb] == sv) {
              any = true;
              A.affected[nb] = 1;
            }
          }
          if (__any_sync(0xffffffffu, any) && lane == 0) A.affected[v] = 1;
        }
      }
      __syncthreads();
      if (s_stop != DET_OK) break;
      continue;
    }
    // ---- a long row, by the whole block ----
    const double kv = A.k[v];
    const u32* col = A.col;
    det_row_sums(o0, o1, A.w, A.ordered, [&](u64 q) { return f[col[q]]; }, A.bw, A.bp, A.klist,
                 &s_nk, tile);
    __syncthreads();
    const double wcur = A.bw[cur];
    const double dcur = d_of(cur);
    const u32 nk = s_nk;
    double g = 0.0;
    u32 p = NONE32, kk = NONE32;
    for (u32 i = tid; i < nk; i += DET_THREADS) {
      const u32 c = A.klist[i];
      if (c == cur) continue;
      const double wc = A.bw[c], dc = d_of(c);
      const u32 pc = A.bp[c];
      if (!det_may_gain(wc, dc, wcur, A.tw, A.gamma, kv, dcur)) continue;
      const double gn = move_gain(wc, wcur, A.tw, A.gamma, kv, dcur, dc);
      if (gn > 0.0 && (p == NONE32 || gn > g || (gn == g && pc < p))) {
        g = gn;
        p = pc;
        kk = c;
      }
    }
    det_argmax(g, p, kk, r_g, r_p, r_k);
    if (tid == 0) {
      best = cur;
      double bestg = 0.0;
      if (p != NONE32) {
        best = kk;
        bestg = g;
      }
      if (det_may_gain(0.0, 0.0, wcur, A.tw, A.gamma, kv, dcur)) {
        const double eg = empty_gain(wcur, A.tw, A.gamma, kv, dcur);
        if (eg > bestg) {
          bestg = eg;
          best = DET_EMPTY;
        }
      }
      if (bestg > 0.0) {
        if (best == DET_EMPTY) {
          if ((u64)s_empty >= A.dcap) s_stop = DET_ID_SPACE;
          else best = s_empty++;
        }
        if (s_stop == DET_OK) {
          A.f[v] = best;
          if (fl) fl[v] = best;
          A.changed[v] = 1;
          if (A.mark_moved) A.affected[v] = 1;
          d_put(cur, __dsub_rn(dcur, kv));
          d_put(best, __dadd_rn(d_of(best), kv));
          ++s_moves;
        }
      }
      s_best = best;
      s_bestg = bestg;
    }
    __syncthreads();
    for (u32 i = tid; i < nk; i += DET_THREADS) {
      const u32 c = A.klist[i];
      A.bw[c] = 0.0;
      A.bp[c] = NONE32;
    }
    if (s_stop != DET_OK) break;
    if (s_bestg > 0.0) {
      best = s_best;
      const u32 sv = A.s[v];
      for (u64 q = o0 + tid; q < o1; q += DET_THREADS) {
        const u32 nb = A.col[q];
        if (f[nb] != best) B.set(nb);
        if (A.s[nb] == sv) {
          A.affected[v] = 1;
          A.affected[nb] = 1;
        }
      }
    }
    __syncthreads();
  }
  if (trav) atomicAdd(&s_trav, trav);
  __syncthreads();
  if (tid == 0) {
    A.out[0] = s_pops;
    A.out[1] = s_moves;
    A.out[2] = s_trav;
    A.out[3] = s_stop;
    A.out[4] = s_empty;
  }
}

__global__ void k_fill_u32_det(u32* p, u32 v, u64 n) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    p[i] = v;
}

static void det_status(Engine& E, const u64* out, const char* stage) {
  if (out[3] == DET_POP_LIMIT)
    throw Error(HL_ERR_TIMEOUT, std::string(stage) + ": the sequential loop reached its step bound");
  if (out[3] == DET_ID_SPACE)
    throw Error(HL_ERR_UNSUPPORTED,
                std::string(stage) + ": more empty-community moves in one call than ids below 2n+2");
  (void)E;
}

static std::atomic<bool> g_det_attr[64];

// The deterministic branch of inc_movement, after seeding and d(C) (`act`: the
// active bit set).  Returns moves and traversed entries.
void inc_movement_det(Engine& E, Level& L, const u32* act, double* d, size_t dcap,
                      bool mark_moved, u64* moves, u64* traversed) {
  Scratch& S = E.sc;
  cudaStream_t st = E.stream;
  const u32 n = L.g.n;
  const u64 n0 = ((u64)n + 31) / 32, n1 = (n0 + 31) / 32, n2 = (n1 + 31) / 32;
  const bool bits_local = n <= DET_BITS_LOCAL, f_local = n <= DET_F_LOCAL;
  if (!bits_local) S.det_bits.ensure(E.mem, n0 + n1 + n2);
  const bool d_local = n <= DET_D_LOCAL;
  size_t smem = sizeof(DetSmem) + (bits_local ? 4 * (n0 + n1 + n2) : 0) +
                (f_local ? 4 * (size_t)n : 0);
  if (d_local) smem = ((smem + 7) & ~(size_t)7) + 8 * (size_t)n;
  // bit sets: n / 8 bytes and a little more than a 32nd of that above them
  constexpr auto bits = [](size_t x) { return x / 8 + x / 128; };
  static_assert(sizeof(DetSmem) + 12 * DET_D_LOCAL + bits(DET_D_LOCAL) <= DET_SMEM_MAX &&
                    sizeof(DetSmem) + 4 * DET_F_LOCAL + bits(DET_F_LOCAL) <= DET_SMEM_MAX &&
                    sizeof(DetSmem) + bits(DET_BITS_LOCAL) <= DET_SMEM_MAX,
                "the largest levels kept in shared memory fit it");
  const int dev = E.device;
  if (dev >= 0 && dev < 64 && !g_det_attr[dev]) {
    HL_CUDA(cudaFuncSetAttribute(k_det_move, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)DET_SMEM_MAX));
    g_det_attr[dev] = true;
  }
  S.det_bw.ensure(E.mem, dcap);
  S.det_bp.ensure(E.mem, dcap);
  S.det_keys.ensure(E.mem, dcap);
  S.det_out.ensure(E.mem, 8);
  HL_CUDA(cudaMemsetAsync(S.det_bw.p, 0, sizeof(double) * dcap, st));
  ++E.nlaunch, k_fill_u32_det<<<grid_for(dcap), 256, 0, st>>>(S.det_bp.p, NONE32, dcap);
  HL_CUDA(cudaMemsetAsync(S.det_out.p, 0, 8 * sizeof(u64), st));
  HL_LAUNCH_CHECK();
  DetMoveArgs A;
  A.n = n;
  A.off = L.g.off.p;
  A.col = L.g.col.p;
  A.w = L.g.w.p;
  A.f = L.f.p;
  A.s = L.s_cur.p;
  A.k = L.k.p;
  A.d = d;
  A.dcap = dcap;
  A.act = act;
  A.f_local = f_local;
  A.d_local = d_local;
  A.gbits = bits_local ? nullptr : S.det_bits.p;
  A.changed = S.changed.p;
  A.affected = S.affected.p;
  A.mark_moved = mark_moved;
  A.bw = S.det_bw.p;
  A.bp = S.det_bp.p;
  A.klist = S.det_keys.p;
  A.tw = L.tw;
  A.gamma = E.cfg.resolution;
  A.next_empty = n;  // ids were compacted below n: the reference's community_degrees.len()
  A.ordered = !E.integral;
  A.max_pops = 4096ull * (u64)n + (1ull << 20);
  A.out = reinterpret_cast<unsigned long long*>(S.det_out.p);
  ++E.nlaunch, k_det_move<<<1, DET_THREADS, smem, st>>>(A);
  HL_LAUNCH_CHECK();
  u64 out[8];
  HL_CUDA(cudaMemcpyAsync(E.hs.p, S.det_out.p, 8 * sizeof(u64), cudaMemcpyDeviceToHost, st));
  E.sync();
  std::memcpy(out, E.hs.p, sizeof(out));
  det_status(E, out, "deterministic movement");
  *moves = out[1];
  *traversed = out[2];
}

// ----------------------------------------------------------------------------
// Sequential singleton merges with the live T-filter.
// ----------------------------------------------------------------------------
struct DetRefArgs {
  const u64* off;
  const u32* col;
  const double* w;
  const u32* f;
  u32* s;
  const double* k;
  double* dS;          // sub-community degrees (ordered sums, then step updates)
  u32* sizes;
  const double* dcomm; // d_parent: Σ k over each community, node order
  const u32* rlist;    // R sorted by (k, node)
  u32 nr;
  double* bw;
  u32* bp;
  u32* klist;
  double* wsp;         // cached w(S, C_parent)
  u8* wvalid;
  const u32* members;  // nodes sorted by (s, node) at the start of the merges
  const u32* mstart;   // per S: first index of its members (NONE32: none)
  const u32* mcount;   // per S: number of initial members
  u32* xhead;          // per S: merged singletons, ascending linked list
  u32* xnext;          // per node: next merged singleton of the same S
  double tw, gamma;
  bool ordered;
  unsigned long long* out;  // [0] merges
};

// w(S, C_parent) (hit_leiden.rs:1528-1541): S's members (the initial ones and
// those merged since, two ascending lists), each member's row, entries whose
// neighbour lies in C_parent.
//
// Integral weights, in any order: thread t's share of nt (whole warps).  A lane
// takes a member, rows above 32 entries the whole warp.
__device__ __forceinline__ double det_wsp_any(const DetRefArgs& A, u32 S, u32 parent, u32 t,
                                              u32 nt) {
  const u32 lane = t & 31;
  const u32 ms = A.mstart[S];
  const u32 mc = ms == NONE32 ? 0u : A.mcount[S];
  const u32* f = A.f;
  const u32* col = A.col;
  const double* w = A.w;
  double acc = 0.0;
  for (u32 i0 = t - lane; i0 < mc; i0 += nt) {
    const u32 m = i0 + lane < mc ? A.members[ms + i0 + lane] : NONE32;
    const u64 a = m != NONE32 ? A.off[m] : 0, b = m != NONE32 ? A.off[m + 1] : 0;
    if (b - a <= 32)
      for (u64 q = a; q < b; ++q)
        if (f[col[q]] == parent) acc += w[q];
    for (u32 big = __ballot_sync(0xffffffffu, b - a > 32); big; big &= big - 1) {
      const u32 j = __ffs(big) - 1;
      const u64 bb = __shfl_sync(0xffffffffu, b, j);
      for (u64 q = __shfl_sync(0xffffffffu, a, j) + lane; q < bb; q += 32)
        if (f[col[q]] == parent) acc += w[q];
    }
  }
  for (u32 x = A.xhead[S]; x != NONE32; x = A.xnext[x])
    for (u64 q = A.off[x] + t; q < A.off[x + 1]; q += nt)
      if (f[col[q]] == parent) acc += w[q];
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// Other weights, by one warp: members in node order, rows in CSR order.
__device__ __forceinline__ double det_wsp_ordered(const DetRefArgs& A, u32 S, u32 parent) {
  const u32 ms = A.mstart[S];
  const u32 mc = ms == NONE32 ? 0u : A.mcount[S];
  const u32* f = A.f;
  const u32* col = A.col;
  const double* w = A.w;
  double acc = 0.0;
  u32 i = 0;
  u32 x = A.xhead[S];
  while (i < mc || x != NONE32) {
    u32 m;
    if (x == NONE32 || (i < mc && A.members[ms + i] < x)) {
      m = A.members[ms + i];
      ++i;
    } else {
      m = x;
      x = A.xnext[x];
    }
    acc = warp_ordered_sum(A.off[m], A.off[m + 1], acc, [&](u64 t) { return w[t]; },
                           [&](u64 t) { return f[col[t]] == parent; });
  }
  return acc;
}

// The same by the block; thread 0 holds it.
__device__ double det_wsp(const DetRefArgs& A, u32 S, u32 parent, double* r_g) {
  const u32 tid = threadIdx.x;
  double acc = 0.0;
  if (!A.ordered) {
    acc = det_wsp_any(A, S, parent, tid, DET_THREADS);
    if ((tid & 31) == 0) r_g[tid >> 5] = acc;
    __syncthreads();
    if (tid == 0)
      for (u32 x = 1; x < DET_WARPS; ++x) acc += r_g[x];
  } else if (tid < 32) {
    acc = det_wsp_ordered(A, S, parent);
  }
  __syncthreads();
  return acc;
}

// The merge of v into `best` (lane 0 / thread 0).  w(best, C) grows by v's own
// w(v, C) (`wv`), exactly so with integral weights; otherwise (wv < 0: not
// known) it is summed again when next needed.
__device__ __forceinline__ void det_merge(const DetRefArgs& A, u32 v, u32 cs, u32 best, double kv,
                                          double wv) {
  A.s[v] = best;
  A.sizes[cs] -= 1u;
  A.sizes[best] += 1u;
  A.dS[cs] = __dsub_rn(A.dS[cs], kv);
  A.dS[best] = __dadd_rn(A.dS[best], kv);
  // v joins best's members, in node order
  u32* link = &A.xhead[best];
  while (*link != NONE32 && *link < v) link = &A.xnext[*link];
  A.xnext[v] = *link;
  *link = v;
  if (wv < 0.0) A.wvalid[best] = 0;
  else if (A.wvalid[best]) A.wsp[best] += wv;
}

// Entries of a sub-community from which the block sums w(S, C): a warp takes some
// 1.5 us for 32 short rows or 32 entries of a long one, the block's barriers 2.
constexpr double DET_WSP_BLOCK = 4096.0;

enum : u32 { DET_STAYS = 0, DET_MERGED = 1, DET_BLOCK = 2 };

// One singleton by one warp (rows of up to DET_WARP_ROW entries): per-key sums
// in the warp's table, the candidates in gain order until the T-filter lets one
// pass.  No block barriers: they were most of a step.  DET_BLOCK: the step is the
// block's, a candidate is too large for one warp; nothing has changed then.
__device__ __forceinline__ u32 det_refine_warp(const DetRefArgs& A, DetWarp& T, u32 v, u32 cs) {
  const u32 lane = threadIdx.x & 31;
  const u64 o0 = A.off[v];
  const u32 deg = (u32)(A.off[v + 1] - o0);
  const u32 cc = A.f[v];
  const double kv = A.k[v];
  const double dcs = A.dS[cs], dpar = A.dcomm[cc];
  u32 cap = 64;
  while (cap < 2 * deg) cap <<= 1;
  const u32 mask = cap - 1;
  for (u32 x = lane; x < cap; x += 32) T.tk[x] = NONE32;
  u32 cq[DET_WARP_ROW / 32];
#pragma unroll
  for (u32 j = 0; j < DET_WARP_ROW / 32; ++j) {
    const u32 q = 32 * j + lane;
    cq[j] = q < deg ? A.col[o0 + q] : NONE32;
    if (q < deg) T.sw[q] = A.w[o0 + q];
  }
#pragma unroll
  for (u32 j = 0; j < DET_WARP_ROW / 32; ++j)
    if (cq[j] != NONE32) cq[j] = A.f[cq[j]] == cc ? A.s[cq[j]] : NONE32;
  double wv = -1.0;  // w(v, C), kept with integral weights
  if (!A.ordered) {
    wv = 0.0;
#pragma unroll
    for (u32 j = 0; j < DET_WARP_ROW / 32; ++j)
      if (cq[j] != NONE32) wv += T.sw[32 * j + lane];
    for (int o = 16; o; o >>= 1) wv += __shfl_xor_sync(0xffffffffu, wv, o);
  }
  __syncwarp();
#pragma unroll
  for (u32 j = 0; j < DET_WARP_ROW / 32; ++j) {
    if (32 * j >= deg) break;
    const u32 c = cq[j];
    const u32 grp = __match_any_sync(0xffffffffu, c);
    if (c != NONE32 && !(grp & ((1u << lane) - 1u))) {
      u32 slot = ((c * 2654435761u) >> 7) & mask;
      while (true) {  // the table holds at most deg < cap keys
        const u32 prev = atomicCAS(&T.tk[slot], NONE32, c);
        if (prev == NONE32 || prev == c) {
          double sum = prev == NONE32 ? 0.0 : T.tv[slot];
          for (u32 m = grp; m; m &= m - 1) sum = __dadd_rn(sum, T.sw[32 * j + __ffs(m) - 1]);
          T.tv[slot] = sum;
          if (prev == NONE32) T.tp[slot] = 32 * j + lane;
          break;
        }
        slot = (slot + 1) & mask;
      }
    }
    __syncwarp();
  }
  double wcur = 0.0;
  bool found = false;
  for (u32 x = lane; x < cap; x += 32)
    if (T.tk[x] == cs) {
      wcur = T.tv[x];
      found = true;
    }
  const u32 fm = __ballot_sync(0xffffffffu, found);
  wcur = __shfl_sync(0xffffffffu, wcur, fm ? __ffs(fm) - 1 : 0);
  if (!fm) wcur = 0.0;
  // gains in place of the sums; candidates without a positive one leave the table
  for (u32 x = lane; x < cap; x += 32) {
    const u32 c = T.tk[x];
    if (c == NONE32) continue;
    double gn = 0.0;
    if (c != cs) {
      const double dc = A.dS[c];
      if (det_may_gain(T.tv[x], dc, wcur, A.tw, A.gamma, kv, dcs))
        gn = move_gain(T.tv[x], wcur, A.tw, A.gamma, kv, dcs, dc);
    }
    if (gn > 0.0) T.tv[x] = gn;
    else T.tk[x] = NONE32;
  }
  __syncwarp();
  // The best candidate the T-filter lets through wins (the same choice as the
  // reference's strict '>' over the filtered list).
  while (true) {
    double g = 0.0;
    u32 p = NONE32, at = 0;
    for (u32 x = lane; x < cap; x += 32) {
      if (T.tk[x] == NONE32) continue;
      const double gn = T.tv[x];
      const u32 pc = T.tp[x];
      if (p == NONE32 || gn > g || (gn == g && pc < p)) {
        g = gn;
        p = pc;
        at = x;
      }
    }
    const u32 bl = det_warp_best(g, p);
    if (bl == 32) return DET_STAYS;
    const u32 slot = __shfl_sync(0xffffffffu, at, bl);
    const u32 cand = T.tk[slot];
    const double ds = A.dS[cand];  // (:1514-1548)
    bool skip = false;
    if (ds > 0.0) {
      double x;
      if (A.wvalid[cand]) {
        x = A.wsp[cand];
      } else {
        // (an integral d_S is at least the number of S's entries)
        if (!A.ordered && ds > DET_WSP_BLOCK) return DET_BLOCK;
        x = A.ordered ? det_wsp_ordered(A, cand, cc) : det_wsp_any(A, cand, cc, lane, 32);
        if (lane == 0) {
          A.wsp[cand] = x;
          A.wvalid[cand] = 1;
        }
      }
      skip = remove_gain(x, A.tw, A.gamma, ds, dpar) > 1e-9;
    }
    __syncwarp();
    if (!skip) {
      if (lane == 0) det_merge(A, v, cs, cand, kv, wv);
      __syncwarp();
      return DET_MERGED;
    }
    if (lane == 0) T.tk[slot] = NONE32;
    __syncwarp();
  }
}

// hit_leiden.rs:1392-1413 → try_merge_singleton_refinement (:1419-1511) with
// should_skip_candidate_t_filter (:1514-1548).
__global__ void __launch_bounds__(DET_THREADS) k_det_refine(DetRefArgs A) {
  __shared__ u32 s_nk, s_best, s_v, s_go;
  __shared__ double s_bestg, s_wsp;
  __shared__ double r_g[DET_WARPS];
  __shared__ u32 r_p[DET_WARPS], r_k[DET_WARPS];
  __shared__ double tile[32];
  const u32 tid = threadIdx.x;
  unsigned long long merges = 0;
  __shared__ DetWarp s_warp;
  __shared__ u32 s_i;
  for (u32 i = 0;; ++i) {
    // the first warp walks until a step needs the block
    if (tid < 32) {
      for (; i < A.nr; ++i) {
        const u32 v = A.rlist[i];
        const u32 cs = A.s[v];
        if (A.sizes[cs] != 1u) continue;  // singleton check (:1398-1400)
        if (A.off[v + 1] - A.off[v] > DET_WARP_ROW) break;
        const u32 r = det_refine_warp(A, s_warp, v, cs);
        if (r == DET_BLOCK) break;
        if (r == DET_MERGED) ++merges;
      }
      if (tid == 0) s_i = i;
    }
    __syncthreads();
    i = s_i;
    if (i >= A.nr) break;
    // ---- a long row or a large candidate, by the whole block ----
    const u32 v = A.rlist[i];
    const u32 cs = A.s[v];
    const u32 cc = A.f[v];
    const double kv = A.k[v];
    if (tid == 0) s_nk = 0;
    __syncthreads();
    const u32* f = A.f;
    const u32* col = A.col;
    const u32* s = A.s;
    det_row_sums(A.off[v], A.off[v + 1], A.w, A.ordered,
                 [&](u64 q) {
                   const u32 nb = col[q];
                   return f[nb] == cc ? s[nb] : NONE32;
                 },
                 A.bw, A.bp, A.klist, &s_nk, tile);
    __syncthreads();
    const double wcur = A.bw[cs];
    const double dcs = A.dS[cs];
    const double dpar = A.dcomm[cc];
    const u32 nk = s_nk;
    // Candidates in gain order; the best one the T-filter lets through wins
    // (the same choice as the reference's strict '>' over the filtered list).
    if (tid == 0) {
      s_best = cs;
      s_bestg = 0.0;
      s_go = 1;
    }
    __syncthreads();
    while (s_go) {
      double g = 0.0;
      u32 p = NONE32, kk = NONE32;
      for (u32 j = tid; j < nk; j += DET_THREADS) {
        const u32 c = A.klist[j];
        if (c == cs || A.bp[c] == NONE32 - 1u) continue;  // current, or filtered out
        const double gn = move_gain(A.bw[c], wcur, A.tw, A.gamma, kv, dcs, A.dS[c]);
        const u32 pc = A.bp[c];
        if (gn > 0.0 && (p == NONE32 || gn > g || (gn == g && pc < p))) {
          g = gn;
          p = pc;
          kk = c;
        }
      }
      det_argmax(g, p, kk, r_g, r_p, r_k);
      if (tid == 0) {
        s_v = p == NONE32 ? NONE32 : kk;
        s_bestg = g;
      }
      __syncthreads();
      const u32 cand = s_v;
      if (cand == NONE32) {
        if (tid == 0) s_go = 0;
        __syncthreads();
        break;
      }
      // T-filter of the candidate (:1514-1548)
      const double ds = A.dS[cand];
      bool skip = false;
      if (ds > 0.0) {
        double x;
        if (A.wvalid[cand]) {
          x = A.wsp[cand];
        } else {
          x = det_wsp(A, cand, cc, r_g);
          if (tid == 0) {
            A.wsp[cand] = x;
            A.wvalid[cand] = 1;
          }
        }
        if (tid == 0) s_wsp = x;
        __syncthreads();
        skip = remove_gain(s_wsp, A.tw, A.gamma, ds, dpar) > 1e-9;
      }
      if (tid == 0) {
        if (skip) {
          A.bp[cand] = NONE32 - 1u;  // filtered out for this vertex
        } else {
          s_best = cand;
          s_go = 0;
        }
      }
      __syncthreads();
    }
    const u32 best = s_best;
    const double bestg = s_bestg;
    // w(v, C), which w(best, C) grows by (integral weights: kept, not summed again)
    double wv = -1.0;
    if (!A.ordered && best != cs) {
      double acc = 0.0;
      for (u32 j = tid; j < nk; j += DET_THREADS) acc += A.bw[A.klist[j]];
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if ((tid & 31) == 0) r_g[tid >> 5] = acc;
      __syncthreads();
      if (tid == 0) {
        wv = 0.0;
        for (u32 x = 0; x < DET_WARPS; ++x) wv += r_g[x];
      }
    }
    __syncthreads();
    for (u32 j = tid; j < nk; j += DET_THREADS) {
      const u32 c = A.klist[j];
      A.bw[c] = 0.0;
      A.bp[c] = NONE32;
    }
    __syncthreads();
    if (best != cs && bestg > 0.0) {
      if (tid == 0) {
        det_merge(A, v, cs, best, kv, wv);
        ++merges;
      }
      __syncthreads();
    }
    __syncthreads();
  }
  if (tid == 0) A.out[0] = merges;
}

__global__ void k_member_index(const u32* sorted_s, u32 n, u32* mstart, u32* mcount) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
    const u32 c = sorted_s[i];
    if (i == 0 || sorted_s[i - 1] != c) mstart[c] = (u32)i;
    atomicAdd(&mcount[c], 1u);
  }
}

__global__ void k_k_keys(const u32* verts, u32 nv, const double* k, u64* keys) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < nv; i += (u64)gridDim.x * blockDim.x)
    keys[i] = double_key(k[verts[i]]);
}

__global__ void k_iota_det(u32* p, u32 n) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    p[i] = (u32)i;
}

// The deterministic merge step of inc_refinement: refined vertices `rv`
// (ascending, nr of them), sub-community sizes and degrees for ids < scap,
// d_parent per community.  Returns the number of merges.
u64 merge_singletons_det(Engine& E, Level& L, const u32* rv, u32 nr, u32* sizes, double* dS,
                         const double* dcomm, size_t scap) {
  Scratch& S = E.sc;
  cudaStream_t st = E.stream;
  const u32 n = L.g.n;
  u32* s = L.s_cur.p;
  // R sorted by k ascending, stable (hit_leiden.rs:1373-1374)
  S.det_k64.ensure(E.mem, nr);
  S.det_k64b.ensure(E.mem, nr);
  S.det_rsort.ensure(E.mem, nr);
  ++E.nlaunch, k_k_keys<<<grid_for(nr), 256, 0, st>>>(rv, nr, L.k.p, S.det_k64.p);
  HL_LAUNCH_CHECK();
  {
    u64* ki = S.det_k64.p;
    u64* ko = S.det_k64b.p;
    const u32* vi = rv;
    u32* vo = S.det_rsort.p;
    cub_run(E, [&](void* t, size_t& b) {
      return cub::DeviceRadixSort::SortPairs(t, b, ki, ko, vi, vo, (int64_t)nr, 0, 64, st);
    });
  }
  // nodes by (s, node): the initial members of every sub-community
  S.det_mkey.ensure(E.mem, n);
  S.det_mkey2.ensure(E.mem, n);
  S.det_mval.ensure(E.mem, n);
  S.det_members.ensure(E.mem, n);
  S.det_mstart.ensure(E.mem, scap);
  S.det_mcount.ensure(E.mem, scap);
  S.det_xhead.ensure(E.mem, scap);
  S.det_xnext.ensure(E.mem, n);
  S.det_wsp.ensure(E.mem, scap);
  S.det_wvalid.ensure(E.mem, scap);
  S.det_bw.ensure(E.mem, scap);
  S.det_bp.ensure(E.mem, scap);
  S.det_keys.ensure(E.mem, scap);
  S.det_out.ensure(E.mem, 8);
  HL_CUDA(cudaMemcpyAsync(S.det_mkey.p, s, sizeof(u32) * n, cudaMemcpyDeviceToDevice, st));
  ++E.nlaunch, k_iota_det<<<grid_for(n), 256, 0, st>>>(S.det_mval.p, n);
  HL_LAUNCH_CHECK();
  {
    u32* ki = S.det_mkey.p;
    u32* ko = S.det_mkey2.p;
    u32* vi = S.det_mval.p;
    u32* vo = S.det_members.p;
    cub_run(E, [&](void* t, size_t& b) {
      return cub::DeviceRadixSort::SortPairs(t, b, ki, ko, vi, vo, (int64_t)n, 0,
                                             bits_for(scap), st);
    });
  }
  ++E.nlaunch, k_fill_u32_det<<<grid_for(scap), 256, 0, st>>>(S.det_mstart.p, NONE32, scap);
  HL_CUDA(cudaMemsetAsync(S.det_mcount.p, 0, sizeof(u32) * scap, st));
  ++E.nlaunch, k_member_index<<<grid_for(n), 256, 0, st>>>(S.det_mkey2.p, n, S.det_mstart.p,
                                                            S.det_mcount.p);
  ++E.nlaunch, k_fill_u32_det<<<grid_for(scap), 256, 0, st>>>(S.det_xhead.p, NONE32, scap);
  ++E.nlaunch, k_fill_u32_det<<<grid_for(scap), 256, 0, st>>>(S.det_bp.p, NONE32, scap);
  HL_CUDA(cudaMemsetAsync(S.det_wvalid.p, 0, scap, st));
  HL_CUDA(cudaMemsetAsync(S.det_bw.p, 0, sizeof(double) * scap, st));
  HL_CUDA(cudaMemsetAsync(S.det_out.p, 0, 8 * sizeof(u64), st));
  HL_LAUNCH_CHECK();
  DetRefArgs A;
  A.off = L.g.off.p;
  A.col = L.g.col.p;
  A.w = L.g.w.p;
  A.f = L.f.p;
  A.s = s;
  A.k = L.k.p;
  A.dS = dS;
  A.sizes = sizes;
  A.dcomm = dcomm;
  A.rlist = S.det_rsort.p;
  A.nr = nr;
  A.bw = S.det_bw.p;
  A.bp = S.det_bp.p;
  A.klist = S.det_keys.p;
  A.wsp = S.det_wsp.p;
  A.wvalid = S.det_wvalid.p;
  A.members = S.det_members.p;
  A.mstart = S.det_mstart.p;
  A.mcount = S.det_mcount.p;
  A.xhead = S.det_xhead.p;
  A.xnext = S.det_xnext.p;
  A.tw = L.tw;
  A.gamma = E.cfg.resolution;
  A.ordered = !E.integral;
  A.out = reinterpret_cast<unsigned long long*>(S.det_out.p);
  ++E.nlaunch, k_det_refine<<<1, DET_THREADS, 0, st>>>(A);
  HL_LAUNCH_CHECK();
  return E.read_u64(S.det_out.p);
}

}  // namespace hl
