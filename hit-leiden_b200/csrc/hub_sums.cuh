// hub_sums.cuh — per-key sums of one long row by a whole block, and the best
// move from them.
//
// With f64 weights every key's sum has to be extended in CSR order.  Instead of
// walking the row tile by tile with a barrier and a serial fold per tile, the
// block sorts the row's weights by key once: every key gets a dense id, each
// warp counts its consecutive stretch of the row per id, prefix sums over
// (id, warp) give every stretch its place, and a second walk moves the weights
// there in CSR order.  A key's sum is then one chain over consecutive terms, and
// the keys' chains run side by side, one per lane.
#pragma once
#include "hl_internal.cuh"

namespace hl {

constexpr u32 HUB_TAB = 4096;     // hash slots
constexpr u32 HUB_KEYS = 2048;    // distinct keys at most
constexpr u32 HUB_MAXDEG = 16384; // entries at most (16-bit ids, counts and scratch)
constexpr u32 HUB_LANE = 48;      // chains up to this length: a lane each

__device__ __forceinline__ u32 hub_hash(u32 x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

template <u32 WARPS>
struct HubSmem {
  double sum[HUB_KEYS];                // per id; integral weights: the integer sum's bits
  double chain[WARPS][CHAIN_TILE];
  u32 tab[HUB_TAB];                    // keys
  u32 key[HUB_KEYS];                   // per id
  u32 pos[HUB_KEYS];                   // first CSR position
  u32 start[HUB_KEYS + 1];             // first term in the sorted row
  u32 wsum[WARPS + 1];
  u32 used, over;
  unsigned short id[HUB_TAB];          // per slot
  unsigned short cnt[WARPS][HUB_KEYS]; // per warp stretch and id
  double red_g[WARPS];
  u32 red_p[WARPS], red_k[WARPS];
  double wcur;
};

// Dense id of `key`, claimed on first sight; HUB_KEYS when the row has too many
// (H.over is set then).  Ids are published by the claiming lane; other lanes
// look the id up after a block barrier.
template <u32 WARPS>
__device__ __forceinline__ u32 hub_slot(HubSmem<WARPS>& H, u32 key) {
  u32 slot = hub_hash(key) & (HUB_TAB - 1);
  while (!*reinterpret_cast<volatile u32*>(&H.over)) {
    const u32 prev = atomicCAS(&H.tab[slot], NONE32, key);
    if (prev == key) return slot;
    if (prev == NONE32) {
      const u32 d = atomicAdd(&H.used, 1u);
      if (d < HUB_KEYS) {
        H.id[slot] = (unsigned short)d;
        H.key[d] = key;
      } else {
        H.over = 1;
      }
      return slot;
    }
    slot = (slot + 1) & (HUB_TAB - 1);
  }
  return slot;
}

// Sums of row [o0, o1) per key_of(neighbour) (NONE32: skipped) into H.key / sum /
// pos, ids 0..H.used-1.  False (for the whole block) when the row has more than
// HUB_KEYS distinct keys.  `gslot` / `gw` are the block's scratch of HUB_MAXDEG
// entries.  All threads of the block call it.
template <u32 WARPS, typename K>
__device__ __forceinline__ bool hub_sums(HubSmem<WARPS>& H, u64 o0, u64 o1, const u32* col,
                                         const double* w, bool integral, K key_of,
                                         unsigned short* gslot, double* gw) {
  constexpr u32 NT = WARPS * 32;
  const u32 tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const u32 lt = (1u << lane) - 1u;
  const u32 D = (u32)(o1 - o0);
  for (u32 i = tid; i < HUB_TAB; i += NT) H.tab[i] = NONE32;
  if (tid == 0) {
    H.used = 0;
    H.over = 0;
  }
  __syncthreads();
  // ---- keys and their slots ----
  for (u32 q0 = tid; q0 < D; q0 += 4 * NT) {
    u32 k[4];
#pragma unroll
    for (u32 j = 0; j < 4; ++j) k[j] = q0 + j * NT < D ? col[o0 + q0 + j * NT] : NONE32;
#pragma unroll
    for (u32 j = 0; j < 4; ++j) k[j] = k[j] != NONE32 ? key_of(k[j]) : NONE32;
#pragma unroll
    for (u32 j = 0; j < 4; ++j)
      if (q0 + j * NT < D)
        gslot[q0 + j * NT] =
            k[j] == NONE32 ? (unsigned short)0xFFFF : (unsigned short)hub_slot(H, k[j]);
  }
  __syncthreads();
  if (H.over) return false;
  const u32 U = H.used;
  // ---- per warp stretch, entries per id ----
  const u32 per = ((D + WARPS - 1) / WARPS + 31) & ~31u;
  const u32 lo = min(D, wib * per), hi = min(D, lo + per);
  if (integral) {
    for (u32 i = tid; i < U; i += NT) {
      H.sum[i] = 0.0;  // integer 0
      H.pos[i] = NONE32;
    }
    __syncthreads();
    for (u32 q0 = lo; q0 < hi; q0 += 32) {
      const u32 q = q0 + lane;
      const u32 sl = q < hi ? gslot[q] : 0xFFFFu;
      const bool ok = sl != 0xFFFFu;
      const u32 d = ok ? H.id[sl] : NONE32 - lane;
      unsigned long long x = ok ? (unsigned long long)w[o0 + q] : 0ull;
      const u32 grp = __match_any_sync(0xffffffffu, d);
      // the lanes of one id add up first: a row's heavy key would otherwise
      // queue 32 atomics on one word
      u32 multi = __ballot_sync(0xffffffffu, ok && (grp & (grp - 1)) && !(grp & lt));
      while (multi) {
        const u32 l = __ffs(multi) - 1;
        const u32 gm = __shfl_sync(0xffffffffu, grp, l);
        unsigned long long s = (gm >> lane) & 1u ? x : 0ull;
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == l) x = s;
        multi &= multi - 1;
      }
      if (ok && !(grp & lt)) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&H.sum[d]), x);
        atomicMin(&H.pos[d], q);
      }
    }
    __syncthreads();
    for (u32 i = tid; i < U; i += NT)
      H.sum[i] = (double)(unsigned long long)__double_as_longlong(H.sum[i]);
    __syncthreads();
    return true;
  }
  unsigned short* cw = H.cnt[wib];
  for (u32 i = lane; i < U; i += 32) cw[i] = 0;
  __syncwarp();
  for (u32 q0 = lo; q0 < hi; q0 += 32) {
    const u32 q = q0 + lane;
    const u32 sl = q < hi ? gslot[q] : 0xFFFFu;
    const u32 d = sl != 0xFFFFu ? H.id[sl] : NONE32;
    const u32 grp = __match_any_sync(0xffffffffu, d);
    if (d != NONE32 && !(grp & lt)) cw[d] += (unsigned short)__popc(grp);
    __syncwarp();
  }
  __syncthreads();
  // ---- starts: prefix over ids, stretches before this one added ----
  constexpr u32 IDS = HUB_KEYS / NT;  // consecutive ids of a thread
  u32 tot[IDS], mine = 0;
#pragma unroll
  for (u32 j = 0; j < IDS; ++j) {
    const u32 d = tid * IDS + j;
    u32 t = 0;
    if (d < U)
      for (u32 x = 0; x < WARPS; ++x) {
        const u32 c = H.cnt[x][d];
        H.cnt[x][d] = (unsigned short)t;
        t += c;
      }
    tot[j] = t;
    mine += t;
  }
  u32 inc = mine;
#pragma unroll
  for (u32 o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) H.wsum[wib] = inc;
  __syncthreads();
  u32 at = inc - mine;
  for (u32 x = 0; x < wib; ++x) at += H.wsum[x];
#pragma unroll
  for (u32 j = 0; j < IDS; ++j) {
    H.start[tid * IDS + j] = at;
    at += tot[j];
  }
  if (tid == NT - 1) H.start[HUB_KEYS] = at;
  __syncthreads();
  // ---- weights into (id, CSR) order ----
  for (u32 q0 = lo; q0 < hi; q0 += 32) {
    const u32 q = q0 + lane;
    const u32 sl = q < hi ? gslot[q] : 0xFFFFu;
    const double x = q < hi ? w[o0 + q] : 0.0;
    const u32 d = sl != 0xFFFFu ? H.id[sl] : NONE32;
    const u32 grp = __match_any_sync(0xffffffffu, d);
    if (d != NONE32) {
      const u32 rank = cw[d] + __popc(grp & lt);
      gw[H.start[d] + rank] = x;
      if (rank == 0) H.pos[d] = q;
    }
    __syncwarp();
    if (d != NONE32 && !(grp & lt)) cw[d] += (unsigned short)__popc(grp);
    __syncwarp();
  }
  __syncthreads();
  // ---- one chain per id ----
  for (u32 d0 = wib * 32; d0 < U; d0 += NT) {
    const u32 d = d0 + lane;
    const u32 a = d < U ? H.start[d] : 0, b = d < U ? H.start[d + 1] : 0;
    if (b - a <= HUB_LANE && d < U) {
      double x = 0.0;
      u32 t = a;
      for (; t + 4 <= b; t += 4) {
        const double y0 = gw[t], y1 = gw[t + 1], y2 = gw[t + 2], y3 = gw[t + 3];
        x = __dadd_rn(x, y0);
        x = __dadd_rn(x, y1);
        x = __dadd_rn(x, y2);
        x = __dadd_rn(x, y3);
      }
      for (; t < b; ++t) x = __dadd_rn(x, gw[t]);
      H.sum[d] = x;
    }
  }
  // the long ones by a warp each, spread over the warps
  for (u32 d0 = 0, turn = 0; d0 < U; d0 += 32) {
    const u32 d = d0 + lane;
    u32 m = __ballot_sync(0xffffffffu, d < U && H.start[d + 1] - H.start[d] > HUB_LANE);
    for (; m; m &= m - 1, ++turn) {
      if (turn % WARPS != wib) continue;
      const u32 l = d0 + __ffs(m) - 1;
      const double x = warp_chain_sum(H.start[l], H.start[l + 1], 0.0, gw, H.chain[wib]);
      if (lane == 0) H.sum[l] = x;
    }
  }
  __syncthreads();
  return true;
}

// Best key by gain (ties: the first CSR position) over H's ids but `cur`;
// valid in thread 0, with w(v, cur) in H.wcur for everyone.
template <u32 WARPS, typename D>
__device__ __forceinline__ void hub_best(HubSmem<WARPS>& H, u32 cur, double tw, double gamma,
                                         double kv, double dcur, D d_of, double& g, u32& p,
                                         u32& kk) {
  constexpr u32 NT = WARPS * 32;
  const u32 tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const u32 U = H.used;
  if (tid == 0) H.wcur = 0.0;
  __syncthreads();
  for (u32 i = tid; i < U; i += NT)
    if (H.key[i] == cur) H.wcur = H.sum[i];
  __syncthreads();
  const double wcur = H.wcur;
  g = -1.0;
  p = NONE32;
  kk = cur;
  if (tw != 0.0) {
    GainScreen scr;  // exact gains only for candidates that may win
    scr.init(wcur, tw, gamma, kv, dcur);
    for (u32 i = tid; i < U; i += NT) {
      const u32 key = H.key[i];
      if (key == cur) continue;
      const double dk = d_of(key), x = H.sum[i];
      if (!scr.keep(x, dk)) continue;
      const double gn = move_gain(x, wcur, tw, gamma, kv, dcur, dk);
      const u32 pp = H.pos[i];
      if (p == NONE32 || gn > g || (gn == g && pp < p)) {
        g = gn;
        p = pp;
        kk = key;
      }
    }
  }
  for (int o = 16; o; o >>= 1) {
    const double og = __shfl_xor_sync(0xffffffffu, g, o);
    const u32 op = __shfl_xor_sync(0xffffffffu, p, o);
    const u32 ok = __shfl_xor_sync(0xffffffffu, kk, o);
    if (op != NONE32 && (p == NONE32 || og > g || (og == g && op < p))) {
      g = og;
      p = op;
      kk = ok;
    }
  }
  if (lane == 0) {
    H.red_g[wib] = g;
    H.red_p[wib] = p;
    H.red_k[wib] = kk;
  }
  __syncthreads();
  if (tid == 0)
    for (u32 x = 1; x < WARPS; ++x)
      if (H.red_p[x] != NONE32 &&
          (p == NONE32 || H.red_g[x] > g || (H.red_g[x] == g && H.red_p[x] < p))) {
        g = H.red_g[x];
        p = H.red_p[x];
        kk = H.red_k[x];
      }
}

}  // namespace hl
