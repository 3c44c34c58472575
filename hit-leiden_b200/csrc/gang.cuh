// gang.cuh — one launch for a whole stage of the update path.
//
// A batch on a small or mid-size level is bound by its launches and by the
// host reads between them, not by memory: a stage is some twenty dependent
// steps of a few microseconds each.  The gang kernels run all steps of a stage
// in one launch, with a barrier over all of their blocks between steps and
// every size kept on the device; the host reads one small result per stage.
//
// The blocks of a gang are one block, one thread-block cluster (its hardware
// barrier costs a fraction of a microsecond, and clusters of different graphs
// run side by side) or a cooperative grid of one block per SM for the large
// levels.  All of them execute every barrier: branches around a barrier are
// taken on values that every block reads alike.
//
// Arrays that a kernel writes and reads again after a barrier carry no
// __restrict__ / const __restrict__ qualifiers (they must not go through the
// non-coherent cache).
#pragma once
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>

#include "hl_engine.cuh"

namespace hl {

constexpr u32 GANG_THREADS = 512;
constexpr u32 GANG_WARPS = GANG_THREADS / 32;
constexpr u32 GANG_MAX_BLOCKS = 148;
constexpr u32 GSORT_CHUNK = 1024;  // records sorted by one block at a time
constexpr u32 GANG_WORDS = 2048;   // 64-bit words of a block's shared memory (GangSmem)
constexpr u32 GSORT_ILP = 8;       // chunks a record's rank is looked up in at once

struct Gang {
  u32 rank, nct;
  bool grid;
  __device__ __forceinline__ u32 thread() const { return rank * GANG_THREADS + threadIdx.x; }
  __device__ __forceinline__ u32 threads() const { return nct * GANG_THREADS; }
  // consecutive warps sit on different blocks, so a short list spreads out
  __device__ __forceinline__ u32 warp() const { return (threadIdx.x >> 5) * nct + rank; }
  __device__ __forceinline__ u32 warps() const { return nct * GANG_WARPS; }
  __device__ __forceinline__ void sync() const {
    if (grid) {
      cooperative_groups::this_grid().sync();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    }
  }
};

__device__ __forceinline__ Gang gang_make(bool grid) {
  Gang G;
  G.rank = blockIdx.x;
  G.nct = gridDim.x;
  G.grid = grid;
  return G;
}

// A stage's counters: one of two blocks of GANG_CNT zeroed words by turns, and
// every launch clears the block of the next one (the one before it is done
// with it).  The result goes straight to the engine's pinned block.  A memset
// before and a copy after each launch cost 5-8 us of a stage's 40-100.
constexpr u32 GANG_CNT = 64;
__device__ __forceinline__ void gang_clear_next(const Gang& G, u32* next) {
  if (G.thread() < GANG_CNT) next[G.thread()] = 0;
}

// Shared memory of the primitives below (one instance per kernel, static or
// at the start of the dynamic block).
struct GangSmem {
  u64 key[GANG_WORDS];
  u32 val[GSORT_CHUNK];
  u32 wsum[GANG_WARPS + 1];
  u32 bcast[2];
};

// Sum of x over the block's threads, and the sum over the threads before this
// one (exclusive).  Two block barriers.
__device__ __forceinline__ u32 block_scan(GangSmem& S, u32 x, u32& total) {
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  u32 inc = x;
#pragma unroll
  for (u32 o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) S.wsum[wib] = inc;
  __syncthreads();
  u32 before = 0, tot = 0;
#pragma unroll
  for (u32 i = 0; i < GANG_WARPS; ++i) {
    const u32 y = S.wsum[i];
    if (i < wib) before += y;
    tot += y;
  }
  __syncthreads();
  total = tot;
  return before + inc - x;
}

// d[c] += x for the lanes with `on` (the whole warp calls it), where sums are
// exact in any order.  One community may hold most of a level, and 2M atomics on
// its word take 3 ms: the ids of the first two lanes left are looked for in the
// others, and what eight lanes or more share adds up before its atomic.
__device__ __forceinline__ void warp_add_by_id(double* d, u32 c, double x, bool on) {
  const u32 lane = threadIdx.x & 31;
  u32 rest = __ballot_sync(0xffffffffu, on);
#pragma unroll
  for (u32 t = 0; t < 2; ++t) {
    if (!rest) return;
    const u32 l = __ffs(rest) - 1;
    const u32 cl = __shfl_sync(0xffffffffu, c, l);
    const u32 same = __ballot_sync(0xffffffffu, ((rest >> lane) & 1u) && c == cl);
    const bool mine = (same >> lane) & 1u;
    if (__popc(same) >= 8) {
      double y = mine ? x : 0.0;
      for (u32 o = 16; o; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      if (lane == l) atomicAdd(&d[c], y);
    } else if (mine) {
      atomicAdd(&d[c], x);
    }
    rest &= ~same;
  }
  if ((rest >> lane) & 1u) atomicAdd(&d[c], x);
}

// Exclusive prefix sums of val(0..N-1), handed to out(i, prefix); returns the
// total.  val is evaluated twice.  One gang barrier inside; the caller places
// one before it reads what out wrote (which also frees `part`, nct words).
template <typename V, typename O>
__device__ __forceinline__ u32 gang_scan(const Gang& G, GangSmem& S, u32 N, V val, O out,
                                         u32* part) {
  const u32 per = ((N + G.nct - 1) / G.nct + GANG_THREADS - 1) / GANG_THREADS * GANG_THREADS;
  const u32 lo = min(N, G.rank * per), hi = min(N, lo + per);
  u32 base = 0, total = 0;
  if (G.nct > 1) {
    u32 sum = 0;
    for (u32 i = lo + threadIdx.x; i < hi; i += GANG_THREADS) sum += val(i);
    u32 tot;
    block_scan(S, sum, tot);
    if (threadIdx.x == 0) part[G.rank] = tot;
    G.sync();
    if (threadIdx.x < 32) {
      u32 b = 0, t = 0;
      for (u32 r = threadIdx.x; r < G.nct; r += 32) {
        const u32 y = part[r];
        if (r < G.rank) b += y;
        t += y;
      }
      b = __reduce_add_sync(0xffffffffu, b);
      t = __reduce_add_sync(0xffffffffu, t);
      if (threadIdx.x == 0) {
        S.bcast[0] = b;
        S.bcast[1] = t;
      }
    }
    __syncthreads();
    base = S.bcast[0];
    total = S.bcast[1];
    __syncthreads();
  }
  u32 run = base;
  for (u32 i0 = lo; i0 < hi; i0 += GANG_THREADS) {
    const u32 i = i0 + threadIdx.x;
    const u32 x = i < hi ? val(i) : 0u;
    u32 tot;
    const u32 ex = block_scan(S, x, tot);
    if (i < hi) out(i, run + ex);
    run += tot;
  }
  if (G.nct == 1) total = run;
  return total;
}

// Ascending sort of the P (key, value) records (a power of two from 64 to
// GSORT_CHUNK) in S.key / S.val by (key, value), by the block: every warp sorts
// 32 records through its lanes, then runs merge pairwise, each record finding
// its place by a bisection in the sibling run.
//
// What bounds it: a sort runs once or twice per launch, so straight-line code
// costs its instruction fetches: with the 15 lane stages unrolled four times,
// 2048 records took 55 us, 29 us of it in those stages; rolled and shared by all
// sorts of a kernel, 33 us.  512 records take 8 us, 1024 take 15; chunks above
// that lose more than a rank among fewer chunks gains.
static __device__ __noinline__ void block_sort(GangSmem* Sp, u32 P) {
  __builtin_assume(__isShared(Sp));
  GangSmem& S = *Sp;
  constexpr u32 PER = GSORT_CHUNK / GANG_THREADS;
  const u32 tid = threadIdx.x, lane = tid & 31;
  const u32 per = (P + GANG_THREADS - 1) / GANG_THREADS;  // uniform
  u64 k[PER];
  u32 v[PER], pos[PER];
#pragma unroll
  for (u32 j = 0; j < PER; ++j) {
    const u32 e = tid + j * GANG_THREADS;
    k[j] = e < P ? S.key[e] : ~0ull;
    v[j] = e < P ? S.val[e] : NONE32;
  }
#pragma unroll 1
  for (u32 size = 2; size <= 32; size <<= 1) {
#pragma unroll 1
    for (u32 stride = size >> 1; stride; stride >>= 1) {
      const bool want_less = ((lane & size) == 0) == ((lane & stride) == 0);
#pragma unroll
      for (u32 j = 0; j < PER; ++j) {
        if (j >= per) break;
        const u64 ok = __shfl_xor_sync(0xffffffffu, k[j], stride);
        const u32 ov = __shfl_xor_sync(0xffffffffu, v[j], stride);
        const bool less = ok < k[j] || (ok == k[j] && ov < v[j]);
        const bool differ = ok != k[j] || ov != v[j];
        if (differ && less == want_less) {
          k[j] = ok;
          v[j] = ov;
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (u32 j = 0; j < PER; ++j) {
    const u32 e = tid + j * GANG_THREADS;
    if (e >= P) continue;
    S.key[e] = k[j];
    S.val[e] = v[j];
  }
  __syncthreads();
#pragma unroll 1
  for (u32 run = 32; run < P; run <<= 1) {
#pragma unroll
    for (u32 j = 0; j < PER; ++j) pos[j] = 0;
#pragma unroll 1
    for (u32 half = run; half; half >>= 1) {
#pragma unroll
      for (u32 j = 0; j < PER; ++j) {
        if (j >= per) break;
        const u32 e = tid + j * GANG_THREADS;
        if (e >= P || pos[j] + half > run) continue;
        const u32 sib = (e & ~(run - 1)) ^ run;
        const u32 at = sib + pos[j] + half - 1;
        const u64 x = S.key[at];
        bool before = x < k[j];
        if (x == k[j]) {  // equal records: the left run's come first
          const u32 y = S.val[at];
          before = y < v[j] || (y == v[j] && sib < e);
        }
        if (before) pos[j] += half;
      }
    }
    __syncthreads();
#pragma unroll
    for (u32 j = 0; j < PER; ++j) {
      const u32 e = tid + j * GANG_THREADS;
      if (e >= P) continue;
      const u32 to = (e & ~(2 * run - 1)) + (e & (run - 1)) + pos[j];
      S.key[to] = k[j];
      S.val[to] = v[j];
    }
    __syncthreads();
#pragma unroll
    for (u32 j = 0; j < PER; ++j) {
      const u32 e = tid + j * GANG_THREADS;
      if (e >= P) continue;
      k[j] = S.key[e];
      v[j] = S.val[e];
    }
  }
}

// How many records of the sorted chunks first, first + GSORT_ILP, ... come
// before record (k, v) of chunk `mine` (tk / tv: N records in chunks of ch);
// GSORT_ILP bisections side by side; equal records: earlier chunks first.
static __device__ __noinline__ u32 gang_rank(const u64* tk, const u32* tv, u32 N, u32 ch, u32 nch,
                                             u32 first, u32 step, u32 mine, u64 k, u32 v) {
  u32 rank = 0;
#pragma unroll 1
  for (u32 c0 = first; c0 < nch; c0 += step) {
    u32 pos[GSORT_ILP];
#pragma unroll
    for (u32 j = 0; j < GSORT_ILP; ++j) pos[j] = 0;
#pragma unroll 1
    for (u32 half = ch; half; half >>= 1) {
      u64 probe[GSORT_ILP];
      bool in[GSORT_ILP];
#pragma unroll
      for (u32 j = 0; j < GSORT_ILP; ++j) {
        const u32 c = c0 + j;
        const u32 at = c * ch + pos[j] + half;  // one past the probed record
        in[j] = c < nch && c != mine && pos[j] + half <= ch && at <= N;
        probe[j] = in[j] ? tk[at - 1] : 0ull;
      }
#pragma unroll
      for (u32 j = 0; j < GSORT_ILP; ++j) {
        if (!in[j] || probe[j] > k) continue;
        if (probe[j] == k) {
          const u32 y = tv[(c0 + j) * ch + pos[j] + half - 1];
          if (y > v || (y == v && c0 + j > mine)) continue;
        }
        pos[j] += half;
      }
    }
#pragma unroll
    for (u32 j = 0; j < GSORT_ILP; ++j) rank += pos[j];
  }
  return rank;
}

// Ascending sort of N (key, value) records by (key, value); with the record's
// index as its value, the stable sort by key.  Blocks sort chunks of up to
// GSORT_CHUNK records in shared memory; after a barrier every record
// finds its rank by a bisection in each other chunk and is handed to
// emit(rank, key, value).  `tk`/`tv` take the sorted chunks.  Two gang barriers
// inside (one when a single chunk holds everything); the caller's emitted
// output is visible after the last one.
//
// For a few thousand records this takes 10-20 us; a radix sort of the same keys
// is six to nine dependent kernel launches.
template <typename K, typename VL, typename EM>
__device__ __forceinline__ void gang_sort(const Gang& G, GangSmem& S, u32 N, K key_of, VL val_of,
                                          u64* tk, u32* tv, EM emit) {
  const u32 tid = threadIdx.x;
  // Few chunks, because a record's rank costs one bisection per chunk, and at
  // most one a block: on a grid 32 (a rank among 32 chunks takes four lanes what
  // one among 8 takes one).
  u32 ch = 64;
  while (ch < GSORT_CHUNK && ch * min(G.nct, 32u) < N) ch <<= 1;
  const u32 nch = (N + ch - 1) / ch;
  for (u32 c = G.rank; c < nch; c += G.nct) {
    const u32 base = c * ch;
    const u32 cnt = min(ch, N - base);
    u32 P = 64;  // the padded length of this chunk
    while (P < cnt) P <<= 1;
    for (u32 i = tid; i < P; i += GANG_THREADS) {
      S.key[i] = i < cnt ? key_of(base + i) : ~0ull;
      S.val[i] = i < cnt ? val_of(base + i) : NONE32;
    }
    __syncthreads();
    block_sort(&S, P);
    for (u32 i = tid; i < cnt; i += GANG_THREADS) {
      if (nch == 1) {
        emit(i, S.key[i], S.val[i]);
      } else {
        tk[base + i] = S.key[i];
        tv[base + i] = S.val[i];
      }
    }
    __syncthreads();
  }
  G.sync();
  if (nch == 1) return;
  // a warp takes 32 / L records, L lanes a record share its chunks; consecutive
  // warps sit on different blocks, which spreads the probes over the chip
  u32 L = 1;
  while (L < 32 && L * GSORT_ILP < nch) L <<= 1;
  const u32 per = 32 / L, g = (tid & 31) / per;
  for (u32 e0 = G.warp() * per; e0 < N; e0 += G.warps() * per) {
    const u32 e = e0 + ((tid & 31) & (per - 1));
    const bool on = e < N;
    const u64 k = on ? tk[e] : 0ull;
    const u32 v = on ? tv[e] : 0u;
    const u32 mine = e / ch;
    u32 rank = 0;
    if (on) rank = gang_rank(tk, tv, N, ch, nch, g * GSORT_ILP, L * GSORT_ILP, mine, k, v);
    for (u32 o = per; o < 32; o <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (on && g == 0) emit(rank + e - mine * ch, k, v);
  }
  G.sync();
}

// Stable counting sort of the vertices 0..n-1 by a label below 2^bits: sorted
// labels in `lab`, vertices in `idx`, both ascending within.  8 bits a pass;
// every warp of the gang owns a consecutive run of records, counts it per
// digit (`hist`, 256 words a warp, digit-major), and after a scan places it in
// order.  lab2 / idx2 are the other halves of the double buffers; the result is
// in the buffers that *second names.  All barriers inside; the output is
// visible on return.
template <typename L0>
__device__ __forceinline__ void gang_label_sort(const Gang& G, GangSmem& S, u32 n, u32 bits,
                                                L0 label, u32* lab, u32* idx, u32* lab2,
                                                u32* idx2, u32* hist, u32* part, bool* second) {
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  // consecutive runs for consecutive (block, warp): run order is record order
  const u32 run = G.rank * GANG_WARPS + wib, runs = G.warps();
  const u32 per = ((n + runs - 1) / runs + 31) & ~31u;
  const u32 lo = min(n, run * per), hi = min(n, lo + per);
  u32* cnt = reinterpret_cast<u32*>(S.key) + wib * 256;  // 16 warps x 256 words
  bool from_label = true;
  u32 *ki = nullptr, *vi = nullptr, *ko = lab, *vo = idx;
  for (u32 shift = 0; shift < bits; shift += 8) {
    for (u32 d = lane; d < 256; d += 32) cnt[d] = 0;
    __syncwarp();
    for (u32 i0 = lo; i0 < hi; i0 += 32) {
      const u32 i = i0 + lane;
      const u32 k = i < hi ? (from_label ? label(i) : ki[i]) : 0u;
      const u32 d = i < hi ? (k >> shift) & 255u : 256u;
      const u32 grp = __match_any_sync(0xffffffffu, d);
      if (i < hi && lane == (u32)(__ffs(grp) - 1)) cnt[d] += __popc(grp);
      __syncwarp();
    }
    for (u32 d = lane; d < 256; d += 32) hist[d * runs + run] = cnt[d];
    G.sync();
    gang_scan(
        G, S, 256 * runs, [&](u32 i) { return hist[i]; }, [&](u32 i, u32 ex) { hist[i] = ex; },
        part);
    G.sync();
    for (u32 d = lane; d < 256; d += 32) cnt[d] = hist[d * runs + run];
    __syncwarp();
    for (u32 i0 = lo; i0 < hi; i0 += 32) {
      const u32 i = i0 + lane;
      const u32 k = i < hi ? (from_label ? label(i) : ki[i]) : 0u;
      const u32 v = i < hi ? (from_label ? i : vi[i]) : 0u;
      const u32 d = i < hi ? (k >> shift) & 255u : 256u;
      const u32 grp = __match_any_sync(0xffffffffu, d);
      if (i < hi) {
        const u32 at = cnt[d] + __popc(grp & ((1u << lane) - 1u));
        ko[at] = k;
        vo[at] = v;
      }
      __syncwarp();
      if (i < hi && lane == (u32)(__ffs(grp) - 1)) cnt[d] += __popc(grp);
      __syncwarp();
    }
    __syncthreads();  // cnt aliases S.key, which gang_scan does not touch
    G.sync();
    from_label = false;
    *second = ko == lab2;
    u32* t = ko;
    ko = t == lab ? lab2 : lab;
    ki = t;
    t = vo;
    vo = t == idx ? idx2 : idx;
    vi = t;
  }
}

// Ordered sums of x over the segments of equal values in the ascending labels
// lab[0..n): done(label, sum) is called by one lane per segment.  A warp takes
// 32 positions and the segments that start there; one that ends within the next
// position is the last of its 32, found by a 32-way search.  Segments of up to
// 16 terms take a lane, longer ones the warp (`buf`: CHAIN_TILE doubles of it).
// ANY_ORDER: sums that are exact in every order, the long ones lane by lane.
// init(label): what a segment's sum starts from.
struct FromZero {
  template <typename T>
  __device__ __forceinline__ double operator()(T) const { return 0.0; }
};
template <bool ANY_ORDER = false, typename T, typename DN, typename IN = FromZero>
__device__ __forceinline__ void gang_segment_sums(const Gang& G, u32 n, const T* lab,
                                                  const double* x, double* buf, DN done,
                                                  IN init = IN{}) {
  const u32 lane = threadIdx.x & 31;
  for (u32 t0 = G.warp() * 32; t0 < n; t0 += G.warps() * 32) {
    const u32 t = t0 + lane;
    const T c = t < n ? lab[t] : T(0);
    const T before = t < n && t > 0 ? lab[t - 1] : T(0);
    const u32 hm = __ballot_sync(0xffffffffu, t < n && (t == 0 || before != c));
    if (!hm) continue;
    // the last segment's end
    const u32 last = 31 - __clz(hm);
    const T cl = __shfl_sync(0xffffffffu, c, last);
    u32 lo = t0 + last, hi = n;  // lab[lo] == cl
    u32 step = 1;                // most segments are short: gallop first
    while (true) {
      const u64 p = (u64)lo + (u64)step * (lane + 1);
      const u32 m = __ballot_sync(0xffffffffu, p < hi && lab[p] == cl);
      const u32 j = (u32)__popc(m);
      if (j == 32) {
        lo += 32 * step;
        step *= 32;
        continue;
      }
      const u64 nhi = (u64)lo + (u64)step * (j + 1);
      lo += step * j;
      hi = nhi < hi ? (u32)nhi : hi;
      if (step == 1) break;
      step /= 32;
    }
    const u32 end_last = lo + 1;
    const bool head = (hm >> lane) & 1u;
    const u32 above = hm & ~((2u << lane) - 1u);
    const u32 end = above ? t0 + __ffs(above) - 1 : end_last;
    const u32 len = head ? end - t : 0;
    if (len && len <= 16) {
      double s = init(c);
      u32 q = t;
      for (; q + 4 <= end; q += 4) {
        const double y0 = x[q], y1 = x[q + 1], y2 = x[q + 2], y3 = x[q + 3];
        s = __dadd_rn(s, y0);
        s = __dadd_rn(s, y1);
        s = __dadd_rn(s, y2);
        s = __dadd_rn(s, y3);
      }
      for (; q < end; ++q) s = __dadd_rn(s, x[q]);
      done(c, s);
    }
    for (u32 bm = __ballot_sync(0xffffffffu, len > 16); bm; bm &= bm - 1) {
      const u32 l = __ffs(bm) - 1;
      const u32 e = __shfl_sync(0xffffffffu, end, l);
      double s = init(__shfl_sync(0xffffffffu, c, l));
      if (ANY_ORDER) {
#pragma unroll 8
        for (u32 q = t0 + l + lane; q < e; q += 32) s += x[q];
        for (u32 o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      } else {
        s = warp_long_sum(t0 + l, e, s, x, buf);
      }
      if (lane == l) done(c, s);
    }
  }
}

// ---------------------------------------------------------------------------
// Host side: the shape of a gang.
// ---------------------------------------------------------------------------
struct GangShape {
  u32 blocks;
  bool grid;  // cooperative grid instead of a cluster
};

constexpr u64 GANG_BLOCK_WORK = 4096;           // entries up to which one block takes a stage
u64 gang_cluster_work(const Engine& E);          // ... a cluster of 8
// Shape for a stage that touches about `work` entries.
GangShape gang_shape(Engine& E, u64 work);
// Launch of a gang kernel with one argument struct.
u32* gang_counters(Engine& E, u32** next);  // this launch's block, the next one's
void gang_turn(Engine& E);                  // a launch that clears *next is on its way
void gang_launch(Engine& E, const void* kernel, const GangShape& s, size_t smem, void* args);

}  // namespace hl
