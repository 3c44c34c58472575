// gang_refine.cu — inc-refinement in one launch (hit_leiden.rs:1265-1390,
// :1554-1637; throughput.rs:239-359).
//
// The same steps and results as inc_refinement in refine.cu, on lists instead
// of whole-level passes: the vertices of affected sub-communities, the
// components split off, the refined singletons, their candidate
// sub-communities and those candidates' members.  The kernel leaves a step to
// the multi-kernel path, before it changes anything that step reads, when a
// list outgrows its room, a candidate needs the ordered T-filter sum, or a
// singleton's row does not fit a warp's table; the status word says which.
#include "csr_rebuild.cuh"
#include "gang.cuh"

namespace hl {

// Entries of a row a warp takes: an edge's union is a chain of dependent L2
// accesses, so long slices leave the other warps idle (20k nodes with 360k
// entries on 8 blocks: 390 us with 1024 entries and a find per union, 30-50 us
// with 256 and single neighbours hooked directly).
constexpr u32 REF_SLICE = 256;
constexpr u32 REF_MAXDEG = 256;    // singleton rows evaluated here
constexpr u32 REF_TAB = 2 * REF_MAXDEG;
constexpr u32 REF_MAX_REC = 65536;  // records sorted here (as AGG_MAX_REC)

struct RefCnt {  // zeroed by the host
  u32 smax, nitems, nsplit, nrefined, nsingle, nsitems, nbig, ncand;
  u32 nmitems, nrec, namb, merges, not_identity, pad_;
};

struct RefOut {
  u32 status, smax, nsplit, nrefined, nsingle, merges, pad_[2];
};

struct RefSmem {
  double tv[GANG_WARPS][REF_TAB];
  u32 tk[GANG_WARPS][REF_TAB];
  u32 tp[GANG_WARPS][REF_TAB];
  double sw[GANG_WARPS][32];
};

struct GangRefArgs {
  u32 n;
  const u64* off;
  const u32* col;
  const double* w;
  const u32* f;
  u32* s;
  const double* k;
  const u8* affected;
  u8* refined;           // padded to whole words
  u32 s_words;           // words of a bit set over the ids below the level's s bound
  u32 c_words;           // ... below that bound plus n
  u32 f_words;           // ... over the community ids
  bool same_f, throughput, integral, force_ordered, grid;
  u32 *affsc, *cand, *parent;  // bit sets over sub-communities / communities
  u32 *par, *root, *csize, *newid;
  u64* keep;
  u64 *items, *sitems, *mitems;  // (vertex << 32 | slice)
  u64 *skey, *skey2;             // split components (s << 32 | root)
  u32 *sidx, *sidx2;
  u32* origin;           // per new id: the sub-community it was split from
  u32 *rlist, *single, *clist;
  u64 *rec, *rid, *rtmp;  // (id << 33 | is community << 32 | vertex)
  u32 *ridx, *rtidx;
  double* rval;
  double *dS, *dcomm, *wsp;
  unsigned long long* wcnt;
  u32* minmem;
  u8* blocked;
  u32* to;
  double* gain;
  double tw, gamma;
  u32* part;
  RefCnt* cnt;
  u32* cnt_next;
  RefOut* out;
};

__device__ __forceinline__ bool bit_test(const u32* b, u32 i) { return (b[i >> 5] >> (i & 31)) & 1u; }
// Sets bit i; true for the one caller that set it.
__device__ __forceinline__ bool bit_first(u32* b, u32 i) {
  const u32 m = 1u << (i & 31);
  if (b[i >> 5] & m) return false;
  return (atomicOr(&b[i >> 5], m) & m) == 0;
}

// The slices of v's row onto a work list.
__device__ __forceinline__ void push_row(u64* list, u32* count, u32 v, u64 deg) {
  const u32 ns = deg ? (u32)((deg + REF_SLICE - 1) / REF_SLICE) : 1u;
  const u32 at = atomicAdd(count, ns);
  for (u32 x = 0; x < ns; ++x) list[at + x] = ((u64)v << 32) | x;
}

// Parents are read from L2: the other blocks hook roots meanwhile.
__device__ __forceinline__ u32 gr_find(u32* par, u32 x) {
  u32 p = __ldcg(&par[x]);
  while (p != x) {
    const u32 gp = __ldcg(&par[p]);
    if (gp != p) __stcg(&par[x], gp);  // path halving (always an ancestor)
    x = p;
    p = gp;
  }
  return x;
}

// Hooks the larger root under the smaller, so a root is its component's
// minimum vertex.
__device__ __forceinline__ void gr_unite(u32* par, u32 a, u32 b) {
  while (true) {
    a = gr_find(par, a);
    b = gr_find(par, b);
    if (a == b) return;
    const u32 lo = min(a, b), hi = max(a, b);
    if (atomicCAS(&par[hi], hi, lo) == hi) return;
  }
}

__device__ __forceinline__ u32 gr_hash(u32 x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// Best same-community neighbour sub-community of singleton v on the snapshot
// (throughput.rs:291-359), by one warp: per-key sums in CSR order, the first
// CSR position on ties.
__device__ __forceinline__ void gr_eval(const GangRefArgs& A, RefSmem& W, u32 v, u32& to_out,
                                        double& gain_out) {
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  u32* tk = W.tk[wib];
  u32* tp = W.tp[wib];
  double* tv = W.tv[wib];
  double* sw = W.sw[wib];
  const u64 o0 = A.off[v], o1 = A.off[v + 1];
  const u32 fv = A.f[v], cur = A.s[v];
  const double kv = A.k[v];
  u32 cap = 64;
  while (cap < 2 * (o1 - o0)) cap <<= 1;
  const u32 mask = cap - 1;
  for (u32 x = lane; x < cap; x += 32) tk[x] = NONE32;
  __syncwarp();
  for (u64 b0 = o0; b0 < o1; b0 += 32) {
    const u64 q = b0 + lane;
    u32 key = NONE32;
    double wv = 0.0;
    if (q < o1) {
      const u32 nb = A.col[q];
      wv = A.w[q];
      if (A.f[nb] == fv) key = A.s[nb];
    }
    sw[lane] = wv;
    __syncwarp();
    const u32 grp = __match_any_sync(0xffffffffu, key);
    if (key != NONE32 && lane == (u32)(__ffs(grp) - 1)) {
      u32 slot = gr_hash(key) & mask;
      while (true) {  // the table holds at most deg < cap keys
        const u32 prev = atomicCAS(&tk[slot], NONE32, key);
        if (prev == NONE32 || prev == key) {
          double sum = prev == NONE32 ? 0.0 : tv[slot];
          for (u32 m = grp; m; m &= m - 1) sum = __dadd_rn(sum, sw[__ffs(m) - 1]);
          tv[slot] = sum;
          if (prev == NONE32) tp[slot] = (u32)(q - o0);
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
    if (tk[x] == cur) {
      wcur = tv[x];
      found = true;
    }
  const u32 fm = __ballot_sync(0xffffffffu, found);
  wcur = __shfl_sync(0xffffffffu, wcur, fm ? __ffs(fm) - 1 : 0);
  if (!fm) wcur = 0.0;
  double g = -1.0;
  u32 p = NONE32, kk = cur;
  if (A.tw != 0.0) {
    const double dcur = A.dS[cur];
    for (u32 x = lane; x < cap; x += 32) {
      const u32 key = tk[x];
      if (key == NONE32 || key == cur || A.blocked[key]) continue;
      const double gn = move_gain(tv[x], wcur, A.tw, A.gamma, kv, dcur, A.dS[key]);
      const u32 pp = tp[x];
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
  __syncwarp();
  const bool pos = p != NONE32 && g > 0.0;
  to_out = pos ? kk : cur;
  gain_out = pos ? g : 0.0;
}

__device__ __forceinline__ void gr_result(const Gang& G, const GangRefArgs& A, u32 status) {
  if (G.thread() != 0) return;
  A.out->status = status;
  A.out->smax = A.cnt->smax;
  A.out->nsplit = A.cnt->nsplit;
  A.out->nrefined = A.cnt->nrefined;
  A.out->nsingle = A.cnt->nsingle;
  A.out->merges = A.cnt->merges;
}

// What bounds it: a chain of some fifteen dependent steps of 1-10 us each
// (barriers, L2 round trips); on hub levels the unions.  Against the
// multi-kernel form (some fifty launches and six host reads a level), the
// stage of one level: 5 levels of 250-400 nodes 330 -> 27 us, 3 levels of
// 7-10k nodes 370 -> 51 us, 10 levels of 10-50k nodes 445 -> 88 us, 10 levels
// of 0.13-1M nodes with f64 weights 235 -> 66 us (events around the launch).
__global__ void __launch_bounds__(GANG_THREADS, 1) k_gang_refine(GangRefArgs A) {
  extern __shared__ __align__(16) unsigned char gr_raw[];
  RefSmem& W = *reinterpret_cast<RefSmem*>(gr_raw);
  __shared__ GangSmem S;
  const Gang G = gang_make(A.grid);
  const u32 lane = threadIdx.x & 31;
  const u32 gt = G.thread(), gts = G.threads();
  RefCnt& C = *A.cnt;
  gang_clear_next(G, A.cnt_next);
  // ---- clear; the largest sub-community id ----
  for (u32 i = gt; i < A.s_words; i += gts) A.affsc[i] = 0;
  for (u32 i = gt; i < (A.n + 3) / 4; i += gts) reinterpret_cast<u32*>(A.refined)[i] = 0;
  {
    u32 mx = 0;
    for (u32 v = gt; v < A.n; v += gts) mx = max(mx, A.s[v]);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(&C.smax, mx);
  }
  G.sync();
  // ---- affected sub-communities and their vertices ----
  for (u32 v = gt; v < A.n; v += gts)
    if (A.affected[v]) bit_first(A.affsc, A.s[v]);
  G.sync();
  const u32 smax = C.smax;
  for (u32 v = gt; v < A.n; v += gts) {
    const u32 sv = A.s[v];
    if (!bit_test(A.affsc, sv)) continue;
    A.par[v] = v;
    A.csize[v] = 0;
    A.keep[sv] = 0;
    push_row(A.items, &C.nitems, v, A.off[v + 1] - A.off[v]);
  }
  G.sync();
  // ---- components over edges inside a sub-community, each edge once ----
  const u32 nitems = C.nitems;
  for (u32 i = G.warp(); i < nitems; i += G.warps()) {
    const u64 it = A.items[i];
    const u32 v = (u32)(it >> 32);
    const u64 lo = A.off[v] + (u64)(u32)it * REF_SLICE;
    const u64 hi = min(A.off[v + 1], lo + REF_SLICE);
    if (hi <= lo || A.col[hi - 1] <= v) continue;  // each edge once, from its lower end
    const u32 sv = A.s[v], fv = A.f[v];
    const u32 rv = __ldcg(&A.par[v]);  // v or an ancestor of v
    for (u64 p0 = lo + lane; p0 < hi; p0 += 128) {
      u32 nb[4], sn[4], fn[4], pn[4];
      bool open[4];  // not known to share v's tree yet
#pragma unroll
      for (int j = 0; j < 4; ++j) nb[j] = p0 + 32 * j < hi ? A.col[p0 + 32 * j] : v;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sn[j] = sv + 1;
        if (nb[j] > v) {
          sn[j] = A.s[nb[j]];
          fn[j] = A.same_f ? A.f[nb[j]] : fv;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        open[j] = sn[j] == sv && fn[j] == fv;
        if (open[j]) pn[j] = __ldcg(&A.par[nb[j]]);
      }
      // a neighbour that is still alone is hooked under v's side at once (its
      // id is larger, so parents stay below their children); the rest unite
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (open[j] && (pn[j] == rv || (pn[j] == nb[j] &&
                                        atomicCAS(&A.par[nb[j]], nb[j], rv) == nb[j])))
          open[j] = false;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (open[j]) gr_unite(A.par, v, nb[j]);
    }
  }
  G.sync();
  // ---- roots and sizes (the forest no longer changes) ----
  for (u32 i = gt; i < nitems; i += gts) {
    const u64 it = A.items[i];
    if ((u32)it) continue;
    const u32 v = (u32)(it >> 32);
    u32 r = v;
    while (A.par[r] != r) r = A.par[r];
    A.root[v] = r;
    atomicAdd(&A.csize[r], 1u);
  }
  G.sync();
  // ---- the largest component keeps the id, the last one on ties ----
  for (u32 i = gt; i < nitems; i += gts) {
    const u64 it = A.items[i];
    const u32 v = (u32)(it >> 32);
    if ((u32)it || A.root[v] != v) continue;
    atomicMax(reinterpret_cast<unsigned long long*>(&A.keep[A.s[v]]),
              ((unsigned long long)A.csize[v] << 32) | v);
  }
  G.sync();
  for (u32 i = gt; i < nitems; i += gts) {
    const u64 it = A.items[i];
    const u32 v = (u32)(it >> 32);
    if ((u32)it || A.root[v] != v) continue;
    const u32 sv = A.s[v];
    if ((u32)A.keep[sv] != v) A.skey[atomicAdd(&C.nsplit, 1u)] = ((u64)sv << 32) | v;
  }
  G.sync();
  const u32 m = C.nsplit;
  if (m > REF_MAX_REC) {
    gr_result(G, A, REF_HOST_ALL);
    return;
  }
  if (m) {
    // ---- fresh ids in (sub-community, minimum vertex) order ----
    gang_sort(
        G, S, m, [&](u32 i) { return A.skey[i]; }, [](u32 i) { return i; }, A.skey2, A.sidx2,
        [&](u32 r, u64 key, u32) {
          A.newid[(u32)key] = smax + 1 + r;
          A.origin[r] = (u32)(key >> 32);
        });
    for (u32 i = gt; i < nitems; i += gts) {
      const u64 it = A.items[i];
      if ((u32)it) continue;
      const u32 v = (u32)(it >> 32), r = A.root[v];
      if ((u32)A.keep[A.s[v]] == r) continue;  // A.s[v] is still v's own old id
      A.s[v] = A.newid[r];
      A.refined[v] = 1;
      A.rlist[atomicAdd(&C.nrefined, 1u)] = v;
      if (A.csize[r] == 1) A.single[atomicAdd(&C.nsingle, 1u)] = v;
    }
    G.sync();
  }
  {
    // is_initial (hit_leiden.rs:1333-1339): s is the identity => R = all
    u32 bad = 0;
    for (u32 v = gt; v < A.n && !bad; v += gts) bad = A.s[v] != v ? 1u : 0u;
    __syncwarp();
    if (__any_sync(0xffffffffu, bad != 0) && lane == 0) atomicOr(&C.not_identity, 1u);
  }
  G.sync();
  const bool all = C.not_identity == 0;
  if (all) {
    for (u32 v = gt; v < A.n; v += gts) {
      A.refined[v] = 1;
      A.rlist[v] = v;
      A.single[v] = v;
    }
    G.sync();
    if (gt == 0) C.nrefined = C.nsingle = A.n;
    G.sync();
  }
  const u32 nr = C.nrefined, ns = C.nsingle;
  if (!A.throughput && nr) {
    gr_result(G, A, REF_HOST_MERGE);
    return;
  }
  if (!ns) {
    gr_result(G, A, REF_DONE);
    return;
  }
  // many singletons (s is the identity: all of the level): the multi-kernel
  // path spreads them over the whole GPU at full occupancy (9,877 on a cluster
  // of 8 blocks: 0.7 ms a load slower here)
  if (A.force_ordered || ns > 16 * G.warps()) {
    gr_result(G, A, REF_HOST_MERGE);
    return;
  }
  // ---- refined singletons ----
  for (u32 i = gt; i < A.c_words; i += gts) A.cand[i] = 0;
  for (u32 i = gt; i < A.f_words; i += gts) A.parent[i] = 0;
  for (u32 i = gt; i < ns; i += gts) {
    const u32 v = A.single[i];
    const u64 deg = A.off[v + 1] - A.off[v];
    A.dS[A.s[v]] = A.k[v];  // its own sub-community holds v alone
    if (deg > REF_MAXDEG) atomicAdd(&C.nbig, 1u);
    push_row(A.sitems, &C.nsitems, v, deg);
  }
  G.sync();
  // ---- candidate sub-communities of the T-filter (hit_leiden.rs:1567-1586) ----
  const u32 nsitems = C.nsitems;
  for (u32 i = G.warp(); i < nsitems; i += G.warps()) {
    const u64 it = A.sitems[i];
    const u32 v = (u32)(it >> 32);
    const u64 lo = A.off[v] + (u64)(u32)it * REF_SLICE;
    const u64 hi = min(A.off[v + 1], lo + REF_SLICE);
    const u32 sv = A.s[v], fv = A.f[v];
    for (u64 p0 = lo + lane; p0 < hi; p0 += 128) {
      u32 nb[4], fn[4], sn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) nb[j] = p0 + 32 * j < hi ? A.col[p0 + 32 * j] : NONE32;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (nb[j] != NONE32) {
          fn[j] = A.f[nb[j]];
          sn[j] = A.s[nb[j]];
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const u32 x = sn[j];
        if (nb[j] == NONE32 || fn[j] != fv || x == sv || !bit_first(A.cand, x)) continue;
        A.clist[atomicAdd(&C.ncand, 1u)] = x;
        A.minmem[x] = NONE32;
        A.wsp[x] = 0.0;
        A.wcnt[x] = 0;
        A.dS[x] = 0.0;
      }
    }
  }
  G.sync();
  // ---- their members ----
  const u32 ncand = C.ncand;
  if (ncand) {
    for (u32 v0 = gt - lane; v0 < A.n; v0 += gts) {
      const u32 v = v0 + lane;
      const u32 x = v < A.n ? A.s[v] : 0;
      const bool on = v < A.n && bit_test(A.cand, x);
      if (A.integral) warp_add_by_id(A.dS, x, on ? A.k[v] : 0.0, on);
      if (!on) continue;
      atomicMin(&A.minmem[x], v);
      push_row(A.mitems, &C.nmitems, v, A.off[v + 1] - A.off[v]);
      if (!A.integral) {
        const u32 at = atomicAdd(&C.nrec, 1u);
        if (at < REF_MAX_REC) A.rec[at] = ((u64)x << 33) | v;
      }
    }
    G.sync();
    for (u32 i = gt; i < ncand; i += gts) {
      const u32 c = A.f[A.minmem[A.clist[i]]];
      if (bit_first(A.parent, c)) A.dcomm[c] = 0.0;
    }
    G.sync();
    // ---- w(S, C_parent) in any order, d of the parents ----
    const u32 nm = C.nmitems;
    for (u32 i = G.warp(); i < nm; i += G.warps()) {
      const u64 it = A.mitems[i];
      const u32 v = (u32)(it >> 32), x = A.s[v];
      const u64 lo = A.off[v] + (u64)(u32)it * REF_SLICE;
      const u64 hi = min(A.off[v + 1], lo + REF_SLICE);
      const u32 parent = A.f[A.minmem[x]];
      double sum = 0.0;
      u32 c = 0;
      for (u64 p0 = lo + lane; p0 < hi; p0 += 128) {
        u32 nb[4];
        double y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          nb[j] = p0 + 32 * j < hi ? A.col[p0 + 32 * j] : NONE32;
          y[j] = p0 + 32 * j < hi ? A.w[p0 + 32 * j] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (nb[j] != NONE32 && A.f[nb[j]] == parent) {
            sum += y[j];
            ++c;
          }
      }
      for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      c = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0 && c) {
        atomicAdd(&A.wsp[x], sum);
        atomicAdd(&A.wcnt[x], (unsigned long long)c);
      }
    }
    for (u32 v0 = gt - lane; v0 < A.n; v0 += gts) {
      const u32 v = v0 + lane;
      const u32 c = v < A.n ? A.f[v] : 0;
      const bool on = v < A.n && bit_test(A.parent, c);
      if (A.integral) {
        warp_add_by_id(A.dcomm, c, on ? A.k[v] : 0.0, on);
      } else if (on) {
        const u32 at = atomicAdd(&C.nrec, 1u);
        if (at < REF_MAX_REC) A.rec[at] = ((u64)c << 33) | (1ull << 32) | v;
      }
    }
    G.sync();
    const u32 nrec = C.nrec;
    if (nrec > REF_MAX_REC) {
      gr_result(G, A, REF_HOST_MERGE);
      return;
    }
    if (nrec) {
      // ---- d_S and d_C, each over its members in node order ----
      gang_sort(
          G, S, nrec, [&](u32 i) { return A.rec[i]; }, [](u32 i) { return i; }, A.rtmp, A.rtidx,
          [&](u32 r, u64 key, u32) {
            A.rid[r] = key >> 32;
            A.rval[r] = A.k[(u32)key];
          });
      gang_segment_sums(G, nrec, A.rid, A.rval, W.tv[threadIdx.x >> 5], [&](u64 id, double x) {
        (id & 1 ? A.dcomm : A.dS)[id >> 1] = x;
      });
      G.sync();
    }
    // ---- T-filter decisions (the rounding window of k_blocked_bounds) ----
    u32 amb = 0;
    for (u32 i = gt; i < ncand; i += gts) {
      const u32 x = A.clist[i];
      const double ds = A.dS[x];
      u8 b = 0;
      if (ds > 0.0) {
        const double dpar = A.dcomm[A.f[A.minmem[x]]];
        const double sum = A.wsp[x];
        const unsigned long long N = A.wcnt[x];
        if (A.integral || N <= 1) {
          b = remove_gain(sum, A.tw, A.gamma, ds, dpar) > 1e-9 ? 1 : 0;
        } else {
          const double err = __dmul_rn(__dmul_rn(sum, (double)N), 0x1p-50);
          const double lo = fmax(__dsub_rn(sum, err), 0.0);
          const double hi = __dadd_rn(sum, err);
          if (remove_gain(hi, A.tw, A.gamma, ds, dpar) > 1e-9) b = 1;
          else if (remove_gain(lo, A.tw, A.gamma, ds, dpar) > 1e-9) ++amb;
        }
      }
      A.blocked[x] = b;
    }
    if (amb) atomicAdd(&C.namb, amb);
    G.sync();
    if (C.namb) {
      gr_result(G, A, REF_HOST_MERGE);
      return;
    }
  }
  if (C.nbig) {
    gr_result(G, A, REF_HOST_EVAL);
    return;
  }
  // ---- Jacobi singleton merge ----
  for (u32 i = G.warp(); i < ns; i += G.warps()) {
    u32 to;
    double g;
    gr_eval(A, W, A.single[i], to, g);
    if (lane == 0) {
      A.to[i] = to;
      A.gain[i] = g;
    }
  }
  G.sync();
  u32 merged = 0;
  for (u32 i = gt; i < ns; i += gts)
    if (A.gain[i] > 0.0) {
      A.s[A.single[i]] = A.to[i];
      ++merged;
    }
  if (merged) atomicAdd(&C.merges, merged);
  G.sync();
  gr_result(G, A, REF_DONE);
}

static std::atomic<bool> g_ref_attr[64];

// The bootstrap refines every vertex of every level from the identity: worth
// one launch while one block per SM has few singletons a warp.
bool gang_refine_fits(Engine& E, const Level& L) {
  return !E.lean && L.g.n > 0 && L.g.n < (1u << 30) &&
         (!E.in_bootstrap || L.g.n <= 16 * GANG_WARPS * GANG_MAX_BLOCKS);
}

// One launch of the refinement.  The caller continues on the multi-kernel path
// from the step *status names (REF_*).
u32 gang_refine(Engine& E, Level& L, bool cc_same_community, RefineOut& out) {
  Scratch& S = E.sc;
  const u32 n = L.g.n;
  const int dev = E.device;
  if (dev >= 0 && dev < 64 && !g_ref_attr[dev]) {
    HL_CUDA(cudaFuncSetAttribute(k_gang_refine, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RefSmem)));
    g_ref_attr[dev] = true;
  }
  const u64 nslice = L.g.nnz / REF_SLICE + 1;
  const u64 scap = (u64)L.s_bound + n;
  const GangShape shape =
      gang_shape(E, 2ull * n + L.g.nnz / 8 + (E.in_bootstrap ? 128ull * n : 0));
  S.refined.ensure(E.mem, ((size_t)n + 3) & ~(size_t)3);
  S.gr_bits.ensure(E.mem, (L.s_bound + 31) / 32 + (scap + 31) / 32 + (2ull * n + 33) / 32);
  S.par.ensure(E.mem, n);
  S.uroot.ensure(E.mem, n);
  S.csize.ensure(E.mem, n);
  S.newid.ensure(E.mem, n);
  S.keep.ensure(E.mem, scap);
  S.gr_items.ensure(E.mem, 3 * (n + nslice));
  S.gkey.ensure(E.mem, n);
  S.gkey2.ensure(E.mem, n);
  S.order2.ensure(E.mem, n);
  S.origin.ensure(E.mem, n);
  S.act.ensure(E.mem, n);
  S.cand_idx.ensure(E.mem, n);
  S.cand_node.ensure(E.mem, scap);
  const u64 nrec = E.integral ? 1 : std::min<u64>(2ull * n, REF_MAX_REC);
  S.rkeys.ensure(E.mem, nrec);
  S.rkeys2.ensure(E.mem, nrec);
  S.keys.ensure(E.mem, nrec);
  S.idx.ensure(E.mem, nrec);
  S.fvals.ensure(E.mem, nrec);
  S.dS.ensure(E.mem, scap);
  S.dcomm.ensure(E.mem, 2 * (size_t)n + 2);
  S.wsp.ensure(E.mem, scap);
  S.wcnt.ensure(E.mem, scap);
  S.minmem.ensure(E.mem, scap);
  S.blocked.ensure(E.mem, scap);
  S.cand_to.ensure(E.mem, n);
  S.cand_gain.ensure(E.mem, n);
  S.gang_part.ensure(E.mem, GANG_MAX_BLOCKS);
  GangRefArgs A{};
  A.n = n;
  A.off = L.g.off.p;
  A.col = L.g.col.p;
  A.w = L.g.w.p;
  A.f = L.f.p;
  A.s = L.s_cur.p;
  A.k = L.k.p;
  A.affected = S.affected.p;
  A.refined = S.refined.p;
  A.s_words = (L.s_bound + 31) / 32;
  A.c_words = (u32)((scap + 31) / 32);
  A.f_words = (u32)((2ull * n + 33) / 32);
  A.same_f = cc_same_community;
  A.throughput = E.cfg.mode != HL_MODE_DETERMINISTIC;
  A.integral = E.integral;
  A.force_ordered = g_exact_tfilter.load() != 0;
  A.grid = shape.grid;
  A.affsc = S.gr_bits.p;
  A.cand = A.affsc + A.s_words;
  A.parent = A.cand + A.c_words;
  A.par = S.par.p;
  A.root = S.uroot.p;
  A.csize = S.csize.p;
  A.newid = S.newid.p;
  A.keep = S.keep.p;
  A.items = S.gr_items.p;
  A.sitems = A.items + n + nslice;
  A.mitems = A.sitems + n + nslice;
  A.skey = S.gkey.p;
  A.skey2 = S.gkey2.p;
  A.sidx2 = S.order2.p;
  A.origin = S.origin.p;
  A.rlist = S.act.p;
  A.single = S.cand_idx.p;
  A.clist = S.cand_node.p;
  A.rec = S.rkeys.p;
  A.rid = S.rkeys2.p;
  A.rtmp = S.keys.p;
  A.rtidx = S.idx.p;
  A.rval = S.fvals.p;
  A.dS = S.dS.p;
  A.dcomm = S.dcomm.p;
  A.wsp = S.wsp.p;
  A.wcnt = reinterpret_cast<unsigned long long*>(S.wcnt.p);
  A.minmem = S.minmem.p;
  A.blocked = S.blocked.p;
  A.to = S.cand_to.p;
  A.gain = S.cand_gain.p;
  A.tw = L.tw;
  A.gamma = E.cfg.resolution;
  A.part = S.gang_part.p;
  A.cnt = reinterpret_cast<RefCnt*>(gang_counters(E, &A.cnt_next));
  A.out = reinterpret_cast<RefOut*>(E.hs.p);
  cudaEvent_t ev = E.kt_begin();
  gang_launch(E, reinterpret_cast<const void*>(&k_gang_refine), shape, sizeof(RefSmem), &A);
  gang_turn(E);
  E.kt_end(KT_GANG_REFINE, ev);
  RefOut o;
  E.sync();
  std::memcpy(&o, E.hs.p, sizeof(o));
  if (o.status == REF_HOST_ALL) return o.status;
  out.smax_before = o.smax;
  out.splits = o.nsplit;
  out.refined = o.nrefined;
  out.merges = o.merges;
  out.singles = o.nsingle;
  E.n_new = o.nsplit;
  E.new_base = o.smax + 1;
  L.s_bound = std::max(n, o.smax + o.nsplit + 1);
  return o.status;
}

}  // namespace hl
