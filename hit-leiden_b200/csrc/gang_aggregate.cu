// gang_aggregate.cu — inc-aggregation in one launch (hit_leiden.rs:1639-1731),
// with the growth of the next level before it and the communities' projection
// onto it.
//
// The same steps and results as inc_aggregation, graph_grow_nodes,
// inherit_new_nodes and project_up: ΔH records in the reference's push order,
// sorted stably by key, each key summed in that order, |w| <= 1e-9 dropped.
// More than AGG_MAX_REC records are left to the multi-kernel aggregation
// (nothing but the next level's new nodes and projection has changed then).
#include "csr_rebuild.cuh"
#include "gang.cuh"

namespace hl {

constexpr u32 AGG_SLICE = 512;       // entries of a row a warp emits
constexpr u32 AGG_LANE = 16;         // sums up to this length: a lane each
// Records sorted here: those of a largest batch (GANG_BATCH_MAX), two an update;
// the sort's ranks grow with the square, and the radix sort takes over.
constexpr u32 AGG_MAX_REC = 65536;

struct AggCnt {  // zeroed by the host
  u32 nitems, nlong;
  unsigned long long total;  // records of the changed rows
  u32 pad_[28];
};

struct AggOut {
  u32 status, count, records, pad_;
};

struct GangAggArgs {
  // level p
  u32 n;
  const u64* off;
  const u32* col;
  const double* w;
  const u32* f;
  const u32* s_cur;
  u32* s_pre;
  const u8* refined;
  // level p + 1: nodes [hn_old, hn) are new
  u32 hn_old, hn, new_base, n_new;
  u64 h_nnz;
  u64* h_off;
  u32 *h_f, *h_g, *h_spre, *h_scur;
  double* h_k;
  const u32* origin;
  u8* kflag;
  u32* last;
  // ΔG
  const u32* du;
  const u32* dv;
  const double* dw;
  u32 dk;
  bool aggregate, grid;
  u64 *items, *items2, *itmp;  // changed rows: (vertex << 32 | slice)
  u32 *itv, *icnt, *ipos;
  u64 *keys, *keys2, *ktmp;
  u32 *ktv;
  double *vals, *sw, *xs;
  u32* longs;
  u32* part;
  u32 *ou, *ov;
  double* ow;
  AggCnt* cnt;
  u32* cnt_next;
  AggOut* out;
};

__device__ __forceinline__ u64 gg_pair(u32 a, u32 b) {
  return a <= b ? ((u64)a << 32) | b : ((u64)b << 32) | a;
}

// Weight of v's self-loop in the aggregation: half the sum of its two stored
// entries; 0 when it has none.
__device__ __forceinline__ double gg_loop(const GangAggArgs& A, u32 v, u64 o0, u64 o1) {
  double x = 0.0;
  for (u64 p = lower_bound_u32(A.col, o0, o1, v); p < o1 && A.col[p] == v; ++p)
    x = __dadd_rn(x, A.w[p]);
  return x / 2.0;
}

// Records of one slice: counted, or written from position `at` on.
template <bool EMIT>
__device__ __forceinline__ u32 gg_slice(const GangAggArgs& A, u64 it, u32 at) {
  const u32 lane = threadIdx.x & 31;
  const u32 v = (u32)(it >> 32);
  const u64 o0 = A.off[v], o1 = A.off[v + 1];
  const u64 lo = o0 + (u64)(u32)it * AGG_SLICE;
  const u64 hi = min(o1, lo + AGG_SLICE);
  const u32 sp = A.s_pre[v], sc = A.s_cur[v];
  u32 c = 0;
  for (u64 b0 = lo; b0 < hi; b0 += 128) {
    u32 nb[4], np_[4], nc[4];
    u8 rf[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const u64 p = b0 + 32 * j + lane;
      nb[j] = p < hi ? A.col[p] : NONE32;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (nb[j] != NONE32) {
        np_[j] = A.s_pre[nb[j]];
        nc[j] = A.s_cur[nb[j]];
        rf[j] = A.refined[nb[j]];
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool emit =
          nb[j] != NONE32 && nb[j] != v && (nc[j] == np_[j] || v < nb[j] || !rf[j]);
      const u32 m = __ballot_sync(0xffffffffu, emit);
      if (EMIT && emit) {
        const u32 t = at + c + 2 * __popc(m & ((1u << lane) - 1u));
        const double x = A.w[b0 + 32 * j + lane];
        A.keys[t] = gg_pair(sp, np_[j]);
        A.vals[t] = -x;
        A.keys[t + 1] = gg_pair(sc, nc[j]);
        A.vals[t + 1] = x;
      }
      c += 2 * __popc(m);
    }
  }
  if (hi == o1) {  // the row's last slice: its self-loop
    const double x = gg_loop(A, v, o0, o1);
    if (fabs(x) > 1e-12) {
      if (EMIT && lane == 0) {
        A.keys[at + c] = gg_pair(sp, sp);
        A.vals[at + c] = -x;
        A.keys[at + c + 1] = gg_pair(sc, sc);
        A.vals[at + c + 1] = x;
      }
      c += 2;
    }
  }
  return c;
}

// What bounds it: the chain of its two sorts, scans and barriers.  Against the
// multi-kernel form (some thirty launches and five host reads a level), the
// stage with the next level's growth and projection: 5 levels of 250-400 nodes
// 290 -> 22 us, 10 levels of 10-50k nodes 370 -> 79 us, 10 levels of 0.13-1M
// nodes 420 -> 61 us (events around the launch).
__global__ void __launch_bounds__(GANG_THREADS, 1) k_gang_aggregate(GangAggArgs A) {
  __shared__ GangSmem S;
  __shared__ __align__(16) double chain[GANG_WARPS][CHAIN_TILE];
  const Gang G = gang_make(A.grid);
  const u32 lane = threadIdx.x & 31;
  const u32 gt = G.thread(), gts = G.threads();
  AggCnt& C = *A.cnt;
  gang_clear_next(G, A.cnt_next);
  // ---- new nodes of the level above start isolated with identity maps ----
  for (u32 x = gt; x < A.hn; x += gts) {
    A.last[x] = 0;
    A.kflag[x] = 0;
    if (x < A.hn_old) continue;
    A.h_off[x + 1] = A.h_nnz;
    A.h_f[x] = A.h_g[x] = A.h_spre[x] = A.h_scur[x] = x;
    A.h_k[x] = 0.0;
  }
  // ---- changed rows ----
  if (A.aggregate)
    for (u32 v = gt; v < A.n; v += gts) {
      if (!A.refined[v] || A.s_cur[v] == A.s_pre[v]) continue;
      const u64 deg = A.off[v + 1] - A.off[v];
      const u32 ns = deg ? (u32)((deg + AGG_SLICE - 1) / AGG_SLICE) : 1u;
      const u32 at = atomicAdd(&C.nitems, ns);
      for (u32 x = 0; x < ns; ++x) A.items[at + x] = ((u64)v << 32) | x;
    }
  G.sync();
  // a split-off node takes over from the node it was split from (M6) and joins
  // K (M8); the last member of every node above
  for (u32 i = gt; i < A.n_new; i += gts) {
    const u32 x = A.new_base + i, o = A.origin[i];
    A.h_spre[x] = A.h_spre[o];
    A.h_scur[x] = A.h_scur[o];
    A.h_g[x] = A.h_g[o];
    A.kflag[x] = 1;
  }
  for (u32 v = gt; v < A.n; v += gts) atomicMax(&A.last[A.s_cur[v]], v + 1);
  G.sync();
  // ---- f of the level above, from the last member (M5) ----
  for (u32 x = gt; x < A.hn; x += gts) {
    const u32 l = A.last[x];
    if (!l) continue;
    const u32 nf = A.f[l - 1];
    if (A.h_f[x] != nf) {
      A.h_f[x] = nf;
      A.kflag[x] = 1;
    }
  }
  if (!A.aggregate) {
    if (gt == 0) {
      A.out->status = 0;
      A.out->count = 0;
      A.out->records = 0;
    }
    return;
  }
  u32 R = A.dk;
  const u32 nitems = C.nitems;
  // Everything is counted before anything is sorted: the sort's ranks cost
  // nitems^2 / 1024 searches (a split star of 1M leaves: 27 ms), and the total
  // of up to AGG_MAX_REC slices fits 32 bits.
  bool fits = nitems <= AGG_MAX_REC;
  if (fits && nitems) {
    unsigned long long mine = 0;
    for (u32 i = G.warp(); i < nitems; i += G.warps()) {
      const u32 c = gg_slice<false>(A, A.items[i], 0);
      if (lane == 0) A.ipos[i] = c;
      mine += c;
    }
    if (lane == 0 && mine) atomicAdd(&C.total, mine);
    G.sync();
    fits = C.total + A.dk <= AGG_MAX_REC;
  }
  if (!fits) {
    if (gt == 0) {
      A.out->status = 1;
      A.out->count = 0;
      A.out->records = 0;
    }
    return;
  }
  if (nitems) {
    // ---- records of every changed row, in vertex and CSR order ----
    gang_sort(
        G, S, nitems, [&](u32 i) { return A.items[i]; }, [](u32 i) { return i; }, A.itmp, A.itv,
        [&](u32 r, u64 key, u32 i) {
          A.items2[r] = key;
          A.icnt[r] = A.ipos[i];
        });
    R += gang_scan(
        G, S, nitems, [&](u32 i) { return A.icnt[i]; }, [&](u32 i, u32 ex) { A.ipos[i] = ex; },
        A.part);
    G.sync();
    for (u32 i = G.warp(); i < nitems; i += G.warps())
      gg_slice<true>(A, A.items2[i], A.dk + A.ipos[i]);
  }
  for (u32 i = gt; i < A.dk; i += gts) {
    A.keys[i] = gg_pair(A.s_pre[A.du[i]], A.s_pre[A.dv[i]]);
    A.vals[i] = A.dw ? A.dw[i] : 1.0;
  }
  G.sync();
  // ---- the level's s_pre catches up (no later step reads it) ----
  for (u32 v = gt; v < A.n; v += gts)
    if (A.refined[v]) A.s_pre[v] = A.s_cur[v];
  u32 count = 0;
  if (R) {
    // ---- records by key, their weights in that order ----
    gang_sort(
        G, S, R, [&](u32 i) { return A.keys[i]; }, [](u32 i) { return i; }, A.ktmp, A.ktv,
        [&](u32 r, u64 key, u32 i) {
          A.keys2[r] = key;
          A.sw[r] = A.vals[i];
        });
    // ---- every key's sum in push order; xs is 0 where nothing is kept ----
    for (u32 t = gt; t < R; t += gts) {
      const u64 key = A.keys2[t];
      double x = 0.0;
      if (t == 0 || A.keys2[t - 1] != key) {
        x = A.sw[t];
        u32 j = t + 1;
        if (j < R && A.keys2[j] == key) {
          x = __dadd_rn(0.0, x);
          for (; j < R && j < t + AGG_LANE && A.keys2[j] == key; ++j) x = __dadd_rn(x, A.sw[j]);
          if (j < R && A.keys2[j] == key) {
            A.longs[atomicAdd(&C.nlong, 1u)] = t;
            x = 0.0;
          }
        }
      }
      A.xs[t] = fabs(x) > 1e-9 ? x : 0.0;
    }
    G.sync();
    const u32 nlong = C.nlong;
    if (nlong) {
      for (u32 i = G.warp(); i < nlong; i += G.warps()) {
        const u32 t = A.longs[i];
        const u32 b = warp_bound_u64<true>(A.keys2, t, R, A.keys2[t]);
        const double x = warp_long_sum(t, b, 0.0, A.sw, chain[threadIdx.x >> 5]);
        if (lane == 0) A.xs[t] = fabs(x) > 1e-9 ? x : 0.0;
      }
      G.sync();
    }
    // ---- the kept ones, in ascending key order ----
    count = gang_scan(
        G, S, R, [&](u32 i) { return A.xs[i] != 0.0 ? 1u : 0u; },
        [&](u32 i, u32 ex) {
          const double x = A.xs[i];
          if (x == 0.0) return;
          const u64 key = A.keys2[i];
          A.ou[ex] = (u32)(key >> 32);
          A.ov[ex] = (u32)key;
          A.ow[ex] = x;
        },
        A.part);
  }
  if (gt == 0) {
    A.out->status = 0;
    A.out->count = count;
    A.out->records = R;
  }
}

bool gang_aggregate_fits(Engine& E, const Level& L, const DevEdges& delta) {
  return !E.lean && L.g.n > 0 && delta.k <= AGG_MAX_REC;
}

// Grows level H to `hn` nodes, projects the communities of L onto it and, with
// `aggregate`, compresses ΔH into (ou, ov, ow).  Returns false when the records
// did not fit: the caller then runs inc_aggregation.
bool gang_aggregate(Engine& E, Level& L, Level& H, const DevEdges& delta, bool aggregate,
                    DBuf<u32>& ou, DBuf<u32>& ov, DBuf<double>& ow, u64* count) {
  Scratch& S = E.sc;
  const u32 n = L.g.n, h_old = H.g.n;
  const u32 hn = std::max(h_old, E.new_base + E.n_new);
  const GangShape shape = gang_shape(E, 2ull * n + L.g.nnz / 8 + 32ull * delta.k);
  if (hn > h_old) {
    H.g.off.ensure(E.mem, (size_t)hn + 1, true);
    H.f.ensure(E.mem, hn, true);
    H.gm.ensure(E.mem, hn, true);
    H.s_pre.ensure(E.mem, hn, true);
    H.s_cur.ensure(E.mem, hn, true);
    H.k.ensure(E.mem, hn, true);
  }
  S.kflag.ensure(E.mem, hn ? hn : 1);
  S.minmem.ensure(E.mem, (size_t)hn + 1);
  S.gang_part.ensure(E.mem, GANG_MAX_BLOCKS);
  GangAggArgs A{};
  if (aggregate) {
    const u64 nit = (u64)n + L.g.nnz / AGG_SLICE + 1;
    // records: ΔG, and two per entry of the changed rows
    const u64 rec = std::min<u64>(AGG_MAX_REC, delta.k + 2 * L.g.nnz + 2ull * n) + 1;
    S.gr_items.ensure(E.mem, 3 * nit);
    S.order.ensure(E.mem, nit);
    S.order2.ensure(E.mem, nit);
    S.used.ensure(E.mem, nit);
    S.keys.ensure(E.mem, rec);
    S.keys2.ensure(E.mem, rec);
    S.rkeys.ensure(E.mem, rec);
    S.idx.ensure(E.mem, rec);
    S.neww.ensure(E.mem, rec);
    S.fvals.ensure(E.mem, rec);
    S.ew.ensure(E.mem, rec);
    S.idx2.ensure(E.mem, rec);
    ou.ensure(E.mem, rec);
    ov.ensure(E.mem, rec);
    ow.ensure(E.mem, rec);
    A.items = S.gr_items.p;
    A.items2 = A.items + nit;
    A.itmp = A.items2 + nit;
    A.itv = S.order.p;
    A.icnt = S.order2.p;
    A.ipos = S.used.p;
    A.keys = S.keys.p;
    A.keys2 = S.keys2.p;
    A.ktmp = S.rkeys.p;
    A.ktv = S.idx.p;
    A.vals = S.neww.p;
    A.sw = S.fvals.p;
    A.xs = S.ew.p;
    A.longs = S.idx2.p;
    A.ou = ou.p;
    A.ov = ov.p;
    A.ow = ow.p;
  }
  A.n = n;
  A.off = L.g.off.p;
  A.col = L.g.col.p;
  A.w = L.g.w.p;
  A.f = L.f.p;
  A.s_cur = L.s_cur.p;
  A.s_pre = L.s_pre.p;
  A.refined = S.refined.p;
  A.hn_old = h_old;
  A.hn = hn;
  A.new_base = E.new_base;
  A.n_new = E.n_new;
  A.h_nnz = H.g.nnz;
  A.h_off = H.g.off.p;
  A.h_f = H.f.p;
  A.h_g = H.gm.p;
  A.h_spre = H.s_pre.p;
  A.h_scur = H.s_cur.p;
  A.h_k = H.k.p;
  A.origin = S.origin.p;
  A.kflag = S.kflag.p;
  A.last = S.minmem.p;
  A.du = delta.u;
  A.dv = delta.v;
  A.dw = delta.w;
  A.dk = (u32)delta.k;
  A.aggregate = aggregate;
  A.grid = shape.grid;
  A.part = S.gang_part.p;
  A.cnt = reinterpret_cast<AggCnt*>(gang_counters(E, &A.cnt_next));
  A.out = reinterpret_cast<AggOut*>(E.hs.p);
  cudaEvent_t ev = E.kt_begin();
  gang_launch(E, reinterpret_cast<const void*>(&k_gang_aggregate), shape, 0, &A);
  gang_turn(E);
  E.kt_end(KT_GANG_AGG, ev);
  H.g.n = hn;
  if (H.s_bound && H.s_bound < hn) H.s_bound = hn;
  if (!aggregate) {
    *count = 0;
    return true;
  }
  AggOut o;
  E.sync();
  std::memcpy(&o, E.hs.p, sizeof(o));
  *count = o.count;
  // lifted ΔG, the maps, the records written and read once, the output
  E.kagg[KT_GANG_AGG].bytes += 32ull * delta.k + 13ull * n + 42ull * o.records + 16ull * o.count;
  return o.status == 0;
}

}  // namespace hl
