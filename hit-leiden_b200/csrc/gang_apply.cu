// gang_apply.cu — G ← G ⊕ ΔG in one launch (in_memory.rs:103-137).
//
// The same steps and results as apply_delta in graph.cu, for batches of up to
// GANG_BATCH_MAX edges: batch keys sorted, every key resolved against the CSR
// (existing weight, then the batch's weights in batch order), weight changes
// written in place, inserts and deletes sorted as row-operations and merged
// into the level's second CSR buffer, the degrees of the changed rows, 2m.
#include "csr_rebuild.cuh"
#include "gang.cuh"

namespace hl {

struct ApplyCnt {  // zeroed by the host
  u32 ins_loops, del_loops, nops, nrows, nlong, work, err, pad_;
};

struct ApplyOut {
  u64 nnz_new;
  double tw;
  u32 nops, ins_loops, del_loops, err;
};

struct GangApplyArgs {
  u32 n;
  u64 nnz;
  const u64* off;
  const u32* col;
  double* w;
  u64* noff;
  u32* ncol;
  double* nw;
  double* k;
  const u32* bu;
  const u32* bv;
  const double* bw;
  u32 kb;
  bool integral, grid, structure_only, finish_only;
  u64 *keys, *keys2;   // batch keys, sorted chunks / sorted keys
  u32 *idx, *idx2;
  double* neww;        // per position of the sorted batch (heads only)
  u64 *rkeys, *rkeys2; // row-operations (row << 32 | neighbour)
  u32 *rvals, *rvals2;
  u32* dpre;           // deletes before each sorted row-operation
  u64* opos;           // position of each sorted row-operation in the old entries (= rkeys)
  u32* touched;        // bit per row: its weights changed
  u32* rows;           // those rows, listed
  u32* longrows;       // ... and those of LONG_SUM entries or more
  double *red, *red2;
  u32* part;
  ApplyCnt* cnt;
  u32* cnt_next;
  ApplyOut* out;
};

// Rows of this many entries are summed first: with integral weights by a whole
// block each, otherwise one ordered chain (about 10 cycles an entry) must not
// start behind shorter ones.
constexpr u64 LONG_SUM = 2048;

__device__ __forceinline__ void ga_touch(const GangApplyArgs& A, u32 v, u64 deg) {
  const u32 bit = 1u << (v & 31);
  if (atomicOr(&A.touched[v >> 5], bit) & bit) return;
  if (deg >= LONG_SUM) A.longrows[atomicAdd(&A.cnt->nlong, 1u)] = v;
  else A.rows[atomicAdd(&A.cnt->nrows, 1u)] = v;
}

// Tile sums of the fixed-shape pairwise sum (tiles of 1024, +0.0 padded,
// folded by stride halving).
__device__ __forceinline__ void ga_tree_tiles(const Gang& G, GangSmem& S, const double* x, u64 n,
                                              double* out) {
  double* s = reinterpret_cast<double*>(S.key);
  const u32 tid = threadIdx.x;
  const u64 tiles = (n + 1023) / 1024;
  for (u64 t = G.rank; t < tiles; t += G.nct) {
    const u64 a = t * 1024 + tid;
    const double x0 = a < n ? x[a] : 0.0;
    const double x1 = a + 512 < n ? x[a + 512] : 0.0;
    s[tid] = __dadd_rn(x0, x1);
    __syncthreads();
    for (u32 st = 256; st >= 32; st >>= 1) {
      if (tid < st) s[tid] = __dadd_rn(s[tid], s[tid + st]);
      __syncthreads();
    }
    if (tid < 32) {
      double y = s[tid];
#pragma unroll
      for (u32 st = 16; st >= 1; st >>= 1) y = __dadd_rn(y, __shfl_down_sync(0xffffffffu, y, st));
      if (tid == 0) out[t] = y;
    }
    __syncthreads();
  }
}

// What bounds it: on large levels the rewrite of the CSR (24 bytes an entry:
// 29.0M entries in 173 us, 4.0 TB/s), on small ones the chain of sorts,
// searches and barriers.  Against the multi-kernel form it replaces (some
// forty launches and five host reads a level), the whole stage of one level:
// 5 levels of 250-400 nodes 240 -> 36 us, 10 levels of 10-50k nodes 460 -> 113
// us, 10 levels of 0.13-1M nodes with f64 weights 830 -> 350 us (of which the
// rewrite 90-220, the chains of hub rows 40-110, two sorts 65; events around
// the launch).
__global__ void __launch_bounds__(GANG_THREADS, 1) k_gang_apply(GangApplyArgs A) {
  __shared__ GangSmem S;
  __shared__ __align__(16) double chain[GANG_WARPS][CHAIN_TILE];
  const Gang G = gang_make(A.grid);
  const u32 tid = threadIdx.x, lane = tid & 31;
  ApplyCnt& C = *A.cnt;
  gang_clear_next(G, A.cnt_next);
  if (!A.finish_only) {
    // ---- the batch by key, stable (batch order within a key) ----
    for (u32 i = G.thread(); i < (A.n + 31) / 32; i += G.threads()) A.touched[i] = 0;
    gang_sort(
        G, S, A.kb,
        [&](u32 i) {
          const u32 a = A.bu[i], b = A.bv[i];
          return a < b ? ((u64)a << 32) | b : ((u64)b << 32) | a;
        },
        [](u32 i) { return i; }, A.keys, A.idx,
        [&](u32 r, u64 key, u32 i) {
          A.keys2[r] = key;
          A.idx2[r] = i;
        });
    // ---- every distinct key: existing weight, then the batch's in order ----
    for (u32 t = G.thread(); t < A.kb; t += G.threads()) {
      const u64 key = A.keys2[t];
      if (t && A.keys2[t - 1] == key) continue;
      const u32 a = (u32)(key >> 32), b = (u32)key;
      const u64 o0 = A.off[a], o1 = A.off[a + 1];
      const u64 p = lower_bound_u32(A.col, o0, o1, b);
      const bool present = p < o1 && A.col[p] == b;
      double x = present ? A.w[p] : 0.0;
      for (u32 j = t; j < A.kb && A.keys2[j] == key; ++j)
        x = __dadd_rn(x, A.bw ? A.bw[A.idx2[j]] : 1.0);
      const bool live = x > 1e-12;
      if (!present && !live) continue;
      A.neww[t] = x;
      const u64 q0 = A.off[b], q1 = A.off[b + 1];
      ga_touch(A, a, o1 - o0);
      if (a != b) ga_touch(A, b, q1 - q0);
      if (present && live) {
        A.w[p] = x;
        if (a == b) A.w[p + 1] = x;
        else A.w[lower_bound_u32(A.col, q0, q1, a)] = x;
        continue;
      }
      if (a == b) atomicAdd(present ? &C.del_loops : &C.ins_loops, 1u);
      const u32 at = atomicAdd(&C.nops, 2u);
      const u32 val = present ? DEL_MARK : t;
      A.rkeys[at] = ((u64)a << 32) | b;
      A.rvals[at] = val;
      A.rkeys[at + 1] = ((u64)b << 32) | a;
      A.rvals[at + 1] = val;
    }
    G.sync();
  }
  const u32 R = C.nops;
  u64 nnz_new = A.nnz;
  if (R && !A.finish_only) {
    // ---- row-operations by (row, neighbour); equal ones are a loop's pair ----
    gang_sort(
        G, S, R, [&](u32 i) { return A.rkeys[i]; }, [&](u32 i) { return A.rvals[i]; }, A.keys,
        A.idx,
        [&](u32 r, u64 key, u32 v) {
          A.rkeys2[r] = key;
          A.rvals2[r] = v;
        });
    for (u32 t = G.thread(); t < R; t += G.threads())
      A.opos[t] = rowop_position(t, A.rkeys2, A.rvals2, A.off, A.col);
    const u32 ndel = gang_scan(
        G, S, R, [&](u32 i) { return A.rvals2[i] == DEL_MARK ? 1u : 0u; },
        [&](u32 i, u32 ex) { A.dpre[i] = ex; }, A.part);
    if (G.thread() == 0) A.dpre[R] = ndel;
    G.sync();
  }
  if (R) nnz_new = A.nnz + R - 2ull * A.dpre[R];
  if (A.structure_only) {
    if (G.thread() == 0) {
      A.out->nnz_new = nnz_new;
      A.out->nops = R;
    }
    return;
  }
  if (R) {
    // ---- the new CSR ----
    const RowOps O{R, A.rkeys2, A.rvals2, A.dpre, A.opos};
    rebuild_inserts(O, A.neww, A.ncol, A.nw, nnz_new, &C.err, G.thread(), G.threads());
    rebuild_offsets(O, A.n, A.off, A.noff, G.warp(), G.warps());
    rebuild_entries(O, A.nnz, A.col, A.w, A.ncol, A.nw, nnz_new, &C.err, G.warp(), G.warps());
    G.sync();
  }
  // ---- degrees of the changed rows, in CSR order; the long ones first ----
  const u64* off = R ? A.noff : A.off;
  const double* w = R ? A.nw : A.w;
  const u32 nlong = C.nlong, nrows = C.nrows;
  if (A.integral) {  // exact in any order: a block per long row, then a warp per row
    double* sred = reinterpret_cast<double*>(S.key);
    for (u32 i = G.rank; i < nlong; i += G.nct) {
      const u32 v = A.longrows[i];
      double s = 0.0;
      for (u64 p = off[v] + tid; p < off[v + 1]; p += GANG_THREADS) s += w[p];
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) sred[tid >> 5] = s;
      __syncthreads();
      if (tid == 0) {
        double t = 0.0;
        for (u32 x = 0; x < GANG_WARPS; ++x) t += sred[x];
        A.k[v] = t;
      }
      __syncthreads();
    }
    for (u32 i = G.warp(); i < nrows; i += G.warps()) {
      const u32 v = A.rows[i];
      double s = 0.0;
      for (u64 p = off[v] + lane; p < off[v + 1]; p += 32) s += w[p];
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) A.k[v] = s;
    }
  } else {
    double* buf = chain[tid >> 5];
    for (u32 i = G.warp(); i < nlong + nrows;) {
      const u32 v = i < nlong ? A.longrows[i] : A.rows[i - nlong];
      const double s = warp_long_sum(off[v], off[v + 1], 0.0, w, buf);
      if (lane == 0) {
        A.k[v] = s;
        i = G.warps() + atomicAdd(&C.work, 1u);  // the next row not yet taken
      }
      i = __shfl_sync(0xffffffffu, i, 0);
    }
  }
  G.sync();
  // ---- 2m ----
  const double* src = A.k;
  double* dst = A.red;
  double* other = A.red2;
  u64 cur = A.n;
  while (true) {
    const u64 tiles = (cur + 1023) / 1024;
    ga_tree_tiles(G, S, src, cur, dst);
    if (tiles == 1) break;
    G.sync();
    src = dst;
    cur = tiles;
    double* t = dst;
    dst = other;
    other = t;
  }
  // ---- the result; block 0 took the last tile ----
  if (G.thread() == 0) {
    A.out->tw = dst[0];
    A.out->nnz_new = nnz_new;
    A.out->nops = R;
    A.out->ins_loops = C.ins_loops;
    A.out->del_loops = C.del_loops;
    A.out->err = C.err;
  }
}

constexpr u64 GANG_ROOM_MAX = 1ull << 22;  // entries

bool gang_apply_fits(Engine& E, const Level& L, const DevEdges& b, bool drop_loops) {
  return !E.lean && b.k > 0 && b.k <= GANG_BATCH_MAX && !drop_loops && L.g.n > 0;
}

void gang_apply(Engine& E, Level& L, const DevEdges& b) {
  Scratch& S = E.sc;
  DevGraph& Gr = L.g;
  const u32 n = Gr.n;
  const u32 k = (u32)b.k;
  const u32 rmax = 2 * k;
  // A sorted record costs about 64 streamed entries (17.5k updates: two sorts
  // 310 us on 8 blocks, 140 us on 148), and less while a single block sorts all
  // of them in one go (70 updates of 1.3k entries: 25 us on one block, 40 on 8).
  const GangShape shape = gang_shape(E, Gr.nnz + n + (k <= 128 ? 16ull : 64ull) * k);
  S.keys.ensure(E.mem, rmax);
  S.idx.ensure(E.mem, rmax);
  S.keys2.ensure(E.mem, k);
  S.idx2.ensure(E.mem, k);
  S.neww.ensure(E.mem, k);
  S.rkeys.ensure(E.mem, rmax);
  S.rkeys2.ensure(E.mem, rmax);
  S.rvals.ensure(E.mem, rmax);
  S.rvals2.ensure(E.mem, rmax);
  S.opdelpre.ensure(E.mem, rmax + 1);
  S.ga_touched.ensure(E.mem, (n + 31) / 32);
  S.rowlist.ensure(E.mem, rmax);
  S.longrows.ensure(E.mem, std::min<u64>(rmax, Gr.nnz / LONG_SUM + 1));
  S.newoff.ensure(E.mem, (size_t)n + 1);
  const u64 tiles = ((u64)n + 1023) / 1024;
  S.red.ensure(E.mem, tiles + 1);
  S.red2.ensure(E.mem, (tiles + 1023) / 1024 + 1);
  S.gang_part.ensure(E.mem, GANG_MAX_BLOCKS);
  GangApplyArgs A{};
  A.n = n;
  A.nnz = Gr.nnz;
  A.off = Gr.off.p;
  A.col = Gr.col.p;
  A.w = Gr.w.p;
  A.noff = S.newoff.p;
  A.k = L.k.p;
  A.bu = b.u;
  A.bv = b.v;
  A.bw = b.w;
  A.kb = k;
  A.integral = E.integral;
  A.grid = shape.grid;
  A.keys = S.keys.p;
  A.keys2 = S.keys2.p;
  A.idx = S.idx.p;
  A.idx2 = S.idx2.p;
  A.neww = S.neww.p;
  A.rkeys = S.rkeys.p;
  A.rkeys2 = S.rkeys2.p;
  A.rvals = S.rvals.p;
  A.rvals2 = S.rvals2.p;
  A.dpre = S.opdelpre.p;
  A.opos = S.rkeys.p;  // the unsorted keys are done with
  A.touched = S.ga_touched.p;
  A.rows = S.rowlist.p;
  A.longrows = S.longrows.p;
  A.red = S.red.p;
  A.red2 = S.red2.p;
  A.part = S.gang_part.p;
  A.cnt = reinterpret_cast<ApplyCnt*>(gang_counters(E, &A.cnt_next));
  A.out = reinterpret_cast<ApplyOut*>(E.hs.p);
  const u64 bound = Gr.nnz + rmax;
  cudaEvent_t ev = E.kt_begin();
  ApplyOut o;
  const void* fn = reinterpret_cast<const void*>(&k_gang_apply);
  auto result = [&]() {
    E.sync();
    std::memcpy(&o, E.hs.p, sizeof(o));
  };
  // Room for every update to insert, where that is small (a handle with a
  // budget does not): the launch that finds the exact size first costs
  // 17 us on a level of 40k entries.
  if ((Gr.col2.cap < bound || Gr.w2.cap < bound) && bound <= GANG_ROOM_MAX && !E.mem.budget) {
    Gr.col2.ensure_slack(E.mem, bound);
    Gr.w2.ensure_slack(E.mem, bound);
  }
  if (Gr.col2.cap < bound || Gr.w2.cap < bound) {
    // the second buffer may have to grow: only by what the batch needs
    A.structure_only = true;
    gang_launch(E, fn, shape, 0, &A);
    gang_turn(E);  // the second launch goes on with these counters
    result();
    if (o.nops) {
      Gr.col2.ensure_slack(E.mem, o.nnz_new ? o.nnz_new : 1);
      Gr.w2.ensure_slack(E.mem, o.nnz_new ? o.nnz_new : 1);
    }
    A.structure_only = false;
    A.finish_only = true;
  }
  A.ncol = Gr.col2.p;
  A.nw = Gr.w2.p;
  gang_launch(E, fn, shape, 0, &A);
  if (!A.finish_only) gang_turn(E);
  result();
  E.kt_end(KT_GANG_APPLY, ev);
  if (o.err)
    throw Error(HL_ERR_CUDA, "internal error: CSR merge produced an out-of-range position");
  if (o.nops) {
    E.kagg[KT_GANG_APPLY].bytes += 16ull * ((u64)n + 1) + 12ull * (Gr.nnz + o.nnz_new);
    Gr.col.swap(Gr.col2);
    Gr.w.swap(Gr.w2);
    Gr.off.swap(S.newoff);
    Gr.nnz = o.nnz_new;
    Gr.self_loop_entries = Gr.self_loop_entries + 2ull * o.ins_loops - 2ull * o.del_loops;
  }
  L.tw = o.tw;
}

}  // namespace hl
