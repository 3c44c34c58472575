// graph.cu — device CSR maintenance: G ← G ⊕ ΔG (K1), degrees, 2m.
//
// apply_delta restates in_memory.rs:103-137: every ΔG edge is keyed by
// (min, max); a key's new weight is its existing weight followed by the
// batch's deltas in batch order (a stable sort keeps that order); keys whose
// weight ends at <= 1e-12 disappear.  Instead of rebuilding a hash map of all
// m edges, only the changed keys are resolved: weight updates are written in
// place, and inserts/deletes become sorted row-operations by which every
// surviving entry moves into a fresh CSR (csr_rebuild.cuh).
#include "csr_rebuild.cuh"
#include "hl_engine.cuh"

namespace hl {

__global__ void k_fill_u8(u8* p, u8 v, u64 n) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void k_iota(u32* p, u32 n) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    p[i] = (u32)i;
}

__global__ void k_fill_u64_range(u64* p, u64 v, u64 lo, u64 hi) {
  for (u64 i = lo + blockIdx.x * (u64)blockDim.x + threadIdx.x; i < hi;
       i += (u64)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void k_fill_f64_range(double* p, double v, u64 lo, u64 hi) {
  for (u64 i = lo + blockIdx.x * (u64)blockDim.x + threadIdx.x; i < hi;
       i += (u64)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void k_iota_range(u32* p, u64 lo, u64 hi) {
  for (u64 i = lo + blockIdx.x * (u64)blockDim.x + threadIdx.x; i < hi;
       i += (u64)gridDim.x * blockDim.x)
    p[i] = (u32)i;
}

static inline u32 grid_for(u64 n, u32 block = 256) {
  u64 g = (n + block - 1) / block;
  if (g > 148u * 64u) g = 148u * 64u;
  return g ? (u32)g : 1u;
}

void graph_init_empty(Engine& E, Level& L, u32 n) {
  L.g.n = n;
  L.g.nnz = 0;
  L.g.self_loop_entries = 0;
  L.g.off.ensure(E.mem, (size_t)n + 1);
  HL_CUDA(cudaMemsetAsync(L.g.off.p, 0, sizeof(u64) * ((size_t)n + 1), E.stream));
  L.g.col.ensure(E.mem, 1);
  L.g.w.ensure(E.mem, 1);
  L.f.ensure(E.mem, n ? n : 1);
  L.gm.ensure(E.mem, n ? n : 1);
  L.s_pre.ensure(E.mem, n ? n : 1);
  L.s_cur.ensure(E.mem, n ? n : 1);
  L.k.ensure(E.mem, n ? n : 1);
  if (n) {
    ++E.nlaunch, k_iota<<<grid_for(n), 256, 0, E.stream>>>(L.f.p, n);
    ++E.nlaunch, k_iota<<<grid_for(n), 256, 0, E.stream>>>(L.gm.p, n);
    ++E.nlaunch, k_iota<<<grid_for(n), 256, 0, E.stream>>>(L.s_pre.p, n);
    ++E.nlaunch, k_iota<<<grid_for(n), 256, 0, E.stream>>>(L.s_cur.p, n);
    HL_CUDA(cudaMemsetAsync(L.k.p, 0, sizeof(double) * n, E.stream));
  }
  L.tw = 0.0;
  L.s_bound = n;
  HL_LAUNCH_CHECK();
}

// New nodes start isolated with identity maps (PartitionState::identity).
void graph_grow_nodes(Engine& E, Level& L, u32 n) {
  u32 old = L.g.n;
  if (n <= old) return;
  L.g.off.ensure(E.mem, (size_t)n + 1, true);
  ++E.nlaunch, k_fill_u64_range<<<grid_for(n - old), 256, 0, E.stream>>>(L.g.off.p, L.g.nnz, (u64)old + 1,
                                                             (u64)n + 1);
  L.f.ensure(E.mem, n, true);
  L.gm.ensure(E.mem, n, true);
  L.s_pre.ensure(E.mem, n, true);
  L.s_cur.ensure(E.mem, n, true);
  L.k.ensure(E.mem, n, true);
  ++E.nlaunch, k_iota_range<<<grid_for(n - old), 256, 0, E.stream>>>(L.f.p, old, n);
  ++E.nlaunch, k_iota_range<<<grid_for(n - old), 256, 0, E.stream>>>(L.gm.p, old, n);
  ++E.nlaunch, k_iota_range<<<grid_for(n - old), 256, 0, E.stream>>>(L.s_pre.p, old, n);
  ++E.nlaunch, k_iota_range<<<grid_for(n - old), 256, 0, E.stream>>>(L.s_cur.p, old, n);
  ++E.nlaunch, k_fill_f64_range<<<grid_for(n - old), 256, 0, E.stream>>>(L.k.p, 0.0, old, n);
  L.g.n = n;
  if (L.s_bound && L.s_bound < n) L.s_bound = n;
  HL_LAUNCH_CHECK();
}

__global__ void k_check_endpoints(const u32* u, const u32* v, u64 k, u32 n, u32* bad) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < k; i += (u64)gridDim.x * blockDim.x)
    if (u[i] >= n || v[i] >= n) atomicAdd(bad, 1u);
}

void check_endpoints(Engine& E, const DevEdges& b, u32 n) {
  if (!b.k) return;
  E.sc.cnt.ensure(E.mem, 16);
  HL_CUDA(cudaMemsetAsync(E.sc.cnt.p, 0, sizeof(u32), E.stream));
  ++E.nlaunch, k_check_endpoints<<<grid_for(b.k), 256, 0, E.stream>>>(b.u, b.v, b.k, n, E.sc.cnt.p);
  HL_LAUNCH_CHECK();
  u32 bad = E.read_u32(E.sc.cnt.p);
  require(bad == 0, "edge endpoint exceeds node_count (" + std::to_string(bad) + " edges)");
}

__global__ void k_integral(const double* w, u64 k, u32* bad) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < k; i += (u64)gridDim.x * blockDim.x) {
    double x = w[i];
    if (!(x == floor(x)) || fabs(x) > 4294967296.0) atomicAdd(bad, 1u);
  }
}

bool edges_integral(Engine& E, const DevEdges& b) {
  if (!b.k || !b.w) return true;
  E.sc.cnt.ensure(E.mem, 16);
  HL_CUDA(cudaMemsetAsync(E.sc.cnt.p + 1, 0, sizeof(u32), E.stream));
  ++E.nlaunch, k_integral<<<grid_for(b.k), 256, 0, E.stream>>>(b.w, b.k, E.sc.cnt.p + 1);
  HL_LAUNCH_CHECK();
  return E.read_u32(E.sc.cnt.p + 1) == 0;
}

__global__ void k_delta_keys(const u32* u, const u32* v, u64 k, u64* keys, u32* idx) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < k; i += (u64)gridDim.x * blockDim.x) {
    u32 a = u[i], b = v[i];
    u32 lo = a < b ? a : b, hi = a < b ? b : a;
    keys[i] = ((u64)lo << 32) | hi;
    idx[i] = (u32)i;
  }
}

__global__ void k_heads(const u64* sk, u64 k, u32* head) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < k; i += (u64)gridDim.x * blockDim.x)
    head[i] = (i == 0 || sk[i] != sk[i - 1]) ? 1u : 0u;
}

__global__ void k_seg_start(const u32* head, const u32* segid, u64 k, u32* seg_start) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < k; i += (u64)gridDim.x * blockDim.x)
    if (head[i]) seg_start[segid[i]] = (u32)i;
}

enum : u8 { OP_NONE = 0, OP_UPD = 1, OP_INS = 2, OP_DEL = 3 };

// One thread per distinct key: existing weight, then the batch's deltas in
// batch order (in_memory.rs:133-137), then the > 1e-12 filter (:110).
__global__ void k_resolve(u32 U, const u32* seg_start, u64 k, const u64* sk, const u32* sidx,
                          const double* bw, const u64* off, const u32* col, double* w,
                          bool keep_loops, u8* op, double* neww, u8* ktouched, u32* nops_del,
                          u32* nops_ins, u32* loop_counts) {
  for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < U; j += (u64)gridDim.x * blockDim.x) {
    u64 t0 = seg_start[j];
    u64 t1 = (j + 1 < U) ? seg_start[j + 1] : k;
    u64 key = sk[t0];
    u32 a = (u32)(key >> 32), b = (u32)key;
    u64 o0 = off[a], o1 = off[a + 1];
    u64 p = lower_bound_u32(col, o0, o1, b);
    bool present = p < o1 && col[p] == b;
    if (a == b && !keep_loops) present = false;
    double x = present ? w[p] : 0.0;
    for (u64 t = t0; t < t1; ++t) x = __dadd_rn(x, bw ? bw[sidx[t]] : 1.0);
    u8 o = OP_NONE;
    u32 nd = 0, ni = 0;
    if (present) {
      if (x > 1e-12) {
        o = OP_UPD;
        w[p] = x;
        if (a == b) {
          w[p + 1] = x;
        } else {
          u64 q = lower_bound_u32(col, off[b], off[b + 1], a);
          w[q] = x;
        }
      } else {
        o = OP_DEL;
        nd = 2;
        if (a == b) atomicAdd(&loop_counts[1], 1u);
      }
    } else if (x > 1e-12) {
      o = OP_INS;
      ni = 2;
      if (a == b) atomicAdd(&loop_counts[0], 1u);
    }
    op[j] = o;
    neww[j] = x;
    nops_del[j] = nd;
    nops_ins[j] = ni;
    if (o != OP_NONE) {
      ktouched[a] = 1;
      ktouched[b] = 1;
    }
  }
}

__global__ void k_emit_rowops(u32 U, const u32* seg_start, const u64* sk, const u8* op,
                              const u32* pos_del, const u32* pos_ins, u64 ins_base, u64* rkeys,
                              u32* rvals) {
  for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < U; j += (u64)gridDim.x * blockDim.x) {
    u8 o = op[j];
    if (o != OP_DEL && o != OP_INS) continue;
    u64 key = sk[seg_start[j]];
    u32 a = (u32)(key >> 32), b = (u32)key;
    u64 p = (o == OP_DEL) ? pos_del[j] : ins_base + pos_ins[j];
    u32 val = (o == OP_DEL) ? DEL_MARK : (u32)j;
    rkeys[p] = ((u64)a << 32) | b;
    rvals[p] = val;
    rkeys[p + 1] = ((u64)b << 32) | a;
    rvals[p + 1] = val;
  }
}

__global__ void k_count_loops(u32 n, const u64* off, const u32* col, u32* total) {
  u32 local = 0;
  for (u64 v = blockIdx.x * (u64)blockDim.x + threadIdx.x; v < n; v += (u64)gridDim.x * blockDim.x) {
    u64 o0 = off[v], o1 = off[v + 1];
    u64 p = lower_bound_u32(col, o0, o1, (u32)v);
    while (p < o1 && col[p] == (u32)v) {
      ++local;
      ++p;
    }
  }
  if (local) atomicAdd(total, local);
}

// Existing self-loops are dropped by the reference's apply_delta
// (collect_canonical_edges keeps node < neighbor only, in_memory.rs:125).
__global__ void k_emit_loop_drops(u32 n, const u64* off, const u32* col, u64* rkeys, u32* rvals,
                                  u64 base, u64 limit, u32* counter, u8* ktouched, u32* err) {
  for (u64 v = blockIdx.x * (u64)blockDim.x + threadIdx.x; v < n; v += (u64)gridDim.x * blockDim.x) {
    u64 o0 = off[v], o1 = off[v + 1];
    u64 p = lower_bound_u32(col, o0, o1, (u32)v);
    u32 c = 0;
    while (p + c < o1 && col[p + c] == (u32)v) ++c;
    if (c) {
      u32 at = atomicAdd(counter, c);
      for (u32 i = 0; i < c; ++i) {
        if (base + at + i >= limit) {
          atomicAdd(err, 1u);
          break;
        }
        rkeys[base + at + i] = ((u64)v << 32) | (u32)v;
        rvals[base + at + i] = DEL_MARK;
      }
      ktouched[v] = 1;
    }
  }
}

__global__ void k_del_flags(const u32* rvals, u64 R, u32* flag) {
  for (u64 t = blockIdx.x * (u64)blockDim.x + threadIdx.x; t <= R; t += (u64)gridDim.x * blockDim.x)
    flag[t] = (t < R && rvals[t] == DEL_MARK) ? 1u : 0u;
}

__global__ void k_rowop_positions(const u64* rkeys, const u32* rvals, u64 R, const u64* off,
                                  const u32* col, u64* opos) {
  for (u64 t = blockIdx.x * (u64)blockDim.x + threadIdx.x; t < R; t += (u64)gridDim.x * blockDim.x)
    opos[t] = rowop_position((u32)t, rkeys, rvals, off, col);
}

// The new CSR from the old one and its row-operations (csr_rebuild.cuh).
__global__ void __launch_bounds__(256) k_rebuild(RowOps O, u32 n, u64 nnz, const u64* off,
                                                 const u32* col, const double* w,
                                                 const double* neww, u64* noff, u32* ncol,
                                                 double* nw, u64 nnz_new, u32* err) {
  const u64 thread = blockIdx.x * (u64)blockDim.x + threadIdx.x;
  const u64 threads = (u64)gridDim.x * blockDim.x;
  rebuild_inserts(O, neww, ncol, nw, nnz_new, err, thread, threads);
  rebuild_offsets(O, n, off, noff, thread >> 5, threads >> 5);
  rebuild_entries(O, nnz, col, w, ncol, nw, nnz_new, err, thread >> 5, threads >> 5);
}

LongList long_list(Engine& E, u64 total, u32 nseg) {
  Scratch& S = E.sc;
  const u64 cap = std::min<u64>(total / LONG_SEG + 1, nseg ? nseg : 1);
  S.longseg.ensure(E.mem, cap);
  S.longcnt.ensure(E.mem, 1);
  HL_CUDA(cudaMemsetAsync(S.longcnt.p, 0, sizeof(u32), E.stream));
  return LongList{S.longseg.p, S.longcnt.p};
}

// Row sums in CSR order (hit_leiden.rs:1063), left to right: the exact
// rounding of the reference for any weights.  A warp takes 32 rows at a time
// and sums those whose flag is set (all without flags) one after another; the
// long ones are listed for k_row_sum_serial_long.
__global__ void __launch_bounds__(256) k_row_sum_serial(u32 n, const u64* off, const double* w,
                                                        double* k, const u8* flags, LongList ll) {
  __shared__ __align__(16) double chain[8][CHAIN_TILE];
  const u32 lane = threadIdx.x & 31;
  const u64 warp = (blockIdx.x * (u64)blockDim.x + threadIdx.x) >> 5;
  const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 v0 = warp * 32; v0 < n; v0 += nwarps * 32) {
    const u64 v = v0 + lane;
    bool on = v < n && (!flags || flags[v]);
    const u64 a = on ? off[v] : 0, b = on ? off[v + 1] : 0;
    if (b - a >= LONG_SEG) {
      ll.seg[atomicAdd(ll.cnt, 1u)] = (u32)v;
      on = false;
    }
    double mine = 0.0;
    for (u32 m = __ballot_sync(0xffffffffu, on); m; m &= m - 1) {
      const u32 j = __ffs(m) - 1;
      const double s = warp_long_sum(__shfl_sync(0xffffffffu, a, j),
                                      __shfl_sync(0xffffffffu, b, j), 0.0, w,
                                      chain[threadIdx.x >> 5]);
      if (lane == j) mine = s;
    }
    if (on) k[v] = mine;
  }
}

// The listed rows, a warp each.
__global__ void __launch_bounds__(256) k_row_sum_serial_long(LongList ll, const u64* off,
                                                             const double* w, double* k) {
  __shared__ __align__(16) double chain[8][CHAIN_TILE];
  const u32 cnt = *ll.cnt;
  for (u32 i = blockIdx.x * 8 + (threadIdx.x >> 5); i < cnt; i += gridDim.x * 8) {
    const u32 v = ll.seg[i];
    const double s = warp_long_sum(off[v], off[v + 1], 0.0, w, chain[threadIdx.x >> 5]);
    if ((threadIdx.x & 31) == 0) k[v] = s;
  }
}

// Left-to-right sums of the segments [off[i], off[i+1]) of x from `init`:
// the library's own choice (path 0), the run fold (1) or the shuffled fold (2).
template <int PATH>
__global__ void __launch_bounds__(256) k_seq_sums(u32 nseg, const u64* off, const double* x,
                                                  double init, double* out) {
  __shared__ __align__(16) double chain[8][CHAIN_TILE];
  const u32 lane = threadIdx.x & 31;
  const u64 warp = (blockIdx.x * (u64)blockDim.x + threadIdx.x) >> 5;
  const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 i = warp; i < nseg; i += nwarps) {
    const u64 a = off[i], b = off[i + 1];
    const double s = PATH == 0   ? warp_long_sum(a, b, init, x, chain[threadIdx.x >> 5])
                     : PATH == 1 ? warp_fold_runs(a, b, init, x)
                                 : warp_ordered_sum(a, b, init, [&](u64 p) { return x[p]; },
                                                    [](u64) { return true; });
    if (lane == 0) out[i] = s;
  }
}

void seq_sums(Engine& E, u32 nseg, const u64* off, const double* x, double init, int path,
              double* out) {
  if (!nseg) return;
  const u32 grid = grid_for((u64)nseg * 32);
  if (path == 2)
    ++E.nlaunch, k_seq_sums<2><<<grid, 256, 0, E.stream>>>(nseg, off, x, init, out);
  else if (path == 1)
    ++E.nlaunch, k_seq_sums<1><<<grid, 256, 0, E.stream>>>(nseg, off, x, init, out);
  else
    ++E.nlaunch, k_seq_sums<0><<<grid, 256, 0, E.stream>>>(nseg, off, x, init, out);
  HL_LAUNCH_CHECK();
}

// Ordered row sums of the flagged rows (all rows without flags).
static void row_sums_ordered(Engine& E, Level& L, const u8* flags) {
  const LongList ll = long_list(E, L.g.nnz, L.g.n);
  ++E.nlaunch, k_row_sum_serial<<<grid_for(L.g.n), 256, 0, E.stream>>>(
      L.g.n, L.g.off.p, L.g.w.p, L.k.p, flags, ll);
  ++E.nlaunch, k_row_sum_serial_long<<<LONG_BLOCKS, 256, 0, E.stream>>>(ll, L.g.off.p, L.g.w.p,
                                                                        L.k.p);
}

// Warp-parallel row sums; only used when every weight is integral, where any
// summation order gives the same bits.
__global__ void k_row_sum_warp(u32 n, const u64* off, const double* w, double* k,
                               const u8* flags, LongList ll) {
  const u32 lane = threadIdx.x & 31;
  const u64 warp = (blockIdx.x * (u64)blockDim.x + threadIdx.x) >> 5;
  const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 v0 = warp * 32; v0 < n; v0 += nwarps * 32) {
    const u64 v = v0 + lane;
    bool on = v < n && (!flags || flags[v]);
    const u64 a = on ? off[v] : 0, b = on ? off[v + 1] : 0;
    if (b - a >= LONG_SEG) {
      ll.seg[atomicAdd(ll.cnt, 1u)] = (u32)v;
      on = false;
    }
    double mine = 0.0;
    for (u32 m = __ballot_sync(0xffffffffu, on); m; m &= m - 1) {
      const u32 j = __ffs(m) - 1;
      const u64 hi = __shfl_sync(0xffffffffu, b, j);
      u64 p = __shfl_sync(0xffffffffu, a, j) + lane;
      double s = 0.0;
      for (; p + 224 < hi; p += 256) {  // 8 loads in flight
        double y[8];
#pragma unroll
        for (u32 i = 0; i < 8; ++i) y[i] = w[p + 32 * i];
#pragma unroll
        for (u32 i = 0; i < 8; ++i) s += y[i];
      }
      for (; p < hi; p += 32) s += w[p];
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == j) mine = s;
    }
    if (on) k[v] = mine;
  }
}

// The listed rows, a block each.
__global__ void __launch_bounds__(256) k_row_sum_warp_long(LongList ll, const u64* off,
                                                           const double* w, double* k) {
  __shared__ double sh[8];
  const u32 cnt = *ll.cnt;
  for (u32 i = blockIdx.x; i < cnt; i += gridDim.x) {
    const u32 v = ll.seg[i];
    const double s = block_sum_any(w, off[v], off[v + 1], sh);
    if (threadIdx.x == 0) k[v] = s;
  }
}

// Row sums in any order of the flagged rows (all rows without flags).
static void row_sums_integral(Engine& E, Level& L, const u8* flags) {
  const LongList ll = long_list(E, L.g.nnz, L.g.n);
  ++E.nlaunch, k_row_sum_warp<<<grid_for(L.g.n), 256, 0, E.stream>>>(
      L.g.n, L.g.off.p, L.g.w.p, L.k.p, flags, ll);
  ++E.nlaunch, k_row_sum_warp_long<<<LONG_BLOCKS, 256, 0, E.stream>>>(ll, L.g.off.p, L.g.w.p,
                                                                      L.k.p);
}

// Fixed-shape pairwise sum: tiles of 1024 (+0.0 padded) folded by stride
// halving; repeated on the tile sums until one value remains.
__global__ void k_tree_tile(const double* x, u64 n, double* out) {
  __shared__ double s[1024];
  u64 base = (u64)blockIdx.x * 1024;
  for (u32 i = threadIdx.x; i < 1024; i += blockDim.x) {
    u64 idx = base + i;
    s[i] = idx < n ? x[idx] : 0.0;
  }
  __syncthreads();
  for (u32 st = 512; st >= 1; st >>= 1) {
    for (u32 i = threadIdx.x; i < st; i += blockDim.x) s[i] = __dadd_rn(s[i], s[i + st]);
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = s[0];
}

double tree_sum(Engine& E, const double* x, u64 n) {
  if (n == 0) return 0.0;
  u64 tiles = (n + 1023) / 1024;
  E.sc.red.ensure(E.mem, tiles + 1);
  E.sc.red2.ensure(E.mem, (tiles + 1023) / 1024 + 1);
  const double* src = x;
  double* a = E.sc.red.p;
  double* b = E.sc.red2.p;
  u64 cur = n;
  while (true) {
    u64 t = (cur + 1023) / 1024;
    ++E.nlaunch, k_tree_tile<<<(u32)t, 256, 0, E.stream>>>(src, cur, a);
    HL_LAUNCH_CHECK();
    if (t == 1) break;
    src = a;
    cur = t;
    std::swap(a, b);
  }
  return E.read_f64(a);
}

// Rows whose flag is set (no list, so no count to read back first).
static void recompute_flagged_rows(Engine& E, Level& L, const u8* flags) {
  const u32 n = L.g.n;
  if (!n) return;
  cudaEvent_t ev = E.kt_begin();
  if (E.integral) row_sums_integral(E, L, flags);
  else row_sums_ordered(E, L, flags);
  HL_LAUNCH_CHECK();
  E.kt_end(KT_ROW_SUMS, ev);
}

void recompute_all_degrees(Engine& E, Level& L) {
  u32 n = L.g.n;
  if (n) {
    if (E.integral) row_sums_integral(E, L, nullptr);
    else row_sums_ordered(E, L, nullptr);
    HL_LAUNCH_CHECK();
  }
  L.tw = tree_sum(E, L.k.p, n);
}

struct FlagToIndex {
  const u8* f;
  __host__ __device__ bool operator()(const u32& i) const { return f[i] != 0; }
};

void apply_delta(Engine& E, Level& L, const DevEdges& b, u32 new_n, bool keep_loops) {
  Scratch& S = E.sc;
  cudaStream_t st = E.stream;
  if (new_n > L.g.n) graph_grow_nodes(E, L, new_n);
  const u32 n = L.g.n;
  const bool drop_loops = !keep_loops && L.g.self_loop_entries > 0;
  if (b.k == 0 && !drop_loops) return;
  if (gang_apply_fits(E, L, b, drop_loops)) {
    gang_apply(E, L, b);
    return;
  }
  const u64 k = b.k;

  S.ktouched.ensure(E.mem, n ? n : 1);
  HL_CUDA(cudaMemsetAsync(S.ktouched.p, 0, n ? n : 1, st));
  S.cnt.ensure(E.mem, 16);
  HL_CUDA(cudaMemsetAsync(S.cnt.p, 0, 16 * sizeof(u32), st));  // [0] ins loops [1] del loops [2] drops

  u32 U = 0;
  cudaEvent_t ev_ds = E.kt_begin();
  if (k) {
    S.keys.ensure(E.mem, k);
    S.keys2.ensure(E.mem, k);
    S.idx.ensure(E.mem, k);
    S.idx2.ensure(E.mem, k);
    S.segid.ensure(E.mem, k);
    S.seg_start.ensure(E.mem, k + 1);
    S.rowlist.ensure(E.mem, k);
    ++E.nlaunch, k_delta_keys<<<grid_for(k), 256, 0, st>>>(b.u, b.v, k, S.keys.p, S.idx.p);
    HL_LAUNCH_CHECK();
    u64* kin = S.keys.p;
    u64* kout = S.keys2.p;
    u32* vin = S.idx.p;
    u32* vout = S.idx2.p;
    cub_run(E, [&](void* t, size_t& bytes) {
      // keys (u << 32) | v with u, v < n
      return cub::DeviceRadixSort::SortPairs(t, bytes, kin, kout, vin, vout, (int64_t)k, 0,
                                             32 + bits_for(n ? n - 1 : 0), st);
    });
    ++E.nlaunch, k_heads<<<grid_for(k), 256, 0, st>>>(kout, k, S.rowlist.p);
    HL_LAUNCH_CHECK();
    u32* head = S.rowlist.p;
    u32* segid = S.segid.p;
    cub_run(E, [&](void* t, size_t& bytes) {
      return cub::DeviceScan::ExclusiveSum(t, bytes, head, segid, (int64_t)k, st);
    });
    ++E.nlaunch, k_seg_start<<<grid_for(k), 256, 0, st>>>(head, segid, k, S.seg_start.p);
    HL_LAUNCH_CHECK();
    u32 lh[2];
    E.read_u32s({segid + (k - 1), head + (k - 1)}, lh);
    U = lh[0] + lh[1];

    S.op.ensure(E.mem, U);
    S.neww.ensure(E.mem, U);
    S.nops_del.ensure(E.mem, U + 1);
    S.nops_ins.ensure(E.mem, U + 1);
    S.pos_del.ensure(E.mem, U + 1);
    S.pos_ins.ensure(E.mem, U + 1);
    ++E.nlaunch, k_resolve<<<grid_for(U), 256, 0, st>>>(U, S.seg_start.p, k, kout, vout, b.w, L.g.off.p,
                                           L.g.col.p, L.g.w.p, keep_loops, S.op.p, S.neww.p,
                                           S.ktouched.p, S.nops_del.p, S.nops_ins.p, S.cnt.p);
    HL_LAUNCH_CHECK();
    HL_CUDA(cudaMemsetAsync(S.nops_del.p + U, 0, sizeof(u32), st));
    HL_CUDA(cudaMemsetAsync(S.nops_ins.p + U, 0, sizeof(u32), st));
    u32* nd = S.nops_del.p;
    u32* pd = S.pos_del.p;
    u32* ni = S.nops_ins.p;
    u32* pi = S.pos_ins.p;
    cub_run(E, [&](void* t, size_t& bytes) {
      return cub::DeviceScan::ExclusiveSum(t, bytes, nd, pd, (int64_t)U + 1, st);
    });
    cub_run(E, [&](void* t, size_t& bytes) {
      return cub::DeviceScan::ExclusiveSum(t, bytes, ni, pi, (int64_t)U + 1, st);
    });
  }
  E.kt_end(KT_DELTA_SORT, ev_ds);
  u64 n_del_keys = 0, n_ins = 0;
  if (U) {
    u32 di[2];
    E.read_u32s({S.pos_del.p + U, S.pos_ins.p + U}, di);
    n_del_keys = di[0];
    n_ins = di[1];
  }

  // Existing self-loops to drop (reference behaviour) — counted first.
  u64 n_drop = 0;
  if (drop_loops) {
    HL_CUDA(cudaMemsetAsync(S.cnt.p + 3, 0, sizeof(u32), st));
    ++E.nlaunch, k_count_loops<<<grid_for(n), 256, 0, st>>>(n, L.g.off.p, L.g.col.p, S.cnt.p + 3);
    HL_LAUNCH_CHECK();
    n_drop = E.read_u32(S.cnt.p + 3);
  }
  u64 R = n_del_keys + n_drop + n_ins;

  if (R == 0) {
    // Weight updates only: no structural change.
    if (U) {
      recompute_flagged_rows(E, L, S.ktouched.p);
      L.tw = tree_sum(E, L.k.p, n);
    }
    return;
  }

  S.rkeys.ensure(E.mem, R);
  S.rkeys2.ensure(E.mem, R);
  S.rvals.ensure(E.mem, R);
  S.rvals2.ensure(E.mem, R);
  if (U)
    ++E.nlaunch, k_emit_rowops<<<grid_for(U), 256, 0, st>>>(U, S.seg_start.p, S.keys2.p, S.op.p, S.pos_del.p,
                                               S.pos_ins.p, n_del_keys + n_drop, S.rkeys.p,
                                               S.rvals.p);
  if (drop_loops && n_drop)
    ++E.nlaunch, k_emit_loop_drops<<<grid_for(n), 256, 0, st>>>(n, L.g.off.p, L.g.col.p, S.rkeys.p, S.rvals.p,
                                                   n_del_keys, n_del_keys + n_drop, S.cnt.p + 2,
                                                   S.ktouched.p, S.cnt.p + 4);
  HL_LAUNCH_CHECK();
  {
    u64* kin = S.rkeys.p;
    u64* kout = S.rkeys2.p;
    u32* vin = S.rvals.p;
    u32* vout = S.rvals2.p;
    cub_run(E, [&](void* t, size_t& bytes) {
      // keys (row << 32) | neighbour with both < n
      return cub::DeviceRadixSort::SortPairs(t, bytes, kin, kout, vin, vout, (int64_t)R, 0,
                                             32 + bits_for(n ? n - 1 : 0), st);
    });
  }
  require(R < 0xFFFFFFFFull, "too many row operations in one batch");
  // deletes before every operation, and its position in the old entries
  S.opdel.ensure(E.mem, R + 1);
  S.opdelpre.ensure(E.mem, R + 1);
  ++E.nlaunch, k_del_flags<<<grid_for(R + 1), 256, 0, st>>>(S.rvals2.p, R, S.opdel.p);
  HL_LAUNCH_CHECK();
  {
    u32* a = S.opdel.p;
    u32* o = S.opdelpre.p;
    cub_run(E, [&](void* t, size_t& bytes) {
      return cub::DeviceScan::ExclusiveSum(t, bytes, a, o, (int64_t)R + 1, st);
    });
  }
  u64* opos = S.rkeys.p;  // the unsorted keys are done with
  ++E.nlaunch, k_rowop_positions<<<grid_for(R), 256, 0, st>>>(S.rkeys2.p, S.rvals2.p, R,
                                                               L.g.off.p, L.g.col.p, opos);
  HL_LAUNCH_CHECK();
  S.newoff.ensure(E.mem, (size_t)n + 1);
  DevGraph& G = L.g;
  const u64 nnz_new = G.nnz + R - 2ull * E.read_u32(S.opdelpre.p + R);
  DBuf<u32>& ncol = G.col2;
  DBuf<double>& nw = G.w2;
  ncol.ensure_slack(E.mem, nnz_new ? nnz_new : 1);
  nw.ensure_slack(E.mem, nnz_new ? nnz_new : 1);
  cudaEvent_t kev = E.kt_begin();
  const RowOps O{(u32)R, S.rkeys2.p, S.rvals2.p, S.opdelpre.p, opos};
  ++E.nlaunch, k_rebuild<<<grid_for(G.nnz / 8 + R + n), 256, 0, st>>>(
      O, n, G.nnz, G.off.p, G.col.p, G.w.p, S.neww.p, S.newoff.p, ncol.p, nw.p, nnz_new,
      S.cnt.p + 4);
  HL_LAUNCH_CHECK();
  E.kt_end(KT_MERGE_ROWS, kev);
  // old and new offsets, old and new (col, w) entries
  E.kagg[KT_MERGE_ROWS].bytes += 16ull * ((u64)n + 1) + 12ull * (G.nnz + nnz_new);
  u32 ce[3];  // merge errors, inserted and deleted self-loops
  E.read_u32s({S.cnt.p + 4, S.cnt.p + 0, S.cnt.p + 1}, ce);
  if (ce[0] != 0)
    throw Error(HL_ERR_CUDA, "internal error: CSR merge produced an out-of-range position");
  G.col.swap(ncol);
  G.w.swap(nw);
  G.off.swap(S.newoff);
  G.nnz = nnz_new;
  {
    u32 ins_loops = ce[1];
    u32 del_loops = ce[2];
    if (drop_loops)
      G.self_loop_entries = 2ull * ins_loops;
    else
      G.self_loop_entries = G.self_loop_entries + 2ull * ins_loops - 2ull * del_loops;
  }
  // Degrees of every row whose weights changed, then 2m.
  recompute_flagged_rows(E, L, S.ktouched.p);
  L.tw = tree_sum(E, L.k.p, n);
}

}  // namespace hl
