// gang_modularity.cu — Q = (Σ_intra w − Σ_C d(C)²/2m) / 2m in one launch
// (hit_leiden.rs:121-161), and first-seen label canonicalisation in one
// (hit_leiden.rs:358-376).
//
// Each undirected edge appears twice in the CSR (a self-loop twice in its own
// row), so the CSR intra sum equals the reference's 2·Σ_intra over its edge
// list and the row sums equal its node degrees.  Every partial sum is carried as
// a double-double (error-free TwoSum); d(C) is the ordered sum of its members'
// degrees, so Q agrees with any faithful ordering to ~1e-15 relative.
#include "csr_rebuild.cuh"
#include "gang.cuh"

namespace hl {

struct DD {
  double hi, lo;
};

__device__ __forceinline__ DD dd_add(DD a, double b) {
  const double s = __dadd_rn(a.hi, b);
  const double bb = __dsub_rn(s, a.hi);
  const double err = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  return {s, __dadd_rn(a.lo, err)};
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  DD r = dd_add(a, b.hi);
  r.lo = __dadd_rn(r.lo, b.lo);
  return r;
}
__device__ __forceinline__ DD dd_shfl_xor(DD a, u32 o) {
  return {__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
}

struct ModCnt {  // zeroed by the host
  u32 maxlab, work;
};

struct GangModArgs {
  u32 n;
  const u64* off;
  const u32* col;
  const double* w;
  const double* k;
  const u32* part;
  double tw;
  bool grid, integral;
  u32 *lab, *idx, *lab2, *idx2, *hist, *gpart;
  double* kval;
  double* partial;  // per block: intra hi, lo, expected hi, lo
  ModCnt* cnt;
  u32* cnt_next;
  double* out;      // intra, expected
};

constexpr u32 MOD_ROWS = 32;      // rows a warp takes at a time
constexpr u32 MOD_AHEAD = 4;      // groups of four rows whose loads are in flight together
constexpr u32 MOD_LONG = 256;     // rows above this take the whole warp

// Sum of the 32 lanes' double-doubles of this warp's share, block by block, to
// partial[2 q], partial[2 q + 1].
__device__ __forceinline__ void mod_block_sum(DD x, DD* sh, double* out) {
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  for (u32 o = 16; o; o >>= 1) x = dd_add(x, dd_shfl_xor(x, o));
  if (lane == 0) sh[wib] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    DD s{0.0, 0.0};
    for (u32 i = 0; i < GANG_WARPS; ++i) s = dd_add(s, sh[i]);
    out[0] = s.hi;
    out[1] = s.lo;
  }
  __syncthreads();
}

// What bounds it: reading the CSR and gathering the neighbours' labels (16
// bytes an entry); a large community's ordered degree sum is one warp's (8-11
// cycles a member, 700k vertices in two communities: 2.45 ms a call) beside it.  500k vertices, 12M entries, 4,000
// communities: row sums 133 us, ordered degrees 56 us and some twenty launches
// with five host reads, 520 us a call, become one launch and 375 us (with one
// group of rows in flight a warp and 128 rows taken at a time: 458).
__global__ void __launch_bounds__(GANG_THREADS, 1) k_gang_modularity(GangModArgs A) {
  __shared__ GangSmem S;
  __shared__ __align__(16) double chain[GANG_WARPS][CHAIN_TILE];
  __shared__ DD sh[GANG_WARPS];
  const Gang G = gang_make(A.grid);
  const u32 lane = threadIdx.x & 31;
  const u32 gt = G.thread(), gts = G.threads();
  ModCnt& C = *A.cnt;
  gang_clear_next(G, A.cnt_next);
  // ---- the largest label ----
  {
    u32 mx = 0;
    for (u32 v = gt; v < A.n; v += gts) mx = max(mx, A.part[v]);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(&C.maxlab, mx);
  }
  G.sync();
  DD expected{0.0, 0.0}, intra{0.0, 0.0};
  auto square = [&](u32, double x) {
    expected = dd_add(expected, __ddiv_rn(__dmul_rn(x, x), A.tw));
  };
  if (A.integral && C.maxlab < A.n) {
    // ---- Σ_C d(C)²/2m: integral degrees add up in any order, in shared memory
    // while the labels fit it: no label sort and no ordered sum (300k vertices in
    // 2 and 30 communities: 289 and 332 us in the multi-kernel form, 182 and 184
    // so).
    const u32 nc = C.maxlab + 1;
    const bool local = nc <= GANG_WORDS;
    for (u32 c = gt; c < nc; c += gts) A.kval[c] = 0.0;
    if (local)
      for (u32 c = threadIdx.x; c < nc; c += GANG_THREADS) S.key[c] = 0;
    __syncthreads();
    G.sync();
    for (u32 t0 = G.warp() * 32; t0 < A.n; t0 += G.warps() * 32) {
      const u32 v = t0 + lane;
      const bool ok = v < A.n;
      const u32 c = ok ? A.part[v] : 0;
      unsigned long long x = ok ? (unsigned long long)A.k[v] : 0ull;
      const u32 grp = __match_any_sync(0xffffffffu, ok ? c : NONE32);
      const bool lead = ok && lane == (u32)(__ffs(grp) - 1);
      // lanes of one community add up first
      for (u32 m = __ballot_sync(0xffffffffu, lead && (grp & (grp - 1))); m; m &= m - 1) {
        const u32 l = __ffs(m) - 1;
        const u32 gm = __shfl_sync(0xffffffffu, grp, l);
        unsigned long long y = (gm >> lane) & 1u ? x : 0ull;
        for (u32 o = 16; o; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (lane == l) x = y;
      }
      if (!lead) continue;
      if (local) atomicAdd(reinterpret_cast<unsigned long long*>(&S.key[c]), x);
      else atomicAdd(&A.kval[c], (double)x);
    }
    __syncthreads();
    if (local)
      for (u32 c = threadIdx.x; c < nc; c += GANG_THREADS)
        if (S.key[c]) atomicAdd(&A.kval[c], (double)S.key[c]);
    G.sync();
    for (u32 c = gt; c < nc; c += gts) square(c, A.kval[c]);
  } else {
    // ---- members by community, their degrees in that order ----
    const u32 bits = C.maxlab ? 32 - __clz(C.maxlab) : 1;
    bool second;
    gang_label_sort(G, S, A.n, bits, [&](u32 i) { return A.part[i]; }, A.lab, A.idx, A.lab2,
                    A.idx2, A.hist, A.gpart, &second);
    const u32* lab = second ? A.lab2 : A.lab;
    const u32* idx = second ? A.idx2 : A.idx;
    for (u32 t = gt; t < A.n; t += gts) A.kval[t] = A.k[idx[t]];
    G.sync();
    // ---- Σ_C d(C)²/2m ----
    if (A.integral)
      gang_segment_sums<true>(G, A.n, lab, A.kval, chain[threadIdx.x >> 5], square);
    else
      gang_segment_sums(G, A.n, lab, A.kval, chain[threadIdx.x >> 5], square);
  }
  // ---- intra weight: eight lanes a row, taken by the warps as they come ----
  const u32 sub = lane & 7;
  const u32 chunks = (A.n + MOD_ROWS - 1) / MOD_ROWS;
  while (true) {
    u32 ch = 0;
    if (lane == 0) ch = atomicAdd(&C.work, 1u);
    ch = __shfl_sync(0xffffffffu, ch, 0);
    if (ch >= chunks) break;
    // MOD_AHEAD groups of four rows at once: a group is a chain of three
    // dependent loads (offsets, neighbours, labels) that one warp would wait
    // for in turn
    for (u32 r = 0; r < MOD_ROWS; r += 4 * MOD_AHEAD) {
      u64 a[MOD_AHEAD], b[MOD_AHEAD];
      u32 c[MOD_AHEAD], nb[MOD_AHEAD][4];
      double x[MOD_AHEAD][4];
#pragma unroll
      for (u32 k = 0; k < MOD_AHEAD; ++k) {
        const u64 v = (u64)ch * MOD_ROWS + r + 4 * k + (lane >> 3);
        const bool live = v < A.n;
        a[k] = live ? A.off[v] : 0;
        b[k] = live ? A.off[v + 1] : 0;
        c[k] = live ? A.part[v] : 0;
      }
#pragma unroll
      for (u32 k = 0; k < MOD_AHEAD; ++k) {
        const u64 stop = b[k] - a[k] > MOD_LONG ? a[k] : b[k];
#pragma unroll
        for (u32 j = 0; j < 4; ++j) {
          const u64 p = a[k] + sub + 8 * j;
          nb[k][j] = p < stop ? A.col[p] : NONE32;
          x[k][j] = p < stop ? A.w[p] : 0.0;
        }
      }
#pragma unroll
      for (u32 k = 0; k < MOD_AHEAD; ++k)
#pragma unroll
        for (u32 j = 0; j < 4; ++j)
          if (nb[k][j] == NONE32 || A.part[nb[k][j]] != c[k]) x[k][j] = 0.0;
#pragma unroll
      for (u32 k = 0; k < MOD_AHEAD; ++k) {
        const bool big = b[k] - a[k] > MOD_LONG;
        DD s{0.0, 0.0};
#pragma unroll
        for (u32 j = 0; j < 4; ++j)
          if (x[k][j] != 0.0) s = dd_add(s, x[k][j]);
        if (!big)
          for (u64 p0 = a[k] + sub + 32; p0 < b[k]; p0 += 32) {
            u32 m[4];
            double y[4];
#pragma unroll
            for (u32 j = 0; j < 4; ++j) m[j] = p0 + 8 * j < b[k] ? A.col[p0 + 8 * j] : NONE32;
#pragma unroll
            for (u32 j = 0; j < 4; ++j) y[j] = m[j] != NONE32 ? A.w[p0 + 8 * j] : 0.0;
#pragma unroll
            for (u32 j = 0; j < 4; ++j)
              if (m[j] != NONE32 && A.part[m[j]] == c[k]) s = dd_add(s, y[j]);
          }
        for (u32 o = 4; o; o >>= 1) s = dd_add(s, dd_shfl_xor(s, o));
        // a row's sum is rounded before the total, as the reference adds rows
        if (!big && sub == 0) intra = dd_add(intra, s.hi + s.lo);
        for (u32 bm = __ballot_sync(0xffffffffu, big && sub == 0); bm; bm &= bm - 1) {
          const u32 l = __ffs(bm) - 1;
          const u64 ba = __shfl_sync(0xffffffffu, a[k], l), bb = __shfl_sync(0xffffffffu, b[k], l);
          const u32 bc = __shfl_sync(0xffffffffu, c[k], l);
          DD t{0.0, 0.0};
          for (u64 p = ba + lane; p < bb; p += 32)
            if (A.part[A.col[p]] == bc) t = dd_add(t, A.w[p]);
          for (u32 o = 16; o; o >>= 1) t = dd_add(t, dd_shfl_xor(t, o));
          if (lane == 0) intra = dd_add(intra, t.hi + t.lo);
        }
      }
    }
  }
  // ---- totals ----
  mod_block_sum(intra, sh, A.partial + 4 * G.rank);
  mod_block_sum(expected, sh, A.partial + 4 * G.rank + 2);
  G.sync();
  if (gt == 0) {
    DD si{0.0, 0.0}, se{0.0, 0.0};
    for (u32 r = 0; r < G.nct; ++r) {
      si = dd_add(si, DD{A.partial[4 * r], A.partial[4 * r + 1]});
      se = dd_add(se, DD{A.partial[4 * r + 2], A.partial[4 * r + 3]});
    }
    A.out[0] = si.hi + si.lo;
    A.out[1] = se.hi + se.lo;
  }
}

double modularity(Engine& E, Level& L, const u32* part) {
  const u32 n = L.g.n;
  if (!n || L.tw == 0.0) return 0.0;
  Scratch& S = E.sc;
  GangShape shape = gang_shape(E, 8ull * n + L.g.nnz);
  // a tight budget: no label sort where none is needed, digit counts (16 KB a
  // block) of no more than 8 bytes a vertex, and nothing stays
  E.plan_scratch(0, 0, 0, 1);
  if (E.lean && shape.grid && n / 2048 < shape.blocks) shape = GangShape{8, false};
  if (E.lean && !shape.grid && n / 2048 < shape.blocks) shape = GangShape{1, false};
  const bool keep_kval = !E.lean || S.fvals.cap > 0;
  if (E.lean) S.cnt.ensure(E.mem, 16);
  if (!E.lean || !E.integral || reduce_max_u32(E, part, n, S.cnt.p + 12) >= n) {
    S.used.ensure(E.mem, n);
    S.rank.ensure(E.mem, n);
    S.order.ensure(E.mem, n);
    S.order2.ensure(E.mem, n);
    S.gm_hist.ensure(E.mem, (size_t)256 * GANG_WARPS * shape.blocks);
  }
  S.fvals.ensure(E.mem, n);
  S.gang_part.ensure(E.mem, GANG_MAX_BLOCKS);
  S.red.ensure(E.mem, 4 * GANG_MAX_BLOCKS);
  GangModArgs A{};
  A.n = n;
  A.off = L.g.off.p;
  A.col = L.g.col.p;
  A.w = L.g.w.p;
  A.k = L.k.p;
  A.part = part;
  A.tw = L.tw;
  A.integral = E.integral;
  A.grid = shape.grid;
  A.lab = S.used.p;
  A.lab2 = S.rank.p;
  A.idx = S.order.p;
  A.idx2 = S.order2.p;
  A.hist = S.gm_hist.p;
  A.gpart = S.gang_part.p;
  A.kval = S.fvals.p;
  A.partial = S.red.p;
  A.cnt = reinterpret_cast<ModCnt*>(gang_counters(E, &A.cnt_next));
  A.out = reinterpret_cast<double*>(E.hs.p);
  gang_launch(E, reinterpret_cast<const void*>(&k_gang_modularity), shape, 0, &A);
  gang_turn(E);
  E.sync();
  double q[2];
  std::memcpy(q, E.hs.p, sizeof(q));
  if (E.lean) S.gm_hist.release();
  if (!keep_kval) S.fvals.release();
  return (q[0] - q[1]) / L.tw;
}

// ---------------------------------------------------------------------------
// First-seen relabelling: a label's new id is the rank of its first index.
// ---------------------------------------------------------------------------
struct GangCanonArgs {
  u32 n, bound;      // labels are below bound
  const u32* lab;
  u32 *first, *rank; // per label
  u32* out;
  u32* part;
  bool grid;
};

__global__ void __launch_bounds__(GANG_THREADS, 1) k_gang_canonical(GangCanonArgs A) {
  __shared__ GangSmem S;
  const Gang G = gang_make(A.grid);
  const u32 gt = G.thread(), gts = G.threads();
  for (u32 c = gt; c < A.bound; c += gts) A.first[c] = NONE32;
  G.sync();
  const u32 lane = threadIdx.x & 31;
  for (u32 v0 = gt - lane; v0 < A.n; v0 += gts) {
    const u32 v = v0 + lane;
    const u32 c = v < A.n ? A.lab[v] : NONE32;
    // the lanes of one label ask once (its lowest lane has the lowest index)
    const u32 grp = __match_any_sync(0xffffffffu, c);
    if (v < A.n && !(grp & ((1u << lane) - 1u))) atomicMin(&A.first[c], v);
  }
  G.sync();
  gang_scan(
      G, S, A.n, [&](u32 v) { return A.first[A.lab[v]] == v ? 1u : 0u; },
      [&](u32 v, u32 ex) {
        const u32 c = A.lab[v];
        if (A.first[c] == v) A.rank[c] = ex;
      },
      A.part);
  G.sync();
  for (u32 v = gt; v < A.n; v += gts) A.out[v] = A.rank[A.lab[v]];
}

void canonicalize_bounded(Engine& E, const u32* labels, u32 n, u32 bound, u32* out) {
  if (!n) return;
  Scratch& S = E.sc;
  const GangShape shape = gang_shape(E, 4ull * n + bound);
  S.used.ensure(E.mem, bound);
  S.rank.ensure(E.mem, bound);
  S.gang_part.ensure(E.mem, GANG_MAX_BLOCKS);
  GangCanonArgs A{};
  A.n = n;
  A.bound = bound;
  A.lab = labels;
  A.first = S.used.p;
  A.rank = S.rank.p;
  A.out = out;
  A.part = S.gang_part.p;
  A.grid = shape.grid;
  gang_launch(E, reinterpret_cast<const void*>(&k_gang_canonical), shape, 0, &A);
}

}  // namespace hl
