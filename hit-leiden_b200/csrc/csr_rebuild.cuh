// csr_rebuild.cuh — a CSR rewritten by sorted row-operations, entry-parallel.
// Shared by the multi-kernel and the single-launch delta application.
//
// The operations are sorted by (row, neighbour); a self-loop's come in pairs,
// and deletes of a key come before inserts of the same key (a dropped loop
// replaced by an inserted one).  Operation t has a position e[t] in the old
// entries: where a deleted entry stands, or before which an insert lands.  e
// ascends, so with s = the number of operations at positions <= p and dpre the
// deletes before each operation, a surviving old entry p moves to
//     p + s - 2 dpre[s]        (s - dpre[s] inserts before it, dpre[s] deletes)
// and an insert t goes to
//     e[t] + t - 2 dpre[t].
// No row is walked: all entries between two operations move by the same
// distance, touched row or not, so the copy streams, and rows of any length
// split evenly.
#pragma once
#include "hl_internal.cuh"

namespace hl {

// Value of a row-operation that deletes (an insert carries the index of its
// weight).
constexpr u32 DEL_MARK = 0xFFFFFFFFu;

struct RowOps {
  u32 R;
  const u64* keys;  // row << 32 | neighbour, ascending
  const u32* vals;
  const u32* dpre;  // deletes before each operation, R + 1 entries
  const u64* e;
};

// Position of operation t (keys and values as in RowOps).
__device__ __forceinline__ u64 rowop_position(u32 t, const u64* keys, const u32* vals,
                                              const u64* off, const u32* col) {
  const u64 key = keys[t];
  const u32 row = (u32)(key >> 32);
  u64 e = lower_bound_u32(col, off[row], off[row + 1], (u32)key);
  for (u32 x = t; x > 0 && keys[x - 1] == key; --x)
    if (vals[x - 1] == DEL_MARK) ++e;  // a loop's second copy; an insert after its deletes
  return e;
}

// First index in [lo, hi) of the ascending a with a[i] >= x / > x.
__device__ __forceinline__ u32 lb_u64(const u64* a, u32 lo, u32 hi, u64 x) {
  while (lo < hi) {
    const u32 mid = lo + (hi - lo) / 2;
    if (a[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ u32 ub_u64(const u64* a, u32 lo, u32 hi, u64 x) {
  while (lo < hi) {
    const u32 mid = lo + (hi - lo) / 2;
    if (a[mid] <= x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The same searches by a whole warp for one x: 32 probes a step.
template <bool UPPER>
__device__ __forceinline__ u32 warp_bound_u64(const u64* a, u32 lo, u32 hi, u64 x) {
  const u32 lane = threadIdx.x & 31;
  while (hi - lo > 32) {
    const u32 step = (hi - lo + 31) / 32;
    const u64 p = (u64)lo + (u64)step * lane;
    const bool below = p < hi && (UPPER ? a[p] <= x : a[p] < x);
    const u32 m = __ballot_sync(0xffffffffu, below);
    if (!m) return lo;  // not even a[lo]
    const u32 j = 31 - __clz(m);
    const u64 nhi = (u64)lo + (u64)step * (j + 1);
    lo = lo + step * j + 1;
    hi = nhi < hi ? (u32)nhi : hi;
  }
  const bool below = lo + lane < hi && (UPPER ? a[lo + lane] <= x : a[lo + lane] < x);
  return lo + (u32)__popc(__ballot_sync(0xffffffffu, below));
}

// New row offsets, a warp per 256 rows: off[v] plus the net insertions of the
// rows before v.  The few operations of those rows sit in the lanes.
__device__ __forceinline__ void rebuild_offsets(const RowOps& O, u32 n, const u64* off, u64* noff,
                                                u64 warp, u64 warps) {
  const u32 lane = threadIdx.x & 31;
  for (u64 v0 = warp * 256; v0 <= n; v0 += warps * 256) {
    const u64 v1 = v0 + 255 < n ? v0 + 255 : n;
    const u32 t0 = warp_bound_u64<false>(O.keys, 0, O.R, v0 << 32);
    const u32 t1 = warp_bound_u64<false>(O.keys, t0, O.R, v1 << 32);
    u64 o[8];
#pragma unroll
    for (u32 j = 0; j < 8; ++j) {
      const u64 v = v0 + 32 * j + lane;
      o[j] = v <= v1 ? off[v] : 0;
    }
    if (t1 - t0 < 32) {
      const u32 row = t0 + lane < t1 ? (u32)(O.keys[t0 + lane] >> 32) : NONE32;
      const u32 dp = t0 + lane <= t1 ? O.dpre[t0 + lane] : 0u;
#pragma unroll
      for (u32 j = 0; j < 8; ++j) {
        const u64 v = v0 + 32 * j + lane;
        u32 c = 0;
        for (u32 i = 0; i < t1 - t0; ++i)
          c += __shfl_sync(0xffffffffu, row, i) < (u32)v ? 1u : 0u;
        const u32 d = __shfl_sync(0xffffffffu, dp, c);
        if (v <= v1) noff[v] = o[j] + (t0 + c) - 2ull * d;
      }
    } else {
#pragma unroll
      for (u32 j = 0; j < 8; ++j) {
        const u64 v = v0 + 32 * j + lane;
        if (v > v1) continue;
        const u32 t = lb_u64(O.keys, t0, t1, v << 32);
        noff[v] = o[j] + t - 2ull * O.dpre[t];
      }
    }
  }
}

// Surviving old entries, a warp per 256.
__device__ __forceinline__ void rebuild_entries(const RowOps& O, u64 nnz, const u32* col,
                                                const double* w, u32* ncol, double* nw,
                                                u64 nnz_new, u32* err, u64 warp, u64 warps) {
  const u32 lane = threadIdx.x & 31;
  for (u64 p0 = warp * 256; p0 < nnz; p0 += warps * 256) {
    const u64 p1 = p0 + 256 < nnz ? p0 + 256 : nnz;
    u32 c[8];
    double x[8];
#pragma unroll
    for (u32 j = 0; j < 8; ++j) {
      const u64 p = p0 + 32 * j + lane;
      if (p < p1) {
        c[j] = col[p];
        x[j] = w[p];
      }
    }
    const u32 s0 = warp_bound_u64<true>(O.e, 0, O.R, p0);
    const u32 s1 = warp_bound_u64<true>(O.e, s0, O.R, p1 - 1);
    const u64 d0 = O.dpre[s0];
#pragma unroll
    for (u32 j = 0; j < 8; ++j) {
      const u64 p = p0 + 32 * j + lane;
      if (p >= p1) continue;
      u32 s = s0;
      u64 d = d0;
      if (s0 != s1) {
        s = ub_u64(O.e, s0, s1, p);
        d = O.dpre[s];
      }
      if (s && O.e[s - 1] == p && O.vals[s - 1] == DEL_MARK) continue;
      const u64 q = p + s - 2 * d;
      if (q >= nnz_new) {
        atomicAdd(err, 1u);
        continue;
      }
      ncol[q] = c[j];
      nw[q] = x[j];
    }
  }
}

// Inserted entries, a thread per operation.
__device__ __forceinline__ void rebuild_inserts(const RowOps& O, const double* neww, u32* ncol,
                                                double* nw, u64 nnz_new, u32* err, u64 thread,
                                                u64 threads) {
  for (u64 t = thread; t < O.R; t += threads) {
    const u32 val = O.vals[t];
    if (val == DEL_MARK) continue;
    const u64 q = O.e[t] + t - 2ull * O.dpre[t];
    if (q >= nnz_new) {
      atomicAdd(err, 1u);
      continue;
    }
    ncol[q] = (u32)O.keys[t];
    nw[q] = neww[val];
  }
}

}  // namespace hl
