// gang_move.cu — inc-movement in one launch (hit_leiden.rs:1024-1101 →
// throughput.rs:80-236 → parallel_frontier.rs:133-239).
//
// Seeding, community degrees and whole movement rounds, with every size kept on
// the device: per round the frontier's best moves on the snapshot (a warp per
// vertex, a block per hub), the positive candidates sorted by (gain desc, node
// asc), the decoupled selection by reservations, the accepted moves, the next
// frontier and the K marks; the rules, bits and order of the multi-kernel
// rounds.  A round is atomic: the kernel hands the loop back at a round
// boundary (frontier as bytes in S.active) when the frontier outgrows its lists
// or a hub its tables, and the host continues with the multi-kernel rounds.
#include "csr_rebuild.cuh"
#include "gang.cuh"
#include "hub_sums.cuh"
#include "prune.cuh"

namespace hl {

constexpr u32 GM_MAXDEG = 256;      // rows a warp evaluates
constexpr u32 GM_TAB = 2 * GM_MAXDEG;
constexpr u32 GM_SLICE = 512;       // entries of a moved row a warp marks
constexpr u32 GM_MAX_SELECT = 64;   // reservation rounds before the serial finish

enum : u32 { GM_EMIT = 1, GM_ACC = 2 };
enum : u32 { GM_UNDECIDED = 0, GM_ACCEPTED = 1, GM_REJECTED = 2 };

struct MoveRound {  // of one parity; the other one's is cleared meanwhile
  u32 nv, nh, ncand, nops, nitems, work, hwork, big, wv, wh;
  u32 huge, whuge;  // a row of the frontier (to evaluate) outgrows the hub tables
};

// No hub table holds a row of this round: nothing further is taken up.
__device__ __forceinline__ void gm_big(MoveRound& R) {
  R.big = 1;
  atomicMax(&R.work, 1u << 30);
  atomicMax(&R.hwork, 1u << 30);
}

struct MoveCnt {  // zeroed by the host
  MoveRound r[2];
  u32 maxlab, und[2], pad_;
  unsigned long long moves, cands, trav, nfront, pruned;
};

struct MoveOutDev {
  u32 status, it, round, frontier;
  u64 epoch;
  unsigned long long moves, cands, trav, nfront, pruned;
};

struct WarpTabs {
  double tv[GANG_WARPS][GM_TAB];
  u32 tk[GANG_WARPS][GM_TAB];
  u32 tp[GANG_WARPS][GM_TAB];
  double sw[GANG_WARPS][GM_MAXDEG];
};
union MoveSmem {
  WarpTabs w;
  HubSmem<GANG_WARPS> h;
};

struct GangMoveArgs {
  u32 n;
  const u64* off;
  const u32* col;
  const double* w;
  u32* f;
  const u32* s;
  const double* k;
  double* d;
  u64 dcap;
  u8* active;    // frontier as bytes: on entry without setup, and on hand-back
  u8* changed;   // byte arrays padded to whole words
  u8* affected;
  const u8* kflag;  // K marks handed up from the level below, or null
  const u32* du;
  const u32* dv;
  const double* dw;
  u32 dk;
  bool setup, all_active, mark_moved, integral, grid;
  double tw, gamma;
  u32* bits[2];      // frontier bit sets
  u32* verts[2];     // frontier: rows of up to GM_MAXDEG entries
  u32* hubs[2];      // ... and longer ones
  u32 list_cap;      // entries of a list
  u32 max_frontier;  // vertices up to which a round stays in this launch
  u32 *wverts, *whubs;  // those of them that need an evaluation
  Prune prune;
  u32* to;           // per vertex: its candidate's target
  u64* ckey;
  u32* cnode;
  u64* skey;
  u32* sval;
  u32 *sel_node, *sel_from, *sel_to;
  u8 *status, *nmask;
  u32* role;
  unsigned long long* res;
  u64 *okey, *okey2, *otmp;  // d(C) updates: (community << 32 | 2 rank + enters), sorted:
  double* oterm;             // the communities and the signed degrees
  u32 *otv;
  u64* items;                // moved rows: (rank << 32 | slice)
  u32 items_cap;
  u32 *lab, *idx, *lab2, *idx2, *hist;
  double* kval;
  unsigned short* gslot;
  double* gw;
  u32* part;
  u32 it0, max_rounds, round0;
  bool more;  // max_rounds is this launch's own limit, not the movement's
  u64 epoch0;
  u32 label_bits;
  MoveCnt* cnt;
  u32* cnt_next;
  MoveOutDev* out;
};

__device__ __forceinline__ u32 gm_role(u32 r, u32 round) { return (r >> 2) == round ? (r & 3u) : 0u; }

// Vertex v joins the frontier of parity b (once).
__device__ __forceinline__ void gm_activate(const GangMoveArgs& A, u32 b, u32 v) {
  const u32 m = 1u << (v & 31);
  u32* word = &A.bits[b][v >> 5];
  if ((*word & m) || (atomicOr(word, m) & m)) return;
  MoveRound& R = A.cnt->r[b];
  const u64 deg = A.off[v + 1] - A.off[v];
  if (deg <= GM_MAXDEG) {
    const u32 at = atomicAdd(&R.nv, 1u);
    if (at < A.list_cap) A.verts[b][at] = v;
  } else {
    if (deg > HUB_MAXDEG) R.huge = 1;
    const u32 at = atomicAdd(&R.nh, 1u);
    if (at < A.list_cap) A.hubs[b][at] = v;
  }
}

// The decision from the best neighbour community: a positive gain wins, then
// the empty community n + v on a strict improvement.  Positive candidates are
// listed.
__device__ __forceinline__ void gm_finish(const GangMoveArgs& A, MoveRound& R, u32 v, u32 cur,
                                          double kv, double wcur, double dcur, double g, u32 p,
                                          u32 kk, bool bound, double shift) {
  u32 to = cur;
  double gain = 0.0;
  if (p != NONE32 && g > 0.0) {
    gain = g;
    to = kk;
  }
  if (A.tw != 0.0) {
    const double eg = empty_gain(wcur, A.tw, A.gamma, kv, dcur);
    if (bound && A.prune.b)
      prune_store(A.prune, shift, v, p != NONE32 && g > eg ? g : eg, kv, dcur, A.tw, A.gamma);
    if (eg > gain) {
      gain = eg;
      to = A.n + v;
    }
  }
  if (gain > 0.0) {
    const u32 at = atomicAdd(&R.ncand, 1u);
    A.ckey[at] = ~double_key(gain);
    A.cnode[at] = v;
    A.to[v] = to;
  }
}

// Best move of v by one warp: up to 256 entries loaded together, their labels
// gathered together, then folded in CSR order into the warp's table.
__device__ __forceinline__ void gm_eval(const GangMoveArgs& A, WarpTabs& W, MoveRound& R, u32 v,
                                        double shift, unsigned long long& trav) {
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  u32* tk = W.tk[wib];
  u32* tp = W.tp[wib];
  double* tv = W.tv[wib];
  double* sw = W.sw[wib];
  const u64 o0 = A.off[v];
  const u32 deg = (u32)(A.off[v + 1] - o0);
  const u32 cur = A.f[v];
  const double kv = A.k[v];
  const double dcur = A.d[cur];
  if (lane == 0) trav += deg;
  u32 cap = 64;
  while (cap < 2 * deg) cap <<= 1;
  const u32 mask = cap - 1;
  u32 key[GM_MAXDEG / 32];
#pragma unroll
  for (u32 j = 0; j < GM_MAXDEG / 32; ++j) {
    key[j] = NONE32;
    if (j * 32 >= deg) continue;
    const u32 q = j * 32 + lane;
    if (q < deg) {
      key[j] = A.col[o0 + q];
      sw[q] = A.w[o0 + q];
    }
  }
  for (u32 x = lane; x < cap; x += 32) tk[x] = NONE32;
#pragma unroll
  for (u32 j = 0; j < GM_MAXDEG / 32; ++j)  // self-loops skipped (parallel_frontier.rs:164-166)
    if (key[j] != NONE32) key[j] = key[j] == v ? NONE32 : A.f[key[j]];
  __syncwarp();
#pragma unroll
  for (u32 j = 0; j < GM_MAXDEG / 32; ++j) {
    if (j * 32 >= deg) break;  // warp-uniform
    const u32 grp = __match_any_sync(0xffffffffu, key[j]);
    if (key[j] != NONE32 && lane == (u32)(__ffs(grp) - 1)) {
      u32 slot = hub_hash(key[j]) & mask;
      while (true) {  // the table holds at most deg < cap keys
        const u32 prev = atomicCAS(&tk[slot], NONE32, key[j]);
        if (prev == NONE32 || prev == key[j]) {
          double sum = prev == NONE32 ? 0.0 : tv[slot];
          for (u32 m = grp; m; m &= m - 1) sum = __dadd_rn(sum, sw[j * 32 + __ffs(m) - 1]);
          tv[slot] = sum;
          if (prev == NONE32) tp[slot] = j * 32 + lane;
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
    GainScreen scr;  // exact gains only for candidates that may win
    scr.init(wcur, A.tw, A.gamma, kv, dcur);
    for (u32 x0 = lane; x0 < cap; x0 += 128) {
      u32 kq[4];
      double dk[4];
#pragma unroll
      for (u32 j = 0; j < 4; ++j) {
        kq[j] = x0 + 32 * j < cap ? tk[x0 + 32 * j] : NONE32;
        if (kq[j] == cur) kq[j] = NONE32;
      }
#pragma unroll
      for (u32 j = 0; j < 4; ++j) dk[j] = kq[j] != NONE32 ? A.d[kq[j]] : 0.0;
#pragma unroll
      for (u32 j = 0; j < 4; ++j) {
        const u32 x = x0 + 32 * j;
        if (kq[j] == NONE32 || !scr.keep(tv[x], dk[j])) continue;
        const double gn = move_gain(tv[x], wcur, A.tw, A.gamma, kv, dcur, dk[j]);
        const u32 pp = tp[x];
        if (p == NONE32 || gn > g || (gn == g && pp < p)) {
          g = gn;
          p = pp;
          kk = kq[j];
        }
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
  if (lane == 0)
    gm_finish(A, R, v, cur, kv, wcur, dcur, g, p, kk, deg > PRUNE_MIN_DEG, shift);
  __syncwarp();
}

// What bounds it: the chain of its steps (barriers and dependent L2 accesses);
// with many active rows, the gathers of their neighbours' labels.  Against the
// multi-kernel rounds and the one-block rounds it replaces, the stage of one
// level: 5 levels of 250-400 nodes 88 -> 23 us, 3 levels of 7-10k nodes
// 415 -> 79 us, 10 levels of 10-50k nodes 410 -> 54 us, one level of 100k nodes
// 570 -> 210 us, 10 levels of 0.13-1M nodes with f64 weights 750 -> 440 us (events
// around the launch).
__global__ void __launch_bounds__(GANG_THREADS, 1) k_gang_move(GangMoveArgs A) {
  extern __shared__ __align__(16) unsigned char gm_raw[];
  MoveSmem& M = *reinterpret_cast<MoveSmem*>(gm_raw);
  __shared__ GangSmem S;
  __shared__ u32 s_next;
  const Gang G = gang_make(A.grid);
  const u32 tid = threadIdx.x, lane = tid & 31;
  const u32 gt = G.thread(), gts = G.threads();
  MoveCnt& C = *A.cnt;
  gang_clear_next(G, A.cnt_next);
  const u32 words = (A.n + 31) / 32;
  unsigned long long trav = 0, trav_round = 0, pruned = 0;
  u32 b = 0;  // parity of the current frontier
  // ---- clear; the largest label ----
  for (u32 i = gt; i < words; i += gts) A.bits[0][i] = A.bits[1][i] = 0;
  if (A.setup) {
    u32 mx = 0;
    for (u32 i = gt; i < (A.n + 3) / 4; i += gts) {
      reinterpret_cast<u32*>(A.changed)[i] = 0;
      reinterpret_cast<u32*>(A.affected)[i] = 0;
    }
    for (u32 v = gt; v < A.n; v += gts) mx = max(mx, A.f[v]);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && mx) atomicMax(&C.maxlab, mx);
    for (u64 c = gt; c < A.dcap; c += gts) A.d[c] = 0.0;
    if (A.prune.b) {
      for (u32 i = gt; i < words; i += gts) A.prune.valid[i] = 0;
      for (u64 c = gt; c < A.dcap; c += gts) A.prune.drop[c] = 0.0;
      if (gt == 0) {
        *A.prune.shift = 0.0;
        *A.prune.worst = 0;
      }
    }
  }
  G.sync();
  if (A.setup) {
    if (C.maxlab >= A.n) {  // ids must stay below n: n + v is v's empty community
      if (gt == 0) A.out->status = MOVE_LABELS;
      return;
    }
    // ---- seeding (hit_leiden.rs:1037-1057) ----
    for (u32 i = gt; i < A.dk; i += gts) {
      const u32 x = A.du[i], y = A.dv[i];
      const double al = A.dw ? A.dw[i] : 1.0;
      const bool same_f = A.f[x] == A.f[y];
      if ((al > 0.0 && !same_f) || (al < 0.0 && same_f)) {
        gm_activate(A, 0, x);
        gm_activate(A, 0, y);
      }
      if (A.s[x] == A.s[y]) {
        A.affected[x] = 1;
        A.affected[y] = 1;
      }
    }
    if (A.kflag)
      for (u32 v = gt; v < A.n; v += gts)
        if (A.kflag[v]) A.affected[v] = 1;
    if (A.all_active)
      for (u32 v = gt; v < A.n; v += gts) gm_activate(A, 0, v);
    // ---- community degrees (hit_leiden.rs:1060-1066) ----
    if (A.integral) {
      for (u32 v0 = gt - lane; v0 < A.n; v0 += gts) {
        const u32 v = v0 + lane;
        const bool on = v < A.n;
        warp_add_by_id(A.d, on ? A.f[v] : 0, on ? A.k[v] : 0.0, on);
      }
    } else {
      bool second;
      gang_label_sort(G, S, A.n, A.label_bits, [&](u32 i) { return A.f[i]; }, A.lab, A.idx,
                      A.lab2, A.idx2, A.hist, A.part, &second);
      const u32* lab = second ? A.lab2 : A.lab;
      const u32* idx = second ? A.idx2 : A.idx;
      for (u32 t = gt; t < A.n; t += gts) A.kval[t] = A.k[idx[t]];
      G.sync();
      gang_segment_sums(G, A.n, lab, A.kval, M.w.sw[tid >> 5],
                        [&](u32 c, double x) { A.d[c] = x; });
    }
    G.sync();
  } else {
    for (u32 v = gt; v < A.n; v += gts)
      if (A.active[v]) gm_activate(A, 0, v);
    G.sync();
  }
  u32 it = A.it0, round = A.round0;
  u64 epoch = A.epoch0;
  u32 status = MOVE_DONE;
  u32 m_last = 0;  // candidates of the round before
  while (true) {
    MoveRound& R = C.r[b];
    const u32 nv = R.nv, nh = R.nh;
    double shift = 0.0;
    if (A.prune.b) {
      shift = *A.prune.shift + prune_worst_now(A.prune);
      for (u32 r = gt; r < m_last; r += gts)
        if (A.status[r] == GM_ACCEPTED) A.prune.drop[A.sel_from[r]] = 0.0;
      m_last = 0;
    }
    if (it >= A.max_rounds || nv + nh == 0) {
      if (A.more && nv + nh) status = MOVE_BIG_FRONTIER;
      break;
    }
    if (nv > A.max_frontier || nh > A.max_frontier || nv + nh > A.max_frontier) {
      status = MOVE_BIG_FRONTIER;
      break;
    }
    // ---- best moves on the snapshot: hubs by block, the rest by warp ----
    if (gt == 0) {
      MoveRound& N = C.r[b ^ 1];
      N.nv = N.nh = N.ncand = N.nops = N.nitems = N.work = N.hwork = N.big = N.wv = N.wh = 0;
      N.huge = N.whuge = 0;
    }
    const u32 *verts = A.verts[b], *hubs = A.hubs[b];
    u32 ev = nv, eh = nh;  // vertices to evaluate
    unsigned long long pruned_round = 0;
    // a row too long for the tables hands the round back before any evaluation,
    // unless its bound rules it out
    bool huge = R.huge != 0;
    if (A.prune.b && it > 0) {
      // rows of earlier rounds hold bounds: most need no evaluation
      for (u32 i = gt; i < nv + nh; i += gts) {
        const bool hub = i >= nv;
        const u32 v = hub ? hubs[i - nv] : verts[i];
        if (prune_valid(A.prune, v) &&
            prune_rules_out(A.prune, shift, v, A.k[v], A.d[A.f[v]], A.tw, A.gamma)) {
          pruned_round += A.off[v + 1] - A.off[v];
        } else if (hub) {
          if (A.off[v + 1] - A.off[v] > HUB_MAXDEG) R.whuge = 1;
          A.whubs[atomicAdd(&R.wh, 1u)] = v;
        } else {
          A.wverts[atomicAdd(&R.wv, 1u)] = v;
        }
      }
      G.sync();
      ev = R.wv;
      eh = R.wh;
      verts = A.wverts;
      hubs = A.whubs;
      huge = R.whuge != 0;
    }
    if (huge) {
      status = MOVE_BIG_HUB;
      break;
    }
    if (eh) {
      for (;;) {
        __syncthreads();
        if (tid == 0) s_next = atomicAdd(&R.hwork, 1u);
        __syncthreads();
        const u32 i = s_next;
        if (i >= eh) break;
        const u32 v = hubs[i];
        const u64 o0 = A.off[v], o1 = A.off[v + 1];
        const u32 cur = A.f[v];
        if (!hub_sums<GANG_WARPS>(
                M.h, o0, o1, A.col, A.w, A.integral,
                [&](u32 nb) { return nb == v ? NONE32 : A.f[nb]; },
                A.gslot + (size_t)G.rank * HUB_MAXDEG,
                A.gw ? A.gw + (size_t)G.rank * HUB_MAXDEG : nullptr)) {
          if (tid == 0) gm_big(R);
          continue;
        }
        const double kv = A.k[v], dcur = A.d[cur];
        double g;
        u32 p, kk;
        hub_best<GANG_WARPS>(M.h, cur, A.tw, A.gamma, kv, dcur, [&](u32 c) { return A.d[c]; }, g,
                             p, kk);
        if (tid == 0) {
          trav_round += o1 - o0;
          gm_finish(A, R, v, cur, kv, M.h.wcur, dcur, g, p, kk, true, shift);
        }
      }
      __syncthreads();
    }
    for (u32 i = G.warp(); i < ev;) {
      gm_eval(A, M.w, R, verts[i], shift, trav_round);
      if (lane == 0) i = G.warps() + atomicAdd(&R.work, 1u);
      i = __shfl_sync(0xffffffffu, i, 0);
    }
    G.sync();
    if (R.big) {
      status = MOVE_BIG_HUB;
      break;
    }
    trav += trav_round;
    pruned += pruned_round;
    trav_round = 0;
    const u32 m = R.ncand;
    ++it;
    if (gt == 0) {
      C.cands += m;
      C.nfront += ev + eh;
    }
    if (m == 0) {
      b ^= 1;  // nothing selected: the next frontier is empty
      break;
    }
    // ---- candidates by (gain desc, node asc) ----
    ++round;
    gang_sort(
        G, S, m, [&](u32 i) { return A.ckey[i]; }, [&](u32 i) { return A.cnode[i]; }, A.skey,
        A.sval, [&](u32 r, u64, u32 v) {
          A.sel_node[r] = v;
          A.sel_from[r] = A.f[v];
          A.sel_to[r] = A.to[v];
          A.status[r] = GM_UNDECIDED;
        });
    // ---- decoupled selection (throughput.rs:204-236) by reservations ----
    for (u32 iter = 0;; ++iter) {
      ++epoch;
      if (gt == 0) C.und[iter & 1] = 0;
      for (u32 r = gt; r < m; r += gts) {
        if (A.status[r] != GM_UNDECIDED) continue;
        const u32 x = A.sel_from[r], y = A.sel_to[r];
        const u32 bx = gm_role(A.role[x], round), by = gm_role(A.role[y], round);
        if ((bx & GM_ACC) || (by & GM_EMIT)) {
          A.status[r] = GM_REJECTED;
          continue;
        }
        const unsigned long long key = (epoch << 32) | (0xFFFFFFFFu - r);
        u8 mk = 0;
        if (bx == 0) {
          mk |= 1;
          atomicMax(&A.res[x], key);
        }
        if (by == 0) {
          mk |= 2;
          atomicMax(&A.res[y], key);
        }
        A.nmask[r] = mk;
      }
      G.sync();
      u32 left = 0;
      for (u32 r = gt; r < m; r += gts) {
        if (A.status[r] != GM_UNDECIDED) continue;
        const u32 x = A.sel_from[r], y = A.sel_to[r];
        const u8 mk = A.nmask[r];
        const unsigned long long key = (epoch << 32) | (0xFFFFFFFFu - r);
        if (((mk & 1) && A.res[x] != key) || ((mk & 2) && A.res[y] != key)) {
          ++left;
          continue;
        }
        A.status[r] = GM_ACCEPTED;
        if (x == y) {
          A.role[x] = (round << 2) | GM_EMIT | GM_ACC;
        } else {
          A.role[x] = (round << 2) | GM_EMIT;
          A.role[y] = (round << 2) | GM_ACC;
        }
      }
      if (left) atomicAdd(&C.und[iter & 1], left);
      G.sync();
      if (!C.und[iter & 1]) break;
      if (iter + 1 >= GM_MAX_SELECT) {
        // every earlier-ranked candidate is final: the greedy rule in rank order
        if (gt == 0)
          for (u32 r = 0; r < m; ++r) {
            if (A.status[r] != GM_UNDECIDED) continue;
            const u32 x = A.sel_from[r], y = A.sel_to[r];
            const u32 bx = gm_role(A.role[x], round), by = gm_role(A.role[y], round);
            if ((bx & GM_ACC) || (by & GM_EMIT)) {
              A.status[r] = GM_REJECTED;
              continue;
            }
            A.status[r] = GM_ACCEPTED;
            A.role[x] = (round << 2) | bx | GM_EMIT;
            A.role[y] = (round << 2) | gm_role(A.role[y], round) | GM_ACC;
          }
        G.sync();
        break;
      }
    }
    // ---- the accepted moves (throughput.rs:182-187) ----
    if (gt == 0 && A.prune.b) {
      *A.prune.shift = shift;
      *A.prune.worst = 0;
    }
    m_last = m;
    for (u32 r = gt; r < m; r += gts) {
      if (A.status[r] != GM_ACCEPTED) continue;
      const u32 v = A.sel_node[r], from = A.sel_from[r], to = A.sel_to[r];
      prune_moved(A.prune, v, from, A.k[v]);
      A.f[v] = to;
      A.changed[v] = 1;
      if (A.mark_moved) A.affected[v] = 1;
      const u32 at = atomicAdd(&R.nops, 2u);
      if (A.integral) {
        const double kv = A.k[v];
        atomicAdd(&A.d[from], -kv);
        atomicAdd(&A.d[to], kv);
      } else {
        A.okey[at] = ((u64)from << 32) | (2 * r);
        A.okey[at + 1] = ((u64)to << 32) | (2 * r + 1);
      }
      const u64 deg = A.off[v + 1] - A.off[v];
      const u32 ns = deg ? (u32)((deg + GM_SLICE - 1) / GM_SLICE) : 0u;
      if (ns) {
        const u32 i0 = atomicAdd(&R.nitems, ns);
        for (u32 x = 0; x < ns; ++x)
          if (i0 + x < A.items_cap) A.items[i0 + x] = ((u64)r << 32) | x;
      }
    }
    for (u32 i = gt; i < nv; i += gts) A.bits[b][A.verts[b][i] >> 5] = 0;
    for (u32 i = gt; i < nh; i += gts) A.bits[b][A.hubs[b][i] >> 5] = 0;
    G.sync();
    const u32 nops = R.nops;
    if (gt == 0) C.moves += nops / 2;
    if (!A.integral && nops) {
      // d(C) -= k / += k in selected order, per community: an ordered sum that
      // starts from d(C) (a community that gains or loses thousands of vertices
      // in a round is one long chain)
      gang_sort(
          G, S, nops, [&](u32 i) { return A.okey[i]; }, [](u32 i) { return i; }, A.otmp, A.otv,
          [&](u32 r, u64 key, u32) {
            const u32 op = (u32)key;
            const double kv = A.k[A.sel_node[op >> 1]];
            A.okey2[r] = key >> 32;
            A.oterm[r] = (op & 1) ? kv : -kv;
          });
      gang_segment_sums(
          G, nops, A.okey2, A.oterm, M.w.sw[tid >> 5], [&](u64 c, double x) { A.d[c] = x; },
          [&](u64 c) { return A.d[c]; });
    }
    // ---- the next frontier and K (throughput.rs:189-199), after all moves ----
    const u32 nitems = min(R.nitems, A.items_cap);
    for (u32 i = G.warp(); i < nitems; i += G.warps()) {
      const u64 item = A.items[i];
      const u32 v = A.sel_node[(u32)(item >> 32)], to = A.sel_to[(u32)(item >> 32)];
      const u32 from = A.sel_from[(u32)(item >> 32)];
      if (lane == 0 && (u32)item == 0) prune_worst(A.prune, from);
      const u64 lo = A.off[v] + (u64)(u32)item * GM_SLICE;
      const u64 hi = min(A.off[v + 1], lo + GM_SLICE);
      const u32 sv = A.s[v];
      bool any = false;
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
          if (nb[j] == NONE32) continue;
          if (fn[j] != to) {
            gm_activate(A, b ^ 1, nb[j]);
            if (prune_valid(A.prune, nb[j]))
              prune_raise(A.prune, nb[j], fn[j], from, A.w[p0 + 32 * j]);
          }
          if (sn[j] == sv) {
            A.affected[nb[j]] = 1;
            any = true;
          }
        }
      }
      if (__any_sync(0xffffffffu, any) && lane == 0) A.affected[v] = 1;
    }
    b ^= 1;
    G.sync();
  }
  for (int o = 16; o; o >>= 1) trav += __shfl_xor_sync(0xffffffffu, trav, o);
  for (int o = 16; o; o >>= 1) pruned += __shfl_xor_sync(0xffffffffu, pruned, o);
  if (lane == 0 && trav) atomicAdd(&C.trav, trav);
  if (lane == 0 && pruned) atomicAdd(&C.pruned, pruned);
  if (status != MOVE_DONE)  // the frontier for the host's rounds
    for (u32 v = gt; v < A.n; v += gts) A.active[v] = (A.bits[b][v >> 5] >> (v & 31)) & 1u;
  G.sync();
  if (gt == 0) {
    if (A.prune.b) {  // for the host's rounds
      *A.prune.shift += prune_worst_now(A.prune);
      *A.prune.worst = 0;
    }
    A.out->status = status;
    A.out->frontier = C.r[b].nv + C.r[b].nh;
    A.out->it = it;
    A.out->round = round;
    A.out->epoch = epoch;
    A.out->moves = C.moves;
    A.out->cands = C.cands;
    A.out->trav = C.trav;
    A.out->nfront = C.nfront;
    A.out->pruned = C.pruned;
  }
}

static std::atomic<bool> g_move_attr[64];

bool gang_move_fits(Engine& E, const Level& L) {
  return !E.lean && L.g.n > 0 &&
         (E.cfg.mode == HL_MODE_DETERMINISTIC || !(E.cfg.flags & HL_FLAG_NO_SMALL_ROUNDS));
}

// Movement rounds from the seeds (`setup`) or from the frontier in S.active.  In
// deterministic mode the setup alone: the active set is left in S.gm_bits.
// Returns MOVE_DONE, or why the host's rounds continue from S.active
// (MOVE_LABELS: the labels need compaction first; nothing else has happened).
u32 gang_move(Engine& E, Level& L, const DevEdges& delta, bool setup, bool all_active,
              bool mark_moved, u32 frontier, u32& it, GangMoveStats& ms) {
  Scratch& S = E.sc;
  const u32 n = L.g.n;
  const int dev = E.device;
  if (dev >= 0 && dev < 64 && !g_move_attr[dev]) {
    HL_CUDA(cudaFuncSetAttribute(k_gang_move, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(MoveSmem)));
    g_move_attr[dev] = true;
  }
  const u64 avg = L.g.nnz / n + 1;
  const GangShape shape = gang_shape(E, n + 4ull * std::min(n, frontier) * avg);
  const size_t nflag = (((size_t)n + 3) & ~(size_t)3);
  const size_t ncap = 2 * (size_t)n + 2;
  const u32 fr = std::min(n, GM_FRONTIER);
  S.active.ensure(E.mem, nflag);
  S.next.ensure(E.mem, nflag);
  S.changed.ensure(E.mem, nflag);
  S.affected.ensure(E.mem, nflag);
  ensure_comm_arrays(E, ncap);
  S.gm_bits.ensure(E.mem, 2 * (((size_t)n + 31) / 32));
  S.sm_list_a.ensure(E.mem, 4 * (size_t)fr);
  S.sm_list_b.ensure(E.mem, 2 * (size_t)fr);
  S.cand_to.ensure(E.mem, n);
  S.gkey.ensure(E.mem, fr);
  S.gkey2.ensure(E.mem, fr);
  S.cand_node.ensure(E.mem, fr);
  S.cand_idx.ensure(E.mem, fr);
  S.sel_node.ensure(E.mem, fr);
  S.sel_from.ensure(E.mem, fr);
  S.sel_to.ensure(E.mem, fr);
  S.status.ensure(E.mem, fr);
  S.nmask.ensure(E.mem, fr);
  const u64 items_cap = (u64)fr + L.g.nnz / GM_SLICE + 1;
  S.gr_items.ensure(E.mem, items_cap);
  GangMoveArgs A{};
  if (!E.integral) {
    S.keys.ensure(E.mem, 2 * (size_t)fr);
    S.keys2.ensure(E.mem, 2 * (size_t)fr);
    S.rkeys.ensure(E.mem, 2 * (size_t)fr);
    S.idx.ensure(E.mem, 2 * (size_t)fr);
    A.okey = S.keys.p;
    A.okey2 = S.keys2.p;
    A.otmp = S.rkeys.p;
    A.otv = S.idx.p;
    S.fvals.ensure(E.mem, std::max<size_t>(n, 2 * (size_t)fr));
    A.oterm = S.fvals.p;
    if (setup) {
      S.used.ensure(E.mem, n);
      S.rank.ensure(E.mem, n);
      S.order.ensure(E.mem, n);
      S.order2.ensure(E.mem, n);
      S.gm_hist.ensure(E.mem, (size_t)256 * GANG_WARPS * shape.blocks);
      A.lab = S.used.p;
      A.lab2 = S.rank.p;
      A.idx = S.order.p;
      A.idx2 = S.order2.p;
      A.hist = S.gm_hist.p;
      A.kval = S.fvals.p;  // before any round
    }
  }
  if (L.g.nnz > GM_MAXDEG) {  // a row may be a hub
    S.gm_slot.ensure(E.mem, (size_t)HUB_MAXDEG * shape.blocks);
    A.gslot = S.gm_slot.p;
    if (!E.integral) {
      S.gm_w.ensure(E.mem, (size_t)HUB_MAXDEG * shape.blocks);
      A.gw = S.gm_w.p;
    }
  }
  S.gang_part.ensure(E.mem, GANG_MAX_BLOCKS);
  static_assert(sizeof(MoveCnt) <= GANG_CNT * sizeof(u32), "fits the counter block");
  static_assert(sizeof(MoveOutDev) <= 64 * sizeof(u64), "fits the pinned block");
  selection_room(E);
  const u32 max_rounds =
      E.cfg.mode == HL_MODE_DETERMINISTIC ? 0 : E.cfg.max_rounds ? E.cfg.max_rounds : 20;
  A.n = n;
  A.off = L.g.off.p;
  A.col = L.g.col.p;
  A.w = L.g.w.p;
  A.f = L.f.p;
  A.s = L.s_cur.p;
  A.k = L.k.p;
  A.d = S.d.p;
  A.dcap = ncap;
  A.active = S.active.p;
  A.changed = S.changed.p;
  A.affected = S.affected.p;
  A.kflag = E.k_flags_set ? S.kflag.p : nullptr;
  A.du = delta.u;
  A.dv = delta.v;
  A.dw = delta.w;
  A.dk = setup ? (u32)delta.k : 0;
  A.setup = setup;
  A.all_active = all_active;
  A.mark_moved = mark_moved;
  A.integral = E.integral;
  A.grid = shape.grid;
  A.tw = L.tw;
  A.gamma = E.cfg.resolution;
  A.bits[0] = S.gm_bits.p;
  A.bits[1] = S.gm_bits.p + ((size_t)n + 31) / 32;
  A.verts[0] = S.sm_list_a.p;
  A.verts[1] = S.sm_list_b.p;
  A.hubs[0] = S.sm_list_a.p + fr;
  A.hubs[1] = S.sm_list_b.p + fr;
  A.wverts = S.sm_list_a.p + 2 * (size_t)fr;
  A.whubs = S.sm_list_a.p + 3 * (size_t)fr;
  A.list_cap = fr;
  // A launch whose blocks were chosen for a few vertices must not go on when the
  // frontier has grown to what the whole GPU should evaluate (20k vertices with
  // 320k entries, 40-2,000 updates that wake them all: 13-14.5 ms on 8 blocks,
  // 3.0-3.8 with the hand-over, 8.3-10.3 by multi-kernel rounds).  A cluster may
  // take twice the work it was chosen for; one block 32 times, because a
  // hand-over costs 30 us (8 times: 2,000 updates of 3,000 vertices 4.0 -> 4.3 ms).
  A.max_frontier = fr;
  if (!shape.grid) {
    const u64 work = shape.blocks > 1 ? 2 * gang_cluster_work(E) : 32 * GANG_BLOCK_WORK;
    const u64 most = work > n ? (work - n) / (4 * avg) : 0;
    A.max_frontier = (u32)std::min<u64>(fr, std::max<u64>(most, 64));
  }
  A.prune = E.prune;
  A.to = S.cand_to.p;
  A.ckey = S.gkey.p;
  A.cnode = S.cand_node.p;
  A.skey = S.gkey2.p;
  A.sval = S.cand_idx.p;
  A.sel_node = S.sel_node.p;
  A.sel_from = S.sel_from.p;
  A.sel_to = S.sel_to.p;
  A.status = S.status.p;
  A.nmask = S.nmask.p;
  A.role = S.role.p;
  A.res = reinterpret_cast<unsigned long long*>(S.res.p);
  A.items = S.gr_items.p;
  A.items_cap = (u32)std::min<u64>(items_cap, 0xFFFFFFFFull);
  A.part = S.gang_part.p;
  A.it0 = it;
  A.more = max_rounds > it && max_rounds - it > SEL_ROUNDS;
  A.max_rounds = A.more ? it + SEL_ROUNDS : max_rounds;
  A.round0 = E.sel_round;
  A.epoch0 = E.epoch;
  A.label_bits = (u32)bits_for(n - 1);
  A.cnt = reinterpret_cast<MoveCnt*>(gang_counters(E, &A.cnt_next));
  A.out = reinterpret_cast<MoveOutDev*>(E.hs.p);
  cudaEvent_t ev = E.kt_begin();
  gang_launch(E, reinterpret_cast<const void*>(&k_gang_move), shape, sizeof(MoveSmem), &A);
  gang_turn(E);
  E.kt_end(KT_GANG_MOVE, ev);
  MoveOutDev o;
  E.sync();
  std::memcpy(&o, E.hs.p, sizeof(o));
  if (o.status == MOVE_LABELS) return o.status;
  if (setup) E.k_flags_set = false;
  it = o.it;
  ms.frontier = o.frontier;
  ms.moves += o.moves;
  ms.cands += o.cands;
  ms.trav += o.trav + o.pruned;  // rows ruled out count as traversed
  E.sel_round = o.round;
  E.epoch = o.epoch;
  E.kagg[KT_GANG_MOVE].bytes += 52ull * o.nfront + 16ull * o.trav + 8ull * o.cands;
  E.kagg[KT_GANG_MOVE].items += o.nfront;
  return o.status;
}

}  // namespace hl
