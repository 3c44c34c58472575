// hl_engine.cuh — device state of one graph handle and the stage entry points.
#pragma once
#include <atomic>
#include <initializer_list>
#include <cub/cub.cuh>

#include "hl_internal.cuh"

namespace hl {

// Undirected weighted CSR on the device: both directions stored, rows sorted
// by neighbour id, a self-loop stored twice in its row (in_memory.rs:20-72).
struct DevGraph {
  u32 n = 0;
  u64 nnz = 0;
  u64 self_loop_entries = 0;
  DBuf<u64> off;  // n+1
  DBuf<u32> col;
  DBuf<double> w;
  DBuf<u32> col2;  // the other half of the double buffer used by apply_delta
  DBuf<double> w2;
};

// One hierarchy level (state.rs:19-32): supergraph G^p and its maps.
struct Level {
  DevGraph g;
  DBuf<u32> f;      // community_mapping_per_level[p]
  DBuf<u32> gm;     // refined_community_mapping_per_level[p]
  DBuf<u32> s_pre;  // previous_subcommunity_mapping_per_level[p]
  DBuf<u32> s_cur;  // current_subcommunity_mapping_per_level[p]
  DBuf<double> k;   // weighted degree of each level-p node
  double tw = 0.0;  // 2m of G^p
  u32 s_bound = 0;  // every id in s_pre and s_cur is below this (0: not known)
};

// An edge list on the device (GraphInput): w == nullptr means weight 1.0.
struct DevEdges {
  const u32* u = nullptr;
  const u32* v = nullptr;
  const double* w = nullptr;
  u64 k = 0;
};

// Scratch reused by every stage; grown on demand, never shrunk.
struct Scratch {
  DBuf<u8> cub_tmp;
  // edge-list staging (host batches, aggregation output)
  DBuf<u32> eu, ev, eu2, ev2;
  DBuf<double> ew, ew2;
  // delta application
  DBuf<u64> keys, keys2, rkeys, rkeys2;
  DBuf<u32> idx, idx2, segid, seg_start, rvals, rvals2;
  DBuf<u8> op, ktouched;
  DBuf<double> neww;
  DBuf<u32> nops_del, nops_ins, pos_del, pos_ins;
  DBuf<u32> opdel, opdelpre;  // apply_delta: delete flags of the sorted operations, their scan
  DBuf<u64> newoff;
  DBuf<u32> rowlist;
  // node flags (level size)
  DBuf<u8> active, next, changed, affected, refined;
  DBuf<u32> act, cand_idx, cnt;
  DBuf<u32> cand_to, cand_node;
  DBuf<double> cand_gain;
  DBuf<u64> gkey, gkey2;
  DBuf<u32> sel_from, sel_to, sel_node, order, order2;
  DBuf<u8> status, nmask;
  DBuf<u32> role;
  DBuf<u64> res;
  DBuf<double> d;       // community degrees (2n)
  DBuf<u32> used, rank;
  // refinement
  DBuf<u32> par, uroot, csize, newid, minmem;
  DBuf<u64> keep;
  DBuf<u8> affsc, cand_sc, blocked;
  DBuf<u32> sizes;
  DBuf<double> dS, wsp, dcomm;
  DBuf<u64> wcnt;       // T-filter: terms of each any-order sum
  DBuf<u8> amb;         // T-filter: S whose decision needs the ordered sum
  DBuf<u32> longrows;   // T-filter: member rows summed by a whole block
  // reductions
  DBuf<double> red, red2;
  DBuf<u64> red64;
  DBuf<u32> origin;
  // global tables of the block-per-vertex kernel's second pass (rows with
  // more than 2048 distinct keys)
  DBuf<u32> huge_key, huge_pos, huge_list;
  DBuf<u32> ovf, ovf_cnt;  // block kernel: rows deferred to the pass with global regions
  DBuf<u32> acc_cnt;       // inc-movement: accepted moves over all rounds
  DBuf<u32> hubk, hubk2, hubv;  // block bin ordered by degree (keys, sorted keys, list)
  DBuf<u32> longseg, longcnt;   // long rows or segments, summed apart, and their count
  DBuf<double> fvals;           // ordered sums: the terms gathered into sum order
  DBuf<double> huge_val;
  // deterministic mode (det.cu)
  DBuf<u32> det_bits, det_bp, det_keys, det_rsort, det_mkey, det_mkey2, det_mval, det_members,
      det_mstart, det_mcount, det_xhead, det_xnext;
  DBuf<double> det_bw, det_wsp;
  DBuf<u64> det_out, det_k64, det_k64b;
  DBuf<u8> det_wvalid;
  // partitioned second pass of the block kernel (integral weights)
  DBuf<u32> pb_nb, pb_nc, pb_bbase, pb_cbase, pb_rowfail, pb_fail, pb_failcnt, pb_ktmp, pb_ekey,
      pb_epos, pb_bcnt, pb_boff, pb_bp, pb_bk;
  DBuf<u64> pb_ne, pb_ebase, pb_ro0;
  DBuf<double> pb_wcur, pb_ew, pb_bg, pb_rkv, pb_rdcur;
  DBuf<u32> pb_brow, pb_crow, pb_rv, pb_rfv, pb_rcur;  // bucket / chunk -> row; row scalars
  DBuf<u32> pb_okey, pb_okey2, pb_oval, pb_ord, pb_fwork;  // fold order (largest bucket first)
  DBuf<unsigned long long> mark_long;  // (rank << 32 | segment) of long moved rows
  DBuf<u32> mark_long_cnt;
  // batch statistics accumulated on the device and read once at the end of
  // the call: [0..7] traversed / candidates of the four evaluation bins,
  // [8] accepted moves, [9] refinement merges, [10] |B^1|, [11] entries of
  // vertices whose bound ruled a move out
  DBuf<u64> bacc;
  DBuf<u8> kflag;     // K marks for the next level (M8), level-size bytes
  // movement bounds (prune.cuh)
  DBuf<double> pr_b, pr_shift, pr_drop;
  DBuf<u32> pr_valid;
  // movement in one launch (gang_move.cu): frontier lists
  DBuf<u32> sm_list_a, sm_list_b;
  // per-level output: the level's s_cur before the batch, the changed nodes
  DBuf<u32> lvl_prev, lvl_nodes, lvl_ids;
  DBuf<u8> lvl_flag;
  // single-launch stages (gang.cuh)
  DBuf<u32> canon;  // the canonical partition before it is copied out
  DBuf<u32> gang_part, gang_cnt, ga_touched, gr_bits, gm_bits, gm_hist;
  DBuf<unsigned short> gm_slot;
  DBuf<double> gm_w;
  DBuf<u64> gr_items;
};

// Per-kernel device timing (CUDA events on the engine's stream), enabled by
// HL_FLAG_KERNEL_TIMING; bytes are the algorithmic bytes the stage moved.
struct KernelAgg {
  u64 launches = 0;
  double ms = 0.0;
  u64 bytes = 0;
  u64 items = 0;  // vertices / records processed, where meaningful
};
enum KernelId : int {
  KT_MOVE_EVAL = 0,
  KT_REFINE_EVAL,
  KT_SELECT,
  KT_MERGE_ROWS,
  KT_AGGREGATE,
  KT_EVAL_SMALL,   // sub-warp bins (both evaluation kinds)
  KT_EVAL_MID,     // warp-per-vertex bin
  KT_EVAL_BIG,     // warp-per-vertex wide bin (129..512)
  KT_EVAL_HUGE,    // block-per-vertex bin (> 512), both passes
  KT_COMM_DEG,     // per-community / per-sub-community degree sums
  KT_MARK_NEXT,    // accepted-move application and frontier marking
  KT_REFINE_CC,    // connected components of affected sub-communities
  KT_TFILTER,      // T-filter sums and decisions
  KT_ROW_SUMS,     // vertex degrees of touched rows
  KT_DELTA_SORT,   // batch key sort and resolution in apply_delta
  KT_STAGE_APPLY,  // whole stages of the level loop (including host waits)
  KT_STAGE_MOVE,
  KT_STAGE_REFINE,
  KT_STAGE_AGGREGATE,
  KT_HOST_SYNC,    // host waits on the stream (launches = count; no time)
  KT_GANG_APPLY,   // whole delta applications in one launch (gang_apply.cu)
  KT_GANG_MOVE,    // movement rounds of small frontiers in one launch (gang_move.cu)
  KT_EVAL_PB,      // the partitioned pass of the block bin (inside KT_EVAL_HUGE)
  KT_GANG_REFINE,  // whole refinements in one launch (gang_refine.cu)
  KT_GANG_AGG,     // whole aggregations in one launch (gang_aggregate.cu)
  KT_COUNT
};

// Bounds that rule a move out without reading the row (prune.cuh): from one
// movement's start to its end.
struct Prune {
  double* b = nullptr;    // per vertex, where `valid` is set
  u32* valid = nullptr;   // bit per vertex
  double* shift = nullptr;// S: how far any community's degree may have fallen
  double* drop = nullptr; // per community: degree leaving it in this round
  unsigned long long* worst = nullptr;  // bits of the largest of them, not yet in S
};

struct Engine {
  // the staging block and the buffers go back with nothing in flight
  ~Engine() {
    if (side) cudaStreamSynchronize(side);
    if (stream) cudaStreamSynchronize(stream);
    if (side_go) cudaEventDestroy(side_go);
    if (side_done) cudaEventDestroy(side_done);
    if (side) cudaStreamDestroy(side);
  }
  hl_config cfg{};
  int device = 0;
  cudaStream_t stream = nullptr;
  // A second stream for launches that need nothing from the engine's current
  // ones (created by the first large frontier that has both kinds of rows):
  // side_begin lets it start where the engine's stream is now, side_end makes
  // the engine's stream wait for all of it, before anything reads or frees what
  // it uses.
  cudaStream_t side = nullptr;
  cudaEvent_t side_go = nullptr, side_done = nullptr;
  void side_begin();
  cudaError_t side_end();
  MemCtx mem;
  Scratch sc;
  std::vector<Level> levels;
  bool multilevel = false;
  bool integral = true;  // every weight integral: all FP64 sums exact in any order
  bool in_bootstrap = false;  // hl_create's bootstrap is running
  HostScalars hs;
  u64 epoch = 1;         // selection epochs (reservation keys)
  u32 sel_round = 0;     // role tag of the current selection
  u32 gang_set = 0;      // counter block of the next gang launch
  u64 stats_sel_iters = 0;
  u64 nlaunch = 0;       // launches of this library's kernels
  u64 launch_mark = 0;
  // per-call statistics
  hl_batch_stats st{};
  // sub-community ids of the last refinement's splits: new_base ..
  // new_base + n_new - 1, split from the ids in Scratch::origin
  u32 n_new = 0, new_base = 0;
  // K marks handed to the next level's inc_movement (M8): the nodes it gained
  // from splits below and the nodes whose community the projection changed
  bool k_flags_set = false;
  u32 prune_rounds = 0;  // multi-kernel evaluations of the running movement
  Prune prune;           // the running movement's bounds (b == nullptr: off)
  bool shared = false;   // other graphs are being updated on the GPU meanwhile
  // The handle's budget may not hold what the one-launch stages and the movement
  // bounds take: this call keeps to the multi-kernel stages, which size their
  // scratch by what they find (plan_scratch).
  bool lean = false;
  void plan_scratch(u64 n, u64 entries, u64 updates, u64 nlevels);
  u64 sum_nv_batch = 0;  // frontier sizes of the multi-kernel evaluations, this call
  // degree-bin thresholds picked by the autotuner (0 = compile-time default)
  struct Tune {
    u32 mid_max = 0, wide_max = 0;
    u32 hub_defer = 0;  // integral weights: hub rows above this many entries skip pass 1
    bool done = false;
    u32 frontier = 0;
    float best_ms = 0.f;
  } tune;
  // per-level output (hl_set_level_callback): called after each level's refinement
  hl_level_fn level_fn = nullptr;
  void* level_user = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // kernel timing
  bool ktiming = false;
  KernelAgg kagg[KT_COUNT];
  std::vector<cudaEvent_t> ev_pool;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> ev_pending;
  // on `s`, or on the engine's stream
  cudaEvent_t kt_begin(cudaStream_t s = nullptr);
  void kt_end(int id, cudaEvent_t a, cudaStream_t s = nullptr);
  void kt_collect();

  u64 read_u64(const u64* dptr);
  u32 read_u32(const u32* dptr);
  // Several device scalars with one wait: out[i] = *ptrs[i] (at most 16).
  void read_u32s(std::initializer_list<const u32*> ptrs, u32* out);
  double read_f64(const double* dptr);
  void sync();
};

// CUB helper: query temp bytes, grow the shared temp buffer, run.
template <typename F>
inline void cub_run(Engine& E, F f) {
  size_t bytes = 0;
  HL_CUDA(f((void*)nullptr, bytes));
  E.sc.cub_tmp.ensure(E.mem, bytes + 16);
  HL_CUDA(f((void*)E.sc.cub_tmp.p, bytes));
}

// ---- stage entry points (one .cu file each) --------------------------------
// graph.cu
void graph_init_empty(Engine& E, Level& L, u32 n);
void graph_grow_nodes(Engine& E, Level& L, u32 n);
void apply_delta(Engine& E, Level& L, const DevEdges& b, u32 new_n, bool keep_loops);
void recompute_all_degrees(Engine& E, Level& L);
double tree_sum(Engine& E, const double* x, u64 n);
void seq_sums(Engine& E, u32 nseg, const u64* off, const double* x, double init, int path,
              double* out);
// Kernels that take 32 rows or segments a warp leave those of LONG_SEG terms or
// more to a second launch: hub rows stand side by side (R-MAT's first vertices),
// and one warp would sum all of its 32 one after another.  List (and zeroed
// count) with room for every such segment of `total` terms.
constexpr u64 LONG_SEG = 512;
constexpr u32 LONG_BLOCKS = 148 * 4;
struct LongList {
  u32* seg;
  u32* cnt;
};
LongList long_list(Engine& E, u64 total, u32 nseg);
bool edges_integral(Engine& E, const DevEdges& b);
void check_endpoints(Engine& E, const DevEdges& b, u32 n);

// gang_apply.cu: apply_delta in one launch, for batches it fits
// Updates: where the in-kernel sorts (chunks ranked among each other) have caught
// up with the radix sorts.  Kernel time of the stage, one launch and multi-kernel:
// 0.09 and 0.12 ms for 2,048 updates of 20k vertices, 0.22 and 0.22 for 32,768;
// of 400k vertices 0.13 and 0.14, 0.32 and 0.25.  The multi-kernel form adds five
// host reads, 0.4-0.6 ms.
constexpr u64 GANG_BATCH_MAX = 32768;
bool gang_apply_fits(Engine& E, const Level& L, const DevEdges& b, bool drop_loops);
void gang_apply(Engine& E, Level& L, const DevEdges& b);

// move.cu
struct MoveOut {
  u32 iterations = 0;
  u64 moves = 0, candidates = 0, traversed = 0, changed = 0;
};
MoveOut inc_movement(Engine& E, Level& L, const DevEdges& delta, bool all_active,
                     bool mark_moved);
void recompute_comm_degrees(Engine& E, Level& L, const u32* part, u32 ncomm_cap, double* d);
void compact_labels_if_needed(Engine& E, u32* labels, u32 n, u32 limit);
void select_decoupled_dev(Engine& E, u32 M);
void ensure_comm_arrays(Engine& E, size_t ncap);
// Rounds one launch of gang_move runs at most before it hands back, so that a
// movement without a cap that never settles is a chain of launches of some 10 ms
// (10 us a round) and not one without an end; a round takes at most 65 epochs.
constexpr u32 SEL_ROUNDS = 1024;
void selection_room(Engine& E);
void prune_begin(Engine& E, const Level& L);
void run_eval(Engine& E, int kind, const u32* verts, u32 nv, const Level& L, const u32* s,
              const double* d, const u8* blocked, bool allow_empty, u32* out_to, double* out_gain,
              unsigned long long* traversed);

// refine.cu
struct RefineOut {
  u64 splits = 0, merges = 0, refined = 0;
  u64 tfilter_exact = 0;  // candidates decided from the ordered sum
  u32 smax_before = 0;
  u32 singles = 0;  // refined singletons (gang_refine)
};
RefineOut inc_refinement(Engine& E, Level& L, bool cc_same_community);
u32 reduce_max_u32(Engine& E, const u32* x, u32 n, u32* out);

// gang_refine.cu: the refinement in one launch; the status names the step the
// multi-kernel path continues from
enum : u32 { REF_DONE = 0, REF_HOST_ALL = 1, REF_HOST_MERGE = 2, REF_HOST_EVAL = 3 };
bool gang_refine_fits(Engine& E, const Level& L);
u32 gang_refine(Engine& E, Level& L, bool cc_same_community, RefineOut& out);

// api.cu: device-side batch statistics (Scratch::bacc)
void stats_acc_u64(Engine& E, const unsigned long long* src, u32 count, u32 slot);
void stats_acc_u32(Engine& E, const u32* src, u32 slot);
void stats_count_flags(Engine& E, const u8* flags, u32 n, u32 slot);

// gang_move.cu: the movement in one launch; the status says why the host's
// rounds go on from S.active
enum : u32 { MOVE_DONE = 0, MOVE_BIG_FRONTIER = 1, MOVE_BIG_HUB = 2, MOVE_LABELS = 3 };
struct GangMoveStats {
  u64 moves = 0, cands = 0, trav = 0;
  u32 frontier = 0;  // of the round the last launch handed over
};
// Frontier (and candidate) limit.  Where it lies hardly matters: first passes of
// the 1M-vertex f64 graph, whose rounds have 37-50k vertices, take 130, 139, 138
// and 127 ms with 32768, 65536, 131072 and 1M; the smallest keeps the lists small.
constexpr u32 GM_FRONTIER = 32768;
bool gang_move_fits(Engine& E, const Level& L);
u32 gang_move(Engine& E, Level& L, const DevEdges& delta, bool setup, bool all_active,
              bool mark_moved, u32 frontier, u32& it, GangMoveStats& ms);

// eval.cu: degree-bin autotuner (once per handle)
void autotune_bins(Engine& E, const u32* verts, u32 nv, const Level& L, const u32* s,
                   const double* d, u32* out_to, double* out_gain);

// det.cu: the sequential (RunMode::Deterministic) steps
void inc_movement_det(Engine& E, Level& L, const u32* act, double* d, size_t dcap,
                      bool mark_moved, u64* moves, u64* traversed);
u64 merge_singletons_det(Engine& E, Level& L, const u32* rv, u32 nr, u32* sizes, double* dS,
                         const double* dcomm, size_t scap);

// Test switch: decide every T-filter candidate from the ordered sum.
extern std::atomic<int> g_exact_tfilter;
// Test switch: table slots of the partitioned hub pass (eval.cu).
extern std::atomic<u32> g_pb_slots;
extern std::atomic<u32> g_dbg_hub_defer;
extern std::atomic<u64> g_dbg_pb_round;

// aggregate.cu
// gang_aggregate.cu: the next level's growth and projection and the aggregation
// in one launch
bool gang_aggregate_fits(Engine& E, const Level& L, const DevEdges& delta);
bool gang_aggregate(Engine& E, Level& L, Level& H, const DevEdges& delta, bool aggregate,
                    DBuf<u32>& ou, DBuf<u32>& ov, DBuf<double>& ow, u64* count);
u64 inc_aggregation(Engine& E, Level& L, const DevEdges& delta, u32* next_n,
                    bool changed_only, bool edge_weight_loops);  // output in sc.eu2/ev2/ew2
u64 aggregate_full(Engine& E, Level& L, const u32* s, u32* out_u, u32* out_v, double* out_w);
void project_up(Engine& E, Level& lo, Level& hi, u8* changed_flags = nullptr);
void top_down(Engine& E);
void inherit_new_nodes(Engine& E, Level& hi);

// gang_modularity.cu
double modularity(Engine& E, Level& L, const u32* part);
void canonicalize_bounded(Engine& E, const u32* labels, u32 n, u32 bound, u32* out);
// modularity.cu
void canonicalize_device(Engine& E, u32* labels, u64 n, u32* out);
u32 rank_compact(Engine& E, u32* labels, u32 n, u32 id_bound);

// kernels used by more than one stage
__global__ void k_fill_u8(u8* p, u8 v, u64 n);
__global__ void k_iota(u32* p, u32 n);

}  // namespace hl
