// gang.cu — shapes and launches of the single-launch stage kernels (gang.cuh).
#include "gang.cuh"

namespace hl {

static u32 sm_count(int device) {
  static std::atomic<u32> cached[64];
  if (device >= 0 && device < 64 && cached[device].load()) return cached[device].load();
  int v = 0;
  HL_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device));
  if (device >= 0 && device < 64) cached[device].store((u32)v);
  return (u32)v;
}

// One block up to a few thousand entries (its barrier is a block barrier), a
// portable cluster of 8 up to a few hundred thousand, above that one block
// per SM.  While other graphs are being updated too, a grid that needs every SM
// at once waits for all of their kernels: there clusters go on to a few million
// entries (48 graphs of 1k-30k vertices on 16 host threads: 18.5 ms a batch
// each with grids, 12 ms with clusters; one graph at a time: 97 and 104 ms).
constexpr u64 GANG_CLUSTER_WORK = 400000;
constexpr u64 GANG_SHARED_WORK = 4000000;

u64 gang_cluster_work(const Engine& E) { return E.shared ? GANG_SHARED_WORK : GANG_CLUSTER_WORK; }

GangShape gang_shape(Engine& E, u64 work) {
  if (work <= GANG_BLOCK_WORK) return GangShape{1, false};
  if (work <= gang_cluster_work(E)) return GangShape{8, false};
  const u32 sms = sm_count(E.device);
  return GangShape{sms < GANG_MAX_BLOCKS ? sms : GANG_MAX_BLOCKS, true};
}

u32* gang_counters(Engine& E, u32** next) {
  Scratch& S = E.sc;
  if (!S.gang_cnt.p) {
    S.gang_cnt.ensure(E.mem, 2 * GANG_CNT);
    HL_CUDA(cudaMemsetAsync(S.gang_cnt.p, 0, 2 * GANG_CNT * sizeof(u32), E.stream));
    E.gang_set = 0;
  }
  *next = S.gang_cnt.p + (E.gang_set ^ 1u) * GANG_CNT;
  return S.gang_cnt.p + E.gang_set * GANG_CNT;
}
void gang_turn(Engine& E) { E.gang_set ^= 1u; }

void gang_launch(Engine& E, const void* kernel, const GangShape& s, size_t smem, void* args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(s.blocks);
  cfg.blockDim = dim3(GANG_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = E.stream;
  cudaLaunchAttribute at[1];
  cfg.attrs = at;
  if (s.grid) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.numAttrs = 1;
  } else if (s.blocks > 1) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = s.blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  void* params[1] = {args};
  ++E.nlaunch;
  HL_CUDA(cudaLaunchKernelExC(&cfg, kernel, params));
}

}  // namespace hl
