// modularity.cu — first-seen label canonicalisation of arbitrary labels
// (hit_leiden.rs:358-376); gang_modularity.cu holds the modularity and the
// canonicalisation of a handle's own labels.
#include "hl_engine.cuh"

namespace hl {

static inline u32 grid_for(u64 n, u32 block = 256) {
  u64 g = (n + block - 1) / block;
  if (g > 148u * 64u) g = 148u * 64u;
  return g ? (u32)g : 1u;
}

// First-seen relabelling: a label's new id is the rank of its first index.
__global__ void k_first_index(const u32* lab, u64 n, u32* first) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    atomicMin(&first[lab[i]], (u32)i);
}
__global__ void k_is_first(const u32* lab, u64 n, const u32* first, u32* flag) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    flag[i] = first[lab[i]] == (u32)i ? 1u : 0u;
}
__global__ void k_apply_first(const u32* lab, u64 n, const u32* first, const u32* rank, u32* out) {
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    out[i] = rank[first[lab[i]]];
}

void canonicalize_device(Engine& E, u32* labels, u64 n, u32* out) {
  if (!n) return;
  Scratch& S = E.sc;
  cudaStream_t st = E.stream;
  S.cnt.ensure(E.mem, 16);
  u32* o = S.cnt.p + 14;
  cub_run(E, [&](void* t, size_t& b) {
    return cub::DeviceReduce::Max(t, b, labels, o, (int64_t)n, st);
  });
  u64 nc = (u64)E.read_u32(o) + 1;
  DBuf<u32> first, flag, rank;
  first.ensure(E.mem, nc);
  flag.ensure(E.mem, n);
  rank.ensure(E.mem, n);
  HL_CUDA(cudaMemsetAsync(first.p, 0xFF, sizeof(u32) * nc, st));
  ++E.nlaunch, k_first_index<<<grid_for(n), 256, 0, st>>>(labels, n, first.p);
  ++E.nlaunch, k_is_first<<<grid_for(n), 256, 0, st>>>(labels, n, first.p, flag.p);
  HL_LAUNCH_CHECK();
  u32* a = flag.p;
  u32* r = rank.p;
  cub_run(E, [&](void* t, size_t& b) {
    return cub::DeviceScan::ExclusiveSum(t, b, a, r, (int64_t)n, st);
  });
  ++E.nlaunch, k_apply_first<<<grid_for(n), 256, 0, st>>>(labels, n, first.p, rank.p, out);
  HL_LAUNCH_CHECK();
  E.sync();
}

}  // namespace hl
