// Test build of the lockstep kernel's split 15 (librsx_lists.so; not part of librsx.so): the block's mesh lists so short that a
// few contact-heavy arenas fill every one of them, counters of the ways past a full list, and a StaticData whose trees are
// deeper than the walk's path keys hold.
#include <cuda_runtime.h>
#include <stdint.h>
#define RSX_LS_MAXT 448
#define RSX_LS_WIDE_REGS    // split 15 only
#define RSX_LS_SMALL_LISTS
// a job lost to a full list, to a deep tree; done by its lane alone; waiting for another round; a SAT past the list; a lost
// wheel-ray job
enum { kCountFull, kCountDeep, kCountAlone, kCountWait, kCountSat, kCountRayAlone, kCounts };
__device__ uint32_t rsx_ls_count[kCounts];
#define LS_COUNT(which) atomicAdd(&rsx_ls_count[which], 1u)
#include "kern_lockstep.cu"

// one decision of n arenas on `grid` blocks of `block` threads in claims of `width`; counts: kCounts words on the host
extern "C" int rsx_lists_decide(uint32_t* d_states, uint32_t n, const void* d_statics, const uint8_t* d_sd_index, const void* d_controls,
                                uint32_t* d_result, uint32_t* d_event_or, uint32_t width, uint32_t grid, uint32_t block, uint32_t* counts,
                                void* stream) {
  const uint32_t zero[kCounts] = {};
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyToSymbolAsync(rsx_ls_count, zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      L_NAME(d_states, d_statics, d_sd_index, d_controls, d_result, d_event_or, nullptr, nullptr, n, width, grid, block, 15, 1, kTicksPerDecision,
             s) != cudaSuccess ||
      cudaMemcpyFromSymbolAsync(counts, rsx_ls_count, sizeof(zero), 0, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -2;
  return 0;
}

// `levels` nodes of one child each above every mesh's root: the walks reach the same leaves in the same order, that much
// deeper.  0, or -1 where the node array has no room.
extern "C" int rsx_lists_deepen(uint32_t* static_words, uint32_t levels) {
  StaticData& D = *reinterpret_cast<StaticData*>(static_words);
  uint32_t at = 0;
  for (int m = 0; m < kMeshes; ++m) {
    const uint32_t end = D.meshes[m].node_first + D.meshes[m].node_count;
    at = end > at ? end : at;
  }
  for (int m = 0; m < kMeshes; ++m) {
    const uint32_t first = D.meshes[m].node_first;
    if (D.meshes[m].node_count == 0) continue;
    for (uint32_t l = 0; l < levels; ++l) {
      if (at >= (uint32_t)kMaxNodes) return -1;
      D.nodes[at] = D.nodes[first];  // the root so far, below its new one
      WideNode& root = D.nodes[first];
      for (int i = 0; i < 4; ++i) {
        root.lo_x[i] = root.lo_y[i] = root.lo_z[i] = -1e9f;
        root.hi_x[i] = root.hi_y[i] = root.hi_z[i] = 1e9f;
        root.child[i] = at - first;
      }
      root.n_child = root.valid = 1;
      ++at;
    }
  }
  return 0;
}
