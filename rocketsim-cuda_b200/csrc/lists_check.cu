// Test build of the lockstep kernel's split 15 (librsx_lists.so; not part of librsx.so): the block's mesh lists so short that a
// few contact-heavy arenas fill every one of them, and counters of the ways past a full list.
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
