// The launch shape of a lockstep decision: the blocks and the threads of each to launch, the arenas a warp claims at a
// time, and whether it claims them from the queue.  Host code without CUDA calls; capi.cu launches what it says.
#pragma once
#include <stdint.h>

namespace rsx {

constexpr uint32_t kSpreadSplit = 15;  // the lockstep split whose kernels exist in every register budget

// The blocks to launch of `grid` asked for, on a device of `sms` SMs that each hold per_sm() such blocks at once.  Arenas
// are dealt out over the blocks at the start, so a block that waited for another to leave its SM would step its share a
// whole decision later (4,096 headline arenas on 1,480 blocks of 64 threads: 16.3 ms, of which an SM holds three), and
// blocks on one SM step out of lockstep with one another: no more than hold the arenas, the same number on every SM (the
// same call on 148: 4.8 ms), and no more than the device holds.
template <class PerSm>
inline uint32_t lockstep_grid(uint32_t n, uint32_t grid, uint32_t block, uint32_t sms, PerSm&& per_sm) {
  if (grid <= sms || sms == 0) return grid;
  const uint64_t lanes = (uint64_t)sms * block;
  uint64_t most = (n + lanes - 1) / lanes;  // blocks per SM
  if (most > 1) {
    const uint32_t held = per_sm();
    if (held != 0 && most > held) most = held;
  }
  return most * sms < grid ? (uint32_t)(most * sms) : grid;
}

struct LockstepPlan {
  uint32_t block, width;
  bool queue;
};
// n arenas on `grid` blocks of at most `block` threads
inline LockstepPlan lockstep_plan(uint32_t n, uint32_t grid, uint32_t block, uint32_t split) {
  const uint64_t lanes = (uint64_t)grid * block;
  const uint64_t rounds = (n + lanes - 1) / lanes;
  const uint32_t per = (uint32_t)((n + rounds * grid - 1) / (rounds * grid));  // a block's arenas in one round
  LockstepPlan p;
  // Blocks no larger than their arenas need: a scheduler's registers are its warps', 255 each for 8 warps a block, 168 for 12,
  // 128 for 14 and 16.  20,000 headline arenas (136 per SM): 6.5 ms in 256 threads; 7.3 in 448, and 7.8 in 256 threads held
  // to 128 registers, so it is the registers that pay and not the fewer warps at a barrier.  56,000 (379): 9.7 in 384, 10.1
  // in 448.  Uneven rounds are evened out the same way: 70,001 arenas in two rounds of 256 threads rather than one of 448
  // and a rest.
  p.block = block;
  if (split == kSpreadSplit && per <= 384 && block > 384) p.block = 384;
  if (split == kSpreadSplit && per <= 256 && block > 256) p.block = 256;
  // Few arenas a block: one warp per SM until it is full, then more.  A warp's lanes share its instruction fetches, which
  // bound an SM that runs few warps; spread over more warps the lanes diverge less but each warp fetches for itself.
  // 2,048 arenas: headline states 3.4 ms in one warp of 14, 3.6 in seven of 2; kickoffs, which hardly diverge, 1.3 and 2.1
  // ms; 4,096: 4.15 and 1.4 ms in one warp, 4.05 and 1.9 in four.  Up to three arenas get a warp each, where the block has
  // the warps (444 arenas on 148 blocks of one warp, claimed one by one: kickoffs 3.9 ms, in one claim 1.7): 300 arenas
  // 1.8 ms, 1.9 in one warp (contact-heavy 2.1 both ways; kickoffs 1.3 and 1.1).
  const uint32_t warps = p.block / 32;
  p.width = per <= 3 && per <= warps ? 1u : per < 32 ? per : 32u;
  p.queue = rounds > 1;  // one round is dealt out evenly by the kernel (10,007 arenas left 125 of 148 SMs idle: 9.6 ms, now 5.3)
  return p;
}

}  // namespace rsx
