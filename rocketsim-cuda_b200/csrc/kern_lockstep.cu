// The SM-lockstep persistent decision kernel.
//
// Why: one decision runs ~10^5 dependent instructions per arena through a simulator whose machine code is about a
// megabyte (P1 and P3b alone are ~450 KB each), far beyond an SM's instruction cache.  When the warps of an SM drift
// into different phases, every warp's instruction fetches evict the others' and the SM stalls on instruction misses
// (measured on the one-thread-per-arena launch: ~26 cycles of "no instruction" stall per issued instruction, issue
// active 4% of cycles).  Here the warps of a block step their arenas phase by phase together: a __syncthreads()
// after each of the ten phases (split 1: also after each car's pre-tick inside P1; split 2: P1 of each car in three
// parts, pre-tick head / wheel rays / wheel response; split 3: also a barrier after every step of P3b's pair / leaf
// loop; split 6: split 2 with P5 as rows / iterations / integration and P8 as cars / the rest; split 7: split 6 with
// P3a one dynamic body at a time; splits 4 and 5 leave
// the barriers out between P3b (4) or P4 (5) and P8, to measure what they buy), so that at any time the block's warps
// fetch from one piece of code.  Splits 9 and 10 add the pooled contact work below; split 11 is split 10 with P3a in
// one piece again (once P3b and the rays were pooled, P3a's per-body barriers cost more than they kept together);
// split 14 is split 11 with the box-triangle SATs' feature pairs computed by the whole block; split 15 runs all of a
// tick's mesh work (the wheel rays of both cars, every mesh pair of P3b) in one round each, its BVH walks too by the whole
// block, level by level.
//
// Work: `gridDim.x` resident blocks (normally one per SM, `blockDim.x` up to RSX_LS_MAXT threads); every warp claims
// `width` (up to 32) consecutive entries of `order` (arena indices; identity when null) whenever its previous arenas have
// finished this launch's ticks (t_first..t_last of the decision's 8), with one atomicAdd on `counter` (zero at launch) or,
// when counter is null, its own share of the entries in turn, and loads them at the next tick boundary.  A claim narrower
// than a warp leaves its other lanes without an arena; they still take part in the block's pooled work.  A decision split
// over several launches carries each arena's progress in its result word (scored tick, unimplemented bit) and event
// word; an arena scored in an earlier launch is not stepped again.  The block leaves when no warp holds work.  Lanes past
// n and order entries past n store nothing (they step nothing, or a copy in the splits that pool nothing).
//
// Results: each arena's decision is the decide() sequence of sim/physics.cuh (controls before every tick, all 8 ticks
// stepped, the state after the first scored tick kept, event OR up to that tick), so states, result words and event
// words equal those of every other decision kernel, whatever grid, block, split or order.
//
// Compiled once per register budget (RSX_LS_MAXT threads per block, one block per SM; a scheduler holds a quarter of the
// registers and of the warps): 256 threads -> 255 registers, 384 -> 168, 448 and 512 -> 128.  The first two hold split 15
// only (RSX_LS_WIDE_REGS).
#include "kern_common.cuh"

#ifndef RSX_LS_MAXT
#define RSX_LS_MAXT 512
#endif
#define RSX_CAT2(a, b) a##b
#define RSX_CAT(a, b) RSX_CAT2(a, b)
#define K_NAME RSX_CAT(k_sim8_lockstep_t, RSX_LS_MAXT)
// Zone timers of the profiling build (RSX_ZONES; empty markers otherwise): warp cycles in each piece of the tick
// (ids 40-49 and 29-30: P0, P1 head, P1 rays, P1 response, P2, P3a, P3b, P4, P5, P6, P7, P8), at the barrier after it
// (ids 50-59 and 31-32 likewise), and inside the pooled P3b (33 heads and walks, 34 pooled tests, 35 additions).
#define LS_SYNC(id)          \
  do {                       \
    RSX_ZONE_BEGIN(zb_);     \
    __syncthreads();         \
    RSX_ZONE_END(zb_, id);   \
  } while (0)
#define L_NAME RSX_CAT(rsx_launch_sim8_lockstep_t, RSX_LS_MAXT)
// Counters of the test build (lists_check.cu; empty otherwise): how often split 15's ways past a full list are taken
#ifndef LS_COUNT
#define LS_COUNT(which)
#endif

namespace {
// ---- split 9: P3b with the leaf tests of every arena of the block pooled ----
// Each round, every lane whose arena has P3b work runs its pair heads up to its next mesh job and takes up to
// sim::kLeafChunk leaves of the job's BVH walk; the jobs and their (job, leaf) tests are published in shared memory
// (slots from a block-wide prefix sum); all threads of the block then run the tests, kPoolPairs at most, one test per
// thread at a time; each owner adds its hits in walk order and closes the job when its walk is done.  A heavy arena's
// leaves (a ball against a wall: up to ~30 triangles in one tick) are thus tested side by side instead of one after
// another on one lane, while the order-dependent part (the manifold updates) stays on the owner.  Jobs past the pool's
// capacity test their own leaves, as in the other splits.  Words equal every other split's: the walk / test / add
// separation is exact (sim/narrow.cuh, P3b driver).
constexpr int kPoolJobs = 128;
constexpr int kPoolPairs = 512;
// split 14: up to kDeferSat box-triangle SATs of a round that reach their 47 feature pairs have those pairs computed by
// the whole block (stage B) before their owners' threads finish them (stage C); the pairs overlay the job records, which
// no thread reads after the first stage of the tests.
constexpr int kDeferSat = 18;
struct PoolSmem {
  union {
    struct {
      sim::LeafJob job[kPoolJobs];
      const StaticData* jd[kPoolJobs];
      uint32_t pair_job[kPoolPairs];
      uint32_t pair_tri[kPoolPairs];
    };
    sim::FeatPair feat[kDeferSat][sim::kPairs];
  };
  sim::LeafHit hit[kPoolPairs];
  sim::SatFront front[kDeferSat];
  uint32_t front_pair[kDeferSat];
};
static_assert(sizeof(sim::FeatPair) * kDeferSat * sim::kPairs <=
                  sizeof(sim::LeafJob) * kPoolJobs + sizeof(void*) * kPoolJobs + sizeof(uint32_t) * 2 * kPoolPairs,
              "the feature pairs fit over the job records");
// split 10: the wheel rays' mesh leaves pooled too (sim/ray.cuh: evaluated anywhere, replayed on the owner)
constexpr int kRayJobs = 64;
constexpr int kRayPairs = 512;
constexpr int kRayJobsLane = 4;
constexpr int kRayLeavesLane = 48;
struct RayPoolSmem {
  sim::RayMeshJob job[kRayJobs];
  const StaticData* jd[kRayJobs];
  uint32_t pair_job[kRayPairs];  // job slot | mesh index << 16
  uint32_t pair_leaf[kRayPairs];
  sim::RayLeaf out[kRayPairs];
};
// split 15: mesh walks by the whole block.  Jobs (a body's query box against a mesh body) are listed in shared memory,
// the block walks all their BVHs level by level (front: the nodes of one level with their path keys, sim/ray.cuh
// walk_expand), and the leaves found are put in each job's stack-walk order by a counting sort by job and a ranking by
// key within the job.  A job that loses a node, a leaf or a hit to a full list, or whose tree is deeper than the keys hold,
// is marked and done by its own lane (in P3b a full list is tried again first); the other jobs are whole.
constexpr uint32_t kJobMask = 511u, kHeadMask = 8191u;
constexpr int kJobBits = 9, kHeadBits = 13;  // job, then mesh (4 bits), then node or leaf
constexpr uint32_t kLostFull = 1u, kLostDeep = 2u;  // marks of lost[]
template <int JOBS, int FRONT, int LEAVES>
struct WalkLists {
  uint32_t cnt[JOBS], seg[JOBS], fill[JOBS], lost[JOBS];
  uint32_t front[2][FRONT];     // job | mesh | node
  uint16_t fkey[2][FRONT];      // its path key
  uint32_t leaf[LEAVES];        // as found: job | mesh | leaf
  uint16_t key[LEAVES];         // its path key
  uint16_t byjob[LEAVES];       // the entries above, by job
  uint32_t njobs, nfront[sim::kWalkLevels + 1], nleaf;
};
#ifndef RSX_LS_SMALL_LISTS
constexpr int kWalkRayJobs = 144, kWalkRayFront = 384, kWalkRayLeaves = 400;
constexpr int kWalkPairJobs = 208, kWalkPairFront = 640, kWalkPairLeaves = 704;
constexpr int kWalkHits = 128;
constexpr int kWalkSats = 48;      // SATs of a round whose feature pairs the block computes, kWalkFeat at a time
constexpr int kWalkFeat = 15;
#else  // the test build: a few contact-heavy arenas fill every list
constexpr int kWalkRayJobs = 16, kWalkRayFront = 24, kWalkRayLeaves = 24;
constexpr int kWalkPairJobs = 24, kWalkPairFront = 32, kWalkPairLeaves = 32;
constexpr int kWalkHits = 4;
constexpr int kWalkSats = 2;
constexpr int kWalkFeat = 1;
#endif
constexpr int kWalkRayLane = 8;  // jobs of one lane (both cars)
struct RayWalkSmem {
  sim::RayMeshJob job[kWalkRayJobs];
  Box3 jbox[kWalkRayJobs];
  uint16_t jbody[kWalkRayJobs], jsd[kWalkRayJobs];
  WalkLists<kWalkRayJobs, kWalkRayFront, kWalkRayLeaves> w;
  sim::RayLeaf out[kWalkRayLeaves];
  uint32_t at[kWalkRayLeaves];  // mesh | leaf << 4 of out[]
};
constexpr int kWalkPairLane = 8;   // jobs of one lane in one round
constexpr int kWalkPairRounds = 3; // from this round on a job lost to a full list is done by its lane alone
struct PairJob {                   // a sim::LeafJob without what the static data holds
  uint8_t kind, mesh, body;
  union {
    struct { Aff box_xf, mesh_to_box; };
    struct { V3 center; float radius, rt, rt2; };
  };
};
struct PairWalkSmem {
  union {
    PairJob job[kWalkPairJobs];
    sim::FeatPair feat[kWalkFeat][sim::kPairs];  // over the job records, which nobody reads after the tests
  };
  Box3 jbox[kWalkPairJobs];
  uint16_t jsd[kWalkPairJobs];
  WalkLists<kWalkPairJobs, kWalkPairFront, kWalkPairLeaves> w;
  sim::LeafHit hit[kWalkHits];
  uint16_t at_tri[kWalkPairLeaves];  // in walk order: the leaf's triangle, and its hit's index + 1 (0: no contact)
  uint16_t at_hit[kWalkPairLeaves];
  sim::SatFront front[kWalkSats];
  uint32_t front_at[kWalkSats];      // place | job << 16
  uint32_t nsat, nhit;
};
static_assert(sizeof(sim::FeatPair) * kWalkFeat * sim::kPairs <= sizeof(PairJob) * kWalkPairJobs, "the feature pairs fit over the jobs");
static_assert(sizeof(RayWalkSmem) + 256 <= 63 * 1024 && sizeof(PairWalkSmem) + 256 <= 63 * 1024, "a 64 KB carveout");
static_assert(kWalkPairFront >= kWalkPairJobs, "every job starts as an entry of the first level");
static_assert(kWalkPairJobs <= 512 && kWalkRayJobs <= 512 && kMeshes <= 16 && kWalkPairLeaves < 65536 && kMaxTris < 65536 &&
                  kWalkHits < 65535 && kMaxNodes < (1 << 19) && kMaxLeaves < (1 << 19),
              "the lists' fields hold their values");
// one shared buffer for the pools (they serve different pieces of the tick) and the prefix sums
struct Pools {
  union {
    PoolSmem p3b;
    RayPoolSmem rays;
    RayWalkSmem ray_walk;
    PairWalkSmem pair_walk;
  };
  uint32_t warp_sum[32];
  uint32_t limit;
  uint32_t deferred;  // split 14: SATs of this round whose feature pairs the block computes
};
extern __shared__ uint4 smem_pools[];  // sizeof(Pools) bytes for the splits that pool (9 on)
__device__ __forceinline__ Pools& pools() { return *reinterpret_cast<Pools*>(smem_pools); }

// block-wide exclusive prefix sum of v (every thread calls it); returns the exclusive sum, *total the block's sum
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* total, Pools& sm) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if (lane >= (uint32_t)d) x += y;
  }
  if (lane == 31) sm.warp_sum[warp] = x;
  if (threadIdx.x == 0) {
    sm.limit = 0;
    sm.deferred = 0;
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < nw ? sm.warp_sum[lane] : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, d);
      if (lane >= (uint32_t)d) w += y;
    }
    sm.warp_sum[lane] = w;
  }
  __syncthreads();
  *total = sm.warp_sum[nw - 1];
  return (warp ? sm.warp_sum[warp - 1] : 0u) + x - v;
}

// P3b of the thread's arena (have) with pooled leaf tests; every thread of the block calls it.  SplitSat (split 14): the
// box-triangle SATs that reach their feature pairs have them computed by the whole block.
template <bool SplitSat>
__device__ __noinline__ void p3b_pooled(ArenaState& s, const StaticData* D, bool have, int* un) {
  Pools& u = pools();
  PoolSmem& sm = u.p3b;
  sim::P3bLoop L;
  bool more = have;
  if (have) sim::p3b_begin(s, L);
  uint32_t tris[sim::kLeafChunk];
  for (;;) {
    int k = 0;
    bool job = false;
    RSX_ZONE_BEGIN(zo);
    if (more) {
      if (sim::p3b_open(s, *D, L) == sim::NEAR_DONE) {
        more = false;
      } else {
        job = true;
        k = sim::p3b_collect(*D, L, tris, sim::kLeafChunk);
      }
    }
    RSX_ZONE_END(zo, 33);
    // (the barrier also orders the last round's reads of the pool before this round's writes)
    RSX_ZONE_BEGIN(zb0);
    const bool any = __syncthreads_or(job);
    RSX_ZONE_END(zb0, 56);
    if (!any) break;
    uint32_t total;
    const uint32_t v = k > 0 ? ((1u << 16) | (uint32_t)k) : 0u;
    const uint32_t ex = block_scan(v, &total, u);
    const uint32_t slot = ex >> 16, off = ex & 0xFFFFu;
    // pooled jobs are a prefix in scan order (slot and off only grow), so the pool's pairs are [0, limit)
    const bool pooled = k > 0 && slot < (uint32_t)kPoolJobs && off + (uint32_t)k <= (uint32_t)kPoolPairs;
    if (pooled) {
      sim::leaf_job_of(L, sm.job[slot]);
      sm.jd[slot] = D;
      for (int i = 0; i < k; ++i) {
        sm.pair_job[off + i] = slot;
        sm.pair_tri[off + i] = tris[i];
      }
      atomicMax(&u.limit, off + (uint32_t)k);
    }
    LS_SYNC(56);
    const uint32_t npairs = u.limit;
    RSX_ZONE_BEGIN(zt);
    for (uint32_t p = threadIdx.x; p < npairs; p += blockDim.x) {
      const uint32_t j = sm.pair_job[p];
      sim::LeafHit h;
      if (!SplitSat) {
        sim::leaf_test(sm.job[j], *sm.jd[j], sm.pair_tri[p], &h);
      } else {
        sim::SatFront f;
        if (!sim::leaf_test_front(sm.job[j], *sm.jd[j], sm.pair_tri[p], &h, &f)) {
          const uint32_t d = atomicAdd(&u.deferred, 1u);
          if (d < (uint32_t)kDeferSat) {  // the block computes its feature pairs below
            sm.front[d] = f;
            sm.front_pair[d] = p;
            continue;
          }
          sim::FeatPair P[sim::kPairs];  // past the deferred capacity: this thread computes them itself
          sim::enum_pairs(f.hu, f.q, f.e, P);
          sim::leaf_test_back(f, P, &h);
        }
      }
      sm.hit[p] = h;
    }
    RSX_ZONE_END(zt, 34);
    LS_SYNC(56);
    if (SplitSat) {
      const uint32_t nd = min(u.deferred, (uint32_t)kDeferSat);
      if (nd != 0) {  // (uniform: every thread read the count after the barrier)
        RSX_ZONE_BEGIN(zf);
        for (uint32_t w = threadIdx.x; w < nd * (uint32_t)sim::kPairs; w += blockDim.x) {
          const uint32_t d = w / (uint32_t)sim::kPairs, i = w % (uint32_t)sim::kPairs;
          sm.feat[d][i] = sim::feat_pair(sm.front[d], (int)i);
        }
        RSX_ZONE_END(zf, 34);
        LS_SYNC(56);
        RSX_ZONE_BEGIN(zg);
        for (uint32_t d = threadIdx.x; d < nd; d += blockDim.x) {
          sim::LeafHit h;
          sim::leaf_test_back(sm.front[d], sm.feat[d], &h);
          sm.hit[sm.front_pair[d]] = h;
        }
        RSX_ZONE_END(zg, 34);
        LS_SYNC(56);
      }
    }
    RSX_ZONE_BEGIN(zc);
    if (pooled) {
      for (int i = 0; i < k; ++i)
        if (sm.hit[off + i].found) sim::p3b_add_hit(s, *D, L, tris[i], sm.hit[off + i]);
    } else if (k > 0) {  // past the pool's capacity: this lane tests its own leaves
      sim::LeafJob jb;
      sim::leaf_job_of(L, jb);
      for (int i = 0; i < k; ++i) {
        sim::LeafHit h;
        if (sim::leaf_test(jb, *D, tris[i], &h)) sim::p3b_add_hit(s, *D, L, tris[i], h);
      }
    }
    if (job && L.walk_done) sim::p3b_close(s, *D, L);
    RSX_ZONE_END(zc, 35);
  }
  if (have && L.unimplemented != 0) *un = 1;
}

// The wheel rays of car ci of the thread's arena (act) with the mesh leaves of the whole block pooled; every thread of
// the block calls it.  A mesh body's walk reads only the body-local rays' box, and a leaf's evaluation made with the
// starting fractions at 1 serves any later ones (sim/ray.cuh), so each lane first walks every mesh candidate of its
// packet (up to kRayJobsLane bodies, kRayLeavesLane leaves), the block evaluates all those leaves at once, and each
// owner then runs its candidates in order: mesh bodies by replaying their evaluated leaves against the fractions held
// at that point, the plane, ball and car bodies by testing them in place.  One pool round per car; results equal
// vehicle_rays'.  Lanes past the pool's capacity or their own budget run vehicle_rays' sequence.
__device__ __noinline__ void rays_pooled(ArenaState& s, const StaticData* D, bool act, int ci, sim::WheelHit hits[kWheels]) {
  Pools& u = pools();
  RayPoolSmem& sm = u.rays;
  sim::RayPacket pk;
  uint32_t cand[kHandles];
  int nk = 0;
  RSX_ZONE_BEGIN(zr0);
  if (act) {
    sim::vehicle_rays_begin(s, *D, ci, pk);
    nk = sim::grid_candidates(s, *D, &pk, cand);
  }
  uint32_t leaves[kRayLeavesLane];
  uint8_t meshes[kRayLeavesLane], jcand[kRayJobsLane], jstart[kRayJobsLane], jcount[kRayJobsLane];
  int nj = 0, nl = 0;
  bool fits = true;
  RSX_ZONE_BEGIN(zr6);
  for (int k = 0; k < nk && fits; ++k) {
    const uint32_t w = cand[k];
    const uint32_t shape = D->bodies[w].shape;
    if (shape == sim::SHAPE_BOX || shape == sim::SHAPE_SPHERE || shape == sim::SHAPE_PLANE) continue;
    if (nj == kRayJobsLane) {
      fits = false;
      break;
    }
    sim::LocalRays lr;
    sim::RayBox rb;
    sim::ray_body_setup(s, *D, w, &pk, lr, rb);
    sim::RayWalk wk;
    sim::ray_walk_seek(wk, *D, w, rb.box, 0);
    int mesh;
    uint32_t leaf;
    const int first = nl;
    while (sim::ray_walk_next(wk, *D, w, rb.box, &mesh, &leaf)) {
      if (nl == kRayLeavesLane) {
        fits = false;
        break;
      }
      leaves[nl] = leaf;
      meshes[nl] = (uint8_t)mesh;
      ++nl;
    }
    jcand[nj] = (uint8_t)k;
    jstart[nj] = (uint8_t)first;
    jcount[nj] = (uint8_t)(nl - first);
    ++nj;
  }
  RSX_ZONE_END(zr6, 9);
  if (!fits) nj = nl = 0;
  RSX_ZONE_END(zr0, 5);
  RSX_ZONE_BEGIN(zr1);
  uint32_t total;
  const uint32_t ex = block_scan(((uint32_t)nj << 16) | (uint32_t)nl, &total, u);
  const uint32_t slot = ex >> 16, off = ex & 0xFFFFu;
  // all of a lane's bodies or none; pooled lanes are a prefix in scan order
  const bool pooled = nj > 0 && slot + (uint32_t)nj <= (uint32_t)kRayJobs && off + (uint32_t)nl <= (uint32_t)kRayPairs;
  if (pooled) {
    for (int j = 0; j < nj; ++j) {  // no body has been tested yet: the packet's fractions are all still 1
      sim::LocalRays lr;
      sim::RayBox rb;
      sim::ray_body_setup(s, *D, cand[jcand[j]], &pk, lr, rb);
      sim::ray_mesh_job(lr, rb, sm.job[slot + j]);
      sm.jd[slot + j] = D;
      for (int t = 0; t < jcount[j]; ++t) {
        sm.pair_job[off + jstart[j] + t] = (slot + j) | ((uint32_t)meshes[jstart[j] + t] << 16);
        sm.pair_leaf[off + jstart[j] + t] = leaves[jstart[j] + t];
      }
    }
    atomicMax(&u.limit, off + (uint32_t)nl);
  }
  __syncthreads();
  RSX_ZONE_END(zr1, 8);
  RSX_ZONE_BEGIN(zr2);
  const uint32_t npairs = u.limit;
  for (uint32_t p = threadIdx.x; p < npairs; p += blockDim.x) {
    const uint32_t j = sm.pair_job[p] & 0xFFFFu;
    const StaticData& Dj = *sm.jd[j];
    sim::ray_leaf_eval(sm.job[j], Dj, Dj.meshes[sm.pair_job[p] >> 16], sm.pair_leaf[p], nullptr, &sm.out[p]);
  }
  RSX_ZONE_END(zr2, 6);
  RSX_ZONE_BEGIN(zr3);
  __syncthreads();
  RSX_ZONE_END(zr3, 8);
  RSX_ZONE_BEGIN(zr4);
  if (act) {
    int j = 0;
    for (int k = 0; k < nk; ++k) {
      const uint32_t w = cand[k];
      if (pooled && j < nj && jcand[j] == k) {
        sim::LocalRays lr;
        sim::RayBox rb;
        sim::ray_body_setup(s, *D, w, &pk, lr, rb);
        for (int t = 0; t < jcount[j]; ++t) {
          const int q = jstart[j] + t;
          sim::ray_leaf_replay(&lr, rb.lmax, *D, D->meshes[meshes[q]], leaves[q], sm.out[off + q]);
        }
        ++j;
      } else {
        sim::ray_body(s, *D, w, &pk);
      }
    }
    sim::wheel_packet_hits(s, *D, pk, hits);
  }
  RSX_ZONE_END(zr4, 7);
  RSX_ZONE_BEGIN(zr5);
  __syncthreads();  // the pool is read above: the next piece's writes come after every lane's reads
  RSX_ZONE_END(zr5, 8);
}

template <class Lists>
__device__ __forceinline__ void mark_lost(Lists& w, uint32_t q, uint32_t why) {
  atomicOr(&w.lost[q], why);
  LS_COUNT(why == kLostDeep ? kCountDeep : kCountFull);
}
// The levels of a walk and the order of its leaves (split 15; every thread of the block calls it, after a barrier behind
// the jobs' writes).  box(q): job q's box; expand(item, key, level, emit): the children of a front item whose boxes meet
// the job's; keep(entry): whether a leaf entry is kept.  Afterwards each kept leaf's entry is in byjob[seg[q] ..
// seg[q] + cnt[q]) of its job, in no order: rank_of gives its place in the stack walk's order.
template <int JOBS, int FRONT, int LEAVES, class Expand, class Keep>
__device__ __forceinline__ void walk_levels(WalkLists<JOBS, FRONT, LEAVES>& w, Expand&& expand, Keep&& keep) {
  for (int level = 0; level < sim::kWalkLevels; ++level) {
    const uint32_t F = min(w.nfront[level], (uint32_t)FRONT);
    if (F == 0) break;  // (uniform: written only before the barrier above)
    const int cur = level & 1;
    for (uint32_t i = threadIdx.x; i < F; i += blockDim.x) {
      const uint32_t it = w.front[cur][i], head = it & kHeadMask, q = it & kJobMask;
      expand(it, w.fkey[cur][i], level, [&](uint32_t ch, uint32_t key) {
        if (ch & 0x80000000u) {
          const uint32_t entry = head | ((ch & 0x7FFFFFFFu) << kHeadBits);
          if (!keep(entry)) return;
          const uint32_t e = atomicAdd(&w.nleaf, 1u);
          if (e < (uint32_t)LEAVES) {
            w.leaf[e] = entry;
            w.key[e] = (uint16_t)key;
            atomicAdd(&w.cnt[q], 1u);
          } else {
            mark_lost(w, q, kLostFull);
          }
        } else if (level + 1 == sim::kWalkLevels) {
          mark_lost(w, q, kLostDeep);
        } else {
          const uint32_t f = atomicAdd(&w.nfront[level + 1], 1u);
          if (f < (uint32_t)FRONT) {
            w.front[cur ^ 1][f] = head | (ch << kHeadBits);
            w.fkey[cur ^ 1][f] = (uint16_t)key;
          } else {
            mark_lost(w, q, kLostFull);
          }
        }
      });
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) {  // seg: the exclusive prefix sum of cnt
    const uint32_t J = min(w.njobs, (uint32_t)JOBS);
    uint32_t base = 0;
    for (uint32_t q0 = 0; q0 < J; q0 += 32) {
      const uint32_t q = q0 + threadIdx.x, c = q < J ? w.cnt[q] : 0u;
      uint32_t x = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (threadIdx.x >= (uint32_t)d) x += y;
      }
      if (q < J) w.seg[q] = base + x - c;
      base += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
  }
  __syncthreads();
  const uint32_t nl = min(w.nleaf, (uint32_t)LEAVES);
  for (uint32_t e = threadIdx.x; e < nl; e += blockDim.x) {
    const uint32_t q = w.leaf[e] & kJobMask;
    w.byjob[w.seg[q] + atomicAdd(&w.fill[q], 1u)] = (uint16_t)e;
  }
  __syncthreads();
}
// the place of leaf entry e of job q among the block's leaves: its job's segment, then the number of lower keys there
// (a job's keys are distinct: a key is the path to the leaf)
template <class Lists>
__device__ __forceinline__ uint32_t rank_of(const Lists& w, uint32_t e, uint32_t q) {
  const uint32_t b = w.seg[q], n = w.cnt[q], key = w.key[e];
  uint32_t at = b;
  for (uint32_t i = 0; i < n; ++i) at += w.key[w.byjob[b + i]] < key ? 1u : 0u;
  return at;
}
template <class Lists>
__device__ __forceinline__ void lists_clear(Lists& w) {
  for (uint32_t q = threadIdx.x; q < sizeof(w.cnt) / 4; q += blockDim.x) w.cnt[q] = w.fill[q] = w.lost[q] = 0;
  if (threadIdx.x <= (uint32_t)sim::kWalkLevels) w.nfront[threadIdx.x] = 0;
  if (threadIdx.x == 0) w.njobs = w.nleaf = 0;
}

// The wheel rays of both cars of the thread's arena (act[ci]) in one round (split 15); every thread of the block calls
// it.  The rays read poses, flags and static data only, and between car 0's rays and car 1's the tick changes none that
// car 1's rays read: car 0's response writes velocities and wheel states, and car 1's pre-tick head moves a car only when
// it respawns, which casts no rays; so both cars' rays can be cast after car 0's head.  Each lane lists the mesh bodies
// among its candidates as jobs, the block walks them and evaluates their leaves, and each owner runs its candidates in
// order, replaying the mesh ones.  Results equal vehicle_rays'.
// What bounds it: the barriers behind the slowest lane's candidate search and replays, and the walk's levels.  One round
// for both cars pays them once: with a round per car it took 414 thousand cycles a tick, together 316 thousand (65,536
// arenas, 448 threads, of 2.97 and 2.48 million in all).
__device__ __noinline__ void rays_walk_both(ArenaState& s, const StaticData* sds, uint32_t di, bool act0, bool act1, sim::WheelHit hits[kCars][kWheels]) {
  Pools& u = pools();
  RayWalkSmem& sm = u.ray_walk;
  const StaticData* D = sds + di;
  lists_clear(sm.w);
  __syncthreads();
  sim::RayPacket pk[kCars];
  uint32_t cand[kCars][kHandles];
  int nk[kCars] = {0, 0};
  uint32_t jslot[kWalkRayLane];  // job | candidate << 16 | car << 24
  int nj = 0;
  RSX_ZONE_BEGIN(zr0);
#pragma unroll 1
  for (int ci = 0; ci < kCars; ++ci) {
    if (!(ci ? act1 : act0)) continue;
    sim::vehicle_rays_begin(s, *D, ci, pk[ci]);
    nk[ci] = sim::grid_candidates(s, *D, &pk[ci], cand[ci]);
    for (int k = 0; k < nk[ci] && nj < kWalkRayLane; ++k) {
      const uint32_t w = cand[ci][k], shape = D->bodies[w].shape;
      if (shape == sim::SHAPE_BOX || shape == sim::SHAPE_SPHERE || shape == sim::SHAPE_PLANE) continue;
      const uint32_t q = atomicAdd(&sm.w.njobs, 1u);
      if (q >= (uint32_t)kWalkRayJobs) break;  // past the pool: this lane walks the rest itself
      jslot[nj++] = q | ((uint32_t)k << 16) | ((uint32_t)ci << 24);
      sim::LocalRays lr;  // no body has been tested yet: the packet's fractions are all still 1
      sim::RayBox rb;
      sim::ray_body_setup(s, *D, w, &pk[ci], lr, rb);
      sim::ray_mesh_job(lr, rb, sm.job[q]);
      sm.jsd[q] = (uint16_t)di;
      sm.jbox[q] = rb.box;
      sm.jbody[q] = (uint16_t)w;
    }
  }
  RSX_ZONE_END(zr0, 5);
  RSX_ZONE_BEGIN(zr1);
  __syncthreads();
  RSX_ZONE_END(zr1, 8);
  RSX_ZONE_BEGIN(zr6);
  const uint32_t J = min(sm.w.njobs, (uint32_t)kWalkRayJobs);
  if (J != 0) {  // (uniform: written only before the barrier)
    // the jobs' meshes: every mesh of the job's body whose root box meets the job's box, in mesh order by key
    for (uint32_t i = threadIdx.x; i < J * (uint32_t)kMeshes; i += blockDim.x) {
      const uint32_t q = i / (uint32_t)kMeshes;
      const int m = (int)(i % (uint32_t)kMeshes);
      const StaticData& Dj = sds[sm.jsd[q]];
      if (Dj.meshes[m].body == sm.jbody[q] && box_overlap(sm.jbox[q], Dj.meshes[m].root_box)) {
        const uint32_t f = atomicAdd(&sm.w.nfront[0], 1u);
        if (f < (uint32_t)kWalkRayFront) {
          sm.w.front[0][f] = q | ((uint32_t)m << kJobBits);
          sm.w.fkey[0][f] = (uint16_t)sim::walk_root_key(m);
        } else {
          mark_lost(sm.w, q, kLostFull);
        }
      }
    }
    __syncthreads();
    walk_levels(
        sm.w,
        [&](uint32_t it, uint32_t key, int level, auto&& emit) {
          const uint32_t q = it & kJobMask;
          sim::walk_expand(sds[sm.jsd[q]], (int)((it >> kJobBits) & 15u), it >> kHeadBits, key, level, sm.jbox[q], emit);
        },
        [](uint32_t) { return true; });
    RSX_ZONE_END(zr6, 9);
    RSX_ZONE_BEGIN(zr2);
    const uint32_t nl = min(sm.w.nleaf, (uint32_t)kWalkRayLeaves);
    for (uint32_t e = threadIdx.x; e < nl; e += blockDim.x) {
      const uint32_t v = sm.w.leaf[e], q = v & kJobMask, m = (v >> kJobBits) & 15u;
      const uint32_t at = rank_of(sm.w, e, q);
      const StaticData& Dj = sds[sm.jsd[q]];
      sim::ray_leaf_eval(sm.job[q], Dj, Dj.meshes[m], v >> kHeadBits, nullptr, &sm.out[at]);
      sm.at[at] = v >> kJobBits;
    }
    RSX_ZONE_END(zr2, 6);
    RSX_ZONE_BEGIN(zr3);
    __syncthreads();
    RSX_ZONE_END(zr3, 8);
  }
  RSX_ZONE_BEGIN(zr4);
  int j = 0;
#pragma unroll 1
  for (int ci = 0; ci < kCars; ++ci) {
    if (!(ci ? act1 : act0)) continue;
    for (int k = 0; k < nk[ci]; ++k) {
      const uint32_t w = cand[ci][k];
      const uint32_t slot = j < nj ? jslot[j] : ~0u, q = slot & kJobMask;
      if ((slot >> 16) == ((uint32_t)k | ((uint32_t)ci << 8))) {
        ++j;
        if (!sm.w.lost[q]) {
          sim::LocalRays lr;
          sim::RayBox rb;
          sim::ray_body_setup(s, *D, w, &pk[ci], lr, rb);
          const uint32_t b = sm.w.seg[q], n = sm.w.cnt[q];
          for (uint32_t t = 0; t < n; ++t) {
            const uint32_t v = sm.at[b + t];
            sim::ray_leaf_replay(&lr, rb.lmax, *D, D->meshes[v & 15u], v >> 4, sm.out[b + t]);
          }
          continue;
        }
        LS_COUNT(kCountRayAlone);
      }
      sim::ray_body(s, *D, w, &pk[ci]);
    }
    sim::wheel_packet_hits(s, *D, pk[ci], hits[ci]);
  }
  RSX_ZONE_END(zr4, 7);
  RSX_ZONE_BEGIN(zr5);
  __syncthreads();  // the lists are read above: the next piece's writes come after every lane's reads
  RSX_ZONE_END(zr5, 8);
}

__device__ __forceinline__ sim::LeafJob leaf_job(const PairJob& p, const StaticData& D) {
  sim::LeafJob j;
  j.kind = p.kind;
  j.tri_first = D.meshes[p.mesh].tri_first;
  if (p.kind == sim::NEAR_BOX_JOB) {
    const BodyConst& bc = D.bodies[p.body];
    j.box_xf = p.box_xf;
    j.mesh_to_box = p.mesh_to_box;
    j.half = bc.box_half;
    j.margin = bc.box_margin;
    j.maxd = fadd(bc.box_margin, rmin(bc.breaking_threshold, D.bodies[p.mesh].breaking_threshold));
  } else {
    j.center = p.center;
    j.radius = p.radius;
    j.rt = p.rt;
    j.rt2 = p.rt2;
  }
  return j;
}

// P3b of the thread's arena (have) with the tick's mesh jobs found, walked and tested before the pairs run (split 15);
// every thread of the block calls it.  The jobs depend on nothing that P3b changes (sim/narrow.cuh near_peek), so each
// lane lists its pairs' jobs, the block walks all of them level by level and tests their leaves (SAT feature pairs by the
// whole block, kWalkFeat SATs at a time), and each owner then runs its pairs in order, adding the hits of each job it
// opens.  A lane whose next job found no room waits for the next round.
// What bounds it: the slowest lane's pairs, and the barriers around it.  p3b_pooled (split 14) needs a round per mesh pair
// of the arena with the most (4.6 a tick on headline states), each as long as its slowest head and walk: 1,346 thousand
// cycles a tick; here 892 thousand (65,536 arenas).  The lists are sized for a 64 KB carveout, which holds the 131 jobs
// (at most 182 seen), 345 leaves and 39 hits a block has on headline states; twice the lists in 118 KB saved a round on
// contact-heavy states but cost every phase L1 for the arenas' states: 12.55 against 11.7 - 11.9 ms a decision, and 24.0
// against 20.5 - 21.5 ms on the contact-heavy mix.
__device__ __noinline__ void p3b_walk_all(ArenaState& s, const StaticData* sds, uint32_t di, bool have, int* un) {
  Pools& u = pools();
  PairWalkSmem& sm = u.pair_walk;
  const StaticData* D = sds + di;
  sim::P3bLoop L;
  bool more = have;
  if (have) sim::p3b_begin(s, L);
  for (int round = 0;; ++round) {
    uint32_t listed = 0;            // the pairs listed
    lists_clear(sm.w);
    if (threadIdx.x == 0) sm.nsat = sm.nhit = 0;
    RSX_ZONE_BEGIN(zb0);
    __syncthreads();
    RSX_ZONE_END(zb0, 56);
    uint32_t jslot[kWalkPairLane];  // job | pair << 16
    int nj = 0;
    RSX_ZONE_BEGIN(zo);
    if (more) {
      for (uint32_t i = L.kind != sim::NEAR_DONE ? L.i - 1 : L.i; i < L.n && nj < kWalkPairLane; ++i) {
        const Pair p = s.pairs[i];
        sim::BoxJob bj;
        sim::SphereJob sj;
        const int kind = sim::near_peek(s, *D, D->proxies[p.h0].body, D->proxies[p.h1].body, bj, sj);
        if (kind == sim::NEAR_DONE) continue;
        const bool isbox = kind == sim::NEAR_BOX_JOB;
        const uint32_t m = isbox ? bj.mesh_body : sj.mesh_body;
        listed |= 1u << i;
        if ((isbox ? bj.cu.n : sj.cu.n) == 0) continue;  // the mesh's root box is out of reach: no leaves
        const uint32_t q = atomicAdd(&sm.w.njobs, 1u);
        if (q >= (uint32_t)kWalkPairJobs) {
          listed &= ~(1u << i);
          break;
        }
        jslot[nj++] = q | (i << 16);
        PairJob& job = sm.job[q];
        job.kind = (uint8_t)kind;
        job.mesh = (uint8_t)m;
        if (isbox) {
          job.body = (uint8_t)bj.car;
          job.box_xf = bj.box_xf;
          job.mesh_to_box = bj.mesh_to_box;
        } else {
          job.body = (uint8_t)sj.sph;
          job.center = sj.center;
          job.radius = sj.radius;
          job.rt = sj.rt;
          job.rt2 = sj.rt2;
        }
        sm.jsd[q] = (uint16_t)di;
        sm.jbox[q] = isbox ? bj.box : sj.box;
        const uint32_t f = atomicAdd(&sm.w.nfront[0], 1u);
        sm.w.front[0][f] = q | (m << kJobBits);
        sm.w.fkey[0][f] = 0;
      }
    }
    RSX_ZONE_END(zo, 33);
    LS_SYNC(56);
    if (sm.w.njobs != 0) {  // (uniform: written only before the barrier)
      RSX_ZONE_BEGIN(zw);
      walk_levels(
          sm.w,
          [&](uint32_t it, uint32_t key, int level, auto&& emit) {
            const uint32_t q = it & kJobMask;
            sim::walk_expand(sds[sm.jsd[q]], (int)((it >> kJobBits) & 15u), it >> kHeadBits, key, level, sm.jbox[q], emit);
          },
          [&](uint32_t v) {
            const uint32_t q = v & kJobMask;
            if (sm.job[q].kind != sim::NEAR_BOX_JOB) return true;
            const StaticData& Dj = sds[sm.jsd[q]];
            const MeshInfo& m = Dj.meshes[(v >> kJobBits) & 15u];
            return sim::tri_meets_box(Dj.tris[m.tri_first + Dj.leaves[m.leaf_first + (v >> kHeadBits)].tri], sm.jbox[q]);
          });
      RSX_ZONE_END(zw, 36);
      auto put = [&](uint32_t at, uint32_t q, const sim::LeafHit& h) {
        uint32_t i = 0;
        if (h.found) {
          i = atomicAdd(&sm.nhit, 1u) + 1;
          if (i <= (uint32_t)kWalkHits) sm.hit[i - 1] = h;
          else mark_lost(sm.w, q, kLostFull);
        }
        sm.at_hit[at] = (uint16_t)(i <= (uint32_t)kWalkHits ? i : 0u);
      };
      RSX_ZONE_BEGIN(zt);
      const uint32_t nl = min(sm.w.nleaf, (uint32_t)kWalkPairLeaves);
      for (uint32_t e = threadIdx.x; e < nl; e += blockDim.x) {
        const uint32_t v = sm.w.leaf[e], q = v & kJobMask;
        const uint32_t at = rank_of(sm.w, e, q);
        const StaticData& Dj = sds[sm.jsd[q]];
        const uint32_t tri = Dj.leaves[Dj.meshes[(v >> kJobBits) & 15u].leaf_first + (v >> kHeadBits)].tri;
        sm.at_tri[at] = (uint16_t)tri;
        sim::LeafHit h;
        sim::SatFront f;
        if (!sim::leaf_test_front(leaf_job(sm.job[q], Dj), Dj, tri, &h, &f)) {
          const uint32_t d = atomicAdd(&sm.nsat, 1u);
          if (d < (uint32_t)kWalkSats) {  // the block computes its feature pairs below
            sm.front[d] = f;
            sm.front_at[d] = at | (q << 16);
            continue;
          }
          LS_COUNT(kCountSat);
          sim::FeatPair P[sim::kPairs];  // past the list: this thread computes them itself
          sim::enum_pairs(f.hu, f.q, f.e, P);
          sim::leaf_test_back(f, P, &h);
        }
        put(at, q, h);
      }
      RSX_ZONE_END(zt, 34);
      LS_SYNC(56);
      const uint32_t ns = min(sm.nsat, (uint32_t)kWalkSats);
      for (uint32_t d0 = 0; d0 < ns; d0 += (uint32_t)kWalkFeat) {  // (the pairs overlay the job records, which are read by now)
        const uint32_t nd = min(ns - d0, (uint32_t)kWalkFeat);
        RSX_ZONE_BEGIN(zf);
        for (uint32_t w = threadIdx.x; w < nd * (uint32_t)sim::kPairs; w += blockDim.x) {
          const uint32_t d = w / (uint32_t)sim::kPairs, i = w % (uint32_t)sim::kPairs;
          sm.feat[d][i] = sim::feat_pair(sm.front[d0 + d], (int)i);
        }
        RSX_ZONE_END(zf, 34);
        LS_SYNC(56);
        RSX_ZONE_BEGIN(zg);
        for (uint32_t d = threadIdx.x; d < nd; d += blockDim.x) {
          sim::LeafHit h;
          sim::leaf_test_back(sm.front[d0 + d], sm.feat[d], &h);
          put(sm.front_at[d0 + d] & 0xFFFFu, sm.front_at[d0 + d] >> 16, h);
        }
        RSX_ZONE_END(zg, 34);
        LS_SYNC(56);
      }
    }
    RSX_ZONE_BEGIN(zc);
    if (more) {
      more = false;
      for (int j = 0; j < nj; ++j)
        if (sm.w.lost[jslot[j] & kJobMask]) listed &= ~(1u << (jslot[j] >> 16));
      int j = 0;
      while (sim::p3b_open(s, *D, L, listed) != sim::NEAR_DONE) {
        const uint32_t pair = L.i - 1;
        while (j < nj && (jslot[j] >> 16) < pair) ++j;
        const bool has = j < nj && (jslot[j] >> 16) == pair;
        if ((listed >> pair) & 1u) {
          if (has) {
            const uint32_t q = jslot[j] & kJobMask, b = sm.w.seg[q], n = sm.w.cnt[q];
            for (uint32_t t = 0; t < n; ++t) {
              const uint32_t i = sm.at_hit[b + t];
              if (i != 0) sim::p3b_add_hit(s, *D, L, sm.at_tri[b + t], sm.hit[i - 1]);
            }
          }
          L.walk_done = true;
          sim::p3b_close(s, *D, L);
        } else if (has && (round >= kWalkPairRounds || (sm.w.lost[jslot[j] & kJobMask] & kLostDeep))) {  // (no round holds a deep tree)
          LS_COUNT(kCountAlone);
          sim::p3b_job_alone(s, *D, L);
        } else {  // its job found no room: the next round
          LS_COUNT(kCountWait);
          more = true;
          break;
        }
      }
    }
    RSX_ZONE_END(zc, 35);
    RSX_ZONE_BEGIN(zd);
    const bool again = __syncthreads_or(more);  // (the lists are read above)
    RSX_ZONE_END(zd, 56);
    if (!again) break;
  }
  if (have && L.unimplemented != 0) *un = 1;
}

}  // namespace

template <int SPLIT>
__global__ void __launch_bounds__(RSX_LS_MAXT, 1) K_NAME(uint32_t* states, const StaticData* sds, const uint8_t* sd_index,
                                                        const Controls* controls, uint32_t* result, uint32_t* ev_or,
                                                        const uint32_t* order, uint32_t* counter, uint32_t n, uint32_t width,
                                                        uint32_t t_first, uint32_t t_last) {
  const uint32_t lane = threadIdx.x & 31u;
  ArenaState s;
  Controls c0, c1;
  const StaticData* D = sds;
  uint32_t a = 0, di = 0, t = 0, scored = 0, unimpl = 0, ev = 0;
  // without a queue the claims are dealt out evenly: split 15 over the identity order each block's in a row (neighbouring
  // arenas on one SM: 2% faster at 65,536 arenas than the blocks in turn; the splits below 9 are up to 9% slower so), else
  // the blocks in turn (another order's costliest arenas come first)
  const bool rows = SPLIT >= 15 && !order;
  const uint32_t nw = blockDim.x >> 5, warp = threadIdx.x >> 5, claims = (n + width - 1) / width;
  const uint32_t first = rows ? (uint32_t)((uint64_t)claims * blockIdx.x / gridDim.x) : blockIdx.x, step = rows ? 1u : gridDim.x;
  const uint32_t end = rows ? (uint32_t)((uint64_t)claims * (blockIdx.x + 1) / gridDim.x) : claims;
  uint32_t next = first + warp * step;
  bool busy = false;               // the warp holds a claim (uniform over the warp)
  bool have = false, live = false, ovf = false;  // the lane steps an arena, which is its own
  for (;;) {
    // a warp without arenas claims its next ones
    if (!busy) {
      uint32_t base = 0;
      if (lane == 0) {
        if (counter) {
          base = atomicAdd(counter, width);
        } else {
          base = next < end ? next * width : n;
          next += nw * step;
        }
      }
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base < n) {
        busy = true;
        t = t_first;
        // A lane past the claim's arenas, or at an order entry past n (not a permutation): where the block pools its work it
        // steps nothing (a copy's jobs would fill the pools); else it steps a copy of its warp's first arena and stores
        // nothing, so that the branches on `have` are uniform over a warp, for the compiler too (65,536 arenas, splits 1 and
        // 7: 3 - 4% faster).
        const uint32_t i = base + lane;
        a = lane < width && i < n ? (order ? order[i] : i) : n;
        live = a < n;
        have = live;
        if (SPLIT < 9) {
          const uint32_t own = __ballot_sync(0xFFFFFFFFu, live);
          const uint32_t first_a = __shfl_sync(0xFFFFFFFFu, a, __ffs(own) - 1);
          if (!live) a = first_a;
          have = own != 0;
        }
        if (have) {
          di = sd_index ? sd_index[a] : 0;
          D = sds + di;
          RSX_ZONE_BEGIN(zl);
          load_tick(&s, states, a);
          RSX_ZONE_END(zl, 60);
          c0 = controls[(size_t)a * kCars];
          c1 = controls[(size_t)a * kCars + 1];
          scored = unimpl = ev = 0;
          if (t_first > 1) {  // a later launch of a split decision: the progress so far rides in the result / event words
            uint32_t r0 = result[a];
            scored = r0 & kScoredMask;
            unimpl = r0 & kUnimplemented;
            ev = ev_or ? ev_or[a] : 0u;
            if (scored) {  // decided in an earlier launch: the buffer holds its goal state
              live = false;
              if (SPLIT >= 9) have = false;
            }
          }
          ovf = false;
        }
      }
    }
    if (!__syncthreads_or(busy)) break;
    // one tick, phase by phase in lockstep (every thread reaches every barrier)
    int un = 0;
    if (have) {
      s.cars[0].controls = c0;
      s.cars[1].controls = c1;
    }
    if (SPLIT >= 2) {
      {
        RSX_ZONE_BEGIN(z0);
        if (have) sim::t_p0(s, *D);
        RSX_ZONE_END(z0, 40);
      }
      LS_SYNC(50);
      if (have) {
        sim::flip_zdamp(s, *D, 0);
        sim::flip_zdamp(s, *D, 1);
      }
      if (SPLIT >= 15) {
        // P1: car 0's head, both cars' wheel rays, car 0's response, car 1's head and response
        bool act0 = false, act1 = false;
        float thr0 = 0.0f, thr1 = 0.0f;
        uint32_t was0 = 0, was1 = 0;
        {
          RSX_ZONE_BEGIN(z1);
          if (have) {
            was0 = s.cars[0].on_ground;
            act1 = !s.cars[1].is_demoed;
            act0 = sim::car_pre_tick_head(s, *D, 0, &thr0);
          }
          RSX_ZONE_END(z1, 41);
        }
        LS_SYNC(51);
        sim::WheelHit hits[kCars][kWheels];
        {
          RSX_ZONE_BEGIN(z2);
          rays_walk_both(s, sds, di, act0, act1, hits);
          RSX_ZONE_END(z2, 42);
        }
#pragma unroll 1
        for (int ci = 0; ci < kCars; ++ci) {
          if (ci) {
            RSX_ZONE_BEGIN(z1);
            if (have) {
              was1 = s.cars[1].on_ground;
              act1 = sim::car_pre_tick_head(s, *D, 1, &thr1);
            }
            RSX_ZONE_END(z1, 41);
            LS_SYNC(51);
          }
          RSX_ZONE_BEGIN(z3);
          if (have) {
            if (ci ? act1 : act0) {
              sim::vehicle_response(s, *D, ci, sim::kTickTime, s.cars[ci].handbrake_val, ci ? thr1 : thr0, D->cars[ci].three_wheels != 0, hits[ci]);
              sim::car_pre_tick_tail(s, *D, ci);
            }
            if (!(ci ? was1 : was0) && s.cars[ci].on_ground) s.events |= 1u << (EV_LANDED + ci);
          }
          RSX_ZONE_END(z3, 43);
          LS_SYNC(53);
        }
      } else
#pragma unroll 1
      for (int ci = 0; ci < kCars; ++ci) {
        // P1 for car ci in three barrier-separated parts: pre-tick head, wheel rays, wheel response + tail
        bool act = false;
        float rthr = 0.0f;
        uint32_t was = 0;
        RSX_ZONE_BEGIN(z1);
        if (SPLIT == 8) {  // the pre-tick head in three parts
          sim::PreTick pt;
          if (have) {
            was = s.cars[ci].on_ground;
            act = sim::car_pre_tick_wheels(s, *D, ci, pt);
          }
          __syncthreads();
          if (have && act) sim::car_pre_tick_jumps(s, *D, ci, pt);
          __syncthreads();
          if (have && act) rthr = sim::car_pre_tick_air(s, *D, ci, pt);
        } else if (have) {
          was = s.cars[ci].on_ground;
          act = sim::car_pre_tick_head(s, *D, ci, &rthr);
        }
        RSX_ZONE_END(z1, 41);
        LS_SYNC(51);
        sim::WheelHit hits[kWheels];
        {
          RSX_ZONE_BEGIN(z2);
          if (SPLIT >= 10)
            rays_pooled(s, D, have && act, ci, hits);
          else if (have && act)
            sim::vehicle_rays(s, *D, ci, hits);
          RSX_ZONE_END(z2, 42);
        }
        LS_SYNC(52);
        {
          RSX_ZONE_BEGIN(z3);
          if (have) {
            if (act) {
              sim::vehicle_response(s, *D, ci, sim::kTickTime, s.cars[ci].handbrake_val, rthr, D->cars[ci].three_wheels != 0, hits);
              sim::car_pre_tick_tail(s, *D, ci);
            }
            if (!was && s.cars[ci].on_ground) s.events |= 1u << (EV_LANDED + ci);
          }
          RSX_ZONE_END(z3, 43);
        }
        LS_SYNC(53);
      }
#pragma unroll 1
      for (int k = 2; k < sim::kPhases; ++k) {
        // split 4: no barrier between P3b and P8 (warps without contact work run ahead to the tick's end);
        // split 5: none between P4 and P8
        const bool bar = !((SPLIT == 4 && k >= 4 && k < sim::kPhases - 1) || (SPLIT == 5 && k >= 5 && k < sim::kPhases - 1));
        // zone ids of phase k's pieces and of the barriers after them
        const int zp = k <= 7 ? 42 + k : 21 + k, zb = zp + (k <= 7 ? 10 : 2);
        (void)zp;
        (void)zb;
        if (SPLIT >= 7 && SPLIT < 11 && k == 3) {  // P3a: one dynamic body at a time (from split 11: one piece)
#pragma unroll 1
          for (uint32_t d = 0; d < (uint32_t)kDyn; ++d) {
            {
              RSX_ZONE_BEGIN(za);
              if (have) sim::t_p3a_body(s, *D, d);
              RSX_ZONE_END(za, zp);
            }
            LS_SYNC(zb);
          }
          continue;
        }
        if (SPLIT >= 6 && k == 6) {  // P5: rows, iterations, integration
          sim::Solver sv;
          RSX_ZONE_BEGIN(z5a);
          if (have) sim::t_p5_setup(s, *D, sv);
          RSX_ZONE_END(z5a, zp);
          LS_SYNC(zb);
          RSX_ZONE_BEGIN(z5b);
          if (have) sim::t_p5_iterate(sv);
          RSX_ZONE_END(z5b, zp);
          LS_SYNC(zb);
          RSX_ZONE_BEGIN(z5c);
          if (have) sim::t_p5_finish(s, *D, sv);
          RSX_ZONE_END(z5c, zp);
          LS_SYNC(zb);
          continue;
        }
        if (SPLIT >= 6 && k == 9) {  // P8: cars, then pads / ball / tick count
          RSX_ZONE_BEGIN(z8a);
          if (have) sim::t_p8_cars(s);
          RSX_ZONE_END(z8a, zp);
          LS_SYNC(zb);
          RSX_ZONE_BEGIN(z8b);
          if (have) sim::t_p8_rest(s, *D);
          RSX_ZONE_END(z8b, zp);
          LS_SYNC(zb);
          continue;
        }
        if (SPLIT == 4 || SPLIT == 5) {
          if (have && sim::run_phase(k, s, *D) != sim::PHASE_OK) un = 1;
          if (bar) __syncthreads();
          continue;
        }
        if (SPLIT >= 9 && k == 4) {  // P3b with the block's leaf tests pooled
          if (SPLIT >= 15)
            p3b_walk_all(s, sds, di, have, &un);
          else
            p3b_pooled<(SPLIT >= 14)>(s, D, have, &un);
          continue;
        }
        if (SPLIT == 3 && k == 4) {
          // P3b with a barrier after every step of the pair / leaf loop
          sim::P3bLoop L;
          bool more = have;
          if (have) sim::p3b_begin(s, L);
          while (__syncthreads_or(more))
            if (more) more = sim::t_p3b_step(s, *D, L);
          if (have && L.unimplemented != 0) un = 1;
          continue;
        }
        {
          RSX_ZONE_BEGIN(zk);
          if (have && sim::run_phase(k, s, *D) != sim::PHASE_OK) un = 1;
          RSX_ZONE_END(zk, zp);
        }
        LS_SYNC(zb);
      }
    } else if (SPLIT) {
      if (have) sim::t_p0(s, *D);
      __syncthreads();
      if (have) {
        sim::flip_zdamp(s, *D, 0);
        sim::flip_zdamp(s, *D, 1);
      }
#pragma unroll 1
      for (int ci = 0; ci < kCars; ++ci) {
        if (have) {
          uint32_t was = s.cars[ci].on_ground;
          sim::car_pre_tick(s, *D, ci);
          if (!was && s.cars[ci].on_ground) s.events |= 1u << (EV_LANDED + ci);
        }
        __syncthreads();
      }
#pragma unroll 1
      for (int k = 2; k < sim::kPhases; ++k) {
        if (have && sim::run_phase(k, s, *D) != sim::PHASE_OK) un = 1;
        __syncthreads();
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < sim::kPhases; ++k) {
        if (have && sim::run_phase(k, s, *D) != sim::PHASE_OK) un = 1;
        __syncthreads();
      }
    }
    // the tick hooks of decide(): event OR, goal state, and the end of the decision
    if (have) {
      if (scored == 0) {
        if (un) unimpl = kUnimplemented;
        ev |= s.events;
        if (sim::ball_scored(s, *D)) {
          scored = t;
          if (live) store_tick(states, a, &s);
          ovf = sim::any_overflow(s);
        }
      }
      if (t == t_last) {  // the end of this launch's ticks (tick 8: of the decision)
        RSX_ZONE_BEGIN(zs);
        if (scored == 0) {
          if (live) store_tick(states, a, &s);
          ovf = sim::any_overflow(s);
        }
        RSX_ZONE_END(zs, 61);
        if (live) {
          if (ev_or) ev_or[a] = ev;
          result[a] = scored | unimpl | (ovf ? kOverflow : 0u);
        }
      }
    }
    if (busy && t++ == t_last) busy = have = false;
  }
}

using Kernel = void (*)(uint32_t*, const StaticData*, const uint8_t*, const Controls*, uint32_t*, uint32_t*, const uint32_t*, uint32_t*,
                        uint32_t, uint32_t, uint32_t, uint32_t);
static Kernel kernel_of(int split) {
  switch (split) {
    case 15: return K_NAME<15>;
#ifndef RSX_LS_WIDE_REGS
    case 14: return K_NAME<14>;
    case 11: return K_NAME<11>;
    case 10: return K_NAME<10>;
    case 9: return K_NAME<9>;
    case 8: return K_NAME<8>;
    case 7: return K_NAME<7>;
    case 6: return K_NAME<6>;
    case 5: return K_NAME<5>;
    case 4: return K_NAME<4>;
    case 3: return K_NAME<3>;
    case 2: return K_NAME<2>;
    case 1: return K_NAME<1>;
    case 0: return K_NAME<0>;
#endif
    default: return nullptr;
  }
}
static size_t pool_bytes(int split) { return split >= 9 ? sizeof(Pools) : 0; }
static cudaError_t allow_pool(Kernel k, size_t pool) {
  return pool ? cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pool) : cudaSuccess;
}

cudaError_t L_NAME(uint32_t* states, const void* sds, const uint8_t* sd_index, const void* controls, uint32_t* result, uint32_t* ev_or,
                   const uint32_t* order, uint32_t* counter, uint32_t n, uint32_t width, uint32_t grid, uint32_t block, int split,
                   uint32_t t_first, uint32_t t_last, cudaStream_t s) {
  const Kernel k = kernel_of(split);
  if (!k) return cudaErrorInvalidValue;
  const size_t pool = pool_bytes(split);
  const cudaError_t e = allow_pool(k, pool);
  if (e != cudaSuccess) return e;
  k<<<grid, block, pool, s>>>(states, (const StaticData*)sds, sd_index, (const Controls*)controls, result, ev_or, order, counter, n, width,
                              t_first, t_last);
  return cudaGetLastError();
}

// how many blocks of `block` threads of the split's kernel one SM of the current device holds at once
cudaError_t RSX_CAT(rsx_lockstep_blocks_per_sm_t, RSX_LS_MAXT)(int split, uint32_t block, int* blocks) {
  const Kernel k = kernel_of(split);
  if (!k) return cudaErrorInvalidValue;
  const size_t pool = pool_bytes(split);
  const cudaError_t e = allow_pool(k, pool);
  return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, (int)block, pool);
}

#ifdef RSX_ZONES
// Zone-timer profiling build (not part of librsx.so): one decision of this kernel with zone sums over all warps.
__device__ unsigned long long rsx_zone_acc[148 * 16][64];
extern "C" int rsx_zones_lockstep(uint32_t* d_states, uint32_t n, const void* d_statics, const uint8_t* d_sd_index, const void* d_controls,
                                  uint32_t* d_result, uint32_t* d_counter, uint32_t block, int split, unsigned long long* zone_cycles) {
  static unsigned long long acc[148 * 16][64];
  memset(acc, 0, sizeof(acc));
  if (cudaMemcpyToSymbol(rsx_zone_acc, acc, sizeof(acc)) != cudaSuccess) return -2;
  if (cudaMemset(d_counter, 0, 4) != cudaSuccess) return -2;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
  if (L_NAME(d_states, d_statics, d_sd_index, d_controls, d_result, nullptr, nullptr, d_counter, n, 32, sms < 148 ? sms : 148, block, split, 1,
             kTicksPerDecision, 0) != cudaSuccess)
    return -2;
  if (cudaDeviceSynchronize() != cudaSuccess) return -2;
  if (cudaMemcpyFromSymbol(acc, rsx_zone_acc, sizeof(acc)) != cudaSuccess) return -2;
  for (int z = 0; z < 64; ++z) {
    zone_cycles[z] = 0;
    for (int w = 0; w < 148 * 16; ++w) zone_cycles[z] += acc[w][z];
  }
  return 0;
}
#endif
