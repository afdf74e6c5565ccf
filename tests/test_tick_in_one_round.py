"""The orders in which the lockstep kernel's split 15 runs a tick's pieces, arena by arena on the host build, against the
phases they replace, word for word on contact-rich play with demolitions and respawns: both cars' wheel rays before car
0's response (P1), and P3b with its mesh jobs found, walked level by level and tested before any pair runs.  On the same
play P3a's sort, which every split shares, against its rule restated one step at a time (one loop per end and direction)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rocketsim-cuda_b200", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <cstdint>
#include <vector>
#include "state.cuh"
#include "sim/physics.cuh"
using namespace rsx;
using namespace rsx::sim;
extern "C" int rsx_build_static(uint32_t* words, uint64_t seed, int p0, int p1);
extern "C" int rsx_make_states_multi(const uint32_t* sds, uint32_t count, const uint8_t* idx, uint32_t* out, uint32_t n,
                                     uint64_t seed, const float* mix);
// P1 with both cars' rays after car 0's head
static bool p1_both(ArenaState& S, const StaticData& D) {
  flip_zdamp(S, D, 0);
  flip_zdamp(S, D, 1);
  float thr[2] = {0.0f, 0.0f};
  WheelHit hits[2][kWheels];
  const uint32_t was0 = S.cars[0].on_ground;
  const bool act1 = !S.cars[1].is_demoed;
  const bool act0 = car_pre_tick_head(S, D, 0, &thr[0]);
  if (act0) vehicle_rays(S, D, 0, hits[0]);
  if (act1) vehicle_rays(S, D, 1, hits[1]);
  bool same = true;
  for (int ci = 0; ci < 2; ++ci) {
    bool act = act0;
    uint32_t was = was0;
    if (ci) {
      was = S.cars[1].on_ground;
      act = car_pre_tick_head(S, D, 1, &thr[1]);
      same = act == act1;
    }
    if (act) {
      vehicle_response(S, D, ci, kTickTime, S.cars[ci].handbrake_val, thr[ci], D.cars[ci].three_wheels != 0, hits[ci]);
      car_pre_tick_tail(S, D, ci);
    }
    if (!was && S.cars[ci].on_ground) S.events |= 1u << (EV_LANDED + ci);
  }
  return same;
}
// one end of a handle past its neighbours, one step at a time (the sort's rule)
static void pass(ArenaState& S, const StaticData& D, int axis, uint32_t at, bool up, bool min_edge, long* passed) {
  Edge* e = S.edges[axis];
  const uint32_t moving = e[at].handle;
  while (up ? at + 1 < (uint32_t)kEdges && e[at + 1].handle != 0 && e[at].pos >= e[at + 1].pos : at > 0 && e[at].pos < e[at - 1].pos) {
    const uint32_t to = up ? at + 1 : at - 1, other = e[to].handle;
    const bool other_max = is_max_edge(e[to]);
    const int d = up ? -1 : 1;
    if (other_max == min_edge && overlap2d(S, moving, other, axis)) {
      if (min_edge ? !up : up) add_pair(S, D, moving, other);
      else remove_pair(S, D, moving, other);
    }
    if (other_max) S.handle_edges[other].hi[axis] = (uint16_t)(S.handle_edges[other].hi[axis] + d);
    else S.handle_edges[other].lo[axis] = (uint16_t)(S.handle_edges[other].lo[axis] + d);
    if (min_edge) S.handle_edges[moving].lo[axis] = (uint16_t)(S.handle_edges[moving].lo[axis] - d);
    else S.handle_edges[moving].hi[axis] = (uint16_t)(S.handle_edges[moving].hi[axis] - d);
    std::swap(e[at], e[to]);
    at = to;
    ++*passed;
  }
}
static void axes_plain(ArenaState& S, const StaticData& D, uint32_t h, const uint16_t qmin[3], const uint16_t qmax[3], long* passed) {
  for (int ax = 0; ax < 3; ++ax) {
    Edge* e = S.edges[ax];
    const uint32_t mi = S.handle_edges[h].lo[ax], ma = S.handle_edges[h].hi[ax];
    const int dmin = (int)qmin[ax] - (int)e[mi].pos, dmax = (int)qmax[ax] - (int)e[ma].pos;
    if (dmin == 0 && dmax == 0) continue;
    e[mi].pos = qmin[ax];
    e[ma].pos = qmax[ax];
    if (dmin < 0) pass(S, D, ax, mi, false, true, passed);
    if (dmax > 0) pass(S, D, ax, ma, true, false, passed);
    if (dmin > 0) pass(S, D, ax, mi, true, true, passed);
    if (dmax < 0) pass(S, D, ax, ma, false, false, passed);
  }
}
// P3b with its mesh jobs found first; pairs whose bit is set in `drop` find no room and are done by their owner alone
static uint32_t p3b_found(ArenaState& S, const StaticData& D, uint32_t drop, long* jobs, long* hits) {
  struct Found { uint32_t pair; std::vector<uint32_t> tri; std::vector<LeafHit> hit; };
  std::vector<Found> found;
  P3bLoop L;
  p3b_begin(S, L);
  uint32_t listed = 0;
  for (uint32_t i = 0; i < L.n; ++i) {
    P3bLoop J;
    J.kind = near_peek(S, D, D.proxies[S.pairs[i].h0].body, D.proxies[S.pairs[i].h1].body, J.bj, J.sj);
    if (J.kind == NEAR_DONE || ((drop >> i) & 1u)) continue;
    const bool box = J.kind == NEAR_BOX_JOB;
    listed |= 1u << i;
    if ((box ? J.bj.cu.n : J.sj.cu.n) == 0) continue;
    ++*jobs;
    const uint32_t m = box ? J.bj.mesh_body : J.sj.mesh_body;
    const Box3& b = box ? J.bj.box : J.sj.box;
    std::vector<std::pair<uint32_t, uint32_t>> front = {{0u, 0u}}, next, leaves;  // key, node or leaf
    for (int level = 0; level < kWalkLevels && !front.empty(); ++level) {
      next.clear();
      for (auto& f : front)
        walk_expand(D, (int)m, f.second, f.first, level, b, [&](uint32_t ch, uint32_t key) {
          if (ch & 0x80000000u) leaves.push_back({key, ch & 0x7FFFFFFFu});
          else next.push_back({key, ch});
        });
      front.swap(next);
    }
    std::sort(leaves.begin(), leaves.end());
    LeafJob job;
    leaf_job_of(J, job);
    Found f;
    f.pair = i;
    for (auto& l : leaves) {
      const uint32_t tri = D.leaves[D.meshes[m].leaf_first + l.second].tri;
      if (box && !tri_meets_box(D.tris[D.meshes[m].tri_first + tri], b)) continue;
      LeafHit h;
      if (leaf_test(job, D, tri, &h)) {
        f.tri.push_back(tri);
        f.hit.push_back(h);
        ++*hits;
      }
    }
    found.push_back(f);
  }
  while (p3b_open(S, D, L, listed) != NEAR_DONE) {
    const uint32_t pair = L.i - 1;
    if (!((listed >> pair) & 1u)) {
      p3b_job_alone(S, D, L);
      continue;
    }
    for (auto& f : found)
      if (f.pair == pair)
        for (size_t k = 0; k < f.tri.size(); ++k) p3b_add_hit(S, D, L, f.tri[k], f.hit[k]);
    L.walk_done = true;
    p3b_close(S, D, L);
  }
  return L.unimplemented;
}
int main() {
  const int n = 1536, ticks = 120;
  std::vector<uint32_t> sds((size_t)49 * kStaticWords);
  for (int p = 0; p < 7; ++p)
    for (int q = 0; q < 7; ++q) rsx_build_static(&sds[(size_t)(p * 7 + q) * kStaticWords], 7, p, q);
  std::vector<uint8_t> idx(n);
  for (int a = 0; a < n; ++a) idx[a] = (uint8_t)((a * 37u + 11u) % 49u);
  std::vector<uint32_t> st((size_t)n * kArenaWords);
  const float mix[5] = {0.1f, 0.2f, 0.2f, 0.4f, 0.1f};
  rsx_make_states_multi(sds.data(), 49, idx.data(), st.data(), n, 11, mix);
  long bad1 = 0, bad3 = 0, bad3b = 0, passed = 0, jobs = 0, hits = 0, demos = 0;
  ArenaState* T = new ArenaState;
  for (int a = 0; a < n; ++a) {
    ArenaState& S = *reinterpret_cast<ArenaState*>(&st[(size_t)a * kArenaWords]);
    const StaticData& D = *reinterpret_cast<const StaticData*>(&sds[(size_t)idx[a] * kStaticWords]);
    for (int t = 0; t < ticks; ++t) {
      for (int c = 0; c < 2; ++c) {
        Controls& k = S.cars[c].controls;
        k.throttle = (float)(((a + t / 7 + c) % 3) - 1);
        k.steer = (float)(((a * 7 + t / 3 + c) % 3) - 1);
        k.jump = ((a + t / 5 + c) % 4) == 0;
        k.boost = ((a + t / 2) % 3) == 0;
        if ((a * 13 + t + c * 29) % 61 == 0 && !S.cars[c].is_demoed) {  // a demolition, its respawn a few ticks later
          S.cars[c].is_demoed = 1;
          S.cars[c].demo_respawn_timer = 3.0f / 120.0f;
          ++demos;
        }
      }
      t_p0(S, D);
      std::memcpy(T, &S, sizeof S);
      t_p1(S, D);
      if (!p1_both(*T, D) || std::memcmp(T, &S, sizeof S) != 0) ++bad1;
      t_p2(S, D);
      std::memcpy(T, &S, sizeof S);
      for (uint32_t d = 0; d < (uint32_t)kDyn; ++d) {
        phase3a_body(S, D, d);
        const uint32_t h = D.dyn_handle[d];
        if (S.bodies[d].flags & CF_STATIC) continue;
        uint16_t qmin[3], qmax[3];
        quantize_point(D, S.dyn_proxy[d].box.lo, 0, qmin);
        quantize_point(D, S.dyn_proxy[d].box.hi, 1, qmax);
        axes_plain(*T, D, h, qmin, qmax, &passed);
        if (std::memcmp(T->edges, S.edges, sizeof S.edges) != 0 || std::memcmp(T->handle_edges, S.handle_edges, sizeof S.handle_edges) != 0 ||
            T->n_pairs != S.n_pairs || std::memcmp(T->pairs, S.pairs, sizeof S.pairs) != 0 ||
            std::memcmp(T->manifolds, S.manifolds, sizeof S.manifolds) != 0 || T->n_manifolds != S.n_manifolds)
          ++bad3;
      }
      std::memcpy(T, &S, sizeof S);
      const uint32_t u0 = t_p3b(S, D), u1 = p3b_found(*T, D, (a + t) % 3 == 0 ? 0x5555u << ((a + t) & 1) : 0u, &jobs, &hits);
      if (u0 != u1 || std::memcmp(T, &S, sizeof S) != 0) ++bad3b;
      t_p4(S, D); t_p5(S, D); t_p6(S, D); t_p7(S, D); t_p8(S, D);
    }
  }
  std::printf("demos %ld passed %ld jobs %ld hits %ld mismatches %ld %ld %ld\n", demos, passed, jobs, hits, bad1, bad3, bad3b);
  return bad1 + bad3 + bad3b != 0;
}
"""


def test_tick_orders_equal_the_phases(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    libdir = os.path.join(ROOT, "rocketsim-cuda_b200")
    if not os.path.exists(os.path.join(libdir, "librsx.so")):
        pytest.skip("librsx.so is not built")
    src = tmp_path / "tick_orders.cpp"
    exe = tmp_path / "tick_orders"
    src.write_text(PROGRAM)
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-L", libdir, "-lrsx", f"-Wl,-rpath,{libdir}",
           "-o", str(exe)]
    cuda_lib = "/usr/local/cuda/lib64"
    if os.path.isdir(cuda_lib):
        cmd[-2:-2] = ["-L", cuda_lib, f"-Wl,-rpath,{cuda_lib}"]
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    words = out.stdout.split()
    for name in ("demos", "passed", "jobs", "hits"):  # each path is exercised
        assert int(words[words.index(name) + 1]) > 500, out.stdout
