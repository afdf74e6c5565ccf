"""The launch shapes of the decision by size (one lane per SM, the lockstep kernel's register budgets, one round dealt
out or several from the queue, narrow claims) at the sizes where the shape changes, the lockstep kernel's lists past their
capacity and trees deeper than its walks hold: the words, results and events of the persistent kernel without barriers,
which steps each arena on one lane (every word the same, no tolerance)."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 148


class Arenas:
    """n contact-heavy arenas of two car pairings, made on the device, and a reference decision of them."""

    def __init__(self, rsx, dev, n, pairings=2, change=None):
        """change: applied to each pairing's StaticData words."""
        import torch

        self.t, self.rsx, self.dev, self.n = torch, rsx, dev, n
        L = self.L = rsx.lib()
        statics = np.stack([rsx.build_static(7, p, q) for p, q in [(0, 0), (2, 6)][:pairings]])
        if change:
            for words in statics:
                change(words)
        self.sd = dev.upload_static(statics)
        self.idx = (torch.arange(n, device=dev.device) % pairings).to(torch.uint8)
        self.ctl = dev.upload_controls(rsx.random_controls(np.random.default_rng(n), n))
        self.counter = torch.zeros(1, dtype=torch.int32, device=dev.device)
        self.ds = dev.alloc_states(n)
        self.words = rsx.aosoa_words(n)
        self.start = torch.empty(self.words, dtype=torch.int32, device=dev.device)
        torch.cuda.synchronize()
        mix = (ctypes.c_float * 5)(*rsx.MIX_CONTACT_HEAVY)
        rsx.check(L.rsx_reset_arenas_raw(self.ds.ptr(), n, self.sd.ptr(), self.idx.data_ptr(), 3, mix, None, None, None, dev.stream_ptr()), "reset")
        self.reference()
        self.reference()  # the states two decisions in
        rsx.check(L.rsx_copy_raw(self.start.data_ptr(), self.ds.ptr(), self.words * 4, dev.stream_ptr()), "copy")
        self.want = self.step(self.reference)

    def outputs(self):
        self.res = self.t.full((self.n,), -1, dtype=self.t.int32, device=self.dev.device)
        self.ev = self.t.full((self.n,), -1, dtype=self.t.int32, device=self.dev.device)
        self.t.cuda.synchronize()

    def reference(self):
        self.outputs()
        self.rsx.check(self.L.rsx_sim8_persistent_raw(self.ds.ptr(), self.n, self.sd.ptr(), self.idx.data_ptr(), self.ctl.data_ptr(),
                                                      self.res.data_ptr(), self.ev.data_ptr(), None, self.counter.data_ptr(), SMS * 4, 64, 1,
                                                      self.dev.stream_ptr()), "persistent")

    def step(self, f):
        self.rsx.check(self.L.rsx_copy_raw(self.ds.ptr(), self.start.data_ptr(), self.words * 4, self.dev.stream_ptr()), "copy")
        self.outputs()
        f()
        out = self.t.empty(self.words, dtype=self.t.int32, device=self.dev.device)
        self.rsx.check(self.L.rsx_copy_raw(out.data_ptr(), self.ds.ptr(), self.words * 4, self.dev.stream_ptr()), "copy")
        self.dev.sync()
        return out, self.res.clone(), self.ev.clone()

    def same(self, f, events=True):
        got = self.step(f)
        for g, w, name in zip(got, self.want, ("states", "results", "events")):
            assert (name == "events" and not events) or self.t.equal(g, w), name

    def multi(self, block=32):
        self.rsx.check(self.L.rsx_sim8_multi_raw(self.ds.ptr(), self.n, self.sd.ptr(), self.idx.data_ptr(), self.ctl.data_ptr(),
                                                 self.res.data_ptr(), self.ev.data_ptr(), block, self.dev.stream_ptr()), "multi")

    def sim8(self):
        self.rsx.check(self.L.rsx_sim8_raw(self.ds.ptr(), self.n, self.sd.ptr(), self.ctl.data_ptr(), self.res.data_ptr(), 32, None,
                                           self.dev.stream_ptr()), "sim8")

    def lockstep(self, grid=SMS, block=448, order=None, ticks=8, split=15):
        self.rsx.check(self.L.rsx_sim8_lockstep_ex(self.ds.ptr(), self.n, self.sd.ptr(), self.idx.data_ptr(), self.ctl.data_ptr(),
                                                   self.res.data_ptr(), self.ev.data_ptr(), order, self.counter.data_ptr(), grid, block, split,
                                                   ticks, self.dev.stream_ptr()), "lockstep")

    def free(self):
        self.dev.sync()
        self.ds.free()
        self.sd.free()


@pytest.fixture(scope="module")
def dev(rsx):
    d = rsx.SimDevice(0)
    yield d
    d.close()


# one lane per SM up to SMS / 8; claims of 1 up to 3 arenas a block, then as wide as the block's share, 32 from there; 256
# threads up to 256 a block
@pytest.mark.parametrize("n", [1, SMS // 8, SMS // 8 + 1, 3 * SMS, 3 * SMS + 1, 31 * SMS + 5, 32 * SMS + 1, 64 * SMS + 33])
def test_one_launch_decisions(rsx, dev, n):
    a = Arenas(rsx, dev, n)
    a.same(a.multi)
    a.same(a.lockstep)
    a.free()
    b = Arenas(rsx, dev, n, pairings=1)
    b.same(b.sim8, events=False)  # sim8 writes no events
    b.free()


# the register budgets' edges (256 and 384 arenas a block), one round and two, full blocks of contact-heavy arenas (more mesh
# jobs than the lists hold), a block of one warp, up to three arenas a block in fewer warps than that, more blocks than the
# device holds at once (one round and several, both register budgets)
@pytest.mark.parametrize("n,grid,block", [(256, 1, 448), (257, 1, 448), (384, 1, 448), (385, 1, 448), (448, 1, 448), (449, 1, 448),
                                          (512, 1, 512), (1345, 3, 448), (2000, 5, 64), (33, 1, 32), (2050, 4, 512),
                                          (444, 148, 32), (444, 148, 64), (4096, 1480, 64), (600, 296, 224),
                                          (40001, 296, 224), (40001, 1480, 64)])
def test_lockstep_blocks(rsx, dev, n, grid, block):
    a = Arenas(rsx, dev, n)
    a.same(lambda: a.lockstep(grid, block))
    perm = a.t.from_numpy(np.random.default_rng(5).permutation(n).astype(np.int32)).to(dev.device)
    a.same(lambda: a.lockstep(grid, block, perm.data_ptr(), ticks=4))
    a.free()


def test_rounds_and_plain_at_size(rsx, dev):
    """Two even rounds of the smaller budget, and the plain launch above the lockstep kernel's sizes, block 32 and 64."""
    n = SMS * 448 + 77
    a = Arenas(rsx, dev, n)
    a.same(a.lockstep)
    a.same(a.multi)
    a.same(lambda: a.multi(64))
    a.free()


# an order that leaves arenas out (entries of n or more step nothing): some of a claim, the whole of another; lanes past the
# arenas step copies below split 9 and nothing from there
@pytest.mark.parametrize("split", [0, 1, 7, 9, 14, 15])
@pytest.mark.parametrize("grid,block,ticks", [(2, 64, 8), (148, 448, 4)])
def test_orders_with_holes(rsx, dev, split, grid, block, ticks):
    n = 203
    a = Arenas(rsx, dev, n)
    rng = np.random.default_rng(8)
    order = rng.permutation(n).astype(np.int32)
    holes = np.r_[5:9, 64:128, n - 2]  # positions 64 .. 127 hold a whole claim of the wide launches
    left_out = np.sort(order[holes])
    order[holes] = n + np.arange(len(holes), dtype=np.int32)
    d_order = a.t.from_numpy(order).to(dev.device)
    got = a.step(lambda: a.lockstep(grid, block, d_order.data_ptr(), ticks, split))
    kept = np.ones(n, bool)
    kept[left_out] = False
    for g, w, name in zip(got[1:], a.want[1:], ("results", "events")):
        g, w = g.cpu().numpy(), w.cpu().numpy()
        assert np.array_equal(g[kept], w[kept]) and (g[~kept] == -1).all(), name
    states, want, start = (rsx.unpack(x.cpu().numpy().view(np.uint32), n) for x in (got[0], a.want[0], a.start))
    assert np.array_equal(states[kept][:, :rsx.TICK_WORDS], want[kept][:, :rsx.TICK_WORDS])
    assert np.array_equal(states[~kept], start[~kept])
    a.free()


def test_a_first_launch_inside_a_capture(rsx, dev):
    """A grid past the SMs (whose blocks the library counts first) and a small one-launch decision, captured and replayed."""
    a = Arenas(rsx, dev, 4096)
    for f in (lambda: a.lockstep(1480, 96), a.multi):
        s = a.t.cuda.ExternalStream(dev.stream_ptr(), device=dev.device)

        def captured():
            g = a.t.cuda.CUDAGraph()
            with a.t.cuda.graph(g, stream=s):
                f()
            with a.t.cuda.stream(s):
                g.replay()

        a.same(captured)
    a.free()


# ---- split 15's mesh lists, in the build with short lists and counters (csrc/lists_check.cu) ----
COUNTS = ("full", "deep", "alone", "wait", "sat", "ray_alone")


@pytest.fixture(scope="module")
def lists(rsx):
    lib = ctypes.CDLL(os.path.join(os.path.dirname(rsx.LIB_PATH), "librsx_lists.so"))
    vp, u32 = ctypes.c_void_p, ctypes.c_uint32
    lib.rsx_lists_decide.argtypes = [vp, u32, vp, vp, vp, vp, vp, u32, u32, u32, vp, vp]
    lib.rsx_lists_deepen.argtypes = [vp, u32]
    return lib


def decide_counted(lists, a, width, grid, block, counts):
    c = (ctypes.c_uint32 * len(COUNTS))()
    rc = lists.rsx_lists_decide(a.ds.ptr(), a.n, a.sd.ptr(), a.idx.data_ptr(), a.ctl.data_ptr(), a.res.data_ptr(), a.ev.data_ptr(), width, grid,
                                block, c, a.dev.stream_ptr())
    assert rc == 0
    counts.update(zip(COUNTS, c))


@pytest.mark.parametrize("n,grid,block", [(448, 1, 448), (200, 1, 224), (900, 4, 256)])
def test_every_way_past_a_full_list(rsx, dev, lists, n, grid, block):
    a, counts = Arenas(rsx, dev, n), {}
    a.same(lambda: decide_counted(lists, a, 32, grid, block, counts))
    assert counts["deep"] == 0 and all(counts[k] > 0 for k in COUNTS if k != "deep"), counts
    a.free()


# the worlds' trees have five levels and the keys hold six: one more, the first that is too deep, and a chain that every walk
# leaves before it reaches the tree.  One arena a block: no list is full, so a deep job is its lane's in the round that finds it
@pytest.mark.parametrize("levels", [1, 2, 6])
def test_trees_deeper_than_the_keys(rsx, dev, lists, levels):
    def deepen(words):
        assert lists.rsx_lists_deepen(words.ctypes.data, levels) == 0

    n, counts = 96, {}
    plain, a = Arenas(rsx, dev, n), Arenas(rsx, dev, n, change=deepen)
    for deep, flat, name in zip(a.want, plain.want, ("states", "results", "events")):
        assert a.t.equal(deep, flat), name  # the walks reach the same leaves
    a.same(lambda: decide_counted(lists, a, 1, n, 32, counts))
    assert (counts["deep"] > 0) == (levels > 1), counts
    if levels == 6:
        assert counts["full"] == 0 and counts["wait"] == 0 and counts["alone"] > 0 and counts["ray_alone"] > 0, counts
    for block in (32, 256):  # the library's kernel
        a.same(lambda: a.lockstep(n, block))
    a.free()
    plain.free()
