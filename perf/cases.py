"""The calls whose time matters to a program that uses this framework, over the sizes it meets, through the public entry
points (rsx.SimDevice, runner.DecisionRunner, predictor.ContactPredictor).

The decision is the product: one 8-tick decision of a batch of arenas, from one arena (somebody watching or driving a
single match) through the 1,024 kickoff arenas of the plain configuration and a few thousand arenas (an evaluation, a
small learner) to the 65,536 and 262,144 arenas of the headline and batching configurations.  Around it stand the rollout
step (the learned order, the decision, the restart of finished episodes, the observations), the observation kernel by
itself, and the contact predictor's inference and training step.

A decision changes its states, so every pass first copies the batch's snapshot back (rsx_copy_raw, as a search that
branches from one state does): all passes then do the same work.  Start states are the device generator's, played a few
decisions on with random controls and restarts, so that cars are against walls, balls in the air and pads taken.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys
import weakref

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "rocketsim-cuda_b200"))

import rsx  # noqa: E402
import predictor as P  # noqa: E402
from runner import DecisionRunner  # noqa: E402

PAIRINGS = [(p, q) for p in range(7) for q in range(7)]
MIXES = {"kickoff": rsx.MIX_KICKOFF, "headline": rsx.MIX_HEADLINE, "contact": rsx.MIX_CONTACT_HEAVY}
WEIGHTS = (10.0, 0.5, 0.2, 1.0, -1.0, 0.1, 0.05, 0.1)  # a learner's reward weights
PLAYED = 5  # decisions played before the measured one

_once: dict = {}


def _device() -> "rsx.SimDevice":
    if "dev" not in _once:
        _once["dev"] = rsx.SimDevice(0)
    return _once["dev"]


def _statics(count: int) -> np.ndarray:
    """The world's StaticData, one per car pairing (built once by a program)."""
    if count not in _once:
        _once[count] = np.stack([rsx.build_static(7, p, q) for p, q in PAIRINGS[:count]])
    return _once[count]


def _stream():
    """The stream of a program's batch: its decisions follow one another."""
    if "stream" not in _once:
        _once["stream"] = torch.cuda.Stream()
    return _once["stream"]


class _Filled(rsx.SimDevice):
    """A device whose uploaded states are only allocated: the generator on the device fills them."""

    def __init__(self, dev):
        self.__dict__.update(dev.__dict__)

    def upload_states(self, states):
        return self.alloc_states(states.shape[0])


class _Words:
    """The words of a state buffer as a tensor that keeps its owner alive."""

    def __init__(self, owner, ptr: int, words: int):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (words,), "typestr": "<i4", "data": (ptr, False), "version": 2}


def _words(owner, ptr, n):
    return torch.as_tensor(_Words(owner, ptr, rsx.aosoa_words(n)), device="cuda")


def _controls(gen, n: int):
    """Random controls on the device: axes in {-1, 0, 1}, jump / boost / handbrake on half the time."""
    c = torch.empty((n, 2, rsx.CONTROL_WORDS), dtype=torch.int32, device="cuda")
    c[:, :, :5] = torch.randint(-1, 2, (n, 2, 5), generator=gen, device="cuda").to(torch.float32).view(torch.int32)
    c[:, :, 5:] = torch.randint(0, 2, (n, 2, 3), generator=gen, device="cuda", dtype=torch.int32)
    return c


def _gen(seed: int):
    return torch.Generator(device="cuda").manual_seed(seed)


def _reset(states_ptr, n, statics_ptr, index_ptr, seed, mix, result_ptr, stream):
    m = (ctypes.c_float * 5)(*mix)
    rsx.check(rsx.lib().rsx_reset_arenas_raw(states_ptr, n, statics_ptr, index_ptr, seed, m, result_ptr, None, None, stream), "reset")


# ---- the states of the cases ---------------------------------------------------------------------------------------
class Match:
    """Arenas of one car pairing on a SimDevice, stepped by sim8 (the reference-shaped calls)."""

    def __init__(self, case, seed):
        self.n = n = case["arenas"]
        self.dev = dev = _device()
        gen = _gen(seed)
        self.sd = dev.upload_static(_statics(1))
        self.ds = dev.alloc_states(n)
        weakref.finalize(self, self.sd.free)
        weakref.finalize(self, self.ds.free)
        self.res = dev.alloc_result(n)
        _reset(self.ds.ptr(), n, self.sd.ptr(), None, seed, MIXES[case["mix"]], None, dev.stream_ptr())
        for _ in range(PLAYED):
            self.ctl = _controls(gen, n)
            dev.sim8(self.ds, self.sd, self.ctl, self.res)
            dev.sync()
        self.ctl = _controls(gen, n)
        self.bytes = rsx.aosoa_words(n) * 4
        self.snap = torch.empty(rsx.aosoa_words(n), dtype=torch.int32, device="cuda")
        rsx.check(rsx.lib().rsx_copy_raw(self.snap.data_ptr(), self.ds.ptr(), self.bytes, dev.stream_ptr()), "rsx_copy_raw")
        dev.sync()

    def run(self):
        rsx.check(rsx.lib().rsx_copy_raw(self.ds.ptr(), self.snap.data_ptr(), self.bytes, self.dev.stream_ptr()), "rsx_copy_raw")
        self.dev.sim8(self.ds, self.sd, self.ctl, self.res)
        return {"states": _words(self, self.ds.ptr(), self.n), "result": self.res}


class Batch:
    """Arenas of all 49 car pairings in a DecisionRunner."""

    def __init__(self, case, seed):
        n = case["arenas"]
        gen = _gen(seed)
        sds = _statics(len(PAIRINGS))
        index = torch.randint(0, len(PAIRINGS), (n,), generator=gen, device="cuda", dtype=torch.uint8)
        self.runner = r = DecisionRunner(_Filled(_device()), sds, index.cpu().numpy(), np.broadcast_to(np.zeros(1, np.uint32), (n, 1)), stream=_stream())
        weakref.finalize(self, r.free)
        self.mix = MIXES[case["mix"]]
        self.seed = seed
        self.config = None
        _reset(r.ds.ptr(), n, r.dsd.ptr(), r.didx.data_ptr(), seed, self.mix, None, r.sptr)
        for d in range(PLAYED):
            ctl = _controls(gen, n)
            torch.cuda.synchronize()
            r.step(ctl.data_ptr())
            _reset(r.ds.ptr(), n, r.dsd.ptr(), r.didx.data_ptr(), seed + 1 + d, self.mix, r.res.data_ptr(), r.sptr)
            torch.cuda.synchronize()
        self.ctl = _controls(gen, n)
        if case["path"] == "plain":
            self.config = {"mode": "plain", "block": 32}
        if case["path"] == "rollout":
            r.train_predictor(control_seed=seed, decisions=2, epochs=1)
            self.config = {"mode": "levels", "block": 448, "grid": r.sms, "split": 15, "threshold": 0.5, "levels": 16, "weights": [1.0] * P.LABELS}
        self.snap = r.snapshot()
        if case["path"] == "observe":
            r.step(self.ctl.data_ptr())
        torch.cuda.synchronize()

    def step(self):
        r = self.runner
        r.restore(self.snap)
        r.step(self.ctl.data_ptr(), self.config)
        return {"states": _words(self, r.ds.ptr(), r.n), "result": r.res, "events": r.ev}

    def rollout(self):
        r = self.runner
        out = self.step()
        obs, reward = r.observe(WEIGHTS)
        _reset(r.ds.ptr(), r.n, r.dsd.ptr(), r.didx.data_ptr(), self.seed + 100, self.mix, r.res.data_ptr(), r.sptr)
        return dict(out, observations=obs, reward=reward)

    def observe(self):
        obs, reward = self.runner.observe(WEIGHTS)
        return {"observations": obs, "reward": reward}


def _features(gen, n):
    """Feature rows as the framework stores them: BF16 values of magnitude around one."""
    return torch.randn((n, P.FEATURES), generator=gen, device="cuda").clamp_(-3.0, 3.0).to(torch.bfloat16).view(torch.int16)


class Network:
    """The contact predictor with the rows of one call."""

    def __init__(self, case, seed):
        gen = _gen(seed)
        self.n = case["rows"]
        self.pred = P.ContactPredictor(torch.device("cuda", 0), seed=seed % 1000)
        self.X = _features(gen, self.n)
        self.Y = torch.randint(0, 64, (self.n,), generator=gen, device="cuda", dtype=torch.uint8)
        self.Z = torch.empty((self.n, 8), dtype=torch.float32, device="cuda")
        # a program keeps its weights; each pass takes its step from these, so that all passes are the same step
        self.start = (self.pred.w.clone(), self.pred.m.clone(), self.pred.v.clone())

    def predict(self):
        return {"logits": self.pred.logits(self.X, self.n, out=self.Z)[:, :P.LABELS]}

    def train(self):
        p = self.pred
        for dst, src in zip((p.w, p.m, p.v), self.start):
            dst.copy_(src)
        rsx.check(p.L.rsx_pred_to_bf16_raw(p.w.data_ptr(), p.wb.data_ptr(), p.stream), "rsx_pred_to_bf16_raw")
        p.step = 0
        p.train_step(self.X, self.Y, self.n, lr=1e-3)
        return {"gradient": p.grad, "loss": p.loss, "weights": p.w}


# ---- the cases -----------------------------------------------------------------------------------------------------
def listed():
    return [
        # one match, as somebody who drives or watches a single game steps it: latency is all there is
        {"name": "sim8_1", "path": "sim8", "arenas": 1, "mix": "headline"},
        # an odd handful of matches
        {"name": "sim8_37", "path": "sim8", "arenas": 37, "mix": "headline"},
        # the plain configuration: 1,024 Octane vs Octane kickoffs
        {"name": "sim8_1024_kickoff", "path": "sim8", "arenas": 1024, "mix": "kickoff"},
        # a small batch of mixed pairings on the plain launch, which the autotuner keeps at this size
        {"name": "plain_4096", "path": "plain", "arenas": 4096, "mix": "headline"},
        # a ragged medium batch on the runner's default configuration
        {"name": "lockstep_10007", "path": "lockstep", "arenas": 10007, "mix": "headline"},
        # the headline
        {"name": "lockstep_65536", "path": "lockstep", "arenas": 65536, "mix": "headline"},
        # the batching configuration: several claim rounds a decision
        {"name": "lockstep_262144", "path": "lockstep", "arenas": 262144, "mix": "headline"},
        # a learner's step over contact-heavy play: learned order, decision, observations and rewards, restarts
        {"name": "rollout_49153", "path": "rollout", "arenas": 49153, "mix": "contact"},
        # observations and rewards of a learner whose decisions run elsewhere in its loop
        {"name": "observe_65536", "path": "observe", "arenas": 65536, "mix": "headline"},
        # the predictor's inference over a headline batch and its training step
        {"name": "predict_65536", "path": "predict", "rows": 65536},
        {"name": "train_8192", "path": "train", "rows": 8192},
    ]


def _spread(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n | 1 if rng.random() < 0.5 else n))


def draw(rng):
    path = rng.choice(["sim8", "sim8", "plain", "lockstep", "lockstep", "lockstep", "rollout", "observe", "predict", "train"])
    if path == "sim8":
        return {"path": path, "arenas": _spread(rng, 1, 4096), "mix": rng.choice(["kickoff", "headline", "contact"])}
    if path == "predict":
        return {"path": path, "rows": _spread(rng, 1000, 262144)}
    if path == "train":
        return {"path": path, "rows": _spread(rng, 1024, 32768)}
    lo, hi = {"plain": (64, 8192), "lockstep": (1024, 200000), "rollout": (8192, 100000), "observe": (1024, 200000)}[path]
    return {"path": path, "arenas": _spread(rng, lo, hi), "mix": rng.choice(["headline", "headline", "contact"])}


def prepare(case, seed):
    path = case["path"]
    if path == "sim8":
        return ("sim8", Match(case, seed))
    if path in ("predict", "train"):
        return (path, Network(case, seed))
    return (path, Batch(case, seed))


def run(state):
    path, s = state
    if path == "sim8":
        return s.run()
    if path == "predict":
        return s.predict()
    if path == "train":
        return s.train()
    if path == "rollout":
        return s.rollout()
    if path == "observe":
        return s.observe()
    return s.step()


LAYERS = ((P.HIDDEN, P.FEATURES), (P.HIDDEN, P.HIDDEN), (P.HIDDEN, P.HIDDEN), (8, P.HIDDEN))


def work(case):
    path = case["path"]
    if path in ("predict", "train"):
        n = case["rows"]
        macs = sum(a * b for a, b in LAYERS)
        if path == "predict":
            return {"bytes": n * (P.FEATURES * 2 + P.LABELS * 4) + P.PARAMS * 2, "flops": 2 * n * macs}
        # forward, the layers' input gradients (not the first layer's) and the weight gradients; weights and moments
        # read and written, the gradient written
        return {"bytes": n * (P.FEATURES * 2 + 1) + P.PARAMS * 4 * 7, "flops": 2 * n * (3 * macs - P.HIDDEN * P.FEATURES)}
    n = case["arenas"]
    obs = n * 2 * (rsx.OBS_DIM * 2 + 4)
    if path == "observe":
        # what the rows hold: ball, cars, controls and pad times (638 B an arena), result and events; rows and rewards
        return {"bytes": n * (638 + 8) + obs, "flops": 0}
    # the snapshot's words read and the new state's words written, the controls, the result and event words; the arithmetic
    # is scalar and branches by contact: it has no fixed count
    b = n * (rsx.ARENA_WORDS * 4 * 2 + 64 + 8)
    return {"bytes": b + (obs if path == "rollout" else 0), "flops": 0}


def tolerance(case):
    """The simulator's words, result words, events, observation bits and rewards are fixed bit for bit.  The network
    computes in BF16 with FP32 sums: `exact` keeps its activations in 64 bits, and the weights after one Adam step differ
    in sign(g) * lr where a gradient is near zero."""
    if case["path"] == "predict":
        return {"rel": 1.5e-2}
    if case["path"] == "train":
        return {"rel": 1.5e-2}
    return "exact"


def exact(case, seed):
    """The network in 64 bits (weights and features as the path reads them: rounded to BF16); the simulator has no
    implementation here but its own."""
    if case["path"] not in ("predict", "train"):
        return None
    gen = _gen(seed)
    X = _features(gen, case["rows"]).view(torch.bfloat16).double()
    Y = torch.randint(0, 64, (case["rows"],), generator=gen, device="cuda", dtype=torch.uint8)
    flat = torch.from_numpy(P.init_params(seed % 1000)).cuda()
    params = []
    for name, shape in zip(("W1", "b1", "W2", "b2", "W3", "b3", "W4", "b4"),
                           [s for l in LAYERS for s in (l, (l[0],))]):
        o, size = P.OFF[name]
        w = flat[o:o + size].reshape(shape)
        params.append((w.to(torch.bfloat16) if name[0] == "W" else w).double().requires_grad_(case["path"] == "train"))
    h = X
    for k in range(0, 6, 2):
        h = torch.relu(h @ params[k].t() + params[k + 1])
    z = (h @ params[6].t() + params[7])[:, :P.LABELS]
    if case["path"] == "predict":
        return {"logits": z}
    bits = ((Y[:, None].long() >> torch.arange(P.LABELS, device="cuda")) & 1).double()
    loss = torch.nn.functional.binary_cross_entropy_with_logits(z, bits, reduction="sum")
    g = torch.cat([x.reshape(-1) for x in torch.autograd.grad(loss / case["rows"], params)])
    # the first Adam step: both moments' bias corrections cancel their decay
    return {"gradient": g, "loss": loss.detach().reshape(1), "weights": flat.double() - 1e-3 * g / (g.abs() + 1e-8)}
