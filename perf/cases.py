"""What the performance of this framework is measured on.

Each case is one pass of work that a user's program has the framework do, through its
public Python entry points (``Simulation``, ``Batch``, ``Server``):

* ``step``    advance one world by ``frames`` frames in one call, with edits on the first
              (``restart``: from a starting grid kept in device memory, each time);
* ``loop``    one iteration of the game loop: advance with the light field kept, then the
              composited image in device memory;
* ``colour``  advance one frame and render the colour image;
* ``batch``   give many independent worlds their grids, advance them together and read every
              grid back;
* ``serve``   a request per session to the live server, waited for, and the grids read back.

Worlds evolve from pass to pass, as a running program's do; where long runs would settle
into a world at rest, each pass restarts instead.  Sizes are those of the workloads
(``sandengine_gb300/workloads.py``) and tests, or generic ones.

Grids are whole material ids and have no 64-bit counterpart.  Colours subtract
``fract(sin(q) * 43758.5453)`` of binary32 arguments ``q``: evaluated in 64 bits these are
unrelated numbers, so ``exact`` gives no value for images either.
"""
import math
import random

import numpy as np
import torch

import sandengine_gb300 as se
from sandengine_gb300 import workloads as wl
from sandengine_gb300.batch import Batch
from sandengine_gb300.serving import Server

# A rule that reads the block's position and the frame counter: such rule sets cannot use
# the block transition table and take the generated-rules path.
LEDGE_RULE = """
  ledge:
    if: isType_EMPTY(DOWN) and pos.x + pos.y * 3 - frame % 7 > 11
    do: SWAP SELF DOWN
"""
ROUNDS = 16  # edit rounds prepared per state, used in turn


def listed():
    return [
        # the reference's default window: one iteration of its main loop on a 64 x 64 world
        {"name": "loop_64", "kind": "loop", "rules": "twelve", "w": 64, "h": 64, "frames": 1, "edits": 1},
        # an interactive session on the 256 x 256 workload: one frame per call, one brush stroke
        {"name": "brush_256", "kind": "step", "rules": "four", "w": 256, "h": 256, "frames": 1, "edits": 1},
        # the same world: a rollout of a second
        {"name": "second_256", "kind": "step", "rules": "four", "w": 256, "h": 256, "frames": 60, "edits": 0,
         "restart": True},
        # an odd-sized world (width not a multiple of 4): half a second, with edits
        {"name": "ragged_1001x777", "kind": "step", "rules": "twelve", "w": 1001, "h": 777, "frames": 30, "edits": 8,
         "restart": True},
        # the game loop at a full-screen size
        {"name": "loop_1920x1080", "kind": "loop", "rules": "twelve", "w": 1920, "h": 1080, "frames": 1, "edits": 2},
        # frames rendered as colour images, odd sides
        {"name": "colour_3001x2003", "kind": "colour", "rules": "twelve", "w": 3001, "h": 2003, "frames": 1,
         "edits": 0},
        # rules that read positions: the generated-rules path
        {"name": "ledge_2048", "kind": "step", "rules": "ledge", "w": 2048, "h": 2048, "frames": 30, "edits": 4,
         "restart": True},
        # the 4096 x 4096 workload: nearly every block is in motion
        {"name": "second_4096", "kind": "step", "rules": "four", "w": 4096, "h": 4096, "frames": 60, "edits": 0,
         "restart": True},
        # a large world whose every frame is wanted: one frame per call
        {"name": "frame_8192", "kind": "step", "rules": "twelve", "w": 8192, "h": 8192, "frames": 1, "edits": 0},
        # the 16384 x 16384 workload: a second with a round of 32 edits
        {"name": "second_16384", "kind": "step", "rules": "twelve", "w": 16384, "h": 16384, "frames": 60, "edits": 32},
        # rollouts of many worlds of different sizes: grids uploaded, final grids read back
        {"name": "rollouts_60", "kind": "batch", "rules": "twelve", "worlds": 60, "lo": 64, "hi": 1024,
         "frames": 600},
        # a burst of requests to the live server, results read back
        {"name": "serve_24", "kind": "serve", "rules": "twelve", "sessions": 24, "lo": 128, "hi": 2048, "frames": 300,
         "edits": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds: sides log-uniform (odd ones among them)."""
    kind = rng.choice(["step", "step", "step", "step", "loop", "loop", "colour", "batch", "serve"])
    if kind == "step":
        rules = rng.choice(["four", "twelve", "twelve", "ledge"])
        top = 2048 if rules == "ledge" else 12000
        frames = rng.choice([1, 1, _log(rng, 2, 60), _log(rng, 2, 60)])
        return {"kind": kind, "rules": rules, "w": _log(rng, 64, top), "h": _log(rng, 64, top), "frames": frames,
                "edits": rng.choice([0, 0, _log(rng, 1, 32)]), "restart": frames > 1}
    if kind == "loop":
        return {"kind": kind, "rules": rng.choice(["four", "twelve", "twelve"]), "w": _log(rng, 64, 4096),
                "h": _log(rng, 64, 4096), "frames": rng.choice([1, 1, _log(rng, 2, 8)]), "edits": rng.choice([0, 1, 4])}
    if kind == "colour":
        return {"kind": kind, "rules": "twelve", "w": _log(rng, 64, 8192), "h": _log(rng, 64, 8192), "frames": 1,
                "edits": rng.choice([0, 1])}
    if kind == "batch":
        return {"kind": kind, "rules": rng.choice(["four", "twelve"]), "worlds": _log(rng, 8, 60), "lo": 64,
                "hi": _log(rng, 256, 1024), "frames": _log(rng, 60, 600)}
    return {"kind": kind, "rules": "twelve", "sessions": _log(rng, 4, 24), "lo": 128, "hi": _log(rng, 256, 2048),
            "frames": _log(rng, 30, 300), "edits": rng.choice([0, 4])}


# ---- what a program has in hand ----------------------------------------------------------

_rulesets = {}


def _ruleset(name):
    """A program parses its rule set once."""
    if name not in _rulesets:
        if name == "ledge":
            text = wl.ruleset_text(wl.FOUR).replace("rules:\n", "rules:\n" + LEDGE_RULE.lstrip("\n"), 1)
            text = text.replace("base_rules: [fall]", "base_rules: [fall, ledge]")
        else:
            text = wl.ruleset_text(wl.TWELVE if name == "twelve" else wl.FOUR)
        _rulesets[name] = se.parse_string(text)
    return _rulesets[name]


def _fill(rules, w, h, gen):
    """Initial cells on the GPU: i.i.d. materials for the four-material rules, 64 x 64 patches
    of one material (16 x 16 in small worlds) for the twelve-material ones."""
    ids, probs = wl.twelve_fill_spec() if rules == "twelve" else wl.FOUR_FILL
    patch = 1 if rules != "twelve" else 64 if min(w, h) >= 512 else 16
    pw, ph = -(-w // patch), -(-h // patch)
    cum = torch.tensor(np.cumsum(probs)[:-1], dtype=torch.float32, device="cuda")
    pick = torch.searchsorted(cum, torch.rand((ph, pw), generator=gen, device="cuda"), right=True)
    cells = torch.tensor(ids, dtype=torch.int32, device="cuda")[pick]
    if patch > 1:
        cells = cells.repeat_interleave(patch, 0)[:h].repeat_interleave(patch, 1)[:, :w]
    return cells.contiguous()


def _edits(rng, w, h, count):
    """Circles of EMPTY or sand (radius 1-16 on small worlds, 8-64 on large ones)."""
    lo, hi = (8, 64) if min(w, h) >= 512 else (1, 16)
    return [se.SimModification((rng.randrange(w), rng.randrange(h)), 0, rng.randint(lo, hi), rng.choice([0, 3]))
            for _ in range(count)]


class _DeviceArray:
    """A device buffer of a simulation as torch sees it (keeps the simulation alive)."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(state, ptr, floats):
    """The tensor over one of the simulation's buffers (it has a few; each is wrapped once)."""
    t = state["views"].get(ptr)
    if t is None:
        w, h = state["sim"].size
        a = _DeviceArray(state["sim"], ptr, (h, w, 4) if floats else (h, w), "<f4" if floats else "<i4")
        t = state["views"][ptr] = torch.as_tensor(a, device="cuda")
    return t


def _sizes(rng, count, lo, hi):
    """World sizes, sides log-uniform; every fourth world has odd sides."""
    out = []
    for i in range(count):
        w, h = _log(rng, lo, hi), _log(rng, lo, hi)
        out.append((w | 1, h | 1) if i % 4 == 3 else (w & ~7, h & ~7))
    return [(min(w, hi), min(h, hi)) for w, h in out]


def prepare(case, seed):
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rules, kind = case["rules"], case["kind"]
    rs = _ruleset(rules)
    if kind == "batch":
        sizes = _sizes(random.Random(5), case["worlds"], case["lo"], case["hi"])
        grids = [_fill(rules, w, h, gen).cpu().numpy().view(np.uint32) for w, h in sizes]
        return {"kind": kind, "batch": Batch(rs, sizes), "frames": case["frames"], "grids": grids,
                "starts": [rng.randint(1, 1000) for _ in sizes]}
    if kind == "serve":
        sizes = _sizes(random.Random(6), case["sessions"], case["lo"], case["hi"])
        srv = Server(rs, 4 << 30)
        requests = []
        for w, h in sizes:
            sid = srv.open_session(w, h, _fill(rules, w, h, gen).cpu().numpy().view(np.uint32), rng.randint(1, 1000))
            requests.append((sid, case["frames"] - (sid * case["frames"]) // (2 * len(sizes)),
                             [_edits(rng, w, h, case["edits"]) for _ in range(ROUNDS)]))
        srv.start()
        return {"kind": kind, "server": srv, "requests": requests, "round": 0}
    w, h = case["w"], case["h"]
    sim = se.Simulation(rs, (w, h))
    state = {"kind": kind, "sim": sim, "frames": case["frames"], "views": {}, "round": 0,
             "edits": [_edits(rng, w, h, case["edits"]) for _ in range(ROUNDS)]}
    cells, state["start"] = _fill(rules, w, h, gen), rng.randint(1, 1000)
    _view(state, sim.device_grid_ptr(), False).copy_(cells)
    sim.params.frame = state["start"]
    if case.get("restart"):
        state["cells"], state["stream"] = cells, torch.cuda.ExternalStream(sim.stream)
    if kind == "loop":
        sim.set_light(True)
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        for i, (cells, frame) in enumerate(zip(state["grids"], state["starts"])):
            b.set_grid(i, cells)
            b.set_frame(i, frame)
        b.step(state["frames"])
        return [b.grid(i) for i in range(len(b))]
    if kind == "serve":
        srv, k = state["server"], state["round"] % ROUNDS
        state["round"] += 1
        ids = [srv.submit(sid, frames, edits[k]) for sid, frames, edits in state["requests"]]
        for i in ids:
            srv.wait(i)
        return [srv.grid(sid) for sid, _, _ in state["requests"]]
    sim = state["sim"]
    if "cells" in state:
        with torch.cuda.stream(state["stream"]):
            _view(state, sim.device_grid_ptr(), False).copy_(state["cells"])
        sim.params.frame = state["start"]
    edits = state["edits"][state["round"] % ROUNDS]
    state["round"] += 1
    if state["frames"] == 1:
        sim.modifications.extend(edits)
        sim.run()
    else:
        sim.run_frames(state["frames"], edits)
    if kind == "loop":
        return [_view(state, sim.composite_device(), True), _view(state, sim.device_grid_ptr(), False)]
    if kind == "colour":
        return [_view(state, sim.render_color_device(), True), _view(state, sim.device_grid_ptr(), False)]
    return _view(state, sim.device_grid_ptr(), False)


def work(case):
    """Bytes of one pass: every grid read and written once (4 B a cell each), the light field
    once each way per frame (16 B each), an image written once (16 B); grids that come from the
    host are written and results that go to it are read once more.  The updates are integer work: only the light and the images
    count as floating-point operations."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        n = case["worlds"] if kind == "batch" else case["sessions"]
        sizes = _sizes(random.Random(5 if kind == "batch" else 6), n, case["lo"], case["hi"])
        return {"bytes": (16.0 if kind == "batch" else 12.0) * sum(w * h for w, h in sizes), "flops": 0.0}
    cells = float(case["w"] * case["h"])
    if kind == "loop":
        return {"bytes": cells * (8 + 32 + 16), "flops": cells * (100 * case["frames"] + 150)}
    if kind == "colour":
        return {"bytes": cells * (8 + 16), "flops": cells * 8}
    return {"bytes": cells * 8, "flops": 0.0}


def exact(case, seed):
    return None
