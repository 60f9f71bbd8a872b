"""The calls whose time matters to a user of this framework.

Every case goes through the package's public API: models stepped, rendered and
read (``CellularAutomaton``, ``model.gpu``), ensembles run from host memory to
host memory (``Ensemble.run``) and simulation requests served (``Server``).
States evolve from pass to pass, as a running simulation does.

All outputs are cells, pixels or totals: whole numbers, equal or wrong.
"""
import functools
import operator

import numpy as np
import torch

from xentica_gb300 import _native, core, seeds, serve
from xentica_gb300.batch import Ensemble, ensemble_seeds
from xentica_gb300.core import canonical, color_effects
from xentica_gb300.seeds.random import RandInt, RandPoisson
from xentica_gb300.tools import xmath
from xentica_gb300.tools.rules import LifeLike


class Life(core.CellularAutomaton):
    """Life-like CA on a 2-D Moore torus, its rule an interactive parameter."""

    state = core.IntegerProperty(max_val=1)
    rule = core.Parameter(default=LifeLike.golly2int("B3/S23"), interactive=True)

    class Topology:
        dimensions = 2
        lattice = core.OrthogonalLattice()
        neighborhood = core.MooreNeighborhood()
        border = core.TorusBorder()

    def emit(self):
        for buf in self.buffers:
            buf.state = self.main.state

    def absorb(self):
        alive = core.IntegerVariable()
        for i in range(len(self.buffers)):
            alive += self.neighbors[i].buffer.state
        is_born = (self.rule >> alive) & 1
        is_sustain = (self.rule >> 9 >> alive) & 1
        self.main.state = is_born | is_sustain & self.main.state

    @color_effects.MovingAverage
    def color(self):
        return (self.main.state * 255, self.main.state * 255, self.main.state * 255)


class LifeStatic(Life):
    """The same inside a border of dead cells."""

    class Topology(Life.Topology):
        border = core.StaticBorder(0)


class Life3D(Life):
    """B13,14,17-19/S13-26 (cloud-like blobs) on a 3-D Moore torus."""

    class Topology(Life.Topology):
        dimensions = 3

    def absorb(self):
        alive = core.IntegerVariable()
        for i in range(len(self.buffers)):
            alive += self.neighbors[i].buffer.state
        is_born = (0xE6000 >> alive) & 1
        is_sustain = (0x7FFE000 >> alive) & 1
        self.main.state = is_born | is_sustain & self.main.state


class Life3DFaces(Life):
    """B2/S23 on a 3-D von Neumann lattice inside a border of dead cells."""

    class Topology(Life.Topology):
        dimensions = 3
        neighborhood = core.VonNeumannNeighborhood()
        border = core.StaticBorder(0)

    def absorb(self):
        alive = core.IntegerVariable()
        for i in range(len(self.buffers)):
            alive += self.neighbors[i].buffer.state
        self.main.state = ((4 >> alive) & 1) | ((12 >> alive) & 1) & self.main.state


class ForestFire(core.CellularAutomaton):
    """Empty ground (0) grows trees (1) at random; a tree beside a burning
    cell (2) or struck by lightning burns, and is empty ground after that.
    No kernel family of its own: it runs on the interpreter."""

    ground = core.IntegerProperty(max_val=2)
    rng = core.RandomProperty()

    class Topology:
        dimensions = 2
        lattice = core.OrthogonalLattice()
        neighborhood = core.MooreNeighborhood()
        border = core.TorusBorder()

    def emit(self):
        for buf in self.buffers:
            buf.ground = self.main.ground

    def absorb(self):
        burning = core.IntegerVariable()
        for i in range(len(self.buffers)):
            burning += self.neighbors[i].buffer.ground == 2
        chance = core.IntegerVariable()
        chance += xmath.int(self.main.rng.uniform * 1000)
        grows = (self.main.ground == 0) & (chance < 30)
        tree = self.main.ground == 1
        burns = tree & ((burning > 0) | (chance < 1))
        self.main.ground = grows + tree + burns

    @color_effects.MovingAverage
    def color(self):
        red = (self.main.ground == 2) * 255
        green = (self.main.ground == 1) * 160
        return (red, green, self.main.ground * 20)


SOUP = {"state": RandInt(0, 1)}

#: kind -> (model, its starting state, experiment settings), as their own examples set them
MODELS = {
    "life": (Life, SOUP, {}),
    "life_static": (LifeStatic, SOUP, {}),
    "life3d": (Life3D, SOUP, {}),
    "life3d_faces": (Life3DFaces, SOUP, {}),
    "evolife": (canonical.EvoLifeProgram,
                {"energy": RandInt(0, 255), "rule": RandInt(0, 2 ** 18 - 1),
                 "rng": RandInt(0, 2 ** 16 - 1)},
                {"fade_in": 18, "fade_out": 3, "death_speed": 15, "max_genes": 9,
                 "mutation_prob": 0.0}),
    "mass": (canonical.MassTransferProgram, {"mass": RandPoisson(4)}, {}),
    "lifecolor": (canonical.LifeColorProgram,
                  {"state": RandInt(0, 1), "red": RandInt(0, 255), "green": RandInt(0, 255),
                   "blue": RandInt(0, 255)},
                  {"fade_in": 255, "fade_out": 10, "smooth_factor": 1}),
    "noise": (canonical.NoiseProgram, {"rng": RandInt(0, 2 ** 16 - 1)},
              {"fade_in": 40, "fade_out": 25, "smooth_factor": 1}),
    "gravity": (canonical.GravityProgram, {"energy": RandInt(0, 1) * 1, "gravity": 0}, {}),
    "forest": (ForestFire, {"ground": RandInt(0, 1), "rng": RandInt(0, 2 ** 16 - 1)},
               {"fade_in": 60, "fade_out": 20, "smooth_factor": 1}),
}

#: kind -> (packed cell bytes, colour bytes kept per cell, operations per cell-update of the rule
#: as written: one addition per neighbour and property, the rule, the colour)
COSTS = {
    "life": (1, 0, 12), "life_static": (1, 0, 12), "life3d": (1, 0, 30), "life3d_faces": (1, 0, 10),
    "evolife": (8, 12, 300), "mass": (4, 0, 20), "lifecolor": (4, 12, 50), "noise": (2, 12, 15),
    "gravity": (8, 12, 100), "forest": (4, 12, 40),
}


def listed():
    return [
        # the viewer on a small lattice: a few generations a frame, each its own call; launches
        # and host work count
        {"name": "view_life_160x120", "do": "view", "model": "life", "x": 160, "y": 120,
         "rule": "B3/S23", "generations": 8},
        # Conway's Life on the configured 512x512 torus, 1000 generations between looks
        {"name": "life_512", "do": "steps", "model": "life", "x": 512, "y": 512,
         "rule": "B3/S23", "generations": 1000},
        # the largest side that requests have, a rule other than Conway's
        {"name": "life_4096", "do": "steps", "model": "life", "x": 4096, "y": 4096,
         "rule": "B36/S23", "generations": 1000},
        # a Life-like rule in three dimensions
        {"name": "life3d_128", "do": "steps", "model": "life3d", "x": 128, "y": 128, "z": 128,
         "generations": 100},
        # the evolving-genome model at its configured size, a frame for every generation
        {"name": "evolife_1080p", "do": "frames", "model": "evolife", "x": 1920, "y": 1080,
         "generations": 64},
        # sand transfer at its configured size: a projection and the checked total for every
        # generation
        {"name": "mass_256", "do": "frames", "model": "mass", "x": 256, "y": 256, "z": 256,
         "generations": 64},
        # the other example models at full-HD size, watched
        {"name": "lifecolor_1080p", "do": "frames", "model": "lifecolor", "x": 1920, "y": 1080,
         "generations": 64},
        {"name": "noise_1080p", "do": "frames", "model": "noise", "x": 1920, "y": 1080,
         "generations": 64},
        {"name": "gravity_1080p", "do": "frames", "model": "gravity", "x": 1920, "y": 1080,
         "generations": 64},
        # a user's own model, at the examples' usual size
        {"name": "forest_640x360", "do": "frames", "model": "forest", "x": 640, "y": 360,
         "generations": 64},
        # the configured ensemble: random rules, ragged sizes, host memory to host memory
        {"name": "ensemble_4096", "do": "ensemble", "lattices": 4096, "mix": 2041, "side": 1024,
         "generations": 256},
        # requests of every kind at once
        {"name": "serve_32", "do": "serve", "requests": 32, "mix": 11, "generations": 2000},
    ]


def draw(rng):
    def near(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    do = rng.choice(["view", "life", "life", "life3d", "evolife", "mass", "lifecolor", "noise",
                     "gravity", "forest", "ensemble", "serve"])
    if do == "view":
        return {"do": "view", "model": rng.choice(["life", "life_static"]), "x": near(64, 640),
                "y": near(48, 360), "rule": "B3/S23", "generations": rng.randint(1, 16)}
    if do == "life":
        return {"do": "steps", "model": rng.choice(["life", "life_static"]), "x": near(64, 4000),
                "y": near(64, 4000), "rule": rng.choice(["B3/S23", "B36/S23", "B34/S34"]),
                "generations": near(100, 1000)}
    if do == "life3d":
        return {"do": "steps", "model": rng.choice(["life3d", "life3d_faces"]), "x": near(32, 192),
                "y": near(32, 192), "z": near(32, 192), "generations": near(16, 100)}
    if do == "mass":
        return {"do": rng.choice(["frames", "steps"]), "model": "mass", "x": near(64, 256),
                "y": near(64, 256), "z": near(64, 256), "generations": near(16, 64)}
    if do == "forest":
        return {"do": "frames", "model": do, "x": near(64, 1280), "y": near(48, 720),
                "generations": near(16, 64)}
    if do == "ensemble":
        return {"do": "ensemble", "lattices": near(64, 2048), "mix": rng.randrange(1000),
                "side": rng.choice([256, 512, 1024]), "generations": near(32, 256)}
    if do == "serve":
        return {"do": "serve", "requests": rng.randint(4, 32), "mix": rng.randrange(1000),
                "generations": near(200, 1000)}
    return {"do": rng.choice(["frames", "steps"]), "model": do, "x": near(160, 1920),
            "y": near(120, 1080), "generations": near(16, 64)}


def requests(case):
    """The requests of a serving case: kinds, sizes and rules are the case's."""
    return serve.serving_workload(case["requests"], seed=case["mix"], sides2d=(32, 2048),
                                  sides3d=(64, 192), generations=(100, case["generations"]))


def lattices(case):
    """Widths, heights, rules, densities and seeds of an ensemble case's lattices."""
    sides = [s for s in (64, 128, 256, 512, 1024) if s <= case["side"]]
    return ensemble_seeds(case["lattices"], case["mix"], sides)


def cells_of(case):
    return functools.reduce(operator.mul, (case[k] for k in "xyz" if k in case))


def prepare(case, seed):
    if case["do"] == "ensemble":
        widths, heights, rules, densities, words = lattices(case)
        ens = Ensemble(widths, heights, rules)
        ens.tune(case["generations"])
        ens.seed_bernoulli(words ^ np.uint32(seed & 0xFFFFFFFF), densities)
        cells = [_native.PinnedBuffer(ens.total_cells) for _ in range(2)]
        ens.download(cells[0].array)
        return {"ensemble": ens, "in": cells[0], "out": cells[1], **case}
    if case["do"] == "serve":
        jobs = []
        for i, spec in enumerate(requests(case)):
            cells = serve.make_cells({**spec, "seed": seed * 1000 + i})
            jobs.append((spec["kind"], cells, spec["rule"], spec["generations"]))
        return {"server": serve.Server(4 << 30, host_bytes=1 << 30), "jobs": jobs, **case}
    model, start, settings = MODELS[case["model"]]
    settings = dict(settings, word="CASES %d" % seed, zoom=1, pos=[0, 0],
                    size=tuple(case[k] for k in "xyz" if k in case),
                    seed=seeds.patterns.PrimordialSoup(vals=start))
    if "rule" in case:
        settings["rule"] = LifeLike.golly2int(case["rule"])
    ca = model(type("CaseExperiment", (core.Experiment,), settings))
    ca.set_viewport((case["x"], case["y"]))
    state = {**case, "model": ca, "kind": case["model"], "golly": settings.get("rule")}
    if case["do"] == "frames":
        state["frames"] = torch.empty((case["generations"], 3 * case["x"] * case["y"]),
                                      dtype=torch.uint8, device="cuda")
    return state


def run(state):
    n = state["generations"]
    if state["do"] == "ensemble":
        state["ensemble"].run(state["in"].array, state["out"].array, n)
        return state["out"].array
    if state["do"] == "serve":
        queued = [state["server"].submit(*job) for job in state["jobs"]]
        return [r.result() for r in queued]
    ca = state["model"]
    if state["golly"] is not None:
        ca.rule = state["golly"]      # a parameter belongs to the class: other models set it too
    if state["do"] == "view":
        for _ in range(n):
            ca.step()
        return ca.render()
    if state["do"] == "frames":
        ca.gpu.step_frames(n, ca.width, ca.height, 1, 0, 0, state["frames"].data_ptr(),
                           on_device=True)
        out = [state["frames"]]
    else:
        ca.gpu.step(n)
        out = [ca.gpu.main_plane()]
    if state["kind"] == "mass":
        out.append(ca.gpu.mass_totals(n))
    return out


def work(case):
    """The state read and written once, the pixels written, and the rule's operations."""
    n = case["generations"]
    if case["do"] == "ensemble":
        widths, heights = lattices(case)[:2]
        cells = int((widths.astype(np.int64) * heights).sum())
        return {"bytes": 2 * cells, "flops": 12 * n * cells}
    if case["do"] == "serve":
        total = {"bytes": 0, "flops": 0}
        for spec in requests(case):
            size, _, ops = COSTS["mass" if spec["kind"] == "mass" else
                                 "life" if spec["kind"] == "life2d" else "life3d_faces"]
            cells = int(np.prod(spec["shape"]))
            total["bytes"] += 2 * size * cells
            total["flops"] += ops * spec["generations"] * cells
        return total
    cells = cells_of(case)
    size, colour, ops = COSTS[case["model"]]
    moved = 2 * (size + colour) * cells
    if case["do"] == "frames":
        moved += 3 * case["x"] * case["y"] * n
    elif case["do"] == "view":
        moved += 3 * case["x"] * case["y"]
    return {"bytes": moved, "flops": ops * n * cells}


def exact(case, seed):
    """No output is a rounded number: cells, pixels and totals are whole."""
    return None
