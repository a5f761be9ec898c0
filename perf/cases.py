"""What a user of plume_b200 has it do, as cases to be timed, each through the package's public entry points.

Kinds of case
- "step": one Stepper.step of a grid, loaded beforehand with a moving, smoking state (the six arrays that carry
  a run from one substep to the next are copied in, as a program that resumes a captured state does).
- "project": pressure.project with a Multigrid solve, for programs that call the operators one by one.
- "frame": FrameRenderer.render of a smoking grid to a host image, in either channel layout.
- "fit": FlowFit.loss_and_grad, a few substeps forward and their adjoints back.
- "batch": Batch.run of an uneven parameter sweep from a given state, after Batch.reset.

Recipes: "plain" is the benchmark's step (4 V-cycles, confinement, drag, a hard-edged emitter); "puff" is the
smoke-puff recipe's physics (2 V-cycles, noisy emitter, strong confinement, turbulence, drag, dissipation).

`exact` restates each path in float64 torch, from the equations alone.
"""

import dataclasses
import math

import numpy as np
import torch

from plume_b200.adjoint import FlowFit
from plume_b200.recipe.derived import derive
from plume_b200.recipe.load import resolve_table
from plume_b200.recipe.schema import NORMAL_LAYOUT, SHADE_LAYOUT
from plume_b200.recipe.variation import sweep_table
from plume_b200.render.camera import sheet_domain_view
from plume_b200.render.frame_renderer import FrameRenderer
from plume_b200.sim.batch import Batch
from plume_b200.sim.grid import make_grid
from plume_b200.sim.multigrid import Multigrid
from plume_b200.sim.pressure import project
from plume_b200.sim.stepper import Stepper
from plume_b200.workloads import batch_base_table, plain_step_recipe

DEVICE = "cuda:0" if torch.cuda.is_available() else "cpu"
STORAGE = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
FIELDS = ("u", "v", "w", "smoke", "temperature")
LARGEST_CELLS = 256 * 384 * 256


def step_case(name, cells, recipe="plain", storage="f32", faces="open", solver="multigrid"):
    return {"name": name, "kind": "step", "nx": cells[0], "ny": cells[1], "nz": cells[2], "recipe": recipe,
            "storage": storage, "faces": faces, "solver": solver}


def listed():
    return [
        # the smoke puff's preview run (48 cells on the longest axis): a designer's turn-around, all latency
        step_case("step_preview_puff", (38, 48, 38), recipe="puff"),
        # the small puff run of the benchmark configurations
        step_case("step_64x96x64", (64, 96, 64)),
        # the full smoke-puff recipe's own grid (2 m x 2.5 m x 2 m at 0.025 m)
        step_case("step_puff_80x100x80", (80, 100, 80), recipe="puff"),
        # a ragged grid in a closed box, half storage: no axis halves evenly, rows are odd
        step_case("step_odd_f16_closed", (75, 113, 91), storage="f16", faces="closed"),
        # the operator-level benchmark grid
        step_case("step_128x192x128", (128, 192, 128)),
        # the largest grid of the sweeps, stored as bfloat16
        step_case("step_bf16_160x240x160", (160, 240, 160), storage="bf16"),
        # the headline benchmark step
        step_case("step_256x384x256", (256, 384, 256)),
        # the projection on its own, on an uneven grid
        {"name": "project_odd", "kind": "project", "nx": 129, "ny": 97, "nz": 141, "cycles": 4, "faces": "open"},
        # a sheet frame with the light volume (shade layout), as every frame of a run renders one
        {"name": "frame_shade_128", "kind": "frame", "nx": 128, "ny": 192, "nz": 128, "layout": "shade"},
        # a sheet frame with the normal field (normal layout)
        {"name": "frame_normal_96", "kind": "frame", "nx": 96, "ny": 144, "nz": 96, "layout": "normal"},
        # gradients through the step, for fitting a source field and forces to an image
        {"name": "fit_96x144x96", "kind": "fit", "nx": 96, "ny": 144, "nz": 96, "substeps": 4},
        # a parameter sweep of uneven small grids, two frames of every instance
        {"name": "batch_sweep", "kind": "batch", "small": 4, "middle": 2, "large": 1, "frames": 2},
    ]


def draw(rng):
    """One more case: mostly steps, of log-spread sizes, odd ones among them."""
    kind = rng.choices(("step", "project", "frame", "fit", "batch"), weights=(10, 2, 4, 1, 1))[0]
    most = {"step": LARGEST_CELLS, "project": 6_000_000, "frame": 4_000_000, "fit": 1_400_000, "batch": 0}[kind]
    if kind == "batch":
        return {"kind": "batch", "small": rng.randint(1, 4), "middle": rng.randint(0, 2), "large": rng.randint(0, 1),
                "frames": rng.randint(1, 2)}
    cells = math.exp(rng.uniform(math.log(40_000), math.log(0.9 * most)))
    tall, deep = rng.uniform(1.0, 1.6), rng.uniform(0.8, 1.2)
    nx = max(16, round((cells / (tall * deep)) ** (1.0 / 3.0)))
    ny, nz = max(16, round(nx * tall)), max(16, round(nx * deep))
    if rng.random() < 0.5:  # half of the grids are multiples of eight, as recipes choose them
        nx, ny, nz = (max(16, n // 8 * 8) for n in (nx, ny, nz))
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "step":
        case["recipe"] = rng.choice(("plain", "plain", "puff"))
        case["storage"] = rng.choice(("f32", "f32", "f32", "bf16", "f16"))
        case["faces"] = rng.choice(("open", "open", "open", "closed"))
        case["solver"] = "gauss_seidel" if nx * ny * nz < 1_000_000 and rng.random() < 0.15 else "multigrid"
    elif kind == "project":
        case["cycles"] = rng.randint(1, 4)
        case["faces"] = rng.choice(("open", "closed"))
    elif kind == "frame":
        case["layout"] = rng.choice(("shade", "shade", "normal"))
    else:
        case["substeps"] = rng.randint(2, 4)
    return case


# ---- recipes and states ---------------------------------------------------------------------------------------

CLOSED_FACES = dict.fromkeys(("bottom", "top", "left", "right", "back", "front"), "closed")


def puff_recipe(cells):
    """The smoke-puff recipe's physics on any grid: a domain 2 m wide."""
    nx, ny, nz = cells
    cell_m = 2.0 / nx
    return resolve_table({
        "seed": 7,
        "domain": {"size_m": [nx * cell_m, ny * cell_m, nz * cell_m], "cell_m": cell_m},
        "time": {"duration_s": 2.4, "frames": 64},
        "emitter": [{"name": "puff", "center_m": [0.0, 0.35, 0.0], "radius_m": 0.3, "edge_softness": 0.6, "end_s": 0.2,
                     "smoke_per_s": 14.0, "temperature_k": 318.0, "velocity_mps": [0.0, 0.35, 0.0],
                     "noise": {"scale_m": 0.12, "strength": 0.7}}],
        "forces": {"vorticity_confinement": 3.0, "drag_per_s": 0.5,
                   "turbulence": {"scale_m": 0.2, "strength_mps2": 0.12, "speed_mps": 0.2}},
        "dissipation": {"smoke_per_s": 1.6, "cooling_per_s": 1.0},
        "render": {"opacity_per_density": 4.0},
    }, "puff")


def recipe_of(case):
    cells = (case["nx"], case["ny"], case["nz"])
    recipe = puff_recipe(cells) if case.get("recipe") == "puff" else plain_step_recipe(cells, case.get("cycles", 4))
    if case.get("faces") == "closed":
        recipe = dataclasses.replace(recipe, domain=dataclasses.replace(
            recipe.domain, faces=dataclasses.replace(recipe.domain.faces, **CLOSED_FACES)))
    if case.get("solver") == "gauss_seidel":
        recipe = dataclasses.replace(recipe, solver=dataclasses.replace(recipe.solver, pressure_solver="gauss_seidel"))
    if case.get("layout"):
        recipe = dataclasses.replace(
            recipe, camera=dataclasses.replace(recipe.camera, elevation_deg=15.0, azimuth_deg=30.0),
            output=dataclasses.replace(recipe.output,
                                       channels=SHADE_LAYOUT if case["layout"] == "shade" else NORMAL_LAYOUT))
    return recipe


def smooth_noise(shape, generator, passes=3):
    x = torch.rand(shape, generator=generator, device=DEVICE) * 2.0 - 1.0
    for _ in range(passes):
        x = torch.nn.functional.avg_pool3d(
            torch.nn.functional.pad(x[None, None], (1, 1, 1, 1, 1, 1), mode="replicate"), 3, stride=1)[0, 0]
    return x


def moving_state(cells, ambient_k, warmth_k, cell_speed, seed):
    """A plume under way: a rising jet of up to 0.6 cells a step over smooth noise (0.08 cells a step rms), a
    ragged cloud of smoke around it, warm where there is smoke. `cell_speed`: one cell per step, in m/s."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    nx, ny, nz = cells
    axis = [(torch.arange(n, device=DEVICE, dtype=torch.float32) + 0.5) / n - 0.5 for n in cells]
    x, y, z = axis[0][:, None, None], axis[1][None, :, None], axis[2][None, None, :]
    across = x * x + z * z
    state = {}
    for name, shape in (("u", (nx + 1, ny, nz)), ("v", (nx, ny + 1, nz)), ("w", (nx, ny, nz + 1))):
        noise = smooth_noise(shape, g)
        state[name] = noise * (0.08 * cell_speed / noise.std())
    lift = 0.6 * cell_speed * torch.exp(-across / 0.02) * torch.exp(-((y + 0.15) ** 2) / 0.08)
    state["v"][:, 1:, :] += lift
    cloud = smooth_noise(cells, g)
    cloud = 0.5 + 0.25 * cloud / cloud.std()
    body = across + 0.7 * (y + 0.1) ** 2
    state["smoke"] = torch.where(body < 0.08, cloud.clamp(0.0, 1.0), torch.zeros_like(cloud))
    state["temperature"] = ambient_k + warmth_k * state["smoke"]
    return {name: value.contiguous() for name, value in state.items()}


def state_of(case, recipe, derived, seed, storage=torch.float32):
    warmth = 25.0 if case.get("recipe") == "puff" else 0.8
    state = moving_state(derived.cells, recipe.domain.ambient_k, warmth, recipe.domain.cell_m / derived.dt_s, seed)
    return {name: value.to(storage) for name, value in state.items()}


def new_grid(recipe, derived, storage=torch.float32):
    d = recipe.domain
    return make_grid(derived, d.cell_m, d.faces, d.ambient_k, DEVICE, storage=storage)


def load(grid, state):
    torch._foreach_copy_([getattr(grid, name).data for name in FIELDS], [state[name] for name in FIELDS])
    grid.pressure.zero_()


def fields_of(grid):
    return {name: getattr(grid, name).data for name in FIELDS}


STEP_TIME_S = 0.1  # every emitter is active


# ---- prepare and run ------------------------------------------------------------------------------------------

BATCH_GRIDS = {"small": (48, 48, 48), "middle": (64, 96, 64), "large": (96, 144, 96)}


def batch_recipes(case):
    """The sweep's instances: uneven grids of the same 2 m wide domain, their forces and emitters spread."""
    variations = []
    for size in ("small", "middle", "large"):
        nx, ny, nz = BATCH_GRIDS[size]
        cell_m = 2.0 / nx
        for n in range(case[size]):
            variations.append([f"seed={7 + len(variations)}", f"domain.size_m={[nx * cell_m, ny * cell_m, nz * cell_m]!r}",
                               f"domain.cell_m={cell_m!r}", f"emitter.puff.radius_m={(5.0 + n) * cell_m!r}",
                               f"forces.heat_buoyancy={0.6 + 0.2 * n!r}", f"forces.drag_per_s={0.1 * (n + 1)!r}",
                               f"forces.vorticity_confinement={0.2 + 0.1 * n!r}"])
    return sweep_table(batch_base_table(case["frames"]), variations, "sweep")


def batch_states(case, recipes, seed):
    # the fastest gas crosses about four cells a frame, so that the step cap plans about four substeps of each
    return [moving_state(derive(r).cells, r.domain.ambient_k, 0.8, 4.0 * r.domain.cell_m / derive(r).dt_s, seed + n)
            for n, r in enumerate(recipes)]


FIT_SOURCE = (8, 8, 8)


def fit_parts(case, seed):
    recipe = recipe_of(case)
    derived = derive(recipe)
    view = sheet_domain_view(recipe, derived)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    source = torch.rand(FIT_SOURCE, generator=g, device=DEVICE) * 8.0
    target = torch.rand((view.height_px, view.width_px), generator=g, device=DEVICE) * 0.5
    corner = tuple(max(0, n // 2 - 4) if a != 1 else max(0, n // 8) for a, n in enumerate(derived.cells))
    return recipe, derived, view, source, target, corner


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        recipes = batch_recipes(case)
        states = batch_states(case, recipes, seed)

        def fill(index, grid):
            load(grid, states[index])

        return {"kind": kind, "batch": Batch(recipes, DEVICE, initial_state=fill)}
    if kind == "fit":
        recipe, _, _, source, target, corner = fit_parts(case, seed)
        return {"kind": kind, "fit": FlowFit(recipe, FIT_SOURCE, corner, case["substeps"], DEVICE), "source": source,
                "target": target}
    recipe = recipe_of(case)
    derived = derive(recipe)
    storage = STORAGE[case.get("storage", "f32")]
    state = state_of(case, recipe, derived, seed, storage)
    grid = new_grid(recipe, derived, storage)
    load(grid, state)
    held = {"kind": kind, "grid": grid, "state": state}
    if kind == "step":
        held["stepper"], held["dt"] = Stepper(grid, recipe), derived.dt_s
    elif kind == "project":
        held["solve"] = Multigrid(grid, recipe.solver.multigrid_cycles, recipe.solver.multigrid_sweeps)
    else:
        view = sheet_domain_view(recipe, derived)
        held["renderer"] = FrameRenderer(view, recipe.render, derived.cells, recipe.output.channels, DEVICE)
    return held


def run(state):
    kind = state["kind"]
    if kind == "step":
        load(state["grid"], state["state"])
        state["stepper"].step(STEP_TIME_S, state["dt"])
        return {**fields_of(state["grid"]), "pressure": state["grid"].pressure}
    if kind == "project":
        load(state["grid"], state["state"])
        project(state["grid"], state["solve"])
        return {**{n: getattr(state["grid"], n).data for n in "uvw"}, "pressure": state["grid"].pressure}
    if kind == "frame":
        return state["renderer"].render(state["grid"])
    if kind == "fit":
        loss, source, scalars, thickness = state["fit"].loss_and_grad(state["source"], state["target"])
        return {"loss": loss, "source": source, "scalars": scalars, "thickness": thickness}
    batch = state["batch"]
    batch.reset()
    batch.run()
    return [fields_of(grid) for grid in batch.grids]


def work(case):
    """Bytes: each array that carries the state read once and written once. Flops: the equations' operations."""
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for size in BATCH_GRIDS:
            cells = math.prod(BATCH_GRIDS[size])
            steps = 4 * case["frames"] * case[size]
            total["bytes"] += 48.0 * cells * steps
            total["flops"] += 2400.0 * cells * steps
        return total
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "step":
        width = 4.0 if case["storage"] == "f32" else 2.0
        cycles = 2 if case["recipe"] == "puff" else 4
        solve = 130.0 * cycles if case["solver"] == "multigrid" else 11.0 * 60
        # five MacCormack fields (two traces, eight trilinear samples each), forces; turbulence: 24 lattice blends
        return {"bytes": (10 * width + 8.0) * cells,
                "flops": (1500.0 + solve + (1500.0 if case["recipe"] == "puff" else 0.0)) * cells}
    if kind == "project":
        return {"bytes": 32.0 * cells, "flops": (20.0 + 130.0 * case["cycles"]) * cells}
    recipe = recipe_of(case)
    view = sheet_domain_view(recipe, derive(recipe))
    pixels = view.height_px * view.width_px
    if kind == "frame":
        # samples of the march inside the cloud (about a third of its length), and for the shade layout the light
        # of the cloud's cells (about a tenth of the grid), each marched to the edge at half-cell steps
        depth = 2.0 * max(case["nx"], case["nz"])
        flops = pixels * depth / 3 * 80.0
        flops += cells * 0.1 * depth * 40.0 if case["layout"] == "shade" else cells * 70.0
        return {"bytes": 8.0 * cells + 20.0 * pixels, "flops": flops}
    return {"bytes": (48.0 * 3 * cells) * case["substeps"] + 12.0 * pixels, "flops": 6000.0 * cells * case["substeps"]}


# ---- the same paths in float64 --------------------------------------------------------------------------------

F64 = torch.float64


def lerp(a, b, t):
    return a * (1.0 - t) + b * t


def corner_axis(g, n):
    x = g.clamp(0.0, float(n - 1))
    lower = x.floor()
    i0 = lower.long()
    return i0, (i0 + 1).clamp(max=n - 1), x - lower


def sample(f, g, with_range=False):
    """Trilinear sample of `f` at index-space coordinates g = (x, y, z), clamped to the array."""
    (i0, i1, tx), (j0, j1, ty), (k0, k1, tz) = (corner_axis(x, n) for x, n in zip(g, f.shape))
    flat, (_, n1, n2) = f.reshape(-1), f.shape

    def at(i, j, k):
        return flat[(i * n1 + j) * n2 + k]

    corners = [at(i, j, k) for i in (i0, i1) for j in (j0, j1) for k in (k0, k1)]
    c00, c01 = lerp(corners[0], corners[4], tx), lerp(corners[1], corners[5], tx)
    c10, c11 = lerp(corners[2], corners[6], tx), lerp(corners[3], corners[7], tx)
    value = lerp(lerp(c00, c10, ty), lerp(c01, c11, ty), tz)
    if not with_range:
        return value
    lo = hi = corners[0]
    for c in corners[1:]:
        lo, hi = torch.minimum(lo, c), torch.maximum(hi, c)
    return value, lo, hi


FACE = {"u": (0.0, 0.5, 0.5), "v": (0.5, 0.0, 0.5), "w": (0.5, 0.5, 0.0)}
CENTRE = (0.5, 0.5, 0.5)


def positions(shape, offset, device):
    idx = [torch.arange(n, device=device, dtype=F64) + o for n, o in zip(shape, offset)]
    return [x.expand(shape) for x in (idx[0][:, None, None], idx[1][None, :, None], idx[2][None, None, :])]


def velocity_at(velocity, p):
    return [sample(velocity[n], [x - o for x, o in zip(p, FACE[n])]) for n in "uvw"]


def trace(velocity, p, dt_over_cell):
    mid = [x - v * (0.5 * dt_over_cell) for x, v in zip(p, velocity_at(velocity, p))]
    return [x - v * dt_over_cell for x, v in zip(p, velocity_at(velocity, mid))]


def beyond_open(p, box):
    outside = torch.zeros_like(p[0], dtype=torch.bool)
    for x, n, lo, hi in zip(p, box.cells, box.open_lo, box.open_hi):
        if lo:
            outside |= x < 0.0
        if hi:
            outside |= x > n
    return outside


def maccormack(data, offset, velocity, dt_over_cell, box=None, outside=0.0):
    """(next, hat): the clamped MacCormack result and the semi-Lagrangian one; `box`: the value beyond its open
    faces is `outside`."""
    p = positions(data.shape, offset, data.device)
    src = trace(velocity, p, dt_over_cell)
    hat, lo, hi = sample(data, [x - o for x, o in zip(src, offset)], with_range=True)
    if box is not None:
        gone = beyond_open(src, box)
        hat, lo, hi = (torch.where(gone, outside, x) for x in (hat, lo, hi))
    del src
    back_at = trace(velocity, p, -dt_over_cell)
    back = sample(hat, [x - o for x, o in zip(back_at, offset)])
    if box is not None:
        back = torch.where(beyond_open(back_at, box), outside, back)
    corrected = hat + 0.5 * (data - back)
    return torch.where(corrected < lo, lo, torch.where(corrected > hi, hi, corrected)), hat


class Box:
    """The grid in float64: cell counts, spacing, origin and which faces are open."""

    def __init__(self, recipe, derived):
        f = recipe.domain.faces
        self.cells, self.cell_m, self.origin = derived.cells, recipe.domain.cell_m, derived.domain_min_m
        self.open_lo = [k == "open" for k in (f.left, f.bottom, f.back)]
        self.open_hi = [k == "open" for k in (f.right, f.top, f.front)]


def hash32(x):
    x = x ^ (x >> 16)
    x = x * 0x7FEB352D & 0xFFFFFFFF
    x = x ^ (x >> 15)
    x = x * 0x846CA68B & 0xFFFFFFFF
    return x ^ (x >> 16)


def lattice(seed, stream, i, j, k):
    shift = 1048576
    h = hash32(torch.tensor(seed + shift & 0xFFFFFFFF, device=i.device))
    h = hash32(h ^ (stream + shift & 0xFFFFFFFF))
    for x in (i, j, k):
        h = hash32(h ^ (x + shift & 0xFFFFFFFF))
    return (h >> 8).to(F64) * (2.0 / 16777215.0) - 1.0


def fade(t):
    return t * t * (3.0 - 2.0 * t)


def value_noise(seed, stream, p):
    low = [x.floor() for x in p]
    i, j, k = (x.long() for x in low)
    tx, ty, tz = (fade(x - f) for x, f in zip(p, low))

    def row(dj, dk):
        return lerp(lattice(seed, stream, i, j + dj, k + dk), lattice(seed, stream, i + 1, j + dj, k + dk), tx)

    return lerp(lerp(row(0, 0), row(1, 0), ty), lerp(row(0, 1), row(1, 1), ty), tz)


def soft_edge(distance, extent, softness):
    inner = extent * (1.0 - softness)
    t = (distance - inner) / max(extent - inner, 1e-300)
    return torch.where(distance <= inner, 1.0, torch.where(distance >= extent, 0.0, 1.0 - fade(t)))


def emit(s, box, recipe, time_s, dt):
    for stream, e in enumerate(recipe.emitter):
        if not e.start_s <= time_s < e.end_s:
            continue
        for name in FIELDS:
            offset = FACE.get(name, CENTRE)
            x = [o + p * box.cell_m for o, p in zip(box.origin, positions(s[name].shape, offset, s[name].device))]
            off = [a - c for a, c in zip(x, e.center_m)]
            amount = soft_edge((off[0] ** 2 + off[1] ** 2 + off[2] ** 2).sqrt(), e.radius_m, e.edge_softness)
            if e.noise.strength > 0.0:
                breakup = 1.0 + e.noise.strength * value_noise(recipe.seed, stream, [a / e.noise.scale_m for a in x])
                amount = amount * breakup.clamp(min=0.0)
            amount = amount.clamp(max=1.0)
            blend = 1.0 - (1.0 - amount) ** (dt * 80.0)
            if name == "smoke":
                s[name] = s[name] + e.smoke_per_s * amount * dt
            else:
                target = e.temperature_k if name == "temperature" else e.velocity_mps["uvw".index(name)]
                s[name] = torch.where(amount > 0.0, lerp(s[name], target, blend), s[name])


def neighbours(f, axis):
    """The values one cell below and above along `axis`, clamped at the ends, and the cells between the two."""
    n = f.shape[axis]
    idx = torch.arange(n, device=f.device)
    lo, hi = (idx - 1).clamp(min=0), (idx + 1).clamp(max=n - 1)
    span = (hi - lo).to(F64).reshape([-1 if a == axis else 1 for a in range(3)])
    return f.index_select(axis, lo), f.index_select(axis, hi), span


def difference(f, axis, cell_m):
    lo, hi, span = neighbours(f, axis)
    return torch.where(span > 0.0, (hi - lo) / (span.clamp(min=1.0) * cell_m), 0.0)


def confine(s, box, strength, dt):
    centre = [0.5 * (s[n].narrow(a, 0, box.cells[a]) + s[n].narrow(a, 1, box.cells[a])) for a, n in enumerate("uvw")]
    d = [[difference(c, a, box.cell_m) for c in centre] for a in range(3)]
    curl = [d[1][2] - d[2][1], d[2][0] - d[0][2], d[0][1] - d[1][0]]
    spin = (curl[0] ** 2 + curl[1] ** 2 + curl[2] ** 2).sqrt()
    toward = [difference(spin, a, box.cell_m) for a in range(3)]
    length = (toward[0] ** 2 + toward[1] ** 2 + toward[2] ** 2).sqrt()
    still = length < 1.0e-12
    n = [torch.where(still, 0.0, t / torch.where(still, 1.0, length)) for t in toward]
    cross = [n[1] * curl[2] - n[2] * curl[1], n[2] * curl[0] - n[0] * curl[2], n[0] * curl[1] - n[1] * curl[0]]
    for a, name in enumerate("uvw"):
        push = cross[a] * (strength * box.cell_m)
        faces = torch.arange(box.cells[a] + 1, device=push.device)
        below = push.index_select(a, (faces - 1).clamp(min=0))
        above = push.index_select(a, faces.clamp(max=box.cells[a] - 1))
        s[name] = s[name] + 0.5 * (below + above) * dt


def stir(s, box, recipe, time_s, dt):
    t = recipe.forces.turbulence
    pattern_time, to_lattice = time_s * t.speed_mps / t.scale_m, box.cell_m / t.scale_m
    base, blend = math.floor(pattern_time), fade(pattern_time - math.floor(pattern_time))

    def potential(component, p):
        first = (1 << 24) + 3 * base + component
        p = [x * to_lattice for x in p]
        return lerp(value_noise(recipe.seed, first, p), value_noise(recipe.seed, first + 3, p), blend)

    for a, name in enumerate("uvw"):
        p, b, c = positions(s[name].shape, FACE[name], s[name].device), (a + 1) % 3, (a + 2) % 3

        def moved(axis, by):
            return [x + by if n == axis else x for n, x in enumerate(p)]

        curl = potential(c, moved(b, 0.5)) - potential(c, moved(b, -0.5))
        curl = curl - (potential(b, moved(c, 0.5)) - potential(b, moved(c, -0.5)))
        s[name] = s[name] + t.strength_mps2 * (curl / to_lattice) * dt


class Poisson:
    """One level of the pressure solve: couplings, update and residual."""

    def __init__(self, cells, cell_m, box, fill, gap, device):
        self.cells, self.cell_m, self.fill, self.gap, self.box, self.device = cells, cell_m, fill, gap, box, device
        widths = []
        for a, n in enumerate(cells):
            w = torch.ones(n, dtype=F64, device=device)
            w[n - 1] = fill[a]
            widths.append(w.reshape([-1 if b == a else 1 for b in range(3)]))
        self.volume = widths[0] * widths[1] * widths[2]
        self.total = torch.zeros(cells, dtype=F64, device=device)
        self.pairs = []  # per axis: the coupling across each inner face
        for a, n in enumerate(cells):
            area = widths[(a + 1) % 3] * widths[(a + 2) % 3]
            w = widths[a]
            inner = None
            if n > 1:
                inner = (area / (0.5 * (w.narrow(a, 0, n - 1) + w.narrow(a, 1, n - 1))))
                inner = inner.expand([n - 1 if b == a else cells[b] for b in range(3)])
                self.total.narrow(a, 0, n - 1).add_(inner)
                self.total.narrow(a, 1, n - 1).add_(inner)
            if box.open_lo[a]:
                self.total.narrow(a, 0, 1).add_(area / (0.5 * w.narrow(a, 0, 1) + gap))
            if box.open_hi[a]:
                self.total.narrow(a, n - 1, 1).add_(area / (0.5 * w.narrow(a, n - 1, 1) + gap))
            self.pairs.append(inner)
        idx = [torch.arange(n, device=device) for n in cells]
        self.red = ((idx[0][:, None, None] + idx[1][None, :, None] + idx[2][None, None, :]) & 1) == 0

    def gathered(self, q):
        out = torch.zeros_like(q)
        for a, n in enumerate(self.cells):
            if n > 1:
                out.narrow(a, 1, n - 1).add_(self.pairs[a] * q.narrow(a, 0, n - 1))
                out.narrow(a, 0, n - 1).add_(self.pairs[a] * q.narrow(a, 1, n - 1))
        return out

    def sweep(self, q, rhs, count, relaxation):
        source = self.volume * self.cell_m ** 2 * rhs
        coupled = self.total > 0.0
        for _ in range(count):
            for colour in (self.red, ~self.red):
                target = (self.gathered(q) - source) / torch.where(coupled, self.total, 1.0)
                q = torch.where(colour & coupled, q + relaxation * (target - q), q)
        return q

    def residual(self, q, rhs):
        return rhs - (self.gathered(q) - self.total * q) / (self.volume * self.cell_m ** 2)


def poisson_levels(box, device):
    levels, cells, depth = [], box.cells, 0
    while True:
        scale = 2.0 ** depth
        fill = tuple(top / scale - (n - 1) for top, n in zip(box.cells, cells))
        levels.append(Poisson(cells, box.cell_m * scale, box, fill, 0.5 / scale, device))
        if min(cells) <= 2 or len(levels) == 8:
            return levels
        cells, depth = tuple((n + 1) // 2 for n in cells), depth + 1


def v_cycle(levels, q, rhs, sweeps):
    level = levels[0]
    if len(levels) == 1:
        return level.sweep(q, rhs, max(20, 4 * max(level.cells)), 1.5)
    q = level.sweep(q, rhs, sweeps, 1.0)
    coarse = levels[1]
    padding = [x for a in (2, 1, 0) for x in (0, 2 * coarse.cells[a] - level.cells[a])]

    def children(x):
        return torch.nn.functional.avg_pool3d(torch.nn.functional.pad(x, padding)[None, None], 2)[0, 0]

    restricted = children(level.residual(q, rhs)) / children(torch.ones_like(q))
    e = v_cycle(levels[1:], torch.zeros(coarse.cells, dtype=F64, device=q.device), restricted, sweeps)
    p = positions(level.cells, (0.0, 0.0, 0.0), q.device)
    return level.sweep(q + sample(e, [0.5 * x - 0.25 for x in p]), rhs, sweeps, 1.0)


def make_divergence_free(s, box, solver, pressure):
    for a, name in enumerate("uvw"):
        if not box.open_lo[a]:
            s[name].select(a, 0).zero_()
        if not box.open_hi[a]:
            s[name].select(a, box.cells[a]).zero_()
    rhs = sum(s[n].narrow(a, 1, box.cells[a]) - s[n].narrow(a, 0, box.cells[a]) for a, n in enumerate("uvw")) / box.cell_m
    levels = poisson_levels(box, pressure.device)
    if solver.pressure_solver == "gauss_seidel":
        pressure = levels[0].sweep(pressure, rhs, solver.pressure_iterations, 1.5)
    else:
        for _ in range(solver.multigrid_cycles):
            pressure = v_cycle(levels, pressure, rhs, solver.multigrid_sweeps)
    for a, name in enumerate("uvw"):
        n = box.cells[a]
        f = s[name]
        f.narrow(a, 1, n - 1).sub_((pressure.narrow(a, 1, n - 1) - pressure.narrow(a, 0, n - 1)) / box.cell_m)
        if box.open_lo[a]:
            f.narrow(a, 0, 1).sub_(pressure.narrow(a, 0, 1) / box.cell_m)
        if box.open_hi[a]:
            f.narrow(a, n, 1).add_(pressure.narrow(a, n - 1, 1) / box.cell_m)
    return pressure


def exact_step(s, pressure, box, recipe, time_s, dt):
    """One substep of the state `s` (float64 arrays, replaced); returns the pressure."""
    forces, ambient = recipe.forces, recipe.domain.ambient_k
    emit(s, box, recipe, time_s, dt)
    rows = torch.arange(box.cells[1] + 1, device=pressure.device)
    below, above = (rows - 1).clamp(min=0), rows.clamp(max=box.cells[1] - 1)
    heat, density = (0.5 * (s[n].index_select(1, below) + s[n].index_select(1, above)) for n in ("temperature", "smoke"))
    lift = forces.heat_buoyancy * (heat - ambient) / ambient - forces.smoke_weight * density
    s["v"] = s["v"] + forces.gravity_mps2 * lift * dt
    if forces.vorticity_confinement > 0.0:
        confine(s, box, forces.vorticity_confinement, dt)
    if forces.turbulence.strength_mps2 != 0.0:
        stir(s, box, recipe, time_s, dt)
    if forces.drag_per_s != 0.0:
        keep = math.exp(-forces.drag_per_s * dt)
        for a, name in enumerate("uvw"):
            s[name] = forces.wind_mps[a] + (s[name] - forces.wind_mps[a]) * keep
    over = dt / box.cell_m
    before = {n: s[n] for n in "uvw"}
    for name in "uvw":
        s[name] = maccormack(before[name], FACE[name], before, over)[0]
    del before
    pressure = make_divergence_free(s, box, recipe.solver, pressure)
    velocity = {n: s[n] for n in "uvw"}
    smoke, hat = maccormack(s["smoke"], CENTRE, velocity, over, box, 0.0)
    was, plain, total = (float(x.sum()) for x in (s["smoke"], hat, smoke))
    s["smoke"] = smoke * (max(plain, min(total, was)) / total if total > 0.0 else 1.0)
    s["temperature"] = maccormack(s["temperature"], CENTRE, velocity, over, box, ambient)[0]
    loss = recipe.dissipation
    if loss.smoke_per_s != 0.0 or loss.cooling_per_s != 0.0:
        s["smoke"] = s["smoke"] * math.exp(-loss.smoke_per_s * dt)
        s["temperature"] = ambient + (s["temperature"] - ambient) * math.exp(-loss.cooling_per_s * dt)
    return pressure


def slab(origin, direction, low, high):
    """Where the rays enter and leave the box; rays parallel to an axis never start outside it here."""
    enter = torch.full_like(origin[0], -1.0e30)
    leave = torch.full_like(origin[0], 1.0e30)
    for o, d, a, b in zip(origin, direction, low, high):
        if abs(d) < 1.0e-12:
            miss = (o < a) | (o > b)
            enter, leave = torch.where(miss, 1.0, enter), torch.where(miss, 0.0, leave)
            continue
        t0, t1 = (a - o) / d, (b - o) / d
        enter, leave = torch.maximum(enter, torch.minimum(t0, t1)), torch.minimum(leave, torch.maximum(t0, t1))
    return enter, leave


def light_volume(smoke, toward, cell_m, opacity):
    """exp(-opacity * column toward the light) at every cell, marched at steps of at most half a cell."""
    start = [x.reshape(-1) for x in positions(smoke.shape, CENTRE, smoke.device)]
    _, length = slab(start, toward, (0.0, 0.0, 0.0), [float(n) for n in smoke.shape])
    steps = (length / 0.5).ceil()
    step = length / steps
    column = torch.zeros_like(length)
    alive = torch.arange(length.numel(), device=smoke.device)
    for n in range(int(steps.max())):
        alive = alive[steps[alive] > n]
        t = (n + 0.5) * step[alive]
        density = sample(smoke, [x[alive] - 0.5 + d * t for x, d in zip(start, toward)]).clamp(min=0.0)
        column[alive] += density * step[alive]
    return torch.exp(-opacity * column * cell_m).reshape(smoke.shape)


def blurred_gradient(smoke, sigma):
    radius = math.ceil(3.0 * sigma) if sigma > 0 else 0
    taps = np.exp(-np.arange(-radius, radius + 1) ** 2 / (2.0 * sigma ** 2)) if radius else np.ones(1)
    taps = taps / taps.sum()
    f = smoke
    for a in range(3):
        idx = torch.arange(f.shape[a], device=f.device)
        f = sum(float(w) * f.index_select(a, (idx + o).clamp(0, f.shape[a] - 1))
                for w, o in zip(taps, range(-radius, radius + 1)))
    return [difference(f, a, 1.0) for a in range(3)]


def march(smoke, temperature, box, view, settings, layout):
    """The raw frame (H, W, 5) of an orthographic view; with `layout` None, the thickness alone."""
    device, cam, cell = smoke.device, view.camera, box.cell_m
    right, up, toward = (np.asarray(v, dtype=np.float64) for v in (cam.right, cam.up, cam.toward))
    px = (view.left_m + (torch.arange(view.width_px, device=device, dtype=F64) + 0.5) * view.pixel_m)[None, :]
    py = (view.top_m - (torch.arange(view.height_px, device=device, dtype=F64) + 0.5) * view.pixel_m)[:, None]
    origin = [(float(right[a]) * px + float(up[a]) * py + float(toward[a]) * 1.0e4).reshape(-1) for a in range(3)]
    direction = [-float(t) for t in toward]
    low = box.origin
    high = [o + n * cell for o, n in zip(low, box.cells)]
    enter, leave = slab(origin, direction, low, high)
    hit = leave > enter
    length = torch.where(hit, leave - enter, 0.0)
    steps = (length / (0.5 * cell)).ceil()
    step = torch.where(hit, length / steps.clamp(min=1.0), 0.0)
    through = torch.ones_like(length)
    heat, shade = torch.zeros_like(length), torch.zeros_like(length)
    normal = [torch.zeros_like(length) for _ in range(3)]
    light = slope_of = None
    if layout == "shade":
        x, y, z = settings.light_dir
        to_light = x * right + y * up + z * toward
        to_light = to_light / np.linalg.norm(to_light)
        light = light_volume(smoke, [float(t) for t in to_light], cell, settings.opacity_per_density)
    elif layout == "normal":
        slope_of = blurred_gradient(smoke, settings.normal_blur_cells)
    for n in range(int(steps.max())):
        live = steps > n
        t = enter + (n + 0.5) * step
        g = [(o + d * t - b) / cell - 0.5 for o, d, b in zip(origin, direction, low)]
        density = sample(smoke, g).clamp(min=0.0)
        alpha = torch.where(live, 1.0 - torch.exp(-settings.opacity_per_density * density * step), 0.0)
        if layout:
            glow = torch.where(live, (sample(temperature, g) - settings.glow_start_k).clamp(min=0.0), 0.0)
            heat = heat + glow * step * through ** settings.smoke_hides_heat
        if light is not None:
            shade = shade + through * alpha * (settings.shade_fill + (1.0 - settings.shade_fill) * sample(light, g))
        if slope_of is not None:
            slope = [sample(f, g) for f in slope_of]
            size = (slope[0] ** 2 + slope[1] ** 2 + slope[2] ** 2).sqrt()
            steep = size > 1.0e-9
            normal = [s - torch.where(steep, a / torch.where(steep, size, 1.0), 0.0) * through * alpha
                      for s, a in zip(normal, slope)]
        through = through * (1.0 - alpha)
    thickness = 1.0 - through
    size = (view.height_px, view.width_px)
    if layout is None:
        return thickness.reshape(size)
    zero = torch.zeros_like(heat)
    if layout == "shade":
        return torch.stack([heat, thickness, shade, zero, zero], dim=-1).reshape(*size, 5)
    seen = [sum(float(axis[a]) * normal[a] for a in range(3)) for axis in (right, up, toward)]
    length = (seen[0] ** 2 + seen[1] ** 2 + seen[2] ** 2).sqrt()
    known = length > 1.0e-9
    unit = [torch.where(known, c / torch.where(known, length, 1.0), 0.0) for c in seen]
    weight = (thickness / settings.normal_fade_thickness).clamp(0.0, 1.0)
    facing = [lerp(0.0, unit[0], weight), lerp(0.0, unit[1], weight), lerp(1.0, unit[2].abs(), weight)]
    length = (facing[0] ** 2 + facing[1] ** 2 + facing[2] ** 2).sqrt()
    unit = [torch.where(known, c / length, d) for c, d in zip(facing, (0.0, 0.0, 1.0))]
    return torch.stack([heat, thickness, *unit], dim=-1).reshape(*size, 5)


def wide(state):
    return {name: value.to(F64) for name, value in state.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        recipes = batch_recipes(case)
        return [exact_run(r, wide(s)) for r, s in zip(recipes, batch_states(case, recipes, seed))]
    if kind == "fit":
        return exact_fit(case, seed)
    recipe = recipe_of(case)
    derived = derive(recipe)
    box = Box(recipe, derived)
    s = wide(state_of(case, recipe, derived, seed, STORAGE[case.get("storage", "f32")]))
    pressure = torch.zeros(derived.cells, dtype=F64, device=s["u"].device)
    if kind == "step":
        pressure = exact_step(s, pressure, box, recipe, STEP_TIME_S, derived.dt_s)
        return {**s, "pressure": pressure}
    if kind == "project":
        pressure = make_divergence_free(s, box, recipe.solver, pressure)
        return {**{n: s[n] for n in "uvw"}, "pressure": pressure}
    view = sheet_domain_view(recipe, derived)
    return march(s["smoke"], s["temperature"], box, view, recipe.render, case["layout"])


def exact_run(recipe, s):
    """A whole run with its step cap: each frame split so that the fastest gas crosses at most max_cells_per_step."""
    derived = derive(recipe)
    box, solver = Box(recipe, derived), recipe.solver
    pressure = torch.zeros(derived.cells, dtype=F64, device=s["u"].device)
    length = derived.steps_per_frame * derived.dt_s
    for frame in range(recipe.time.frames):
        speed = max(float(s[n].abs().max()) for n in "uvw")
        steps = max(derived.steps_per_frame, math.ceil(speed * length / (solver.max_cells_per_step * box.cell_m)))
        for n in range(steps):
            pressure = exact_step(s, pressure, box, recipe, frame * length + n * length / steps, length / steps)
    return s


def exact_fit(case, seed):
    """The loss and the thickness image; the gradients are those of a converged projection, not of these cycles."""
    recipe, derived, view, source, target, corner = fit_parts(case, seed)
    box, cells = Box(recipe, derived), derived.cells
    shapes = {"u": (cells[0] + 1, cells[1], cells[2]), "v": (cells[0], cells[1] + 1, cells[2]),
              "w": (cells[0], cells[1], cells[2] + 1), "smoke": cells, "temperature": cells}
    s = {n: torch.zeros(shape, dtype=F64, device=source.device) for n, shape in shapes.items()}
    s["temperature"] += recipe.domain.ambient_k
    pressure = torch.zeros(cells, dtype=F64, device=source.device)
    window = tuple(slice(c, c + n) for c, n in zip(corner, FIT_SOURCE))
    for n in range(case["substeps"]):
        s["smoke"][window] += derived.dt_s * source.to(F64)
        pressure = exact_step(s, pressure, box, recipe, n * derived.dt_s, derived.dt_s)
    thickness = march(s["smoke"], s["temperature"], box, view, recipe.render, None)
    error = thickness - target.to(F64)
    return {"loss": float((error * error).sum()), "source": None, "scalars": None, "thickness": thickness}
