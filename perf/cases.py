"""The solver's performance cases: what programs that use this framework have it do, as calls of
hnanosolver_b200.lib (and, where a call takes device pointers that the binding has no method for,
of the C ABI below it). Each case is a dict of plain values; listed() has the standing ones, draw()
more of the same ranges.

Kinds of call:
  operators     the three SOP operators one after the other (HNanoAdvectVelocity, HNanoAdvect,
                HNanoProjectNonDivergent) on device arrays
  step          the SOP chain as one FP32 step (hns_step_plain), with both kinds of wall, a fixed
                iteration count or a tolerance
  advance       the all-in-one FP32 step of the HNanoSolver SOP on the context's named fields
                (hns_advance_model), set from and read back to device arrays
  mixed         the SOP chain on BF16/FP16 storage with the FP64-refined solve (hns_step_mixed)
  mixed_host    the same from and to the host application's FP32 arrays (hns_step_mixed_host)
  fire          the all-in-one step on BF16/FP16 storage (hns_advance_mixed)
  adjoint_step  the reverse pass of one FP32 step (hns_adjoint_step_plain)
  adjoint_fire  the reverse pass of one mixed fire step (hns_adjoint_advance_mixed)
  topology      a grid built on the device from its active voxels (hns_create_from_voxels)

Grids are those of hnanosolver_b200.synth: full boxes, narrow-band shells, unions of spheres.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from hnanosolver_b200 import lib as hl
from hnanosolver_b200 import synth

DX = 0.1  # voxel size of every configuration of this repository
FIELDS_ORDER = ("density", "temperature", "fuel", "waste", "flame")


# ---- the cases ---------------------------------------------------------------------------------

def _grid(shape, extent, count=0, rmin=0.0, rmax=0.0, grid_seed=0):
    return {"shape": shape, "extent": extent, "count": count, "rmin": rmin, "rmax": rmax, "grid_seed": grid_seed}


def listed():
    return [
        # A SOP network's three operator nodes on a small sparse smoke: latency and launches count.
        {"name": "operators_spheres64", "kind": "operators", **_grid("spheres", 64, 2, 8.0, 16.0, 3), "speed": 3.0,
         "dt": 0.1, "iterations": 20, "omega": 1.0},
        # The smallest configuration: one FP32 step of a 64^3 box, 40 iterations.
        {"name": "step_box64", "kind": "step", **_grid("box", 64), "speed": 1.0, "dt": 0.1, "scalars": 1, "walls": "open",
         "iterations": 40, "omega": 1.0, "tolerance": 0.0, "check_every": 0},
        # The sparse plume's grid with the zero-gradient walls its configuration names.
        {"name": "step_plume256_walls", "kind": "step", **_grid("spheres", 256, 8, 20.0, 60.0), "speed": 1.0,
         "dt": 1.0 / 24.0, "scalars": 1, "walls": "closed", "iterations": 100, "omega": 1.8, "tolerance": 0.0,
         "check_every": 0},
        # The narrow-band shell in full FP32, solved to 1e-5 under a generous iteration cap.
        {"name": "step_shell512", "kind": "step", **_grid("shell", 512), "speed": 1.0, "dt": 0.1, "scalars": 1,
         "walls": "open", "iterations": 1000, "omega": 1.82, "tolerance": 1e-5, "check_every": 10},
        # The sparse plume's FP32 fire step: rate burn, buoyancy, confinement, 100 iterations.
        {"name": "advance_plume256", "kind": "advance", **_grid("spheres", 256, 8, 20.0, 60.0), "speed": 1.0,
         "dt": 1.0 / 24.0, "burn": "rate", "iterations": 100, "substeps": 1, "resolve": False, "factor_scale": 1.0},
        # HNS_Advance as the SOP calls it: the oxygen burn, two substeps, the disturbance re-solve.
        {"name": "advance_oxygen_spheres160", "kind": "advance", **_grid("spheres", 160, 5, 14.0, 37.0, 5), "speed": 2.0,
         "dt": 1.0 / 24.0, "burn": "oxygen", "iterations": 40, "substeps": 2, "resolve": True, "factor_scale": 0.5},
        # The headline: one mixed step of the narrow-band shell, multigrid inside the refinement.
        {"name": "mixed_shell512", "kind": "mixed", **_grid("shell", 512), "speed": 1.0, "dt": 0.1, "scalars": 1,
         "inner": "multigrid", "omega": 1.92, "inner_iterations": 2, "max_outer": 8},
        # A host application's frame: FP32 arrays in host memory, red-black inner solves.
        {"name": "mixed_host_plume256", "kind": "mixed_host", **_grid("spheres", 256, 8, 20.0, 60.0), "speed": 1.0,
         "dt": 1.0 / 24.0, "scalars": 1, "inner": "red-black", "omega": 1.9, "inner_iterations": 30, "max_outer": 12},
        # The largest: the 1024^3 sparse fire, 95.6M voxels, solved to 1e-5.
        {"name": "fire_1024", "kind": "fire", **_grid("spheres", 1024, 32, 30.0, 120.0), "speed": 1.0, "dt": 1.0 / 24.0,
         "burn": "rate", "inner": "multigrid", "omega": 1.97, "inner_iterations": 2, "max_outer": 16},
        # The differentiable rollout's reverse step: 128^3 box, 60 iterations.
        {"name": "adjoint_step_box128", "kind": "adjoint_step", **_grid("box", 128), "speed": 1.0, "dt": 0.1, "scalars": 1,
         "iterations": 60, "omega": 1.0},
        # The reverse pass of the mid-size fire's step.
        {"name": "adjoint_fire512", "kind": "adjoint_fire", **_grid("spheres", 512, 32, 15.0, 60.0), "speed": 1.0,
         "dt": 1.0 / 24.0, "burn": "rate", "inner": "multigrid", "omega": 1.95, "inner_iterations": 2, "max_outer": 16},
        # A frame's new domain: the band's active voxels, dilated by two, to a solver grid.
        {"name": "topology_shell512", "kind": "topology", **_grid("shell", 512), "padding": 2, "band": 12.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _drawn_grid(rng, largest):
    """A grid of 64^3-box size up to about `largest` voxels, of any of the three shapes."""
    target = _log(rng, 5e4, largest)
    shape = rng.choice(("box", "spheres", "spheres", "spheres", "shell"))
    seed = rng.randrange(1000)
    if shape == "box":
        return _grid("box", 8 * max(2, round(target ** (1.0 / 3.0) / 8.0)))
    if shape == "shell":  # a band about 48 voxels thick around a sphere
        extent = 8 * max(8, min(64, round(math.sqrt(target / (math.pi * 48.0)) / 0.78 / 8.0)))
        return _grid("shell", extent, grid_seed=seed)
    # About `count` spheres of mean radius 0.16 extent (padded by the leaf half-diagonal), a third overlapping.
    count = rng.randrange(2, 12)
    radius = (target / (0.7 * count * 4.19)) ** (1.0 / 3.0)
    extent = 8 * max(5, min(64, round(radius / 0.16 / 8.0)))
    return _grid("spheres", extent, count, round(0.08 * extent, 1), round(0.24 * extent, 1), seed)


def draw(rng):
    kind = rng.choice(("operators", "step", "step", "advance", "advance", "mixed", "mixed", "mixed_host", "fire", "fire",
                       "adjoint_step", "adjoint_fire", "topology"))
    largest = {"operators": 6e6, "step": 6e6, "advance": 6e6, "mixed": 2.5e7, "mixed_host": 6e6, "fire": 2.5e7,
               "adjoint_step": 4e6, "adjoint_fire": 1.2e7, "topology": 2.5e7}[kind]
    case = {"kind": kind, **_drawn_grid(rng, largest)}
    if kind == "topology":
        return {**case, "padding": rng.choice((0, 1, 2, 3, 5)), "band": float(rng.choice((6, 9, 12)))}
    case.update(speed=rng.choice((0.5, 1.0, 2.0, 4.0)), dt=rng.choice((0.1, 1.0 / 24.0)))
    if kind in ("operators", "step", "adjoint_step"):
        case.update(iterations=rng.randrange(8, 101), omega=round(rng.uniform(1.0, 1.85), 2))
    if kind in ("step", "adjoint_step", "mixed", "mixed_host"):
        case["scalars"] = rng.choice((0, 1, 1, 1, 2, 3))
    if kind == "step":
        case.update(walls=rng.choice(("open", "open", "closed")), tolerance=0.0, check_every=0)
        if case["walls"] == "open" and rng.random() < 0.4:
            case.update(iterations=rng.randrange(200, 501), tolerance=1e-4, check_every=rng.choice((10, 20)))
    if kind == "advance":
        case.update(burn=rng.choice(("rate", "oxygen", "none")), iterations=rng.randrange(10, 101),
                    substeps=rng.choice((1, 1, 2)), resolve=rng.random() < 0.5, factor_scale=rng.choice((0.5, 1.0, 2.0)))
    if kind in ("fire", "adjoint_fire"):
        case["burn"] = rng.choice(("rate", "rate", "oxygen"))
    if kind in ("mixed", "mixed_host", "fire", "adjoint_fire"):
        if rng.random() < 0.65:
            case.update(inner="multigrid", omega=1.9, inner_iterations=rng.choice((1, 2, 2, 3)), max_outer=16)
        else:
            case.update(inner="red-black", omega=1.9, inner_iterations=rng.choice((30, 36, 40)), max_outer=16)
    return case


# ---- grids and fields ----------------------------------------------------------------------------

@functools.lru_cache(maxsize=16)
def _origins(shape, extent, count, rmin, rmax, grid_seed):
    if shape == "box":
        return synth.sort_leaves_nanovdb(synth._box_leaves(extent))
    if shape == "shell":
        return synth.shell_topology(extent, 200.0 * extent / 512.0, 16.0, grid_seed)
    return synth.spheres_topology(extent, count, rmin, rmax, grid_seed)


def _leaves(case):
    return _origins(case["shape"], case["extent"], case["count"], case["rmin"], case["rmax"], case["grid_seed"])


def _noise(origins, generator):
    """Value noise in [0, 1] on the leaves' slots (synth.value_noise_leaves, made on the device)."""
    dev = torch.device("cuda")
    o = torch.from_numpy(origins).to(dev).long() >> 3
    cell = o - o.min(dim=0).values
    lattice = torch.rand(tuple(int(v) + 2 for v in cell.max(dim=0).values), device=dev, generator=generator)
    t = torch.from_numpy(synth.local_offsets()).to(dev).float() / 8.0
    weights, corners = [], []
    for q in range(8):
        d = (q >> 2, (q >> 1) & 1, q & 1)
        weights.append(torch.stack([t[:, k] if d[k] else 1.0 - t[:, k] for k in range(3)]).prod(dim=0))
        corners.append(lattice[cell[:, 0] + d[0], cell[:, 1] + d[1], cell[:, 2] + d[2]])
    w, c = torch.stack(weights), torch.stack(corners, dim=1)
    out = torch.zeros((len(origins), 512), device=dev)
    for q in range(8):
        out.addcmul_(c[:, q:q + 1], w[q:q + 1])
    return out.reshape(-1)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _velocity(case, origins, gen):
    return torch.stack([(2.0 * _noise(origins, gen) - 1.0) * case["speed"] for _ in range(3)], dim=1).contiguous()


def _scalar_names(burn):
    return {"rate": ("density", "temperature", "fuel", "flame"), "none": ("density", "temperature"),
            "oxygen": ("density", "temperature", "fuel", "waste", "flame")}[burn]


def _fire_inputs(case, origins, seed):
    """FP32 fields and sources of a burning state: warm smoke with fuel in it, and an emitter."""
    gen = _generator(seed)
    fields = {"velocity": _velocity(case, origins, gen)}
    for name in _scalar_names(case["burn"]):
        f = _noise(origins, gen)
        fields[name] = 2.0 * f if name == "temperature" else 0.4 * f if name in ("fuel", "waste") else f
    c = torch.from_numpy(origins).cuda().float()
    pos = (c[:, None, :] + torch.from_numpy(synth.local_offsets()).cuda().float()[None]).reshape(-1, 3)
    centre = c[len(origins) // 3] + 3.5
    emitter = (torch.linalg.vector_norm(pos - centre, dim=1) <= 10.0).float()
    return fields, {"temperature": 2.0 * emitter, "fuel": emitter.clone()}


def _params(case):
    p = hl.CombustionParams()
    p.expansionRate, p.temperatureRelease = 0.1, 0.5
    p.vorticityScale, p.factorScale = 0.3, case.get("factor_scale", 1.0)
    p.disturbanceEnable = 1.0 if case.get("resolve") else 0.0
    p.substeps = case.get("substeps", 1)
    if case["burn"] == "oxygen":  # the reference's buoyancy and gravity, a warm ambient
        p.buoyancyStrength, p.ambientTemp, p.gravity = 1.0, 0.5, 1.0
    else:
        p.buoyancyStrength, p.ambientTemp, p.gravity = 0.5, 0.0, 0.0
    m = hl.ForceModel(combustion={"oxygen": 0, "rate": 1, "none": 2}[case["burn"]], burn_rate=0.5, heat_release=1.0,
                      ignition_temp=0.0, density_buoyancy=0.0 if case["burn"] == "oxygen" else 0.1)
    return p, m


def _mixed_desc(case, dt):
    return hl.MixedDesc(dt=dt, omega=case["omega"], tolerance=1e-5, max_outer=case["max_outer"],
                        inner_iterations=case["inner_iterations"],
                        flags=hl.SOLVE_MULTIGRID if case["inner"] == "multigrid" else 0)


def _half(fields):
    return {k: v.to(torch.bfloat16 if v.ndim == 2 else torch.float16) for k, v in fields.items()}


def _band_voxels(case, seed):
    """Active voxels (n, 3) int32 on the device: those that a frame would have active (a band of the
    shell, about 7/8 of the voxels of other grids), shifted by some voxels, in random leaf order."""
    origins = _leaves(case)
    gen = _generator(seed)
    o = torch.from_numpy(origins).cuda()[torch.randperm(len(origins), device="cuda", generator=gen)]
    pos = (o[:, None, :] + torch.from_numpy(synth.local_offsets()).cuda()[None]).reshape(-1, 3)
    if case["shape"] == "shell":
        centre = torch.from_numpy(origins).cuda().float().mean(dim=0) + 3.5
        d = torch.linalg.vector_norm(pos.float() - centre, dim=1) - 200.0 * case["extent"] / 512.0
        keep = d.abs() <= case["band"]
    else:
        keep = torch.rand(len(pos), device="cuda", generator=gen) < 0.875
    shift = torch.randint(-40, 41, (3,), device="cuda", generator=gen, dtype=torch.int32)
    return (pos[keep].int() + shift).contiguous()


# ---- what a program has before the call ------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "topology":
        # The program keeps the new grid's leaf list in an array of its own.
        s = {"case": case, "voxels": _band_voxels(case, seed),
             "leaves": np.zeros((8 * len(_leaves(case)) + 4096, 3), np.int32)}
        torch.cuda.synchronize()
        return s
    origins = _leaves(case)
    s = {"case": case, "grid": hl.Grid(origins, voxel_size=DX)}
    if kind in ("advance", "fire", "adjoint_fire"):
        fields, sources = _fire_inputs(case, origins, seed)
        s["params"], s["model"] = _params(case)
        if kind == "advance":
            s.update(fields=fields, sources=sources, out={k: torch.empty_like(v) for k, v in fields.items()})
        else:
            s.update(fields=_half(fields), sources=_half(sources), desc=_mixed_desc(case, 0.0))
            if kind == "fire":
                s["out"] = {k: torch.empty_like(v) for k, v in s["fields"].items()}
            else:
                gen = _generator(seed + 500)
                s["out_bar"] = {k: torch.randn(v.shape, device="cuda", generator=gen) for k, v in fields.items()}
                s["in_bar"] = {k: torch.empty_like(v) for k, v in fields.items()}
    else:
        gen = _generator(seed)
        vel = _velocity(case, origins, gen)
        scalars = [_noise(origins, gen) for _ in range(case.get("scalars", 1))]
        if kind == "mixed":
            s.update(vel=vel.bfloat16(), scalars=[x.half() for x in scalars], desc=_mixed_desc(case, case["dt"]))
        elif kind == "mixed_host":
            s.update(pinned=[t.cpu().pin_memory() for t in (vel, *scalars)], desc=_mixed_desc(case, case["dt"]))
            s["host"] = [t.numpy() for t in s["pinned"]]
        else:
            s.update(vel=vel, scalars=scalars)
        if kind == "step":
            s["desc"] = hl.StepDesc(dt=case["dt"], max_iterations=case["iterations"], omega=case["omega"],
                                    tolerance=case["tolerance"], check_every=case["check_every"],
                                    flags=hl.SOLVE_NEUMANN if case["walls"] == "closed" else 0)
        if kind in ("operators", "step", "mixed"):
            s.update(vel_out=torch.empty_like(s["vel"]), scalars_out=[torch.empty_like(x) for x in s["scalars"]])
        if kind == "adjoint_step":
            s.update(vel_bar=torch.randn(vel.shape, device="cuda", generator=gen),
                     scalars_bar=[torch.randn(x.shape, device="cuda", generator=gen) for x in scalars],
                     vel_in_bar=torch.empty_like(vel), scalars_in_bar=[torch.empty_like(x) for x in scalars])
    if kind.startswith("adjoint"):  # the program zeroes the gradients on the stream that the solver works on
        s["stream"] = torch.cuda.Stream()
        s["grid"].set_stream(s["stream"].cuda_stream)
    torch.cuda.synchronize()
    return s


# ---- one pass --------------------------------------------------------------------------------------

def run(state):
    case, g = state["case"], state.get("grid")
    kind = case["kind"]
    if kind == "operators":
        g.advect_vec3(state["vel"], state["vel_out"], case["dt"])
        g.advect_scalar(state["vel"], state["scalars"][0], state["scalars_out"][0], case["dt"])
        g.project(state["vel_out"], case["iterations"], case["omega"], info=False)
        return [state["vel_out"], state["scalars_out"][0]]
    if kind == "step":
        g.step_plain(state["vel"], state["vel_out"], state["scalars"], state["scalars_out"], state["desc"])
        return [state["vel_out"], *state["scalars_out"]]
    if kind == "advance":
        c = hl.lib
        for name, t in state["fields"].items():
            hl.check(c.hns_field_set(g.handle, name.encode(), 3 if t.ndim == 2 else 1, t.data_ptr(), 1))
        for name, t in state["sources"].items():
            hl.check(c.hns_field_set(g.handle, b"src_" + name.encode(), 1, t.data_ptr(), 1))
        g.advance(case["iterations"], case["dt"], state["params"], state["model"])
        for name, t in state["out"].items():
            hl.check(c.hns_field_get(g.handle, name.encode(), ctypes.c_void_p(t.data_ptr()), 1))
        return state["out"]
    if kind == "mixed":
        g.step_mixed(state["vel"], state["vel_out"], state["scalars"], state["scalars_out"], state["desc"])
        return [state["vel_out"], *state["scalars_out"]]
    if kind == "mixed_host":  # in place: the next pass goes on from this one's fields
        g.step_mixed_host(state["host"][0], state["host"][1:], state["desc"])
        return list(state["host"])
    if kind == "fire":
        g.advance_mixed(state["fields"], state["out"], state["sources"], case["dt"], state["params"], state["model"],
                        state["desc"])
        return state["out"]
    if kind == "adjoint_step":
        with torch.cuda.stream(state["stream"]):
            state["vel_in_bar"].zero_()
            for t in state["scalars_in_bar"]:
                t.zero_()
            g.adjoint_step_plain(state["vel"], state["scalars"], state["vel_bar"], state["scalars_bar"],
                                 state["vel_in_bar"], state["scalars_in_bar"], case["dt"], case["iterations"],
                                 case["omega"])
        return [state["vel_in_bar"], *state["scalars_in_bar"]]
    if kind == "adjoint_fire":
        with torch.cuda.stream(state["stream"]):
            for t in state["in_bar"].values():
                t.zero_()
            g.adjoint_advance_mixed(state["fields"], state["sources"], state["out_bar"], state["in_bar"], case["dt"],
                                    state["params"], state["model"], state["desc"])
        return state["in_bar"]
    if kind == "topology":
        grid = hl.Grid(voxels=state["voxels"], padding=case["padding"], voxel_size=DX)
        state["leaves"][:grid.num_leaves] = grid.leaf_origins()
        grid.close()
        return state["leaves"]
    raise ValueError(kind)


# ---- the work a pass cannot do without -------------------------------------------------------------

def work(case):
    n = 512.0 * len(_leaves(case))
    kind, scalars = case["kind"], case.get("scalars", 1)
    advect_v, advect_s, relax = 170.0, 60.0, 10.0  # operations per voxel: MacCormack, one red-black iteration
    project = 8.0 + 12.0
    if kind == "topology":
        return {"bytes": 12.0 * 0.6 * n + 12.0 * n / 512, "flops": 0.0}
    if kind in ("operators", "step"):
        return {"bytes": n * (24 + 8 * scalars), "flops": n * (advect_v + scalars * advect_s + project +
                                                                 relax * min(case["iterations"], 470))}
    if kind == "adjoint_step":
        return {"bytes": n * (36 + 12 * scalars), "flops": n * (2 * (advect_v + scalars * advect_s) + project +
                                                                  relax * case["iterations"])}
    # A solve to 1e-5: about six multigrid cycles, or a few hundred red-black iterations.
    solve = 6 * 60.0 if case.get("inner") == "multigrid" else 180 * relax
    if kind in ("mixed", "mixed_host"):
        size = 2.0 if kind == "mixed" else 4.0
        return {"bytes": n * size * 2 * (3 + scalars), "flops": n * (advect_v + scalars * advect_s + project + solve)}
    names = len(_scalar_names(case["burn"]))
    forces = 150.0
    if kind == "advance":
        its = case["iterations"] + (max(2, case["iterations"] // 2) if case["resolve"] else 0)
        return {"bytes": n * 4 * (2 * (3 + names) + 2),
                "flops": n * case["substeps"] * (advect_v + names * advect_s + project + forces + relax * its)}
    if kind == "fire":
        return {"bytes": n * 2 * (2 * (3 + names) + 2), "flops": n * (advect_v + names * advect_s + project + forces + solve)}
    return {"bytes": n * (2 * (3 + names + 2) + 8 * (3 + names)),
            "flops": 2 * n * (advect_v + names * advect_s + project + forces + solve)}


# ---- the same in 64 bits -----------------------------------------------------------------------------

class _Exact:
    """The step's operators in FP64 on slot-ordered arrays. A missing voxel reads the entry past the
    last slot (0), or slot 0 in the multi-field advection, as the reference does."""

    def __init__(self, origins):
        dev = torch.device("cuda")
        self.n = 512 * len(origins)
        o = torch.from_numpy(origins).to(dev).long()
        self.lo = (o.min(dim=0).values >> 3) - 1
        dims = (o.max(dim=0).values >> 3) - self.lo + 2
        self.dims = [int(v) for v in dims]
        self.table = torch.full(self.dims, -1, device=dev, dtype=torch.int64)
        c = (o >> 3) - self.lo
        self.table[c[:, 0], c[:, 1], c[:, 2]] = torch.arange(len(origins), device=dev)
        self.pos = (o[:, None, :] + torch.from_numpy(synth.local_offsets()).to(dev).long()[None]).reshape(-1, 3)
        self.leaf_nbr = [self.table[c[:, 0] + d[0], c[:, 1] + d[1], c[:, 2] + d[2]] for d in self._dirs()]
        self.nbr = [self.slots(*(self.pos[:, k] + d[k] for k in range(3))) for d in self._dirs()]

    @staticmethod
    def _dirs():
        return ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))

    def slots(self, i, j, k):
        c = [(v >> 3) - self.lo[q] for q, v in enumerate((i, j, k))]
        inside = torch.ones_like(i, dtype=torch.bool)
        for q in range(3):
            inside &= (c[q] >= 0) & (c[q] < self.dims[q])
            c[q] = c[q].clamp(0, self.dims[q] - 1)
        leaf = torch.where(inside, self.table[c[0], c[1], c[2]], -1)
        return torch.where(leaf >= 0, leaf * 512 + ((i & 7) << 6) + ((j & 7) << 3) + (k & 7), self.n)

    @staticmethod
    def at(f, idx):
        return torch.cat([f, f.new_zeros(1)]).index_select(0, idx)

    def cell(self, x):
        base = [torch.floor(v).long() for v in x]
        frac = [v - b for v, b in zip(x, base)]
        taps = [self.slots(*(base[k] + ((q >> (2 - k)) & 1) for k in range(3))) for q in range(8)]
        return taps, frac

    def sample(self, f, cell):
        taps, (tx, ty, tz) = cell
        out = 0.0
        for q in range(8):
            w = (tx if q & 4 else 1 - tx) * (ty if q & 2 else 1 - ty) * (tz if q & 1 else 1 - tz)
            out = out + w * self.at(f, taps[q])
        return out

    def traces(self, vel, sdt, fallback=None):
        """Back and forward cells of the MacCormack trace; fallback: the slot a missing tap reads."""
        def mapped(cell):
            return cell if fallback is None else ([torch.where(t == self.n, fallback, t) for t in cell[0]], cell[1])
        back = [self.pos[:, k].double() - vel[:, k] * sdt for k in range(3)]
        cb = mapped(self.cell(back))
        cf = mapped(self.cell([back[k] + self.sample(vel[:, k], cb) * sdt for k in range(3)]))
        return cb, cf

    def corrected(self, f, cells, nbr):
        pf, pb = self.sample(f, cells[0]), self.sample(f, cells[1])
        around = [f, pf] + [self.at(f, s) for s in nbr]
        low, high = functools.reduce(torch.minimum, around), functools.reduce(torch.maximum, around)
        return torch.maximum(low, torch.minimum(pf + 0.5 * (f - pb), high))

    def advect(self, vel, fields, dt):
        cells = self.traces(vel, dt / DX)
        v = torch.stack([self.corrected(vel[:, k], cells, self.nbr) for k in range(3)], dim=1)
        return v, [self.corrected(f, cells, self.nbr) for f in fields]

    def advect_many(self, vel, fields, dt):
        cells = self.traces(vel, dt / DX, fallback=0)
        nbr = [torch.where(s == self.n, 0, s) for s in self.nbr]
        return [self.corrected(f, cells, nbr) for f in fields]

    def divergence(self, v):
        return sum(self.at(v[:, k], self.nbr[2 * k]) - self.at(v[:, k], self.nbr[2 * k + 1]) for k in range(3)) * (0.5 / DX)

    def subtract_gradient(self, v, p, closed=False):
        def side(s):
            return torch.where(s == self.n, p, self.at(p, s)) if closed else self.at(p, s)
        return v - torch.stack([side(self.nbr[2 * k]) - side(self.nbr[2 * k + 1]) for k in range(3)], dim=1) * (0.5 / DX)

    def without_mean(self, div):
        """Removes the mean of each face-connected component of leaves."""
        label = torch.arange(len(self.leaf_nbr[0]), device=div.device)
        while True:
            new = label
            for l in self.leaf_nbr:
                new = torch.where(l >= 0, torch.minimum(new, label[l.clamp(min=0)]), new)
            new = torch.minimum(new, new[new])
            if torch.equal(new, label):
                break
            label = new
        per = label.repeat_interleave(512)
        sums = torch.zeros_like(label, dtype=torch.float64).index_add_(0, per, div)
        count = torch.zeros_like(sums).index_add_(0, per, torch.ones_like(div))
        return div - (sums / count.clamp(min=1.0))[per]

    def relax(self, div, iterations, omega, closed=False):
        b = div * DX * DX
        red = (self.pos.sum(dim=1) & 1) == 0
        sides = 6.0 if not closed else sum((s != self.n).double() for s in self.nbr)
        p = torch.zeros_like(b)
        for _ in range(iterations):
            for colour in (red, ~red):
                target = (sum(self.at(p, s) for s in self.nbr) - b) / sides
                p = torch.where(colour, p + omega * (target - p), p)
        return p

    def solve(self, div, steps=20000):
        """L p = div dx^2 by conjugate gradients to 1e-12, p = 0 outside."""
        b = -div * DX * DX
        p, r = torch.zeros_like(b), b.clone()
        d, rr = r.clone(), r.dot(r)
        stop = 1e-24 * float(rr)
        for it in range(steps):
            if it % 32 == 0 and float(rr) <= stop:
                break
            q = 6.0 * d - sum(self.at(d, s) for s in self.nbr)
            a = rr / d.dot(q)
            p.add_(a * d)
            r.sub_(a * q)
            new = r.dot(r)
            d = r + (new / rr) * d
            rr = new
        return p

    def confine(self, v, dt, scale, offset):
        def curl(side):
            h = 0.5 / DX
            d = [[self.at(v[:, c], side[2 * k]) - self.at(v[:, c], side[2 * k + 1]) for c in range(3)] for k in range(3)]
            return (d[1][2] - d[2][1]) * h, (d[2][0] - d[0][2]) * h, (d[0][1] - d[1][0]) * h
        w = curl(self.nbr)
        if offset == 0:
            return v
        grad = []
        for k in range(3):
            mags = []
            for sign in (1, -1):
                at = [self.pos[:, q] + (sign * offset if q == k else 0) for q in range(3)]
                c = curl([self.slots(*(at[q] + d[q] for q in range(3))) for d in self._dirs()])
                mags.append(torch.sqrt(c[0] ** 2 + c[1] ** 2 + c[2] ** 2))
            grad.append((mags[0] - mags[1]) * 0.5 / DX)
        n = torch.sqrt(sum(x * x for x in grad)) + 1e-5
        nx, ny, nz = (x / n for x in grad)
        force = torch.stack([ny * w[2] - nz * w[1], nz * w[0] - nx * w[2], nx * w[1] - ny * w[0]], dim=1)
        return v + scale * dt * force

    def fire(self, case, fields, sources, pressure):
        p, m = _params(case)
        f = {k: v.double() for k, v in fields.items()}
        src = {k: v.double() for k, v in sources.items()}
        dt = case["dt"] / max(1, p.substeps)
        for _ in range(max(1, p.substeps)):
            v, _ = self.advect(f["velocity"], [], dt)
            v = self.confine(v, dt, p.vorticityScale, int(p.factorScale))
            for k, s in src.items():
                if k in f:
                    f[k] = f[k] + dt * s
            v = v - torch.tensor([0.0, p.gravity * dt, 0.0], device=v.device, dtype=v.dtype)
            div = self.divergence(v)
            if case["burn"] == "oxygen":
                fuel = torch.where(f["fuel"] < 0.001, 0.0, f["fuel"])
                room = 1.0 - fuel - f["waste"]
                burn = torch.where(room < 0, 0.0, torch.minimum(room, fuel))
                f["fuel"], f["waste"] = fuel - burn, f["waste"] + 2.0 * burn
                f["temperature"] = f["temperature"] + burn * p.temperatureRelease
                f["flame"] = torch.where(room < 0, f["flame"], torch.maximum(f["flame"], (10.0 * burn).clamp(max=1.0)))
                div = div + burn * p.expansionRate
            elif case["burn"] == "rate":
                burn = torch.where((f["fuel"] > 0) & (f["temperature"] >= m.ignition_temp),
                                   f["fuel"].clamp(max=m.burn_rate * dt), 0.0)
                f["fuel"], f["temperature"] = f["fuel"] - burn, f["temperature"] + burn * m.heat_release
            t = f["temperature"]
            lift = torch.where(t > p.ambientTemp, ((t - p.ambientTemp) * p.buoyancyStrength).clamp(min=0.0), 0.0)
            lift = lift - m.density_buoyancy * f["density"]
            pushed = torch.stack([v[:, 0], v[:, 1] + lift * dt, v[:, 2]], dim=1)
            if p.disturbanceEnable > 0:
                press = pressure(self.divergence(pushed), True)
            else:
                press = pressure(div, False)
            f["velocity"] = self.subtract_gradient(pushed, press)
            names = [k for k in f if k != "velocity"]
            f.update(zip(names, self.advect_many(f["velocity"], [f[k] for k in names], dt)))
        return f


def exact(case, seed):
    kind = case["kind"]
    n = 512 * len(_leaves(case))
    if kind in ("topology", "adjoint_fire"):  # whole numbers; a derivative at rounded inputs' ties is not unique
        return None
    if n > 30e6:  # too long in 64 bits
        return None
    s = prepare(case, seed)
    s.pop("grid").close()
    x = _Exact(_leaves(case))
    if kind in ("operators", "step"):
        closed = case.get("walls") == "closed"
        v, out = x.advect(s["vel"].double(), [t.double() for t in s["scalars"]], case["dt"])
        div = x.divergence(v)
        if closed:
            div = x.without_mean(div)
        p = x.solve(div) if case.get("tolerance") else x.relax(div, case["iterations"], case["omega"], closed)
        return [x.subtract_gradient(v, p, closed), *out]
    if kind in ("mixed", "mixed_host"):
        fields = [t.cuda().double() for t in (s["pinned"] if kind == "mixed_host" else [s["vel"], *s["scalars"]])]
        v, out = x.advect(fields[0], fields[1:], case["dt"])
        return [x.subtract_gradient(v, x.solve(x.divergence(v))), *out]
    if kind == "advance":
        omega = 2.0 / (1.0 + math.sin(3.14159 * DX))
        its = case["iterations"]
        return x.fire(case, s["fields"], s["sources"],
                      lambda div, again: x.relax(div, max(2, its // 2) if again else its, omega))
    if kind == "fire":
        return x.fire(case, s["fields"], s["sources"], lambda div, again: x.solve(div))
    # adjoint_step: the transpose of the step's derivative, by differentiating the 64-bit step.
    inputs = [s["vel"].double().requires_grad_()] + [t.double().requires_grad_() for t in s["scalars"]]
    v, out = x.advect(inputs[0], inputs[1:], case["dt"])
    outs = [x.subtract_gradient(v, x.relax(x.divergence(v), case["iterations"], case["omega"])), *out]
    return list(torch.autograd.grad(outs, inputs, [s["vel_bar"].double()] + [t.double() for t in s["scalars_bar"]]))
