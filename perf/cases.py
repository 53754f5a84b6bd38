"""The work this framework is used for, as cases that can be timed and checked one by one.

Every case goes through the package's public interface the way a program using it does:

* ``box``      a periodic D3Q19 box (the Taylor-Green benchmark, HIT runs): ``set_level_box``,
               ``set_equilibrium_dense``, steps, ``get_macros_dense``;
* ``channel``  a D3Q19 channel between bounce-back walls (one moving), driven by a body force;
* ``cavity``   the D2Q9 lid-driven cavity on a Morton node list, populations read back to the host;
* ``exchange`` the drop-in use from a host program: FP64 populations up, steps, populations and
               fields down through pinned host memory;
* ``flow``     the packaged multi-level flows (cylinder, cube) with immersed boundaries;
* ``learned``  LES with the learned closure evaluated inside the collision;
* ``fine``     the closure's training data: a fine run and its box filter;
* ``train``    optimiser steps of the closure network.

A pass continues the run its state holds by ``steps`` time steps, so a state can be run any number of
times.  Inputs come from the seed alone.  ``exact`` restates the single-level cases in FP64 torch.
"""
import ctypes
import math

import numpy as np
import torch

import zllbm_b200 as zl
from zllbm_b200 import cube_flow, cylinder_flow
from zllbm_b200.hit import hit_velocity, initial_net

ELEM = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # the 256^2 lid-driven cavity (Re 100) in the parity storage: the smallest grid in use, where a
        # step is a few microseconds and launches count
        {"name": "cavity_256_f64", "kind": "cavity", "nx": 257, "ny": 257, "collision": "srt", "steps": 100},
        # the 64^3 Taylor-Green vortex in the parity storage: it fits the caches
        {"name": "tgv_64_f64", "kind": "box", "nx": 64, "ny": 64, "nz": 64, "collision": "mrt", "storage": "f64",
         "rounding": "nearest", "les": False, "block": "default", "graph": True, "steps": 100},
        # the benchmark's own workload, two nodes per thread (what its autotuner picks)
        {"name": "tgv_256_f32", "kind": "box", "nx": 256, "ny": 256, "nz": 256, "collision": "mrt", "storage": "f32",
         "rounding": "nearest", "les": False, "block": "pair", "graph": True, "steps": 20},
        # the same with half the memory: FP16, stochastic rounding, one warp per row
        {"name": "tgv_256_f16", "kind": "box", "nx": 256, "ny": 256, "nz": 256, "collision": "mrt", "storage": "f16",
         "rounding": "stochastic", "les": False, "block": "row", "graph": True, "steps": 20},
        # wall-bounded, forced, odd extents
        {"name": "channel_161x97x81_f32", "kind": "channel", "nx": 161, "ny": 97, "nz": 81, "collision": "srt",
         "storage": "f32", "les": False, "graph": True, "steps": 40},
        # a host program's exchange in both directions around a short run
        {"name": "exchange_128_f64", "kind": "exchange", "nx": 128, "ny": 128, "nz": 128, "collision": "mrt",
         "steps": 20},
        # coarse LES runs on decaying HIT: Smagorinsky, stepped call by call as the HIT driver does
        {"name": "hit_les_256", "kind": "box", "nx": 256, "ny": 256, "nz": 256, "collision": "srt", "storage": "f32",
         "rounding": "nearest", "les": True, "block": "default", "graph": False, "steps": 20},
        # the same with the network evaluated in every step
        {"name": "hit_learned_128", "kind": "learned", "n": 128, "collision": "srt", "storage": "f32", "every": 1,
         "steps": 20},
        # fine HIT run and the filter that makes the coarse reference and the training data
        {"name": "hit_fine_256", "kind": "fine", "n": 256, "factor": 4, "steps": 16},
        # eight optimiser steps on the HIT driver's batch
        {"name": "train_37888", "kind": "train", "batch": 37888, "steps": 8},
        # flow past a cube: three levels, Smagorinsky, 24,578 immersed-boundary vertices
        {"name": "cube_flow_f32", "kind": "flow", "body": "cube", "storage": "f32", "steps": 64},
        # flow past a cylinder: four levels of which three hold about 5,000 nodes each
        {"name": "cylinder_flow_f32", "kind": "flow", "body": "cylinder", "storage": "f32", "steps": 128},
    ]


def _size(rng, lo, hi, even=False):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n + (n & 1) if even else n


def draw(rng):
    """A case of the listed kinds, with sizes over the whole range (odd ones among them)."""
    kind = rng.choices(("box", "channel", "cavity", "exchange", "flow", "learned", "fine", "train"),
                       weights=(6, 3, 2, 1, 2, 2, 1, 1))[0]
    coll = rng.choice(("srt", "mrt"))
    if kind == "box":
        storage = rng.choice(("f64", "f32", "f32", "f16", "bf16"))
        block = "default" if storage == "f64" else rng.choice(("default", "pair", "row" if ELEM[storage] == 2 else "pair"))
        les = rng.random() < 0.3
        if les:  # (MRT with Smagorinsky is a reduced-precision combination)
            block, coll = "default", "srt" if storage == "f64" else coll
        nx = rng.choice((128, 256)) if block == "row" else _size(rng, 24, 256, even=block == "pair")
        return {"kind": kind, "nx": nx, "ny": _size(rng, 24, 200), "nz": _size(rng, 24, 200), "collision": coll,
                "storage": storage, "rounding": rng.choice(("nearest", "stochastic")) if ELEM[storage] == 2 else "nearest",
                "les": les, "block": block, "graph": rng.random() < 0.5, "steps": 2 * rng.randint(4, 10)}
    if kind == "channel":
        storage, les = rng.choice(("f64", "f32", "f32")), rng.random() < 0.4
        return {"kind": kind, "nx": _size(rng, 24, 256), "ny": _size(rng, 20, 128), "nz": _size(rng, 20, 160),
                "collision": "srt" if les and storage == "f64" else coll, "storage": storage, "les": les,
                "graph": rng.random() < 0.5, "steps": 2 * rng.randint(5, 20)}
    if kind == "cavity":
        return {"kind": kind, "nx": _size(rng, 33, 1100), "ny": _size(rng, 33, 1100), "collision": coll,
                "steps": 2 * rng.randint(10, 50)}
    if kind == "exchange":
        return {"kind": kind, "nx": _size(rng, 24, 128), "ny": _size(rng, 24, 128), "nz": _size(rng, 24, 128),
                "collision": coll, "steps": 2 * rng.randint(2, 10)}
    if kind == "flow":
        body = rng.choice(("cube", "cylinder"))
        return {"kind": kind, "body": body, "storage": rng.choice(("f32", "f64")),
                "steps": rng.randint(4, 24) if body == "cube" else rng.randint(8, 127)}
    if kind == "learned":
        return {"kind": kind, "n": _size(rng, 32, 160), "collision": coll, "storage": "f32",
                "every": rng.choice((1, 8, 16)), "steps": 2 * rng.randint(4, 10)}
    if kind == "fine":
        factor = rng.choice((2, 4))
        return {"kind": kind, "n": factor * _size(rng, 16, 63), "factor": factor, "steps": 2 * rng.randint(2, 8)}
    return {"kind": "train", "batch": _size(rng, 1000, 150000), "steps": rng.randint(2, 12)}


# ---------------------------------------------------------------- inputs
NU_LES = 0.0005          # lattice viscosity of the LES runs (tau 0.5015)
U0, NU_TGV = 0.05, (0.55 - 0.5) / 3.0
FORCE, U_WALL, NU_CHANNEL = 2e-6, 0.02, 0.02
U_LID = 0.1
STORAGE = zl.STORAGE_NAMES
COLLISION = {"srt": zl.SRT, "mrt": zl.MRT}


def _tgv_fields(nx, ny, nz, seed):
    """Density [nz, ny, nx] and velocity [nz, ny, nx, 3] (FP32) of a Taylor-Green vortex with seeded
    phases and a second, weaker seeded mode."""
    g = np.random.default_rng(seed)
    ph = g.uniform(0.0, 2.0 * math.pi, 6)
    dev = "cuda"
    ax = [2.0 * math.pi * torch.arange(n, device=dev, dtype=torch.float64) / n for n in (nx, ny, nz)]
    x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    a, b, c = x + ph[0], y + ph[1], z + ph[2]
    u = torch.stack([(U0 * torch.sin(a) * torch.cos(b) * torch.cos(c) + 0.1 * U0 * torch.sin(2 * z + ph[3])).expand(nz, ny, nx),
                     (-U0 * torch.cos(a) * torch.sin(b) * torch.cos(c) + 0.1 * U0 * torch.sin(2 * x + ph[4])).expand(nz, ny, nx),
                     (0.1 * U0 * torch.sin(2 * y + ph[5])).expand(nz, ny, nx)], dim=-1)
    p = U0 * U0 / 16.0 * (torch.cos(2 * a) + torch.cos(2 * b)) * (torch.cos(2 * c) + 2.0)
    return (1.0 + 3.0 * p).float().contiguous(), u.float().contiguous()


def _channel_fields(nx, ny, nz, seed):
    """A wall-to-wall profile with seeded streamwise-periodic disturbances."""
    g = np.random.default_rng(seed)
    ph = g.uniform(0.0, 2.0 * math.pi, 3)
    dev = "cuda"
    x = (2.0 * math.pi * torch.arange(nx, device=dev, dtype=torch.float64) / nx)[None, None, :]
    z = (2.0 * math.pi * torch.arange(nz, device=dev, dtype=torch.float64) / nz)[:, None, None]
    s = ((torch.arange(ny, device=dev, dtype=torch.float64) + 0.5) / ny)[None, :, None]
    env = s * (1.0 - s)
    u = torch.stack([(U_WALL * s + 0.16 * env + 0.02 * env * torch.sin(z + ph[0])).expand(nz, ny, nx),
                     (0.02 * env * torch.sin(x + ph[1]) * torch.cos(z)).expand(nz, ny, nx),
                     (0.02 * env * torch.sin(2 * x + ph[2])).expand(nz, ny, nx)], dim=-1)
    return torch.ones(nz, ny, nx, device=dev), u.float().contiguous()


def _hit_fields(n, seed):
    return torch.ones(n, n, n, device="cuda"), hit_velocity(n, seed=seed).reshape(n, n, n, 3)


def _net(seed):
    """A closure network whose inputs are normalised by the features' usual magnitudes."""
    typical = [1.0, 3e-4, 1e-4, 1.0, 1e-4, 1.0, 1e-4, 1.0, 1e-4] + [3e-3, 1e-4] * 2 + [1e-3] * 3 + [1e-4] * 3 + \
              [1e-4, 2e-5, 5e-8, 5e-3, 2e-3]
    return initial_net(seed, None, 1.0 / np.array(typical))


def _train_data(batch, steps, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(steps, batch, zl.MLP_IN, device="cuda", generator=g)
    y = (1.0 + 0.5 * torch.tanh(x[..., 9] * x[..., 11]) + 0.3 * x[..., 22]).clamp(0.0, 8.0).contiguous()
    return x, y


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _dp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _exchange_populations(case, seed):
    """FP64 populations [n, 19] of the stored nodes (the duplicated maximum planes included), x fastest."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rho, u = _tgv_fields(nx, ny, nz, seed)
    f = Lattice(3).feq(rho.double(), u.double().movedim(-1, 0))
    idx = [torch.arange(n + 1, device=f.device) % n for n in (nz, ny, nx)]
    f = f[:, idx[0]][:, :, idx[1]][:, :, :, idx[2]]
    return f.reshape(19, -1).T.contiguous()


def _cavity_populations(case, seed):
    g = np.random.default_rng(seed)
    x = np.arange(case["nx"])[None, :] / (case["nx"] - 1)
    y = np.arange(case["ny"])[:, None] / (case["ny"] - 1)
    psi = np.sin(np.pi * x) ** 2 * np.sin(np.pi * y) ** 2
    k, amp = g.uniform(1.0, 2.0), 0.03 + 0.02 * g.random()
    ux = amp * np.sin(np.pi * x) ** 2 * np.sin(2 * np.pi * y * k) * psi
    uy = -amp * np.sin(2 * np.pi * x * k) * np.sin(np.pi * y) ** 2 * psi
    u = torch.from_numpy(np.stack([ux, uy])).reshape(2, 1, case["ny"], case["nx"])
    f = Lattice(2).feq(torch.ones(1, case["ny"], case["nx"], dtype=torch.float64), u)
    return f.reshape(9, -1).T.contiguous()


# ---------------------------------------------------------------- what a program holds before the call
class State:
    """A run: its context and the buffers it reads into."""

    def __init__(self, case):
        self.case = case
        self.ctx = None

    def __del__(self):
        if self.ctx is not None:
            self.ctx.close()


def _box(case, cfg, extent, fields):
    """A full-box level started from dense fields."""
    rho, u = fields
    st = State(case)
    st.ctx = zl.Context(cfg)
    st.ctx.set_level_box(0, (0, 0, 0), extent)
    torch.cuda.synchronize()
    st.ctx.set_equilibrium_dense(0, rho.data_ptr(), u.data_ptr())
    st.rho, st.u = torch.empty_like(rho), torch.empty_like(u)
    return st


def prepare(case, seed):
    st = _prepare(case, seed)
    torch.cuda.synchronize()
    return st


def _prepare(case, seed):
    kind = case["kind"]
    periodic = (zl.BC_PERIODIC,) * 6
    if kind == "box":
        n = (case["nx"], case["ny"], case["nz"])
        les = zl.LES_SMAGORINSKY if case["les"] else zl.LES_OFF
        fields = _hit_fields(n[0], seed) if case["les"] and n[0] == n[1] == n[2] else _tgv_fields(*n, seed)
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=COLLISION[case["collision"]], storage=STORAGE[case["storage"]],
                              viscosity=NU_LES if case["les"] else NU_TGV, bc_kind=periodic, domain_min=(0, 0, 0),
                              domain_max=n, les=les, les_cs=0.1,
                              storage_rounding=zl.ROUND_NEAREST if case["rounding"] == "nearest" else zl.ROUND_STOCHASTIC)
        st = _box(case, cfg, n, fields)
        if case["block"] == "pair":
            st.ctx.set_block(0, -128 if n[0] > 128 else -64, 1)
        elif case["block"] == "row":
            st.ctx.set_block(0, zl.BLOCK_ROW, 2)
        st.ctx.set_graph(case["graph"])
    elif kind == "channel":
        n = (case["nx"], case["ny"], case["nz"])
        wall = zl.BC_BOUNCE_BACK
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=COLLISION[case["collision"]], storage=STORAGE[case["storage"]],
                              viscosity=NU_CHANNEL, bc_kind=periodic[:2] + (wall, wall) + periodic[:2],
                              bc_velocity=((0.0,) * 3,) * 3 + ((U_WALL, 0.0, 0.0),) + ((0.0,) * 3,) * 2,
                              domain_min=(0, 0, 0), domain_max=(n[0], n[1] - 1, n[2]), forcing=1,
                              constant_force=(FORCE, 0.0, 0.0), les=zl.LES_SMAGORINSKY if case["les"] else zl.LES_OFF,
                              les_cs=0.1)
        st = _box(case, cfg, n, _channel_fields(*n, seed))
        st.ctx.set_graph(case["graph"])
    elif kind == "learned":
        n = (case["n"],) * 3
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=COLLISION[case["collision"]], storage=STORAGE[case["storage"]],
                              viscosity=NU_LES, bc_kind=periodic, domain_min=(0, 0, 0), domain_max=n,
                              les=zl.LES_LEARNED, les_cs=0.1)
        st = _box(case, cfg, n, _hit_fields(case["n"], seed))
        st.ctx.set_closure(_net(seed))
        st.ctx.set_closure_interval(case["every"])
    elif kind == "fine":
        n = (case["n"],) * 3
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=zl.SRT, storage=zl.STORAGE_F32, viscosity=0.002,
                              bc_kind=periodic, domain_min=(0, 0, 0), domain_max=n)
        st = _box(case, cfg, n, _hit_fields(case["n"], seed))
        del st.rho, st.u
        st.filtered = torch.empty((case["n"] // case["factor"]) ** 3, 29, device="cuda")
    elif kind == "train":
        st = State(case)
        st.x, st.y = _train_data(case["batch"], case["steps"], seed)
        st.trainer = zl.Trainer(initial_net(seed))
        st.trainer.set_stream(torch.cuda.current_stream().cuda_stream or None)
    elif kind == "cavity":
        nx, ny = case["nx"], case["ny"]
        wall = zl.BC_BOUNCE_BACK
        cfg = zl.SolverConfig(lattice=zl.D2Q9, collision=COLLISION[case["collision"]], storage=zl.STORAGE_F64,
                              viscosity=U_LID * nx / 100.0, bc_kind=(wall,) * 4 + (0, 0),
                              bc_velocity=((0.0,) * 3,) * 3 + ((U_LID, 0.0, 0.0),) + ((0.0,) * 3,) * 2,
                              domain_min=(1, 1, 0), domain_max=(nx, ny, 0))
        st = State(case)
        st.ctx = zl.Context(cfg)
        st.ctx.set_level_nodes(0, zl.box_codes(2, (1, 1), (nx, ny)))
        st.ctx.set_populations(0, None, _cavity_populations(case, seed).numpy())
        st.ctx.set_graph(True)
        st.f = _pinned(nx * ny, 9)
    elif kind == "exchange":
        n = (case["nx"], case["ny"], case["nz"])
        cfg = zl.SolverConfig(lattice=zl.D3Q19, collision=COLLISION[case["collision"]], storage=zl.STORAGE_F64,
                              viscosity=NU_TGV, bc_kind=periodic, domain_min=(1, 1, 1),
                              domain_max=tuple(v + 1 for v in n))
        st = State(case)
        st.ctx = zl.Context(cfg)
        st.ctx.set_level_nodes(0, zl.box_codes(3, (1, 1, 1), tuple(v + 1 for v in n)))
        f = _exchange_populations(case, seed)
        st.f0, st.f = _pinned(*f.shape), _pinned(*f.shape)
        st.f0.copy_(f)
        st.rho, st.u = _pinned(f.shape[0]), _pinned(f.shape[0], 3)
        st.ctx.set_graph(True)
    else:
        st = _prepare_flow(case, seed)
    return st



def _prepare_flow(case, seed):
    """A packaged flow whose body's surface moves: the cylinder spins, the cube's surface blows and sucks
    weakly (both seeded)."""
    mod = cube_flow if case["body"] == "cube" else cylinder_flow
    st = State(case)
    built = mod.build(mod.DEFAULT_TOPOLOGY, STORAGE[case["storage"]])
    st.ctx, meta, st.nodes = built[:3]
    st.levels = meta["levels"]
    g = np.random.default_rng(seed)
    amp, ph = g.uniform(0.1, 0.3), g.uniform(0.0, 2.0 * math.pi)
    if case["body"] == "cube":
        cx, cy, cz, edge = (float(v) for v in meta["cube"].split(","))
        xyz, area = cube_flow.cube_vertices((cx, cy, cz), edge, 1.0 / (1 << st.levels))
        vel = np.zeros_like(xyz)
        vel[:, 1] = amp * cube_flow.U_IN * np.sin(2.0 * math.pi * (xyz[:, 0] - cx) / edge + ph)
    else:
        cx, cy, r = (float(v) for v in meta["circle"].split(","))
        t = 2.0 * math.pi * np.arange(cylinder_flow.VERTICES) / cylinder_flow.VERTICES
        xyz = np.stack([cx + r * np.cos(t), cy + r * np.sin(t), np.zeros(t.size)], axis=1)
        area = np.full(t.size, 2.0 * math.pi * r / t.size)
        spin = amp * cylinder_flow.U_IN * math.cos(ph)
        vel = np.stack([-spin * np.sin(t), spin * np.cos(t), np.zeros(t.size)], axis=1)
    st.ctx.ib_set_vertices(st.levels, xyz, vel, area)
    st.ctx.set_graph(True)
    dims = st.ctx.config.dims
    st.rho = [_pinned(n) for n in st.nodes]
    st.u = [_pinned(n, dims) for n in st.nodes]
    return st


# ---------------------------------------------------------------- one pass
def run(state):
    case, ctx = state.case, state.ctx
    kind = case["kind"]
    if kind in ("box", "channel") and case["graph"]:
        ctx.advance(case["steps"])
    elif kind in ("box", "channel", "learned", "fine"):
        for _ in range(case["steps"]):
            ctx.step_level(0)
    if kind in ("box", "channel", "learned"):
        ctx.get_macros_dense(0, state.rho.data_ptr(), state.u.data_ptr())
        return {"rho": state.rho, "u": state.u}
    if kind == "fine":
        ctx.filter_level(0, case["factor"], state.filtered.data_ptr())
        return {"filtered": state.filtered}
    if kind == "train":
        for k in range(case["steps"]):
            state.trainer.step(state.x[k].data_ptr(), state.y[k].data_ptr(), case["batch"], 1e-3)
        return {"gradients": state.trainer.gradients().flat()[:zl.MLP_TRAINABLE],
                "weights": state.trainer.weights().flat()[:zl.MLP_TRAINABLE]}
    if kind == "cavity":
        ctx.advance(case["steps"])
        ctx._check(ctx.lib.zl_get_populations(ctx.handle, 0, None, _dp(state.f), state.f.shape[0]))
        return {"f": state.f}
    if kind == "exchange":
        n = state.f.shape[0]
        ctx._check(ctx.lib.zl_set_populations(ctx.handle, 0, None, _dp(state.f0), n))
        ctx.advance(case["steps"])
        ctx._check(ctx.lib.zl_get_populations(ctx.handle, 0, None, _dp(state.f), n))
        ctx._check(ctx.lib.zl_get_macros(ctx.handle, 0, None, _dp(state.rho), _dp(state.u), n))
        return {"f": state.f, "rho": state.rho, "u": state.u}
    # flow: the vertex forces and every level's fields, FP32 runs kept in FP32 on the device for analysis
    ctx.advance(case["steps"])
    out = {}
    for lv, n in enumerate(state.nodes):
        ctx._check(ctx.lib.zl_get_macros(ctx.handle, lv, None, _dp(state.rho[lv]), _dp(state.u[lv]), n))
        out[f"rho{lv}"], out[f"u{lv}"] = state.rho[lv], state.u[lv]
    out["forces"], out["total"] = ctx.ib_get_forces(state.levels)
    if case["storage"] == "f32":
        for k, v in out.items():
            out[k] = v.to("cuda", non_blocking=True).float() if isinstance(v, torch.Tensor) else v.astype(np.float32)
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes and operations of one pass.  A time step reads and writes every population of every node
    once (a level's populations are the state between steps); outputs are written once."""
    kind = case["kind"]
    if kind in ("box", "channel", "exchange", "learned", "fine"):
        n = case["n"] ** 3 if "n" in case else case["nx"] * case["ny"] * case["nz"]
        elem = ELEM[case.get("storage", "f64" if kind == "exchange" else "f32")]
        flops = 2 * 19 * 19 + 150 if elem == 8 and case["collision"] == "mrt" else 250
        moved, done = n * 2 * 19 * elem * case["steps"], n * flops * case["steps"]
        if kind == "learned":
            done += n * 2 * (24 * 64 + 64 * 64 + 64) * -(-case["steps"] // case["every"])
        if kind == "exchange":
            moved += n * 8 * (19 + 19 + 4)
        elif kind == "fine":
            moved += n * 19 * elem + (case["n"] // case["factor"]) ** 3 * 29 * 4
        else:
            moved += n * (19 * elem + 16)
        return {"bytes": moved, "flops": done}
    if kind == "cavity":
        n = case["nx"] * case["ny"]
        return {"bytes": n * 2 * 9 * 8 * case["steps"] + n * 9 * 8, "flops": n * 120 * case["steps"]}
    if kind == "train":
        n = case["batch"] * case["steps"]
        return {"bytes": n * 25 * 4, "flops": n * 3 * 2 * (24 * 64 + 64 * 64 + 64)}
    # node updates of a coarse step, sum of nodes x 2^level, of the packaged grids
    lups = 7929639 if case["body"] == "cube" else 592829
    nodes = 5334255 if case["body"] == "cube" else 538789
    q, dims = (19, 3) if case["body"] == "cube" else (9, 2)
    elem = ELEM[case["storage"]]
    return {"bytes": lups * 2 * q * elem * case["steps"] + nodes * (q * elem + 8 * (dims + 1)),
            "flops": lups * 13 * q * case["steps"]}


# ---------------------------------------------------------------- the same in FP64 torch
class Lattice:
    """D2Q9 / D3Q19 with SRT or MRT collision, Smagorinsky and a body force, on f[q, z, y, x] in FP64."""

    def __init__(self, dims):
        self.dims = dims
        if dims == 3:
            self.c = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0),
                      (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1),
                      (0, -1, 1), (0, 1, -1), (0, -1, -1)]
            self.w = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
            rates = [0, 1.5, 1.4, 0, 1.2, 0, 1.2, 0, 1.2, -1, 1.4, -1, 1.4, -1, -1, -1, 1.98, 1.98, 1.98]
        else:
            self.c = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0),
                      (1, -1, 0)]
            self.w = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
            rates = [0, 1.4, 1.4, 0, 1.2, 0, 1.2, -1, -1]
        self.rates = torch.tensor(rates, dtype=torch.float64)
        self.opp = [self.c.index(tuple(-v for v in c)) for c in self.c]
        x, y, z = (torch.tensor([c[a] for c in self.c], dtype=torch.float64) for a in range(3))
        r = x * x + y * y + z * z
        if dims == 3:
            xx, yz = 3 * x * x - r, y * y - z * z
            rows = [x * 0 + 1, 19 * r - 30, (21 * r * r - 53 * r + 24) / 2, x, (5 * r - 9) * x, y, (5 * r - 9) * y, z,
                    (5 * r - 9) * z, xx, (3 * r - 5) * xx, yz, (3 * r - 5) * yz, x * y, y * z, x * z, yz * x,
                    (z * z - x * x) * y, (x * x - y * y) * z]
        else:
            rows = [x * 0 + 1, 3 * r - 4, (9 * r * r - 21 * r + 8) / 2, x, (3 * r - 5) * x, y, (3 * r - 5) * y,
                    x * x - y * y, x * y]
        self.m = torch.stack(rows)
        self.minv = self.m.T / (self.m * self.m).sum(dim=1)

    def dot(self, q, v):
        s = 0.0
        for a in range(self.dims):
            if self.c[q][a]:
                s = s + self.c[q][a] * v[a]
        return s

    def feq(self, rho, u):
        uu = (u * u).sum(dim=0)
        out = torch.empty((len(self.c),) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
        for q, w in enumerate(self.w):
            cu = self.dot(q, u)
            out[q] = w * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * uu)
        return out

    def macros(self, f):
        rho = f.sum(dim=0)
        j = torch.zeros((self.dims,) + tuple(rho.shape), dtype=torch.float64, device=f.device)
        for q, c in enumerate(self.c):
            for a in range(self.dims):
                if c[a]:
                    j[a] += c[a] * f[q]
        return rho, j

    def stress(self, neq):
        pairs = [(a, b) for a in range(self.dims) for b in range(a, self.dims)]
        out = {}
        for a, b in pairs:
            out[a, b] = sum(c[a] * c[b] * neq[q] for q, c in enumerate(self.c) if c[a] * c[b])
        return out

    def collide(self, f, tau, mrt, les_c=None, force=None, closure=None):
        """les_c: the constant 18 Cs^2; closure(rho, neq, stress): the same per node."""
        rho, u = self.macros(f)
        if force is not None:
            for a in range(self.dims):
                u[a] += 0.5 * force[a]
        u /= rho
        neq = f - self.feq(rho, u)
        t = tau
        if les_c is not None or closure is not None:
            pi = self.stress(neq)
            if closure is not None:
                les_c = closure(rho, neq, pi)
            if force is not None:
                for (a, b), v in pi.items():
                    pi[a, b] = v + (force[a] * u[a] if a == b else 0.5 * (force[a] * u[a] + force[b] * u[b]))
            pp = sum((1.0 if a == b else 2.0) * v * v for (a, b), v in pi.items())
            t = tau + 0.5 * (torch.sqrt(tau * tau + les_c * torch.sqrt(2.0 * pp)) - tau)
        term = None
        if force is not None:
            uf = sum(u[a] * force[a] for a in range(self.dims))
            term = torch.stack([self.w[q] * (3.0 * (self.dot(q, force) - uf) + 9.0 * self.dot(q, u) * self.dot(q, force))
                                for q in range(len(self.c))])
        if not mrt:
            out = f - neq / t
            return out if term is None else out + (1.0 - 0.5 / t) * term
        m, minv, rates = (v.to(f.device) for v in (self.m, self.minv, self.rates))

        def relax(x, of_rate):
            mom = torch.tensordot(m, x, dims=1)
            for k, s in enumerate(rates.tolist()):
                mom[k] *= of_rate(1.0 / t if s < 0 else s)
            return torch.tensordot(minv, mom, dims=1)

        out = f - relax(neq, lambda s: s)
        return out if term is None else out + relax(term, lambda s: 1.0 - 0.5 * s)

    def stream(self, post):
        out = torch.empty_like(post)
        for q, c in enumerate(self.c):
            out[q] = torch.roll(post[q], shifts=(c[2], c[1], c[0]), dims=(0, 1, 2))
        return out


def _walls(lat, f, post, faces):
    """Bounce back on faces [(axis, side, velocity)], in that order; in 2D an x wall reflects the diagonals
    specularly."""
    for axis, side, vel in faces:
        inward = 1 if side == 0 else -1
        at = [slice(None)] * 3
        at[2 - axis] = 0 if side == 0 else -1
        for q, c in enumerate(lat.c):
            if c[axis] != inward:
                continue
            o = lat.c.index((-c[0], c[1], 0)) if lat.dims == 2 and axis == 0 else lat.opp[q]
            f[(q, *at)] = post[(o, *at)] - 6.0 * lat.w[o] * lat.dot(o, vel)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _closure(lat, net, tau0):
    """The learned constant 18 c per node from the closure network."""
    v = torch.from_numpy(net.flat()).double().to(_device())
    w1, b1, w2, b2, w3, b3, mean, inv = torch.split(v, [64 * 24, 64, 64 * 64, 64, 64, 1, 24, 24])
    w1, w2 = w1.reshape(64, 24), w2.reshape(64, 64)
    m = lat.m.to(v.device)

    def constant(rho, neq, pi):
        x = torch.zeros((24,) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
        x[:19] = torch.tensordot(m, neq, dims=1) / rho
        x[[0, 3, 5, 7]] = 0.0
        s = {k: -1.5 * p / (rho * tau0) for k, p in pi.items()}
        norm = lambda t: sum((1.0 if a == b else 2.0) * p * p for (a, b), p in t.items())
        x[19] = s[0, 0] + s[1, 1] + s[2, 2]
        x[20] = norm(s)
        d = {k: p - (x[19] / 3.0 if k[0] == k[1] else 0.0) for k, p in s.items()}
        x[21] = 3.0 * (d[0, 0] * (d[1, 1] * d[2, 2] - d[1, 2] ** 2) - d[0, 1] * (d[0, 1] * d[2, 2] - d[1, 2] * d[0, 2])
                       + d[0, 2] * (d[0, 1] * d[1, 2] - d[1, 1] * d[0, 2]))
        x[22] = torch.sqrt(2.0 * norm(d))
        x[23] = 0.5 * (torch.sqrt(tau0 * tau0 + 0.18 * torch.sqrt(2.0 * norm(pi))) - tau0)
        x = x.reshape(24, -1)
        y = torch.empty(x.shape[1], dtype=torch.float64, device=x.device)
        for i in range(0, x.shape[1], 1 << 20):
            h = (x[:, i:i + (1 << 20)].T - mean) * inv
            h = torch.nn.functional.gelu(h @ w1.T + b1, approximate="tanh")
            h = torch.nn.functional.gelu(h @ w2.T + b2, approximate="tanh")
            y[i:i + (1 << 20)] = h @ w3 + b3
        return 0.18 * y.clamp(0.0, 8.0).reshape(rho.shape)

    return constant


def _exact_train(case, seed):
    x, y = _train_data(case["batch"], case["steps"], seed)
    flat = torch.from_numpy(initial_net(seed).flat()).double().to(x.device)
    w = flat[:zl.MLP_TRAINABLE].clone().requires_grad_(True)
    m, v, grad = torch.zeros_like(w), torch.zeros_like(w), None
    for k in range(case["steps"]):
        w1, b1, w2, b2, w3, b3 = torch.split(w, [64 * 24, 64, 64 * 64, 64, 64, 1])
        h = torch.nn.functional.gelu(x[k].double() @ w1.reshape(64, 24).T + b1, approximate="tanh")
        h = torch.nn.functional.gelu(h @ w2.reshape(64, 64).T + b2, approximate="tanh")
        loss = ((h @ w3 + b3 - y[k].double()) ** 2).mean()
        grad, = torch.autograd.grad(loss, w)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad * grad
            w = w - 1e-3 * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
        w = w.detach().requires_grad_(True)
    return {"gradients": grad, "weights": w.detach()}


def exact(case, seed):
    """What ``run`` returns for a new state, in FP64.  The multi-level flows have none: a restatement of
    the grids' transfers and immersed boundaries would be a solver of its own."""
    kind = case["kind"]
    if kind == "flow":
        return None
    if kind == "train":
        return _exact_train(case, seed)
    mrt = case.get("collision") == "mrt"
    if kind == "cavity":
        lat = Lattice(2)
        nx, ny = case["nx"], case["ny"]
        f = _cavity_populations(case, seed).to(_device()).T.reshape(9, 1, ny, nx).contiguous()
        tau = 3.0 * U_LID * nx / 100.0 + 0.5
        rest = (0.0, 0.0, 0.0)
        for _ in range(case["steps"]):
            post = lat.collide(f, tau, mrt)
            f = lat.stream(post)
            _walls(lat, f, post, [(0, 0, rest), (1, 0, rest), (0, 1, rest), (1, 1, (U_LID, 0.0, 0.0))])
        return {"f": f.reshape(9, -1).T.contiguous()}
    lat = Lattice(3)
    if kind == "exchange":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        f = _exchange_populations(case, seed).T.reshape(19, nz + 1, ny + 1, nx + 1)[:, :nz, :ny, :nx].contiguous()
        for _ in range(case["steps"]):
            f = lat.stream(lat.collide(f, 3.0 * NU_TGV + 0.5, mrt))
        idx = [torch.arange(n + 1, device=f.device) % n for n in (nz, ny, nx)]
        f = f[:, idx[0]][:, :, idx[1]][:, :, :, idx[2]]
        rho, j = lat.macros(f)
        return {"f": f.reshape(19, -1).T.contiguous(), "rho": rho.reshape(-1),
                "u": (j / rho).reshape(3, -1).T.contiguous()}
    if kind == "box":
        n = (case["nx"], case["ny"], case["nz"])
        rho, u = _hit_fields(n[0], seed) if case["les"] and n[0] == n[1] == n[2] else _tgv_fields(*n, seed)
        nu = NU_LES if case["les"] else NU_TGV
    elif kind == "channel":
        rho, u = _channel_fields(case["nx"], case["ny"], case["nz"], seed)
        nu = NU_CHANNEL
    else:
        rho, u = _hit_fields(case["n"], seed)
        nu = NU_LES if kind == "learned" else 0.002
    f = lat.feq(rho.double(), u.double().movedim(-1, 0))
    tau = 3.0 * nu + 0.5
    les_c = 18.0 * 0.1 ** 2 if case.get("les") else None
    force = (FORCE, 0.0, 0.0) if kind == "channel" else None
    closure = _closure(lat, _net(seed), tau) if kind == "learned" else None
    kept = None

    def constant(rho, neq, pi):
        nonlocal kept
        if step % case["every"] == 0:
            kept = closure(rho, neq, pi)
        return kept

    for step in range(case["steps"]):
        post = lat.collide(f, tau, mrt, les_c, force, constant if closure else None)
        f = lat.stream(post)
        if kind == "channel":
            rest = (0.0, 0.0, 0.0)
            _walls(lat, f, post, [(1, 0, rest), (1, 1, (U_WALL, 0.0, 0.0))])
        del post
    rho, j = lat.macros(f)
    u = j / rho
    if kind == "fine":
        k, fac = case["n"] // case["factor"], case["factor"]
        neq = f - lat.feq(rho, u)
        cols = [rho, u[0], u[1], u[2], u[0] ** 2, u[1] ** 2, u[2] ** 2, u[0] * u[1], u[0] * u[2], u[1] * u[2]]
        cols += [neq[q] for q in range(19)]
        return {"filtered": torch.stack([v.reshape(k, fac, k, fac, k, fac).mean(dim=(1, 3, 5)).reshape(-1) for v in cols],
                                        dim=1)}
    return {"rho": rho, "u": u.movedim(0, -1).contiguous()}
