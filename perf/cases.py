"""What a user of the particle-to-surface pipeline has it do, as measurable cases.

A case names a scene (which particles), an operation (which calls of the public
API) and the options of config.txt that change the work: the smoothing radius
(h = ratio * spacing), the scalar grid (cell = spacing / sc) and the band.
Inputs are made on the GPU from the seed alone, by the same constructions as
postmps_gb300/synth.py's frames (jittered lattices advected by analytic fields).

A program keeps one context for all of its frames, and so do these cases: one
context per configuration, fed with frame after frame.  Meshes and diffuse
particles reach page-locked host buffers that the program also keeps.

    listed()          the cases
    draw(rng)         one more of the same ranges
    prepare(case, s)  the inputs a program has in hand (and, once, its context)
    run(state)        one pass through the public calls
    work(case)        bytes and operations a pass cannot do without
    exact(case, s)    outputs in 64 bits, where they can be stated
"""
from __future__ import annotations

import ctypes as C
import math
import os
import tempfile

import numpy as np
import torch

from postmps_gb300 import learned, pms, synth

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # a small frame, as in an interactive preview or a unit of a parameter sweep: latency and launches
        {"name": "block_4k", "scene": "block", "op": "mesh", "n": 4096, "ratio": 2, "sc": 2, "band": "plain"},
        # a frame whose welded mesh with normals goes to a renderer
        {"name": "block_27k_weld", "scene": "block", "op": "weld", "n": 27000, "ratio": 2, "sc": 2, "band": "plain"},
        # the plain water block, an ordinary frame
        {"name": "block_262k", "scene": "block", "op": "mesh", "n": 262144, "ratio": 2, "sc": 2, "band": "plain"},
        # droplets, a thin sheet and stray particles, an odd count, the wide kernel of ratio 3
        {"name": "spray_151k", "scene": "spray", "op": "mesh", "n": 151003, "ratio": 3, "sc": 2, "band": "plain"},
        # density and velocity at the mesh vertices, for shading
        {"name": "block_110k_values", "scene": "block", "op": "values", "n": 110592, "ratio": 2, "sc": 2, "band": "plain"},
        # the benchmark's crown splash: two consecutive frames from the host, mesh and diffuse particles back
        {"name": "crown_2m_sequence", "scene": "crown", "op": "sequence", "n": 2000000, "ratio": 2, "sc": 2, "band": "plain", "frames": 2},
        # the crown's surface through the learned band
        {"name": "crown_2m_learned", "scene": "crown", "op": "mesh", "n": 2000000, "ratio": 2, "sc": 2, "band": "learned"},
        # the largest frame: the dam break
        {"name": "dam_8m", "scene": "dam", "op": "mesh", "n": 8000000, "ratio": 2, "sc": 2, "band": "plain"},
        # sloshing-tank frames of many sizes in one batch, from the host, meshes back inside the graph
        {"name": "slosh_batch_8", "scene": "slosh", "op": "batch", "n": 3600000, "ratio": 2, "sc": 2, "band": "plain", "frames": 8},
        # config.txt's defaults make diffuse particles and no surface: three consecutive frames
        {"name": "crown_1m_diffuse", "scene": "crown", "op": "diffuse", "n": 1000003, "ratio": 2, "sc": 2, "band": "plain", "frames": 3},
        # the band network's loss and gradient over given samples (a trainer's batch, from the host)
        {"name": "grad_8k", "scene": "samples", "op": "grad", "n": 8192, "ratio": 2, "sc": 2, "band": "plain"},
    ]


# per operation: the scenes it is used on, and its range of particle counts (samples for grad)
_RANGE = {
    "mesh": (("block", "spray", "crown", "dam"), 3000, 3000000),
    "weld": (("block", "spray", "crown"), 3000, 600000),
    "values": (("block", "spray", "crown"), 3000, 250000),
    "sequence": (("crown",), 40000, 1800000),
    "batch": (("slosh",), 60000, 3600000),
    "diffuse": (("crown", "dam"), 40000, 2000000),
    "grad": (("samples",), 500, 100000),
}
_WEIGHTED = ("mesh",) * 5 + ("weld", "values", "sequence", "sequence", "batch", "diffuse", "grad")


def draw(rng):
    op = rng.choice(_WEIGHTED)
    scenes, lo, hi = _RANGE[op]
    case = {"scene": rng.choice(scenes), "op": op, "ratio": 2, "sc": 2, "band": "plain"}
    if op == "grad":
        case["n"] = int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1
        return case
    if op in ("mesh", "weld", "values", "diffuse"):
        case["ratio"] = rng.choice((2, 2, 2, 3, 4))
    if op in ("mesh", "weld", "sequence"):
        case["sc"] = rng.choice((1, 2, 2, 2, 3))
    if op in ("mesh", "batch"):
        case["band"] = rng.choice(("plain", "plain", "plain", "certified", "learned"))
    # wider kernels and finer grids cost more per particle: fewer particles
    cost = (case["ratio"] / 2.0) ** 3 * max(1.0, (case["sc"] / 2.0) ** 3)
    # (droplets have nothing but surface)
    cost *= 12.0 if case["scene"] == "spray" else 1.0
    hi = max(2 * lo, int(hi / cost))
    case["n"] = int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1
    if op in ("sequence", "diffuse"):
        case["frames"] = rng.choice((2, 3))
    if op == "batch":
        case["frames"] = rng.choice((2, 3, 5, 8))
    return case


# ---------------------------------------------------------------------------
# scenes, on the GPU
# ---------------------------------------------------------------------------
def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt * 7919 + 17) % (1 << 62))
    return g


def _lattice(nx, ny, nz, spacing, g):
    """Jittered lattice (+-0.1 spacing) in the first octant, float64 (n, 3)."""
    n = nx * ny * nz
    i = torch.arange(n, device="cuda")
    p = torch.stack([i // (ny * nz), (i // nz) % ny, i % nz], 1).double()
    return (p + 0.5 + 0.2 * (torch.rand(n, 3, device="cuda", dtype=torch.float64, generator=g) - 0.5)) * spacing


def _thin(p, n, g):
    """n of the particles, in their order (counts need not be products)."""
    if len(p) == n:
        return p
    keep = torch.randperm(len(p), device="cuda", generator=g)[:n].sort().values
    return p[keep]


def _box(n, ax, ay, az, spacing, g):
    """About ax : ay : az, n particles of a lattice."""
    s = (n / (ax * ay * az)) ** (1.0 / 3.0)
    nx, ny = max(1, round(ax * s)), max(1, round(ay * s))
    nz = max(1, -(-n // (nx * ny)))
    return _thin(_lattice(nx, ny, nz, spacing, g), n, g)


def _block(n, sp, seed, frame=0):
    """A turning block of water."""
    p = _box(n, 1, 1, 1, sp, _gen(seed, 1))
    d = p - p.mean(0)
    return p, torch.stack([-d[:, 1], d[:, 0], 0.3 * d[:, 0]], 1) * (1.0 / d[:, 0].max())


def _dam(n, sp, seed, frame=0):
    g = _gen(seed, 2)
    p = _box(n, 4, 1, 2, sp, g)
    h, length = p[:, 2].max(), p[:, 0].max()
    s = (p[:, 2] / h).clamp(0, 1)
    vx = 2.0 * torch.sqrt(9.81 * h) * (1 - s) * (p[:, 0] / length)
    vz = -0.5 * torch.sqrt(9.81 * h) * s * (p[:, 0] / length)
    v = torch.stack([vx, torch.zeros_like(vx), vz], 1)
    t = 0.1 * float((n / 8.0e6) ** (1.0 / 6.0)) + 0.02 * frame
    ox = length * (1.2 + 0.2 * torch.rand(1, device="cuda", dtype=torch.float64, generator=g))
    q = p + v * t
    q[:, 2] += torch.where(q[:, 0] > ox, 0.1 * torch.exp(-(((q[:, 0] - ox) / 0.05) ** 2)), torch.zeros_like(vx))
    return q, v


def _crown(n, sp, seed, frame=0):
    g = _gen(seed, 3)
    s = (n / 2.0e6) ** (1.0 / 3.0)
    n_ring = n // 5
    slab = _box(n - n_ring, 5, 5, 1, sp, g)
    side, top = slab[:, 0].max(), slab[:, 2].max()
    layers = max(2, round(10 * s))
    radius = 0.3 * side
    rs = radius + sp * (torch.arange(layers, device="cuda", dtype=torch.float64) + 0.5)
    per = torch.clamp(torch.round(2 * math.pi * rs / sp), min=1).long()
    lay0 = torch.repeat_interleave(torch.arange(layers, device="cuda"), per)
    start = torch.cumsum(per, 0) - per
    ang0 = (torch.arange(len(lay0), device="cuda") - start[lay0]).double() / per[lay0].double()
    levels = -(-n_ring // len(lay0))
    lay, ang = lay0.repeat(levels)[:n_ring], ang0.repeat(levels)[:n_ring] * 2 * math.pi
    lev = torch.arange(levels, device="cuda").repeat_interleave(len(lay0))[:n_ring].double()
    jit = (torch.rand(n_ring, 3, device="cuda", dtype=torch.float64, generator=g) - 0.5) * 0.2 * sp
    r0, th = rs[lay] + jit[:, 0], ang + jit[:, 1] / rs[lay]
    z0 = top + sp * (lev + 0.5) + jit[:, 2]
    speed = 1.5 + 0.3 * torch.randn(n_ring, device="cuda", dtype=torch.float64, generator=g)
    tilt = 0.4 + 0.8 * (z0 - top) / (sp * levels)
    dn = torch.sqrt(1 + tilt * tilt)
    v = torch.stack([speed * torch.cos(th) / dn, speed * torch.sin(th) / dn, speed * tilt / dn], 1)
    t = 0.05 * s + 0.02 * frame
    c = torch.stack([side / 2, side / 2, torch.zeros_like(side)])
    p = torch.stack([r0 * torch.cos(th), r0 * torch.sin(th), z0], 1) + c + v * t
    p[:, 2] -= 0.5 * 9.81 * t * t
    v[:, 2] -= 9.81 * t
    return torch.cat([slab, p]), torch.cat([torch.zeros_like(slab), v])


def _spray(n, sp, seed, frame=0):
    """Droplets of 10 to 400 particles, a thin sheet, 2 % stray particles."""
    g = _gen(seed, 4)
    n_stray, n_sheet = n // 50, n // 4
    n_drop = n - n_stray - n_sheet
    side = sp * (12.0 * n) ** (1.0 / 3.0)
    m = max(4, n_drop // 100)
    size = 10 + 390 * torch.rand(m, device="cuda", dtype=torch.float64, generator=g) ** 3
    rad = sp * (size * 3 / (4 * math.pi)) ** (1.0 / 3.0)
    centre = torch.rand(m, 3, device="cuda", dtype=torch.float64, generator=g) * side
    which = torch.searchsorted(torch.cumsum(size, 0) / size.sum(), torch.rand(n_drop, device="cuda", dtype=torch.float64, generator=g)).clamp(max=m - 1)
    d = torch.randn(n_drop, 3, device="cuda", dtype=torch.float64, generator=g)
    d = d / d.norm(dim=1, keepdim=True) * torch.rand(n_drop, 1, device="cuda", dtype=torch.float64, generator=g) ** (1.0 / 3.0)
    drops = centre[which] + d * rad[which, None]
    k = max(2, int(math.ceil(math.sqrt(n_sheet / 2.0))))
    sheet = _thin(_lattice(k, k, 2, sp, g), n_sheet, g)
    sheet = sheet + torch.tensor([0.0, 0.0, 0.5], device="cuda", dtype=torch.float64) * side
    stray = torch.rand(n_stray, 3, device="cuda", dtype=torch.float64, generator=g) * side
    p = torch.cat([drops, sheet, stray])
    v = torch.randn(len(p), 3, device="cuda", dtype=torch.float64, generator=g)
    return p[torch.randperm(len(p), device="cuda", generator=g)], v


def _slosh(n, sp, seed, frame=0):
    """A tank of about n particles whose surface sloshes."""
    g = _gen(seed, 5 + frame)
    p = _box(n, 2, 1, 0.4, sp, g)
    length, depth = p[:, 0].max(), p[:, 2].max()
    t = frame / 16.0
    amp = 0.08 * depth
    mode = torch.cos(math.pi * p[:, 0] / length) * (p[:, 2] / depth)
    v = torch.zeros_like(p)
    v[:, 2] = amp * 2 * math.pi * math.cos(2 * math.pi * t) * mode
    p[:, 2] += amp * math.sin(2 * math.pi * t + 0.3) * mode
    return p, v


_SCENES = {"block": (_block, 0.01), "dam": (_dam, 0.005), "crown": (_crown, 0.005), "spray": (_spray, 0.01), "slosh": (_slosh, 0.01)}


def _frame(case, n, seed, frame=0):
    make, sp = _SCENES[case["scene"]]
    p, v = make(n, sp, seed, frame)
    return p.float().contiguous(), v.float().contiguous()


def _batch_sizes(case):
    """Frames from about a seventh to the double of the mean, the same for every seed."""
    k = case["frames"]
    w = [0.15 + 0.85 * ((0.37 + 0.618034 * f) % 1.0) for f in range(k)]
    return [max(64, int(case["n"] * x / sum(w)) | 1) for x in w]


# ---------------------------------------------------------------------------
# the program around the library: its context and its host buffers
# ---------------------------------------------------------------------------
def _config(case):
    keys = {"sim.particlespacing": _SCENES[case["scene"]][1], "surface.smoothingradiusratio": case["ratio"],
            "domain.sclargridsizescale": case["sc"]}
    if case["op"] in ("sequence", "diffuse"):
        keys = dict(synth.CROWN_KEYS, **keys)
        keys["config.isdiffusegeneration"] = "true"
    if case["op"] == "diffuse":
        keys["config.issurfacereconstruct"] = "false"
    fd, path = tempfile.mkstemp(suffix=".txt")
    with os.fdopen(fd, "w") as f:
        f.write(synth.config_text(**keys))
    try:
        return pms.load_config(path)
    finally:
        os.unlink(path)


class _Program:
    """One configuration's context, and how large the program makes its host buffers
    (from a frame of its own; whatever the seed, outputs have these shapes)."""

    def __init__(self, case):
        self.ctx = pms.Context(_config(case), 0)
        if case["band"] == "learned":
            self.ctx.set_band_model(learned.load_model())
        if case["op"] != "batch":
            self.ctx.set_band_mode(case["band"])
        self.waiting = None               # the state whose streamed mesh was not waited for yet
        self.rows, self.live = [], 0
        op, k = case["op"], case.get("frames", 1)
        room = lambda n: int(n * (1.5 if case["scene"] == "spray" else 1.2)) + 8192  # noqa: E731
        if op == "batch":
            frames = [_frame(case, m, 1, f) for f, m in enumerate(_batch_sizes(case))]
            torch.cuda.synchronize()
            self.ctx.run_batch([(p.data_ptr(), v.data_ptr(), None, len(p)) for p, v in frames], learned=case["band"])
            self.rows = [room(self.ctx.batch_mesh_range(f)[1]) for f in range(k)]
            return
        for f in range(k):
            p, v = _frame(case, case["n"], 1, f)
            torch.cuda.synchronize()
            _upload(self.ctx, p, v)
            self.ctx.run_frame()
            c = self.ctx.counts()
            self.rows.append(room(c.n_mesh_vertices))
            self.live = max(self.live, room(1.2 * c.n_diffuse))
        if op == "weld":
            self.rows = [_weld_rows(case), self.rows[0]]


_programs = {}


def _program(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _programs:
        _programs.clear()                 # one program at a time
        _programs[key] = _Program(case)
    return _programs[key]


def _weld_rows(case):
    """Room for a welded mesh (one vertex per crossed grid edge)."""
    if case["scene"] == "spray":
        return int(2.4 * case["sc"] ** 2 * case["n"]) + 4096
    return int((10.0 if case["scene"] == "block" else 45.0) * case["sc"] ** 2 * case["n"] ** (2.0 / 3.0)) + 4096


def _pinned(rows, columns):
    return torch.zeros((rows, columns), dtype=torch.float32, pin_memory=True)


def prepare(case, seed):
    op, n = case["op"], case["n"]
    state = {"op": op, "band": case["band"]}
    if op == "grad":
        g = np.random.default_rng(seed)
        # features are coarse densities: 0 in air, about 1 in fluid, between at the surface
        level = g.random((n, 1), dtype=np.float32) * 2.4 - 0.7
        x = np.clip(level + g.normal(0, 0.35, (n, pms.MLP_INPUTS)).astype(np.float32), 0, 1.6)
        bits = np.ascontiguousarray(x, np.float32).view(np.uint32)
        state["x"] = ((bits + 0x7FFF + ((bits >> 16) & 1)) >> 16).astype(np.uint16)
        state["y"] = (np.abs(level[:, 0] - 0.5) < 0.3).astype(np.uint8)
        state["trainer"] = pms.Trainer(0, seed % 1000 + 1)
        return state
    program = state["program"] = _program(case)
    rows = program.rows
    if op == "batch":
        frames = [_frame(case, m, seed, f) for f, m in enumerate(_batch_sizes(case))]
        state["frames"] = frames = [(p.cpu().pin_memory(), v.cpu().pin_memory()) for p, v in frames]
        state["calls"] = [(p.data_ptr(), v.data_ptr(), None, len(p)) for p, v in frames]
    elif op in ("sequence", "diffuse"):
        frames = [_frame(case, n, seed, f) for f in range(case["frames"])]
        if op == "sequence":              # from the host
            frames = [(p.cpu().pin_memory().numpy(), v.cpu().pin_memory().numpy()) for p, v in frames]
        state["frames"] = frames
        state["live"] = [_pinned(program.live, 8) for _ in frames]
    else:
        state["frame"] = _frame(case, n, seed)
    if op in ("mesh", "batch", "sequence"):
        state["mesh"] = [_pinned(r, 3) for r in rows]
    elif op == "weld":
        state["pos"], state["normal"] = _pinned(rows[0], 3), _pinned(rows[0], 3)
        state["triangles"] = torch.zeros(rows[1], dtype=torch.int32, pin_memory=True)
    elif op == "values":
        state["vel"], state["len"], state["rho"] = _pinned(rows[0], 3), _pinned(rows[0], 1), _pinned(rows[0], 1)
    return state


def _upload(ctx, p, v):
    if isinstance(p, torch.Tensor):
        ctx.upload_device(p.data_ptr(), v.data_ptr(), None, len(p))
    else:
        ctx.upload(p, v)


def _mesh_size(ctx):
    """The frame's mesh vertices (the size query of the download call; it waits for nothing)."""
    n = C.c_uint64()
    pms.lib().pms_download_mesh(ctx.handle, None, None, 0, C.byref(n))
    return n.value


def run(state):
    op = state["op"]
    if op == "grad":
        g, loss = state["trainer"].grad(state["x"], state["y"], 4.0)
        return {"grad": g, "loss": loss}
    program = state["program"]
    ctx, lib = program.ctx, pms.lib()
    if op == "mesh":
        # a frame loop with frames in flight: this frame's mesh travels to its own host buffer
        # while the next frame runs; the loop waits for the frame before
        if program.waiting is state:
            ctx.wait_mesh()
            program.waiting = None
        mesh = state["mesh"][0]
        ctx.stream_mesh_to_host(mesh.data_ptr(), None, len(mesh))
        _upload(ctx, *state["frame"])
        ctx.run_frame()
        if program.waiting is not None:
            ctx.wait_mesh()
        program.waiting = state
        return {"n": _mesh_size(ctx), "mesh": mesh}
    if op == "weld":
        _upload(ctx, *state["frame"])
        ctx.run_frame()
        ctx._call("pms_weld_mesh", 1)
        nv, ni = C.c_uint64(), C.c_uint64()
        pos, nrm, tri = state["pos"], state["normal"], state["triangles"]
        ctx._call("pms_download_welded_mesh", pos.data_ptr(), nrm.data_ptr(), len(pos), tri.data_ptr(), len(tri),
                  C.byref(nv), C.byref(ni))
        return {"n": [nv.value, ni.value], "pos": pos, "normal": nrm, "triangles": tri}
    if op == "values":
        _upload(ctx, *state["frame"])
        ctx.run_frame()
        ctx._call("pms_scalar_values")
        n, vel = C.c_uint64(), state["vel"]
        ctx._call("pms_download_scalar_values", vel.data_ptr(), state["len"].data_ptr(), state["rho"].data_ptr(),
                  len(vel), C.byref(n))
        return {"n": n.value, "vel": vel, "vel_len": state["len"], "rhop": state["rho"]}
    if op == "batch":
        ctx.run_batch(state["calls"], learned=state["band"])
        sizes = []
        for f, mesh in enumerate(state["mesh"]):
            n = C.c_uint64()
            ctx._call("pms_batch_mesh", f, mesh.data_ptr(), len(mesh), C.byref(n))
            sizes.append(n.value)
        return {"n": sizes, "mesh": state["mesh"]}
    # a sequence: the diffuse particles are carried from frame to frame
    surface = op == "sequence"
    ctx.reset_diffuse()
    for f, (p, v) in enumerate(state["frames"]):
        if surface:
            ctx.stream_mesh_to_host(state["mesh"][f].data_ptr(), None, len(state["mesh"][f]))
        ctx.stream_diffuse_to_host(state["live"][f].data_ptr(), len(state["live"][f]))
        _upload(ctx, p, v)
        ctx.run_frame()
    out = []
    for f, live in enumerate(state["live"]):
        whole = live.view(torch.int32)    # pms_diffuse_particle: pos, ttl, vel, type
        one = {"n": ctx.wait_diffuse(), "pos": live[:, 0:3], "vel": live[:, 4:7], "ttl": whole[:, 3], "type": whole[:, 7]}
        if surface:
            one["n_mesh"], one["mesh"] = ctx.wait_mesh(), state["mesh"][f]
        out.append(one)
    return out


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once, results written once, and the operations of the sums that
    define the results: density over the particles within h (volume of the ball in
    spacings), the moments within 2h of surface particles, the field at the vertices
    around the surface, the diffuse sums.  Surface shares and mesh sizes are the
    scenes' own, in round numbers."""
    n = case["n"]
    if case["op"] == "grad":
        return {"bytes": 129 * n + 8 * pms.MLP_PARAMS, "flops": n * (2 * 64 * 64 * 2 + 8 * 64)}
    r, sc = case["ratio"], case["sc"]
    ball = 4.18879 * r ** 3
    edge = n ** (1.0 / 3.0)
    area = {"block": 6.0 * edge ** 2, "dam": 6.0 * edge ** 2, "slosh": 8.0 * edge ** 2,
            "crown": 15.0 * edge ** 2, "spray": 1.5 * n}[case["scene"]]       # in spacing^2
    if case["op"] == "batch":
        area *= case["frames"] ** (1.0 / 3.0)
    surface = min(n, 2.0 * area)
    frames = case.get("frames", 1) if case["op"] != "batch" else 1
    flops = n * ball * 12.0
    moved = 24.0 * n
    if case["op"] != "diffuse":
        soup = 6.0 * area * sc * sc
        flops += surface * 8 * ball * 30.0 + area * sc * sc * 2 * sc * ball * 0.5 * 18.0
        moved += 12.0 * soup
        if case["op"] == "values":
            flops += soup * ball * 0.5 * 20.0
            moved += 8.0 * soup
    if case["op"] in ("sequence", "diffuse"):
        flops += 0.3 * n * 4.18879 * 1.732 ** 3 * 40.0
        moved += 0.2 * n * 32.0
    return {"bytes": frames * moved, "flops": frames * flops}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["op"] == "grad":
        return _exact_grad(case, seed)
    if case["op"] == "weld" and case["n"] <= 40000 and case["ratio"] == 2 and case["sc"] <= 2:
        p, _ = _frame(case, case["n"], seed)
        pos, nrm = _exact_weld(p, _SCENES[case["scene"]][1], case["ratio"], case["sc"])
        rows = torch.zeros((2, _weld_rows(case), 3), device=pos.device, dtype=torch.float64)
        rows[0, :len(pos)], rows[1, :len(nrm)] = pos, nrm
        return {"n": None, "pos": rows[0], "normal": rows[1], "triangles": None}
    return None      # the soup's triangles follow the case tables, the particles a chain of decisions


def _exact_grad(case, seed):
    """Mean weighted cross-entropy of relu(x W1 + b1) w2 + b2 and its gradient, with the
    model as the network reads it (first-layer and w2 weights in bf16)."""
    s = prepare(case, seed)
    m = s["trainer"].model().arrays()
    bf = lambda b: (np.asarray(b).astype(np.uint32) << 16).view(np.float32).astype(np.float64)  # noqa: E731
    w1, w2, b1, b2 = bf(m["w1"]).reshape(64, 64), bf(m["w2"]), m["b1"].astype(np.float64), m["b2"]
    x, y, pw, n = bf(s["x"]), s["y"].astype(np.float64), 4.0, len(s["y"])
    pre = x @ w1 + b1
    h = np.maximum(pre, 0)
    z = h @ w2 + b2
    weight = np.where(y > 0, pw, 1.0)
    loss = float((weight * (np.logaddexp(0, z) - y * z)).mean())
    dz = weight * (1 / (1 + np.exp(-z)) - y) / n
    dh = np.outer(dz, w2) * (pre > 0)
    grad = np.concatenate([(x.T @ dh).reshape(-1), dh.sum(0), h.T @ dz, [dz.sum()]])
    return {"grad": grad, "loss": loss}


def _exact_weld(pos32, spacing, ratio, sc, iso=0.5, min_neighbours=25):
    """Welded mesh vertices and normals with every sum in 64 bits.  Grid positions and
    cells are the 32-bit ones that the method defines."""
    dev, f32, f64 = pos32.device, np.float32, torch.float64
    sp = f32(spacing)
    h = f32(ratio) * sp
    cell, vcell = f32(float(sp) * 1.5), sp / f32(sc)
    lo, hi = pos32.min(0).values.cpu().numpy(), pos32.max(0).values.cpu().numpy()
    smin, smax = lo - f32(4) * h, hi + f32(4) * h
    vmin, vmax = lo - f32(2) * h, hi + f32(2) * h
    sres = ((smax - smin) / cell).astype(np.int64)
    vres = (((vmax - vmin) / vcell).astype(np.float64) + 0.5).astype(np.int64)
    t32 = lambda a: torch.tensor(a, device=dev, dtype=torch.float32)  # noqa: E731
    c = ((pos32 - t32(smin)) / t32(cell)).long()
    key = (c[:, 2] * int(sres[1]) + c[:, 1]) * int(sres[0]) + c[:, 0]
    order = torch.sort(key, stable=True).indices
    pos32, key, c = pos32[order], key[order], c[order]
    p, n, H = pos32.to(f64), len(pos32), float(h)
    # surface cells: occupied, with an empty cell among the 27
    occ = torch.zeros(tuple(int(k) for k in sres[::-1]), device=dev)
    occ[c[:, 2], c[:, 1], c[:, 0]] = 1
    full = -torch.nn.functional.max_pool3d(-occ[None, None], 3, 1, 1)[0, 0]
    surf = full[c[:, 2], c[:, 1], c[:, 0]] == 0
    mass, sigma = 1.0, 315 / (64 * math.pi)
    rho = torch.empty(n, device=dev, dtype=f64)
    G = torch.eye(3, device=dev, dtype=f64).repeat(n, 1, 1) / H
    normal, flag = torch.zeros(n, 3, device=dev, dtype=f64), torch.zeros(n, device=dev, dtype=torch.bool)
    for a in range(0, n, 1024):
        i = slice(a, min(a + 1024, n))
        u = p[None] - p[i, None]
        d2 = (u * u).sum(2)
        rho[i] = (torch.clamp(1 - d2 / H ** 2, min=0) ** 3).sum(1) * sigma / H ** 3 * mass
        w = torch.clamp(1 - (d2.sqrt() / (2 * H)) ** 3, min=0)
        s0 = w.sum(1)
        o = (w[..., None] * u).sum(1) / s0[:, None]
        q = u - o[:, None]
        cov = (torch.einsum("ij,ija,ijb->iab", w, q, q) + H * H * torch.eye(3, device=dev, dtype=f64)) / s0[:, None, None]
        e, U = torch.linalg.eigh(cov)
        few = (d2 <= H * H).sum(1) < min_neighbours
        flag[i] = few | (e[:, 0] <= e[:, 2] * 0.25)
        nv = torch.where(few[:, None], torch.tensor([1.0, 0, 0], device=dev, dtype=f64), U[:, :, 0])
        normal[i] = torch.where(((nv * -o).sum(1) < 0)[:, None], -nv, nv)
        e = torch.maximum(e, e[:, 2:] / 4)
        k = e.prod(1, keepdim=True) ** (1.0 / 3.0) / H / e
        g = torch.where(few[:, None, None], torch.eye(3, device=dev, dtype=f64) / H, torch.einsum("iak,ik,ibk->iab", U, k, U))
        G[i] = torch.where(surf[i, None, None], g, G[i])
    weight = mass / rho * sigma * torch.linalg.det(G)
    # band: vertices within the box p +- h on the outer side, then one step along each axis
    rx, rxy, size = int(vres[0]), int(vres[0] * vres[1]), int(vres.prod())
    band = torch.zeros(size + rxy + 1, device=dev, dtype=torch.bool)
    sidx = surf.nonzero()[:, 0]
    ps = pos32[sidx]
    base = ((ps - t32(vmin)) / t32(vcell)).long()
    ext = int(np.ceil(h / vcell))
    off = torch.cartesian_prod(*[torch.arange(-ext, ext + 1, device=dev)] * 3)
    top = torch.tensor(vres - 1, device=dev)
    for a in range(0, len(sidx), 4096):
        b = slice(a, a + 4096)
        v = torch.minimum((base[b, None] + off[None]).clamp(min=0), top)
        x = v.float() * t32(vcell) + t32(vmin)
        q = ps[b, None]
        inside = ((x >= q - t32(h)) & (x <= q + t32(h))).all(2)
        side = flag[sidx[b], None] | (((x.to(f64) - q.to(f64)) * normal[sidx[b], None]).sum(2) > 0)
        band[(v[..., 2] * rxy + v[..., 1] * rx + v[..., 0])[inside & side]] = True
    ids = band.nonzero()[:, 0]
    for step in (1, rx, rxy):
        band[ids + step] = True
    ids = band[:size].nonzero()[:, 0]
    xyz = torch.stack([ids % rx, (ids // rx) % int(vres[1]), ids // rxy], 1)
    vpos = (xyz.float() * t32(vcell) + t32(vmin)).to(f64)
    # field: the sum in cell order, ended after the cell that takes it past 2 iso
    last = torch.cat([(key[1:] != key[:-1]).nonzero()[:, 0], torch.tensor([n - 1], device=dev)])
    cell_end = last[torch.searchsorted(last, torch.arange(n, device=dev))]
    field = torch.zeros(size, device=dev, dtype=f64)
    for a in range(0, len(ids), 1024):
        v = vpos[a:a + 1024]
        near = ((p > v.min(0).values - 2.6 * H) & (p < v.max(0).values + 2.6 * H)).all(1).nonzero()[:, 0]
        r = p[None, near] - v[:, None]
        m2 = torch.einsum("jab,ijb->ija", G[near], r).square_().sum(2)
        s = torch.cumsum(weight[near] * torch.clamp(1 - m2, min=0) ** 3, 1)
        past = s > 2 * iso
        end = torch.searchsorted(near, cell_end[near[past.int().argmax(1)]], right=True) - 1
        field[ids[a:a + 1024]] = torch.where(past.any(1), s.gather(1, end[:, None])[:, 0], s[:, -1])
    # cubes with eight band corners; their crossed edges, by lower corner and axis
    corner = torch.tensor([x + y * rx + z * rxy for z in (0, 1) for y in (0, 1) for x in (0, 1)], device=dev)
    cid = ids[:, None] + corner
    whole = (cid < size).all(1)
    cid = cid[whole]
    cid = cid[band[cid].all(1)]
    below = field[cid] <= iso
    keys = []
    for axis, bit in ((0, 1), (1, 2), (2, 4)):
        for k in range(8):
            if not k & bit:
                keys.append(3 * cid[below[:, k] != below[:, k | bit], k] + axis)
    keys = torch.unique(torch.cat(keys))
    va, axis = keys // 3, keys % 3
    vb = va + torch.tensor([1, rx, rxy], device=dev)[axis]
    coords = lambda i: torch.stack([i % rx, (i // rx) % int(vres[1]), i // rxy], 1)  # noqa: E731
    xa, xb = ((coords(i).float() * t32(vcell) + t32(vmin)).to(f64) for i in (va, vb))
    t = ((iso - field[va]) / (field[vb] - field[va]))[:, None]

    def gradient(i):
        x, out = coords(i), []
        for a, step in enumerate((1, rx, rxy)):
            left = torch.where(x[:, a] > 0, field[(i - step).clamp(min=0)], torch.zeros((), device=dev, dtype=f64))
            right = torch.where(x[:, a] + 1 < int(vres[a]), field[(i + step).clamp(max=size - 1)], torch.zeros((), device=dev, dtype=f64))
            out.append(left - right)
        return torch.nn.functional.normalize(torch.stack(out, 1), dim=1)

    na, nb = gradient(va), gradient(vb)
    return xa + t * (xb - xa), torch.nn.functional.normalize(na + t * (nb - na), dim=1)
