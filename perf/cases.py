"""The work that users of fluide_engine_b200 have it do, as cases that can be timed and compared.

A case is a dict of plain values.  `kind` says which public path it takes:

  step      a resident scene advances one substep (Scene.restore of a checkpoint, Scene.step, particles read into
            device tensors): what a simulation loop, a parameter sweep or a resumed job does
  frame     the same through Scene.advance_frame (the reference's AdvanceSingleFrame, CFL-adaptive)
  roundtrip a caller that owns the particles: set_particles and set_pressure, one substep, get_particles, with
            device tensors or pinned host buffers (`buffers`), in the caller's own particle order
  batch     many scenes of uneven sizes and mixed transfers advanced by one Batch.step
  surface   the fluid surface of the particles (GetSurface per frame): build, then the mesh into device tensors
  mesh      Mesh2SDF of a triangle mesh onto a node grid (scene initialisation, emitters, colliders)

Every input is made from the seed alone.  Fluid bodies are the benchmark's dam break and pool with a falling sphere,
with wavy free surfaces, a smooth swirl and a little spray, so cell marks, extrapolation and the
pressure system look as they do in mid-run; the pressure starts from one that about balances gravity, a guess like
the previous substep's pressure in a running scene.  Resident scenes hold their particles in the order a running
scene keeps them (cell tiles, as of the substep before).
"""
import ctypes
import math

import numpy as np
import torch

import fluide_engine_b200 as fe
from fluide_engine_b200._abi import check, ptr

SOLVERS = {"PIC": fe.PIC, "FLIP": fe.FLIP, "APIC": fe.APIC}
GRAVITY = 9.81
BLEND = 0.05


def listed():
    return [
        # the smallest call: one display frame of a 16^3 preview, a chain of launches on a few thousand particles
        dict(name="flip_frame_16", kind="frame", nx=16, ny=16, nz=16, solver="FLIP", body="dam", dt=1 / 60, tol=1e-6,
             cfl=1.0),
        # the reference's first configuration: 32^3 FLIP dam break, 63 thousand particles
        dict(name="flip_32", kind="step", nx=32, ny=32, nz=32, solver="FLIP", body="dam", dt=1 / 240, tol=1e-6,
             cfl=1.0),
        # a caller with its own device arrays, PIC transfer, ordinary size
        dict(name="pic_64_device", kind="roundtrip", buffers="device", nx=64, ny=64, nz=64, solver="PIC", body="dam",
             dt=1 / 240, tol=1e-6, cfl=1.0),
        # odd extents, no power of two, the reference's default maxCfl of 3 (three extrapolation passes and RK2 steps)
        dict(name="apic_ragged", kind="roundtrip", buffers="device", nx=61, ny=90, nz=47, solver="APIC", body="pool",
             dt=1 / 240, tol=1e-6, cfl=3.0),
        # end to end from pinned host buffers and back, as the benchmark's end-to-end figure takes it
        dict(name="flip_96_host", kind="roundtrip", buffers="host", nx=96, ny=96, nz=96, solver="FLIP", body="dam",
             dt=1 / 240, tol=1e-6, cfl=1.0),
        # the headline scene: 128^3 FLIP dam break, four million particles
        dict(name="flip_128", kind="step", nx=128, ny=128, nz=128, solver="FLIP", body="dam", dt=1 / 240, tol=1e-6,
             cfl=1.0),
        # the largest scene: 256^3 APIC sphere drop into a pool, 42 million particles, pressure to 1e-8
        dict(name="apic_pool_256", kind="step", nx=256, ny=256, nz=256, solver="APIC", body="pool", dt=1 / 480,
             tol=1e-8, cfl=1.0),
        # a server's batch: scenes of 32^3 .. 128^3, all three transfers
        dict(name="batch_16", kind="batch", scenes=16, nmin=32, nmax=128, dt=1 / 240, tol=1e-6, cfl=1.0),
        # viscosity switched on (the value of the reference's example program)
        dict(name="flip_64_viscous", kind="step", nx=64, ny=64, nz=64, solver="FLIP", body="dam", dt=1 / 240, tol=1e-6,
             cfl=1.0, viscosity=0.01),
        # a solid box in the dam break's path
        dict(name="flip_64_collider", kind="step", nx=64, ny=64, nz=64, solver="FLIP", body="dam", dt=1 / 240,
             tol=1e-6, cfl=1.0, collider=True),
        # one frame's surface mesh for a renderer
        dict(name="surface_128", kind="surface", nx=128, ny=128, nz=128, solver="FLIP", body="dam"),
        # scene initialisation from a mesh of 1280 triangles
        dict(name="mesh_sdf_96", kind="mesh", nx=96, ny=96, nz=96, subdiv=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes spread over their logarithm, cubes and ragged boxes, every transfer and option."""
    kind = rng.choice(["step", "step", "step", "step", "roundtrip", "roundtrip", "frame", "batch", "surface", "mesh"])
    if kind == "batch":
        return dict(kind="batch", scenes=rng.randint(4, 16), nmin=rng.choice([16, 24, 32]), nmax=_log_int(rng, 40, 128),
                    dt=1 / rng.choice([120, 240, 480]), tol=1e-6, cfl=rng.choice([1.0, 2.0]))
    n = _log_int(rng, 16, 176 if kind == "step" else 112)
    if rng.random() < 0.5:
        nx, ny, nz = (max(12, int(n * rng.uniform(0.6, 1.4))) for _ in range(3))
    else:
        nx = ny = nz = n
    if kind == "mesh":
        return dict(kind="mesh", nx=nx, ny=ny, nz=nz, subdiv=rng.randint(1, 4))
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz, solver=rng.choice(["PIC", "FLIP", "FLIP", "APIC"]),
                body=rng.choice(["dam", "dam", "pool"]))
    if kind == "surface":
        return case
    case.update(dt=1 / rng.choice([120, 240, 480]), tol=rng.choice([1e-6, 1e-6, 1e-8]), cfl=rng.choice([1.0, 1.0, 2.0, 3.0]))
    if kind == "roundtrip":
        case["buffers"] = rng.choice(["device", "host"])
    if kind == "step" and max(nx, ny, nz) <= 80:
        extra = rng.random()
        if extra < 0.2:
            case["viscosity"] = rng.choice([0.001, 0.01, 0.1])
        elif extra < 0.4 and case["solver"] != "PIC":
            case["collider"] = True
    return case


# ------------------------------------------------------------------------------------------------ inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _extent(n):
    h = 1.0 / max(n)
    return tuple(k * h for k in n), h


def _batch_specs(case):
    """The scenes of a batch: (n, solver, body), a fixed spread of sizes over [nmin, nmax] and all transfers."""
    specs = []
    for k in range(case["scenes"]):
        t = (k * 0.618034) % 1.0
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** t)) & ~3
        n = max(12, n) if k % 8 else case["nmax"]  # every eighth scene is one of the largest
        specs.append(((n, n, n), ("FLIP", "APIC", "PIC")[k % 3], "pool" if k % 4 == 3 else "dam"))
    return specs


def fluid(n, body, dt, seed, tile_order):
    """Particles of a fluid body on the device: positions and velocities (float32), APIC matrices, and a pressure
    (float64, z y x) that about balances gravity in the cells that hold particles."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(1000003 * int(seed) + 17)
    r = np.random.RandomState(sum((k + 1) * m for k, m in enumerate(n)) + (7919 if body == "dam" else 0))
    size, h = _extent(n)
    ph = r.uniform(0, 2 * math.pi, 5)  # the body's shape is the scene's; its particles and their motion are the seed's
    wave = [float(a) for a in r.uniform(0.7, 1.3, 4) * 0.012]
    axis = [(torch.arange(2 * n[a], device=dev, dtype=torch.float32) + 0.5) * (0.5 * h) for a in range(3)]
    X, Y, Z = axis[0][:, None, None], axis[1][None, :, None], axis[2][None, None, :]
    if body == "dam":
        side = 0.4 * size[0] + wave[0] * torch.sin(9.0 * Y + ph[0]) + wave[1] * torch.sin(14.0 * Z + ph[1])
        top = 0.6 * size[1] + wave[2] * torch.sin(11.0 * X + ph[2]) + wave[3] * torch.sin(8.0 * Z + ph[3])
        inside = (X < side) & (Y < top)
        ball = None
    else:
        top = 0.3 * size[1] + wave[2] * torch.sin(11.0 * X + ph[2]) + wave[3] * torch.sin(8.0 * Z + ph[3])
        ball = (0.5 * size[0], 0.6 * size[1], 0.5 * size[2], 0.15 * min(size))
        inside = (Y < top) | ((X - ball[0]) ** 2 + (Y - ball[1]) ** 2 + (Z - ball[2]) ** 2 < ball[3] ** 2)
    at = torch.nonzero(inside.expand(2 * n[0], 2 * n[1], 2 * n[2]))
    count = at.shape[0]
    pos = (at.to(torch.float32) + torch.rand((count, 3), generator=g, device=dev)) * (0.5 * h)
    del at, inside
    spray = torch.rand((max(8, count // 1000), 3), generator=g, device=dev) * torch.tensor(
        [0.98 * size[0], 0.35 * size[1], 0.98 * size[2]], device=dev) + torch.tensor(
        [0.01 * size[0], 0.6 * size[1], 0.01 * size[2]], device=dev)
    pos = torch.cat([pos, spray])
    hi = torch.tensor([s * (1 - 1e-6) for s in size], device=dev, dtype=torch.float32)
    pos = torch.minimum(pos, hi).contiguous()
    x, y, z = pos[:, 0], pos[:, 1], pos[:, 2]
    # a swirl without divergence or flow through the walls, as the previous substep's projection leaves it
    kx, ky, kz = math.pi / size[0], math.pi / size[1], 2.0 * math.pi / size[2]
    c0 = float(np.random.RandomState(int(seed) % (1 << 31)).uniform(0, 2 * math.pi))
    a0, a1 = 0.5 / ky, 0.25 / ky
    vel = torch.empty_like(pos)
    along = a0 * (1.0 + 0.3 * torch.cos(2.0 * z + c0))
    vel[:, 0] = ky * along * torch.sin(kx * x) * torch.cos(ky * y)
    vel[:, 1] = -kx * along * torch.cos(kx * x) * torch.sin(ky * y) + kz * a1 * torch.sin(ky * y) * torch.cos(kz * z)
    vel[:, 2] = -ky * a1 * torch.cos(ky * y) * torch.sin(kz * z)
    del along
    vel += 0.005 * torch.randn(vel.shape, generator=g, device=dev)
    vel[count:] *= 2.0
    if ball is not None:
        drop = (x - ball[0]) ** 2 + (y - ball[1]) ** 2 + (z - ball[2]) ** 2 < ball[3] ** 2
        vel[drop, 1] -= 2.0
    C = 0.3 * torch.randn((pos.shape[0], 9), generator=g, device=dev)
    if tile_order:  # the order of the cells of one substep earlier, 8^3 cells a tile
        c = [((pos[:, a] - dt * vel[:, a]) / h).long().clamp_(0, n[a] - 1) for a in range(3)]
        t = [(k + 7) // 8 for k in n]
        key = (((c[2] >> 3) * t[1] + (c[1] >> 3)) * t[0] + (c[0] >> 3)) * 512 + (c[2] & 7) * 64 + (c[1] & 7) * 8 + (c[0] & 7)
        order = torch.argsort(key, stable=True)
        pos, vel, C = pos[order].contiguous(), vel[order].contiguous(), C[order].contiguous()
    cells = [(pos[:, a] / h).long().clamp_(0, n[a] - 1) for a in range(3)]
    full = torch.zeros(n[2] * n[1] * n[0], dtype=torch.float64, device=dev)
    full[(cells[2] * n[1] + cells[1]) * n[0] + cells[0]] = 1.0
    mark = full.view(n[2], n[1], n[0]) > 0
    b = torch.zeros(mark.shape, dtype=torch.float64, device=dev)
    b[:, 0, :] = -GRAVITY * dt / h
    p = _conjugate_gradient(b, mark, h, 2 * max(n))
    return pos, vel, C, p.contiguous()


def icosphere(subdiv, seed):
    """A closed, gently bumpy triangle mesh in the unit cube: vertices (V, 3) and triangles (T, 3)."""
    r = np.random.RandomState((int(seed) * 104729 + 5) % (1 << 31))
    t = (1.0 + 5 ** 0.5) / 2.0
    V = [(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t), (t, 0, -1),
         (t, 0, 1), (-t, 0, -1), (-t, 0, 1)]
    F = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2), (10, 7, 6),
         (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10), (8, 6, 7),
         (9, 8, 1)]
    V = [np.array(v, float) / np.linalg.norm(v) for v in V]
    for _ in range(subdiv):
        seen, finer = {}, []

        def mid(a, b):
            k = (min(a, b), max(a, b))
            if k not in seen:
                m = V[a] + V[b]
                V.append(m / np.linalg.norm(m))
                seen[k] = len(V) - 1
            return seen[k]

        for a, b, c in F:
            ab, bc, ca = mid(a, b), mid(b, c), mid(c, a)
            finer += [(a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca)]
        F = finer
    V = np.array(V)
    bump = 1.0 + 0.05 * np.sin(4 * V @ r.uniform(-1, 1, (3, 3)) + r.uniform(0, 6, 3)).sum(1, keepdims=True)
    return V * bump * 0.27, np.array(F, dtype=np.int64)


def box_collider():
    """The box [0.55, 0.8] x [0, 0.3] x [0.35, 0.65]: vertices, triangles with a normal id, unit face normals."""
    lo, hi = np.array([0.55, 0.0, 0.35]), np.array([0.8, 0.3, 0.65])
    V = np.array([[(lo, hi)[(c >> a) & 1][a] for a in range(3)] for c in range(8)])
    tri = []
    for a, b, c, d in [(0, 2, 3, 1), (4, 5, 7, 6), (0, 1, 5, 4), (2, 6, 7, 3), (0, 4, 6, 2), (1, 3, 7, 5)]:
        tri += [(a, b, c), (a, c, d)]
    T = np.array([[a, b, c, t] for t, (a, b, c) in enumerate(tri)], dtype=np.int64)
    N = np.cross(V[T[:, 1]] - V[T[:, 0]], V[T[:, 2]] - V[T[:, 0]])
    return V, T, N / np.linalg.norm(N, axis=1, keepdims=True)


# ------------------------------------------------------------------------------------------------ prepare and run

class _Resident:
    """A scene with its start state as a checkpoint and device tensors for its particles."""

    def __init__(self, n, solver, body, dt, tol, cfl, seed, viscosity=0.0, collider=False):
        size, h = _extent(n)
        pos, vel, C, p = fluid(n, body, dt, seed, tile_order=True)
        torch.cuda.synchronize()
        self.apic = solver == "APIC"
        self.scene = fe.Scene(n, solver=SOLVERS[solver], size=size, flip_blend=BLEND, max_cfl=cfl, cg_rel_tol=tol,
                              cg_max_it=4000, max_refine=24, viscosity=viscosity)
        if collider:
            V, T, N = box_collider()
            self.scene.add_mesh_collider(V * np.array(size), T, N, n, (0.0, 0.0, 0.0), (h, h, h))
        self.scene.set_particles(pos, vel, C if self.apic else None)
        check(fe.lib().fe_scene_set_pressure(self.scene.handle, ptr(p)))
        self.start = self.scene.checkpoint()
        self.pos, self.vel, self.C = torch.empty_like(pos), torch.empty_like(vel), torch.empty_like(C) if self.apic else None

    def read(self):
        check(fe.lib().fe_scene_get_particles(self.scene.handle, ptr(self.pos), ptr(self.vel), ptr(self.C),
                                              self.pos.shape[0]))
        return {"pos": self.pos, "vel": self.vel, "C": self.C} if self.apic else {"pos": self.pos, "vel": self.vel}


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "mesh":
        n = (case["nx"], case["ny"], case["nz"])
        size, h = _extent(n)
        V, T = icosphere(case["subdiv"], seed)
        state.update(V=V + 0.5 * np.array(size), T=T, n=n, h=h)
        return state
    if kind == "batch":
        state["members"] = [_Resident(n, solver, body, case["dt"], case["tol"], case["cfl"], seed * 64 + k)
                            for k, (n, solver, body) in enumerate(_batch_specs(case))]
        state["batch"] = fe.Batch([m.scene for m in state["members"]])
        for _ in range(10):  # a batch in service runs from its captured graph
            _restore(state["members"])
            state["batch"].step(case["dt"], 1, stats=False)
        torch.cuda.synchronize()
        return state
    n = (case["nx"], case["ny"], case["nz"])
    size, _ = _extent(n)
    if kind == "surface":
        pos, vel, _, _ = fluid(n, case["body"], 1 / 240, seed, tile_order=True)
        torch.cuda.synchronize()
        state["scene"] = fe.Scene(n, solver=SOLVERS[case["solver"]], size=size, max_cfl=1.0)
        state["scene"].set_particles(pos, vel)
        room = n[0] * n[1] * n[2] // 3 + 8192  # a renderer's buffers, larger than any frame's mesh
        state.update(vertices=torch.zeros((room, 3), dtype=torch.float64, device="cuda"),
                     normals=torch.zeros((room, 3), dtype=torch.float64, device="cuda"),
                     triangles=torch.zeros((2 * room, 4), dtype=torch.int64, device="cuda"))
        return state
    if kind == "roundtrip":
        pos, vel, C, p = fluid(n, case["body"], case["dt"], seed, tile_order=False)
        if case["buffers"] == "host":
            pos, vel, C, p = (t.cpu().pin_memory() for t in (pos, vel, C, p))
        torch.cuda.synchronize()
        apic = case["solver"] == "APIC"
        state["scene"] = fe.Scene(n, solver=SOLVERS[case["solver"]], size=size, flip_blend=BLEND, max_cfl=case["cfl"],
                                  cg_rel_tol=case["tol"], cg_max_it=4000, max_refine=24, max_particles=pos.shape[0])
        like = (lambda t: torch.empty_like(t, pin_memory=True)) if case["buffers"] == "host" else torch.empty_like
        state.update(pos=pos, vel=vel, C=C if apic else None, p=p, pos1=like(pos), vel1=like(vel),
                     C1=like(C) if apic else None)
        return state
    state["resident"] = _Resident(n, case["solver"], case["body"], case["dt"], case["tol"], case["cfl"], seed,
                                  case.get("viscosity", 0.0), case.get("collider", False))
    return state


def _restore(members):
    for m in members:
        m.scene.restore(m.start)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        m = state["resident"]
        m.scene.restore(m.start)
        m.scene.step(case["dt"], 1)
        return m.read()
    if kind == "frame":
        m = state["resident"]
        m.scene.restore(m.start)
        count = m.scene.advance_frame(case["dt"])
        return {"substeps": count, **m.read()}
    if kind == "roundtrip":
        L, s = fe.lib(), state["scene"]
        s.set_particles(state["pos"], state["vel"], state["C"])
        check(L.fe_scene_set_pressure(s.handle, ptr(state["p"])))
        s.step(case["dt"], 1)
        check(L.fe_scene_get_particles(s.handle, ptr(state["pos1"]), ptr(state["vel1"]), ptr(state["C1"]),
                                       state["pos1"].shape[0]))
        out = {"pos": state["pos1"], "vel": state["vel1"]}
        if state["C1"] is not None:
            out["C"] = state["C1"]
        return out
    if kind == "batch":
        _restore(state["members"])
        state["batch"].step(case["dt"], 1)
        return [m.read() for m in state["members"]]
    if kind == "surface":
        L, s = fe.lib(), state["scene"]
        nv, nt = ctypes.c_uint64(), ctypes.c_uint64()
        check(L.fe_scene_build_surface(s.handle, ctypes.byref(nv), ctypes.byref(nt)))
        if nv.value > state["vertices"].shape[0] or nt.value > state["triangles"].shape[0]:
            raise RuntimeError("the mesh does not fit the buffers: %d vertices" % nv.value)
        mesh = {k: state[k] for k in ("vertices", "normals", "triangles")}
        check(L.fe_scene_get_surface(s.handle, ptr(mesh["vertices"]), ptr(mesh["normals"]), ptr(mesh["triangles"])))
        return {"n_vertices": nv.value, "n_triangles": nt.value, **mesh}
    return fe.mesh_to_sdf(state["V"], state["T"], state["n"], (0.0, 0.0, 0.0), (state["h"],) * 3)


# ------------------------------------------------------------------------------------------------ work

def _particles_of(n, body):
    """About how many particles the body holds (8 a cell)."""
    cells = n[0] * n[1] * n[2]
    return 8.0 * cells * (0.24 if body == "dam" else 0.3 + 4.19 * 0.15 ** 3)


def _substep_bytes(n, body, solver):
    """Particles in and out once, pressure in and out once (the warm start), the velocity grid and marks out."""
    cells = n[0] * n[1] * n[2]
    state = 4 * (15 if solver == "APIC" else 6)
    return 2.0 * state * _particles_of(n, body) + (2 * 8 + 3 * 4 + 1) * cells


def work(case):
    kind = case["kind"]
    if kind == "batch":
        specs = _batch_specs(case)
        return {"bytes": sum(_substep_bytes(n, b, s) for n, s, b in specs),
                "flops": sum(400.0 * _particles_of(n, b) for n, _, b in specs)}
    n = (case["nx"], case["ny"], case["nz"])
    cells = n[0] * n[1] * n[2]
    if kind == "mesh":
        return {"bytes": 8.0 * cells, "flops": 30.0 * cells}
    if kind == "surface":  # positions in; a mesh of about two vertices and four triangles a surface cell out
        surface = 2.5 * cells ** (2 / 3)
        return {"bytes": 12.0 * _particles_of(n, case["body"]) + surface * (2 * 48 + 4 * 32),
                "flops": 30.0 * _particles_of(n, case["body"])}
    return {"bytes": _substep_bytes(n, case["body"], case["solver"]), "flops": 400.0 * _particles_of(n, case["body"])}


# ------------------------------------------------------------------------------------------------ 64-bit values

def _bary(x, size):
    """Index and fraction of a sample position on `size` values, clamped to the last interval."""
    f = torch.floor(x)
    i = f.long()
    t = x - f
    t = torch.where(i < 0, torch.zeros_like(t), torch.where(i > size - 2, torch.ones_like(t), t))
    return i.clamp(0, size - 2), t


def _stencil(P, org, h, sizes):
    """The 8 corners (i, j, k) and per-axis weights of trilinear interpolation at P."""
    return [_bary((P[:, a] - org[a]) / h, sizes[a]) for a in range(3)]


def _corners(st):
    for t in range(8):
        ijk, w = [], 1.0
        for a in range(3):
            up = (t >> a) & 1
            ijk.append(st[a][0] + up)
            w = w * (st[a][1] if up else 1.0 - st[a][1])
        yield t, ijk, w


def _sample(A, P, org, h):
    """Trilinear sample of a (z, y, x) array at P."""
    out = 0.0
    sz, sy, sx = A.shape
    for _, (i, j, k), w in _corners(_stencil(P, org, h, (sx, sy, sz))):
        out = out + w * A[k, j, i]
    return out


def _shift(A, d, step, fill):
    """A's neighbour values at +1 / -1 along dimension d."""
    out = torch.full_like(A, fill)
    n = A.shape[d]
    if step > 0:
        out.narrow(d, 0, n - 1).copy_(A.narrow(d, 1, n - 1))
    else:
        out.narrow(d, 1, n - 1).copy_(A.narrow(d, 0, n - 1))
    return out


def _extrapolate(A, valid, depth):
    for _ in range(depth):
        total, count = torch.zeros_like(A), torch.zeros_like(A)
        for d in range(3):
            for step in (1, -1):
                ok = _shift(valid, d, step, False)
                total += torch.where(ok, _shift(A, d, step, 0.0), torch.zeros_like(A))
                count += ok
        take = ~valid & (count > 0)
        A = torch.where(take, total / count.clamp(min=1), A)
        valid = valid | take
    return A


def _walls(U):
    for c, A in enumerate(U):
        d = 2 - c
        A.narrow(d, 0, 1).zero_()
        A.narrow(d, A.shape[d] - 1, 1).zero_()


def _conjugate_gradient(b, mark, h, most=20000):
    """The pressure: per fluid cell the 7-point row (walls mirrored, air 0), solved to the 64-bit rounding."""
    inside = torch.ones_like(mark)
    m = mark.to(b.dtype)
    diag = sum(_shift(inside, d, s, False).to(b.dtype) for d in range(3) for s in (1, -1))

    def apply(x):
        y = diag * x
        for d in range(3):
            n = x.shape[d]
            y.narrow(d, 0, n - 1).sub_(x.narrow(d, 1, n - 1))
            y.narrow(d, 1, n - 1).sub_(x.narrow(d, 0, n - 1))
        return y.mul_(m)

    b = (b * m) * (h * h)
    inv = m / diag
    x, r = torch.zeros_like(b), b.clone()
    z = inv * r
    p, rz = z.clone(), (r * z).sum()
    stop = 1e-12 * float(b.norm())
    for it in range(most):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 32 == 31 and not float(r.norm()) > stop:
            break
        z = inv * r
        rz, old = (r * z).sum(), rz
        p.mul_(rz / old).add_(z)
    return x


def substep64(n, solver, body, dt, cfl, seed, tile_order):
    """One substep in 64 bits: transfer to the grid, marks, extrapolation, walls and gravity, pressure, extrapolation,
    transfer back and advection."""
    pos32, vel32, C32, _ = fluid(n, body, dt, seed, tile_order)
    size, h = _extent(n)
    nx, ny, nz = n
    dev, f8 = pos32.device, torch.float64
    count = pos32.shape[0]
    chunks = [slice(a, min(a + (1 << 22), count)) for a in range(0, count, 1 << 22)]
    faces = [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)]
    orgs = [[0.0 if a == c else 0.5 * h for a in range(3)] for c in range(3)]
    lo, hi = [0.5 * h] * 3, [s - 0.5 * h for s in size]

    def transverse(P, c):  # APIC: the particle clamped by half a cell on the two other axes
        return torch.stack([P[:, a] if a == c else P[:, a].clamp(lo[a], hi[a]) for a in range(3)], 1)

    U, valid, mark = [], [], torch.zeros(nz * ny * nx, dtype=torch.bool, device=dev)
    for c in range(3):
        fz, fy, fx = faces[c]
        clamp = (fx, fy, fz) if solver == "FLIP" else (nx, ny, nz)
        num, den = torch.zeros(fz * fy * fx, dtype=f8, device=dev), torch.zeros(fz * fy * fx, dtype=f8, device=dev)
        seen = torch.zeros(fz * fy * fx, dtype=torch.bool, device=dev)
        for s in chunks:
            P, v = pos32[s].to(f8), vel32[s, c].to(f8)
            row = C32[s, 3 * c:3 * c + 3].to(f8)
            Pc = transverse(P, c)
            for _, (i, j, k), w in _corners(_stencil(P, orgs[c], h, clamp)):
                at = (k * fy + j) * fx + i
                val = v
                if solver == "APIC":
                    for a, q in enumerate((i, j, k)):
                        val = val + row[:, a] * (orgs[c][a] + h * q.to(f8) - Pc[:, a])
                num.index_add_(0, at, w * val)
                den.index_add_(0, at, w)
                seen[at] = True
        U.append(torch.where(den > 0, num / den.clamp(min=1e-300), num).view(faces[c]))
        valid.append(seen.view(faces[c]))
    radius = 1.2 * h / math.sqrt(2.0)
    for s in chunks:
        P = pos32[s].to(f8)
        base = torch.floor(P / h - 0.5).long()
        for t in range(8):
            node = base + torch.tensor([(t >> a) & 1 for a in range(3)], device=dev)
            ok = ((node >= 0) & (node < torch.tensor(n, device=dev))).all(1)
            d2 = ((P - (node.to(f8) + 0.5) * h) ** 2).sum(1)
            ok &= d2 < radius * radius
            q = node[ok]
            mark[(q[:, 2] * ny + q[:, 1]) * nx + q[:, 0]] = True
    mark = mark.view(nz, ny, nx)
    before = [A.clone() for A in U]
    depth = math.ceil(cfl)
    U = [_extrapolate(A, m, depth) for A, m in zip(U, valid)]
    U[1] = U[1] - GRAVITY * dt
    _walls(U)
    b = torch.zeros((nz, ny, nx), dtype=f8, device=dev)
    for c, A in enumerate(U):
        d = 2 - c
        b += (A.narrow(d, 1, n[c]) - A.narrow(d, 0, n[c])) / h
    p = _conjugate_gradient(b, mark, h)
    for c, A in enumerate(U):  # faces toward + of a fluid cell, walls left alone
        d = 2 - c
        low = mark.narrow(d, 0, n[c] - 1)
        A.narrow(d, 1, n[c] - 1).add_(torch.where(low, (p.narrow(d, 1, n[c] - 1) - p.narrow(d, 0, n[c] - 1)) / h,
                                                  torch.zeros_like(p.narrow(d, 0, n[c] - 1))))
    U = [_extrapolate(A, m, depth) for A, m in zip(U, valid)]
    _walls(U)
    delta = [A - B for A, B in zip(U, before)]
    pos, vel, C = torch.empty_like(pos32, dtype=f8), torch.empty_like(vel32, dtype=f8), torch.empty_like(C32, dtype=f8)
    steps = max(int(cfl), 1)
    for s in chunks:
        P = pos32[s].to(f8)
        at = lambda Q: torch.stack([_sample(U[c], Q, orgs[c], h) for c in range(3)], 1)  # noqa: E731
        pic = at(P)
        v = pic
        if solver == "FLIP":
            d = torch.stack([_sample(delta[c], P, orgs[c], h) for c in range(3)], 1)
            blend = float(np.float32(BLEND))
            v = (1.0 - blend) * (vel32[s].to(f8) + d) + blend * pic
        if solver == "APIC":
            for c in range(3):
                st = _stencil(transverse(P, c), orgs[c], h, n)
                rows = [0.0, 0.0, 0.0]
                for t, (i, j, k), _ in _corners(st):
                    f = U[c][k, j, i]
                    w = [st[a][1] if (t >> a) & 1 else 1.0 - st[a][1] for a in range(3)]
                    sign = [1.0 if (t >> a) & 1 else -1.0 for a in range(3)]
                    rows[0] = rows[0] + sign[0] / h * w[1] * w[2] * f
                    rows[1] = rows[1] + sign[1] / h * w[0] * w[2] * f
                    rows[2] = rows[2] + sign[2] / h * w[0] * w[1] * f
                C[s, 3 * c:3 * c + 3] = torch.stack(rows, 1)
        v = v.clone()
        Q = P
        for t in range(steps):
            v0 = pic if t == 0 else at(Q)
            Q = Q + dt / steps * at(Q + 0.5 * dt / steps * v0)
        top = torch.tensor(size, dtype=f8, device=dev)
        v[(Q <= 0) | (Q >= top)] = 0.0
        pos[s], vel[s] = torch.minimum(Q.clamp(min=0.0), top), v
    return {"pos": pos, "vel": vel, "C": C} if solver == "APIC" else {"pos": pos, "vel": vel}


def exact(case, seed):
    kind = case["kind"]
    n = (case.get("nx"), case.get("ny"), case.get("nz"))
    if kind in ("surface", "mesh") or case.get("viscosity") or case.get("collider"):
        return None  # fixed 64-bit algorithms whose result is their own order of operations
    if kind == "batch":
        return [substep64(m, solver, body, case["dt"], case["cfl"], seed * 64 + k, True)
                for k, (m, solver, body) in enumerate(_batch_specs(case))]
    out = substep64(n, case["solver"], case["body"], case["dt"], case["cfl"], seed, kind != "roundtrip")
    return {"substeps": None, **out} if kind == "frame" else out
