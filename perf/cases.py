"""The work users have this library do, as timed cases.

A case names a kind and its sizes. The kinds:

frame   one rendered frame of a scene through `Simulator`: the node state of
        a checkpoint written from pinned memory, the frame's substeps, the
        positions and velocities read back to pinned memory -- a host
        program's frame loop.
splats  the deformation of a body's bound Gaussians from written positions
        and their depth sort, read back.
sort    the stable radix sort of 32-bit keys on device arrays.
cloud   a Gaussian cloud on the device voxelised, the occupancy read back.
serve   a batch of requests run by the session server, every session's
        positions read back; the sessions go on from where they are.
"""
import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "visionary-sim_gb300"))

H = 0.016  # cell edge of the scenes, metres


def listed():
    return [
        # The smallest scene: a 16 x 4 x 4 bar pinned at one end, no contact
        # (a single test body; every launch counts).
        dict(name="frame bar 16x4x4", kind="frame", scene="bar", nx=16, ny=4, nz=4, steps=10, stretch=0.0),
        # A bar with the stretch limit on, dragged compliantly by one end: the
        # limit's 24 extra passes a substep.
        dict(name="frame limited bar 31x9x10", kind="frame", scene="bar", nx=31, ny=9, nz=10, steps=10, stretch=1.15),
        # An interactive scene: a few bodies in a tank in contact with each
        # other, ~14,000 nodes, one dragged by the hard law.
        dict(name="frame pile of 6", kind="frame", scene="pile", bodies=6, n=12, steps=8),
        # One large body folded onto itself: ground and self contact.
        dict(name="frame blob 64", kind="frame", scene="blob", nx=64, ny=64, nz=64, steps=10),
        # Many independent bodies of uneven sizes in one simulator, no contact.
        dict(name="frame batch of 256", kind="frame", scene="batch", bodies=256, lo=4, hi=48, steps=10),
        # The largest scene: a blob and a thin sheet over it, two sweeps a
        # substep, contact, self contact, odd sides.
        dict(name="frame large 161x150x157", kind="frame", scene="large", nx=161, ny=150, nz=157, steps=20),
        # A million Gaussians in the body they move with: the renderer's frame.
        dict(name="splats 1M", kind="splats", n=64, count=1_000_000, axes=False),
        # A captured object for a renderer that stores rotations and scales.
        dict(name="splats 120k axes", kind="splats", n=27, count=120_001, axes=True),
        # Depth keys of a small cloud, and of a very large one.
        dict(name="sort 30k", kind="sort", count=30_011, bits=32),
        dict(name="sort 20M", kind="sort", count=20_000_000, bits=32),
        # A scanned capture of two million Gaussians to a ~230^3 grid.
        dict(name="cloud 2M", kind="cloud", count=2_000_000, across=227),
        # A small pool of sessions of uneven sizes, a request of 1-3 frames
        # each, half of them dragging a node.
        dict(name="serve 20 sessions", kind="serve", sessions=20, lo=8, hi=44),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bar", "pile", "blob", "batch", "large", "splats", "sort", "cloud", "serve"])
    if kind == "bar":
        return dict(kind="frame", scene="bar", nx=_log(rng, 6, 60), ny=_log(rng, 3, 14), nz=_log(rng, 3, 14),
                    steps=rng.randint(4, 12), stretch=rng.choice([0.0, 1.05 + 0.3 * rng.random()]))
    if kind == "pile":
        return dict(kind="frame", scene="pile", bodies=rng.randint(2, 12), n=rng.randint(6, 20),
                    steps=rng.randint(4, 12))
    if kind == "blob":
        return dict(kind="frame", scene="blob", nx=_log(rng, 14, 110), ny=_log(rng, 14, 90), nz=_log(rng, 14, 110),
                    steps=rng.randint(6, 12))
    if kind == "batch":
        return dict(kind="frame", scene="batch", bodies=_log(rng, 8, 300), lo=rng.randint(3, 6),
                    hi=rng.randint(16, 46), steps=rng.randint(6, 10))
    if kind == "large":
        return dict(kind="frame", scene="large", nx=rng.randint(90, 160), ny=rng.randint(90, 150),
                    nz=rng.randint(90, 157), steps=rng.randint(8, 20))
    if kind == "splats":
        return dict(kind="splats", n=rng.randint(12, 72), count=_log(rng, 10_000, 3_000_000),
                    axes=rng.random() < 0.3)
    if kind == "sort":
        return dict(kind="sort", count=_log(rng, 2_000, 20_000_000), bits=rng.choice([32, 32, 32, 24, 17]))
    if kind == "cloud":
        return dict(kind="cloud", count=_log(rng, 20_000, 2_000_000), across=rng.randint(40, 227))
    return dict(kind="serve", sessions=rng.randint(6, 24), lo=rng.randint(6, 9), hi=rng.randint(20, 44))


# ------------------------------------------------------------- the scenes --

def _noise(dims, gen):
    """Three octaves of value noise on a (z, y, x) grid, about half of it above 0.5."""
    nx, ny, nz = dims
    total = torch.zeros((nz, ny, nx), dtype=torch.float32)
    for octave in range(3):
        f = 4 * 2 ** octave + 1
        lattice = torch.rand((1, 1, f, f, f), generator=gen)
        total += 0.5 ** octave * torch.nn.functional.interpolate(lattice, size=(nz, ny, nx), mode="trilinear",
                                                                 align_corners=True)[0, 0]
    return total / 1.75


def _material(**changes):
    m = dict(youngs_modulus=1.2e5, poisson_ratio=0.40, density=1000.0, friction=0.4, damping=0.6, relaxation=0.012,
             max_stretch=0.0)
    m.update(changes)
    return m


def _body(dims, origin, occupancy=None, static=None, h=H, **material):
    occ = np.ones(dims[0] * dims[1] * dims[2], np.uint8) if occupancy is None else \
        np.ascontiguousarray(occupancy, np.uint8).ravel()
    return dict(dims=tuple(dims), origin=tuple(float(v) for v in origin), h=h, occ=occ, mat=_material(**material),
                static=np.zeros(0, np.uint32) if static is None else static)


def _rest(b):
    nx, ny, nz = (d + 1 for d in b["dims"])
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    ijk = np.stack([i.ravel(), j.ravel(), k.ravel()], 1).astype(np.float64)
    return ijk * b["h"] + np.asarray(b["origin"])


def _settled(rest, gen, floor, sag):
    """Rest positions (metres, y up) sagged under their weight -- the lower part of the body squeezed most,
    folding it into contact with itself -- with a bend and a small jitter, and the velocities of such a motion."""
    p = torch.from_numpy(rest)
    lo, hi = p.min(0).values, p.max(0).values
    size = (hi - lo).clamp_min(1e-6)
    t = (p - lo) / size
    p = p.clone()
    p[:, 1] = floor + size[1] * (t[:, 1] - sag * (1 - (1 - t[:, 1]) ** 3) / 3)
    phase = torch.rand(6, generator=gen, dtype=torch.float64) * 6.28
    for a in range(3):
        p[:, a] += 0.3 * H * torch.sin(6.28 * t[:, (a + 1) % 3] * 1.5 + phase[a])
    p += 0.05 * H * (torch.rand(p.shape, generator=gen, dtype=torch.float64) - 0.5)
    p[:, 1] = p[:, 1].clamp_min(floor)
    v = 0.15 * torch.sin(6.28 * t + phase[3:]) + 0.05 * torch.randn(p.shape, generator=gen, dtype=torch.float64)
    return p.numpy(), v.numpy()


def _face(dims):
    """The nodes of the x = 0 face."""
    nx, ny, nz = (d + 1 for d in dims)
    return (np.arange(ny * nz) * nx).astype(np.uint32)


def _scene(case, seed):
    """Bodies, tank, options, and a checkpoint (positions, velocities, xyz float32) of a frame case."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    rnd = lambda lo, hi: lo + (hi - lo) * float(torch.rand(1, generator=gen, dtype=torch.float64))  # noqa: E731
    logr = lambda lo, hi: math.exp(rnd(math.log(lo), math.log(hi)))  # noqa: E731
    inf = float("inf")
    s = dict(step=1 / 600, steps=case["steps"], iterations=1, contact=True, self_contact=False, isolated=False,
             tank=((-inf,) * 3, (inf,) * 3), hold=None, law="hard")
    kind = case["scene"]
    sizes = np.random.RandomState(12)  # a case's body sizes do not depend on the seed
    pos, vel = [], []
    if kind == "bar":
        dims = (case["nx"], case["ny"], case["nz"])
        s.update(contact=False)
        b = _body(dims, (0, 0, 0), static=_face(dims), youngs_modulus=logr(5e4, 4e5), poisson_ratio=0.45,
                  max_stretch=case["stretch"])
        s["bodies"] = [b]
        p = _rest(b)
        x = p[:, 0].copy()
        p[:, 1] -= 0.4 * x * x + 0.02 * x * math.sin(rnd(0, 6.28))  # bent under its weight
        pos.append(p + (x > 0)[:, None] * rnd(0.01, 0.03) * H * np.sin(37 * p))
        vel.append(0.3 * x[:, None] * np.array([0.1, -1.0, rnd(-0.5, 0.5)]))
        if case["stretch"] > 1:
            ny, nz = dims[1] + 1, dims[2] + 1
            tip = (np.arange(ny * nz) * (dims[0] + 1) + dims[0]).astype(np.uint32)[: 4 * ny]
            anchor = p[tip[0]]
            s.update(law="compliant", hold=(tip, p[tip] - anchor, anchor, anchor + [0.02, 0.01, rnd(-0.02, 0.02)]))
    elif kind == "pile":
        n, count = case["n"], case["bodies"]
        side = int(math.ceil(math.sqrt(count)))
        s["bodies"] = []
        for q in range(count):
            dims = tuple(int(v) for v in np.maximum(3, n + sizes.randint(-3, 4, 3)))
            gap = (n + 4) * 0.92 * H  # neighbours overlap a little: they touch
            origin = ((q % side) * gap, 0.5 * H, (q // side) * gap)
            noise = _noise(dims, gen)
            b = _body(dims, origin, (noise > 0.42).numpy(), youngs_modulus=logr(3e4, 3e5), friction=rnd(0.2, 0.6),
                      poisson_ratio=rnd(0.3, 0.47), density=rnd(600, 1400))
            if not b["occ"].any():
                b["occ"][:] = 1
            s["bodies"].append(b)
            p, v = _settled(_rest(b), gen, 0.0, 0.3)
            pos.append(p)
            vel.append(v + np.array([rnd(-0.4, 0.4), rnd(-1.0, 0.0), rnd(-0.4, 0.4)]))
        extent = side * (n + 4) * H
        s.update(tank=((-0.1, 0.0, -0.1), (extent + 0.1, 3 * extent + 0.5, extent + 0.1)))
        b = s["bodies"][0]
        material = _corner_counts(b) > 0
        node = int(np.flatnonzero(material)[-1])
        nodes = np.array([node], np.uint32)
        anchor = pos[0][node]
        s.update(hold=(nodes, np.zeros((1, 3)), anchor, anchor + [0.01, 0.02, rnd(-0.02, 0.02)]))
    elif kind in ("blob", "large"):
        dims = (case["nx"], case["ny"], case["nz"])
        occ = (_noise(dims, gen) > 0.5).numpy()
        occ[: max(1, dims[2] // 4), 0, 0] = True
        half = [0.5 * d * H for d in dims]
        # soft enough to stay folded: a settled body under its own weight
        blob = _body(dims, (-half[0], 0.0, -half[2]), occ, youngs_modulus=logr(6e3, 1.5e4), poisson_ratio=0.45)
        s.update(bodies=[blob], self_contact=True)
        p, v = _settled(_rest(blob), gen, 0.0, 0.85)
        pos.append(p)
        vel.append(v)
        top = dims[1] * H
        if kind == "large":
            sheet = _body((dims[0], 2, dims[2]), (-half[0], top + 2 * H, -half[2]), youngs_modulus=5e5,
                          poisson_ratio=0.48)
            s["bodies"].append(sheet)
            s.update(step=1 / 1200, iterations=2)
            q = _rest(sheet)
            q[:, 1] += -1.4 * H + 0.8 * H * np.sin(9 * q[:, 0]) * np.cos(8 * q[:, 2])
            pos.append(q)
            vel.append(np.array([0.0, -1.0, 0.0]) + 0.1 * np.sin(11 * q))
        margin = 0.1 * max(dims) * H + 4 * H
        s.update(tank=((-half[0] - margin, 0.0, -half[2] - margin), (half[0] + margin, top + 6 * H + margin,
                                                                     half[2] + margin)))
    elif kind == "batch":
        s.update(contact=False, bodies=[])
        count = case["bodies"]
        side = int(math.ceil(math.sqrt(count)))
        pitch = (case["hi"] + 4) * H
        sides = np.exp(math.log(case["lo"]) + math.log(case["hi"] / case["lo"]) * sizes.rand(count, 3))
        for q in range(count):
            dims = tuple(int(round(v)) for v in sides[q])
            b = _body(dims, ((q % side) * pitch, 0.01, (q // side) * pitch), static=_face(dims),
                      youngs_modulus=logr(1e4, 2e5), poisson_ratio=rnd(0.30, 0.48), density=rnd(700, 1500))
            s["bodies"].append(b)
            p = _rest(b)
            x = p[:, 0] - p[0, 0]
            p[:, 1] -= 0.03 * x * x
            pos.append(p)
            vel.append(x[:, None] * np.array([0.0, -0.5, rnd(-0.5, 0.5)]))
        s.update(tank=((-1.0, 0.0, -1.0), (side * pitch + 1.0, 2.0, side * pitch + 1.0)))
    s["pos"] = np.concatenate(pos).astype(np.float32)
    s["vel"] = np.concatenate(vel).astype(np.float32)
    return s


def _vsim_bodies(bodies):
    from vsim.scenes import Body

    return [Body(b["dims"], b["origin"], b["h"], b["occ"], dict(b["mat"]), b["static"]) for b in bodies]


def _fp(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def _up(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_uint32))


def _quads(xyz):
    """(n, 3) values as pinned xyzw quadruples."""
    t = torch.zeros((xyz.shape[0], 4), dtype=torch.float32, pin_memory=True)
    t[:, :3] = torch.as_tensor(xyz)
    return t


def _pinned(shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


# ---------------------------------------------------------------- prepare --

def _prepare_frame(case, seed):
    from vsim import Scene, Simulator

    s = _scene(case, seed)
    scene = Scene(_vsim_bodies(s["bodies"]), s["tank"], step_duration=s["step"], substeps=s["steps"],
                  iterations=s["iterations"], contact=s["contact"], self_contact=s["self_contact"])
    sim = Simulator(scene)
    if s["hold"]:
        nodes, offsets, place, target = s["hold"]
        sim.set_drive_law(s["law"])
        sim.hold(nodes, offsets.astype(np.float32))
    n = sim.node_count
    return dict(kind="frame", sim=sim, n=n, steps=s["steps"], hold=s["hold"], pos=_quads(s["pos"]),
                vel=_quads(s["vel"]), out_pos=_pinned((n, 4)), out_vel=_pinned((n, 4)))


def _splat_inputs(case, seed):
    """A blob with `count` Gaussians in its occupied cells, and a deformed state of its nodes."""
    n, count = case["n"], case["count"]
    s = _scene(dict(scene="blob", nx=n, ny=n, nz=n, steps=1), seed)
    b = s["bodies"][0]
    gen = torch.Generator().manual_seed(int(seed) * 104729 + 3)
    occ = torch.from_numpy(np.flatnonzero(b["occ"]))
    cell = occ[torch.randint(0, occ.numel(), (count,), generator=gen)].numpy()
    ijk = np.stack([cell % n, cell // n % n, cell // (n * n)], 1)
    means = (np.asarray(b["origin"]) + (ijk + torch.rand((count, 3), generator=gen).numpy()) * H).astype(np.float32)
    quats = torch.randn((count, 4), generator=gen)
    quats = (quats / quats.norm(dim=1, keepdim=True)).numpy()
    scales = torch.exp(torch.rand((count, 3), generator=gen) * math.log(10.0) + math.log(1e-3)).numpy()
    return s, means, quats, scales


VIEW = (0.0, -0.6, -0.8)


def _prepare_splats(case, seed):
    from vsim import Scene, Simulator

    s, means, quats, scales = _splat_inputs(case, seed)
    sim = Simulator(Scene(_vsim_bodies(s["bodies"]), s["tank"], step_duration=s["step"], contact=False))
    sim.bind_splats(0, means, quats, scales)
    count = case["count"]
    state = dict(kind="splats", sim=sim, n=sim.node_count, count=count, axes=case["axes"], pos=_quads(s["pos"]),
                 means=_pinned((count, 3)), cov=_pinned((count, 6)), order=_pinned((count,), torch.int32))
    if case["axes"]:
        state.update(rotation=_pinned((count, 4)), scale=_pinned((count, 3)))
    return state


def _prepare_sort(case, seed):
    from vsim._ffi import check, lib

    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    # depths of a cloud seen from outside, as ordered float bits: most keys
    # share their leading digits
    depth = 2.0 + 0.5 * torch.randn(case["count"], device="cuda", generator=gen)
    keys = (depth.clamp(0.1, 10.0).view(torch.int32) & ((1 << case["bits"]) - 1 if case["bits"] < 32 else -1))
    need = C.c_size_t()
    check(lib().vsim_radix_sort_u32(None, None, case["count"], case["bits"], None, C.byref(need), None))
    return dict(kind="sort", keys=keys, order=torch.empty_like(keys), n=case["count"], bits=case["bits"],
                temp=torch.empty(need.value, dtype=torch.uint8, device="cuda"), temp_bytes=need)


def _prepare_cloud(case, seed):
    from vsim._ffi import CloudOptions

    count, radius = case["count"], 0.3
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rand = lambda *shape: torch.rand(shape, device="cuda", generator=gen)  # noqa: E731
    # a scan: Gaussians on a lumpy closed surface, nothing behind it
    i = torch.arange(count, device="cuda", dtype=torch.float64)
    y = 1 - 2 * (i + 0.5) / count
    ring = torch.sqrt((1 - y * y).clamp_min(0))
    theta = math.pi * (3 - math.sqrt(5)) * i
    unit = torch.stack([torch.cos(theta) * ring, y, torch.sin(theta) * ring], 1)
    phase = 6.28 * rand(1).double()
    r = radius * (1 + 0.08 * torch.sin(5 * unit[:, 0] + phase) * torch.cos(4 * unit[:, 1]) +
                  0.005 * torch.randn(count, device="cuda", generator=gen, dtype=torch.float64))
    positions = (unit * r[:, None]).float().contiguous()
    spacing = math.sqrt(4 * math.pi * radius * radius / count)
    scales = (0.4 * spacing * torch.exp(rand(count, 3) * math.log(4.0))).contiguous()
    quats = torch.randn((count, 4), device="cuda", generator=gen)
    quats = (quats / quats.norm(dim=1, keepdim=True)).contiguous()
    h = 2.1 * radius / case["across"]
    most = (case["across"] + 40) ** 3
    options = CloudOptions(element_size=h, sigma=2.0, padding=2, seal=2, fill=1)
    return dict(kind="cloud", arrays=(positions, quats, scales), n=count, options=options,
                occupancy=_pinned((most,), torch.uint8).zero_())


def _serve_inputs(case, seed):
    """Session bodies (blobs above the ground), one request each, drags for half of them."""
    gen = torch.Generator().manual_seed(int(seed) * 31 + 5)
    rnd = lambda lo, hi: lo + (hi - lo) * float(torch.rand(1, generator=gen, dtype=torch.float64))  # noqa: E731
    bodies, frames, drags = [], [], []
    for q in range(case["sessions"]):
        # sizes log-spaced over the range (the mix does not depend on the seed), jittered
        t = (q + 0.5) / case["sessions"]
        n = int(round(math.exp(math.log(case["lo"]) + t * math.log(case["hi"] / case["lo"]))))
        occ = (_noise((n, n, n), gen) > 0.47).numpy()
        occ[n // 3: n // 3 + 3, :3, n // 3] = True
        b = _body((n, n, n), (-0.5 * n * H, 0.7 * H, -0.5 * n * H), occ, youngs_modulus=math.exp(rnd(9.2, 13.8)),
                  poisson_ratio=0.45)
        bodies.append(b)
        frames.append(1 + q % 3)
        drag = None
        if q % 2:
            inside = _corner_counts(b)
            surface = np.flatnonzero((inside > 0) & (inside < 8))
            node = int(surface[int(rnd(0, surface.size - 1e-9))])
            p0 = _rest(b)[node]
            steps = 0.05 * torch.randn((3, 3), generator=gen, dtype=torch.float64).numpy()
            control = np.vstack([p0, p0 + steps[0], p0 + steps[0] + steps[1], p0 + steps.sum(0)])
            drag = (node, control.astype(np.float32), 0.5)
        drags.append(drag)
    extent = 2 * case["hi"] * H
    return bodies, frames, drags, ((-extent, 0.0, -extent), (extent, 2 * extent, extent))


def _prepare_serve(case, seed):
    from vsim.server import Server

    bodies, frames, drags, tank = _serve_inputs(case, seed)
    server = Server(_vsim_bodies(bodies), tank)
    first = np.concatenate([[0], np.cumsum([np.prod([d + 1 for d in b["dims"]]) for b in bodies])]).astype(int)
    return dict(kind="serve", server=server, frames=frames, flags=[d is not None for d in drags], drags=drags,
                sessions=list(range(len(bodies))), first=first, out=_pinned((int(first[-1]), 4)))


def prepare(case, seed):
    return {"frame": _prepare_frame, "splats": _prepare_splats, "sort": _prepare_sort, "cloud": _prepare_cloud,
            "serve": _prepare_serve}[case["kind"]](case, seed)


# -------------------------------------------------------------------- run --

def run(state):
    from vsim import _ffi
    from vsim._ffi import check, lib

    kind, L = state["kind"], lib()
    if kind == "frame":
        sim, n = state["sim"], state["n"]
        check(L.vsim_write_state(sim.handle, _fp(state["pos"]), None, _fp(state["vel"]), n))
        if state["hold"]:
            sim.place_grab(state["hold"][2])
            sim.move_grab(state["hold"][3])
        sim.dispatch(state["steps"])
        check(L.vsim_read_state(sim.handle, _fp(state["out_pos"]), None, _fp(state["out_vel"]), n))
        return {"pos": state["out_pos"], "vel": state["out_vel"]}
    if kind == "splats":
        sim, count = state["sim"], state["count"]
        check(L.vsim_write_state(sim.handle, _fp(state["pos"]), None, None, state["n"]))
        if state["axes"]:
            sim.deform_splats_axes(VIEW)
        else:
            sim.deform_splats(VIEW)
        sim.sort_splats()
        out = {"means": state["means"], "cov": state["cov"], "order": state["order"]}
        check(L.vsim_splats_read(sim.handle, _fp(state["means"]), _fp(state["cov"]), _up(state["order"]), count))
        if state["axes"]:
            check(L.vsim_splats_read_axes(sim.handle, _fp(state["rotation"]), _fp(state["scale"]), count))
            out.update(rotation=state["rotation"], scale=state["scale"])
        return out
    if kind == "sort":
        check(L.vsim_radix_sort_u32(_up(state["keys"]), _up(state["order"]), state["n"], state["bits"],
                                    C.c_void_p(state["temp"].data_ptr()), C.byref(state["temp_bytes"]),
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["order"]
    if kind == "cloud":
        volume = C.c_void_p()
        pos, rot, scale = state["arrays"]
        check(L.vsim_voxelize_cloud_device(_fp(pos), _fp(rot), _fp(scale), state["n"], C.byref(state["options"]),
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(volume)))
        try:
            grid = _ffi.CloudGrid()
            check(L.vsim_cloud_volume_grid(volume, C.byref(grid)))
            check(L.vsim_cloud_volume_read(volume, C.cast(state["occupancy"].data_ptr(), C.POINTER(C.c_uint8)),
                                           state["occupancy"].numel()))
        finally:
            L.vsim_cloud_volume_destroy(volume)
        return {"dims": [int(d) for d in grid.dims], "filled": int(grid.filled),
                "occupied": int(grid.occupied), "cells": state["occupancy"]}
    server = state["server"]
    server.run(None, state["sessions"], state["frames"], state["flags"], state["drags"], keep=0)
    first, out = state["first"], state["out"]
    for i in state["sessions"]:
        a, b = int(first[i]), int(first[i + 1])
        check(L.vsim_server_read_positions(server._h, i, _fp(out[a:b]), b - a))
    return out


# ------------------------------------------------------------------- work --

# Arithmetic of one cell's projection: six tetrahedra, each its deformation
# gradient (27), norm, determinant and cofactors (48), two gradient sets (66),
# Gram sums and rates (126), the 2x2 solve (24) and four corner updates (44).
TET_FLOPS = 335


def _node_total(bodies):
    return sum(int(np.prod([d + 1 for d in b["dims"]])) for b in bodies)


def _cell_guess(case):
    """Nodes and occupied cells of a case's scene, near enough for a count of its work."""
    if case["kind"] == "serve":
        sides = [math.exp(math.log(case["lo"]) + (q + 0.5) / case["sessions"] * math.log(case["hi"] / case["lo"]))
                 for q in range(case["sessions"])]
        return sum((n + 1) ** 3 for n in sides), [0.6 * n ** 3 for n in sides]
    s = case["scene"]
    if s == "pile":
        return case["bodies"] * (case["n"] + 1) ** 3, 0.7 * case["bodies"] * case["n"] ** 3
    if s == "batch":
        span = math.log(case["hi"] / case["lo"])
        side = (case["hi"] - case["lo"]) / span  # mean of a log-uniform side
        return case["bodies"] * (side + 1) ** 3, case["bodies"] * side ** 3
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    cells = case["nx"] * case["ny"] * case["nz"]
    if s == "bar":
        return nodes, cells
    if s == "large":
        return nodes + 3 * (case["nx"] + 1) * (case["nz"] + 1), 0.5 * cells + 2 * case["nx"] * case["nz"]
    return nodes, 0.5 * cells


def work(case):
    kind = case["kind"]
    if kind == "frame":
        nodes, cells = _cell_guess(case)
        sweeps = 2 if case["scene"] == "large" else 1
        # state in and out (positions and velocities), a cell record each
        return {"bytes": 64.0 * nodes + 16.0 * cells, "flops": cells * case["steps"] * sweeps * 6.0 * TET_FLOPS}
    if kind == "splats":
        per = 44 + 40 + (28 if case["axes"] else 0)
        return {"bytes": float(case["count"] * per + 16 * (case["n"] + 1) ** 3), "flops": 330.0 * case["count"]}
    if kind == "sort":
        return {"bytes": 8.0 * case["count"], "flops": 0.0}
    if kind == "cloud":
        return {"bytes": 40.0 * case["count"] + 1.2 * case["across"] ** 3, "flops": 400.0 * case["count"]}
    nodes, cells = _cell_guess(case)
    return {"bytes": 16.0 * nodes + 32.0 * nodes,
            "flops": sum(c * (1 + q % 3) for q, c in enumerate(cells)) * 10 * 6.0 * TET_FLOPS}


# ------------------------------------------------------ the 64-bit answers --

TETS = ((0, 1, 3, 7), (0, 5, 1, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 4, 5, 7), (0, 6, 4, 7))


def _corner_counts(b):
    """Occupied cells around each node, in node order."""
    nx, ny, nz = b["dims"]
    occ = np.zeros((nz + 2, ny + 2, nx + 2), np.int32)
    occ[1:-1, 1:-1, 1:-1] = b["occ"].reshape(nz, ny, nx)
    return sum(occ[c:c + nz + 1, r:r + ny + 1, q:q + nx + 1] for c in (0, 1) for r in (0, 1)
               for q in (0, 1)).ravel()


class _Exact:
    """The solver's substep in 64 bits with plain tensor operations."""

    def __init__(self, bodies, tank, step, iterations, contact, self_contact, isolated):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev, self.dt, self.iterations = dev, step, iterations
        self.contact, self.self_contact, self.isolated = contact, self_contact, isolated
        T = lambda a, dtype=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=dev)  # noqa: E731
        self.tank = (T(tank[0]), T(tank[1]))
        offset = np.concatenate([[0], np.cumsum([_node_total([b]) for b in bodies])]).astype(np.int64)
        self.n = int(offset[-1])
        w, body_of = np.zeros(self.n), np.zeros(self.n, np.int64)
        cells = [[] for _ in range(8)]
        recs, coords, radius, boxes = [], [], [], []
        for q, b in enumerate(bodies):
            nx, ny, nz = b["dims"]
            count = _corner_counts(b)
            mass = b["mat"]["density"] * b["h"] ** 3 / 8 * count
            inv = np.divide(1.0, mass, out=np.zeros(count.size), where=count > 0)
            inv[b["static"].astype(np.int64)] = 0.0
            w[offset[q]:offset[q + 1]] = inv
            body_of[offset[q]:offset[q + 1]] = q
            c = np.flatnonzero(b["occ"])
            i, j, k = c % nx, c // nx % ny, c // (nx * ny)
            colour = (i & 1) | (j & 1) << 1 | (k & 1) << 2
            n0 = offset[q] + i + (nx + 1) * (j + (ny + 1) * k)
            for col in range(8):
                at = n0[colour == col]
                cells[col].append(np.stack([at, np.full(at.size, q), np.full(at.size, nx + 1),
                                            np.full(at.size, (nx + 1) * (ny + 1))], 1))
            s = np.flatnonzero((count > 0) & (count < 8))
            recs.append(offset[q] + s)
            coords.append(np.stack([s % (nx + 1), s // (nx + 1) % (ny + 1), s // ((nx + 1) * (ny + 1))], 1))
            radius.append(np.full(s.size, b["h"] / 2))
            boxes.append((np.asarray(b["origin"]), np.asarray(b["origin"]) + np.asarray(b["dims"]) * b["h"]))
        self.w, self.body_of = T(w), T(body_of, torch.int64)
        self.active = T(w, torch.float64) > 0
        mats = [b["mat"] for b in bodies]
        hs = np.array([b["h"] for b in bodies])
        nu = np.clip([m["poisson_ratio"] for m in mats], 0.25, 0.49)
        e = np.maximum(1.0, [m["youngs_modulus"] for m in mats])
        mu, lam = e / (2 * (1 + nu)), e * nu / ((1 + nu) * (1 - 2 * nu))
        self.lame = (mu, lam)
        volume = hs ** 3 / 6
        per = dict(adev=1 / (mu * volume) / step ** 2, ahyd=1 / (lam * volume) / step ** 2, gamma=1 + mu / lam,
                   relax=np.array([m["relaxation"] for m in mats]) / step, h=hs,
                   stretch=np.array([m["max_stretch"] for m in mats]))
        self.friction = T([m["friction"] for m in mats])
        self.damp = T(np.exp(-np.array([m["damping"] for m in mats]) * step))
        self.limited = bool((per["stretch"] > 1).any())
        self.colours = []
        for col in range(8):
            c = np.concatenate(cells[col])
            if not c.size:
                continue
            n0, q, sy, sz = c.T
            ids = np.stack([n0 + (v & 1) + (v >> 1 & 1) * sy + (v >> 2) * sz for v in range(8)])
            self.colours.append((T(ids, torch.int64), {k: T(v[q]) for k, v in per.items()}))
        self.rest_inverse = []
        for tet in TETS:
            corner = np.array([[v & 1, v >> 1 & 1, v >> 2] for v in tet], np.float64)
            self.rest_inverse.append(T(np.linalg.inv((corner[1:] - corner[0]).T)))
        self.rec = T(np.concatenate(recs), torch.int64)
        self.coord = T(np.concatenate(coords), torch.int64)
        self.radius = T(np.concatenate(radius))
        self.grids(boxes, hs, tank, T)

    def grids(self, boxes, hs, tank, T):
        """The contact grid each body bins into: the tank's, or its own where bodies are isolated."""
        origin, size, dims, base = [], [], [], []
        at = 0
        for (lo, hi), h in zip(boxes, hs):
            if self.isolated:
                pad = np.maximum(0.25 * (hi - lo), 4 * h)
                mn, mx, edge = np.maximum(tank[0], lo - pad), np.minimum(tank[1], hi + pad), h
            else:
                mn, mx, edge = np.asarray(tank[0]), np.asarray(tank[1]), hs.max()
            if not np.isfinite(mn).all():  # no contact in such a scene
                mn, mx = np.zeros(3), np.ones(3)
            d = np.maximum(1, np.ceil((mx - mn) / edge)).astype(np.int64) + 2
            origin.append(mn - edge)
            size.append(edge)
            dims.append(d)
            base.append(at)
            at += int(np.prod(d)) if self.isolated else 0
        self.grid = (T(np.array(origin)), T(np.array(size)), T(np.array(dims), torch.int64),
                     T(np.array(base), torch.int64))

    def project(self, ids, k, limit_only):
        p, prev, w = list(self.pos[ids]), self.prev[ids], self.w[ids]
        dot = lambda a, b: (a * b).sum(-1)  # noqa: E731
        if not limit_only:
            for t, tet in enumerate(TETS):
                B = self.rest_inverse[t]
                E = torch.stack([p[v] - p[tet[0]] for v in tet[1:]], -1)
                F = (E @ B) / k["h"][:, None, None]
                c_dev = F.flatten(1).norm(dim=1)
                f = F.unbind(-1)
                cof = torch.stack([torch.linalg.cross(f[1], f[2]), torch.linalg.cross(f[2], f[0]),
                                   torch.linalg.cross(f[0], f[1])], -1)
                c_hyd = dot(f[0], cof[..., 0]) - k["gamma"]
                inv = torch.where(c_dev > 1e-9, 1 / c_dev, torch.zeros_like(c_dev))
                D = (F * inv[:, None, None]) @ B.T / k["h"][:, None, None]
                Hy = cof @ B.T / k["h"][:, None, None]
                d, h = list(D.unbind(-1)), list(Hy.unbind(-1))
                d, h = [-(d[0] + d[1] + d[2])] + d, [-(h[0] + h[1] + h[2])] + h
                ws = [w[v] for v in tet]
                gx = sum(a * dot(x, x) for a, x in zip(ws, d))
                gy = sum(a * dot(x, y) for a, x, y in zip(ws, d, h))
                gz = sum(a * dot(y, y) for a, y in zip(ws, h))
                moved = [p[v] - prev[v] for v in tet]
                rx, ry = sum(dot(x, m) for x, m in zip(d, moved)), sum(dot(y, m) for y, m in zip(h, moved))
                stiff = 1 + k["relax"]
                a00, a01, a11 = gx * stiff + k["adev"], gy * stiff, gz * stiff + k["ahyd"]
                det = a00 * a11 - a01 * a01
                bx, by = -(c_dev + rx * k["relax"]), -(c_hyd + ry * k["relax"])
                ok = (det >= 1e-20) & (sum(ws) > 0)
                safe = torch.where(ok, det, torch.ones_like(det))
                lx = torch.where(ok, (a11 * bx - a01 * by) / safe, torch.zeros_like(det))
                ly = torch.where(ok, (a00 * by - a01 * bx) / safe, torch.zeros_like(det))
                for v, a, x, y in zip(tet, ws, d, h):
                    p[v] = p[v] + (x * lx[:, None] + y * ly[:, None]) * a[:, None]
        if self.limited:
            on = k["stretch"] > 1
            for _ in range(2):
                for a in range(8):
                    for b in range(a + 1, 8):
                        delta = p[b] - p[a]
                        length = delta.norm(dim=1)
                        most = math.sqrt(bin(a ^ b).count("1")) * k["h"] * k["stretch"]
                        weight = w[a] + w[b]
                        go = on & (length > most) & (weight > 0)
                        f = torch.where(go, (length - most) / (length * weight).clamp_min(1e-300),
                                        torch.zeros_like(length))
                        p[a] = p[a] + delta * (f * w[a])[:, None]
                        p[b] = p[b] - delta * (f * w[b])[:, None]
        self.pos[ids] = torch.stack(p)

    def collide(self):
        """Corrections averaged over the overlapping records of the 27 buckets around each record (at most 32
        records of a bucket take part)."""
        node = self.rec
        body = self.body_of[node]
        P, moved, w = self.pos[node], self.pos[node] - self.prev[node], self.w[node]
        origin, size, dims, base = (g[body] for g in self.grid)
        c = torch.floor((P - origin) / size[:, None]).long()
        c = torch.minimum(c.clamp_min(0), dims - 1)
        linear = lambda q: base + q[:, 0] + dims[:, 0] * (q[:, 1] + dims[:, 1] * q[:, 2])  # noqa: E731
        key, order = torch.sort(linear(c), stable=True)
        buckets, held = torch.unique_consecutive(key, return_counts=True)
        start = torch.cumsum(held, 0) - held
        seen = held.clamp_max(32)
        total = torch.zeros_like(P)
        hits = torch.zeros(P.shape[0], dtype=P.dtype, device=P.device)
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    q = c + torch.tensor([dx, dy, dz], device=c.device)
                    inside = ((q >= 0) & (q < dims)).all(1)
                    near = linear(q)
                    at = torch.searchsorted(buckets, near).clamp_max(buckets.numel() - 1)
                    n = torch.where(inside & (buckets[at] == near), seen[at], torch.zeros_like(at))
                    me = torch.repeat_interleave(torch.arange(P.shape[0], device=P.device), n)
                    if not me.numel():
                        continue
                    k = torch.arange(me.numel(), device=P.device) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
                    mate = order[start[at][me] + k]
                    apart = ((self.coord[me] - self.coord[mate]).abs() > 1).any(1)
                    other = body[me] != body[mate]
                    ok = (other & (not self.isolated)) | (~other & apart & self.self_contact)
                    d = P[me] - P[mate]
                    reach = self.radius[me] + self.radius[mate]
                    ok &= ((d * d).sum(1) < reach * reach) & (w[me] + w[mate] > 0)
                    me, mate, d, reach = me[ok], mate[ok], d[ok], reach[ok]
                    share = w[me] / (w[me] + w[mate])
                    dist = d.norm(dim=1)
                    up = torch.zeros_like(d)
                    up[:, 1] = torch.where(node[me] < node[mate], 1.0, -1.0).to(d.dtype)
                    normal = torch.where((dist > 1e-9)[:, None], d / dist.clamp_min(1e-300)[:, None], up)
                    depth = reach - dist
                    slide = moved[me] - moved[mate]
                    tangent = slide - normal * (slide * normal).sum(1, keepdim=True)
                    slid = tangent.norm(dim=1)
                    mu = torch.minimum(self.friction[body[me]], self.friction[body[mate]])
                    grip = torch.where(slid > 1e-9, (mu * depth / slid.clamp_min(1e-300)).clamp_max(1.0),
                                       torch.zeros_like(slid))
                    fix = normal * (depth * share)[:, None] - tangent * (share * grip)[:, None]
                    total.index_add_(0, me, fix)
                    hits.index_add_(0, me, torch.ones_like(depth))
        self.pos[node] = P + torch.where((hits > 0)[:, None], total / hits.clamp_min(1)[:, None],
                                         torch.zeros_like(total))

    def plane(self, p, axis, sign, depth, friction):
        normal = torch.zeros(3, dtype=p.dtype, device=p.device)
        normal[axis] = sign
        q = p + normal * depth[:, None]
        delta = q - self.prev
        tangent = delta - normal * (delta @ normal)[:, None]
        length = tangent.norm(dim=1)
        grip = torch.where(length > 1e-9, (friction * depth / length.clamp_min(1e-300)).clamp_max(1.0),
                           torch.zeros_like(length))
        return torch.where((depth > 0)[:, None], q - tangent * grip[:, None], p)

    def substep(self, live=None, drive=None):
        """One substep of the live nodes (all by default); drive: (nodes, goals, velocity, law)."""
        dt = self.dt
        saved = (self.pos.clone(), self.prev.clone(), self.vel.clone()) if live is not None else None
        go = self.active[:, None]
        g = torch.tensor([0.0, -9.81, 0.0], dtype=self.pos.dtype, device=self.dev)
        v = self.vel + g * dt
        self.prev = torch.where(go, self.pos, self.prev)
        self.vel = torch.where(go, v, self.vel)
        self.pos = torch.where(go, self.pos + v * dt, self.pos)
        if drive is not None:
            nodes, goal, velocity, law = drive
            here = self.pos[nodes]
            if law == "hard":
                step, to_goal = velocity * dt, goal - here
                short = (step * step).sum(-1, keepdim=True) >= (to_goal * to_goal).sum(-1, keepdim=True)
                there = here + torch.where(short, to_goal, step)
                self.prev[nodes], self.pos[nodes], self.vel[nodes] = here, there, (there - here) / dt
            else:
                self.pos[nodes] = here + (goal - here) * (dt * dt / (dt * dt + 0.05 * 0.05))
        for _ in range(self.iterations):
            for ids, k in self.colours:
                self.project(ids, k, False)
        if self.limited:
            for _ in range(3):
                for ids, k in self.colours:
                    self.project(ids, k, True)
        if self.contact:
            self.collide()
        friction = self.friction[self.body_of]
        mn, mx = self.tank
        p = self.pos
        p = self.plane(p, 1, 1.0, mn[1] - p[:, 1], friction)
        p = self.plane(p, 0, 1.0, mn[0] - p[:, 0], friction)
        p = self.plane(p, 0, -1.0, p[:, 0] - mx[0], friction)
        p = self.plane(p, 2, 1.0, mn[2] - p[:, 2], friction)
        p = self.plane(p, 2, -1.0, p[:, 2] - mx[2], friction)
        go = self.active[:, None]
        self.vel = torch.where(go, (p - self.prev) / dt * self.damp[self.body_of][:, None], self.vel)
        self.pos = torch.where(go, p, self.pos)
        if live is not None:
            keep = ~live[:, None]
            self.pos, self.prev, self.vel = (torch.where(keep, a, b)
                                             for a, b in zip(saved, (self.pos, self.prev, self.vel)))

    def start(self, pos, vel):
        self.pos = torch.as_tensor(pos, dtype=torch.float64, device=self.dev).clone()
        self.vel = torch.as_tensor(vel, dtype=torch.float64, device=self.dev).clone()
        self.prev = self.pos.clone()

    def hard_hold(self, nodes):
        self.w[nodes] = 0.0
        self.active[nodes] = False


def _quad_out(t):
    return torch.cat([t, torch.zeros_like(t[:, :1])], 1).cpu()


def _exact_frame(case, seed):
    s = _scene(case, seed)
    x = _Exact(s["bodies"], s["tank"], s["step"], s["iterations"], s["contact"], s["self_contact"], False)
    x.start(s["pos"], s["vel"])
    drive = None
    if s["hold"]:
        nodes, offsets, place, target = s["hold"]
        at = torch.as_tensor(nodes.astype(np.int64), device=x.dev)
        vec = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=x.dev)  # noqa: E731
        velocity = (vec(target) - vec(place)) / (s["steps"] * s["step"])
        drive = (at, vec(target) + vec(offsets), velocity, s["law"])
        if s["law"] == "hard":
            x.hard_hold(at)
    for _ in range(s["steps"]):
        x.substep(drive=drive)
    return {"pos": _quad_out(x.pos), "vel": _quad_out(x.vel)}


def _exact_splats(case, seed):
    s, means, quats, scales = _splat_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    D = lambda a: torch.as_tensor(a, device=dev).double()  # noqa: E731
    b, n = s["bodies"][0], case["n"]
    grid = (D(means) - torch.tensor(b["origin"], dtype=torch.float32).to(dev).double()) / float(np.float32(H))
    cell = torch.floor(grid).clamp(0, n - 1)
    local, at = grid - cell, cell.long()
    pos = D(s["pos"])
    position = torch.zeros_like(grid)
    F = torch.zeros(grid.shape[0], 3, 3, dtype=torch.float64, device=dev)
    for c in range(8):
        bit = torch.tensor([c & 1, c >> 1 & 1, c >> 2], device=dev)
        f = torch.where(bit.bool(), local, 1 - local)
        sign = 2.0 * bit - 1.0
        q = at + bit
        p = pos[q[:, 0] + (n + 1) * (q[:, 1] + (n + 1) * q[:, 2])]
        position += p * f.prod(1, keepdim=True)
        grad = torch.stack([sign[0] * f[:, 1] * f[:, 2], sign[1] * f[:, 0] * f[:, 2], sign[2] * f[:, 0] * f[:, 1]], 1)
        F += p[:, :, None] * grad[:, None, :] / float(np.float32(H))
    x, y, z, w = D(quats).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
    A = F @ R * D(scales)[:, None, :]
    S = A @ A.transpose(1, 2)
    cov = torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 0, 2], S[:, 1, 1], S[:, 1, 2], S[:, 2, 2]], 1)
    out = {"means": position.cpu(), "cov": cov.cpu(), "order": None}
    if case["axes"]:  # an axis pair is the same turned about: no single answer
        out.update(rotation=None, scale=None)
    return out


def _bezier(c, t):
    u = 1 - t
    p = u ** 3 * c[0] + 3 * u * u * t * c[1] + 3 * u * t * t * c[2] + t ** 3 * c[3]
    return p, 3 * u * u * (c[1] - c[0]) + 6 * u * t * (c[2] - c[1]) + 3 * t * t * (c[3] - c[2])


def _exact_serve(case, seed):
    bodies, frames, drags, tank = _serve_inputs(case, seed)
    x = _Exact(bodies, tank, 1 / 600, 1, True, True, True)
    first = np.concatenate([[0], np.cumsum([_node_total([b]) for b in bodies])]).astype(np.int64)
    x.start(np.concatenate([_rest(b) for b in bodies]).astype(np.float32), np.zeros((int(first[-1]), 3)))
    held = [(q, int(first[q]) + d[0], d[1].astype(np.float64), d[2]) for q, d in enumerate(drags) if d is not None]
    nodes = torch.tensor([n for _, n, _, _ in held], dtype=torch.int64, device=x.dev)
    x.hard_hold(nodes)
    t = [0.0] * len(held)
    place = [c[0] for _, _, c, _ in held]
    frame_dt = 10 / 600
    for f in range(max(frames)):
        live = torch.as_tensor(np.repeat([f < n for n in frames], np.diff(first)), device=x.dev)
        goal, velocity = [], []
        for i, (q, _, c, speed) in enumerate(held):
            t[i] = min(1.0, t[i] + speed * frame_dt / max(float(np.linalg.norm(_bezier(c, t[i])[1])), 1e-9))
            p = _bezier(c, t[i])[0]
            goal.append(p)
            velocity.append((p - place[i]) / frame_dt)
            place[i] = p
        D = lambda a: torch.as_tensor(np.array(a), device=x.dev).view(-1, 3)  # noqa: E731
        for _ in range(10):
            x.substep(live, (nodes, D(goal), D(velocity), "hard"))
    return _quad_out(x.pos)


def exact(case, seed):
    """What run() returns in 64 bits by plain tensor operations; None for whole numbers (a permutation, a grid)."""
    if case["kind"] == "frame":
        return _exact_frame(case, seed)
    if case["kind"] == "splats":
        return _exact_splats(case, seed)
    if case["kind"] == "serve":
        return _exact_serve(case, seed)
    return None
