"""Cells of stiff bodies near rest, where the two constraints' gradients are
parallel but for roundings and the 2 x 2 system's determinant comes out
negative: the multipliers are then 0 (xpbdCouple.wgsl:58-71), in the branch-free
arithmetic (csrc/step_device.cuh projectTetInRange) as in the IEEE one. Through
the row pass, the one-launch frame of a small scene, the ticks of a server and
its session kernel, against the oracle, bit for bit (such cells can blow up: where
the oracle has NaN the device has it too)."""
import numpy as np
import pytest

F = np.float32
KUHN = ((0, 1, 3, 7), (0, 5, 1, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 4, 5, 7), (0, 6, 4, 7))
# Young's modulus, Poisson's ratio, density, cell edge, step
ALUMINIUM = (7e10, 0.33, 2700.0, 0.016, 1 / 60)
STEEL = (2e11, 0.3, 7800.0, 0.005, 1 / 60)
LIGHT = (2e11, 0.3, 1000.0, 0.016, 1 / 60)
STIFF = pytest.mark.parametrize("stiff", [ALUMINIUM, STEEL, LIGHT], ids=["aluminium", "steel", "light"])
INF = float("inf")


def box(dims, stiff, seed=3):
    """A box, and its nodes 1e-5 of a cell off rest."""
    import vsim.scenes as sc

    youngs, poisson, density, h, _ = stiff
    mat = dict(sc.DEFAULT_MATERIAL, youngs_modulus=youngs, poisson_ratio=poisson, density=density)
    body = sc.Body(dims, (0.0, 0.0, 0.0), h, np.ones(int(np.prod(dims)), np.uint8), mat)
    rest = sc.rest_positions(body).astype(np.float64)
    off = rest + 1e-5 * h * np.random.default_rng(seed).standard_normal(rest.shape)
    return body, np.concatenate([off, np.zeros((len(off), 1))], 1).astype(F)


def determinants(body, pos, step):
    """The determinants of every cell's six 2 x 2 systems at `pos`, in float32
    (inner nodes' masses; not rounding for rounding the kernels')."""
    nx, ny, nz = body.node_dims
    grid = pos[:, :3].reshape(nz, ny, nx, 3)
    corner = [grid[k >> 2:nz - 1 + (k >> 2), k >> 1 & 1:ny - 1 + (k >> 1 & 1), k & 1:nx - 1 + (k & 1)].reshape(-1, 3)
              for k in range(8)]
    m, h = body.material, body.h
    mu = m["youngs_modulus"] / (2 * (1 + m["poisson_ratio"]))
    lame = 2 * mu * m["poisson_ratio"] / (1 - 2 * m["poisson_ratio"])
    alpha = [F(1 / (c * h ** 3 / 6)) / F(step) ** 2 for c in (mu, lame)]
    stiffened = F(1) + F(m["relaxation"]) / F(step)
    weight, s = F(1 / (m["density"] * h ** 3)), F(1) / F(h)
    out = []
    for tet in KUHN:
        shape = [[(tet[c] >> r & 1) - (tet[0] >> r & 1) for c in (1, 2, 3)] for r in range(3)]
        inverse = np.rint(np.linalg.inv(shape)).astype(F) * s
        f = np.stack([corner[tet[c]] - corner[tet[0]] for c in (1, 2, 3)], 2) @ inverse
        norm = np.sqrt((f * f).sum((1, 2), dtype=F))[:, None, None]
        cofactor = np.stack([np.cross(f[:, :, (c + 1) % 3], f[:, :, (c + 2) % 3]) for c in range(3)], 2)
        dev, hyd = ((g, -g.sum(2, dtype=F)[:, :, None]) for g in (f / norm @ inverse.T, cofactor @ inverse.T))
        dev, hyd = np.concatenate(dev, 2), np.concatenate(hyd, 2)
        xx, xy, yy = (weight * (a * b).sum((1, 2), dtype=F) for a, b in ((dev, dev), (dev, hyd), (hyd, hyd)))
        a01 = xy * stiffened
        out.append(((xx * stiffened + alpha[0]).astype(np.float64) * (yy * stiffened + alpha[1]) - a01 * a01).astype(F))
    return np.concatenate(out)


@STIFF
def test_the_inputs_have_negative_determinants(stiff):
    import vsim.scenes as sc

    body, pos = box((20, 7, 6), stiff)
    det = determinants(body, pos, stiff[-1])
    assert np.mean(det < 0) > 0.05 and np.mean(det > 1) > 0.3
    body, pos = box((20, 7, 6), (1.2e5, 0.4, 1000.0, sc.H, 1 / 600))
    assert (determinants(body, pos, 1 / 600) > 1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,launches", [((16, 4, 4), 1), ((70, 9, 8), None)], ids=["one launch", "row passes"])
@STIFF
def test_frames(vsimlib, gpu, stiff, dims, launches):
    import pyoracle
    import vsim.scenes as sc
    from vsim import Simulator

    body, pos = box(dims, stiff)
    scene = sc.Scene([body], ((-INF,) * 3, (INF,) * 3), step_duration=stiff[-1], substeps=3, contact=False)
    sim, orc = Simulator(scene), pyoracle.Oracle(scene, 32)
    rest = np.zeros_like(pos)
    sim.write_state(pos, pos, rest)
    orc.set_state(pos, pos, rest)
    assert (sim.frame_launches(3) == 1) == (launches == 1)
    for frame in range(3):
        sim.dispatch(3)
        orc.dispatch(3)
        for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
            assert np.array_equal(g, o, equal_nan=True), f"frame {frame}: {name}"
    sim.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("engine,block,cluster", [(0, 0, 0), (1, 1 << 30, 0), (1, 0, 1 << 30)],
                         ids=["ticks", "session blocks", "session clusters"])
@STIFF
def test_sessions(vsimlib, gpu, stiff, engine, block, cluster):
    import pyoracle
    import vsim.scenes as sc
    from vsim.server import Server

    made = [box(dims, stiff, seed) for seed, dims in enumerate([(12, 5, 4), (40, 3, 6)])]
    bodies = [b for b, _ in made]
    tank = ((-10.0,) * 3, (10.0,) * 3)
    server = Server(bodies, tank, step_duration=stiff[-1], substeps=4, self_contact=False)
    server.set_engine(engine, block, cluster)
    for q, (_, pos) in enumerate(made):
        server.write_state(q, pos, pos, np.zeros_like(pos))
    server.run(None, np.arange(2), np.array([2, 3]), np.zeros(2, int))
    for q, frames in enumerate((2, 3)):
        scene = sc.Scene([bodies[q]], tank, step_duration=stiff[-1], substeps=4, contact=True, isolated=True)
        orc = pyoracle.Oracle(scene, 32)
        orc.set_state(made[q][1], made[q][1], np.zeros_like(made[q][1]))
        for _ in range(frames):
            orc.dispatch(4)
        for name, g, o in zip(("pos", "prev", "vel"), server.read_state(q), orc.state()):
            assert np.array_equal(g, o, equal_nan=True), f"session {q}: {name}"
    server.destroy()
