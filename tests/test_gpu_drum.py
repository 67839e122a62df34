"""The rotating drum: spheres and rigid clumps against a triangle mesh that
turns about its axis, on the GPU against the CPU oracle (which tests every
triangle of the mesh, so the GPU's grid-pruned candidates must give the same
contacts), bit-exactly, including the mesh pose."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def small_drum(sd, omega=20.0, seed=0, engine=None):
    from stardust_gb300 import scenes
    d = scenes.drum_scene(n_spheres=650, radius=0.04, length=0.04, n_around=24, n_along=6, n_rings=3,
                          r_range=(0.002, 0.0028), omega=omega, seed=seed)
    if engine is not None:
        d["cfg"].collision_engine = engine
    eng = sd.DEMEngine(d["cfg"])
    scenes.add_drum_scene(eng, d)
    eng.prepare()
    eng.step(d["dt"], 0)  # builds the step (and the mesh's per-step rotation)
    eng.sync()
    return eng, d


def body_tables(d, n):
    body_of = np.full(n, -1, np.int32)
    r0 = np.zeros((n, 4), np.float32)
    first, count = [], []
    i = 0
    for b, (rel, *_r) in enumerate(d["clumps"]):
        first.append(i)
        count.append(len(rel))
        body_of[i:i + len(rel)] = b
        r0[i:i + len(rel), :3] = rel[:, :3]
        i += len(rel)
    return body_of, r0, np.array(first, np.uint32), np.array(count, np.uint32)


@pytest.mark.parametrize("steps", [1, 50, 400])
@pytest.mark.parametrize("engine", ["SHP", "SAP"])
def test_drum_bit_exact(sdlib, orc, steps, engine):
    """Either collision engine: sphere-triangle candidates from the mesh's
    static grid (SHP) or from sweep and prune along the drum axis (SAP)."""
    from stardust_gb300 import _abi
    eng, d = small_drum(sdlib, engine=getattr(_abi, "SD_ENGINE_" + engine))
    n = eng.n
    body_of, r0, first, count = body_tables(d, n)
    pos, vel, omg = eng.positions(), eng.velocities(), eng.omegas()
    ids = np.arange(n, dtype=np.uint32)
    omg.view(np.uint32)[:, 3] = np.where(body_of >= 0, ids | np.uint32(0x80000000), ids)
    b0 = {"pos": eng.bodies(_abi.SD_BODY_POSITION), "vel": eng.bodies(_abi.SD_BODY_VELOCITY),
          "quat": eng.bodies(_abi.SD_BODY_QUATERNION), "omega": eng.bodies(_abi.SD_BODY_OMEGA),
          "angmom": eng.bodies(_abi.SD_BODY_ANGMOM), "inv": eng.bodies(_abi.SD_BODY_INV_INERTIA),
          "first": first, "count": count}
    mesh = orc.make_mesh(d["tris"], d["patch"], d["centre"], eng.mesh_state())
    p = orc.params_checked(d["cfg"], pos[:, 3], d["dt"], eng.params())
    op, ov, ow, ob = orc.run_full(p, pos, vel, omg, steps, b0, r0, body_of, mesh)
    eng.step(d["dt"], steps)
    eng.sync()
    assert eng.stats()["device_errors"] == 0
    un = lambda a: orc.unsort(a, ow)
    assert np.array_equal(bits(eng.positions()), bits(un(op)))
    assert np.array_equal(bits(eng.velocities()), bits(un(ov)))
    assert np.array_equal(bits(eng.bodies(_abi.SD_BODY_QUATERNION)), bits(ob["quat"]))
    assert np.array_equal(bits(eng.mesh_state()), bits(np.array(mesh.state, np.float32)))
    eng.close()


def test_drum_keeps_spheres_inside_and_drags_the_bed(sdlib):
    """The bed stays inside the turning cylinder and picks up angular
    momentum about the drum axis in the drum's sense of rotation."""
    eng, d = small_drum(sdlib, omega=30.0, seed=1)
    eng.step(d["dt"], 20000)
    eng.sync()
    assert eng.stats()["device_errors"] == 0
    p = eng.positions().astype(np.float64)
    v = eng.velocities().astype(np.float64)
    c = np.array(d["centre"])
    rad = np.hypot(p[:, 1] - c[1], p[:, 2] - c[2])
    assert np.all(rad + p[:, 3] < 0.04 * 1.01)
    assert np.all(np.abs(p[:, 0] - c[0]) + p[:, 3] < 0.02 * 1.01)
    # angular momentum about the x axis through the centre: sense of +omega
    Lx = (v[:, 3] * ((p[:, 1] - c[1]) * v[:, 2] - (p[:, 2] - c[2]) * v[:, 1])).sum()
    assert Lx > 0
    eng.close()


@pytest.mark.parametrize("clumps", [0, 200])
@pytest.mark.parametrize("n", [800_000, 800_001])
def test_large_drum_register_budgets(sdlib, n, clumps):
    """Either side of the size from which the list kernel of a swept mesh is
    the one of five blocks per SM: with it, with four, and with the grid's
    candidates, the same bits."""
    from stardust_gb300 import _abi, scenes
    rng = np.random.default_rng(n)
    r, radius, length = 0.002, 0.25, 0.5
    a = 1.995 * r
    ys = np.arange(r, 2 * radius - r, a)
    sites = np.stack(np.meshgrid(ys, ys, np.arange(r, length - r, a), indexing="ij"), -1).reshape(-1, 3)[:, ::-1]
    sites = sites[((sites[:, 1:] - radius) ** 2).sum(1) < (radius - 0.99 * r) ** 2][:n - 3 * clumps]
    assert len(sites) == n - 3 * clumps
    tris, patch = scenes.drum_mesh(radius, length, 32, 8, 2, (0.5 * length, radius, radius))
    tet = np.array([[1, 1, 1, 0], [1, -1, -1, 0], [-1, 1, -1, 0], [-1, -1, 1, 0]]) * (0.3 * r) + (0, 0, 0, 0.5 * r)
    pos = np.concatenate([sites[clumps:], np.full((len(sites) - clumps, 1), r)], 1).astype(np.float32)
    vel = rng.uniform(-0.5, 0.5, pos.shape).astype(np.float32)
    vel[:, 3] = 1e-4
    got, old = [], _abi.tune_get("listed_blocks")
    try:
        for engine, blocks in ((_abi.SD_ENGINE_SAP, 5), (_abi.SD_ENGINE_SAP, 4), (_abi.SD_ENGINE_SHP, 5)):
            _abi.tune_set("listed_blocks", blocks)
            cfg = sdlib.EngineConfig(box_hi=(length, 2 * radius, 2 * radius), walls=0, cell=2.01 * r,
                                     pair_capacity=1 << 22, collision_engine=engine)
            eng = sdlib.DEMEngine(cfg)
            for c in sites[:clumps]:
                eng.add_clump(tet.astype(np.float32), 1e-4, tuple(c))
            eng.add_spheres(pos, vel)
            eng.add_mesh(tris, (0.5 * length, radius, radius), (1.0, 0.0, 0.0), 20.0, patch)
            eng.prepare()
            eng.step(2e-6, 5)
            eng.sync()
            st = eng.stats()
            assert st["device_errors"] == 0 and st["listed_steps"] > 0
            got.append([bits(eng.positions()), bits(eng.velocities()), bits(eng.omegas())])
            eng.close()
    finally:
        _abi.tune_set("listed_blocks", old)
    for other in got[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(got[0], other))
