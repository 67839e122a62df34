"""The incremental re-sort against the oracle: the step merges the few
spheres whose cell key changed into the previous slot order instead of
radix-sorting every key, and must give exactly the stable sort's order
(the oracle's), so positions, velocities, spins and the contact list stay
bit-identical.  Scenes are set moving so that the number of changed keys
per step ranges from 0 to about a third of all spheres, on both sides of
the knob's limit (the radix passes take over above it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def moving_scene(n, moved_per_step, seed):
    """Settling-box spheres with random velocities sized so that about
    `moved_per_step` keys change per step (a key changes when a centre
    crosses a cell face; z faces are twice as dense)."""
    from stardust_gb300 import scenes
    pos, vel, cfg, dt, phi = scenes.settling_rsa(n, box=scenes.scaled_box(n), seed=seed)
    pos = pos.copy()
    vel = vel.copy()
    rng = np.random.default_rng(seed)
    speed = moved_per_step / n * cfg.cell / (2.0 * dt)
    vel[:, :3] = (rng.standard_normal((n, 3)) * speed).astype(np.float32)
    return pos, vel, cfg, dt


@pytest.mark.parametrize("resort_max,moved", [(0, 200), (2, 200), (256, 200), (1024, 200), (1024, 0),
                                              (1024, 700), (512, 9000)])
def test_incremental_resort_bit_exact(sdlib, orc, resort_max, moved):
    from stardust_gb300 import _abi
    old = _abi.tune_get("resort_max")
    try:
        _abi.tune_set("resort_max", resort_max)
        n = 30_000
        pos, vel, cfg, dt = moving_scene(n, moved, seed=7)
        eng = sdlib.DEMEngine(cfg)
        eng.add_spheres(pos, vel)
        eng.prepare()
        steps = 12
        seen = []
        for _ in range(steps):
            eng.step(dt, 1)
            seen.append(eng.stats()["moved_keys"])
        eng.sync()
        assert eng.stats()["device_errors"] == 0
        if resort_max == 0:
            assert max(seen) == 0
        elif moved == 0:
            assert max(seen) <= 8
        else:
            assert 0.3 * moved < np.median(seen) < 3 * moved
        p = orc.params_checked(cfg, pos[:, 3], dt, eng.params())
        op, ov, ow = orc.run(p, pos, vel, orc.with_ids(np.zeros_like(pos), np.arange(n)), steps)
        assert np.array_equal(bits(eng.positions()), bits(orc.unsort(op, ow)))
        assert np.array_equal(bits(eng.velocities()), bits(orc.unsort(ov, ow)))
        assert np.array_equal(bits(eng.omegas())[:, :3], bits(orc.unsort(ow, ow))[:, :3])
        sp, sv, sw, _, cs = orc.prepare(p, eng.positions(), eng.velocities(),
                                        orc.with_ids(eng.omegas(), np.arange(n)))
        assert np.array_equal(eng.pairs(), orc.contact_pairs(p, sp, sw, cs))
        eng.close()
    finally:
        _abi.tune_set("resort_max", old)


def test_resort_mixes_with_radix_steps(sdlib, orc):
    """A strong gravity accelerates the spheres from rest, so the changed-key
    count grows from tens to about a thousand per step: the early steps
    re-sort incrementally, the later ones run the radix passes, and the
    state stays exact throughout."""
    from stardust_gb300 import _abi, scenes
    old = _abi.tune_get("resort_max")
    try:
        _abi.tune_set("resort_max", 256)
        n = 30_000
        pos, vel, cfg, dt, phi = scenes.settling_rsa(n, box=scenes.scaled_box(n), seed=3)
        cfg.gravity = (0.0, 0.0, -3e5)
        eng = sdlib.DEMEngine(cfg)
        eng.add_spheres(pos, vel)
        eng.prepare()
        seen = []
        for _ in range(30):
            eng.step(dt, 1)
            seen.append(eng.stats()["moved_keys"])
        assert min(seen) <= 256 < max(seen)
        p = orc.params_checked(cfg, pos[:, 3], dt, eng.params())
        op, ov, ow = orc.run(p, pos, vel, orc.with_ids(np.zeros_like(pos), np.arange(n)), 30)
        assert np.array_equal(bits(eng.positions()), bits(orc.unsort(op, ow)))
        assert np.array_equal(bits(eng.velocities()), bits(orc.unsort(ov, ow)))
        eng.close()
    finally:
        _abi.tune_set("resort_max", old)


def test_step_kernel_count(sdlib):
    """The plain radix step launches the contact stage, two passes and the
    reorder; with the re-sort the step adds the plan kernel (which orders the
    moved slots the contact stage listed) and the radix fallback's histogram
    (both return at once when not needed, like the passes), and the reorder
    becomes two in-place phases (gather the positions whose source moved,
    copy them back); stats report the graph's kernel nodes."""
    from stardust_gb300 import _abi
    old = _abi.tune_get("resort_max")
    counts = {}
    try:
        for rm in (0, 1024):
            _abi.tune_set("resort_max", rm)
            pos, vel, cfg, dt = moving_scene(20_000, 50, seed=1)
            eng = sdlib.DEMEngine(cfg)
            eng.add_spheres(pos, vel)
            eng.prepare()
            assert eng.stats()["step_kernels"] == 0
            eng.step(dt, 2)
            counts[rm] = eng.stats()["step_kernels"]
            eng.close()
    finally:
        _abi.tune_set("resort_max", old)
    assert counts[0] >= 4 and counts[1024] == counts[0] + 3


@pytest.mark.parametrize("n,resort_max,moved,items", [(30_000, 1024, 2, 16), (30_000, 1024, 200, 16),
                                                      (30_000, 1024, 700, 16), (30_000, 512, 9000, 16),
                                                      (30_000, 512, 9000, 8), (300, 1024, 20, 16), (300, 8, 200, 16),
                                                      (257, 1024, 100, 8), (150_000, 1024, 300, 16)])
def test_runs_of_steps_bit_exact(sdlib, orc, n, resort_max, moved, items):
    """Calls of several steps (one kernel after each contact stage, several
    steps to a graph): 0 to 9,000 changed keys per step, on both sides of the
    re-sort's limit, calls of 3, 8, 5, 13 and 1 steps one after the other."""
    from stardust_gb300 import _abi
    knobs = {"resort_max": resort_max, "sort_items": items}
    old = {k: _abi.tune_get(k) for k in knobs}
    try:
        for k, v in knobs.items():
            _abi.tune_set(k, v)
        pos, vel, cfg, dt = moving_scene(n, moved, seed=11)
        eng = sdlib.DEMEngine(cfg)
        eng.add_spheres(pos, vel)
        eng.prepare()
        kernels = []
        for steps in (3, 8, 5, 13, 1):
            eng.step(dt, steps)
            kernels.append(eng.stats()["step_kernels"])
        eng.sync()
        assert kernels[1] < kernels[0] and kernels[1] == kernels[2] == kernels[3] and kernels[4] == kernels[0]
        assert eng.stats()["device_errors"] == 0
        assert eng.stats()["steps"] == 30
        p = orc.params_checked(cfg, pos[:, 3], dt, eng.params())
        op, ov, ow = orc.run(p, pos, vel, orc.with_ids(np.zeros_like(pos), np.arange(n)), 30)
        assert np.array_equal(bits(eng.positions()), bits(orc.unsort(op, ow)))
        assert np.array_equal(bits(eng.velocities()), bits(orc.unsort(ov, ow)))
        assert np.array_equal(bits(eng.omegas())[:, :3], bits(orc.unsort(ow, ow))[:, :3])
        sp, sv, sw, _, cs = orc.prepare(p, eng.positions(), eng.velocities(),
                                        orc.with_ids(eng.omegas(), np.arange(n)))
        assert np.array_equal(eng.pairs(), orc.contact_pairs(p, sp, sw, cs))
        eng.close()
    finally:
        for k, v in old.items():
            _abi.tune_set(k, v)


def _state(eng):
    eng.sync()
    assert eng.stats()["device_errors"] == 0
    return [bits(eng.positions()), bits(eng.velocities()), bits(eng.omegas())[:, :3]]


@pytest.mark.parametrize("items,fix_blocks", [(8, 4), (16, 8)])
def test_run_fallback_with_more_tiles_than_blocks(sdlib, items, fix_blocks):
    """The step kernel's radix passes when its blocks take several tiles each
    (one block per SM and tiles of 2,048 keys: 196 tiles for 152 blocks; two
    and 4,096: 329 for 304), against the separate kernels of one-step calls."""
    from stardust_gb300 import _abi
    knobs = {"resort_max": 256, "sort_items": items, "fix_blocks": fix_blocks}
    old = {k: _abi.tune_get(k) for k in knobs}
    n = 400_000 if items == 8 else 1_345_000
    try:
        for k, v in knobs.items():
            _abi.tune_set(k, v)
        small, vel, cfg, dt = moving_scene(50_000, 900, seed=5)
        copies = -(-n // len(small))  # side by side along x, in one box
        width = float(cfg.box_hi[0])
        pos = np.concatenate([small + np.float32([c * width, 0, 0, 0]) for c in range(copies)])[:n]
        vel = np.concatenate([np.roll(vel, c, 0) for c in range(copies)])[:n]
        cfg.box_hi = (copies * width, *cfg.box_hi[1:])
        got = []
        for calls in ([9], [1] * 9):
            eng = sdlib.DEMEngine(cfg)
            eng.add_spheres(pos, vel)
            eng.prepare()
            moved = []
            for k in calls:
                eng.step(dt, k)
                moved.append(eng.stats()["moved_keys"])
            assert min(moved) > 256
            got.append(_state(eng))
            eng.close()
        assert all(np.array_equal(a, b) for a, b in zip(*got))
    finally:
        for k, v in old.items():
            _abi.tune_set(k, v)


def test_engines_in_runs_beside_each_other(sdlib):
    """Two engines in runs of steps from two threads, each step a kernel whose
    blocks meet: the states that each reaches alone."""
    import threading
    scenes = [moving_scene(60_000, 300, seed=3), moving_scene(20_000, 2_000, seed=4)]

    def run(k, out):
        pos, vel, cfg, dt = scenes[k]
        eng = sdlib.DEMEngine(cfg)
        eng.add_spheres(pos, vel)
        eng.prepare()
        for _ in range(10):
            eng.step(dt, 16)
        out[k] = _state(eng)
        eng.close()

    alone, beside = {}, {}
    for k in (0, 1):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, beside)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert all(np.array_equal(a, b) for a, b in zip(alone[k], beside[k]))
