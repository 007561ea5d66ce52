"""Calls that are refused leave what was there before them as it was."""
import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu


def refused_table(vxp, n, statics, why):
    """A table of n bodies, the first of them static, that set_bodies refuses."""
    b = np.zeros(n, dtype=vxp.abi.BODY_DTYPE)
    b["id"] = np.arange(1000, 1000 + n)
    b["body_type"] = vxp.abi.BODY_DYNAMIC
    b["body_type"][:statics] = vxp.abi.BODY_STATIC
    b["rotation"][:, 3] = 1.0
    if why == "duplicate id":
        b["id"][-1] = b["id"][0]
    else:
        b["body_type"][-1] = 3
    return b


@pytest.mark.parametrize("why", ["duplicate id", "bad body_type"])
@pytest.mark.parametrize("n", [29, 200, 300])
@pytest.mark.parametrize("mode", [0, 1])
def test_refused_bodies_leave_the_world(vxp, n, why, mode):
    """27 boxes resting on two static bodies; then a table is refused that is
    larger than any before it (within the body capacity of 256 and past it),
    with more static bodies: the bodies read back as they were, and the next
    steps are the oracle's."""
    sc = vxp.scenes.config2(mass_fn=O.mass_fn, n_side=3, seed=8)
    dt = np.float32(sc.dt)
    settled = O.OracleWorld(substeps=8)
    settled.load_scene(sc)
    for _ in range(180):
        settled.step(dt)
    assert {1, 2} & {int(m["body_a_id"]) for m in settled.manifolds()}
    sc.bodies = settled.get_bodies()
    settled.close()
    r = O.OracleWorld(substeps=8)
    r.load_scene(sc)
    g = vxp.VoxelPhysicsSystem(substeps=8)
    g.load_scene(sc)
    g.set_launch_mode(mode)
    for s in range(3):
        with pytest.raises(vxp.system.VxpError) as e:
            g.set_bodies(refused_table(vxp, n, 9, why))
        assert e.value.code == vxp.abi.VXP_ERR_ARG and why.split()[0] in str(e.value)
        assert g.get_bodies().tobytes() == r.get_bodies().tobytes(), f"step {s}: the refused table was felt"
        pairs = r.pairs()
        assert g.pairs().tobytes() == pairs.tobytes(), f"step {s}"
        g.step(dt, pairs)
        r.step(dt, pairs)
        assert g.get_bodies().tobytes() == r.get_bodies().tobytes(), f"step {s}: bodies differ"
    # an accepted table in another order than its ids'
    b = r.get_bodies()[::-1].copy()
    g.set_bodies(b)
    r.set_bodies(b)
    for s in range(3):
        g.step(dt)
        r.step(dt)
        assert g.get_bodies().tobytes() == r.get_bodies().tobytes(), f"reversed table, step {s}: bodies differ"
    g.close()
    r.close()


@pytest.mark.parametrize("why", ["duplicate id", "bad body_type"])
@pytest.mark.parametrize("n", [20, 400])
def test_refused_batch_world_leaves_the_slot(vxp, n, why):
    """A table refused for a stepped slot of a batch, smaller and larger than
    the slot's buffers: the slot's world and its neighbour's step on as the
    oracle's do; refused for an empty slot, the slot stays empty."""
    dt = np.float32(1 / 60)
    rng = np.random.default_rng(12)
    worlds = [vxp.scenes.world_for_batch(rng, k, O.mass_fn) for k in (30, 12)]
    b = vxp.VoxelWorldBatch(3, substeps=4)
    refs = []
    for i, sc in enumerate(worlds):
        b.load_scene(i, sc, collider_offset=1000 * (i + 1))
        r = O.OracleWorld(substeps=4)
        r.load_scene(sc)
        refs.append(r)
    touching = 0
    for s in range(130):
        if s in (110, 120):
            for w in (0, 2):
                with pytest.raises(vxp.system.VxpError) as e:
                    b.set_world(w, refused_table(vxp, n, 9, why))
                assert e.value.code == vxp.abi.VXP_ERR_ARG and why.split()[0] in str(e.value)
            assert b.lib.vxp_batch_world_bytes(b.b, 2) == 0
        b.step(dt)
        b.synchronize()
        for r in refs:
            r.step(dt)
        touching += s >= 110 and len(refs[0].manifolds()) > 0
        if s >= 109:
            for i, r in enumerate(refs):
                got, want = b.get_world(i), r.get_bodies()
                for f in got.dtype.names:
                    if f != "collider_id":
                        assert got[f].tobytes() == want[f].tobytes(), f"step {s}, world {i}: {f} differs"
    assert touching >= 10, "the refusals fell into free flight"
    b.close()


@pytest.mark.parametrize("fresh", [False, True])
def test_batch_world_without_memory_leaves_an_empty_slot(vxp, fresh):
    """A world whose pair buffers no GPU holds (2^28 pairs, about 400 GB), for
    a stepped slot and for one that never held a world: the slot is empty
    afterwards and out of the launches, its neighbour steps on as the oracle's
    world does, and the slot takes the next world."""
    dt = np.float32(1 / 60)
    rng = np.random.default_rng(13)
    worlds = [vxp.scenes.world_for_batch(rng, k, O.mass_fn) for k in (12, 25)]
    tables = []
    b = vxp.VoxelWorldBatch(2, substeps=4)
    for i, sc in enumerate(worlds):
        for c in sc.colliders:
            b.add_collider(1000 * i + c.id, c.voxel_size, c.bricks)
        t = sc.bodies.copy()
        t["collider_id"] += 1000 * i
        tables.append(t)
    refs = [O.OracleWorld(substeps=4) for _ in worlds]
    for r, sc in zip(refs, worlds):
        r.load_scene(sc)

    def check(i):
        got, want = b.get_world(i), refs[i].get_bodies()
        for f in got.dtype.names:
            if f != "collider_id":
                assert got[f].tobytes() == want[f].tobytes(), f"world {i}: {f} differs"

    b.set_world(1, tables[1])
    if not fresh:
        b.set_world(0, tables[0])
    for _ in range(90):
        b.step(dt)
        refs[1].step(dt)
    b.synchronize()
    with pytest.raises(vxp.system.VxpError) as e:
        b.set_world(0, tables[0], pair_capacity=1 << 28)
    assert e.value.code == vxp.abi.VXP_ERR_OOM
    assert b.lib.vxp_batch_world_bytes(b.b, 0) == 0
    out = np.zeros(len(tables[0]), dtype=vxp.abi.BODY_DTYPE)
    assert b.lib.vxp_batch_world_get(b.b, 0, vxp.abi.ptr(out), len(out)) != 0
    b.times()  # the last step's launch table is gone with the slot
    check(1)
    for _ in range(10):
        b.step(dt)
        refs[1].step(dt)
    b.synchronize()
    check(1)
    b.set_world(0, tables[0])
    for _ in range(70):
        b.step(dt)
        for r in refs:
            r.step(dt)
    b.synchronize()
    b.times()
    check(0)
    check(1)
    b.close()


def test_times_after_a_world_is_released(vxp):
    """The per-world times of the last step outlive the buffers of a world
    released since (the launch table that names them does not)."""
    rng = np.random.default_rng(14)
    b = vxp.VoxelWorldBatch(3, substeps=4)
    for i, sc in enumerate(vxp.scenes.world_for_batch(rng, k, O.mass_fn) for k in (12, 20, 16)):
        b.load_scene(i, sc, collider_offset=1000 * (i + 1))
    b.step(np.float32(1 / 60), 3)
    b.release_world(1)
    total, per = b.times()
    assert total > 0 and per[0] > 0 and per[2] > 0 and per[1] == 0
    b.synchronize()
    b.step(np.float32(1 / 60), 1)
    b.synchronize()
    _, per = b.times()
    assert per[0] > 0 and per[2] > 0 and per[1] == 0
    b.close()
