"""Bulk state export (vxp_bodies_export, vxp_batch_world_export): the
per-handle getters of the reference (getPosition, getRotation,
getLinearVelocity, getAngularVelocity, getWorldAABB, isSleeping;
src/system.zig:963-1017) for a range of bodies in one call, into host arrays
or into device memory that a CUDA consumer reads on its own stream."""
import ctypes

import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu


def _stepped(vxp, steps=40):
    sc = vxp.scenes.config1(mass_fn=O.mass_fn, n_side=3, seed=4)
    g = vxp.VoxelPhysicsSystem()
    g.load_scene(sc)
    r = O.OracleWorld()
    r.load_scene(sc)
    dt = np.float32(sc.dt)
    for _ in range(steps):
        p = r.pairs()
        g.step(dt, p)
        r.step(dt, p)
    assert g.get_bodies().tobytes() == r.get_bodies().tobytes()
    return g, r


def test_export_matches_bodies_and_oracle_aabbs(vxp):
    g, r = _stepped(vxp)
    b = g.get_bodies()
    e = g.export_state()
    assert e["position"].tobytes() == np.ascontiguousarray(b["position"]).tobytes()
    assert e["rotation"].tobytes() == np.ascontiguousarray(b["rotation"]).tobytes()
    assert e["linear_velocity"].tobytes() == np.ascontiguousarray(b["linear_velocity"]).tobytes()
    assert e["angular_velocity"].tobytes() == np.ascontiguousarray(b["angular_velocity"]).tobytes()
    assert (e["sleeping"] == b["is_sleeping"]).all()
    mn, mx = r.world_aabbs()
    assert e["aabb_min"].tobytes() == mn.tobytes()
    assert e["aabb_max"].tobytes() == mx.tobytes()
    # a range, some fields only
    part = g.export_state(fields=("rotation", "aabb_max"), first=5, n=7)
    assert set(part) == {"rotation", "aabb_max"}
    assert part["rotation"].tobytes() == e["rotation"][5:12].tobytes()
    assert part["aabb_max"].tobytes() == mx[5:12].tobytes()
    g.close()
    r.close()


def test_export_into_device_memory_for_a_consumer_stream(vxp):
    import torch

    g, r = _stepped(vxp, steps=25)
    n = g.n_bodies
    dev = {"position": torch.full((n, 3), -1.0, device="cuda:0"), "aabb_min": torch.full((n, 3), -1.0, device="cuda:0"),
           "sleeping": torch.full((n,), 7, dtype=torch.uint8, device="cuda:0")}
    s = torch.cuda.Stream(device="cuda:0")
    g.export_state_to_device({k: v.data_ptr() for k, v in dev.items()}, consumer_stream=s.cuda_stream)
    with torch.cuda.stream(s):
        got = {k: v.clone() for k, v in dev.items()}  # the consumer, ordered after the export
    s.synchronize()
    want = g.export_state(fields=("position", "aabb_min", "sleeping"))
    for k in got:
        assert got[k].cpu().numpy().tobytes() == want[k].tobytes(), k
    g.close()
    r.close()


def test_export_rejects_bad_arguments(vxp):
    g, r = _stepped(vxp, steps=2)
    n = g.n_bodies
    host = np.zeros((n, 3), dtype=np.float32)
    view = vxp.abi.StateView()
    view.position = host.ctypes.data
    # host memory passed as device memory: rejected before any launch
    assert g.lib.vxp_bodies_export(g.ctx, ctypes.byref(view), 0, n, 1, None) == vxp.abi.VXP_ERR_ARG
    # a range past the bodies
    assert g.lib.vxp_bodies_export(g.ctx, ctypes.byref(view), 1, n, 0, None) == vxp.abi.VXP_ERR_ARG
    assert g.lib.vxp_bodies_export(g.ctx, None, 0, n, 0, None) == vxp.abi.VXP_ERR_ARG
    # the context is still usable
    assert g.export_state(fields=("position",))["position"].shape == (n, 3)
    g.close()
    r.close()


def test_batch_world_export(vxp):
    sc = [vxp.scenes.config1(mass_fn=O.mass_fn, n_side=2, seed=s) for s in (1, 2)]
    bt = vxp.VoxelWorldBatch(2)
    for w, scene in enumerate(sc):
        bt.load_scene(w, scene, collider_offset=1000 * w)
    bt.step(np.float32(sc[0].dt), 20)
    for w in range(2):
        b = bt.get_world(w)
        e = bt.export_world(w, fields=("position", "angular_velocity", "sleeping"))
        assert e["position"].tobytes() == np.ascontiguousarray(b["position"]).tobytes()
        assert e["angular_velocity"].tobytes() == np.ascontiguousarray(b["angular_velocity"]).tobytes()
        assert (e["sleeping"] == b["is_sleeping"]).all()
    bt.close()


@pytest.mark.parametrize("fields,n", [([], None), (None, 0), (None, 500), (None, None)])
def test_export_reports_a_pending_error(vxp, fields, n):
    """A step left undone for want of pair buffers (200 bodies in one place) is
    reported by the next export to host memory, also one without a field, one
    of no bodies and one past the bodies; the report clears it."""
    b = np.zeros(200, dtype=vxp.abi.BODY_DTYPE)
    b["id"] = np.arange(1, 201)
    b["body_type"] = vxp.abi.BODY_DYNAMIC
    b["inv_mass"] = 1.0
    b["rotation"][:, 3] = 1.0
    g = vxp.VoxelPhysicsSystem(max_pairs=1024)
    g.add_collider(0, 0.1, vxp.scenes.readme_box(8))
    g.set_bodies(b)
    g.step(np.float32(1 / 60))
    with pytest.raises(vxp.system.VxpError) as e:
        g.export_state(fields, n=n)
    assert e.value.code == vxp.abi.VXP_ERR_CAP
    assert g.export_state(["position"])["position"].tobytes() == b["position"].tobytes()
    g.close()


def test_large_tables_first_and_later(vxp):
    """Body tables of more than 1 MB (9000 bodies), which the first calls of a
    context copy to and from pageable memory and later ones through pinned
    memory: every byte comes back, in both directions and from an export."""
    rng = np.random.default_rng(18)
    n = 9000
    g = vxp.VoxelPhysicsSystem(max_bodies=n)
    g.add_collider(0, 0.1, vxp.scenes.readme_box(8))
    for turn in range(4):
        b = np.zeros(n, dtype=vxp.abi.BODY_DTYPE)
        b["id"] = rng.permutation(n) + 1
        b["body_type"] = rng.integers(0, 3, size=n)
        b["inv_mass"] = rng.uniform(0.1, 1.0, size=n)
        b["inv_inertia_local"][:, [0, 4, 8]] = rng.uniform(0.1, 1.0, size=(n, 3))
        b["position"] = rng.uniform(-500, 500, size=(n, 3))
        b["linear_velocity"] = rng.uniform(-1, 1, size=(n, 3))
        b["rotation"] = vxp.scenes.shoemake_quat(rng, n)
        g.set_bodies(b)
        if turn != 1:
            assert g.get_bodies().tobytes() == b.tobytes(), f"turn {turn}"
        for _ in range(2):
            out = g.export_state()
            for f in ("position", "rotation", "linear_velocity"):
                assert out[f].tobytes() == np.ascontiguousarray(b[f]).tobytes(), f"turn {turn}: {f}"
    g.close()
