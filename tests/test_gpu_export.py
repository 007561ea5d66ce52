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
    """Body tables of more than a pinned buffer holds (9000 bodies, over 1 MB), in
    a context's first calls and later: every byte comes back, in both directions
    and from an export."""
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


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4096, 4097, 6145])
def test_tables_at_the_edges_of_upload_buffers(vxp, n):
    """Tables of about one, two and three buffers of 2048 bodies, ids in another
    order than the table's, cubes resting on static ones on both sides of each
    edge: the table comes back, and the pair list and the steps (which read the
    id order and the list of static bodies) are the oracle's."""
    rng = np.random.default_rng(n)
    b = np.zeros(n, dtype=vxp.abi.BODY_DTYPE)
    b["id"] = rng.permutation(n) + 1
    b["body_type"] = vxp.abi.BODY_DYNAMIC
    b["inv_mass"] = 1.0
    b["inv_inertia_local"][:, [0, 4, 8]] = 1.0
    b["friction"] = 0.5
    b["rotation"][:, 3] = 1.0
    b["position"] = np.stack(np.meshgrid(*[np.arange(19)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n] * 3.0
    edges = sorted({i for e in range(0, n + 1, 2048) for i in (e - 1, e) if 0 <= i < n} | {n - 1})
    for i in edges:
        b["body_type"][i] = vxp.abi.BODY_STATIC
        b["inv_mass"][i] = 0.0
        on = (i + n // 2) % n
        if on in edges:
            on = (on + 7) % n
        b["position"][on] = b["position"][i] + np.array([0.1, 0.78, 0.05], dtype=np.float32)
    g = vxp.VoxelPhysicsSystem(substeps=4, max_bodies=n)
    r = O.OracleWorld(substeps=4)
    for w in (g, r):
        w.add_collider(0, 0.1, vxp.scenes.readme_box(8))
    dt = np.float32(1 / 60)
    for turn in range(2):
        for w in (g, r):
            w.set_bodies(b)
        assert g.get_bodies().tobytes() == b.tobytes()
        for s in range(2):
            pairs = r.pairs()
            assert g.pairs().tobytes() == pairs.tobytes()
            g.step(dt)
            r.step(dt, pairs)
            assert len(r.manifolds()) >= len(edges) // 2
            assert g.manifolds().tobytes() == r.manifolds().tobytes()
            assert g.get_bodies().tobytes() == r.get_bodies().tobytes()
        b = b[::-1].copy()
    g.close()
    r.close()


@pytest.mark.parametrize("n", [6800, 13600, 13625, 27500])
def test_exports_of_several_pinned_buffers(vxp, n):
    """Exports of half a megabyte to two, through a buffer of one, every field and some, whole
    and of a range: the values set."""
    rng = np.random.default_rng(n)
    b = np.zeros(n, dtype=vxp.abi.BODY_DTYPE)
    b["id"] = np.arange(1, n + 1)
    b["body_type"] = vxp.abi.BODY_DYNAMIC
    b["position"] = rng.uniform(-500, 500, size=(n, 3))
    b["rotation"] = vxp.scenes.shoemake_quat(rng, n)
    b["linear_velocity"] = rng.uniform(-1, 1, size=(n, 3))
    b["angular_velocity"] = rng.uniform(-1, 1, size=(n, 3))
    b["is_sleeping"] = rng.integers(0, 2, size=n)
    g = vxp.VoxelPhysicsSystem(max_bodies=n)
    g.set_bodies(b)  # no collider: a body's box is its position
    for fields in (None, ["rotation", "sleeping"], ["position", "aabb_max", "angular_velocity"]):
        for first, k in ((0, n), (1, n - 2)):
            out = g.export_state(fields, first=first, n=k)
            for f, v in out.items():
                want = b[{"aabb_min": "position", "aabb_max": "position", "sleeping": "is_sleeping"}.get(f, f)]
                assert (np.asarray(v).reshape(k, -1) == want[first : first + k].reshape(k, -1)).all(), (fields, first, f)
    g.close()


@pytest.mark.parametrize("cap", [0, 1, 1023, 1024, 2046, 2047, 2197, 4000])
def test_collider_read_of_several_pinned_buffers(vxp, cap):
    """2197 bricks, more than the 2046 that one buffer holds, read with room for
    none, one, half a buffer's, a buffer's and all of them."""
    rng = np.random.default_rng(5)
    bricks = vxp.scenes.readme_box(104)
    assert len(bricks) == 2197
    bricks["voxels"][:, rng.integers(0, 512, size=200)] = 0
    g = vxp.VoxelPhysicsSystem()
    g.add_collider(3, 0.1, bricks)
    whole_info, whole = g.read_collider(3)
    order = np.lexsort(whole["pos"].T)
    assert whole[order].tobytes() == bricks[np.lexsort(bricks["pos"].T)].tobytes()
    info = np.zeros(1, dtype=vxp.abi.COLLIDER_INFO_DTYPE)
    out = np.zeros(max(cap, 1), dtype=vxp.abi.BRICK_DTYPE)
    n = ctypes.c_uint32(0)
    rc = g.lib.vxp_collider_read(g.ctx, 3, vxp.abi.ptr(info), vxp.abi.ptr(out) if cap else None, cap, ctypes.byref(n))
    assert rc == 0 and n.value == 2197
    assert info[0].tobytes() == whole_info.tobytes()
    k = min(cap, 2197)
    assert out[:k].tobytes() == whole[:k].tobytes()
    assert not out[k:]["voxels"].any()
    g.close()
