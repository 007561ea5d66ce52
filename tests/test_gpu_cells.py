"""The pair list by cells, where its cells and rows have edges: boxes whose
corners lie on cell faces, bodies that touch very many others, and worlds of
mostly large bodies, moving and static."""
import time

import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu


def table(vxp, n):
    b = np.zeros(n, dtype=vxp.abi.BODY_DTYPE)
    b["id"] = np.arange(1, n + 1)
    b["body_type"] = vxp.abi.BODY_DYNAMIC
    b["inv_mass"] = 1.0
    b["inv_inertia_local"][:, [0, 4, 8]] = 1.0
    b["rotation"][:, 3] = 1.0
    return b


@pytest.mark.parametrize("n,mode", [(700, 0), (4800, 1)])
def test_boxes_on_cell_faces(vxp, n, mode):
    """Unrotated boxes of 1 x 1 x 0.5 m (diagonal 1.5) at a margin of 1/16 have
    cells of exactly 2 m.  Each axis of each box puts the inflated box's lower or
    its upper end on a cell face, on both sides of the origin, or leaves it at a
    multiple of 1/16: boxes that just touch across a face are pairs, as for the
    oracle."""
    margin = np.float32(0.0625)
    rng = np.random.default_rng(n)
    half = int(0.6 * n ** (1 / 3)) + 1
    b = table(vxp, n)
    b["body_type"][:: 7] = vxp.abi.BODY_STATIC
    face = 2.0 * rng.integers(-half, half + 1, size=(n, 3))
    lower = face + 0.0625
    upper = face - 0.0625 - np.array([1.0, 1.0, 0.5])
    free = rng.integers(-32 * half, 32 * half + 1, size=(n, 3)) / 16.0
    b["position"] = np.choose(rng.integers(0, 3, size=(n, 3)), [lower, upper, free]).astype(np.float32)
    g = vxp.VoxelPhysicsSystem(pair_margin=margin, substeps=2, max_bodies=n, max_pairs=1 << 16)
    r = O.OracleWorld(substeps=2)
    for w in (g, r):
        w.add_collider(0, 0.125, vxp.scenes.solid_box(8, 8, 4))
        w.set_bodies(b)
    g.set_launch_mode(mode)
    pairs = r.pairs(margin)
    lo = b["position"] - margin
    hi = b["position"] + np.array([1.0, 1.0, 0.5], dtype=np.float32) + margin
    i, j = pairs["body_a"].astype(int) - 1, pairs["body_b"].astype(int) - 1
    touching = (lo[i] == hi[j]) | (hi[i] == lo[j])
    assert (touching & (np.mod(np.where(lo[i] == hi[j], lo[i], hi[i]), 2.0) == 0)).any(axis=1).sum() > 50
    assert g.pairs(margin).tobytes() == pairs.tobytes()
    dt = np.float32(1 / 120)
    g.step(dt)
    r.step(dt, pairs)
    gs, rs = g.stats(), r.stats()
    assert gs["pairs_tested"] == rs["pairs_tested"] > 100
    assert g.manifolds().tobytes() == r.manifolds().tobytes()
    assert g.get_bodies().tobytes() == r.get_bodies().tobytes()
    g.close()
    r.close()


def add_box_colliders(vxp, *worlds):
    """0: cubes of 0.8 m, 1: of 8 m, 2: of 400 m."""
    for w in worlds:
        for c, voxel in enumerate((0.1, 1.0, 50.0)):
            w.add_collider(c, voxel, vxp.scenes.readme_box(8))


@pytest.mark.parametrize("n,mode", [(300, 0), (900, 0), (4800, 1), (9000, 1)])
@pytest.mark.parametrize("large,static", [(0.002, 1.0), (0.002, 0.0), (0.3, 0.5), (0.9, 1.0), (0.6, 0.0)])
def test_large_bodies_among_small(vxp, n, mode, large, static):
    """Bodies too large for the cells, few or most, moving or static, and three
    that every other one touches, the first, a middle and the last of their ids
    (two static, one moving): the oracle's list, and its steps."""
    rng = np.random.default_rng(n)
    b = table(vxp, n)
    big = rng.random(n) < large
    b["collider_id"] = big
    b["body_type"][big & (rng.random(n) < static)] = vxp.abi.BODY_STATIC
    side = 0.5 * (n * (0.8 ** 3 * (1 - large) + 8.0 ** 3 * large)) ** (1 / 3) + 1.0
    b["position"] = rng.uniform(-side, side, size=(n, 3)).astype(np.float32)
    b["rotation"] = vxp.scenes.shoemake_quat(rng, n)
    wide = [0, n // 2, n - 1]
    b["collider_id"][wide] = 2
    b["position"][wide] = -200.0
    b["rotation"][wide] = (0, 0, 0, 1)
    b["body_type"][wide] = (vxp.abi.BODY_STATIC, vxp.abi.BODY_DYNAMIC, vxp.abi.BODY_STATIC)
    b["id"] = rng.permutation(n) + 1
    order = np.argsort(b["id"])
    b["id"][wide] = b["id"][order[[0, n // 2, n - 1]]]
    b["id"][np.setdiff1d(np.arange(n), wide)] = rng.permutation(
        np.setdiff1d(np.arange(1, n + 1), [1, n // 2 + 1, n]))
    # no contacts: the list alone is in question, not 400 m bodies' overlap regions
    g = vxp.VoxelPhysicsSystem(substeps=1, max_bodies=n, max_pairs=1 << 20)
    r = O.OracleWorld(substeps=1)
    add_box_colliders(vxp, g, r)
    for w in (g, r):
        w.set_bodies(b)
    for margin in (0.1, 0.0):
        pairs = r.pairs(margin)
        counts = np.bincount(pairs["body_a"])
        assert counts.max() > n // 4
        assert g.pairs(margin).tobytes() == pairs.tobytes(), f"margin {margin}"
    if mode == 0:
        # the list as a step on one CTA builds it: its pairs, by their number
        # and by what they do
        g.set_launch_mode(0)
        dt = np.float32(1 / 120)
        pairs = r.pairs()
        g.step(dt)
        r.step(dt, pairs)
        gs, rs = g.stats(), r.stats()
        assert gs["pairs_tested"] == rs["pairs_tested"] == len(pairs)
        assert g.manifolds().tobytes() == r.manifolds().tobytes()
        assert g.get_bodies().tobytes() == r.get_bodies().tobytes()
    g.close()
    r.close()


@pytest.mark.parametrize("at", [1, 40000, 66000])
def test_row_longer_than_its_bitmap(vxp, at):
    """One body that 65999 others touch, none of which touch each other: its row
    is longer than the 65536 columns put in order at a time."""
    n = 66000
    b = table(vxp, n)
    s = 41
    pos = np.stack(np.meshgrid(*[np.arange(s)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n]
    b["position"] = pos * 2.0
    wide = at - 1
    b["collider_id"][wide] = 2
    b["position"][wide] = -10.0
    b["body_type"][wide] = vxp.abi.BODY_STATIC
    g = vxp.VoxelPhysicsSystem(max_bodies=n, max_pairs=1 << 17)
    add_box_colliders(vxp, g)
    g.set_bodies(b)
    others = np.setdiff1d(np.arange(1, n + 1), [at])
    want = np.zeros(n - 1, dtype=vxp.abi.PAIR_DTYPE)
    want["body_a"] = np.minimum(others, at)
    want["body_b"] = np.maximum(others, at)
    assert g.pairs(0.1).tobytes() == want.tobytes()
    g.close()


@pytest.mark.parametrize("kind,limit", [("wide", 10), ("level", 2)])
def test_time_of_lists_with_large_bodies(vxp, kind, limit):
    """15000 cubes' own list of 0.14 million pairs against two of as many bodies:
    64 static ones under all the cubes (a million pairs in rows of up to 15000,
    once 30 times as long, each pair looked for in its whole row), and a level of
    14000 static chunks ten times the cubes' size with 1000 cubes (0.03 million
    pairs, once 4.8 times as long, every chunk tested against every body)."""
    n, s = 15000, 25
    rng = np.random.default_rng(3)
    b = table(vxp, n)
    b["position"] = np.stack(np.meshgrid(*[np.arange(s)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n]
    b["position"] += rng.uniform(-0.2, 0.2, size=(n, 3)).astype(np.float32)
    b["rotation"] = vxp.scenes.shoemake_quat(rng, n)
    g = vxp.VoxelPhysicsSystem(max_bodies=n, max_pairs=1 << 21)
    add_box_colliders(vxp, g)

    def fastest_s():
        g.set_bodies(b)
        out = []
        for _ in range(9):
            t0 = time.perf_counter()
            g.pairs(0.1)
            out.append(time.perf_counter() - t0)
        return min(out)

    plain = fastest_s()
    if kind == "wide":
        b["collider_id"][:64] = 2
        b["position"][:64] = -100.0
        b["rotation"][:64] = (0, 0, 0, 1)
        b["body_type"][:64] = vxp.abi.BODY_STATIC
    else:
        chunks = np.arange(n) % 15 != 0
        b["collider_id"][chunks] = 1
        b["body_type"][chunks] = vxp.abi.BODY_STATIC
        b["position"] *= 3.5
    assert fastest_s() < limit * plain
    g.close()
