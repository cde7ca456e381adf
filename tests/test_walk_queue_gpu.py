"""Ray-set walks over stacked triangles, where every ray reaches leaf after leaf: few rays walk one per warp (three
triangles per lane and step), more fill the persistent walk's triangle queue (up to 24 per node and lane against room
for 64 per warp, so that most go back to the ray's stack and are queued again). Hits must equal the oracle's, at ray
counts around a warp's 32 lanes, beside the largest one-per-warp launch (12 rays per block) and above it."""
import numpy as np
import pytest

import oracle
from sparkle_gb300 import abi, native, scenes

from parity import INVALID, classify_hits, oracle_hits

pytestmark = pytest.mark.gpu


def stacked_triangles(layers: int):
    """`layers` large triangles, one above the other and slightly tilted, as two instances (one turned and scaled),
    with an analytic sphere between them."""
    rng = np.random.default_rng(layers)
    z = np.linspace(0.0, 1.0, layers)
    base = np.array([[-4.0, -3.0], [4.0, -3.0], [0.0, 5.0]])
    pos = np.zeros((layers, 3, 3))
    pos[:, :, :2] = base
    pos[:, :, 2] = z[:, None] + rng.uniform(-0.3, 0.3, (layers, 3)) / layers
    pos = pos.reshape(-1, 3)
    nrm = np.tile([0.0, 0.0, 1.0], (len(pos), 1))
    mesh = abi.Mesh(pos, nrm, np.arange(len(pos)).reshape(-1, 3))
    mats = [abi.Material.lambertian((0.5, 0.5, 0.5))]
    lin = scenes._rot_z(0.4) @ np.diag([1.2, 0.9, 1.1])
    inst = [abi.Instance(0, 0), abi.Instance(0, 0, scenes._affine(lin, (0.2, -0.1, -3.0))),
            abi.Instance(0, 0, scenes._affine(np.eye(3), (0.5, 0.5, -1.0)), sphere=True, radius=0.8)]
    return abi.Scene([mesh], inst, mats, abi.Sky(), name=f"stack{layers}")


@pytest.mark.parametrize("layers", [1, 24, 200])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 4097, 12768, 12769, 34049])
def test_stacked_triangles_match_the_oracle(layers, count):
    scene = stacked_triangles(layers)
    rng = np.random.default_rng(count)
    target = np.stack([rng.uniform(-3, 3, count), rng.uniform(-2, 3, count), rng.uniform(-3, 1, count)], 1)
    origin = np.stack([rng.uniform(-3, 3, count), rng.uniform(-3, 3, count), np.where(rng.random(count) < 0.5, 6.0, -8.0)], 1)
    d = target - origin
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = abi.rays_to_array(origin, d)
    ref_scene = oracle.OracleScene(scene)
    ctx = native.Context(0)
    ctx.set_scene(scene)
    got = ctx.trace(rays)
    assert ctx.stats()["error_flags"] == 0
    assert ctx.stats()["extension_rays"] == count
    ref, _ = oracle_hits(ref_scene, rays, oracle.PRUNED)
    c = classify_hits(got, ref)
    assert c["exact"] + c["tie"] == count, c
    any_hit = ctx.trace(rays, any_hit=True)
    sphere = ref["face"][ref["prim"] != INVALID] == INVALID  # (an any-hit query takes a sphere behind the ray too)
    assert not ((any_hit["prim"] == INVALID) & (ref["prim"] != INVALID)).any(), sphere.sum()
    ctx.close()


def test_edge_rays_are_the_same_whatever_walks_them():
    """Rays that leave an axis-aligned box from a point of its walls, nearly along them: whether Moeller-Trumbore
    accepts a wall's edge, and whether the ray enters its flat box, are both decided by the last bit. A large launch
    (a ray per lane) and small ones (a ray per warp) have to decide alike."""
    scene, _ = scenes.cornell_box(0)
    ctx = native.Context(0)
    ctx.set_scene(scene)
    lo, hi = (np.asarray(v, np.float32) for v in scene.world_bounds())
    rng = np.random.default_rng(3)
    n = 200_000
    o = (lo + (hi - lo) * rng.random((n, 3))).astype(np.float32)
    d = rng.standard_normal((n, 3))
    axis, side = rng.integers(0, 3, n), rng.integers(0, 2, n)
    rows = np.arange(n)
    o[rows, axis] = np.where(side == 1, hi[axis], lo[axis])
    d[rows, axis] = np.where(side == 1, 1, -1) * 10 ** rng.uniform(-7, -2, n)
    near = (axis + 1) % 3  # close to a neighbouring wall, towards it
    o[rows, near] = (lo[near] + (hi[near] - lo[near]) * 10 ** rng.uniform(-6, -2, n)).astype(np.float32)
    d[rows, near] = -np.abs(d[rows, near])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d.astype(np.float32)], 1).astype(np.float32)
    whole = ctx.trace(rays)
    for a in range(0, n, 8192):
        part = ctx.trace(rays[a:a + 8192])
        for f in ("t", "u", "v", "prim", "face"):
            assert np.array_equal(whole[f][a:a + 8192].view(np.uint32), part[f].view(np.uint32)), (f, a)
    ctx.close()


@pytest.mark.parametrize("layers", [1, 24, 200])
@pytest.mark.parametrize("count", [1, 33, 12768, 12769, 34049])
def test_any_hit_over_stacked_triangles_is_the_oracles(layers, count):
    """Any-hit flags both ways: a hit missed, and a hit reported for a ray that has none (a queued triangle credited to
    another lane's ray would do that). Half of the rays pass beside the stack."""
    scene = stacked_triangles(layers)
    rng = np.random.default_rng(1000 + count)
    target = np.stack([rng.uniform(-5, 5, count), rng.uniform(-4, 5, count), rng.uniform(-3, 1, count)], 1)
    origin = np.stack([rng.uniform(-3, 3, count), rng.uniform(-3, 3, count), np.where(rng.random(count) < 0.5, 6.0, -8.0)], 1)
    d = target - origin
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = abi.rays_to_array(origin, d)
    want, _ = oracle.OracleScene(scene).trace(rays, any_hit=True)
    hit = want["prim"] != INVALID
    assert count < 1000 or 0.2 < hit.mean() < 0.8
    ctx = native.Context(0)
    ctx.set_scene(scene)
    got = ctx.trace(rays, any_hit=True)
    assert ctx.stats()["error_flags"] == 0
    assert np.array_equal(got["prim"] != INVALID, hit)
    ctx.close()


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("count", [33, 8512, 8513, 12769, 34047, 34049, 200_000])
def test_scenes_of_few_nodes(count, any_hit):
    """The box (8 instances of few triangles each), whose walks test triangles as they reach them, at ray counts on both
    sides of where the walks and the grid change: the same as the same rays in launches of 4096, which walk one per
    warp, and the oracle's hits (a ray that grazes an edge may differ: 2 in 4096, as the smoke test has it)."""
    scene, _ = scenes.cornell_box(0)
    rays = scenes.random_rays(*scene.world_bounds(), count, seed=count)
    ctx = native.Context(0)
    ctx.set_scene(scene)
    assert len(ctx.bvh_nodes()) <= 16
    got = ctx.trace(rays, any_hit=any_hit)
    st = ctx.stats()
    assert st["error_flags"] == 0 and st["extension_rays"] == count
    parts = np.concatenate([ctx.trace(rays[a:a + 4096], any_hit=any_hit) for a in range(0, count, 4096)])
    ctx.close()
    ref_scene = oracle.OracleScene(scene)
    if any_hit:
        assert np.array_equal(got["prim"] != INVALID, parts["prim"] != INVALID)
        want, _ = ref_scene.trace(rays, any_hit=True)
        wrong = int(((got["prim"] != INVALID) != (want["prim"] != INVALID)).sum())
    else:
        assert got.tobytes() == parts.tobytes()
        c = classify_hits(got, oracle_hits(ref_scene, rays, oracle.PRUNED)[0])
        wrong = count - c["exact"] - c["tie"]
    assert wrong <= max(2, count // 2048)


def test_edge_rays_one_per_warp():
    """Rays that leave the box from a point of its walls, nearly along them (their hits are decided by the last bit), in
    launches of 4096, which walk one ray per warp there, against one launch of all."""
    scene, _ = scenes.cornell_box(0)
    lo, hi = (np.asarray(v, np.float32) for v in scene.world_bounds())
    rng = np.random.default_rng(11)
    n = 65_536
    axis, rows = rng.integers(0, 3, n), np.arange(n)
    side = rng.integers(0, 2, n) == 1
    near = (axis + 1) % 3
    o = (lo + (hi - lo) * rng.random((n, 3))).astype(np.float32)
    o[rows, axis] = np.where(side, hi[axis], lo[axis])
    o[rows, near] = (lo[near] + (hi[near] - lo[near]) * 10 ** rng.uniform(-6, -2, n)).astype(np.float32)
    d = rng.standard_normal((n, 3))
    d[rows, axis] = np.where(side, 1, -1) * 10 ** rng.uniform(-7, -2, n)
    d[rows, near] = -np.abs(d[rows, near])
    rays = abi.rays_to_array(o, d / np.linalg.norm(d, axis=1, keepdims=True))
    ctx = native.Context(0)
    ctx.set_scene(scene)
    for any_hit in (False, True):
        whole = ctx.trace(rays, any_hit=any_hit)
        parts = np.concatenate([ctx.trace(rays[a:a + 4096], any_hit=any_hit) for a in range(0, n, 4096)])
        if any_hit:
            assert np.array_equal(whole["prim"] != INVALID, parts["prim"] != INVALID)
        else:
            assert whole.tobytes() == parts.tobytes()
    ctx.close()
