"""Casts without work counters take the plain-ray iteration (vx_regular.cuh); casts with
counters the general one.  Both against the oracle, bit for bit (0 ulp: every result is
discrete or the same IEEE operations), where the two may part: directions around the
thresholds of the regular form (1/550, 1e-5, 1e-8), axes of either sign, origins on the box,
on voxel planes and far away, worlds with other sizes than a power of two, other minima and
other t ranges (needs a B200)."""
import numpy as np
import pytest

from test_gpu_parity import assert_hits_equal, gpu_cast, scene_from_oracle

pytestmark = pytest.mark.gpu

FLT_MAX = 3.4028234663852886e38


def edge_rays(wmin, wmax, n, seed):
    """Rays whose directions have components at and around every threshold, from origins inside,
    on planes of voxels and of the box, and outside (some beyond the plain form's range)."""
    rng = np.random.default_rng(seed)
    wmin, wmax = np.asarray(wmin, np.float32), np.asarray(wmax, np.float32)
    size = wmax - wmin
    o = (wmin + size * rng.uniform(-0.2, 1.2, size=(n, 3))).astype(np.float32)
    on_plane = rng.random((n, 3)) < 0.25
    o = np.where(on_plane, np.round(o), o).astype(np.float32)
    k = rng.random((n, 3))
    o = np.where(k < 0.05, wmin, np.where(k > 0.95, wmax, o)).astype(np.float32)
    far = rng.random(n) < 0.05
    away = rng.choice(np.array([2e2, 5e4, 9.9e4, 2e5, 3e7], np.float32), size=(n, 1))
    d = rng.normal(size=(n, 3)).astype(np.float32)
    o[far] = (wmin + size / 2 - d[far] / np.linalg.norm(d[far], axis=1, keepdims=True) * away[far]).astype(np.float32)
    mags = np.array([0.0, 1e-12, 0.99e-8, 1.01e-8, 1e-7, 0.99e-5, 1.01e-5, 1e-4, 1.0 / 560, 1.0 / 540, 0.003], np.float32)
    small = (rng.random((n, 3)) < 0.3) & ~far[:, None]
    sign = rng.choice(np.array([-1.0, 1.0], np.float32), size=(n, 3))
    d = np.where(small, mags[rng.integers(0, mags.size, size=(n, 3))] * sign, d).astype(np.float32)
    d[rng.random(n) < 0.02] *= np.float32(1e-18)  # |d|^2 outside the ordinary range
    return np.concatenate([o, d], axis=1).astype(np.float32)


def sparse_scene(vo, wmin, wmax, depth, seed, count):
    rng = np.random.default_rng(seed)
    lo, hi = np.ceil(wmin).astype(int), np.floor(wmax).astype(int)
    p = np.unique(rng.integers(lo, hi, size=(count, 3)), axis=0)
    return vo.OracleScene.from_positions([tuple(float(v) for v in q) for q in p], wmin, wmax, depth)


SCENES = [((0.0, 0.0, 0.0), (64.0, 64.0, 64.0), 6, 9000), ((0.0, 0.0, 0.0), (40.0, 40.0, 40.0), 6, 2500),
          ((-40.0, -16.0, 3.0), (24.0, 48.0, 67.0), 6, 4000), ((0.0, 0.0, 0.0), (128.0, 128.0, 128.0), 7, 30000),
          ((0.0, 0.0, 0.0), (3.0, 3.0, 3.0), 2, 9)]


@pytest.mark.parametrize("case", SCENES, ids=lambda c: f"{c[0][0]:g}_{c[1][0]:g}")
@pytest.mark.parametrize("t", [(0.0, FLT_MAX), (0.0, 30.0), (17.5, 60.0)], ids=lambda t: f"t{t[0]:g}")
def test_plain_rays_equal_oracle(vx, vo, cuda, case, t):
    wmin, wmax, depth, count = case
    o = sparse_scene(vo, wmin, wmax, depth, 5, count)
    scene = vx.Scene(scene_from_oracle(vx, o, (wmin, wmax), depth))
    rays = edge_rays(wmin, wmax, 60001, 7)
    want = o.cast_rays(rays, *t)
    for with_counters in (False, True):
        g, _, cnt = gpu_cast(vx, scene, rays, *t, with_counters=with_counters)
        assert_hits_equal(g, want, cnt, f"counters={with_counters}")


@pytest.mark.parametrize("lod", [(0.0, 0.004), (0.5, 0.03)])
def test_plain_rays_lod_equal_oracle(vx, vo, cuda, lod):
    import torch
    wmin, wmax = (0.0, 0.0, 0.0), (128.0, 128.0, 128.0)
    o = sparse_scene(vo, wmin, wmax, 7, 6, 20000)
    scene = vx.Scene(scene_from_oracle(vx, o, (wmin, wmax), 7))
    rays = edge_rays(wmin, wmax, 40003, 8)
    r = torch.from_numpy(rays).cuda()
    hits = torch.zeros((rays.shape[0], 4), dtype=torch.int32, device="cuda")
    scene.cast_rays_dev(r, hits, lod=lod)
    torch.cuda.synchronize()
    assert_hits_equal(hits.cpu().numpy().view(vx.HIT_DTYPE).reshape(-1), o.cast_rays_lod(rays, lod), None, "lod")


@pytest.mark.parametrize("tuning", [(128, 32, 1, 0), (256, 64, 0, 0), (256, 32, 1, 7), (128, 64, 0, 1)],
                         ids=lambda t: "b%d_k%d_s%d_g%d" % t)
def test_plain_rays_batched_equal_oracle(vx, vo, cuda, tuning):
    """Static lanes, stack in shared and local memory, with and without an iteration budget (the
    second launch casts the rays set aside), two scenes of different shapes in one launch."""
    import torch
    shapes = [SCENES[0], SCENES[2]]
    oracles = [sparse_scene(vo, c[0], c[1], c[2], 9, c[3]) for c in shapes]
    scenes = [vx.Scene(scene_from_oracle(vx, o, (c[0], c[1]), c[2])) for o, c in zip(oracles, shapes)]
    parts = [edge_rays(c[0], c[1], m, 11) for c, m in zip(shapes, (20011, 7))]
    rays = torch.from_numpy(np.concatenate(parts)).cuda()
    begin = torch.tensor([0, 20011, 20018], dtype=torch.int32, device="cuda")
    hits = torch.zeros((20018, 4), dtype=torch.int32, device="cuda")
    batch = vx.Batch(scenes)
    block, k, shared, budget = tuning
    batch.set_tuning(block, k, shared, 0, budget)
    batch.cast(rays, begin, hits)
    torch.cuda.synchronize()
    g = hits.cpu().numpy().view(vx.HIT_DTYPE).reshape(-1)
    assert_hits_equal(g[:20011], oracles[0].cast_rays(parts[0]), None, "scene 0")
    assert_hits_equal(g[20011:], oracles[1].cast_rays(parts[1]), None, "scene 1")
    batch.close()


def test_bricks_away_from_their_slots(vx, vo, cuda):
    """A scene whose grid slots name bricks with other coordinates is accepted; its casts march the
    brick's own box, with and without counters."""
    wmin, wmax, depth, count = SCENES[0]
    o = sparse_scene(vo, wmin, wmax, depth, 12, count)
    a = scene_from_oracle(vx, o, (wmin, wmax), depth)
    a.brick_coord = np.roll(a.brick_coord, 3)
    scene = vx.Scene(a)
    rays = edge_rays(wmin, wmax, 20001, 13)
    plain, _, _ = gpu_cast(vx, scene, rays, with_counters=False)
    general, _, _ = gpu_cast(vx, scene, rays, with_counters=True)
    np.testing.assert_array_equal(plain, general)
    assert (plain["flags"] & 1).any()
