"""Scenes that the plain-ray kernels do not take (a world minimum beyond 1e5, a world taller than
wide): every entry point sends them to the general kernels.  Hits against the oracle, bit for bit,
and the time against the same cast with counters, which is the general kernel's own (needs a B200)."""
import dataclasses

import numpy as np
import pytest

from test_gpu_parity import assert_hits_equal, scene_from_oracle

pytestmark = pytest.mark.gpu

FAR = 131072.0
WORLDS = {"moved": ((FAR, FAR, FAR), (FAR + 64, FAR + 64, FAR + 64)), "tall": ((0.0, 0.0, 0.0), (64.0, 80.0, 64.0)),
          "ordinary": ((0.0, 0.0, 0.0), (64.0, 64.0, 64.0))}


def build(vx, vo, world, seed=4):
    wmin, wmax = WORLDS[world]
    rng = np.random.default_rng(seed)
    p = np.unique(rng.integers(0, 64, size=(6000, 3)), axis=0) + np.asarray(wmin)
    o = vo.OracleScene.from_positions([tuple(float(v) for v in q) for q in p], wmin, wmax, 6)
    return o, vx.Scene(scene_from_oracle(vx, o, (wmin, wmax), 6))


def rays_for(world, n, seed):
    rng = np.random.default_rng(seed)
    wmin, wmax = (np.asarray(v, np.float32) for v in WORLDS[world])
    o = wmin + (wmax - wmin) * rng.uniform(-0.3, 1.3, size=(n, 3)).astype(np.float32)
    return np.concatenate([o, rng.normal(size=(n, 3)).astype(np.float32)], axis=1).astype(np.float32)


def to_hits(vx, t):
    return t.cpu().numpy().view(vx.HIT_DTYPE).reshape(-1)


@pytest.mark.parametrize("world", ["moved", "tall"])
def test_every_single_scene_entry(vx, vo, cuda, world):
    import torch
    from vx_b200 import workloads as W
    o, scene = build(vx, vo, world)
    rays = rays_for(world, 20003, 1)
    d = torch.from_numpy(rays).cuda()
    n = rays.shape[0]
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    scene.cast_rays_dev(d, hits)
    want = o.cast_rays(rays)
    assert_hits_equal(to_hits(vx, hits), want, None, "cast")
    assert_hits_equal(scene.cast_rays_host(rays[:777])[0], want[:777], None, "host")
    lod = (0.0, 0.02)
    lod_hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    scene.cast_rays_dev(d, lod_hits, lod=lod)
    assert_hits_equal(to_hits(vx, lod_hits), o.cast_rays_lod(rays, lod), None, "lod")
    # shadow rays: the compacted cast against the cast of all slots
    light = W.light_dir(3)
    shadow, slots = torch.zeros((n, 4), dtype=torch.int32, device="cuda"), torch.zeros((n, 6), device="cuda")
    scene.cast_shadow_rays_dev(d, hits, light, shadow)
    vx.spawn_shadow_rays(d, hits, light, slots)
    all_slots = slots.cpu().numpy()
    got = to_hits(vx, shadow)
    live = (want["flags"] & 1).astype(bool)
    sw = o.cast_rays(all_slots[live])
    assert live.any()
    assert_hits_equal(got[live], sw, None, "shadow")
    # the rendered image's and the forward pass's hits against the cast of their camera's rays
    wmin = WORLDS[world][0]
    cam = W.look_camera([wmin[0] + 30.5, wmin[1] + 31.5, wmin[2] - 60.0], [0.05, 0.02, 1.0], 60.0, 101, 67)
    cr = vx.camera_rays(cam, 101, 67)
    cw = o.cast_rays(cr)
    assert (cw["flags"] & 1).any()
    rec = torch.zeros((101 * 67, 4), dtype=torch.int32, device="cuda")
    scene.render_dev(cam, 101, 67, hits=rec)
    assert_hits_equal(to_hits(vx, rec), cw, None, "render")
    attr = torch.rand(scene.download().brick_count * 1536, device="cuda")
    image = torch.zeros((101 * 67, 3), device="cuda")
    rec.zero_()
    vx.diff_forward(scene, cam, 101, 67, 0, attr, None, image, rec)
    assert_hits_equal(to_hits(vx, rec), cw, None, "forward")


@pytest.mark.parametrize("worlds", [["moved"], ["moved", "ordinary"], ["tall"] * 7 + ["ordinary"],
                                    ["moved"] * 8 + ["ordinary"]], ids=len)
@pytest.mark.parametrize("tuning", [(256, 32, 1, 0), (128, 64, 0, 0), (256, 32, 1, 5), (128, 32, 0, 3)],
                         ids=lambda t: "b%d_s%d_g%d" % (t[0], t[2], t[3]))
def test_batches_of_both_kinds(vx, vo, cuda, worlds, tuning):
    """Batches on both sides of the rule (one ordinary scene in eight), with and without a budget."""
    import torch
    built = {w: build(vx, vo, w) for w in set(worlds)}
    parts = [rays_for(w, 1501 + 7 * i, i) for i, w in enumerate(worlds)]
    begin = np.concatenate([[0], np.cumsum([p.shape[0] for p in parts])])
    rays = torch.from_numpy(np.concatenate(parts)).cuda()
    d_begin = torch.from_numpy(begin.astype(np.int32)).cuda()
    scenes = [built[w][1] for w in worlds]
    batch = vx.Batch(scenes)
    block, k, shared, budget = tuning
    batch.set_tuning(block, k, shared, 0, budget)
    outs = []
    for _ in range(2):
        outs.append(torch.zeros((int(begin[-1]), 4), dtype=torch.int32, device="cuda"))
    batch.cast(rays, d_begin, outs[0])
    vx.cast_batch_noalloc(scenes, rays, d_begin, outs[1])
    torch.cuda.synchronize()
    for out in outs:
        g = to_hits(vx, out)
        for i, w in enumerate(worlds):
            assert_hits_equal(g[begin[i]:begin[i + 1]], built[w][0].cast_rays(parts[i]), None, f"scene {i}")
    batch.close()


def test_general_scenes_run_the_general_kernel(vx, cuda):
    """The cast of a scene away from the origin takes no longer than with counters (the general kernel
    and 16 more bytes a ray); through the plain kernel, whose rays would all go out of line, it took
    1.22 times as long."""
    import torch
    from vx_b200 import workloads as W
    bits = vx.synth_noise(256, 16, 3, 0.3, 5, False)
    arrays = vx.build_dense(bits, 256, 8)
    moved = dataclasses.replace(arrays, world_min=(FAR,) * 3, world_max=(FAR + 256,) * 3)
    scene = vx.Scene(moved)
    cam = W.empty_voxel_camera(bits, 256, 5, 60.0, 1024, 768)
    rays = vx.camera_rays(cam, 1024, 768)
    rays[:, :3] += np.float32(FAR)
    d = torch.from_numpy(rays).cuda()
    hits = torch.zeros((rays.shape[0], 4), dtype=torch.int32, device="cuda")
    counters = torch.zeros((rays.shape[0], 4), dtype=torch.int32, device="cuda")
    best = {}
    for _ in range(8):
        for name, c in (("plain call", None), ("with counters", counters)):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                scene.cast_rays_dev(d, hits, None, c)
            b.record()
            torch.cuda.synchronize()
            best[name] = min(best.get(name, 1e9), a.elapsed_time(b))
    assert best["plain call"] < 1.1 * best["with counters"], best


@pytest.mark.parametrize("keep", [0.001, 0.05, 0.1, 0.5])
def test_trees_with_children_beyond_their_nodes(vx, cuda, keep):
    """A tree cut off after some of its nodes is accepted: a ray that would enter a missing child
    stands still up to the reference's cap.  The same hits with and without counters, alone and in a
    batch beside the whole tree, and no more time without counters than with (the plain kernel, which
    would run the cap out, took 4 to 7 times as long)."""
    import torch
    from vx_b200 import workloads as W
    bits = vx.synth_noise(256, 16, 3, 0.3, 5, False)
    arrays = vx.build_dense(bits, 256, 8)
    k = max(1, int(arrays.node_count * keep))
    cut = vx.Scene(dataclasses.replace(arrays, nodes=arrays.nodes[:2 * k].copy(), node_brick=arrays.node_brick[:k].copy()))
    whole = vx.Scene(arrays)
    n = 200003
    d = torch.from_numpy(W.random_rays(n, 256, seed=8)).cuda()
    out = [torch.zeros((n, 4), dtype=torch.int32, device="cuda") for _ in range(2)]
    counters = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    best = [1e9, 1e9]
    for _ in range(6):
        for i, c in enumerate((None, counters)):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                cut.cast_rays_dev(d, out[i], None, c)
            b.record()
            torch.cuda.synchronize()
            best[i] = min(best[i], a.elapsed_time(b))
    assert torch.equal(out[0], out[1])
    assert best[0] < 1.1 * best[1], best
    whole_hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    whole.cast_rays_dev(d, whole_hits)
    batch = vx.Batch([cut, whole])
    begin = torch.tensor([0, n, 2 * n], dtype=torch.int32, device="cuda")
    both = torch.zeros((2 * n, 4), dtype=torch.int32, device="cuda")
    batch.cast(torch.cat([d, d]).contiguous(), begin, both)
    torch.cuda.synchronize()
    assert torch.equal(both[:n], out[1]) and torch.equal(both[n:], whole_hits)
    batch.close()


def test_the_device_builders_children_are_nodes(vx, cuda):
    """Scenes built on the device are taken as ordinary without a check: every child that may be
    entered is one of their nodes."""
    for R, levels in ((64, 6), (192, 8), (256, 8), (64, 23)):
        bits = vx.synth_noise_dev(R, 8, 3, 0.4, R, False)
        nodes = vx.scene_from_dense_dev(bits, R, levels).download().nodes.reshape(-1, 2)
        inner = ~(nodes[:, 1] >> 8) & nodes[:, 1] & 0xFF
        count = np.array([bin(v).count("1") for v in range(256)])[inner]
        assert np.all((count == 0) | (nodes[:, 0].astype(np.int64) + count <= nodes.shape[0]))
