"""Batches of different sizes in one process (needs a B200): a kernel's shared-memory limit is the
kernel's, so preparing a small batch must not refuse the launches of a larger one prepared before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuning", [(256, 32, 1, 0), (256, 32, 1, 8), (128, 32, 1, 0)],
                         ids=lambda t: "b%d_r%d" % (t[0], t[3]))
def test_a_small_batch_after_a_large_one(vx, cuda, tuning):
    import torch
    from vx_b200 import workloads as W
    bits = vx.synth_noise(64, 8, 3, 0.3, 2, False)
    scene = vx.Scene(W.scene_from_bits(bits, 64, None, 2, max_levels=23))
    n = 3001
    rays = torch.from_numpy(W.random_rays(n, 64, seed=3)).cuda()
    want = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    scene.cast_rays_dev(rays, want)
    sizes = (256, 2)
    batches = [vx.Batch([scene] * s) for s in sizes]
    begins = [torch.tensor([0] + [n] * s, dtype=torch.int32, device="cuda") for s in sizes]
    for b in batches:
        b.set_tuning(*tuning)
    for k in (0, 1, 0):
        hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
        batches[k].cast(rays, begins[k], hits)
        torch.cuda.synchronize()
        assert torch.equal(hits, want)
    vx.cast_batch_noalloc([scene], rays, begins[1][:2].contiguous(), hits)
    batches[0].cast(rays, begins[0], hits)
    torch.cuda.synchronize()
    assert torch.equal(hits, want)
    for b in batches:
        b.close()
