"""Host-buffer casts on both sides of the small-cast limit (5,000 rays) against the device-buffer
cast of the same rays, colours included, calls of growing and shrinking size on one scene
(needs a B200)."""
import numpy as np
import pytest

from test_gpu_parity import gpu_cast

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("color", ["rgba8", "dxt1", None])
def test_small_host_casts_equal_device_casts(vx, cuda, color):
    from vx_b200 import workloads as W
    bits = vx.synth_noise(64, 8, 3, 0.4, 21, True)
    scene = vx.Scene(W.scene_from_bits(bits, 64, color, 21))
    for n in (1, 5000, 33, 5001, 4999, 2):
        rays = W.random_rays(n, 64, seed=n)
        g, c, _ = gpu_cast(vx, scene, rays, with_counters=False)
        h, hc = scene.cast_rays_host(rays)
        np.testing.assert_array_equal(h, g)
        if color:
            np.testing.assert_array_equal(hc.view(np.uint32), c.view(np.uint32))
        lod = (0.0, 0.02)
        hl, _ = scene.cast_rays_host(rays, lod=lod)
        gl, _ = scene.cast_rays_host(np.concatenate([rays, W.random_rays(6000, 64, seed=1)]), lod=lod)
        np.testing.assert_array_equal(hl, gl[:n])
