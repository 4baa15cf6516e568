"""Device noise generator against the host one (needs a B200): identical bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,spacing,octaves,fill,shell", [(64, 16, 3, 0.1, True), (128, 32, 4, 0.1, True),
                                                         (256, 64, 5, 0.5, False), (128, 16, 2, 0.0, True),
                                                         (64, 8, 1, 1.0, False)])
def test_device_noise_equals_host(vx, cuda, R, spacing, octaves, fill, shell):
    host = vx.synth_noise(R, spacing, octaves, fill, 1234, shell)
    dev = vx.synth_noise_dev(R, spacing, octaves, fill, 1234, shell).cpu().numpy().view(np.uint64)
    np.testing.assert_array_equal(dev, host)


@pytest.mark.parametrize("R,spacing,octaves,fill,shell", [
    (192, 12, 3, 0.3, False),       # rows side by side in a block leave threads over
    (320, 20, 3, 0.37, True),       # the last segment of a row is short
    (64, 1, 1, 0.5, False),         # one lattice cell per voxel
    (128, 1 << 15, 16, 0.25, True),  # the most octaves, the coarsest far larger than the grid
    (128, 256, 9, 0.62, False),
    (64, 1 << 30, 1, 0.5, False),   # nearly all values alike: more values in one bin than candidates
    (64, 1 << 20, 2, 0.001, False), (128, 8, 3, 1e-7, False), (64, 5, 2, 0.9999, True)])
def test_device_noise_edges_equal_host(vx, cuda, R, spacing, octaves, fill, shell):
    """Odd tile shapes, every register form (4, 8, 16 octaves), both ways to the threshold."""
    host = vx.synth_noise(R, spacing, octaves, fill, 99, shell)
    dev = vx.synth_noise_dev(R, spacing, octaves, fill, 99, shell).cpu().numpy().view(np.uint64)
    np.testing.assert_array_equal(dev, host)


@pytest.mark.parametrize("spacing,octaves,fill", [(32, 3, 0.1), (32, 3, 0.37), (27, 2, 0.1)])
def test_device_noise_rounds_like_the_host(vx, cuda, spacing, octaves, fill):
    """134 M voxels: several per binary32 value, so a value off by one unit in the last place near
    the threshold changes bits (products and sums fused into one rounding change tens of them)."""
    host = vx.synth_noise(512, spacing, octaves, fill, 5, False)
    dev = vx.synth_noise_dev(512, spacing, octaves, fill, 5, False).cpu().numpy().view(np.uint64)
    np.testing.assert_array_equal(dev, host)


def test_device_noise_from_several_threads(vx, cuda):
    """Calls of different sizes at once, each thread on a stream of its own: every launch has the
    shared memory its size needs, whatever size another thread launches with."""
    import ctypes
    import threading

    import torch
    sizes = [(512, 1 << 15, 16), (64, 16, 1), (320, 4, 3), (128, 32, 4)]
    want = [vx.synth_noise(R, s, o, 0.3, 7, False) for R, s, o in sizes]
    outs = [torch.zeros(R * R * (R // 64), dtype=torch.int64, device="cuda") for R, _, _ in sizes]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()
    status = [[] for _ in sizes]

    def work(k):
        R, s, o = sizes[k]
        for _ in range(40):
            status[k].append(vx.lib().vx_synth_noise_dev(R, s, o, 0.3, 7, 0, ctypes.c_void_p(outs[k].data_ptr()),
                                                         ctypes.c_void_p(streams[k].cuda_stream)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [set(x) for x in status] == [{vx.VX_OK}] * len(sizes)
    for o, w in zip(outs, want):
        np.testing.assert_array_equal(o.cpu().numpy().view(np.uint64), w)
