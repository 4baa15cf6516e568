"""Bounce-ray compaction at the edges of its chunks of 1,024 primary rays: scenes with one ray, a
chunk less one, a chunk, a chunk and one, none; the compacted rays per scene, in bin order and
inside a bin first (k = 0) then second bounce rays in primary order; bounce hits equal those of
the uncompacted frame (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bin_of(d):
    octant = (d[:, 0] > 0).astype(int) | ((d[:, 1] > 0).astype(int) << 1) | ((d[:, 2] > 0).astype(int) << 2)
    a = np.abs(d)
    ax, ay, az = a[:, 0], a[:, 1], a[:, 2]
    major = np.where((ax >= ay) & (ax >= az), 0, np.where(ay >= az, 1, 2))
    minor = np.where((ax < ay) & (ax < az), 0, np.where(ay < az, 1, 2))
    nxt = (major + 1) % 3
    return octant * 6 + major * 2 + np.where(minor == nxt, 0, 1)


@pytest.mark.parametrize("sizes", [(1,), (1023,), (1024, 1025), (1, 2047, 0, 2049, 31), (5000, 3, 0)])
def test_chunk_edges(vx, cuda, sizes):
    import torch
    from vx_b200 import workloads as W
    bits = vx.synth_noise(64, 8, 3, 0.4, 3, True)
    scene = vx.Scene(W.scene_from_bits(bits, 64, None, 3))
    n = sum(sizes)
    rays = torch.from_numpy(W.random_rays(n, 64, seed=n)).cuda()
    begin = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()

    def buffers(m):
        return torch.zeros((m, 4), dtype=torch.int32, device="cuda")

    got = {}
    for compact in (True, False):
        batch = vx.Batch([scene] * len(sizes))
        hits, bounce, bhits = buffers(n), torch.zeros((2 * n, 6), device="cuda"), buffers(2 * n)
        torch.cuda.synchronize()
        if compact:
            batch.capture_frame_compact(rays, begin, hits, bounce, bhits, 77, stream.cuda_stream)
        else:
            batch.capture_frame(rays, begin, hits, bounce, begin * 2, bhits, 77, stream.cuda_stream)
        batch.launch_frame()
        torch.cuda.synchronize()
        got[compact] = (hits.cpu().numpy(), bhits.cpu().numpy(), bounce.cpu().numpy())
        if compact:
            scene_begin, slot = batch.frame_compaction()
    np.testing.assert_array_equal(got[True][0], got[False][0])
    np.testing.assert_array_equal(got[True][1], got[False][1])
    hit = (got[True][0].view(vx.HIT_DTYPE).reshape(-1)["flags"] & 1).astype(bool)
    edges = np.concatenate([[0], np.cumsum(sizes)])
    for s in range(len(sizes)):
        lo, hi = int(scene_begin[s]), int(scene_begin[s + 1])
        primary = np.flatnonzero(hit[edges[s]:edges[s + 1]]) + edges[s]
        assert hi - lo == 2 * primary.size
        np.testing.assert_array_equal(got[True][2][lo:hi], got[False][2][slot[lo:hi]])
        want = np.concatenate([2 * primary + k for k in (0, 1)])          # k first, then primary order ...
        chunk = (want // 2 - edges[s]) // 1024                            # ... inside a chunk,
        order = np.lexsort((np.arange(want.size), chunk, bin_of(got[False][2][want, 3:])))  # chunks inside a bin
        np.testing.assert_array_equal(slot[lo:hi], want[order])
