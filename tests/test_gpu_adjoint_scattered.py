"""The adjoint over records that are not in runs: the same few places again and again, apart in a
warp (needs a B200).  Sums against FP64: m binary32 terms summed in any order are off by at most m
units of roundoff of the sum of their magnitudes, and a term by four roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def records(n, places, order, kind, seed):
    """Hits on `places` voxels (kind 1: blocks), in random order or in turn, a few misses between."""
    rng = np.random.default_rng(seed)
    place = rng.integers(0, places, size=n) if order == "random" else np.arange(n) % places
    brick, voxel = place // 16, place % 16 * (16 if kind else 1)
    hit = rng.random(n) < 0.95
    rec = np.zeros((n, 4), np.uint32)
    rec[:, 1] = np.where(hit, brick, 0xFFFFFFFF)
    rec[:, 3] = np.where(hit, voxel | ((1 | 16) << 16), 0xFFFF)  # face x: the Lambert factor 0.3 + 0.7 / sqrt 3
    return rec, hit, brick, voxel


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("order", ["random", "turn"])
@pytest.mark.parametrize("n,places", [(33, 1), (7, 2), (1003, 2), (1003, 3), (20011, 4), (20011, 9), (20011, 16),
                                      (20011, 31), (50021, 200)])
def test_sums_of_places_apart(vx, cuda, kind, order, n, places):
    import torch
    rng = np.random.default_rng(n + places)
    rec, hit, brick, voxel = records(n, places, order, kind, places)
    bricks = 16
    image, target = rng.random((n, 3), dtype=np.float32), rng.random((n, 3), dtype=np.float32)
    idx = rng.integers(0, 2 ** 32, size=bricks * 32, dtype=np.uint64).astype(np.uint32)
    size = bricks * 512 * 3 if kind == 0 else bricks * 32 * 6
    g = 2.0 * (image.astype(np.float64) - target) * (0.3 + 0.7 / np.sqrt(3.0))
    want, mag, cnt = np.zeros(size), np.zeros(size), np.zeros(size)
    for ch in range(3):
        if kind == 0:
            terms = [((brick * 512 + voxel) * 3 + ch, g[:, ch])]
        else:
            block = brick * 32 + (voxel >> 4)
            w = np.array([1, 0, 2 / 3, 1 / 3])[(idx[block] >> (2 * (voxel & 15)).astype(np.uint32)) & 3]
            terms = [(block * 6 + ch, w * g[:, ch]), (block * 6 + 3 + ch, (1 - w) * g[:, ch])]
        for at, v in terms:
            np.add.at(want, at[hit], v[hit])
            np.add.at(mag, at[hit], np.abs(v[hit]))
            np.add.at(cnt, at[hit], 1)
    d = [torch.from_numpy(a).cuda() for a in (idx.view(np.int32), rec.view(np.int32), image, target)]
    for offset in (0, 1):
        grad = torch.zeros(size + 2, device="cuda")
        vx.diff_backward(kind, d[0], d[1], d[2], d[3], grad[offset:offset + size])
        torch.cuda.synchronize()
        got = grad[offset:offset + size].cpu().numpy().astype(np.float64)
        assert np.all(np.abs(got - want) <= (cnt + 4) * 2.0 ** -23 * mag)


def test_places_in_turn_cost_no_more_than_runs(vx, cuda):
    """Pixels that hit two voxels in turn, eight voxels in all, against the same pixels in runs of
    nine: without adding the turns up first, eleven times the time (the reductions of a warp queue at
    two addresses); with it, less."""
    import torch
    n = 2000000
    i = np.arange(n)
    image = torch.rand((n, 3), device="cuda")
    target = torch.rand((n, 3), device="cuda")
    grad = torch.zeros(16 * 512 * 3, device="cuda")
    times = []
    for place in (i // 9 % 8, (i // 64 * 2 + i % 2) % 8):
        rec = np.zeros((n, 4), np.uint32)
        rec[:, 3] = place | ((1 | 16) << 16)
        d = torch.from_numpy(rec.view(np.int32)).cuda()
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                vx.diff_backward(0, None, d, image, target, grad)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] < 3.0 * times[0]
