"""The adjoint's run sums against an FP64 sum of the same records (needs a B200): runs of every
length, across warp edges, misses between them, ragged ends, gradients on and off 8-byte
alignment, with and without the loss.  Tolerance: m binary32 terms summed in any order are off by
at most m units of roundoff of the sum of their magnitudes, and a term by four roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A = 1.0 / np.sqrt(3.0)


def records(n, longest, bricks, seed):
    rng = np.random.default_rng(seed)
    lengths = rng.integers(1, longest + 1, size=n)
    run = np.repeat(np.arange(n), lengths)[:n]
    brick, voxel = rng.integers(0, bricks, size=n)[run], rng.integers(0, 512, size=n)[run]
    if longest > 32:
        voxel[: n // 2] = 7
        brick[: n // 2] = 1
    hit = (rng.random(n) < 0.85)[run]
    axis, neg = rng.integers(0, 3, size=n), rng.integers(0, 2, size=n)
    rec = np.zeros((n, 4), np.uint32)
    rec[:, 1] = np.where(hit, brick, 0xFFFFFFFF)
    rec[:, 2] = rec[:, 1]
    flags = 1 | (axis << 1) | (neg << 3)
    rec[:, 3] = np.where(hit, voxel | (flags << 16), 0xFFFF)
    return rec, hit, brick, voxel, axis, neg


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n,longest", [(1, 1), (31, 3), (33, 40), (257, 2), (4099, 9), (100003, 70), (700001, 3)])
def test_run_sums(vx, cuda, kind, n, longest):
    import torch
    rng = np.random.default_rng(n + kind)
    bricks = 37
    rec, hit, brick, voxel, axis, neg = records(n, longest, bricks, n)
    image, target = rng.random((n, 3), dtype=np.float32), rng.random((n, 3), dtype=np.float32)
    idx = rng.integers(0, 2 ** 32, size=bricks * 32, dtype=np.uint64).astype(np.uint32)
    size = bricks * 512 * 3 if kind == 0 else bricks * 32 * 6
    facing = np.where(neg == 1, -1.0, 1.0) * np.array([A, A, -A])[axis]
    g = 2.0 * (image.astype(np.float64) - target) * (0.3 + 0.7 * np.maximum(facing, 0.0))[:, None]
    want, mag, cnt = np.zeros(size), np.zeros(size), np.zeros(size)

    def add(at, v):
        np.add.at(want, at[hit], v[hit])
        np.add.at(mag, at[hit], np.abs(v[hit]))
        np.add.at(cnt, at[hit], 1)

    for ch in range(3):
        if kind == 0:
            add((brick * 512 + voxel) * 3 + ch, g[:, ch])
        else:
            block = brick * 32 + (voxel >> 4)
            sel = (idx[block] >> (2 * (voxel & 15)).astype(np.uint32)) & 3
            add(block * 6 + ch, np.array([1, 0, 2 / 3, 1 / 3])[sel] * g[:, ch])
            add(block * 6 + 3 + ch, np.array([0, 1, 1 / 3, 2 / 3])[sel] * g[:, ch])
    bound = (cnt + 4) * 2.0 ** -23 * mag
    d = [torch.from_numpy(a).cuda() for a in (idx.view(np.int32), rec.view(np.int32), image, target)]
    for offset in (0, 1):
        grad = torch.zeros(size + 2, device="cuda")
        loss = torch.zeros(1, device="cuda") if offset == 0 else None
        vx.diff_backward(kind, d[0], d[1], d[2], d[3], grad[offset:offset + size], loss)
        torch.cuda.synchronize()
        got = grad[offset:offset + size].cpu().numpy().astype(np.float64)
        assert np.all(np.abs(got - want) <= bound)
        if loss is not None:
            ref = float(((image.astype(np.float64) - target) ** 2).sum())
            assert abs(float(loss) - ref) <= (3 * n + 4) * 2.0 ** -23 * ref
