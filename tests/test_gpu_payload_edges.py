"""Payload encoders on the device against the host ones, bit for bit, where the device forms
part from them: the normal encoder's tables of results (runs of equal blocks, no two equal, more
bricks than one per warp, two streams at once), the DXT1 encoder's paired searches (ties, equal
texels, infinities and NaN, colours off 16-byte alignment), the palette's vector stores (ragged
ends, ids of both tables) (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def normal_bricks(n, seed):
    """Solid, empty, layered, sparse and random bricks in runs."""
    rng = np.random.default_rng(seed)
    occ = rng.integers(0, 2 ** 32, size=(n, 16), dtype=np.uint64).astype(np.uint32)
    kind = np.repeat(rng.integers(0, 6, size=n // 7 + 1), 7)[:n]
    occ[kind == 0] = 0xFFFFFFFF
    occ[kind == 1] = 0
    occ[kind == 2] &= rng.integers(0, 2 ** 32, size=(int((kind == 2).sum()), 16), dtype=np.uint64).astype(np.uint32)
    occ[kind == 3, 8:] = 0
    occ[kind == 3, :8] = 0xFFFFFFFF
    occ[kind == 4] = np.uint32(0x0F0F0F0F)
    return occ


@pytest.mark.parametrize("n", [1, 31, 2369, 8191, 8192, 16383, 16384, 30011])
def test_normals_with_result_tables(vx, cuda, n):
    import torch
    occ = normal_bricks(n, n)
    o = torch.from_numpy(occ.view(np.int32)).cuda()
    out = torch.full((n * 64,), -1, dtype=torch.int64, device="cuda")
    want = vx.build_normals(occ).reshape(-1)
    for _ in range(2):
        vx.build_normals_dev(o, out)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)


def test_normals_on_two_streams(vx, cuda):
    import torch
    sets = [normal_bricks(20000, s) for s in (1, 2)]
    dev = [torch.from_numpy(o.view(np.int32)).cuda() for o in sets]
    outs = [torch.zeros(20000 * 64, dtype=torch.int64, device="cuda") for _ in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    for _ in range(8):
        for d, o, s in zip(dev, outs, streams):
            vx.build_normals_dev(d, o, s.cuda_stream)
    torch.cuda.synchronize()
    for occ, o in zip(sets, outs):
        np.testing.assert_array_equal(o.cpu().numpy().view(np.uint64), vx.build_normals(occ).reshape(-1))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 5, 1203])
def test_dxt1_pairs(vx, cuda, n, offset):
    import torch
    rng = np.random.default_rng(n)
    rgb = rng.random((n, 32, 16, 3)).astype(np.float32)
    kind = rng.integers(0, 8, size=(n, 32))
    rgb[kind == 0] = np.float32(0.25)                                     # all texels alike
    rgb[kind == 1] = rng.choice(np.array([0.0, 0.5, 1.0], np.float32), size=(int((kind == 1).sum()), 16, 3))  # ties
    rgb[kind == 2] = np.round(rgb[kind == 2] * 4) / 4
    for k, v in ((3, np.inf), (4, np.nan), (5, -np.inf), (6, 3e38)):
        where = (kind == k)[..., None, None] & (rng.random((n, 32, 16, 3)) < 0.15)
        rgb[where] = v
    occ = rng.integers(0, 2 ** 32, size=(n, 16), dtype=np.uint64).astype(np.uint32)
    occ[rng.random((n, 16)) < 0.3] = 0xFFFFFFFF
    occ[rng.random((n, 16)) < 0.1] = 0
    buf = torch.zeros(n * 1536 + 4, dtype=torch.float32, device="cuda")
    d_rgb = buf[offset:offset + n * 1536]
    d_rgb.copy_(torch.from_numpy(rgb.reshape(-1)))
    out = torch.zeros(n * 32, dtype=torch.int64, device="cuda")
    vx.build_dxt1_dev(d_rgb, torch.from_numpy(occ.view(np.int32)).cuda(), out)
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        want = vx.build_dxt1(rgb.reshape(n, 512, 3), occ)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 5 * 1024 + 3, 400001])
def test_material_colours(vx, cuda, n, offset):
    import torch
    rng = np.random.default_rng(n)
    words = rng.integers(0, 70, size=n, dtype=np.uint64).astype(np.uint32)
    words[rng.random(n) < 0.2] = rng.integers(0, 2 ** 32, dtype=np.uint64)
    words[:: 7] = rng.integers(0, 1024, size=words[::7].size)
    buf = torch.full((3 * n + 8,), -5.0, dtype=torch.float32, device="cuda")
    d_words = torch.zeros(n + 1, dtype=torch.int32, device="cuda")[offset % 2:][:n]
    d_words.copy_(torch.from_numpy(words.view(np.int32)))
    vx.material_rgb_dev(d_words, buf[offset:offset + 3 * n])
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + 3 * n].view(np.uint32), vx.material_rgb(words).reshape(-1).view(np.uint32))
    assert np.all(got[:offset] == -5.0) and np.all(got[offset + 3 * n:] == -5.0)
