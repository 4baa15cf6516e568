"""The palette's output at every offset from a 16-byte boundary (needs a B200): the same colours as
the host's, nothing beside them written, and no more than half again the time of an aligned one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 1023, 1024, 1025, 2048, 70001])
def test_colours_at_every_offset(vx, cuda, n, offset):
    import torch
    words = np.random.default_rng(n).integers(0, 600, size=n, dtype=np.uint64).astype(np.uint32)
    buf = torch.full((3 * n + 8,), -5.0, dtype=torch.float32, device="cuda")
    vx.material_rgb_dev(torch.from_numpy(words.view(np.int32)).cuda(), buf[offset:offset + 3 * n])
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    want = vx.material_rgb(words).reshape(-1)
    np.testing.assert_array_equal(got[offset:offset + 3 * n].view(np.uint32), want.view(np.uint32))
    assert np.all(got[:offset] == -5.0) and np.all(got[offset + 3 * n:] == -5.0)


def test_an_offset_costs_little(vx, cuda):
    """Single stores of an output off 16 bytes took 2.6 times an aligned one's time."""
    import torch
    n = 16 << 20
    words = torch.full((n,), 33, dtype=torch.int32, device="cuda")
    buf = torch.zeros(3 * n + 4, dtype=torch.float32, device="cuda")
    best = {}
    for _ in range(8):
        for offset in (0, 1):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                vx.material_rgb_dev(words, buf[offset:offset + 3 * n])
            b.record()
            torch.cuda.synchronize()
            best[offset] = min(best.get(offset, 1e9), a.elapsed_time(b))
    assert best[1] < 1.5 * best[0], best
