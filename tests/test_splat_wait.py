"""SphContext.splat returns finished images, also on torch's default stream, while the context still has steps queued."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("own_stream", [False, True])
def test_splat_waits_for_the_images(sphlib, own_stream):
    torch = pytest.importorskip("torch")
    n = 100 ** 3
    box = (3.0, 3.0, 3.0)
    pos = sphlib.dam_break_scene((100, 100, 100), box, 1)
    ctx = sphlib.SphContext(box, n)
    ctx.upload(pos)
    with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
        for _ in range(6):
            torch.full((480, 640), 7, dtype=torch.int32, device="cuda")  # (memory that the images may take over)
            ctx.step(3)
            cnt, dep = ctx.splat(0, 2, 640, 480)
            assert int(cnt.sum()) == n
            x = ctx.download()["pos"]
            px = [np.clip(np.floor((x[:, a] + np.float32(b / 2)) * np.float32(k / b)), 0, k - 1).astype(int)
                  for a, b, k in ((0, 3.0, 640), (1, 3.0, 480))]
            want = np.bincount(px[1] * 640 + px[0], minlength=640 * 480).reshape(480, 640)
            assert np.array_equal(cnt, want)
            assert np.array_equal(np.isfinite(dep), want > 0)
    ctx.close()
