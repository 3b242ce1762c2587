"""The fused detail map's tiles (30 columns, 62 or 30 rows, rows in pairs): two
overlapping crops of one frame put the same samples at other places of the
tiles and row pairs; away from the crops' edges their outputs agree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr

KERNELS = {"lanczos4": dict(kernel="lanczos", taps=4), "spline36": dict(kernel="spline36"),
           "bicubic": dict(kernel="bicubic"), "lanczos2": dict(kernel="lanczos", taps=2)}
MARGIN = 48             # beyond the windows of the base, the detail map and the transfer


def crop(planes, x, y, w, h, sw, sh):
    return [torch.from_numpy(np.ascontiguousarray(planes[0][y:y + h, x:x + w])).cuda()] + \
        [torch.from_numpy(np.ascontiguousarray(p[y >> sh:(y + h) >> sh, x >> sw:(x + w) >> sw])).cuda()
         for p in planes[1:]]


@pytest.mark.parametrize("dx,dy", [(2, 2), (30, 0), (0, 62), (28, 30), (16, 34)])
@pytest.mark.parametrize("sub", [(1, 1), (1, 0)])
@pytest.mark.parametrize("kernel", list(KERNELS))
def test_crops_agree(kernel, sub, dx, dy):
    sw, sh = sub
    rng = np.random.default_rng(3)
    W, H, w, h = 260, 300, 226, 230
    planes = [rng.random((H, W), np.float32)] + \
        [rng.random((H >> sh, W >> sw), np.float32) - np.float32(0.5) for _ in range(2)]
    r = lgcr.Recon(lgcr.video_format(w, h, 32, sw, sh, True), algo=6, sparse=0, **KERNELS[kernel])

    def call(x, y):
        f = crop(planes, x, y, w, h, sw, sh)
        out = r.frame(f, out=[torch.empty((h, w), device="cuda") for _ in range(3)])
        torch.cuda.synchronize()
        return [p.cpu().numpy() for p in out]

    a, b = call(0, 0), call(dx, dy)
    rows, cols = slice(MARGIN + dy, h - MARGIN), slice(MARGIN + dx, w - MARGIN)
    moved = slice(MARGIN, h - MARGIN - dy), slice(MARGIN, w - MARGIN - dx)
    for p in (1, 2):
        # 32-bit positions below 256 are known to 2^-16 of a sample and the
        # planes change by at most 1 from sample to sample; ten such terms
        np.testing.assert_allclose(a[p][rows, cols], b[p][moved], rtol=0, atol=10 * 2.0 ** -16)
