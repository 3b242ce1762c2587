"""The consensus and affine statistics of the detail transfer by tiles: two
overlapping crops of one frame agree away from their edges, a non-finite sample
changes nothing outside its windows (dense and sparse statistics), and flat
frames from below one tile up stay flat."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr

MARGIN = 48


def call(r, planes):
    f = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in planes]
    out = r.frame(f, out=[torch.empty(f[0].shape, device="cuda") for _ in range(3)])
    torch.cuda.synchronize()
    return [p.cpu().numpy() for p in out]


def scene(W, H, sw, sh, seed):
    rng = np.random.default_rng(seed)
    return [rng.random((H, W), np.float32)] + \
        [rng.random((H >> sh, W >> sw), np.float32) - np.float32(0.5) for _ in range(2)]


@pytest.mark.parametrize("sub", [(1, 1), (1, 0), (0, 1)])
@pytest.mark.parametrize("dx,dy", [(2, 0), (0, 2), (34, 66)])
def test_crops_agree(sub, dx, dy):
    sw, sh = sub
    planes = scene(300, 300, sw, sh, 11)
    w, h = 230, 230
    r = lgcr.Recon(lgcr.video_format(w, h, 32, sw, sh, True), algo=6, sparse=0, kernel="spline36")

    def at(x, y):
        return [planes[0][y:y + h, x:x + w]] + [p[y >> sh:(y + h) >> sh, x >> sw:(x + w) >> sw] for p in planes[1:]]

    a, b = call(r, at(0, 0)), call(r, at(dx, dy))
    rows, cols = slice(MARGIN + dy, h - MARGIN), slice(MARGIN + dx, w - MARGIN)
    moved = slice(MARGIN, h - MARGIN - dy), slice(MARGIN, w - MARGIN - dx)
    for p in (1, 2):
        # 32-bit positions below 256 are known to 2^-16 of a sample and the
        # planes change by at most 1 from sample to sample; ten such terms
        np.testing.assert_allclose(a[p][rows, cols], b[p][moved], rtol=0, atol=10 * 2.0 ** -16)


@pytest.mark.parametrize("sparse", [0, 1])
@pytest.mark.parametrize("sub", [(1, 1), (0, 1)])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_samples_stay_near(sub, sparse, value):
    sw, sh = sub
    w, h = 230, 130
    r = lgcr.Recon(lgcr.video_format(w, h, 32, sw, sh, True), algo=6, sparse=sparse, kernel="spline36")
    clean = scene(w, h, sw, sh, 12)
    spoiled = [p.copy() for p in clean]
    spoiled[0][64, 100] = value
    spoiled[1][64 >> sh, 100 >> sw] = value
    a, b = call(r, clean), call(r, spoiled)
    far = np.ones((h, w), bool)
    far[64 - MARGIN:64 + MARGIN, 100 - MARGIN:100 + MARGIN] = False
    for p in (0, 1, 2):
        assert np.isfinite(a[p]).all()
        np.testing.assert_array_equal(a[p][far], b[p][far])


@pytest.mark.parametrize("w,h", [(16, 8), (62, 34), (66, 64), (130, 66)])
def test_flat_frames_stay_flat(w, h):
    # constant planes: zero variances, every quotient 0 / (0 + eps)
    r = lgcr.Recon(lgcr.video_format(w, h, 32, 1, 1, True), algo=6, sparse=0, kernel="spline36")
    planes = [np.full((h, w), 0.25, np.float32)] + [np.full((h // 2, w // 2), v, np.float32) for v in (0.125, -0.375)]
    out = call(r, planes)
    for p, v in ((1, 0.125), (2, -0.375)):
        np.testing.assert_array_equal(out[p], np.full((h, w), v, np.float32))
