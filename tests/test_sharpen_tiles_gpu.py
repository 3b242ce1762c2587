"""Sharpen against a plain torch float32 evaluation of the same filter at the
edges of its tiles (32 x 16 samples) and planes, for the self-guided planes of
4:4:4 and for luma; the last case's similarity denominators leave the fast
reciprocal's range (2^64).

Tolerance: a sample is c0 + alpha * hp / wsum with |hp / wsum| at most the
window's range R. Sums of 24 float products in another order, reciprocals and
quotients rounded once each: relative error of hp and wsum within 30 * 2^-24
of sum n |c0 - s| and sum n, so alpha * R * 2 * 30 * 2^-24, plus two roundings
of the result: 2^-23 * (|c0| + R)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr


def sharpen_plane(s, alpha=0.3, sigma=0.01, sratio=0.15, g=1.2):
    h, w = s.shape
    p = torch.nn.functional.pad(s[None, None], (2, 2, 2, 2), mode="replicate")[0, 0]
    at = lambda j, i: p[2 + j:2 + j + h, 2 + i:2 + i + w]
    window = torch.stack([at(j, i) for j in range(-2, 3) for i in range(-2, 3)])
    reach = (window - s).abs().amax(0)
    step = torch.stack([(at(j, i) - s).abs() for j, i in ((0, 1), (0, -1), (1, 0), (-1, 0))]).sort(0).values
    sig = torch.maximum(torch.clamp(sratio * reach, min=sigma), 3.0 * 0.5 * (step[1] + step[2]))
    hp, total = torch.zeros_like(s), torch.zeros_like(s)
    for j in range(-2, 3):
        for i in range(-2, 3):
            if i or j:
                d = at(j, i) - s
                n = 1.0 / (1.0 + (i * i + j * j) / (g * g)) / (1.0 + d * d / (sig * sig))
                hp, total = hp - n * d, total + n
    out = torch.where(total > 1e-6, s + alpha * hp / total, s)
    return torch.minimum(torch.maximum(out, window.amin(0)), window.amax(0)), window.amax(0) - window.amin(0)


@pytest.mark.parametrize("w,h", [(1, 1), (31, 15), (32, 16), (33, 17), (67, 35)])
@pytest.mark.parametrize("scale,sigma", [(1.0, 0.01), (1e12, 1e-3)])
def test_tiles_against_torch(w, h, scale, sigma):
    rng = np.random.default_rng(w * 100 + h)
    planes = [(scale * rng.random((h, w))).astype(np.float32) for _ in range(3)]
    if scale > 1:                                # flat areas with one spike: sigma stays small
        planes = [np.zeros((h, w), np.float32) for _ in range(3)]
        planes[0][h // 2, w // 2] = scale
    kw = dict(sigma=sigma, sratio=0.15 if scale == 1.0 else 1e-20)
    got = lgcr.Sharpen(lgcr.video_format(w, h, 32, 0, 0), alpha=0.3, **kw).frame(planes)
    for p in range(3):
        s = torch.from_numpy(planes[p])
        ref, span = sharpen_plane(s, sigma=np.float32(kw["sigma"]), sratio=np.float32(kw["sratio"]))
        bound = 0.3 * span * 2 * 30 * 2.0 ** -24 + 2.0 ** -23 * (s.abs() + span)
        assert bool(((torch.from_numpy(got[p]) - ref).abs() <= bound + 1e-30).all())
