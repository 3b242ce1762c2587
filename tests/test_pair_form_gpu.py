"""Which frames take column pairs, by the launches of a batch: the guided stage is
one launch for frames in the pixel form, two (contexts, taps) or, with jinc
frames, three (extrema before them) for pairs, and both kinds where a batch
holds both. The comparisons of the two forms rest on frames that do take
different ones."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S
from test_guided_pairs_gpu import FORMATS, KERNELS, device, outputs
from test_pair_scratch_gpu import run_batch


def launches(fmt, sizes, kw):
    recons = [lgcr.Recon(lgcr.video_format(w, h, fmt.bits, fmt.ssw, fmt.ssh), **kw) for w, h in sizes]
    frames = [device(S.make_frame(w, h, fmt, seed=3)) for w, h in sizes]
    return run_batch(recons, frames, [outputs(r, f) for r, f in zip(recons, frames)])[1][0]


@pytest.mark.parametrize("kernel", list(KERNELS))
@pytest.mark.parametrize("fmt", list(FORMATS))
def test_small_frames_pair_beside_a_large_one(fmt, kernel):
    f, jinc = FORMATS[fmt], kernel.startswith("jinc")
    kw = dict(algo=4 if jinc else 2, sparse=0, **KERNELS[kernel])
    alone, large = launches(f, [(66, 34)], kw), launches(f, [(1600, 1000)], kw)
    assert large == alone + (2 if jinc else 1)          # pixels alone, pairs
    assert launches(f, [(66, 34), (1600, 1000)], kw) == large


@pytest.mark.parametrize("kw", [dict(algo=4, kernel="jinc", taps=3, cedge=1), dict(algo=2, kernel="jinc", taps=3),
                                dict(algo=2, kernel="bilinear"), dict(algo=2, kernel="lanczos", taps=5)])
def test_frames_that_never_pair(kw):
    kw = dict(kw, sparse=0)
    assert launches(S.YUV420P10, [(1600, 1000)], kw) == launches(S.YUV420P10, [(66, 34)], kw)
