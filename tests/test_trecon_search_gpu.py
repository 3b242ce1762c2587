"""TRecon block matching at the edges of its two forms: search windows up to
tsearch 42 are staged in shared memory, wider ones are read from the plane.
On clips of whole-sample motion within the smaller range both find the same
motion, so the frames are equal; sizes leave partial blocks on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S
from trecon_seq import make_clip

MOTIONS = [(0, 0), (2, -1), (-3, 2)]
CASES = [("420P10", S.YUV420P10, 98, 66), ("422P10", S.YUV422P10, 50, 35),
         ("444P8", S.FrameFormat(8, 0, 0), 33, 17), ("420PS", S.YUV420PS, 64, 48)]


@pytest.mark.parametrize("name,fmt,w,h", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("trad", [1, 2])
def test_staged_and_direct_search_agree(name, fmt, w, h, trad):
    clip = [tuple(np.ascontiguousarray(p) for p in f) for f in make_clip(w, h, fmt, MOTIONS, seed=31, noise=0.0)]
    out = []
    for search in (42, 43):
        tr = lgcr.TRecon(lgcr.video_format(w, h, fmt.bits, fmt.ssw, fmt.ssh), len(clip), trad=trad,
                         tsearch=search)
        out.append([tr.frame(n, lambda i: clip[i]) for n in range(len(clip))])
    for a, b in zip(*out):
        for p in range(3):
            assert np.array_equal(a[p], b[p])
