"""Block matching of float frames with NaN and infinite samples: the call ends,
and output samples whose search windows hold none of them equal the clean
frame's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("sub", [(1, 1), (0, 0)])
def test_samples_far_away_are_untouched(sub, value):
    fmt = S.FrameFormat(32, *sub)
    w, h = 200, 120
    planes = S.make_frame(w, h, fmt, seed=4)
    rec = lgcr.Recon(lgcr.video_format(w, h, 32, *sub), algo=2, bm=1, kernel="lanczos", taps=3, sparse=0)
    clean = rec.frame(planes, -1)
    edited = [p.copy() for p in planes]
    edited[0][40:70, 30:90] = value                  # covers whole search windows
    edited[1][5, 20] = value
    got = rec.frame(edited, -1)
    # the guided taps and maps reach less than 16 output samples, a candidate
    # patch ends 16 from its anchor and the group's patches as far again
    for p in (1, 2):
        assert np.array_equal(got[p][:, 150:], clean[p][:, 150:])
    again = rec.frame(edited, -1)
    for p in range(3):
        assert np.array_equal(got[p], again[p], equal_nan=True)
