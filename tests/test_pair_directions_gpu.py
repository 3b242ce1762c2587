"""Column pairs whose direction is not finite: a NaN, infinite or overflowing
luma sample makes the smoothed tensor of its neighbours NaN, and with it the
bump term of the taps. The pixel form multiplies that term by a rescue weight
of zero where the column has none, which is NaN (the sample falls back to the
bilinear one); the pair form must come to the same sample. With ms = 0 the
mutual gate, which is NaN there too, does not hide the difference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from lgcr import synthetic as S
from test_guided_pairs_gpu import check

KERNELS = {"lanczos2": dict(algo=2, kernel="lanczos", taps=2), "lanczos4": dict(algo=2, kernel="lanczos", taps=4),
           "jinc2": dict(algo=4, kernel="jinc", taps=2), "jinc3": dict(algo=4, kernel="jinc", taps=3)}
FORMATS = {"420": (1, 1), "422": (1, 0), "444": (0, 0)}


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30])
@pytest.mark.parametrize("sub", list(FORMATS))
@pytest.mark.parametrize("kernel", list(KERNELS))
def test_directions_that_are_not_finite(kernel, sub, value):
    def edit(planes):
        planes = [p.copy() for p in planes]
        for y, x in ((7, 9), (8, 24), (19, 40), (26, 51)):   # both parities of row and column
            planes[0][y, x] = value
        return planes
    check(S.FrameFormat(32, *FORMATS[sub]), dict(KERNELS[kernel], sparse=0, ms=0.0), [(74, 34)], -1, edit)
