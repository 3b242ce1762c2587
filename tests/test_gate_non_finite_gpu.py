"""Non-finite samples in the middle of a float frame: the gate's sample
positions stay inside its tile, and samples out of reach are unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr


@pytest.mark.parametrize("algo,sparse", [(2, 0), (2, 1), (6, 0)])
@pytest.mark.parametrize("plane", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_far_samples_unchanged(value, plane, algo, sparse):
    w, h, reach = 642, 514, 48
    rng = np.random.default_rng(21)
    clean = [rng.random((h, w), np.float32)] + [rng.random((h // 2, w // 2), np.float32) - np.float32(0.5) for _ in range(2)]
    r = lgcr.Recon(lgcr.video_format(w, h, 32, 1, 1, True), algo=algo, sparse=sparse, kernel="spline36")

    def call(planes):
        f = [torch.from_numpy(p).cuda() for p in planes]
        out = r.frame(f, out=[torch.empty((h, w), device="cuda") for _ in range(3)])
        torch.cuda.synchronize()
        return [p.cpu().numpy() for p in out]

    spoiled = [p.copy() for p in clean]
    s = 1 if plane else 0
    spoiled[plane][300 >> s, 400 >> s] = value
    a, b = call(clean), call(spoiled)
    far = np.ones((h, w), bool)
    far[300 - reach:300 + reach, 400 - reach:400 + reach] = False
    for p in range(3):
        np.testing.assert_array_equal(a[p][far], b[p][far])
