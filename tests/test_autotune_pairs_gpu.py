"""What the autotuners report of the guided stage: variants belong to the pixel
form, so they are timed where a frame of the layout takes it, and a layout
whose frames all take column pairs says so and keeps its settings."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S
from test_guided_pairs_gpu import device, outputs

PAIRS, PIXELS = (1600, 1000), (320, 180)       # of a launch by itself


@pytest.mark.parametrize("process_wide", [False, True])
@pytest.mark.parametrize("sizes,pixel_form", [([PAIRS], False), ([PIXELS], True)])
def test_report_names_what_ran(sizes, pixel_form, process_wide):
    lib = lgcr.library()
    kw = dict(algo=2, kernel="lanczos", taps=4)
    recons = [lgcr.Recon(lgcr.video_format(w, h, 10, 1, 1), **kw) for w, h in sizes]
    frames = [device(S.make_frame(w, h, S.YUV420P10, seed=5)) for w, h in sizes]
    outs = [outputs(r, f) for r, f in zip(recons, frames)]
    items = (lgcr.BatchItem * len(sizes))()
    for i in range(len(sizes)):
        items[i].filter = recons[i].handle
        items[i].inp = lgcr.planes_desc(frames[i])
        items[i].out = lgcr.planes_desc(outs[i])
        items[i].chroma_location = -1
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    report = ctypes.create_string_buffer(8192)
    if process_wide:
        status = lib.lgcr_autotune(items, len(sizes), ctypes.c_void_p(stream.cuda_stream), report, 8192)
    else:
        handle = ctypes.c_void_p()
        assert lib.lgcr_batch_create(ctypes.byref(handle)) == 0
        status = lib.lgcr_batch_autotune(handle, items, len(sizes), ctypes.c_void_p(stream.cuda_stream), report, 8192)
        lib.lgcr_batch_destroy(handle)
    assert status == 0, lib.lgcr_last_error().decode()
    line = [l for l in report.value.decode().splitlines() if l.startswith("reconstructChroma:")]
    assert len(line) == 1
    if pixel_form:
        assert "2-blocks=" in line[0] and "staged=" in line[0], line
    else:
        assert line[0] == "reconstructChroma: column pairs", line
