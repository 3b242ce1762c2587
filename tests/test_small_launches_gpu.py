"""The work split of small launches and the chained stage launches: a frame
alone (short walks), the same frame in a batch with larger ones (long walks)
and many calls in flight on two streams give the same samples. Sizes leave
partial strips, words and tiles."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S


def device(planes):
    return [torch.from_numpy(p.view(np.int16) if p.dtype == np.uint16 else p).cuda() for p in planes]


def batch(recons, frames):
    lib = lgcr.library()
    items = (lgcr.BatchItem * len(frames))()
    outs = []
    for i, (r, f) in enumerate(zip(recons, frames)):
        outs.append([torch.empty((r.out_h, r.out_w), dtype=f[0].dtype, device="cuda") for _ in range(3)])
        items[i].filter = r.handle
        items[i].inp = lgcr.planes_desc(f)
        items[i].out = lgcr.planes_desc(outs[-1])
        items[i].chroma_location = -1
    handle = ctypes.c_void_p()
    assert lib.lgcr_batch_create(ctypes.byref(handle)) == 0
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    assert lib.lgcr_batch_run(handle, items, len(frames), ctypes.c_void_p(stream.cuda_stream), 1) == 0
    stream.synchronize()
    lib.lgcr_batch_destroy(handle)
    return outs


@pytest.mark.parametrize("algo", [2, 4, 6])
@pytest.mark.parametrize("w,h", [(34, 18), (226, 66), (418, 130)])
def test_alone_batched_and_in_flight(algo, w, h):
    fmt = S.YUV420P10
    kw = dict(algo=algo, kernel="lanczos", taps=3)
    small = lgcr.Recon(lgcr.video_format(w, h, 10, 1, 1), **kw)
    large = lgcr.Recon(lgcr.video_format(1920, 1080, 10, 1, 1), **kw)
    frames = [device(S.make_frame(w, h, fmt, seed=40 + i)) for i in range(3)]
    big = device(S.make_frame(1920, 1080, fmt, seed=50))

    def call(f, stream=None):
        out = [torch.empty((h, w), dtype=f[0].dtype, device="cuda") for _ in range(3)]
        return small.frame(f, out=out, stream=stream)

    alone = []
    for f in frames:
        alone.append(call(f))
        torch.cuda.synchronize()
    mixed = batch([small] * 3 + [large], frames + [big])[:3]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    flying = [[call(f, streams[(i + k) % 2]) for i, f in enumerate(frames)] for k in range(8)]
    torch.cuda.synchronize()
    for i in range(3):
        for p in range(3):
            assert torch.equal(alone[i][p], mixed[i][p])
            for run in flying:
                assert torch.equal(alone[i][p], run[i][p])
