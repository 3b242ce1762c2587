"""The guided pass by column pairs against the pixel form: a small frame alone
takes the pixel form, the same frame in one batch with a frame large enough
for the pair form takes pairs. Both are the same arithmetic, so the samples
are equal (integer and float, with NaN and infinite float samples too)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S

KERNELS = {"lanczos2": dict(kernel="lanczos", taps=2), "lanczos3": dict(kernel="lanczos", taps=3),
           "lanczos4": dict(kernel="lanczos", taps=4), "bicubic": dict(kernel="bicubic"),
           "spline36": dict(kernel="spline36"), "jinc2": dict(kernel="jinc", taps=2),
           "jinc3": dict(kernel="jinc", taps=3), "jinc4": dict(kernel="jinc", taps=4)}
FORMATS = {"420P10": S.YUV420P10, "420P8": S.YUV420P8, "420PS": S.YUV420PS, "422P10": S.YUV422P10,
           "444PS": S.YUV444PS}


def device(planes):
    return [torch.from_numpy(p.view(np.int16) if p.dtype == np.uint16 else p).cuda() for p in planes]


def outputs(r, f):
    return [torch.empty((r.out_h, r.out_w), dtype=f[0].dtype, device="cuda") for _ in range(3)]


def batch(recons, frames, locations):
    lib = lgcr.library()
    items = (lgcr.BatchItem * len(frames))()
    outs = [outputs(r, f) for r, f in zip(recons, frames)]
    for i, (r, f) in enumerate(zip(recons, frames)):
        items[i].filter = r.handle
        items[i].inp = lgcr.planes_desc(f)
        items[i].out = lgcr.planes_desc(outs[i])
        items[i].chroma_location = locations[i]
    handle = ctypes.c_void_p()
    assert lib.lgcr_batch_create(ctypes.byref(handle)) == 0
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    # one launch per stage over all frames, whatever their sizes
    assert lib.lgcr_batch_run(handle, items, len(frames), ctypes.c_void_p(stream.cuda_stream), 0) == 0
    stream.synchronize()
    lib.lgcr_batch_destroy(handle)
    return outs


def check(fmt, kw, sizes, location, edit=None, scale=None):
    large = lgcr.Recon(lgcr.video_format(1600, 1000, fmt.bits, fmt.ssw, fmt.ssh), **kw)
    big = device(S.make_frame(1600, 1000, fmt, seed=3))
    recons, frames = [], []
    for k, (w, h) in enumerate(sizes):
        size = dict(width=int(w * scale), height=int(h * scale)) if scale else {}
        recons.append(lgcr.Recon(lgcr.video_format(w, h, fmt.bits, fmt.ssw, fmt.ssh), **kw, **size))
        planes = S.make_frame(w, h, fmt, seed=60 + k, antialias=bool(scale))
        frames.append(device(edit(planes) if edit else planes))
    alone = []
    for r, f in zip(recons, frames):
        alone.append(r.frame(f, location, out=outputs(r, f)))
        torch.cuda.synchronize()
    mixed = batch(recons + [large], frames + [big], [location] * len(frames) + [-1])
    for a, b in zip(alone, mixed):
        for p in range(3):
            x, y = a[p], b[p]
            assert bool(((x == y) | ((x != x) & (y != y))).all())


@pytest.mark.parametrize("kernel", list(KERNELS))
@pytest.mark.parametrize("fmt", list(FORMATS))
def test_pairs_equal_pixels(fmt, kernel):
    f = FORMATS[fmt]
    sizes = [(64, 34), (66, 30), (130, 66)] if f.ssw else [(64, 33), (65, 31), (131, 66)]
    kw = dict(algo=4 if kernel.startswith("jinc") else 2, sparse=1, **KERNELS[kernel])
    check(f, kw, sizes, -1)
    check(f, dict(kw, sparse=0, algo=4), sizes[:1], -1)


@pytest.mark.parametrize("location", range(6))
@pytest.mark.parametrize("kernel", ["lanczos4", "jinc3"])
def test_sitings(kernel, location):
    check(S.YUV420P10, dict(algo=4, sparse=0, **KERNELS[kernel]), [(66, 34), (34, 18)], location)


@pytest.mark.parametrize("kernel", ["lanczos3", "jinc3"])
@pytest.mark.parametrize("scale", [0.5, 0.8, 1.5, 2.0, 2.1])
def test_resized(kernel, scale):
    algo = 4 if kernel == "jinc3" else 2
    check(S.YUV420PS, dict(algo=algo, **KERNELS[kernel]), [(66, 50), (130, 34)], -1, scale=scale)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e30])
@pytest.mark.parametrize("kernel", ["lanczos4", "jinc3"])
def test_special_samples(kernel, value):
    def edit(planes):
        planes = [p.copy() for p in planes]
        planes[0][7, 9] = value
        planes[1][5, 20] = value
        planes[2][12, 3] = value
        return planes
    check(S.YUV420PS, dict(algo=4 if kernel == "jinc3" else 2, sparse=0, **KERNELS[kernel]), [(66, 34)], -1, edit)
