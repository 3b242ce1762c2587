"""The plain stage by row pairs: a small frame alone is evaluated one output row
at a time, the same frame in one batch with a large one in pairs of rows. Both
give the same samples (odd heights, windows 0, 1 and more rows apart, clamped
taps, listed pixels, NaN and infinite float samples), and finite float frames
are the separable sums of the axis tables."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr

KERNELS = {"lanczos3": dict(kernel="lanczos", taps=3), "lanczos4": dict(kernel="lanczos", taps=4),
           "bicubic": dict(kernel="bicubic"), "bilinear": dict(kernel="bilinear")}
# width, height, subsampling (w, h), output size
GEOMETRY = [(70, 18, 1, 1, 70, 18), (134, 131, 1, 0, 134, 131), (66, 35, 0, 0, 132, 71), (66, 50, 0, 0, 99, 75),
            (130, 131, 0, 0, 97, 65), (200, 130, 1, 1, 70, 37)]


def axis(r, which, n):
    lib = lgcr.library()
    lib.lgcr_debug_axis.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_double] + [ctypes.c_void_p] * 9 + \
        [ctypes.POINTER(ctypes.c_int)]
    sup = ctypes.c_int()
    lib.lgcr_debug_axis(r.handle, which, 0.0, *[None] * 9, ctypes.byref(sup))
    start, w = np.zeros(n, np.int32), np.zeros((n, sup.value), np.float32)
    act = np.zeros((n, sup.value), np.uint8)
    lib.lgcr_debug_axis(r.handle, which, 0.0, start.ctypes.data, w.ctypes.data, act.ctypes.data, *[None] * 6,
                        ctypes.byref(sup))
    return start, w.astype(np.float64) * (act != 0), act != 0


def separable(r, plane):
    """Normalised separable sums held to the hull of the active taps, in 64 bits (horizontal sums rounded to 32)."""
    h, w = plane.shape
    xs, wx, ax = axis(r, 0, r.out_w)
    ys, wy, ay = axis(r, 1, r.out_h)
    xi = np.clip(xs[:, None] + np.arange(wx.shape[1]), 0, w - 1)
    yi = np.clip(ys[:, None] + np.arange(wy.shape[1]), 0, h - 1)
    p = plane.astype(np.float64)
    rows = np.einsum("hxi,xi->hx", p[:, xi], wx).astype(np.float32).astype(np.float64)
    v = np.einsum("yjx,yj->yx", rows[yi], wy)
    sums = wy.sum(1)[:, None] * wx.sum(1)[None]
    lo = np.where(ax, p[:, xi], np.inf).min(2)
    hi = np.where(ax, p[:, xi], -np.inf).max(2)
    lo = np.where(ay[:, :, None], lo[yi], np.inf).min(1)
    hi = np.where(ay[:, :, None], hi[yi], -np.inf).max(1)
    assert (sums > 0.05 * np.abs(wy).sum(1)[:, None] * np.abs(wx).sum(1)[None]).all()
    return np.clip(v / sums, lo, hi)


def run(recons, frames):
    lib = lgcr.library()
    items = (lgcr.BatchItem * len(frames))()
    outs = [[torch.empty((r.out_h, r.out_w), dtype=f[0].dtype, device="cuda") for _ in range(3)]
            for r, f in zip(recons, frames)]
    for i, (r, f) in enumerate(zip(recons, frames)):
        items[i].filter, items[i].inp, items[i].out = r.handle, lgcr.planes_desc(f), lgcr.planes_desc(outs[i])
        items[i].chroma_location = 1
    handle = ctypes.c_void_p()
    assert lib.lgcr_batch_create(ctypes.byref(handle)) == 0
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    assert lib.lgcr_batch_run(handle, items, len(frames), ctypes.c_void_p(stream.cuda_stream), 1) == 0
    stream.synchronize()
    lib.lgcr_batch_destroy(handle)
    return [[p.cpu().numpy() for p in o] for o in outs]


def frame(w, h, sw, sh, seed, special=False):
    rng = np.random.default_rng(seed)
    planes = [rng.random((h, w), np.float32)] + \
        [(rng.random(((h + sh) >> sh, (w + sw) >> sw), np.float32) - 0.5) for _ in range(2)]
    if special:
        for p in planes[1:]:
            p[rng.integers(p.shape[0]), rng.integers(p.shape[1])] = np.nan
            p[rng.integers(p.shape[0]), rng.integers(p.shape[1])] = np.inf
            p[rng.integers(p.shape[0]), rng.integers(p.shape[1])] = -3e38
    return [torch.from_numpy(p).cuda() for p in planes]


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("algo,strength", [(2, 0.0), (2, 0.8), (4, 0.8), (6, 0.8)])
@pytest.mark.parametrize("kernel", list(KERNELS))
def test_pairs_equal_single_rows_and_the_separable_sums(kernel, algo, strength, special):
    for i, (w, h, sw, sh, ow, oh) in enumerate(GEOMETRY):
        kw = dict(algo=algo, strength=strength, width=ow, height=oh, **KERNELS[kernel])
        small = lgcr.Recon(lgcr.video_format(w, h, 32, sw, sh, True), **kw)
        large = lgcr.Recon(lgcr.video_format(3840, 2160, 32, 1, 1, True), algo=algo, strength=strength,
                           **KERNELS[kernel])
        f = frame(w, h, sw, sh, 7 * i + 1, special)
        alone = run([small], [f])[0]
        beside = run([small, large], [f, frame(3840, 2160, 1, 1, 5)])[0]
        for a, b in zip(alone, beside):
            np.testing.assert_array_equal(a, b)
        if strength == 0.0 and not special and kernel != "bilinear":   # (interpolated in 32 bits, without the sums)
            for p in (1, 2):
                plane = f[p].cpu().numpy()
                want = separable(small, plane)
                # a row sum can round to the next 32-bit value: 2^-23 of it, of
                # samples up to 0.5 and absolute weights up to twice their sum
                # on either axis, so 2^-23 * 0.5 * 2 * 2; twice that, and the
                # rounding of the result
                assert np.abs(alone[p] - want).max() <= 2 * 2.0 ** -22 + 2.0 ** -24
