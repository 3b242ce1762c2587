"""Device memory of the guided pass by column pairs, and its chunks.

A frame's workspace holds the same planes whether or not the frame may take
pairs; what the pair form's kernels hand on lives in one scratch per launch,
whose size does not follow the number of frames. A launch with more list
entries than the scratch holds goes through it chunk by chunk, with the same
samples."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

import lgcr
from lgcr import synthetic as S
from test_guided_pairs_gpu import device, outputs

ENTRIES = 8 << 20                       # most entries of the scratch (PairScratch::kMost)


def scratch(pairs, jinc):
    """Bytes of the scratch of one launch with that many column pairs."""
    return min(pairs, ENTRIES) * (112 if jinc else 64)


def run_batch(recons, frames, outs):
    lib = lgcr.library()
    items = (lgcr.BatchItem * len(frames))()
    for i, (r, f) in enumerate(zip(recons, frames)):
        items[i].filter = r.handle
        items[i].inp = lgcr.planes_desc(f)
        items[i].out = lgcr.planes_desc(outs[i])
        items[i].chroma_location = -1
    handle = ctypes.c_void_p()
    assert lib.lgcr_batch_create(ctypes.byref(handle)) == 0
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    launches = []
    for _ in range(2):
        assert lib.lgcr_batch_run(handle, items, len(frames), ctypes.c_void_p(stream.cuda_stream), 0) == 0, \
            lib.lgcr_last_error().decode()
        launches.append(lib.lgcr_batch_launch_count(handle))
    stream.synchronize()
    free = torch.cuda.mem_get_info()[0]
    lib.lgcr_batch_destroy(handle)
    return free, launches


# filter, source size, output scale, bytes of a workspace's planes per output
# pixel (rounded up: converted planes, tensor, masks, list, float outputs,
# (u, v) pairs; separable kernels 16 for the horizontal table and 24 for the
# window extrema, the selector 6 per source pixel), whether the frames pair
FILTERS = {"jinc selector 2x": (dict(algo=4, kernel="jinc", taps=3), (960, 540), 2, 22, True),
           "jinc guided 2x": (dict(algo=2, kernel="jinc", taps=3), (960, 540), 2, 22, False),
           "jinc selector, chroma edges": (dict(algo=4, kernel="jinc", taps=3, cedge=1), (1920, 1080), 1, 45, False),
           "lanczos guided": (dict(algo=2, kernel="lanczos", taps=4), (1920, 1080), 1, 79, True),
           "lanczos selector": (dict(algo=4, kernel="lanczos", taps=4), (1920, 1080), 1, 85, True)}


@pytest.mark.parametrize("name", list(FILTERS))
def test_workspaces_hold_their_planes_alone(name):
    kw, (w, h), scale, per_pixel, pair = FILTERS[name]
    if scale != 1:
        kw = dict(kw, width=scale * w, height=scale * h)
    count = 24
    planes = device(S.make_frame(w, h, S.YUV420P10, seed=8))
    taken = []
    for n in (1, 1, 1 + count):         # the first loads the kernels
        rec = lgcr.Recon(lgcr.video_format(w, h, 10, 1, 1), **kw)
        outs = [outputs(rec, planes) for _ in range(n)]
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        after, _ = run_batch([rec] * n, [planes] * n, outs)
        taken.append(before - after)
        del rec
    pixels = w * h * scale * scale
    # 2 MiB: an allocation's granule; upscaling frames take a launch each
    limit = count * (per_pixel * pixels + (2 << 20))
    if pair and scale == 1:
        limit += scratch((1 + count) * pixels // 2, kw["kernel"] == "jinc")
    assert taken[2] - taken[1] <= limit, ((taken[2] - taken[1]) / count / pixels, taken)


@pytest.mark.parametrize("kernel", [dict(kernel="lanczos", taps=3, algo=2), dict(kernel="jinc", taps=3, algo=4)])
@pytest.mark.parametrize("fmt", [S.YUV420P8, S.YUV420PS])
def test_chunks_give_the_same_samples(kernel, fmt):
    """Frames of one launch in more chunks than one, the chunk borders inside
    frames; each frame in a launch of its own takes one chunk."""
    w, h = 1502, 1002
    kw = dict(kernel, sparse=0)
    pairs = w // 2 * h
    n = 2 * ENTRIES // pairs + 1
    assert pairs < ENTRIES < 2 * ENTRIES < n * pairs
    rec = lgcr.Recon(lgcr.video_format(w, h, fmt.bits, 1, 1), **kw)
    some = [device(S.make_frame(w, h, fmt, seed=90 + k)) for k in range(3)]
    frames = [some[k % 3] for k in range(n)]
    alone, mixed = [outputs(rec, f) for f in some], [outputs(rec, f) for f in frames]
    single = [run_batch([rec], [f], [o])[1][0] for f, o in zip(some, alone)][0]
    _, launches = run_batch([rec] * n, frames, mixed)
    passes = 3 if kernel["kernel"] == "jinc" else 2
    assert launches == [single + 2 * passes] * 2
    for k, out in enumerate(mixed):
        for p in range(3):
            assert bool((alone[k % 3][p] == out[p]).all())


@pytest.mark.parametrize("kernel", [dict(kernel="lanczos", taps=3, algo=2), dict(kernel="jinc", taps=3, algo=4)])
def test_more_frames_than_one_prefix_table(kernel):
    """A launch of more frames than a block's table of list lengths holds
    (1024): the frames past it continue the entries of those before."""
    w, h, n = 66, 34, 1030
    rec = lgcr.Recon(lgcr.video_format(w, h, 10, 1, 1), **dict(kernel, sparse=0))
    some = [device(S.make_frame(w, h, S.YUV420P10, seed=70 + k)) for k in range(3)]
    alone, mixed = [outputs(rec, f) for f in some], [outputs(rec, some[0]) for _ in range(n)]
    single = [run_batch([rec], [f], [o])[1][0] for f, o in zip(some, alone)][0]
    _, launches = run_batch([rec] * n, [some[k % 3] for k in range(n)], mixed)
    # the guided stage's one launch becomes two or three
    assert launches == [single + (2 if kernel["kernel"] == "jinc" else 1)] * 2
    for k, out in enumerate(mixed):
        for p in range(3):
            assert bool((alone[k % 3][p] == out[p]).all())


def test_a_growing_batch():
    """One batch object meeting larger and larger launches: its scratch grows
    in powers of two, and the samples stay those of a launch alone."""
    lib = lgcr.library()
    rec = lgcr.Recon(lgcr.video_format(640, 360, 10, 1, 1), kernel="lanczos", taps=3, algo=2)
    frame = device(S.make_frame(640, 360, S.YUV420P10, seed=12))
    outs = [outputs(rec, frame) for _ in range(24)]
    alone = rec.frame(frame, -1, out=outputs(rec, frame))
    items = (lgcr.BatchItem * len(outs))()
    for i, out in enumerate(outs):
        items[i].filter = rec.handle
        items[i].inp = lgcr.planes_desc(frame)
        items[i].out = lgcr.planes_desc(out)
        items[i].chroma_location = -1
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    handle = ctypes.c_void_p()
    assert lib.lgcr_batch_create(ctypes.byref(handle)) == 0
    for n in range(1, len(outs) + 1):           # 0.2 to 5.5 million pixels: pairs from 7 frames on
        for out in outs[:n]:
            for p in out:
                p.zero_()
        stream.wait_stream(torch.cuda.current_stream())
        assert lib.lgcr_batch_run(handle, items, n, ctypes.c_void_p(stream.cuda_stream), n % 2) == 0, \
            lib.lgcr_last_error().decode()
        stream.synchronize()
        for out in outs[:n]:
            for p in range(3):
                assert bool((out[p] == alone[p]).all()), (n, p)
    lib.lgcr_batch_destroy(handle)
