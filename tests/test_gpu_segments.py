"""Uploads and copies back segment by segment: a context that decodes a second
batch of the layout of the one before starts each concurrent segment on its
own inputs and copies its output as it joins.  Every kind of output, page-locked
and ordinary memory, several tickets in flight; compared with the oracle byte
for byte."""
import ctypes as C

import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import GpuDecoder, pack_pinned, pinned_empty, split_planes  # noqa: E402
from oracle import oracle as O  # noqa: E402

W, H, TILE = 616, 424, 128  # 5 x 4 tiles, the last column and row cropped


def tiles(seed):
    s = synth.SynthSet()
    places = []
    for y in range(0, H, TILE):
        for x in range(0, W, TILE):
            s.add(synth.intra_cfg(seed * 1000 + len(places), TILE, TILE, bit_depth=10))
            places.append((x, y, TILE, TILE))
    return s, s.pictures(), places


def output(kind, places, orientation=0, order=None):
    if order is not None:
        places = [places[i] for i in order]
    arr = (abi.TilePlace * len(places))(*[abi.TilePlace(*p) for p in places])
    out = abi.Output(kind, abi.MATRIX_SMPTE170M, 1, W, H, C.cast(arr, C.c_void_p))
    out.orientation = orientation
    return out, arr


def check_planes(got, ref):
    for g, r in zip(got, ref):
        for c in range(3):
            assert np.array_equal(g[c].astype(np.uint16), r[c])


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("kind,orientation,backwards", [(abi.OUT_RGB8, 0, False), (abi.OUT_RGB8, 0, True),
                                                        (abi.OUT_RGB8, abi.ORIENT_ROTATE90, False),
                                                        (abi.OUT_YUV_CANVAS, 0, False)])
def test_canvas(pinned, kind, orientation, backwards):
    with GpuDecoder(0, max_inflight=2) as dec:
        pending = []
        for seed in range(5):
            s, pics, places = tiles(seed)
            order = list(range(len(places)))[::-1] if backwards else None  # later tiles lie before earlier ones
            out, arr = output(kind, places, orientation, order)
            _, ref = O.decode_batch(pics, out)
            dst = keep = None
            if pinned:
                pics, keep = pack_pinned(pics)
                dst, dk = pinned_empty(np.asarray(ref).nbytes)
                out.host_dst, out.host_dst_bytes = dst.ctypes.data, dst.nbytes
                keep = (keep, dk)
            pending.append((dec.submit(pics, out), dst, ref, (s, arr, keep)))
            if len(pending) == 2 or seed % 2:
                t, d, r, _ = pending.pop(0)
                dec.wait(t)
                assert np.array_equal(dec.read(t, d).ravel(), np.asarray(r).view(np.uint8).ravel())
        for t, d, r, _ in pending:
            dec.wait(t)
            assert np.array_equal(dec.read(t, d).ravel(), np.asarray(r).view(np.uint8).ravel())


def test_planes():
    with GpuDecoder(0) as dec:
        for seed in range(3):
            s, pics, _ = tiles(10 + seed)
            ref, _ = O.decode_batch(pics)
            t = dec.submit(pics)
            dec.wait(t)
            check_planes(split_planes(pics, dec.read(t)), ref)


def test_canvas_buffers():
    """One page-locked buffer per canvas, tiles of the canvases interleaved."""
    with GpuDecoder(0) as dec:
        for seed in range(3):
            s, pics, _ = tiles(20 + seed)
            places = [((i // 2 % 5) * TILE, (i // 10) * TILE, TILE, TILE, i % 2) for i in range(len(pics))]
            arr = (abi.TilePlace * len(places))(*[abi.TilePlace(*p) for p in places])
            cv = (abi.Canvas * 2)(abi.Canvas(600, 256, abi.MATRIX_BT709, 1), abi.Canvas(640, 250, abi.MATRIX_SMPTE170M, 0))
            out = abi.Output(abi.OUT_RGB8, 0, 0, 0, 0, C.cast(arr, C.c_void_p), None, 0, 2, C.cast(cv, C.c_void_p))
            _, ref = O.decode_batch(pics, out)
            bufs = [pinned_empty(600 * 256 * 3), pinned_empty(640 * 250 * 3)]
            ptrs = (C.c_void_p * 2)(*[b[0].ctypes.data for b in bufs])
            out.canvas_dst = C.cast(ptrs, C.c_void_p)
            t = dec.submit(pics, out)
            dec.wait(t)
            dec.read(t, np.empty(dec.output_size(t), np.uint8))
            got = np.concatenate([b[0] for b in bufs])
            want = np.concatenate([np.asarray(r).ravel() for r in ref]) if isinstance(ref, (list, tuple)) else np.asarray(ref).ravel()
            assert np.array_equal(got, want)
