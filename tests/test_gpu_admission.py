"""HBM admission: a context never holds more than its budget.  What a batch
makes it hold is counted here from the formats of the public structures: the
input arena, the reconstruction planes, the final planes where they are
separate, the residual planes, the edge words and work list of the wavefront
and the canvas.  A budget below that is refused (before anything is copied),
one with room for the small tables beside it decodes."""
import ctypes as C

import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import GpuDecoder  # noqa: E402
from oracle import oracle as O  # noqa: E402

TABLES = 64 << 10  # picture table, prefix, counters


def up(v, a):
    return -(-v // a) * a


def planes_bytes(w, h, cw, ch, size):
    return up(w * h * size, 256) + 2 * up(cw * ch * size, 256)


def held_bytes(pics, canvas, separate_final):
    arr = (abi.Picture * len(pics))(*pics)
    arena = abi.lib().hpvcd_gpu_packed_size(arr, len(pics))
    total = up(arena + arena // 4, 1 << 20) + canvas
    referenced = {r for p in pics for row in p.ref_slot for r in row}
    for i, p in enumerate(pics):
        g = synth.geometry(p)
        w, h, cw, ch = g["w"], g["h"], g["cw"], g["ch"]
        total += planes_bytes(w, h, cw, ch, g["bytes_per_sample"]) * (2 if separate_final or i in referenced else 1)
        total += up(up(w, 16) * h * 2, 256) + 2 * up(up(cw, 16) * ch * 2, 256)
        ctb, sw, sh = 1 << p.log2_ctb, 2 if p.chroma_idc in (1, 2) else 1, 2 if p.chroma_idc == 1 else 1
        words = ctb // 2 + (2 * (ctb // sw // 4 + ctb // sh // 4) if p.chroma_idc else 0)
        total += g["ctb_cols"] * g["ctb_rows"] * (8 * words + 8)
    return total


def check(pics, out, canvas, separate_final):
    need = held_bytes(pics, canvas, separate_final)
    with GpuDecoder(0, max_inflight=1, hbm_budget=need - 1) as dec:
        with pytest.raises(abi.HpvcdError) as e:
            dec.submit(pics, out)
        assert e.value.status == abi.ERR_ALLOC
    with GpuDecoder(0, max_inflight=1, hbm_budget=need + TABLES) as dec:
        got = dec.decode_rgb8(pics, out)
    _, ref = O.decode_batch(pics, out, want_planes=False)
    assert np.array_equal(got, ref)


def batch(idc, log2_ctb, sao):
    s = synth.SynthSet()
    for i in range(2):
        c = synth.intra_cfg(90 + i, 512, 512, bit_depth=8, chroma_idc=idc, sao=sao)
        c.log2_ctb = log2_ctb
        s.add(c)
    place = (abi.TilePlace * 2)(abi.TilePlace(0, 0, 512, 512), abi.TilePlace(512, 0, 512, 512))
    return s, abi.Output(abi.OUT_RGB8, abi.MATRIX_SMPTE170M, 1, 1024, 512, C.cast(place, C.c_void_p)), place


@pytest.mark.parametrize("idc", [0, 1, 2, 3])
@pytest.mark.parametrize("log2_ctb", [4, 6])
def test_edge_words_are_counted(idc, log2_ctb):
    s, out, place = batch(idc, log2_ctb, True)
    check(s.pictures(), out, 1024 * 512 * 3, True)


@pytest.mark.parametrize("canvas_only", [False, True])
@pytest.mark.parametrize("sao", [False, True])
def test_kept_final_planes_are_counted(canvas_only, sao):
    s, out, place = batch(1, 6, sao)
    out.options = abi.OUTPUT_CANVAS_ONLY if canvas_only else 0
    check(s.pictures(), out, 1024 * 512 * 3, sao or not canvas_only)
