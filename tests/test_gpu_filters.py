"""The tile filter where its packed arithmetic can go wrong: every SAO type,
class and band position with offsets at both ends of a byte and beyond it, at
every bit depth; deblocking with the strongest and weakest thresholds;
pictures whose tiles are cropped on either side; RGB8 of every matrix and
range from extreme samples.  Compared with the oracle sample for sample
(integer work: no tolerance)."""
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


def picture(seed, w, h, depth, idc, offsets, qp):
    """An intra picture with its SAO parameters redrawn and its cells' QP set."""
    rng = np.random.default_rng(seed)
    s = synth.SynthSet()
    s.add(synth.intra_cfg(seed, w, h, bit_depth=depth, chroma_idc=idc))
    p = s.picture(0)
    g = synth.geometry(p)
    n = g["ctb_cols"] * g["ctb_rows"]
    sao = np.zeros(n, abi.SAO_DTYPE)
    sao["comp"]["type_idx"] = rng.integers(0, 3, (n, 3))
    sao["comp"]["band_pos"] = rng.integers(0, 32, (n, 3))
    sao["comp"]["eo_class"] = rng.integers(0, 4, (n, 3))
    sao["comp"]["offsets"] = rng.choice(np.asarray(offsets, np.int16), (n, 3, 4))
    raw = np.ctypeslib.as_array((C.c_uint8 * (g["gw"] * g["gh"] * 4)).from_address(p.cells)).copy()
    cells = raw.view(abi.CELL_DTYPE)
    cells["qp_y"] = rng.choice(np.asarray(qp, np.int8), cells.size)
    p.sao, p.cells = sao.ctypes.data, cells.ctypes.data
    return p, (s, sao, cells)


@pytest.mark.parametrize("depth", [8, 10, 12])
@pytest.mark.parametrize("idc", [0, 1, 2, 3])
@pytest.mark.parametrize("offsets", [(-128, 127, 0, 1, -1), (-129, 128, 300, -5)])
def test_planes(depth, idc, offsets):
    for k, (w, h) in enumerate([(8, 8), (64, 72), (136, 128), (200, 264)]):
        p, keep = picture(10 * depth + idc + k, w, h, depth, idc, offsets, (0, 20, 37, 51))
        ref, _ = O.decode_batch([p])
        with GpuDecoder(0) as dec:
            got = dec.decode_yuv([p])
        for c in range(3):
            if ref[0][c].size:
                assert np.array_equal(got[0][c].astype(np.uint16), ref[0][c]), (w, h, c)
        del keep


@pytest.mark.parametrize("matrix", [abi.MATRIX_IDENTITY, abi.MATRIX_BT709, abi.MATRIX_SMPTE170M, abi.MATRIX_YCGCO,
                                    abi.MATRIX_BT2020NCL])
@pytest.mark.parametrize("full", [0, 1])
@pytest.mark.parametrize("depth,idc", [(8, 0), (8, 1), (10, 2), (12, 3), (12, 1)])
def test_rgb8(matrix, full, depth, idc):
    p, keep = picture(depth + idc, 136, 72, depth, idc, (-100, 100, 7), (30,))
    for w, h, dx in ((136, 72, 0), (133, 70, 3)):
        place = (abi.TilePlace * 1)(abi.TilePlace(dx, 1, w, h))
        out = abi.Output(abi.OUT_RGB8, matrix, full, w + 5, h + 2, C.cast(place, C.c_void_p))
        _, ref = O.decode_batch([p], out)
        with GpuDecoder(0) as dec:
            got = dec.decode_rgb8([p], out)
        assert np.array_equal(got, ref)
    del keep
