"""The residual kernel at the sizes and values where its paths can go wrong.

Every TB of a CTA step is filed under its size class and taken by a warp, an
eight-lane group or one lane; the step's record count follows the batch size,
levels are read as vectors when the pool is aligned, and dequantisation is
done in 32-bit arithmetic.  Each case is decoded through the host-buffer API
and compared with the oracle sample for sample (integer work: no tolerance).
"""
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


def check(pics):
    ref, _ = O.decode_batch(pics, threads=4)
    with GpuDecoder(0) as dec:
        got = dec.decode_yuv(pics)
    for g, r in zip(got, ref):
        for c in range(3):
            if r[c].size:
                assert np.array_equal(g[c].astype(np.uint16), r[c])


def edit(p, shift, levels, qp, narrow):
    """Picture p with a pool displaced by `shift` levels, its levels replaced
    and its QP set where given; returns what must outlive its use."""
    tus = synth.tus_of(p).copy()
    lv = synth.coeffs_of(p).astype(np.int64)
    rng = np.random.default_rng(p.n_tus)
    if levels is not None:
        lv = rng.choice(np.asarray(levels), lv.size)
        tus["nx"] = 0
    if qp is not None:
        tus["qp_y"] = rng.choice(np.asarray(qp, np.int8), tus.size)
    pool = np.zeros(lv.size + shift, np.int8 if narrow else np.int16)
    pool[shift:] = lv
    tus["coeff_off"] += shift
    p.tus, p.coeffs, p.n_coeffs = tus.ctypes.data, pool.ctypes.data, pool.size
    if narrow:
        p.flags |= abi.PIC_COEFF8
    return tus, pool


# one record; one 32-record step and a remainder; several steps per CTA
@pytest.mark.parametrize("w,h,chroma", [(8, 8, 0), (64, 64, 1), (72, 136, 3), (1024, 768, 2), (2048, 2048, 1)])
@pytest.mark.parametrize("depth", [8, 10])
def test_sizes(w, h, chroma, depth):
    s = synth.SynthSet()
    s.add(synth.residual_cfg(w + h, w, h, bit_depth=depth, chroma_idc=chroma))
    s.add(synth.residual_cfg(w, 32, 32, bit_depth=depth, chroma_idc=chroma))
    check(s.pictures())


# the whole int16 range at both ends of the QP range, flat and with scaling
# lists: the largest products and both shift directions of the dequantisation
@pytest.mark.parametrize("depth", [8, 10, 12])
@pytest.mark.parametrize("scaling", [False, True])
def test_extreme_levels(depth, scaling):
    s = synth.SynthSet()
    c = synth.residual_cfg(depth, 256, 192, bit_depth=depth)
    c.scaling = int(scaling)
    s.add(c)
    for levels, qp in (([-32768, 32767, -1, 0, 1], [-6 * (depth - 8), 51]), ([-300, 7, 0, 255], [0, 17, 37])):
        p = s.picture(0)
        keep = edit(p, 0, levels, qp, False)
        check([p])
        del keep


# pools whose TBs start at any alignment
@pytest.mark.parametrize("shift", [1, 4, 7])
@pytest.mark.parametrize("narrow", [False, True])
def test_unaligned_pools(shift, narrow):
    s = synth.SynthSet()
    s.add(synth.residual_cfg(5, 320, 200, bit_depth=10))
    p = s.picture(0)
    keep = edit(p, shift, [-128, 127, 3, 0, 0, 0], None, narrow)
    check([p])
    del keep


# inter TBs added to the motion-compensated plane (rows of every chroma
# alignment) beside intra TBs of the same picture
@pytest.mark.parametrize("w,h,depth", [(136, 72, 8), (136, 72, 10), (264, 200, 8)])
def test_added_in_plane(w, h, depth):
    s = synth.SynthSet()
    s.add(synth.intra_cfg(1, w, h, bit_depth=depth))
    s.add(synth.inter_cfg(2, w, h, bit_depth=depth, intra_cu_p=0.5))
    check(s.pictures())


# a launch large enough for the longest sorted lists, over pictures whose ends
# fall inside a CTA step and beside others of a few records
def test_long_lists():
    s = synth.SynthSet()
    for i in range(13):
        s.add(synth.residual_cfg(70 + i, 1016 + 8 * (i % 3), 776, bit_depth=8 + 2 * (i & 1), chroma_idc=3))
        s.add(synth.residual_cfg(90 + i, 16, 8))
    pics = s.pictures()
    assert sum(p.n_tus for p in pics) > 2 * 148 * 1024
    check(pics)
