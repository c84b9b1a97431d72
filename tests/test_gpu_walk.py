"""The intra walk where its per-TB entries can go wrong: reference lines that
are one run of available samples (substituted by a clamp) beside lines that are
not (slice boundaries, constrained intra prediction), at every CTB size and
chroma format, ragged pictures included.  Compared with the oracle sample for
sample (integer work: no tolerance)."""
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
    for i, (g, r) in enumerate(zip(got, ref)):
        for c in range(3):
            if r[c].size:
                assert np.array_equal(g[c].astype(np.uint16), r[c]), f"picture {i} component {c}"


@pytest.mark.parametrize("log2_ctb", [4, 5, 6])
@pytest.mark.parametrize("idc", [0, 1, 2, 3])
@pytest.mark.parametrize("regions", [0, 1, 2])
def test_lines(log2_ctb, idc, regions):
    s = synth.SynthSet()
    for k, (w, h) in enumerate([(8, 8), (200, 136), (320, 256)]):
        c = synth.intra_cfg(100 * log2_ctb + 10 * idc + regions + k, w, h, bit_depth=8 + 2 * (k % 2), chroma_idc=idc)
        c.log2_ctb = log2_ctb
        c.regions = regions if w > 8 else 0
        s.add(c)
    check(s.pictures())


@pytest.mark.parametrize("idc", [1, 2, 3])
@pytest.mark.parametrize("log2_ctb", [5, 6])
def test_lines_constrained(idc, log2_ctb):
    s = synth.SynthSet()
    a = synth.intra_cfg(7, 256, 192, bit_depth=8, chroma_idc=idc)
    a.log2_ctb = log2_ctb
    s.add(a)
    c = synth.inter_cfg(8, 256, 192, bit_depth=8, intra_cu_p=0.5)
    c.chroma_idc = idc
    c.log2_ctb = log2_ctb
    c.regions = 1
    c.pic_flags |= abi.PIC_CONSTRAINED_INTRA
    s.add(c)
    check(s.pictures())


# one TB size after another: every mode of it, with and without residual
@pytest.mark.parametrize("mix", [(1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 1)])
@pytest.mark.parametrize("cbf", [0.0, 0.5])
@pytest.mark.parametrize("depth", [8, 12])
def test_sizes(mix, cbf, depth):
    s = synth.SynthSet()
    c = synth.intra_cfg(int(sum(m << i for i, m in enumerate(mix))), 512, 384, bit_depth=depth, cbf_p=cbf)
    for i, m in enumerate(mix):
        c.tu_mix[i] = m
    s.add(c)
    check(s.pictures())


# Cr TBs whose modes differ from Cb's: the two components share no table then
@pytest.mark.parametrize("idc", [1, 2, 3])
@pytest.mark.parametrize("share", [1.0, 0.02])
def test_cr_modes_of_their_own(idc, share):
    s = synth.SynthSet()
    s.add(synth.intra_cfg(31 + idc, 320, 192, bit_depth=10, chroma_idc=idc))
    p = s.picture(0)
    rng = np.random.default_rng(idc)
    tus = synth.tus_of(p).copy()
    cr = (tus["comp"] == 2) & (rng.random(tus.size) < share)
    tus["mode"][cr] = rng.integers(0, 35, int(cr.sum()))
    p.tus = tus.ctypes.data
    check([p])
