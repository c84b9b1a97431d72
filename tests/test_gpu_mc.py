"""Motion compensation where its tiles and packed fetches can go wrong: PU
shapes that are not multiples of a tile (4-wide and asymmetric parts), every
fraction, references far outside the picture, pictures smaller than a tile
row, missing references, every chroma format and sample size.  Compared with
the oracle sample for sample (integer work: no tolerance)."""
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


def split_pus(pus, rng, mv_range):
    """Every PU cut into two parts along a multiple of four, motion vectors
    over +-mv_range quarter samples, now and then a reference that is not there."""
    out = []
    for u in pus:
        w, h = int(u["w"]), int(u["h"])
        cut = 4 * int(rng.integers(1, max(w, h) // 4)) if max(w, h) > 4 else 0
        parts = [(0, 0, w, h)]
        if cut and rng.random() < 0.7:
            if w >= h:
                parts = [(0, 0, cut, h), (cut, 0, w - cut, h)]
            else:
                parts = [(0, 0, w, cut), (0, cut, w, h - cut)]
        for dx, dy, pw, ph in parts:
            q = u.copy()
            q["x"], q["y"], q["w"], q["h"] = u["x"] + dx, u["y"] + dy, pw, ph
            q["mv"] = rng.integers(-mv_range, mv_range + 1, (2, 2))
            if rng.random() < 0.1:
                q["ref_idx"][int(rng.integers(0, 2))] = 15
            out.append(q)
    return np.array(out, abi.PU_DTYPE)


@pytest.mark.parametrize("idc", [0, 1, 2, 3])
@pytest.mark.parametrize("depth", [8, 10, 12])
@pytest.mark.parametrize("weighted", [False, True])
def test_shapes(idc, depth, weighted):
    rng = np.random.default_rng(100 * idc + depth + weighted)
    for w, h, mv_range in ((8, 8, 40), (24, 200, 300), (200, 72, 4000)):
        s = synth.SynthSet()
        s.add(synth.intra_cfg(1, w, h, bit_depth=depth, chroma_idc=idc))
        for k in range(2):
            c = synth.inter_cfg(2 + k, w, h, bit_depth=depth, weighted=weighted, n_refs=2)
            c.chroma_idc = idc
            s.add(c)
        pics, keep = s.pictures(), []
        for p in pics[1:]:
            pus = split_pus(synth.pus_of(p), rng, mv_range)
            p.pus, p.n_pus = pus.ctypes.data, len(pus)
            keep.append(pus)
        check(pics)
