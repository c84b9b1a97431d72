"""Motion compensation where a warp's luma and chroma tasks follow one another
in the same shared-memory block: pictures with several tasks for every warp, of
large PUs (runs of tiles of one PU) and of the smallest, every chroma format
and sample size.  Compared with the oracle sample for sample (integer work: no
tolerance)."""
import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import DevicePlan  # noqa: E402
from oracle import oracle as O  # noqa: E402


def grid_pus(w, h, size, rng):
    """Bi-predicted PUs of size x size over the picture, fractions of every kind."""
    out = np.zeros((h // size) * (w // size), abi.PU_DTYPE)
    out["x"] = np.tile(np.arange(0, w, size), h // size)
    out["y"] = np.repeat(np.arange(0, h, size), w // size)
    out["w"] = out["h"] = size
    out["mv"] = rng.integers(-64, 65, (out.size, 2, 2))
    out["flags"] = abi.PU_L0 | abi.PU_L1
    return out


@pytest.mark.parametrize("idc", [1, 2, 3])
@pytest.mark.parametrize("depth", [8, 10])
@pytest.mark.parametrize("size", [8, 64])
def test_luma_and_chroma_tasks_of_a_warp(idc, depth, size):
    w, h = 1024, 512
    s = synth.SynthSet()
    s.add(synth.intra_cfg(1, w, h, bit_depth=depth, chroma_idc=idc))
    c = synth.inter_cfg(2, w, h, bit_depth=depth, n_refs=1, intra_cu_p=0.0)
    c.chroma_idc = idc
    s.add(c)
    pics = s.pictures()
    pus = grid_pus(w, h, size, np.random.default_rng(idc + depth + size))
    pics[1].pus, pics[1].n_pus = pus.ctypes.data, len(pus)
    ref, _ = O.decode_batch(pics, threads=4)
    plan = DevicePlan(pics)
    for _ in range(3):
        plan.launch()
        assert plan.status() == abi.OK
        for i in range(2):
            for g, r in zip(plan.planes(i), ref[i]):
                assert np.array_equal(g.astype(np.uint16), r)
    plan.close()
