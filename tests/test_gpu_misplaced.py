"""Intra TB records that are not at a multiple of their size.  No coding
quadtree makes one, and the walk reads and writes a TB's samples in words, so
the kernel's own check has to leave such a record out and report
HPVCD_ERR_BITSTREAM; the device stays usable and decodes the proper picture
sample for sample."""
import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import DevicePlan  # noqa: E402
from oracle import oracle as O  # noqa: E402


def decode(pics):
    plan = DevicePlan(pics)
    plan.launch()
    status = plan.status()
    planes = [plan.planes(i) for i in range(len(pics))]
    plan.close()
    return status, planes


@pytest.mark.parametrize("inter", [False, True])
@pytest.mark.parametrize("log2n,comp", [(2, 0), (3, 0), (4, 0), (5, 0), (2, 1), (3, 2), (4, 1)])
@pytest.mark.parametrize("dx,dy", [(1, 0), (2, 0), (0, 1), (3, 2)])
def test_record_off_its_grid(inter, log2n, comp, dx, dy):
    s = synth.SynthSet()
    s.add(synth.intra_cfg(61, 320, 192, bit_depth=10))
    if inter:
        s.add(synth.inter_cfg(62, 320, 192, bit_depth=10, n_refs=1, intra_cu_p=0.5))
    pics = s.pictures()
    p, n, ctb = pics[-1], 1 << log2n, 64 >> (comp > 0)
    good = p.tus
    tus = synth.tus_of(p).copy()
    hit = (tus["comp"] == comp) & (tus["log2n"] == log2n) & ((tus["flags"] & abi.TU_INTRA) != 0)
    hit &= (tus["x"] % ctb + n + dx <= ctb) & (tus["y"] % ctb + n + dy <= ctb)  # stays in its CTU
    at = np.flatnonzero(hit)
    assert at.size >= 2
    for k in (at[0], at[-1]):
        tus["x"][k] += dx
        tus["y"][k] += dy
    p.tus = tus.ctypes.data
    assert decode(pics)[0] == abi.ERR_BITSTREAM
    p.tus = good
    status, planes = decode(pics)
    assert status == abi.OK
    ref, _ = O.decode_batch(pics)
    for g, r in zip(planes, ref):
        for c in range(3):
            assert np.array_equal(g[c].astype(np.uint16), r[c])
