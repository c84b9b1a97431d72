"""The flags by which the walk takes its entries, with as many entries as a CTU
can hold (every TB 4x4) and with few, in both builds of the wavefront kernel
(other numbers of threads share them out), every chroma format.  Compared with
the oracle sample for sample (integer work: no tolerance)."""
import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import DevicePlan  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("idc", [0, 1, 2, 3])
@pytest.mark.parametrize("chroma_warps", [1, 2])
@pytest.mark.parametrize("mix", [(1, 0, 0, 0), (0.5, 0.5, 0, 0), (0, 0, 0, 1)])
@pytest.mark.parametrize("wave", [0, 1])
def test_flags(idc, chroma_warps, mix, wave):
    s = synth.SynthSet()
    c = synth.intra_cfg(41 + idc, 320, 256, bit_depth=10, chroma_idc=idc)
    for i, m in enumerate(mix):
        c.tu_mix[i] = m
    s.add(c)
    pics = s.pictures()
    if mix[0] == 1:
        t = synth.tus_of(pics[0])
        start = np.ctypeslib.as_array((np.ctypeslib.ctypes.c_uint32 * 21).from_address(pics[0].ctu_tu_start))
        assert max(int((t["comp"][a:b] == 0).sum()) for a, b in zip(start, start[1:])) == 256
    ref, _ = O.decode_batch(pics)
    plan = DevicePlan(pics, sched=abi.Sched(0, chroma_warps, 0, wave))
    plan.launch()
    assert plan.status() == abi.OK
    for g, r in zip(plan.planes(0), ref[0]):
        if r.size:
            assert np.array_equal(g.astype(np.uint16), r)
    plan.close()
