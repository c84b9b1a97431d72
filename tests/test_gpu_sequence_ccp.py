"""Sequences whose later pictures use cross-component prediction: the residuals
of every picture but the first, the luma-derived chroma residuals among them,
are computed on a side stream beside the first picture.  Directly and as a
CUDA graph, several launches in a row; compared with the oracle sample for
sample (integer work: no tolerance), and the launches counted."""
import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import DevicePlan  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("depth", [8, 12])
@pytest.mark.parametrize("ccp", [(0, 1), (1, 0, 0), (0, 0, 1, 1), (1, 1, 1)])
def test_later_pictures(depth, ccp):
    s = synth.SynthSet()
    for i, on in enumerate(ccp):
        make = synth.inter_cfg if i else synth.intra_cfg
        c = make(70 + i, 256, 192, bit_depth=depth)
        c.chroma_idc = 3
        c.ccp_p = 0.7 if on else 0.0
        s.add(c)
    pics = s.pictures()
    for p, on in zip(pics, ccp):
        assert bool(p.flags & abi.PIC_CROSS_COMPONENT) == bool(on)
    ref, _ = O.decode_batch(pics)
    plan, stream = DevicePlan(pics), torch.cuda.Stream()
    for stages in (abi.STAGE_ALL, abi.STAGE_ALL, abi.STAGE_ALL | abi.STAGE_GRAPH, abi.STAGE_ALL | abi.STAGE_GRAPH):
        plan.launch(stages, stream)
        assert plan.status(stream) == abi.OK
        for i, r in enumerate(ref):
            for c, g in enumerate(plan.planes(i)):
                assert np.array_equal(g.astype(np.uint16), r[c]), f"picture {i} component {c}"
    # residual and cross-component launches of the first picture and of the rest, then
    # wavefront and filter of every picture and motion compensation of the inter ones
    n = len(ccp)
    assert plan.launches_per_run == 2 + ccp[0] + any(ccp[1:]) + 2 * n + (n - 1)
    before = abi.lib().hpvcd_kernel_launch_count()
    plan.launch()
    assert abi.lib().hpvcd_kernel_launch_count() - before == plan.launches_per_run
    plan.close()
