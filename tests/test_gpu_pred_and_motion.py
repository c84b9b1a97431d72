"""Pictures flagged both HPVCD_PIC_PRED_IN_PLANE and HPVCD_PIC_INTER: the planes
start as the given prediction, motion compensation overwrites the PUs, then
every TB adds its residual to the plane, under a PU or not.  Alone, in the
middle of a sequence and as its last picture, through a plan and through a
context; compared with the oracle sample for sample (integer work: no
tolerance)."""
import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import DevicePlan, GpuDecoder  # noqa: E402
from oracle import oracle as O  # noqa: E402

W, H = 328, 200


def sequence(depth, idc, n, both):
    """n pictures (0 intra, the others inter); `both` start from a prediction
    of their own and keep two thirds of their PUs."""
    rng = np.random.default_rng(depth + idc + n)
    s = synth.SynthSet()
    for i in range(n):
        c = synth.inter_cfg(80 + i, W, H, bit_depth=depth, n_refs=2) if i or n == 1 else synth.intra_cfg(
            80, W, H, bit_depth=depth)
        c.chroma_idc = idc
        if idc == 3:
            c.ccp_p = 0.5
        s.add(c)
    pics, keep = s.pictures(), [s]
    for i in both:
        p, g = pics[i], synth.geometry(pics[i])
        p.flags |= abi.PIC_PRED_IN_PLANE
        for k in range(3 if idc else 1):
            shape = (g["h"], g["w"]) if k == 0 else (g["ch"], g["cw"])
            pred = rng.integers(0, 1 << depth, shape).astype(np.uint8 if depth == 8 else np.uint16)
            p.pred[k] = pred.ctypes.data
            keep.append(pred)
        pus = synth.pus_of(p)
        pus = pus[rng.random(pus.size) < 2 / 3].copy()
        p.pus, p.n_pus = pus.ctypes.data, len(pus)
        if n == 1:
            for l in range(2):
                for r in range(abi.MAX_REFS):
                    p.ref_slot[l][r] = -1
        keep.append(pus)
    return pics, keep


@pytest.mark.parametrize("depth", [8, 10])
@pytest.mark.parametrize("idc", [1, 2, 3])
@pytest.mark.parametrize("n,both", [(1, (0,)), (2, (1,)), (4, (2,)), (4, (1, 3))])
def test_prediction_then_motion_then_residual(depth, idc, n, both):
    pics, keep = sequence(depth, idc, n, both)
    ref, _ = O.decode_batch(pics)

    def check(planes, what):
        for i, (g, r) in enumerate(zip(planes, ref)):
            for c in range(3):
                assert np.array_equal(g[c].astype(np.uint16), r[c]), f"{what}: picture {i} component {c}"

    plan, stream = DevicePlan(pics), torch.cuda.Stream()
    for stages in (abi.STAGE_ALL, abi.STAGE_ALL | abi.STAGE_GRAPH):
        plan.launch(stages, stream)
        assert plan.status(stream) == abi.OK
        check([plan.planes(i) for i in range(n)], f"plan, stages {stages:#x}")
    plan.close()
    with GpuDecoder(0) as dec:
        for _ in range(2):
            check(dec.decode_yuv(pics), "context")
