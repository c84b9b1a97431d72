"""A submit that fails half way.  The first canvas of a batch of concurrent
segments has no destination, so the copy of the first segment's output is
refused while the other segments run.  The call reports it and leaves nothing
in flight: the slot's next batches, other inputs of the same layout, decode
byte for byte as the oracle does."""
import ctypes as C

import numpy as np
import pytest

from hpvcd_b200 import abi, synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from hpvcd_b200.gpu import GpuDecoder, pack_pinned, pinned_empty  # noqa: E402
from oracle import oracle as O  # noqa: E402

N, SIDE = 16, 256


def batch(seed):
    s = synth.SynthSet()
    for i in range(N):
        s.add(synth.intra_cfg(seed * 100 + i, SIDE, SIDE, bit_depth=10))
    pics = s.pictures()
    place = (abi.TilePlace * N)(*[abi.TilePlace(0, 0, SIDE, SIDE, i) for i in range(N)])
    cv = (abi.Canvas * N)(*[abi.Canvas(SIDE, SIDE, abi.MATRIX_BT709, 1) for _ in range(N)])
    out = abi.Output(abi.OUT_RGB8, 0, 0, 0, 0, C.cast(place, C.c_void_p), None, 0, N, C.cast(cv, C.c_void_p))
    return s, pics, out, (place, cv)


@pytest.mark.parametrize("pinned", [False, True])
def test_next_batch_of_the_slot(pinned):
    buf, keep = pinned_empty(N * SIDE * SIDE * 3)
    each = [buf[i * SIDE * SIDE * 3:(i + 1) * SIDE * SIDE * 3] for i in range(N)]
    good = (C.c_void_p * N)(*[b.ctypes.data for b in each])
    bad = (C.c_void_p * N)(None, *[b.ctypes.data for b in each[1:]])
    with GpuDecoder(0, max_inflight=1) as dec:
        for seed in range(6):
            s, pics, out, tables = batch(seed)
            ref = O.decode_batch(pics, out, want_planes=False)[1]
            if pinned:
                pics, arena = pack_pinned(pics)
            if seed in (1, 2, 4):  # after a batch of this layout, and twice in a row
                out.canvas_dst = C.cast(bad, C.c_void_p)
                with pytest.raises(abi.HpvcdError) as e:
                    dec.submit(pics, out)
                assert e.value.status == abi.ERR_CUDA
                continue
            out.canvas_dst = C.cast(good, C.c_void_p)
            t = dec.submit(pics, out)
            dec.wait(t)
            dec.read(t, np.empty(dec.output_size(t), np.uint8))
            want = np.concatenate([np.asarray(r).ravel() for r in ref]) if isinstance(ref, (list, tuple)) else np.asarray(ref).ravel()
            assert np.array_equal(buf, want)
