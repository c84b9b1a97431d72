"""The work this framework is used for, as timed cases.

Each case is one use of a public entry point over inputs with the shapes and
distributions of the repository's own configurations (hpvcd_b200/synth.py):

* ``residual`` -- one residual-only picture through a device plan;
* ``picture``  -- one intra picture through a device plan to its planes;
* ``grid``     -- a HEIC grid of tiles to one RGB8 or native YCbCr canvas,
  through a device plan or, ``host``, through the host-buffer context from
  host memory back to host memory;
* ``batch``    -- many images of uneven sizes fused into one plan, replayed as
  a CUDA graph;
* ``video``    -- an intra frame and its inter frames, as one device plan
  replayed as a CUDA graph or, ``host``, frame by frame through the context
  with its decoded-picture buffer.

Outputs are whole: every final plane or canvas byte of the pass.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from hpvcd_b200 import abi, synth
from hpvcd_b200.gpu import DevicePlan, Dpb, GpuDecoder, pack_pinned, pinned_empty

_MASK = (1 << 62) - 1


def listed():
    return [
        # the smallest reconstruction call: the plain residual configuration
        dict(name="residual_512", kind="residual", width=512, height=512, depth=8, chroma=1),
        # a gallery thumbnail, host buffers in, RGB8 out: call latency
        dict(name="thumbnail_host", kind="grid", width=320, height=240, tile=512, depth=8, chroma=1, out="rgb8",
             host=True, pinned=False, narrow=False, orientation=0),
        # one HEIC tile on its own: the intra wavefront at its shortest
        dict(name="tile_512_10bit", kind="picture", width=512, height=512, depth=10, chroma=1, log2_ctb=6, tools=False),
        # the 12-megapixel 10-bit photo, buffers already in HBM
        dict(name="grid_12mp", kind="grid", width=4032, height=3024, tile=512, depth=10, chroma=1, out="rgb8",
             host=False, pinned=True, narrow=True, orientation=0),
        # the same photo from page-locked host memory to a page-locked canvas
        dict(name="grid_12mp_host", kind="grid", width=4032, height=3024, tile=512, depth=10, chroma=1, out="rgb8",
             host=True, pinned=True, narrow=True, orientation=0),
        # screen content and graphics: 8-bit 4:4:4, native YCbCr out, ragged edge tiles
        dict(name="grid_444_yuv", kind="grid", width=2040, height=1352, tile=512, depth=8, chroma=3, out="yuv",
             host=False, pinned=True, narrow=False, orientation=0),
        # the mixed-size serving batch: 8 / 10 bit, 4:2:0 / 4:4:4, 256..4096 a side
        dict(name="batch_24_mixed", kind="batch", images=24, max_side=4096, mix=2),
        # an ungridded 4K still: one picture's wavefront bounds it
        dict(name="intra_4k_10bit", kind="picture", width=3840, height=2160, depth=10, chroma=1, log2_ctb=6,
             tools=False),
        # 4:2:2 with scaling lists, transform skip, bypass, I_PCM and slices; ragged, small CTBs
        dict(name="tools_422", kind="picture", width=1288, height=968, depth=10, chroma=2, log2_ctb=5, tools=True),
        # 1080p video, 8 bit, four references: the inter configuration
        dict(name="video_1080p", kind="video", width=1920, height=1080, depth=8, frames=12, refs=4, weighted=False,
             host=False),
        # 4K 10-bit inter frames with two references, as the schedule selector meets them
        dict(name="video_4k_10bit", kind="video", width=3840, height=2160, depth=10, frames=3, refs=2, weighted=False,
             host=False),
        # a ragged 10-bit stream with explicit weights, one submit per frame
        dict(name="video_host_weighted", kind="video", width=1192, height=664, depth=10, frames=6, refs=3,
             weighted=True, host=True),
    ]


def _side(rng, lo, hi):
    """A multiple of 8 in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, 8 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 8)))


def draw(rng):
    kind = rng.choice(["residual", "picture", "grid", "grid", "batch", "video", "video"])
    if kind == "residual":
        return dict(kind=kind, width=_side(rng, 64, 2048), height=_side(rng, 64, 2048), depth=rng.choice([8, 10]),
                    chroma=rng.choice([1, 1, 3]))
    if kind == "picture":
        return dict(kind=kind, width=_side(rng, 128, 3840), height=_side(rng, 128, 2160), depth=rng.choice([8, 10]),
                    chroma=rng.choice([0, 1, 1, 2, 3]), log2_ctb=rng.choice([4, 5, 6, 6]), tools=rng.random() < 0.25)
    if kind == "grid":
        out = rng.choice(["rgb8", "rgb8", "yuv"])
        host = rng.random() < 0.4
        return dict(kind=kind, width=_side(rng, 256, 4096), height=_side(rng, 256, 3072), tile=rng.choice([512, 256]),
                    depth=rng.choice([8, 10]), chroma=rng.choice([1, 1, 3]), out=out, host=host,
                    pinned=rng.random() < 0.5, narrow=rng.random() < 0.5,
                    orientation=abi.ORIENT_ROTATE90 if out == "rgb8" and rng.random() < 0.25 else 0)
    if kind == "batch":
        return dict(kind=kind, images=rng.randint(3, 20), max_side=_side(rng, 512, 2816) // 64 * 64,
                    mix=rng.randrange(1 << 20))
    return dict(kind=kind, width=_side(rng, 320, 2560), height=_side(rng, 240, 1440), depth=rng.choice([8, 10]),
                frames=rng.randint(3, 8), refs=rng.randint(1, 4), weighted=rng.random() < 0.3,
                host=rng.random() < 0.4)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _sub(seed, i):
    return (int(seed) * 1_000_003 + 7919 * (i + 1)) & _MASK


def _tool_cfg(cfg):
    cfg.scaling = 1
    cfg.tskip_p = 0.2
    cfg.tqb_p = 0.05
    cfg.pcm_p = 0.05
    cfg.regions = 1
    return cfg


def _picture_cfg(case, seed):
    if case["kind"] == "residual":
        return synth.residual_cfg(seed, case["width"], case["height"], case["depth"], case["chroma"])
    cfg = synth.intra_cfg(seed, case["width"], case["height"], case["depth"], case["chroma"])
    cfg.log2_ctb = case["log2_ctb"]
    return _tool_cfg(cfg) if case["tools"] else cfg


def _one(cfg):
    s = synth.SynthSet()
    s.add(cfg)
    return s


def _make_all(cfgs):
    """Every configuration as a picture of its own set, generated in threads."""
    with ThreadPoolExecutor(8) as ex:
        sets = list(ex.map(_one, cfgs))
    return sets, [s.picture(0) for s in sets]


def _tiles(width, height, tile):
    """Places of a grid's tiles on its canvas."""
    return [(x, y, tile, tile) for y in range(0, height, tile) for x in range(0, width, tile)]


def _batch_images(case):
    return synth.config2_images(case["mix"], case["images"], case["max_side"])


def _video_cfgs(case, seed):
    w, h, bd = case["width"], case["height"], case["depth"]
    cfgs = [synth.intra_cfg(_sub(seed, 0), w, h, bit_depth=bd, chroma_idc=1)]
    for i in range(1, case["frames"]):
        cfgs.append(synth.inter_cfg(_sub(seed, i), w, h, bit_depth=bd, weighted=case["weighted"],
                                    n_refs=case["refs"]))
    return cfgs


class _DeviceArray:
    """Device memory of a plan as torch sees it (no copy); the tensor made of
    it keeps this object, and so the plan, for as long as it lives."""

    def __init__(self, plan, ptr, shape, typestr):
        self.plan = plan
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _device_tensor(plan, ptr, shape, wide=False):
    return torch.as_tensor(_DeviceArray(plan, ptr, shape, "<i2" if wide else "|u1"), device="cuda")


def _plan_planes(plan, pics, which):
    """The final planes of pictures `which`, as tensors over the plan's memory."""
    out = []
    for i in which:
        g = synth.geometry(pics[i])
        ptr = [C.c_void_p() for _ in range(3)]
        abi.check(abi.lib().hpvcd_plan_planes(plan._h, i, *(C.byref(p) for p in ptr)), "hpvcd_plan_planes")
        shapes = [(g["h"], g["w"])] + [(g["ch"], g["cw"])] * (2 if pics[i].chroma_idc else 0)
        out += [_device_tensor(plan, p.value, s, g["bytes_per_sample"] == 2) for p, s in zip(ptr, shapes)]
    return out


@functools.cache
def _stream():
    """The program's decoding stream (a graph replay needs one of its own)."""
    return torch.cuda.Stream()


def _canvas_tensor(plan, wide):
    ptr, nbytes = plan.canvas_ptr()
    return _device_tensor(plan, ptr, (nbytes // 2 if wide else nbytes,), wide)


# ---------------------------------------------------------------------------
# What a program has in hand before the call
# ---------------------------------------------------------------------------

def _prepare_grid(case, seed):
    places = _tiles(case["width"], case["height"], case["tile"])
    keep, pics = _make_all([synth.intra_cfg(_sub(seed, i), case["tile"], case["tile"], case["depth"], case["chroma"])
                            for i in range(len(places))])
    pools = synth.narrow_coeffs(pics) if case["narrow"] else []
    arr = (abi.TilePlace * len(places))(*[abi.TilePlace(*p) for p in places])
    kind = abi.OUT_RGB8 if case["out"] == "rgb8" else abi.OUT_YUV_CANVAS
    out = abi.Output(kind, abi.MATRIX_SMPTE170M, 1, case["width"], case["height"], C.cast(arr, C.c_void_p))
    out.orientation = case["orientation"]
    if case["out"] == "rgb8":
        out.options = abi.OUTPUT_CANVAS_ONLY
    wide = case["out"] == "yuv" and case["depth"] > 8
    if not case["host"]:
        plan = DevicePlan(pics, out)
        return dict(plan=plan, stages=abi.STAGE_ALL, outputs=[_canvas_tensor(plan, wide)], keep=(out, arr))
    per = 3.0 if case["out"] == "rgb8" else {0: 1, 1: 1.5, 3: 3}[case["chroma"]] * (2 if wide else 1)
    nbytes = int(case["width"] * case["height"] * per)
    if case["pinned"]:
        pics, packed = pack_pinned(pics)
        dst, dst_keep = pinned_empty(nbytes)
        out.host_dst, out.host_dst_bytes = dst.ctypes.data, nbytes
    else:
        packed, dst, dst_keep = None, np.empty(nbytes, np.uint8), None
    return dict(dec=GpuDecoder(0), batches=[(pics, out)], dst=[dst], in_flight=1,
                keep=(keep, pools, arr, packed, dst_keep))


def _prepare_batch(case, seed):
    cfgs, places, canvases = [], [], []
    for k, (w, h, depth, chroma) in enumerate(_batch_images(case)):
        for x, y, tw, th in _tiles(w, h, 512):
            cfgs.append(synth.intra_cfg(_sub(seed, len(cfgs)), tw, th, depth, chroma))
            places.append((x, y, tw, th, k))
        canvases.append(abi.Canvas(w, h, abi.MATRIX_SMPTE170M if k % 3 else abi.MATRIX_BT709, k % 2))
    keep, pics = _make_all(cfgs)  # kept until the upload is done
    pl = (abi.TilePlace * len(places))(*[abi.TilePlace(*p) for p in places])
    cv = (abi.Canvas * len(canvases))(*canvases)
    out = abi.Output(abi.OUT_RGB8, 0, 0, 0, 0, C.cast(pl, C.c_void_p), None, 0, len(canvases), C.cast(cv, C.c_void_p))
    out.options = abi.OUTPUT_CANVAS_ONLY
    plan = DevicePlan(pics, out)
    del keep, pics
    return dict(plan=plan, stages=abi.STAGE_ALL | abi.STAGE_GRAPH, stream=_stream(),
                outputs=[_canvas_tensor(plan, False)], keep=(out, pl, cv))


def _prepare_video(case, seed):
    s = synth.SynthSet()
    for cfg in _video_cfgs(case, seed):
        s.add(cfg)
    pics = s.pictures()
    if not case["host"]:
        plan = DevicePlan(pics)
        return dict(plan=plan, stages=abi.STAGE_ALL | abi.STAGE_GRAPH, stream=_stream(),
                    outputs=_plan_planes(plan, pics, range(len(pics))))
    # one frame per submit: frame k is kept in entry k and read from there
    batches, dst, keep = [], [], [s]
    for k, p in enumerate(pics):
        p.flags |= abi.PIC_STORE_DPB(k)
        for lst in range(2):
            for r in range(abi.MAX_REFS):
                slot = p.ref_slot[lst][r]
                p.ref_slot[lst][r] = abi.REF_DPB(slot) if slot >= 0 else -1
        (q,), packed = pack_pinned([p])
        g = synth.geometry(p)
        nbytes = (g["w"] * g["h"] + 2 * g["cw"] * g["ch"]) * g["bytes_per_sample"]
        buf, buf_keep = pinned_empty(nbytes)
        out = abi.Output(abi.OUT_YUV)
        out.host_dst, out.host_dst_bytes = buf.ctypes.data, nbytes
        batches.append(([q], out))
        dst.append(buf)
        keep.append((packed, buf_keep))
    dec, dpb = GpuDecoder(0, max_inflight=2), Dpb(0, len(pics))
    dec.set_dpb(dpb)
    return dict(dec=dec, batches=batches, dst=dst, in_flight=2, keep=(keep, dpb))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        return _prepare_grid(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "video":
        return _prepare_video(case, seed)
    s = _one(_picture_cfg(case, _sub(seed, 0)))
    pics = s.pictures()
    plan = DevicePlan(pics)
    return dict(plan=plan, stages=abi.STAGE_ALL, outputs=_plan_planes(plan, pics, [0]))


def run(state):
    if "plan" in state:
        state["plan"].launch(state["stages"], state.get("stream"))
        return state["outputs"]
    dec, pending, out = state["dec"], [], []

    def finish():
        ticket, dst = pending.pop(0)
        dec.wait(ticket)
        out.append(dec.read(ticket, dst))

    for (pics, output), dst in zip(state["batches"], state["dst"]):
        pending.append((dec.submit(pics, output), dst))
        if len(pending) == state["in_flight"]:
            finish()
    while pending:
        finish()
    return out


# ---------------------------------------------------------------------------
# What the work cannot do without
# ---------------------------------------------------------------------------

def _samples(width, height, chroma):
    return width * height * {0: 1.0, 1: 1.5, 2: 2.0, 3: 3.0}[chroma]


def _input_bytes(cfg, narrow=False):
    """Bytes of one picture's flat buffers, by the density of a 512 x 512 one."""
    area = cfg.width * cfg.height
    cfg.width = cfg.height = 512
    s = synth.SynthSet()
    if cfg.kind == abi.SYNTH_INTER:  # the pictures it refers to
        s.add(synth.intra_cfg(1, 512, 512, cfg.bit_depth, cfg.chroma_idc))
    p = s.picture(s.add(cfg))
    sample = 1 if cfg.bit_depth == 8 else 2
    n = 16 * p.n_tus + 20 * p.n_pus + (1 if narrow else 2) * p.n_coeffs
    if p.cells:
        n += 4 * 128 * 128
    if p.sao:
        n += 36 * (512 >> p.log2_ctb) ** 2
    if p.flags & abi.PIC_PRED_IN_PLANE:
        n += _samples(512, 512, cfg.chroma_idc) * sample
    return n * area / (512 * 512)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = 0.0
        for w, h, depth, chroma in _batch_images(case):
            tiles = len(_tiles(w, h, 512))
            total += tiles * _input_bytes(synth.intra_cfg(1, 512, 512, depth, chroma)) + 3 * w * h
        return {"bytes": total, "flops": 0}
    w, h, depth = case["width"], case["height"], case["depth"]
    sample = 1 if depth == 8 else 2
    if kind == "grid":
        tile = synth.intra_cfg(1, case["tile"], case["tile"], depth, case["chroma"])
        out = 3 * w * h if case["out"] == "rgb8" else _samples(w, h, case["chroma"]) * sample
        return {"bytes": len(_tiles(w, h, case["tile"])) * _input_bytes(tile, case["narrow"]) + out, "flops": 0}
    if kind == "video":
        total = sum(_input_bytes(cfg) for cfg in _video_cfgs(case, 1))
        return {"bytes": total + case["frames"] * _samples(w, h, 1) * sample, "flops": 0}
    total = _input_bytes(_picture_cfg(case, 1))
    return {"bytes": total + _samples(w, h, case["chroma"]) * sample, "flops": 0}


# ---------------------------------------------------------------------------
# The residual picture in plain numpy: dequantisation and inverse transform of
# ITU-T H.265 (8.6.2 - 8.6.4.2) in 64-bit integers
# ---------------------------------------------------------------------------

def _dct(n):
    """The n-point basis: the 32-point one decimated, from its angle magnitudes."""
    mag = [64, 90, 90, 90, 89, 88, 87, 85, 83, 82, 80, 78, 75, 73, 70, 67, 64, 61, 57, 54, 50, 46, 43, 38, 36, 31, 25,
           22, 18, 13, 9, 4, 0]
    t = np.full((n, n), 64, np.int64)
    for k in range(1, n):
        for m in range(n):
            j = k * (32 // n) * (2 * m + 1) % 128
            j = min(j, 128 - j)
            t[k, m] = mag[j] if j <= 32 else -mag[64 - j]
    return t


_DST = np.array([[29, 55, 74, 84], [74, 74, 0, -74], [84, -29, -74, 55], [55, -84, 74, -29]], np.int64)


def _chroma_qp(qpi, chroma):
    if chroma != 1:
        return min(qpi, 51)
    return qpi if qpi < 30 else qpi - 6 if qpi > 43 else [29, 30, 31, 32, 33, 33, 34, 34, 35, 35, 36, 36, 37, 37][qpi - 30]


def exact(case, seed):
    if case["kind"] != "residual":
        return None  # a whole picture's prediction, sample after sample: far over the time there is
    s = _one(_picture_cfg(case, _sub(seed, 0)))
    p = s.picture(0)
    depth, chroma = case["depth"], case["chroma"]
    dt = np.uint8 if depth == 8 else np.uint16
    planes = []
    for c in range(3):
        w, h = (p.width, p.height) if c == 0 or chroma == 3 else (p.width // 2, p.height // 2)
        raw = (C.c_uint8 * (w * h * dt().itemsize)).from_address(p.pred[c])
        planes.append(np.frombuffer(raw, dt).reshape(h, w).astype(np.int64))
    levels, bases = synth.coeffs_of(p).astype(np.int64), {n: _dct(n) for n in (4, 8, 16, 32)}
    offset, top = 6 * (depth - 8), (1 << depth) - 1
    for t in synth.tus_of(p):
        c, n, flags = int(t["comp"]), 1 << int(t["log2n"]), int(t["flags"])
        if not flags & abi.TU_CBF:
            continue
        qp = int(t["qp_y"])
        if c:
            pps = p.pps_cb_qp_offset if c == 1 else p.pps_cr_qp_offset
            qp = _chroma_qp(max(-offset, min(57, qp + pps + int(t["cqp_off"]))), chroma)
        qp += offset
        at = int(t["coeff_off"])
        lv = levels[at:at + n * n].reshape(n, n)
        shift = depth + int(t["log2n"]) - 5
        d = (lv * ([40, 45, 51, 57, 64, 72][qp % 6] << (qp // 6)) * 16 + (1 << (shift - 1))) >> shift
        d = np.clip(d, -32768, 32767)
        basis = _DST if n == 4 and c == 0 and flags & abi.TU_INTRA else bases[n]
        e = np.clip((basis.T @ d + 64) >> 7, -32768, 32767)
        r = (e @ basis + (1 << (19 - depth))) >> (20 - depth)
        x, y = int(t["x"]), int(t["y"])
        view = planes[c][y:y + n, x:x + n]
        view[:] = np.clip(view + r[:view.shape[0], :view.shape[1]], 0, top)
    kept = np.uint8 if depth == 8 else np.int16
    return [torch.from_numpy(q.astype(kept)) for q in planes]
