"""What is timed of this framework: whole calls of its C API (include/msnhnet_capi.h) as a user's program makes them,
host images in, logits / maps / boxes out.

A case names a net of `topologies`, its input size, the element type of the plan, the images per forward (`batch`), the
forwards per call (`steps`) and the call:

    batch      msnhB200RunClassifyBatch / RunYoloBatch: float images in ordinary host memory, one forward, synchronous
    stream     msnhB200RunClassifyStream / RunYoloStream: float images in pinned memory, forwards pipelined
    stream_u8  the same for raw 8-bit images of any size (`width` x `height`), preprocessed on the device
    list       runYoloList: one raw 8-bit image, the reference's own detection entry point

Weights are the seeded, calibrated stand-ins the benchmark uses; images are seeded uniform noise in the range the
preprocessing produces (8-bit ones as fine as the net's input sees them, so that the resize leaves that noise as it is). The C API holds one net per process, as a program that serves one model does: it is built when a
case first asks for it and kept while the cases that follow want the same one.
"""
import ctypes as C

import numpy as np
import torch

from msnhnet_b200 import _ffi, synth, topologies
from msnhnet_b200.net import Net

MAX_BOXES = 1024     # rows per image of the box buffers a caller passes (the reference's own MaxBBoxNum)

# net: (convolution GFLOP per image, at this input size, range of input sizes)
NETS = {
    "mobilenetv2": (0.605, 224, (96, 320)),
    "resnet18": (3.63, 224, (224, 320)),
    "yolov3_tiny": (5.57, 416, (256, 608)),
    "yolov4": (128.39, 608, (256, 608)),
    "yolov5m": (52.19, 640, (256, 640)),
    "fcns": (64.54, 320, (96, 416)),
}
DETECTORS = ("yolov3_tiny", "yolov4", "yolov5m")


def case(net, size, dtype, batch, call, steps=1, width=0, height=0):
    return {"net": net, "size": size, "dtype": dtype, "batch": batch, "call": call, "steps": steps, "width": width, "height": height}


def listed():
    return [
        # one image at a time: latency, launches and host work
        dict(case("mobilenetv2", 224, "fp16", 1, "batch"), name="mobilenetv2-224 fp16 1"),          # a classifier on an edge of a pipeline
        dict(case("resnet18", 224, "fp32", 1, "batch"), name="resnet18-224 fp32 1"),                # the default element type
        dict(case("yolov3_tiny", 416, "fp32", 1, "batch"), name="yolov3tiny-416 fp32 1"),           # fp32 detection, exact arithmetic
        dict(case("yolov4", 608, "fp16", 1, "list", width=1280, height=720), name="yolov4-608 fp16 list"),   # a camera frame
        # a few images per call: an offline classifier, an odd number of images on an odd plane, fp32 detection
        dict(case("resnet18", 224, "fp32", 32, "batch"), name="resnet18-224 fp32 32"),
        dict(case("yolov4", 416, "fp16", 5, "batch"), name="yolov4-416 fp16 5"),
        dict(case("yolov5m", 352, "fp32", 3, "batch"), name="yolov5m-352 fp32 3"),
        # throughput: the benchmark's workloads, streamed
        dict(case("mobilenetv2", 224, "fp16", 64, "stream", 4), name="mobilenetv2-224 fp16 4x64"),
        dict(case("yolov3_tiny", 416, "fp16", 16, "stream", 6), name="yolov3tiny-416 fp16 6x16"),
        dict(case("fcns", 320, "fp16", 16, "stream", 4), name="fcns-320 fp16 4x16"),                # segmentation: a map comes back
        dict(case("yolov4", 608, "fp16", 8, "stream", 6), name="yolov4-608 fp16 6x8"),              # the headline
        dict(case("yolov5m", 640, "fp16", 32, "stream_u8", 4, width=1280, height=720), name="yolov5m-640 fp16 4x32 u8"),
    ]


def gflop(c):
    per, ref, _ = NETS[c["net"]]
    return per * (c["size"] / ref) ** 2 * c["batch"] * c["steps"]


def image_bytes(c):
    n = c["batch"] * c["steps"] * 3
    return n * c["width"] * c["height"] if c["call"] in ("stream_u8", "list") else n * 4 * c["size"] ** 2


def draw(rng):
    while True:
        net = rng.choice(sorted(NETS))
        lo, hi = NETS[net][2]
        size = 32 * rng.randint(lo // 32, hi // 32)
        dtype = rng.choice(("fp16", "fp16", "fp16", "fp32"))
        call = rng.choice(("batch", "batch", "stream", "stream_u8") + (("list",) if net in DETECTORS else ()))
        batch = 1 if call == "list" else round(2 ** rng.uniform(0, 6))
        steps = rng.randint(2, 6) if call.startswith("stream") else 1
        width = height = 0
        if call in ("stream_u8", "list"):       # camera and file sizes: larger than the net's input, upright ones too
            width = rng.randint(3 * size // 2, 1920)
            height = rng.randint(width // 2, width)
            if rng.random() < 0.25:
                width, height = height, width
        c = case(net, size, dtype, batch, call, steps, width, height)
        if call == "stream_u8" and width * height > 4 * size * size:
            continue
        if net == "yolov5m" and batch * steps < 3:      # under random weights one image in three holds nothing that this net sees
            continue
        # fp32 detection runs on the CUDA cores at a few percent of the tensor rate, tf32 at half of it
        most = 6000 if dtype == "fp16" else 160 if net in DETECTORS else 2500
        if gflop(c) > most or image_bytes(c) > (350e6 if call == "stream_u8" else 250e6 if call == "stream" else 100e6):
            continue
        return c


def _topology(c):
    """The net's text. Under random weights the confidence threshold at which an image holds some ten to hundred boxes, as
    a photograph does, differs from net to net and with what the image looks like (8-bit images come with gray bars and
    a little smoothed)."""
    raw = c["call"] in ("stream_u8", "list")
    conf = {"yolov3_tiny": 0.18, "yolov4": 0.33 if raw else 0.4, "yolov5m": 0.2 if c["size"] < 512 else 0.6}
    kw = {"conf": conf[c["net"]]} if c["net"] in DETECTORS else {}
    return topologies.NETS[c["net"]](size=c["size"], **kw)


_blobs = {}


def _blob(net, text):
    """A net's weights. Their order and number hardly ever depend on the input size, so sizes share them."""
    key = (net, tuple(synth.weight_layout(text)))
    if key not in _blobs:
        if len(_blobs) == 4:
            _blobs.clear()
        _blobs[key] = synth.make_blob(text, synth.load_factors(net))
    return _blobs[key]


_built = {"key": None, "net": None}


def _net(c):
    key = (c["net"], c["size"], c["dtype"], c["batch"], c["call"] in ("stream_u8", "list"))
    if _built["key"] != key:
        if _built["net"] is not None:
            _built["net"].close()
        _built.update(key=None, net=None)
        text = _topology(c)
        _built.update(net=Net(text, _blob(c["net"], text), c["dtype"] == "fp16", batch=c["batch"]), key=key)
    return _built["net"]


def prepare(c, seed):
    net = _net(c)
    n = c["batch"] * c["steps"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    u8 = c["call"] in ("stream_u8", "list")
    shape = (n, c["height"], c["width"], 3) if u8 else (n, 3, c["size"], c["size"])
    dtype = torch.uint8 if u8 else torch.float32
    host = torch.empty(shape, dtype=dtype, pin_memory=c["call"].startswith("stream"))
    if u8:      # one random colour per pixel of the net's input, enlarged to the image's size
        side = max(c["height"], c["width"])
        rows = torch.arange(c["height"], device="cuda") * c["size"] // side
        cols = torch.arange(c["width"], device="cuda") * c["size"] // side
    for k in range(n):      # image by image: no second batch in device memory
        if u8:
            host[k].copy_(torch.randint(0, 256, (c["size"], c["size"], 3), dtype=dtype, device="cuda", generator=g)[rows][:, cols])
        else:
            host[k].copy_(torch.rand(shape[1:], device="cuda", generator=g))
    state = {"case": c, "host": host, "images": C.c_void_p(host.data_ptr()), "msg": C.c_char_p()}
    if net.is_yolo:
        state["boxes"] = np.zeros((n, MAX_BOXES, 8), np.float32)
        state["counts"] = np.zeros(n, np.int32)
    else:
        state["out"] = np.zeros((n,) + net.last_shape, np.float32)
    return state


def run(state):
    c = state["case"]
    lib, msg, images = _net(c).lib, C.byref(state["msg"]), state["images"]
    batch, steps, call = c["batch"], c["steps"], c["call"]
    if "boxes" in state:
        boxes = state["boxes"].ctypes.data_as(C.POINTER(_ffi.BBox))
        counts = state["counts"].ctypes.data_as(C.POINTER(C.c_int))
        if call == "batch":
            rc = lib.msnhB200RunYoloBatch(msg, images, batch, boxes, MAX_BOXES, counts)
        elif call == "stream":
            rc = lib.msnhB200RunYoloStream(msg, images, steps, boxes, MAX_BOXES, counts)
        elif call == "stream_u8":
            rc = lib.msnhB200RunYoloStreamU8(msg, images, c["width"], c["height"], 1, steps, boxes, MAX_BOXES, counts)
        else:
            container = C.cast(boxes, C.POINTER(_ffi.BBoxContainer))
            rc = lib.runYoloList(msg, images, c["width"], c["height"], 3, container, counts, 1, 1)
    else:
        out = state["out"].ctypes.data_as(C.POINTER(C.c_float))
        if call == "batch":
            rc = lib.msnhB200RunClassifyBatch(msg, images, batch, out, state["out"].size)
        elif call == "stream":
            rc = lib.msnhB200RunClassifyStream(msg, images, steps, out, state["out"].size)
        else:
            rc = lib.msnhB200RunClassifyStreamU8(msg, images, c["width"], c["height"], _ffi.PREP_UNIT, 1, None, None, steps, out, state["out"].size)
    if rc != 1:
        raise RuntimeError(state["msg"].value.decode())
    if "boxes" not in state:
        return state["out"]
    # a row is x, y, w, h, objectness, class score, class (an integer), angle; rows past an image's count are zero
    return {"counts": state["counts"], "boxes": state["boxes"][..., :6], "classes": state["boxes"].view(np.int32)[..., 6]}


def work(c):
    """The images and the weights (in the plan's element type) read once, the result written once; convolution FLOPs."""
    text = _topology(c)
    weights = sum(count for _, _, count, _ in synth.weight_layout(text)) * (2 if c["dtype"] == "fp16" else 4)
    n = c["batch"] * c["steps"]
    if c["net"] in DETECTORS:
        out = n * 100 * 32           # about a hundred boxes an image
    else:
        out = n * 4 * (2 * c["size"] ** 2 if c["net"] == "fcns" else 1000)
    return {"bytes": image_bytes(c) + weights + out, "flops": gflop(c) * 1e9}


def tolerance(c):
    if c["dtype"] == "fp16":
        return {"rel": 1e-2, "differ": 0.005}       # fp16 storage; near-tied class scores may swap
    if c["net"] in DETECTORS:
        return {"rel": 1e-4, "differ": 0.005}       # fp32 sums through some hundred layers and an exp
    return {"rel": 3e-3}                            # tf32 products (10 mantissa bits), fp32 sums
