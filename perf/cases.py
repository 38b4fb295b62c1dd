"""What a user of this encoder has it do, as cases to time: single frames of the smallest to the largest sizes
(device-resident and host input), the one-call Python entry point, several live streams, a batch of mixed
resolutions, learned decisions, and one gradient of the decision network's training.

Every encode returns the user's output buffers with the whole .jxl files and their sizes; the gradient returns the whole gradient and the per-sample
statistics. Frames come from a seeded generator on the GPU with the content of cujpegxl_b200.synth: a gradient,
1/f^1.5 noise, hard edges, fine stripes, smooth chroma. Distances and sizes are those of this repository's tests
and benchmark, and 7680x4320 as the largest frame of a video pipeline."""

import math

import numpy as np
import torch

import cujpegxl_b200 as jxl
from cujpegxl_b200 import _capi
from cujpegxl_b200.acsnet import DEFAULT_WEIGHTS, QF, SPLIT, AcsNet, Trainer, unpack_blob

DEV = "cuda"
QF_WEIGHT = 0.5
TRAIN_TILES = 512


def listed():
    return [
        # The smallest call: a thumbnail or preview of one AC group, where only latency counts.
        {"name": "preview_256x256", "kind": "device", "width": 256, "height": 256, "distance": 1.0, "pad": 0},
        # The one-call Python entry point on a host array: a script that encodes a frame now and then.
        {"name": "oneshot_1280x720", "kind": "oneshot", "width": 1280, "height": 720, "distance": 1.0, "pad": 0},
        # A decoder's or a renderer's 720p frame, already on the device.
        {"name": "device_1280x720", "kind": "device", "width": 1280, "height": 720, "distance": 1.0, "pad": 0},
        # A camera's 1080p frame in host memory through a kept encoder.
        {"name": "host_1920x1080", "kind": "host", "width": 1920, "height": 1080, "distance": 1.0, "pad": 0},
        # A cropped picture: partial tiles and groups on both sides, a pitch of its own, a stronger compression.
        {"name": "ragged_1000x1480", "kind": "device", "width": 1000, "height": 1480, "distance": 2.5, "pad": 40},
        # The headline frame: 3840x2160 at distance 1.
        {"name": "device_3840x2160", "kind": "device", "width": 3840, "height": 2160, "distance": 1.0, "pad": 0},
        # The same frame for an archive: more tokens, larger files.
        {"name": "archive_3840x2160", "kind": "device", "width": 3840, "height": 2160, "distance": 0.4, "pad": 0},
        # The largest single frame.
        {"name": "device_7680x4320", "kind": "device", "width": 7680, "height": 4320, "distance": 1.0, "pad": 0},
        # Learned split and quant field on the headline frame.
        {"name": "learned_3840x2160", "kind": "learned", "width": 3840, "height": 2160, "distance": 1.0, "pad": 0},
        # A server with eight live 1080p streams: one frame of each, asynchronously, files into page-locked memory.
        {"name": "streams_8x1080p", "kind": "streams", "count": 8, "width": 1920, "height": 1080, "distance": 1.0,
         "pad": 0},
        # A transcoding job's batch of uneven resolutions.
        {"name": "batch_16_mixed", "kind": "batch", "distance": 1.0,
         "mix": "1280x720:4 1920x1080:4 2560x1440:4 3840x2160:2 4096x2160:2"},
        # Training of the decision network: the gradient of one batch.
        {"name": "train_gradient_1024", "kind": "train", "samples": 1024, "distance": 1.0},
    ]


def draw(rng):
    kind = rng.choice(["device"] * 6 + ["host"] * 2 + ["oneshot"] + ["learned"] * 2 + ["streams"] * 2 + ["batch"] * 2 +
                      ["train"])
    distance = round(math.exp(rng.uniform(math.log(0.3), math.log(6.0))), 3)

    def side(lo, hi):
        return 8 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 8))

    if kind == "train":
        return {"kind": kind, "samples": int(math.exp(rng.uniform(math.log(64), math.log(4096)))), "distance": distance}
    if kind == "batch":
        sizes = ["640x360", "1280x720", "1920x1080", "2560x1440", "1080x1920", "1000x1480", "3840x2160"]
        mix = ["%s:%d" % (s, rng.randint(1, 4)) for s in rng.sample(sizes, rng.randint(2, 3))]
        return {"kind": kind, "distance": distance, "mix": " ".join(mix)}
    if kind == "streams":
        return {"kind": kind, "count": rng.randint(2, 8), "width": side(264, 1920), "height": side(264, 1080),
                "distance": distance, "pad": 8 * rng.choice([0, 0, 1, 5])}
    top = 2048 if kind == "oneshot" else 7680
    width = side(64, top)
    height = side(64, top * 9 / 16)
    return {"kind": kind, "width": width, "height": height, "distance": distance,
            "pad": 0 if kind in ("host", "oneshot") else 8 * rng.choice([0, 0, 1, 5])}


def _sizes(case):
    """Every frame's (width, height) in the order of the outputs."""
    if case["kind"] == "batch":
        out = []
        for part in case["mix"].split():
            wh, n = part.split(":")
            w, h = wh.split("x")
            out += [(int(w), int(h))] * int(n)
        return out
    return [(case["width"], case["height"])] * case.get("count", 1)


# ---- inputs ----

def _frequency(h, w):
    fy = torch.fft.fftfreq(h, device=DEV)[:, None]
    fx = torch.fft.rfftfreq(w, device=DEV)[None, :]
    return fy * fy + fx * fx


def _frame(width, height, seed):
    """One NV12 frame: (luma [H][W], chroma [H/2][W]) uint8 on the device."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    x = torch.arange(width, device=DEV, dtype=torch.float32)[None, :]
    y = torch.arange(height, device=DEV, dtype=torch.float32)[:, None]
    luma = 64.0 + 96.0 * (0.6 * x / width + 0.4 * y / height)
    spec = torch.fft.rfft2(torch.randn((height, width), generator=gen, device=DEV))
    f2 = _frequency(height, width)
    f2[0, 0] = 1.0
    amp = f2 ** -0.75
    amp[0, 0] = 0.0
    noise = torch.fft.irfft2(spec * amp, s=(height, width))
    luma = luma + noise * (12.0 / noise.std())
    for i in range(40):
        rw, rh = int(rng.integers(64, 513)), int(rng.integers(64, 513))
        x0, y0 = int(rng.integers(0, max(1, width - rw + 1))), int(rng.integers(0, max(1, height - rh + 1)))
        step = float(rng.uniform(30.0, 80.0)) * (1.0 if rng.random() < 0.5 else -1.0)
        part = luma[y0:y0 + rh, x0:x0 + rw]
        sx, sy = x[:, :part.shape[1]], y[:part.shape[0]]
        if i < 20:
            at = float(rng.random())
            mask = (sx >= at * part.shape[1]) if rng.random() < 0.5 else (sy >= at * part.shape[0])
        else:
            angle = float(rng.uniform(0.0, math.pi))
            mask = (sx - part.shape[1] * float(rng.random())) * math.cos(angle) + \
                (sy - part.shape[0] * float(rng.random())) * math.sin(angle) >= 0.0
        part += step * mask
    luma = luma.round().clamp(0, 255)
    for _ in range(8):
        x0, y0 = int(rng.integers(0, max(1, width - 63))), int(rng.integers(0, max(1, height - 63)))
        period = int(rng.integers(1, 3))
        part = luma[y0:y0 + 64, x0:x0 + 64]
        along = x[:, :part.shape[1]] if rng.random() < 0.5 else y[:part.shape[0]]
        part[:] = torch.where((along / period).floor() % 2 == 0, 16.0, 235.0)
    ch, cw = height // 2, width // 2
    blur = torch.exp(-2.0 * (math.pi * 8.0) ** 2 * _frequency(ch, cw))
    chroma = torch.empty((ch, cw, 2), device=DEV)
    for c in range(2):
        p = torch.fft.irfft2(torch.fft.rfft2(torch.randn((ch, cw), generator=gen, device=DEV)) * blur, s=(ch, cw))
        chroma[:, :, c] = 128.0 + 20.0 * p / p.abs().max()
    return luma.to(torch.uint8), chroma.round().clamp(0, 255).to(torch.uint8).reshape(ch, width)


def _device_frame(width, height, pad, seed):
    """A frame as a decoder hands it over: (planes kept alive, (luma, chroma, luma_pitch, chroma_pitch))."""
    luma, chroma = _frame(width, height, seed)
    pitch = width + pad
    planes = torch.zeros((height + height // 2, pitch), dtype=torch.uint8, device=DEV)
    planes[:height, :width] = luma
    planes[height:, :width] = chroma
    at = planes.data_ptr()
    return planes, (at, at + height * pitch, pitch, pitch)


def _host_frame(width, height, seed):
    luma, chroma = _frame(width, height, seed)
    return torch.cat([luma.reshape(-1), chroma.reshape(-1)]).cpu().numpy()


def _room(width, height):
    """Bytes of a user's output buffer for one file (several times what the smallest distance here needs)."""
    return width * height + 65536


def _flags(width, height):
    return jxl.SINGLE_GROUP if width <= 256 and height <= 256 else 0


def _train_inputs(case, seed):
    """Tiles of XYB-like pictures, labels, and the soft targets the trainer takes."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n = case["samples"]
    spec = torch.fft.rfft2(torch.randn((TRAIN_TILES, 3, 64, 64), generator=gen, device=DEV))
    f2 = _frequency(64, 64)
    f2[0, 0] = 1.0
    p = torch.fft.irfft2(spec * f2 ** -0.75, s=(64, 64))[:, :, :34, :34]
    p = p / p.std()
    scale = torch.tensor([0.004, 0.12, 0.12], device=DEV)[None, :, None, None]
    shift = torch.tensor([0.0, 0.45, 0.45], device=DEV)[None, :, None, None]
    tiles = (p * scale + shift).contiguous()
    index = torch.randint(0, TRAIN_TILES, (n,), generator=gen, device=DEV, dtype=torch.int32)
    log2d = torch.rand((n,), generator=gen, device=DEV) * 3.0 - 1.0 + math.log2(case["distance"]) * 0.25
    cls = torch.randint(0, 17, (n,), generator=gen, device=DEV).to(torch.int8)
    qf = torch.rand((n, 16), generator=gen, device=DEV) * 2.0 + 2.0
    soft = torch.softmax(4.0 * torch.randn((n, 17), generator=gen, device=DEV), dim=1).contiguous()
    return tiles, index, log2d, cls, qf, soft


def prepare(case, seed):
    kind = case["kind"]
    d = case["distance"]
    if kind == "train":
        params, norm = unpack_blob(DEFAULT_WEIGHTS.read_bytes())
        return {"kind": kind, "trainer": Trainer(params, norm, case["samples"]), "data": _train_inputs(case, seed)}
    sizes = _sizes(case)
    w, h = sizes[0]
    if kind == "oneshot":
        # The one-call entry point takes frames of more than one AC group.
        w = max(w, 264)
        return {"kind": kind, "nv12": _host_frame(w, h, seed), "width": w, "height": h, "distance": d,
                "files": [np.zeros(_room(w, h), np.uint8)]}
    if kind == "host":
        return {"kind": kind, "nv12": _host_frame(w, h, seed), "enc": jxl.Encoder(w, h, d, flags=_flags(w, h)),
                "files": [np.zeros(_room(w, h), np.uint8)]}
    frames = [_device_frame(fw, fh, case.get("pad", 0), seed + 1000 * i) for i, (fw, fh) in enumerate(sizes)]
    state = {"kind": kind, "planes": [f[0] for f in frames], "inputs": [f[1] for f in frames]}
    if kind != "streams":
        state["files"] = [np.zeros(_room(fw, fh), np.uint8) for fw, fh in sizes]
    if kind == "batch":
        state["batch"] = jxl.Batch([(fw, fh, d) for fw, fh in sizes])
        return state
    state["enc"] = [jxl.Encoder(fw, fh, d, flags=_flags(fw, fh)) for fw, fh in sizes]
    if kind == "learned":
        state["net"] = AcsNet.load()
        for e in state["enc"]:
            e.set_acsnet(state["net"], margin=0.2, flags=SPLIT | QF)
    if kind == "streams":
        state["files"] = [torch.zeros(_room(fw, fh), dtype=torch.uint8, pin_memory=True) for fw, fh in sizes]
        state["words"] = torch.zeros((len(sizes), 2), dtype=torch.int64, pin_memory=True)
    return state


def _keep(state, i, data):
    """A file into its place in the program's output buffer; its size."""
    state["files"][i][:len(data)] = np.frombuffer(data, np.uint8)
    return len(data)


def run(state):
    kind = state["kind"]
    if kind == "train":
        tiles, index, log2d, cls, qf, soft = state["data"]
        grad, stats = state["trainer"].gradient(tiles, index, log2d, cls, qf, QF_WEIGHT, soft)
        return {"grad": grad, "stats": stats}
    if kind == "device" or kind == "learned":
        f = state["files"][0]
        sizes = [state["enc"][0].encode_device_into(*state["inputs"][0], f.ctypes.data, f.size)]
    elif kind == "host":
        sizes = [_keep(state, 0, state["enc"].encode_host(state["nv12"]))]
    elif kind == "oneshot":
        sizes = [_keep(state, 0, jxl.encode(state["nv12"], state["width"], state["height"],
                                            distance=state["distance"]))]
    elif kind == "streams":
        lib = _capi.lib()
        for i, e in enumerate(state["enc"]):
            e.enqueue(*state["inputs"][i])
            f = state["files"][i]
            _capi.check("enqueue_readback", lib.cujpegxl_b200_encoder_enqueue_readback(
                e.handle, f.data_ptr(), f.numel(), state["words"][i].data_ptr()))
        sizes = [e.result()[0] for e in state["enc"]]
    else:
        b = state["batch"]
        b.encode(state["inputs"])
        b.sync()
        sizes = [_keep(state, i, b.read(i)) for i in range(len(state["inputs"]))]
    return {"files": state["files"], "sizes": sizes}


def work(case):
    if case["kind"] == "train":
        n = case["samples"]
        # Multiply-adds of the four layers (16x16, 8x8, 4x4 and 4x4 outputs of 32 channels): forward, weight
        # gradient, and data gradient of all layers but the first.
        macs = [256 * 32 * 36, 64 * 32 * 288, 16 * 32 * 288, 16 * 18 * 288]
        return {"bytes": 4.0 * (min(n, TRAIN_TILES) * 3 * 34 * 34 + n * (2 + 16 + 17 + 4) + 2 * 30336),
                "flops": 2.0 * n * (3 * sum(macs) - macs[0])}
    pixels = sum(w * h for w, h in _sizes(case))
    # NV12 in once, the file (about 0.5 bit a pixel at distance 1) out once. Operations of the float path that no
    # encoder of these files avoids: colour conversion, sharpening and one separable transform of three channels.
    return {"bytes": pixels * (1.5 + 0.0625 / max(case["distance"], 0.25)), "flops": pixels * 400.0}


def tolerance(case):
    # Files are compared byte for byte. The gradient's BF16 activations and weights are rounded at every layer.
    return {"rel": 0.02} if case["kind"] == "train" else "exact"


def exact(case, seed):
    if case["kind"] != "train":
        return None
    params, norm = unpack_blob(DEFAULT_WEIGHTS.read_bytes())
    tiles, index, log2d, cls, qf, soft = _train_inputs(case, seed)
    f64 = torch.float64
    flat = torch.tensor(params, device=DEV, dtype=f64, requires_grad=True)
    ks = [80, 288, 288, 288]
    at, ws = 0, []
    for k in ks:
        ws.append(flat[at:at + 32 * k].reshape(32, k))
        at += 32 * k
    bs = [flat[at + 32 * i:at + 32 * (i + 1)] for i in range(4)]
    norm = torch.tensor(norm, device=DEV, dtype=f64)
    x = (tiles.to(f64)[index.long()] - norm[4:7][None, :, None, None]) * norm[0:3][None, :, None, None]
    dist = ((log2d.to(f64) - norm[7]) * norm[3])[:, None, None, None].expand(-1, 1, 34, 34)
    x = torch.cat([x, dist, torch.zeros((x.shape[0], 4, 34, 34), device=DEV, dtype=f64)], dim=1)
    for i, (stride, pad) in enumerate(((2, 0), (2, 1), (2, 1), (1, 1))):
        cin = x.shape[1]
        kernel = ws[i][:, :9 * cin].reshape(32, 3, 3, cin).permute(0, 3, 1, 2)
        # Unfolded by hand: the convolution as one product in 64 bits.
        cols = torch.nn.functional.unfold(x, 3, padding=pad, stride=stride)
        x = (kernel.reshape(32, -1) @ cols + bs[i][None, :, None])
        side = int(round(math.sqrt(x.shape[2])))
        x = x.reshape(x.shape[0], 32, side, side)
        if i < 3:
            x = torch.relu(x)
    out = x.reshape(x.shape[0], 32, 16)
    logits = out[:, 1:18].sum(dim=2) / 16.0
    ce = torch.logsumexp(logits, dim=1) - (soft.to(f64) * logits).sum(dim=1)
    sq = ((out[:, 0] - qf.to(f64)) ** 2).mean(dim=1)
    grad, = torch.autograd.grad((ce + QF_WEIGHT * sq).mean(), flat)
    top2 = torch.softmax(logits, dim=1).topk(2, dim=1).values
    hit = (logits.argmax(dim=1) == cls.long()).to(f64)
    stats = torch.stack([ce, sq, hit, top2[:, 0] - top2[:, 1]], dim=1).detach()
    return {"grad": grad, "stats": stats}
