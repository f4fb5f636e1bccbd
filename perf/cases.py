"""Workloads of the image-transform-and-batch path, as programs that use this package run them.

A case names a chain of ops ("chain"), where its samples come from ("feed": tensors in GPU memory,
ordinary numpy arrays, arrays in page-locked memory, JPEG files held in memory), where the batches go
("out"), the form of the pixels in them ("cast": the bytes, x / 255, or the channel-normalised form)
and sizes.  Image heights and widths are drawn from ``h0..h1`` x ``w0..w1`` with the case's own
``shapes`` number, so a case always means the same work; the pixels (and the random crops and flips)
come from the seed.

Sizes follow the five configurations of ``mlx-data_b200/workloads.py`` where one exists.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

MEAN, STD = (0.485, 0.456, 0.406, 0.5), (0.229, 0.224, 0.225, 0.25)
CHANNELS_OF_GRAY = 1


def _package():
    """The package directory has a hyphen in its name, so it is loaded by path."""
    if "mlx_data_b200" not in sys.modules:
        root = os.path.join(os.getcwd(), "mlx-data_b200")
        spec = importlib.util.spec_from_file_location(
            "mlx_data_b200", os.path.join(root, "__init__.py"), submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["mlx_data_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["mlx_data_b200"]


def _case(name, chain, n, h, w, size, crop, c=3, cast="norm", feed="device", out="device", batches=1, shapes=0, **more):
    d = dict(chain=chain, n=n, h0=h[0], h1=h[1], w0=w[0], w1=w[1], c=c, size=size, crop=crop, cast=cast, feed=feed,
             out=out, batches=batches, shapes=shapes, **more)
    if name:
        d["name"] = name
    return d


def listed():
    return [
        # an inference service: one camera image already on the GPU, brought to a network's input
        _case("serve_1", "eval", 1, (480, 480), (640, 640), 256, 224),
        # small photographs in small batches, validation transform (configuration c1)
        _case("eval_32", "eval", 32, (200, 500), (200, 500), 256, 224, cast="scale"),
        # classification training: random area crop, resize, flip, normalise (c2)
        _case("train_256", "train", 256, (256, 800), (256, 800), 224, 224),
        # detection: shorter side to 320, every image padded to the largest of its batch (c3)
        _case("pad_64", "pad", 64, (160, 1024), (160, 1024), 320, 0, cast="scale"),
        # grey-level training data, kept as bytes in the batch (c3 with the channel reduction)
        _case("gray_96", "gray", 96, (240, 640), (240, 640), 320, 224, cast="bytes"),
        # augmentation by rotation, a per-sample angle (c4)
        _case("rotate_128", "rotate", 128, (512, 512), (512, 512), 0, 448, cast="scale"),
        # full-HD video frames in throughput-sized batches (c5)
        _case("frames_512", "train_frames", 512, (1080, 1080), (1920, 1920), 512, 512),
        # tiny images, no resize: random crop and flip, per-sample overhead counts
        _case("tiny_1024", "crop", 1024, (40, 40), (40, 40), 0, 32),
        # tiny images enlarged to a network's input
        _case("enlarge_128", "resize", 128, (32, 32), (32, 32), 224, 0),
        # what a plain script does: numpy samples in, numpy batches out, look-ahead of four
        _case("numpy_4x32", "eval", 32, (256, 640), (256, 640), 256, 224, feed="numpy", out="host", batches=4),
        # frames in page-locked memory feeding a training loop on the GPU
        _case("pinned_3x8", "eval", 8, (1080, 1080), (1920, 1920), 512, 512, feed="pinned", batches=3),
        # training from JPEG files: decode, random area crop, resize, flip, normalise
        _case("jpeg_2x32", "train", 32, (300, 500), (300, 500), 224, 224, feed="jpeg", batches=2, quality=88, sub420=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# what one draw may move at most: bytes of the largest listed case per kind of feed
_MOST = {"device": 3.4e9, "numpy": 1.4e8, "pinned": 1.6e8, "jpeg": 6e7}


def draw(rng):
    while True:
        feed = rng.choice(["device"] * 6 + ["numpy", "pinned", "jpeg"])
        chain = rng.choice(["eval", "train", "pad", "gray", "rotate", "train_frames", "crop", "resize"])
        c = rng.choice([3, 3, 3, 3, 1, 4]) if chain != "gray" and feed != "jpeg" else 3
        cast = rng.choice(["norm", "norm", "scale", "bytes"])
        shapes = rng.randrange(1 << 20)
        more = {}
        batches = 1 if feed == "device" else rng.choice([2, 3, 4])
        n = _log_int(rng, 1, 1024) if feed == "device" else _log_int(rng, 4, 48)
        if chain == "crop":
            lo = _log_int(rng, 28, 512)
            hi = rng.choice([lo, rng.randint(lo, 2 * lo)])
            size, crop = 0, rng.randint(max(8, lo // 2), lo)
        elif chain == "rotate":
            lo = _log_int(rng, 64, 768)
            hi = lo
            size, crop = 0, rng.randint(lo // 2, lo)
        elif chain == "resize":
            lo = _log_int(rng, 24, 512)
            hi = rng.choice([lo, rng.randint(lo, 2 * lo)])
            size, crop = _log_int(rng, 64, 448), 0
        else:
            lo = _log_int(rng, 96, 1080)
            hi = rng.randint(lo, min(1920, 4 * lo))
            size = _log_int(rng, max(48, hi // 10), 512)
            crop = rng.randint(size // 2, size)
        if feed == "jpeg":
            if hi > 1100:
                continue
            more = dict(quality=rng.randint(70, 95), sub420=rng.random() < 0.75)
        out = "device" if feed == "device" else rng.choice(["host", "device"])
        case = _case(None, chain, n, (lo, hi), (lo, hi), size, crop, c, cast, feed, out, batches, shapes, **more)
        w = work(case)["bytes"]
        if 2e4 < w <= _MOST[feed]:
            return case


# ------------------------------------------------------------------ shapes and work
def _shapes(case):
    rng = np.random.default_rng(case["shapes"])
    n = case["n"] * case["batches"]
    hs = rng.integers(case["h0"], case["h1"] + 1, n)
    ws = rng.integers(case["w0"], case["w1"] + 1, n)
    return [(int(h), int(w)) for h, w in zip(hs, ws)]


def _resized(case, h, w):
    """Output size of the resize, and the source pixels it has to read along each axis."""
    size, crop = case["size"], case["crop"]
    if case["chain"] == "resize":
        return size, size, h, w
    if case["chain"] == "train":
        return size, size, h * math.sqrt(0.54), w * math.sqrt(0.54)   # mean area of the random crop
    scale = size / min(h, w)
    th, tw = round(h * scale), round(w * scale)
    if case["chain"] in ("pad",):
        return th, tw, h, w
    return min(th, crop), min(tw, crop), h * min(1.0, crop / th), w * min(1.0, crop / tw)


def work(case):
    """Every source pixel the chain needs read once, every batch value written once; the multiply-adds of a
    two-pass triangle filter over the taps that its definition gives."""
    c, n = case["c"], case["n"]
    co = CHANNELS_OF_GRAY if case["chain"] == "gray" else c
    elem = 1 if case["cast"] == "bytes" else 4
    read = wrote = flops = 0.0
    shapes = _shapes(case)
    for b in range(case["batches"]):
        slot_h = slot_w = 0
        for h, w in shapes[b * n:(b + 1) * n]:
            if case["chain"] in ("crop", "rotate"):
                oh, ow, fh, fw = case["crop"], case["crop"], case["crop"], case["crop"]
            else:
                oh, ow, fh, fw = _resized(case, h, w)
                ty, tx = 2 * max(1.0, fh / oh), 2 * max(1.0, fw / ow)
                flops += 2 * c * (oh * fw * ty + oh * ow * tx)
            read += fh * fw * c * (0.15 if case["feed"] == "jpeg" else 1.0)
            slot_h, slot_w = max(slot_h, oh), max(slot_w, ow)
        wrote += n * slot_h * slot_w * co * elem
    return {"bytes": read + wrote, "flops": flops}


def tolerance(case):
    """Crops, flips, rotations, bytes and casts are exact.  A resize sums in float32 and then rounds to a byte:
    another order of the same sums moves about one value in ten thousand by one level of 255."""
    if case["chain"] in ("crop", "rotate"):
        return "exact"
    return {"rel": 1e-4, "max": 0.05, "differ": 1e-4}


# ------------------------------------------------------------------ inputs
def _images(shapes, c, seed):
    """uint8 [H, W, C] tensors that look like photographs to a filter: smooth fields with fine noise."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out = []
    for h, w in shapes:
        coarse = torch.rand((1, c, h // 24 + 2, w // 24 + 2), device="cuda", generator=gen) * 230 + 12
        img = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear")[0].permute(1, 2, 0)
        img = img + torch.randn((h, w, c), device="cuda", generator=gen) * 6
        out.append(img.clamp_(0, 255).to(torch.uint8).contiguous())
    return out


# The luminance tables of the JPEG standard's annex K: quantisation in row order, Huffman code counts and symbols.
_ZIGZAG = [k for s in range(15) for k in sorted((k for k in range(64) if k // 8 + k % 8 == s),
                                                key=lambda k: k // 8 if s % 2 else k % 8)]
_QUANT = np.array([
    16, 11, 10, 16, 24, 40, 51, 61, 12, 12, 14, 19, 26, 58, 60, 55, 14, 13, 16, 24, 40, 57, 69, 56, 14, 17, 22, 29, 51, 87,
    80, 62, 18, 22, 37, 56, 68, 109, 103, 77, 24, 35, 55, 64, 81, 104, 113, 92, 49, 64, 78, 87, 103, 121, 120, 101, 72, 92,
    95, 98, 112, 100, 103, 99])
_DC_BITS, _DC_SYMBOLS = [0, 1, 5, 1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0], list(range(12))
_AC_BITS = [0, 2, 1, 3, 3, 2, 4, 3, 5, 5, 4, 4, 0, 0, 1, 0x7D]
_AC_SYMBOLS = list(bytes.fromhex(
    "01020300041105122131410613516107227114328191a1082342b1c11552d1f02433627282090a161718191a25262728292a3435363738393a"
    "434445464748494a535455565758595a636465666768696a737475767778797a838485868788898a92939495969798999aa2a3a4a5a6a7a8a9"
    "aab2b3b4b5b6b7b8b9bac2c3c4c5c6c7c8c9cad2d3d4d5d6d7d8d9dae1e2e3e4e5e6e7e8e9eaf1f2f3f4f5f6f7f8f9fa"))


def _codes(bits, symbols):
    code, at = 0, 0
    value, length = np.zeros(256, np.int64), np.zeros(256, np.int64)
    for n in range(16):
        for _ in range(bits[n]):
            value[symbols[at]], length[symbols[at]] = code, n + 1
            code += 1
            at += 1
        code <<= 1
    return value, length


def _jpeg(img, quality, sub420):
    """A baseline JPEG file of a uint8 [H, W, 3] array (numpy), as bytes in a uint8 array."""
    h, w, _ = img.shape
    scale = 5000 / quality if quality < 50 else 200 - 2 * quality
    quant = np.clip((_QUANT * scale + 50) // 100, 1, 255).astype(np.int64)
    rgb = img.astype(np.float32)
    y = rgb @ np.float32([0.299, 0.587, 0.114])
    planes = [y, (rgb[..., 2] - y) * np.float32(0.5 / 0.886) + 128, (rgb[..., 0] - y) * np.float32(0.5 / 0.701) + 128]
    f = 2 if sub420 else 1
    mh, mw = -(-h // (8 * f)), -(-w // (8 * f))
    k = np.arange(8)
    dct = np.cos((2 * k[None] + 1) * k[:, None] * np.pi / 16) * np.where(k[:, None] == 0, math.sqrt(0.125), 0.5)
    dct = dct.astype(np.float32)
    blocks = []   # per component: [mcus, blocks of the mcu, 64] in zigzag order
    for i, p in enumerate(planes):
        p = np.pad(p, ((0, mh * 8 * f - h), (0, mw * 8 * f - w)), mode="edge") - 128
        g = f if i == 0 else 1
        if i > 0 and f == 2:
            p = (p[::2, ::2] + p[1::2, ::2] + p[::2, 1::2] + p[1::2, 1::2]) * np.float32(0.25)
        b = p.reshape(mh, g, 8, mw, g, 8).transpose(0, 3, 1, 4, 2, 5).reshape(mh * mw, g * g, 8, 8)
        b = np.rint((dct @ b @ dct.T).reshape(mh * mw, g * g, 64) / quant).astype(np.int64)
        blocks.append(b[:, :, _ZIGZAG])
    zz = np.concatenate(blocks, axis=1)
    comp = np.concatenate([[i] * b.shape[1] for i, b in enumerate(blocks)])
    for i in range(3):
        dc = zz[:, comp == i, 0].reshape(-1)
        zz[:, comp == i, 0] = np.diff(dc, prepend=0).reshape(len(zz), -1)
    zz = zz.reshape(-1, 64)
    dc_code, dc_len = _codes(_DC_BITS, _DC_SYMBOLS)
    ac_code, ac_len = _codes(_AC_BITS, _AC_SYMBOLS)

    def magnitude(v):
        size = np.frexp(np.abs(v).astype(np.float64))[1].astype(np.int64)
        return size, np.where(v < 0, v + (1 << size) - 1, v)

    size, extra = magnitude(zz[:, 0])
    order = [np.arange(len(zz)) * 256]
    value = [(dc_code[size] << size) | extra]
    length = [dc_len[size] + size]
    blk, pos = np.nonzero(zz[:, 1:])
    pos = pos + 1
    first = np.ones(len(blk), bool)
    first[1:] = blk[1:] != blk[:-1]
    run = pos - np.where(first, 0, np.concatenate([[0], pos[:-1]])) - 1
    size, extra = magnitude(zz[blk, pos])
    symbol = (run % 16) * 16 + size
    order.append(blk * 256 + pos * 2 + 1)
    value.append((ac_code[symbol] << size) | extra)
    length.append(ac_len[symbol] + size)
    zrl = np.repeat(np.arange(len(blk)), run // 16)
    order.append(blk[zrl] * 256 + pos[zrl] * 2)
    value.append(np.full(len(zrl), ac_code[0xF0]))
    length.append(np.full(len(zrl), ac_len[0xF0]))
    eob = np.nonzero(zz[:, 63] == 0)[0]
    order.append(eob * 256 + 200)
    value.append(np.full(len(eob), ac_code[0]))
    length.append(np.full(len(eob), ac_len[0]))
    at = np.argsort(np.concatenate(order), kind="stable")
    value, length = np.concatenate(value)[at], np.concatenate(length)[at]
    ends = np.cumsum(length)
    shift = np.repeat(ends, length) - 1 - np.arange(ends[-1])
    data = np.packbits(np.concatenate([((np.repeat(value, length) >> shift) & 1).astype(np.uint8),
                                       np.ones(-int(ends[-1]) % 8, np.uint8)]))
    data = np.insert(data, np.nonzero(data == 255)[0] + 1, 0)

    def segment(marker, body):
        return bytes([0xFF, marker]) + (len(body) + 2).to_bytes(2, "big") + bytes(body)

    s = 0x22 if sub420 else 0x11
    head = b"\xff\xd8" + segment(0xDB, bytes([0]) + bytes(int(quant[k]) for k in _ZIGZAG))
    head += segment(0xC0, bytes([8]) + h.to_bytes(2, "big") + w.to_bytes(2, "big") +
                    bytes([3, 1, s, 0, 2, 0x11, 0, 3, 0x11, 0]))
    head += segment(0xC4, bytes([0x00] + _DC_BITS + _DC_SYMBOLS)) + segment(0xC4, bytes([0x10] + _AC_BITS + _AC_SYMBOLS))
    head += segment(0xDA, bytes([3, 1, 0, 2, 0, 3, 0, 0, 63, 0]))
    return np.frombuffer(head + data.tobytes() + b"\xff\xd9", dtype=np.uint8)


def _chain(ds, case):
    """The fluent calls of a user's program between the source and the batch node."""
    k, size, crop = case["chain"], case["size"], case["crop"]
    if k == "eval":
        return ds.image_resize_smallest_side("image", size).image_center_crop("image", crop, crop)
    if k == "train":
        ds = ds.image_random_area_crop("image", area_range=(0.08, 1.0), aspect_ratio_range=(3 / 4, 4 / 3))
        return ds.image_resize("image", size, size).image_random_h_flip("image", 0.5)
    if k == "train_frames":
        ds = ds.image_resize_smallest_side("image", size).image_center_crop("image", crop, crop)
        return ds.image_random_h_flip("image", 0.5)
    if k == "pad":
        return ds.image_resize_smallest_side("image", size)
    if k == "gray":
        ds = ds.image_resize_smallest_side("image", size).image_center_crop("image", crop, crop)
        return ds.image_channel_reduction("image", "default")
    if k == "rotate":
        ds = ds.image_rotate("image", angle=0.0, angle_key="angle", crop=True).image_random_h_flip("image", 0.5)
        return ds.image_center_crop("image", crop, crop)
    if k == "crop":
        return ds.image_random_crop("image", crop, crop).image_random_h_flip("image", 0.5)
    return ds.image_resize("image", size, size)


def prepare(case, seed):
    dx = _package()
    dx.core.set_device(torch.cuda.current_device())
    dx.core.set_rgba_resize_independent(True)
    shapes = _shapes(case)
    if case["feed"] == "jpeg":
        files = [_jpeg(t.cpu().numpy(), case["quality"], case["sub420"]) for t in _images(shapes[:16], 3, seed)]
        arrays = [files[i % len(files)] for i in range(len(shapes))]
    else:
        arrays = _images(shapes, case["c"], seed)
        if case["feed"] == "numpy":
            arrays = [t.cpu().numpy() for t in arrays]
        elif case["feed"] == "pinned":
            held = []
            for t in arrays:
                held.append(dx.core.pinned_empty(list(t.shape), "uint8"))
                held[-1][...] = t.cpu().numpy()
            arrays = held
    samples = [{"image": a} for a in arrays]
    if case["chain"] == "rotate":
        for s, a in zip(samples, np.random.default_rng(seed).uniform(-30.0, 30.0, len(samples))):
            s["angle"] = np.float64(a)
    # where batches go is fixed when the batch node is built
    dx.core.set_device_output(case["out"] == "device")
    dx.core.set_stream(torch.cuda.current_stream().cuda_stream, case["feed"] == "device")
    ds = dx.buffer_from_vector(samples)
    if case["feed"] == "jpeg":
        # files are decoded by worker threads, the batches after them are made in order
        ds = ds.load_image("image", from_memory=True).ordered_prefetch(32, 8)
    ds = _chain(ds, case).batch(case["n"])
    if case["cast"] != "bytes":
        c = case["c"] if case["chain"] != "gray" else 1
        ds = ds.key_cast("image", **({} if case["cast"] == "scale" else dict(mean=list(MEAN[:c]), std=list(STD[:c]))))
    # a chain that draws at random stays on one thread, so that its draws come in one order
    if case["feed"] in ("numpy", "pinned"):
        ds = ds.ordered_prefetch(4, 1 if case["chain"] in ("train", "train_frames", "rotate", "crop") else 4)
    torch.cuda.synchronize()
    return {"package": dx, "pipe": ds, "seed": seed, "device": case["out"] == "device", "single": case["feed"] == "device"}


def run(state):
    """One epoch over the state's samples: a batch from GPU memory, or a few from the host through the look-ahead."""
    dx = state["package"]
    dx.core.set_state(state["seed"])
    if state["single"]:
        batches = [state["pipe"][0]["image"]]
    else:
        state["pipe"].reset()
        batches = [b["image"] for b in state["pipe"]]
    if state["device"]:
        return [torch.as_tensor(b, device="cuda") for b in batches]
    return batches
