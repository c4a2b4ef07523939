"""What the framework is timed on: the record path from encoded records in host memory to augmented batches, and the batch
kernels alone.  Each case is a configuration a training or serving program runs, at the sizes this repository's own
benchmark and tests use.

The records are synthetic, made on the GPU from a seed: pictures with the spectrum of photographs (octaves of smooth noise,
flat shapes with hard edges, a little sensor noise) as baseline JPEG files with the standard's own quantiser and Huffman
tables, MJPEG clips in AVI files, PNG masks, 16-bit audio.
"""
import ctypes as C
import json
import math
import struct
import zlib

import numpy as np
import torch

from aeon_b200 import _lib as L
from aeon_b200 import kernels as K
from aeon_b200.provider import Provider

MEAN, STD = [123.7 / 255, 116.3 / 255, 103.5 / 255], [58.4 / 255, 57.1 / 255, 57.4 / 255]
# random-area crop + flip, and the same with every photometric stage: how classification networks are trained
AUG_CROP = {"type": "image", "crop_enable": True, "center": False, "do_area_scale": True, "scale": [0.08, 1.0],
            "horizontal_distortion": [0.75, 1.3333334], "flip_enable": True}
AUG_PHOTO = dict(AUG_CROP, contrast=[0.6, 1.4], brightness=[0.6, 1.4], saturation=[0.6, 1.4], hue=[-18, 18], lighting=[0.0, 0.1],
                 mean=MEAN, stddev=STD)
CLASSES = ["class%02d" % i for i in range(20)]
SSD_SAMPLERS = [{"max_sample": 1, "max_trials": 1}] + [
    {"max_sample": 1, "max_trials": 50, "sampler": {"scale": [0.3, 1.0], "aspect_ratio": [0.5, 2.0]}, "sample_constraint": c}
    for c in ({"min_jaccard_overlap": 0.1}, {"min_jaccard_overlap": 0.3}, {"min_jaccard_overlap": 0.5},
              {"min_jaccard_overlap": 0.7}, {"min_jaccard_overlap": 0.9}, {"max_jaccard_overlap": 1.0})]


def listed():
    return [
        # one request of a serving program: one photo, centre crop, normalised float; nothing but latency
        {"name": "serve_one", "kind": "classify", "batch": 1, "out": 224, "lo": 375, "hi": 500, "quality": 90, "sampling": "420",
         "restart": False, "aug": "eval", "dtype": "float", "deliver": "device", "depth": 1},
        # a training step of a classification network that takes bytes from host memory
        {"name": "cls_u8_b128_host", "kind": "classify", "batch": 128, "out": 224, "lo": 256, "hi": 512, "quality": 90, "sampling": "420",
         "restart": False, "aug": "crop", "dtype": "uint8_t", "deliver": "host", "depth": 1},
        # the same with the full photometric chain and normalised floats left on the GPU, one batch at a time
        {"name": "cls_f32_b256", "kind": "classify", "batch": 256, "out": 224, "lo": 256, "hi": 512, "quality": 90, "sampling": "420",
         "restart": False, "aug": "photo", "dtype": "float", "deliver": "device", "depth": 1},
        # a stretch of an epoch: four such batches in flight, as a training loop keeps them
        {"name": "cls_f32_b256_x4", "kind": "classify", "batch": 256, "out": 224, "lo": 256, "hi": 512, "quality": 90, "sampling": "420",
         "restart": False, "aug": "photo", "dtype": "float", "deliver": "device", "depth": 4},
        # the three batch kernels of that configuration alone, compressed scans and tables resident in device memory
        {"name": "kernels_f32_b256", "kind": "kernels", "batch": 256, "out": 224, "lo": 256, "hi": 512, "quality": 90, "sampling": "420",
         "restart": False, "aug": "photo", "dtype": "float"},
        # photos as cameras write them (4:2:2, a restart marker after every MCU row), shrunk with area averaging to HWC bytes
        {"name": "camera_area_b32", "kind": "classify", "batch": 32, "out": 224, "lo": 900, "hi": 1400, "quality": 92, "sampling": "422",
         "restart": True, "aug": "area", "dtype": "uint8_t", "deliver": "device", "depth": 1},
        # single-shot detection: expand, patch sampling against the boxes, 300 x 300 floats and the box buffers
        {"name": "ssd_b32", "kind": "ssd", "batch": 32, "out": 300, "lo": 375, "hi": 500, "quality": 90},
        # action recognition: MJPEG clips of 16 frames
        {"name": "video_b32", "kind": "video", "batch": 32, "frames": 16, "width": 171, "height": 128, "out": 112, "quality": 90},
        # speech: log-mel with 20 ms frames, and cepstra with 25 ms frames
        {"name": "logmel_b64", "kind": "audio", "batch": 64, "seconds": 16.0, "frame": 320, "filters": 64, "cepstra": 0},
        {"name": "mfcc_b32", "kind": "audio", "batch": 32, "seconds": 16.0, "frame": 400, "filters": 40, "cepstra": 13},
        # region-proposal detection: 1000 x 1000 pictures with anchor labels and regression targets
        {"name": "rcnn_b4", "kind": "rcnn", "batch": 4, "out": 1000, "lo": 375, "hi": 500, "quality": 90, "scale": 1.6},
        # segmentation: photo and class mask rotated and cropped together
        {"name": "segment_b16", "kind": "segment", "batch": 16, "out": 256, "lo": 375, "hi": 500, "quality": 90, "angle": 15},
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["classify"] * 5 + ["kernels", "ssd", "video", "audio", "audio", "rcnn", "segment"])
    quality = rng.choice([75, 85, 90, 95])
    if kind in ("classify", "kernels"):
        lo = size(96, 512)
        c = {"kind": kind, "batch": size(1, 256), "out": size(64, 320), "lo": lo, "hi": min(640, int(lo * rng.uniform(1.0, 2.0)) + 1),
             "quality": quality, "sampling": rng.choice(["420", "420", "420", "422", "444", "grey"]), "restart": rng.random() < 0.2,
             "aug": rng.choice(["crop", "photo", "photo", "eval", "area"]), "dtype": rng.choice(["uint8_t", "float"])}
        if kind == "classify":
            c.update(deliver=rng.choice(["device", "device", "host"]), depth=rng.choice([1, 1, 1, 3]))
        if c["aug"] == "area" and kind == "kernels":
            c["aug"] = "crop"
        if c["aug"] in ("photo", "eval"):
            c["dtype"] = "float"  # their outputs are normalised
        if c["lo"] > 320:
            c["batch"] = max(1, c["batch"] // 2)  # no dearer than the largest listed case
        return c
    if kind == "ssd":
        return {"kind": kind, "batch": size(2, 64), "out": rng.choice([300, 512]), "lo": 300, "hi": 500, "quality": quality}
    if kind == "video":
        w = size(100, 320)
        return {"kind": kind, "batch": size(1, 32), "frames": rng.choice([8, 16, 32]), "width": w, "height": int(0.75 * w), "out": size(64, 128),
                "quality": quality}
    if kind == "audio":
        cepstra = rng.choice([0, 13, 20])
        return {"kind": kind, "batch": size(1, 64), "seconds": float(size(2, 16)), "frame": rng.choice([256, 320, 400, 400, 441, 512]),
                "filters": rng.choice([26, 40] if cepstra else [26, 40, 64, 80]), "cepstra": cepstra}
    if kind == "rcnn":
        return {"kind": kind, "batch": size(1, 8), "out": 1000, "lo": 333, "hi": 500, "quality": quality, "scale": 1.6}
    return {"kind": kind, "batch": size(1, 32), "out": size(96, 320), "lo": 256, "hi": 500, "quality": quality, "angle": rng.choice([10, 20, 30])}


# ---------------------------------------------------------------------------------------------------------------------
# synthetic records
# ---------------------------------------------------------------------------------------------------------------------

# ITU-T T.81 annex K: quantiser steps (zig-zag order), code counts and symbols of the typical Huffman tables
ZIGZAG = [0, 1, 8, 16, 9, 2, 3, 10, 17, 24, 32, 25, 18, 11, 4, 5, 12, 19, 26, 33, 40, 48, 41, 34, 27, 20, 13, 6, 7, 14, 21, 28,
          35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, 30, 37, 44, 51, 58, 59, 52, 45, 38, 31, 39, 46, 53, 60, 61, 54, 47, 55, 62, 63]
Q_LUMA = [16, 11, 12, 14, 12, 10, 16, 14, 13, 14, 18, 17, 16, 19, 24, 40, 26, 24, 22, 22, 24, 49, 35, 37, 29, 40, 58, 51, 61, 60, 57, 51,
          56, 55, 64, 72, 92, 78, 64, 68, 87, 69, 55, 56, 80, 109, 81, 87, 95, 98, 103, 104, 103, 62, 77, 113, 121, 112, 100, 120, 92, 101, 103, 99]
Q_CHROMA = [17, 18, 18, 24, 21, 24, 47, 26, 26, 47, 99, 66, 56, 66] + [99] * 50
DC_LUMA = (bytes([0, 1, 5, 1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0]), bytes(range(12)))
DC_CHROMA = (bytes([0, 3, 1, 1, 1, 1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0]), bytes(range(12)))
AC_LUMA = (bytes([0, 2, 1, 3, 3, 2, 4, 3, 5, 5, 4, 4, 0, 0, 1, 0x7d]), bytes.fromhex(
    "01020300041105122131410613516107227114328191a1082342b1c11552d1f02433627282090a161718191a25262728292a3435363738393a434445464748"
    "494a535455565758595a636465666768696a737475767778797a838485868788898a92939495969798999aa2a3a4a5a6a7a8a9aab2b3b4b5b6b7b8b9bac2c3"
    "c4c5c6c7c8c9cad2d3d4d5d6d7d8d9dae1e2e3e4e5e6e7e8e9eaf1f2f3f4f5f6f7f8f9fa"))
AC_CHROMA = (bytes([0, 2, 1, 2, 4, 4, 3, 4, 7, 5, 4, 4, 0, 1, 2, 0x77]), bytes.fromhex(
    "0001020311040521310612415107617113223281081442 91a1b1c109233352f0156272d10a162434e125f11718191a262728292a35363738393a434445464748"
    "494a535455565758595a636465666768696a737475767778797a82838485868788898a92939495969798999aa2a3a4a5a6a7a8a9aab2b3b4b5b6b7b8b9bac2"
    "c3c4c5c6c7c8c9cad2d3d4d5d6d7d8d9dae2e3e4e5e6e7e8e9eaf2f3f4f5f6f7f8f9fa".replace(" ", "")))


def code_table(dht, dev):
    """(code, length) by symbol of a Huffman table in DHT form."""
    code, k, out = 0, 0, np.zeros((2, 256), np.int64)
    for ln, count in enumerate(dht[0], 1):
        for _ in range(count):
            out[0, dht[1][k]], out[1, dht[1][k]] = code, ln
            code, k = code + 1, k + 1
        code <<= 1
    return torch.from_numpy(out).to(dev)


def pictures(gen, n, h, w, dev):
    """n pictures of h x w pixels, float R,G,B in 0..255: octaves of smooth noise (amplitude falls by a third as the frequency
    doubles), a few flat shapes, a flat sky in some, sensor noise of about three levels."""
    rnd = lambda *s: torch.rand(*s, generator=gen, device=dev)  # noqa: E731
    img = 60 + 140 * rnd(n, 3, 1, 1).expand(n, 3, h, w)
    cells, amp = 3, 48.0
    while cells < max(h, w):
        grid = torch.randn(n, 1, cells, cells, generator=gen, device=dev) + 0.3 * torch.randn(n, 3, cells, cells, generator=gen, device=dev)
        img = img + amp * torch.nn.functional.interpolate(grid, size=(h, w), mode="bilinear", align_corners=False)
        cells, amp = cells * 2, amp * 0.68
    yy, xx = torch.arange(h, device=dev).view(1, h, 1), torch.arange(w, device=dev).view(1, 1, w)
    for _ in range(4):
        cx, cy, r = rnd(n, 1, 1) * w, rnd(n, 1, 1) * h, (0.05 + 0.15 * rnd(n, 1, 1)) * min(h, w)
        inside = (torch.maximum((xx - cx).abs(), (yy - cy).abs()) < r).unsqueeze(1)
        img = torch.where(inside, 255 * rnd(n, 3, 1, 1), img)
    sky = (yy < (0.25 * h * (rnd(n, 1, 1) < 0.3))).unsqueeze(1)
    img = torch.where(sky, 150 + 90 * rnd(n, 3, 1, 1), img)
    return (img + 3.0 * torch.randn(n, 3, h, w, generator=gen, device=dev)).clamp(0, 255)


def jpeg_files(gen, sizes, quality, sampling, restart, dev):
    """Baseline JPEG files of synthetic pictures, sizes = [(width, height)]; `restart`: a marker after every MCU row."""
    comps = {"420": [(2, 2), (1, 1), (1, 1)], "422": [(2, 1), (1, 1), (1, 1)], "444": [(1, 1)] * 3, "grey": [(1, 1)]}[sampling]
    hs, vs = comps[0]
    scale = 5000 // quality if quality < 50 else 200 - 2 * quality
    quant = [np.clip((np.array(q) * scale + 50) // 100, 1, 255) for q in (Q_LUMA, Q_CHROMA)]
    head = b"\xff\xd8" + b"".join(b"\xff\xdb\x00\x43" + bytes([t]) + bytes(quant[t].astype(np.uint8)) for t in (0, 1))
    dht = b"".join(b"\xff\xc4" + struct.pack(">HB", 19 + len(t[1]), slot) + t[0] + t[1]
                   for slot, t in ((0, DC_LUMA), (0x10, AC_LUMA), (1, DC_CHROMA), (0x11, AC_CHROMA)))
    sos = b"\xff\xda" + struct.pack(">HB", 6 + 2 * len(comps), len(comps)) + b"".join(bytes([c + 1, 0x11 if c else 0]) for c in range(len(comps))) + b"\x00\x3f\x00"
    files, step = [], max(1, (1 << 23) // max(w * h for w, h in sizes))
    for first in range(0, len(sizes), step):
        part = sizes[first:first + step]
        grid = [(-(-w // (8 * hs)), -(-h // (8 * vs))) for w, h in part]
        streams, begin = encode(gen, grid, comps, quant, restart, dev)
        for (w, h), (mx, _), own in zip(part, grid, begin):
            sof = b"\xff\xc0" + struct.pack(">HBHHB", 8 + 3 * len(comps), 8, h, w, len(comps)) + b"".join(
                bytes([c + 1, s[0] * 16 + s[1], 1 if c else 0]) for c, s in enumerate(comps))
            dri = b"\xff\xdd" + struct.pack(">HH", 4, mx) if restart else b""
            body = b"".join((b"" if i == 0 else bytes([0xff, 0xd0 + (i - 1) % 8])) + streams[a:b] for i, (a, b) in enumerate(own))
            files.append(head + sof + dht + dri + sos + body + b"\xff\xd9")
    return files


def encode(gen, grid, comps, quant, restart, dev):
    """Entropy-coded segments of one picture per (mcux, mcuy) of `grid`: (bytes, [[(begin, end) of each segment]])."""
    n, W, H = len(grid), max(g[0] for g in grid), max(g[1] for g in grid)
    hs, vs = comps[0]
    rgb = pictures(gen, n, 8 * vs * H, 8 * hs * W, dev)
    mat = torch.tensor([[0.299, 0.587, 0.114], [-0.168736, -0.331264, 0.5], [0.5, -0.418688, -0.081312]], device=dev)
    ycc = torch.einsum("ij,njhw->nihw", mat, rgb)
    k = torch.arange(8, dtype=torch.float64)
    dct = (torch.cos((2 * k[None, :] + 1) * k[:, None] * math.pi / 16) * torch.where(k == 0, math.sqrt(1 / 8), 0.5)[:, None]).float().to(dev)
    zz = torch.tensor(ZIGZAG, device=dev)
    grids = torch.tensor(grid, device=dev)
    keep = (torch.arange(W, device=dev).view(1, 1, W) < grids[:, 0].view(n, 1, 1)) & (torch.arange(H, device=dev).view(1, H, 1) < grids[:, 1].view(n, 1, 1))
    where = keep.nonzero()  # MCUs in file order: picture, row, column
    blocks = []
    for c, (bw, bh) in enumerate(comps):
        plane = ycc[:, c] - (128 if c == 0 else 0)
        if c and (hs, vs) != (1, 1):
            plane = torch.nn.functional.avg_pool2d(plane.unsqueeze(1), (vs, hs)).squeeze(1)
        b = plane.view(n, H, bh, 8, W, bw, 8).permute(0, 1, 4, 2, 5, 3, 6)  # n, mcu row, mcu column, bh, bw, 8, 8
        b = dct @ b[keep] @ dct.T
        b = b.reshape(len(where), bw * bh, 64)[..., zz] / torch.from_numpy(quant[min(c, 1)]).float().to(dev)
        blocks.append(b.round().long())
    coef = torch.cat(blocks, 1)  # MCU, block, zig-zag position
    bpm = coef.shape[1]
    comp = torch.tensor([c for c, (bw, bh) in enumerate(comps) for _ in range(bw * bh)], device=dev)
    new = torch.ones(len(where), dtype=torch.bool, device=dev)  # MCUs that start a segment: the DC predictors are zero there
    new[1:] = (where[1:, 0] != where[:-1, 0]) | ((where[1:, 1] != where[:-1, 1]) if restart else False)
    for c in range(len(comps)):
        idx = (comp == c).nonzero().flatten()
        dc = coef[:, idx, 0]
        flat = dc.flatten()
        prev = torch.cat([flat.new_zeros(1), flat[:-1]]).view_as(dc)
        prev[:, 0] = torch.where(new, torch.zeros_like(prev[:, 0]), prev[:, 0])
        coef[:, idx, 0] = dc - prev
    segment = (torch.cumsum(new, 0) - 1).repeat_interleave(bpm)
    table = (comp > 0).long().repeat(len(where))
    coef = coef.view(-1, 64)
    N = len(coef)
    size = torch.frexp(coef.float()).exponent.long()  # bit length of the magnitude, 0 for 0
    value = torch.where(coef < 0, coef + (1 << size) - 1, coef)
    pos = torch.arange(64, device=dev).expand(N, 64)
    last = torch.cummax(torch.where((coef != 0) | (pos == 0), pos, torch.zeros_like(pos)), 1).values  # last coded position so far
    run = pos[:, 1:] - last[:, :-1] - 1
    ac = torch.stack([code_table(AC_LUMA, dev), code_table(AC_CHROMA, dev)])
    dct_ = torch.stack([code_table(DC_LUMA, dev), code_table(DC_CHROMA, dev)])
    bits, length = torch.zeros(N, 65, dtype=torch.long, device=dev), torch.zeros(N, 65, dtype=torch.long, device=dev)
    bits[:, 0] = dct_[table, 0, size[:, 0]] << size[:, 0] | value[:, 0]
    length[:, 0] = dct_[table, 1, size[:, 0]] + size[:, 0]
    t, symbol = table.view(N, 1).expand(N, 63), (run & 15) << 4 | size[:, 1:]
    code, ln = ac[t, 0, symbol], ac[t, 1, symbol]
    for _ in range(3):  # runs of sixteen zeros in front of a coefficient
        more = run >= 16 * (_ + 1)
        zrl, zln = ac[t, 0, torch.full_like(t, 0xf0)], ac[t, 1, torch.full_like(t, 0xf0)]
        code, ln = torch.where(more, zrl << ln | code, code), torch.where(more, ln + zln, ln)
    live = coef[:, 1:] != 0
    bits[:, 1:64] = torch.where(live, code << size[:, 1:] | value[:, 1:], 0)
    length[:, 1:64] = torch.where(live, ln + size[:, 1:], 0)
    open_end = last[:, 63] < 63  # end-of-block code
    bits[:, 64], length[:, 64] = torch.where(open_end, ac[table, 0, 0], 0), torch.where(open_end, ac[table, 1, 0], 0)
    used = length > 0
    seg, bits, length = segment.view(N, 1).expand(N, 65)[used], bits[used], length[used]
    S = int(segment[-1]) + 1
    total = torch.zeros(S, dtype=torch.long, device=dev).index_add_(0, seg, length)
    nbytes = (total + 7) // 8
    base = torch.cumsum(nbytes, 0) - nbytes
    begin = torch.cumsum(length, 0) - length
    shift = base * 8 - (torch.cumsum(total, 0) - total)
    at = begin + shift[seg]
    pad = nbytes * 8 - total  # the last byte of a segment is filled with ones
    at, bits, length = torch.cat([at, base * 8 + total]), torch.cat([bits, (1 << pad) - 1]), torch.cat([length, pad])
    words = torch.zeros(int(nbytes.sum()) // 4 + 4, dtype=torch.long, device=dev)
    for w in range(3):
        s = (at & 31) + length - 32 * (w + 1)
        piece = torch.where(s >= 0, bits >> s.clamp(min=0, max=63), torch.where(s > -32, bits << (-s).clamp(min=0, max=31), 0)) & 0xffffffff
        words.index_add_(0, (at >> 5) + w, piece)
    raw = torch.stack([words >> 24, words >> 16 & 255, words >> 8 & 255, words & 255], 1).flatten()[:int(nbytes.sum())]
    ff = (raw == 255).long()  # a zero byte follows every 0xff
    moved = torch.cumsum(ff, 0) - ff
    out = torch.zeros(len(raw) + int(ff.sum()), dtype=torch.uint8, device=dev)
    out[torch.arange(len(raw), device=dev) + moved] = raw.to(torch.uint8)
    edge = torch.cat([base, nbytes.sum().view(1)])
    edge = (edge + torch.cat([moved, ff.sum().view(1)])[edge]).cpu().tolist()
    counts = [g[1] if restart else 1 for g in grid]
    begin, i = [], 0
    for k in counts:
        begin.append([(edge[j], edge[j + 1]) for j in range(i, i + k)])
        i += k
    return out.cpu().numpy().tobytes(), begin


def avi_file(frames, width, height):
    """MJPEG frames as a plain AVI file with an index, as OpenCV's and ffmpeg's writers lay it out."""
    chunk = lambda tag, body: tag + struct.pack("<I", len(body)) + body + b"\0" * (len(body) & 1)  # noqa: E731
    avih = struct.pack("<14I", 40000, 0, 0, 0x10, len(frames), 0, 1, 0, width, height, 0, 0, 0, 0)
    strh = b"vidsMJPG" + struct.pack("<12I", 0, 0, 0, 1, 25, 0, len(frames), 0, 0xffffffff, 0, 0, width | height << 16)
    strf = struct.pack("<3I2H6I", 40, width, height, 1, 24, 0x47504a4d, width * height * 3, 0, 0, 0, 0)
    hdrl = chunk(b"LIST", b"hdrl" + chunk(b"avih", avih) + chunk(b"LIST", b"strl" + chunk(b"strh", strh) + chunk(b"strf", strf)))
    movi, index = b"movi", b""
    for f in frames:
        index += b"00dc" + struct.pack("<3I", 0x10, len(movi), len(f))
        movi += chunk(b"00dc", f)
    body = b"AVI " + hdrl + chunk(b"LIST", movi) + chunk(b"idx1", index)
    return b"RIFF" + struct.pack("<I", len(body)) + body


def png_file(mask):
    """An 8-bit grey PNG."""
    h, w = mask.shape
    chunk = lambda tag, body: struct.pack(">I", len(body)) + tag + body + struct.pack(">I", zlib.crc32(tag + body))  # noqa: E731
    rows = np.concatenate([np.zeros((h, 1), np.uint8), mask], 1).tobytes()
    return (b"\x89PNG\r\n\x1a\n" + chunk(b"IHDR", struct.pack(">IIBBBBB", w, h, 8, 0, 0, 0, 0)) + chunk(b"IDAT", zlib.compress(rows, 6)) +
            chunk(b"IEND", b""))


def annotation(rng, w, h):
    """Objects of a picture in the JSON form the localisation providers read."""
    objs = []
    for _ in range(int(rng.integers(1, 9))):
        x0, y0 = int(rng.integers(0, w - 40)), int(rng.integers(0, h - 40))
        objs.append({"name": CLASSES[int(rng.integers(20))], "difficult": bool(rng.integers(2)),
                     "bndbox": {"xmin": x0, "ymin": y0, "xmax": int(rng.integers(x0 + 24, w)), "ymax": int(rng.integers(y0 + 24, h))}})
    return json.dumps({"object": objs, "size": {"width": w, "height": h, "depth": 3}}).encode()


def audio_clips(gen, rng, n, seconds, dev):
    """Voiced-like clips: a few harmonics with a slow envelope over a noise floor, 16 kHz, between 1/16 and all of `seconds`."""
    clips = []
    for _ in range(n):
        m = int(16000 * seconds * rng.uniform(1 / 16, 1.0))
        t = torch.arange(m, device=dev, dtype=torch.float32) / 16000
        f0, env = rng.uniform(90, 300), 0.5 + 0.5 * torch.sin(2 * math.pi * rng.uniform(1, 5) * t + rng.uniform(0, 6.28))
        x = sum(rng.uniform(0.3, 1.0) / k * torch.sin(2 * math.pi * f0 * k * t + rng.uniform(0, 6.28)) for k in range(1, 9))
        x = 0.12 * env * x + 0.01 * torch.randn(m, generator=gen, device=dev)
        clips.append((x * 32767).clamp(-32768, 32767).to(torch.int16).cpu().numpy().tobytes())
    return clips


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------

_CTX = []


def context():
    """The program's one context."""
    if not _CTX:
        _CTX.append(K.Context(0))
    return _CTX[0]


def config(case, seed):
    kind, out = case["kind"], case.get("out")
    label = {"type": "label", "binary": True}
    if kind == "classify":
        img = {"type": "image", "height": out, "width": out, "channels": 3, "output_type": case["dtype"], "channel_major": case["aug"] != "area",
               "bgr_to_rgb": case["dtype"] == "float"}
        aug = {"crop": AUG_CROP, "photo": AUG_PHOTO,
               "eval": {"type": "image", "crop_enable": True, "center": True, "scale": [0.875, 0.875], "mean": MEAN, "stddev": STD},
               "area": {"type": "image", "crop_enable": True, "center": False, "scale": [0.5, 1.0], "flip_enable": True,
                        "interpolation_method": "AREA"}}[case["aug"]]
        etl = [img, label]
    elif kind == "ssd":
        etl = [{"type": "localization_ssd", "height": out, "width": out, "max_gt_boxes": 64, "class_names": CLASSES},
               {"type": "image", "height": out, "width": out, "output_type": "float"}]
        aug = {"type": "image", "crop_enable": False, "flip_enable": True, "expand_ratio": [1.0, 4.0], "expand_probability": 0.5,
               "emit_constraint_type": "center", "batch_samplers": SSD_SAMPLERS}
    elif kind == "video":
        etl = [{"type": "video", "max_frame_count": case["frames"], "frame": {"height": out, "width": out, "channels": 3}}, label]
        aug = {"type": "image", "frame": {"type": "image", "scale": [0.875, 0.875], "center": False, "flip_enable": True}}
    elif kind == "audio":
        etl = [{"type": "audio", "frame_length": case["frame"], "frame_stride": 160, "max_samples": int(16000 * case["seconds"]),
                "num_filters": case["filters"], "sample_rate": 16000, "window_type": "hann",
                "feature_type": "mfcc" if case["cepstra"] else "mfsc", "num_cepstra": case["cepstra"] or 1}, label]
        aug = None
    elif kind == "rcnn":
        etl = [{"type": "image", "height": out, "width": out},
               {"type": "localization_rcnn", "height": out, "width": out, "max_gt_boxes": 64, "class_names": CLASSES, "debug_deterministic": True}]
        aug = {"type": "image", "fixed_aspect_ratio": True, "fixed_scaling_factor": case["scale"], "crop_enable": False, "flip_enable": True}
    else:
        etl = [{"type": "image", "height": out, "width": out, "output_type": "float"},
               {"type": "pixelmask", "height": out, "width": out, "channels": 1, "output_type": "uint8_t"}]
        aug = {"type": "image", "crop_enable": True, "center": False, "scale": [0.5, 1.0], "flip_enable": True, "angle": [-case["angle"], case["angle"]]}
    return {"batch_size": case["batch"], "random_seed": 1 + seed % 1000003, "etl": etl, "augmentation": [aug] if aug else []}


def sizes_of(case, rng, n):
    return [(int(rng.integers(case["lo"], case["hi"] + 1)), int(rng.integers(case["lo"], case["hi"] + 1))) for _ in range(n)]


def records(case, gen, rng, n, dev):
    """n encoded records: a tuple of bytes each, one element per etl entry."""
    kind, label = case["kind"], lambda: struct.pack("<i", int(rng.integers(0, 1000)))
    if kind == "classify":
        files = jpeg_files(gen, sizes_of(case, rng, n), case["quality"], case["sampling"], case["restart"], dev)
        return [(f, label()) for f in files]
    if kind == "video":
        w, h, t = case["width"], case["height"], case["frames"]
        files = jpeg_files(gen, [(w, h)] * (n * t), case["quality"], "420", False, dev)
        return [(avi_file(files[i * t:(i + 1) * t], w, h), label()) for i in range(n)]
    if kind == "audio":
        return [(c, label()) for c in audio_clips(gen, rng, n, case["seconds"], dev)]
    if kind == "rcnn":
        sizes = [(int(rng.integers(case["lo"], case["hi"] + 1)), case["lo"]) for _ in range(n)]
    else:
        sizes = sizes_of(case, rng, n)
    files = jpeg_files(gen, sizes, case["quality"], "420", False, dev)
    if kind == "segment":
        out = []
        for f, (w, h) in zip(files, sizes):
            field = torch.nn.functional.interpolate(torch.rand(1, 1, 6, 6, generator=gen, device=dev), size=(h, w), mode="bicubic")[0, 0]
            out.append((f, png_file((field * 21).clamp(0, 20).to(torch.uint8).cpu().numpy())))
        return out
    boxes = [annotation(rng, w, h) for w, h in sizes]
    return list(zip(boxes, files)) if kind == "ssd" else list(zip(files, boxes))


def output_buffers(prov, case, dev):
    """A set of output buffers a program keeps: device tensors, or pinned host arrays."""
    out = {}
    for name, dims, dt, _ in prov.outputs:
        shape, dtype = (prov.batch_size,) + dims, K._TORCH_DTYPE[dt]
        if case.get("deliver") == "host":
            out[name] = torch.zeros(shape, dtype=dtype).pin_memory().numpy()
        else:
            out[name] = torch.zeros(shape, dtype=dtype, device=dev)
    return out


def prepare(case, seed):
    ctx = context()
    dev = torch.device("cuda", ctx.device)
    gen = torch.Generator(device=dev).manual_seed(seed)
    rng = np.random.default_rng(seed)
    if case["kind"] == "kernels":
        return prepare_kernels(case, seed, ctx, gen, rng, dev)
    depth = case.get("depth", 1)
    n = case["batch"] * depth
    recs = records(case, gen, rng, min(n, 512), dev)
    recs = [recs[i] for i in rng.permutation(n) % len(recs)]
    batches = [recs[i * case["batch"]:(i + 1) * case["batch"]] for i in range(depth)]
    prov = Provider(ctx, config(case, seed))
    outs = [output_buffers(prov, case, dev) for _ in range(depth)]
    # a program has been running: the provider's threads and buffers are up (other records than the pass sees, three calls, as
    # many as it has buffer sets)
    warm = records(case, gen, rng, min(case["batch"], 8), dev)
    warm = [warm[i % len(warm)] for i in range(case["batch"])]
    state = {"prov": prov, "batches": batches, "outs": outs, "host": case.get("deliver") == "host"}
    for _ in range(3):
        run(dict(state, batches=[warm], outs=outs[:1]))
    return state


def run(state):
    if "kernels" in state:
        ctx, ed, jd, idesc, n, layout, out = state["kernels"]
        L.check(ctx.lib.aeonb_jpeg_entropy_batch(ctx.handle, ed, n))
        L.check(ctx.lib.aeonb_jpeg_backend_batch(ctx.handle, jd, n))
        L.check(ctx.lib.aeonb_image_batch(ctx.handle, idesc, n, C.byref(layout)))
        return {"image": out, "status": state["status"]}
    prov = state["prov"]
    if len(state["batches"]) == 1:
        call = prov.run_host if state["host"] else prov.run_device
        return call(state["batches"][0], state["outs"][0])
    submit = prov.submit_host if state["host"] else prov.submit_device
    for ticket in [submit(b, o) for b, o in zip(state["batches"], state["outs"])]:
        prov.wait(ticket)
    return state["outs"]


def prepare_kernels(case, seed, ctx, gen, rng, dev):
    """Descriptors of the three batch kernels with everything they read resident in device memory; only the MCUs a record's crop
    box can touch are decoded, as the provider does it."""
    lib, n, size = ctx.lib, case["batch"], case["out"]
    files = jpeg_files(gen, sizes_of(case, rng, n), case["quality"], case["sampling"], case["restart"], dev)
    f32 = case["dtype"] == "float"
    photo = case["aug"] == "photo"
    aug = {"crop": AUG_CROP, "photo": AUG_PHOTO, "eval": {"type": "image", "center": True, "scale": [0.875, 0.875]}}[case["aug"]]
    infos = [K.jpeg_parse(f) for f in files]
    ws, hs = (C.c_int32 * n)(*[i.width for i in infos]), (C.c_int32 * n)(*[i.height for i in infos])
    drawn = (C.c_double * (24 * n))()
    L.check(lib.aeonb_draw_params(json.dumps(aug).encode(), 1 + seed % 1000003, n, n, ws, hs, size, size, drawn))
    p = np.array(drawn).reshape(n, 24)
    ed, jd, idesc = (L.EntropyDesc * n)(), (L.JpegDesc * n)(), (L.ImageDesc * n)()
    dtype = torch.float32 if f32 else torch.uint8
    out = torch.zeros((n, 3, size, size), dtype=dtype, device=dev)
    status = torch.full((n,), -1, dtype=torch.int32, device=dev)
    keep = []

    def room(nbytes):
        keep.append(torch.zeros(max(int(nbytes), 16), dtype=torch.uint8, device=dev))
        return keep[-1].data_ptr()

    def resident(a):
        keep.append(torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).to(dev))
        return keep[-1].data_ptr()

    for i, data in enumerate(files):
        info, quant, tables, off = L.JpegInfo(), np.zeros(192, np.uint16), np.zeros(1088, np.uint8), C.c_size_t()
        buf = (C.c_char * len(data)).from_buffer_copy(data)
        x, d, e = ed[i], jd[i], idesc[i]
        L.check(lib.aeonb_jpeg_entropy_prepare(buf, len(data), C.byref(info), quant.ctypes.data_as(C.POINTER(C.c_uint16)),
                                               tables.ctypes.data_as(C.POINTER(C.c_uint8)), C.byref(x), C.byref(off)))
        cx, cy, cw, ch = (int(v) for v in p[i, 0:4])
        roi = (C.c_int32 * 4)()
        L.check(lib.aeonb_jpeg_roi_for_crop(C.byref(info), cx, cy, cw, ch, roi))
        x.scan = resident(np.frombuffer(data, np.uint8)[off.value:off.value + x.scan_size])
        x.tables, x.status = resident(tables), status.data_ptr() + 4 * i
        x.scratch_bytes = int(lib.aeonb_jpeg_entropy_scratch_bytes(C.byref(x)))
        x.scratch = room(x.scratch_bytes)
        q = resident(quant)
        for k in range(4):
            x.roi[k] = roi[k]
        rx, ry = roi[0] * 8 * info.hs[0], roi[1] * 8 * info.vs[0]
        d.width, d.height = min(info.width, roi[2] * 8 * info.hs[0]) - rx, min(info.height, roi[3] * 8 * info.vs[0]) - ry
        d.ncomp = info.ncomp
        for c in range(info.ncomp):
            d.hs[c], d.vs[c] = info.hs[c], info.vs[c]
            d.blocks_w[c], d.blocks_h[c] = (roi[2] - roi[0]) * info.hs[c], (roi[3] - roi[1]) * info.vs[c]
            x.coef[c] = d.coef[c] = room(d.blocks_w[c] * d.blocks_h[c] * 128)
            d.quant[c] = q + 128 * c
        d.dst_pitch, d.dst_pixel_stride = (d.width * 3 + 15) // 16 * 16, 3
        d.dst = e.src = room(d.dst_pitch * d.height)
        e.src_pitch, e.src_w, e.src_h, e.src_pixel_stride = d.dst_pitch, d.width, d.height, 3
        e.canvas_w, e.canvas_h, e.canvas_x, e.canvas_y = info.width, info.height, rx, ry
        e.crop_x, e.crop_y, e.crop_w, e.crop_h = cx, cy, cw, ch
        e.out_w, e.out_h, e.interp, e.flip = size, size, L.INTERP_LINEAR, int(p[i, 6])
        light = (C.c_float * 3)(*[float(v) for v in p[i, 12:15]])
        L.check(lib.aeonb_image_desc_set_photometric(C.byref(e), float(p[i, 9]), float(p[i, 10]), float(p[i, 11]), int(p[i, 8]),
                                                     light if photo else None, float(p[i, 15])))
        e.dst = out.data_ptr() + i * out.stride(0) * out.element_size()
    norm = f32 and case["aug"] != "crop"
    layout = K.make_layout(size, size, L.F32 if f32 else L.U8, True, f32, MEAN if norm else None, STD if norm else None)
    torch.cuda.synchronize(dev)
    return {"kernels": (ctx, ed, jd, idesc, n, layout, out), "status": status, "keep": keep}


# bytes of a coded pixel of the pictures above, by JPEG quality (measured; 4:2:0)
BYTES_PER_PIXEL = {75: 0.10, 85: 0.14, 90: 0.185, 92: 0.21, 95: 0.30}


def work(case):
    """Each encoded record read once, each output written once; the transforms of the audio path as operations."""
    kind, n, out = case["kind"], case["batch"], case.get("out", 0)
    if kind == "audio":
        frames = int((16000 * case["seconds"] - case["frame"]) // 160 + 1)
        live = 0.53 * frames  # clips are between 1/16 and all of the longest
        width = case["cepstra"] or case["filters"]
        flops = n * live * (2.5 * case["frame"] * math.log2(case["frame"]) + 6 * case["frame"] + 2 * case["cepstra"] * case["filters"])
        return {"bytes": n * (2 * 16000 * case["seconds"] * 0.53 + 4.0 * frames * width), "flops": flops}
    bpp = BYTES_PER_PIXEL[case["quality"]] * {"422": 1.13, "444": 1.4, "grey": 0.85}.get(case.get("sampling"), 1.0)
    if kind == "video":
        return {"bytes": n * case["frames"] * (case["width"] * case["height"] * bpp + 3 * out * out), "flops": 0}
    pixels = (0.5 * (case["lo"] + case["hi"])) ** 2
    size = 1 if case.get("dtype") == "uint8_t" or kind == "rcnn" else 4
    produced = 3.0 * out * out * size
    if kind == "rcnn":
        produced += 48.0 * (out // 16) ** 2 * 9  # regression targets and their mask (4 floats each), two label planes and theirs
    if kind == "segment":
        produced += out * out
    return {"bytes": case.get("depth", 1) * n * (pixels * bpp + produced), "flops": 0}


def tolerance(case):
    """Bytes, counts and box buffers are exact.  Normalised floats are one multiply-add of a byte: a few units in the last place.
    Spectra are 32-bit transforms; a mel band with next to no energy carries the rounding of the whole frame into its logarithm
    (against a 64-bit transform: rel 8e-7, max 2.3e-4 over 64 clips)."""
    if case["kind"] == "audio":
        return {"rel": 4e-6, "max": 1e-3}
    return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}
