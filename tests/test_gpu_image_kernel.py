"""Parity of the image augmentation/packing kernel with the CPU oracle, through the C ABI.

Bar: bit-exact for uint8 outputs (geometry and photometric alike, since the oracle restates
OpenCV's integer / float32 arithmetic), 1e-6 absolute for standardised float outputs."""
import os

import numpy as np
import pytest
import torch

from oracle import image_ops as ops
from tests.synth import gradient_image

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_kernel(ctx, srcs, params, slot_w, slot_h, output_type="uint8_t", channel_major=True, bgr_to_rgb=False,
               mean=None, stddev=None, pixel_stride=3):
    from aeon_b200 import kernels as K
    dt = K.DTYPE_BY_NAME[output_type]
    dev = torch.device("cuda", ctx.device)
    with torch.cuda.stream(ctx.torch_stream):
        tsrc = []
        for s in srcs:
            if s is None:
                tsrc.append(None)
                continue
            if pixel_stride == 4:
                s = np.concatenate([s, np.full(s.shape[:2] + (1,), 77, np.uint8)], -1)
            tsrc.append(torch.from_numpy(np.ascontiguousarray(s)).to(dev))
        shape = (len(srcs), 3, slot_h, slot_w) if channel_major else (len(srcs), slot_h, slot_w, 3)
        out = torch.full(shape, 99, dtype=K._TORCH_DTYPE[dt], device=dev)
        lay = K.make_layout(slot_w, slot_h, dt, channel_major, bgr_to_rgb, mean, stddev)
        K.image_batch(ctx, tsrc, params, out, lay)
        ctx.synchronize()
        return out.cpu().numpy()


def oracle(src, p, slot_w, slot_h, **kw):
    img = ops.transform_single_image(src, p)
    canvas = np.zeros((slot_h, slot_w, 3), np.uint8)
    canvas[:img.shape[0], :img.shape[1]] = img
    full = ops.load_image(canvas, **kw)
    if kw.get("mean") is not None and (img.shape[0] != slot_h or img.shape[1] != slot_w):
        # the reference standardises only the image region of a fixed-aspect canvas
        z = ops.load_image(np.zeros_like(canvas), kw.get("channel_major", True), kw.get("bgr_to_rgb", False),
                           kw.get("output_type", "uint8_t"))
        roi = ops.load_image(img, **kw)
        if kw.get("channel_major", True):
            z[:, :img.shape[0], :img.shape[1]] = roi
        else:
            z[:img.shape[0], :img.shape[1]] = roi
        full = z
    return full


def random_params(rng, w, h, ow, oh, photometric):
    cw = int(rng.integers(2, w + 1))
    ch = int(rng.integers(2, h + 1))
    kw = dict(cropbox=(int(rng.integers(0, w - cw + 1)), int(rng.integers(0, h - ch + 1)), cw, ch),
              output_size=(ow, oh), flip=bool(rng.integers(2)))
    if photometric:
        kw.update(contrast=float(np.float32(rng.uniform(0.6, 1.4))), brightness=float(np.float32(rng.uniform(0.6, 1.4))),
                  saturation=float(np.float32(rng.uniform(0.6, 1.4))), hue=int(rng.integers(-18, 19)),
                  lighting=[float(v) for v in rng.normal(0, 0.1, 3).astype(np.float32)], color_noise_std=0.1)
    return ops.ImageParams(**kw)


@pytest.mark.parametrize("pixel_stride", [3, 4])
def test_geometry_uint8_chw_bit_exact(ctx, pixel_stride):
    rng = np.random.default_rng(11)
    srcs, params = [], []
    for _ in range(24):
        h, w = (int(v) for v in rng.integers(256, 513, 2))
        srcs.append(gradient_image(rng, h, w))
        params.append(random_params(rng, w, h, 224, 224, False))
    got = run_kernel(ctx, srcs, params, 224, 224, pixel_stride=pixel_stride)
    for i in range(len(srcs)):
        want = oracle(srcs[i], params[i], 224, 224)
        assert np.array_equal(got[i], want), "record %d differs" % i


def test_full_photometric_float_normalised(ctx):
    rng = np.random.default_rng(12)
    mean = [123.7 / 255, 116.3 / 255, 103.5 / 255]
    std = [58.4 / 255, 57.1 / 255, 57.4 / 255]
    srcs, params = [], []
    for _ in range(24):
        h, w = (int(v) for v in rng.integers(256, 513, 2))
        srcs.append(gradient_image(rng, h, w))
        params.append(random_params(rng, w, h, 224, 224, True))
    got = run_kernel(ctx, srcs, params, 224, 224, "float", True, True, mean, std)
    got_u8 = run_kernel(ctx, srcs, params, 224, 224, "uint8_t", False, False)
    for i in range(len(srcs)):
        want_u8 = ops.transform_single_image(srcs[i], params[i])
        assert np.array_equal(got_u8[i], want_u8), "uint8 photometric output of record %d differs" % i
        want = oracle(srcs[i], params[i], 224, 224, channel_major=True, bgr_to_rgb=True, output_type="float",
                      mean=mean, stddev=std)
        assert np.abs(got[i] - want).max() <= 1e-6


def test_each_photometric_stage_alone(ctx):
    rng = np.random.default_rng(13)
    src = rng.integers(0, 256, (97, 131, 3), dtype=np.uint8)  # full-range noise exercises saturation
    base = dict(cropbox=(0, 0, 131, 97), output_size=(131, 97))
    cases = [dict(brightness=1.4), dict(saturation=0.6), dict(brightness=0.7, saturation=1.3),
             dict(hue=-18), dict(hue=17), dict(hue=-1), dict(contrast=0.6), dict(contrast=1.4),
             dict(lighting=[0.2, -0.1, 0.05], color_noise_std=0.1), dict(flip=True, hue=5)]
    params = [ops.ImageParams(**base, **c) for c in cases]
    got = run_kernel(ctx, [src] * len(cases), params, 131, 97, "uint8_t", False)
    for i, p in enumerate(params):
        assert np.array_equal(got[i], ops.transform_single_image(src, p)), cases[i]


def test_hsv_round_trip_all_inputs(ctx):
    """Every 8-bit BGR triple through hue shifts, 4096 x 4096 pixels in 16 bands."""
    v = np.arange(256, dtype=np.uint8)
    b, g, r = np.meshgrid(v, v, v, indexing="ij")
    img = np.stack([b, g, r], -1).reshape(4096, 4096, 3)
    for hue in (-7, 11):
        for band in (0, 5, 15):
            src = np.ascontiguousarray(img[band * 256:(band + 1) * 256, :1000])
            p = ops.ImageParams(cropbox=(0, 0, 1000, 256), output_size=(1000, 256), hue=hue)
            got = run_kernel(ctx, [src], [p], 1000, 256, "uint8_t", False)[0]
            assert np.array_equal(got, ops.transform_single_image(src, p))


@pytest.mark.parametrize("shape", [(1, 1), (2, 3), (7, 5), (16, 16), (17, 17), (33, 9)])
def test_tiny_and_odd_sizes(ctx, shape):
    rng = np.random.default_rng(14)
    h, w = shape
    src = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    params = [ops.ImageParams(cropbox=(0, 0, w, h), output_size=(ow, oh), flip=f, contrast=c)
              for (ow, oh, f, c) in [(w, h, False, 1.0), (13, 11, True, 1.0), (31, 17, False, 0.8), (5, 40, True, 1.3)]]
    for p in params:
        ow, oh = p.output_size
        got = run_kernel(ctx, [src], [p], ow, oh, "uint8_t", False)[0]
        assert np.array_equal(got, ops.transform_single_image(src, p))


def test_crop_at_borders_and_upscale(ctx):
    rng = np.random.default_rng(15)
    src = gradient_image(rng, 90, 120)
    boxes = [(0, 0, 40, 30), (80, 0, 40, 30), (0, 60, 40, 30), (80, 60, 40, 30), (0, 0, 120, 90), (119, 89, 1, 1)]
    params = [ops.ImageParams(cropbox=b, output_size=(224, 224), flip=bool(i & 1)) for i, b in enumerate(boxes)]
    got = run_kernel(ctx, [src] * len(boxes), params, 224, 224)
    for i, p in enumerate(params):
        assert np.array_equal(got[i], oracle(src, p, 224, 224)), boxes[i]


def test_expand_canvas_and_padding(ctx):
    rng = np.random.default_rng(16)
    src = gradient_image(rng, 75, 100)
    p1 = ops.ImageParams(expand_ratio=2.0, expand_offset=(37, 21), expand_size=(200, 150), cropbox=(10, 5, 160, 130),
                         output_size=(300, 300), flip=True)
    p2 = ops.ImageParams(cropbox=(0, 0, 100, 75), output_size=(100, 75), padding=4, padding_crop_offset=(1, 7))
    got1 = run_kernel(ctx, [src], [p1], 300, 300, "float", True)[0]
    assert np.array_equal(got1, oracle(src, p1, 300, 300, output_type="float"))
    got2 = run_kernel(ctx, [src], [p2], 100, 75, "uint8_t", False)[0]
    assert np.array_equal(got2, ops.transform_single_image(src, p2))


def test_fixed_aspect_slot_zero_fill_and_null_source(ctx):
    rng = np.random.default_rng(17)
    src = gradient_image(rng, 60, 90)
    p = ops.ImageParams(cropbox=(0, 0, 90, 60), output_size=(48, 32))
    got = run_kernel(ctx, [src, None], [p, p], 64, 64, "uint8_t", True)
    assert np.array_equal(got[0], oracle(src, p, 64, 64))
    assert not got[1].any()
    mean, std = [0.4, 0.5, 0.6], [0.2, 0.0, 0.3]
    gotf = run_kernel(ctx, [src], [p], 64, 64, "float", True, False, mean, std)[0]
    want = oracle(src, p, 64, 64, channel_major=True, output_type="float", mean=mean, stddev=std)
    assert np.abs(gotf - want).max() <= 1e-6
    assert not gotf[:, 32:, :].any() and not gotf[:, :, 48:].any()


@pytest.mark.parametrize("otype", ["int8_t", "int16_t", "uint16_t", "int32_t", "double"])
def test_output_types_and_hwc(ctx, otype):
    rng = np.random.default_rng(18)
    src = gradient_image(rng, 64, 64)
    p = ops.ImageParams(cropbox=(3, 5, 50, 40), output_size=(30, 20), flip=True)
    for cm in (True, False):
        got = run_kernel(ctx, [src], [p], 30, 20, otype, cm, True)[0]
        want = ops.load_image(ops.transform_single_image(src, p), cm, True, otype)
        assert np.array_equal(got, want.astype(got.dtype))


def test_nearest_interpolation(ctx):
    rng = np.random.default_rng(19)
    src = gradient_image(rng, 70, 55)
    p = ops.ImageParams(cropbox=(2, 3, 50, 60), output_size=(33, 47), interpolation_method="NEAREST")
    got = run_kernel(ctx, [src], [p], 33, 47, "uint8_t", False)[0]
    assert np.array_equal(got, ops.transform_single_image(src, p))


def test_reference_golden_train_vector(ctx, golden_dir):
    """aeon test/test_provider.cpp:96-179: crop (50,50,171x201) + flip + 224 LINEAR + RGB CHW float standardise."""
    import cv2
    import os
    enc = np.fromfile(os.path.join(golden_dir, "img_2112_70.jpg"), np.uint8)
    img = cv2.imdecode(enc, cv2.IMREAD_COLOR)
    p = ops.ImageParams(cropbox=(50, 50, 171, 201), output_size=(224, 224), flip=True)
    got = run_kernel(ctx, [img], [p], 224, 224, "float", True, True, [0.485, 0.456, 0.406], [0.229, 0.224, 0.225])[0]
    gold = np.fromfile(os.path.join(golden_dir, "augment_output_linear_train.bin"), np.float32).reshape(3, 224, 224)
    assert np.abs(got - gold).max() <= 1e-5


def test_invalid_descriptors_are_rejected(ctx):
    from aeon_b200._lib import AeonError
    rng = np.random.default_rng(20)
    src = gradient_image(rng, 32, 32)
    bad = ops.ImageParams(cropbox=(10, 10, 30, 30), output_size=(16, 16))
    with pytest.raises(AeonError, match="outside"):
        run_kernel(ctx, [src], [bad], 16, 16)
    big = ops.ImageParams(cropbox=(0, 0, 32, 32), output_size=(40, 16))
    with pytest.raises(AeonError, match="does not fit"):
        run_kernel(ctx, [src], [big], 16, 16)



SIZES_AT_ONCE = """
import sys, threading
import numpy as np, torch
from aeon_b200 import kernels as K
from oracle import image_ops as ops
from tests.test_gpu_specgram import run as specgram
barrier, failures = threading.Barrier(4), []
rng = np.random.default_rng(0)
src = torch.from_numpy(rng.integers(0, 256, (64, 64, 4), dtype=np.uint8)).cuda()
clip = rng.integers(-999, 999, 12000, dtype=np.int16)
box = np.array([[10, 10, 60, 60]], np.float32)

def work(size, frame, anchors):
    ctx = K.Context(0)
    def attempt(what, fn):
        torch.cuda.synchronize()
        barrier.wait(60)
        try:
            fn()
        except Exception as e:
            failures.append((what, str(e)))
    for dt in K._TORCH_DTYPE:
        for stride in (3, 4):
            out = torch.zeros((1, size, size, 3), dtype=K._TORCH_DTYPE[dt], device="cuda")
            lay = K.make_layout(size, size, dt, False)
            p = ops.ImageParams(cropbox=(0, 0, 64, 64), output_size=(size, size))
            attempt(("image", size, dt, stride), lambda: (K.image_batch(ctx, [src[:, :, :stride].contiguous()], [p], out, lay), ctx.synchronize()))
    for _ in range(20):
        attempt(("specgram", frame), lambda: specgram(ctx, [clip], frame_length=frame, frame_stride=frame, max_time_steps=2, num_filters=0))
        attempt(("rcnn", anchors), lambda: K.rcnn_label_batch(ctx, np.tile(box, (anchors, 1)), [box], [(100, 100)]))

threads = [threading.Thread(target=work, args=a) for a in ((32, 131, 100), (400, 6007, 60000), (240, 1009, 30000), (64, 257, 25600))]
[t.start() for t in threads]
[t.join() for t in threads]
print(len(failures), failures[:4])
sys.exit(1 if failures else 0)
"""


def test_launches_of_several_sizes_at_once(ctx):
    """Four threads with contexts of their own launch every variant of the image kernel for the first time in the process, and the
    direct-sum spectrogram and the anchor kernel, each with another amount of shared memory: no thread's launch may find the limit that
    another has set for a smaller one."""
    import subprocess
    import sys
    for _ in range(3):
        done = subprocess.run([sys.executable, "-c", SIZES_AT_ONCE], capture_output=True, text=True, timeout=180, cwd=ROOT)
        assert done.returncode == 0, done.stdout[-2000:] + done.stderr[-2000:]


@pytest.mark.parametrize("otype", ["uint8_t", "int8_t", "uint16_t", "float", "double"])
@pytest.mark.parametrize("layout", ["planes", "planes apart", "lines apart", "side by side", "side by side, lines apart", "strides"])
@pytest.mark.parametrize("records", [3, 260])
def test_outputs_that_do_not_start_on_16_bytes(ctx, records, otype, layout):
    """Every way a band is stored (260 records have enough blocks for the stores in runs, three only where bytes go out as they are), at widths
    around a piece of 16 bytes, slots larger than the picture, one row to many bands, first elements at every place of a piece: what lies in the
    slots equals an output of aligned lines, what lies between them is left alone."""
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(21)
    dt, dev = K.DTYPE_BY_NAME[otype], torch.device("cuda", ctx.device)
    for w, h, margin in [(1, 1, 0), (3, 7, 2), (15, 16, 0), (16, 9, 1), (17, 33, 0), (31, 5, 3), (225, 40, 0), (229, 301, 5), (500, 64, 0), (1000, 61, 0)]:
        if records > 3:
            h = min(h, 33)
        srcs = [torch.from_numpy(gradient_image(rng, 40 + 9 * k, 70 + 5 * k)).to(dev) for k in range(3)]
        srcs = [srcs[k % 3] for k in range(records)]
        params = [random_params(rng, s.shape[1], s.shape[0], max(w - margin, 1), max(h - margin, 1), False) for s in srcs]
        pitch = (w + 31) // 16 * 16
        with torch.cuda.stream(ctx.torch_stream):
            want = torch.full((records, 3, h, pitch), 99, dtype=K._TORCH_DTYPE[dt], device=dev)
            K.image_batch(ctx, srcs, params, want, K.make_layout(w, h, dt, strides=(h * pitch, pitch, 1)))
            sc, sy, sx = {"planes": (h * w, w, 1), "planes apart": (h * w + 5, w, 1), "lines apart": (h * (w + 3), w + 3, 1),
                          "side by side": (1, 3 * w, 3), "side by side, lines apart": (1, 3 * w + 7, 3), "strides": (2, 7 * w, 7)}[layout]
            if w % 16 == 0 and layout in ("planes", "lines apart"):
                sc, sy = h * (w + 1), w + 1
            slot = 2 * sc + (h - 1) * sy + (w - 1) * sx + 1
            for lead in range(0, 16, 1 if w == 17 and records == 3 else 5):
                room = torch.full((lead + records * (slot + 4) + 16,), 77, dtype=K._TORCH_DTYPE[dt], device=dev)
                got = torch.as_strided(room, (records, 3, h, w), (slot + 4, sc, sy, sx), lead)
                expect = room.clone()
                torch.as_strided(expect, (records, 3, h, w), (slot + 4, sc, sy, sx), lead).copy_(want[..., :w])
                K.image_batch(ctx, srcs, params, got, K.make_layout(w, h, dt, strides=(sc, sy, sx)), record_stride=slot + 4)
                ctx.synchronize()
                assert torch.equal(room, expect), (w, h, lead)


@pytest.mark.parametrize("n, w", [(47, 256), (48, 255), (48, 256), (60, 301)])
def test_doubles_side_by_side(ctx, n, w):
    """8-byte elements with the channels side by side go out in runs from 384 blocks (eight a picture here) and 256 columns on."""
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(22)
    h, dt, dev = 37, K.DTYPE_BY_NAME["double"], torch.device("cuda", ctx.device)
    srcs = [torch.from_numpy(gradient_image(rng, 50, 80)).to(dev) for _ in range(n)]
    params = [random_params(rng, 80, 50, w, h, False) for _ in srcs]
    with torch.cuda.stream(ctx.torch_stream):
        want = torch.full((n, 3, h, w), 99, dtype=K._TORCH_DTYPE[dt], device=dev)
        K.image_batch(ctx, srcs, params, want, K.make_layout(w, h, dt))
        for lead in (0, 1):
            room = torch.full((lead + n * h * w * 3 + 8,), 77, dtype=K._TORCH_DTYPE[dt], device=dev)
            got = room[lead:lead + n * h * w * 3].view(n, h, w, 3)
            K.image_batch(ctx, srcs, params, got, K.make_layout(w, h, dt, channel_major=False))
            ctx.synchronize()
            assert torch.equal(got, want.permute(0, 2, 3, 1)) and torch.all(room[:lead] == 77) and torch.all(room[lead + n * h * w * 3:] == 77)
