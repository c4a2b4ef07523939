"""Rotation pre-pass (image::rotate, src/image.cpp:53-75) through the C ABI against the oracle: bit-exact."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import image_ops as ops

pytestmark = pytest.mark.gpu


def rotate_gpu(ctx, images, angles, src_stride=3, dst_stride=3, nearest=False):
    from aeon_b200 import _lib as L
    dev = torch.device("cuda", ctx.device)
    n = len(images)
    descs = (L.RotateDesc * n)()
    keep, outs = [], []
    for i, (img, angle) in enumerate(zip(images, angles)):
        h, w = img.shape[:2]
        if src_stride == 4:
            img = np.concatenate([img, np.full((h, w, 1), 201, np.uint8)], -1)
        src = torch.from_numpy(np.ascontiguousarray(img)).to(dev)
        pitch = (w * dst_stride + 15) // 16 * 16
        dst = torch.full((h, pitch), 123, dtype=torch.uint8, device=dev)
        d = descs[i]
        d.src, d.src_pitch, d.src_pixel_stride = src.data_ptr(), w * src_stride, src_stride
        d.width, d.height, d.angle, d.nearest = w, h, int(angle), int(nearest)
        d.dst, d.dst_pitch, d.dst_pixel_stride = dst.data_ptr(), pitch, dst_stride
        keep += [src, dst]
        outs.append(torch.as_strided(dst, (h, w, dst_stride), (pitch, dst_stride, 1)))
    torch.cuda.synchronize(dev)
    L.check(ctx.lib.aeonb_rotate_batch(ctx.handle, descs, n))
    ctx.synchronize()
    return [o.cpu().numpy()[..., :3] for o in outs]


@pytest.mark.parametrize("strides", [(3, 3), (4, 3), (3, 4)])
def test_rotation_matches_oracle(ctx, strides):
    rng = np.random.default_rng(91)
    cases = [(40, 60, 7), (97, 131, -13), (64, 64, 20), (200, 150, 3), (33, 70, -20), (256, 384, 45), (50, 50, 90), (31, 17, 180),
             (120, 80, -1), (1, 1, 5), (2, 300, 11), (375, 500, 19), (512, 512, -20)]
    images = [rng.integers(0, 256, (h, w, 3), dtype=np.uint8) for h, w, _ in cases]
    got = rotate_gpu(ctx, images, [a for _, _, a in cases], *strides)
    for img, (h, w, angle), g in zip(images, cases, got):
        assert np.array_equal(g, ops.rotate(img, angle)), (h, w, angle)


def test_rotation_matches_opencv_binary(ctx):
    import cv2
    rng = np.random.default_rng(92)
    images = [rng.integers(0, 256, (int(rng.integers(20, 300)), int(rng.integers(20, 300)), 3), dtype=np.uint8) for _ in range(24)]
    angles = [int(a) for a in rng.integers(-45, 46, len(images))]
    got = rotate_gpu(ctx, images, angles)
    for img, angle, g in zip(images, angles, got):
        h, w = img.shape[:2]
        ref = cv2.warpAffine(img, cv2.getRotationMatrix2D((w // 2, h // 2), angle, 1.0), (w, h), flags=cv2.INTER_LINEAR,
                             borderMode=cv2.BORDER_CONSTANT, borderValue=(0, 0, 0, 0))
        assert np.array_equal(g, ref), (h, w, angle)


def test_rotation_without_interpolation_for_masks(ctx):
    """image::rotate(.., interpolate = false) as the pixelmask / depthmap transformers call it (src/etl_pixel_mask.cpp:71-73):
    against the oracle and against cv2.warpAffine(INTER_NEAREST) itself; grey pictures stored as B = G = R."""
    import cv2
    rng = np.random.default_rng(93)
    images, angles = [], []
    for _ in range(24):
        h, w = int(rng.integers(1, 300)), int(rng.integers(1, 300))
        grey = rng.integers(0, 256, (h, w, 1), dtype=np.uint8)
        images.append(np.repeat(grey, 3, axis=2) if rng.integers(2) else rng.integers(0, 256, (h, w, 3), dtype=np.uint8))
        angles.append(int(rng.integers(-180, 181)) or 13)
    got = rotate_gpu(ctx, images, angles, nearest=True)
    for img, angle, g in zip(images, angles, got):
        h, w = img.shape[:2]
        ref = cv2.warpAffine(img, cv2.getRotationMatrix2D((w // 2, h // 2), angle, 1.0), (w, h), flags=cv2.INTER_NEAREST,
                             borderMode=cv2.BORDER_CONSTANT, borderValue=(0, 0, 0, 0))
        assert np.array_equal(g, ops.rotate(img, angle, interpolate=False)), (h, w, angle)
        assert np.array_equal(g, ref.reshape(img.shape)), (h, w, angle)


def test_bad_arguments(ctx):
    from aeon_b200 import _lib as L
    d = (L.RotateDesc * 1)()
    assert ctx.lib.aeonb_rotate_batch(ctx.handle, d, 1) == L.ERR_INVALID
    assert ctx.lib.aeonb_rotate_batch(ctx.handle, d, 0) == 0


@pytest.mark.parametrize("nearest", [False, True])
@pytest.mark.parametrize("tiles", [False, True])
def test_rotation_at_the_edges_of_tiles_and_words(ctx, nearest, tiles):
    """Widths and heights around a tile (512 x 8) and four pixels, sources at every alignment: rows, and nothing beside them, are written as
    the oracle has them.  Launches of at least 2**22 pixels (masks: a quarter) of pictures at least 128 wide, with destinations of three bytes per pixel on
    words, go through tiles, others through a thread per pixel, with destinations at every alignment."""
    from aeon_b200 import _lib as L
    rng = np.random.default_rng(93)
    dev = torch.device("cuda", ctx.device)
    cases = [(h, w) for w in (1, 2, 3, 4, 5, 128, 129, 511, 512, 513, 1030) for h in (1, 8, 9)] + [(17, 515)]
    if tiles:
        cases = [c for c in cases if c[1] >= 128] + [(2051, 2047)]      # the last one brings the pixels
    pixels = sum(h * w for h, w in cases) * (4 if nearest else 1)
    assert (pixels >= 1 << 22) == tiles
    descs = (L.RotateDesc * len(cases))()
    keep = []
    for i, (h, w) in enumerate(cases):
        img = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
        angle, lead, pitch, at = int(rng.integers(-30, 31)), i % 4, 3 * w + i % 3, (i // 4) % 4
        if tiles:
            pitch, at = (3 * w + 3) // 4 * 4, 4 * (i % 2)
        src = torch.zeros(8 + h * 3 * w, dtype=torch.uint8, device=dev)
        src[lead:lead + img.size] = torch.from_numpy(img.reshape(-1)).to(dev)
        dst = torch.full((8 + h * pitch,), 123, dtype=torch.uint8, device=dev)
        d = descs[i]
        d.src, d.src_pitch, d.src_pixel_stride = src.data_ptr() + lead, 3 * w, 3
        d.width, d.height, d.angle, d.nearest = w, h, angle, int(nearest)
        d.dst, d.dst_pitch, d.dst_pixel_stride = dst.data_ptr() + at, pitch, 3
        want = np.full(8 + h * pitch, 123, np.uint8)
        turned = ops.rotate(img, angle, False) if nearest else ops.rotate(img, angle)
        for y in range(h):
            want[at + y * pitch:at + y * pitch + 3 * w] = turned[y].reshape(-1)
        keep.append((src, dst, want))
    torch.cuda.synchronize(dev)
    L.check(ctx.lib.aeonb_rotate_batch(ctx.handle, descs, len(cases)))
    ctx.synchronize()
    for (h, w), (_, dst, want) in zip(cases, keep):
        assert np.array_equal(dst.cpu().numpy(), want), (h, w)


def test_rotation_on_either_side_of_the_rule_for_tiles(ctx):
    """The same pictures in launches that go through tiles and in ones that one property each keeps from it: too few pixels, a narrow picture,
    a destination off a word, four bytes per pixel."""
    from aeon_b200 import _lib as L
    rng = np.random.default_rng(94)
    dev = torch.device("cuda", ctx.device)
    shapes = [(1025, 2048), (1024, 2048)]
    images = [rng.integers(0, 256, (h, w, 3), dtype=np.uint8) for h, w in shapes]
    small = rng.integers(0, 256, (40, 127, 3), dtype=np.uint8)
    want = [ops.rotate(img, 13) for img in images] + [ops.rotate(small, 13)]
    for name, pictures, at, stride in [("tiles", images, 0, 3), ("few pixels", images[1:], 0, 3), ("narrow", images + [small], 0, 3), ("off a word", images, 2, 3),
                                       ("four bytes", images, 0, 4)]:
        descs, keep = (L.RotateDesc * len(pictures))(), []
        for d, img in zip(descs, pictures):
            h, w = img.shape[:2]
            src, dst = torch.from_numpy(img).to(dev), torch.zeros(at + h * w * stride, dtype=torch.uint8, device=dev)
            d.src, d.src_pitch, d.src_pixel_stride = src.data_ptr(), 3 * w, 3
            d.width, d.height, d.angle = w, h, 13
            d.dst, d.dst_pitch, d.dst_pixel_stride = dst.data_ptr() + at, w * stride, stride
            keep.append((src, dst))
        torch.cuda.synchronize(dev)
        L.check(ctx.lib.aeonb_rotate_batch(ctx.handle, descs, len(pictures)))
        ctx.synchronize()
        for img, (_, dst), ref in zip(pictures, keep, want[1:] if len(pictures) == 1 else want):
            got = dst[at:].cpu().numpy().reshape(img.shape[0], img.shape[1], stride)[..., :3]
            assert np.array_equal(got, ref), (name, img.shape)
