"""Parity of host entropy decode + GPU JPEG back end with cv2.imdecode and the numpy oracle (bit-exact)."""
import os

import numpy as np
import pytest

from oracle import jpeg as ojpeg
from tests.synth import gradient_image, jpeg_bytes

pytestmark = pytest.mark.gpu


def decode_gpu(ctx, blobs, pixel_stride=3):
    from aeon_b200 import kernels as K
    outs, _ = K.jpeg_decode_batch(ctx, blobs, pixel_stride)
    return [o.cpu().numpy()[..., :3] for o in outs]


@pytest.mark.parametrize("pixel_stride", [3, 4])
def test_batch_420_matches_opencv(ctx, pixel_stride):
    import cv2
    rng = np.random.default_rng(21)
    blobs = []
    for _ in range(16):
        h, w = (int(v) for v in rng.integers(256, 513, 2))
        blobs.append(jpeg_bytes(gradient_image(rng, h, w), 90))
    got = decode_gpu(ctx, blobs, pixel_stride)
    for i, b in enumerate(blobs):
        ref = cv2.imdecode(np.frombuffer(b, np.uint8), cv2.IMREAD_COLOR)
        assert np.array_equal(got[i], ref), "image %d" % i


def test_sampling_modes_odd_sizes_restart_and_grey(ctx):
    import cv2
    rng = np.random.default_rng(22)
    cases = []
    for (h, w) in [(8, 8), (1, 1), (17, 16), (37, 53), (64, 80), (33, 47), (15, 130), (200, 9)]:
        for extra in ([], [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444],
                      [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422],
                      [cv2.IMWRITE_JPEG_RST_INTERVAL, 3]):
            cases.append(jpeg_bytes(rng.integers(0, 256, (h, w, 3), dtype=np.uint8), int(rng.integers(30, 100)), extra))
    cases.append(jpeg_bytes(gradient_image(rng, 45, 30)[..., 0], 85))
    got = decode_gpu(ctx, cases)
    for i, b in enumerate(cases):
        ref = cv2.imdecode(np.frombuffer(b, np.uint8), cv2.IMREAD_COLOR)
        assert np.array_equal(got[i], ref), "case %d" % i
        assert np.array_equal(got[i], ojpeg.decode(b)), "oracle case %d" % i


def test_reference_fixtures(ctx, golden_dir):
    """aeon's own test images: img_2112_70.jpg (480x360) and flowers.jpg (restart interval 38)."""
    import cv2
    blobs = [open(os.path.join(golden_dir, n), "rb").read() for n in ("img_2112_70.jpg", "flowers.jpg")]
    got = decode_gpu(ctx, blobs)
    for g, b in zip(got, blobs):
        assert np.array_equal(g, cv2.imdecode(np.frombuffer(b, np.uint8), cv2.IMREAD_COLOR))


def test_corrupt_streams_raise(ctx):
    from aeon_b200 import kernels as K
    from aeon_b200._lib import AeonError
    for blob in (b"", b"\x00" * 64, b"\xff\xd8\xff\xd9"):
        with pytest.raises(AeonError, match="Decoding image failed"):
            K.jpeg_entropy_decode(blob)


def test_region_decode_equals_the_same_pixels_of_the_full_decode(ctx):
    """Only the MCUs a crop box can touch are decoded; inside the box the pixels must equal the full decode."""
    import ctypes as C
    import cv2
    import torch
    from aeon_b200 import _lib as L, kernels as K
    rng = np.random.default_rng(23)
    dev = torch.device("cuda", ctx.device)
    for (h, w), extra in [((300, 420), []), ((97, 131), []), ((256, 256), [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422]),
                          ((64, 64), [cv2.IMWRITE_JPEG_RST_INTERVAL, 5])]:
        blob = jpeg_bytes(gradient_image(rng, h, w), 90, extra)
        ref = cv2.imdecode(np.frombuffer(blob, np.uint8), cv2.IMREAD_COLOR)
        info = K.jpeg_parse(blob)
        for _ in range(6):
            cw, ch = int(rng.integers(1, w + 1)), int(rng.integers(1, h + 1))
            cx, cy = int(rng.integers(0, w - cw + 1)), int(rng.integers(0, h - ch + 1))
            roi = (C.c_int32 * 4)()
            L.check(ctx.lib.aeonb_jpeg_roi_for_crop(C.byref(info), cx, cy, cw, ch, roi))
            mw, mh = 8 * info.hs[0], 8 * info.vs[0]
            rx, ry = roi[0] * mw, roi[1] * mh
            rw, rh = min(w, roi[2] * mw) - rx, min(h, roi[3] * mh) - ry
            assert rx <= cx and ry <= cy and rx + rw >= cx + cw and ry + rh >= cy + ch
            d = (L.JpegDesc * 1)()
            d[0].width, d[0].height, d[0].ncomp = rw, rh, info.ncomp
            coefs, quants, keep = [], [], []
            for c in range(info.ncomp):
                bw, bh = (roi[2] - roi[0]) * info.hs[c], (roi[3] - roi[1]) * info.vs[c]
                coefs.append(np.zeros(bw * bh * 64, np.int16))
                quants.append(np.zeros(64, np.uint16))
                d[0].hs[c], d[0].vs[c], d[0].blocks_w[c], d[0].blocks_h[c] = info.hs[c], info.vs[c], bw, bh
            cp = (C.c_void_p * 3)(*[c.ctypes.data for c in coefs])
            qp = (C.c_void_p * 3)(*[q.ctypes.data for q in quants])
            buf = (C.c_char * len(blob)).from_buffer_copy(blob)
            L.check(ctx.lib.aeonb_jpeg_entropy_decode_roi(buf, len(blob), roi, cp, qp))
            with torch.cuda.stream(ctx.torch_stream):
                for c in range(info.ncomp):
                    ct, qt = torch.from_numpy(coefs[c]).to(dev), torch.from_numpy(quants[c].view(np.int16)).to(dev)
                    keep += [ct, qt]
                    d[0].coef[c], d[0].quant[c] = ct.data_ptr(), qt.data_ptr()
                pitch = (rw * 3 + 15) // 16 * 16
                out = torch.zeros((rh, pitch), dtype=torch.uint8, device=dev)
                d[0].dst, d[0].dst_pitch, d[0].dst_pixel_stride = out.data_ptr(), pitch, 3
                L.check(ctx.lib.aeonb_jpeg_backend_batch(ctx.handle, d, 1))
                ctx.synchronize()
            got = out.cpu().numpy()[:, :rw * 3].reshape(rh, rw, 3)
            assert np.array_equal(got[cy - ry:cy - ry + ch, cx - rx:cx - rx + cw], ref[cy:cy + ch, cx:cx + cw]), (h, w, cx, cy, cw, ch)


def test_progressive_streams_match_opencv(ctx):
    """Progressive files (SOF2) are entropy-decoded on the host, scan by scan; the GPU back end is the same."""
    import cv2
    rng = np.random.default_rng(29)
    cases = []
    for (h, w) in [(64, 64), (37, 53), (200, 150), (8, 8), (1, 1), (375, 500), (33, 47)]:
        for extra in ([], [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444],
                      [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422], [cv2.IMWRITE_JPEG_RST_INTERVAL, 3]):
            cases.append(jpeg_bytes(gradient_image(rng, h, w), int(rng.integers(30, 100)), [cv2.IMWRITE_JPEG_PROGRESSIVE, 1] + extra))
    cases.append(jpeg_bytes(gradient_image(rng, 45, 30)[..., 0], 85, [cv2.IMWRITE_JPEG_PROGRESSIVE, 1]))
    assert all(b"\xff\xc2" in c for c in cases)
    got = decode_gpu(ctx, cases)
    for i, b in enumerate(cases):
        assert np.array_equal(got[i], cv2.imdecode(np.frombuffer(b, np.uint8), cv2.IMREAD_COLOR)), "case %d" % i


def test_exif_orientation_is_applied_as_opencv_does(ctx):
    import cv2
    from tests.synth import with_exif_orientation
    rng = np.random.default_rng(30)
    cases = []
    for o in range(1, 9):
        h, w = (int(v) for v in rng.integers(20, 200, 2))
        cases.append(with_exif_orientation(jpeg_bytes(gradient_image(rng, h, w), 90), o, big_endian=bool(o % 2)))
    got = decode_gpu(ctx, cases)
    for i, b in enumerate(cases):
        ref = cv2.imdecode(np.frombuffer(b, np.uint8), cv2.IMREAD_COLOR)
        assert got[i].shape == ref.shape and np.array_equal(got[i], ref), "orientation %d" % (i + 1)


def test_440_and_411_sampling(ctx):
    """4:4:0 (libjpeg's vertical-only triangle filter) and 4:1:1 (replication), baseline and progressive, odd sizes."""
    import cv2
    rng = np.random.default_rng(33)
    cases = []
    for (h, w) in [(8, 8), (1, 1), (17, 16), (37, 53), (64, 80), (33, 47), (15, 130), (200, 9), (375, 500)]:
        for factor in (cv2.IMWRITE_JPEG_SAMPLING_FACTOR_440, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_411):
            for extra in ([], [cv2.IMWRITE_JPEG_PROGRESSIVE, 1], [cv2.IMWRITE_JPEG_RST_INTERVAL, 2]):
                cases.append(jpeg_bytes(rng.integers(0, 256, (h, w, 3), dtype=np.uint8), int(rng.integers(30, 100)),
                                        [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, factor] + extra))
    got = decode_gpu(ctx, cases)
    for i, b in enumerate(cases):
        assert np.array_equal(got[i], cv2.imdecode(np.frombuffer(b, np.uint8), cv2.IMREAD_COLOR)), "case %d" % i


@pytest.mark.parametrize("pitch_step", [4, 8])
def test_422_and_420_rows_at_the_edges_of_the_eight_pixel_groups(ctx, pitch_step):
    """Widths around multiples of eight and sixteen (the last group of a row takes the generic path), strips of one and two MCU rows, and
    destinations whose rows are 4-byte but not 8-byte aligned."""
    import ctypes as C
    import cv2
    import torch
    from aeon_b200 import _lib as L, kernels as K
    rng = np.random.default_rng(24)
    dev = torch.device("cuda", ctx.device)
    blobs = [jpeg_bytes(rng.integers(0, 256, (h, w, 3), dtype=np.uint8), 95, [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, mode])
             for mode in (cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420)
             for h, w in [(1, 7), (8, 8), (9, 9), (16, 15), (17, 16), (33, 17), (40, 23), (7, 24), (24, 25), (31, 31), (64, 32), (5, 33), (48, 257)]]
    descs, keep, outs = (L.JpegDesc * len(blobs))(), [], []
    for d, blob in zip(descs, blobs):
        info, coefs, quants = K.jpeg_entropy_decode(blob)
        pitch = (info.width * 3 + 3) // 4 * 4
        pitch += 4 if pitch % 8 != pitch_step % 8 else 0
        out = torch.full((info.height + 1, pitch), 77, dtype=torch.uint8, device=dev)
        d.width, d.height, d.ncomp = info.width, info.height, info.ncomp
        for c in range(info.ncomp):
            d.hs[c], d.vs[c], d.blocks_w[c], d.blocks_h[c] = info.hs[c], info.vs[c], info.blocks_w[c], info.blocks_h[c]
            t, q = torch.from_numpy(coefs[c]).to(dev), torch.from_numpy(quants[c].view(np.int16)).to(dev)
            keep += [t, q]
            d.coef[c], d.quant[c] = t.data_ptr(), q.data_ptr()
        d.dst, d.dst_pitch, d.dst_pixel_stride = out.data_ptr(), pitch, 3
        outs.append(out)
    torch.cuda.synchronize(dev)
    L.check(ctx.lib.aeonb_jpeg_backend_batch(ctx.handle, descs, len(blobs)))
    ctx.synchronize()
    for d, blob, out in zip(descs, blobs, outs):
        want = cv2.imdecode(np.frombuffer(blob, np.uint8), cv2.IMREAD_COLOR)
        got = out.cpu().numpy()
        assert np.array_equal(got[:-1, :d.width * 3].reshape(want.shape), want), (want.shape, d.dst_pitch)
        assert (got[-1] == 77).all()


@pytest.mark.parametrize("mode,widest", [("420", 3440), ("422", 5376), ("444", 3584), (None, 10752)])
def test_pictures_as_wide_as_two_mcu_rows_in_shared_memory_allow(ctx, mode, widest):
    """The sample planes of two MCU rows and the warps' 32 KB of coefficients take 200 KB at most: 50 bytes a column in 4:2:0, 32 in 4:2:2,
    48 in 4:4:4, 16 in grey.  The widest picture decodes, the next one is refused."""
    import cv2
    from aeon_b200._lib import AeonError
    rng = np.random.default_rng(25)
    extra = [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, getattr(cv2, "IMWRITE_JPEG_SAMPLING_FACTOR_" + mode)] if mode else []
    blobs = [jpeg_bytes(gradient_image(rng, 40, w) if mode else gradient_image(rng, 40, w)[..., 0], 90, extra) for w in (widest, widest - 5, widest + 1)]
    for got, blob in zip(decode_gpu(ctx, blobs[:2]), blobs):
        assert np.array_equal(got, cv2.imdecode(np.frombuffer(blob, np.uint8), cv2.IMREAD_COLOR))
    with pytest.raises(AeonError, match="too wide"):
        decode_gpu(ctx, blobs[2:])


@pytest.mark.parametrize("n", [1, 53, 54, 59, 60])
def test_batches_around_the_size_that_travels_with_a_launch(ctx, n):
    """Descriptors go with the launch up to 8064 bytes and through device memory beyond: 53 streams or images, 59 pictures of one strip of MCU
    rows with their work lists.  The same pictures on either side."""
    import ctypes as C
    from aeon_b200 import _lib as L
    near = 8064
    assert near // C.sizeof(L.EntropyDesc) == near // C.sizeof(L.ImageDesc) == 53 and near // (C.sizeof(L.JpegDesc) + 8) == 59
    from aeon_b200.provider import Provider
    from tests.pipeline_oracle import PipelineOracle
    rng = np.random.default_rng(80 + n)
    recs = [(jpeg_bytes(gradient_image(rng, int(rng.integers(20, 33)), int(rng.integers(20, 90))), 90),) for _ in range(n)]
    cfg = {"batch_size": n, "random_seed": 3, "etl": [{"type": "image", "height": 64, "width": 48}],
           "augmentation": [{"type": "image", "crop_enable": True, "center": False, "scale": [0.5, 1.0], "flip_enable": True}]}
    prov = Provider(ctx, cfg)
    try:
        assert np.array_equal(prov.run_host(recs)["image"], PipelineOracle(cfg).batch(recs)["image"])
    finally:
        prov.close()
