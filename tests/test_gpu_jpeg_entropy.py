"""Device entropy decoders (a cluster of thread blocks per JPEG stream, or a block, decoding segments speculatively; a block per run of
intervals for streams with restart markers; one warp per stream) against the host decoder and against the oracle: identical coefficient
planes.

Launches of up to 66 streams, none longer than about 120 KB and none with more than six blocks in an MCU, go through the kernel that spreads
a stream over a cluster; padded to 67 (1024 threads at most) or 149 (512) they go through the one with a block per stream."""
import ctypes as C
import os

import numpy as np
import pytest

from tests.synth import gradient_image, jpeg_bytes

pytestmark = pytest.mark.gpu


def host_planes(blob, roi=None):
    from aeon_b200 import _lib as L
    from aeon_b200 import kernels as K
    if roi is None:
        info, coefs, quants = K.jpeg_entropy_decode(blob)
        return info, coefs, quants
    lib = L.load()
    info = K.jpeg_parse(blob)
    nb = [(roi[2] - roi[0]) * info.hs[c] * (roi[3] - roi[1]) * info.vs[c] for c in range(info.ncomp)]
    coefs = [np.zeros(max(n * 64, 1), np.int16) for n in nb] + [np.zeros(1, np.int16)] * (3 - info.ncomp)
    quants = [np.zeros(64, np.uint16) for _ in range(3)]
    cp = (C.c_void_p * 3)(*[c.ctypes.data for c in coefs])
    qp = (C.c_void_p * 3)(*[q.ctypes.data for q in quants])
    buf = (C.c_char * len(blob)).from_buffer_copy(blob)
    r = (C.c_int32 * 4)(*roi)
    L.check(lib.aeonb_jpeg_entropy_decode_roi(buf, len(blob), r, cp, qp))
    return info, coefs[:info.ncomp], quants[:info.ncomp]


@pytest.fixture(params=[True, False], ids=["block-parallel", "one-warp"])
def parallel(request):
    return request.param


def check(ctx, blobs, rois=None, parallel=True):
    from aeon_b200 import kernels as K
    got = K.jpeg_entropy_decode_device(ctx, blobs, rois, parallel)
    for i, blob in enumerate(blobs):
        info, planes, quant, status = got[i]
        assert status == 0, "record %d status %d" % (i, status)
        hinfo, hcoefs, hquants = host_planes(blob, None if rois is None else rois[i])
        assert info.ncomp == hinfo.ncomp
        for c in range(info.ncomp):
            assert np.array_equal(planes[c].cpu().numpy(), hcoefs[c][:planes[c].numel()]), "record %d component %d" % (i, c)
            assert np.array_equal(quant[c], hquants[c])


def test_sampling_modes_sizes_and_restarts(ctx, parallel):
    import cv2
    rng = np.random.default_rng(61)
    blobs = []
    for (h, w) in [(8, 8), (1, 1), (17, 16), (37, 53), (64, 80), (33, 47), (15, 130), (200, 9), (256, 256)]:
        for extra in ([], [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444],
                      [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422],
                      [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_440],
                      [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_411],
                      [cv2.IMWRITE_JPEG_RST_INTERVAL, 3], [cv2.IMWRITE_JPEG_OPTIMIZE, 1]):
            blobs.append(jpeg_bytes(rng.integers(0, 256, (h, w, 3), dtype=np.uint8), int(rng.integers(30, 101)), extra))
    blobs.append(jpeg_bytes(gradient_image(rng, 45, 30)[..., 0], 85))
    check(ctx, blobs, parallel=parallel)


def test_noise_at_quality_100_exercises_long_codes_and_stuffing(ctx, parallel):
    rng = np.random.default_rng(62)
    blobs = [jpeg_bytes(rng.integers(0, 256, (96, 160, 3), dtype=np.uint8), 100) for _ in range(4)]
    assert any(b"\xff\x00" in b for b in blobs)
    check(ctx, blobs, parallel=parallel)


def test_natural_batch_and_reference_fixtures(ctx, golden_dir, parallel):
    rng = np.random.default_rng(63)
    blobs = [jpeg_bytes(gradient_image(rng, int(rng.integers(256, 513)), int(rng.integers(256, 513))), 90) for _ in range(32)]
    blobs += [open(os.path.join(golden_dir, n), "rb").read() for n in ("img_2112_70.jpg", "flowers.jpg")]
    check(ctx, blobs, parallel=parallel)


@pytest.mark.parametrize("parallel, n", [(True, 12), (True, 67), (True, 149), (False, 12)])
def test_regions(ctx, parallel, n):
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(64)
    blobs, rois = [], []
    for _ in range(12):
        h, w = (int(v) for v in rng.integers(100, 400, 2))
        blob = jpeg_bytes(gradient_image(rng, h, w), 85)
        info = K.jpeg_parse(blob)
        mcux, mcuy = info.blocks_w[0] // info.hs[0], info.blocks_h[0] // info.vs[0]
        x0, y0 = int(rng.integers(0, mcux)), int(rng.integers(0, mcuy))
        x1, y1 = int(rng.integers(x0 + 1, mcux + 1)), int(rng.integers(y0 + 1, mcuy + 1))
        blobs.append(blob)
        rois.append((x0, y0, x1, y1))
    check(ctx, [blobs[i % 12] for i in range(n)], [rois[i % 12] for i in range(n)], parallel)


@pytest.mark.parametrize("parallel, n", [(True, 3), (True, 67), (True, 149), (False, 3)])
def test_malformed_stream_sets_status_and_returns(ctx, parallel, n):
    """A scan of 0xFF filler and one of random bytes: the kernel flags them (or decodes garbage) and terminates."""
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(65)
    good = jpeg_bytes(gradient_image(rng, 128, 128), 90)
    sos = good.index(b"\xff\xda")
    head = good[:sos + 14]
    truncated = good[:sos + 14 + 200] + b"\xff\xd9"
    noise = head + bytes(rng.integers(0, 255, 3000, dtype=np.uint8)) + b"\xff\xd9"
    got = K.jpeg_entropy_decode_device(ctx, [good, truncated, noise] + [good] * (n - 3), None, parallel)
    assert [g[3] for g in got[:1] + got[3:]] == [0] * (n - 2)
    assert got[1][3] in (0, 1) and got[2][3] in (0, 1)
    # and the context is still usable
    check(ctx, [good] * (n - 2), parallel=parallel)


def test_large_picture_and_many_streams(ctx, parallel):
    """A 2048x1536 picture (segments of several KB per thread) and a launch of 600 small streams (more blocks than fit at once)."""
    rng = np.random.default_rng(66)
    big = jpeg_bytes(gradient_image(rng, 1536, 2048), 92)
    assert len(big) > 400_000
    check(ctx, [big], parallel=parallel)
    small = [jpeg_bytes(gradient_image(rng, int(rng.integers(16, 64)), int(rng.integers(16, 64))), 80) for _ in range(40)]
    check(ctx, [small[i % 40] for i in range(600)], parallel=parallel)


def test_device_decoder_against_the_oracle_planes(ctx, golden_dir, parallel):
    """Both device kernels against oracle/jpeg.py's own Huffman decoder (not only against the library's host decoder)."""
    import cv2
    from aeon_b200 import kernels as K
    from oracle import jpeg as ojpeg
    rng = np.random.default_rng(67)
    blobs = [jpeg_bytes(gradient_image(rng, 40, 56), 90), jpeg_bytes(gradient_image(rng, 33, 47), 75, [cv2.IMWRITE_JPEG_RST_INTERVAL, 2]),
             jpeg_bytes(rng.integers(0, 256, (24, 24, 3), dtype=np.uint8), 100, [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444]),
             open(os.path.join(golden_dir, "img_2112_70.jpg"), "rb").read()]
    got = K.jpeg_entropy_decode_device(ctx, blobs, None, parallel)
    for i, blob in enumerate(blobs):
        info, planes, quant, status = got[i]
        co = ojpeg.entropy_decode(blob)
        assert status == 0 and (info.width, info.height, info.ncomp) == (co.width, co.height, co.ncomp)
        for c in range(info.ncomp):
            mine = planes[c].cpu().numpy().reshape(info.blocks_h[c], info.blocks_w[c], 8, 8).transpose(0, 1, 3, 2)  # column-major blocks
            assert np.array_equal(mine, co.blocks[c]), (i, c)


def test_streams_with_more_segments_than_the_smallest_segment_allows(ctx, golden_dir):
    """Streams longer than threads x smallest segment get longer segments, and their last, short segment can end a few
    bits before a checkpoint position.  The fixture is a 90 KB stream of the benchmark's generator (507 segments of 176
    bytes) whose last segment ends 8 bits before its second checkpoint: a run that stepped over that position with its
    last symbol once left a note there that a later run fell into step with, and the stream was reported as malformed
    although every coefficient was right."""
    blob = open(os.path.join(golden_dir, "entropy_stream_507_segments.jpg"), "rb").read()
    check(ctx, [blob])
    info = host_planes(blob)[0]
    mcux, mcuy = info.blocks_w[0] // info.hs[0], info.blocks_h[0] // info.vs[0]
    rois = [(0, 0, mcux, mcuy), (3, 5, mcux - 2, mcuy), (0, mcuy - 1, mcux, mcuy), (0, 0, mcux, mcuy - 1)]
    for n in (4, 68, 149):
        check(ctx, [blob] * n, [rois[i % 4] for i in range(n)])
    rng = np.random.default_rng(77)
    big = []
    for k in range(24):   # 84-140 KB: segments of 164 to 280 bytes, last segments of every length
        h, w = int(rng.integers(440, 513)), int(rng.integers(440, 513))
        img = np.clip(gradient_image(rng, h, w).astype(np.int16) + rng.integers(-28 - k, 29 + k, (h, w, 3)), 0, 255).astype(np.uint8)
        big.append(jpeg_bytes(img, 92))
    assert min(len(b) for b in big) > 84000
    check(ctx, big)
    check(ctx, [big[i % 24] for i in range(67)])


def restart_offsets(blob):
    """Positions of the restart markers of a file (of their 0xFF)."""
    start = blob.index(b"\xff\xda")
    return [i for i in range(start, len(blob) - 1) if blob[i] == 0xFF and 0xD0 <= blob[i + 1] <= 0xD7]


@pytest.mark.parametrize("interval", [1, 2, 7, 64, 65, 1000])
def test_restart_intervals(ctx, interval):
    """Interval decoding at the edges of its partition: intervals of one MCU (more of them than a part takes, fewer bytes than a
    segment), of many MCUs (several segments each), more than the picture has; pictures with a ragged last interval; regions that
    end inside an interval.  Identical planes to the host decoder."""
    import cv2
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(680 + interval)
    blobs, rois = [], []
    for (h, w), mode in [((8, 8), None), ((75, 333), None), ((210, 190), cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422),
                         ((130, 260), cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444), ((520, 700), cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420)]:
        extra = [cv2.IMWRITE_JPEG_RST_INTERVAL, interval] + ([cv2.IMWRITE_JPEG_SAMPLING_FACTOR, mode] if mode else [])
        for quality in (60, 95, 100):   # at 100 the noise brings stuffed bytes at every place of a vector
            img = gradient_image(rng, h, w) if quality < 100 else rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
            blob = jpeg_bytes(img, quality, extra)
            info = K.jpeg_parse(blob)
            mcux, mcuy = info.blocks_w[0] // info.hs[0], info.blocks_h[0] // info.vs[0]
            x0, y0 = int(rng.integers(0, mcux)), int(rng.integers(0, mcuy))
            blobs += [blob, blob]
            rois += [(0, 0, mcux, mcuy), (x0, y0, int(rng.integers(x0 + 1, mcux + 1)), int(rng.integers(y0 + 1, mcuy + 1)))]
    check(ctx, blobs, rois)
    check(ctx, blobs[:1], rois[:1])


@pytest.mark.parametrize("n", [1, 15, 16, 33, 34, 66, 67])
def test_restart_index_over_clusters(ctx, n):
    """Launches at the edges of the number of blocks that look for a stream's markers: streams of a few vectors, whose blocks are mostly
    empty, beside one of 100 KB, markers at every place of a vector and on both sides of a block's share."""
    import cv2
    rng = np.random.default_rng(690 + n)
    long = jpeg_bytes(rng.integers(0, 256, (230, 400, 3), dtype=np.uint8), 95, [cv2.IMWRITE_JPEG_RST_INTERVAL, 1])
    assert len(long) > 100_000
    small = [jpeg_bytes(gradient_image(rng, int(rng.integers(8, 60)), int(rng.integers(8, 60))), 85, [cv2.IMWRITE_JPEG_RST_INTERVAL, int(rng.integers(1, 5))])
             for _ in range(8)]
    check(ctx, [long if i == n // 2 else small[i % 8] for i in range(n)])
    check(ctx, [small[i % 8] for i in range(n)])


def test_damaged_restart_streams_are_left_to_the_serial_decoder(ctx):
    """Streams whose intervals are not all there, or do not end where they should: with and without a work area the same status,
    and the same planes where the status is good."""
    import cv2
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(69)
    good = jpeg_bytes(gradient_image(rng, 200, 330), 90, [cv2.IMWRITE_JPEG_RST_INTERVAL, 5])
    at = restart_offsets(good)
    assert len(at) > 30
    a, b = at[10], at[11]
    damaged = [good[:a] + good[a + 2:],                       # a marker lost
               good[:a] + good[b:],                           # an interval lost
               good[:a] + b"\xff" + good[a:],                 # a fill byte in front of a marker
               good[:a] + b"\xff\xd3" + good[a:],             # an empty interval
               good[:a] + bytes(40) + good[a:],               # bytes behind an interval's last block, few and many
               good[:a] + bytes(90) + good[a:],
               good[:a - 3] + good[a:],                       # an interval cut short
               good[:b] + b"\xff\xd9",                        # the end of the stream lost
               good[:a + 9] + b"\xff\xfe" + good[a + 9:],     # a foreign marker inside an interval
               good[:a + 4] + bytes(rng.integers(0, 255, b - a - 8, dtype=np.uint8)) + good[b - 4:]]
    blobs = [good] + damaged + [good]
    serial = K.jpeg_entropy_decode_device(ctx, blobs, None, parallel=False)
    got = K.jpeg_entropy_decode_device(ctx, blobs, None, parallel=True)
    assert serial[0][3] == 0 and {s[3] for s in serial} == {0, 1}
    for i, (g, s) in enumerate(zip(got, serial)):
        assert g[3] == s[3], i
        for c in range(3):
            assert s[3] != 0 or np.array_equal(g[1][c].cpu().numpy(), s[1][c].cpu().numpy()), (i, c)
    check(ctx, [good])


@pytest.mark.parametrize("copies", [1, 148, 149])
def test_block_sizes_on_either_side_of_a_stream_per_sm(ctx, golden_dir, copies):
    """Up to one stream per SM a stream gets a thread per piece of the storing pass, above that a thread per segment and less shared
    memory.  A stream of 507 segments, noise at quality 100 (long codes, blocks that end at coefficient 63 without an end-of-block code)
    and a stream too long for the shared memory of a block that shares its SM."""
    rng = np.random.default_rng(78)
    blobs = [open(os.path.join(golden_dir, "entropy_stream_507_segments.jpg"), "rb").read(),
             jpeg_bytes(rng.integers(0, 256, (168, 200, 3), dtype=np.uint8), 100),
             jpeg_bytes(rng.integers(0, 256, (300, 400, 3), dtype=np.uint8), 97),
             jpeg_bytes(gradient_image(rng, 24, 40), 75)]
    assert len(blobs[2]) > 115_000
    for blob in blobs if copies == 1 else [None]:
        check(ctx, [blob] if blob else [blobs[i % len(blobs)] for i in range(copies)])


def test_streams_that_fit_with_fewer_segments(ctx):
    """Streams around the longest that two blocks on an SM can hold: the launch's longest one decides how many segments there is room for
    beside it (382 of them at 57 KB, 128 at 69 KB; behind that the copy goes to global memory)."""
    rng = np.random.default_rng(79)
    img = np.clip(gradient_image(rng, 400, 900).astype(np.int16) + rng.integers(-24, 25, (400, 900, 3)), 0, 255).astype(np.uint8)
    blobs, w = [], 240
    for size in (54_000, 58_000, 62_000, 66_000, 68_500, 71_000):
        while len(jpeg_bytes(img[:, :w], 90)) < size:
            w += 4
        blobs.append(jpeg_bytes(img[:, :w], 90))
        assert len(blobs[-1]) < size + 1500
    for longest in range(1, len(blobs) + 1):
        check(ctx, [blobs[longest - 1 - i % min(longest, 2)] for i in range(149)])


def decode_descs(ctx, blobs, rois=None, lead=0, scratch=True, scan_bytes=None):
    """Entropy decode with the descriptors in hand: (status, [planes], work area, descriptor) of every record.  `lead`: offset of a scan from a
    16-byte boundary; `scan_bytes`: cuts the scans off; work areas are zeroed before."""
    import torch
    from aeon_b200 import _lib as L
    lib, dev = ctx.lib, torch.device("cuda", ctx.device)
    descs = (L.EntropyDesc * len(blobs))()
    status = torch.full((len(blobs),), -1, dtype=torch.int32, device=dev)
    keep, out = [], []
    for i, (d, blob) in enumerate(zip(descs, blobs)):
        info, quant, tables, off = L.JpegInfo(), np.zeros(192, np.uint16), np.zeros(1088, np.uint8), C.c_size_t()
        buf = (C.c_char * len(blob)).from_buffer_copy(blob)
        L.check(lib.aeonb_jpeg_entropy_prepare(buf, len(blob), C.byref(info), quant.ctypes.data_as(C.POINTER(C.c_uint16)),
                                               tables.ctypes.data_as(C.POINTER(C.c_uint8)), C.byref(d), C.byref(off)))
        d.scan_size = d.scan_size if scan_bytes is None else min(d.scan_size, scan_bytes)
        scan = np.full(d.scan_size + 64, 0xFF, np.uint8)
        scan[lead:lead + d.scan_size] = np.frombuffer(blob, np.uint8)[off.value:off.value + d.scan_size]
        scan, tables = torch.from_numpy(scan).to(dev), torch.from_numpy(tables).to(dev)
        for k in range(4 if rois else 0):
            d.roi[k] = rois[i][k]
        planes = [torch.full(((d.roi[2] - d.roi[0]) * d.hs[c] * (d.roi[3] - d.roi[1]) * d.vs[c] * 64,), 0x5555, dtype=torch.int16, device=dev)
                  for c in range(info.ncomp)]
        for c, p in enumerate(planes):
            d.coef[c] = p.data_ptr()
        d.scan, d.tables, d.status = scan.data_ptr() + lead, tables.data_ptr(), status.data_ptr() + 4 * i
        d.scratch_bytes = int(lib.aeonb_jpeg_entropy_scratch_bytes(C.byref(d)))
        work = torch.zeros(d.scratch_bytes, dtype=torch.uint8, device=dev)
        d.scratch = work.data_ptr() if scratch else None
        keep += [scan, tables]
        out.append((planes, work))
    torch.cuda.synchronize(dev)
    L.check(lib.aeonb_jpeg_entropy_batch(ctx.handle, descs, len(blobs)))
    ctx.synchronize()
    return [(int(s), [p.cpu().numpy() for p in planes], work.cpu().numpy(), d)
            for s, (planes, work), d in zip(status.cpu().numpy(), out, descs)]


@pytest.mark.parametrize("interval", [1, 3, 1000])
def test_restart_streams_without_a_byte_of_data(ctx, interval):
    """A file with restart markers that ends behind its scan header, alone in a batch and beside a whole one: whatever the work area
    holds, the status is the serial decoder's."""
    import cv2
    blob = jpeg_bytes(gradient_image(np.random.default_rng(70), 64, 96), 90, [cv2.IMWRITE_JPEG_RST_INTERVAL, interval])
    want = decode_descs(ctx, [blob], scratch=False, scan_bytes=0)[0]
    for lead in (0, 5):
        for got in (decode_descs(ctx, [blob], lead=lead, scan_bytes=0), decode_descs(ctx, [blob] * 3, lead=lead, scan_bytes=0)):
            for status, planes, _, _ in got:
                assert status == want[0]
                assert status != 0 or all(np.array_equal(a, b) for a, b in zip(planes, want[1]))
    assert want[0] == (1 if interval < 1000 else 0)


def coded_grey(rng, size, whole):
    """A grey JPEG whose entropy-coded data takes `size` bytes: its table gives the end of a block nine bits, eight ones and a zero.  Without
    the end of the last block (`whole` false) the data ends at a byte's end just in front of it."""
    dc = [("00", 0), ("01", 1), ("10", 5)]
    ac = [("0", 0x01), ("10", 0x02), ("110", 0x11), ("1110", 0x03), ("11110", 0x04), ("111110", 0x22), ("1111110", 0x05), ("11111110", 0x31)]
    plain = [a for a in ac if a[1] < 16]
    out, bits, blocks = bytearray(), "", 0

    def put(code, value_bits=0):
        nonlocal bits
        bits += code + (format(int(rng.integers(1 << value_bits)), "b").zfill(value_bits) if value_bits else "")
        while len(bits) >= 8:
            out.append(int(bits[:8], 2))
            if out[-1] == 0xFF:
                out.append(0)
            bits = bits[8:]

    def symbol(table):
        code, sym = table[rng.integers(len(table))]
        put(code, sym & 15)

    while len(out) < size - (20 if size < 10000 else 60):
        symbol(dc)
        for _ in range(rng.integers(0, 6) if size < 10000 else 55):      # a picture has at most 8191 blocks in a row
            symbol(ac if size < 10000 else plain)
        put("111111110")
        blocks += 1
    kept = bytes(out), bits
    while True:      # the last block: symbols until the data ends where it should
        out[:], bits = kept
        symbol(dc)
        for _ in range(60):
            if len(out) == size and (not whole) and bits == "":
                break
            if whole and len(out) + 3 > size:
                put("111111110")
                if bits:
                    put("1" * (8 - len(bits)))
                break
            symbol(plain)
        if len(out) == size and bits == "":
            break
    blocks += 1
    mark = lambda m, body: bytes([0xFF, m]) + (len(body) + 2).to_bytes(2, "big") + body  # noqa: E731
    dht = lambda cls, lens, syms: mark(0xC4, bytes([cls]) + bytes(lens + [0] * (16 - len(lens))) + bytes(syms))  # noqa: E731
    return (b"\xff\xd8" + mark(0xDB, bytes([0]) + bytes([1] * 64)) +
            mark(0xC0, bytes([8, 0, 8]) + (8 * blocks).to_bytes(2, "big") + bytes([1, 1, 0x11, 0])) +
            dht(0x00, [0, 3], [s for _, s in dc]) + dht(0x10, [1] * 9, [s for _, s in ac] + [0]) +
            mark(0xDA, bytes([1, 1, 0, 0, 63, 0])) + bytes(out) + b"\xff\xd9" + bytes(20))


@pytest.mark.parametrize("n, tile", [(1, 8192), (67, 4096), (149, 4096), (67, 8192), (1, 13 * 16384)])
def test_streams_that_end_at_the_edge_of_a_tile(ctx, n, tile):
    """The end marker at every place around a multiple of the bytes a block copies at a time -- 16 for each of its threads: 512 of a cluster's
    only block, 256 of the blocks that short streams get in launches of more than 66, 1024 and the copy in the work area for
    the long one: a whole stream decodes, one cut short in front of its last code is reported, also where the marker's first byte is
    the last of a tile."""
    rng = np.random.default_rng(tile)
    for size, lead in [(tile - 2, 0), (tile - 1, 0), (tile, 0), (tile + 1, 0), (tile - 1 - 6, 6), (tile - 1 - 15, 15)][:6 if tile < 10000 else 3]:
        blob = coded_grey(rng, size, True)
        want = host_planes(blob)[1][0]
        for status, planes, _, _ in decode_descs(ctx, [blob] * n, lead=lead):
            assert status == 0 and np.array_equal(planes[0], want[:planes[0].size]), (size, lead)
        cut = decode_descs(ctx, [coded_grey(rng, size, False)] * n, lead=lead)
        assert all(status == 1 for status, _, _, _ in cut), (size, lead)


def left_to_the_serial_decoder(work, d):
    """The first word of the work area's header: not 0 where the interval decoder has given a stream up."""
    mcus, bpm = d.mcux * d.mcuy, sum(d.hs[c] * d.vs[c] for c in range(d.ncomp))
    intervals = -(-mcus // d.restart_interval)
    parts = intervals if intervals < 96 else intervals // 256 + 96
    at = (d.scan_size + 64 * (parts + 2) + 15) // 16 * 16 + (mcus * bpm * 2 + 15) // 16 * 16
    return int(work[at:at + 4].view(np.uint32)[0])


@pytest.mark.parametrize("interval", [2, 7, 13, 40, 64, 1000])
def test_regions_that_end_inside_a_restart_interval(ctx, interval):
    """A region whose last row is not the end of an interval: the rest of that interval is not looked at, and the stream stays with the
    interval decoder.  Every last row of a picture of 13 x 9 MCUs, and the same planes as the host decoder."""
    import cv2
    blob = jpeg_bytes(gradient_image(np.random.default_rng(71), 9 * 16 - 3, 13 * 16 - 5), 90, [cv2.IMWRITE_JPEG_RST_INTERVAL, interval])
    rois = [(x0, y0, x1, y1) for y1 in range(1, 10) for x0, x1, y0 in ((0, 13, 0), (3, 9, y1 // 2))]
    for roi, (status, planes, work, d) in zip(rois, decode_descs(ctx, [blob] * len(rois), rois)):
        _, want, _ = host_planes(blob, roi)
        assert status == 0 and all(np.array_equal(p, w[:p.size]) for p, w in zip(planes, want)), roi
        assert left_to_the_serial_decoder(work, d) == 0, roi


@pytest.mark.parametrize("h, w, interval, parts_of", [(16 * 20 - 3, 16 * 26 - 5, 1, 6), (16 * 16, 16 * 16, 1, 3), (16 * 40, 16 * 40, 2, 9), (24, 16 * 400, 1, 9)])
def test_many_restart_intervals(ctx, h, w, interval, parts_of):
    """More than 256 intervals, the most that a block takes, and as many as that (the work area's layout changes at 96 and with every 256):
    identical planes, and the stream stays with the interval decoder, for the whole picture and for regions.  `parts_of`: one stream in a
    launch, or beside enough others that its parts hold more intervals."""
    import cv2
    rng = np.random.default_rng(73)
    blob = jpeg_bytes(gradient_image(rng, h, w), 85, [cv2.IMWRITE_JPEG_RST_INTERVAL, interval])
    mcux, mcuy = -(-w // 16), -(-h // 16)
    assert -(-mcux * mcuy // interval) >= 256
    whole, part = (0, 0, mcux, mcuy), (1, mcuy // 3, mcux - 2, max(mcuy - 1, mcuy // 3 + 1))
    for n in (1, parts_of, 40):
        rois = [whole if i % 2 == 0 else part for i in range(n)]
        for roi, (status, planes, work, d) in zip(rois, decode_descs(ctx, [blob] * n, rois)):
            _, want, _ = host_planes(blob, roi)
            assert status == 0 and all(np.array_equal(p, x[:p.size]) for p, x in zip(planes, want)), roi
            assert left_to_the_serial_decoder(work, d) == 0, roi


def recode(blob, dc_lengths, ac_lengths, interval=0):
    """The same coefficients coded with other Huffman tables, one for DC and one for AC symbols: code lengths by symbol.  With `interval`, a
    restart marker after every so many MCUs."""
    import struct
    from aeon_b200 import kernels as K
    info, coefs, _ = K.jpeg_entropy_decode(blob)
    zz = [0, 8, 1, 2, 9, 16, 24, 17, 10, 3, 4, 11, 18, 25, 32, 40, 33, 26, 19, 12, 5, 6, 13, 20, 27, 34, 41, 48, 56, 49, 42, 35, 28, 21, 14, 7,
          15, 22, 29, 36, 43, 50, 57, 58, 51, 44, 37, 30, 23, 31, 38, 45, 52, 59, 60, 53, 46, 39, 47, 54, 61, 62, 55, 63]  # column-major

    def canonical(lengths):
        codes, code, last = {}, 0, 0
        for sym, ln in sorted(lengths.items(), key=lambda s: (s[1], s[0])):
            code <<= ln - last
            codes[sym], code, last = (code, ln), code + 1, ln
        counts = bytes(sum(v == ln for v in lengths.values()) for ln in range(1, 17))
        return codes, counts + bytes(s for s, _ in sorted(lengths.items(), key=lambda s: (s[1], s[0])))

    (dc, dc_table), (ac, ac_table) = canonical(dc_lengths), canonical(ac_lengths)
    bits, body = [], b""

    def put(code, value, size):
        bits.append(format(code[0], "0%db" % code[1]))
        if size:
            bits.append(format(value if value > 0 else value + (1 << size) - 1, "0%db" % size))

    def whole_bytes():
        text = "".join(bits)
        text += "1" * (-len(text) % 8)
        bits.clear()
        return bytes(int(text[i:i + 8], 2) for i in range(0, len(text), 8)).replace(b"\xff", b"\xff\x00")

    pred = [0] * info.ncomp
    for m in range((info.blocks_w[0] // info.hs[0]) * (info.blocks_h[0] // info.vs[0])):
        mx, my = m % (info.blocks_w[0] // info.hs[0]), m // (info.blocks_w[0] // info.hs[0])
        if interval and m and m % interval == 0:
            body += whole_bytes() + bytes([0xFF, 0xD0 + (m // interval - 1) % 8])
            pred = [0] * info.ncomp
        for c in range(info.ncomp):
            for y in range(info.vs[c]):
                for x in range(info.hs[c]):
                    at = ((my * info.vs[c] + y) * info.blocks_w[c] + mx * info.hs[c] + x) * 64
                    block = [int(coefs[c][at + zz[k]]) for k in range(64)]
                    diff, pred[c] = block[0] - pred[c], block[0]
                    put(dc[abs(diff).bit_length()], diff, abs(diff).bit_length())
                    run = 0
                    for k in range(1, 64):
                        if block[k] == 0:
                            run += 1
                            continue
                        for _ in range(run // 16):
                            put(ac[0xf0], 0, 0)
                        size = abs(block[k]).bit_length()
                        put(ac[run % 16 << 4 | size], block[k], size)
                        run = 0
                    if run:
                        put(ac[0], 0, 0)
    body += whole_bytes()
    out, p = blob[:2], 2
    while blob[p + 1] != 0xDA:          # the other segments as they are, without the tables
        end = p + 2 + struct.unpack(">H", blob[p + 2:p + 4])[0]
        out += blob[p:end] if blob[p + 1] != 0xC4 else b""
        p = end
    out += b"\xff\xdd" + struct.pack(">HH", 4, interval) if interval else b""
    for kind, table in ((0, dc_table), (0x10, ac_table)):
        out += b"\xff\xc4" + struct.pack(">H", 3 + len(table)) + bytes([kind]) + table
    sos = bytearray(blob[p:p + 2 + struct.unpack(">H", blob[p + 2:p + 4])[0]])
    for c in range(info.ncomp):
        sos[6 + 2 * c] = 0
    return out + bytes(sos) + body + b"\xff\xd9"


@pytest.mark.parametrize("dc_long, ac_long, ac_short", [(5, 10, 2), (9, 11, 3), (10, 12, 3), (12, 12, 4), (16, 16, 1), (5, 16, 2)])
def test_tables_with_codes_longer_than_the_lookup_windows(ctx, dc_long, ac_long, ac_short):
    """Canonical tables with a few short codes and the rest of one length: just inside the windows (9 bits DC, 11 AC), just outside, and
    so long that they do not start near the end of the code space, where the tables expect codes beyond the windows.  In one stream of
    a launch only, in the kernel for few streams, in the one with a block per stream, in shared memory and too long for it, and in the one
    for restart markers."""
    import cv2
    rng = np.random.default_rng(70)
    img = gradient_image(rng, 90, 130)
    plain = jpeg_bytes(img, 88)
    dc = {s: (2 if s in (2, 3) else dc_long) for s in range(12)}
    short = [0x01, 0x00, 0x02, 0x11][:ac_short]
    ac = {r << 4 | s: ac_long for r in range(16) for s in range(1, 11)}
    ac.update({0x00: ac_long, 0xf0: ac_long})
    ac.update({s: k + 1 for k, s in enumerate(short)})
    assert sum(2.0 ** -v for v in ac.values()) < 1 and sum(2.0 ** -v for v in dc.values()) < 1
    blob = recode(plain, dc, ac)
    assert np.array_equal(cv2.imdecode(np.frombuffer(blob, np.uint8), 1), cv2.imdecode(np.frombuffer(plain, np.uint8), 1))
    check(ctx, [plain, blob, jpeg_bytes(img, 88, [cv2.IMWRITE_JPEG_OPTIMIZE, 1])])
    check(ctx, [blob])
    for n in (67, 149):
        check(ctx, [plain] * (n - 1) + [blob])
    restart = [recode(plain, dc, ac, interval) for interval in (1, 9, 1000)]
    assert np.array_equal(cv2.imdecode(np.frombuffer(restart[0], np.uint8), 1), cv2.imdecode(np.frombuffer(plain, np.uint8), 1))
    for status, planes, work, d in decode_descs(ctx, restart):
        assert status == 0 and all(np.array_equal(p, x[:p.size]) for p, x in zip(planes, host_planes(plain)[1]))
        assert left_to_the_serial_decoder(work, d) == 0
    tall = recode(jpeg_bytes(np.concatenate([img[:80]] * 26), 98), dc, ac)
    assert len(tall) > 227 * 1024
    check(ctx, [tall])


@pytest.mark.parametrize("n", [1, 15, 16, 34, 66, 67])
def test_streams_spread_over_clusters(ctx, n):
    """Launches at the edges of the number of blocks a stream is spread over, with streams of every length in one launch (one MCU up to
    more than the longest one's share per block), of every number of places in an MCU, of regions, of pictures so flat that a
    run entered at a wrong bit stays out of step to the end of the flat part, and of streams that a marker ends early."""
    import cv2
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(710 + n)
    modes = [cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422,
             cv2.IMWRITE_JPEG_SAMPLING_FACTOR_411, None]
    blobs, rois = [], []
    for i in range(n + 5):
        h, w = [(430, 470), (8, 8), (300, 200), (64, 500), (17, 33)][i % 5]
        img = gradient_image(rng, h, w)
        kind = (i // 5) % 4 if n > 1 else i
        if kind == 1:
            img[h // 4:] = 128          # flat from a quarter on
        elif kind == 2:
            img = np.full((h, w, 3), int(rng.integers(0, 256)), np.uint8)
        elif kind == 3:
            img = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
        mode = modes[(i // 3) % 5]
        blob = (jpeg_bytes(img[..., 0], 90) if mode is None else jpeg_bytes(img, int(rng.choice([60, 90, 97])), [cv2.IMWRITE_JPEG_SAMPLING_FACTOR, mode]))
        info = K.jpeg_parse(blob)
        mcux, mcuy = info.blocks_w[0] // info.hs[0], info.blocks_h[0] // info.vs[0]
        x0, y0 = int(rng.integers(0, mcux)), int(rng.integers(0, mcuy))
        blobs.append(blob)
        rois.append((0, 0, mcux, mcuy) if i % 2 else (x0, y0, int(rng.integers(x0 + 1, mcux + 1)), int(rng.integers(y0 + 1, mcuy + 1))))
    for first in (0, 5):
        check(ctx, blobs[first:first + n], rois[first:first + n])
    if n == 1:
        for blob, roi in zip(blobs, rois):
            check(ctx, [blob], [roi])


def test_more_noted_states_than_there_is_room_for(ctx):
    """Noise of which hardly any run falls into step with another: more states on the way than a block has room for."""
    from tests.entropy_model import SPREAD_EXTRA, simulate_spread
    rng = np.random.default_rng(74)
    blobs = [jpeg_bytes(rng.integers(0, 256, (160, 120 + 40 * k, 3), dtype=np.uint8), 100) for k in range(3)]
    for blob in blobs:
        assert max(simulate_spread(blob, len(blobs))["noted"]) > SPREAD_EXTRA
    check(ctx, blobs)


@pytest.mark.parametrize("n", [2, 67, 149])
def test_streams_cut_short(ctx, n):
    """A stream of which a part is missing: the status is 1 unless the region needs none of it, at cuts around the places where the
    blocks of a cluster share the stream out; bytes behind the end marker are no part of the stream."""
    from aeon_b200 import kernels as K
    rng = np.random.default_rng(72)
    blob = jpeg_bytes(np.clip(gradient_image(rng, 320, 448).astype(np.int16) + rng.integers(-20, 21, (320, 448, 3)), 0, 255).astype(np.uint8), 92)
    start = blob.index(b"\xff\xda") + 14
    info = K.jpeg_parse(blob)
    mcux, mcuy = info.blocks_w[0] // info.hs[0], info.blocks_h[0] // info.vs[0]
    size = len(blob) - 2 - start
    tail = bytes(rng.integers(0, 256, 3000, dtype=np.uint8))
    whole, upper = (0, 0, mcux, mcuy), (0, 0, mcux, 2)
    small = jpeg_bytes(gradient_image(rng, 8, 8), 90)
    for cut in sorted({0, 1, size // 2, size - 1, *(size * r // 8 // 16 * 16 + d for r in range(1, 8) for d in (-1, 0, 1))}):
        for k in (0, 3000):
            data = blob[:start + cut] + b"\xff\xd9" + tail[:k]
            got = K.jpeg_entropy_decode_device(ctx, [data, data] + [small] * (n - 2), [whole, upper] + [None] * (n - 2))
            assert got[0][3] == 1, (cut, k)
            if cut > size // 4:
                assert got[1][3] == 0, (cut, k)
                want = host_planes(blob, upper)[1]
                for c in range(info.ncomp):
                    assert np.array_equal(got[1][1][c].cpu().numpy(), want[c][:got[1][1][c].numel()]), (cut, k, c)
    check(ctx, [blob + tail])
