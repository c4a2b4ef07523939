"""The bookkeeping of the block-parallel entropy kernels, as a model on the CPU (tests/entropy_model.py): what the kernels
count must be what the stream holds, every piece of the storing pass must start at the right block in a known state."""
import os

import cv2
import numpy as np
import pytest

from tests.entropy_model import SPREAD_EXTRA, simulate, simulate_spread
from tests.synth import gradient_image


def test_stream_whose_last_segment_ends_just_before_a_checkpoint(golden_dir):
    blob = open(os.path.join(golden_dir, "entropy_stream_507_segments.jpg"), "rb").read()
    r = simulate(blob)
    assert (r["segment"], r["segments"]) == (176, 507) and r["counted"] == r["total_blocks"] == 6144 and not r["problems"]
    # with a checkpoint allowed past the segment's end, the last segment takes an older run's count: three blocks missing
    old = simulate(blob, checkpoint_past_end=True)
    assert old["counted"] == 6141 and ("segment count", 506, 8, 11) in old["problems"]


@pytest.mark.parametrize("seed", range(3))
def test_random_streams_in_every_sampling_mode_and_block_size(seed):
    rng = np.random.default_rng(100 + seed)
    modes = [cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422, None]
    for k in range(12):
        h, w = int(rng.integers(40, 520)), int(rng.integers(40, 520))
        noise = int(rng.integers(1, 40))
        img = np.clip(gradient_image(rng, h, w).astype(np.int16) + rng.integers(-noise, noise + 1, (h, w, 3)), 0, 255).astype(np.uint8)
        quality = int(rng.choice([60, 75, 90, 95, 100]))
        mode = modes[k % 4]
        if mode is None:
            ok, enc = cv2.imencode(".jpg", cv2.cvtColor(img, cv2.COLOR_BGR2GRAY), [cv2.IMWRITE_JPEG_QUALITY, quality])
        else:
            ok, enc = cv2.imencode(".jpg", img, [cv2.IMWRITE_JPEG_QUALITY, quality, cv2.IMWRITE_JPEG_SAMPLING_FACTOR, mode])
        assert ok
        r = simulate(enc.tobytes(), threads=int(rng.choice([512, 256, 128])))
        assert r["counted"] == r["total_blocks"] and not r["problems"], (seed, k, r)


@pytest.mark.parametrize("quality", [75, 95])
def test_a_thread_for_every_piece_of_the_storing_pass(golden_dir, quality):
    """1024 threads, as for streams that have an SM to themselves: segments are lengthened so that the pieces fill whole rounds."""
    rng = np.random.default_rng(quality)
    blobs = [open(os.path.join(golden_dir, "entropy_stream_507_segments.jpg"), "rb").read()] if quality == 95 else []
    for h, w in ((300, 420), (500, 375), (90, 60)):
        blobs.append(cv2.imencode(".jpg", gradient_image(rng, h, w), [cv2.IMWRITE_JPEG_QUALITY, quality])[1].tobytes())
    for blob in blobs:
        r = simulate(blob, threads=1024)
        assert r["counted"] == r["total_blocks"] and not r["problems"], r
        pieces = 4 * r["segments"]
        assert pieces <= 1024 or r["segment"] == 160 or pieces % 1024 == 0 or pieces % 1024 > 256, r


def spread_streams(rng):
    """Streams of one to a thousand segments, of two to six places in an MCU, with much, little and nothing to fall into step on."""
    modes = [cv2.IMWRITE_JPEG_SAMPLING_FACTOR_420, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_444, cv2.IMWRITE_JPEG_SAMPLING_FACTOR_422,
             cv2.IMWRITE_JPEG_SAMPLING_FACTOR_411, None]
    for k, (h, w) in enumerate([(300, 400), (8, 8), (33, 47), (430, 470), (120, 160)] * 4):
        img = gradient_image(rng, h, w, int(rng.integers(2, 40)))
        if k // 5 == 1:
            img[h // 3:] = 128
        elif k // 5 == 2:
            img[:] = (np.arange(w) // 8 % 2 * 255)[None, :, None]
        elif k // 5 == 3:
            img = rng.integers(0, 256, img.shape, dtype=np.uint8)
        mode = modes[(k + k // 5) % 5]
        blob = cv2.imencode(".jpg", img if mode else img[..., 0], [cv2.IMWRITE_JPEG_QUALITY, int(rng.choice([60, 90, 97]))] +
                            ([cv2.IMWRITE_JPEG_SAMPLING_FACTOR, mode] if mode else []))[1].tobytes()
        yield k, blob


@pytest.mark.parametrize("streams", [1, 16, 66])
def test_streams_spread_over_clusters(streams):
    for k, blob in spread_streams(np.random.default_rng(200 + streams)):
        if len(blob) < 110_000:
            r = simulate_spread(blob, streams)
            assert not r["problems"], (k, r)


@pytest.mark.parametrize("room", [0, 1, 30])
def test_more_states_than_there_is_room_for(room):
    """A run that notes no state makes the piece in front of it longer, and nothing else."""
    rng = np.random.default_rng(205)
    for img in (gradient_image(rng, 300, 400), rng.integers(0, 256, (100, 150, 3), dtype=np.uint8)):
        r = simulate_spread(cv2.imencode(".jpg", img, [cv2.IMWRITE_JPEG_QUALITY, 90])[1].tobytes(), extra_room=room)
        assert max(r["noted"]) > room and not r["problems"], r
    noise = cv2.imencode(".jpg", rng.integers(0, 256, (160, 200, 3), dtype=np.uint8), [cv2.IMWRITE_JPEG_QUALITY, 100])[1].tobytes()
    r = simulate_spread(noise)
    assert max(r["noted"]) > SPREAD_EXTRA and not r["problems"], r
