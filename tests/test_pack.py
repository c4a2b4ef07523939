"""How the Python provider hands records over: the address and size of every element, for every kind of buffer, on both sides of the number of
elements that are converted one by one."""
import ctypes as C

import numpy as np
import pytest

from aeon_b200.provider import Provider


def packed(records, k):
    p = object.__new__(Provider)
    p.input_count, p.handle = k, None
    ptrs, sizes, keep = p._pack(records)
    assert len(sizes) == len(records) * k
    return [C.string_at(ptrs[i], sizes[i]) if sizes[i] else b"" for i in range(len(records) * k)]


@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("n", [0, 1, 2, 3, 4, 7, 8, 9, 300])
def test_elements_of_every_kind(n, k):
    rng = np.random.default_rng(10 * n + k)
    blobs = [[bytes(rng.integers(0, 256, int(rng.integers(0, 40)), dtype=np.uint8)) for _ in range(k)] for _ in range(n)]
    want = [b for rec in blobs for b in rec]
    assert packed([tuple(rec) for rec in blobs], k) == want
    assert packed(blobs, k) == want
    for kind in (bytearray, memoryview, lambda b: np.frombuffer(b, np.uint8)):
        assert packed([[kind(b) if i % 3 == 0 else b for i, b in enumerate(rec)] for rec in blobs], k) == want


def test_records_of_another_length():
    for n in (1, 20):
        with pytest.raises(ValueError, match="record %d has 1 elements, the configuration needs 2" % (n - 1)):
            packed([(b"a", b"b")] * (n - 1) + [(b"a",)], 2)
