"""Block CRCs on the GPU against zlib's: lengths around the words, the 4 KiB batches and the warps' chunks of the
bit-sliced form, at every alignment, for launches of few blocks (8 warps each) and of many (4 warps)."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LENGTHS = [*range(0, 40), 127, 128, 129, 4093, 4094, 4095, 4096, 4097, 4098, 4099, 4100, 8191, 8192, 8193, 16383, 16384, 16385,
           32767, 32768, 32769, 65535, 65536, 65537, 262143, 262144, 262147, 1 << 20]


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_lengths_and_alignments(shift, many):
    import zero_cuda as Z
    r = np.random.default_rng(shift)
    data = r.integers(0, 256, (1 << 20) + 8, dtype=np.uint8)
    # stored blocks, decoded back to back: a block's output starts where the one before it ends
    lens = [shift] + [n for k in LENGTHS for n in (k, (4 - k) % 4 + (shift and 4))] + ([3] * 1100 if many else [])
    parts = [data[:n] if k % 2 else data[8:8 + n] for k, n in enumerate(lens)]
    n = np.array(lens, np.uint32)
    at = np.concatenate([[0], np.cumsum(n, dtype=np.uint64)[:-1]]).astype(np.uint64)
    with Z.CudaCodec() as codec:
        raw, crcs, err = codec.decompress_arrays(np.concatenate(parts), at, n, np.zeros(n.size, np.uint8), n)
    assert not err.any()
    assert [int(c) for c in crcs] == [zlib.crc32(p.tobytes()) for p in parts]
