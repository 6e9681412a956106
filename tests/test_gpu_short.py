"""Blocks far shorter than the launch's block size: their segments are the shortest there are (32 bytes), at counts of
segments on both sides of a warp's, a CTA's and the next segment size.  Payloads against the CPU codec's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [1, 5, 9])
@pytest.mark.parametrize("block_log", [16, 18, 20])
def test_bytes(block_log, level):
    import datagen as G
    import oracle as O
    import zero_cuda as Z
    sizes = [0, 1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 96, 300, 1023, 1024, 1025, 3000, 8191, 8192, 8193, 20000, 32767, 32768, 32769, 40000]
    text, noise = G.text_mix(sum(sizes), 5), np.random.default_rng(5).integers(0, 3, sum(sizes), dtype=np.uint8)
    for data in (text, noise, np.zeros(sum(sizes), np.uint8)):
        lens = np.array(sizes, np.uint32)
        offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
        with Z.CudaCodec(level=level) as codec:
            m, n, _, pay, at = codec.compress_batch_arrays(data, offs, lens, block_log)
        for b, size in enumerate(sizes):
            blk = data[int(offs[b]): int(offs[b]) + size].tobytes()
            want = O.Port.compress_block(blk, O.depth_for_level(level)) if size else b""
            assert m[b] == (len(want) < size), size
            if m[b]:
                assert pay[int(at[b]): int(at[b]) + int(n[b])].tobytes() == want, size
