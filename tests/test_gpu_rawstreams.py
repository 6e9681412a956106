"""Raw (not rANS-coded) streams in the decoder: lengths and alignments around the word copy, in every stream.  A block
whose bytes do not compress as symbols but that holds long matches keeps its literals raw; short blocks keep all
their streams raw."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [20, 33, 64, 65, 66, 67, 300, 1001, 5002, 30003, 65535])
@pytest.mark.parametrize("tokens", [1, 2, 5, 40])
def test_round_trip(size, tokens):
    import oracle as O
    import zero_cuda as Z
    r = np.random.default_rng(size * 100 + tokens)
    src = r.integers(0, 256, size, dtype=np.uint8)
    at = r.integers(0, max(size - 20, 1), tokens)
    data = np.concatenate([src] + [src[int(a): int(a) + int(n)] for a, n in zip(at, r.integers(10, 4000, tokens))])[:131072]
    with Z.CudaCodec() as codec:
        m, n, crcs, pay, offs = codec.compress_arrays(data, 17)
        want = O.Port.compress_block(data.tobytes(), O.depth_for_level(5))
        if len(want) < data.size:
            assert m[0] == 1 and pay[: int(n[0])].tobytes() == want
        # three copies of the payload at different alignments
        body = pay[: int(n[0])] if m[0] else data
        parts = [body, r.integers(0, 256, 1, dtype=np.uint8), body, r.integers(0, 256, 2, dtype=np.uint8), body]
        starts = np.cumsum([0] + [p.size for p in parts])[[0, 2, 4]].astype(np.uint64)
        raw, got, err = codec.decompress_arrays(np.concatenate(parts), starts, np.full(3, body.size, np.uint32),
                                                np.full(3, m[0], np.uint8), np.full(3, data.size, np.uint32))
    assert not err.any() and (got == crcs[0]).all() and np.array_equal(raw, np.tile(data, 3))
