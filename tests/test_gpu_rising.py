"""Data whose candidates get longer the farther back they are (runs of one value among few others, a short period with
faults): each beats the one before by a byte or two, so extending one candidate of a position at a time takes as many
turns as it has candidates.  Payloads against the CPU codec's, and the time of a call against what the encoder took when
it compared every position's candidates (B200, ms, the limits below)."""
import numpy as np
import pytest

from test_gpu_runs import milliseconds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    import zero_cuda as Z
    with Z.CudaCodec(level=5) as c:
        yield c


def rising(kind, n):
    r = np.random.default_rng(7)
    a = np.zeros(n, np.uint8)
    if kind == "faulty period":
        a = np.resize(r.integers(0, 256, 7, dtype=np.uint8), n)
    if kind == "two values":
        return np.resize(np.repeat(np.arange(n // 10, dtype=np.uint8) % 2, np.exp(r.uniform(0, 6, n // 10)).astype(int) + 1), n)
    at = r.integers(0, n, n // (100 if kind == "sparse" else 200))
    a[at] = r.integers(0, 256, at.size)
    return a


@pytest.mark.parametrize("kind,block_log,limit", [("sparse", 16, 12.5), ("faulty period", 16, 9.9), ("two values", 18, 19.5)])
def test_time(codec, kind, block_log, limit):
    assert milliseconds(codec, np.resize(rising(kind, 1 << 22), 1 << 26), block_log, 9) <= limit


@pytest.mark.parametrize("level", [1, 5, 9])
@pytest.mark.parametrize("block_log", [16, 18])
@pytest.mark.parametrize("kind", ["sparse", "faulty period", "two values"])
def test_bytes(codec, kind, block_log, level):
    import oracle as O
    data, B = rising(kind, (2 << block_log) + 4099), 1 << block_log
    m, lens, _, pay, offs = codec.compress_arrays(data, block_log, level=level)
    for b in range(len(m)):
        blk = data[b * B: (b + 1) * B].tobytes()
        want = O.Port.compress_block(blk, O.depth_for_level(level))
        assert m[b] == (len(want) < len(blk))
        if m[b]:
            assert pay[int(offs[b]): int(offs[b]) + int(lens[b])].tobytes() == want, b
