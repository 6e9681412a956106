"""Data that repeats itself (one value, a long period): the parse's chain then jumps whole segments and its walks never
meet.  Payloads against the CPU codec's, byte for byte, and the time of a call against what the encoder took when it
compared every position's candidates (B200, ms, the limits below): a parse that hands such a chain from segment
to segment, or extends its matches again for every walk and candidate, takes two to five times as long."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    import zero_cuda as Z
    with Z.CudaCodec(level=5) as c:
        yield c


def repeating(period, n):
    return np.resize(np.random.default_rng(1).integers(0, 256, period, dtype=np.uint8), n)


def milliseconds(codec, data, block_log, level):
    """The least of five device-resident compress calls."""
    import torch
    B, n = 1 << block_log, data.size
    nb = (n + B - 1) // B
    z = lambda k, t: torch.zeros(k, dtype=t, device="cuda")  # noqa: E731
    d_in = z(n + 64, torch.uint8)
    d_in[:n] = torch.from_numpy(data).cuda()
    offs = torch.arange(nb, device="cuda") * B
    lens = torch.clamp(n - offs, max=B).to(torch.int32)
    out = (z(nb, torch.uint8), z(nb, torch.int32), z(nb, torch.int32), z(n, torch.uint8), z(nb, torch.int64), z(1, torch.int64))
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        codec.compress_device(d_in, offs, lens, nb, block_log, *out, stream=torch.cuda.current_stream().cuda_stream, level=level)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return min(times[2:])


@pytest.mark.parametrize("period,n,block_log,level,limit", [
    (1, 1 << 18, 18, 5, 1.19), (1, 1 << 20, 20, 5, 3.61), (300, 1 << 18, 18, 5, 1.28), (300, 1 << 20, 20, 5, 3.74),
    (5000, 1 << 18, 18, 5, 1.82), (5000, 1 << 20, 20, 5, 6.06), (1, 1 << 26, 16, 1, 2.43), (5000, 1 << 28, 20, 9, 18.9)])
def test_time(codec, period, n, block_log, level, limit):
    assert milliseconds(codec, repeating(period, n), block_log, level) <= limit


@pytest.mark.parametrize("level", [1, 5, 9])
@pytest.mark.parametrize("block_log", [16, 18, 20])
@pytest.mark.parametrize("period", [1, 2, 33, 300, 511, 512, 5000, 70000])
def test_bytes(codec, period, block_log, level):
    """Segments of 256 to 1024 bytes, entered where the chain's last jump lands, and a last segment that is short."""
    import oracle as O
    for n in (1 << block_log, (1 << block_log) - 4097, 3 * 4096 + 5):
        data = repeating(period, n)
        data[n // 2] ^= 1  # (one byte that breaks the period)
        m, lens, _, pay, offs = codec.compress_arrays(data, block_log, level=level)
        want = O.Port.compress_block(data.tobytes(), O.depth_for_level(level))
        assert m[0] == (len(want) < n)
        if m[0]:
            assert pay[int(offs[0]): int(offs[0]) + int(lens[0])].tobytes() == want, n
