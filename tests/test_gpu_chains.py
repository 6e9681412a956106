"""Blocks whose output is one long chain of near copies (two symbols at random, coded with short chains): extracting
one must not take longer than a warp by itself takes, and such blocks come out right among all others, in every form of a
launch.  (Several warps that share such a block pass every copied word to one another: 1.5 times as long.)"""
import numpy as np
import pytest

from test_gpu_fill_launch import check, device_launch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    import zero_cuda as Z
    with Z.CudaCodec(level=1) as c:
        yield c


def records(codec, raw, block_log):
    lens = np.array([b.size for b in raw], np.uint32)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
    m, n, crc, pay, at = codec.compress_batch_arrays(np.concatenate(raw), offs, lens, block_log)
    return [(int(m[b]), pay[int(at[b]): int(at[b]) + int(n[b])] if m[b] else raw[b]) for b in range(len(raw))], crc


def chain(kind, n, r):
    if kind == "bits":
        return r.integers(0, 2, n, dtype=np.uint8)
    if kind == "counter":
        return (np.arange(n // 8 + 1, dtype=np.uint64) * 24 + 0x7F0000000000).view(np.uint8)[:n]
    a, b = np.array([0], np.uint8), np.array([0, 1], np.uint8)
    while b.size < n:
        a, b = b, np.concatenate([b, a])
    return b[:n].copy()


# ms of a call when every block had one warp (B200)
@pytest.mark.parametrize("kind,block_log,nb,limit", [
    ("bits", 16, 1, 0.92), ("bits", 18, 1, 3.58), ("bits", 18, 256, 4.13), ("bits", 20, 1, 14.1), ("bits", 20, 64, 15.8),
    ("counter", 16, 1, 2.53), ("counter", 18, 1, 9.99), ("counter", 18, 256, 10.6), ("counter", 20, 64, 41.7)])
def test_time(codec, kind, block_log, nb, limit):
    import torch
    raw = [chain(kind, 1 << block_log, np.random.default_rng(7))]
    launch = device_launch(raw, *records(codec, raw, block_log), nb, 0)
    check(codec, launch, block_log)
    args, out, out_at = launch[:3]
    crc, err = torch.zeros(nb, dtype=torch.int32, device="cuda"), torch.zeros(nb, dtype=torch.int32, device="cuda")
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        codec.decompress_device(*args, block_log, out, out_at, crc, err, stream=torch.cuda.current_stream().cuda_stream)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    assert min(times[2:]) <= limit


@pytest.mark.parametrize("nb", [1, 7, 296, 592, 888, 889])
@pytest.mark.parametrize("block_log", [16, 18])
def test_bytes(codec, block_log, nb):
    """From no literal to one byte in eight, one to six bits a symbol, whole and short; chains between text and noise."""
    import datagen as G
    r = np.random.default_rng(nb)
    raw = []
    for n in (1 << block_log, (1 << block_log) - 1234):
        for kind in ("bits", "fibonacci", "counter"):
            for piece in (9000, 20000, 70000):
                parts = [chain(kind, piece, r), G.text_mix(piece, nb), chain(kind, 2 * piece + 77, r), G.random_bytes(piece // 3, nb)]
                raw.append(np.resize(np.concatenate(parts), n))
    for n in (1 << block_log, (1 << block_log) - 77, 5000, 300, 33):
        for share in (0, 40, 18, 16, 14, 8):
            for symbols in (2, 4, 16, 64):
                a = r.integers(0, symbols, n, dtype=np.uint8)
                if share:
                    at = r.integers(0, n, n // share)
                    a[at] = r.integers(0, 256, at.size)
                raw.append(a)
    raw = [raw[i] for i in r.permutation(len(raw))]
    check(codec, device_launch(raw, *records(codec, raw, block_log), nb, 1 + nb % 5), block_log)
