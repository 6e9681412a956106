"""The parse's finishing of matches (warp_finish) and its split into segments and walks, at the sizes where they can
go wrong: match lengths on both sides of the 16- and 32-byte compares, the 64-byte extension steps and the longest
match, equal lengths at several distances, chains longer than the depth, and launches that take each segment
count.  Every comparison is of whole payloads, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    import zero_cuda as Z
    with Z.CudaCodec(level=5) as c:
        yield c


def lengths(rng):
    """Copies of one source cut to every length where a compare ends, each followed by fresh bytes."""
    src = rng.integers(0, 256, 9000, dtype=np.uint8)
    parts = []
    for n in (3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 48, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 4095, 4096, 4097, 8192):
        parts += [src[:n], rng.integers(0, 256, 7, dtype=np.uint8)]
    return np.concatenate([src] + parts * 2)


def rows(rng):
    """Lines that share long prefixes and differ late: many long candidates, equal lengths at several distances."""
    base = rng.integers(97, 123, 500, dtype=np.uint8)
    out = []
    for _ in range(260):
        b = base[: int(rng.integers(5, 500))].copy()
        b[int(rng.integers(3, b.size)):][:1] ^= 1
        out.append(b)
    return np.concatenate(out)


DATA = {
    "lengths": lengths,
    "rows": rows,
    "runs": lambda r: np.repeat(r.integers(0, 3, 60, dtype=np.uint8), r.integers(1, 5000, 60)),
    "period_33": lambda r: np.resize(r.integers(0, 256, 33, dtype=np.uint8), 70001),
    "two_symbols": lambda r: r.integers(0, 2, 65537, dtype=np.uint8),
    "one_value": lambda r: np.full(66000, 7, np.uint8),
    "tiny": lambda r: np.resize(r.integers(0, 256, 5, dtype=np.uint8), 11),
}


@pytest.mark.parametrize("level", [1, 5, 9])
@pytest.mark.parametrize("name", sorted(DATA))
def test_finished_matches(codec, name, level):
    import oracle as O
    data = DATA[name](np.random.default_rng(11))
    for block_log in (16, 18):
        B = 1 << block_log
        methods, lens, _, pay, offs = codec.compress_arrays(data, block_log, level=level)
        for b in range(len(methods)):
            blk = data[b * B:(b + 1) * B].tobytes()
            want = O.Port.compress_block(blk, O.depth_for_level(level))
            got = pay[int(offs[b]): int(offs[b]) + int(lens[b])].tobytes() if methods[b] else blk
            assert got == (want if len(want) < len(blk) else blk), f"block {b} of {name} at 2^{block_log}"


@pytest.mark.parametrize("level", [1, 5])
def test_segment_counts(codec, level):
    """One device launch of 1408 blocks of 256 KiB (512-byte segments) against launches of 16 blocks (256-byte segments):
    the blocks repeat, so their payloads must."""
    import datagen as G
    import torch
    block_log, nb, reps = 18, 128, 11
    B = 1 << block_log
    tile = G.lz_mix(nb << block_log, block_log, 3)
    small = []
    for k in range(0, nb, 16):
        m, n, _, p, o = codec.compress_arrays(tile[k << block_log:(k + 16) << block_log], block_log, level=level)
        small += [p[int(a): int(a) + int(b)].tobytes() for a, b in zip(o, n)]
        assert m.all()
    total = nb * reps
    z = lambda k, t: torch.zeros(k, dtype=t, device="cuda")  # noqa: E731
    d_in = z(total * B + 64, torch.uint8)
    d_in[: total * B] = torch.from_numpy(tile).cuda().repeat(reps)
    offs, lens = torch.arange(total, device="cuda") * B, torch.full((total,), B, dtype=torch.int32, device="cuda")
    m, n, crc, out, at, end = (z(total, torch.uint8), z(total, torch.int32), z(total, torch.int32), z(total * B, torch.uint8),
                               z(total, torch.int64), z(1, torch.int64))
    codec.compress_device(d_in, offs, lens, total, block_log, m, n, crc, out, at, end, level=level)
    m, n, at, out = m.cpu().numpy(), n.cpu().numpy(), at.cpu().numpy(), out[: int(end.item())].cpu().numpy()
    assert m.all()
    for b in range(total):
        assert out[int(at[b]): int(at[b]) + int(n[b])].tobytes() == small[b % nb], f"block {b}"


def test_walks_a_warp(codec):
    """Launches whose warps take 2, 4, 8, 16 and 32 walks each give the same blocks the same payloads, which are the
    CPU codec's."""
    import datagen as G
    import oracle as O
    block_log, B = 16, 1 << 16
    data = np.concatenate([G.text_mix(256 * B, 1), G.lz_mix(256 * B, block_log, 2)])[::-1].copy()
    want = {}
    for nb in (1, 32, 64, 128, 256, 512):  # (256 walks a block; 4736 warps at most, or 2 walks a warp)
        m, n, _, p, o = codec.compress_arrays(data[: nb * B], block_log, level=5)
        for b in range(nb):
            got = p[int(o[b]): int(o[b]) + int(n[b])].tobytes() if m[b] else None
            if b not in want:
                want[b] = got
                if b in (0, 31, 300):
                    blk = data[b * B:(b + 1) * B].tobytes()
                    ref = O.Port.compress_block(blk, O.depth_for_level(5))
                    assert got == (ref if len(ref) < len(blk) else None)
            assert got == want[b], (nb, b)
