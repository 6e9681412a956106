"""The decoder fill's launch forms: one warp a block, and 4, 8 or 16 warps sharing one, on both sides of the block
counts where the form changes, with uneven blocks (empty ones, ones shorter than a line), outputs at any alignment,
and matches that repeat their own bytes at every short period."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    import zero_cuda as Z
    with Z.CudaCodec(level=5) as c:
        yield c


def material(n, seed):
    """Text, LZ-structured bytes, runs of periods 1 .. 40 between short literals, and incompressible stretches."""
    import datagen as G
    r = np.random.default_rng(seed)
    parts = [G.text_mix(n // 4, seed), G.lz_mix(n // 4, 16, seed + 1)]
    size = 0
    while size < n // 4:
        p = int(r.integers(1, 41))
        parts.append(np.resize(r.integers(0, 256, p, dtype=np.uint8), int(r.integers(p + 1, 300))))
        size += parts[-1].size
    parts.append(G.random_bytes(n // 4, seed + 2))
    return np.concatenate(parts)


def round_trip(codec, data, offs, lens, block_log):
    methods, clens, crcs, pay, poffs = codec.compress_batch_arrays(data, offs, lens, block_log)
    bodies = [pay[int(poffs[b]): int(poffs[b]) + int(clens[b])] if methods[b] else data[int(offs[b]): int(offs[b]) + int(lens[b])]
              for b in range(len(lens))]
    n = np.array([x.size for x in bodies], np.uint64)
    at = np.concatenate([[0], np.cumsum(n)[:-1]]).astype(np.uint64)
    raw, got, err = codec.decompress_arrays(np.concatenate(bodies + [np.zeros(1, np.uint8)]), at, n, methods, lens)
    assert not err.any() and np.array_equal(got, crcs)
    want = np.concatenate([data[int(o): int(o) + int(k)] for o, k in zip(offs, lens)] + [np.zeros(0, np.uint8)])
    assert np.array_equal(raw, want)


@pytest.mark.parametrize("nb", [1, 2, 296, 297, 592, 593, 888, 889, 1480, 1481])
def test_block_counts(codec, nb):
    data = material(1 << 20, nb)
    r = np.random.default_rng(nb)
    lens = r.integers(0, 6000, nb).astype(np.uint32)
    lens[:: 7] = r.integers(0, 140, lens[:: 7].size)
    offs = r.integers(0, data.size - 6000, nb).astype(np.uint64)
    round_trip(codec, data, offs, lens, 16)


@pytest.mark.parametrize("words", [1, 2, 4])
@pytest.mark.parametrize("ring_log,warps", [(11, 8), (13, 4), (15, 1)])
def test_shapes_of_one_warp_a_block(codec, ring_log, warps, words):
    """More blocks than the form with several warps a block takes, in each shape of the other one."""
    default = codec.get_shape(16, 5)
    codec.set_shape(16, 5, fill_ring_log=ring_log, fill_warps=warps, fill_words=words)
    try:
        data = material(1 << 20, 7)
        r = np.random.default_rng(8)
        lens = r.integers(0, 6000, 900).astype(np.uint32)
        lens[:: 90] = 65536
        offs = r.integers(0, data.size - 65536, 900).astype(np.uint64)
        round_trip(codec, data, offs, lens, 16)
    finally:
        codec.set_shape(16, 5, **default)


@pytest.mark.parametrize("block_log", [16, 18, 20])
def test_whole_blocks(codec, block_log):
    """Blocks of the full size behind one of odd length, so every output line is unaligned; far sources leave the
    ring of recent output."""
    B = 1 << block_log
    data = np.concatenate([material(3 * B, 5), material(B, 6)])
    lens = np.array([77, B, B, B - 1, 1], np.uint32)
    round_trip(codec, data, np.cumsum(np.concatenate([[0], lens[:-1]])).astype(np.uint64), lens, block_log)


@pytest.mark.parametrize("copies", [0, 1, 3, 4, 5, 2047, 2048, 2049, 4097, 9000])
def test_token_counts(codec, copies):
    """About as many tokens as copies: on both sides of the token scan's four a thread and 2048 a tile, with groups of up
    to 255 tokens and offsets that repeat (recent-offset symbols naming tokens of this tile and earlier ones)."""
    r = np.random.default_rng(copies + 1)
    src = r.integers(0, 256, 3000, dtype=np.uint8)
    out = [src]
    for k in range(copies):
        at = int(r.integers(0, 2900)) if k % 3 else 40 * (k % 7)
        out += [src[at: at + int(r.integers(5, 25))], r.integers(0, 256, int(r.integers(0, 2)), dtype=np.uint8)]
    data = np.concatenate(out)
    assert data.size < 1 << 18
    round_trip(codec, data, np.zeros(1, np.uint64), np.array([data.size], np.uint32), 18)
