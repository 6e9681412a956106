"""The hash sort and the chain marking at the edges of their warps and tiles: blocks at odd offsets whose last tile or
round holds one entry, all but one or exactly all, with digits all equal, of two values, nearly all equal and all
different.  A wrong order of the sort changes the matches, so whole payloads are compared, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a block of n bytes sorts n - 3 entries: 32 a round, 256 a warp, 2048 a chain tile, 4096 a sort tile
SIZES = [4, 5, 34, 35, 36, 258, 259, 260, 2050, 2051, 2052, 4098, 4099, 4100, 8195, 65535, 65536]


def nearly_one(r, n):
    a = np.full(n, 9, np.uint8)
    a[r.integers(0, n, n // 300 + 1)] = r.integers(0, 256, n // 300 + 1)
    return a


DATA = {
    "one_value": lambda r, n: np.full(n, 5, np.uint8),
    "two_values": lambda r, n: (np.arange(n) & 1).astype(np.uint8),
    "nearly_one_value": nearly_one,
    "two_symbols": lambda r, n: r.integers(0, 2, n, dtype=np.uint8),
    "bytes": lambda r, n: r.integers(0, 256, n, dtype=np.uint8),
    "repeated_bytes": lambda r, n: np.resize(r.integers(0, 256, n // 3 + 1, dtype=np.uint8), n),
}


@pytest.mark.parametrize("level", [1, 9])
@pytest.mark.parametrize("name", sorted(DATA))
def test_sort_edges(name, level):
    import oracle as O
    import torch
    import zero_cuda as Z
    rng = np.random.default_rng(5)
    blocks = [DATA[name](rng, n) for n in SIZES]
    at, offs = 3, []
    for b in blocks:  # (odd offsets: every alignment within a word)
        offs.append(at)
        at += b.size + 1
    raw = np.zeros(at + 64, np.uint8)
    for o, b in zip(offs, blocks):
        raw[o: o + b.size] = b
    nb = len(blocks)
    z = lambda k, t: torch.zeros(k, dtype=t, device="cuda")  # noqa: E731
    m, n, crc, out, to, end = z(nb, torch.uint8), z(nb, torch.int32), z(nb, torch.int32), z(at, torch.uint8), z(nb, torch.int64), z(1, torch.int64)
    with Z.CudaCodec(level=level) as codec:
        codec.compress_device(torch.from_numpy(raw).cuda(), torch.tensor(offs, dtype=torch.int64, device="cuda"),
                              torch.tensor(SIZES, dtype=torch.int32, device="cuda"), nb, 16, m, n, crc, out, to, end, level=level)
        m, n, to, out = m.cpu().numpy(), n.cpu().numpy(), to.cpu().numpy(), out.cpu().numpy()
    for k, b in enumerate(blocks):
        want = O.Port.compress_block(b.tobytes(), O.depth_for_level(level))
        got = out[int(to[k]): int(to[k]) + int(n[k])].tobytes() if m[k] else b.tobytes()
        assert got == (want if len(want) < b.size else b.tobytes()), f"{name}, {b.size} bytes"
