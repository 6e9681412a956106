"""The stream writer's tiles (8, 16 or 32 warps a block by the launch's block count): groups that end at 255 tokens or
span tiles, literal runs copied by a lane, a warp or the CTA, offset bits carried from tile to tile.  Whole payloads,
byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def far_groups(r):
    """Tokens whose sources all lie in the block's first part: groups run to their 255-token limit."""
    head = r.integers(0, 256, 20000, dtype=np.uint8)
    at = r.integers(0, 19900, 4000)
    return np.concatenate([head] + [head[int(p): int(p) + int(k)] for p, k in zip(at, r.integers(5, 14, 4000))])


def long_literals(r):
    """Literal runs of 14 .. 40000 bytes between copies."""
    src = r.integers(0, 256, 400, dtype=np.uint8)
    parts = [src]
    for n in (14, 15, 16, 31, 32, 33, 2047, 2048, 2049, 15000, 40000, 5):
        parts += [r.integers(0, 256, n, dtype=np.uint8), src[:200]]
    return np.concatenate(parts)


def near_offsets(r):
    """Short copies at small offsets: groups of a token or two, recent offsets everywhere."""
    out = list(r.integers(0, 256, 64))
    while len(out) < 30000:
        d, n = int(r.integers(1, 60)), int(r.integers(4, 30))
        out += [out[len(out) - d + k % d] for k in range(n)] + list(r.integers(0, 256, int(r.integers(0, 3))))
    return np.array(out, np.uint8)


DATA = {"far_groups": far_groups, "long_literals": long_literals, "near_offsets": near_offsets}


@pytest.mark.parametrize("copies", [1, 149, 445])
@pytest.mark.parametrize("name", sorted(DATA))
def test_payloads(name, copies):
    import oracle as O
    import zero_cuda as Z
    data = DATA[name](np.random.default_rng(21))
    want = O.Port.compress_block(data.tobytes(), O.depth_for_level(5))
    lens = np.full(copies, data.size, np.uint32)
    with Z.CudaCodec(level=5) as codec:
        at = np.arange(copies, dtype=np.uint64) * np.uint64(data.size)
        m, n, _, pay, offs = codec.compress_batch_arrays(np.tile(data, copies), at, lens, 17)
    for b in range(copies):
        assert m[b] == 1 and pay[int(offs[b]): int(offs[b]) + int(n[b])].tobytes() == want, f"copy {b}"
