"""The decoder's fill with all blocks in one launch, whose count picks the form: up to 888 blocks several warps share
one (16, 8 or 4 of them), beyond that a warp each in the set shape.  (A host call cuts its blocks into launches of its
own.)  Blocks of the full size among short ones, so that the rings of recent output wrap and far sources are read back
from the output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    import zero_cuda as Z
    with Z.CudaCodec(level=5) as c:
        yield c


def blocks(codec, block_log, seed):
    """Raw blocks and their records: text, near and far matches, short periods, runs, noise; whole, short and empty."""
    import datagen as G
    B = 1 << block_log
    r = np.random.default_rng(seed)
    periods = np.concatenate([np.resize(r.integers(0, 256, p, dtype=np.uint8), 1 + 40 * p) for p in range(1, 60)])
    far = np.concatenate([G.random_bytes(B // 2, seed), G.random_bytes(B // 2, seed)])  # (a copy half a block back)
    whole = [G.text_mix(B, seed), G.lz_mix(B, block_log, seed + 1), far, np.resize(periods, B), np.zeros(B, np.uint8), G.random_bytes(B, seed + 2)]
    raw = whole + [w[: int(n)] for w in whole for n in (0, 1, 131, 5000, B - 1)]
    lens = np.array([b.size for b in raw], np.uint32)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
    m, n, crc, pay, at = codec.compress_batch_arrays(np.concatenate(raw), offs, lens, block_log)
    return raw, [(int(m[b]), pay[int(at[b]): int(at[b]) + int(n[b])] if m[b] else raw[b]) for b in range(len(raw))], crc


def device_launch(raw, body, crc, nb, head):
    """The arguments of one call that decodes nb blocks, the given ones in turn, from output byte `head` on."""
    import torch
    pick = np.arange(nb) % len(raw)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, d)).cuda()  # noqa: E731
    size = np.array([body[k][1].size for k in range(len(raw))])
    at = np.concatenate([[0], np.cumsum(size)[:-1]])
    comp = t(np.concatenate([b for _, b in body] + [np.zeros(64, np.uint8)]), np.uint8)
    rlen = np.array([raw[k].size for k in pick])
    out_at = head + np.concatenate([[0], np.cumsum(rlen)[:-1]])
    out = torch.zeros(head + int(rlen.sum()) + 16, dtype=torch.uint8, device="cuda")
    want = torch.cat([torch.zeros(head, dtype=torch.uint8, device="cuda")] + [t(raw[k], np.uint8) for k in pick] +
                     [torch.zeros(16, dtype=torch.uint8, device="cuda")])
    args = (comp, t(at[pick], np.int64), t(size[pick], np.int32), t([body[k][0] for k in pick], np.uint8), t(rlen, np.int32), nb)
    return args, out, t(out_at, np.int64), want, t(crc[pick].view(np.int32), np.int32)


def check(codec, launch, block_log):
    import torch
    args, out, out_at, want, want_crc = launch
    nb = args[-1]
    out.zero_()
    crc, err = torch.zeros(nb, dtype=torch.int32, device="cuda"), torch.zeros(nb, dtype=torch.int32, device="cuda")
    codec.decompress_device(*args, block_log, out, out_at, crc, err)
    torch.cuda.synchronize()
    assert not err.any() and torch.equal(crc, want_crc) and torch.equal(out, want)


@pytest.mark.parametrize("nb", [296, 297, 592, 593, 888, 889])
@pytest.mark.parametrize("block_log", [16, 18])
def test_forms(codec, block_log, nb):
    check(codec, device_launch(*blocks(codec, block_log, 3), nb, 1 + nb % 7), block_log)


@pytest.mark.parametrize("block_log", [16, 18])
def test_shapes(codec, block_log):
    """Every shape that fits, 889 blocks."""
    default = codec.get_shape(block_log, 5)
    codec.prepare(block_log)
    launch = device_launch(*blocks(codec, block_log, 4), 889, 5)
    try:
        n = 0
        for ring_log in (11, 12, 13, 14, 15):
            for warps in (1, 2, 4, 8):
                for words in (1, 2, 4):
                    if warps * ((1 << ring_log) + 1536 * words) > 227 * 1024:
                        continue
                    codec.set_shape(block_log, 5, fill_ring_log=ring_log, fill_warps=warps, fill_words=words)
                    check(codec, launch, block_log)
                    n += 1
        assert n == 57
    finally:
        codec.set_shape(block_log, 5, **default)
        codec.prepare(18)
