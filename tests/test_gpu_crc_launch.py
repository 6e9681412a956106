"""Block CRCs of one launch against zlib's: every length around the words, the 4 KiB batches and the warps' chunks of
the bit-sliced form, each at every alignment of the output, in a launch of few blocks (8 warps each) and in one of
more than 1024 (4 warps each).  A device call, so that the blocks are one launch and lie where they are put."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LENGTHS = [*range(0, 40), 127, 128, 129, 4093, 4094, 4095, 4096, 4097, 4098, 4099, 4100, 8191, 8192, 8193, 16383, 16384, 16385,
           32767, 32768, 32769, 65535, 65536, 65537, 131071, 131072, 131073, 262143, 262144, 262147, (1 << 20) - 1, 1 << 20]


@pytest.mark.parametrize("few", [True, False])
def test_every_length_at_every_alignment(few):
    import torch
    import zero_cuda as Z
    lens, shifts = np.array([(n, s) for n in LENGTHS for s in range(4)] + [(3, 1)] * (0 if few else 1025 - 4 * len(LENGTHS))).T
    assert lens.size <= 1024 if few else lens.size == 1025
    slots = (lens + 3 + 15) // 16 * 16  # each output in a 16-byte aligned slot of its own, `shift` bytes into it
    out_at = np.concatenate([[0], np.cumsum(slots)[:-1]]) + shifts
    in_at = np.concatenate([[0], np.cumsum(lens)[:-1]])
    data = np.random.default_rng(5).integers(0, 256, int(lens.sum()) + 64, dtype=np.uint8)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, d)).cuda()  # noqa: E731
    nb = lens.size
    out, err, crc = torch.zeros(int(slots.sum()) + 64, dtype=torch.uint8, device="cuda"), t(np.zeros(nb), np.int32), t(np.zeros(nb), np.int32)
    assert out.data_ptr() % 16 == 0
    with Z.CudaCodec() as codec:
        codec.decompress_device(t(data, np.uint8), t(in_at, np.int64), t(lens, np.int32), t(np.zeros(nb), np.uint8),
                                t(lens, np.int32), nb, 20, out, t(out_at, np.int64), crc, err)
        torch.cuda.synchronize()
    assert not err.any()
    want = [zlib.crc32(data[a: a + n].tobytes()) for a, n in zip(in_at, lens)]
    assert crc.cpu().numpy().view(np.uint32).tolist() == want
    got = out.cpu().numpy()
    assert all(np.array_equal(got[o: o + n], data[a: a + n]) for o, a, n in zip(out_at, in_at, lens))
