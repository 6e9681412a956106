"""A context's first host call: its scratch is allocated once, for the largest of its chunks, so the call takes about as
long as reserving that scratch and then calling.  (Scratch that grows with the chunks is freed and allocated twice more
between them, each time after waiting for the chunk before: 1.5 times as long for 256 MiB, whose chunks are 64, 128
and 64 MiB.)"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pinned(n, dtype=np.uint8):
    import torch
    return torch.zeros(n * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)


def test_scratch_is_allocated_once():
    import datagen as G
    import zero_cuda as Z
    block_log, n, chunk = 18, 256 << 20, 128 << 20
    nb = n >> block_log
    data, out = pinned(n), (pinned(nb), pinned(nb, np.uint32), pinned(nb, np.uint32), pinned(n), pinned(nb, np.uint64))
    raw, raw_lens = pinned(n), np.full(nb, 1 << block_log, np.uint32)
    data[:] = np.resize(G.lz_mix(32 << 20, block_log, 1), n)

    def both_ways(codec):
        m, lens, _, pay, offs = codec.compress_arrays(data, block_log, out=out)
        got, _, err = codec.decompress_arrays(pay, offs, lens, m, raw_lens, out=raw)
        assert not err.any()
        return got

    plain, reserved = [], []
    for _ in range(6):  # (the first warms the process up; the least of the others: allocation times vary)
        for times, reserve in ((plain, False), (reserved, True)):
            with Z.CudaCodec(level=5) as codec:
                t = time.perf_counter()
                if reserve:
                    codec._check(Z.lib().zc_reserve(codec._ctx, block_log, chunk >> block_log))
                got = both_ways(codec)
                times.append(time.perf_counter() - t)
    assert np.array_equal(got, data)
    assert min(plain[1:]) <= 1.15 * min(reserved[1:])
